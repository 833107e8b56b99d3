"""Programs traced as bare prims, grouped by the fusion pass, lowered to a plan and run on a B200 against the oracle
evaluating the unfused graph."""

import numpy as np
import pytest
import torch

from lumen_b200 import functional as F
from lumen_b200 import prims, tracer
from lumen_b200.compiler import compile_graph
from lumen_b200.plan import Plan
from lumen_b200.runtime import TORCH_DTYPES, device_status
from tests.helpers import bf16, run_oracle, to_numpy, to_torch

pytestmark = pytest.mark.gpu


def run_plan(g, inputs, cuda):
    compiled = compile_graph(g)
    outs = [torch.empty(g.types[v].shape, dtype=TORCH_DTYPES[g.types[v].dtype], device=cuda) for v in g.outputs]
    Plan(compiled, cuda).run([to_torch(x, cuda) for x in inputs], outs)
    device_status()
    return compiled, [to_numpy(o) for o in outs]


def test_softmax_program_from_bare_prims(cuda):
    def program(x, w):
        p = F.softmax(x, -1)
        return p, F.sum(p * w, -1) * 0.5

    g = tracer.trace(program, ("float32", (512, 1024)), ("float32", (512, 1024)))
    rng = np.random.default_rng(0)
    inputs = [rng.standard_normal((512, 1024), dtype=np.float32), rng.standard_normal((512, 1024), dtype=np.float32)]
    compiled, got = run_plan(g, inputs, cuda)
    assert len(compiled.labels) <= 2
    want = run_oracle(g, inputs)
    np.testing.assert_allclose(got[0], want[0], rtol=1e-5, atol=1e-7)
    np.testing.assert_allclose(got[1], want[1], rtol=1e-5, atol=1e-6)


def test_mlp_block_from_bare_prims_uses_gemm_epilogues(cuda):
    dims = (((1,), (0,)), ((), ()))

    def program(x, w1, w2, r):
        h = F.relu(prims.dot_general(x, w1, dims, "float32", "bfloat16"))
        return prims.dot_general(h, w2, dims, "float32", "bfloat16") + r

    g = tracer.trace(program, ("bfloat16", (384, 256)), ("bfloat16", (256, 512)), ("bfloat16", (512, 256)), ("bfloat16", (384, 256)))
    rng = np.random.default_rng(1)
    inputs = [bf16(rng.standard_normal((384, 256)) / 16), bf16(rng.standard_normal((256, 512)) / 16),
              bf16(rng.standard_normal((512, 256)) / 16), bf16(rng.standard_normal((384, 256)))]
    compiled, got = run_plan(g, inputs, cuda)
    assert compiled.labels == ["dot_general_relu", "dot_general_add"]
    want = run_oracle(g, inputs)[0].astype(np.float32)
    np.testing.assert_allclose(got[0].astype(np.float32), want, rtol=2**-6, atol=2**-6 * np.abs(want).max())


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("m, n, k", [
    (1, 8, 8), (200, 520, 64), (200, 4096, 1024),  # narrow tiles: one, ragged ones, K cut over a cluster
    (2100, 2056, 40), (2304, 2048, 64),  # pairs of large tiles, with and without ragged ones
    (128, 40008, 64), (70, 50002, 40), (2100, 2047, 40), (300, 513, 24),  # one row block; rows of the result that are not 16-byte aligned
    (1024, 1024, 8192), (1024, 1021, 8192),  # K cut into ranges whose sums another kernel adds
    (30, 33, 17), (300, 513, 25)])  # rows that the tensor cores' copies do not take
def test_relu_beside_its_product_and_what_a_maximum_passes_back_on_the_gpu(cuda, m, n, k, dtype):
    """Each kernel's epilogue bit for bit against the product of the same sizes by itself and the two primitives after it: where the
    operand is zero (rows of zeros), infinite or not a number too."""
    from lumen_b200 import autograd
    from lumen_b200.runtime import gemm, gemm_scratch_bytes

    torch_dtype, dims = TORCH_DTYPES[dtype], (((1,), (1,)), ((), ()))

    def program(x, w, v, dy):
        h = prims.dot_general(x, w, dims, "float32", dtype)
        a, pull = autograd.vjp(F.relu, h)
        y = F.matmul(a, v, "float32", dtype)
        back = prims.dot_general(dy, w, dims, "float32", dtype)
        return y, a, pull(back)[0], h * 1.0

    g = tracer.trace(program, (dtype, (m, k)), (dtype, (n, k)), (dtype, (n, 8)), (dtype, (m, k)))
    compiled = compile_graph(g)
    assert "dot_general_relu_beside" in compiled.labels and "dot_general_max_backward" in compiled.labels
    gen = torch.Generator(device=cuda).manual_seed(n)
    x, w, v, dy = (torch.randn(s, generator=gen, device=cuda).to(torch_dtype) for s in ((m, k), (n, k), (n, 8), (m, k)))
    x[::5] = 0
    if m > 7:
        x[3, 0], x[6, 1], dy[10 % m, 0] = float("inf"), float("nan"), -float("inf")
    outs = [torch.empty(s, dtype=torch_dtype, device=cuda) for s in ((m, 8), (m, n), (m, n), (m, n))]
    Plan(compiled).run([x, w, v, dy], outs)

    def product(a):
        scratch = torch.empty(gemm_scratch_bytes(m, n, k), dtype=torch.uint8, device=cuda)
        return gemm(a, w.t(), torch.empty(m, n, dtype=torch_dtype, device=cuda), scratch=scratch if scratch.numel() else None)

    h, back = product(x), product(dy)
    factor = torch.where(h > 0, 1.0, torch.where(h == 0, 0.5, 0.0)).to(torch_dtype)
    for got, want in ((outs[3], h), (outs[1], torch.clamp(h, min=0)), (outs[2], back * factor)):  # clamp keeps a NaN
        assert torch.equal(torch.isnan(got), torch.isnan(want))
        assert torch.equal(got.nan_to_num(0.0, None, None), want.nan_to_num(0.0, None, None))
    device_status()


def test_compile_surface_runs_a_traced_function(cuda, tmp_path):
    """`lumen_b200.compile(fn, device="cuda")`: traced on the first call per signature, results owned by the compiled
    function and overwritten by the next call, a second signature compiles its own plan."""
    import lumen_b200

    def fn(x, w, scale):
        return F.relu(x * w) * scale, F.sum(x, -1)

    f = lumen_b200.compile(fn, device="cuda", use_graphs=True)
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.standard_normal((256, 512), dtype=np.float32)).to(cuda)
    w = torch.from_numpy(rng.standard_normal((256, 512), dtype=np.float32)).to(cuda)
    for _ in range(3):  # plain run, recording, replay
        y, s = f(x, w, 0.5)
        device_status()
        torch.testing.assert_close(y, torch.relu(x * w) * 0.5, rtol=1e-6, atol=0)
        torch.testing.assert_close(s, x.sum(-1), rtol=1e-5, atol=1e-5)
    assert "reduce_sum" in str(f) and len(f.steps()) <= 2
    first = y
    y2, _ = f(x * 2, w, 0.5)
    assert y2.data_ptr() == first.data_ptr()  # the compiled function owns its results
    small, _ = f(x[:64], w[:64], 0.5)
    assert small.shape == (64, 512) and len(f.signatures) == 2
    written = f.dump_code(str(tmp_path))
    kernels = [p for p in written if p.endswith(".cu")]
    assert len(kernels) == len(f.steps()) and all("fused_kernel" in open(p).read() for p in kernels)


def test_compiled_function_with_attention_and_projection(cuda):
    """`F.flash_attention` inside a compiled function: the q/k/v projection GEMM, the attention fusion reading strided
    views of it in place, and an output projection with a residual add in its epilogue."""
    import lumen_b200

    b, s, n, h = 2, 256, 2, 64
    d = n * h
    dims = (((1,), (0,)), ((), ()))

    def block(x, wqkv, wo):
        qkv = prims.dot_general(x, wqkv, dims, "float32", "bfloat16")
        q, k, v = (prims.slice(qkv, (0, i * d), (b * s, (i + 1) * d)).reshape(b, s, n, h) for i in range(3))
        o, _ = F.flash_attention(q, k, v, causal=True)
        return prims.dot_general(o.reshape(b * s, d), wo, dims, "float32", "bfloat16") + x

    rng = np.random.default_rng(7)
    x, wqkv, wo = (bf16(rng.standard_normal(shape) / np.sqrt(shape[0] if len(shape) > 1 else 1))
                   for shape in ((b * s, d), (d, 3 * d), (d, d)))
    f = lumen_b200.compile(block)
    got = f(to_torch(x, cuda), to_torch(wqkv, cuda), to_torch(wo, cuda))
    device_status()
    assert [st["label"] for st in f.steps()] == ["dot_general", "flash_attention", "dot_general_add"]
    g = tracer.trace(block, ("bfloat16", x.shape), ("bfloat16", wqkv.shape), ("bfloat16", wo.shape))
    want = run_oracle(g, [x, wqkv, wo])[0].astype(np.float32)
    np.testing.assert_allclose(to_numpy(got).astype(np.float32), want, rtol=2e-2, atol=2e-2 * np.abs(want).max())


def test_normalisations_and_the_adamw_step_beside_the_training_path(cuda):
    """`rms_norm`, `log_softmax`, a clamp chain and the AdamW step (tests/test_front_ops.py pins them to float64 on the
    oracle) through the fusion pass and the generated kernels: one kernel each, rtol 1e-5 against the oracle
    (elementwise values of the AdamW step bit-exact: one rounding per primitive, no reduction)."""
    from tests.test_front_ops import adamw_graph, adamw_inputs, clamp_program, log_softmax_program, rms_program

    rng = np.random.default_rng(9)
    x = (2 * rng.standard_normal((300, 1000))).astype(np.float32)
    w = rng.uniform(0.5, 1.5, 1000).astype(np.float32)
    for program, inputs in ((rms_program, [x, w]), (log_softmax_program, [x]), (clamp_program, [x])):
        g = tracer.trace(program, *[("float32", a.shape) for a in inputs])
        compiled, got = run_plan(g, inputs, cuda)
        assert len(compiled.labels) == 1, (program.__name__, compiled.labels)
        np.testing.assert_allclose(got[0], run_oracle(g, inputs)[0], rtol=1e-5, atol=1e-6)
    for dtype in ("float32", "bfloat16"):
        g = adamw_graph(dtype, (129, 520), 7, lr=1e-2, weight_decay=0.1)
        inputs = adamw_inputs(dtype, (129, 520), seed=3)
        compiled, got = run_plan(g, inputs, cuda)
        assert compiled.labels == ["adamw_update"]
        want = run_oracle(g, inputs)
        for a, b in zip(got, want):
            # division and square root are correctly rounded on both sides
            np.testing.assert_array_equal(a.astype(np.float32), b.astype(np.float32))


def test_compile_takes_dlpack_arrays_in_place(cuda):
    """Arguments that are not torch tensors but export DLPack are imported without a copy (same device pointer)."""
    import lumen_b200

    class Foreign:  # stands for another framework's array
        def __init__(self, t):
            self.t = t

        def __dlpack__(self, **kw):
            return self.t.__dlpack__(**kw)

        def __dlpack_device__(self):
            return self.t.__dlpack_device__()

    f = lumen_b200.compile(lambda x, y: F.relu(x - y), device="cuda")
    x = torch.randn((64, 128), device=cuda)
    y = torch.randn((64, 128), device=cuda)
    got = f(Foreign(x), Foreign(y))
    torch.testing.assert_close(got, torch.relu(x - y), rtol=0, atol=0)
    assert f.latest.keep[0][0].data_ptr() == x.data_ptr()


def test_a_recorded_call_is_not_replayed_for_other_memory(cuda):
    """With `use_graphs` a call that returns to other argument memory runs on that memory, from its first call there on."""
    import lumen_b200

    f = lumen_b200.compile(lambda x: x + x, use_graphs=True)
    a, b = (torch.full((64, 64), v, device=cuda) for v in (1.0, 10.0))
    for x in (a, a, a, b, b, b, b, a, b, a, a, a, a):
        assert torch.equal(f(x), x + x)
