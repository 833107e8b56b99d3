"""`lb_compile`, the backend's own C++ lowering of a module that has been through the passes (the counterpart of
`Cuda::lower(module, device)`, lumen/graph_compiler/device.rs:88-112): on the CPU it parses the module, generates and
compiles every fused kernel and builds the plan - steps, places, workspace size - or rejects the module with a message
naming the primitive it has no kernel for (lumen/codegen/devices/cuda/mod.rs:140-189 does the same)."""

import ctypes
import json

import pytest

from lumen_b200 import _lib, autograd, prims, tracer
from lumen_b200 import functional as F
from lumen_b200.attention_pass import match_attention
from lumen_b200.fusion_pass import fuse
from lumen_b200.plan import _bind, lower_native
from lumen_b200.simplify import clean


def plan_of(graph, **kwargs):
    handle = lower_native(graph, **kwargs)
    lib = _bind()
    steps = [(s["kind"], s["label"]) for s in json.loads(lib.lb_plan_steps_json(handle).decode())]
    workspace = lib.lb_plan_workspace_bytes(handle)
    lib.lb_plan_destroy(handle)
    return steps, workspace


def chain(x, g, b):
    y = F.relu(x * g + b)
    return y, F.sum(y * y, 1)


CHAIN_TYPES = (("float32", (64, 256)), ("float32", (256,)), ("float32", (256,)))


def test_fused_chain_is_one_step_written_into_the_outputs():
    steps, workspace = plan_of(fuse(clean(tracer.trace(chain, *CHAIN_TYPES))))
    assert steps == [("fusion", "row")] and workspace == 0  # both results are graph outputs: nothing lives in the workspace


def test_products_become_gemm_steps_with_their_relu():
    def mlp(x, w1, w2):
        return F.matmul(F.relu(F.matmul(x, w1, "float32", "bfloat16")), w2, "float32", "bfloat16")

    g = fuse(clean(tracer.trace(mlp, ("bfloat16", (256, 128)), ("bfloat16", (128, 512)), ("bfloat16", (512, 64)))))
    steps, workspace = plan_of(g)
    assert [k for k, _ in steps] == ["gemm", "gemm"]
    assert workspace == 256 * 512 * 2  # the hidden activation; the result is produced in the output


def test_intermediates_share_the_workspace_by_live_range():
    """A chain of four products: each intermediate is dead once the next product has read it, so the workspace holds two
    of the three at a time - the size the optimising lowering gives the same module."""
    from lumen_b200.compiler import compile_graph

    def chain4(x, a, b, c, d):
        for w in (a, b, c, d):
            x = F.matmul(x, w, "float32", "bfloat16")
        return x

    types = [("bfloat16", (512, 256))] + [("bfloat16", (256, 256))] * 4
    g = tracer.trace(chain4, *types)
    _, workspace = plan_of(fuse(clean(g)))
    assert workspace == 2 * 512 * 256 * 2 == compile_graph(g).workspace_bytes


def test_attention_forward_and_backward_with_and_without_determinism():
    def program(q, k, v, do):
        def loss(q_, k_, v_):
            return F.sum(F.flash_attention(q_, k_, v_, causal=True)[0].float() * do.float())

        value, grads = autograd.value_and_grad(loss, (0, 1, 2))(q, k, v)
        return (value, *grads)

    g = fuse(match_attention(clean(tracer.trace(program, *[("bfloat16", (2, 128, 4, 64))] * 4))))
    steps, pair = plan_of(g)
    assert [k for k, _ in steps].count("attn_fwd") == 1 and [k for k, _ in steps].count("attn_bwd") == 1
    _, atomic = plan_of(g, deterministic=False)
    assert atomic >= pair  # the float32 dQ accumulator of the single-kernel backward lives (only) at the backward step


def test_attention_written_from_prims_is_lowered_after_the_matcher():
    g = match_attention(clean(tracer.trace(lambda q, k, v: F.attention_forward_prims(q, k, v, 0.125, True)[0], *[("bfloat16", (2, 128, 4, 64))] * 3)))
    steps, _ = plan_of(fuse(g))
    assert steps == [("attn_fwd", "flash_attention")]


def test_a_module_that_skipped_the_fusion_pass_is_rejected_by_primitive():
    with pytest.raises(_lib.LumenError, match="primitive `broadcast_in_dim` outside a fusion"):
        lower_native(tracer.trace(chain, *CHAIN_TYPES))
    with pytest.raises(_lib.LumenError):
        _lib.check(_bind().lb_compile(b"not a module", -1, None, None))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_the_whole_training_step_is_lowered(dtype):
    """Forward, backward and SGD update of the transformer step as the passes leave it: generated kernels, products with
    their relu / residual-add / relu-backward epilogues, attention forward and backward on sliced views of the packed
    projection, the embedding's scatter-add, the attention gradients produced inside the concatenation that packs them."""
    from lumen_b200 import transformer as T

    cfg = T.Config(vocab=64, d_model=128, heads=2, hidden=256, layers=1, seq=128, dtype=dtype)
    g, _, _ = T.trace_train_step(cfg, 2)
    steps, workspace = plan_of(fuse(match_attention(clean(g))))
    kinds = [k for k, _ in steps]
    assert kinds.count("gemm") == 15 and kinds.count("attn_fwd") == 1 and kinds.count("attn_bwd") == 1 and kinds.count("scatter_add") == 1
    assert kinds.count("copy") == 0 and workspace > 0  # the attention gradients are produced inside their concatenation
    assert kinds.count("multi") == 1 and [label for k, label in steps if k == "multi"] == ["sgd_update_x13"]  # the 13 updates as one launch


def test_the_data_parallel_step_gets_its_collective_steps():
    """The 2-rank training step: all-reduced gradients side by side in the arena, cut into buckets, each with an
    `all_reduce` step after its last gradient and a `wait` before its first reader - as many collectives, in the same
    places, and the same workspace as the Python lowering gives the same module."""
    from lumen_b200 import transformer as T
    from lumen_b200.compiler import compile_graph

    cfg = T.Config(vocab=64, d_model=128, heads=2, hidden=256, layers=1, seq=128, dtype="bfloat16")
    g, _, donate = T.trace_train_step(cfg, 2, world=2)
    handle = lower_native(fuse(match_attention(clean(g))), True, donate, 100_000)
    lib = _bind()
    kinds = [s["kind"] for s in json.loads(lib.lb_plan_steps_json(handle).decode())]
    python = compile_graph(g, donate, bucket_bytes=100_000)
    python_kinds = [line.split()[1] for line in python.text.splitlines() if line.startswith("s ")]

    def places(ks):  # (kind, number of kernel steps before it) of every collective step
        out, n = [], 0
        for k in ks:
            if k in ("all_reduce", "wait"):
                out.append((k, n))
            elif k not in ("copy", "fill", "transpose"):
                n += 1
        return out

    assert lib.lb_plan_num_collectives(handle) == len(python.buckets) == 3
    assert places(kinds) == places(python_kinds)
    assert lib.lb_plan_workspace_bytes(handle) == python.workspace_bytes
    lib.lb_plan_destroy(handle)


def test_a_concatenation_of_other_values_is_copied_into_place():
    """Operands that are not attention gradients (here two products) are copied into the concatenation by pitched
    copies."""
    def program(x, a, b):
        return F.cat([F.matmul(x, a, "float32", "bfloat16"), F.matmul(x, b, "float32", "bfloat16")], 1)

    g = fuse(clean(tracer.trace(program, ("bfloat16", (256, 128)), ("bfloat16", (128, 64)), ("bfloat16", (128, 192)))))
    steps, _ = plan_of(g)
    assert [k for k, _ in steps] == ["gemm", "gemm", "copy", "copy"]


def test_both_lowerings_make_the_same_steps_of_a_differentiated_program():
    """A SwiGLU MLP step differentiated by autograd returns its weight gradients as transposed views of the products
    that made them: `lb_compile` writes them into the outputs with the transpose kernel, names every product by its
    epilogue and needs the same workspace as the Python lowering of the same program; the plan keeps its own text."""
    from lumen_b200.compiler import compile_graph

    def step(x, y, gate, up, down):
        def loss(g, u, d):
            h = F.swiglu(F.matmul(x, g, "float32", "float32"), F.matmul(x, u, "float32", "float32"))
            r = F.matmul(h, d, "float32", "float32") - y
            return F.mean(r * r)

        value, grads = autograd.value_and_grad(loss, (0, 1, 2))(gate, up, down)
        return (value, *grads)

    types = [("float32", s) for s in ((256, 64), (256, 32), (64, 128), (64, 128), (128, 32))]
    g = tracer.trace(step, *types)
    python = compile_graph(g)
    handle = lower_native(fuse(match_attention(clean(g))))
    lib = _bind()
    labels = [s["label"] for s in json.loads(lib.lb_plan_steps_json(handle).decode())]
    assert labels == python.labels and labels.count("output_transpose") == 3
    assert lib.lb_plan_workspace_bytes(handle) == python.workspace_bytes
    text = lib.lb_plan_text(handle).decode()
    assert text.count("\ns transpose output_transpose ") == 3 and text.rstrip().endswith("end")
    lib.lb_plan_destroy(handle)


def test_both_lowerings_place_the_same_collectives_in_random_data_parallel_steps():
    """Random configurations (1 - 3 layers, float32 and bfloat16, SGD and AdamW), world sizes 2 - 8 and bucket sizes from
    one gradient per bucket to everything in one: both lowerings queue as many collectives, at the same places among the
    kernel steps, make the same steps and need the same workspace."""
    import numpy as np

    from lumen_b200 import transformer as T
    from lumen_b200.compiler import compile_graph

    lib = _bind()

    def places(ks):
        out, n = [], 0
        for k in ks:
            if k in ("all_reduce", "wait"):
                out.append((k, n))
            elif k not in ("copy", "fill", "transpose"):
                n += 1
        return out

    for seed in range(8):
        rng = np.random.default_rng(seed + 300)
        dtype = ["float32", "bfloat16"][int(rng.integers(2))]
        d = int(rng.choice([64, 128]))
        cfg = T.Config(vocab=int(rng.choice([64, 200])), d_model=d, heads=d // 64 if dtype == "bfloat16" else int(rng.choice([2, 4])),
                       hidden=int(rng.choice([128, 256])), layers=int(rng.integers(1, 4)), seq=int(rng.choice([64, 128])), dtype=dtype,
                       optimizer=["sgd", "adamw"][int(rng.integers(2))])
        world = int(rng.choice([2, 4, 8]))
        bucket = int(rng.choice([1, 50_000, 400_000, 1 << 30]))
        g, _, donate = T.trace_train_step(cfg, 2, world=world)
        handle = lower_native(fuse(match_attention(clean(g))), True, donate, bucket)
        steps = json.loads(lib.lb_plan_steps_json(handle).decode())
        python = compile_graph(g, donate, bucket_bytes=bucket)
        python_kinds = [line.split()[1] for line in python.text.splitlines() if line.startswith("s ")]
        what = (seed, cfg, world, bucket)
        assert lib.lb_plan_num_collectives(handle) == len(python.buckets) >= 1, what
        assert places([s["kind"] for s in steps]) == places(python_kinds), what
        assert [s["label"] for s in steps] == python.labels, what
        assert lib.lb_plan_workspace_bytes(handle) == python.workspace_bytes, what
        lib.lb_plan_destroy(handle)


@pytest.mark.parametrize("dtype, k, split", [("float32", 8192, False), ("bfloat16", 8192, True), ("bfloat16", 8191, False)])
def test_products_on_cuda_cores_take_no_split_scratch(dtype, k, split):
    """K is cut by the tensor-core kernels alone: float32 products and rows of 16 bits that are not 16-byte aligned take no memory for
    partial tiles and count as one launch, in both lowerings."""
    from lumen_b200.compiler import compile_graph

    g = tracer.trace(lambda x, w: F.matmul(x, w, "float32", dtype), (dtype, (1024, k)), (dtype, (k, 1024)))
    lib, native, python = _bind(), lower_native(fuse(clean(g))), ctypes.c_void_p()
    compiled = compile_graph(g)
    _lib.check(lib.lb_plan_create(compiled.text.encode(), ctypes.byref(python)))
    assert lib.lb_plan_workspace_bytes(native) == compiled.workspace_bytes and (compiled.workspace_bytes > 0) == split
    for handle in (native, python):
        assert lib.lb_plan_kernel_launches(handle) == 1 + split
        lib.lb_plan_destroy(handle)


@pytest.mark.parametrize("m, n, k, copied", [(2048, 4096, 64, True), (2040, 4096, 64, False), (2048, 4096, 60, False), (2048, 4088, 64, False), (1024, 4096, 32, False), (4096, 4096, 32, True)])
def test_weights_of_much_larger_products_are_transposed(m, n, k, copied):
    """A K-major copy of a weight with long rows: in both lowerings, and never one that the tensor cores do not read."""
    from lumen_b200.compiler import compile_graph

    g = tracer.trace(lambda x, w: F.matmul(x, w, "float32", "bfloat16"), ("bfloat16", (m, k)), ("bfloat16", (k, n)))
    steps, _ = plan_of(fuse(clean(g)))
    assert [label for _, label in steps] == compile_graph(g).labels == ["weight_transpose"] * copied + ["dot_general"]


@pytest.mark.parametrize("m, n, k, across, copied", [
    (24576, 4096, 256, False, True), (24575, 4096, 256, False, False), (24576, 4096, 248, False, False), (131072, 8192, 128, False, False), (12288, 4096, 256, True, False),
    (12288, 4096, 512, True, True), (12280, 4096, 512, True, False), (12288, 4096, 512, False, False), (24576, 8192, 4096, False, True), (24576, 8200, 4096, False, False)])
def test_weights_are_transposed_where_it_pays(m, n, k, across, copied):
    """By M and K, and by which way the other operand lies."""
    from lumen_b200.compiler import compile_graph

    g = tracer.trace(lambda x, w: F.matmul(prims.transpose(x, (1, 0)) if across else x, w, "float32", "bfloat16"),
                     ("bfloat16", (k, m) if across else (m, k)), ("bfloat16", (k, n)))
    steps, _ = plan_of(fuse(clean(g)))
    assert [label for _, label in steps] == compile_graph(g).labels == ["weight_transpose"] * copied + ["dot_general"]


def test_a_plan_text_with_too_little_scratch_is_refused():
    """Partial sums take what the library's kernels need now, whatever wrote the text."""
    from lumen_b200.compiler import compile_graph

    g = tracer.trace(lambda x: F.sum(x, 0), ("float32", (4096, 512)))
    lines = compile_graph(g).text.splitlines(keepends=True)
    (at,) = [i for i, line in enumerate(lines) if line.startswith("t ") and " uint8 " in line]
    lib, plan = _bind(), ctypes.c_void_p()
    _lib.check(lib.lb_plan_create("".join(lines).encode(), ctypes.byref(plan)))
    lib.lb_plan_destroy(plan)
    words = lines[at].split()
    words[6] = str(int(words[6]) - 4)
    lines[at] = " ".join(words) + "\n"
    with pytest.raises(_lib.LumenError, match="scratch"):
        _lib.check(lib.lb_plan_create("".join(lines).encode(), ctypes.byref(plan)))


@pytest.mark.parametrize("shapes, chained, launches", [
    ([(64, 64, 64), (128, 32, 512)], False, 1), ([(64, 64, 64)] * 2, True, 2), ([(64, 64, 64)] * 5, False, 2), ([(64, 0, 64), (64, 64, 0)], False, 1),
    ([(1088, 1152, 64), (64, 64, 64), (64, 64, 64)], False, 2)])  # 17 x 18 tiles of 64 x 64: two for each of 148 SMs, a launch of their own
def test_float32_products_beside_one_another_share_a_launch(shapes, chained, launches):
    """Those of which none reads another's result, four to a launch."""
    def program(*x):
        y = []
        for i in range(len(shapes)):
            y.append(F.matmul(y[-1] if chained and y else x[2 * i], x[2 * i + 1], "float32", "float32"))
        return tuple(y)

    g = tracer.trace(program, *[("float32", s) for m, n, k in shapes for s in ((m, k), (k, n))])
    lib, native = _bind(), lower_native(fuse(clean(g)))
    assert lib.lb_plan_kernel_launches(native) == launches
    lib.lb_plan_destroy(native)


@pytest.mark.parametrize("m, n, k, split", [
    (1024, 1024, 8192, True), (768, 768, 8192, True),  # 128 blocks of K for two ranges of narrow tiles: the line
    (768, 768, 8128, False), (512, 512, 4096, False),  # shorter ranges
    (384, 3072, 6144, False), (384, 1536, 8192, False),  # more units than pairs of SMs: 384 rows are two row tiles
    (128, 9216, 4096, False), (16, 8192, 4096, False), (128, 4096, 12288, False),  # the one-CTA kernel
    (816, 512, 17376, True), (128, 9216, 12288, True), (16, 4864, 16384, True),  # 130 blocks an SM and 2.25 times the large tiles'
    (1664, 256, 14296, True), (896, 496, 11008, False),  # 112 and 86 blocks, the result covered by whole tiles
    (384, 1536, 16384, False), (384, 3072, 16384, False),  # 128 blocks; 256, twice the large tiles'
    (128, 8192, 17000, True),  # longer ranges than the narrow tiles take
])
def test_long_products_that_narrow_tiles_fit_are_cut_on_large_tiles_only_where_that_is_faster(m, n, k, split):
    lib = _bind()
    assert (lib.lb_gemm_step_scratch_bytes(m, n, k) > 0) == split
    if split:
        assert lib.lb_gemm_step_scratch_bytes(m, n, k) == lib.lb_gemm_scratch_bytes(m, n, k, 1)


def test_products_into_donated_inputs_are_counted_where_they_lie():
    """A product written into an input that its neighbour reads has a launch of its own, as in a run; without donation they share one."""
    def program(x, y, z):
        return F.matmul(z, y, "float32", "float32"), F.matmul(x, y, "float32", "float32")

    g = fuse(clean(tracer.trace(program, *[("float32", (64, 64))] * 3)))
    lib = _bind()
    for donate, launches in (({1: 2}, 2), (None, 1)):
        native = lower_native(g, donate=donate)
        assert lib.lb_plan_kernel_launches(native) == launches
        lib.lb_plan_destroy(native)
