"""The native call path (lumen_b200._host) on stand-ins for tensors: what it reads, what it refuses and which calls it leaves to the
general path. No GPU: entries that get as far as the library raise its error."""

import pytest
import torch

from lumen_b200 import _lib
from lumen_b200.runtime import desc


class Array:
    """An array of another framework: the attributes the package reads, `shape` and `stride()` as any sequence."""

    def __init__(self, shape, dtype="float32", strides=None, sequence=tuple, cuda=True):
        self.shape, self.dtype, self.is_cuda, self._sequence = sequence(shape), dtype, cuda, sequence
        dense = [1] * len(shape)
        for d in range(len(shape) - 2, -1, -1):
            dense[d] = dense[d + 1] * shape[d + 1]
        self._strides = dense if strides is None else strides

    def data_ptr(self):
        return 1 << 20

    def stride(self):
        return self._sequence(self._strides)


def gemm(a, b, out):
    _lib.host().gemm(a, b, out, None, 0, 0, 0, 0, 0)


@pytest.mark.parametrize("sequence", [tuple, list, torch.Size])
def test_shapes_and_strides_are_any_sequence(sequence):
    a, b, out = Array((4, 8), sequence=sequence), Array((8, 6), sequence=sequence), Array((4, 5), sequence=sequence)
    with pytest.raises(_lib.LumenError, match=r"\[1,4,8\] x \[1,8,6\] -> \[1,4,5\]"):  # read right: the shapes do not match
        gemm(a, b, out)
    d = desc(a)
    assert (d.rank, list(d.shape[:2]), list(d.stride[:2])) == (2, [4, 8], [8, 1])


def test_what_is_not_a_tensor_on_the_gpu_is_refused():
    a, b, out = Array((4, 8)), Array((8, 6)), Array((4, 6))
    with pytest.raises(ValueError, match="expected a CUDA tensor"):
        gemm(Array((4, 8), cuda=False), b, out)
    with pytest.raises(TypeError, match="at most 8 integers"):
        gemm(Array((1,) * 9), b, out)
    with pytest.raises(TypeError, match="as many strides as dimensions"):
        gemm(Array((4, 8), strides=[1]), b, out)
    with pytest.raises(TypeError, match="no lumen dtype"):
        gemm(Array((4, 8), dtype=complex), b, out)
    with pytest.raises(AttributeError):
        gemm(3.0, b, out)
    with pytest.raises(TypeError, match="expected 9 arguments"):
        _lib.host().gemm(a, b)


class Torch(Array):
    """A torch tensor's further attributes."""

    def __init__(self, shape, dtype="float32", cuda=True, contiguous=True, device=0):
        super().__init__(shape, dtype, cuda=cuda)
        self._contiguous, self._device = contiguous, device

    def is_contiguous(self):
        return self._contiguous

    def get_device(self):
        return self._device


class Parameter(Torch):
    pass


def ran():
    """What a call that finds a signature comes to: the stand-in plan is null."""
    return pytest.raises(_lib.LumenError, match="null plan")


def table(*signatures, device=-1):
    t = _lib.host().CallTable()
    for args in signatures:
        t.add(args, tuple(isinstance(a, Torch) for a in args), device, 0, 0, (0,), "signature", "returned")
    return t


def test_a_call_runs_the_signature_that_its_arguments_match():
    t = table((Array((4, 8)), Array((8,))), (Array((4, 9)), Array((9,))))
    for n in (8, 9):
        with ran():
            t.call((Array((4, n)), Array((n,))), 1, -1)
        assert t.latest == "signature"
    with ran():
        table(()).call((), 1, -1)  # a function without arguments


@pytest.mark.parametrize("args", [
    (),
    (Array((4, 8)),),
    (Array((4, 8)), Array((8,)), Array((8,))),
    (Array((4, 8)), Array((9,))),
    (Array((8, 4)), Array((8,))),
    (Array((4, 8, 1)), Array((8,))),
    (Array((4, 8), "bfloat16"), Array((8,))),
    (Array((4, 8)), Torch((8,))),  # another class
    (Array((4, 8)), 0.5),
    (Array((4, 8)), None),
    (Array((4, 8)),) * 65,
])
def test_calls_that_match_no_signature_are_left_to_the_general_path(args):
    assert table((Array((4, 8)), Array((8,)))).call(args, 1, -1) is None


def test_torch_tensors_have_to_be_readable_in_place():
    t = table((Torch((4, 8)),))
    assert t.call((Torch((4, 8), cuda=False),), 1, -1) is None
    assert t.call((Torch((4, 8), contiguous=False),), 1, -1) is None
    assert t.call((Parameter((4, 8)),), 1, -1) is None
    t.add((Parameter((4, 8)),), (True,), -1, 0, 0, (0,), "signature", "returned")
    for x in (Torch((4, 8)), Parameter((4, 8))):
        with ran():
            t.call((x,), 1, -1)


def test_a_signature_belongs_to_the_device_of_its_memory():
    """After a first call on GPU 0, tensors of the same shape on GPU 1, with that one current, are another signature."""
    t = table((Torch((4, 8), device=0),), device=0)
    assert t.call((Torch((4, 8), device=1),), 1, 1) is None
    assert t.call((Torch((4, 8), device=1),), 1, 0) is None
    assert t.call((Torch((4, 8), device=0),), 1, 1) is None
    with ran():
        t.call((Torch((4, 8), device=0),), 1, 0)
    t.add((Torch((4, 8)),), (True,), 1, 0, 0, (0,), "signature of GPU 1", "returned")
    with ran():
        t.call((Torch((4, 8), device=1),), 1, 1)
    assert t.latest == "signature of GPU 1"


def test_a_call_costs_the_same_among_many_signatures():
    """Found by a hash: the time of a call does not grow with the number of signatures (a search one by one takes 0.1 us each:
    here over 400 us a call against one or two)."""
    import time

    few, many = table((Array((4, 1)),)), table(*((Array((4, n)),) for n in range(1, 4097)))

    def cost(t, x):
        best = 1e9
        for _ in range(5):
            t0 = time.perf_counter()
            for _ in range(200):
                assert t.call((x,), 1, -1) is None
            best = min(best, (time.perf_counter() - t0) / 200)
        return best

    missing = Array((5, 4096))
    assert cost(many, missing) < 10 * cost(few, missing)


def test_errors_of_an_argument_are_raised():
    class Broken(Array):
        @property
        def shape(self):
            raise RuntimeError("no shape")

        @shape.setter
        def shape(self, value):
            pass

    t = _lib.host().CallTable()
    with pytest.raises(RuntimeError, match="no shape"):
        t.add((Broken((4,)),), (False,), -1, 0, 0, (0,), "signature", "returned")
    with pytest.raises(TypeError):
        t.add([Array((4,))], (False,), -1, 0, 0, (0,), "signature", "returned")
    with pytest.raises(TypeError):
        t.call([Array((4,))], 1, -1)


def test_threads_add_and_call_at_once():
    import threading

    t = table((Array((1, 1)),))
    failures = []

    def work(k):
        try:
            for n in range(200):
                x = Array((k + 2, n + 1))
                t.add((x,), (False,), -1, 0, 0, (0,), "signature", "returned")
                with ran():
                    t.call((Array((k + 2, n + 1)),), 1, -1)
                with ran():
                    t.call((Array((1, 1)),), 1, -1)
        except BaseException as e:
            failures.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not failures


def test_calls_of_a_fusion_share_no_partial_sums(monkeypatch):
    """A call that another thread or stream makes before the first one's second kernel is queued gets memory of its own."""
    from lumen_b200 import prims, runtime, tracer

    f = runtime.Fusion(tracer.trace(lambda x: prims.reduce_sum(x, (0,), "float32"), ("float32", (512, 100))))
    assert f.scratch_bytes > 0
    x, seen = torch.zeros(512, 100), []

    def launch(self, descs, scratch=None, stream=None):
        seen.append(scratch)
        if len(seen) == 1:
            f(x)

    monkeypatch.setattr(runtime, "require_cuda", lambda: None)
    monkeypatch.setattr(runtime, "desc", lambda t: t)
    monkeypatch.setattr(runtime.Fusion, "launch_raw", launch)
    f(x)
    assert len(seen) == 2 and seen[0] != seen[1]


def test_temporaries_of_a_call_come_from_its_stream(monkeypatch):
    """The backward's delta and dQ sums and the scatter-add's sums are dropped when the call returns, with its kernels in flight: they
    are memory of the stream that the call names."""
    from lumen_b200 import runtime

    asked = []

    class Nothing:
        def __getattr__(self, name):
            return lambda *a: 0

    def workspace(like, shape, dtype, stream):
        asked.append((tuple(shape), dtype, stream))
        return torch.empty(shape, dtype=runtime.TORCH_DTYPES[dtype])

    monkeypatch.setattr(runtime, "require_cuda", lambda: None)
    monkeypatch.setattr(runtime, "_workspace", workspace)
    monkeypatch.setattr(runtime._lib, "host", Nothing)
    q = torch.zeros(2, 8, 4, 64, dtype=torch.bfloat16)
    lse = torch.zeros(2, 4, 8)
    runtime.attention_backward(q, q, q, q, q, lse, stream=7)
    assert asked == [((2, 4, 8), "float32", 7)]
    runtime.attention_backward(q, q, q, q, q, lse, stream=7, deterministic=False)
    assert asked[1:] == [((2, 4, 8), "float32", 7), ((2, 8, 4, 64), "float32", 7)]
    monkeypatch.setattr(runtime, "desc", lambda t: runtime._lib.strided(0, "float32", t.shape, t.stride()))

    class Answer:
        def __init__(self, value):
            self.value = value

        def __call__(self, *a):
            return self.value

    class Library:
        lb_scatter_add_scratch_bytes, lb_scatter_add_rows = Answer(640), Answer(0)

    monkeypatch.setattr(runtime._lib, "lib", Library)
    runtime.scatter_add_rows(torch.zeros(4, 40), torch.zeros(3, dtype=torch.int64), torch.zeros(3, 40), stream=9)
    assert asked[3:] == [((640,), "uint8", 9)]


def test_results_come_from_a_region_of_the_current_device(monkeypatch):
    from lumen_b200 import device, runtime

    on = [0]

    class Region:
        def __init__(self, nbytes):
            self.device = on[0]

        def empty(self, shape, dtype):
            return self

    monkeypatch.setattr(device, "Region", Region)
    monkeypatch.setattr(device, "current_device", lambda: on[0])
    for name in ("_regions", "_workspaces"):
        monkeypatch.setattr(runtime, name, type(getattr(runtime, name, {}))(), raising=False)
    for on[0] in (0, 1, 0):
        assert runtime._empty_like_input(Array((4,)), (4,), "float32").device == on[0]
        assert runtime._workspace(Array((4,)), (4,), "float32", 5).device == on[0]
