"""Where the attention backward's scratch for dS comes from: regions that are kept once they are large enough, and memory that is there."""

import pytest
import torch

from lumen_b200 import _lib, device, runtime

DS = 37 << 20


class Block:
    def __init__(self, region, at, nbytes):
        self.region, self.at, self.nbytes = region, at, nbytes

    def data_ptr(self):
        return self.at + 1

    def __del__(self):
        self.region.live.remove((self.at, self.nbytes))


class Region:
    """First fit in blocks of 256 bytes, as lb_region_alloc."""

    made, refuses = [], None

    def __init__(self, capacity):
        self.capacity, self.live, self.error = capacity, [], "region out of memory: it is full"
        if Region.refuses and Region.refuses(capacity):
            self.capacity, self.error = 0, "region: reserving failed: out of memory"
        Region.made.append(self)

    def empty(self, shape, dtype):
        nbytes = device.ITEMSIZE[dtype]
        for n in shape:
            nbytes *= n
        nbytes, at = max(256, (nbytes + 255) // 256 * 256), 0
        for start, size in sorted(self.live):
            if start - at >= nbytes:
                break
            at = start + size
        if at + nbytes > self.capacity:
            raise _lib.LumenError(3, self.error)
        self.live.append((at, nbytes))
        return Block(self, at, nbytes)

    def stats(self):
        return {"live_bytes": sum(size for _, size in self.live)}


class Native:
    """A tensor of no framework."""

    is_cuda, dtype = True, "bfloat16"

    def __init__(self, shape):
        self.shape = shape


class Host:
    nbytes, calls = DS, []

    def attention_bwd_scratch_bytes(self, *a):
        return Host.nbytes

    def attention_bwd(self, *a):
        Host.calls.append(a[14:16])


@pytest.fixture
def native(monkeypatch):
    Region.made, Region.refuses, Host.nbytes, Host.calls = [], None, DS, []
    monkeypatch.setattr(device, "Region", Region)
    monkeypatch.setattr(device, "current_device", lambda: 0)
    monkeypatch.setattr(runtime, "require_cuda", lambda: None)
    monkeypatch.setattr(runtime._lib, "host", Host)
    for name in ("_regions", "_workspaces"):
        monkeypatch.setattr(runtime, name, type(getattr(runtime, name))())
    q = Native((2, 1024, 16, 128))

    def backward(**options):
        runtime.attention_backward(q, q, q, q, q, None, stream=5, **options)
        return runtime._workspaces[(0, 5)]

    return backward


def test_a_region_that_holds_all_of_a_call_is_kept(native):
    """delta and then dS from one region, which is too small for both at first."""
    native()
    region, made = native(), len(Region.made)
    assert native() is region and native() is region and len(Region.made) == made
    assert all(pointer and nbytes == DS for pointer, nbytes in Host.calls) and not region.live


def test_regions_that_cannot_be_had(native):
    """Without memory for dS it is computed twice, and delta's region stays."""
    Region.refuses = lambda capacity: 32 << 20 < capacity < 256 << 20  # (results are there)
    region = native()
    assert native() is region and Host.calls == [(0, 0), (0, 0)]
    Region.refuses, Host.nbytes = None, 300 << 20  # more than is kept for a stream
    assert native() is region and Host.calls[-1] == (0, 0)


def test_a_limit_of_the_caller(native):
    native(max_scratch=0), native(max_scratch=-1), native(max_scratch=1 << 20), native(max_scratch=1 << 40)
    assert [nbytes for _, nbytes in Host.calls] == [0, 0, 1 << 20, DS]


@pytest.fixture
def short(monkeypatch):
    """A backward of torch tensors, what its requests are answered with, and the allocator's counts."""
    Host.nbytes, Host.calls = DS, []
    asked, counts, answer = [], {"num_alloc_retries": 0, "num_ooms": 0}, []

    def workspace(like, shape, dtype, stream):
        if dtype == "uint8":
            asked.append(shape)
            if answer:
                raise answer[0]
        return torch.empty(shape if dtype != "uint8" else 1, dtype=runtime.TORCH_DTYPES[dtype])

    monkeypatch.setattr(runtime, "require_cuda", lambda: None)
    monkeypatch.setattr(runtime, "_workspace", workspace)
    monkeypatch.setattr(runtime._lib, "host", Host)
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda device: counts)
    q = torch.zeros(1, 8, 2, 128, dtype=torch.bfloat16)
    return lambda: runtime.attention_backward(q, q, q, q, q, torch.zeros(1, 2, 8), stream=7), asked, counts, answer


def test_what_does_not_fit_is_not_asked_for_again(short):
    backward, asked, counts, answer = short
    Host.nbytes = 4 << 30
    answer.append(torch.OutOfMemoryError("CUDA out of memory."))
    backward()
    assert len(asked) == 1 and Host.calls[-1] == (0, 0)
    counts["num_alloc_retries"] = 1  # what that request left
    backward()
    assert len(asked) == 1 and Host.calls[-1] == (0, 0)
    answer.clear()
    Host.nbytes = 64 << 20
    backward()
    assert len(asked) == 2 and Host.calls[-1][1] == 64 << 20


@pytest.mark.parametrize("error", [RuntimeError("CUDA error: an illegal memory access was encountered"), _lib.LumenError(3, "launch failure")])
def test_other_errors_are_the_callers(short, error):
    backward, _, _, answer = short
    answer.append(error)
    with pytest.raises(RuntimeError, match=str(error)):
        backward()
    assert not Host.calls


@pytest.mark.gpu
def test_a_failed_reservation_leaves_no_error_behind():
    """The next launch's check reports its own error alone."""
    region = device.Region(1 << 46)
    with pytest.raises(_lib.LumenError, match="out of memory"):
        region.empty((16,), "uint8")
    q = torch.randn(1, 40, 2, 32, device="cuda")
    o, lse = runtime.attention_forward(q, q, q)
    torch.testing.assert_close(o, torch.nn.functional.scaled_dot_product_attention(*[q.transpose(1, 2)] * 3).transpose(1, 2), atol=1e-5, rtol=1e-4)
    runtime.device_status()


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [0, 1 << 20, None])
def test_results_are_the_same_with_any_limit(limit):
    gen = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, g = (torch.randn(2, 512, 4, 128, generator=gen, device="cuda").bfloat16() for _ in range(4))
    o, lse = runtime.attention_forward(q, k, v, causal=True)
    want = runtime.attention_backward(q, k, v, o, g, lse, causal=True)
    for x, y in zip(runtime.attention_backward(q, k, v, o, g, lse, causal=True, max_scratch=limit), want):
        assert torch.equal(x, y)
