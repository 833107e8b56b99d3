"""Where the backward's dS lies between its dK/dV kernel and its dQ kernel (csrc/attention_dq.h), built for the host: what is read has been
written, nothing is written twice, and everything lies within the scratch."""

import ctypes
import os
import subprocess

import pytest

from lumen_b200 import _lib

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lumen_b200", "csrc")
CUDA = "/usr/local/cuda/include"

HOST = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include "attention_dq.h"
using namespace lb;
#define CHECK(x) do { if (!(x)) { std::printf("Sq %lld Sk %lld causal %d offset %lld: %s\n", Sq, Sk, causal, offset, #x); return 1; } } while (0)
static int check(long long Sq, long long Sk, int causal, long long offset) {
    DsLayout ds;
    ds.query_blocks = (int)((Sq + 127) / 128) * 2, ds.key_tiles = (int)((Sk + 127) / 128), ds.causal = causal, ds.offset = causal ? (int)(offset / 64) : 0;
    const long long bytes = ds.head_bytes();
    std::map<long long, int> written;  // place -> the key tile, half and query block whose it is
    auto name = [](int j, int half, int qb) { return (j * 2 + half) * 4096 + qb; };
    long long before = 0;
    for (int j = 0; j < ds.key_tiles; j++) {  // as the dK/dV kernel walks its queries
        const long long r0 = 128LL * j, first_q = causal ? std::min(Sq, std::max(0LL, r0 - offset)) : 0;
        const long long stream0 = first_q / 64 * 64, per_head = first_q >= Sq ? 0 : (Sq - stream0 + 127) / 128;
        CHECK(ds.blocks_before(j) == before);
        before += 2 * per_head;
        for (long long it = 0; it < per_head; it++)
            for (int wg = 0; wg < 2; wg++)
                for (int half = 0; half < 2; half++) {
                    const long long at = ds.at(j, half, (int)(stream0 / 64)) + wg * kDsHalfBytes + it * 2 * kDsHalfBytes;
                    CHECK(at >= 0 && at + kDsHalfBytes <= bytes && at % kDsHalfBytes == 0 && !written.count(at));
                    written[at] = name(j, half, (int)(stream0 / 64 + 2 * it + wg));
                }
    }
    CHECK(bytes == (long long)written.size() * kDsHalfBytes && bytes == 2 * before * kDsHalfBytes);
    long long read = 0;
    for (int tile = 0; 256LL * tile < Sq; tile++) {  // as the dQ kernel walks its keys
        const int qb0 = tile * 4, blocks = std::min(4, ds.query_blocks - qb0);
        const int seen0 = ds.tiles_seen(qb0), seen1 = blocks == 4 ? ds.tiles_seen(qb0 + 2) : 0;
        CHECK((blocks == 2 || blocks == 4) && (blocks == 2 || (seen1 >= seen0 && seen1 <= seen0 + 1) || !causal));
        for (int j = 0; j < std::max(seen0, seen1); j++)
            for (int half = 0; half < 2; half++) {
                const int skip = j < seen0 ? 0 : 2, count = (j < seen1 ? 4 : 2) - skip;
                CHECK(skip + count <= blocks && count > 0);
                for (int u = skip; u < skip + count; u++, read++) {
                    auto it = written.find(ds.at(j, half, qb0 + skip) + (u - skip) * (long long)kDsHalfBytes);
                    CHECK(it != written.end() && it->second == name(j, half, qb0 + u));
                }
            }
        // every key that a query of the tile sees is in a tile that is read
        for (long long q = 256LL * tile; q < std::min(Sq, 256LL * (tile + 1)); q++) {
            const long long last = causal ? std::min(Sk - 1, q + offset) : Sk - 1;
            if (last >= 0) CHECK(last / 128 < (q < 256LL * tile + 128 ? seen0 : seen1));
        }
    }
    CHECK(read == (long long)written.size());
    return 0;
}
int main() {
    for (long long Sq : {1, 64, 127, 128, 129, 256, 257, 384, 600, 1024, 1531})
        for (long long Sk : {1, 127, 128, 200, 256, 500, 1024, 1531}) {
            if (check(Sq, Sk, 0, 0)) return 1;
            for (long long offset = -2048; offset <= 2048; offset += 128)
                if (check(Sq, Sk, 1, offset)) return 1;
        }
    return 0;
}
"""


def test_what_is_read_was_written(tmp_path):
    if not os.path.exists(os.path.join(CUDA, "cuda.h")):
        pytest.skip("no CUDA headers")
    (tmp_path / "ds.cpp").write_text(HOST)
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", CSRC, "-I", CUDA, "-I", os.path.join(CSRC, "../../include"), "-o", str(tmp_path / "ds"), str(tmp_path / "ds.cpp")], check=True)
    done = subprocess.run([str(tmp_path / "ds")], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout


def scratch_bytes(b, sq, sk, n, nkv, h, causal, offset=None, dtype="bfloat16"):
    desc = _lib.LbAttnDesc(1.0, int(causal), sk - sq if offset is None else offset)
    q, k = _lib.dense(1 << 20, dtype, (b, sq, n, h)), _lib.dense(1 << 20, dtype, (b, sk, nkv, h))
    return _lib.lib().lb_attention_bwd_scratch_bytes(ctypes.byref(desc), ctypes.byref(q), ctypes.byref(k))


def test_when_and_how_much():
    unit = 16384
    assert scratch_bytes(1, 256, 256, 1, 1, 128, False) == 8 * unit
    assert scratch_bytes(2, 256, 256, 6, 3, 128, True) == 12 * 6 * unit
    assert scratch_bytes(1, 256, 512, 1, 1, 128, True) == (4 + 4 + 4 + 2) * unit
    for left_out in ((1, 256, 256, 1, 1, 64, True), (1, 64, 256, 1, 1, 128, False), (1, 320, 256, 1, 1, 128, False), (1, 256, 320, 1, 1, 128, True),
                     (0, 256, 256, 1, 1, 128, True), (1, 0, 256, 1, 1, 128, False), (1, 512, 256, 1, 1, 128, True, -1024)):
        assert scratch_bytes(*left_out) == 0, left_out
    assert scratch_bytes(1, 256, 256, 1, 1, 128, True, dtype="float32") == 0
    # more than the limit: rounds of as many batch entries each, or of heads of one entry, and none where not even one fits
    one = scratch_bytes(1, 4096, 4096, 32, 32, 128, True)
    assert one == 32 * 32 * 33 * unit and scratch_bytes(8, 4096, 4096, 32, 32, 128, True) == 8 * one
    assert scratch_bytes(16, 4096, 4096, 32, 32, 128, True) == 8 * one and scratch_bytes(10, 4096, 4096, 32, 32, 128, True) == 5 * one
    assert scratch_bytes(1, 8192, 8192, 128, 128, 128, True) == 64 * 64 * 65 * unit
    # ... or where the rounds would have few CTAs
    assert scratch_bytes(3, 16384, 16384, 32, 8, 128, True) == 0 and scratch_bytes(1, 1 << 17, 1 << 17, 32, 32, 128, True) == 0


SHAPES = [
    # b, sq, sk, n, nkv, causal, and the heads a round takes by the scratch it is given (0: all)
    (1, 128, 128, 1, 1, True, 0), (1, 128, 128, 1, 1, False, 0), (2, 256, 256, 2, 1, True, 0), (1, 384, 384, 3, 1, True, 0), (1, 600, 600, 2, 2, True, 0),
    (1, 600, 600, 2, 2, False, 0), (2, 1531, 1531, 4, 2, True, 0), (1, 100, 1000, 2, 1, False, 0), (1, 1000, 72, 2, 1, False, 0), (1, 512, 768, 2, 1, True, 0),
    (1, 768, 512, 2, 1, True, 0), (1, 513, 641, 2, 2, True, 0), (3, 640, 640, 6, 2, True, 0), (48, 512, 512, 32, 32, True, 24 * 32),
    (1, 256, 256, 3200, 3200, True, 1600), (1, 256, 256, 3200, 1600, False, 1599),
]


@pytest.mark.gpu
@pytest.mark.parametrize("b, sq, sk, n, nkv, causal, heads", SHAPES)
def test_dq_from_dS_that_was_left(b, sq, sk, n, nkv, causal, heads):
    """Both ways to dQ round the same values of dS and add the same products in the order of the keys: every bit is the same."""
    import torch

    from lumen_b200 import runtime

    gen = torch.Generator(device="cuda").manual_seed(sq * 7 + sk)
    q, d_o = (torch.randn(b, sq, n, 128, generator=gen, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(b, sk, nkv, 128, generator=gen, device="cuda").bfloat16() for _ in range(2))
    o, lse = runtime.attention_forward(q, k, v, causal=causal)
    nbytes = scratch_bytes(b, sq, sk, n, nkv, 128, causal)
    assert nbytes > 0
    if heads:
        nbytes = nbytes // (b * nkv) * heads + 12345
    few = heads == 1599  # rounds of so few that dS is computed twice

    def backward(nbytes):
        scratch = torch.full((nbytes + 16,), 255, dtype=torch.uint8, device="cuda")  # NaNs wherever a value is read that was not written
        grads = [torch.full_like(t, float("nan")) for t in (q, k, v)]
        delta = torch.empty(b, n, sq, device="cuda")
        runtime._lib.host().attention_bwd(128**-0.5, causal, sk - sq, q, k, v, o, d_o, lse, delta, None, *grads, scratch.data_ptr() if nbytes else 0, nbytes,
                                          torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert (scratch[nbytes:] == 255).all()
        return grads, bool((scratch[:nbytes] != 255).any())

    (want, _), (got, used) = backward(0), backward(nbytes)
    assert used != few
    for name, x, y in zip(("dq", "dk", "dv"), got, want):
        assert torch.equal(x, y), (name, (x.float() - y.float()).norm() / y.float().norm())
    runtime.device_status()
