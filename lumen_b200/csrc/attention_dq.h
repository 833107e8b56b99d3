// dS handed from the backward's dK/dV kernel to its dQ kernel (attention_dq.cu), and where it lies.
//
// A unit is the dS of 64 queries and 128 keys in bfloat16, 16 KB, as two halves of 64 keys; a half lies as the operand of a product
// with the queries as its rows: [8 queries x 8][64 keys][8 queries], 16 bytes a key. Units of a key tile's half lie one after the other
// in the order of their queries, from the first block of 64 that sees any of the tile's keys, so that a tile of 256 queries is one copy.
#pragma once
#include <stdint.h>

#include "device.h"

namespace lb {

constexpr int kDsHalfBytes = 64 * 64 * 2;

struct DsLayout {
    int query_blocks = 0;  // of 64 queries, an even number
    int key_tiles = 0;     // of 128 keys
    int causal = 0;
    int offset = 0;        // the causal offset in blocks of 64, even

    // First query block with units of key tile `j`; query_blocks where there is none. Nondecreasing in j.
    __host__ __device__ int first_block(int j) const {
        if (!causal) return 0;
        const int s = 2 * j - offset;
        return s < 0 ? 0 : s > query_blocks ? query_blocks : s;
    }
    // Query blocks of the key tiles before `j`, added up.
    __host__ __device__ long long blocks_before(int j) const {
        long long left_out = 0;
        if (causal) {
            int from = offset / 2 + 1, to = (query_blocks + offset) / 2;  // between: first_block is 2 j - offset; from `to` on query_blocks
            from = from < 0 ? 0 : from, to = to < from ? from : to;
            const int a = from < j ? from : j, b = to < j ? to : j;
            left_out = (long long)(a + b - 1) * (b - a) - (long long)offset * (b - a) + (long long)(j - b) * query_blocks;
        }
        return (long long)j * query_blocks - left_out;
    }
    // Key tiles, from the first on, that have a unit of query block `qb`
    __host__ __device__ int tiles_seen(int qb) const {
        if (!causal) return key_tiles;
        const int n = qb + offset < 0 ? 0 : (qb + offset) / 2 + 1;
        return n < key_tiles ? n : key_tiles;
    }
    // Of one head, from its first byte: half `half` of the unit of key tile `j` and query block `qb`
    __host__ __device__ long long at(int j, int half, int qb) const {
        const int first = first_block(j);
        return (2 * blocks_before(j) + (long long)half * (query_blocks - first) + (qb - first)) * kDsHalfBytes;
    }
    __host__ __device__ long long head_bytes() const { return 2 * blocks_before(key_tiles) * kDsHalfBytes; }
};

struct DqArgs {
    DsLayout ds;
    const uint8_t* scores;  // the units of the heads of this launch, one head after the other
    int N, Nkv, Sq, Sk;
    int batch0, head0, heads;  // the first batch entry and query head of this launch, and its heads a batch entry
    void* dq;
    long long sb, ss, sn;
    int* status;
};
void attention_dq_launch(const CUtensorMap& keys, int batches, const DqArgs& p, cudaStream_t s);  // `keys`: tiles of 64 rows

}  // namespace lb
