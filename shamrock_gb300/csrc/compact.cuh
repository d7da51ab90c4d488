// Ordered compaction in two launches: per-block counts, whose last block scans them, and a
// pass that places each selected item.  Items are taken 32 at a time by a warp, so loads are
// coalesced and the places follow from ballots.  A block owns a run of whole tiles; at most
// four blocks an SM, as the counts' last-block counter costs about 10 ns a block.  The flags
// are evaluated twice instead of being stored with their offsets (nine and five bytes an
// item, five launches): leaves and rows of 9.1 M particles 71 us together against 240, of
// 5,887 14 us in four launches against 22 in ten.
#pragma once

#include "gbsph_ctx.cuh"

#include <algorithm>

namespace gbsph {
namespace {

constexpr u32 kCompactRounds = 16, kCompactTile = 256 * kCompactRounds;

// the warp's selected items of one tile, as a ballot per round
template<class Flag>
__device__ __forceinline__ u32 tile_ballots(const Flag &flag, u32 n, u32 first, u32 (&b)[kCompactRounds]) {
    u32 sum = 0;
#pragma unroll
    for (u32 k = 0; k < kCompactRounds; k++) {
        const u32 i = first + k * 32;
        b[k]        = __ballot_sync(0xffffffffu, i < n && flag(i));
        sum += __popc(b[k]);
    }
    return sum;
}

template<class Flag>
__global__ void __launch_bounds__(256) k_compact_count(Flag flag, u32 n, u32 tiles, u32 *__restrict__ counts,
                                                       u32 *__restrict__ total, u32 *ticket) {
    __shared__ u32 ws[8];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    u32 sum = 0, b[kCompactRounds];
    for (u32 t = 0; t < tiles; t++) {
        const u32 tile = blockIdx.x * tiles + t;
        sum += tile_ballots(flag, n, tile * kCompactTile + w * (32 * kCompactRounds) + lane, b);
    }
    if (lane == 0) ws[w] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (u32 k = 1; k < 8; k++) sum += ws[k];
        counts[blockIdx.x] = sum;
    }
    if (!last_block(ticket)) return;
    // exclusive scan of the blocks' counts
    u32 carry = 0;
    for (u32 base = 0; base < gridDim.x; base += 256) {
        const u32 i = base + threadIdx.x, v = i < gridDim.x ? __ldcg(&counts[i]) : 0u;
        u32 inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 x = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (u32) o) inc += x;
        }
        __syncthreads();
        if (lane == 31) ws[w] = inc;
        __syncthreads();
        u32 before = carry;
        for (u32 k = 0; k < 8; k++) {
            if (k < w) before += ws[k];
            carry += ws[k];
        }
        if (i < gridDim.x) counts[i] = before + inc - v;
    }
    if (threadIdx.x == 0) *total = carry;
}

template<class Flag, class Place>
__global__ void __launch_bounds__(256) k_compact_place(Flag flag, Place place, u32 n, u32 tiles,
                                                       const u32 *__restrict__ offsets,
                                                       const u32 *__restrict__ total) {
    __shared__ u32 ws[8];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    u32 at = offsets[blockIdx.x], b[kCompactRounds];
    for (u32 t = 0; t < tiles; t++) {
        const u32 first = (blockIdx.x * tiles + t) * kCompactTile + w * (32 * kCompactRounds) + lane;
        const u32 sum   = tile_ballots(flag, n, first, b);
        __syncthreads();
        if (lane == 0) ws[w] = sum;
        __syncthreads();
        u32 pos = at;
        for (u32 k = 0; k < 8; k++) {
            if (k < w) pos += ws[k];
            at += ws[k];
        }
#pragma unroll
        for (u32 k = 0; k < kCompactRounds; k++) {
            if ((b[k] >> lane) & 1u) place(first + k * 32, pos + __popc(b[k] & ((1u << lane) - 1u)));
            pos += __popc(b[k]);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) place.end(*total);
}

template<class Flag, class Place>
cudaError_t compact(Ctx &c, const Flag &flag, const Place &place, u32 n, u32 *total) {
    const u32 all    = std::max(div_up(n, kCompactTile), 1u);
    const u32 tiles  = div_up(all, 4 * c.sms), blocks = div_up(all, tiles);
    cudaError_t e    = c.scan_scratch.ensure(sizeof(u32) * (size_t) blocks, c.stream);
    if (e != cudaSuccess) return e;
    u32 *counts = c.scan_scratch.as<u32>();
    { k_compact_count<<<blocks, 256, 0, c.stream>>>(flag, n, tiles, counts, total, &c.d_scalars.as<Scalars>()->ticket); GBSPH_COUNTED; }
    { k_compact_place<<<blocks, 256, 0, c.stream>>>(flag, place, n, tiles, counts, total); GBSPH_COUNTED; }
    return cudaGetLastError();
}

} // namespace
} // namespace gbsph
