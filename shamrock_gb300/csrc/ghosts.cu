// Periodic ghost layer for one patch covering the simulation box —
//   interface search shammodels/sph/src/BasicSPHGhosts.cpp:260-360 (offsets in x-outer,
//   z-inner order, the zero offset skipped), interaction range
//   shammodels/sph/include/shammodels/sph/SPHUtilities.hpp:79-95 (max h * htol * Rkern),
//   selection by half-open box shamrock/include/shamrock/patch/Patch.hpp:210-215 in
//   particle order (BasicSPHGhosts.cpp:512-530), ghosts appended after the locals in
//   interface order (shammodels/sph/include/shammodels/sph/BasicSPHGhosts.hpp:452-517).
//
// Per axis the interface interval depends only on that axis' offset, so each
// particle classifies itself once per axis (3 x 3 tests) and the 26 memberships are
// products of those.  Ghost slots are assigned by an order-preserving multi-list
// compaction: per-block counts per interface, a scan per interface, then a scatter
// that uses warp ballots for the in-block order.

#include "gbsph_ctx.cuh"

#include <algorithm>

namespace gbsph {

namespace {

constexpr int kGhostThreads = 256;
constexpr int kNoff         = 26;

struct GhostTable {
    long long lo[9]; // [3 axis + offset + 1], the bounds as ord64 patterns
    long long hi[9];
    f64 off[kNoff][3];
};

// largest h, and the interfaces' bounds and offsets from it in the last block
__global__ void __launch_bounds__(512) k_ghost_table(const f64 *__restrict__ h, u32 n, Scalars *sc, f64 htol,
                                                     f64 b0, f64 b1, f64 b2, f64 e0, f64 e1, f64 e2,
                                                     GhostTable *tab) {
    u64 m = 0;
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        u64 o = f64_to_ordered(h[i]);
        m     = o > m ? o : m;
    }
    m = block_reduce(m, OpMaxU64{}, 0ull);
    if (threadIdx.x == 0) raise_u64(&sc->hmax, m);
    if (!last_block(&sc->ticket)) return;
    const f64 bmin[3] = {b0, b1, b2}, bmax[3] = {e0, e1, e2};
    const u32 t = threadIdx.x;
    if (t < 9) {
        const int c  = t / 3;
        const f64 R  = __dmul_rn(__dmul_rn(ordered_to_f64(__ldcg(&sc->hmax)), htol), kRkern);
        f64 off      = __dmul_rn((f64) ((int) (t % 3) - 1), __dsub_rn(bmax[c], bmin[c]));
        f64 rlo      = __dadd_rn(__dsub_rn(bmin[c], R), -off);
        f64 rhi      = __dadd_rn(__dadd_rn(bmax[c], R), -off);
        const f64 lo = fmax(bmin[c], rlo), hi = fmin(bmax[c], rhi);
        // no coordinate satisfies a comparison with NaN
        tab->lo[t] = lo == lo ? ord64(lo) : 0x7fffffffffffffffll;
        tab->hi[t] = hi == hi ? ord64(hi) : (long long) 0x8000000000000000ull;
    }
    if (t < 3 * kNoff) {
        const int k = t / 3, c = t % 3, all = k < 13 ? k : k + 1; // the zero offset skipped
        const int o = (c == 0 ? all / 9 : (c == 1 ? all / 3 % 3 : all % 3)) - 1;
        tab->off[k][c] = __dmul_rn((f64) o, __dsub_rn(bmax[c], bmin[c]));
    }
    __syncthreads();
    if (t == 0) sc->hmax = 0;
}

// The bounds of one block's tests: 0-8 lower, 9-17 upper
__device__ __forceinline__ void stage_bounds(const GhostTable *tab, long long *b) {
    if (threadIdx.x < 9) {
        b[threadIdx.x]     = tab->lo[threadIdx.x];
        b[9 + threadIdx.x] = tab->hi[threadIdx.x];
    }
}

// bit k set iff the particle lies in interface k
__device__ __forceinline__ u32 ghost_mask(const long long *b, f64 x, f64 y, f64 z) {
    const long long p[3] = {ord64(x), ord64(y), ord64(z)};
    u32 ax[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        u32 m = 0;
#pragma unroll
        for (int o = 0; o < 3; o++)
            m |= (b[3 * c + o] <= p[c] && p[c] < b[9 + 3 * c + o]) ? (1u << o) : 0u;
        ax[c] = m;
    }
    u32 mask = 0;
    if (!((ax[0] | ax[1] | ax[2]) & 5u)) return 0; // near no face: most particles
    int k = 0;
#pragma unroll
    for (int xo = 0; xo < 3; xo++)
#pragma unroll
        for (int yo = 0; yo < 3; yo++)
#pragma unroll
            for (int zo = 0; zo < 3; zo++) {
                if (xo == 1 && yo == 1 && zo == 1) continue;
                bool in = ((ax[0] >> xo) & 1) && ((ax[1] >> yo) & 1) && ((ax[2] >> zo) & 1);
                mask |= in ? (1u << k) : 0u;
                k++;
            }
    return mask;
}

// Both passes read 24 bytes a particle and compare them with 18 bounds, by integers; the
// ballots of the 26 interfaces are taken only for those that a particle of the warp lies in.
// Both at 1,048,576 particles: 102 -> 24 us, 8.5 M 650 -> 163 us.
__global__ void __launch_bounds__(kGhostThreads) k_ghost_count(
    const f64 *__restrict__ x, const f64 *__restrict__ y, const f64 *__restrict__ z, u32 vs, u32 n,
    const GhostTable *__restrict__ tab, u32 nblocks, u32 *__restrict__ block_counts) {
    __shared__ long long bounds[18];
    __shared__ u32 cnt[kNoff];
    stage_bounds(tab, bounds);
    if (threadIdx.x < kNoff) cnt[threadIdx.x] = 0;
    __syncthreads();
    u32 i    = blockIdx.x * blockDim.x + threadIdx.x;
    u32 mask = 0;
    if (i < n) mask = ghost_mask(bounds, x[(size_t) i * vs], y[(size_t) i * vs], z[(size_t) i * vs]);
    int lane = threadIdx.x & 31;
    for (u32 any = __reduce_or_sync(0xffffffffu, mask); any; any &= any - 1) {
        const int k = __ffs(any) - 1;
        u32 b       = __ballot_sync(0xffffffffu, (mask >> k) & 1u);
        if (lane == 0) atomicAdd(&cnt[k], (u32) __popc(b));
    }
    __syncthreads();
    if (threadIdx.x < kNoff) block_counts[threadIdx.x * nblocks + blockIdx.x] = cnt[threadIdx.x];
}

// one block per interface: exclusive scan of its block counts in place; the last block turns
// the interfaces' totals into their bases
__global__ void k_ghost_scan(u32 *__restrict__ block_counts, u32 nblocks, u32 *__restrict__ totals, Scalars *sc) {
    u32 *bc = block_counts + blockIdx.x * nblocks;
    __shared__ u32 carry_s;
    __shared__ u32 warp_tot[32];
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    for (u32 base = 0; base < nblocks; base += blockDim.x) {
        u32 i = base + threadIdx.x;
        u32 v = (i < nblocks) ? bc[i] : 0;
        // block exclusive scan
        int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        u32 inc = v;
        for (int o = 1; o < 32; o <<= 1) {
            u32 t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) warp_tot[wid] = inc;
        __syncthreads();
        u32 wpre = 0, tot = 0;
        for (int w = 0; w < (int) (blockDim.x >> 5); w++) {
            if (w < wid) wpre += warp_tot[w];
            tot += warp_tot[w];
        }
        if (i < nblocks) bc[i] = carry_s + wpre + inc - v;
        __syncthreads();
        if (threadIdx.x == 0) carry_s += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry_s;
    if (!last_block(&sc->ticket) || threadIdx.x >= 32) return;
    const u32 k = threadIdx.x, v = k < kNoff ? __ldcg(&totals[k]) : 0u;
    u32 inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        u32 x = __shfl_up_sync(0xffffffffu, inc, o);
        if (k >= (u32) o) inc += x;
    }
    if (k < kNoff) totals[k] = inc - v; // the base of interface k
    if (k == 31) sc->ghost_total = inc;
}

__global__ void __launch_bounds__(kGhostThreads) k_ghost_scatter(
    const f64 *__restrict__ x, const f64 *__restrict__ y, const f64 *__restrict__ z, u32 vs, u32 n,
    const GhostTable *__restrict__ tab, u32 nblocks, const u32 *__restrict__ block_offsets,
    const u32 *__restrict__ bases, u32 *__restrict__ ghost_src, u8 *__restrict__ ghost_oid) {
    constexpr int kWarps = kGhostThreads / 32;
    __shared__ long long bounds[18];
    __shared__ u32 wcnt[kNoff * kWarps];
    stage_bounds(tab, bounds);
    if (threadIdx.x < kNoff * kWarps) wcnt[threadIdx.x] = 0;
    __syncthreads();
    u32 i    = blockIdx.x * blockDim.x + threadIdx.x;
    u32 mask = 0;
    if (i < n) mask = ghost_mask(bounds, x[(size_t) i * vs], y[(size_t) i * vs], z[(size_t) i * vs]);
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    u32 lt        = (1u << lane) - 1u;
    const u32 any = __reduce_or_sync(0xffffffffu, mask);
    for (u32 m = any; m; m &= m - 1) {
        const int k = __ffs(m) - 1;
        u32 b       = __ballot_sync(0xffffffffu, (mask >> k) & 1u);
        if (lane == 0) wcnt[k * kWarps + wid] = __popc(b);
    }
    __syncthreads();
    for (u32 m = any; m; m &= m - 1) {
        const int k = __ffs(m) - 1;
        u32 b       = __ballot_sync(0xffffffffu, (mask >> k) & 1u);
        if ((mask >> k) & 1u) {
            u32 pre = 0;
            for (int w = 0; w < wid; w++) pre += wcnt[k * kWarps + w];
            u32 pos = bases[k] + block_offsets[k * nblocks + blockIdx.x] + pre + (u32) __popc(b & lt);
            ghost_src[pos] = i;
            ghost_oid[pos] = (u8) k;
        }
    }
}

// Locals and ghosts in merged order.  BBOX: also their bounding box, widened by nextafter
// (BuildTrees.cpp:50-55), and the Morton grid step, by the last block; a pass of its own over
// the merged positions and three small launches otherwise: 9.1 M particles 126 -> 99 us,
// 5,887 14 -> 9 us without the gaps between the launches.
template<bool BBOX>
__global__ void __launch_bounds__(512) k_merge(const f64 *__restrict__ x, const f64 *__restrict__ y,
                        const f64 *__restrict__ z, u32 vs, const f64 *__restrict__ h, u32 n, u32 G,
                        const u32 *__restrict__ ghost_src, const u8 *__restrict__ ghost_oid,
                        const GhostTable *__restrict__ tab, f64 *__restrict__ mx,
                        f64 *__restrict__ my, f64 *__restrict__ mz, f64 *__restrict__ mh,
                        Scalars *sc, BBox *bb, u32 val_count) {
    u64 mn[3] = {~0ull, ~0ull, ~0ull}, top[3] = {0, 0, 0};
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n + G; i += gridDim.x * blockDim.x) {
        f64 p[3];
        if (i < n) {
            p[0]  = x[(size_t) i * vs];
            p[1]  = y[(size_t) i * vs];
            p[2]  = z[(size_t) i * vs];
            mh[i] = h[i];
        } else {
            u32 k   = i - n;
            u32 src = ghost_src[k];
            u32 o   = ghost_oid[k];
            p[0]    = __dadd_rn(x[(size_t) src * vs], tab->off[o][0]);
            p[1]    = __dadd_rn(y[(size_t) src * vs], tab->off[o][1]);
            p[2]    = __dadd_rn(z[(size_t) src * vs], tab->off[o][2]);
            mh[i]   = h[src];
        }
        mx[i] = p[0];
        my[i] = p[1];
        mz[i] = p[2];
        if (BBOX) {
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const u64 o = f64_to_ordered(p[c]);
                mn[c]       = o < mn[c] ? o : mn[c];
                top[c]      = o > top[c] ? o : top[c];
            }
        }
    }
    if (!BBOX) return;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const u64 a = block_reduce(mn[c], OpMinU64{}, ~0ull);
        const u64 b = block_reduce(top[c], OpMaxU64{}, 0ull);
        if (threadIdx.x == 0) {
            raise_u64(&sc->bbox_min[c], ~a);
            raise_u64(&sc->bbox_max[c], b);
        }
    }
    if (!last_block(&sc->ticket) || threadIdx.x >= 3) return;
    const int c      = threadIdx.x;
    const f64 inf    = __longlong_as_double(0x7ff0000000000000ll);
    const f64 lo     = nextafter(ordered_to_f64(~__ldcg(&sc->bbox_min[c])), -inf);
    const f64 hi     = nextafter(ordered_to_f64(__ldcg(&sc->bbox_max[c])), inf);
    const f64 f      = __ddiv_rn(__dsub_rn(hi, lo), (f64) val_count);
    bb->lo[c]        = lo;
    bb->hi[c]        = hi;
    bb->fact[c]      = f;
    bb->inv[c]       = f > 1e-300 && f < 1e300 ? __ddiv_rn(1.0, f) : 0.0;
    sc->bbox_min[c]  = 0;
    sc->bbox_max[c]  = 0;
}

} // namespace

cudaError_t periodic_ghosts(Ctx &c, const f64 *x, const f64 *y, const f64 *z, u32 vs,
                            const f64 *h, u32 n, const f64 *bmin, const f64 *bmax, f64 htol) {
    cudaStream_t s = c.stream;
    cudaError_t e;
    Scalars *dsc = c.d_scalars.as<Scalars>();
    u32 nblocks  = div_up(n, kGhostThreads);
    if (nblocks == 0) nblocks = 1;
    if ((e = c.d_ghost_offsets.ensure(sizeof(GhostTable), s)) != cudaSuccess) return e;
    if ((e = c.ghost_block_counts.ensure(sizeof(u32) * ((size_t) kNoff * nblocks + kNoff), s)) !=
        cudaSuccess)
        return e;
    GhostTable *tab = c.d_ghost_offsets.as<GhostTable>();
    u32 *bc         = c.ghost_block_counts.as<u32>();
    u32 *totals     = bc + (size_t) kNoff * nblocks;
    int pg = c.prof.on ? prof_begin(c, kProfGhosts, n) : -1;
    { k_ghost_table<<<std::min(div_up(n, 512), 2 * c.sms), 512, 0, s>>>(h, n, dsc, htol, bmin[0], bmin[1], bmin[2],
                                                                       bmax[0], bmax[1], bmax[2], tab); GBSPH_COUNTED; }
    { k_ghost_count<<<nblocks, kGhostThreads, 0, s>>>(x, y, z, vs, n, tab, nblocks, bc); GBSPH_COUNTED; }
    { k_ghost_scan<<<kNoff, 1024, 0, s>>>(bc, nblocks, totals, dsc); GBSPH_COUNTED; }
    if (pg >= 0) prof_end(c, pg);
    if ((e = sync_scalars(c)) != cudaSuccess) return e;
    ProfScope ps(c, kProfGhosts, 0);
    u32 G     = c.h_scalars->ghost_total;
    c.n_ghost = G;
    if ((e = c.ghost_src.ensure(sizeof(u32) * ((size_t) G + 1), s)) != cudaSuccess) return e;
    if ((e = c.ghost_oid.ensure((size_t) G + 1, s)) != cudaSuccess) return e;
    if (G)
        { k_ghost_scatter<<<nblocks, kGhostThreads, 0, s>>>(x, y, z, vs, n, tab, nblocks, bc, totals,
                                                          c.ghost_src.as<u32>(),
                                                          c.ghost_oid.as<u8>()); GBSPH_COUNTED; }
    return cudaGetLastError();
}

cudaError_t merge_positions(Ctx &c, const f64 *x, const f64 *y, const f64 *z, u32 vs,
                            const f64 *h, u32 n, bool bbox) {
    cudaStream_t s = c.stream;
    cudaError_t e;
    u32 N = n + c.n_ghost;
    if ((e = c.mx.ensure(sizeof(f64) * (size_t) N, s)) != cudaSuccess) return e;
    if ((e = c.my.ensure(sizeof(f64) * (size_t) N, s)) != cudaSuccess) return e;
    if ((e = c.mz.ensure(sizeof(f64) * (size_t) N, s)) != cudaSuccess) return e;
    if ((e = c.mh.ensure(sizeof(f64) * (size_t) N, s)) != cudaSuccess) return e;
    if ((e = c.d_ghost_offsets.ensure(sizeof(GhostTable), s)) != cudaSuccess) return e;
    ProfScope ps(c, kProfMerge, N);
    auto kern = bbox ? k_merge<true> : k_merge<false>;
    { kern<<<std::min(div_up(N, 512), 2 * c.sms), 512, 0, s>>>(
        x, y, z, vs, h, n, c.n_ghost, c.ghost_src.as<u32>(), c.ghost_oid.as<u8>(), c.d_ghost_offsets.as<GhostTable>(),
        c.mx.as<f64>(), c.my.as<f64>(), c.mz.as<f64>(), c.mh.as<f64>(), c.d_scalars.as<Scalars>(),
        c.d_bbox.as<BBox>(), 1024u); GBSPH_COUNTED; }
    return cudaGetLastError();
}

} // namespace gbsph
