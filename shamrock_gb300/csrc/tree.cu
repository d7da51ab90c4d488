// Compressed-leaf BVH build on the GPU: Morton keys, bitonic key/value sort, leaf
// reduction, Karras radix tree, AABB and interaction radius of leaves and nodes.
// Bit-exact with the reference semantics (see the oracle restatement):
//   Morton     shamtree/src/MortonCodeSet.cpp:63-118, shammath/sfc/morton.hpp:46-230
//   sort       shamalgs/src/details/algorithm/bitonicSort_updated_usm.cpp:26-396
//   reduction  shamtree/src/kernels/reduction_alg.cpp:62-85,196-244,274-295,413-456
//   Karras     shamtree/src/KarrasRadixTree.cpp:45-143
//   AABB/field shamtree/src/KarrasRadixTreeAABB.cpp:33-140,
//              shamtree/include/shamtree/KarrasRadixTreeField.hpp:134-222,
//              shammodels/sph/src/Solver.cpp:1322-1356
// The reference propagates node boxes with tree_depth full sweeps; here a node's box is
// united from the few boxes of an 8-ary hierarchy over the leaves that make up its range,
// with the same exact min/max.

#include "compact.cuh"
#include "lean64.cuh"

#include <type_traits>
#include <utility>

namespace gbsph {

namespace {

// ---------------------------------------------------------------- Morton
template<class K>
struct Morton;
template<>
struct Morton<u32> {
    static constexpr u32 val_count = 1024, max_val = 1023;
    static constexpr u32 err       = 0xFFFFFFFFu;
    __device__ static u32 expand(u32 x) {
        x &= 0x3ffU;
        x = (x | x << 16U) & 0x30000ffU;
        x = (x | x << 8U) & 0x300f00fU;
        x = (x | x << 4U) & 0x30c30c3U;
        x = (x | x << 2U) & 0x9249249U;
        return x;
    }
    __device__ static u32 encode(u32 x, u32 y, u32 z) { return expand(x) * 4 + expand(y) * 2 + expand(z); }
    __device__ static int clz(u32 v) { return __clz(v); }
};
template<>
struct Morton<u64> {
    static constexpr u32 val_count = 2097152, max_val = 2097151;
    static constexpr u64 err       = 0xFFFFFFFFFFFFFFFFull;
    __device__ static u64 expand(u64 x) {
        x &= 0x1fffffULL;
        x = (x | x << 32ULL) & 0x1f00000000ffffULL;
        x = (x | x << 16ULL) & 0x1f0000ff0000ffULL;
        x = (x | x << 8ULL) & 0x100f00f00f00f00fULL;
        x = (x | x << 4ULL) & 0x10c30c30c30c30c3ULL;
        x = (x | x << 2ULL) & 0x1249249249249249ULL;
        return x;
    }
    __device__ static u64 encode(u64 x, u64 y, u64 z) { return expand(x) * 4 + expand(y) * 2 + expand(z); }
    __device__ static int clz(u64 v) { return __clzll((long long) v); }
};

// 24 bytes read and 8 written a particle; bound by the FP64 pipe until the cell took two FP64
// instructions a coordinate: 1,048,576 particles 81 -> 24 us, 8.5 M 590 -> 172 us.
template<class K>
__global__ void k_morton(const f64 *__restrict__ x, const f64 *__restrict__ y,
                         const f64 *__restrict__ z, u32 n, u32 P, const BBox *__restrict__ bb,
                         K *__restrict__ keys, u32 *__restrict__ vals) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    vals[i] = i;
    if (i >= n) {
        keys[i] = Morton<K>::err;
        return;
    }
    const u32 gx = grid_cell(x[i], bb->lo[0], bb->hi[0], bb->fact[0], bb->inv[0], Morton<K>::max_val);
    const u32 gy = grid_cell(y[i], bb->lo[1], bb->hi[1], bb->fact[1], bb->inv[1], Morton<K>::max_val);
    const u32 gz = grid_cell(z[i], bb->lo[2], bb->hi[2], bb->fact[2], bb->inv[2], Morton<K>::max_val);
    keys[i]      = Morton<K>::encode(gx, gy, gz);
}

// ---------------------------------------------------------------- bitonic sort
// Compare-exchange of the reference network (bitonicSort_updated_usm.cpp:29-39):
// swap iff reverse ^ (a < b), reverse = ((length << 1) & i) == 0.
template<class K>
__device__ __forceinline__ void cmpx(K &a, K &b, u32 &va, u32 &vb, bool reverse) {
    bool swap = reverse ^ (a < b);
    if (swap) {
        K t = a;
        a   = b;
        b   = t;
        u32 tv = va;
        va     = vb;
        vb     = tv;
    }
}

// The tile of the shared-memory passes.  A thread holds the elements that differ in up to
// four neighbouring index bits, the lowest of them bit 0, 4 or 8; with the low four bits
// exchanged with the next four (an XOR, so the places of a group follow from one) 16
// consecutive lanes always meet all 16 pairs of banks.
__device__ __forceinline__ u32 tile_place(u32 i) { return i ^ ((i >> 4) & 15u); }
template<class K, int TILE>
struct SortTile {
    K k[TILE];
    u32 v[TILE];
    __device__ __forceinline__ void get(u32 p, K &a, u32 &b) const { a = k[p], b = v[p]; }
    __device__ __forceinline__ void put(u32 p, K a, u32 b) { k[p] = a, v[p] = b; }
};
template<int TILE>
struct SortTile<u32, TILE> {
    uint2 kv[TILE];
    __device__ __forceinline__ void get(u32 p, u32 &a, u32 &b) const {
        const uint2 e = kv[p];
        a = e.x, b = e.y;
    }
    __device__ __forceinline__ void put(u32 p, u32 a, u32 b) { kv[p] = make_uint2(a, b); }
};

// the stages of increments S / 2 ... 1 among S elements in registers
template<class K, int S>
__device__ __forceinline__ void reg_stages(K (&x)[S], u32 (&v)[S], bool reverse) {
#pragma unroll
    for (int d = S / 2; d >= 1; d >>= 1)
#pragma unroll
        for (int k = 0; k < S; k++)
            if ((k & d) == 0) cmpx(x[k], x[k + d], v[k], v[k + d], reverse);
}

// BITS consecutive stages (increments 2^(bit + BITS - 1) ... 2^bit) of one merge step;
// from: where the first of a merge's rounds finds the elements, null once they are in s
template<class K, int TILE, int BITS>
__device__ __forceinline__ void tile_round(SortTile<K, TILE> &s, u32 tile, u32 base, u32 dir, int bit,
                                           const K *from_k = nullptr, const u32 *from_v = nullptr) {
    constexpr int S = 1 << BITS;
    for (u32 g = threadIdx.x; g < tile >> BITS; g += blockDim.x) {
        const u32 i = ((g >> bit) << (bit + BITS)) | (g & ((1u << bit) - 1u)), p = tile_place(i);
        K x[S];
        u32 v[S];
#pragma unroll
        for (int k = 0; k < S; k++) {
            if (from_k) x[k] = from_k[base + i + ((u32) k << bit)], v[k] = from_v[base + i + ((u32) k << bit)];
            else s.get(p ^ tile_place((u32) k << bit), x[k], v[k]);
        }
        reg_stages<K, S>(x, v, (dir & (base + i)) == 0);
#pragma unroll
        for (int k = 0; k < S; k++) s.put(p ^ tile_place((u32) k << bit), x[k], v[k]);
    }
    __syncthreads();
}

// The stages within tiles, up to four at a time in registers.  MERGE: the last
// log2(TILE) stages of one merge step, else all steps of lengths below `tile`.  Bound by
// issue and shared memory about alike: a pair costs about six instructions a stage, and the
// tile is read and written once for four.  2^22 keys, all launches: 624 us with a stage at a
// time in shared memory, 398 with three in registers, 208 with four.
template<class K, int TILE, bool MERGE>
__global__ void __launch_bounds__(256) k_bitonic_smem(K *__restrict__ keys, u32 *__restrict__ vals,
                                                      u32 tile, u32 length) {
    __shared__ SortTile<K, TILE> s;
    constexpr int kBits = TILE == 4096 ? 12 : 11, kTop = kBits - 8;
    const u32 base = blockIdx.x * tile;
    if (MERGE) {
        tile_round<K, TILE, kTop>(s, TILE, base, length << 1, 8, keys, vals);
        tile_round<K, TILE, 4>(s, TILE, base, length << 1, 4);
        tile_round<K, TILE, 4>(s, TILE, base, length << 1, 0);
    } else {
        for (u32 k = threadIdx.x; k < tile; k += 256) s.put(tile_place(k), keys[base + k], vals[base + k]);
        __syncthreads();
        for (u32 len = 1; len < tile; len <<= 1) {
            int left = 32 - __clz(len); // stages of the step
            if (left % 4 == 1) tile_round<K, TILE, 1>(s, tile, base, len << 1, left - 1);
            if (left % 4 == 2) tile_round<K, TILE, 2>(s, tile, base, len << 1, left - 2);
            if (left % 4 == 3) tile_round<K, TILE, 3>(s, tile, base, len << 1, left - 3);
            for (left -= left % 4; left > 0; left -= 4) tile_round<K, TILE, 4>(s, tile, base, len << 1, left - 4);
        }
    }
    for (u32 k = threadIdx.x; k < tile; k += 256) s.get(tile_place(k), keys[base + k], vals[base + k]);
}

// LEVELS consecutive stages (inc, inc/2, ...) of one merge step in registers,
// as the reference's order_kernel<2^LEVELS> (bitonicSort_updated_usm.cpp:111-281).
template<class K, int LEVELS>
__global__ void __launch_bounds__(256) k_bitonic_global(K *__restrict__ keys, u32 *__restrict__ vals,
                                                        u32 nthreads, u32 length, u32 inc) {
    constexpr int S = 1 << LEVELS;
    u32 t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nthreads) return;
    u32 sub  = inc >> (LEVELS - 1);
    u32 low  = t & (sub - 1);
    u32 i    = ((t - low) << LEVELS) + low;
    bool reverse = ((length << 1) & i) == 0;
    K x[S];
    u32 v[S];
#pragma unroll
    for (int k = 0; k < S; k++) {
        x[k] = keys[i + k * sub];
        v[k] = vals[i + k * sub];
    }
#pragma unroll
    for (int d = S / 2; d >= 1; d >>= 1) {
#pragma unroll
        for (int k = 0; k < S; k++) {
            if ((k & d) == 0) cmpx(x[k], x[k + d], v[k], v[k + d], reverse);
        }
    }
#pragma unroll
    for (int k = 0; k < S; k++) {
        keys[i + k * sub] = x[k];
        vals[i + k * sub] = v[k];
    }
}

template<class K>
cudaError_t bitonic_sort(K *keys, u32 *vals, u32 len, cudaStream_t s) {
    constexpr int TILE = (sizeof(K) == 4) ? 4096 : 2048;
    if (len <= 1) return cudaSuccess;
    u32 tile = len < (u32) TILE ? len : (u32) TILE;
    { k_bitonic_smem<K, TILE, false><<<len / tile, 256, 0, s>>>(keys, vals, tile, 0); GBSPH_COUNTED; }
    for (u32 length = TILE; length < len; length <<= 1) {
        u32 inc = length;
        while (inc >= (u32) TILE) {
            int avail  = __builtin_ctz(inc) - __builtin_ctz((u32) TILE) + 1;
            int levels = avail < 4 ? avail : 4;
            u32 nth    = len >> levels;
            u32 blocks = div_up(nth, 256);
            switch (levels) {
            case 4: { k_bitonic_global<K, 4><<<blocks, 256, 0, s>>>(keys, vals, nth, length, inc); GBSPH_COUNTED; } break;
            case 3: { k_bitonic_global<K, 3><<<blocks, 256, 0, s>>>(keys, vals, nth, length, inc); GBSPH_COUNTED; } break;
            case 2: { k_bitonic_global<K, 2><<<blocks, 256, 0, s>>>(keys, vals, nth, length, inc); GBSPH_COUNTED; } break;
            default: { k_bitonic_global<K, 1><<<blocks, 256, 0, s>>>(keys, vals, nth, length, inc); GBSPH_COUNTED; } break;
            }
            inc >>= levels;
        }
        { k_bitonic_smem<K, TILE, true><<<len / TILE, 256, 0, s>>>(keys, vals, TILE, length); GBSPH_COUNTED; }
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------- radix sort
// Stable LSD radix sort of n u32 keys with u32 values, four 8-bit digits.  Per pass: a
// per-block digit histogram (bucket-major), its exclusive scan (the global start of each
// block's elements of each digit), and a scatter that walks the block's tile in index
// order, 256 elements per round: lanes with equal digits are ranked with a warp match,
// warps by an exclusive prefix of their per-warp counts, so every pass is stable.  With
// distinct keys the result is the unique sorted order, hence the bitonic network's.
constexpr u32 kRadixItems = 8, kRadixTile = 256 * kRadixItems;

__global__ void __launch_bounds__(256) k_radix_hist(const u32 *__restrict__ keys, u32 n, int shift,
                                                    u32 nblocks, u32 *__restrict__ hist) {
    __shared__ u32 h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const u32 base = blockIdx.x * kRadixTile;
#pragma unroll
    for (u32 r = 0; r < kRadixItems; r++) {
        const u32 i = base + r * 256 + threadIdx.x;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

__global__ void __launch_bounds__(256) k_radix_scatter(const u32 *__restrict__ kin,
                                                       const u32 *__restrict__ vin, u32 n, int shift,
                                                       u32 nblocks, const u32 *__restrict__ offs,
                                                       u32 *__restrict__ kout, u32 *__restrict__ vout) {
    __shared__ u32 cnt[256];   // next output slot of each digit for this block
    __shared__ u32 wc[8][256]; // per-warp digit counts, then their exclusive prefix
    const u32 t = threadIdx.x, lane = t & 31u, w = t >> 5;
    cnt[t]         = offs[t * nblocks + blockIdx.x];
    const u32 base = blockIdx.x * kRadixTile;
    for (u32 r = 0; r < kRadixItems; r++) {
        for (u32 k = lane; k < 256; k += 32) wc[w][k] = 0;
        __syncthreads();
        const u32 i     = base + r * 256 + t;
        const bool valid = i < n;
        const u32 key   = valid ? kin[i] : 0u;
        const u32 val   = valid ? vin[i] : 0u;
        const u32 d     = (key >> shift) & 255u;
        // invalid lanes match only themselves (values above 255)
        const u32 peers = __match_any_sync(0xffffffffu, valid ? d : (0x100u | lane));
        const u32 lower = __popc(peers & ((1u << lane) - 1u));
        if (valid && lower == 0) wc[w][d] = __popc(peers);
        __syncthreads();
        u32 run = cnt[t];
#pragma unroll
        for (u32 ww = 0; ww < 8; ww++) {
            const u32 c = wc[ww][t];
            wc[ww][t]   = run;
            run += c;
        }
        cnt[t] = run;
        __syncthreads();
        if (valid) {
            const u32 pos = wc[w][d] + lower;
            kout[pos]     = key;
            vout[pos]     = val;
        }
        __syncthreads();
    }
}

__global__ void k_adjacent_dup(const u32 *__restrict__ keys, u32 n, u32 *__restrict__ flag) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i + 1 < n && keys[i] == keys[i + 1]) atomicOr(flag, 1u);
}

// sorts keys[0..n) / vals[0..n) in place (four passes end in the input buffers)
cudaError_t radix_sort_u32(Ctx &c, u32 *keys, u32 *vals, u32 n, cudaStream_t s) {
    cudaError_t e;
    if (n < 2) return cudaSuccess;
    const u32 nb = div_up(n, kRadixTile);
    if ((e = c.radix_k.ensure(sizeof(u32) * (size_t) n, s)) != cudaSuccess) return e;
    if ((e = c.radix_v.ensure(sizeof(u32) * (size_t) n, s)) != cudaSuccess) return e;
    if ((e = c.radix_hist.ensure(sizeof(u32) * 256 * (size_t) nb, s)) != cudaSuccess) return e;
    if ((e = c.radix_off.ensure(sizeof(u32) * 256 * (size_t) nb, s)) != cudaSuccess) return e;
    Scalars *dsc = c.d_scalars.as<Scalars>();
    u32 *ka = keys, *va = vals, *kb = c.radix_k.as<u32>(), *vb = c.radix_v.as<u32>();
    for (int shift = 0; shift < 32; shift += 8) {
        { k_radix_hist<<<nb, 256, 0, s>>>(ka, n, shift, nb, c.radix_hist.as<u32>()); GBSPH_COUNTED; }
        if ((e = scan_exclusive_u32(c.radix_hist.as<u32>(), c.radix_off.as<u32>(), 256 * nb,
                                    &dsc->total2, c.scan_scratch, s)) != cudaSuccess)
            return e;
        { k_radix_scatter<<<nb, 256, 0, s>>>(ka, va, n, shift, nb, c.radix_off.as<u32>(), kb, vb); GBSPH_COUNTED; }
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------- leaf reduction
template<class K>
__device__ __forceinline__ i32 karras_delta(i32 x, i32 y, u32 len, const K *__restrict__ m) {
    if ((u32) y > len - 1 || y < 0) return -1;
    return Morton<K>::clz(m[x] ^ m[y]);
}

template<class K>
__global__ void k_split(const K *__restrict__ m, u32 cnt, u8 *__restrict__ out) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cnt) return;
    out[i] = (i > 0) ? ((m[i - 1] != m[i]) ? 1 : 0) : 1;
}

template<class K>
__global__ void k_reduce_iter(const K *__restrict__ m, u32 cnt, const u8 *__restrict__ in,
                              u8 *__restrict__ out) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cnt) return;
    u32 before1 = i - 1;
    while (before1 <= cnt - 1 && !in[before1]) before1--;
    u32 before2 = before1 - 1;
    while (before2 <= cnt - 1 && !in[before2]) before2--;
    u32 next1 = i + 1;
    while (next1 <= cnt - 1 && !in[next1]) next1++;
    i32 delt_0  = karras_delta<K>((i32) i, (i32) next1, cnt, m);
    i32 delt_m  = karras_delta<K>((i32) i, (i32) before1, cnt, m);
    i32 delt_mm = karras_delta<K>((i32) before1, (i32) before2, cnt, m);
    out[i] = (!(delt_0 < delt_m && delt_mm < delt_m) && in[i]) ? 1 : 0;
}

// the kept split points become the leaves
struct LeafFlag {
    const u8 *f;
    __device__ __forceinline__ bool operator()(u32 i) const { return f[i] != 0; }
};
template<class K>
struct LeafPlace {
    const K *m;
    u32 *reduc;
    K *reduced;
    u32 cnt;
    __device__ __forceinline__ void operator()(u32 i, u32 o) const {
        reduc[o]   = i;
        reduced[o] = m[i];
    }
    __device__ __forceinline__ void end(u32 L) const {
        reduc[L]     = cnt;
        reduc[L + 1] = 0;
    }
};

// ---------------------------------------------------------------- Karras
template<class K>
__global__ void k_karras(const K *__restrict__ m, u32 L, u32 *__restrict__ lchild,
                         u32 *__restrict__ rchild, u8 *__restrict__ lflag, u8 *__restrict__ rflag,
                         u32 *__restrict__ endrange, u32 *__restrict__ parent) {
    u32 ui = blockIdx.x * blockDim.x + threadIdx.x;
    if (ui == 0) parent[0] = kNone;
    if (ui + 1 >= L) return;
    i32 i = (i32) ui;
    auto DELTA = [&](i32 a, i32 b) { return karras_delta<K>(a, b, L, m); };
    i32 ddelta    = DELTA(i, i + 1) - DELTA(i, i - 1);
    i32 d         = (ddelta == 0) ? 0 : ((ddelta > 0) ? 1 : -1);
    i32 delta_min = DELTA(i, i - d);
    i32 lmax      = 2;
    while (DELTA(i, i + lmax * d) > delta_min) lmax *= 2;
    i32 l = 0;
    i32 t = lmax / 2;
    while (t > 0) {
        if (DELTA(i, i + (l + t) * d) > delta_min) l = l + t;
        t = t / 2;
    }
    u32 j          = (u32) (i + l * d);
    endrange[i]    = j;
    i32 delta_node = DELTA(i, (i32) j);
    i32 s          = 0;
    float div      = 2;
    t              = (i32) ceilf(__fdiv_rn((float) l, div));
    while (true) {
        i32 tmp_ = i + (s + t) * d;
        if (DELTA(i, tmp_) > delta_node) s = s + t;
        if (t <= 1) break;
        div *= 2;
        t = (i32) ceilf(__fdiv_rn((float) l, div));
    }
    i32 gamma  = i + s * d + min(d, 0);
    u32 off    = L - 1;
    bool lleaf = (min(ui, j) == (u32) gamma);
    bool rleaf = (max(ui, j) == (u32) (gamma + 1));
    lchild[i]  = (u32) gamma;
    lflag[i]   = lleaf ? 1 : 0;
    rchild[i]  = (u32) (gamma + 1);
    rflag[i]   = rleaf ? 1 : 0;
    parent[(u32) gamma + (lleaf ? off : 0)]       = ui;
    parent[(u32) (gamma + 1) + (rleaf ? off : 0)] = ui;
}

// ---------------------------------------------------------------- rank-order copies
__global__ void k_permute(const u32 *__restrict__ sort_index, u32 n, const f64 *__restrict__ x,
                          const f64 *__restrict__ y, const f64 *__restrict__ z,
                          const f64 *__restrict__ h, f64 *__restrict__ sx, f64 *__restrict__ sy,
                          f64 *__restrict__ sz, f64 *__restrict__ sh, u32 *__restrict__ rank_of) {
    u32 r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    u32 id     = sort_index[r];
    sx[r]      = x[id];
    sy[r]      = y[id];
    sz[r]      = z[id];
    if (h) sh[r] = h[id];
    rank_of[id] = r;
}

// ---------------------------------------------------------------- node boxes
// A box's six faces and radius as ordered integers (the largest of lo, hi and the radius is
// taken by integer comparisons; on the FP64 pipe each is 16 cycles of the SM)
struct BoxKeys {
    u64 lo[3], hi[3], rint;
};
__device__ __forceinline__ void min_key(u64 &m, u64 k) { m = k < m ? k : m; }
__device__ __forceinline__ void max_key(u64 &m, u64 k) { m = k > m ? k : m; }
// fmin and fmax drop a NaN: the key that never wins
__device__ __forceinline__ bool is_nan_bits(f64 v) {
    const u32 hi = (u32) __double2hiint(v) << 1, lo = (u32) __double2loint(v);
    return (hi | (lo != 0u ? 1u : 0u)) > 0xffe00000u;
}
__device__ __forceinline__ void store_box(NodeBox *b, const BoxKeys &k) {
    double2 *p = (double2 *) b;
    p[0]       = make_double2(ordered_to_f64(k.lo[0]), ordered_to_f64(k.lo[1]));
    p[1]       = make_double2(ordered_to_f64(k.lo[2]), ordered_to_f64(k.rint));
    p[2]       = make_double2(ordered_to_f64(k.hi[0]), ordered_to_f64(k.hi[1]));
    p[3]       = make_double2(ordered_to_f64(k.hi[2]), 0.0);
}

__device__ __forceinline__ BoxKeys no_box() {
    BoxKeys k;
#pragma unroll
    for (int c = 0; c < 3; c++) k.lo[c] = ~0ull, k.hi[c] = 0ull;
    k.rint = 0ull;
    return k;
}
__device__ __forceinline__ void unite(BoxKeys &k, const BoxKeys &o) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
        min_key(k.lo[c], o.lo[c]);
        max_key(k.hi[c], o.hi[c]);
    }
    max_key(k.rint, o.rint);
}
__device__ __forceinline__ BoxKeys load_keys(const NodeBox *__restrict__ b) {
    const double2 *s = (const double2 *) b;
    const double2 s0 = s[0], s1 = s[1], s2 = s[2];
    const f64 hz = ((const f64 *) b)[6];
    return BoxKeys{{f64_to_ordered(s0.x), f64_to_ordered(s0.y), f64_to_ordered(s1.x)},
                   {f64_to_ordered(s2.x), f64_to_ordered(s2.y), f64_to_ordered(hz)},
                   is_nan_bits(s1.y) ? 0ull : f64_to_ordered(s1.y)};
}
__device__ __forceinline__ NodeBoxF box_f32(const BoxKeys &k) {
    NodeBoxF f;
    f.lo = make_float4(narrow64(ordered_to_f64(k.lo[0])), narrow64(ordered_to_f64(k.lo[1])),
                       narrow64(ordered_to_f64(k.lo[2])), narrow64(__dmul_rn(ordered_to_f64(k.rint), kRkern)));
    f.hi = make_float4(narrow64(ordered_to_f64(k.hi[0])), narrow64(ordered_to_f64(k.hi[1])),
                       narrow64(ordered_to_f64(k.hi[2])), 0.f);
    return f;
}

// a node's box, its FP32 copy, and the copy in its parent's child-pair record
__device__ __forceinline__ void put_node(u32 node, u32 off, const BoxKeys &k, const u32 *__restrict__ lchild,
                                         const u8 *__restrict__ lflag, const u32 *__restrict__ parent,
                                         NodeBox *__restrict__ boxes, NodeBoxF *__restrict__ fb,
                                         NodePairF *__restrict__ rec) {
    store_box(&boxes[node], k);
    NodeBoxF f = box_f32(k);
    fb[node]   = f;
    const u32 p = parent[node];
    if (p == kNone) return;
    f.hi.w = __uint_as_float(node);
    if (lchild[p] + off * (u32) lflag[p] == node) rec[p].l = f;
    else rec[p].r = f;
}

// Boxes of the nodes without a walk up the tree: an internal node covers a range of leaves,
// whose box is united from the few nodes of the 8-ary hierarchy that make it up (minimum and
// maximum are exact, so the order does not matter).  A walk with arrival counters is a chain
// of one to two microseconds a level.  Leaves, levels and nodes together, against the walk and
// the hierarchy built after it: 1,399 leaves 23 us against 31, 35,981 33 against 49, 239,928 79
// against 103, 2.0 M 373 against 446 (bytes: 0.28 GB of boxes and records there, 45 us).
__global__ void __launch_bounds__(256) k_leaf_boxes(const u32 *__restrict__ reduc, u32 L, const f64 *__restrict__ sx,
                                                    const f64 *__restrict__ sy, const f64 *__restrict__ sz,
                                                    const f64 *__restrict__ sh, f64 htol,
                                                    const u32 *__restrict__ lchild, const u8 *__restrict__ lflag,
                                                    const u32 *__restrict__ parent, NodeBox *__restrict__ boxes,
                                                    NodeBoxF *__restrict__ fb, NodePairF *__restrict__ rec) {
    u32 l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= L) return;
    const f64 big = 1.7976931348623157e308;
    BoxKeys k;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        k.lo[c] = f64_to_ordered(big);
        k.hi[c] = f64_to_ordered(-big);
    }
    u64 hm = f64_to_ordered(-big);
    const u32 end = reduc[l + 1];
    for (u32 r = reduc[l]; r < end; r++) {
        const f64 p[3] = {sx[r], sy[r], sz[r]};
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const bool nan = is_nan_bits(p[c]);
            const u64 o    = f64_to_ordered(p[c]);
            min_key(k.lo[c], nan ? ~0ull : o);
            max_key(k.hi[c], nan ? 0ull : o);
        }
        if (sh) {
            const f64 h = sh[r];
            max_key(hm, is_nan_bits(h) ? 0ull : f64_to_ordered(h));
        }
    }
    k.rint = f64_to_ordered(sh ? __dmul_rn(ordered_to_f64(hm), htol) : 0.0);
    put_node(L - 1 + l, L - 1, k, lchild, lflag, parent, boxes, fb, rec);
}

// three levels of the hierarchy above n boxes: 512 of them to 64, 8 and 1 per block
__device__ __forceinline__ BoxKeys unite8(BoxKeys k) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        BoxKeys x;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            x.lo[c] = __shfl_xor_sync(0xffffffffu, k.lo[c], o);
            x.hi[c] = __shfl_xor_sync(0xffffffffu, k.hi[c], o);
        }
        x.rint = __shfl_xor_sync(0xffffffffu, k.rint, o);
        unite(k, x);
    }
    return k;
}
__global__ void __launch_bounds__(512) k_box_levels(const NodeBox *__restrict__ in, LevelPlan lp, int m,
                                                    NodeBox *__restrict__ lb, NodeBoxF *__restrict__ wb) {
    __shared__ BoxKeys s1[64], s2[8];
    const u32 t = threadIdx.x, i = blockIdx.x * 512 + t;
    auto put = [&](int level, u32 o, const BoxKeys &k) {
        if (level > lp.top || o >= lp.n[level]) return;
        store_box(&lb[lp.at[level] + o], k);
        wb[lp.at[level] + o] = box_f32(k);
    };
    BoxKeys k = unite8(i < lp.n[m] ? load_keys(&in[i]) : no_box());
    if ((t & 7) == 0) {
        s1[t / 8] = k;
        put(m + 1, blockIdx.x * 64 + t / 8, k);
    }
    __syncthreads();
    if (t < 64) {
        k = unite8(s1[t]);
        if ((t & 7) == 0) {
            s2[t / 8] = k;
            put(m + 2, blockIdx.x * 8 + t / 8, k);
        }
    }
    __syncthreads();
    if (t < 32) {
        k = unite8(t < 8 ? s2[t] : no_box());
        if (t == 0) put(m + 3, blockIdx.x, k);
    }
}

__global__ void __launch_bounds__(256) k_node_boxes(u32 L, LevelPlan lp, const u32 *__restrict__ endrange,
                                                    const u32 *__restrict__ lchild, const u8 *__restrict__ lflag,
                                                    const u32 *__restrict__ parent, const NodeBox *__restrict__ lb,
                                                    NodeBox *boxes, NodeBoxF *__restrict__ fb,
                                                    NodePairF *__restrict__ rec) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i + 1 >= L) return;
    const u32 j = endrange[i];
    u32 a = min(i, j), b = max(i, j) + 1; // the nodes [a, b) of level m
    const NodeBox *level = boxes + (L - 1);
    BoxKeys k            = no_box();
    for (int m = 0; a < b; m++) {
        const bool top = m == lp.top;
        while (a < b && ((a & 7u) || top)) unite(k, load_keys(&level[a++]));
        while (a < b && (b & 7u)) unite(k, load_keys(&level[--b]));
        a >>= 3;
        b >>= 3;
        level = lb + lp.at[min(m + 1, lp.top)];
    }
    put_node(i, L - 1, k, lchild, lflag, parent, boxes, fb, rec);
}

// Up to this many keys (padded to a power of two) the network sorts at once.  Where keys are
// distinct it costs what the radix sort does (2^20: 105 us against 100, and 14 launches
// against 23; 2^19: 67 against 88; 2^13: 20 us in 3 launches against 68 in 21; at 2^21 192
// against 119), and where they are not, as in most states that are no lattice, the radix
// sort's work and the tree passes up to its sync are lost (disc of 1,000,003: 4242 -> 4053 us
// a step).
constexpr u32 kNetworkKeys = 1u << 20;

template<class K>
cudaError_t tree_build_impl(Ctx &c, const f64 *x, const f64 *y, const f64 *z, const f64 *h, u32 n,
                            u32 level, f64 htol, u32 morton_count, bool fast_sort,
                            const std::function<cudaError_t()> &between) {
    cudaStream_t s = c.stream;
    cudaError_t e;
    u32 P = morton_count;
    if (P == 0) {
        P = 1;
        while (P < n) P <<= 1;
    }
    c.n_obj        = n;
    c.morton_count = P;
    c.key_bits     = (int) sizeof(K) * 8;
    c.has_rint     = (h != nullptr);
#define ENS(buf, bytes)                                                                          \
    if ((e = (buf).ensure((bytes), s)) != cudaSuccess) return e;
    ENS(c.keys, sizeof(K) * P);
    ENS(c.sort_index, sizeof(u32) * P);
    ENS(c.flags_a, n);
    ENS(c.flags_b, n);
    ENS(c.reduc, sizeof(u32) * ((size_t) n + 2));
    ENS(c.reduced, sizeof(K) * (size_t) n);
    ENS(c.rank_of, sizeof(u32) * (size_t) n);
    ENS(c.sx, sizeof(f64) * (size_t) n);
    ENS(c.sy, sizeof(f64) * (size_t) n);
    ENS(c.sz, sizeof(f64) * (size_t) n);
    ENS(c.sh, sizeof(f64) * (size_t) n);

    K *keys = c.keys.as<K>();
    u32 *vals = c.sort_index.as<u32>();
    const u32 T = 256;
    Scalars *dsc = c.d_scalars.as<Scalars>();
    u8 *fa = c.flags_a.as<u8>(), *fb = c.flags_b.as<u8>();
    u8 *fin = (level % 2 == 0) ? fa : fb;
    // For many keys the radix sort is tried first when allowed; equal keys (whose order is
    // the network's) send the build back to the bitonic sort, found at the sync below.
    const bool radix = fast_sort && std::is_same<K, u32>::value && P > kNetworkKeys;
    bool posted = false;
    for (int attempt = radix ? 0 : 1; attempt < 2; attempt++) {
        {
            ProfScope ps(c, kProfSort, P);
            { k_morton<K><<<div_up(P, T), T, 0, s>>>(x, y, z, n, P, c.d_bbox.as<BBox>(), keys, vals); GBSPH_COUNTED; }
            if (attempt == 0) {
                if ((e = cudaMemsetAsync(&dsc->dup_keys, 0, sizeof(u32), s)) != cudaSuccess) return e;
                if ((e = radix_sort_u32(c, (u32 *) keys, vals, n, s)) != cudaSuccess) return e;
                { k_adjacent_dup<<<div_up(n, T), T, 0, s>>>((const u32 *) keys, n, &dsc->dup_keys); GBSPH_COUNTED; }
            } else {
                if ((e = bitonic_sort<K>(keys, vals, P, s)) != cudaSuccess) return e;
            }
        }
        int prof_tree = c.prof.on ? prof_begin(c, kProfTree, n) : -1;
        // leaf reduction: ping-pong split tables, final table is a for even levels
        { k_split<K><<<div_up(n, T), T, 0, s>>>(keys, n, fa); GBSPH_COUNTED; }
        for (u32 it = 1; it <= level; it++) {
            if (it % 2 == 0) { k_reduce_iter<K><<<div_up(n, T), T, 0, s>>>(keys, n, fb, fa); GBSPH_COUNTED; }
            else { k_reduce_iter<K><<<div_up(n, T), T, 0, s>>>(keys, n, fa, fb); GBSPH_COUNTED; }
        }
        if ((e = compact(c, LeafFlag{fin}, LeafPlace<K>{keys, c.reduc.as<u32>(), c.reduced.as<K>(), n}, n,
                         &dsc->total)) != cudaSuccess)
            return e;
        if (prof_tree >= 0) prof_end(c, prof_tree);
        if (attempt == 0) {
            if ((e = sync_scalars(c)) != cudaSuccess) return e;
            if (!c.h_scalars->dup_keys) break;
        } else {
            if ((e = post_scalars(c)) != cudaSuccess) return e;
            posted = true;
        }
    }
    { k_permute<<<div_up(n, T), T, 0, s>>>(vals, n, x, y, z, h, c.sx.as<f64>(), c.sy.as<f64>(),
                                         c.sz.as<f64>(), c.sh.as<f64>(), c.rank_of.as<u32>()); GBSPH_COUNTED; }
    if (between && (e = between()) != cudaSuccess) return e;
    if (posted && (e = wait_scalars(c)) != cudaSuccess) return e;
    ProfScope ps_tree(c, kProfTree, 0);
    u32 L        = c.h_scalars->total;
    c.leaf_count = L;
    u32 I        = L - 1;
    u32 Tn       = 2 * L - 1;
    ENS(c.lchild, sizeof(u32) * (I + 1));
    ENS(c.rchild, sizeof(u32) * (I + 1));
    ENS(c.lflag, I + 1);
    ENS(c.rflag, I + 1);
    ENS(c.endrange, sizeof(u32) * (I + 1));
    ENS(c.parent, sizeof(u32) * Tn);
    ENS(c.boxes, sizeof(NodeBox) * Tn);
    ENS(c.fboxes, sizeof(NodeBoxF) * Tn);
    ENS(c.fpairs, sizeof(NodePairF) * (size_t) L);
    const LevelPlan lp = level_plan(L);
    ENS(c.lboxes, sizeof(NodeBox) * ((size_t) lp.total + 1));
    ENS(c.wboxes, sizeof(NodeBoxF) * ((size_t) lp.total + 1));
#undef ENS
    { k_karras<K><<<div_up(L, T), T, 0, s>>>(c.reduced.as<K>(), L, c.lchild.as<u32>(),
                                           c.rchild.as<u32>(), c.lflag.as<u8>(), c.rflag.as<u8>(),
                                           c.endrange.as<u32>(), c.parent.as<u32>()); GBSPH_COUNTED; }
    NodeBox *boxes = c.boxes.as<NodeBox>();
    { k_leaf_boxes<<<div_up(L, T), T, 0, s>>>(c.reduc.as<u32>(), L, c.sx.as<f64>(), c.sy.as<f64>(), c.sz.as<f64>(),
                                            h ? c.sh.as<f64>() : nullptr, htol, c.lchild.as<u32>(), c.lflag.as<u8>(),
                                            c.parent.as<u32>(), boxes, c.fboxes.as<NodeBoxF>(),
                                            c.fpairs.as<NodePairF>()); GBSPH_COUNTED; }
    for (int m = 0; m < lp.top; m += 3)
        { k_box_levels<<<div_up(lp.n[m], 512), 512, 0, s>>>(m ? c.lboxes.as<NodeBox>() + lp.at[m] : boxes + (L - 1), lp, m,
                                                          c.lboxes.as<NodeBox>(), c.wboxes.as<NodeBoxF>()); GBSPH_COUNTED; }
    if (L > 1)
        { k_node_boxes<<<div_up(L - 1, T), T, 0, s>>>(L, lp, c.endrange.as<u32>(), c.lchild.as<u32>(), c.lflag.as<u8>(),
                                                    c.parent.as<u32>(), c.lboxes.as<NodeBox>(), boxes,
                                                    c.fboxes.as<NodeBoxF>(), c.fpairs.as<NodePairF>()); GBSPH_COUNTED; }
    return cudaGetLastError();
}

} // namespace

cudaError_t sync_scalars(Ctx &c) {
    cudaError_t e = cudaMemcpyAsync(c.h_scalars, c.d_scalars.p, sizeof(Scalars),
                                    cudaMemcpyDeviceToHost, c.stream);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(c.stream);
}

cudaError_t post_scalars(Ctx &c) {
    cudaError_t e = cudaMemcpyAsync(c.h_scalars, c.d_scalars.p, sizeof(Scalars),
                                    cudaMemcpyDeviceToHost, c.stream);
    return e != cudaSuccess ? e : cudaEventRecord(c.posted, c.stream);
}
cudaError_t wait_scalars(Ctx &c) { return cudaEventSynchronize(c.posted); }

cudaError_t set_bbox_host(Ctx &c, const f64 *bmin, const f64 *bmax, int key_bits) {
    const f64 cells = (f64) (key_bits == 64 ? Morton<u64>::val_count : Morton<u32>::val_count);
    BBox b{};
    for (int k = 0; k < 3; k++) {
        b.lo[k]   = bmin[k];
        b.hi[k]   = bmax[k];
        b.fact[k] = (bmax[k] - bmin[k]) / cells;
        b.inv[k]  = b.fact[k] > 1e-300 && b.fact[k] < 1e300 ? 1.0 / b.fact[k] : 0.0;
    }
    cudaError_t e = cudaMemcpyAsync(c.d_bbox.p, &b, sizeof(BBox), cudaMemcpyHostToDevice, c.stream);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(c.stream);
}

cudaError_t tree_build(Ctx &c, const f64 *x, const f64 *y, const f64 *z, const f64 *h, u32 n,
                       u32 level, f64 htol, int key_bits, u32 morton_count, bool fast_sort,
                       const std::function<cudaError_t()> &between) {
    if (key_bits == 64) return tree_build_impl<u64>(c, x, y, z, h, n, level, htol, morton_count, false, between);
    return tree_build_impl<u32>(c, x, y, z, h, n, level, htol, morton_count, fast_sort, between);
}

// explicit entry points for module-level exports (driver.cu)
template<class K>
cudaError_t sort_keys_dev(K *keys, u32 *vals, u32 len, cudaStream_t s) {
    return bitonic_sort<K>(keys, vals, len, s);
}
template cudaError_t sort_keys_dev<u32>(u32 *, u32 *, u32, cudaStream_t);
template cudaError_t sort_keys_dev<u64>(u64 *, u32 *, u32, cudaStream_t);

} // namespace gbsph

namespace gbsph {

namespace {
template<class K>
__global__ void k_morton_only(const f64 *__restrict__ x, const f64 *__restrict__ y,
                              const f64 *__restrict__ z, u32 n, u32 P, const BBox *__restrict__ bb,
                              K *__restrict__ keys) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    if (i >= n) {
        keys[i] = Morton<K>::err;
        return;
    }
    const u32 gx = grid_cell(x[i], bb->lo[0], bb->hi[0], bb->fact[0], bb->inv[0], Morton<K>::max_val);
    const u32 gy = grid_cell(y[i], bb->lo[1], bb->hi[1], bb->fact[1], bb->inv[1], Morton<K>::max_val);
    const u32 gz = grid_cell(z[i], bb->lo[2], bb->hi[2], bb->fact[2], bb->inv[2], Morton<K>::max_val);
    keys[i]      = Morton<K>::encode(gx, gy, gz);
}

__global__ void k_export_boxes(const NodeBox *__restrict__ b, u32 T, f64 *__restrict__ mn,
                               f64 *__restrict__ mx, f64 *__restrict__ rint) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T) return;
    NodeBox v = b[i];
    if (mn) {
        mn[3 * i] = v.lo[0];
        mn[3 * i + 1] = v.lo[1];
        mn[3 * i + 2] = v.lo[2];
    }
    if (mx) {
        mx[3 * i] = v.hi[0];
        mx[3 * i + 1] = v.hi[1];
        mx[3 * i + 2] = v.hi[2];
    }
    if (rint) rint[i] = v.rint;
}
} // namespace

cudaError_t morton_codes_dev(Ctx &c, const f64 *x, const f64 *y, const f64 *z, u32 n, u32 P,
                             int key_bits, void *out) {
    if (key_bits == 64) {
        { k_morton_only<u64><<<div_up(P, 256), 256, 0, c.stream>>>(x, y, z, n, P, c.d_bbox.as<BBox>(),
                                                                 (u64 *) out); GBSPH_COUNTED; }
    } else {
        { k_morton_only<u32><<<div_up(P, 256), 256, 0, c.stream>>>(x, y, z, n, P, c.d_bbox.as<BBox>(),
                                                                 (u32 *) out); GBSPH_COUNTED; }
    }
    return cudaGetLastError();
}

cudaError_t export_boxes(Ctx &c, f64 *mn, f64 *mx, f64 *rint) {
    u32 T = 2 * c.leaf_count - 1;
    { k_export_boxes<<<div_up(T, 256), 256, 0, c.stream>>>(c.boxes.as<NodeBox>(), T, mn, mx, rint); GBSPH_COUNTED; }
    return cudaGetLastError();
}

} // namespace gbsph
