// Two-stage neighbour cache over the compressed-leaf BVH —
//   shammodels/sph/src/modules/NeighbourCache.cpp:223-596 (start_neighbors_cache_2stages),
//   traversal shamtree/include/shamtree/KarrasTreeTraverser.hpp:70-118 (left-first DFS),
//   criteria shamtree/include/shamtree/kernels/geometry_utils.hpp:62-135,
//   CSR layout shamtree/include/shamtree/TreeTraversal.hpp:375-526.
//
// Stage 1: leaf -> candidate leaves (extended-AABB overlap, both directions), stored
//          as rank ranges: consecutive leaves cover consecutive ranks, so runs of
//          consecutive candidates merge and stage 2 walks fewer, longer runs.
// Owner:   local particle -> leaf (the last leaf, in DFS order, whose box holds it).
// Stage 2: local particle -> interacting particles, pair test
//          !(r^2 > (h_a htol)^2 R^2 && r^2 > (h_b htol)^2 R^2).
// Rows are local particles in Morton order; entries are ranks, so a row lists its
// neighbours in exactly the reference order (ascending leaf, then in-leaf order).

#include "compact.cuh"
#include "split64.cuh"

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <type_traits>

namespace gbsph {

namespace {

constexpr int kStack   = 64;
// Initial one-pass slots: stage-1 leaves per leaf, stage-2 entries per row (multiple of
// 4).  A build that overflows records its largest row and is rerun, still in one pass,
// with slots that fit; the context keeps the grown sizes for later builds.
constexpr u32 kLeafCap = 256;
constexpr u32 kRowCap  = 192;
// Beyond this many slot bytes (or u32 offsets) the exact two-pass builds run instead.
constexpr u64 kMaxSlotBytes = 24ull << 30;

__device__ __forceinline__ void load_box(const NodeBox *__restrict__ b, f64 lo[3], f64 hi[3],
                                         f64 &rint) {
    const double2 *p = (const double2 *) b;
    double2 a = __ldg(p), c = __ldg(p + 1), d = __ldg(p + 2), e = __ldg(p + 3);
    lo[0] = a.x;
    lo[1] = a.y;
    lo[2] = c.x;
    rint  = c.y;
    hi[0] = d.x;
    hi[1] = d.y;
    hi[2] = e.x;
}

struct TreeView {
    const u32 *lchild, *rchild;
    const u8 *lflag, *rflag;
    const NodeBox *boxes;
    const u32 *reduc;
    u32 L;
    __device__ u32 off() const { return L - 1; }
    __device__ u32 left(u32 n) const { return lchild[n] + off() * (u32) lflag[n]; }
    __device__ u32 right(u32 n) const { return rchild[n] + off() * (u32) rflag[n]; }
};

// left-first stack DFS; on_leaf(leaf_index) in ascending leaf order
template<class Crit, class OnLeaf>
__device__ __forceinline__ bool dfs(const TreeView &t, Crit &&crit, OnLeaf &&on_leaf) {
    u32 stack[kStack];
    int top      = 0;
    stack[top++] = 0;
    u32 off      = t.off();
    while (top > 0) {
        u32 node = stack[--top];
        if (!crit(node)) continue;
        if (node >= off) {
            on_leaf(node - off);
        } else {
            if (top + 2 > kStack) return false;
            stack[top++] = t.right(node);
            stack[top++] = t.left(node);
        }
    }
    return true;
}

// Candidate leaves arrive in ascending order; a leaf following the previous run
// directly extends it.  A run of leaves [l0, l1) is stored as its rank range
// [reduc[l0], reduc[l1]).  `c` counts runs; only the first `cap` are stored.
struct RangeWriter {
    uint2 *out;
    const u32 *reduc;
    u32 base, cap, c;
    uint2 cur;
    bool open;
    __device__ RangeWriter(uint2 *o, const u32 *rd, u32 b, u32 cp, bool writes = true)
        : out(writes ? o : nullptr), reduc(rd), base(b), cap(cp), c(0), open(false) {}
    __device__ __forceinline__ void add(u32 r0, u32 r1) {
        if (open && cur.y == r0) {
            cur.y = r1;
            return;
        }
        flush();
        cur  = make_uint2(r0, r1);
        open = true;
    }
    __device__ __forceinline__ void flush() {
        if (!open) return;
        if (out && c < cap) out[base + c] = make_uint2(reduc[cur.x], reduc[cur.y]);
        c++;
        open = false;
    }
};

// ---- stage 1 criterion (NeighbourCache.cpp:289-334)
__device__ __forceinline__ bool cella_neigh_b(const f64 amin[3], const f64 amax[3],
                                              const f64 bmin[3], const f64 bmax[3]) {
    return (fmax(amin[0], bmin[0]) <= fmin(amax[0], bmax[0]))
           && (fmax(amin[1], bmin[1]) <= fmin(amax[1], bmax[1]))
           && (fmax(amin[2], bmin[2]) <= fmin(amax[2], bmax[2]));
}

struct LeafCrit {
    const TreeView &t;
    f64 amin[3], amax[3], amin_ext[3], amax_ext[3];
    __device__ LeafCrit(const TreeView &tv, u32 leaf) : LeafCrit(tv, tv.off() + leaf, 0) {}
    __device__ LeafCrit(const TreeView &tv, u32 leaf_node, int) : t(tv) {
        f64 r;
        load_box(&t.boxes[leaf_node], amin, amax, r);
        f64 ra = __dmul_rn(r, kRkern);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            amin_ext[c] = __dsub_rn(amin[c], ra);
            amax_ext[c] = __dadd_rn(amax[c], ra);
        }
    }
    __device__ bool operator()(u32 node) const {
        f64 nlo[3], nhi[3], r;
        load_box(&t.boxes[node], nlo, nhi, r);
        f64 rn = __dmul_rn(r, kRkern);
        f64 emin[3], emax[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            emin[c] = __dsub_rn(nlo[c], rn);
            emax[c] = __dadd_rn(nhi[c], rn);
        }
        return cella_neigh_b(amin, amax, emin, emax) || cella_neigh_b(amin_ext, amax_ext, nlo, nhi);
    }
};

// The same criterion with the leaf's FP64 box loaded at each call: for the one-pass
// traversals, which decide almost every node in FP32 and come here only inside the
// rounding band; a call keeps its two dozen doubles out of their registers.
static __device__ __noinline__ bool leaf_crit_call(const NodeBox *boxes, u32 leaf_node, u32 node) {
    TreeView t{};
    t.boxes = boxes;
    return LeafCrit(t, leaf_node, 0)(node);
}
struct LazyLeafCrit {
    const TreeView &t;
    u32 leaf_node;
    __device__ LazyLeafCrit(const TreeView &tv, u32 leaf) : t(tv), leaf_node(tv.off() + leaf) {}
    __device__ bool operator()(u32 node) const {
        return leaf_crit_call(t.boxes, leaf_node, node);
    }
};

// exact two-pass stage 1: range counts, then ranges at the scanned offsets
__global__ void k_leaf_count(TreeView t, u32 *__restrict__ cnt, u32 *__restrict__ flags) {
    u32 l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= t.L) return;
    LeafCrit crit(t, l);
    RangeWriter w(nullptr, t.reduc, 0, 0);
    bool ok = dfs(t, crit, [&](u32 leaf) { w.add(leaf, leaf + 1); });
    w.flush();
    if (!ok) atomicOr(flags, kFlagStackOverflow);
    cnt[l] = w.c;
}

__global__ void k_leaf_fill(TreeView t, const u32 *__restrict__ off, uint2 *__restrict__ ent) {
    u32 l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= t.L) return;
    LeafCrit crit(t, l);
    RangeWriter w(ent, t.reduc, off[l], 0xffffffffu);
    dfs(t, crit, [&](u32 leaf) { w.add(leaf, leaf + 1); });
    w.flush();
}

// ---- stage 1, one pass into `cap` slots per leaf, optional FP32 pre-test.
// For boxes a (the leaf) and n (a node) the criterion is
//   C1 || C2,  C1 = a overlaps n grown by r_n,  C2 = a grown by r_a overlaps n,
// which in exact arithmetic is  max_axis s <= max(r_n, r_a)  with the per-axis
// separation s = max(n.lo - a.hi, a.lo - n.hi).  The FP32 estimate of s carries at most
// ~2e-7 of the largest coordinate M plus 1e-7 relative; outside a band of
// 1e-6 (M + R) the FP32 answer is certain, inside it the FP64 criterion decides.
// Stage 1 over the child-pair records.  An internal node loads both children's boxes in one
// record and tests them together; the walk goes on in the left child that passes, and the
// right one waits on the stack if both do.  Every node is tested once, when its parent is
// expanded, so the leaves and their order are those of dfs() with the same criterion; per
// step the traversal waits on one record load instead of a box load and a child-index load
// per node.  leaf_thr (see k_owner): a leaf owning no row gets an empty list, and a node
// below which no owned row can find a pair is dropped (the cache is unchanged).
// Local memory is what this kernel must not touch: each lane's stack stands at its own
// height, so an access is up to 32 lines.  The first twelve places are in shared memory, a
// bank per lane, the FP64 criterion is a call, and the registers are not bounded (72; with
// 64, 40 bytes of spills make it three times slower).  1,048,576 / 8.5 M particles 580 us /
// 3.92 ms with the stack in local memory and every passing child pushed, 538 / 3.56 with
// inner nodes dropped too, 460 / 3.12 now; disc 940 -> 777 us.
constexpr int kNear = 12;
__global__ void __launch_bounds__(128) k_leaf_lists(TreeView t, const NodeBoxF *__restrict__ fb,
                                                    const NodePairF *__restrict__ rec,
                                                    u32 *__restrict__ cnt, u32 *__restrict__ off,
                                                    uint2 *__restrict__ ent, u32 cap, Scalars *sc,
                                                    const u32 *__restrict__ leaf_thr) {
    u32 l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= t.L) return;
    u32 base = l * cap;
    const u32 tb = leaf_thr[l];
    if (tb == 0) { // no row is owned by this leaf: stage 2 never reads its list
        cnt[l] = 0;
        off[l] = base;
        return;
    }
    const float thr_own = __uint_as_float(tb);
    LazyLeafCrit crit(t, l);
    const u32 offn = t.off();
    F8 fa = ldg256(&fb[offn + l]), fr = ldg256(&fb[0]);
    const float4 alo = fa.a, ahi = fa.b, rlo = fr.a, rhi = fr.b;
    float M = fmaxf(fmaxf(fmaxf(fabsf(rlo.x), fabsf(rlo.y)), fmaxf(fabsf(rlo.z), fabsf(rhi.x))),
                    fmaxf(fabsf(rhi.y), fabsf(rhi.z)));
    float band_abs = 1e-6f * M;
    // the criterion with an FP32 decision outside the rounding band
    auto test = [&](u32 node, const float4 &nlo, const float4 &nhi) -> bool {
        float sx = fmaxf(nlo.x - ahi.x, alo.x - nhi.x);
        float sy = fmaxf(nlo.y - ahi.y, alo.y - nhi.y);
        float sz = fmaxf(nlo.z - ahi.z, alo.z - nhi.z);
        float sm = fmaxf(fmaxf(sx, sy), sz);
        float R  = fmaxf(nlo.w, alo.w);
        float band = band_abs + 1e-6f * R;
        if (sm < R - band) return true;
        if (sm > R + band) return false;
        return crit(node);
    };
    // Exact pruning for stage 2: every row owned by this leaf lies in its box, so a
    // pair (a, b) with b in the candidate leaf has r_ab at least the Euclidean gap D
    // between the boxes.  With thr_own >= thr_a of every owned row and
    // (r_leaf R)^2 >= thr_b, D^2 > max of the two makes every pair test fail.  The FP32
    // gaps are shrunk by the rounding band and the bound carries a 1e-5 margin, so the
    // skip is certain.
    auto keep = [&](const float4 &nlo, const float4 &nhi) -> bool {
        float gx = fmaxf(fmaxf(nlo.x - ahi.x, alo.x - nhi.x) - band_abs, 0.f);
        float gy = fmaxf(fmaxf(nlo.y - ahi.y, alo.y - nhi.y) - band_abs, 0.f);
        float gz = fmaxf(fmaxf(nlo.z - ahi.z, alo.z - nhi.z) - band_abs, 0.f);
        float d2 = gx * gx + gy * gy + gz * gz;
        float tmax = fmaxf(thr_own, nlo.w * nlo.w * 1.000001f);
        return !(d2 > tmax * 1.00001f);
    };
    __shared__ u32 s_near[kNear][128]; // the first places of the lanes' stacks, a bank each
    u32 far[kStack - kNear];
    int top = 0;
    bool ok = true;
    RangeWriter w(ent, t.reduc, base, cap);
    u32 n = test(0, rlo, rhi) && keep(rlo, rhi) ? 0u : kNone;
    while (n != kNone) {
        u32 next = kNone;
        if (n >= offn) {
            w.add(n - offn, n - offn + 1);
        } else {
            const F8 bl = ldg256(&rec[n].l), br = ldg256(&rec[n].r);
            const u32 li = __float_as_uint(bl.b.w), ri = __float_as_uint(br.b.w);
            const bool pl = test(li, bl.a, bl.b) && keep(bl.a, bl.b);
            const bool pr = test(ri, br.a, br.b) && keep(br.a, br.b);
            if (top + 2 > kStack) {
                ok = false;
                break;
            }
            if (pl && pr) {
                if (top < kNear) s_near[top][threadIdx.x] = ri;
                else far[top - kNear] = ri;
                top++;
            }
            next = pl ? li : (pr ? ri : kNone);
        }
        if (next == kNone && top > 0) {
            top--;
            next = top < kNear ? s_near[top][threadIdx.x] : far[top - kNear];
        }
        n = next;
    }
    w.flush();
    const u32 c = w.c;
    if (!ok) atomicOr(&sc->flags, kFlagStackOverflow);
    if (c > cap) {
        atomicOr(&sc->flags, kFlagLeafCap);
        atomicMax(&sc->leaf_cnt_max, c);
    }
    cnt[l] = c;
    off[l] = base;
}

// ---- stage 1 on the 8-ary hierarchy over the leaves (LevelPlan), FP32 boxes
// The criterion grows with the boxes and radii (rounding is monotonic), so every leaf that
// passes lies below nodes that pass, whatever the hierarchy; this one needs no pointers, its
// eight children are 256 consecutive bytes, and eight lanes test them together.
struct WideTree {
    const NodeBoxF *level[kWideLevels];
    u32 n[kWideLevels];
    int top;
};

// Stage 1 for few leaves: eight lanes walk the hierarchy for one leaf, testing a node's eight children per
// step; the children that pass are a byte of a 64-bit mask per level, so the next node in
// ascending order is its lowest bit and the walk needs no stack.  Inner nodes pass unless
// no owned row can pair with anything below them; leaves are decided as in LeafCrit too.
// Twice the instructions per leaf of k_leaf_lists (the eights of leaves follow the Morton
// curve, so their boxes are looser than the tree's), but a quarter of its dependent loads
// and eight times its warps.
// A leaf owning no row gets an empty list, and a candidate leaf that no owned row can pair
// with is dropped (leaf_thr, see k_owner; the cache is unchanged).
__global__ void __launch_bounds__(128) k_leaf_lists_wide(TreeView t, const NodeBoxF *__restrict__ fb,
                                                         WideTree wt, u32 *__restrict__ cnt,
                                                         u32 *__restrict__ off,
                                                         uint2 *__restrict__ ent, u32 cap, Scalars *sc,
                                                         const u32 *__restrict__ leaf_thr) {
    const u32 g = threadIdx.x & 7u, shift = threadIdx.x & 24u;
    const u32 l = (blockIdx.x * 128 + threadIdx.x) / 8;
    const u32 base = l * cap;
    const u32 tb   = l < t.L ? leaf_thr[l] : 0; // 0: no row is owned by this leaf
    const float thr_own = __uint_as_float(tb);
    LazyLeafCrit crit(t, l < t.L ? l : 0);
    const F8 fa = ldg256(&wt.level[0][l < t.L ? l : 0]), fr = ldg256(&fb[0]);
    const float4 alo = fa.a, ahi = fa.b, rlo = fr.a, rhi = fr.b;
    float M = fmaxf(fmaxf(fmaxf(fabsf(rlo.x), fabsf(rlo.y)), fmaxf(fabsf(rlo.z), fabsf(rhi.x))),
                    fmaxf(fabsf(rhi.y), fabsf(rhi.z)));
    float band_abs = 1e-6f * M;
    // Every row owned by this leaf lies in its box, so a pair (a, b) with b below a node has
    // r_ab at least the Euclidean gap D between the boxes.  With thr_own >= thr_a of every
    // owned row and (r_node R)^2 >= thr_b, D^2 > max of the two makes every pair test below
    // the node fail.  The FP32 gaps are shrunk by the rounding band and the bound carries a
    // 1e-5 margin, so the skip is certain.
    auto apart = [&](const float4 &nlo, const float4 &nhi) -> bool {
        float gx = fmaxf(fmaxf(nlo.x - ahi.x, alo.x - nhi.x) - band_abs, 0.f);
        float gy = fmaxf(fmaxf(nlo.y - ahi.y, alo.y - nhi.y) - band_abs, 0.f);
        float gz = fmaxf(fmaxf(nlo.z - ahi.z, alo.z - nhi.z) - band_abs, 0.f);
        float d2 = gx * gx + gy * gy + gz * gz;
        float tb2 = fmaxf(thr_own, nlo.w * nlo.w * 1.000001f);
        return d2 > tb2 * 1.00001f;
    };
    // the criterion of the reference for a leaf, in FP64 inside the rounding band
    auto leaf_passes = [&](u32 leaf, const float4 &nlo, const float4 &nhi) -> bool {
        float sx = fmaxf(nlo.x - ahi.x, alo.x - nhi.x);
        float sy = fmaxf(nlo.y - ahi.y, alo.y - nhi.y);
        float sz = fmaxf(nlo.z - ahi.z, alo.z - nhi.z);
        float sm = fmaxf(fmaxf(sx, sy), sz);
        float R  = fmaxf(nlo.w, alo.w);
        float band = band_abs + 1e-6f * R;
        if (sm < R - band) return true;
        if (sm > R + band) return false;
        return crit(t.off() + leaf);
    };
    RangeWriter w(ent, t.reduc, base, cap, g == 0);
    // the node whose children are tested next: index i at level m (m = top + 1: the i-th eight
    // of the top level); pend: children still to visit, byte m - 1 for those at level m
    u32 i = 0, root = 0;
    const u32 roots = (wt.n[wt.top] + 7) / 8;
    int m    = wt.top + 1;
    u64 pend = 0;
    bool run = tb != 0;
    while (__any_sync(0xffffffffu, run)) {
        const u32 child = 8 * i + g;
        bool pass       = false;
        if (run && child < wt.n[m - 1]) {
            const F8 nb = ldg256(&wt.level[m - 1][child]);
            pass = !apart(nb.a, nb.b);
            if (m == 1 && pass) pass = leaf_passes(child, nb.a, nb.b);
        }
        u32 bits = (__ballot_sync(0xffffffffu, pass) >> shift) & 0xffu;
        if (!run) continue;
        if (m == 1) {
            while (bits) { // runs of consecutive leaves
                const u32 s = __ffs(bits) - 1, e = __ffs(~(bits >> s)) - 1;
                w.add(8 * i + s, 8 * i + s + e);
                bits &= ~(((1u << e) - 1u) << s);
            }
        } else {
            pend |= (u64) bits << (8 * (m - 2));
        }
        if (pend) {
            const int p = __ffsll((long long) pend) - 1;
            const int at = p / 8 + 1;                // level of the pending child
            i    = 8 * (i >> (3 * (at + 1 - m))) + (u32) (p & 7);
            m    = at;
            pend &= pend - 1;
        } else {
            root++;
            i   = root;
            m   = wt.top + 1;
            run = root < roots;
        }
    }
    if (l >= t.L || g != 0) return;
    w.flush();
    const u32 c = w.c;
    if (c > cap) {
        atomicOr(&sc->flags, kFlagLeafCap);
        atomicMax(&sc->leaf_cnt_max, c);
    }
    cnt[l] = c;
    off[l] = base;
}

// what a cache build accumulates into: no owned row, no threshold, no flag, no entry
__global__ void k_cache_init(u32 L, u32 *__restrict__ leaf_rows, u32 *__restrict__ head,
                             u32 *__restrict__ leaf_thr, Scalars *sc) {
    u32 l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l == 0)
        sc->flags = sc->leaf_cnt_max = sc->row_cnt_max = sc->rows_left = 0, sc->csr_entries = sc->csr_kept = 0;
    if (l >= L) return;
    leaf_rows[l] = 0;
    head[l]      = kNone;
    leaf_thr[l]  = 0;
}

// ---- rows: local particles in rank order
struct RowFlag {
    const u32 *sort_index;
    u32 n_local;
    __device__ __forceinline__ bool operator()(u32 r) const { return sort_index[r] < n_local; }
};
struct RowPlace {
    const u32 *sort_index;
    u32 *row_rank, *row_local;
    __device__ __forceinline__ void operator()(u32 r, u32 row) const {
        row_rank[row]  = r;
        row_local[row] = sort_index[r];
    }
    __device__ __forceinline__ void end(u32) const {}
};

constexpr u32 kLeafRows = 128;         // rows of a leaf that stage 2 leaves to one warp
constexpr u32 kWideRow  = 0x80000000u; // beside the owner leaf: the leaf is wide for the row

// ---- owner leaf: max leaf index whose box contains the point (inclusive bounds),
// i.e. the last leaf the reference's left-first DFS reports (NeighbourCache.cpp:419-443).
// Right-first traversal over the child-pair records (the first leaf reached is the
// largest); containment is decided in FP32 outside a rounding band, else in FP64.
// The rows of a leaf are linked up to kLeafRows: head[leaf], then next_row[row] (their order does
// not matter).  Rows of leaves that own more, and rows whose pair radius is less than a
// twentieth of the leaf's width, are left to k_part_rows, which finds them by their owner.
// leaf_thr: per leaf, the FP32 bits (rounded up) of the largest pair-test
// threshold thr_a = ((h_a htol)^2) R^2 over the rows it owns, 0 for a leaf owning none.
// The exact containment test inside the FP32 band compares the doubles' ordered bit
// patterns with integer operations (the FP64 pipe is scarce on GB300; particles lie on
// their own leaf's faces, so the band is met often).
__global__ void __launch_bounds__(128) k_owner(TreeView t, const NodeBoxF *__restrict__ fb,
                                               const NodePairF *__restrict__ rec,
                                               const u32 *__restrict__ row_rank, u32 n_rows,
                                               const f64 *__restrict__ sx, const f64 *__restrict__ sy,
                                               const f64 *__restrict__ sz, u32 *__restrict__ leaf_rows,
                                               u32 *__restrict__ head, u32 *__restrict__ next_row, u32 *__restrict__ owner,
                                               Scalars *sc, const f64 *__restrict__ sh,
                                               float h_tol_up, u32 *__restrict__ leaf_thr) {
    u32 row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= n_rows) return;
    u32 r    = row_rank[row];
    const f64 p[3] = {sx[r], sy[r], sz[r]};
    const long long op[3] = {ord64(p[0]), ord64(p[1]), ord64(p[2])};
    float px, py, pz, lo_unused;
    split64(p[0], px, lo_unused);
    split64(p[1], py, lo_unused);
    split64(p[2], pz, lo_unused);
    const F8 fr = ldg256(&fb[0]);
    float M = fmaxf(fmaxf(fmaxf(fabsf(fr.a.x), fabsf(fr.a.y)), fmaxf(fabsf(fr.a.z), fabsf(fr.b.x))),
                    fmaxf(fabsf(fr.b.y), fabsf(fr.b.z)));
    const float band = 1e-6f * M;
    auto inside = [&](u32 node, const float4 &lo, const float4 &hi) -> bool {
        float m = fminf(fminf(fminf(px - lo.x, py - lo.y), fminf(pz - lo.z, hi.x - px)),
                        fminf(hi.y - py, hi.z - pz));
        if (m > band) return true;
        if (m < -band) return false;
        f64 l64[3], h64[3], rr;
        load_box(&t.boxes[node], l64, h64, rr);
        return (ord64(l64[0]) <= op[0]) && (op[0] <= ord64(h64[0])) && (ord64(l64[1]) <= op[1])
               && (op[1] <= ord64(h64[1])) && (ord64(l64[2]) <= op[2]) && (op[2] <= ord64(h64[2]));
    };
    const u32 offn = t.off();
    u32 stack[kStack];
    int top   = 0;
    u32 found = kNone;
    if (inside(0, fr.a, fr.b)) stack[top++] = 0;
    while (top > 0) {
        const u32 n = stack[--top];
        if (n >= offn) {
            found = n - offn;
            break;
        }
        const F8 bl = ldg256(&rec[n].l), br = ldg256(&rec[n].r);
        const u32 li = __float_as_uint(bl.b.w), ri = __float_as_uint(br.b.w);
        const bool cl = inside(li, bl.a, bl.b), cr = inside(ri, br.a, br.b);
        if (top + 2 > kStack) {
            atomicOr(&sc->flags, kFlagStackOverflow);
            break;
        }
        if (cl) stack[top++] = li;
        if (cr) stack[top++] = ri;
    }
    bool wide = false; // the leaf is wide for this row (see stage 2)
    if (found == kNone) {
        atomicOr(&sc->flags, kFlagOwnerMissing); // the build stops at its next sync
        found = 0;
    } else {
        // an FP32 upper bound of thr_a = fl64(fl64(h htol)^2 R^2): every factor rounded up
        // (a float at or above a real number is at or above its nearest double)
        const float rint = __fmul_ru(__double2float_ru(sh[r]), h_tol_up);
        const float thr  = __fmul_ru(__fmul_ru(rint, rint), (float) (kRkern * kRkern));
        atomicMax(&leaf_thr[found], __float_as_uint(thr));
        const F8 lb     = ldg256(&fb[offn + found]);
        const float ext = fmaxf(fmaxf(lb.b.x - lb.a.x, lb.b.y - lb.a.y), lb.b.z - lb.a.z);
        wide            = ext * ext > 400.f * thr;
    }
    owner[row] = wide ? found | kWideRow : found;
    if (!wide) {
        const u32 at = atomicAdd(&leaf_rows[found], 1u);
        if (at < kLeafRows) next_row[row] = atomicExch(&head[found], row);
        wide = at == kLeafRows;
    }
    if (wide) sc->rows_left = 1;
}

// ---- stage 2 (NeighbourCache.cpp:492-591)
// MODE kCount: per-row count, and the count rounded up to 4 into off[] (scanned in
// place into offsets); kFill: entries at off[row]; kOnePass: entries straight into
// `cap` slots per row (off[row] = row * cap), flagging kFlagCsrCap when a row
// overflows so the host reruns the two-pass build.  Either way every row starts on a
// 16-byte boundary, so readers may fetch entries four at a time.
//
// The pair test is r^2 <= max(thr_a, thr_b), thr = ((h htol)^2) R^2 in FP64.  r^2 is
// estimated in FP32 and compared with the FP32 rounding of max(thr_a, thr_b) carried in the
// position records; outside a +-1e-5 relative band the answer is certain, inside it the
// exact FP64 test decides, so the cache is the FP64 one.
//
// A warp walks one leaf that owns up to kLeafRows rows (k_part_rows takes those of more): they
// share the leaf's candidates, so the warp expands the leaf's rank runs once, loads each
// candidate's record once, coalesced, drops those out of reach of the rows' box and keeps the
// others' positions relative to the leaf in
// shared memory; a row is then tested against 64 of them at a time and the accepted lanes are
// placed by ballots, in rank order.  Bound by instruction issue (76 % of the peak at 25 a row
// and 32 candidates).  131,072 / 1,048,576 / homogeneous 8.5 M / clustered 3 M / disc 1 M:
//   a thread per row                       181 / 1000 us / 5.57 ms / - / 1146 us
//   32 at a time, 48 registers             137 /  880    / 5.37 / 1.92 /  915
//   64 at a time, 64 registers             123 /  760    / 4.65 / 1.70 /  804
//   and the rows' box                      118 /  684    / 4.73 / 1.67 /  801
//   with a look at the leaf's row count      - /  689    / 4.85 / 1.69 /  810
// (a thread per row loads a record per candidate and row, 10 L1 wavefronts a request, and its
// lanes diverge; at 48 registers, five blocks an SM, either of the last two steps is a loss).
// Relative positions are rounded to FP32 (u = 2^-24, twice a coordinate): with S the rows'
// largest relative coordinate, a separation errs by u (4 S + 3 |d|) an axis, so r^2 of a pair
// near the threshold by u (8 sqrt(3) S / sqrt(thr) + 9) relative, and by 2.5e-14 M / sqrt(thr)
// for the hi/lo records of coordinates of size M; the threshold's own roundings add 3 u.  A row
// with S <= 10 sqrt(thr) and M <= 1e7 sqrt(thr) stays below 9.3e-6, inside the band; any other
// takes the FP64 test for every candidate.  (An ordinary leaf is a few h wide, S about
// sqrt(thr); rows for which it is wider than 20 sqrt(thr) are left to k_part_rows.  With the
// FP64 test for those too, the cache of a line of 300,000 in leaves of 64 cells took 33 ms
// instead of 8.2.  In between few rows fail: with S <= 6 sqrt(thr) here the builds of a thin
// sheet of 100,000 took 0.68 instead of 0.34 ms a step, with 10 sqrt(thr) in the owner search
// 0.53.)
enum CacheMode { kCount = 0, kFill = 1, kOnePass = 2 };

// the exact test (NeighbourCache.cpp:492-591); a call, as few candidates need it
__device__ __noinline__ bool pair_inside(const f64 *__restrict__ sx, const f64 *__restrict__ sy,
                                         const f64 *__restrict__ sz, const f64 *__restrict__ sh,
                                         f64 h_tol, u32 a, u32 b) {
    const f64 dx = __dsub_rn(sx[a], sx[b]), dy = __dsub_rn(sy[a], sy[b]), dz = __dsub_rn(sz[a], sz[b]);
    const f64 rab2   = dot3_rn(dx, dy, dz);
    const f64 rint_a = __dmul_rn(sh[a], h_tol), rint_b = __dmul_rn(sh[b], h_tol);
    const f64 thr_a  = __dmul_rn(__dmul_rn(rint_a, rint_a), kRkern * kRkern);
    const f64 thr_b  = __dmul_rn(__dmul_rn(rint_b, rint_b), kRkern * kRkern);
    return !(rab2 > thr_a && rab2 > thr_b);
}

__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// least of the lanes' floats (no NaN; -0 and 0 alike)
__device__ __forceinline__ float warp_min(float v) {
    const u32 b = __float_as_uint(v), o = b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u);
    const u32 m = __reduce_min_sync(0xffffffffu, o);
    return __uint_as_float(m ^ ((m >> 31) ? 0x80000000u : 0xffffffffu));
}

// the largest row of the build (sizes the slots of the next one) and the entries
template<int MODE>
__device__ __forceinline__ void cache_totals(u32 c_max, u64 c_sum, Scalars *sc) {
    u64 mx = block_reduce((u64) c_max, OpMaxU64{}, 0ull);
    if (threadIdx.x == 0 && mx) raise_u32(&sc->row_cnt_max, (u32) mx);
    if (MODE != kCount) {
        u64 tot = block_reduce(c_sum, OpAddU64{}, 0ull);
        if (threadIdx.x == 0) atomicAdd((unsigned long long *) &sc->csr_entries, (unsigned long long) tot);
    }
}

constexpr u32 kCandBlock = 256; // candidates of a leaf held at a time

template<int MODE>
__global__ void __launch_bounds__(256, 4) k_part_cache(
    u32 L, const u32 *__restrict__ leaf_rows, const u32 *__restrict__ head, const u32 *__restrict__ next_row,
    const u32 *__restrict__ row_rank, const u32 *__restrict__ leaf_cnt,
    const u32 *__restrict__ leaf_off, const uint2 *__restrict__ leaf_ent,
    const float4 *__restrict__ P, const f64 *__restrict__ sx, const f64 *__restrict__ sy,
    const f64 *__restrict__ sz, const f64 *__restrict__ sh, f64 h_tol, u32 *__restrict__ cnt,
    u32 *__restrict__ off, u32 *__restrict__ ent, Scalars *sc, u32 cap, u32 leaf_cap) {
    __shared__ float4 s_cand[8][kCandBlock];
    __shared__ u32 s_id[8][kCandBlock];
    const u32 lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const u32 below = (1u << lane) - 1u, upto = below | (1u << lane);
    constexpr u32 kAll = 0xffffffffu;
    float4 *cand = s_cand[wid];
    u32 *ids     = s_id[wid];
    const float lo_f = 1.f - 1e-5f, band = (1.f + 1e-5f) / (1.f - 1e-5f), big = 3e38f;
    u32 c_max = 0;
    u64 c_sum = 0;
    for (u32 l = blockIdx.x * 8 + wid; l < L; l += gridDim.x * 8) {
        u32 cur      = leaf_rows[l] <= kLeafRows ? head[l] : kNone;
        const u32 k0 = leaf_off[l], nk = min(leaf_cnt[l], leaf_cap); // (an overflowing list is rebuilt)
        while (cur != kNone) {
            // the next 32 rows at most, a lane each
            u32 row = kNone, m = 0;
            while (m < 32 && cur != kNone) {
                if (lane == m) row = cur;
                cur = next_row[cur];
                m++;
            }
            u32 ra = 0, w = 0, c = 0;
            float4 Ph = make_float4(0, 0, 0, 0), Pl = Ph;
            if (lane < m) {
                ra           = row_rank[row];
                const F8 rec = ldg256(&P[2 * (size_t) ra]);
                Ph = rec.a, Pl = rec.b;
                w = (MODE == kFill) ? off[row] : ((MODE == kOnePass) ? row * cap : 0);
            }
            const float ox = __shfl_sync(kAll, Ph.x, 0), oy = __shfl_sync(kAll, Ph.y, 0),
                        oz = __shfl_sync(kAll, Ph.z, 0);
            const float xa = __fadd_rn(__fsub_rn(Ph.x, ox), Pl.x), ya = __fadd_rn(__fsub_rn(Ph.y, oy), Pl.y),
                        za = __fadd_rn(__fsub_rn(Ph.z, oz), Pl.z), thr = Pl.w;
            float tlo, tmax; // the lower end of the band, and the rows' largest; NaN: decide in FP64
            {
                const float mine = lane < m ? fmaxf(fmaxf(fabsf(xa), fabsf(ya)), fabsf(za)) : 0.f;
                const float S    = __uint_as_float(__reduce_max_sync(kAll, __float_as_uint(mine)));
                const float M    = fmaxf(fmaxf(fabsf(Ph.x), fabsf(Ph.y)), fabsf(Ph.z));
                // S / sqrt(thr) <= 10 and M / sqrt(thr) <= 1e7
                const bool ok = S * S <= 100.f * thr && M * M <= 1e14f * thr && thr > 1e-30f;
                tlo           = ok ? thr * lo_f : __int_as_float(0x7fc00000);
                tmax          = __uint_as_float(__reduce_max_sync(kAll, lane < m && ok ? __float_as_uint(tlo) : 0u));
                if (__any_sync(kAll, lane < m && !ok)) tmax = __int_as_float(0x7fc00000);
            }
            // The rows' box.  Rounding is monotone, so for a candidate outside it every row's
            // rounded separation is at least the box's: one beyond the band of the largest
            // threshold from the box is beyond its own band from every row.
            const float lox = warp_min(lane < m ? xa : big), hix = -warp_min(lane < m ? -xa : big);
            const float loy = warp_min(lane < m ? ya : big), hiy = -warp_min(lane < m ? -ya : big);
            const float loz = warp_min(lane < m ? za : big), hiz = -warp_min(lane < m ? -za : big);
            for (u32 kb = 0; kb < nk; kb += 32) {
                const uint2 run = kb + lane < nk ? leaf_ent[k0 + kb + lane] : make_uint2(0, 0);
                const u32 len   = run.y - run.x;
                u32 end         = len;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const u32 v = __shfl_up_sync(kAll, end, o);
                    if (lane >= o) end += v;
                }
                const u32 total = __shfl_sync(kAll, end, 31), start = end - len;
                for (u32 t = 0; t < total;) {
                    // candidates that no row can pair with are dropped here
                    u32 nb = 0;
                    __syncwarp();
                    for (; t < total && nb + 32 <= kCandBlock; t += 32) {
                        // slot t + lane lies in the last run that starts at or before it
                        const u32 d    = start - t;
                        const u32 here = __reduce_or_sync(kAll, len && d < 32 ? 1u << d : 0u);
                        const u32 past = __popc(__ballot_sync(kAll, len && start < t));
                        const u32 j    = past + __popc(here & upto) - 1;
                        const u32 b    = __shfl_sync(kAll, run.x - start, j) + t + lane;
                        bool keep      = t + lane < total;
                        float4 q;
                        if (keep) {
                            const F8 rec = ldg256(&P[2 * (size_t) b]);
                            q = make_float4(__fadd_rn(__fsub_rn(rec.a.x, ox), rec.b.x),
                                            __fadd_rn(__fsub_rn(rec.a.y, oy), rec.b.y),
                                            __fadd_rn(__fsub_rn(rec.a.z, oz), rec.b.z), rec.b.w * lo_f);
                            const float gx = fmaxf(fmaxf(lox - q.x, q.x - hix), 0.f);
                            const float gy = fmaxf(fmaxf(loy - q.y, q.y - hiy), 0.f);
                            const float gz = fmaxf(fmaxf(loz - q.z, q.z - hiz), 0.f);
                            const float g2 = __fmaf_rn(gz, gz, __fmaf_rn(gy, gy, gx * gx));
                            keep           = !(g2 > max_nan(tmax, q.w) * band);
                        }
                        const u32 kept = __ballot_sync(kAll, keep), at = nb + __popc(kept & below);
                        if (keep) cand[at] = q, ids[at] = b;
                        nb += __popc(kept);
                    }
                    // the last ones are filled up far away
                    for (u32 k = nb + lane; k < ((nb + 63u) & ~63u); k += 32)
                        cand[k] = make_float4(1e30f, 1e30f, 1e30f, 0.f), ids[k] = kNone;
                    __syncwarp();
                    for (u32 r = 0; r < m; r++) {
                        const float x = __shfl_sync(kAll, xa, r), y = __shfl_sync(kAll, ya, r),
                                    z = __shfl_sync(kAll, za, r);
                        // rows decided in FP64 alone: no candidate is certain
                        const float ta = __shfl_sync(kAll, tlo, r);
                        u32 *out       = ent + __shfl_sync(kAll, w, r);
                        u32 cr         = __shfl_sync(kAll, c, r);
#pragma unroll 1
                        for (u32 t = 0; t < nb; t += 64) {
                            // 64 candidates at a time: the second 32 beyond nb are far away
                            const float4 q0 = cand[t + lane], q1 = cand[t + 32 + lane];
                            const float dx0 = x - q0.x, dy0 = y - q0.y, dz0 = z - q0.z;
                            const float dx1 = x - q1.x, dy1 = y - q1.y, dz1 = z - q1.z;
                            const float r20 = __fmaf_rn(dz0, dz0, __fmaf_rn(dy0, dy0, dx0 * dx0));
                            const float r21 = __fmaf_rn(dz1, dz1, __fmaf_rn(dy1, dy1, dx1 * dx1));
                            const float tm0 = max_nan(ta, q0.w), tm1 = max_nan(ta, q1.w);
                            const bool sure0 = r20 < tm0, open0 = !sure0 & !(r20 > tm0 * band);
                            const bool sure1 = r21 < tm1, open1 = !sure1 & !(r21 > tm1 * band);
                            u32 bits0 = __ballot_sync(kAll, sure0), bits1 = __ballot_sync(kAll, sure1);
                            if (__any_sync(kAll, open0 | open1)) {
                                const u32 rr = __shfl_sync(kAll, ra, r);
                                const u32 b0 = open0 ? ids[t + lane] : kNone, b1 = open1 ? ids[t + 32 + lane] : kNone;
                                bits0 |= __ballot_sync(kAll, b0 != kNone && pair_inside(sx, sy, sz, sh, h_tol, rr, b0));
                                bits1 |= __ballot_sync(kAll, b1 != kNone && pair_inside(sx, sy, sz, sh, h_tol, rr, b1));
                            }
                            const u32 at0 = cr + __popc(bits0 & below);
                            cr += __popc(bits0);
                            const u32 at1 = cr + __popc(bits1 & below);
                            cr += __popc(bits1);
                            if (MODE != kCount && (bits0 >> lane & 1u) && (MODE == kFill || at0 < cap)) out[at0] = ids[t + lane];
                            if (MODE != kCount && (bits1 >> lane & 1u) && (MODE == kFill || at1 < cap)) out[at1] = ids[t + 32 + lane];
                        }
                        if (lane == r) c = cr;
                    }
                }
            }
            if (lane < m) {
                if (MODE != kFill) cnt[row] = c;
                if (MODE == kCount) off[row] = (c + 3u) & ~3u;
                if (MODE == kOnePass) {
                    off[row] = w;
                    if (c > cap) atomicOr(&sc->flags, kFlagCsrCap);
                }
                c_max = max(c_max, c);
                c_sum += c;
            }
        }
    }
    cache_totals<MODE>(c_max, c_sum, sc);
}

// The rows of leaves that own more than kLeafRows, as of a clump within one Morton cell, or that
// are wide for them: two rows a warp, the candidates 32 at a time from their records, whose
// hi/lo differences need no common origin.  Caches of 20,000 particles of one cell / of condensed
// profiles r ~ u^2 and r ~ u^3 of 200,000 / of a line of 300,000 in leaves of 64 cells, in ms:
//   a thread per row                       5.2  /   4.7 /    9.9 /   32
//   a warp per leaf whatever its rows   8750    / 253   / 5610   / 2310
//   these rows two (one, four) a warp      0.88 (1.06, 1.19) / 1.9 (2.0, 1.9) / 3.8 (3.9, 4.0) / 8.2 (8.9, 8.6)
// A row here costs about twice the instructions of one above, so the line lies where a leaf's
// warp would make a tail: with it at 32 rows a lattice of 300,000 in leaves of 64 cells takes
// 0.91 instead of 0.44 ms, at 256 the profiles 2.0 and 5.2.
constexpr u32 kRowsAWarp = 2;

template<int MODE>
__global__ void __launch_bounds__(256) k_part_rows(
    const u32 *__restrict__ owner, const u32 *__restrict__ leaf_rows, u32 n_rows,
    const u32 *__restrict__ row_rank, const u32 *__restrict__ leaf_cnt,
    const u32 *__restrict__ leaf_off, const uint2 *__restrict__ leaf_ent,
    const float4 *__restrict__ P, const f64 *__restrict__ sx, const f64 *__restrict__ sy,
    const f64 *__restrict__ sz, const f64 *__restrict__ sh, f64 h_tol, u32 *__restrict__ cnt,
    u32 *__restrict__ off, u32 *__restrict__ ent, Scalars *sc, u32 cap, u32 leaf_cap) {
    const u32 lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    constexpr u32 kAll = 0xffffffffu, R = kRowsAWarp;
    const float lo_f = 1.f - 1e-5f, hi_f = 1.f + 1e-5f;
    u32 c_max = 0;
    u64 c_sum = 0;
    for (u32 i = blockIdx.x * 8 + (threadIdx.x >> 5); i < (n_rows + R - 1) / R; i += gridDim.x * 8) {
        const u32 row = R * i + lane;
        const u32 o   = lane < R && row < n_rows ? owner[row] : kNone, leaf = o & ~kWideRow;
        u32 left = __ballot_sync(kAll, o != kNone && ((o & kWideRow) || leaf_rows[leaf] > kLeafRows));
        while (left) {
            // those of one leaf, lane j the j-th row
            const u32 l    = __shfl_sync(kAll, leaf, __ffs(left) - 1);
            const u32 rows = __ballot_sync(kAll, leaf == l) & left;
            const bool mine = rows >> lane & 1u;
            left &= ~rows;
            const u32 k0 = leaf_off[l], nk = min(leaf_cnt[l], leaf_cap); // (an overflowing list is rebuilt)
            u32 ra = 0, w = 0;
            F8 own{};
            if (mine) {
                ra  = row_rank[row];
                own = ldg256(&P[2 * (size_t) ra]);
                w   = (MODE == kFill) ? off[row] : ((MODE == kOnePass) ? row * cap : 0);
                // the hi/lo records' error stays inside the band, or every candidate is decided in FP64
                const float M = fmaxf(fmaxf(fabsf(own.a.x), fabsf(own.a.y)), fabsf(own.a.z));
                if (!(M * M <= 1e16f * own.b.w && own.b.w > 1e-30f)) own.b.w = __int_as_float(0x7fc00000);
            }
            F8 a[R];
            u32 c[R] = {}, at0[R];
#pragma unroll
            for (u32 j = 0; j < R; j++) {
                auto of = [&](float v) { return __shfl_sync(kAll, v, j); };
                a[j].a  = make_float4(of(own.a.x), of(own.a.y), of(own.a.z), 0.f);
                a[j].b  = make_float4(of(own.b.x), of(own.b.y), of(own.b.z), of(own.b.w));
                at0[j]  = __shfl_sync(kAll, w, j);
            }
            for (u32 k = 0; k < nk; k++) {
                const uint2 run = leaf_ent[k0 + k];
                for (u32 b0 = run.x; b0 < run.y; b0 += 32) {
                    const u32 b     = b0 + lane;
                    const bool real = b < run.y;
                    const F8 q      = ldg256(&P[2 * (size_t) (real ? b : run.x)]);
#pragma unroll
                    for (u32 j = 0; j < R; j++) {
                        if (!(rows >> j & 1u)) continue;
                        const float dx = __fadd_rn(__fsub_rn(a[j].a.x, q.a.x), __fsub_rn(a[j].b.x, q.b.x));
                        const float dy = __fadd_rn(__fsub_rn(a[j].a.y, q.a.y), __fsub_rn(a[j].b.y, q.b.y));
                        const float dz = __fadd_rn(__fsub_rn(a[j].a.z, q.a.z), __fsub_rn(a[j].b.z, q.b.z));
                        const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx)), tm = max_nan(a[j].b.w, q.b.w);
                        bool in        = real && r2 < tm * lo_f;
                        if (__any_sync(kAll, real && !in && !(r2 > tm * hi_f))) {
                            const u32 rr = __shfl_sync(kAll, ra, j);
                            if (real && !in && !(r2 > tm * hi_f)) in = pair_inside(sx, sy, sz, sh, h_tol, rr, b);
                        }
                        const u32 bits = __ballot_sync(kAll, in), at = c[j] + __popc(bits & below);
                        if (MODE != kCount && in && (MODE == kFill || at < cap)) ent[at0[j] + at] = b;
                        c[j] += __popc(bits);
                    }
                }
            }
            u32 found = c[0];
#pragma unroll
            for (u32 j = 1; j < R; j++) found = lane == j ? c[j] : found;
            if (mine) {
                if (MODE != kFill) cnt[row] = found;
                if (MODE == kCount) off[row] = (found + 3u) & ~3u;
                if (MODE == kOnePass) {
                    off[row] = w;
                    if (found > cap) atomicOr(&sc->flags, kFlagCsrCap);
                }
                c_max = max(c_max, found);
                c_sum += found;
            }
        }
    }
    cache_totals<MODE>(c_max, c_sum, sc);
}

// ---- generic object query (CLBVHObjectIterator::rtree_for, CLBVHObjectIterator.hpp:127-169)
template<bool FILL>
__global__ void k_query(TreeView t, const f64 *__restrict__ qx, const f64 *__restrict__ qy,
                        const f64 *__restrict__ qz, u32 nq, int mode, f64 s,
                        const u32 *__restrict__ sort_index, const f64 *__restrict__ sx,
                        const f64 *__restrict__ sy, const f64 *__restrict__ sz,
                        u32 *__restrict__ counts, const u32 *__restrict__ offs, u32 *__restrict__ out,
                        u32 *__restrict__ flags) {
    u32 q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nq) return;
    f64 lo[3] = {__dadd_rn(qx[q], -s), __dadd_rn(qy[q], -s), __dadd_rn(qz[q], -s)};
    f64 hi[3] = {__dadd_rn(qx[q], s), __dadd_rn(qy[q], s), __dadd_rn(qz[q], s)};
    u32 c = 0, w = FILL ? offs[q] : 0;
    bool ok = dfs(
        t,
        [&](u32 node) {
            if (mode == 0) return true;
            f64 nl[3], nh[3], r;
            load_box(&t.boxes[node], nl, nh, r);
            for (int k = 0; k < 3; k++)
                if (!(fmin(nh[k], hi[k]) >= fmax(nl[k], lo[k]))) return false;
            return true;
        },
        [&](u32 leaf) {
            for (u32 rr = t.reduc[leaf]; rr < t.reduc[leaf + 1]; rr++) {
                bool in = true;
                if (mode == 1) {
                    f64 p[3] = {sx[rr], sy[rr], sz[rr]};
                    for (int k = 0; k < 3; k++)
                        if (!(fmin(p[k], hi[k]) >= fmax(p[k], lo[k]))) in = false;
                }
                if (in) {
                    if (FILL) out[w++] = sort_index[rr];
                    c++;
                }
            }
        });
    if (!ok) atomicOr(flags, kFlagStackOverflow);
    if (!FILL) counts[q] = c;
}

// the smallest float at or above v (host)
float up_f32(f64 v) {
    float f = (float) v;
    if ((f64) f < v) f = std::nextafter(f, INFINITY);
    return f;
}

TreeView view(const Ctx &c) {
    return TreeView{c.lchild.as<u32>(), c.rchild.as<u32>(), c.lflag.as<u8>(), c.rflag.as<u8>(),
                    c.boxes.as<NodeBox>(), c.reduc.as<u32>(), c.leaf_count};
}

} // namespace

cudaError_t build_rows(Ctx &c, u32 n_local) {
    cudaStream_t s = c.stream;
    cudaError_t e;
    u32 N = c.n_obj;
    if ((e = c.row_rank.ensure(sizeof(u32) * (size_t) n_local, s)) != cudaSuccess) return e;
    if ((e = c.row_local.ensure(sizeof(u32) * (size_t) n_local, s)) != cudaSuccess) return e;
    const u32 *si = c.sort_index.as<u32>();
    if ((e = compact(c, RowFlag{si, n_local}, RowPlace{si, c.row_rank.as<u32>(), c.row_local.as<u32>()}, N,
                     &c.d_scalars.as<Scalars>()->total2)) != cudaSuccess)
        return e;
    c.n_local = n_local;
    return cudaGetLastError();
}

cudaError_t neigh_cache_build(Ctx &c, f64 h_tol, const float4 *P) {
    cudaStream_t s = c.stream;
    cudaError_t e;
    u32 L = c.leaf_count, n = c.n_local;
    if (L == 0) {
        c.err = "neighbour cache: the tree has no leaves";
        return cudaErrorInvalidValue;
    }
    TreeView t = view(c);
    Scalars *dsc = c.d_scalars.as<Scalars>();
    if ((e = c.leaf_cnt.ensure(sizeof(u32) * (size_t) L, s)) != cudaSuccess) return e;
    if ((e = c.leaf_off.ensure(sizeof(u32) * (size_t) L, s)) != cudaSuccess) return e;
    // Stage 1 in one pass into c.leaf_cap slots per leaf; if a leaf has more candidates
    // the pass is rerun with slots that fit, or, past the slot budget, the exact
    // two-pass build runs.
    if (c.leaf_cap == 0) c.leaf_cap = kLeafCap;
    const u64 budget = c.slot_budget ? c.slot_budget : kMaxSlotBytes;
    auto slots_ok = [&](u64 rows, u32 cap, u64 esize = 4) {
        return rows * cap < 0xffffffffull && rows * cap * esize <= budget;
    };
    const bool s1_one_pass = slots_ok(L, c.leaf_cap, sizeof(uint2));
    // FP32 node boxes and the child-pair records the traversals read (the FP64 boxes
    // decide inside the rounding band), made with the boxes
    const NodeBoxF *fb = c.fboxes.as<NodeBoxF>();
    const NodePairF *rec = c.fpairs.as<NodePairF>();
    // Stage 1 on the 8-ary hierarchy (built with the boxes) while the leaves
    // that own rows (their share is about the rows' share of the particles) would leave an SM
    // fewer than 320 threads of the binary walk, a chain of dependent loads: 119 us for 1,399
    // leaves and 178 us for 35,981, 26,000 of them owners, against 34 and 135 us; 84,255
    // leaves with 29,000 owners 368 against 212, 50,404 owners of a disc 338 against 280.
    // From about 50,000 owners on its throughput wins (60,000 in a Sedov state 210 against
    // 255 us, 75,000 in a disc 379 against 393).
    const bool wide = (u64) L * n <= 320ull * c.sms * c.n_obj;
    const LevelPlan lp = level_plan(L);
    WideTree wt{};
    wt.top = lp.top;
    for (int m = 0; m <= lp.top; m++) {
        wt.level[m] = m ? c.wboxes.as<NodeBoxF>() + lp.at[m] : fb + (L - 1);
        wt.n[m]     = lp.n[m];
    }
    // Owner leaves first: they also record, per leaf, the largest threshold of the rows
    // it owns, which lets stage 1 drop leaves that no owned row can pair with (and skip
    // leaves that own no row); the cache is unchanged.
    if ((e = c.leaf_rows.ensure(sizeof(u32) * (size_t) L, s)) != cudaSuccess) return e;
    if ((e = c.leaf_head.ensure(sizeof(u32) * (size_t) L, s)) != cudaSuccess) return e;
    if ((e = c.next_row.ensure(sizeof(u32) * (size_t) n, s)) != cudaSuccess) return e;
    if ((e = c.owner.ensure(sizeof(u32) * (size_t) n, s)) != cudaSuccess) return e;
    if ((e = c.leaf_thr.ensure(sizeof(u32) * (size_t) L, s)) != cudaSuccess) return e;
    u32 *leaf_thr = c.leaf_thr.as<u32>();
    { k_cache_init<<<div_up(L, 256), 256, 0, s>>>(L, c.leaf_rows.as<u32>(), c.leaf_head.as<u32>(), leaf_thr, dsc); GBSPH_COUNTED; }
    if (n) {
        ProfScope ps(c, kProfOwner, n);
        { k_owner<<<div_up(n, 128), 128, 0, s>>>(t, fb, rec, c.row_rank.as<u32>(), n, c.sx.as<f64>(),
                                               c.sy.as<f64>(), c.sz.as<f64>(), c.leaf_rows.as<u32>(), c.leaf_head.as<u32>(), c.next_row.as<u32>(),
                                               c.owner.as<u32>(), dsc, c.sh.as<f64>(), up_f32(h_tol), leaf_thr); GBSPH_COUNTED; }
    }
    auto stage1 = [&]() -> cudaError_t {
        cudaError_t err = c.leaf_ent.ensure(sizeof(uint2) * ((size_t) L * c.leaf_cap + 1), s);
        if (err != cudaSuccess) return err;
        ProfScope ps(c, kProfStage1, L);
        if (wide) {
            k_leaf_lists_wide<<<div_up(L, 16), 128, 0, s>>>(t, fb, wt, c.leaf_cnt.as<u32>(), c.leaf_off.as<u32>(),
                                                           c.leaf_ent.as<uint2>(), c.leaf_cap, dsc, leaf_thr); GBSPH_COUNTED;
        } else {
            k_leaf_lists<<<div_up(L, 128), 128, 0, s>>>(t, fb, rec, c.leaf_cnt.as<u32>(), c.leaf_off.as<u32>(),
                                                       c.leaf_ent.as<uint2>(), c.leaf_cap, dsc, leaf_thr); GBSPH_COUNTED;
        }
        return cudaGetLastError();
    };
    if (s1_one_pass) {
        if ((e = stage1()) != cudaSuccess) return e;
    } else {
        // slots beyond the budget: flag the overflow so the exact build below runs
        const u32 ovf = kFlagLeafCap;
        if ((e = cudaMemcpyAsync(&dsc->flags, &ovf, sizeof(u32), cudaMemcpyHostToDevice, s)) != cudaSuccess) return e;
        if ((e = cudaMemcpyAsync(&dsc->leaf_cnt_max, &c.leaf_cap, sizeof(u32), cudaMemcpyHostToDevice, s)) != cudaSuccess) return e;
    }
    if ((e = c.csr_cnt.ensure(sizeof(u32) * ((size_t) n + 1), s)) != cudaSuccess) return e;
    if ((e = c.csr_off.ensure(sizeof(u32) * ((size_t) n + 1), s)) != cudaSuccess) return e;
    // the padded one-pass layout needs row * cap to fit the u32 offsets
    if (c.row_cap == 0) c.row_cap = kRowCap;
    auto slots_fit = [&](u32 cap) { return slots_ok(n, cap); };
    // slots that no longer fit (more rows than before): size them from the largest row
    // of the last build, with a quarter of margin, before falling back to two passes
    if (!slots_fit(c.row_cap) && c.row_seen > 0) {
        const u32 cap = (c.row_seen + c.row_seen / 4 + 7u) & ~3u;
        if (cap < c.row_cap && slots_fit(cap)) c.row_cap = cap;
    }
    bool one_pass = slots_fit(c.row_cap);
    if (one_pass)
        if ((e = c.csr_ent.ensure(sizeof(u32) * ((size_t) n * c.row_cap + 4), s)) != cudaSuccess) return e;
    // launch helper for the stage-2 kernel family: a warp per leaf, in six times the four
    // blocks that an SM holds (41 KB of candidates each; with one such grid the leaves'
    // uneven work leaves a tail of 10 %, with a block per eight leaves the blocks' atomics
    // on the totals, 10 ns each, take longer than the build)
    u32 leaf_slots = c.leaf_cap; // no bound for the lists of the exact stage 1
    auto part_rows = [&](auto mode_tag, u32 *cnt, u32 *off, u32 *ent) {
        constexpr int MODE = decltype(mode_tag)::value;
        { k_part_rows<MODE><<<std::min(div_up(n, 8 * kRowsAWarp), 24 * c.sms), 256, 0, s>>>(
            c.owner.as<u32>(), c.leaf_rows.as<u32>(), n, c.row_rank.as<u32>(),
            c.leaf_cnt.as<u32>(), c.leaf_off.as<u32>(), c.leaf_ent.as<uint2>(), P, c.sx.as<f64>(),
            c.sy.as<f64>(), c.sz.as<f64>(), c.sh.as<f64>(), h_tol, cnt, off, ent, dsc, c.row_cap, leaf_slots); GBSPH_COUNTED; }
    };
    auto part = [&](auto mode_tag, u32 *cnt, u32 *off, u32 *ent) {
        constexpr int MODE = decltype(mode_tag)::value;
        const u32 blocks   = std::min(div_up(L, 8), 24 * c.sms);
        { k_part_cache<MODE><<<blocks, 256, 0, s>>>(
            L, c.leaf_rows.as<u32>(), c.leaf_head.as<u32>(), c.next_row.as<u32>(), c.row_rank.as<u32>(),
            c.leaf_cnt.as<u32>(), c.leaf_off.as<u32>(), c.leaf_ent.as<uint2>(), P, c.sx.as<f64>(),
            c.sy.as<f64>(), c.sz.as<f64>(), c.sh.as<f64>(), h_tol, cnt, off, ent, dsc, c.row_cap, leaf_slots); GBSPH_COUNTED; }
    };
    using OnePass = std::integral_constant<int, kOnePass>;
    using Count   = std::integral_constant<int, kCount>;
    using Fill    = std::integral_constant<int, kFill>;
    // all: with the rows left to k_part_rows
    auto stage2 = [&](bool all) -> cudaError_t {
        if (!n || !one_pass) return cudaSuccess;
        ProfScope ps(c, kProfCacheFill, n);
        part(OnePass{}, c.csr_cnt.as<u32>(), c.csr_off.as<u32>(), c.csr_ent.as<u32>());
        if (all) part_rows(OnePass{}, c.csr_cnt.as<u32>(), c.csr_off.as<u32>(), c.csr_ent.as<u32>());
        return cudaGetLastError();
    };
    // Stage 2 follows at once: a list that overflowed its slots is read up to its slots only,
    // and both stages run again.  Whether rows are left to k_part_rows is read with the flags.
    if (s1_one_pass && (e = stage2(false)) != cudaSuccess) return e;
    if ((e = sync_scalars(c)) != cudaSuccess) return e;
    if (c.h_scalars->flags & (kFlagStackOverflow | kFlagOwnerMissing)) {
        c.err = "neighbour cache: tree traversal failed (stack overflow or particle outside every leaf box)";
        return cudaErrorUnknown;
    }
    c.leaf_csr_total = 0;
    if (c.h_scalars->flags & kFlagLeafCap) {
        const u32 cap = (c.h_scalars->leaf_cnt_max + 31u) & ~31u;
        const bool fits = s1_one_pass && slots_ok(L, cap, sizeof(uint2));
        if ((e = cudaMemsetAsync(&dsc->flags, 0, sizeof(u32), s)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(&dsc->row_cnt_max, 0, sizeof(u32), s)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(&dsc->csr_entries, 0, sizeof(u64), s)) != cudaSuccess) return e;
        if (fits) {
            // one pass again with slots that hold the largest list
            c.leaf_cap = leaf_slots = cap;
            if ((e = stage1()) != cudaSuccess) return e;
        } else {
            // exact two-pass build
            ProfScope ps(c, kProfStage1, 0);
            { k_leaf_count<<<div_up(L, 128), 128, 0, s>>>(t, c.leaf_cnt.as<u32>(), &dsc->flags); GBSPH_COUNTED; }
            if ((e = scan_exclusive_u32(c.leaf_cnt.as<u32>(), c.leaf_off.as<u32>(), L, &dsc->total,
                                        c.scan_scratch, s)) != cudaSuccess)
                return e;
            if ((e = sync_scalars(c)) != cudaSuccess) return e;
            c.leaf_csr_total = c.h_scalars->total;
            leaf_slots       = 0xffffffffu;
            if ((e = c.leaf_ent.ensure(sizeof(uint2) * (c.leaf_csr_total + 1), s)) != cudaSuccess) return e;
            { k_leaf_fill<<<div_up(L, 128), 128, 0, s>>>(t, c.leaf_off.as<u32>(), c.leaf_ent.as<uint2>()); GBSPH_COUNTED; }
        }
        // stage 2 ran over cut lists, or not at all
        if ((e = stage2(true)) != cudaSuccess) return e;
        if ((e = sync_scalars(c)) != cudaSuccess) return e;
    } else if (c.h_scalars->rows_left && one_pass) {
        ProfScope ps(c, kProfCacheFill, 0);
        part_rows(OnePass{}, c.csr_cnt.as<u32>(), c.csr_off.as<u32>(), c.csr_ent.as<u32>());
        if ((e = sync_scalars(c)) != cudaSuccess) return e;
    }
    c.csr_total = c.h_scalars->csr_entries;
    if (n && one_pass && (c.h_scalars->flags & kFlagCsrCap)) {
        // a row overflowed: one pass again with slots that hold the largest row
        const u32 cap = (c.h_scalars->row_cnt_max + 3u) & ~3u;
        if (slots_fit(cap)) {
            c.row_cap = cap;
            if ((e = c.csr_ent.ensure(sizeof(u32) * ((size_t) n * cap + 4), s)) != cudaSuccess) return e;
            if ((e = cudaMemsetAsync(&dsc->csr_entries, 0, sizeof(u64), s)) != cudaSuccess) return e;
            if ((e = cudaMemsetAsync(&dsc->flags, 0, sizeof(u32), s)) != cudaSuccess) return e;
            {
                ProfScope ps(c, kProfCacheFill, n);
                part(OnePass{}, c.csr_cnt.as<u32>(), c.csr_off.as<u32>(), c.csr_ent.as<u32>());
                part_rows(OnePass{}, c.csr_cnt.as<u32>(), c.csr_off.as<u32>(), c.csr_ent.as<u32>());
            }
            if ((e = sync_scalars(c)) != cudaSuccess) return e;
            c.csr_total = c.h_scalars->csr_entries;
        } else {
            one_pass = false;
        }
    }
    if (n && (!one_pass || (c.h_scalars->flags & kFlagCsrCap))) {
        // slots beyond the budget: exact two-pass build into a compact CSR
        {
            ProfScope ps(c, kProfCacheCount, n);
            part(Count{}, c.csr_cnt.as<u32>(), c.csr_off.as<u32>(), nullptr);
            part_rows(Count{}, c.csr_cnt.as<u32>(), c.csr_off.as<u32>(), nullptr);
        }
        // rows padded to multiples of 4 entries, scanned in place
        if ((e = scan_exclusive_u32(c.csr_off.as<u32>(), c.csr_off.as<u32>(), n, &dsc->total,
                                    c.scan_scratch, s)) != cudaSuccess)
            return e;
        if ((e = cudaMemsetAsync(&dsc->csr_entries, 0, sizeof(u64), s)) != cudaSuccess) return e;
        if ((e = sync_scalars(c)) != cudaSuccess) return e;
        u64 padded = c.h_scalars->total;
        if ((e = c.csr_ent.ensure(sizeof(u32) * (padded + 4), s)) != cudaSuccess) return e;
        {
            ProfScope ps(c, kProfCacheFill, 0);
            part(Fill{}, nullptr, c.csr_off.as<u32>(), c.csr_ent.as<u32>());
            part_rows(Fill{}, nullptr, c.csr_off.as<u32>(), c.csr_ent.as<u32>());
        }
        if ((e = sync_scalars(c)) != cudaSuccess) return e;
        c.csr_total = c.h_scalars->csr_entries;
    }
    c.row_seen    = c.h_scalars->row_cnt_max;
    c.cache_valid = true;
    return cudaGetLastError();
}

cudaError_t tree_query(Ctx &c, const f64 *qx, const f64 *qy, const f64 *qz, u32 nq, int mode,
                       f64 s, u32 *counts, u32 *offsets, u32 *out, bool fill) {
    TreeView t = view(c);
    Scalars *dsc = c.d_scalars.as<Scalars>();
    if (fill)
        { k_query<true><<<div_up(nq, 128), 128, 0, c.stream>>>(
            t, qx, qy, qz, nq, mode, s, c.sort_index.as<u32>(), c.sx.as<f64>(), c.sy.as<f64>(),
            c.sz.as<f64>(), nullptr, offsets, out, &dsc->flags); GBSPH_COUNTED; }
    else
        { k_query<false><<<div_up(nq, 128), 128, 0, c.stream>>>(
            t, qx, qy, qz, nq, mode, s, c.sort_index.as<u32>(), c.sx.as<f64>(), c.sy.as<f64>(),
            c.sz.as<f64>(), counts, nullptr, nullptr, &dsc->flags); GBSPH_COUNTED; }
    return cudaGetLastError();
}

} // namespace gbsph
