// FP64 SPH pair kernels and integrator.  This translation unit is compiled with
// fused multiply-add disabled so that every expression rounds exactly as the cited
// reference line (and the oracle) evaluates it; the FP64 path is bit-identical to
// the oracle for the same neighbour order.
//
//   h-rho Newton step  shammodels/sph/src/modules/IterateSmoothingLengthDensity.cpp:52-119
//                      shammodels/sph/include/shammodels/sph/math/density.hpp:22-41
//   Omega              shammodels/sph/src/modules/ComputeOmega.cpp:36-73
//   EOS (adiabatic)    shammodels/sph/src/modules/ComputeEos.cpp:162-172,219-236
//   derivatives        shammodels/sph/src/modules/UpdateDerivs.cpp:176-271,
//                      shammodels/sph/include/shammodels/sph/math/forces.hpp:24-226, q_ab.hpp:36-39
//   v_sig              shammodels/sph/src/Solver.cpp:2716-2788
//   CFL                ComputeCFLCourant.hpp:45-60, ComputeCFLForce.hpp:50-62
//   corrector          shamrock/src/math/integrators.cpp:88-120, Solver.cpp:2506-2616
//   predictor + wrap   Solver.cpp:390-524, ForwardEuler.hpp:62-84, integrators.cpp:207-237

#include "gbsph_ctx.cuh"
#include "lean64.cuh"
#include "sph_kernels.cuh"

#include <algorithm>

namespace gbsph {

namespace {

// ---------------------------------------------------------------- M4 (FP64)
__device__ __forceinline__ f64 m4_f(f64 q) {
    f64 t1 = 2 - q;
    f64 t2 = 1 - q;
    t1     = t1 * t1 * t1;
    t2     = t2 * t2 * t2;
    const f64 div1_4 = (1. / 4.);
    t1 *= div1_4;
    t2 *= -1;
    if (q < 1) return t1 + t2;
    else if (q < 2) return t1;
    return 0;
}
__device__ __forceinline__ f64 m4_df(f64 q) {
    const f64 div9_4 = (9. / 4.);
    const f64 div3_4 = (3. / 4.);
    if (q < 1) return -3 * q + div9_4 * q * q;
    else if (q < 2) return -3 + 3 * q - div3_4 * q * q;
    return 0;
}
__device__ __forceinline__ f64 W_3d(f64 r, f64 h) { return kNorm3d * m4_f(r / h) / (h * h * h); }
__device__ __forceinline__ f64 dW_3d(f64 r, f64 h) {
    return kNorm3d * m4_df(r / h) / (h * h * h * h);
}
__device__ __forceinline__ f64 dhW_3d(f64 r, f64 h) {
    return -(kNorm3d) * (3 * m4_f(r / h) + (r / h) * m4_df(r / h)) / (h * h * h * h);
}
__device__ __forceinline__ f64 rho_h(f64 m, f64 h) {
    return m * (kHfact / h) * (kHfact / h) * (kHfact / h);
}
__device__ __forceinline__ f64 inv_sat_positive(f64 v) { return (v >= 1e-9) ? 1. / v : 0.; }
__device__ __forceinline__ f64 inv_sat_zero(f64 v) { return (v != 0 && v == v) ? 1. / v : 0.; }

// M4 and its derivative at q >= 0 in the expressions above with fewer FP64 instructions:
// both pieces share their products (their difference is signs and constants), comparisons
// and exact scalings act on the bits.
__device__ __forceinline__ f64 quarter(f64 v) { return from64(bits64(v) - (2ull << 52)); } // |v| > 2^-1020
__device__ __forceinline__ f64 lean_m4_f(f64 q) {
    f64 t1 = 2 - q;
    f64 t2 = 1 - q;
    t1     = mul64i(mul64i(t1, t1), t1);
    t2     = mul64i(mul64i(t2, t2), t2);
    t1     = quarter(t1); // not zero below q = 2
    const u32 hq = hi64(q);
    const f64 t  = t1 - t2;
    return hq < 0x3FF00000u ? t : (hq < 0x40000000u ? t1 : 0.0);
}
__device__ __forceinline__ f64 lean_m4_df(f64 q) {
    const u32 hq  = hi64(q);
    const bool in = hq < 0x3FF00000u;
    const f64 t = mul64i(3.0, q), u = t - 3;
    const f64 s = mul64i(mul64i(in ? 9. / 4. : -3. / 4., q), q);
    const f64 v = (in ? -t : u) + s;
    return hq < 0x40000000u ? v : 0.0;
}

// FP32 pre-test of a row's pairs from coordinates cut to floats: certainly inside or
// outside a support radius away from a band about it.  Cutting moves a separation by at
// most 2^-22 of the coordinates and r^2 / thr by four times that over the radius; rows
// whose band would not be narrow (or whose radius leaves the float range) decide every
// pair in FP64.
struct RowCut {
    float x, y, z, thr, lo, hi;
    __device__ __forceinline__ RowCut(f64 xa, f64 ya, f64 za, f64 h) {
        x = cut32(xa), y = cut32(ya), z = cut32(za);
        const float r   = 2.f * cut32(h);
        const float M   = fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z));
        const float eps = 2e-6f + 9.6e-7f * (M / r + 1.f);
        thr             = r * r;
        const bool ok   = thr > 1e-30f && thr < 1e30f && eps < 0.05f;
        lo = ok ? 1.f - eps : -1.f;
        hi = ok ? 1.f + eps : __int_as_float(0x7f800000);
    }
    __device__ __forceinline__ float r2(f64 xb, f64 yb, f64 zb) const {
        const float dx = x - cut32(xb), dy = y - cut32(yb), dz = z - cut32(zb);
        return dx * dx + dy * dy + dz * dz;
    }
};

// r^2 of a pair inside the band (a call, so that the walk executes its FP64 for those alone)
__device__ __noinline__ f64 pair_r2(f64 xa, f64 ya, f64 za, f64 xb, f64 yb, f64 zb) {
    const f64 dx = xa - xb, dy = ya - yb, dz = za - zb;
    return dx * dx + dy * dy + dz * dz;
}

// ---------------------------------------------------------------- density sums
// The pair terms of one row at h_a, with the plain operators
__device__ __noinline__ void density_pair_plain(f64 rab2, f64 h_a, f64 &w, f64 &dw) {
    const f64 rab = sqrt(rab2);
    w             = W_3d(rab, h_a);
    dw            = dhW_3d(rab, h_a);
}

// Called by all 32 lanes of a warp (a lane without work passes k0 = k1).  FP64 instructions
// bound this loop (two lanes per clock and SM), so a lane first walks to its next pair
// inside the support in FP32 and all lanes then evaluate one together, with the quotients
// and the root of lean64.cuh: 44 FP64 instructions per pair instead of about 65, and none
// for the cached pairs outside the support.
__device__ __forceinline__ void density_sums(const RowSpace &rs, u32 a, u32 k0, u32 k1, f64 h_a,
                                             f64 pmass, f64 &rho_sum, f64 &sumdWdh) {
    f64 xa = rs.x[a], ya = rs.y[a], za = rs.z[a];
    f64 dint = h_a * h_a * kRkern * kRkern;
    const RowCut cut(xa, ya, za, h_a);
    const Denominator H = denominator(h_a), H3 = denominator(h_a * h_a * h_a),
                      H4 = denominator(h_a * h_a * h_a * h_a);
    rho_sum  = 0;
    sumdWdh  = 0;
    u32 k    = k0;
    while (true) {
        f64 xb = 0, yb = 0, zb = 0;
        bool have = false;
        while (k < k1) {
            const u32 b = rs.ent[k++];
            xb = rs.x[b], yb = rs.y[b], zb = rs.z[b];
            const float r2 = cut.r2(xb, yb, zb);
            if (r2 > cut.thr * cut.hi) continue;
            if (!(r2 < cut.thr * cut.lo) && pair_r2(xa, ya, za, xb, yb, zb) > dint) continue;
            have = true;
            break;
        }
        if (!__any_sync(0xffffffffu, have)) break;
        if (!have) continue;
        const f64 dx = xa - xb, dy = ya - yb, dz = za - zb;
        const f64 rab2 = mul64i(dx, dx) + mul64i(dy, dy) + mul64i(dz, dz);
        bool bad     = false;
        const Root r = root64(rab2, bad);
        const bool zero = zero64(bits64(rab2));
        bad             = bad && !zero;
        const f64 rab = zero ? 0.0 : root_value(r);
        const f64 q   = divide_by(rab, H, bad);
        const f64 f = lean_m4_f(q), df = lean_m4_df(q);
        f64 w  = divide_by(mul64i(kNorm3d, f), H3, bad);
        f64 dw = divide_by(mul64i(-(kNorm3d), mul64i(3.0, f) + mul64i(q, df)), H4, bad);
        if (bad) density_pair_plain(rab2, h_a, w, dw);
        rho_sum += mul64i(pmass, w);
        sumdWdh += mul64i(pmass, dw);
    }
}

// ITERS Newton iterations per row (the reference's global loop is equivalent per
// particle: a particle's update reads only its own h, so it iterates until its own
// eps <= eps_p (1e-6 in the reference), becomes -1, or the iteration cap is reached).
// The rows of a warp iterate together until the last of them is done.
__global__ void __launch_bounds__(128, 7) k_h_iterate(RowSpace rs, const f64 *__restrict__ h_old,
                                                   f64 *__restrict__ h_new, f64 *__restrict__ eps,
                                                   f64 pmass, f64 h_evol_max, f64 h_evol_iter_max,
                                                   u32 iters, f64 eps_p, Scalars *sc) {
    const u32 t      = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = t < rs.n;
    u64 emax = 0, emin = ~0ull;
    u32 used = 0;
    u32 a = 0, k0 = 0, k1 = 0;
    f64 ha_0 = 1, h_a = 1, e = 0;
    if (valid) {
        a    = rs.row_rank ? rs.row_rank[t] : t;
        k0   = rs.off[t];
        k1   = k0 + rs.cnt[t];
        ha_0 = h_old[t];
        h_a  = h_new[t];
        e    = eps[t];
    }
    const f64 h_max_tot_max_evol = h_evol_max;
    const f64 h_max_evol_p       = h_evol_iter_max;
    const f64 h_max_evol_m       = 1 / h_evol_iter_max;
    for (u32 it = 0; it < iters; it++) {
        const bool go = valid && e > eps_p;
        if (!__any_sync(0xffffffffu, go)) break;
        f64 rho_sum, sumdWdh;
        density_sums(rs, a, k0, go ? k1 : k0, h_a, pmass, rho_sum, sumdWdh);
        if (!go) continue;
        used++;
        f64 rho_ha  = rho_h(pmass, h_a);
        f64 f_iter  = rho_sum - rho_ha;
        f64 df_iter = sumdWdh + 3 * rho_ha / h_a;
        f64 new_h   = h_a - f_iter / df_iter;
        if (new_h < h_a * h_max_evol_m) new_h = h_max_evol_m * h_a;
        if (new_h > h_a * h_max_evol_p) new_h = h_max_evol_p * h_a;
        if (new_h < ha_0 * h_max_tot_max_evol) {
            e   = fabs(new_h - h_a) / ha_0;
            h_a = new_h;
        } else {
            h_a = ha_0 * h_max_tot_max_evol;
            e   = -1;
        }
    }
    if (valid) {
        h_new[t] = h_a;
        eps[t]   = e;
        emax     = f64_to_ordered(e);
        emin     = emax;
    }
    emax = block_reduce(emax, OpMaxU64{}, 0ull);
    emin = block_reduce(emin, OpMinU64{}, ~0ull);
    u32 um = block_reduce((u64) used, OpMaxU64{}, 0ull);
    if (threadIdx.x == 0) {
        raise_u64(&sc->eps_max, emax);
        lower_u64(&sc->eps_min, emin);
        raise_u32(&sc->iters_max, um);
    }
}

__global__ void __launch_bounds__(128, 6) k_omega(RowSpace rs, const f64 *__restrict__ h_row,
                                               f64 pmass, f64 *__restrict__ omega_out,
                                               const u32 *__restrict__ out_index) {
    const u32 t      = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = t < rs.n;
    u32 a = 0, k0 = 0, k1 = 0;
    f64 h_a = 1;
    if (valid) {
        a   = rs.row_rank ? rs.row_rank[t] : t;
        k0  = rs.off[t];
        k1  = k0 + rs.cnt[t];
        h_a = h_row[t];
    }
    f64 rho_sum, part_omega_sum;
    density_sums(rs, a, k0, k1, h_a, pmass, rho_sum, part_omega_sum);
    if (!valid) return;
    f64 rho_ha  = rho_h(pmass, h_a);
    f64 omega_a = 1 + (h_a / (3 * rho_ha)) * part_omega_sum;
    omega_out[out_index ? out_index[t] : t] = omega_a;
}

// Five 32-byte records per particle, in arrays of their own of N records each, that the
// FP64 pair loops read with one 256-bit load apiece:
//   0 {x, y, z, h}   1 {vx, vy, vz, u}   2 {P, alpha c_s, -rho / 2, inv_sat_zero(rho^2 Omega)}
//   3 {rho, rho Omega, y(rho Omega), y(h)}   4 {h^4, y(h^4) | lo(h), lo(h^4), lo(rho Omega), -}
// with the reciprocals y and lo of lean64.cuh.  Every factor is the pair loop's own
// expression evaluated once per particle, so it has the same bits.
struct __align__(32) D4 {
    f64 x, y, z, w;
};
__device__ __forceinline__ D4 ldd4(const f64 *base, size_t N, u32 rec, u32 r) {
    const F8 v  = ldg256(base + 4 * (rec * N + r));
    auto two    = [](float lo, float hi) { return __hiloint2double(__float_as_int(hi), __float_as_int(lo)); };
    return D4{two(v.a.x, v.a.y), two(v.a.z, v.a.w), two(v.b.x, v.b.y), two(v.b.z, v.b.w)};
}
__device__ __forceinline__ void std4(f64 *base, size_t N, u32 rec, u32 r, f64 x, f64 y, f64 z, f64 w) {
    *(D4 *) (base + 4 * (rec * N + r)) = D4{x, y, z, w};
}
__device__ __forceinline__ f64 pack_floats(float lo, float hi) {
    return __hiloint2double(__float_as_int(hi), __float_as_int(lo));
}
__device__ __forceinline__ float low_float(f64 v) { return __int_as_float(__double2loint(v)); }
__device__ __forceinline__ float high_float(f64 v) { return __int_as_float(__double2hiint(v)); }

__device__ __forceinline__ void stage_record(f64 *rec, size_t N, u32 r, f64 x, f64 y, f64 z, f64 h,
                                             f64 vx, f64 vy, f64 vz, f64 u, f64 P, f64 acs,
                                             f64 rho, f64 om) {
    const f64 rho_om    = rho * om;
    const Denominator H = denominator(h), H4 = denominator(h * h * h * h), R = denominator(rho_om);
    std4(rec, N, 0, r, x, y, z, h);
    std4(rec, N, 1, r, vx, vy, vz, u);
    std4(rec, N, 2, r, P, acs, -f64(0.5) * rho, inv_sat_zero((rho * rho) * om));
    std4(rec, N, 3, r, rho, rho_om, R.y, H.y);
    std4(rec, N, 4, r, H4.b, H4.y, pack_floats(H.lo, H4.lo), pack_floats(R.lo, 0.f));
}

// gather h, u, v, omega of locals and ghosts into rank order + the equation of state;
// alpha_AV: the constant viscosity (the varying one multiplies its alpha in later, record 2
// then holds c_s here)
__global__ void k_gather_eos(const u32 *__restrict__ sort_index, u32 N, u32 n_local,
                             const u32 *__restrict__ ghost_src, const f64 *__restrict__ h,
                             const f64 *__restrict__ u, const f64 *__restrict__ vx,
                             const f64 *__restrict__ vy, const f64 *__restrict__ vz, u32 vs,
                             const f64 *__restrict__ omega, f64 pmass, EosParams eos, f64 alpha_AV,
                             const f64 *__restrict__ sx, const f64 *__restrict__ sy,
                             const f64 *__restrict__ sz, f64 *__restrict__ scs,
                             f64 *__restrict__ rec, Scalars *sc) {
    u32 r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r == 0) reset_corrector(sc);
    if (r >= N) return;
    u32 id  = sort_index[r];
    u32 src = id < n_local ? id : ghost_src[id - n_local];
    const f64 hh = h[src], uu = u[src];
    const f64 x = sx[r], y = sy[r], z = sz[r];
    const f64 rho = rho_h(pmass, hh);
    f64 P, cs;
    if (eos.kind == 1) {
        // LP07 at the merged (rank-ordered) position
        f64 Rsq   = x * x + y * y + z * z;
        f64 cs_sq = (eos.cs0 * eos.cs0) * pow(Rsq / (eos.r0 * eos.r0), -eos.q);
        P         = cs_sq * rho;
        cs        = sqrt(cs_sq);
    } else {
        P  = (eos.gamma - 1) * rho * uu;
        cs = sqrt(eos.gamma * P / rho);
    }
    scs[r] = cs;
    stage_record(rec, N, r, x, y, z, hh, vx[(size_t) src * vs], vy[(size_t) src * vs],
                 vz[(size_t) src * vs], uu, P, alpha_AV * cs, rho, omega[src]);
}

// the same records from the module's merged arrays
__global__ void k_stage_modules(u32 N, const f64 *__restrict__ x, const f64 *__restrict__ y,
                                const f64 *__restrict__ z, HydroSpace hs, f64 pmass, f64 alpha_AV,
                                f64 *__restrict__ rec) {
    u32 r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= N) return;
    stage_record(rec, N, r, x[r], y[r], z[r], hs.h[r], hs.vx[r], hs.vy[r], hs.vz[r], hs.u[r], hs.P[r],
                 alpha_AV * hs.cs[r], rho_h(pmass, hs.h[r]), hs.omega[r]);
}

// varying viscosity: alpha c_s of record 2 from the updated per-particle alpha
__global__ void k_stage_alpha64(const u32 *__restrict__ sort_index, u32 N, u32 n_local,
                                const u32 *__restrict__ ghost_src, const f64 *__restrict__ alpha,
                                const f64 *__restrict__ scs, f64 *__restrict__ rec) {
    u32 r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= N) return;
    const u32 id  = sort_index[r];
    const u32 src = id < n_local ? id : ghost_src[id - n_local];
    rec[4 * (2 * (size_t) N + r) + 1] = alpha[src] * scs[r];
}

__global__ void k_eos_lp07(u32 n, const f64 *__restrict__ x, const f64 *__restrict__ y,
                           const f64 *__restrict__ z, u32 vs, const f64 *__restrict__ h, f64 pmass,
                           f64 cs0, f64 r0, f64 q, f64 *__restrict__ P, f64 *__restrict__ cs) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    size_t iv = (size_t) i * vs;
    f64 a = x[iv], b = y[iv], c = z[iv];
    f64 Rsq   = a * a + b * b + c * c;
    f64 cs_sq = (cs0 * cs0) * pow(Rsq / (r0 * r0), -q);
    P[i]      = cs_sq * rho_h(pmass, h[i]);
    cs[i]     = sqrt(cs_sq);
}

__global__ void k_eos(u32 n, const f64 *__restrict__ h, const f64 *__restrict__ u, f64 pmass,
                      f64 gamma, f64 *__restrict__ P, f64 *__restrict__ cs) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    f64 rho = rho_h(pmass, h[i]);
    f64 Pa  = (gamma - 1) * rho * u[i];
    P[i]    = Pa;
    cs[i]   = sqrt(gamma * Pa / rho);
}

// ---------------------------------------------------------------- derivatives
struct DerivParams {
    f64 pmass, alpha_u, beta_AV;
    f64 hdt;             // dt / 2 for the corrector
    f64 C_cour, C_force; // CFL factors (already x cfl multiplier)
    ExtAccel ext;        // external acceleration added to the hydro one (may be null)
};

// One row's particle as the pair loop keeps it, in shared memory: four lanes share a row
// and the loop has no registers to spare (a stride of 25 doubles keeps the eight rows of a
// warp in different banks)
struct Row64 {
    struct Vec4 {
        f64 x, y, z, w;
        __device__ __forceinline__ void operator=(const D4 &d) { x = d.x, y = d.y, z = d.z, w = d.w; }
    };
    Vec4 p, v, e; // records 0, 1, 2
    f64 rho, inv_rho_om, c_heat; // rho, 1 / (Omega rho), that times 1 / rho
    f64 yH, h4, yH4;             // Denominator of h and of h^4
    float loH, loH4;
    f64 pad[6];
    __device__ __forceinline__ Denominator H() const { return Denominator{p.w, yH, loH}; }
    __device__ __forceinline__ Denominator H4() const { return Denominator{h4, yH4, loH4}; }
};
static_assert(sizeof(Row64) == 25 * 8, "Row64 stride");

// the pair's contributions: force, the two du/dt terms, and v.r_hat of the forces
struct Pair64 {
    f64 fx, fy, fz, t1, t2, vr;
};

// a pair outside both supports (the exact test, a call for the pairs inside the band)
__device__ __noinline__ bool beyond_both(f64 xa, f64 ya, f64 za, f64 ha, f64 xb, f64 yb, f64 zb, f64 hb) {
    const f64 Rker2 = kRkern * kRkern;
    const f64 r2    = pair_r2(xa, ya, za, xb, yb, zb);
    return r2 > ha * ha * Rker2 && r2 > hb * hb * Rker2;
}

// v / 2 where that is exact
__device__ __forceinline__ f64 half(f64 v, bool &bad) {
    const bool zero = zero64(bits64(v));
    bad |= !zero && (hi64(v) & 0x7FFFFFFFu) - 0x00200000u >= 0x7FD00000u;
    return zero ? v : from64(bits64(v) - (1ull << 52));
}
// fmax(v, 0): 0 for NaN
__device__ __forceinline__ f64 positive(f64 v) {
    return bits64(v) - 1ull < 0x7FF0000000000000ull ? v : 0.0;
}

// (Inlined: ptxas 13.0.88 crashes on these two as calls beside the warp votes of the loop.)
// The pair terms with the plain operators (UpdateDerivs.cpp:176-271), from the records of a
// and b
__device__ __forceinline__ void force_pair_plain(const f64 *__restrict__ rec, size_t N, u32 a, u32 b,
                                              const DerivParams &p, Pair64 &o) {
    const D4 A0 = ldd4(rec, N, 0, a), A1 = ldd4(rec, N, 1, a), A2 = ldd4(rec, N, 2, a),
             A3 = ldd4(rec, N, 3, a);
    const D4 B0 = ldd4(rec, N, 0, b), B1 = ldd4(rec, N, 1, b), B2 = ldd4(rec, N, 2, b),
             B3 = ldd4(rec, N, 3, b);
    const f64 dx = A0.x - B0.x, dy = A0.y - B0.y, dz = A0.z - B0.z;
    const f64 rab = sqrt(dx * dx + dy * dy + dz * dz);
    f64 Fab_a   = dW_3d(rab, A0.w);
    f64 Fab_b   = dW_3d(rab, B0.w);
    f64 vx = A1.x - B1.x, vy = A1.y - B1.y, vz = A1.z - B1.z;
    f64 inv = inv_sat_positive(rab);
    f64 rx = dx * inv, ry = dy * inv, rz = dz * inv;
    f64 vr      = vx * rx + vy * ry + vz * rz;
    f64 bv      = p.beta_AV * fabs(vr);
    f64 vsig_a  = A2.y + bv;
    f64 vsig_b  = B2.y + bv;
    f64 rho_avg = (A3.x + B3.x) * 0.5;
    f64 vsig_u  = sqrt(fabs(A2.x - B2.x) / rho_avg);
    f64 AV_P_a  = A2.x + fmax(A2.z * vsig_a * vr, f64(0));
    f64 AV_P_b  = B2.x + fmax(B2.z * vsig_b * vr, f64(0));
    f64 ca = AV_P_a * A2.w, cb = AV_P_b * B2.w;
    f64 nax = rx * Fab_a, nay = ry * Fab_a, naz = rz * Fab_a;
    f64 nbx = rx * Fab_b, nby = ry * Fab_b, nbz = rz * Fab_b;
    f64 mb = -p.pmass;
    o.fx = mb * (ca * nax + cb * nbx);
    o.fy = mb * (ca * nay + cb * nby);
    o.fz = mb * (ca * naz + cb * nbz);
    const f64 inv_rho_om = 1 / A3.y;
    o.t1 = AV_P_a * (inv_rho_om * (1. / A3.x)) * p.pmass * (vx * nax + vy * nay + vz * naz);
    f64 Fa = Fab_a * inv_rho_om;
    f64 Fb = Fab_b / B3.y;
    o.t2 = p.pmass * p.alpha_u * vsig_u * (A1.w - B1.w) * f64(0.5) * (Fa + Fb);
    o.vr = vr;
}

// v.r_hat of the reference's separate v_sig kernel: r_hat = dr / r, zero below 1e-9
__device__ __forceinline__ f64 sig_speed_plain(const f64 *__restrict__ rec, size_t N, u32 a, u32 b) {
    const D4 A0 = ldd4(rec, N, 0, a), A1 = ldd4(rec, N, 1, a);
    const D4 B0 = ldd4(rec, N, 0, b), B1 = ldd4(rec, N, 1, b);
    const f64 dx = A0.x - B0.x, dy = A0.y - B0.y, dz = A0.z - B0.z;
    const f64 rab = sqrt(dx * dx + dy * dy + dz * dz);
    const f64 vx = A1.x - B1.x, vy = A1.y - B1.y, vz = A1.z - B1.z;
    f64 ux = dx / rab, uy = dy / rab, uz = dz / rab;
    if (rab < 1e-9) ux = uy = uz = 0;
    return fabs(vx * ux + vy * uy + vz * uz);
}

// The in-support pairs of the rows of a warp, four lanes per row: the quad tests its next
// four entries in FP32 and queues those inside in entry order until four are there (or the
// row is done); lane j then holds the j-th.
struct QuadWalk {
    u32 k, k1, n, j, q, shift;
    u32 (*queue)[8];
    __device__ __forceinline__ QuadWalk(u32 (*queue_)[8], u32 k0, u32 k1_) : k(k0), k1(k1_), n(0), queue(queue_) {
        const u32 lane = threadIdx.x & 31u;
        j = lane & 3u, q = lane >> 2, shift = lane & ~3u;
    }
    // inside(entry index) for the lane's candidate; false when the warp has no pairs left.
    // take: pairs of this round; the lane has one (entry index at) if j < take.
    template<class Inside>
    __device__ __forceinline__ bool next(Inside &&inside, u32 &take, u32 &at) {
        while (true) {
            const bool need = n < 4 && k < k1;
            if (!__any_sync(0xffffffffu, need)) break;
            bool in      = false;
            const u32 kk = k + j;
            if (need) {
                if (kk < k1) in = inside(kk);
                k += 4;
            }
            const u32 bits = (__ballot_sync(0xffffffffu, in) >> shift) & 15u;
            if (in) queue[q][n + __popc(bits & ((1u << j) - 1u))] = kk;
            n += __popc(bits);
        }
        __syncwarp();
        if (!__any_sync(0xffffffffu, n > 0)) return false;
        take           = min(n, 4u);
        at             = queue[q][j];
        const u32 rest = queue[q][4 + j];
        __syncwarp();
        queue[q][j] = rest;
        n -= take;
        return true;
    }
};

// The FP64 pair loop, called by all 32 lanes of a warp, four to a row (no row: k0 = k1).
// It is bound by the FP64 pipe (two lanes per clock and SM), so
//  - a quad first walks to its next pairs inside either support in FP32 and its lanes then
//    evaluate four of them together: none of the work goes to the quarter of the cached
//    pairs outside both supports, the pieces of M4 do not diverge and rows of different
//    lengths leave few lanes idle;
//  - quotients, roots and reciprocals are those of lean64.cuh, 33 of the 51 products run on
//    the integer pipes (mul64i; all of them there leaves the FP64 pipe waiting for the
//    other instructions: 2.04 ms against 1.75), and the neighbour's factors are staged;
//  - lane c adds component c (x, y, z, du/dt) of the four pairs in entry order.
// About 95 FP64 instructions per pair, where the plain operators take about 215: 5.12 ->
// 1.75 ms per launch at 131,072 particles of the jittered lattice.  The
// particle itself adds zeros and is skipped unless a field of the row is not finite.
// The v_sig maximum, max over the pairs of c_s + 2 |v.u| with u = dr / r: rounding is
// monotonic, so that of the largest |v.u|, which differs from the forces' v.r_hat = v.(dr
// (1/r)) by a few units in the last place of |v|.  The loop keeps the pairs whose |v.r_hat|
// could be the largest within that margin and evaluates the three quotients for those only
// (every pair of the row where more than kSigCandidates of a lane are that close).
constexpr u32 kSigCandidates = 8;
struct Warp64 {
    Row64 row[8];
    f64 x[8][4][6]; // [quad][pair]{fx, fy, fz, t1, t2, 0}
    u32 queue[8][8];
};

template<bool VSIG>
__device__ __forceinline__ void derivs_row(Warp64 &W, const u32 *__restrict__ ent,
                                           const f64 *__restrict__ rec, size_t N, u32 a, u32 k0,
                                           u32 k1, f64 cs_a, const DerivParams &p, f64 &sum,
                                           f64 &vsig_max) {
    QuadWalk walk(W.queue, k0, k1);
    const u32 j = walk.j, q = walk.q;
    Row64 &A    = W.row[q];
    bool plain_row;
    {
        const D4 r0 = ldd4(rec, N, 0, a), r1 = ldd4(rec, N, 1, a), r2 = ldd4(rec, N, 2, a),
                 r3 = ldd4(rec, N, 3, a), r4 = ldd4(rec, N, 4, a);
        const f64 iro = 1 / r3.y, heat = iro * (1. / r3.x);
        // a sum is finite only if its terms are (or cancel infinities, which gives NaN)
        const f64 all = fabs(r1.x) + fabs(r1.y) + fabs(r1.z) + fabs(r1.w) + fabs(r2.x)
                        + fabs(r2.y) + fabs(r2.z) + fabs(r2.w) + fabs(heat);
        const float lo = low_float(r4.z), lo4 = high_float(r4.z);
        plain_row = !(all < 1e300) || !(lo == lo) || !(lo4 == lo4);
        __syncwarp();
        if (j == 0) {
            A.p = r0, A.v = r1, A.e = r2;
            A.rho = r3.x, A.inv_rho_om = iro, A.c_heat = heat;
            A.yH = r3.w, A.h4 = r4.x, A.yH4 = r4.y;
            A.loH = lo, A.loH4 = lo4;
        }
        W.x[q][j][5] = 0;
        __syncwarp();
    }
    const RowCut cut(A.p.x, A.p.y, A.p.z, A.p.w);
    sum = 0;
    float sig_low = -1.f; // a lower bound of the lane's largest |v.u|
    u32 sig_n     = 0;    // candidates kept
    u32 sig_b[kSigCandidates];
    float sig_up[kSigCandidates];
    bool any_pair = false;
    u32 take, at;
    auto inside = [&](u32 kk) {
        const u32 b = ent[kk];
        const D4 B  = ldd4(rec, N, 0, b);
        const float r2 = cut.r2(B.x, B.y, B.z);
        const float hb = cut32(B.w); // NaN bounds decide nothing
        const float tm = hb < 1e18f ? fmaxf(cut.thr, 4.f * hb * hb) : __int_as_float(0x7fc00000);
        if (r2 > tm * cut.hi) return false;
        if (b == a && !plain_row) {
            any_pair = true;
            return false;
        }
        return r2 < tm * cut.lo || !beyond_both(A.p.x, A.p.y, A.p.z, A.p.w, B.x, B.y, B.z, B.w);
    };
    while (walk.next(inside, take, at)) {
        Pair64 o{0, 0, 0, 0, 0, 0};
        if (j < take) {
            any_pair    = true;
            const u32 b = ent[at];
            const D4 B0 = ldd4(rec, N, 0, b), B1 = ldd4(rec, N, 1, b), B2 = ldd4(rec, N, 2, b),
                     B3 = ldd4(rec, N, 3, b), B4 = ldd4(rec, N, 4, b);
            const f64 dx = A.p.x - B0.x, dy = A.p.y - B0.y, dz = A.p.z - B0.z;
            const f64 rab2 = mul64i(dx, dx) + mul64i(dy, dy) + mul64i(dz, dz);
            bool bad       = plain_row;
            const Root r   = root64(rab2, bad);
            const f64 rab  = root_value(r);
            f64 inv        = root_reciprocal(r, bad);
            if (bits64(rab) < bits64(1e-9)) inv = 0;
            const f64 Fab_a = divide_by(mul64i(kNorm3d, lean_m4_df(divide_by(rab, A.H(), bad))), A.H4(), bad);
            const f64 qb    = divide_by(rab, Denominator{B0.w, B3.w, low_float(B4.z)}, bad);
            const f64 Fab_b = divide_by(mul64i(kNorm3d, lean_m4_df(qb)),
                                        Denominator{B4.x, B4.y, high_float(B4.z)}, bad);
            const f64 vx = A.v.x - B1.x, vy = A.v.y - B1.y, vz = A.v.z - B1.z;
            const f64 rx = mul64i(dx, inv), ry = mul64i(dy, inv), rz = mul64i(dz, inv);
            o.vr             = mul64i(vx, rx) + mul64i(vy, ry) + mul64i(vz, rz);
            const f64 bv     = mul64i(p.beta_AV, fabs(o.vr));
            const f64 vsig_a = A.e.y + bv;
            const f64 vsig_b = B2.y + bv;
            const f64 dp     = fabs(A.e.x - B2.x);
            f64 vsig_u       = 0;
            {
                bool odd      = false;
                const f64 rr  = A.rho + B3.x;
                const f64 qu  = quotient64(dp, half(rr, odd), odd);
                const Root ru = root64(qu, odd);
                const bool eq = zero64(bits64(dp)); // sqrt(0 / rho) = 0
                vsig_u        = eq ? 0.0 : root_value(ru);
                bad |= eq ? !(hi64(rr) - 0x00100000u < 0x7FE00000u) : odd;
            }
            const f64 AV_P_a = A.e.x + positive(mul64i(mul64i(A.e.z, vsig_a), o.vr));
            const f64 AV_P_b = B2.x + positive(mul64i(mul64i(B2.z, vsig_b), o.vr));
            const f64 ca = mul64i(AV_P_a, A.e.w), cb = mul64i(AV_P_b, B2.w);
            const f64 nax = rx * Fab_a, nay = ry * Fab_a, naz = rz * Fab_a;
            const f64 nbx = rx * Fab_b, nby = ry * Fab_b, nbz = rz * Fab_b;
            const f64 mb = -p.pmass;
            o.fx = mb * (ca * nax + cb * nbx);
            o.fy = mb * (ca * nay + cb * nby);
            o.fz = mb * (ca * naz + cb * nbz);
            o.t1 = mul64i(mul64i(mul64i(AV_P_a, A.c_heat), p.pmass),
                          vx * nax + vy * nay + vz * naz);
            const f64 Fa = mul64i(Fab_a, A.inv_rho_om);
            const f64 Fb = divide_by(Fab_b, Denominator{B3.y, B3.z, low_float(B4.w)}, bad);
            o.t2 = mul64i(half(mul64i(mul64i(p.pmass * p.alpha_u, vsig_u), A.v.w - B1.w), bad), Fa + Fb);
            if (bad) force_pair_plain(rec, N, a, b, p, o);
            // a pair at rest adds 0 to the v_sig maximum
            if (VSIG && !zero64(bits64(vx) | bits64(vy) | bits64(vz))) {
                const float vf = fabsf(cut32(vx)) + fabsf(cut32(vy)) + fabsf(cut32(vz));
                const float w  = fabsf(cut32(o.vr)), slack = 3e-7f * w + 1e-14f * vf;
                // NaN or out of the float range: always a candidate
                const float up = w + slack < 1e37f ? w + slack : __int_as_float(0x7f800000);
                if (up >= sig_low) {
                    if (w - slack > sig_low) {
                        sig_low = w - slack;
                        // forget the candidates it overtakes
                        if (sig_n <= kSigCandidates) {
                            u32 m = 0;
                            for (u32 i = 0; i < sig_n; i++)
                                if (sig_up[i] >= sig_low) {
                                    sig_b[m]    = sig_b[i];
                                    sig_up[m++] = sig_up[i];
                                }
                            sig_n = m;
                        }
                    }
                    if (sig_n < kSigCandidates) {
                        sig_b[sig_n]  = b;
                        sig_up[sig_n] = up;
                    }
                    sig_n++;
                }
            }
        }
        f64 *x = W.x[q][j];
        x[0] = o.fx, x[1] = o.fy, x[2] = o.fz, x[3] = o.t1, x[4] = o.t2;
        __syncwarp();
#pragma unroll
        for (u32 s = 0; s < 4; s++) {
            sum += W.x[q][s][j];
            sum += W.x[q][s][j == 3 ? 4 : 5];
        }
        __syncwarp();
    }
    vsig_max = 0;
    if (VSIG) {
        auto quad_max = [](float v) {
            v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
            return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
        };
        const float low = quad_max(sig_low);
        f64 vr          = 0;
        if (__any_sync(0xffffffffu, sig_n > kSigCandidates)) {
            for (u32 k = k0; k < k1; k++) {
                const u32 b = ent[k];
                const D4 B  = ldd4(rec, N, 0, b);
                if (!beyond_both(A.p.x, A.p.y, A.p.z, A.p.w, B.x, B.y, B.z, B.w))
                    vr = fmax(vr, sig_speed_plain(rec, N, a, b));
            }
        } else {
            // each lane steps to its next candidate, then all evaluate one
            for (u32 i = 0; true; i++) {
                while (i < sig_n && !(sig_up[i] >= low)) i++;
                if (!__any_sync(0xffffffffu, i < sig_n)) break;
                if (i < sig_n) vr = fmax(vr, sig_speed_plain(rec, N, a, sig_b[i]));
            }
        }
        vr = fmax(vr, __shfl_xor_sync(0xffffffffu, vr, 1));
        vr = fmax(vr, __shfl_xor_sync(0xffffffffu, vr, 2));
        const u32 any = (__ballot_sync(0xffffffffu, any_pair) >> walk.shift) & 15u;
        if (any) vsig_max = fmax(0.0, 1.0 * cs_a + 2.0 * vr);
    }
}

// module form: reference CSR, outputs a, du (and vsig) by row
template<bool VSIG>
__global__ void __launch_bounds__(128, 4) k_derivs(RowSpace rs, const f64 *__restrict__ rec, u32 N,
                                                const f64 *__restrict__ cs, DerivParams p,
                                                f64 *__restrict__ ax, f64 *__restrict__ ay,
                                                f64 *__restrict__ az, f64 *__restrict__ du,
                                                f64 *__restrict__ vsig) {
    __shared__ Warp64 W[4];
    const u32 t = (blockIdx.x * 128 + threadIdx.x) >> 2, j = threadIdx.x & 3u;
    u32 a = 0, k0 = 0, k1 = 0;
    if (t < rs.n) {
        a  = rs.row_rank ? rs.row_rank[t] : t;
        k0 = rs.off[t];
        k1 = k0 + rs.cnt[t];
    }
    f64 sum, vm;
    derivs_row<VSIG>(W[threadIdx.x >> 5], rs.ent, rec, N, a, k0, k1, cs[a], p, sum, vm);
    if (t >= rs.n) return;
    (j == 0 ? ax : j == 1 ? ay : j == 2 ? az : du)[t] = sum;
    if (VSIG && j == 0) vsig[t] = vm;
}

// pipeline form: the sums by rank, {fx, fy, fz, du | v_sig maximum}
__global__ void __launch_bounds__(128, 4) k_derivs_sums64(RowSpace rs, const f64 *__restrict__ rec, u32 N,
                                                       const f64 *__restrict__ cs, DerivParams p,
                                                       f64 *__restrict__ sums, f64 *__restrict__ vmax) {
    __shared__ Warp64 W[4];
    const u32 t = (blockIdx.x * 128 + threadIdx.x) >> 2, j = threadIdx.x & 3u;
    u32 a = 0, k0 = 0, k1 = 0;
    if (t < rs.n) {
        a  = rs.row_rank[t];
        k0 = rs.off[t];
        k1 = k0 + rs.cnt[t];
    }
    f64 sum, vm;
    derivs_row<true>(W[threadIdx.x >> 5], rs.ent, rec, N, a, k0, k1, cs[a], p, sum, vm);
    if (t >= rs.n) return;
    sums[4 * (size_t) a + j] = sum;
    if (j == 0) vmax[a] = vm;
}

// leapfrog corrector + CFL from the sums, in the caller's order
__global__ void __launch_bounds__(256) k_correct64(u32 n, const u32 *__restrict__ rank_of,
                                                   const f64 *__restrict__ sums,
                                                   const f64 *__restrict__ vmax, DerivParams p,
                                                   LocalFields lf, Scalars *sc) {
    u64 ev2 = 0, dtm = ~0ull;
    f64 v2  = 0;
    for (u32 i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        const u32 r  = rank_of[i];
        const D4 S   = ldd4(sums, 0, 0, r);
        const f64 vm = vmax[r];
        f64 fx = S.x, fy = S.y, fz = S.z;
        const f64 tdu   = S.w;
        const size_t iv = (size_t) i * lf.vs;
        if (p.ext.x) {
            // axyz += axyz_ext (ExternalForces.cpp:342-359)
            fx = fx + p.ext.x[i];
            fy = fy + p.ext.y[i];
            fz = fz + p.ext.z[i];
        }
        f64 ox = lf.ax[iv], oy = lf.ay[iv], oz = lf.az[iv], odu = lf.du[i];
        lf.ax[iv] = fx;
        lf.ay[iv] = fy;
        lf.az[iv] = fz;
        lf.du[i]  = tdu;
        // corrector (integrators.cpp:88-120): incr = hdt * (new - old)
        f64 ix = p.hdt * (fx - ox), iy = p.hdt * (fy - oy), iz = p.hdt * (fz - oz);
        f64 nvx = lf.vx[iv] + ix, nvy = lf.vy[iv] + iy, nvz = lf.vz[iv] + iz;
        lf.vx[iv] = nvx;
        lf.vy[iv] = nvy;
        lf.vz[iv] = nvz;
        f64 iu    = p.hdt * (tdu - odu);
        lf.u[i]   = lf.u[i] + iu;
        const u64 e = f64_to_ordered(ix * ix + iy * iy + iz * iz);
        ev2         = e > ev2 ? e : ev2;
        v2 += nvx * nvx + nvy * nvy + nvz * nvz;
        // CFL with the new acceleration
        f64 h_a  = lf.h[i];
        f64 dt   = __longlong_as_double(0x7ff0000000000000ll);
        f64 dt_c = p.C_cour * h_a / vm;
        dt       = fmin(dt, dt_c);
        f64 abs_a = sqrt(fx * fx + fy * fy + fz * fz);
        f64 dt_f  = p.C_force * sqrt(h_a / abs_a);
        dt        = fmin(dt, dt_f);
        const u64 d = f64_to_ordered(dt);
        dtm         = d < dtm ? d : dtm;
    }
    ev2 = block_reduce(ev2, OpMaxU64{}, 0ull);
    dtm = block_reduce(dtm, OpMinU64{}, ~0ull);
    v2  = block_reduce(v2, OpAddF64{}, 0.0);
    if (threadIdx.x == 0) {
        raise_u64(&sc->epsv2_max, ev2);
        lower_u64(&sc->dt_min, dtm);
        atomicAdd(&sc->sum_v2, v2);
    }
}

// One axis of the periodic box: delt = bmax - bmin, and the patterns of delt and 2 delt (0
// where delt is no positive finite number, which sends every coordinate to the library)
struct WrapAxis {
    f64 bmin, delt;
    u64 d, d2;
};
struct Wrap {
    WrapAxis axis[3];
};
inline Wrap wrap_axes(const f64 *bmin, const f64 *bmax) {
    Wrap w;
    for (int c = 0; c < 3; c++) {
        const f64 d   = bmax[c] - bmin[c];
        const bool ok = d > 0 && d <= 1.7976931348623157e308;
        w.axis[c]     = WrapAxis{bmin[c], d, ok ? bits64(d) : 0, ok ? bits64(2 * d) : 0};
    }
    return w;
}

// fmod(r, d) for d > 0.  fmod is exact (its result is r - n d, which is representable),
// so any exact evaluation gives the same bits: within one period of the box, the
// remainder is r itself or r -+ d (exact by Sterbenz's lemma: d <= |r| <= 2 d); further
// out, and for NaN or infinities, the library fmod decides.  The result takes the sign
// of r, as fmod's does (a zero too).  The comparisons are those of the patterns, by integers.
__device__ __noinline__ f64 fmod_far(f64 r, f64 d) { return fmod(r, d); }
__device__ __forceinline__ f64 fmod_wrap(f64 r, const WrapAxis &w) {
    const u64 b = bits64(r), mag = b & 0x7fffffffffffffffull, sign = b & 0x8000000000000000ull;
    if (mag < w.d) return r;
    if (mag < w.d2) return from64(bits64(r - from64(bits64(w.delt) | sign)) | sign);
    return fmod_far(r, w.delt);
}

// acceleration of the central point mass, component n = -GM x over r^3; the plain operators
// where a quotient or the root fails its proof
__device__ __noinline__ f64 point_mass_plain(f64 x, f64 y, f64 z, f64 n) {
    f64 r  = sqrt(x * x + y * y + z * z);
    f64 r3 = r * r * r;
    return n / r3;
}
__device__ __forceinline__ void point_mass(f64 mGM, f64 x, f64 y, f64 z, f64 *ax, f64 *ay, f64 *az) {
    bool bad     = false;
    const f64 r  = root_value(root64(mul64i(x, x) + mul64i(y, y) + mul64i(z, z), bad));
    const f64 r3 = mul64i(mul64i(r, r), r);
    auto over    = [&](f64 n) {
        const u64 b    = bits64(n), sign = b & 0x8000000000000000ull;
        bool odd       = bad;
        const f64 q    = quotient64(from64(b ^ sign), r3, odd);
        return odd ? point_mass_plain(x, y, z, n) : from64(bits64(q) | sign);
    };
    *ax = over(mul64i(mGM, x));
    *ay = over(mul64i(mGM, y));
    *az = over(mul64i(mGM, z));
}

// leapfrog predictor (half kick, drift, half kick) + periodic wrap, one pass.  Bound by the
// FP64 pipe (16 cycles of an SM for a warp's instruction): its sums are the 23 FP64
// instructions left of about 55, the products go to the integer pipes, comparisons are
// integer ones and the box's constants come from the host: 1,048,576 particles 100 -> 63 us,
// 8.5 M 793 -> 475 us (1.22 GB of fields, 185 us at the copy rate); with the products on
// the FP64 pipe too 75 and 585 us.  With the point mass (a root and three quotients by the
// forms of lean64.cuh) 1,000,003 particles 102 -> 72 us.
__global__ void __launch_bounds__(256, 5) k_predict(LocalFields lf, u32 n, f64 dt, f64 dt_half, int periodic, Wrap wrap, f64 mGM,
                          f64 *__restrict__ ext_x, f64 *__restrict__ ext_y, f64 *__restrict__ ext_z) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    size_t iv = (size_t) i * lf.vs;
    const f64 kx = mul64i(dt_half, lf.ax[iv]), ky = mul64i(dt_half, lf.ay[iv]);
    const f64 kz = mul64i(dt_half, lf.az[iv]), ku = mul64i(dt_half, lf.du[i]);
    f64 vx = lf.vx[iv] + kx, vy = lf.vy[iv] + ky, vz = lf.vz[iv] + kz, u = lf.u[i] + ku;
    f64 x = lf.x[iv] + mul64i(dt, vx), y = lf.y[iv] + mul64i(dt, vy), z = lf.z[iv] + mul64i(dt, vz);
    vx = vx + kx;
    vy = vy + ky;
    vz = vz + kz;
    u  = u + ku;
    if (ext_x) {
        // central point mass at the drifted position, before the wrap
        point_mass(mGM, x, y, z, &ext_x[i], &ext_y[i], &ext_z[i]);
    }
    if (periodic) {
        f64 p[3] = {x, y, z};
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const WrapAxis &w = wrap.axis[c];
            f64 r             = fmod_wrap(p[c] - w.bmin, w);
            r                 = fmod_wrap(r + w.delt, w);
            p[c]              = r + w.bmin;
        }
        x = p[0];
        y = p[1];
        z = p[2];
    }
    lf.x[iv]  = x;
    lf.y[iv]  = y;
    lf.z[iv]  = z;
    lf.vx[iv] = vx;
    lf.vy[iv] = vy;
    lf.vz[iv] = vz;
    lf.u[i]   = u;
}

// ---------------------------------------------------------------- conservation totals
// ConservativeCheck::check_conservation (shammodels/sph/src/modules/ConservativeCheck.cpp:
// 56-180): sum v, sum a, sum (u + v.v / 2) and sum (v.a + du), each times the particle
// mass, in FP64.  Per-block partial sums in a fixed tree order, then one block adds the
// partials in block order: the totals are the same from run to run.
constexpr u32 kConsBlock = 256;

__global__ void __launch_bounds__(kConsBlock) k_cons_partial(LocalFields lf, u32 n,
                                                            f64 *__restrict__ part) {
    __shared__ f64 sm[8][kConsBlock];
    const u32 t = threadIdx.x;
    f64 v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (u32 i = blockIdx.x * kConsBlock + t; i < n; i += gridDim.x * kConsBlock) {
        const size_t iv = (size_t) i * lf.vs;
        const f64 vx = lf.vx[iv], vy = lf.vy[iv], vz = lf.vz[iv];
        const f64 ax = lf.ax[iv], ay = lf.ay[iv], az = lf.az[iv];
        v[0] += vx;
        v[1] += vy;
        v[2] += vz;
        v[3] += ax;
        v[4] += ay;
        v[5] += az;
        v[6] += lf.u[i] + 0.5 * ((vx * vx + vy * vy) + vz * vz);
        v[7] += ((vx * ax + vy * ay) + vz * az) + lf.du[i];
    }
#pragma unroll
    for (int k = 0; k < 8; k++) sm[k][t] = v[k];
    __syncthreads();
    for (u32 s = kConsBlock / 2; s > 0; s >>= 1) {
        if (t < s)
#pragma unroll
            for (int k = 0; k < 8; k++) sm[k][t] += sm[k][t + s];
        __syncthreads();
    }
    if (t < 8) part[(size_t) blockIdx.x * 8 + t] = sm[t][0];
}

__global__ void k_cons_final(const f64 *__restrict__ part, u32 nb, f64 pmass,
                             f64 *__restrict__ out) {
    const u32 k = threadIdx.x;
    if (k >= 8) return;
    f64 s = 0;
    for (u32 b = 0; b < nb; b++) s += part[(size_t) b * 8 + k];
    out[k] = pmass * s;
}

// ---------------------------------------------------------------- varying AV (CD10)
// div v and curl v (DiffOperator.cpp:95-140, 200-245) and d(div v)/dt from the linearly
// corrected gradients (DiffOperatorDtDivv.cpp:116-210) in one pass over the row; each
// sum in the reference's order, so the values equal the three separate kernels'.
__device__ __forceinline__ void inv33(const f64 m[3][3], f64 r[3][3]) {
    const f64 a00 = m[0][0], a01 = m[0][1], a02 = m[0][2];
    const f64 a10 = m[1][0], a11 = m[1][1], a12 = m[1][2];
    const f64 a20 = m[2][0], a21 = m[2][1], a22 = m[2][2];
    const f64 det = (((((-a02 * a11) * a20 + (a01 * a12) * a20) + (a02 * a10) * a21)
                      - (a00 * a12) * a21) - (a01 * a10) * a22) + (a00 * a11) * a22;
    r[0][0] = (-a12 * a21 + a11 * a22) / det;
    r[0][1] = (a02 * a21 - a01 * a22) / det;
    r[0][2] = (-a02 * a11 + a01 * a12) / det;
    r[1][0] = (a12 * a20 - a10 * a22) / det;
    r[1][1] = (-a02 * a20 + a00 * a22) / det;
    r[1][2] = (a02 * a10 - a00 * a12) / det;
    r[2][0] = (-a11 * a20 + a10 * a21) / det;
    r[2][1] = (a01 * a20 - a00 * a21) / det;
    r[2][2] = (-a01 * a10 + a00 * a11) / det;
}
__device__ __forceinline__ void mul33(const f64 a[3][3], const f64 b[3][3], f64 c[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) c[i][j] = (a[i][0] * b[0][j] + a[i][1] * b[1][j]) + a[i][2] * b[2][j];
}

// the pair's e = r / |r| (zero below 1e-9) and F = dW(|r|, h_a) with the plain operators
__device__ __noinline__ void gradient_pair_plain(const f64 r[3], f64 rab2, f64 h_a, f64 e[3], f64 &F) {
    const f64 rab = sqrt(rab2);
    for (int c = 0; c < 3; c++) e[c] = (rab < 1e-9) ? 0.0 : r[c] / rab;
    F = dW_3d(rab, h_a);
}

// Bound by the FP64 pipe like the loop above and arranged like it.  Pairs beyond 2 h_a
// (inside the neighbour's support only) have F = 0 and add zeros, so those that the FP32
// test finds outside are not evaluated.  Each lane of a quad evaluates a pair; lane 0 then
// adds R, lane 1 Dv, lane 2 Da (the same nine products with r, v or w) and lane 3 div and
// curl, in entry order, and lane 0 collects them.  acc: records {ax, ay, az, -} of the last
// evaluation.
constexpr int kVgTerms = 19; // {r, v, w (9), curl terms (3), div term, 0 | m g (3), -1}, padded
struct WarpVg64 {
    f64 z[8][4][kVgTerms]; // [quad][pair]
    u32 queue[8][8];
};

__global__ void __launch_bounds__(128, 4) k_velgrad64(RowSpace rs, const f64 *__restrict__ rec, u32 N,
                                                   const f64 *__restrict__ acc, f64 pmass,
                                                   f64 *__restrict__ divv, f64 *__restrict__ cx,
                                                   f64 *__restrict__ cy, f64 *__restrict__ cz,
                                                   u32 cvs, f64 *__restrict__ dtdivv) {
    __shared__ WarpVg64 Ws[4];
    WarpVg64 &W = Ws[threadIdx.x >> 5];
    const u32 t = (blockIdx.x * 128 + threadIdx.x) >> 2;
    u32 a = 0, k0 = 0, k1 = 0;
    if (t < rs.n) {
        a  = rs.row_rank[t];
        k0 = rs.off[t];
        k1 = k0 + rs.cnt[t];
    }
    QuadWalk walk(W.queue, k0, k1);
    const u32 j = walk.j, q = walk.q;
    const D4 A0 = ldd4(rec, N, 0, a), A1 = ldd4(rec, N, 1, a), A3 = ldd4(rec, N, 3, a),
             A4 = ldd4(rec, N, 4, a), Aa = ldd4(acc, N, 0, a);
    const f64 h_a = A0.w;
    const Denominator H{h_a, A3.w, low_float(A4.z)}, H4{A4.x, A4.y, high_float(A4.z)};
    const RowCut cut(A0.x, A0.y, A0.z, h_a);
    const bool plain_row = !(fabs(A1.x) + fabs(A1.y) + fabs(A1.z) + fabs(Aa.x) + fabs(Aa.y) + fabs(Aa.z) < 1e300)
                           || !(H.lo == H.lo) || !(H4.lo == H4.lo);
    f64 S[8] = {};
    W.z[q][j][13] = 0.0;
    W.z[q][j][17] = -1.0;
    auto inside = [&](u32 kk) {
        const u32 b    = rs.ent[kk];
        const D4 B     = ldd4(rec, N, 0, b);
        const float r2 = cut.r2(B.x, B.y, B.z);
        if (!plain_row && (r2 > cut.thr * cut.hi || b == a)) return false;
        return r2 < cut.thr * cut.lo || !beyond_both(A0.x, A0.y, A0.z, A0.w, B.x, B.y, B.z, B.w);
    };
    u32 take, at;
    while (walk.next(inside, take, at)) {
        f64 r[3] = {0, 0, 0}, v[3] = {0, 0, 0}, w[3] = {0, 0, 0}, mg[3] = {0, 0, 0}, cu[3] = {0, 0, 0}, dv = 0;
        if (j < take) {
            const u32 b = rs.ent[at];
            const D4 B0 = ldd4(rec, N, 0, b), B1 = ldd4(rec, N, 1, b), Ba = ldd4(acc, N, 0, b);
            r[0] = A0.x - B0.x, r[1] = A0.y - B0.y, r[2] = A0.z - B0.z;
            v[0] = A1.x - B1.x, v[1] = A1.y - B1.y, v[2] = A1.z - B1.z;
            w[0] = Aa.x - Ba.x, w[1] = Aa.y - Ba.y, w[2] = Aa.z - Ba.z;
            const f64 rab2  = (mul64i(r[0], r[0]) + mul64i(r[1], r[1])) + mul64i(r[2], r[2]);
            bool bad        = plain_row;
            const Root root = root64(rab2, bad);
            const f64 rab   = root_value(root);
            Denominator D{rab, 0, 0.f};
            root_reciprocal(root, bad, D.y, D.lo);
            bad |= bits64(rab) < bits64(1e-9);
            f64 e[3];
#pragma unroll
            for (int c = 0; c < 3; c++) e[c] = divide_by(r[c], D, bad);
            f64 F = divide_by(mul64i(kNorm3d, lean_m4_df(divide_by(rab, H, bad))), H4, bad);
            if (bad) gradient_pair_plain(r, rab2, h_a, e, F);
            const f64 g[3] = {mul64i(F, e[0]), mul64i(F, e[1]), mul64i(F, e[2])};
            dv    = mul64i(pmass, (mul64i(v[0], g[0]) + mul64i(v[1], g[1])) + mul64i(v[2], g[2]));
            cu[0] = mul64i(pmass, mul64i(v[1], g[2]) - mul64i(v[2], g[1]));
            cu[1] = mul64i(pmass, mul64i(v[2], g[0]) - mul64i(v[0], g[2]));
            cu[2] = mul64i(pmass, mul64i(v[0], g[1]) - mul64i(v[1], g[0]));
#pragma unroll
            for (int c = 0; c < 3; c++) mg[c] = mul64i(g[c], pmass);
        }
        f64 *z = W.z[q][j];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            z[c]      = r[c];
            z[3 + c]  = v[c];
            z[6 + c]  = w[c];
            z[9 + c]  = cu[c];
            z[14 + c] = mg[c];
        }
        z[12] = dv;
        __syncwarp();
        // S = S - u (m g): lanes 0-2 the entries (i, jj) of their matrix but the last, lane 3
        // the three last ones and the curl and div terms (times -1)
        for (u32 s = 0; s < take; s++) {
            const f64 *zs = W.z[q][s];
#pragma unroll
            for (int m = 0; m < 8; m++) {
                const f64 u  = zs[j < 3 ? 3 * j + m / 3 : (m < 3 ? 3 * m + 2 : 6 + m)];
                const f64 gg = zs[j < 3 ? 14 + m % 3 : (m < 3 ? 16 : 17)];
                S[m]         = S[m] - mul64i(u, gg);
            }
        }
        __syncwarp();
    }
    // the quad's sums through shared memory to its first lane
    f64 *out = &W.z[q][0][0];
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 8; m++) out[8 * j + m] = S[m];
    __syncwarp();
    if (t >= rs.n || j != 0) return;
    const f64 inv_rho_omega_a = 1. / A3.y; // 1 / (Omega rho)
    f64 R[3][3], Dv[3][3], Da[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int jj = 0; jj < 3; jj++) {
            const int m = 3 * i + jj;
            R[i][jj]    = out[m < 8 ? m : 24];
            Dv[jj][i]   = out[m < 8 ? 8 + m : 25];
            Da[jj][i]   = out[m < 8 ? 16 + m : 26];
        }
    const f64 sc[3] = {out[27], out[28], out[29]};
    const f64 sdiv  = out[30];
    const u32 i = rs.row_local[t];
    divv[i]     = -inv_rho_omega_a * sdiv;
    cx[(size_t) i * cvs] = -inv_rho_omega_a * sc[0];
    cy[(size_t) i * cvs] = -inv_rho_omega_a * sc[1];
    cz[(size_t) i * cvs] = -inv_rho_omega_a * sc[2];
    f64 Ri[3][3], Gv[3][3], Ga[3][3];
    inv33(R, Ri);
    mul33(Ri, Dv, Gv);
    mul33(Ri, Da, Ga);
    const f64 div_a = (Ga[0][0] + Ga[1][1]) + Ga[2][2];
    const f64 tens  = ((((((((Gv[0][0] * Gv[0][0] + Gv[1][0] * Gv[0][1]) + Gv[2][0] * Gv[0][2])
                            + Gv[0][1] * Gv[1][0]) + Gv[1][1] * Gv[1][1]) + Gv[2][1] * Gv[1][2])
                         + Gv[0][2] * Gv[2][0]) + Gv[1][2] * Gv[2][1]) + Gv[2][2] * Gv[2][2]);
    dtdivv[i] = div_a - tens;
}

// Cullen & Dehnen (2010) switch, one implicit-Euler step (UpdateViscosity.cpp:170-215);
// max / min as comparisons, as in the oracle
// T = f64: the reference's FP64 switch, bit for bit.  T = float: the same expressions in
// FP32 for the mixed path (its velocity gradients are FP32 sums already; the switch's
// divisions would otherwise make this pass FP64-pipe bound on GB300).
template<class T>
__global__ void k_cd10(u32 n, const f64 *__restrict__ divv, const f64 *__restrict__ cx,
                       const f64 *__restrict__ cy, const f64 *__restrict__ cz, u32 cvs,
                       const f64 *__restrict__ dtdivv, const f64 *__restrict__ cs,
                       const f64 *__restrict__ h, const f64 *__restrict__ alpha, f64 dt_,
                       f64 sigma_decay_, f64 alpha_min_, f64 alpha_max_, f64 *__restrict__ alpha_new) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const T eps  = (T) 2.220446049250313e-16; // DBL_EPSILON
    const T dt = (T) dt_, sigma_decay = (T) sigma_decay_, alpha_min = (T) alpha_min_,
            alpha_max = (T) alpha_max_;
    const T cs_a = (T) cs[i], h_a = (T) h[i], alpha_a = (T) alpha[i];
    const T inv_tau = cs_a * sigma_decay / h_a;
    const T fact_t  = dt * inv_tau;
    const T euler   = 1 / (1 + fact_t);
    const T md = -(T) divv[i];
    T fac      = (md > 0) ? md : T(0);
    fac        = fac * fac;
    const size_t iv = (size_t) i * cvs;
    const T cxi = (T) cx[iv], cyi = (T) cy[iv], czi = (T) cz[iv];
    const T traceS  = (cxi * cxi + cyi * cyi) + czi * czi;
    const T balsara = (fac + traceS > eps) ? fac / (fac + traceS) : T(1);
    const T mdt     = -(T) dtdivv[i];
    const T A       = balsara * ((mdt > 0) ? mdt : T(0));
    const T temp    = cs_a * cs_a;
    T alpha_loc     = (cs_a > 0) ? 10 * h_a * h_a * A / temp : alpha_min;
    alpha_loc       = (alpha_loc < alpha_max) ? alpha_loc : alpha_max;
    alpha_loc       = (temp > eps) ? alpha_loc : alpha_min;
    T na = (alpha_a + alpha_loc * fact_t) * euler;
    if (alpha_loc > alpha_a) na = alpha_loc;
    alpha_new[i] = (f64) na;
}

// Morris & Monaghan (1997) switch (UpdateViscosity.cpp:53-118), comparisons as in the oracle
template<class T>
__global__ void k_mm97(u32 n, const f64 *__restrict__ divv, const f64 *__restrict__ cs,
                       const f64 *__restrict__ h, const f64 *__restrict__ alpha, f64 dt_,
                       f64 sigma_decay_, f64 alpha_min_, f64 alpha_max_, f64 *__restrict__ alpha_new) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const T dt = (T) dt_, alpha_min = (T) alpha_min_, alpha_max = (T) alpha_max_;
    const T inv_tau = (T) cs[i] * (T) sigma_decay_ / (T) h[i];
    const T fact_t  = dt * inv_tau;
    const T euler   = 1 / (1 + fact_t);
    const T md      = -(T) divv[i];
    const T source  = (md > 0) ? md : T(0);
    const T na      = ((T) alpha[i] + source * dt + fact_t * alpha_min) * euler;
    alpha_new[i]    = (f64) ((na < alpha_max) ? na : alpha_max);
}

// accelerations of the last evaluation in rank order (ghosts copy their source), one
// 32-byte record per rank
__global__ void k_gather_acc(const u32 *__restrict__ sort_index, u32 N, u32 n_local,
                             const u32 *__restrict__ ghost_src, LocalFields lf,
                             f64 *__restrict__ acc) {
    u32 r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= N) return;
    const u32 id    = sort_index[r];
    const size_t iv = (size_t) (id < n_local ? id : ghost_src[id - n_local]) * lf.vs;
    std4(acc, N, 0, r, lf.ax[iv], lf.ay[iv], lf.az[iv], 0.0);
}

__global__ void k_rank_to_local(u32 n, const u32 *__restrict__ row_rank,
                                const u32 *__restrict__ row_local, const f64 *__restrict__ src,
                                f64 *__restrict__ dst) {
    u32 t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    dst[row_local[t]] = src[row_rank[t]];
}

__global__ void k_scatter_rows(u32 n, const u32 *__restrict__ row_local, const f64 *__restrict__ src,
                               f64 *__restrict__ dst) {
    u32 t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    dst[row_local[t]] = src[t];
}

// start of the h iteration: both h of a row, its eps, and the reductions' identities
__global__ void k_h_start(u32 n, const u32 *__restrict__ row_rank, const f64 *__restrict__ h_rank,
                          f64 *__restrict__ h_old, f64 *__restrict__ h_new, f64 *__restrict__ eps, f64 eps0,
                          Scalars *sc) {
    u32 t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) sc->eps_max = 0, sc->eps_min = ~0ull, sc->iters_max = 0;
    if (t >= n) return;
    const f64 v = h_rank[row_rank[t]];
    h_old[t]    = v;
    h_new[t]    = v;
    eps[t]      = eps0;
}

} // namespace

// ---------------------------------------------------------------- host wrappers
cudaError_t h_iterate64(Ctx &c, const RowSpace &rs, const f64 *h_old, f64 *h_new, f64 *eps,
                        f64 pmass, f64 hev, f64 hevi, u32 iters, f64 eps_p) {
    ProfScope ps(c, kProfHIter, rs.n);
    { k_h_iterate<<<div_up(rs.n, 128), 128, 0, c.stream>>>(rs, h_old, h_new, eps, pmass, hev, hevi,
                                                         iters, eps_p, c.d_scalars.as<Scalars>()); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t omega64(Ctx &c, const RowSpace &rs, const f64 *h_row, f64 pmass, f64 *out,
                    const u32 *out_index) {
    ProfScope ps(c, kProfOmega, rs.n);
    { k_omega<<<div_up(rs.n, 128), 128, 0, c.stream>>>(rs, h_row, pmass, out, out_index); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t eos64(Ctx &c, u32 n, const f64 *h, const f64 *u, f64 pmass, f64 gamma, f64 *P, f64 *cs) {
    { k_eos<<<div_up(n, 256), 256, 0, c.stream>>>(n, h, u, pmass, gamma, P, cs); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t gather_eos64(Ctx &c, u32 N, u32 n_local, const LocalFields &lf, const f64 *omega_local,
                         f64 pmass, const EosParams &eos, f64 alpha_AV) {
    cudaError_t e;
    if ((e = c.scs.ensure(sizeof(f64) * (size_t) N, c.stream)) != cudaSuccess) return e;
    if ((e = c.rec64.ensure(sizeof(f64) * 20 * (size_t) N, c.stream)) != cudaSuccess) return e;
    ProfScope ps(c, kProfGatherEos, N);
    { k_gather_eos<<<div_up(N, 256), 256, 0, c.stream>>>(
        c.sort_index.as<u32>(), N, n_local, c.ghost_src.as<u32>(), lf.h, lf.u, lf.vx, lf.vy, lf.vz,
        lf.vs, omega_local, pmass, eos, alpha_AV, c.sx.as<f64>(), c.sy.as<f64>(), c.sz.as<f64>(),
        c.scs.as<f64>(), c.rec64.as<f64>(), c.d_scalars.as<Scalars>()); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t stage_alpha64(Ctx &c, u32 N, u32 n_local, const f64 *alpha_local) {
    { k_stage_alpha64<<<div_up(N, 256), 256, 0, c.stream>>>(c.sort_index.as<u32>(), N, n_local,
                                                           c.ghost_src.as<u32>(), alpha_local,
                                                           c.scs.as<f64>(), c.rec64.as<f64>()); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t eos_lp07(Ctx &c, u32 n, const f64 *x, const f64 *y, const f64 *z, u32 vs, const f64 *h,
                     f64 pmass, f64 cs0, f64 r0, f64 q, f64 *P, f64 *cs) {
    { k_eos_lp07<<<div_up(n, 256), 256, 0, c.stream>>>(n, x, y, z, vs, h, pmass, cs0, r0, q, P, cs); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t derivs64(Ctx &c, const RowSpace &rs, const HydroSpace &hs, f64 pmass, f64 alpha_u,
                     f64 alpha_AV, f64 beta_AV, f64 *ax, f64 *ay, f64 *az, f64 *du, f64 *vsig) {
    DerivParams p{pmass, alpha_u, beta_AV, 0, 0, 0, ExtAccel{nullptr, nullptr, nullptr}};
    // the caller's merged arrays hold c.n_obj entries
    const u32 N   = c.n_obj;
    cudaError_t e = c.rec64.ensure(sizeof(f64) * 20 * (size_t) N, c.stream);
    if (e != cudaSuccess) return e;
    { k_stage_modules<<<div_up(N, 256), 256, 0, c.stream>>>(N, rs.x, rs.y, rs.z, hs, pmass, alpha_AV,
                                                           c.rec64.as<f64>()); GBSPH_COUNTED; }
    auto kern = vsig ? k_derivs<true> : k_derivs<false>;
    { kern<<<div_up(rs.n, 32), 128, 0, c.stream>>>(rs, c.rec64.as<f64>(), N, hs.cs, p, ax, ay, az, du,
                                                  vsig); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t derivs_step64(Ctx &c, const RowSpace &rs, u32 N, f64 pmass, f64 alpha_u, f64 beta_AV,
                          f64 hdt, f64 C_cour, f64 C_force, const LocalFields &lf,
                          const ExtAccel &ext) {
    DerivParams p{pmass, alpha_u, beta_AV, hdt, C_cour, C_force, ext};
    ProfScope ps(c, kProfDerivs, rs.n);
    void *room    = nullptr;
    cudaError_t e = sums_buffer(c, sizeof(f64) * 5 * (size_t) N, &room);
    if (e != cudaSuccess) return e;
    f64 *sums = (f64 *) room, *vmax = sums + 4 * (size_t) N;
    { k_derivs_sums64<<<div_up(rs.n, 32), 128, 0, c.stream>>>(rs, c.rec64.as<f64>(), N, c.scs.as<f64>(), p,
                                                             sums, vmax); GBSPH_COUNTED; }
    { k_correct64<<<std::min(div_up(rs.n, 256), 6 * c.sms), 256, 0, c.stream>>>(
        rs.n, c.rank_of.as<u32>(), sums, vmax, p, lf, c.d_scalars.as<Scalars>()); GBSPH_COUNTED; }
    return cudaGetLastError();
}
// leapfrog corrector (integrators.cpp:88-120): v += dt/2 (a_new - a_old), u likewise;
// max |dv|^2 and sum |v|^2 for the eps_v rerun test (Solver.cpp:2580-2616)
__global__ void k_kdk_correct(LocalFields lf, u32 n, const f64 *__restrict__ aox,
                              const f64 *__restrict__ aoy, const f64 *__restrict__ aoz, u32 avs,
                              const f64 *__restrict__ du_old, f64 hdt, Scalars *sc) {
    u32 i   = blockIdx.x * blockDim.x + threadIdx.x;
    u64 ev2 = 0;
    f64 v2  = 0;
    if (i < n) {
        size_t iv = (size_t) i * lf.vs, io = (size_t) i * avs;
        f64 ix = hdt * (lf.ax[iv] - aox[io]);
        f64 iy = hdt * (lf.ay[iv] - aoy[io]);
        f64 iz = hdt * (lf.az[iv] - aoz[io]);
        f64 vx = lf.vx[iv] + ix, vy = lf.vy[iv] + iy, vz = lf.vz[iv] + iz;
        lf.vx[iv] = vx;
        lf.vy[iv] = vy;
        lf.vz[iv] = vz;
        lf.u[i]   = lf.u[i] + hdt * (lf.du[i] - du_old[i]);
        ev2       = f64_to_ordered(__dadd_rn(__dadd_rn(ix * ix, iy * iy), iz * iz));
        v2        = __dadd_rn(__dadd_rn(vx * vx, vy * vy), vz * vz);
    }
    ev2 = block_reduce(ev2, OpMaxU64{}, 0ull);
    v2  = block_reduce(v2, OpAddF64{}, 0.0);
    if (threadIdx.x == 0) {
        atomicMax((unsigned long long *) &sc->epsv2_max, (unsigned long long) ev2);
        atomicAdd(&sc->sum_v2, v2);
    }
}

// CFL (ComputeCFLCourant.hpp:45-60, ComputeCFLForce.hpp:50-62) and its minimum
__global__ void k_cfl(u32 n, const f64 *__restrict__ h, const f64 *__restrict__ vsig,
                      const f64 *__restrict__ ax, const f64 *__restrict__ ay,
                      const f64 *__restrict__ az, u32 avs, f64 C_cour, f64 C_force,
                      f64 *__restrict__ dt_part, Scalars *sc) {
    u32 i   = blockIdx.x * blockDim.x + threadIdx.x;
    u64 dtm = ~0ull;
    if (i < n) {
        size_t io = (size_t) i * avs;
        f64 dt    = __longlong_as_double(0x7ff0000000000000ll);
        dt        = fmin(dt, C_cour * h[i] / vsig[i]);
        f64 a0 = ax[io], a1 = ay[io], a2 = az[io];
        f64 abs_a = sqrt(a0 * a0 + a1 * a1 + a2 * a2);
        dt        = fmin(dt, C_force * sqrt(h[i] / abs_a));
        if (dt_part) dt_part[i] = dt;
        dtm = f64_to_ordered(dt);
    }
    dtm = block_reduce(dtm, OpMinU64{}, ~0ull);
    if (threadIdx.x == 0) atomicMin((unsigned long long *) &sc->dt_min, (unsigned long long) dtm);
}

cudaError_t kdk_correct64(Ctx &c, const LocalFields &lf, u32 n, const f64 *aox, const f64 *aoy,
                          const f64 *aoz, u32 avs, const f64 *du_old, f64 dt) {
    { k_kdk_correct<<<div_up(n, 256), 256, 0, c.stream>>>(lf, n, aox, aoy, aoz, avs, du_old, dt / 2,
                                                         c.d_scalars.as<Scalars>()); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t cfl64(Ctx &c, u32 n, const f64 *h, const f64 *vsig, const f64 *ax, const f64 *ay,
                  const f64 *az, u32 avs, f64 C_cour, f64 C_force, f64 *dt_part) {
    { k_cfl<<<div_up(n, 256), 256, 0, c.stream>>>(n, h, vsig, ax, ay, az, avs, C_cour, C_force,
                                                 dt_part, c.d_scalars.as<Scalars>()); GBSPH_COUNTED; }
    return cudaGetLastError();
}

cudaError_t predict64(Ctx &c, const LocalFields &lf, u32 n, f64 dt, int periodic, const f64 *bmin,
                      const f64 *bmax, f64 mGM, f64 *ext_x, f64 *ext_y, f64 *ext_z) {
    ProfScope ps(c, kProfPredict, n);
    { k_predict<<<div_up(n, 256), 256, 0, c.stream>>>(lf, n, dt, dt / 2, periodic, wrap_axes(bmin, bmax), mGM,
                                                   ext_x, ext_y, ext_z); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t velgrad64(Ctx &c, const RowSpace &rs, u32 N, u32 n_local, const LocalFields &lf, f64 pmass,
                      f64 *divv, f64 *cx, f64 *cy, f64 *cz, u32 cvs, f64 *dtdivv) {
    cudaError_t e = c.av_arank.ensure(sizeof(f64) * 4 * (size_t) N, c.stream);
    if (e != cudaSuccess) return e;
    ProfScope ps(c, kProfVelGrad, rs.n);
    { k_gather_acc<<<div_up(N, 256), 256, 0, c.stream>>>(c.sort_index.as<u32>(), N, n_local,
                                                        c.ghost_src.as<u32>(), lf,
                                                        c.av_arank.as<f64>()); GBSPH_COUNTED; }
    { k_velgrad64<<<div_up(rs.n, 32), 128, 0, c.stream>>>(rs, c.rec64.as<f64>(), N, c.av_arank.as<f64>(),
                                                         pmass, divv, cx, cy, cz, cvs, dtdivv); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t cd10_update(Ctx &c, u32 n, const f64 *divv, const f64 *cx, const f64 *cy,
                        const f64 *cz, u32 cvs, const f64 *dtdivv, const f64 *cs, const f64 *h,
                        const f64 *alpha, f64 dt, f64 sigma_decay, f64 alpha_min, f64 alpha_max,
                        f64 *alpha_new, bool fp32) {
    if (fp32) {
        k_cd10<float><<<div_up(n, 256), 256, 0, c.stream>>>(n, divv, cx, cy, cz, cvs, dtdivv, cs, h,
                                                           alpha, dt, sigma_decay, alpha_min,
                                                           alpha_max, alpha_new); GBSPH_COUNTED;
    } else {
        k_cd10<f64><<<div_up(n, 256), 256, 0, c.stream>>>(n, divv, cx, cy, cz, cvs, dtdivv, cs, h,
                                                         alpha, dt, sigma_decay, alpha_min,
                                                         alpha_max, alpha_new); GBSPH_COUNTED;
    }
    return cudaGetLastError();
}
cudaError_t mm97_update(Ctx &c, u32 n, const f64 *divv, const f64 *cs, const f64 *h,
                        const f64 *alpha, f64 dt, f64 sigma_decay, f64 alpha_min, f64 alpha_max,
                        f64 *alpha_new, bool fp32) {
    if (fp32) {
        k_mm97<float><<<div_up(n, 256), 256, 0, c.stream>>>(n, divv, cs, h, alpha, dt, sigma_decay,
                                                           alpha_min, alpha_max, alpha_new); GBSPH_COUNTED;
    } else {
        k_mm97<f64><<<div_up(n, 256), 256, 0, c.stream>>>(n, divv, cs, h, alpha, dt, sigma_decay,
                                                         alpha_min, alpha_max, alpha_new); GBSPH_COUNTED;
    }
    return cudaGetLastError();
}
cudaError_t conservation64(Ctx &c, const LocalFields &lf, u32 n, f64 pmass, f64 *out_dev,
                           f64 *scratch) {
    const u32 nb = 1024;
    { k_cons_partial<<<nb, kConsBlock, 0, c.stream>>>(lf, n, scratch); GBSPH_COUNTED; }
    { k_cons_final<<<1, 32, 0, c.stream>>>(scratch, nb, pmass, out_dev); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t rank_to_local64(Ctx &c, u32 n, const f64 *src_rank, f64 *dst) {
    { k_rank_to_local<<<div_up(n, 256), 256, 0, c.stream>>>(n, c.row_rank.as<u32>(),
                                                           c.row_local.as<u32>(), src_rank,
                                                           dst); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t scatter_rows(Ctx &c, u32 n, const f64 *src, f64 *dst) {
    { k_scatter_rows<<<div_up(n, 256), 256, 0, c.stream>>>(n, c.row_local.as<u32>(), src, dst); GBSPH_COUNTED; }
    return cudaGetLastError();
}
cudaError_t h_start(Ctx &c, u32 n, const f64 *h_rank, f64 *h_old, f64 *h_new, f64 *eps, f64 eps0) {
    { k_h_start<<<div_up(n, 256), 256, 0, c.stream>>>(n, c.row_rank.as<u32>(), h_rank, h_old, h_new, eps, eps0,
                                                     c.d_scalars.as<Scalars>()); GBSPH_COUNTED; }
    return cudaGetLastError();
}

} // namespace gbsph
