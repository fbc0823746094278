// Per-step kernels: the fused force evaluation (anisotropic lipid pair
// potential, lipid-protein, LJ, protein-protein, bonds, global area/volume
// constraint) and the integrators, one thread per particle slot over a full
// neighbour list -- every force and torque is accumulated in registers by the
// thread that owns the particle, so no atomics are needed.
//
//   k_step_langevin   forces + src/integrate_langevin.h:105-146 (one launch per
//                     step; positions ping-pong between two buffers)
//   k_nh_final        forces + post_toque_final_update (src/integrate_nh.h:237-273)
//   k_nh_initial      verlet_initial_bounce_clearforce_update (:178-235)
//   k_forces          forces only (parity hook)
//   k_mesh            FP64 membrane area and enclosed volume per system
//
// Per-system sums are deterministic and take two launches: each warp of a
// step kernel reduces its 32 particles with shuffles and stores one warp
// partial (warp_partials); k_reduce, launched next on the stream, adds the
// warp partials of each reduction group in a fixed tree, and its last block
// adds each system's group sums in a fixed order and applies the thermostat,
// the rebuild rule, the step counter and the buffer parity.  The lite Langevin
// kernel keeps no sums: each warp raises the rebuild flag itself and
// k_advance flips the buffers.
#include "orbc_device.cuh"

#include <type_traits>

namespace orbc {

namespace {

template<class R> struct R3 {
    R x, y, z;
};

template<class R> __device__ __forceinline__ typename Vec<R>::T4 ldg4(const typename Vec<R>::T4 *p);
template<> __device__ __forceinline__ float4 ldg4<float>(const float4 *p) { return __ldg(p); }
template<> __device__ __forceinline__ double4a ldg4<double>(const double4a *p) {
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    double4a r;
    r.x = a.x;
    r.y = a.y;
    r.z = b.x;
    r.w = b.y;
    return r;
}

/* Streaming (evict-first) access for data touched once per step -- the
 * velocity / reference-position state -- so that it does not push out of L2
 * the positions and orientations that the next step gathers again.  The
 * neighbour rows, which every warp prefetches into L1 first, are read through
 * the read-only path. */
template<class R> __device__ __forceinline__ typename Vec<R>::T4 ldcs4(const typename Vec<R>::T4 *p);
template<> __device__ __forceinline__ float4 ldcs4<float>(const float4 *p) { return __ldcs(p); }
template<> __device__ __forceinline__ double4a ldcs4<double>(const double4a *p) {
    const double2 a = __ldcs(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldcs(reinterpret_cast<const double2 *>(p) + 1);
    double4a r;
    r.x = a.x;
    r.y = a.y;
    r.z = b.x;
    r.w = b.y;
    return r;
}
__device__ __forceinline__ void stcs4(float4 *p, const float4 &v) { __stcs(p, v); }
__device__ __forceinline__ void stcs4(double4a *p, const double4a &v) {
    __stcs(reinterpret_cast<double2 *>(p), make_double2(v.x, v.y));
    __stcs(reinterpret_cast<double2 *>(p) + 1, make_double2(v.z, v.w));
}

__device__ __forceinline__ void inv_sqrt(float r2, float &r, float &rinv) {
    rinv = rsqrtf(r2);
    r = r2 * rinv;
}
/* FP64: 1/sqrt(r2) by Newton's iteration for the reciprocal square root,
 * y <- y (3 - r2 y^2) / 2, started from the FP32 hardware estimate.  The
 * relative error e goes to about 1.5 e^2 per step (1e-7 -> 2e-14 -> below
 * the FP64 rounding), so two steps leave only a few ulp of rounding; the
 * protein pairs that call it have 1e-5 < r2 < 7, well inside the FP32 range. */
__device__ __forceinline__ void inv_sqrt(double r2, double &r, double &rinv) {
    double y = double(rsqrtf(float(r2)));
    y = y * (1.5 - 0.5 * r2 * y * y);
    y = y * (1.5 - 0.5 * r2 * y * y);
    rinv = y;
    r = r2 * y;
}
__device__ __forceinline__ float rnorm3(float x, float y, float z) { return rsqrtf(x * x + y * y + z * z); }
__device__ __forceinline__ double rnorm3(double x, double y, double z) { return 1.0 / sqrt(x * x + y * y + z * z); }

/* Lennard-Jones with the WCA cut (src/pairwise_kernel_fused.h:63-77). */
template<class R, bool E>
__device__ __forceinline__ void ljf(const PairP<R> &P, R dx, R dy, R dz, R r2, R3<R> &f, R &e) {
    const R r2inv = R(1) / r2;
    const R r6inv = r2inv * r2inv * r2inv;
    const R fpair = r6inv * (P.lj1 * r6inv - P.lj2) * r2inv;
    f.x += dx * fpair;
    f.y += dy * fpair;
    f.z += dz * fpair;
    if (E) e += R(0.5) * r6inv * (P.lj1 * (R(1) / R(12)) * r6inv - P.lj2 * (R(1) / R(6)));
}

/* Protein-protein repulsion (src/pairwise_kernel_fused.h:79-97). */
template<class R, bool E>
__device__ __forceinline__ void repf(const PairP<R> &P, R dx, R dy, R dz, R r2, R3<R> &f, R &e) {
    R r, rinv;
    inv_sqrt(r2, r, rinv);
    const R rc = P.cut - r;
    const R rc3 = rc * rc * rc;
    const R rc4 = rc * rc3;
    const R fr = P.rep8 * rc3 * rc4 * rinv;
    f.x += fr * dx;
    f.y += fr * dy;
    f.z += fr * dz;
    if (E) e += R(0.5) * P.rep * rc4 * rc4;
}

/* Dispatch of src/compute_pairwise_fused.h:91-236 for a pair without an
 * anisotropic interaction. */
template<class R, bool E>
__device__ __forceinline__ void pair_general(const PairP<R> &P, R dx, R dy, R dz, R r2, R3<R> &f, R &e) {
    if (!(r2 > R(1e-5))) return;
    if (r2 < P.cutsq)
        repf<R, E>(P, dx, dy, dz, r2, f, e);
    else if (r2 < P.ljcutsq)
        ljf<R, E>(P, dx, dy, dz, r2, f, e);
}
__device__ __forceinline__ int wrap_delta(int d, int n) {
    if (2 * d >= n) return d - n;
    if (2 * d < -n) return d + n;
    return d;
}

/* x_j - x_i from the packed cells and offsets (minimum image on periodic axes). */
template<class R, class T4>
__device__ __forceinline__ void rel_pos(const SysDev &sd, int cj, int ci, const T4 &pj, const T4 &pi, R &dx, R &dy,
                                        R &dz) {
    int d0 = cx_of(cj) - cx_of(ci), d1 = cy_of(cj) - cy_of(ci), d2 = cz_of(cj) - cz_of(ci);
    if (sd.per[0]) d0 = wrap_delta(d0, sd.nc[0]);
    if (sd.per[1]) d1 = wrap_delta(d1, sd.nc[1]);
    if (sd.per[2]) d2 = wrap_delta(d2, sd.nc[2]);
    dx = R(d0) * lc_of<R>(sd, 0) + (pj.x - pi.x);
    dy = R(d1) * lc_of<R>(sd, 1) + (pj.y - pi.y);
    dz = R(d2) * lc_of<R>(sd, 2) + (pj.z - pi.z);
}

/* Bond force on i, F_i = kappa(r) (x_j - x_i):  HARMONIC is
 * src/compute_bonded.h:109-115; FENE (expand form) and WLC + 1/r^2 (zero
 * force at r0) are the spectrin springs of the whole-cell workloads. */
template<class R, bool E>
__device__ __forceinline__ R bond_kappa(const BondP<R> &B, R r0, R r, R &e, int &flags) {
    if (B.style == BOND_HARMONIC) {
        if (E) e += R(0.25) * B.K * (r - r0) * (r - r0);
        return B.K * (R(1) - r0 / r);
    } else if (B.style == BOND_FENE) {
        const R s = (r - r0) / B.Rm;
        R s2 = s * s;
        if (s2 >= R(0.99)) {
            flags |= ERRB_BOND;
            s2 = R(0.99);
        }
        if (E) e += R(-0.25) * B.K * B.Rm * B.Rm * R(log(1.0 - double(s2)));
        return B.K * (r - r0) / (r * (R(1) - s2));
    } else {
        const R lmax = B.Rm * r0;
        R x = r / lmax;
        if (x >= R(0.99)) {
            flags |= ERRB_BOND;
            x = R(0.99);
        }
        const R x0 = r0 / lmax;
        const R omx = R(1) - x, omx0 = R(1) - x0;
        const R fw = B.K * (R(0.25) / (omx * omx) - R(0.25) + x);
        const R fw0 = B.K * (R(0.25) / (omx0 * omx0) - R(0.25) + x0);
        const R q = r0 / r;
        if (E) {
            const R uw = B.K * lmax * (x * x * R(0.5) + R(0.25) / (R(1) - x) - x * R(0.25) - R(0.25));
            e += R(0.5) * (uw + fw0 * r0 * q);
        }
        return (fw - fw0 * q * q) / r;
    }
}

/* s += d with Kahan compensation c (one component). */
template<class R> __device__ __forceinline__ void kahan_add(R &s, R &c, R d) {
    const R y = d - c;
    const R t = s + y;
    c = (t - s) - y;
    s = t;
}

/* The 27 cell shifts of the list entries, already multiplied by the cell
 * size: x_i - x_j = (o_i - o_j) + shift(code) (a shift of -1, 0 or +1 cells
 * times Lc is exact, so this rounds as the unscaled product would).  One table
 * per warp (which never straddles two systems), one array per axis: three
 * 4-byte lookups by 32 lanes are three conflict-free wavefronts of the L1 data
 * pipe that the gathers need too, one 16-byte lookup takes more than five. */
template<class R> struct ShiftTab {
    R v[3][32];
};
template<> struct ShiftTab<double> {
    double v[3][32];
    float f[3][32];  // rounded, for the shell test
    float slack;     // bound on the relative error of the rounded r^2 (rounding_slack)
};
template<class R> __device__ __forceinline__ void init_shift(const SysDev &sd, ShiftTab<R> &sh) {
    const int lane = threadIdx.x & 31;
    if (lane < 27) {
        sh.v[0][lane] = R(-(lane % 3 - 1)) * lc_of<R>(sd, 0);
        sh.v[1][lane] = R(-((lane / 3) % 3 - 1)) * lc_of<R>(sd, 1);
        sh.v[2][lane] = R(-(lane / 9 - 1)) * lc_of<R>(sd, 2);
        if constexpr (sizeof(R) == 8)
            for (int d = 0; d < 3; ++d) sh.f[d][lane] = float(sh.v[d][lane]);
        if constexpr (sizeof(R) == 8)
            if (lane == 0) sh.slack = rounding_slack(sd);
    }
    __syncwarp();
}
/* Whether the pair of a shell row is inside r^2 < lim, for the FP64 form: in
 * FP32 where the rounding of the coordinates cannot change the answer
 * (rounding_slack), and by the FP64 distance in the thin shell that remains. */
__device__ __forceinline__ bool shell_inside(const ShiftTab<double> &sh, const double4a &pi, const double4a &pj, int c,
                                             double lim) {
    const float fx = float(pi.x) - float(pj.x) + sh.f[0][c], fy = float(pi.y) - float(pj.y) + sh.f[1][c],
                fz = float(pi.z) - float(pj.z) + sh.f[2][c];
    const float r2 = fx * fx + fy * fy + fz * fz, l = float(lim);
    if (r2 < l * (1.f - sh.slack)) return true;
    if (r2 > l * (1.f + sh.slack)) return false;
    const double dx = __dadd_rn(__dadd_rn(pi.x, -pj.x), sh.v[0][c]);
    const double dy = __dadd_rn(__dadd_rn(pi.y, -pj.y), sh.v[1][c]);
    const double dz = __dadd_rn(__dadd_rn(pi.z, -pj.z), sh.v[2][c]);
    return __fma_rn(dz, dz, __fma_rn(dy, dy, __dmul_rn(dx, dx))) < lim;
}

/* ------------------------------------------------------------------------- */
/* Pair sums of a slot                                                       */
/* ------------------------------------------------------------------------- */
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }

/* 1/sqrt(r2) for 1e-5 <= r2: the hardware estimate in FP32; in FP64 one
 * third-order step from it, y (1 + e/2 + 3 e^2 / 8) with e = 1 - r2 y^2: the
 * error e of the estimate (3e-7) leaves 5 e^3 / 16 < 1e-20, below FP64
 * rounding, in five FP64 operations. */
__device__ __forceinline__ float rsqrt_pair(float r2) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(r2));
    return y;
}
__device__ __forceinline__ double rsqrt_pair(double r2) {
    const double y = double(rsqrt_pair(float(r2)));
    const double e = fma_rn(-mul_rn(r2, y), y, 1.0);
    return fma_rn(mul_rn(fma_rn(e, 0.375, 0.5), e), y, y);
}

/* r2 > 1e-5 and max(x, 0).  In FP64 on the integer pipe, as an FP64 comparison
 * takes as long as a multiplication there: numbers above a positive one
 * compare as their bits do (infinity included, the NaNs above it not). */
__device__ __forceinline__ bool apart(float r2) { return r2 > 1e-5f; }
__device__ __forceinline__ bool apart(double r2) {
    const long long b = __double_as_longlong(r2);
    return b > __double_as_longlong(1e-5) && b <= 0x7ff0000000000000LL;
}
/* infinite or not a number, and +-0, on the integer pipe for the same reason */
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_int(x) & 0x7f800000) == 0x7f800000; }
__device__ __forceinline__ bool not_finite(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }
__device__ __forceinline__ bool is_zero(float x) { return (__float_as_int(x) << 1) == 0; }
__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }
__device__ __forceinline__ float positive_part(float x) { return fmaxf(x, 0.f); }
__device__ __forceinline__ double positive_part(double x) { return __double2hiint(x) < 0 ? 0.0 : x; }

/* The anisotropic pair with a lipid j, by the owner's own parameters, in the
 * form that keeps the neighbour's vectors outermost:
 *   f = sum (cu d + kj n_j) + n_i sum kd,   t = sum (kd d - au n_j)
 * with d = x_i - x_j, niu = n_i.d / r, nju = n_j.d / r and the coefficients of
 * src/pairwise_kernel.h:30-68.  Pairs outside the range enter with r_c - r
 * clamped to 0, so that every coefficient vanishes and no branch is needed; a
 * normal that is not a number would still get through (0 x NaN), so IN_RANGE
 * leaves such pairs out by a branch, for the rare warp that meets one.  Each
 * operation is rounded as written, so the sums do not depend on how the
 * loops around them are compiled. */
template<class R> struct OwnP {
    R cut, rep8, a0, a1, aatt, hrep;  // a0 = 4 att (1 - alpha), a1 = 4 att alpha, hrep = rep / 2
};
constexpr int SHELL_U = 2;  // shell rows tested together
template<class R> __device__ __forceinline__ OwnP<R> own_params(const PairP<R> &q) {
    OwnP<R> P;
    P.cut = q.cut;
    P.rep8 = q.rep8;
    P.a1 = q.att4 * q.alpha;
    P.a0 = q.att4 - P.a1;
    P.aatt = q.aatt;
    P.hrep = R(0.5) * q.rep;
    return P;
}
constexpr int NACC = 7;  // force (3), torque (3), coefficient of n_i
template<class R, bool K> struct PairAcc {
    R s[NACC], c[K ? NACC : 1], e;  // sums, Kahan compensations, energy
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < NACC; ++k) s[k] = R(0);
#pragma unroll
        for (int k = 0; k < (K ? NACC : 1); ++k) c[k] = R(0);
        e = R(0);
    }
};
template<class R, bool E, bool K, bool IN_RANGE>
__device__ __forceinline__ void pair_term(PairAcc<R, K> &A, const OwnP<R> &P, const R d[3], const R n[3], R nix, R niy,
                                          R niz) {
    const R r2 = fma_rn(d[2], d[2], fma_rn(d[1], d[1], mul_rn(d[0], d[0])));
    const R r2c = apart(r2) ? r2 : R(1e30);  // coinciding particles: no force, as outside the range
    const R ri = rsqrt_pair(r2c);
    const R rc = positive_part(fma_rn(-r2c, ri, P.cut));
    const R nn = fma_rn(niz, n[2], fma_rn(niy, n[1], mul_rn(nix, n[0])));
    const R niu = mul_rn(fma_rn(niz, d[2], fma_rn(niy, d[1], mul_rn(nix, d[0]))), ri);
    const R nju = mul_rn(fma_rn(n[2], d[2], fma_rn(n[1], d[1], mul_rn(n[0], d[0]))), ri);
    const R A4 = fma_rn(mul_rn(niu, nju), -P.a1, fma_rn(nn, P.a1, P.a0));  // 4 att A
    const R rc2 = mul_rn(rc, rc), rc4 = mul_rn(rc2, rc2);
    const R fra = mul_rn(mul_rn(rc2, rc), fma_rn(P.rep8, rc4, A4));
    const R au = mul_rn(P.aatt, rc4);
    const R auar = mul_rn(au, ri);
    const R kd = mul_rn(auar, nju), kj = mul_rn(auar, niu);
    const R cu = mul_rn(fma_rn(kd, mul_rn(niu, R(-2)), fra), ri);
    if (IN_RANGE && !(rc > R(0))) return;
    if (K) {
#pragma unroll
        for (int k = 0; k < NACC; ++k) {
            const R t = k < 3   ? fma_rn(cu, d[k % 3], mul_rn(kj, n[k % 3]))
                        : k < 6 ? fma_rn(kd, d[k % 3], -mul_rn(au, n[k % 3]))
                                : kd;
            kahan_add(A.s[k], A.c[k], t);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            A.s[k] = fma_rn(cu, d[k], fma_rn(kj, n[k], A.s[k]));
            A.s[3 + k] = fma_rn(kd, d[k], fma_rn(-au, n[k], A.s[3 + k]));
        }
        A.s[6] = add_rn(A.s[6], kd);
    }
    if (E) A.e = fma_rn(rc4, fma_rn(P.hrep, rc4, mul_rn(A4, R(0.125))), A.e);  // half of rep rc^8 + A att rc^4
}

/* Bring the used rows of this warp's block of neighbour entries (read once
 * per step) into L1 ahead of the pair loops, so the loops' entry loads do not
 * wait on DRAM.  packed = inner count | shell count << 16.  All 32 lanes must
 * call it. */
__device__ __forceinline__ void prefetch_warp_list(const uint32_t *nbr, int i, int cap, int packed) {
    const int rin = __reduce_max_sync(0xffffffffu, unsigned(packed & 0xffff));
    const int rout = __reduce_max_sync(0xffffffffu, unsigned(packed >> 16));
    const uint32_t *base = nbr + nbr_index(i & ~31, 0, cap);
    for (int r = int(threadIdx.x & 31); r < rin + rout; r += 32) {
        const int row = r < rin ? r : cap - 1 - (r - rin);
        asm volatile("prefetch.global.L1 [%0];" ::"l"(base + 32 * row));
    }
}

/* Resident blocks asked of the force kernels: FP32, 16 at 64 registers for
 * batches of two rows (14 at 72 with compensated sums, which need more), 10
 * for batches of four; the FP64 forms are bound by the FP64 pipe and keep all
 * the registers they need (16 blocks and more: 840 -> 850 us on a 250 thousand
 * particle cell). */
template<class R, bool K, int U> constexpr int force_blocks() {
    return sizeof(R) == 8 ? 1 : U == 2 ? (K ? 14 : 16) : 10;
}

/* Pair sums of slot i over its list.  Shell rows are tested first, 32 at a
 * time; a hit is a bit of a mask.  Then the inner rows and the hits go through
 * one loop, U of them at a time: their entries and gathers are issued together
 * and their terms added in row order, so the sums are the same for every U.  A
 * lipid's hits among the proteins that it has anisotropic pairs with take the
 * same arithmetic with their own parameters; the hits that need the general
 * pair table (two proteins, or a type without anisotropic pairs: the list
 * build puts all of these in the shell rows) follow if they are in range.  All
 * 32 lanes of the warp must call it.
 *
 * Bound by the L2 latency of the gathers (every row of a warp waits for its
 * slowest lane) and, behind it, by issue and the L1 data pipe.  On the
 * 1.0M-particle cell a warp spends 9 of 42 thousand cycles on the shell rows, 23
 * on the others, 5 before and 5 after.  A cell with 17 % proteins (0.91M
 * particles) has a lane without anisotropic pairs in almost every warp: 160 us
 * per step kernel against 183 with such lanes left out of the loop without
 * selection, their general hits walked unconditionally and the lipids'
 * protein pairs in a branch of their own; FP64, 0.23M particles, 860 -> 740. */
template<class R, bool E, bool K, int U, bool IN_RANGE>
__device__ __forceinline__ void pair_sums(const KArgs<R> &a, const FFDev<R> &F, const OwnP<R> &P, int i,
                                          const typename Vec<R>::T4 *__restrict__ pos,
                                          const typename Vec<R>::T4 *__restrict__ nrm, int ty, int packed,
                                          const typename Vec<R>::T4 &pi, const typename Vec<R>::T4 &ni,
                                          const ShiftTab<R> &sh, PairAcc<R, K> &A) {
    using T4 = typename Vec<R>::T4;
    int nin = packed & 0xffff;
    const int nout = packed >> 16;
    const uint32_t *__restrict__ nb = a.nbr + nbr_index(i, 0, a.cap);
    const uint32_t *__restrict__ shell = nb + int64_t(a.cap - 1) * 32;  // shell rows run downwards
    const uint32_t self = uint32_t(i) | (13u << NB_SHIFT);              // distance 0: contributes nothing
    auto offset = [&](uint32_t ent, const T4 &pj, R d[3]) {
        const int c = int(ent >> NB_SHIFT);
        d[0] = add_rn(add_rn(pi.x, -pj.x), sh.v[0][c]);
        d[1] = add_rn(add_rn(pi.y, -pj.y), sh.v[1][c]);
        d[2] = add_rn(add_rn(pi.z, -pj.z), sh.v[2][c]);
    };
    auto dist2 = [&](const R d[3]) { return fma_rn(d[2], d[2], fma_rn(d[1], d[1], mul_rn(d[0], d[0]))); };
    auto term = [&](uint32_t ent, const T4 &pj, const T4 &nj) {
        R d[3];
        const R n[3] = {nj.x, nj.y, nj.z};
        offset(ent, pj, d);
        pair_term<R, E, K, IN_RANGE>(A, P, d, n, ni.x, ni.y, ni.z);
    };
    for (int k0 = 0;; k0 += 32) {
        uint32_t hm = 0u, hb = 0u;  // hits: for the rows' loop, for the general table
        const R lim = F.reach2[ty];
        const int nq = min(32, nout - k0);
        const int nqmax = int(__reduce_max_sync(0xffffffffu, unsigned(max(nq, 0))));
        for (int k = 0; k < nqmax; k += SHELL_U) {
            uint32_t ent[SHELL_U];
            T4 pj[SHELL_U];
#pragma unroll
            for (int u = 0; u < SHELL_U; ++u) ent[u] = k + u < nq ? __ldg(shell - (k + u + k0) * 32) : self;
#pragma unroll
            for (int u = 0; u < SHELL_U; ++u) pj[u] = ldg4<R>(pos + (ent[u] & NB_MASK));
#pragma unroll
            for (int u = 0; u < SHELL_U; ++u) {
                if constexpr (sizeof(R) == 8) {
                    const bool in = shell_inside(sh, pi, pj[u], int(ent[u] >> NB_SHIFT), lim);
                    if (k + u < nq && in) {
                        // the general pairs are told apart here, each by its own range: a row of the loop
                        // below costs the FP64 pipe 60 operations
                        const PairP<R> &q = F.pair[ty * NT + w_type(wbits(pj[u].w))];
                        if (q.kind == PAIR_ANISO)
                            hm |= 1u << (k + u);
                        else if (shell_inside(sh, pi, pj[u], int(ent[u] >> NB_SHIFT), q.anysq))
                            hb |= 1u << (k + u);
                    }
                } else {
                    R d[3];
                    offset(ent[u], pj[u], d);
                    if (k + u < nq && dist2(d) < lim) hm |= 1u << (k + u);
                }
            }
        }
        // rows that every lane still has inside (rounded down to whole batches): no selection.  A lane without
        // anisotropic pairs has no rows, and goes along on those of a lane that has: its own parameters make
        // them vanish
        const unsigned with = k0 == 0 ? __ballot_sync(0xffffffffu, P.cut > R(0)) : 0u;
        int kmin = 0;
        if (with) {
            kmin = int(__reduce_min_sync(0xffffffffu, unsigned(P.cut > R(0) ? nin : 0xffff))) / U * U;
            if (!(P.cut > R(0))) {
                nin = kmin;
                nb += __ffs(int(with)) - 1 - int(threadIdx.x & 31);
            }
        }
#pragma unroll 1
        for (int k = 0; k < kmin; k += U) {
            uint32_t ent[U];
            T4 pj[U], nj[U];
#pragma unroll
            for (int u = 0; u < U; ++u) ent[u] = __ldg(nb + (k + u) * 32);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                pj[u] = ldg4<R>(pos + (ent[u] & NB_MASK));
                nj[u] = ldg4<R>(nrm + (ent[u] & NB_MASK));
            }
#pragma unroll
            for (int u = 0; u < U; ++u) term(ent[u], pj[u], nj[u]);
        }
        nb = a.nbr + nbr_index(i, 0, a.cap);
        const int total = int(__reduce_max_sync(0xffffffffu, unsigned(nin + __popc(hm))));
        for (int k = kmin; k < total; k += U) {
            uint32_t ent[U], bit[U];
            T4 pj[U], nj[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool in = k + u < nin;
                bit[u] = in ? 0u : hm & (0u - hm);
                hm ^= bit[u];
                const int row = in ? k + u : a.cap - 1 - k0 - (31 - __clz(int(bit[u])));
                ent[u] = (in || bit[u]) ? __ldg(nb + row * 32) : self;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                pj[u] = ldg4<R>(pos + (ent[u] & NB_MASK));
                nj[u] = ldg4<R>(nrm + (ent[u] & NB_MASK));
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int tj = w_type(wbits(pj[u].w));
                OwnP<R> Q = P;
                R d[3], n[3] = {nj[u].x, nj[u].y, nj[u].z};
                offset(ent[u], pj[u], d);
                if (bit[u] && (tj != 0 || !(P.cut > R(0)))) {
                    // a lipid's pair with a protein has parameters of its own; the rest waits
                    const PairP<R> &q = F.pair[ty * NT + tj];
                    if (ty == 0 && q.kind == PAIR_ANISO) {
                        Q = own_params(q);
                    } else {
                        Q.cut = R(0);
                        n[0] = n[1] = n[2] = R(0);
                        if (dist2(d) < q.anysq) hb |= bit[u];
                    }
                }
                pair_term<R, E, K, IN_RANGE>(A, Q, d, n, ni.x, ni.y, ni.z);
            }
        }
        // the general pairs among the hits
        while (hb) {
            const int k = __ffs(int(hb)) - 1;
            hb &= hb - 1u;
            const uint32_t ent = __ldg(shell - int64_t(k + k0) * 32);
            const T4 pj = ldg4<R>(pos + (ent & NB_MASK));
            R d[3], ee = 0;
            offset(ent, pj, d);
            R3<R> df = {0, 0, 0};
            pair_general<R, E>(F.pair[ty * NT + w_type(wbits(pj.w))], d[0], d[1], d[2], dist2(d), df, ee);
            const R v[3] = {df.x, df.y, df.z};
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                if (K)
                    kahan_add(A.s[q], A.c[K ? q : 0], v[q]);
                else
                    A.s[q] = add_rn(A.s[q], v[q]);
            }
            if (E) A.e = add_rn(A.e, ee);
        }
        if (!__any_sync(0xffffffffu, nout > k0 + 32)) break;
        nin = 0;
    }
}

/* Force of bond b and of face b on the vertex in slot i. */
template<class R, bool E>
__device__ __forceinline__ R3<R> bond_force(const KArgs<R> &a, const FFDev<R> &F, int i, int b, int lp,
                                            const typename Vec<R>::T4 *__restrict__ pos,
                                            const typename Vec<R>::T4 &pi, int ci, const SysDev &sd, R &e, int &flags) {
    const BondSlot bs = a.bond[lp][int64_t(b) * a.npad + i];
    const typename Vec<R>::T4 pj = pos[bs.partner];
    R dx, dy, dz;
    rel_pos<R>(sd, a.cell[lp][bs.partner], ci, pj, pi, dx, dy, dz);
    const R r = sqrt(dx * dx + dy * dy + dz * dz);
    const R kap = bond_kappa<R, E>(F.bond[bs.type], R(bs.r0), r, e, flags);
    return {kap * dx, kap * dy, kap * dz};
}
template<class R>
__device__ __forceinline__ R3<R> face_force(const KArgs<R> &a, int i, int b, int lp,
                                            const typename Vec<R>::T4 *__restrict__ pos,
                                            const typename Vec<R>::T4 &pi, int ci, const SysDev &sd, R cv, R ca) {
    const int2 fs = a.fslot[lp][int64_t(b) * a.npad + i];
    R bx, by, bz, cx, cy, cz;
    rel_pos<R>(sd, a.cell[lp][fs.x], ci, pos[fs.x], pi, bx, by, bz);
    rel_pos<R>(sd, a.cell[lp][fs.y], ci, pos[fs.y], pi, cx, cy, cz);
    const R nx = by * cz - bz * cy, ny = bz * cx - bx * cz, nz = bx * cy - by * cx;  // 6 dV/da
    const R inn = rnorm3(nx, ny, nz);
    const R hx = nx * inn, hy = ny * inn, hz = nz * inn;
    const R ex = bx - cx, ey = by - cy, ez = bz - cz;
    const R gx = ey * hz - ez * hy, gy = ez * hx - ex * hz, gz = ex * hy - ey * hx;  // 2 dA/da
    return {cv * nx + ca * gx, cv * ny + ca * gy, cv * nz + ca * gz};
}

/* Bonds and the mesh constraint of slot i, added to f in order.  A membrane
 * has few vertices (0.8 % of the 4M-particle cell), each with about six bonds
 * and six faces, so a warp's one or two vertices would walk a dozen dependent
 * gathers alone: where a warp holds fewer vertices than its longest walk, its
 * lanes take one bond or face each of one vertex after the other, and the
 * owner adds their forces in the same order.  All 32 lanes must call it. */
template<class R, bool E, bool K>
__device__ __forceinline__ void bond_mesh_forces(const KArgs<R> &a, const FFDev<R> &F, int i, int cur, int lp, int w,
                                                 const typename Vec<R>::T4 &pi, const SysDev &sd, const SysState &ss,
                                                 R3<R> &f, R &e, int &flags) {
    using T4 = typename Vec<R>::T4;
    const bool real = w_type(w) != GHOST;
    const int bd = real ? w_bdeg(w) : 0;
    int fd = real ? w_fdeg(w) : 0;
    if (!__any_sync(0xffffffffu, (bd | fd) != 0)) return;
    const R cv = R(ss.cv) * R(1.0 / 6.0), ca = R(ss.ca) * R(0.5);
    if (ss.cv == 0.0 && ss.ca == 0.0) fd = 0;
    const T4 *__restrict__ pos = a.pos[cur];
    const int ci = bd + fd > 0 ? a.cell[lp][i] : 0;
    R3<R> c = {0, 0, 0};
    auto accumulate = [&](const R3<R> &d) {
        if (K) {
            kahan_add(f.x, c.x, d.x);
            kahan_add(f.y, c.y, d.y);
            kahan_add(f.z, c.z, d.z);
        } else {
            f.x += d.x;
            f.y += d.y;
            f.z += d.z;
        }
    };
    unsigned todo = __ballot_sync(0xffffffffu, bd + fd > 0);
    if (__popc(todo) >= int(__reduce_max_sync(0xffffffffu, unsigned(bd + fd)))) {
        for (int b = 0; b < bd; ++b) {
            R eb = 0;
            accumulate(bond_force<R, E>(a, F, i, b, lp, pos, pi, ci, sd, eb, flags));
            if (E) e += eb;
        }
        for (int b = 0; b < fd; ++b) accumulate(face_force<R>(a, i, b, lp, pos, pi, ci, sd, cv, ca));
        return;
    }
    const int lane = threadIdx.x & 31;
    while (todo) {
        const int o = __ffs(int(todo)) - 1;
        todo &= todo - 1u;
        const int obd = __shfl_sync(0xffffffffu, bd, o), ofd = __shfl_sync(0xffffffffu, fd, o);
        const int oi = __shfl_sync(0xffffffffu, i, o), oci = __shfl_sync(0xffffffffu, ci, o);
        T4 op = pi;
        op.x = __shfl_sync(0xffffffffu, pi.x, o);
        op.y = __shfl_sync(0xffffffffu, pi.y, o);
        op.z = __shfl_sync(0xffffffffu, pi.z, o);
        R3<R> d = {0, 0, 0};
        R eb = 0;
        if (lane < obd)
            d = bond_force<R, E>(a, F, oi, lane, lp, pos, op, oci, sd, eb, flags);
        else if (lane < obd + ofd)
            d = face_force<R>(a, oi, lane - obd, lp, pos, op, oci, sd, cv, ca);
        for (int b = 0; b < obd + ofd; ++b) {
            const R3<R> db = {__shfl_sync(0xffffffffu, d.x, b), __shfl_sync(0xffffffffu, d.y, b),
                              __shfl_sync(0xffffffffu, d.z, b)};
            const R ee = E ? __shfl_sync(0xffffffffu, eb, b) : R(0);
            if (lane == o) {
                accumulate(db);
                if (E && b < obd) e += ee;
            }
        }
    }
}

/* All forces and torques on slot i (all 32 lanes of the warp must call it; a
 * ghost's are zero). */
template<class R, bool E, bool K, int U>
__device__ __forceinline__ void slot_forces(const KArgs<R> &a, const FFDev<R> &F, int i, int cur, int lp, int w,
                                            const typename Vec<R>::T4 &pi, const typename Vec<R>::T4 &ni,
                                            const SysDev &sd, const SysState &ss, int packed,
                                            const ShiftTab<R> &sh, R3<R> &f, R3<R> &t, R &e, int &flags) {
    using T4 = typename Vec<R>::T4;
    const bool real = w_type(w) != GHOST;
    const int ty = real ? w_type(w) : 0;
    const PairP<R> &pl = F.pair[ty * NT];  // with a lipid
    const OwnP<R> P = own_params(pl);
    PairAcc<R, K> A;
    A.clear();
    T4 na = ni;  // not used by a type without anisotropic pairs, which may carry anything there
    if (!(P.cut > R(0))) na.x = na.y = na.z = R(0);
    const T4 *__restrict__ pos = a.pos[cur], *__restrict__ nrm = a.nrm[cur];
    pair_sums<R, E, K, U, false>(a, F, P, i, pos, nrm, ty, packed, pi, na, sh, A);
    // (a normal that is not a number or infinite makes the coefficient of d and so every component of f one)
    if (__any_sync(0xffffffffu, not_finite(A.s[0]))) {
        // again with the pairs in range alone.  What the sums take is read anew: kept in registers until here,
        // it would cost the common path spills
        asm volatile("" ::: "memory");
        const PairP<R> &pl2 = F.pair[ty * NT];
        A.clear();
        pair_sums<R, E, K, 1, true>(a, F, own_params(pl2), i, pos, nrm, ty, __ldcg(a.nnb + i), pi, na, sh, A);
    }
    if (is_zero(A.s[6])) na.x = na.y = na.z = R(0);
    if (K) {
#pragma unroll
        for (int k = 0; k < NACC; ++k) A.s[k] = add_rn(A.s[k], -A.c[K ? k : 0]);
    }
    f.x = fma_rn(A.s[6], na.x, A.s[0]);
    f.y = fma_rn(A.s[6], na.y, A.s[1]);
    f.z = fma_rn(A.s[6], na.z, A.s[2]);
    t.x = A.s[3];
    t.y = A.s[4];
    t.z = A.s[5];
    e = A.e;
    bond_mesh_forces<R, E, K>(a, F, i, cur, lp, w, pi, sd, ss, f, e, flags);
}

__device__ __forceinline__ void philox4(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0, uint32_t k1,
                                        uint32_t o[4]) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
        const uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
        const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0;
        c1 = lo1;
        c2 = n2;
        c3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    o[0] = c0;
    o[1] = c1;
    o[2] = c2;
    o[3] = c3;
}
__device__ __forceinline__ void philox3(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0, uint32_t k1,
                                        uint32_t &o0, uint32_t &o1, uint32_t &o2) {
    uint32_t o[4];
    philox4(c0, c1, c2, c3, k0, k1, o);
    o0 = o[0];
    o1 = o[1];
    o2 = o[2];
}
template<class R> __device__ __forceinline__ R u11(uint32_t u) { return R(u >> 8) * R(1.0 / 8388608.0) - R(1); }


/* Reflective walls (src/integrate_nh.h:124-144) on the axes where the system
 * has them (wlo < whi), applied in the frame of the particle's cell. */
template<class R>
__device__ __forceinline__ void bounce_walls(const SysDev &sd, int c, typename Vec<R>::T4 &p, typename Vec<R>::T4 &v) {
    const int cc[3] = {cx_of(c), cy_of(c), cz_of(c)};
    R *pp[3] = {&p.x, &p.y, &p.z};
    R *vv[3] = {&v.x, &v.y, &v.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (!(sd.wlo[d] < sd.whi[d])) continue;
        const double center = sd.lo[d] + (double(cc[d]) + 0.5) * sd.Lc[d];
        const R lo = R(sd.wlo[d] - center), hi = R(sd.whi[d] - center);
        if (*pp[d] < lo) {
            *pp[d] = lo + (lo - *pp[d]);
            *vv[d] = -*vv[d];
        } else if (*pp[d] > hi) {
            *pp[d] = hi - (*pp[d] - hi);
            *vv[d] = -*vv[d];
        }
    }
}

enum { MODE_LANGEVIN = 0, MODE_NH_FINAL = 1, MODE_NH_INITIAL = 2, MODE_FORCES = 3, MODE_VCOM = 4 };

/* Per-system sums, first level.  Every warp reduces its particles' values --
 * the sums in the working precision (in mixed mode the FP64 pipe would cost
 * more than the force loop), the maximum and the flags on integers -- and
 * lane 0 stores them in FP64 as the warp's partial.  No barrier, fence or
 * atomic: k_reduce, launched next on the stream, sums each system's partials
 * in a fixed order.  Partial layout: ke2, epot, max displacement^2, error
 * flags, lipid sum v (3).  All 32 lanes of the warp must call it; i is the
 * caller's slot (a warp never straddles two systems). */
template<class R>
__device__ __forceinline__ void warp_partials(const KArgs<R> &a, int i, R ke, R ep, float md2, int flags,
                                              R vx = R(0), R vy = R(0), R vz = R(0)) {
    R v[5] = {ke, ep, vx, vy, vz};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 5; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
    // md2 >= 0 (or NaN, flagged separately): the bit order is the value order
    const unsigned wmax = __reduce_max_sync(0xffffffffu, __float_as_uint(md2));
    const int wfl = int(__reduce_or_sync(0xffffffffu, unsigned(flags)));
    if ((threadIdx.x & 31) == 0) {
        double *p = a.partial + int64_t(i >> 5) * NPART;
        p[0] = double(v[0]);
        p[1] = double(v[1]);
        p[2] = double(__uint_as_float(wmax));
        p[3] = double(wfl);
        p[4] = double(v[2]);
        p[5] = double(v[3]);
        p[6] = double(v[4]);
    }
}

/* The larger of two numbers >= 0, or the one that is not a number, by their
 * bits: two FP64 comparisons per step of the tree instead cost k_reduce 2 us of
 * 20 (908 thousand particles). */
__device__ __forceinline__ double max_or_nan(double x, double y) {
    const unsigned long long a = __double_as_longlong(x), b = __double_as_longlong(y);
    return __longlong_as_double((long long)(a > b ? a : b));
}
__device__ __forceinline__ double combine_part(int k, double x, double y) {
    return k == 2 ? max_or_nan(x, y) : (k == 3 ? double(int(x) | int(y)) : x + y);
}

/* Per-system sums, second and third level, after a kernel that wrote warp
 * partials.  Block g sums the RED_GROUP warp partials of reduction group g
 * (RED_GROUP x 32 consecutive slots of one system) in a fixed-shape tree; the
 * last block to finish (ticket) gives each system to one warp, which adds the
 * system's group partials in a fixed order, and applies the mode's update:
 * thermostat, kinetic energy, potential energy, bulk velocity, rebuild rule,
 * step counter, buffer parity. */
template<class R> __global__ void __launch_bounds__(RED_GROUP) k_reduce(KArgs<R> a, int mode, int count_step) {
    if (halted(a.S)) {  // the kernel before it did nothing; its partials are stale
        if (a.has_cond && blockIdx.x == 0 && threadIdx.x == 0)
            cudaGraphSetConditional(a.cond, __ldcg(&a.S->rebuild) ? 1u : 0u);
        return;
    }
    __shared__ double red[7][RED_GROUP];
    __shared__ double wmax[RED_GROUP / 32];
    __shared__ int wfl[RED_GROUP / 32];
    __shared__ int last;
    const int g = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int s = 0;
    while (s + 1 < a.nsys && g >= a.sys[s + 1].gbase) ++s;
    const SysDev &sd = a.sys[s];
    const int gl = g - sd.gbase;
    const int64_t w0 = int64_t(sd.off / 32) + int64_t(gl) * RED_GROUP;
    const int nw = min(RED_GROUP, sd.npad / 32 - gl * RED_GROUP);
    for (int k = 0; k < 7; ++k) red[k][t] = t < nw ? __ldcg(a.partial + (w0 + t) * NPART + k) : 0.0;
    __syncthreads();
    for (int h = RED_GROUP / 2; h > 0; h >>= 1) {
        if (t < h)
            for (int k = 0; k < 7; ++k) red[k][t] = combine_part(k, red[k][t], red[k][t + h]);
        __syncthreads();
    }
    if (t == 0) {
        double *gp = a.gpartial + int64_t(g) * NPART;
        for (int k = 0; k < 7; ++k) gp[k] = red[k][0];
        __threadfence();
        last = atomicAdd(&a.S->blk_counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double mymax = 0.0;
    int myfl = 0;
    for (int q = warp; q < a.nsys; q += RED_GROUP / 32) {
        const SysDev &sq = a.sys[q];
        double v[7];
        for (int k = 0; k < 7; ++k) {
            double acc = 0.0;
            for (int u = lane; u < sq.ngrp; u += 32)
                acc = combine_part(k, acc, __ldcg(a.gpartial + int64_t(sq.gbase + u) * NPART + k));
            v[k] = acc;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            for (int k = 0; k < 7; ++k) v[k] = combine_part(k, v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
        if (lane == 0) {
            SysState &ss = a.ss[q];
            const double k2 = v[0], e = v[1];
            if ((mode == MODE_LANGEVIN || mode == MODE_NH_INITIAL || mode == MODE_VCOM) && sq.nlipid > 0) {
                ss.vcom[0] = v[4] / double(sq.nlipid);
                ss.vcom[1] = v[5] / double(sq.nlipid);
                ss.vcom[2] = v[6] / double(sq.nlipid);
            }
            if (mode == MODE_VCOM) {
                ss.ke2 = k2;
            } else if (mode == MODE_LANGEVIN || mode == MODE_FORCES) {
                if (mode == MODE_LANGEVIN) ss.ke2 = k2;
                ss.epot = e;
            } else {
                // zeta += dt/2Q (sum m v^2 / 2 - 3/2 N kT)  (src/integrate_nh.h:182-185, :241-244)
                const double nreal = double(sq.nreal);
                const double Q = sq.Q > 0 ? sq.Q : 0.01 * nreal;
                ss.zeta += 0.5 * a.dt / Q * (0.5 * k2 - 0.5 * 3.0 * nreal * a.kBT);
                ss.ke2 = k2;
                if (mode == MODE_NH_FINAL) ss.epot = e;
            }
            mymax = max_or_nan(v[2], mymax);
            myfl |= int(v[3]);
        }
    }
    if (lane == 0) {
        wmax[warp] = mymax;
        wfl[warp] = myfl;
    }
    __syncthreads();
    if (t == 0) {
        double m = 0.0;
        int fl = 0;
        for (int w = 0; w < RED_GROUP / 32; ++w) {
            m = max_or_nan(wmax[w], m);
            fl |= wfl[w];
        }
        Scalars *S = a.S;
        S->error |= fl;
        int rebuild = __ldcg(&S->rebuild);
        if (mode == MODE_LANGEVIN || mode == MODE_NH_INITIAL) {
            S->since_rebuild += 1;
            // (a position that is not a number counts as moved: the build drops its particle)
            if (!(m <= double(a.skin_half2)) || (a.rebuild_every > 0 && S->since_rebuild >= a.rebuild_every))
                S->rebuild = rebuild = 1;
        }
        if (mode == MODE_LANGEVIN) {
            S->cur ^= 1;
            S->step += 1;
            S->iters += 1;
        }
        if (mode == MODE_NH_INITIAL) S->nh_half = 1;
        if (mode == MODE_NH_FINAL) {
            S->nh_half = 0;
            if (count_step) {
                S->step += 1;
                S->iters += 1;
            }
        }
        S->blk_counter = 0;
        if (a.has_cond) cudaGraphSetConditional(a.cond, rebuild ? 1u : 0u);
        __threadfence();
    }
}

/* One particle of the fused Langevin step, given its forces and torques:
 * src/integrate_langevin.h:105-146 (rotation, then translation with the
 * counter-based noise).  Writes the new state; returns the squared
 * displacement since the list was built, sum m v^2 and the lipid velocity
 * (for the bulk-velocity removal). */
template<class R>
__device__ __forceinline__ void langevin_particle(const KArgs<R> &a, const FFDev<R> &F, int i, int s, int cur, int lp,
                                                  long long step, const typename Vec<R>::T4 &pi,
                                                  const typename Vec<R>::T4 &ni, int ty, bool zero_bulk, R3<R> f,
                                                  const R3<R> &t, R &ke, float &md2, int &flags, R &vsx, R &vsy,
                                                  R &vsz) {
    using T4 = typename Vec<R>::T4;
    const R dt = R(a.dt);
    T4 v = ldcs4<R>(&a.vel[lp][i]), o = ldcs4<R>(&a.omg[lp][i]);
    if (zero_bulk && ty == 0) {  // zero_bulk_velocity on the lipids (src/zero_bulk_velocity.h:38-45)
        v.x -= R(__ldcg(&a.ss[s].vcom[0]));
        v.y -= R(__ldcg(&a.ss[s].vcom[1]));
        v.z -= R(__ldcg(&a.ss[s].vcom[2]));
    }
    // ROTATION: t <- n x t; o += dt t; n <- normalize(n + (o x n) dt)
    const R tx = ni.y * t.z - ni.z * t.y, ty_ = ni.z * t.x - ni.x * t.z, tz = ni.x * t.y - ni.y * t.x;
    o.x += dt * tx;
    o.y += dt * ty_;
    o.z += dt * tz;
    const R gx = ni.x + (o.y * ni.z - o.z * ni.y) * dt;
    const R gy = ni.y + (o.z * ni.x - o.x * ni.z) * dt;
    const R gz = ni.z + (o.x * ni.y - o.y * ni.x) * dt;
    const R gi = rnorm3(gx, gy, gz);
    T4 nn = ni;
    nn.x = gx * gi;
    nn.y = gy * gi;
    nn.z = gz * gi;
    // TRANSLATION: f -= gamma v + sigma r; v += f dt/m; x += v dt
    uint32_t r0, r1, r2;
    philox3(uint32_t(__ldcs(&a.tag[lp][i])), uint32_t(step), uint32_t((unsigned long long)step >> 32), uint32_t(s),
            uint32_t(a.seed), uint32_t(a.seed >> 32), r0, r1, r2);
    const R gam = F.gamma[ty], sig = F.sigma[ty];
    const R dtm = dt * F.inv_mass[ty];
    f.x -= gam * v.x + sig * u11<R>(r0);
    f.y -= gam * v.y + sig * u11<R>(r1);
    f.z -= gam * v.z + sig * u11<R>(r2);
    v.x += f.x * dtm;
    v.y += f.y * dtm;
    v.z += f.z * dtm;
    T4 p = pi;
    p.x += v.x * dt;
    p.y += v.y * dt;
    p.z += v.z * dt;
    a.pos[cur ^ 1][i] = p;
    a.nrm[cur ^ 1][i] = nn;
    stcs4(&a.vel[lp][i], v);
    stcs4(&a.omg[lp][i], o);
    const T4 xr = ldcs4<R>(&a.xref[lp][i]);
    const R ddx = p.x - xr.x, ddy = p.y - xr.y, ddz = p.z - xr.z;
    md2 = float(ddx * ddx + ddy * ddy + ddz * ddz);
    if (!isfinite(p.x + p.y + p.z + v.x + v.y + v.z)) flags |= ERRB_NAN;
    ke = F.mass[ty] * (v.x * v.x + v.y * v.y + v.z * v.z);
    if (ty == 0) {
        vsx = v.x;
        vsy = v.y;
        vsz = v.z;
    }
}

/* Langevin step with the per-system sums (energy, bulk-velocity removal):
 * the structure of the lite kernel below plus warp partials, summed per
 * system by k_reduce after the kernel. */
template<class R, bool E, bool K, int U>
__global__ void __launch_bounds__(force_threads<R>, force_blocks<R, K, U>()) k_step_langevin(KArgs<R> a) {
    using T4 = typename Vec<R>::T4;
    __shared__ ShiftTab<R> shm[force_threads<R> / 32];
    const int i = blockIdx.x * force_threads<R> + threadIdx.x;
    // the loads that depend on nothing, together
    const int4 sc = __ldcg(reinterpret_cast<const int4 *>(a.S));  // cur, lp, rebuild, error
    const int s = a.nsys > 1 ? a.blk_sys[i / SYS_PAD] : 0;
    const int packed = a.nnb[i];
    if (halted(sc)) return;
    const int cur = sc.x, lp = sc.y;
    const FFDev<R> &F = *a.ff;
    prefetch_warp_list(a.nbr, i, a.cap, packed);
    ShiftTab<R> &sh = shm[threadIdx.x >> 5];
    init_shift<R>(a.sys[s], sh);
    const T4 pi = a.pos[cur][i], ni = a.nrm[cur][i];
    const int w = wbits(pi.w);
    R ke = 0, ep = 0, vsx = 0, vsy = 0, vsz = 0;
    float md2 = 0.f;
    int flags = 0;
    R3<R> f, t;
    slot_forces<R, E, K, U>(a, F, i, cur, lp, w, pi, ni, a.sys[s], a.ss[s], packed, sh, f, t, ep, flags);
    if (w_type(w) != GHOST)
        langevin_particle<R>(a, F, i, s, cur, lp, __ldcg(&a.S->step), pi, ni, w_type(w), a.zero_bulk != 0, f, t, ke,
                             md2, flags, vsx, vsy, vsz);
    warp_partials<R>(a, i, ke, ep, md2, flags, vsx, vsy, vsz);
}

/* Langevin step without per-system sums (no energy, no bulk-velocity
 * removal): small blocks that retire independently, the force-field table read
 * through the read-only path, and no end-of-block reduction -- a warp whose
 * particles moved more than skin/2 raises the rebuild flag itself, and
 * k_advance flips the buffers after the kernel.  The temperature is reduced on
 * demand (k_vcom). */
template<class R, bool K, int U>
__global__ void __launch_bounds__(force_threads<R>, force_blocks<R, K, U>()) k_step_langevin_lite(KArgs<R> a) {
    using T4 = typename Vec<R>::T4;
    __shared__ ShiftTab<R> shm[force_threads<R> / 32];
    const int i = blockIdx.x * force_threads<R> + threadIdx.x;
    // the loads that depend on nothing, together
    const int4 sc = __ldcg(reinterpret_cast<const int4 *>(a.S));  // cur, lp, rebuild, error
    const int s = a.nsys > 1 ? a.blk_sys[i / SYS_PAD] : 0;
    const int packed = a.nnb[i];
    if (halted(sc)) return;
    const int cur = sc.x, lp = sc.y;
    const FFDev<R> &F = *a.ff;
    prefetch_warp_list(a.nbr, i, a.cap, packed);
    ShiftTab<R> &sh = shm[threadIdx.x >> 5];
    init_shift<R>(a.sys[s], sh);
    const T4 pi = a.pos[cur][i], ni = a.nrm[cur][i];
    const int w = wbits(pi.w);
    R ke = 0, ep = 0, vsx = 0, vsy = 0, vsz = 0;
    float md2 = 0.f;
    int flags = 0;
    R3<R> f, t;
    slot_forces<R, false, K, U>(a, F, i, cur, lp, w, pi, ni, a.sys[s], a.ss[s], packed, sh, f, t, ep, flags);
    if (w_type(w) != GHOST)
        langevin_particle<R>(a, F, i, s, cur, lp, __ldcg(&a.S->step), pi, ni, w_type(w), false, f, t, ke, md2, flags,
                             vsx, vsy, vsz);
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(md2));  // md2 >= 0: bit order = value order
    const int fl = int(__reduce_or_sync(0xffffffffu, unsigned(flags)));
    if ((threadIdx.x & 31) == 0) {
        if (double(__uint_as_float(m)) > double(a.skin_half2) || !(__uint_as_float(m) == __uint_as_float(m)))
            a.S->rebuild = 1;
        if (fl) atomicOr(&a.S->error, fl);
    }
}

/* After a lite Langevin step (count_step = 1) or a minimisation step (0):
 * flip the position buffers, advance the step counter and apply the
 * every-k-steps rebuild rule; in a graph, hand the rebuild flag to the next
 * step's conditional node (a kernel of its own for that cost 2 us a step). */
__global__ void k_advance(Scalars *S, int rebuild_every, int count_step, cudaGraphConditionalHandle cond,
                          int has_cond) {
    int rebuild = __ldcg(&S->rebuild);
    if (!halted(S)) {
        S->iters += 1;
        S->cur ^= 1;
        S->step += count_step;
        S->since_rebuild += 1;
        if (rebuild_every > 0 && S->since_rebuild >= rebuild_every) S->rebuild = rebuild = 1;
    }
    if (has_cond) cudaGraphSetConditional(cond, rebuild ? 1u : 0u);
}

/* One step of the energy minimisation (src/openrbc.cpp:88-146): forces,
 * post_torque t <- n x t (src/integrate_nh.h:146-154), the step-limited
 * steepest-descent move of :113-130 and bounce_back (:132).  Positions and
 * orientations ping-pong like the Langevin step; the step counter (the noise
 * key) does not advance. */
template<class R, int U>
__global__ void __launch_bounds__(force_threads<R>, force_blocks<R, false, U>())
    k_minimize(KArgs<R> a, double dr_opt, double dn_opt) {
    using T4 = typename Vec<R>::T4;
    __shared__ ShiftTab<R> shm[force_threads<R> / 32];
    const int i = blockIdx.x * force_threads<R> + threadIdx.x;
    // the loads that depend on nothing, together
    const int4 sc = __ldcg(reinterpret_cast<const int4 *>(a.S));  // cur, lp, rebuild, error
    const int s = a.nsys > 1 ? a.blk_sys[i / SYS_PAD] : 0;
    const int packed = a.nnb[i];
    if (halted(sc)) return;
    const int cur = sc.x, lp = sc.y;
    const FFDev<R> &F = *a.ff;
    prefetch_warp_list(a.nbr, i, a.cap, packed);
    ShiftTab<R> &sh = shm[threadIdx.x >> 5];
    init_shift<R>(a.sys[s], sh);
    const SysDev &sd = a.sys[s];
    const T4 pi = a.pos[cur][i], ni = a.nrm[cur][i];
    const int w = wbits(pi.w);
    const int ty = w_type(w);
    float md2 = 0.f;
    int flags = 0;
    R3<R> f, t;
    R e = 0;
    slot_forces<R, false, false, U>(a, F, i, cur, lp, w, pi, ni, sd, a.ss[s], packed, sh, f, t, e, flags);
    if (ty != GHOST) {
        const R tx = ni.y * t.z - ni.z * t.y, ty_ = ni.z * t.x - ni.x * t.z, tz = ni.x * t.y - ni.y * t.x;
        const R m = F.mass[ty];
        const R dxx = f.x / m, dxy = f.y / m, dxz = f.z / m;
        const R dnx = ty_ * ni.z - tz * ni.y, dny = tz * ni.x - tx * ni.z, dnz = tx * ni.y - ty_ * ni.x;
        const R ndx = sqrt(dxx * dxx + dxy * dxy + dxz * dxz), ndn = sqrt(dnx * dnx + dny * dny + dnz * dnz);
        const R dr = R(dr_opt), dn = R(dn_opt);
        const R h = (ndx > dr || ndn > dn) ? min(dr / ndx, dn / ndn) : R(a.dt);
        const R hm = h / m;
        T4 p = pi;
        p.x += f.x * hm;
        p.y += f.y * hm;
        p.z += f.z * hm;
        const R gx = ni.x + dnx * h, gy = ni.y + dny * h, gz = ni.z + dnz * h;
        const R gi = R(1) / sqrt(gx * gx + gy * gy + gz * gz);
        T4 nn = ni;
        nn.x = gx * gi;
        nn.y = gy * gi;
        nn.z = gz * gi;
        T4 v = a.vel[lp][i];
        const T4 v0 = v;
        bounce_walls<R>(sd, a.cell[lp][i], p, v);
        if (v.x != v0.x || v.y != v0.y || v.z != v0.z) a.vel[lp][i] = v;
        a.pos[cur ^ 1][i] = p;
        a.nrm[cur ^ 1][i] = nn;
        const T4 xr = a.xref[lp][i];
        const R ddx = p.x - xr.x, ddy = p.y - xr.y, ddz = p.z - xr.z;
        md2 = float(ddx * ddx + ddy * ddy + ddz * ddz);
        if (!isfinite(p.x + p.y + p.z + nn.x + nn.y + nn.z)) flags |= ERRB_NAN;
    }
    const unsigned mm = __reduce_max_sync(0xffffffffu, __float_as_uint(md2));
    const int fl = int(__reduce_or_sync(0xffffffffu, unsigned(flags)));
    if ((threadIdx.x & 31) == 0) {
        if (double(__uint_as_float(mm)) > double(a.skin_half2) || !(__uint_as_float(mm) == __uint_as_float(mm)))
            a.S->rebuild = 1;
        if (fl) atomicOr(&a.S->error, fl);
    }
}

/* Nose-Hoover second half (post_toque_final_update, src/integrate_nh.h:237-273)
 * fused with the forces: the lite structure plus warp partials for the
 * kinetic-energy sum that k_reduce turns into the thermostat update. */
template<class R, bool E, bool K, int U>
__global__ void __launch_bounds__(force_threads<R>, force_blocks<R, K, U>()) k_nh_final(KArgs<R> a, int count_step) {
    using T4 = typename Vec<R>::T4;
    __shared__ ShiftTab<R> shm[force_threads<R> / 32];
    const int i = blockIdx.x * force_threads<R> + threadIdx.x;
    // the loads that depend on nothing, together
    const int4 sc = __ldcg(reinterpret_cast<const int4 *>(a.S));  // cur, lp, rebuild, error
    const int s = a.nsys > 1 ? a.blk_sys[i / SYS_PAD] : 0;
    const int packed = a.nnb[i];
    if (halted(sc)) return;
    const int cur = sc.x, lp = sc.y;
    const FFDev<R> &F = *a.ff;
    prefetch_warp_list(a.nbr, i, a.cap, packed);
    ShiftTab<R> &sh = shm[threadIdx.x >> 5];
    init_shift<R>(a.sys[s], sh);
    const T4 pi = a.pos[cur][i], ni = a.nrm[cur][i];
    const int w = wbits(pi.w);
    const int ty = w_type(w);
    R ke = 0, ep = 0;
    int flags = 0;
    R3<R> f, t;
    slot_forces<R, E, K, U>(a, F, i, cur, lp, w, pi, ni, a.sys[s], a.ss[s], packed, sh, f, t, ep, flags);
    if (ty != GHOST) {
        const R dt = R(a.dt);
        const R zeta = R(__ldcg(&a.ss[s].zeta));
        const R im = F.inv_mass[ty];
        T4 v = a.vel[lp][i], o = a.omg[lp][i];
        if (a.zero_bulk && count_step && ty == 0) {  // between the forces and the final half (src/openrbc.cpp:228)
            v.x -= R(__ldcg(&a.ss[s].vcom[0]));
            v.y -= R(__ldcg(&a.ss[s].vcom[1]));
            v.z -= R(__ldcg(&a.ss[s].vcom[2]));
        }
        T4 tq = v;
        tq.x = ni.y * t.z - ni.z * t.y;  // post_torque: t <- n x t
        tq.y = ni.z * t.x - ni.x * t.z;
        tq.z = ni.x * t.y - ni.y * t.x;
        v.x += R(0.5) * dt * (f.x * im - zeta * v.x);
        v.y += R(0.5) * dt * (f.y * im - zeta * v.y);
        v.z += R(0.5) * dt * (f.z * im - zeta * v.z);
        o.x += R(0.5) * dt * tq.x;
        o.y += R(0.5) * dt * tq.y;
        o.z += R(0.5) * dt * tq.z;
        T4 fo = v;
        fo.x = f.x;
        fo.y = f.y;
        fo.z = f.z;
        a.vel[lp][i] = v;
        a.omg[lp][i] = o;
        a.frc[lp][i] = fo;
        a.trq[lp][i] = tq;
        if (!isfinite(v.x + v.y + v.z)) flags |= ERRB_NAN;
        ke = F.mass[ty] * (v.x * v.x + v.y * v.y + v.z * v.z);
    }
    warp_partials<R>(a, i, ke, ep, 0.f, flags);
}

template<class R> __global__ void __launch_bounds__(256) k_nh_initial(KArgs<R> a) {
    if (halted(a.S)) return;
    using T4 = typename Vec<R>::T4;
    const int cur = __ldcg(&a.S->cur), lp = __ldcg(&a.S->lp);
    const int i = blockIdx.x * 256 + threadIdx.x;
    const int s = a.blk_sys[i / SYS_PAD];
    const SysDev &sd = a.sys[s];
    T4 p = a.pos[cur][i];
    const int w = wbits(p.w);
    const int ty = w_type(w);
    R ke = 0, vsx = 0, vsy = 0, vsz = 0;
    float md2 = 0.f;
    int flags = 0;
    if (ty != GHOST) {
        const R dt = R(a.dt);
        const R gamma = R(1) / (R(1) + R(0.5) * dt * R(__ldcg(&a.ss[s].zeta)));
        const R hm = R(0.5) * a.ff->inv_mass[ty];
        T4 v = a.vel[lp][i], o = a.omg[lp][i];
        const T4 f = a.frc[lp][i], t = a.trq[lp][i];
        v.x = (v.x + hm * dt * f.x) * gamma;
        v.y = (v.y + hm * dt * f.y) * gamma;
        v.z = (v.z + hm * dt * f.z) * gamma;
        p.x += v.x * dt;
        p.y += v.y * dt;
        p.z += v.z * dt;
        // bounce back at the walls (src/integrate_nh.h:199-208), in the cell frame
        bounce_walls<R>(sd, a.cell[lp][i], p, v);
        ke = a.ff->mass[ty] * (v.x * v.x + v.y * v.y + v.z * v.z);
        if (ty == 0) {
            vsx = v.x;
            vsy = v.y;
            vsz = v.z;
        }
        o.x += R(0.5) * dt * t.x;
        o.y += R(0.5) * dt * t.y;
        o.z += R(0.5) * dt * t.z;
        T4 n = a.nrm[cur][i];
        const R gx = n.x + (o.y * n.z - o.z * n.y) * dt;
        const R gy = n.y + (o.z * n.x - o.x * n.z) * dt;
        const R gz = n.z + (o.x * n.y - o.y * n.x) * dt;
        const R gi = rnorm3(gx, gy, gz);
        n.x = gx * gi;
        n.y = gy * gi;
        n.z = gz * gi;
        a.pos[cur][i] = p;
        a.nrm[cur][i] = n;
        a.vel[lp][i] = v;
        a.omg[lp][i] = o;
        const T4 xr = a.xref[lp][i];
        const R ddx = p.x - xr.x, ddy = p.y - xr.y, ddz = p.z - xr.z;
        md2 = float(ddx * ddx + ddy * ddy + ddz * ddz);
        if (!isfinite(p.x + p.y + p.z)) flags |= ERRB_NAN;
    }
    warp_partials<R>(a, i, ke, R(0), md2, flags, vsx, vsy, vsz);
}

/* Velocity sums of each system after the velocities were replaced (upload,
 * set_state, assign_temperature): sum m v^2 and the mean lipid velocity; the
 * step kernels keep both current afterwards. */
template<class R> __global__ void __launch_bounds__(256) k_vcom(KArgs<R> a) {
    using T4 = typename Vec<R>::T4;
    const int cur = __ldcg(&a.S->cur), lp = __ldcg(&a.S->lp);
    const int i = blockIdx.x * 256 + threadIdx.x;
    R ke = 0, vsx = 0, vsy = 0, vsz = 0;
    const int ty = w_type(wbits(a.pos[cur][i].w));
    if (ty != GHOST) {
        const T4 v = a.vel[lp][i];
        ke = a.ff->mass[ty] * (v.x * v.x + v.y * v.y + v.z * v.z);
        if (ty == 0) {
            vsx = v.x;
            vsy = v.y;
            vsz = v.z;
        }
    }
    warp_partials<R>(a, i, ke, R(0), 0.f, 0, vsx, vsy, vsz);
}

/* assign_temperature (src/assign_temperature.h:26-44, called at
 * src/openrbc.cpp:160): v = sqrt(2 kT / m) g, g three unit Gaussians from
 * Box-Muller on one Philox4x32-10 block keyed by the seed with counter
 * (tag, 0x6B8B4567, 0x327B23C6, system), u = (word + 1/2) / 2^32.  The factor
 * 2 of the reference is kept.  Computed in FP64, stored in R. */
template<class R> __global__ void __launch_bounds__(256) k_assign_temperature(KArgs<R> a, double kT, uint64_t seed) {
    using T4 = typename Vec<R>::T4;
    const int cur = __ldcg(&a.S->cur), lp = __ldcg(&a.S->lp);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.npad) return;
    const int ty = w_type(wbits(a.pos[cur][i].w));
    if (ty == GHOST) return;
    const int s = a.blk_sys[i / SYS_PAD];
    uint32_t o[4];
    philox4(uint32_t(a.tag[lp][i]), 0x6B8B4567u, 0x327B23C6u, uint32_t(s), uint32_t(seed), uint32_t(seed >> 32), o);
    double u[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) u[k] = (double(o[k]) + 0.5) * (1.0 / 4294967296.0);
    const double r0 = sqrt(-2.0 * log(u[0])), r1 = sqrt(-2.0 * log(u[2]));
    const double twopi = 6.283185307179586;
    const double sc = sqrt(2.0 / double(a.ff->mass[ty]) * kT);
    T4 v = a.vel[lp][i];
    v.x = R(sc * r0 * cos(twopi * u[1]));
    v.y = R(sc * r0 * sin(twopi * u[1]));
    v.z = R(sc * r1 * cos(twopi * u[3]));
    a.vel[lp][i] = v;
}

template<class R, bool K, int U>
__global__ void __launch_bounds__(force_threads<R>, force_blocks<R, K, U>()) k_forces(KArgs<R> a) {
    using T4 = typename Vec<R>::T4;
    __shared__ ShiftTab<R> shm[force_threads<R> / 32];
    const int i = blockIdx.x * force_threads<R> + threadIdx.x;
    // the loads that depend on nothing, together
    const int4 sc = __ldcg(reinterpret_cast<const int4 *>(a.S));  // cur, lp, rebuild, error
    const int s = a.nsys > 1 ? a.blk_sys[i / SYS_PAD] : 0;
    const int packed = a.nnb[i];
    if (halted(sc)) return;
    const int cur = sc.x, lp = sc.y;
    const FFDev<R> &F = *a.ff;
    prefetch_warp_list(a.nbr, i, a.cap, packed);
    ShiftTab<R> &sh = shm[threadIdx.x >> 5];
    init_shift<R>(a.sys[s], sh);
    const T4 pi = a.pos[cur][i], ni = a.nrm[cur][i];
    const int w = wbits(pi.w);
    int flags = 0;
    R3<R> f, t;
    R e = 0;
    slot_forces<R, true, K, U>(a, F, i, cur, lp, w, pi, ni, a.sys[s], a.ss[s], packed, sh, f, t, e, flags);
    if (w_type(w) != GHOST) {
        T4 q = pi;
        q.x = f.x;
        q.y = f.y;
        q.z = f.z;
        a.frc[lp][i] = q;
        q.x = t.x;
        q.y = t.y;
        q.z = t.z;
        a.trq[lp][i] = q;
        a.epart[i] = double(e);
    } else {
        e = 0;
    }
    warp_partials<R>(a, i, R(0), e, 0.f, flags);
}

/* Shell entries of the general pairs (those the build puts there whatever
 * their distance) that were inside their range when the list was built: with
 * the inner entries, the partners in range (profile). */
template<class R> __global__ void __launch_bounds__(256) k_count_general(KArgs<R> a, unsigned long long *out) {
    using T4 = typename Vec<R>::T4;
    const int lp = __ldcg(&a.S->lp);
    const int i = blockIdx.x * 256 + threadIdx.x;
    const SysDev &sd = a.sys[a.blk_sys[i / SYS_PAD]];
    const T4 p = a.xref[lp][i];
    const int ty = w_type(wbits(p.w));
    const int nout = ty != GHOST ? a.nnb[i] >> 16 : 0;
    unsigned c = 0;
    for (int k = 0; k < nout; ++k) {
        const uint32_t ent = a.nbr[nbr_index(i, a.cap - 1 - k, a.cap)];
        const T4 q = a.xref[lp][ent & NB_MASK];
        const int tj = w_type(wbits(q.w)), s = int(ent >> NB_SHIFT);
        const PairP<R> &P = a.ff->pair[ty * NT + tj];
        if (tj == 0 && P.kind == PAIR_ANISO) continue;
        const R dx = p.x - q.x - R(s % 3 - 1) * lc_of<R>(sd, 0), dy = p.y - q.y - R((s / 3) % 3 - 1) * lc_of<R>(sd, 1),
                dz = p.z - q.z - R(s / 9 - 1) * lc_of<R>(sd, 2);
        c += dx * dx + dy * dy + dz * dz < P.anysq ? 1u : 0u;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, (unsigned long long)c);
}

/* FP64 membrane area and enclosed volume of each system's face mesh, and
 * the constraint coefficients for the next force evaluation.  Each block sums
 * MESH_CHUNK faces of one system; the last block adds the block sums of each
 * system in block order (deterministic). */
template<class R> __global__ void __launch_bounds__(256) k_mesh(KArgs<R> a) {
    using T4 = typename Vec<R>::T4;
    const int b = blockIdx.x;
    const int s = a.mesh_blk_sys[b];
    const SysDev &sd = a.sys[s];
    __shared__ double sa[8], sv[8];
    __shared__ bool last;
    const int cur = __ldcg(&a.S->cur), lp = __ldcg(&a.S->lp);
    double ar = 0, vol = 0;
    const int f0 = sd.face_begin + (b - sd.mblk_begin) * MESH_CHUNK;
    const int f1 = min(sd.face_end, f0 + MESH_CHUNK);
    if (f1 > f0) {
        const int ref = a.faces[sd.face_begin].x;
        const T4 pr = a.pos[cur][ref];
        const int cr = a.cell[lp][ref];
        for (int f = f0 + int(threadIdx.x); f < f1; f += blockDim.x) {
            const int4 q = a.faces[f];
            double P[3][3];
            const int idx[3] = {q.x, q.y, q.z};
            for (int k = 0; k < 3; ++k) {
                const T4 pk = a.pos[cur][idx[k]];
                rel_pos<double>(sd, a.cell[lp][idx[k]], cr, pk, pr, P[k][0], P[k][1], P[k][2]);
            }
            const double e1[3] = {P[1][0] - P[0][0], P[1][1] - P[0][1], P[1][2] - P[0][2]};
            const double e2[3] = {P[2][0] - P[0][0], P[2][1] - P[0][1], P[2][2] - P[0][2]};
            const double nx = e1[1] * e2[2] - e1[2] * e2[1], ny = e1[2] * e2[0] - e1[0] * e2[2],
                         nz = e1[0] * e2[1] - e1[1] * e2[0];
            ar += sqrt(nx * nx + ny * ny + nz * nz);  // twice the area
            const double bx = P[1][1] * P[2][2] - P[1][2] * P[2][1], by = P[1][2] * P[2][0] - P[1][0] * P[2][2],
                         bz = P[1][0] * P[2][1] - P[1][1] * P[2][0];
            vol += P[0][0] * bx + P[0][1] * by + P[0][2] * bz;  // six times the volume
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ar += __shfl_xor_sync(0xffffffffu, ar, o);
        vol += __shfl_xor_sync(0xffffffffu, vol, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sa[threadIdx.x >> 5] = ar;
        sv[threadIdx.x >> 5] = vol;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double A = 0, V = 0;
        for (int w = 0; w < 8; ++w) {
            A += sa[w];
            V += sv[w];
        }
        a.mesh_partial[2 * b] = A;
        a.mesh_partial[2 * b + 1] = V;
        __threadfence();
        last = atomicAdd(&a.S->mesh_counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int lane = threadIdx.x & 31;
    for (int q = threadIdx.x >> 5; q < a.nsys; q += 8) {
        const SysDev &sq = a.sys[q];
        double A = 0, V = 0;
        for (int k = sq.mblk_begin + lane; k < sq.mblk_end; k += 32) {
            A += __ldcg(a.mesh_partial + 2 * k);
            V += __ldcg(a.mesh_partial + 2 * k + 1);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            A += __shfl_xor_sync(0xffffffffu, A, o);
            V += __shfl_xor_sync(0xffffffffu, V, o);
        }
        if (lane == 0) {
            A *= 0.5;  // the FP64 division once per system, not per face
            V /= 6.0;
            SysState &ss = a.ss[q];
            ss.area = A;
            ss.volume = V;
            ss.cv = (sq.kv != 0 && sq.V0 != 0) ? -sq.kv * (V - sq.V0) / sq.V0 : 0.0;
            ss.ca = (sq.ka != 0 && sq.A0 != 0) ? -sq.ka * (A - sq.A0) / sq.A0 : 0.0;
        }
    }
    if (threadIdx.x == 0) a.S->mesh_counter = 0;
}

}  // namespace

template<class R> void reduce_sums(const KArgs<R> &a, int mode, int count_step, cudaStream_t st) {
    k_reduce<R><<<a.ngroups, RED_GROUP, 0, st>>>(a, mode, count_step);
}
/* launch(U, blocks) with the batch of rows that the size asks for.  FP32: four
 * rows together while all blocks are resident at once (10 per SM, 152 SMs: up
 * to 97 thousand slots), where the chain of dependent gathers sets the time
 * and nothing else competes for the registers; beyond that two, whose 16
 * resident blocks hide more than the longer batch does.  Step kernel, batches
 * of two / four: 2,048 particles 19.1 / 17.8 us, 32,768: 20.1 / 18.5 us, 97,000: 21.9 /
 * 22.2 us, 131,946: 31.4 / 36.5 us, 1.0M: 166 / 199 us.  FP64: one row (the FP64 pipe is
 * the bound: 0.84 against 0.88 and 0.92 ms on a 250 thousand particle cell). */
template<class R, class L> void by_batch(const KArgs<R> &a, L launch) {
    const int nb = a.npad / force_threads<R>;
    if constexpr (sizeof(R) == 8)
        launch(std::integral_constant<int, 1>(), nb);
    else if (nb <= NUM_SM * force_blocks<R, false, 4>())
        launch(std::integral_constant<int, 4>(), nb);
    else
        launch(std::integral_constant<int, 2>(), nb);
}
template<class R, bool K> void step_langevin_v(const KArgs<R> &a, cudaStream_t st, bool energy) {
    by_batch<R>(a, [&](auto u, int nb) {
        constexpr int U = decltype(u)::value;
        if (energy)
            k_step_langevin<R, true, K, U><<<nb, force_threads<R>, 0, st>>>(a);
        else if (a.zero_bulk)
            k_step_langevin<R, false, K, U><<<nb, force_threads<R>, 0, st>>>(a);
        else
            k_step_langevin_lite<R, K, U><<<nb, force_threads<R>, 0, st>>>(a);
    });
    if (energy || a.zero_bulk)
        reduce_sums<R>(a, MODE_LANGEVIN, 1, st);
    else
        k_advance<<<1, 1, 0, st>>>(a.S, a.rebuild_every, 1, a.cond, a.has_cond);
}
template<class R> void launch_step_langevin(const KArgs<R> &a, cudaStream_t st, bool energy) {
    if (a.kahan)
        step_langevin_v<R, true>(a, st, energy);
    else
        step_langevin_v<R, false>(a, st, energy);
}
template<class R, bool K> void nh_final_v(const KArgs<R> &a, cudaStream_t st, bool energy, int count_step) {
    by_batch<R>(a, [&](auto u, int nb) {
        constexpr int U = decltype(u)::value;
        if (energy)
            k_nh_final<R, true, K, U><<<nb, force_threads<R>, 0, st>>>(a, count_step);
        else
            k_nh_final<R, false, K, U><<<nb, force_threads<R>, 0, st>>>(a, count_step);
    });
    reduce_sums<R>(a, MODE_NH_FINAL, count_step, st);
}
template<class R> void launch_nh_final(const KArgs<R> &a, cudaStream_t st, bool energy) {
    if (a.kahan)
        nh_final_v<R, true>(a, st, energy, 1);
    else
        nh_final_v<R, false>(a, st, energy, 1);
}
template<class R> void launch_nh_prologue(const KArgs<R> &a, cudaStream_t st) {
    if (a.kahan)
        nh_final_v<R, true>(a, st, true, 0);
    else
        nh_final_v<R, false>(a, st, true, 0);
}
template<class R> void launch_nh_initial(const KArgs<R> &a, cudaStream_t st) {
    k_nh_initial<R><<<a.npad / 256, 256, 0, st>>>(a);
    reduce_sums<R>(a, MODE_NH_INITIAL, 0, st);
}
template<class R> void launch_forces(const KArgs<R> &a, cudaStream_t st) {
    by_batch<R>(a, [&](auto u, int nb) {
        constexpr int U = decltype(u)::value;
        if (a.kahan)
            k_forces<R, true, U><<<nb, force_threads<R>, 0, st>>>(a);
        else
            k_forces<R, false, U><<<nb, force_threads<R>, 0, st>>>(a);
    });
    reduce_sums<R>(a, MODE_FORCES, 0, st);
}
template<class R> void launch_mesh(const KArgs<R> &a, cudaStream_t st) {
    if (a.nmblk > 0) k_mesh<R><<<a.nmblk, 256, 0, st>>>(a);
}
template<class R> void launch_minimize(const KArgs<R> &a, double dr_opt, double dn_opt, cudaStream_t st) {
    by_batch<R>(a, [&](auto u, int nb) {
        k_minimize<R, decltype(u)::value><<<nb, force_threads<R>, 0, st>>>(a, dr_opt, dn_opt);
    });
    k_advance<<<1, 1, 0, st>>>(a.S, a.rebuild_every, 0, a.cond, a.has_cond);
}
template<class R> void launch_count_general(const KArgs<R> &a, unsigned long long *out, cudaStream_t st) {
    k_count_general<R><<<a.npad / 256, 256, 0, st>>>(a, out);
}
template<class R> void launch_vcom(const KArgs<R> &a, cudaStream_t st) {
    k_vcom<R><<<a.npad / 256, 256, 0, st>>>(a);
    reduce_sums<R>(a, MODE_VCOM, 0, st);
}
template<class R> void launch_assign_temperature(const KArgs<R> &a, double kT, uint64_t seed, cudaStream_t st) {
    k_assign_temperature<R><<<(a.npad + 255) / 256, 256, 0, st>>>(a, kT, seed);
}

#define ORBC_INST(R)                                                                   \
    template void launch_step_langevin<R>(const KArgs<R> &, cudaStream_t, bool);      \
    template void launch_nh_final<R>(const KArgs<R> &, cudaStream_t, bool);           \
    template void launch_nh_prologue<R>(const KArgs<R> &, cudaStream_t);              \
    template void launch_nh_initial<R>(const KArgs<R> &, cudaStream_t);               \
    template void launch_forces<R>(const KArgs<R> &, cudaStream_t);                   \
    template void launch_vcom<R>(const KArgs<R> &, cudaStream_t);                     \
    template void launch_count_general<R>(const KArgs<R> &, unsigned long long *, cudaStream_t); \
    template void launch_minimize<R>(const KArgs<R> &, double, double, cudaStream_t); \
    template void launch_assign_temperature<R>(const KArgs<R> &, double, uint64_t, cudaStream_t); \
    template void launch_mesh<R>(const KArgs<R> &, cudaStream_t);
ORBC_INST(float)
ORBC_INST(double)
#undef ORBC_INST

}  // namespace orbc
