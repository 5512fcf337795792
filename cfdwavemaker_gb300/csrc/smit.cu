// Smit et al. (2017) s-coordinate second-order kinematics on the GPU
// (vertical_theory smit, the reference's experimental theory).
//
// What is computed follows oystelan/CFDwavemaker v3.1.0 src/Irregular.cpp:
//   u_smit :1622-1771, v_smit :1773-1850, w_smit :1852-1927, dp_smit :1929-2027,
//   the pair cache's H coefficients :924-930, 951-958 (Eq. 10 inverted with the
//   Sharma-Dean alpha), the Wheeler-stretched profiles :121-138.
// At a point below the surface, with eta = eta1 + eta2 there and
// sf = h (h + z) / (h + eta), every profile is the ordinary one at the
// stretched height z* = sf - h in [-h, 0]:
//   cosh(k sf)/cosh(kh) = q(k) (e^{k z*} + e^{-k(z* + 2h)}),
// so the sums have the shape of the Sharma-Dean point sums (one thread per
// point, pair tiles in shared memory, two ex2 per wavenumber) with Smit's
// terms per pair: the bound wave H (u, v, w, p), the particular-solution
// velocity and its s-derivative (u), the Bernoulli products (p), and the
// Lagrangian-to-Eulerian chain term of u from first-order sums.
// Ramps enter as r_i r_m per pair (the theory's AA), and every diagonal term
// is kept (its loops have no filter); the pairs are those of the pair cache.
#include "cfdwm.h"
#include "f32x2.cuh"

#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <type_traits>

namespace cfdwm {

#define CK(x)                                                  \
    do {                                                       \
        cudaError_t e_ = (x);                                  \
        if (e_ != cudaSuccess) {                               \
            std::fprintf(stderr, "cfdwm: CUDA error %s at %s:%d\n", \
                         cudaGetErrorString(e_), __FILE__, __LINE__); \
            return E_CUDA;                                     \
        }                                                      \
    } while (0)

namespace {

constexpr int ST = SMIT_TILE;     // components per tile side
constexpr int SMIT_V = 12, SMIT_P = 6;   // floats per pair record: velocity, pressure
constexpr float L2E = 1.4426950408889634f;

__device__ __forceinline__ void skahan(float &s, float &c, float v) {
    float y = v - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
}
__device__ __forceinline__ void s_cp16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
                 "l"(gmem) : "memory");
}

// e^{kz} (1 +- e^{-2k(z+h)}): the profiles with the normaliser left out
__device__ __forceinline__ void sfg(float k, float zk, float zetak, float &F, float &G) {
    const float e1 = ex2(k * zk), e2 = ex2(k * zetak);
    F = fmaf(e1, e2, e1);       // e1 (1 + e2), one rounding
    G = fmaf(-e1, e2, e1);      // e1 (1 - e2)
}

// Eq. 10 inverted for H with the Sharma-Dean alpha (Irregular.cpp:926-929, 954-957)
__device__ __forceinline__ double smit_h(double g, double om12, double oi, double om, double alpha, double k1dk2,
                                         double sgn) {
    return -g / om12 * (alpha / 2.0 - (oi * oi + om * om + sgn * oi * om) / (2.0 * g) + g * k1dk2 / (2.0 * oi * om));
}

__device__ __forceinline__ double k2_rounded(double ki, double km, double gam) {
    return __dadd_rn(__dadd_rn(__dmul_rn(ki, ki), __dmul_rn(km, km)), __dmul_rn(__dmul_rn(2.0 * ki, km), gam));
}

// One record per (tile pair, entry) of the upper triangle, FP64 -> FP32; tile
// pair (I, M) at M (M + 1) / 2 + I, the records of entries (i, m) and (i, m + 1)
// interleaved.  In r:
//  0 Hp q+ A_i A_m      1 Hm q- A_i A_m       (diagonal: 0.5 A^2 H q(2k))
//  2 k+                 3 k-
//  4 kx+  5 kx-  6 ky+  7 ky-                 (k_i cos th_i +- k_m cos th_m, ...)
//  8 rho (w_i + w_m)    9 rho (w_i - w_m)
// 10 -rho g^2 k_i.k_m / (w_i w_m) A_i A_m [+]  11 the same [-]   (diagonal: 0.5 A^2 ...)
// 12 g kx+ A_i A_m     13 g kx- A_i A_m      (diagonal: 0.25 A^2 g 2k cos th)
// 14 g A_i A_m [+]     15 g A_i A_m [-]      (diagonal: 0.25 A^2 g)
// velocity record: k+-, U+-, V+-, W+-, T+-, S+-; pressure record: k+-, P+-, R+-
// (the sums are above k_smit_points).
__global__ void k_build_smit(SmitIn c, float *tabv, float *tabp) {
    const long t = blockIdx.x;
    int I = (int)t, M = 0;
    while (I > M) I -= ++M;
    const double h = c.depth, g = c.g, gg = g * g, rho = c.rho;
    for (int e = threadIdx.x; e < ST * ST; e += blockDim.x) {
        const int i = I * ST + e / ST, m = M * ST + e % ST;
        double r[16];
        for (int q = 0; q < 16; q++) r[q] = 0.0;
        if (i < c.n && m < c.n && i <= m) {
            const double ki = c.k[i], oi = c.omega[i], Ai = c.A[i];
            const double thi = c.theta[i] + c.mtheta_rad, cti = cos(thi), sti = sin(thi);
            const double Rn = ki * tanh(ki * h), Rsn = sqrt(Rn);
            if (i == m) {
                const double Dnn = (6.0 * Rsn * Rsn * (ki * ki - Rn * Rn)) / (2.0 * Rsn * Rsn - ki * tanh(2.0 * ki * h));
                const double ann = (Dnn - (ki * ki - Rn * Rn)) / Rn + 2.0 * Rn;
                const double om2 = 2.0 * oi;
                const double H = -g / om2 * (ann / 2.0 - (3.0 * oi * oi) / (2.0 * g) + g * ki * ki / (2.0 * oi * oi));
                const double q2 = 1.0 / (1.0 + exp(-4.0 * ki * h));
                const double a2 = Ai * Ai;
                r[0] = 0.5 * a2 * H * q2;
                r[2] = 2.0 * ki;
                r[4] = 2.0 * ki * cti;
                r[6] = 2.0 * ki * sti;
                r[8] = rho * om2;
                r[10] = -0.5 * a2 * rho * gg * ki * ki / (oi * oi);
                r[12] = 0.25 * a2 * g * 2.0 * ki * cti;
                r[14] = 0.25 * a2 * g;
            } else {
                const double km = c.k[m], om = c.omega[m], Am = c.A[m];
                const double thm = c.theta[m] + c.mtheta_rad, ctm = cos(thm), stm = sin(thm);
                const double Rm = km * tanh(km * h), Rsm = sqrt(Rm);
                const bool keep = (oi <= c.cutoff) && (om <= c.cutoff) && (fabs(oi - om) <= c.bandwidth);
                const bool hp = keep && (ki + km) <= c.kmax, hm = keep && (ki != km);
                const double gam = __dadd_rn(__dmul_rn(cti, ctm), __dmul_rn(sti, stm));   // Irregular.cpp:869-871
                const double k1dk2 = ki * km * gam;
                const double AA = Ai * Am;
                const double sp = Rsn + Rsm, sm = Rsn - Rsm, R2p = sp * sp, R2m = sm * sm;
                r[4] = ki * cti + km * ctm;
                r[5] = ki * cti - km * ctm;
                r[6] = ki * sti + km * stm;
                r[7] = ki * sti - km * stm;
                r[8] = rho * (oi + om);
                r[9] = rho * (oi - om);
                if (hp) {
                    const double kp = sqrt(fmax(0.0, k2_rounded(ki, km, gam)));
                    const double den = R2p - kp * tanh(kp * h);
                    const double Dp = (2.0 * R2p * (ki * km * gam - Rn * Rm)) / den +
                                      (sp * (Rsn * (km * km - Rm * Rm) + Rsm * (ki * ki - Rn * Rn))) / den;
                    const double ap = (Dp - (ki * km * gam - Rn * Rm)) / sqrt(Rn * Rm) + (Rn + Rm);
                    const double H = smit_h(g, oi + om, oi, om, ap, k1dk2, 1.0);
                    r[0] = AA * H / (1.0 + exp(-2.0 * kp * h));
                    r[2] = kp;
                    r[10] = -AA * rho * gg * k1dk2 / (oi * om);
                    r[12] = AA * g * r[4];
                    r[14] = AA * g;
                }
                if (hm) {
                    const double kq = sqrt(fmax(0.0, k2_rounded(ki, km, -gam)));
                    const double den = R2m - kq * tanh(kq * h);
                    const double Dm = (2.0 * R2m * (ki * km * gam + Rn * Rm)) / den +
                                      (sm * (-Rsn * (km * km - Rm * Rm) + Rsm * (ki * ki - Rn * Rn))) / den;
                    const double am = (Dm - (ki * km * gam + Rn * Rm)) / sqrt(Rn * Rm) + (Rn + Rm);
                    const double om12 = oi - om;
                    const double H = fabs(om12) > SMALL ? smit_h(g, om12, oi, om, am, k1dk2, -1.0) : 0.0;
                    r[1] = AA * H / (1.0 + exp(-2.0 * kq * h));
                    r[3] = kq;
                    r[11] = -AA * rho * gg * k1dk2 / (oi * om);
                    r[13] = AA * g * r[5];
                    r[15] = AA * g;
                }
            }
        }
        const double v[SMIT_V] = {r[2],          r[3],          -r[0] * r[4], -r[1] * r[5], -r[0] * r[6], -r[1] * r[7],
                                  -r[0] * r[2], -r[1] * r[3], r[12],         r[13],         r[14],         r[15]};
        const double w[SMIT_P] = {r[2], r[3], -r[0] * r[8], -r[1] * r[9], r[10], r[11]};
        const long o = (t * ST * ST + (e & ~1)), lane = e & 1;
        for (int q = 0; q < SMIT_V; q++) tabv[o * SMIT_V + 2 * q + lane] = (float)v[q];
        for (int q = 0; q < SMIT_P; q++) tabp[o * SMIT_P + 2 * q + lane] = (float)w[q];
    }
}

// Per point: eta = eta1 + eta2; zero output above eta + swl; the stretched
// height z*, (1 + s) = (h + z)/(h + eta) and the chain factor -(h + z)/(h + eta)^2.
__global__ void k_smit_prep(long n, const double *z, const double *first, const float *eta2, double depth, double swl,
                            float *zs, float *sp1, float *chain, float *above) {
    long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (p >= n) return;
    const double eta = first[p] + (double)eta2[p];
    const double zz = fmax(-depth, z[p] - swl);
    const double D = depth + eta;
    above[p] = (z[p] > eta + swl) ? 1.f : 0.f;
    zs[p] = (float)(depth * (depth + zz) / D - depth);
    sp1[p] = (float)((depth + zz) / D);
    chain[p] = (float)(-(depth + zz) / (D * D));
}

// ---------------------------------------------------------------------------
// The pair sums.  With X = cos(phi_i + phi_m) F(k+), P = sin(phi_i + phi_m) G(k+)
// and Y, Q the same of the differences, and per component
//   A = k / omega Sh,  E = A + (1 + s) k / omega k h Ch,
//   u = sum U+ X + U- Y + (1 + s) sum T+ (A_i + A_m) cos+ + T- (A_i - A_m) cos-
//   v = sum V+ X + V- Y          w = sum W+ P + W- Q
//   d phi2/ds = h w + sum S+ (E_i + E_m) sin+ + S- (E_i - E_m) sin-
//   dp = sum P+ X + P- Y + R+ (Ch Ch - Sh Sh) cos+ + R- (Ch Ch + Sh Sh) cos-
// (the theory's products, coefficients multiplied out in FP64).  All
// terms are linear in the phasors of i and m, which carry the ramps.
//
// Two neighbouring m share a packed FP32 instruction; records of the two are
// interleaved, velocity and pressure apart.
// ---------------------------------------------------------------------------
struct SmitArgs {
    long n;
    int ntile, cstride;
    const float *tabv, *tabp;  // velocity and pressure records
    const float2 *ph;          // [npad][n] phasors of the point phases
    const float *rr;           // ramps, row stride rs (0 where every component has the same ramp)
    long rs;
    const float *cf;           // [NCF][cstride]
    const float *zs, *sp1, *chain, *above;
    float depth, one;
    int tp_per;                // tile pairs per blockIdx.y
    int alone;                 // the only sums of this call: the other rows are written 0
    float *part;               // [slices][parts][n] partial sums (split launches), or null
    long ldo;
    double *out;               // rows 1..4: u, v, w, dp
};

constexpr int SMIT_PARTS = 7;  // u, v, w, d phi2/ds, eta_x, d phi1/ds; dp
constexpr int SMIT_VPARTS = 6;
// Batches that take k_smit_points_few: up to 8 points, where k_smit_points' blocks
// of 128 are nearly empty, and up to 512 as long as the (pair, point) terms,
// which it reads per point, are at most 8e5.  Measured, the three batches of a
// field, this kernel against k_smit_points: 120 components, 60 points 150 and
// 161 us, 200 points 211 and 183; 60 components, 300 points 164 and 170, 512
// points 176 and 168; 24 components, 512 points 132 and 142.
inline bool smit_few(long n, int npad) {
    return n <= 8 || (n <= 512 && (double)n * (0.5 * npad * (npad + 1)) <= 8e5);
}

struct SmitSums {
    f32x2 u = 0, v = 0, w = 0, t = 0, d = 0, p = 0;
};

// The terms of (i, m), (i, m + 1): px, py, ny = -py, nx = -px duplicated; ca, sa
// the m phasors; VEL: A and E of i (duplicated) and m; else Ch and Sh.
template <bool VEL>
__device__ __forceinline__ void smit_pair(const ulonglong2 *r, f32x2 px, f32x2 py, f32x2 nx, f32x2 ny, f32x2 mc,
                                          f32x2 ms, f32x2 ai, f32x2 bi, f32x2 am, f32x2 bm, f32x2 zk, f32x2 zetak,
                                          f32x2 neg1, SmitSums &s) {
    const ulonglong2 rk = r[0], r1 = r[1], r2 = r[2];
    const f32x2 cc = p_mul(px, mc);
    const f32x2 cp = p_fma(ny, ms, cc), cm = p_fma(py, ms, cc);
    // F = e1 (1 + e2), G = e1 (1 - e2), one rounding each, e1 = e^{kz}, e2 = e^{-2k(z+h)}
    const f32x2 e1p = p_ex2(p_mul(rk.x, zk)), e2p = p_ex2(p_mul(rk.x, zetak));
    const f32x2 e1m = p_ex2(p_mul(rk.y, zk)), e2m = p_ex2(p_mul(rk.y, zetak));
    if (VEL) {
        const ulonglong2 r3 = r[3], r4 = r[4], r5 = r[5];
        const f32x2 sc = p_mul(py, mc);
        const f32x2 sp = p_fma(px, ms, sc), sm = p_fma(nx, ms, sc);
        const f32x2 X = p_mul(cp, p_fma(e1p, e2p, e1p)), Y = p_mul(cm, p_fma(e1m, e2m, e1m));
        const f32x2 P = p_mul(sp, p_fma(e1p, p_mul(e2p, neg1), e1p));
        const f32x2 Q = p_mul(sm, p_fma(e1m, p_mul(e2m, neg1), e1m));
        s.u = p_fma(r1.x, X, p_fma(r1.y, Y, s.u));
        s.v = p_fma(r2.x, X, p_fma(r2.y, Y, s.v));
        s.w = p_fma(r3.x, P, p_fma(r3.y, Q, s.w));
        s.t = p_fma(r4.x, p_mul(p_add(ai, am), cp), p_fma(r4.y, p_mul(p_fma(am, neg1, ai), cm), s.t));
        s.d = p_fma(r5.x, p_mul(p_add(bi, bm), sp), p_fma(r5.y, p_mul(p_fma(bm, neg1, bi), sm), s.d));
    } else {
        const f32x2 X = p_mul(cp, p_fma(e1p, e2p, e1p)), Y = p_mul(cm, p_fma(e1m, e2m, e1m));
        const f32x2 ch = p_mul(ai, am), sh = p_mul(bi, bm);
        s.p = p_fma(r1.x, X, p_fma(r1.y, Y, s.p));
        s.p = p_fma(r2.x, p_mul(p_fma(sh, neg1, ch), cp), p_fma(r2.y, p_mul(p_add(ch, sh), cm), s.p));
    }
}

// Component i at a point: its profile q (F, G), and for the velocity A and E.
template <bool VEL>
__device__ __forceinline__ float2 smit_comp(const SmitArgs &a, int i, float zk, float zetak, float sp1) {
    const float k = a.cf[CF_K * a.cstride + i], q = a.cf[CF_Q * a.cstride + i];
    float F, G;
    sfg(k, zk, zetak, F, G);
    if (!VEL) return make_float2(q * F, q * G);
    // k / omega from the coefficient rows: an FP64 division here, per (point,
    // component, tile pair), kept the FP64 pipe 31% busy
    const float al = a.cf[CF_KW * a.cstride + i], A = al * (q * G);
    return make_float2(A, fmaf(sp1, al * k * a.depth * (q * F), A));
}

template <bool VEL> struct SmitStage {
    static constexpr int REC = VEL ? SMIT_V : SMIT_P;            // floats of a record
    static constexpr int N4 = ST * ST * REC / 4;                 // float4 of a tile pair
    static constexpr int SMEM = 2 * N4 * 16;
    static constexpr int PARTS = VEL ? SMIT_VPARTS : 1;
};

// A thread per point, M outer and I inner: the 16 components of tile M stay in
// registers (phasors and profiles, two by two), the records of tile pair (I, M)
// stream through two shared-memory stages, a row of 16 m is unrolled.  Bound by
// the FMA pipe (38 packed operations for two velocity terms, 20 for two of the
// pressure) beside 8 exponentials.  Before, one term at a time with the m tile
// in shared memory (15 shared-memory wavefronts and 75 instructions a term,
// 41 % of the issue slots): 16411 points, 120 components, velocity 588 us and
// pressure 226; 241 and 134 now.
template <bool VEL>
__global__ void __launch_bounds__(128, 4) k_smit_points(SmitArgs a) {
    using SS = SmitStage<VEL>;
    extern __shared__ float4 smem4[];
    const int tid = threadIdx.x;
    const long p = (long)blockIdx.x * 128 + tid;
    const bool valid = p < a.n;
    const long pc = valid ? p : a.n - 1;
    const float zs = a.zs[pc], sp1 = a.sp1[pc];
    const float zk = zs * L2E, zetak = -2.f * (zs + a.depth) * L2E;
    const f32x2 one2 = p_pack(a.one, a.one), neg1 = p_hold(-1.f, -1.f, one2);
    const f32x2 zk2 = p_hold(zk, zk, one2), zetak2 = p_hold(zetak, zetak, one2);
    float su = 0, cu = 0, sv = 0, cv = 0, sw = 0, cw = 0, stt = 0, ct = 0, sd = 0, cd = 0, sq = 0, cq = 0;
    // first order: u, v, w with the stretched profiles, eta_x and d phi1 / ds of the chain term
    float fu = 0, gu = 0, fv = 0, gv = 0, fw = 0, gw = 0, ex = 0, cex = 0, ps = 0, cps = 0;
    const int ntp = a.ntile * (a.ntile + 1) / 2;
    const int lo = blockIdx.y * a.tp_per, hi = min(lo + a.tp_per, ntp);
    int M = 0, I = lo;                                           // tile pair lo = M (M + 1) / 2 + I
    while (I > M) I -= ++M;
    const float4 *tab = reinterpret_cast<const float4 *>(VEL ? a.tabv : a.tabp);
    auto issue = [&](int t) {
        if (t < hi) {
            const float4 *src = tab + (long)t * SS::N4;
            float4 *dst = smem4 + ((t - lo) & 1) * SS::N4;
#pragma unroll
            for (int e = 0; e < SS::N4; e += 128) s_cp16(dst + e + tid, src + e + tid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(lo);
    for (int t = lo; t < hi; M++, I = 0) {
        f32x2 mc[ST / 2], ms[ST / 2], ma[ST / 2], mb[ST / 2];
#pragma unroll
        for (int mm = 0; mm < ST; mm += 2) {
            const int m = M * ST + mm;
            const float2 p0 = a.ph[(long)m * a.n + pc], p1 = a.ph[(long)(m + 1) * a.n + pc];
            const float r0 = a.rr[(long)m * a.rs + pc], r1 = a.rr[(long)(m + 1) * a.rs + pc];
            const float2 c0 = smit_comp<VEL>(a, m, zk, zetak, sp1), c1 = smit_comp<VEL>(a, m + 1, zk, zetak, sp1);
            mc[mm / 2] = p_hold(r0 * p0.x, r1 * p1.x, one2);
            ms[mm / 2] = p_hold(r0 * p0.y, r1 * p1.y, one2);
            ma[mm / 2] = p_hold(c0.x, c1.x, one2);
            mb[mm / 2] = p_hold(c0.y, c1.y, one2);
        }
        for (; I <= M && t < hi; I++, t++) {
            issue(t + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
            const ulonglong2 *rec = reinterpret_cast<const ulonglong2 *>(smem4 + ((t - lo) & 1) * SS::N4);
            // off the diagonal a row is one branch-free block
            auto rows = [&](auto on_diagonal) {
                constexpr bool diag = decltype(on_diagonal)::value;
                float2 pn = a.ph[(long)(I * ST) * a.n + pc];
                float rn = a.rr[(long)(I * ST) * a.rs + pc];
                for (int ii = 0; ii < ST; ii++) {
                    const int i = I * ST + ii;
                    const float2 pi = make_float2(rn * pn.x, rn * pn.y);
                    if (ii + 1 < ST) {                               // the next row's, under this row's sums
                        pn = a.ph[(long)(i + 1) * a.n + pc];
                        rn = a.rr[(long)(i + 1) * a.rs + pc];
                    }
                    const float2 ci = smit_comp<VEL>(a, i, zk, zetak, sp1);
                    const f32x2 px = p_pack(pi.x, pi.x), py = p_pack(pi.y, pi.y), nx = p_pack(-pi.x, -pi.x),
                                ny = p_pack(-pi.y, -pi.y), ai = p_pack(ci.x, ci.x), bi = p_pack(ci.y, ci.y);
                    const ulonglong2 *row = rec + ii * (ST / 2) * (SS::REC / 2);
                    SmitSums s;
#pragma unroll
                    for (int m4 = 0; m4 < ST; m4 += 4) {
                        if (diag && m4 + 3 < ii) continue;           // below the diagonal (zero records)
#pragma unroll
                        for (int mm = m4; mm < m4 + 4; mm += 2)
                            smit_pair<VEL>(row + (mm / 2) * (SS::REC / 2), px, py, nx, ny, mc[mm / 2], ms[mm / 2], ai, bi,
                                           ma[mm / 2], mb[mm / 2], zk2, zetak2, neg1, s);
                    }
                    if (VEL) {
                        skahan(su, cu, p_hsum(s.u));
                        skahan(sv, cv, p_hsum(s.v));
                        skahan(sw, cw, p_hsum(s.w));
                        skahan(stt, ct, p_hsum(s.t));
                        skahan(sd, cd, p_hsum(s.d));
                    } else {
                        skahan(sq, cq, p_hsum(s.p));
                    }
                    if (diag) {
                        // first order of component i and the first-order sums of the
                        // chain term (Irregular.cpp:1638-1645, 1750-1760)
                        const float2 f = smit_comp<false>(a, i, zk, zetak, sp1);
                        if (VEL) {
                            const float agk = a.cf[CF_AU * a.cstride + i], cth = a.cf[CF_CT * a.cstride + i];   // A g k / w
                            skahan(fu, gu, agk * f.x * cth * pi.x);
                            skahan(fv, gv, agk * f.x * a.cf[CF_ST * a.cstride + i] * pi.x);
                            skahan(fw, gw, agk * f.y * pi.y);
                            skahan(ex, cex, -a.cf[CF_A * a.cstride + i] * a.cf[CF_K * a.cstride + i] * cth * pi.y);
                            skahan(ps, cps, agk * a.depth * f.y * pi.y);
                        } else {
                            skahan(sq, cq, a.cf[CF_AP * a.cstride + i] * f.x * pi.x);
                        }
                    }
                }
            };
            if (I == M) rows(std::true_type{});
            else rows(std::false_type{});
            __syncthreads();
        }
    }
    if (!valid) return;
    const bool up = a.above[p] != 0.f;
    if (VEL) {
        const double w2 = (double)sw - cw;
        const double v[SMIT_VPARTS] = {((double)su - cu) + (double)sp1 * ((double)stt - ct) + ((double)fu - gu),
                                       ((double)sv - cv) + ((double)fv - gv), w2 + ((double)fw - gw),
                                       (double)a.depth * w2 + ((double)sd - cd), (double)ex - cex, (double)ps - cps};
        if (a.part) {
            float *o = a.part + (long)blockIdx.y * SMIT_VPARTS * a.n + p;
            for (int q = 0; q < SMIT_VPARTS; q++) o[(long)q * a.n] = (float)v[q];
            return;
        }
        a.out[1 * a.ldo + p] = up ? 0.0 : v[0] + (double)a.chain[p] * v[4] * (v[5] + v[3]);
        a.out[2 * a.ldo + p] = up ? 0.0 : v[1];
        a.out[3 * a.ldo + p] = up ? 0.0 : v[2];
        if (a.alone) a.out[4 * a.ldo + p] = 0.0;
    } else {
        if (a.part) {
            a.part[(long)blockIdx.y * a.n + p] = sq - cq;
            return;
        }
        a.out[4 * a.ldo + p] = up ? 0.0 : (double)sq - cq;
        if (a.alone)
            for (int q = 1; q < 4; q++) a.out[q * a.ldo + p] = 0.0;
    }
}

// Few points (a scalar call, a short batch): block (point p, slice y), thread
// t takes row ii = t % 16 of tile pair 8 g + t / 16 for g = y, y + nslice, ...
// A row is the inner loop of k_smit_points for one point, velocity and
// pressure, with the m tile's phasors, profiles and ramps formed per term (no
// other point shares them); diagonal tile pairs add the first-order terms of
// component 16 I + ii.  Each thread's rows are Kahan-summed, the block's 128 sums added
// in FP32 into slice y's seven partial sums, and k_smit_finish adds the
// slices in order and forms the chain term.
__global__ void __launch_bounds__(128) k_smit_points_few(SmitArgs a, int ntp, int nslice) {
    __shared__ float s_red[4][SMIT_PARTS];
    const long p = blockIdx.x;
    const float h = a.depth;
    const float zs = a.zs[p], sp1 = a.sp1[p];
    const float zk = zs * L2E, zetak = -2.f * (zs + h) * L2E;
    const f32x2 zk2 = p_pack(zk, zk), zetak2 = p_pack(zetak, zetak), neg1 = p_pack(-1.f, -1.f);
    const int ii = threadIdx.x % ST;
    constexpr int PER = 128 / ST;
    float su = 0, cu = 0, sv = 0, cv = 0, sw = 0, cw = 0, sq = 0, cq = 0, sd = 0, cd = 0;
    float ex = 0, cex = 0, ps = 0, cps = 0;
    for (int g = blockIdx.y; g * PER < ntp; g += nslice) {
        const int tp = g * PER + threadIdx.x / ST;
        if (tp >= ntp) continue;
        int I = tp, M = 0;
        while (I > M) I -= ++M;
        const int i = I * ST + ii;
        const float2 ph = a.ph[(long)i * a.n + p];
        const float ri = a.rr[(long)i * a.rs + p];
        const float2 pi = make_float2(ri * ph.x, ri * ph.y);
        const float2 f = smit_comp<false>(a, i, zk, zetak, sp1), v = smit_comp<true>(a, i, zk, zetak, sp1);
        const f32x2 px = p_pack(pi.x, pi.x), py = p_pack(pi.y, pi.y), nx = p_pack(-pi.x, -pi.x),
                    ny = p_pack(-pi.y, -pi.y);
        const f32x2 va = p_pack(v.x, v.x), vb = p_pack(v.y, v.y), fa = p_pack(f.x, f.x), fb = p_pack(f.y, f.y);
        const long o = (long)tp * ST * ST + ii * ST;
        SmitSums s;
        for (int mm = (M == I) ? ii & ~1 : 0; mm < ST; mm += 2) {
            const int m = M * ST + mm;
            const float2 p0 = a.ph[(long)m * a.n + p], p1 = a.ph[(long)(m + 1) * a.n + p];
            const float r0 = a.rr[(long)m * a.rs + p], r1 = a.rr[(long)(m + 1) * a.rs + p];
            const f32x2 mc = p_pack(r0 * p0.x, r1 * p1.x), ms = p_pack(r0 * p0.y, r1 * p1.y);
            const float2 f0 = smit_comp<false>(a, m, zk, zetak, sp1), f1 = smit_comp<false>(a, m + 1, zk, zetak, sp1);
            const float2 v0 = smit_comp<true>(a, m, zk, zetak, sp1), v1 = smit_comp<true>(a, m + 1, zk, zetak, sp1);
            smit_pair<true>(reinterpret_cast<const ulonglong2 *>(a.tabv + (o + mm) * SMIT_V), px, py, nx, ny, mc, ms,
                            va, vb, p_pack(v0.x, v1.x), p_pack(v0.y, v1.y), zk2, zetak2, neg1, s);
            smit_pair<false>(reinterpret_cast<const ulonglong2 *>(a.tabp + (o + mm) * SMIT_P), px, py, nx, ny, mc, ms,
                             fa, fb, p_pack(f0.x, f1.x), p_pack(f0.y, f1.y), zk2, zetak2, neg1, s);
        }
        const float w2 = p_hsum(s.w);
        skahan(su, cu, fmaf(sp1, p_hsum(s.t), p_hsum(s.u)));
        skahan(sv, cv, p_hsum(s.v));
        skahan(sw, cw, w2);
        skahan(sd, cd, fmaf(h, w2, p_hsum(s.d)));
        skahan(sq, cq, p_hsum(s.p));
        if (M == I) {
            // first order of component i with the stretched profiles and the
            // first-order sums of the chain term (Irregular.cpp:1638-1645, 1750-1760)
            const float agk = a.cf[CF_AU * a.cstride + i], ct = a.cf[CF_CT * a.cstride + i];
            skahan(su, cu, agk * f.x * ct * pi.x);
            skahan(sv, cv, agk * f.x * a.cf[CF_ST * a.cstride + i] * pi.x);
            skahan(sw, cw, agk * f.y * pi.y);
            skahan(sq, cq, a.cf[CF_AP * a.cstride + i] * f.x * pi.x);
            skahan(ex, cex, -a.cf[CF_A * a.cstride + i] * a.cf[CF_K * a.cstride + i] * ct * pi.y);
            skahan(ps, cps, agk * h * f.y * pi.y);
        }
    }
    float v[SMIT_PARTS] = {su - cu, sv - cv, sw - cw, sd - cd, ex - cex, ps - cps, sq - cq};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int f = 0; f < SMIT_PARTS; f++) {
        for (int o = 16; o > 0; o >>= 1) v[f] += __shfl_down_sync(0xffffffffu, v[f], o);
        if (lane == 0) s_red[warp][f] = v[f];
    }
    __syncthreads();
    if (threadIdx.x < SMIT_PARTS) {
        const int f = threadIdx.x;
        a.part[((long)blockIdx.y * SMIT_PARTS + f) * a.n + p] = ((s_red[0][f] + s_red[1][f]) + s_red[2][f]) + s_red[3][f];
    }
}

// The slices of a split launch summed in order, then the chain term: parts
// [slice][np][n], velocity rows from part 0 on (vel), dp's in the last (pr);
// rows not computed are 0 where clear is set.
__global__ void k_smit_finish(long n, int nslice, int np, bool vel, bool pr, bool clear, const float *part,
                              const float *chain, const float *above, long ldo, double *out) {
    long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (p >= n) return;
    double v[SMIT_PARTS] = {};
    for (int q = 0; q < np; q++) {
        float s = 0.f, c = 0.f;
        for (int k = 0; k < nslice; k++) skahan(s, c, part[((long)k * np + q) * n + p]);
        v[q] = (double)s - c;
    }
    const bool up = above[p] != 0.f;
    if (vel) {
        out[1 * ldo + p] = up ? 0.0 : v[0] + (double)chain[p] * v[4] * (v[5] + v[3]);
        out[2 * ldo + p] = up ? 0.0 : v[1];
        out[3 * ldo + p] = up ? 0.0 : v[2];
    }
    if (pr) out[4 * ldo + p] = up ? 0.0 : v[np - 1];
    if (clear && !pr) out[4 * ldo + p] = 0.0;
    if (clear && !vel)
        for (int q = 1; q < 4; q++) out[q * ldo + p] = 0.0;
}

// One group of rows of a batch that is not short.
template <bool VEL>
int smit_points(SmitArgs a, float *split_buf, long split_cap, cudaStream_t stream) {
    using SS = SmitStage<VEL>;
    static const cudaError_t attr =
        cudaFuncSetAttribute(k_smit_points<VEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, SS::SMEM);
    CK(attr);
    static const long slots = [] {
        int dev = 0, nsm = 0, per = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_smit_points<VEL>, 128, SS::SMEM) != cudaSuccess ||
            per < 1) {
            cudaGetLastError();
            return 4L * 152;
        }
        return (long)per * nsm;
    }();
    // the walk of the tile pairs split over blockIdx.y where the points alone do
    // not fill whole waves of the resident blocks (slices summed in order)
    const int ntp = a.ntile * (a.ntile + 1) / 2;
    const long nblk = (a.n + 127) / 128;
    a.tp_per = slice_plan(nblk, ntp, slots, split_buf ? std::max<long>(1, split_cap / (SS::PARTS * a.n)) : 1);
    const int nslice = (ntp + a.tp_per - 1) / a.tp_per;
    a.part = nslice > 1 ? split_buf : nullptr;
    prof_begin(PK_POINT_PAIRS, stream);
    k_smit_points<VEL><<<dim3((unsigned)nblk, (unsigned)nslice), 128, SS::SMEM, stream>>>(a);
    note_launch();
    prof_end(PK_POINT_PAIRS, stream);
    CK(cudaGetLastError());
    if (nslice > 1) {
        k_smit_finish<<<(unsigned)((a.n + 255) / 256), 256, 0, stream>>>(a.n, nslice, SS::PARTS, VEL, !VEL, a.alone != 0,
                                                                         split_buf, a.chain, a.above, a.ldo, a.out);
        note_launch();
        CK(cudaGetLastError());
    }
    return OK;
}

}  // namespace

int smit_build(const SmitIn &c, DevSea &sea, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (sea.d_tab_smit) cudaFree(sea.d_tab_smit);
    sea.d_tab_smit = nullptr;
    sea.npad_s = ((c.n + ST - 1) / ST) * ST;
    if (sea.npad_s == 0) sea.npad_s = ST;
    sea.ntile_s = sea.npad_s / ST;
    if (sea.npad_s > sea.npad_g) return E_BAD_ARGUMENT;
    const long ntiles = (long)sea.ntile_s * (sea.ntile_s + 1) / 2;
    CK(cudaMalloc(&sea.d_tab_smit, sizeof(float) * (size_t)ntiles * ST * ST * (SMIT_V + SMIT_P)));
    k_build_smit<<<(unsigned)ntiles, 256, 0, stream>>>(c, sea.d_tab_smit, sea.d_tab_smit + ntiles * ST * ST * SMIT_V);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

int smit_eval(const DevSea &sea, long n, const double *z, const void *ph, const float *rr, const double *first,
              const float *eta2, float *scratch, float *split_buf, long split_cap, long ldo, double *out,
              int mask, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!sea.d_tab_smit) return E_NOT_INITIALIZED;
    if (n <= 0) return OK;
    float *zs = scratch, *sp1 = scratch + n, *chain = scratch + 2 * n, *above = scratch + 3 * n;
    k_smit_prep<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(n, z, first, eta2, sea.depth, sea.swl, zs, sp1, chain,
                                                                 above);
    note_launch();
    CK(cudaGetLastError());
    const int ntp = sea.ntile_s * (sea.ntile_s + 1) / 2;
    SmitArgs a = {};
    a.n = n; a.ntile = sea.ntile_s; a.cstride = sea.npad_g;
    a.tabv = sea.d_tab_smit; a.tabp = sea.d_tab_smit + (long)ntp * ST * ST * SMIT_V;
    a.ph = static_cast<const float2 *>(ph); a.rr = rr; a.rs = sea.trivial_ramp ? 0 : n; a.cf = sea.d_cf;
    a.zs = zs; a.sp1 = sp1; a.chain = chain; a.above = above;
    a.depth = (float)sea.depth; a.one = 1.f; a.ldo = ldo; a.out = out;
    if (smit_few(n, sea.npad_s) && split_buf) {
        // a block per (point, slice), the rows of 8 tile pairs over its threads
        constexpr int PER = 128 / ST;
        const int npass = (ntp + PER - 1) / PER;
        int nslice = (int)std::min<long>(npass, std::max<long>(1, split_cap / ((long)SMIT_PARTS * n)));
        nslice = std::min(nslice, 65535);
        a.part = split_buf;
        prof_begin(PK_POINT_PAIRS, stream);
        k_smit_points_few<<<dim3((unsigned)n, (unsigned)nslice), 128, 0, stream>>>(a, ntp, nslice);
        note_launch();
        prof_end(PK_POINT_PAIRS, stream);
        CK(cudaGetLastError());
        k_smit_finish<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(n, nslice, SMIT_PARTS, true, true, false, split_buf,
                                                                       chain, above, ldo, out);
        note_launch();
        CK(cudaGetLastError());
        return OK;
    }
    // the velocity sums only where u, v or w is asked for, the pressure sum
    // only where dp is
    const bool vel = (mask & 14) != 0, pr = (mask & 16) != 0 || !vel;
    a.alone = !(vel && pr);
    int rc = vel ? smit_points<true>(a, split_buf, split_cap, stream) : OK;
    if (!rc && pr) rc = smit_points<false>(a, split_buf, split_cap, stream);
    if (rc) return rc;
    return OK;
}

}  // namespace cfdwm
