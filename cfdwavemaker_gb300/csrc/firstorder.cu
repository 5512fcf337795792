// First-order sums over the columns of a regular grid at one time: the
// surface sums and the level sums of the s-grid's tensor-core path, and the
// first-order channels of the learned update.
//
// The columns stand on a regular grid, so a component's phasor there factors,
//   exp i(kx x_i + ky y_j - omega t + phase0) = exp i(kx x_i) exp i(ky y_j - omega t + phase0),
// into two tables of (nx + ny) x components.  Their phases reach 1e3-1e4 rad
// and are formed from float pairs (ffmath.cuh); a column's phasor is one
// complex product of two entries good to 1e-7 (about 1.5e-7 together, where
// the SFU's sine of the whole reduced phase, used before, was within 4e-7).
// Per (column, component) that is 4 FP32 operations for about 50.
//
// Sums (FP32):
//   surface   eta1 and the Taylor gradients phi1_dxdz, phi1_dydz, phi1_dzdz,
//             dp1_dz (Irregular.cpp:178-198, 1107-1192), every term compensated (Kahan)
//   levels    u1, v1, w1 (and dp1) at the level heights (Irregular.cpp:394-447,
//             1107-1120): the components of a wave-number group, at most KGRP = 64, in
//             FP32, then 32 groups, then Kahan
//   features  u, v, w and the pressure head at the levels placed under eta1,
//             each in phase and in quadrature
#include "cfdwm.h"
#include "convtc.h"
#include "f32x2.cuh"
#include "ffmath.cuh"
#include "sgrid_geom.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>

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

constexpr float LOG2E_F = 1.4426950408889634f;
constexpr int REC = 16;          // floats of a component's record:
constexpr int REC_S = 0;         //   surface coefficients A, gx, gy, gz, gp
constexpr int REC_L = 8;         //   level coefficients cu, cv, cw, dp1's, head's (all times the ramp)
constexpr int REC_K = 13;        //   k

struct TabArgs {
    GridCols c;
    const double *phase;         // [7][cstride]: kx, ky, omega, phase0, ramp parameters
    const float *cf;             // [NCF][cstride]
    const int *perm;
    int cstride, ncomp, ncp, trivial_ramp, sx, sy;
    double t, fx, fy;
    float depth;
    float2 *X, *Y, *Xt, *Yt;
    float *rec, *ramp;
};

// blockIdx.x: table component (zero past the last); threads: the x indices, then the y indices.
__global__ void __launch_bounds__(128) k_grid_tab(TabArgs a) {
    const int q = blockIdx.x, cs = a.cstride;
    const bool on = q < a.ncomp;
    const int c = on ? a.perm[q] : q;                // the sea's component
    if (threadIdx.x == 0) {
        float *r = a.rec + (long)q * REC;
        for (int k = 0; k < REC; k++) r[k] = 0.f;
        float rp = 0.f;
        if (on) {
            const int ir = a.trivial_ramp ? 0 : c;
            rp = (float)ff_freq_ramp(a.t, a.phase[4 * cs + ir], a.phase[5 * cs + ir], a.phase[6 * cs + ir]);
            const float *f = a.cf + c;
            r[REC_S] = rp * f[CF_A * cs];
            r[REC_S + 1] = rp * f[CF_GX * cs];
            r[REC_S + 2] = rp * f[CF_GY * cs];
            r[REC_S + 3] = rp * f[CF_GZ * cs];
            r[REC_S + 4] = rp * f[CF_GP * cs];
            const float qn = f[CF_Q * cs], au = rp * (f[CF_AU * cs] * qn), k = f[CF_K * cs];
            r[REC_L] = au * f[CF_CT * cs];
            r[REC_L + 1] = au * f[CF_ST * cs];
            r[REC_L + 2] = au;
            r[REC_L + 3] = rp * (f[CF_AP * cs] * qn);
            r[REC_L + 4] = rp * (f[CF_A * cs] * qn);
            r[REC_K] = k;
        }
        a.ramp[c] = rp;
    }
    float2 kx = make_float2(0.f, 0.f), ky = kx, p0 = kx;
    if (on) {
        kx = ff_from_double(a.phase[c]);
        ky = ff_from_double(a.phase[cs + c]);
        const float2 w = ff_from_double(-a.phase[2 * cs + c]), t = ff_from_double(a.t);
        p0 = ff_add(ff_mul(w.x, w.y, t.x, t.y), ff_from_double(a.phase[3 * cs + c]));
    }
    for (int e = threadIdx.x; e < a.sx + a.sy; e += 128) {
        const bool isx = e < a.sx;
        const int i = isx ? e : e - a.sx;
        const bool in = i < (isx ? a.c.nx : a.c.ny);
        float2 v = make_float2(0.f, 0.f);
        if (on && in) {
            const double d = isx ? a.c.d0 + a.c.dx * (i - a.c.off) - a.fx : a.c.d2 + a.c.dy * (i - a.c.off) - a.fy;
            const float2 p = ff_from_double(d), k = isx ? kx : ky;
            float2 ph = ff_mul(k.x, k.y, p.x, p.y);
            if (!isx) ph = ff_add(ph, p0);
            ff_sincos_poly(ff_reduce_2pi(ph), v.y, v.x);
        }
        if (isx) {
            a.X[(long)q * a.sx + i] = v;
            if (in && a.Xt) a.Xt[(long)i * a.ncp + c] = v;
        } else {
            a.Y[(long)q * a.sy + i] = v;
            if (in && a.Xt) a.Yt[(long)i * a.ncp + c] = v;
        }
    }
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.y, b.x, a.x * b.y));
}
__device__ __forceinline__ void kahan_add(float &s, float &c, float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}
// the same for two lanes
__device__ __forceinline__ void kahan_add2(f32x2 &s, f32x2 &c, f32x2 v, f32x2 neg1) {
    const f32x2 y = p_fma(c, neg1, v);
    const f32x2 t = p_add(s, y);
    c = p_fma(y, neg1, p_fma(s, neg1, t));
    s = t;
}

// the table rows of column p
__device__ __forceinline__ void col_rows(const GridTab &T, const GridCols &c, long p, int &i, int &j) {
    const int q = c.act ? c.act[p] : (int)p;
    i = q / c.ny;
    j = q - i * c.ny;
}

// TILE: block (blockIdx.x, blockIdx.y) holds SR rows of 32 columns of the whole
// grid, and a thread SR columns, whose y entries are one load; else blockIdx.x
// holds SR x 32 listed columns.  Warp w sums the components w, w + nw, ...  Loads
// of table entries bound it where terms are added plainly (one column a thread,
// 65536 columns of 1024 components 144 us, 79 with four, FMA pipe 42 %); here every
// term's rounding error is kept: 14 packed operations a component for two columns
// instead of 9, eight components' loads in flight at two blocks an SM, 76 us with
// the FMA pipe at 75 %.  In a learned update, beside the checked columns' kernels,
// 583 us with 16 plain terms a Kahan step, 597 so (four blocks of two components in
// flight 615, three of four 615, one of eight 610).  With the phase
// formed per (column, component) it was issue-bound, 256 us.  A short list gets
// 32 warps a block (64 columns: 8 warps 54 us, 23; one thread per column
// 180).
constexpr int SR = 4;
template <bool TILE, int NW>
__global__ void __launch_bounds__(32 * NW, TILE ? 2 : 1) k_first_surface(GridTab T, GridCols c, double *first) {
    __shared__ float2 part[NW][5][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int NR = TILE ? SR : 1;
    long p[NR];
    bool valid[NR];
    int i, j;
    if (TILE) {
        j = blockIdx.x * 32 + lane;
        i = blockIdx.y * SR;
#pragma unroll
        for (int r = 0; r < NR; r++) {
            valid[r] = j < c.ny && i + r < c.nx;
            p[r] = (long)(i + r) * c.ny + j;
        }
    } else {
        p[0] = blockIdx.x * 32L + lane;
        valid[0] = p[0] < c.n;
        col_rows(T, c, valid[0] ? p[0] : c.n - 1, i, j);
    }
    // sums s with their carries k, every term compensated; TILE: two rows to a
    // packed operand
    constexpr int NP = TILE ? NR / 2 : 1;
    float s[NR][5] = {}, k[NR][5] = {};
    f32x2 ps[NP][5] = {}, pk[NP][5] = {};
    const f32x2 neg1 = p_pack(-1.f, -1.f);
    for (int q0 = w; q0 < T.ncp; q0 += 128) {
#pragma unroll(128 / NW < 8 ? 128 / NW : 8)
        for (int u = 0; u < 128 / NW; u++) {
            const int q = q0 + NW * u;
            const float2 y = T.Y[(long)q * T.sy + j];
            const float2 *xp = T.X + (long)q * T.sx + i;
            const float *rec = T.rec + (long)q * REC + REC_S;
            const float4 f = *reinterpret_cast<const float4 *>(rec);
            const float cf[5] = {f.x, f.y, f.z, f.w, rec[4]};
            if (TILE) {
#pragma unroll
                for (int r = 0; r < NP; r++) {
                    const float4 x = *reinterpret_cast<const float4 *>(xp + 2 * r);
                    const float2 e0 = cmul(make_float2(x.x, x.y), y), e1 = cmul(make_float2(x.z, x.w), y);
                    const f32x2 ec = p_pack(e0.x, e1.x), es = p_pack(e0.y, e1.y);
#pragma unroll
                    for (int v = 0; v < 5; v++) {
                        const f32x2 a = p_fma(p_pack(cf[v], cf[v]), v == 3 ? es : ec, pk[r][v]);
                        const f32x2 t = p_add(ps[r][v], a);
                        pk[r][v] = p_add(p_fma(t, neg1, ps[r][v]), a);
                        ps[r][v] = t;
                    }
                }
            } else {
                const float2 e = cmul(*xp, y);
#pragma unroll
                for (int v = 0; v < 5; v++) {
                    const float a = fmaf(cf[v], v == 3 ? e.y : e.x, k[0][v]), t = s[0][v] + a;
                    k[0][v] = (s[0][v] - t) + a;
                    s[0][v] = t;
                }
            }
        }
    }
    if (TILE)
#pragma unroll
        for (int r = 0; r < NP; r++)
#pragma unroll
            for (int v = 0; v < 5; v++) {
                const float2 a = p_un(ps[r][v]), b = p_un(pk[r][v]);
                s[2 * r][v] = a.x; k[2 * r][v] = b.x;
                s[(2 * r + 1) % NR][v] = a.y; k[(2 * r + 1) % NR][v] = b.y;
            }
#pragma unroll
    for (int r = 0; r < NR; r++) {
        if (r) __syncthreads();
#pragma unroll
        for (int f = 0; f < 5; f++) part[w][f][lane] = make_float2(s[r][f], k[r][f]);
        __syncthreads();
        if (w < 5 && valid[r]) {
            float S = 0.f, K = 0.f;
            for (int u = 0; u < NW; u++) {
                const float2 v = part[u][w][lane];
                kahan_add(S, K, v.x);
                kahan_add(S, K, v.y);
            }
            first[w * c.n + p[r]] = (double)S - (double)K;
        }
    }
}

struct LevelArgs {
    GridTab T;
    GridCols c;
    int nl;
    float depth;
    const float *z0;             // LEVELS: heights [n nl]
    float *sec;                  // LEVELS: [nf][n nl]
    // FEATURES
    GridGeom g;
    const double *sig;           // stretched coordinates of the levels
    const double *first;         // surface sums [5][n]
    float inv_su, inv_sp;
    float *feat;                 // planes [8 nl][n], or null
    uint4 *xs;                   // the same split (convtc.h), or null
    float *base, *eta1;          // interior columns, or null
    int halo;
    float2 one2;                 // (1, 1)
};

enum { LV_UVW = 0, LV_UVWP = 1, LV_FEAT = 2 };
constexpr int LP = 4;            // level pairs per thread
constexpr int LGRP = 8;          // level groups per block at most
// FEW: a short list of columns; more warps and groups per pass hide the loads' latency
template <int MODE, bool FEW> struct LvCfg {
    static constexpr int LGC = FEW ? 16 : 8;         // component groups per pass
    static constexpr int THREADS = 512;              // FEW

    static constexpr int NC = MODE == LV_FEAT ? 8 : MODE == LV_UVWP ? 4 : 3;   // channels
    static constexpr int NQ = MODE == LV_FEAT ? 2 : 1;                         // float4 of a group's sums
    // groups' wave numbers and sums, twice; FEATURES: the heights above swl, else sums and carries
    static constexpr int smem(int rows, int threads) {
        return 2 * LGC * (8 + rows * NQ * 32 * 16) + (MODE == LV_FEAT ? 8 : 16 * NC) * LP * threads;
    }
};

__device__ __forceinline__ void lv_prefetch(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// A block holds `rows` sets of 32 columns (TILE: rows of the grid, which share
// their y entries; else listed columns), a warp 8 levels of one set.  The depth
// profiles
//   cosh(k(z+h))/cosh(kh) = q (E + D), sinh(k(z+h))/cosh(kh) = q (E - D),
// E = e^{kz}, D = e^{-k(z+2h)}, q in the coefficients, depend on the wave number
// only, and a directional sea has many components of one wave number.  So a
// pass takes LGC groups of one wave number each: first each warp sums the
// (coefficient, phasor) products of its groups' components into shared memory
// (a complex product and 3 to 8 multiply-adds each, loads of table entries),
// then each warp adds all the groups' sums times the profiles to its levels, two
// levels to a packed operation (12 and 4 exponentials a pair of levels).  Groups
// end at 64 components: chains of 64 terms and of 32 groups round less than the one
// chain of 128 components before them, a group of any length would not.  The
// exponents are products of k and the level's z or -(z + 2h); -kz - 2kh, of the
// rounded kz and 2kh, was the larger error near the bed.  1000 directions of one
// frequency in phase, u at the bed: 6.5e-7 of its RMS without the limit and with
// that exponent, 3.6e-7 with the limit, 1.8e-7 now (4.1e-7 with phases by the SFU and
// chains of 128).  The sums of one pass are made while the warps that are done
// with them use those of the pass before.  With the profiles per component the second half was
// bound by the FMA and SFU pipes (58 % and 30 % busy).  16 levels, 1024 components
// in 64 groups, features of 69696 columns: one level at a time with float-float
// phases 1263 us, packed 805, by groups 169; levels of 65536 columns: 675, 660
// and 121 (the kernel alone on the GPU; beside the checked columns of a learned
// update the features take 290).
template <int MODE, bool TILE, bool FEW>
__global__ void __launch_bounds__(512, 1) k_first_levels(LevelArgs a, int rows) {
    using CF = LvCfg<MODE, FEW>;
    constexpr int NC = CF::NC, NQ = CF::NQ, LGC = CF::LGC;
    extern __shared__ __align__(16) uint8_t lv_raw[];
    __shared__ int2 s_ij[8][32];                                 // not TILE: the columns' table rows
    const GridCols &c = a.c;
    f32x2 *s_k = reinterpret_cast<f32x2 *>(lv_raw);              // [2][LGC]: k, k
    float4 *s_q = reinterpret_cast<float4 *>(s_k + 2 * LGC);     // [2][LGC][rows][NQ][32]: the groups' sums
    f32x2 *keep = reinterpret_cast<f32x2 *>(s_q + 2 * LGC * rows * NQ * 32) + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nt = blockDim.x, nw = nt >> 5;
    const int ng = min((a.nl + 2 * LP - 1) / (2 * LP), LGRP), g = w % ng;
    const bool worker = w < rows * ng;                           // FEW: the other warps only sum groups
    const int row = worker ? w / ng : 0, m0 = (blockIdx.z * LGRP + g) * 2 * LP;
    long p;                                                      // this warp's columns
    int ci, cj;
    bool valid;
    if (TILE) {
        ci = blockIdx.y * rows + row;
        cj = blockIdx.x * 32 + lane;
        valid = ci < c.nx && cj < c.ny;
        p = valid ? (long)ci * c.ny + cj : 0;
    } else {
        for (int r = w; r < rows; r += nw)
            col_rows(a.T, c, min((blockIdx.x * (long)rows + r) * 32 + lane, c.n - 1), s_ij[r][lane].x, s_ij[r][lane].y);
        __syncthreads();
        p = (blockIdx.x * (long)rows + row) * 32 + lane;
        valid = p < c.n;
        if (!valid) p = c.n - 1;
        ci = s_ij[row][lane].x;
        cj = s_ij[row][lane].y;
    }
    const f32x2 one = p_pack(a.one2.x, a.one2.y), one2 = p_mul(one, one), neg1 = p_hold(-1.f, -1.f, one);
    f32x2 zk[LP], yk[LP];                                        // z and -(z + 2h), times log2(e)
#pragma unroll
    for (int l = 0; l < LP; l++) {
        float z[2], za[2] = {0.f, 0.f};
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = min(m0 + 2 * l + h, a.nl - 1);
            if (MODE == LV_FEAT) {
                const double zd = d_s2z(a.g, a.sig[m], a.first[p] + a.g.swl);
                z[h] = (float)fmin(0.0, zd);
                za[h] = (float)fmax(0.0, zd - a.g.swl);
            } else {
                z[h] = a.z0[p * a.nl + m];
            }
        }
        zk[l] = p_hold(z[0] * LOG2E_F, z[1] * LOG2E_F, one2);
        yk[l] = p_hold(-(z[0] + 2.f * a.depth) * LOG2E_F, -(z[1] + 2.f * a.depth) * LOG2E_F, one2);
        if (MODE == LV_FEAT) keep[l * nt] = p_pack(za[0], za[1]);
    }
    f32x2 acc[NC][LP];
#pragma unroll
    for (int f = 0; f < NC; f++)
#pragma unroll
        for (int l = 0; l < LP; l++) {
            acc[f][l] = 0;
            if (MODE != LV_FEAT) keep[(f * LP + l) * nt] = keep[((NC + f) * LP + l) * nt] = 0;
        }

    // the groups [g0, g0 + LGC) into buffer buf, two rows at a time
    auto sums = [&](int g0, int buf) {
        const int ngc = min(LGC, a.T.ngrp - g0);
        for (int gi = w; gi < ngc; gi += nw) {
            const int qb = a.T.grp[g0 + gi], qe = a.T.grp[g0 + gi + 1];
            for (int r = 0; r < rows; r += 2) {
                int i[2], j[2];
                if (TILE) {
                    i[0] = blockIdx.y * rows + r;
                    i[1] = i[0] + 1;
                    j[0] = j[1] = blockIdx.x * 32 + lane;
                } else {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        i[h] = s_ij[r + h][lane].x;
                        j[h] = s_ij[r + h][lane].y;
                    }
                }
                float4 sc[2], ss[2];
#pragma unroll
                for (int h = 0; h < 2; h++) sc[h] = ss[h] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll(MODE == LV_FEAT ? 4 : 8)
                for (int q = qb; q < qe; q++) {
                    const float2 *X = a.T.X + (long)q * a.T.sx, *Y = a.T.Y + (long)q * a.T.sy;
                    float2 x[2], y[2];
                    if (TILE) {
                        const float4 xx = *reinterpret_cast<const float4 *>(X + i[0]);
                        x[0] = make_float2(xx.x, xx.y);
                        x[1] = make_float2(xx.z, xx.w);
                        y[0] = y[1] = Y[j[0]];
                    } else {
#pragma unroll
                        for (int h = 0; h < 2; h++) { x[h] = X[i[h]]; y[h] = Y[j[h]]; }
                    }
                    const float *rc = a.T.rec + (long)q * REC + REC_L;
                    const float4 f = *reinterpret_cast<const float4 *>(rc);
                    const float hd = MODE == LV_FEAT ? rc[4] : f.w;
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float2 e = cmul(x[h], y[h]);
                        sc[h].x = fmaf(f.x, e.x, sc[h].x);
                        sc[h].y = fmaf(f.y, e.x, sc[h].y);
                        sc[h].z = fmaf(f.z, MODE == LV_FEAT ? e.x : e.y, sc[h].z);
                        if (MODE != LV_UVW) sc[h].w = fmaf(hd, e.x, sc[h].w);
                        if (MODE == LV_FEAT) {
                            ss[h].x = fmaf(f.x, e.y, ss[h].x);
                            ss[h].y = fmaf(f.y, e.y, ss[h].y);
                            ss[h].z = fmaf(f.z, e.y, ss[h].z);
                            ss[h].w = fmaf(hd, e.y, ss[h].w);
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float4 *d = s_q + (((buf * LGC + gi) * rows + r + h) * NQ) * 32 + lane;
                    d[0] = sc[h];
                    if (MODE == LV_FEAT) d[32] = ss[h];
                }
            }
            if (lane == 0) {
                const float *rc = a.T.rec + (long)qb * REC + REC_K;
                s_k[buf * LGC + gi] = p_pack(rc[0], rc[0]);
            }
        }
    };
    sums(0, 0);
    __syncthreads();
    for (int g0 = 0, buf = 0, since = 1; g0 < a.T.ngrp; g0 += LGC, buf ^= 1, since++) {
        if (g0 + LGC < a.T.ngrp) sums(g0 + LGC, buf ^ 1);
        // the entries of this warp's group of the pass after next, toward L1, many
        // lines an instruction (levels of 65536 columns 123 and 121 us; features
        // alone 169 us with and without; a learned update 592-600 and 577-586 us)
        if (TILE && w < LGC && g0 + 2 * LGC + w < a.T.ngrp) {
            const int qb = a.T.grp[g0 + 2 * LGC + w], qe = a.T.grp[g0 + 2 * LGC + w + 1];
            for (int q = qb + (lane >> 1); q < qe; q += 16) {
                lv_prefetch(a.T.Y + (long)q * a.T.sy + blockIdx.x * 32 + (lane & 1) * 16);
                if (lane & 1) lv_prefetch(a.T.X + (long)q * a.T.sx + blockIdx.y * rows);
                else lv_prefetch(a.T.rec + (long)q * REC + REC_L);
            }
        }
        const int ngc = min(LGC, a.T.ngrp - g0);
        for (int gi = 0; gi < (worker ? ngc : 0); gi++) {
            const f32x2 rk = s_k[buf * LGC + gi];
            const float4 *sq = s_q + (((buf * LGC + gi) * rows + row) * NQ) * 32 + lane;
            const float4 sc = sq[0];
            f32x2 q2[NC];
            if (MODE == LV_FEAT) {
                const float4 ss = sq[32];
                const float v[8] = {sc.x, ss.x, sc.y, ss.y, ss.z, -sc.z, sc.w, ss.w};
#pragma unroll
                for (int f = 0; f < NC; f++) q2[f] = p_hold(v[f], v[f], one2);
            } else {
                const float v[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
                for (int f = 0; f < NC; f++) q2[f] = p_hold(v[f & 3], v[f & 3], one2);
            }
            f32x2 E[LP], D[LP];
#pragma unroll
            for (int l = 0; l < LP; l++) {
                E[l] = p_ex2(p_mul(rk, zk[l]));
                D[l] = p_ex2(p_mul(rk, yk[l]));
            }
#pragma unroll
            for (int l = 0; l < LP; l++) {
                const f32x2 F = p_add(E[l], D[l]), G = p_fma(D[l], neg1, E[l]);
#pragma unroll
                for (int f = 0; f < NC; f++) {
                    const bool sinh = MODE == LV_FEAT ? f == 4 || f == 5 : f == 2;
                    acc[f][l] = p_fma(q2[f], sinh ? G : F, acc[f][l]);
                }
            }
        }
        // a Kahan step every 32 terms
        if (MODE != LV_FEAT && (since % (32 / LGC) == 0 || g0 + LGC >= a.T.ngrp))
#pragma unroll
            for (int f = 0; f < NC; f++)
#pragma unroll
                for (int l = 0; l < LP; l++) {
                    f32x2 sv = keep[(f * LP + l) * nt], cv = keep[((NC + f) * LP + l) * nt];
                    kahan_add2(sv, cv, acc[f][l], neg1);
                    keep[(f * LP + l) * nt] = sv;
                    keep[((NC + f) * LP + l) * nt] = cv;
                    acc[f][l] = 0;
                }
        __syncthreads();
    }
    if (!valid || !worker) return;
    if (MODE != LV_FEAT) {
        const long tot = c.n * a.nl;
#pragma unroll
        for (int f = 0; f < NC; f++)
#pragma unroll
            for (int l = 0; l < LP; l++) {
                const float2 v = p_un(keep[(f * LP + l) * nt]);
                const int m = m0 + 2 * l;
                float *o = a.sec + f * tot + p * a.nl + m;
                if (m < a.nl) o[0] = v.x;
                if (m + 1 < a.nl) o[1] = v.y;
            }
        return;
    }
    const int i = ci - a.halo, j = cj - a.halo;
    const bool inner = i >= 0 && i < a.g.nx && j >= 0 && j < a.g.ny;
    const long col = (long)i * a.g.ny + j, nxy = (long)a.g.nx * a.g.ny;
    float ty[3];
#pragma unroll
    for (int f = 0; f < 3; f++) ty[f] = inner && a.base ? (float)a.first[(long)(1 + f) * c.n + p] : 0.f;
#pragma unroll
    for (int l = 0; l < LP; l++) {
        const float2 za = p_un(keep[l * nt]);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = m0 + 2 * l + h;
            if (m >= a.nl) continue;
            float v[8];
#pragma unroll
            for (int f = 0; f < 8; f++) {
                const float2 d = p_un(acc[f % NC][l]);
                v[f] = h ? d.y : d.x;
            }
            if (inner && a.base)
#pragma unroll
                for (int f = 0; f < 3; f++)
                    a.base[(long)f * nxy * a.nl + col * a.nl + m] = fmaf(ty[f], h ? za.y : za.x, v[2 * f]);
#pragma unroll
            for (int f = 0; f < 8; f++) v[f] *= f < 6 ? a.inv_su : a.inv_sp;
            if (a.feat)
#pragma unroll
                for (int f = 0; f < 8; f++) a.feat[(long)(m * 8 + f) * c.n + p] = v[f];
            if (a.xs) {
                uint4 hi, lo;
                conv_split8(v, hi, lo);
                a.xs[(long)m * c.n + p] = hi;
                a.xs[(long)(a.nl + m) * c.n + p] = lo;
            }
        }
    }
    if (inner && a.eta1 && m0 == 0) a.eta1[col] = (float)a.first[p];
}

__global__ void k_sigma(GridGeom g, double *sig) {
    for (int m = threadIdx.x; m < g.nl; m += blockDim.x) sig[m] = d_sigma_level(g, m);
}

// Tiles of whole rows where at least two thirds of the lanes have a column (and
// the rows, two a block at least, fit the grid's y dimension; the columns of more
// are taken as a list, whose blocks are in x).
bool tiled(const GridCols &c) {
    return !c.act && c.n == (long)c.nx * c.ny && c.nx <= 2 * 65535 && 3 * c.ny >= 2 * ((c.ny + 31) / 32 * 32);
}

template <int MODE, bool TILE, bool FEW>
int launch_levels_t(const LevelArgs &a, cudaStream_t st) {
    using CF = LvCfg<MODE, FEW>;
    const int ng = (a.nl + 2 * LP - 1) / (2 * LP), gpb = std::min(ng, LGRP);
    const int rows = FEW ? 2 : gpb == 1 ? 8 : gpb == 2 ? 4 : 2;
    const int threads = FEW ? CF::THREADS : 32 * gpb * rows, smem = CF::smem(rows, threads);
    static const cudaError_t attr = cudaFuncSetAttribute(
        k_first_levels<MODE, TILE, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    CK(attr);
    dim3 grid(1, 1, (unsigned)((ng + LGRP - 1) / LGRP));
    if (TILE) {
        grid.x = (unsigned)((a.c.ny + 31) / 32);
        grid.y = (unsigned)((a.c.nx + rows - 1) / rows);
    } else {
        grid.x = (unsigned)((a.c.n + 32 * rows - 1) / (32 * rows));
    }
    k_first_levels<MODE, TILE, FEW><<<grid, threads, smem, st>>>(a, rows);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

// FEW where the columns make fewer blocks of 256 threads than two per SM (64
// columns of 16 levels, 1024 components: 99 us without, 52 with).
template <int MODE>
int launch_levels(const LevelArgs &a, cudaStream_t st) {
    const long warps = (a.c.n + 31) / 32 * ((a.nl + 2 * LP - 1) / (2 * LP));
    if (warps < 2 * 152 * 8) return launch_levels_t<MODE, false, true>(a, st);
    return tiled(a.c) ? launch_levels_t<MODE, true, false>(a, st) : launch_levels_t<MODE, false, false>(a, st);
}

int padded(const DevSea &sea) { return (sea.n + 127) / 128 * 128; }
int stride_x(int nx) { return (nx + 7) / 8 * 8; }
int stride_y(int ny) { return (ny + 31) / 32 * 32; }

}  // namespace

size_t grid_tab_bytes(const DevSea &sea, int nx, int ny) {
    return (size_t)padded(sea) * (sizeof(float2) * (stride_x(nx) + stride_y(ny) + nx + ny) + sizeof(float) * (REC + 1));
}

int grid_tab(const DevSea &sea, const GridCols &c, double t, void *mem, bool transposed, GridTab *T, void *stream) {
    if (c.nx < 1 || c.ny < 1 || sea.n < 1) return E_BAD_ARGUMENT;
    TabArgs a;
    a.c = c;
    a.phase = sea.d_phase; a.cf = sea.d_cf; a.cstride = sea.npad_g; a.ncomp = sea.n; a.ncp = padded(sea);
    a.trivial_ramp = sea.trivial_ramp ? 1 : 0;
    a.t = t; a.fx = sea.fx; a.fy = sea.fy; a.depth = (float)sea.depth;
    a.X = (float2 *)mem;
    a.sx = stride_x(c.nx);
    a.sy = stride_y(c.ny);
    a.Y = a.X + (size_t)a.ncp * a.sx;
    a.Xt = a.Y + (size_t)a.ncp * a.sy;
    a.Yt = a.Xt + (size_t)a.ncp * c.nx;
    a.rec = (float *)(a.Yt + (size_t)a.ncp * c.ny);
    a.ramp = a.rec + (size_t)a.ncp * REC;
    a.perm = sea.d_kperm;
    if (!transposed) a.Xt = a.Yt = nullptr;
    k_grid_tab<<<(unsigned)a.ncp, 128, 0, (cudaStream_t)stream>>>(a);
    note_launch();
    CK(cudaGetLastError());
    T->X = a.X; T->Y = a.Y; T->Xt = a.Xt; T->Yt = a.Yt;
    T->rec = a.rec;
    T->ramp = a.ramp;
    T->grp = sea.d_kgrp;
    T->ngrp = sea.ngrp;
    T->ncp = a.ncp;
    T->sx = a.sx;
    T->sy = a.sy;
    return OK;
}

int first_surface(const GridTab &T, const GridCols &c, double *first, void *stream) {
    if (c.n <= 0) return OK;
    const unsigned nb = (unsigned)((c.n + 31) / 32);
    cudaStream_t st = (cudaStream_t)stream;
    if (nb < 152)
        k_first_surface<false, 32><<<nb, 1024, 0, st>>>(T, c, first);
    else if (tiled(c))
        k_first_surface<true, 8><<<dim3((unsigned)((c.ny + 31) / 32), (unsigned)((c.nx + SR - 1) / SR)), 256, 0, st>>>(
            T, c, first);
    else
        k_first_surface<false, 8><<<nb, 256, 0, st>>>(T, c, first);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

int first_levels(const GridTab &T, const GridCols &c, int nl, int nf, double depth, const float *z0, float *sec,
                 void *stream) {
    if (c.n <= 0) return OK;
    LevelArgs a = {};
    a.T = T; a.c = c; a.nl = nl; a.depth = (float)depth; a.z0 = z0; a.sec = sec;
    a.one2 = make_float2(1.f, 1.f);
    return nf == 4 ? launch_levels<LV_UVWP>(a, (cudaStream_t)stream) : launch_levels<LV_UVW>(a, (cudaStream_t)stream);
}

int first_features(const GridTab &T, const GridCols &c, const GridGeom &g, int halo, const double *sig,
                   const double *first, float inv_su, float inv_sp, float *feat, void *xs, float *base, float *eta1,
                   void *stream) {
    if (g.nl > 32) return E_UNSUPPORTED;
    LevelArgs a = {};
    a.T = T; a.c = c; a.nl = g.nl; a.depth = (float)g.depth;
    a.g = g; a.sig = sig; a.first = first; a.inv_su = inv_su; a.inv_sp = inv_sp;
    a.feat = feat; a.xs = (uint4 *)xs; a.base = base; a.eta1 = eta1; a.halo = halo;
    a.one2 = make_float2(1.f, 1.f);
    return launch_levels<LV_FEAT>(a, (cudaStream_t)stream);
}

// Loads the kernels, which the first launch of each would do otherwise (some
// 0.1 ms each, in the middle of a ring step).
int first_order_load() {
    static const cudaError_t rc = [] {
        const void *k[] = {(const void *)k_grid_tab,
                           (const void *)k_first_surface<false, 8>,
                           (const void *)k_first_surface<false, 32>,
                           (const void *)k_first_surface<true, 8>,
                           (const void *)k_first_levels<LV_UVW, false, false>,
                           (const void *)k_first_levels<LV_UVW, false, true>,
                           (const void *)k_first_levels<LV_UVW, true, false>,
                           (const void *)k_first_levels<LV_UVWP, false, false>,
                           (const void *)k_first_levels<LV_UVWP, false, true>,
                           (const void *)k_first_levels<LV_UVWP, true, false>,
                           (const void *)k_first_levels<LV_FEAT, false, false>,
                           (const void *)k_first_levels<LV_FEAT, false, true>,
                           (const void *)k_first_levels<LV_FEAT, true, false>};
        cudaFuncAttributes at;
        for (const void *f : k) {
            const cudaError_t e = cudaFuncGetAttributes(&at, f);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }();
    CK(rc);
    return OK;
}

int grid_sigma_table(const GridGeom &g, double *sig, void *stream) {
    k_sigma<<<1, 128, 0, (cudaStream_t)stream>>>(g, sig);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

}  // namespace cfdwm
