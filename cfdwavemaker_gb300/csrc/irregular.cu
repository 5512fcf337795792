// Irregular second-order (Sharma & Dean) kinematics on the GPU.
//
// What is computed follows the reference (oystelan/CFDwavemaker v3.1.0):
//   first-order sums     Irregular.cpp:178-198, 394-447, 1107-1192
//   eta2 (pair cache)    Irregular.cpp:223-293
//   u2/v2/w2/dp2         Irregular.cpp:450-803   (point API, unfiltered pairs)
//   uvw2 (pair cache)    Irregular.cpp:975-1102  (s-grid)
//   pair cache filters   Irregular.cpp:840-967
//   order dispatch       Irregular.cpp:9-157     (Taylor layer above swl)
//
// How it is computed (GB300 design):
//  * The per-pair transfer functions (D+-, alpha+-) are evaluated ONCE, in FP64
//    on the device, and stored as FP32 coefficients in tiles of the upper
//    triangle of the N x N pair matrix (build kernels below).  Each pair
//    record already folds the amplitudes, 1/(omega_i +- omega_m), the
//    direction factors and the depth normaliser 1/(1+exp(-2 k+- h)).
//  * Phases are formed in FP64 (k.x - omega t + phase0 can reach 1e4 rad) and
//    reduced to [-pi, pi] before an FP32 sincos; the phasors of every
//    (component, point) are written once to a scratch workspace.
//  * The pair sums run on FP32 CUDA cores: each thread owns one point (or one
//    s-grid column with LV levels in registers); the coefficient tile and the
//    phasors of the streamed component tile are staged in shared memory and
//    read as warp-wide broadcasts / conflict-free rows.  The depth factors
//    cosh(k(z+h))/cosh(kh) and sinh(k(z+h))/cosh(kh) use two MUFU ex2 per
//    wavenumber, exp(kz) and exp(-2k(z+h)), both <= 1 below the surface.
//  * Accumulation is compensated: a tile row is summed in FP32, then added to
//    a Kahan (sum, carry) pair per output.
#include "cfdwm.h"
#include "f32x2.cuh"
#include "ffmath.cuh"
#include "ramp.cuh"

#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <vector>

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

constexpr int EATA_NC = 2;    // eta table: A (cc coefficient), B (ss coefficient)
constexpr int GRIDV_NC = 8;   // uvw table: Pu, Mu, Pv, Mv, Pw, Mw, kp, km
// s-grid pressure tables (grid mask, rho folded): Pp, Mp of the phase terms,
// and X, Z of the phase-free terms (products of the first-order profiles for
// a pair, the linear diagonal terms on the diagonal entry)
constexpr int GRIDP_NC = 2;
// point tables (one allocation, in this order): the velocity records Pu, Mu,
// Pv, Mv, Pw, Mw, kp, km; the pressure's phase terms Pp, Mp, kp, km; its
// phase-free products Xpp, Xzz.  A velocity call and a pressure call each read
// their own.  Two neighbouring entries of a row are interleaved (point_at), so
// that a 16-byte word is two packed FP32x2 operands.
constexpr int POINTV_NC = 8, POINTP_NC = 4, POINTK_NC = 2;
__host__ __device__ inline long point_at(long entry, int nc, int q) { return ((entry / 2) * nc + q) * 2 + (entry & 1); }
constexpr float LOG2E_F = 1.4426950408889634f;
constexpr long SPLIT_TARGET_BLOCKS = 4 * 152;   // blocks a column-pair launch aims for
// Batches that the evaluation by points (k_point_few) takes: 20 points, where
// the per-thread kernels' blocks of 128 are nearly empty, and as many more as
// 4e6 (pair, point) terms are, where its terms, read per point, cost less than
// the per-thread path's seven dependent kernels.  Measured, a wave_Kinematics
// and a pressure batch from host arrays, this kernel against the per-thread
// ones: 24 components, 1024 points 75 and 111 us; 128 components, 256 points 105
// and 122, 512 points 145 and 123; 256 components, 64 points 99 and 126, 128
// points 129 and 129; 384 components, 64 points 137 and 147; 4096 components,
// 16 points 1.9 and 2.3 ms, 64 points 7.2 and 2.2.
constexpr long FEW_MAX_POINTS = 4096;
constexpr int FEW_MAX_NPAD = 4096;   // components whose phasors, profiles and ramps fit shared memory
static bool few_points(long n, int npad) {
    return npad <= FEW_MAX_NPAD && n <= FEW_MAX_POINTS &&
           (double)n <= 20.0 + 4e6 / (0.5 * npad * (npad + 1));
}
// the phasors alone (the Smit theory's short batches): a block per point up to
// 300 points (120 components, a velocity and a pressure batch of 200 points 243
// us against 257 with the limit at 1024, of 1000 points 307 against 368)
constexpr long PH_FEW_POINTS = 300;

__device__ __forceinline__ void kahan(float &s, float &c, float v) {
    float y = v - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
}

// Irregular::freq_ramp, Irregular.cpp:200-204 (FP64, as the reference).
__device__ __forceinline__ double d_freq_ramp(double t, double rt, double ts, double du) {
    double rampdown = fmax(fmin(1. - ((t - ts - du + rt) / (rt + SMALL)), 1.), 0.);
    double rampup = fmax(fmin(((t - ts) / (rt + SMALL)), 1.), 0.);
    return rampup * rampdown;
}

__host__ __device__ inline long tile_index(int I, int M, int nt) {
    return (long)I * nt - (long)I * (I - 1) / 2 + (M - I);
}

// ---------------------------------------------------------------------------
// Setup: FP64 component data and pair tables (on device)
// ---------------------------------------------------------------------------
struct CompIn {
    int n, npad;
    const double *omega, *A, *k, *theta;   // device copies (FP64), length n
    double depth, g, rho, mtheta_rad, cutoff, bandwidth, kmax;
};

// ki^2 + km^2 + 2 ki km gam, each product rounded separately (as the
// reference's FP64 expression without contraction)
__device__ __forceinline__ double pair_k2(double ki, double km, double gam) {
    return __dadd_rn(__dadd_rn(__dmul_rn(ki, ki), __dmul_rn(km, km)), __dmul_rn(__dmul_rn(2.0 * ki, km), gam));
}

// One record per (tile, entry).  mode 0: grid mask (eta + uvw tables, and
// the pressure tables tab_gp / tab_gk), mode 1: point-API mask (the u2/v2/w2
// table tab_v and the dp2 tables tab_gp, tab_gk).
__global__ void k_build_tables(CompIn c, int TT, int nt, int mode, float *tab_eta,
                               float *tab_v, float *tab_gp, float *tab_gk) {
    long t = blockIdx.x;
    int I = 0;
    while (tile_index(I, nt - 1, nt) < t) I++;
    int M = (int)(t - tile_index(I, I, nt)) + I;
    for (int e = threadIdx.x; e < TT * TT; e += blockDim.x) {
        int ii = e / TT, mm = e % TT;
        int i = I * TT + ii, m = M * TT + mm;
        double out[12], pr[4] = {0.0, 0.0, 0.0, 0.0};   // pr: Pp, Mp, X, Z (mode 0)
        for (int q = 0; q < 12; q++) out[q] = 0.0;
        double eA = 0.0, eB = 0.0;
        const double h = c.depth, g = c.g, gg = c.g * c.g;
        if (i < c.n && m < c.n && i <= m) {
            double ki = c.k[i], oi = c.omega[i], Ai = c.A[i];
            double thi = c.theta[i] + c.mtheta_rad;
            double cti = cos(thi), sti = sin(thi);
            double Rn = ki * tanh(ki * h), Rsn = sqrt(Rn);
            double agi = Ai * g / oi;
            if (i == m) {
                bool keep = (mode == 1) || (oi <= c.cutoff);
                if (keep) {
                    double Dnn = (6.0 * Rsn * Rsn * (ki * ki - Rn * Rn)) /
                                 (2.0 * Rsn * Rsn - ki * tanh(2.0 * ki * h));
                    double AAd = 0.25 * agi * agi * (Dnn / (2.0 * oi));
                    double q2 = 1.0 / (1.0 + exp(-4.0 * ki * h));
                    out[0] = AAd * (2.0 * ki * cti) * q2;
                    out[2] = AAd * (2.0 * ki * sti) * q2;
                    out[4] = AAd * (2.0 * ki) * q2;
                    if (mode == 1) {
                        out[6] = c.rho * AAd * (2.0 * oi) * q2;
                        out[8] = 2.0 * ki;
                    } else {
                        out[6] = 2.0 * ki;
                        // uvw2 pressure, diagonal (Irregular.cpp:1034-1037): the
                        // 2-phi term and the two terms linear in the profiles
                        pr[0] = c.rho * AAd * (2.0 * oi) * q2;
                        pr[2] = -c.rho * (gg * (2.0 * ki * cti + 2.0 * ki * sti) * 2.0) / (2.0 * oi);
                        pr[3] = c.rho * (gg * (2.0 * ki) * 2.0) / (2.0 * oi);
                        if (2.0 * ki <= c.kmax) {
                            double ann = (Dnn - (ki * ki - Rn * Rn)) / Rn + 2.0 * Rn;
                            double pe = 0.25 * Ai * Ai * ann;
                            eA = pe;
                            eB = -pe;
                        }
                    }
                }
            } else {
                double km = c.k[m], om = c.omega[m], Am = c.A[m];
                double thm = c.theta[m] + c.mtheta_rad;
                double ctm = cos(thm), stm = sin(thm);
                double Rm = km * tanh(km * h), Rsm = sqrt(Rm);
                double agm = Am * g / om;
                bool keep = true, hp = true, hm = (ki != km);
                double gam;
                if (mode == 0) {
                    keep = (oi <= c.cutoff) && (om <= c.cutoff) && (fabs(oi - om) <= c.bandwidth);
                    hp = (ki + km) <= c.kmax;
                    // Irregular.cpp:870, rounded as the reference rounds it (no FMA)
                    gam = __dadd_rn(__dmul_rn(cti, ctm), __dmul_rn(sti, stm));
                } else {
                    gam = cos(thi - thm);               // Irregular.cpp:470
                }
                if (keep && (hp || hm)) {
                    // |k_i +- k_m|; for opposite (equal) directions of equal k the
                    // radicand is 0 up to rounding: clamped so that a -1e-16 does
                    // not turn the whole table into NaN
                    double kp = sqrt(fmax(0.0, pair_k2(ki, km, gam)));
                    double kq = sqrt(fmax(0.0, pair_k2(ki, km, -gam)));
                    double sp = Rsn + Rsm, sm = Rsn - Rsm;
                    double R2p = sp * sp, R2m = sm * sm;
                    double AA = 0.5 * agi * agm;
                    if (hp) {
                        double den = R2p - kp * tanh(kp * h);
                        double Dp = (2.0 * R2p * (ki * km * gam - Rn * Rm)) / den +
                                    (sp * (Rsn * (km * km - Rm * Rm) + Rsm * (ki * ki - Rn * Rn))) / den;
                        double BB = Dp / (oi + om);
                        double qp = 1.0 / (1.0 + exp(-2.0 * kp * h));
                        out[0] = AA * BB * (ki * cti + km * ctm) * qp;
                        out[2] = AA * BB * (ki * sti + km * stm) * qp;
                        out[4] = AA * BB * kp * qp;
                        if (mode == 1) {
                            out[6] = c.rho * AA * BB * (oi + om) * qp;
                            out[8] = kp;
                        } else {
                            out[6] = kp;
                            // uvw2 pressure, sum term and the phase-free
                            // products of the profiles (Irregular.cpp:1074-1077)
                            pr[0] = c.rho * AA * BB * (oi + om) * qp;
                            pr[2] = -c.rho * (gg * (ki * cti * km * ctm + ki * sti * km * stm)) / (oi * om);
                            pr[3] = c.rho * (gg * (ki * km)) / (oi * om);
                            double ap = (Dp - (ki * km * gam - Rn * Rm)) / sqrt(Rn * Rm) + (Rn + Rm);
                            double pe = 0.5 * Ai * Am * ap;
                            eA += pe;
                            eB -= pe;
                        }
                    }
                    if (hm) {
                        double den = R2m - kq * tanh(kq * h);
                        double Dm = (2.0 * R2m * (ki * km * gam + Rn * Rm)) / den +
                                    (sm * (-Rsn * (km * km - Rm * Rm) + Rsm * (ki * ki - Rn * Rn))) / den;
                        double CC = Dm / (oi - om);
                        double qm = 1.0 / (1.0 + exp(-2.0 * kq * h));
                        out[1] = AA * CC * (ki * cti - km * ctm) * qm;
                        out[3] = AA * CC * (ki * sti - km * stm) * qm;
                        out[5] = AA * CC * kq * qm;
                        if (mode == 1) {
                            out[7] = c.rho * AA * CC * (oi - om) * qm;
                            out[9] = kq;
                        } else {
                            out[7] = kq;
                            pr[1] = c.rho * AA * CC * (oi - om) * qm;   // Irregular.cpp:1093
                            double am = (Dm - (ki * km * gam + Rn * Rm)) / sqrt(Rn * Rm) + (Rn + Rm);
                            double pe = 0.5 * Ai * Am * am;
                            eA += pe;
                            eB += pe;
                        }
                    }
                    if (mode == 1) {
                        // the phase-free products of the first-order profiles
                        // in dp2 (Irregular.cpp:786-787)
                        out[10] = -c.rho * (gg * (ki * cti * km * ctm + ki * sti * km * stm)) / (oi * om);
                        out[11] = c.rho * (gg * (ki * km)) / (oi * om);
                    }
                }
            }
        }
        long base = t * (long)TT * TT + e;
        if (mode == 0) {
            tab_eta[base * EATA_NC + 0] = (float)eA;
            tab_eta[base * EATA_NC + 1] = (float)eB;
            for (int q = 0; q < GRIDV_NC; q++) tab_v[base * GRIDV_NC + q] = (float)out[q];
            tab_gp[base * GRIDP_NC + 0] = (float)pr[0];
            tab_gp[base * GRIDP_NC + 1] = (float)pr[1];
            tab_gk[base * GRIDP_NC + 0] = (float)pr[2];
            tab_gk[base * GRIDP_NC + 1] = (float)pr[3];
        } else {
            const int vq[POINTV_NC] = {0, 1, 2, 3, 4, 5, 8, 9}, pq[POINTP_NC] = {6, 7, 8, 9};
            for (int q = 0; q < POINTV_NC; q++) tab_v[point_at(base, POINTV_NC, q)] = (float)out[vq[q]];
            for (int q = 0; q < POINTP_NC; q++) tab_gp[point_at(base, POINTP_NC, q)] = (float)out[pq[q]];
            for (int q = 0; q < POINTK_NC; q++) tab_gk[point_at(base, POINTK_NC, q)] = (float)out[10 + q];
        }
    }
}

// Count of pairs kept by the reference's pair cache (Irregular.cpp:840-967).
__global__ void k_count_pairs(CompIn c, unsigned long long *cnt) {
    long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
    long tot = (long)c.n * c.n;
    unsigned long long local = 0;
    for (; idx < tot; idx += (long)gridDim.x * blockDim.x) {
        int i = (int)(idx / c.n), m = (int)(idx % c.n);
        if (m <= i) continue;
        double oi = c.omega[i], om = c.omega[m];
        if (oi > c.cutoff || om > c.cutoff || fabs(oi - om) > c.bandwidth) continue;
        bool hp = (c.k[i] + c.k[m]) <= c.kmax, hm = c.k[i] != c.k[m];
        if (hp || hm) local++;
    }
    if (local) atomicAdd(cnt, local);
}

__global__ void k_component_coefs(CompIn c, int npad, double fx, double fy, double tofmax,
                                  const double *phase, const double *rt, const double *st,
                                  const double *du, double *ph_out, float *cf, float2 *cfp) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npad) return;
    double v[NCF];
    for (int q = 0; q < NCF; q++) v[q] = 0.0;
    double kx = 0, ky = 0, om = 0, p0 = 0, r0 = 0, r1 = -SMALL, r2 = HUGE_;
    if (i < c.n) {
        double k = c.k[i], w = c.omega[i], A = c.A[i], h = c.depth, g = c.g, gg = g * g;
        double th = c.theta[i] + c.mtheta_rad, ct = cos(th), st_ = sin(th);
        kx = k * ct; ky = k * st_; om = w; p0 = w * tofmax + phase[i];
        r0 = rt[i]; r1 = st[i]; r2 = du[i];
        v[CF_A] = A;
        v[CF_AU] = A * g * k / w;
        v[CF_CT] = ct;
        v[CF_ST] = st_;
        v[CF_K] = k;
        v[CF_Q] = 1.0 / (1.0 + exp(-2.0 * k * h));
        v[CF_AP] = A * c.rho * g;
        v[CF_GX] = ct * A * w * k;
        v[CF_GY] = st_ * A * w * k;
        v[CF_GZ] = A * w * k * (cosh(k * h) / sinh(k * h));
        v[CF_GP] = A * c.rho * g * k;
        v[CF_X1] = -c.rho * (gg * (2 * k * ct + 2 * k * st_) * 2) / (2 * w);
        v[CF_Z1] = c.rho * (gg * (2 * k) * 2) / (2 * w);
        v[CF_KW] = w > 0.0 ? k / w : 0.0;
    }
    ph_out[0 * npad + i] = kx;
    ph_out[1 * npad + i] = ky;
    ph_out[2 * npad + i] = om;
    ph_out[3 * npad + i] = p0;
    ph_out[4 * npad + i] = r0;
    ph_out[5 * npad + i] = r1;
    ph_out[6 * npad + i] = r2;
    for (int q = 0; q < NCF; q++) {
        float2 f;
        ff_split(v[q], f.x, f.y);
        cf[q * npad + i] = f.x;
        cfp[q * npad + i] = f;
    }
}

// floats of a phasor record: kx, ky, -omega, phase0 as float pairs, then A, GX,
// GY, GZ, GP.  Two neighbouring components' records are interleaved, float by
// float, into packed operands (the pair is 28 floats, 7 words of 16 bytes)
constexpr int PH_REC = 14;
constexpr int PH_CHUNK = 128;    // records per shared-memory chunk
__host__ __device__ inline long rec_at(long comp, int q) { return (comp / 2) * (2 * PH_REC) + 2 * q + (comp & 1); }

// The phasor records of all components (time-independent, built once with the sea).
__global__ void k_phasor_records(int n, int npad, const double *phase, const float *cf, int cs, float *rec) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npad) return;
    float v[PH_REC];
    for (int q = 0; q < PH_REC; q++) v[q] = 0.f;
    if (i < n) {
        ff_split(phase[i], v[0], v[1]);
        ff_split(phase[cs + i], v[2], v[3]);
        ff_split(-phase[2 * cs + i], v[4], v[5]);
        ff_split(phase[3 * cs + i], v[6], v[7]);
        v[8] = cf[CF_A * cs + i];
        v[9] = cf[CF_GX * cs + i];
        v[10] = cf[CF_GY * cs + i];
        v[11] = cf[CF_GZ * cs + i];
        v[12] = cf[CF_GP * cs + i];
    }
    for (int q = 0; q < PH_REC; q++) rec[rec_at(i, q)] = v[q];
}

static int point_kin_build(DevSea &sea, cudaStream_t stream);

int sea_build(const Config &cfg, DevSea &sea, bool point_table, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    sea_free(sea);
    int n = (int)cfg.omega.size();
    sea.n = n;
    sea.depth = cfg.depth; sea.swl = cfg.swl; sea.g = cfg.gravity; sea.rho = cfg.rho;
    sea.fx = cfg.x_pos; sea.fy = cfg.y_pos; sea.order = cfg.order;
    sea.npad_g = ((n + GRID_TILE - 1) / GRID_TILE) * GRID_TILE;
    sea.npad_p = ((n + POINT_TILE - 1) / POINT_TILE) * POINT_TILE;
    if (sea.npad_g == 0) sea.npad_g = GRID_TILE;
    if (sea.npad_p == 0) sea.npad_p = POINT_TILE;
    sea.ntile_g = sea.npad_g / GRID_TILE;
    sea.ntile_p = sea.npad_p / POINT_TILE;
    sea.trivial_ramp = true;
    for (int i = 1; i < n; i++)
        if (cfg.ramptime[i] != cfg.ramptime[0] || cfg.starttime[i] != cfg.starttime[0] ||
            cfg.duration[i] != cfg.duration[0])
            sea.trivial_ramp = false;
    double kmax = 0.0;   // Irregular.cpp:833-835
    for (int i = 0; i < n; i++) kmax = std::max(kmax, cfg.k[i]);
    sea.kmax = kmax;

    // FP64 component inputs on the device
    double *d_in = nullptr;
    size_t nn = (size_t)(n > 0 ? n : 1);
    CK(cudaMalloc(&d_in, sizeof(double) * nn * 8));
    const std::vector<double> *src[8] = {&cfg.omega, &cfg.A, &cfg.k, &cfg.theta, &cfg.phase,
                                         &cfg.ramptime, &cfg.starttime, &cfg.duration};
    for (int q = 0; q < 8; q++)
        if (n) CK(cudaMemcpyAsync(d_in + q * nn, src[q]->data(), sizeof(double) * n,
                                  cudaMemcpyHostToDevice, stream));
    CompIn ci;
    ci.n = n; ci.npad = sea.npad_g;
    ci.omega = d_in; ci.A = d_in + nn; ci.k = d_in + 2 * nn; ci.theta = d_in + 3 * nn;
    ci.depth = cfg.depth; ci.g = cfg.gravity; ci.rho = cfg.rho;
    ci.mtheta_rad = cfg.mtheta * PI_IRR / 180.0;
    ci.cutoff = cfg.dw_cutoff; ci.bandwidth = cfg.dw_bandwidth; ci.kmax = kmax;

    CK(cudaMalloc(&sea.d_phase, sizeof(double) * 7 * sea.npad_g));
    CK(cudaMalloc(&sea.d_cf, sizeof(float) * NCF * sea.npad_g));
    CK(cudaMalloc(&sea.d_cfp, sizeof(float2) * NCF * sea.npad_g));
    // records for up to the next multiple of 256 components (the plain
    // precision form pads to 256), zero past the last component
    const int nrec_cap = ((sea.npad_g + 255) / 256) * 256;
    CK(cudaMalloc(&sea.d_phrec, sizeof(float) * PH_REC * nrec_cap));
    k_component_coefs<<<(sea.npad_g + 127) / 128, 128, 0, stream>>>(
        ci, sea.npad_g, cfg.x_pos, cfg.y_pos, cfg.tofmax, d_in + 4 * nn, d_in + 5 * nn,
        d_in + 6 * nn, d_in + 7 * nn, sea.d_phase, sea.d_cf, sea.d_cfp);
    note_launch();
    CK(cudaGetLastError());
    k_phasor_records<<<(nrec_cap + 127) / 128, 128, 0, stream>>>(n, nrec_cap, sea.d_phase, sea.d_cf,
                                                                 sea.npad_g, sea.d_phrec);
    note_launch();
    CK(cudaGetLastError());

    {
        std::vector<int> perm(n), grp(1, 0);
        std::vector<unsigned> key(n);
        for (int i = 0; i < n; i++) {
            const float k = (float)cfg.k[i];
            std::memcpy(&key[i], &k, sizeof(k));
            perm[i] = i;
        }
        std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) { return key[a] < key[b]; });
        // at most KGRP components to a group, whose first stage of summation is plain
        for (int i = 1; i <= n; i++)
            if (i == n || key[perm[i]] != key[perm[i - 1]] || i - grp.back() == KGRP) grp.push_back(i);
        sea.ngrp = (int)grp.size() - 1;
        CK(cudaMalloc(&sea.d_kperm, sizeof(int) * nn));
        CK(cudaMalloc(&sea.d_kgrp, sizeof(int) * grp.size()));
        if (n) CK(cudaMemcpyAsync(sea.d_kperm, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(sea.d_kgrp, grp.data(), sizeof(int) * grp.size(), cudaMemcpyHostToDevice, stream));
        CK(cudaStreamSynchronize(stream));      // the host arrays go out of scope
    }

    if (cfg.order == 2) {
        long ntiles = tile_index(sea.ntile_g - 1, sea.ntile_g - 1, sea.ntile_g) + 1;
        size_t ent = (size_t)ntiles * GRID_TILE * GRID_TILE;
        CK(cudaMalloc(&sea.d_tab_eta, sizeof(float) * ent * EATA_NC));
        CK(cudaMalloc(&sea.d_tab_grid, sizeof(float) * ent * GRIDV_NC));
        CK(cudaMalloc(&sea.d_tab_gp, sizeof(float) * ent * GRIDP_NC));
        CK(cudaMalloc(&sea.d_tab_gk, sizeof(float) * ent * GRIDP_NC));
        k_build_tables<<<(unsigned)ntiles, 256, 0, stream>>>(ci, GRID_TILE, sea.ntile_g, 0,
                                                             sea.d_tab_eta, sea.d_tab_grid, sea.d_tab_gp,
                                                             sea.d_tab_gk);
        note_launch();
        CK(cudaGetLastError());
        if (point_table) {
            long ntp = tile_index(sea.ntile_p - 1, sea.ntile_p - 1, sea.ntile_p) + 1;
            size_t entp = (size_t)ntp * POINT_TILE * POINT_TILE;
            CK(cudaMalloc(&sea.d_tab_point, sizeof(float) * entp * (POINTV_NC + POINTP_NC + POINTK_NC)));
            sea.d_tab_pp = sea.d_tab_point + entp * POINTV_NC;
            sea.d_tab_pk = sea.d_tab_pp + entp * POINTP_NC;
            k_build_tables<<<(unsigned)ntp, 256, 0, stream>>>(ci, POINT_TILE, sea.ntile_p, 1, nullptr,
                                                              sea.d_tab_point, sea.d_tab_pp, sea.d_tab_pk);
            note_launch();
            CK(cudaGetLastError());
            int rc = point_kin_build(sea, stream);
            if (rc) return rc;
        }
        if (cfg.vertical_theory == 1) {
            SmitIn si;
            si.n = n; si.omega = ci.omega; si.A = ci.A; si.k = ci.k; si.theta = ci.theta;
            si.depth = ci.depth; si.g = ci.g; si.rho = ci.rho; si.mtheta_rad = ci.mtheta_rad;
            si.cutoff = ci.cutoff; si.bandwidth = ci.bandwidth; si.kmax = ci.kmax;
            int rc = smit_build(si, sea, stream);
            if (rc) return rc;
            sea.smit = true;
        }
        unsigned long long *d_cnt = nullptr, h_cnt = 0;
        CK(cudaMalloc(&d_cnt, sizeof(unsigned long long)));
        CK(cudaMemsetAsync(d_cnt, 0, sizeof(unsigned long long), stream));
        k_count_pairs<<<256, 256, 0, stream>>>(ci, d_cnt);
        note_launch();
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(&h_cnt, d_cnt, sizeof(h_cnt), cudaMemcpyDeviceToHost, stream));
        CK(cudaStreamSynchronize(stream));
        cudaFree(d_cnt);
        sea.npairs_grid = (long)h_cnt;
    }
    CK(cudaStreamSynchronize(stream));
    cudaFree(d_in);
    return OK;
}

void sea_free(DevSea &sea) {
    if (sea.d_phase) cudaFree(sea.d_phase);
    if (sea.d_cf) cudaFree(sea.d_cf);
    if (sea.d_cfp) cudaFree(sea.d_cfp);
    sea.d_cfp = nullptr;
    if (sea.d_tab_eta) cudaFree(sea.d_tab_eta);
    if (sea.d_tab_grid) cudaFree(sea.d_tab_grid);
    if (sea.d_tab_point) cudaFree(sea.d_tab_point);
    if (sea.d_tab_gp) cudaFree(sea.d_tab_gp);
    if (sea.d_tab_gk) cudaFree(sea.d_tab_gk);
    if (sea.d_tab_smit) cudaFree(sea.d_tab_smit);
    if (sea.d_kin) cudaFree(sea.d_kin);
    sea.d_kin = nullptr;
    if (sea.d_phrec) cudaFree(sea.d_phrec);
    if (sea.d_kperm) cudaFree(sea.d_kperm);
    if (sea.d_kgrp) cudaFree(sea.d_kgrp);
    sea.d_kperm = sea.d_kgrp = nullptr;
    sea.d_tab_smit = nullptr;
    sea.d_phrec = nullptr;
    sea.smit = false;
    sea.d_phase = nullptr; sea.d_cf = nullptr; sea.d_tab_eta = nullptr;
    sea.d_tab_grid = nullptr; sea.d_tab_point = nullptr; sea.d_tab_pp = sea.d_tab_pk = nullptr; sea.d_tab_gp = nullptr; sea.d_tab_gk = nullptr;
}

int workspace_reserve(Workspace &ws, size_t bytes) {
    if (ws.bytes >= bytes) return OK;
    if (ws.base) cudaFree(ws.base);
    ws.base = nullptr;
    ws.bytes = 0;
    CK(cudaMalloc(&ws.base, bytes));
    ws.bytes = bytes;
    return OK;
}
void workspace_free(Workspace &ws) {
    if (ws.base) cudaFree(ws.base);
    ws.base = nullptr;
    ws.bytes = 0;
}

// ---------------------------------------------------------------------------
// Phasor pass: every (point or column, component).
// ---------------------------------------------------------------------------
struct PhArgs {
    long n;
    const double *x, *y, *t;
    long sx, sy, st;        // element strides of x, y, t (0 broadcasts one value)
    int ncomp, npad;
    const double *phase;    // [7][npad_g]
    const float *cf;        // [NCF][npad_g]
    int cstride;            // npad_g
    double fx, fy;
    int trivial_ramp;
    const float *rec;       // phasor records (rec_at)
    int sums;               // which first-order sums: bit q = first[q]
    float2 *ph;             // [npad][n]
    float *rr;              // [npad][n]; with a trivial ramp row 0 only
    double *first;          // [5][n]: eta1, gx, gy, gz, gp
};

__device__ __forceinline__ void ph_kahan(float &s, float &c, float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

// sin and cos of two phases hi + lo, FMA-only: one Cody-Waite reduction to
// |r| <= pi/4 by multiples of pi/2 = A + B + C (A short: n A cancels hi's
// leading bits exactly for |n| < 2^18), then the Taylor polynomials of
// ff_sincos_poly.
__device__ __forceinline__ void ph_sincos(f32x2 hi, f32x2 lo, f32x2 &s, f32x2 &c) {
    auto dup = [](float v) { return p_pack(v, v); };
    const float2 q = p_un(p_mul(hi, dup(0.636619772f)));
    const float n0 = rintf(q.x), n1 = rintf(q.y);
    const f32x2 nn = p_pack(-n0, -n1);
    f32x2 r = p_fma(nn, dup(1.5703125f), hi);
    r = p_fma(nn, dup(4.837512969970703125e-4f), r);
    r = p_fma(nn, dup(7.549789948768648e-8f), r);
    r = p_add(r, lo);
    const f32x2 r2 = p_mul(r, r);
    f32x2 ps = p_fma(r2, dup(2.7557319e-6f), dup(-1.98412698e-4f));
    ps = p_fma(r2, p_fma(r2, ps, dup(8.33333333e-3f)), dup(-0.166666667f));
    f32x2 pc = p_fma(r2, dup(-2.75573192e-7f), dup(2.48015873e-5f));
    pc = p_fma(r2, p_fma(r2, p_fma(r2, pc, dup(-1.38888889e-3f)), dup(4.16666667e-2f)), dup(-0.5f));
    const float2 sr = p_un(p_fma(p_mul(r, r2), ps, r)), cr = p_un(p_fma(r2, pc, dup(1.0f)));
    // quarter n: sine and cosine swap when n is odd; sin is negative for n = 2,
    // 3 and cos for n = 1, 2 (mod 4)
    auto pick = [](float n, float sv, float cv, float &so, float &co) {
        const unsigned k = (unsigned)(int)n;
        const unsigned us = __float_as_uint((k & 1) ? cv : sv), uc = __float_as_uint((k & 1) ? sv : cv);
        so = __uint_as_float(us ^ ((k & 2) << 30));
        co = __uint_as_float(uc ^ (((k + 1) & 2) << 30));
    };
    float s0, c0, s1, c1;
    pick(n0, sr.x, cr.x, s0, c0);
    pick(n1, sr.y, cr.y, s1, c1);
    s = p_pack(s0, s1);
    c = p_pack(c0, c1);
}

// A point's offsets and time as duplicated packed operands
struct PhPoint {
    f32x2 xh, xl, nxh, yh, yl, nyh, th, tl, nth;
    __device__ __forceinline__ PhPoint(float2 dx, float2 dy, float2 t)
        : xh(p_pack(dx.x, dx.x)), xl(p_pack(dx.y, dx.y)), nxh(p_pack(-dx.x, -dx.x)), yh(p_pack(dy.x, dy.x)),
          yl(p_pack(dy.y, dy.y)), nyh(p_pack(-dy.x, -dy.x)), th(p_pack(t.x, t.x)), tl(p_pack(t.y, t.y)),
          nth(p_pack(-t.x, -t.x)) {}
};

// The phases kx x + ky y - omega t + phase0 of two components (records R) as
// pairs (hi, lo): each product exact, the sums error-free in the hi parts.
__device__ __forceinline__ void ph_phase(const ulonglong2 *R, const PhPoint &P, f32x2 &hi, f32x2 &lo) {
    const f32x2 neg1 = p_pack(-1.f, -1.f);
    const ulonglong2 kx = R[0], ky = R[1], w = R[2], p0 = R[3];
    hi = p_mul(kx.x, P.xh);
    lo = p_fma(kx.x, P.xl, p_fma(kx.y, P.xh, p_fma(kx.x, P.xh, p_mul(kx.x, P.nxh))));
    auto add = [&](f32x2 h, f32x2 l) {
        const f32x2 s = p_add(hi, h), bb = p_fma(hi, neg1, s);
        const f32x2 d = p_fma(bb, neg1, s);
        const f32x2 e = p_add(p_fma(d, neg1, hi), p_fma(bb, neg1, h));
        hi = s;
        lo = p_add(p_add(lo, l), e);
    };
    add(p_mul(ky.x, P.yh), p_fma(ky.x, P.yl, p_fma(ky.y, P.yh, p_fma(ky.x, P.yh, p_mul(ky.x, P.nyh)))));
    add(p_mul(w.x, P.th), p_fma(w.x, P.tl, p_fma(w.y, P.th, p_fma(w.x, P.th, p_mul(w.x, P.nth)))));
    add(p0.x, p0.y);
}

// The phasors (cos, sin) and ramps of every component and the first-order
// sums eta1 and the Taylor gradients.  The phase
// kx (x - fx) + ky (y - fy) - omega t + phase0 is formed in float-float from
// the records (the point's coordinates split by integer operations) and
// reduced, then sine and cosine by polynomial (within 1e-7; the SFU's few
// 1e-7 raised the plain form's error against FP64 tenfold); the sums are FP32
// with Kahan compensation.  FP64 per (point, component) -- phase, reduction and FP64
// sums -- kept the FP64 pipe the bound on this GPU.  Only non-trivial
// component ramps are evaluated in FP64 (Irregular.cpp:200-204).
//
// A block takes 32 points, a warp every PH_WARPS-th pair of components of a
// chunk, the lanes the points (so the rows are written 256 bytes at a time);
// the warps' shares of the sums are added in warp order, compensated, and only
// the sums that the call's rows need are formed.  Instruction issue is the
// bound, so two components are worked on at once in packed FP32x2 (89
// instructions a phasor instead of 180).  A ramp that all components share is
// evaluated once per point and written once (row 0).  With a thread per point
// and all components in turn a batch of 5003 points was 40 blocks of one long
// chain: 73 us at 256 components, 20 us now; 65536 points, 128 components: 60
// us then, 38 now (4 warps a block; 2: 39, 8: 44).
constexpr int PH_WARPS = 4;
__global__ void __launch_bounds__(32 * PH_WARPS) k_phasors(PhArgs a) {
    __shared__ __align__(16) float s_rec[PH_CHUNK * PH_REC];
    __shared__ float2 s_off[2];
    __shared__ float2 s_sum[PH_WARPS][5][32];
    __shared__ float s_ramp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long p = blockIdx.x * 32L + lane;
    const bool valid = p < a.n;
    const long pc = valid ? p : 0;
    if (threadIdx.x == 0) {
        ff_split(-a.fx, s_off[0].x, s_off[0].y);
        ff_split(-a.fy, s_off[1].x, s_off[1].y);
    }
    const double tp = a.t[pc * a.st];
    const double *P = a.phase;
    const int cs = a.cstride;
    if (warp == 1 && a.trivial_ramp) {
        const float r0 = (float)d_freq_ramp(tp, P[4 * cs], P[5 * cs], P[6 * cs]);
        s_ramp[lane] = r0;
        if (valid) a.rr[p] = r0;
    }
    __syncthreads();
    const float2 dx = ff_add(ff_from_double(a.x[pc * a.sx]), s_off[0]);
    const float2 dy = ff_add(ff_from_double(a.y[pc * a.sy]), s_off[1]);
    const float2 tt = ff_from_double(tp);
    const float rconst = a.trivial_ramp ? s_ramp[lane] : 0.f;
    // everything below is on two components at once (packed FP32x2), as
    // instruction issue is the bound
    const f32x2 neg1 = p_pack(-1.f, -1.f);
    auto dup = [](float v) { return p_pack(v, v); };
    const PhPoint pt(dx, dy, tt);
    f32x2 S[5] = {0, 0, 0, 0, 0}, C[5] = {0, 0, 0, 0, 0};
    for (int i0 = 0; i0 < a.npad; i0 += PH_CHUNK) {
        const int nrec = min(PH_CHUNK, a.npad - i0);
        __syncthreads();
        for (int e = threadIdx.x; e < nrec * PH_REC / 4; e += blockDim.x)
            reinterpret_cast<float4 *>(s_rec)[e] = reinterpret_cast<const float4 *>(a.rec + (long)i0 * PH_REC)[e];
        __syncthreads();
        for (int ii = 2 * warp; ii < nrec; ii += 2 * PH_WARPS) {
            const int i = i0 + ii;
            const ulonglong2 *R = reinterpret_cast<const ulonglong2 *>(s_rec + ii * PH_REC);
            f32x2 hi, lo;
            ph_phase(R, pt, hi, lo);
            f32x2 c2, s2;
            ph_sincos(hi, lo, s2, c2);
            const float2 c = p_un(c2), s = p_un(s2);
            f32x2 rc = c2, rs = s2;
            if (a.trivial_ramp) {
                const f32x2 r2 = dup(rconst);
                rc = p_mul(r2, c2);
                rs = p_mul(r2, s2);
            } else {
                float r[2];
                for (int q = 0; q < 2; q++)
                    r[q] = i + q < a.ncomp ? (float)d_freq_ramp(tp, P[4 * cs + i + q], P[5 * cs + i + q],
                                                                P[6 * cs + i + q])
                                           : 0.f;
                const f32x2 r2 = p_pack(r[0], r[1]);
                rc = p_mul(r2, c2);
                rs = p_mul(r2, s2);
                if (valid) {
                    a.rr[(long)i * a.n + p] = r[0];
                    a.rr[(long)(i + 1) * a.n + p] = r[1];
                }
            }
            // (records past the last component are zero: phase 0, coefficients 0)
            const ulonglong2 a0 = R[4], a1 = R[5], a2 = R[6];
            const f32x2 cf[5] = {a0.x, a0.y, a1.x, a1.y, a2.x};
#pragma unroll
            for (int q = 0; q < 5; q++) {
                if (!(a.sums & (1 << q))) continue;
                // Kahan: y = v - C, t = S + y, C = (t - S) - y
                const f32x2 y = p_fma(C[q], neg1, p_mul(q == 3 ? rs : rc, cf[q]));
                const f32x2 t = p_add(S[q], y);
                C[q] = p_fma(y, neg1, p_fma(S[q], neg1, t));
                S[q] = t;
            }
            if (valid) {
                a.ph[(long)i * a.n + p] = make_float2(c.x, s.x);
                a.ph[(long)(i + 1) * a.n + p] = make_float2(c.y, s.y);
            }
        }
    }
    float sm[5], cm[5];
    for (int q = 0; q < 5; q++) {        // the two lanes
        const float2 t = p_un(S[q]), u = p_un(C[q]);
        sm[q] = t.x;
        cm[q] = u.x + u.y;
        ph_kahan(sm[q], cm[q], t.y);
    }
    for (int q = 0; q < 5; q++) s_sum[warp][q][lane] = make_float2(sm[q], cm[q]);
    __syncthreads();
    for (int q = warp; q < 5; q += PH_WARPS) {
        if (!valid || !(a.sums & (1 << q))) continue;
        float v = 0.f, c = 0.f;
        for (int w = 0; w < PH_WARPS; w++) {
            const float2 t = s_sum[w][q][lane];
            ph_kahan(v, c, t.x);
            c += t.y;                    // the share is t.x - t.y
        }
        a.first[q * a.n + p] = (double)v - (double)c;
    }
}

// Few points (a scalar call, a short batch): one block per point, the
// components spread over the threads, so that a point's N phasors are formed
// in parallel instead of by one thread in turn.  The same records and
// arithmetic per (point, component) as k_phasors; each thread's share of the
// five first-order sums is Kahan-compensated in FP32 and the 128 shares are
// added in FP64 (per point, not per component).
__global__ void __launch_bounds__(128) k_phasors_few(PhArgs a) {
    __shared__ double s_red[4][5];
    const long p = blockIdx.x;
    float2 off[2];
    ff_split(-a.fx, off[0].x, off[0].y);
    ff_split(-a.fy, off[1].x, off[1].y);
    const double tp = a.t[p * a.st];
    const float2 dx = ff_add(ff_from_double(a.x[p * a.sx]), off[0]);
    const float2 dy = ff_add(ff_from_double(a.y[p * a.sy]), off[1]);
    const float2 tt = ff_from_double(tp);
    const double *P = a.phase;
    const int cs = a.cstride;
    const float rconst = a.trivial_ramp ? (float)d_freq_ramp(tp, P[4 * cs], P[5 * cs], P[6 * cs]) : 0.f;
    float sm[5] = {0, 0, 0, 0, 0}, cm[5] = {0, 0, 0, 0, 0};
    for (int i = threadIdx.x; i < a.npad; i += blockDim.x) {
        float R[PH_REC];
#pragma unroll
        for (int q = 0; q < PH_REC; q++) R[q] = a.rec[rec_at(i, q)];
        float c = 0.f, sn = 0.f, r = 0.f;
        if (i < a.ncomp) {
            float2 ph = ff_add(ff_mul(R[0], R[1], dx.x, dx.y), ff_mul(R[2], R[3], dy.x, dy.y));
            ph = ff_add(ph, ff_mul(R[4], R[5], tt.x, tt.y));
            ph = ff_add(ph, make_float2(R[6], R[7]));
            ff_sincos_poly(ff_reduce_2pi(ph), sn, c);
            r = a.trivial_ramp ? rconst : (float)d_freq_ramp(tp, P[4 * cs + i], P[5 * cs + i], P[6 * cs + i]);
            const float rc = r * c, rs = r * sn;
            ph_kahan(sm[0], cm[0], rc * R[8]);
            ph_kahan(sm[1], cm[1], rc * R[9]);
            ph_kahan(sm[2], cm[2], rc * R[10]);
            ph_kahan(sm[3], cm[3], rs * R[11]);
            ph_kahan(sm[4], cm[4], rc * R[12]);
        }
        a.ph[(long)i * a.n + p] = make_float2(c, sn);
        if (!a.trivial_ramp || i == 0) a.rr[(long)i * a.n + p] = a.trivial_ramp ? rconst : r;
    }
    double v[5];
#pragma unroll
    for (int q = 0; q < 5; q++) {
        v[q] = (double)sm[q] - (double)cm[q];
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int q = 0; q < 5; q++) s_red[warp][q] = v[q];
    __syncthreads();
    if (threadIdx.x < 5)
        a.first[threadIdx.x * a.n + p] = ((s_red[0][threadIdx.x] + s_red[1][threadIdx.x]) + s_red[2][threadIdx.x]) +
                                         s_red[3][threadIdx.x];
}

// ---------------------------------------------------------------------------
// Pair-sum kernels
// ---------------------------------------------------------------------------
struct PairArgs {
    long ncol;           // points / columns
    int nl;              // levels per column
    int nlg;             // level groups per column (power of two, <= 16)
    int ntile;           // component tiles of the table
    const float *tab;    // pair tiles
    const float2 *tabp;  // pressure pair tiles (Pp, Mp), column kernel with pressure
    const float4 *tpp;   // point kernel: pressure tiles (Pp, Mp, kp, km)
    const float4 *tpk;   // and the phase-free products (X, Z)
    float one;           // 1 (p_hold)
    const float2 *ph;    // [npad][ncol]
    const float *rr;     // ramps: row stride rs (0 where every component has the same ramp)
    long rs;
    const float *cf;     // [NCF][cstride]
    int cstride;
    const float *z0;     // column kernel: [ncol*nl] evaluation heights (z0 <= 0 below the surface)
    float depth;
    const double *z;     // point kernel: the points' heights
    double swl, h;
    int order, clamp;    // clamp: the seabed clamp of the wave_* calls (z below -h evaluated at -h)
    float *out;          // [nf][ncol*nl]
    int pairs;           // point kernel; 0: first-order z-dependent sums only
    int first;           // 1: add first-order z-dependent sums
    int tp_per;          // tile pairs per blockIdx.y (split of the pair loop; partial sums
                         // of slice y go to out + y * nf * ncol * nl)
};

// Depth factors with the normaliser folded into the coefficients:
//   F = exp(kz) (1 + exp(-2k(z+h))),  G = exp(kz) (1 - exp(-2k(z+h))).
__device__ __forceinline__ void depth_fg(float k, float zk, float zetak, float &F, float &G) {
    const float e1 = ex2(k * zk);
    const float e2 = ex2(k * zetak);
    F = fmaf(e1, e2, e1);       // e1 (1 + e2), one rounding
    G = fmaf(-e1, e2, e1);      // e1 (1 - e2)
}

// Column mode: u, v, w (PR: and the phase terms of the pressure, with the
// first-order dp1) at LV levels per thread, grid (pair-cache) mask.
template <int TT, int LV, bool PR>
__global__ void __launch_bounds__(128) k_pairs_columns(PairArgs a) {
    extern __shared__ float4 smem4[];
    constexpr int NF = PR ? 4 : 3;
    float *s_tab = reinterpret_cast<float *>(smem4);                       // TT*TT*8
    float2 *s_tp = reinterpret_cast<float2 *>(s_tab + TT * TT * GRIDV_NC); // TT*TT (PR)
    float2 *s_ph = s_tp + (PR ? TT * TT : 0);                             // TT*cols
    const int cols = 128 / a.nlg;
    const int lg = threadIdx.x / cols, cl = threadIdx.x % cols;
    const long col = (long)blockIdx.x * cols + cl;
    const bool valid = col < a.ncol;
    const long colc = valid ? col : 0;
    const long npts = a.ncol * a.nl;
    static_assert(LV % 2 == 0, "levels are processed in pairs");
    constexpr int LP = LV / 2;
    float zk[LV], zetak[LV], yk[LV];   // z log2(e), -2(z + h) log2(e), -(z + 2h) log2(e)
    float2 zk2[LP], yk2[LP];
    float su[LV], cu[LV], sv[LV], cv[LV], sw[LV], cw[LV];
    float sp[PR ? LV : 1], cq[PR ? LV : 1];     // pressure sum and carry
#pragma unroll
    for (int l = 0; l < LV; l++) {
        int lev = lg * LV + l;
        float z = (valid && lev < a.nl) ? a.z0[colc * a.nl + lev] : 0.f;
        zk[l] = z * LOG2E_F;
        zetak[l] = -2.f * (z + a.depth) * LOG2E_F;
        yk[l] = -(z + 2.f * a.depth) * LOG2E_F;
        su[l] = cu[l] = sv[l] = cv[l] = sw[l] = cw[l] = 0.f;
        if (PR) sp[l] = cq[l] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < LP; j++) {
        zk2[j] = make_float2(zk[2 * j], zk[2 * j + 1]);
        yk2[j] = make_float2(yk[2 * j], yk[2 * j + 1]);
    }
    // slice of the tile-pair loop owned by this blockIdx.y (block-uniform)
    const int tp_lo = blockIdx.y * a.tp_per, tp_hi = tp_lo + a.tp_per;
    int tp = -1;
    for (int I = 0; I < a.ntile; I++) {
        for (int M = I; M < a.ntile; M++) {
            tp++;
            if (tp < tp_lo || tp >= tp_hi) continue;
            __syncthreads();
            const float4 *src = reinterpret_cast<const float4 *>(
                a.tab + tile_index(I, M, a.ntile) * (long)TT * TT * GRIDV_NC);
            float4 *dst = reinterpret_cast<float4 *>(s_tab);
            for (int e = threadIdx.x; e < TT * TT * GRIDV_NC / 4; e += blockDim.x) dst[e] = src[e];
            if (PR) {
                const float2 *srp = a.tabp + tile_index(I, M, a.ntile) * (long)TT * TT;
                for (int e = threadIdx.x; e < TT * TT; e += blockDim.x) s_tp[e] = srp[e];
            }
            for (int e = threadIdx.x; e < TT * cols; e += blockDim.x) {
                int mm = e / cols, c2 = e % cols;
                long cc = (long)blockIdx.x * cols + c2;
                s_ph[e] = (cc < a.ncol) ? a.ph[(long)(M * TT + mm) * a.ncol + cc] : make_float2(0.f, 0.f);
            }
            __syncthreads();
            if (!valid) continue;
            for (int ii = 0; ii < TT; ii++) {
                const int i = I * TT + ii;
                const float2 pi = a.ph[(long)i * a.ncol + col];
                const float ri = a.rr[(long)i * a.rs + col];
                // packed FP32x2 over level pairs: per pair and level,
                // E = exp(k z), Y = exp(-k(z + 2h)) = E exp(-2k(z+h)),
                // F = E + Y, G = E - Y (the normaliser is in the record)
                float2 au[LP], av[LP], aw[LP], apr[PR ? LP : 1];
#pragma unroll
                for (int j = 0; j < LP; j++) au[j] = av[j] = aw[j] = make_float2(0.f, 0.f);
#pragma unroll
                for (int j = 0; j < (PR ? LP : 1); j++) apr[j] = make_float2(0.f, 0.f);
                const float2 neg1 = make_float2(-1.f, -1.f);
                const int m0 = (M == I) ? ii : 0;
                for (int mm = m0; mm < TT; mm++) {
                    const float4 c0 = *reinterpret_cast<const float4 *>(s_tab + (ii * TT + mm) * GRIDV_NC);
                    const float4 c1 = *reinterpret_cast<const float4 *>(s_tab + (ii * TT + mm) * GRIDV_NC + 4);
                    const float2 pm = s_ph[mm * cols + cl];
                    const float cc = pi.x * pm.x, ss = pi.y * pm.y;
                    const float sc = pi.y * pm.x, cs = pi.x * pm.y;
                    const float cp = cc - ss, cmn = cc + ss, sp = sc + cs, smn = sc - cs;
                    const float up = c0.x * cp, um = c0.y * cmn, vp = c0.z * cp, vm = c0.w * cmn;
                    const float wp = c1.x * sp, wm = c1.y * smn;
                    const float2 up2 = make_float2(up, up), um2 = make_float2(um, um);
                    const float2 vp2 = make_float2(vp, vp), vm2 = make_float2(vm, vm);
                    const float2 wp2 = make_float2(wp, wp), wm2 = make_float2(wm, wm);
                    const float2 kp2 = make_float2(c1.z, c1.z), km2 = make_float2(c1.w, c1.w);
                    float2 pp2 = make_float2(0.f, 0.f), pm2 = pp2;
                    if (PR) {
                        const float2 tp = s_tp[ii * TT + mm];
                        const float pp = tp.x * cp, pm_ = tp.y * cmn;
                        pp2 = make_float2(pp, pp);
                        pm2 = make_float2(pm_, pm_);
                    }
#pragma unroll
                    for (int j = 0; j < LP; j++) {
                        const float2 ap = __fmul2_rn(kp2, zk2[j]), bp = __fmul2_rn(kp2, yk2[j]);
                        const float2 am = __fmul2_rn(km2, zk2[j]), bm = __fmul2_rn(km2, yk2[j]);
                        const float2 Ep = make_float2(ex2(ap.x), ex2(ap.y));
                        const float2 Yp = make_float2(ex2(bp.x), ex2(bp.y));
                        const float2 Em = make_float2(ex2(am.x), ex2(am.y));
                        const float2 Ym = make_float2(ex2(bm.x), ex2(bm.y));
                        const float2 Fp = __fadd2_rn(Ep, Yp), Gp = __ffma2_rn(Yp, neg1, Ep);
                        const float2 Fm = __fadd2_rn(Em, Ym), Gm = __ffma2_rn(Ym, neg1, Em);
                        au[j] = __ffma2_rn(up2, Fp, __ffma2_rn(um2, Fm, au[j]));
                        av[j] = __ffma2_rn(vp2, Fp, __ffma2_rn(vm2, Fm, av[j]));
                        aw[j] = __ffma2_rn(wp2, Gp, __ffma2_rn(wm2, Gm, aw[j]));
                        if (PR) apr[j] = __ffma2_rn(pp2, Fp, __ffma2_rn(pm2, Fm, apr[j]));
                    }
                }
#pragma unroll
                for (int j = 0; j < LP; j++) {
                    kahan(su[2 * j], cu[2 * j], ri * au[j].x);
                    kahan(su[2 * j + 1], cu[2 * j + 1], ri * au[j].y);
                    kahan(sv[2 * j], cv[2 * j], ri * av[j].x);
                    kahan(sv[2 * j + 1], cv[2 * j + 1], ri * av[j].y);
                    kahan(sw[2 * j], cw[2 * j], ri * aw[j].x);
                    kahan(sw[2 * j + 1], cw[2 * j + 1], ri * aw[j].y);
                    if (PR) {
                        kahan(sp[2 * j], cq[2 * j], ri * apr[j].x);
                        kahan(sp[2 * j + 1], cq[2 * j + 1], ri * apr[j].y);
                    }
                }
            }
            if (a.first && M == I) {
                // first-order u1, v1, w1 at the level heights (Irregular.cpp:394-447)
                for (int mm = 0; mm < TT; mm++) {
                    const int m = M * TT + mm;
                    const float2 pm = s_ph[mm * cols + cl];
                    const float rm = a.rr[(long)m * a.rs + col];
                    const float k = a.cf[CF_K * a.cstride + m], q = a.cf[CF_Q * a.cstride + m];
                    const float au_ = a.cf[CF_AU * a.cstride + m] * q * rm;
                    const float cu_ = au_ * a.cf[CF_CT * a.cstride + m] * pm.x;
                    const float cv_ = au_ * a.cf[CF_ST * a.cstride + m] * pm.x;
                    const float cw_ = au_ * pm.y;
                    // dp1 (Irregular.cpp:1107-1120)
                    const float cp_ = PR ? a.cf[CF_AP * a.cstride + m] * q * rm * pm.x : 0.f;
#pragma unroll
                    for (int l = 0; l < LV; l++) {
                        float F, G;
                        depth_fg(k, zk[l], zetak[l], F, G);
                        kahan(su[l], cu[l], cu_ * F);
                        kahan(sv[l], cv[l], cv_ * F);
                        kahan(sw[l], cw[l], cw_ * G);
                        if (PR) kahan(sp[l], cq[l], cp_ * F);
                    }
                }
            }
        }
    }
    if (!valid) return;
    float *out = a.out + (long)blockIdx.y * NF * npts;
#pragma unroll
    for (int l = 0; l < LV; l++) {
        int lev = lg * LV + l;
        if (lev < a.nl) {
            long o = col * a.nl + lev;
            out[0 * npts + o] = su[l];
            out[1 * npts + o] = sv[l];
            out[2 * npts + o] = sw[l];
            if (PR) out[3 * npts + o] = sp[l];
        }
    }
}

// Sum of the split slices of the column kernel, in slice order.
__global__ void k_sum_slices(long n, int nslice, const float *part, float *out) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= n) return;
    float s = 0.f, c = 0.f;
    for (int k = 0; k < nslice; k++) kahan(s, c, part[(long)k * n + e]);
    out[e] = s;
}

// Tile pair tp of a walk with the column tile M outermost: I = 0..M, so that a
// thread's phasors of tile M stay in registers for M + 1 tile pairs.
__device__ __forceinline__ void walk_at(int tp, int &I, int &M) {
    M = 0;
    while (tp > M) tp -= ++M;
    I = tp;
}

__device__ __forceinline__ void pr_cp16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void pr_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void pr_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// The height of a point's profiles, z0 = min(0, z - swl) (order 2 and 1) or z -
// swl (order 0): z0 and -2 (z0 + h), times log2(e).  In FP64, as an FP32
// z0 = -50 keeps little of z0 + h, on which the first-order vertical velocity near
// the seabed, e^{kz0} (1 - e^{-2k(z0+h)}), lives: RMS error of w over its own RMS within
// 5 m of the bed at 50 m 4.4e-7 with z0 + h in FP32, 2.1e-7 so (within 1 m 2.2e-6 and
// 1.1e-6; at 12 m depth, within 0.2 m, 2.9e-6 and 2.3e-6).
__device__ __forceinline__ void point_height(double z, double swl, double h, int order, int clamp, float &zk,
                                             float &zetak) {
    const double zz = (clamp ? fmax(-h, z) : z) - swl, z0 = order == 0 ? zz : fmin(0.0, zz);
    zk = (float)z0 * LOG2E_F;
    zetak = (float)(-2.0 * (z0 + h)) * LOG2E_F;
}

// Point mode: u, v, w, dp at one height per thread, point-API mask
// (u2/v2/w2/dp2 of the reference, with rho folded into the p records).
// VEL: the velocity sums, PR: the pressure sums (a call that asks for one of
// them does not pay for the other; rows not computed are 0).
//
// Per (pair, point) the velocity sums take 24 FMA-pipe instructions and 4
// exponentials, the pressure's 15 and 4.  A thread keeps its phasors (and for
// the pressure its profiles) of the 16 components of tile M in registers over
// the walk's tiles (I, M), two components to a packed FP32x2 operand, and the
// records, which all points share, come as broadcast reads of such operands
// from a double-buffered stage.  Packing halves the instructions issued (the
// FMA pipe's work is the same): unpacked, with phasors and profiles in shared
// memory, 42 instructions a pair were issued (issue 79 % busy), now 22 (FMA pipe
// 70 % busy, pressure: XU 66 %).  65536 points, 128 components: velocity and
// pressure sums 1331 us together then, 894 now; 5003 points, 256 components 491
// and 264 (tiles of 32 instead of 16 components: 1043 and 383; five blocks an
// SM instead of six: 882 and 307).  In a tile of the diagonal the records below
// it are zero; whole groups of four are skipped.  The pairs' profiles are E + Y and
// E - Y, Y = e^{-k(z+2h)}; as E (1 +- e), e = e^{-2k(z+h)}, which k_point_few takes, they
// cost a packed operation more each (65536 points 1171 us against 1134, with the
// velocity's sign by the integer pipe) for at most 5 % of w's error near the bed (8 and
// 12 m depth; none from 20 m on).
// KIN: the phase-free products of the first-order profiles in the pressure,
// summed here (otherwise the caller adds them from the height table).
template <bool VEL, bool PR, bool KIN>
struct PointStage {
    static constexpr int TT = POINT_TILE;
    static constexpr int V4 = VEL ? TT * TT * POINTV_NC / 4 : 0;      // float4 of a stage: velocity records,
    static constexpr int P4 = PR ? TT * TT * POINTP_NC / 4 : 0;       // pressure phase terms,
    static constexpr int K4 = KIN ? TT * TT * POINTK_NC / 4 : 0;      // phase-free products
    static constexpr int N4 = V4 + P4 + K4;
    static constexpr int SMEM = 2 * N4 * 16;
    static constexpr int ROWS = VEL ? 3 : 1;                          // u, v, w or p
};

template <bool VEL, bool PR, bool KIN>
__global__ void __launch_bounds__(128, KIN ? 2 : 6) k_pairs_points(PairArgs a) {
    static_assert(VEL != PR && (PR || !KIN), "one group of rows a launch");
    using ST = PointStage<VEL, PR, KIN>;
    constexpr int TT = POINT_TILE;
    extern __shared__ float4 smem4[];
    const int tid = threadIdx.x;
    const long p = (long)blockIdx.x * 128 + tid;
    const bool valid = p < a.ncol;
    const long pc = valid ? p : a.ncol - 1;
    float zk, zetak;
    point_height(a.z[pc], a.swl, a.h, a.order, a.clamp, zk, zetak);
    const float yk = zk + zetak;         // -(z + 2h)
    const f32x2 zk2 = p_pack(zk, zk), yk2 = p_pack(yk, yk), neg1 = p_pack(-1.f, -1.f);
    float su = 0, cu = 0, sv = 0, cv = 0, sw = 0, cw = 0, sq = 0, cq = 0;
    // slice of the tile-pair loop owned by this blockIdx.y (block-uniform);
    // without pairs the "walk" is the diagonal tiles
    const int ntp = a.pairs ? a.ntile * (a.ntile + 1) / 2 : a.ntile;
    const int lo = blockIdx.y * a.tp_per, hi = min(lo + a.tp_per, ntp);
    int I = lo, M = lo;
    if (a.pairs) walk_at(lo, I, M);
    int lI = I, lM = M, lt = lo;         // the next tile pair to load
    auto issue = [&]() {
        if (a.pairs && lt < hi) {
            const long e0 = tile_index(lI, lM, a.ntile) * (long)TT * TT;
            float4 *dst = smem4 + ((lt - lo) & 1) * ST::N4;
            if (VEL) {
                const float4 *src = reinterpret_cast<const float4 *>(a.tab) + e0 * (POINTV_NC / 4);
#pragma unroll
                for (int e = 0; e < ST::V4; e += 128) pr_cp16(dst + e + tid, src + e + tid);
            }
            if (PR) {
                const float4 *sp = a.tpp + e0;
#pragma unroll
                for (int e = 0; e < ST::P4; e += 128) pr_cp16(dst + ST::V4 + e + tid, sp + e + tid);
            }
            if (KIN) {
                const float4 *sk = a.tpk + e0 / 2;
#pragma unroll
                for (int e = 0; e < ST::K4; e += 128) pr_cp16(dst + ST::V4 + ST::P4 + e + tid, sk + e + tid);
            }
            if (++lI > lM) { lI = 0; lM++; }
        }
        lt++;
        pr_commit();
    };
    issue();
    const f32x2 one2 = p_pack(a.one, a.one);
    for (int t = lo; t < hi; M++) {
        // cosines and sines of tile M's components two by two, and (KIN) px, pz
        f32x2 pmc[TT / 2], pms[TT / 2], xmx[KIN ? TT / 2 : 1], xmz[KIN ? TT / 2 : 1];
        {
#pragma unroll
            for (int mm = 0; mm < TT; mm += 2) {
                const int m = M * TT + mm;
                const float2 p0 = a.ph[(long)m * a.ncol + pc], p1 = a.ph[(long)(m + 1) * a.ncol + pc];
                pmc[mm / 2] = p_hold(p0.x, p1.x, one2);
                pms[mm / 2] = p_hold(p0.y, p1.y, one2);
                if (KIN) {
                    float F0, G0, F1, G1;
                    depth_fg(a.cf[CF_K * a.cstride + m], zk, zetak, F0, G0);
                    depth_fg(a.cf[CF_K * a.cstride + m + 1], zk, zetak, F1, G1);
                    const float q0 = a.cf[CF_Q * a.cstride + m], q1 = a.cf[CF_Q * a.cstride + m + 1];
                    xmx[mm / 2] = p_hold(q0 * F0, q1 * F1, one2);
                    xmz[mm / 2] = p_hold(q0 * G0, q1 * G1, one2);
                }
            }
        }
        if (!a.pairs) I = M;
        for (; I <= M && t < hi; I++, t++) {
        issue();
        pr_wait1();
        __syncthreads();
        const ulonglong2 *tv = reinterpret_cast<const ulonglong2 *>(smem4) + ((t - lo) & 1) * ST::N4, *tq = tv + ST::V4,
                         *tx = tq + ST::P4;
        if (a.pairs) {
            const float2 *prow = a.ph + (long)(I * TT) * a.ncol + pc;
            const float *rrow = a.rr + (long)(I * TT) * a.rs + pc;
            float2 pn = *prow;
            float rn = *rrow;
            // off the diagonal a row is one branch-free block (its reads and
            // exponentials scheduled across the whole row)
            auto rows = [&](auto diag) {
                constexpr bool DIAG = decltype(diag)::value;
                for (int ii = 0; ii < TT; ii++) {
                    const int i = I * TT + ii;
                    const float2 pi = pn;
                    const float ri = rn;
                    if (ii + 1 < TT) {       // the next row's, under this row's sums
                        prow += a.ncol;
                        rrow += a.rs;
                        pn = *prow;
                        rn = *rrow;
                    }
                    const f32x2 px2 = p_pack(pi.x, pi.x), py2 = p_pack(pi.y, pi.y);
                    const f32x2 nx2 = p_pack(-pi.x, -pi.x), ny2 = p_pack(-pi.y, -pi.y);
                    f32x2 au = 0, av = 0, aw = 0, ap = 0, ax = 0, az = 0;
                    // the row's records; within it every read has a constant offset
                    const ulonglong2 *rv = tv + ii * (2 * TT), *rq = tq + ii * TT, *rx = tx + ii * (TT / 2);
#pragma unroll
                    for (int m4 = 0; m4 < TT; m4 += 4) {
                        if (DIAG && m4 + 3 < ii) continue;
#pragma unroll
                        for (int mm = m4; mm < m4 + 4; mm += 2) {
                            const f32x2 mc = pmc[mm / 2], ms = pms[mm / 2];
                            ulonglong2 r0, r1, r2, rk, rp;
                            if (VEL) {
                                r0 = rv[2 * mm]; r1 = rv[2 * mm + 1]; r2 = rv[2 * mm + 2]; rk = rv[2 * mm + 3];
                            }
                            if (PR) {
                                rp = rq[mm]; rk = rq[mm + 1];
                            }
                            // cos(phi_i +- phi_m), and sin below
                            const f32x2 cc = p_mul(px2, mc);
                            const f32x2 cp = p_fma(ny2, ms, cc), cm = p_fma(py2, ms, cc);
                            // E = exp(kz), Y = exp(-k(z + 2h)): F = E + Y, G = E - Y (the
                            // normaliser is in the record)
                            const f32x2 Ep = p_ex2(p_mul(rk.x, zk2)), Yp = p_ex2(p_mul(rk.x, yk2));
                            const f32x2 Em = p_ex2(p_mul(rk.y, zk2)), Ym = p_ex2(p_mul(rk.y, yk2));
                            // the phase-and-depth products once, then one FMA per coefficient
                            const f32x2 A = p_mul(cp, p_add(Ep, Yp)), B = p_mul(cm, p_add(Em, Ym));
                            if (VEL) {
                                const f32x2 sc = p_mul(py2, mc);
                                const f32x2 sp = p_fma(px2, ms, sc), sm = p_fma(nx2, ms, sc);
                                const f32x2 C = p_mul(sp, p_fma(Yp, neg1, Ep)), D = p_mul(sm, p_fma(Ym, neg1, Em));
                                au = p_fma(r0.x, A, p_fma(r0.y, B, au));
                                av = p_fma(r1.x, A, p_fma(r1.y, B, av));
                                aw = p_fma(r2.x, C, p_fma(r2.y, D, aw));
                            }
                            if (PR) ap = p_fma(rp.x, A, p_fma(rp.y, B, ap));
                            if (KIN) {
                                const ulonglong2 x2 = rx[mm / 2];
                                ax = p_fma(x2.x, xmx[mm / 2], ax);
                                az = p_fma(x2.y, xmz[mm / 2], az);
                            }
                        }
                    }
                    if (VEL) {
                        kahan(su, cu, ri * p_hsum(au));
                        kahan(sv, cv, ri * p_hsum(av));
                        kahan(sw, cw, ri * p_hsum(aw));
                    }
                    if (PR) {
                        float row = p_hsum(ap);
                        if (KIN) {
                            float F, G;
                            depth_fg(a.cf[CF_K * a.cstride + i], zk, zetak, F, G);
                            const float q = a.cf[CF_Q * a.cstride + i];
                            row = fmaf(q * F, p_hsum(ax), fmaf(q * G, p_hsum(az), row));
                        }
                        kahan(sq, cq, ri * row);
                    }
                }
            };
            if (M == I) rows(std::true_type{});
            else rows(std::false_type{});
        }
        if (a.first && M == I) {
            // first-order u1, v1, w1, dp1 and the linear dp2 diagonal terms
            for (int mm = 0; mm < TT; mm++) {
                const int m = M * TT + mm;
                const float2 pv = a.ph[(long)m * a.ncol + pc];
                const float rm = a.rr[(long)m * a.rs + pc];
                float F, G;
                depth_fg(a.cf[CF_K * a.cstride + m], zk, zetak, F, G);
                const float q = a.cf[CF_Q * a.cstride + m];
                const float px = q * F, pz = q * G;
                if (VEL) {
                    const float au_ = a.cf[CF_AU * a.cstride + m] * rm;
                    kahan(su, cu, au_ * px * a.cf[CF_CT * a.cstride + m] * pv.x);
                    kahan(sv, cv, au_ * px * a.cf[CF_ST * a.cstride + m] * pv.x);
                    kahan(sw, cw, au_ * pz * pv.y);
                }
                if (PR) {
                    float pp = a.cf[CF_AP * a.cstride + m] * px * pv.x;
                    if (KIN && a.pairs) pp += a.cf[CF_X1 * a.cstride + m] * px + a.cf[CF_Z1 * a.cstride + m] * pz;
                    kahan(sq, cq, rm * pp);
                }
            }
        }
        __syncthreads();                 // the stage is refilled by the next issue
        }
        I = 0;
    }
    if (!valid) return;
    float *out = a.out + (long)blockIdx.y * ST::ROWS * a.ncol;
    if (VEL) {
        out[p] = su;
        out[a.ncol + p] = sv;
        out[2 * a.ncol + p] = sw;
    } else {
        out[p] = sq;
    }
}

// Elevation mode: eta2 from the pair cache (Irregular.cpp:223-293).  The
// record holds A = P+M and B = M-P so that a pair contributes
// c_i (A c_m) + s_i (B s_m); a row is c_i sum(A c_m) + s_i sum(B s_m).
// (A, B) times (c_m, s_m) is one packed FMA, so a broadcast read of two records
// (two of the shared memory's cycles) has to feed several points or it is the
// bound: a thread takes two points, with their phasors of half a column tile
// (16 components) in registers, two rows a step; the column half is outermost in the
// walk.  65536 points, 128 components 139 us with the records and phasors read
// per point, 90 now; 5003 points, 256 components 49 and 37 (latency of the
// shared-memory reads and row loads; two points, one row a step: 88 and 37; four
// points 117 and 51; a whole tile's columns 93 and 35).
constexpr int ETA_P = 2, ETA_C = 16;                       // points a thread, columns of a walk step
constexpr int ETA_R = 2;                                   // rows of a step
constexpr int ETA_H = GRID_TILE / ETA_C;                   // walk steps of a tile pair
constexpr int ETA_N4 = GRID_TILE * ETA_C * EATA_NC / 4;    // float4 of a stage
constexpr int ETA_SMEM = 2 * ETA_N4 * 16;
__global__ void __launch_bounds__(128) k_pairs_eta(PairArgs a) {
    extern __shared__ float4 smem4[];
    constexpr int TT = GRID_TILE;
    const int tid = threadIdx.x;
    long p[ETA_P];
#pragma unroll
    for (int k = 0; k < ETA_P; k++) p[k] = min((long)blockIdx.x * 128 * ETA_P + 128 * k + tid, a.ncol - 1);
    float se[ETA_P], ce[ETA_P];
#pragma unroll
    for (int k = 0; k < ETA_P; k++) se[k] = ce[k] = 0.f;
    // step t: tile pair t mod (M + 1) of column tile M's part H
    const int nst = a.ntile * (a.ntile + 1) / 2 * ETA_H;
    const int lo = blockIdx.y * a.tp_per, hi = min(lo + a.tp_per, nst);
    int I, M, H;
    {
        int t = lo;
        M = 0;
        while (t >= ETA_H * (M + 1)) { t -= ETA_H * (M + 1); M++; }
        H = t / (M + 1);
        I = t % (M + 1);
    }
    auto next = [](int &i, int &m, int &h) {
        if (++i > m) {
            i = 0;
            if (++h >= ETA_H) { h = 0; m++; }
        }
    };
    int lI = I, lM = M, lH = H, lt = lo;
    auto issue = [&]() {
        if (lt < hi) {
            const float4 *src = reinterpret_cast<const float4 *>(a.tab) +
                                tile_index(lI, lM, a.ntile) * (long)(TT * TT * EATA_NC / 4) + lH * (ETA_C * EATA_NC / 4);
            float4 *dst = smem4 + ((lt - lo) & 1) * ETA_N4;
            constexpr int R4 = ETA_C * EATA_NC / 4;        // float4 of a row's half
#pragma unroll
            for (int e = 0; e < ETA_N4; e += 128)
                pr_cp16(dst + e + tid, src + (e + tid) / R4 * (TT * EATA_NC / 4) + (e + tid) % R4);
            next(lI, lM, lH);
        }
        lt++;
        pr_commit();
    };
    issue();
    const f32x2 one2 = p_pack(a.one, a.one);
    for (int t = lo; t < hi;) {
        f32x2 pm[ETA_P][ETA_C];
        const int m0 = M * TT + H * ETA_C;
        {
#pragma unroll
            for (int mm = 0; mm < ETA_C; mm++)
#pragma unroll
                for (int k = 0; k < ETA_P; k++) {
                    const float2 v = a.ph[(long)(m0 + mm) * a.ncol + p[k]];
                    pm[k][mm] = p_hold(v.x, v.y, one2);
                }
        }
        for (; I <= M && t < hi; I++, t++) {
        issue();
        pr_wait1();
        __syncthreads();
        const ulonglong2 *rec = reinterpret_cast<const ulonglong2 *>(smem4) + ((t - lo) & 1) * ETA_N4;
        // rows past the columns of a diagonal tile are zeros
        const int rows = M == I ? min(TT, (H + 1) * ETA_C) : TT;
        const float2 *prow[ETA_P];
        const float *rrow[ETA_P];
        float2 pn[ETA_R][ETA_P];
        float rn[ETA_R][ETA_P];
#pragma unroll
        for (int k = 0; k < ETA_P; k++) {
            prow[k] = a.ph + (long)(I * TT) * a.ncol + p[k];
            rrow[k] = a.rr + (long)(I * TT) * a.rs + p[k];
#pragma unroll
            for (int r = 0; r < ETA_R; r++) {
                pn[r][k] = prow[k][(long)r * a.ncol];
                rn[r][k] = rrow[k][(long)r * a.rs];
            }
        }
        for (int ii = 0; ii < rows; ii += ETA_R, rec += ETA_R * (ETA_C / 2)) {
            float2 pi[ETA_R][ETA_P];
            float ri[ETA_R][ETA_P];
#pragma unroll
            for (int k = 0; k < ETA_P; k++) {
#pragma unroll
                for (int r = 0; r < ETA_R; r++) {
                    pi[r][k] = pn[r][k];
                    ri[r][k] = rn[r][k];
                }
                if (ii + ETA_R < rows) {                   // the next rows', under these rows' sums
                    prow[k] += ETA_R * a.ncol;
                    rrow[k] += ETA_R * a.rs;
#pragma unroll
                    for (int r = 0; r < ETA_R; r++) {
                        pn[r][k] = prow[k][(long)r * a.ncol];
                        rn[r][k] = rrow[k][(long)r * a.rs];
                    }
                }
            }
            f32x2 acc[ETA_R][ETA_P];                       // sums of A c_m and B s_m
#pragma unroll
            for (int r = 0; r < ETA_R; r++)
#pragma unroll
                for (int k = 0; k < ETA_P; k++) acc[r][k] = 0;
#pragma unroll
            for (int mm = 0; mm < ETA_C; mm += 2)
#pragma unroll
                for (int r = 0; r < ETA_R; r++) {
                    const ulonglong2 c = rec[(r * ETA_C + mm) / 2];
#pragma unroll
                    for (int k = 0; k < ETA_P; k++)
                        acc[r][k] = p_fma(c.y, pm[k][mm + 1], p_fma(c.x, pm[k][mm], acc[r][k]));
                }
#pragma unroll
            for (int r = 0; r < ETA_R; r++)
#pragma unroll
                for (int k = 0; k < ETA_P; k++) {
                    const float2 s2 = p_un(acc[r][k]);
                    kahan(se[k], ce[k], ri[r][k] * fmaf(pi[r][k].x, s2.x, pi[r][k].y * s2.y));
                }
        }
        __syncthreads();
        }
        I = 0;
        if (++H >= ETA_H) { H = 0; M++; }
    }
#pragma unroll
    for (int k = 0; k < ETA_P; k++) {
        const long q = (long)blockIdx.x * 128 * ETA_P + 128 * k + tid;
        if (q < a.ncol) a.out[(long)blockIdx.y * a.ncol + q] = se[k];
    }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
namespace {

struct WsLayout {
    float2 *ph;
    float *rr;
    double *first;
    float *sec;
    float *split;         // partial sums of a split point-pair launch
    long split_cap;       // its floats
    size_t bytes;
};

// Resident blocks of a kernel on the current device (0 where the query fails).
template <typename K>
static long resident_slots(K kernel, int threads, size_t smem) {
    int dev = 0, nsm = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (long)per * nsm;
}
// floats of the split region: room for 7 partial rows per slice and point at
// slices x points = 256 SPLIT_TARGET_BLOCKS; the launches take no more
// slices than the region holds for their batch.  It has that fixed size,
// whatever the batch (a batch's last, short chunk may split while its first
// does not).
static long point_split_floats(long n) {
    (void)n;
    return 7L * 128 * 2 * SPLIT_TARGET_BLOCKS;
}

WsLayout layout(long n, int npad, void *base) {
    WsLayout L;
    size_t off = 0;
    auto take = [&](size_t b) { size_t o = off; off += (b + 255) & ~size_t(255); return o; };
    size_t o_ph = take(sizeof(float2) * (size_t)npad * n);
    size_t o_rr = take(sizeof(float) * (size_t)npad * n);
    size_t o_first = take(sizeof(double) * 5 * (size_t)n);
    size_t o_sec = take(sizeof(float) * 5 * (size_t)n);
    const long scap = point_split_floats(n);
    size_t o_split = take(sizeof(float) * (size_t)std::max<long>(scap, 1));
    char *b = (char *)base;
    L.ph = (float2 *)(b + o_ph);
    L.rr = (float *)(b + o_rr);
    L.first = (double *)(b + o_first);
    L.sec = (float *)(b + o_sec);
    L.split = (float *)(b + o_split);
    L.split_cap = scap;
    L.bytes = off;
    return L;
}

// K(z) of a height table [nz][2] (K, dK/dz) over [-h, 0], by cubic Hermite
__device__ __forceinline__ double kin_at(const double *kin, int nz, double h, double z) {
    const double dz = h / (nz - 1);
    const double t = fmin(fmax((z + h) / dz, 0.0), (double)(nz - 1));
    const int i = min((int)t, nz - 2);
    const double r = t - i;
    const double f0 = kin[2 * i], f1 = kin[2 * i + 2], d0 = kin[2 * i + 1], d1 = kin[2 * i + 3];
    const double a = dz * d0 - (f1 - f0), b = -dz * d1 + (f1 - f0);
    return f0 * (1.0 - r) + f1 * r + r * (1.0 - r) * (a * (1.0 - r) + b * r);
}

// Irregular::eta/u/v/w/dp assembled from the pieces (Irregular.cpp:9-157).
// out has row stride ldo (the full batch length).
// With any row or record of api set, the API rows and records are written
// here (the finishing pass folded in) instead of out.
// kt.kin: the pressure's phase-free part is added here from the height table
// (cubic Hermite in FP64), times the point's ramp.
struct KinTab {
    const double *kin;      // [nz][2] over [-h, 0], or null
    int nz;
    double h, depth;
    const float *rr;
};
__global__ void k_combine(long n, long ldo, int order, double swl, const double *z,
                          const double *first, const float *sec, const float *eta2, int mask,
                          double *out, ApiRows api, KinTab kt) {
    long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (p >= n) return;
    double za = (order == 2) ? fmax(0.0, z[p] - swl) : 0.0;
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (mask & 1) v[0] = swl + first[0 * n + p] + (eta2 ? (double)eta2[p] : 0.0);
    if (mask & 2) v[1] = (double)sec[0 * n + p] + first[1 * n + p] * za;
    if (mask & 4) v[2] = (double)sec[1 * n + p] + first[2 * n + p] * za;
    if (mask & 8) v[3] = (double)sec[2 * n + p] + first[3 * n + p] * za;
    if (mask & 16) v[4] = (double)sec[3 * n + p] + first[4 * n + p] * za;
    if ((mask & 16) && kt.kin) {
        const double z0 = fmin(0.0, fmax(-kt.depth, z[p]) - swl);
        v[4] += (double)kt.rr[p] * kin_at(kt.kin, kt.nz, kt.h, z0);
    }
    if (!api.any()) {
        for (int q = 0; q < 5; q++)
            if (mask & (1 << q)) out[q * ldo + p] = v[q];
        return;
    }
    v[5] = v[4] - api.rho * api.g * v[0];
    api_store(api, p, v);
}

// ---------------------------------------------------------------------------
// Few points (a scalar call, a short batch).  Block (point, slice): every block
// forms the point's phasors in shared memory (two components a thread at once),
// then its threads take items of the sums in turn -- eight terms of a row of a
// tile pair of the velocity, pressure or elevation tables, and the first-order
// terms of a component -- and the block's sums go to its slice's partial sums.
// k_few_finish, launched so that it is there when they are written, adds the
// slices in a fixed order, assembles eta, u, v, w, dp and writes the rows (with one
// slice k_point_few does).  What bounds a call is latency: as separate kernels
// (phasors, heights, elevation and point pairs, slice sums, combining pass) a
// wave_VeloX call of the 128-component sea was five dependent kernels, 26 us; 18 us
// now (a launch and a synchronisation are 8 of these).  The blocks of a point could
// also find out the last of them by a counter, no faster (four scalar calls 75 us with
// the counter, 73 so, 69 with the first order as items of its own), but this way
// nothing carries over from one call to the next, whatever the workspace held and
// whichever streams share it.
//
// Accuracy.  A single value is held to its own size, not to that of the largest
// of a batch, and the first order is nearly all of it.  Its terms are formed in
// float pairs (phase, sine, profiles, coefficients; 1e-8), as is every sum over
// the threads and slices: 40 x 3 components, u 9e-9 RMS of the field, 1.1e-7 with
// FP32 terms.  Heights above the bed, z + h, are taken in FP64: of an FP32 z = -50
// little is left of them, and w = sinh(k(z + h)) lives on that difference.  For
// the same reason the pairs' profiles are e1 (1 +- e2), e2 = e^{-2k(z+h)}, not E +-
// Y with Y = e^{-k(z+2h)}, whose exponents, of up to 40, round apart: w within
// 3 m of the bed, 128 components at 50 m, 3.1e-7 RMS of its maximum with E - Y.
// ---------------------------------------------------------------------------
constexpr int FEW_T = 128;           // threads of a block
constexpr int FEW_Q = 10;            // sums: eta2, u, v, w, dp, then eta1, gx, gy, gz, gp
constexpr int FEW_E = 8;             // terms of an item
struct FewArgs {
    long n, ldo;
    const double *x, *y, *z, *t;
    double swl, depth;
    float2 ox, oy;                   // -fx, -fy
    int ncomp, npad, cstride, trivial_ramp, order, clamp, kin, mask;
    const float *rec, *cf;
    const float2 *cfp;
    const double *phase;
    int ntp, ntg;                    // point and grid table tiles per side
    const float *tabv, *tpp, *tpk, *tabe;
    long nv, np, ne;                 // items of the velocity, pressure and elevation sums
    float2 *part;                    // [slices][FEW_Q][n] sums and their rounding errors
    double *out;
    ApiRows api;
    KinTab kt;
};

// whether a call of this mask needs sum q
__device__ __forceinline__ bool few_needs(int mask, int q) { return mask >> (q < 5 ? q : q - 5) & 1; }

// s + e += v, the rounding errors of s in e
__device__ __forceinline__ void few_add(float2 &s, float v) {
    const float2 t = ff_two_sum(s.x, v);
    s.x = t.x;
    s.y += t.y;
}
__device__ __forceinline__ void few_add(float2 &s, float2 v) {
    few_add(s, v.x);
    s.y += v.y;
}

// (I, M) of tile t of an upper triangle of nt x nt tiles
__device__ __forceinline__ void tile_at(long t, int nt, int &I, int &M) {
    const float b = 2.f * nt + 1.f;
    I = min(nt - 1, max(0, (int)((b - sqrtf(fmaxf(0.f, b * b - 8.f * (float)t))) * 0.5f)));
    while (I > 0 && tile_index(I, I, nt) > t) I--;
    while (I + 1 < nt && tile_index(I + 1, I + 1, nt) <= t) I++;
    M = I + (int)(t - tile_index(I, I, nt));
}

// The first-order terms of component i (Irregular.cpp:178-198, 394-447, 1107-1192)
// at offsets dx, dy and time t, heights z and zeta = -2 (z + h), ramp r.
__device__ __forceinline__ void few_first(const FewArgs &a, int i, float2 dx, float2 dy, float2 t, float2 z, float2 zeta,
                                          float r, float2 S[FEW_Q]) {
    const float *R = a.rec;
    auto rec = [&](int q) { return R[rec_at(i, q)]; };
    auto cf = [&](int q) { return a.cfp[q * a.cstride + i]; };
    float2 ph = ff_add(ff_mul(rec(0), rec(1), dx.x, dx.y), ff_mul(rec(2), rec(3), dy.x, dy.y));
    ph = ff_add(ph, ff_mul(rec(4), rec(5), t.x, t.y));
    ph = ff_add(ph, make_float2(rec(6), rec(7)));
    float2 s, c;
    ff_sincos(ph, s, c);
    c = ff_mul(r, 0.f, c.x, c.y);
    s = ff_mul(r, 0.f, s.x, s.y);
    if (a.mask & 1) few_add(S[5], ff_mul(cf(CF_A), c));
    if (!(a.mask & 30)) return;
    // q E (1 +- e2), E = e^{kz}, e2 = e^{k zeta}
    const float2 k = cf(CF_K);
    float2 p, p2;
    const float T = ff_exp(ff_mul(k, z), p), T2 = ff_exp(ff_mul(k, zeta), p2);
    float2 E = ff_two_sum(1.f, p.x), up = ff_two_sum(1.f + T2, T2 * p2.x), um = ff_two_sum(1.f - T2, -T2 * p2.x);
    E.y += p.y;
    up.y += T2 * p2.y;
    um.y -= T2 * p2.y;
    E = ff_mul(cf(CF_Q), make_float2(T * E.x, T * E.y));
    const float2 F = ff_mul(E, up), G = ff_mul(E, um);
    if (a.mask & 6) {
        const float2 u = ff_mul(ff_mul(cf(CF_AU), F), c);
        few_add(S[1], ff_mul(u, cf(CF_CT)));
        few_add(S[2], ff_mul(u, cf(CF_ST)));
        few_add(S[6], ff_mul(cf(CF_GX), c));
        few_add(S[7], ff_mul(cf(CF_GY), c));
    }
    if (a.mask & 8) {
        few_add(S[3], ff_mul(ff_mul(cf(CF_AU), G), s));
        few_add(S[8], ff_mul(cf(CF_GZ), s));
    }
    if (a.mask & 16) {
        few_add(S[4], ff_mul(ff_mul(cf(CF_AP), F), c));
        if (a.kin) few_add(S[4], r * fmaf(cf(CF_X1).x, F.x, cf(CF_Z1).x * G.x));
        few_add(S[9], ff_mul(cf(CF_GP), c));
    }
}

// Irregular::eta/u/v/w/dp of point p from its sums (Irregular.cpp:9-157); kin: the
// pressure's phase-free part from the height table.
__device__ __forceinline__ void few_rows(const FewArgs &a, long p, const double *sum, double kin) {
    const double za = a.order == 2 ? fmax(0.0, a.z[p] - a.swl) : 0.0;
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (a.mask & 1) v[0] = a.swl + sum[5] + sum[0];
    for (int q = 1; q < 5; q++)
        if (a.mask & (1 << q)) v[q] = sum[q] + sum[5 + q] * za;
    v[4] += kin;
    if (!a.api.any()) {
        for (int q = 0; q < 5; q++)
            if (a.mask & (1 << q)) a.out[q * a.ldo + p] = v[q];
        return;
    }
    v[5] = v[4] - a.api.rho * a.api.g * v[0];
    api_store(a.api, p, v);
}

__global__ void __launch_bounds__(FEW_T) k_point_few(FewArgs a) {
    extern __shared__ float2 s_few[];
    float2 *s_ph = s_few;                                   // phasors [npad]
    float2 *s_px = s_ph + a.npad;                           // kin: profiles px, pz [npad]
    float *s_r = reinterpret_cast<float *>(s_px + (a.kin ? a.npad : 0));   // ramps [npad] (individual ramps)
    __shared__ float2 s_red[FEW_T / 32][FEW_Q];
    __shared__ double s_sum[FEW_Q], s_z0;
    __shared__ float2 s_z, s_zeta;                          // z0, -2 (z0 + h)
    __shared__ float s_ramp;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int tid = threadIdx.x;
    const long p = blockIdx.x;
    const int ns = gridDim.y, slice = blockIdx.y;
    const double xp = a.x[p], yp = a.y[p], tp = a.t[p];
    const double *P = a.phase;
    const int cs = a.cstride;
    // FP64 by one thread (an instruction holds the pipe for 16 cycles a warp; by every
    // thread, 24 components, 4096 points: 178 us a call, 148 so)
    if (tid == 0) {
        const double zz = (a.clamp ? fmax(-a.depth, a.z[p]) : a.z[p]) - a.swl, z0 = a.order == 0 ? zz : fmin(0.0, zz);
        s_z0 = z0;
        s_z = ff_from_double(z0);
        s_zeta = ff_from_double(-2.0 * (z0 + a.depth));
    }
    if (a.trivial_ramp) {
        if (tid == FEW_T - 1) s_ramp = (float)d_freq_ramp(tp, P[4 * cs], P[5 * cs], P[6 * cs]);
    } else {
        for (int i = tid; i < a.npad; i += FEW_T)
            s_r[i] = i < a.ncomp ? (float)d_freq_ramp(tp, P[4 * cs + i], P[5 * cs + i], P[6 * cs + i]) : 0.f;
    }
    const float2 dx = ff_add(ff_from_double(xp), a.ox), dy = ff_add(ff_from_double(yp), a.oy), tt = ff_from_double(tp);
    {
        const PhPoint pt(dx, dy, tt);
        for (int i = 2 * tid; i < a.npad; i += 2 * FEW_T) {
            f32x2 hi, lo, s2, c2;
            ph_phase(reinterpret_cast<const ulonglong2 *>(a.rec + (long)i * PH_REC), pt, hi, lo);
            ph_sincos(hi, lo, s2, c2);
            const float2 c = p_un(c2), s = p_un(s2);
            s_ph[i] = make_float2(c.x, s.x);
            s_ph[i + 1] = make_float2(c.y, s.y);
        }
    }
    __syncthreads();
    const float zk = s_z.x * LOG2E_F, zetak = s_zeta.x * LOG2E_F;
    if (a.kin) {
        for (int i = tid; i < a.npad; i += FEW_T) {
            // cosh(k(z+h))/cosh(kh), sinh(k(z+h))/cosh(kh)
            const float q = a.cf[CF_Q * cs + i];
            float F, G;
            depth_fg(a.cf[CF_K * cs + i], zk, zetak, F, G);
            s_px[i] = make_float2(q * F, q * G);
        }
        __syncthreads();
    }
    auto ramp = [&](int i) { return a.trivial_ramp ? s_ramp : s_r[i]; };
    float2 S[FEW_Q];
#pragma unroll
    for (int q = 0; q < FEW_Q; q++) S[q] = make_float2(0.f, 0.f);
    // pair items, eight terms each, then the components' first order; the records of
    // two neighbouring terms are interleaved (velocity, pressure) or adjacent
    // (elevation)
    const f32x2 zk2 = p_pack(zk, zk), zetak2 = p_pack(zetak, zetak), neg1 = p_pack(-1.f, -1.f);
    const long total = a.nv + a.np + a.ne;
    for (long item = (long)slice * FEW_T + tid; item < total + a.ncomp; item += (long)ns * FEW_T) {
        if (item >= total) {
            const int i = (int)(item - total);
            few_first(a, i, dx, dy, tt, s_z, s_zeta, ramp(i), S);
            continue;
        }
        int I, M, i, m0;
        if (item < a.nv + a.np) {
            const bool vel = item < a.nv;
            const long it = vel ? item : item - a.nv;
            constexpr int TT = POINT_TILE, CH = TT / FEW_E;
            const int ch = (int)(it % CH), ii = (int)(it / CH % TT);
            const long t = it / (CH * TT);
            tile_at(t, a.ntp, I, M);
            i = I * TT + ii;
            m0 = M * TT + ch * FEW_E;
            if (m0 + FEW_E <= i) continue;                  // below the diagonal: zeros
            const long e2 = (t * TT * TT + ii * TT + ch * FEW_E) / 2;
            const float2 pi = s_ph[i];
            const f32x2 px2 = p_pack(pi.x, pi.x), py2 = p_pack(pi.y, pi.y), nx2 = p_pack(-pi.x, -pi.x),
                        ny2 = p_pack(-pi.y, -pi.y);
            const ulonglong2 *RV = reinterpret_cast<const ulonglong2 *>(a.tabv) + e2 * (POINTV_NC / 2);
            const ulonglong2 *RP = reinterpret_cast<const ulonglong2 *>(a.tpp) + e2 * (POINTP_NC / 2);
            const ulonglong2 *RK = reinterpret_cast<const ulonglong2 *>(a.tpk) + e2 * (POINTK_NC / 2);
            f32x2 au = 0, av = 0, aw = 0, ap = 0, ax = 0, az = 0;
#pragma unroll
            for (int k = 0; k < FEW_E / 2; k++) {
                const float2 q0 = s_ph[m0 + 2 * k], q1 = s_ph[m0 + 2 * k + 1];
                const f32x2 mc = p_pack(q0.x, q1.x), ms = p_pack(q0.y, q1.y);
                const f32x2 cc = p_mul(px2, mc);
                const f32x2 cp = p_fma(ny2, ms, cc), cm = p_fma(py2, ms, cc);
                const ulonglong2 rk = vel ? RV[4 * k + 3] : RP[2 * k + 1];
                const f32x2 Ep = p_ex2(p_mul(rk.x, zk2)), ep = p_ex2(p_mul(rk.x, zetak2));
                const f32x2 Em = p_ex2(p_mul(rk.y, zk2)), em = p_ex2(p_mul(rk.y, zetak2));
                const f32x2 A = p_mul(cp, p_fma(Ep, ep, Ep)), B = p_mul(cm, p_fma(Em, em, Em));
                if (vel) {
                    const ulonglong2 r0 = RV[4 * k], r1 = RV[4 * k + 1], r2 = RV[4 * k + 2];
                    const f32x2 sc = p_mul(py2, mc);
                    const f32x2 sp = p_fma(px2, ms, sc), sm = p_fma(nx2, ms, sc);
                    const f32x2 Cc = p_mul(sp, p_fma(Ep, p_mul(ep, neg1), Ep));
                    const f32x2 D = p_mul(sm, p_fma(Em, p_mul(em, neg1), Em));
                    au = p_fma(r0.x, A, p_fma(r0.y, B, au));
                    av = p_fma(r1.x, A, p_fma(r1.y, B, av));
                    aw = p_fma(r2.x, Cc, p_fma(r2.y, D, aw));
                } else {
                    const ulonglong2 rp = RP[2 * k];
                    ap = p_fma(rp.x, A, p_fma(rp.y, B, ap));
                    if (a.kin) {
                        const ulonglong2 x2 = RK[k];
                        const float2 w0 = s_px[m0 + 2 * k], w1 = s_px[m0 + 2 * k + 1];
                        ax = p_fma(x2.x, p_pack(w0.x, w1.x), ax);
                        az = p_fma(x2.y, p_pack(w0.y, w1.y), az);
                    }
                }
            }
            const float ri = ramp(i);
            if (vel) {
                few_add(S[1], ri * p_hsum(au));
                few_add(S[2], ri * p_hsum(av));
                few_add(S[3], ri * p_hsum(aw));
            } else {
                float row = p_hsum(ap);
                if (a.kin) row = fmaf(s_px[i].x, p_hsum(ax), fmaf(s_px[i].y, p_hsum(az), row));
                few_add(S[4], ri * row);
            }
        } else {
            const long it = item - a.nv - a.np;
            constexpr int TT = GRID_TILE, CH = TT / FEW_E;
            const int ch = (int)(it % CH), ii = (int)(it / CH % TT);
            const long t = it / (CH * TT);
            tile_at(t, a.ntg, I, M);
            i = I * TT + ii;
            m0 = M * TT + ch * FEW_E;
            if (m0 + FEW_E <= i) continue;
            const ulonglong2 *RE = reinterpret_cast<const ulonglong2 *>(a.tabe) +
                                   (t * TT * TT + ii * TT + ch * FEW_E) * EATA_NC / 4;
            f32x2 acc = 0;                                  // sums of A c_m and B s_m
#pragma unroll
            for (int k = 0; k < FEW_E / 2; k++) {
                const ulonglong2 c = RE[k];
                const float2 q0 = s_ph[m0 + 2 * k], q1 = s_ph[m0 + 2 * k + 1];
                acc = p_fma(c.y, p_pack(q1.x, q1.y), p_fma(c.x, p_pack(q0.x, q0.y), acc));
            }
            const float2 s2 = p_un(acc), pi = s_ph[i];
            few_add(S[0], ramp(i) * fmaf(pi.x, s2.x, pi.y * s2.y));
        }
    }
    // the block's sums with their rounding errors: at one or a few terms a thread
    // the tree is most of the summation
#pragma unroll
    for (int q = 0; q < FEW_Q; q++) {
        if (!few_needs(a.mask, q)) continue;
        float2 v = S[q];
        for (int o = 16; o > 0; o >>= 1)
            few_add(v, make_float2(__shfl_down_sync(0xffffffffu, v.x, o), __shfl_down_sync(0xffffffffu, v.y, o)));
        if ((tid & 31) == 0) s_red[tid >> 5][q] = v;
    }
    __syncthreads();
    if (tid < FEW_Q && few_needs(a.mask, tid)) {
        float2 v = s_red[0][tid];
        for (int w = 1; w < FEW_T / 32; w++) few_add(v, s_red[w][tid]);
        if (ns > 1) a.part[((long)slice * FEW_Q + tid) * a.n + p] = v;
        else s_sum[tid] = (double)v.x + (double)v.y;
    }
    if (ns > 1) return;
    __syncthreads();
    if (tid == 0) few_rows(a, p, s_sum, (a.mask & 16) && a.kt.kin ? s_ramp * kin_at(a.kt.kin, a.kt.nz, a.kt.h, s_z0) : 0.0);
}

// The slices of a point's sums, a warp a sum in turn, its lanes over the slices.
__global__ void __launch_bounds__(FEW_T) k_few_finish(FewArgs a, int ns) {
    __shared__ double s_sum[FEW_Q];
    const int lane = threadIdx.x & 31;
    const long p = blockIdx.x;
    double kin = 0.0;
    if (threadIdx.x == 0 && (a.mask & 16) && a.kt.kin) {
        const double *P = a.phase + 4 * a.cstride;
        const double z0 = fmin(0.0, (a.clamp ? fmax(-a.depth, a.z[p]) : a.z[p]) - a.swl);
        kin = (float)d_freq_ramp(a.t[p], P[0], P[a.cstride], P[2 * a.cstride]) * kin_at(a.kt.kin, a.kt.nz, a.kt.h, z0);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");       // k_point_few's sums; what is above only reads inputs
    for (int q = threadIdx.x >> 5; q < FEW_Q; q += FEW_T / 32) {
        if (!few_needs(a.mask, q)) continue;
        double v = 0.0;
        for (int k = lane; k < ns; k += 32) {
            const float2 f = a.part[((long)k * FEW_Q + q) * a.n + p];
            v += (double)f.x + (double)f.y;
        }
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) s_sum[q] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) few_rows(a, p, s_sum, kin);
}

}  // namespace

static int launch_phasors(const DevSea &sea, long n, const double *x, const double *y,
                          const double *t, long sx, long sy, long st, int npad, float2 *ph,
                          float *rr, double *first, cudaStream_t stream, int sums = 31) {
    PhArgs a;
    a.sums = sums;
    a.n = n; a.x = x; a.y = y; a.t = t; a.sx = sx; a.sy = sy; a.st = st;
    a.ncomp = sea.n; a.npad = npad; a.phase = sea.d_phase; a.cf = sea.d_cf;
    a.cstride = sea.npad_g; a.fx = sea.fx; a.fy = sea.fy;
    a.trivial_ramp = sea.trivial_ramp ? 1 : 0;
    a.ph = ph; a.rr = rr; a.first = first; a.rec = sea.d_phrec;
    if (!sea.d_phrec || npad > ((sea.npad_g + 255) / 256) * 256) return E_BAD_ARGUMENT;
    prof_begin(PK_PHASORS, stream);
    if (n <= PH_FEW_POINTS)
        k_phasors_few<<<(unsigned)n, 128, 0, stream>>>(a);
    else
        k_phasors<<<(unsigned)((n + 31) / 32), 32 * PH_WARPS, 0, stream>>>(a);
    note_launch();
    prof_end(PK_PHASORS, stream);
    CK(cudaGetLastError());
    return OK;
}

int launch_phasors_public(const DevSea &sea, long n, const double *x, const double *y,
                          const double *t, long sx, long sy, long st, int npad, float2 *ph,
                          float *rr, double *first, cudaStream_t stream) {
    return launch_phasors(sea, n, x, y, t, sx, sy, st, npad, ph, rr, first, stream);
}

int launch_eta_pairs(const DevSea &sea, long n, const float2 *ph, const float *rr, float *out,
                     cudaStream_t stream, float *split_buf = nullptr, long split_cap = 0) {
    PairArgs a{};
    a.ncol = n; a.nl = 1; a.nlg = 1; a.ntile = sea.ntile_g; a.tab = sea.d_tab_eta;
    a.ph = ph; a.rr = rr; a.rs = sea.trivial_ramp ? 0 : n; a.cf = sea.d_cf; a.cstride = sea.npad_g; a.out = out;
    a.first = 0; a.one = 1.f;
    const long nblk = (n + 128 * ETA_P - 1) / (128 * ETA_P);
    const int ntp = sea.ntile_g * (sea.ntile_g + 1) / 2 * ETA_H;   // steps of the walk
    constexpr size_t smem = ETA_SMEM;
    static_assert(smem <= 48 * 1024, "no shared-memory opt-in needed");
    static const long slots = [&] {
        const long v = resident_slots(k_pairs_eta, 128, smem);
        return v > 0 ? v : SPLIT_TARGET_BLOCKS;
    }();
    // the tile-pair loop split over blockIdx.y where the columns alone do
    // not fill whole waves of the resident blocks (slices summed in order)
    a.tp_per = slice_plan(nblk, ntp, slots, split_buf ? split_cap / std::max<long>(1, n) : 1);
    const int nslice = (ntp + a.tp_per - 1) / a.tp_per;
    if (nslice > 1) a.out = split_buf;
    prof_begin(PK_ETA_PAIRS, stream);
    k_pairs_eta<<<dim3((unsigned)nblk, (unsigned)nslice), 128, smem, stream>>>(a);
    note_launch();
    prof_end(PK_ETA_PAIRS, stream);
    CK(cudaGetLastError());
    if (nslice > 1) {
        k_sum_slices<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(n, nslice, split_buf, out);
        note_launch();
        CK(cudaGetLastError());
    }
    return OK;
}

long column_pairs_split_floats(int nl) {
    constexpr int LV = 8;
    int nlg = 1;
    while (nlg * LV < nl) nlg *= 2;
    long cols = 128 / nlg;
    return 4L * nl * cols * 2 * SPLIT_TARGET_BLOCKS;
}

template <bool PR>
static int column_pairs_t(const PairArgs &a, long nblk, int nslice, int cols, cudaStream_t stream) {
    constexpr int LV = 8;
    auto bytes = [](int c) {
        return sizeof(float) * GRID_TILE * GRID_TILE * GRIDV_NC + (PR ? sizeof(float2) * GRID_TILE * GRID_TILE : 0) +
               sizeof(float2) * GRID_TILE * c;
    };
    // set once per process (thread-safe static initialisation)
    static const cudaError_t attr = cudaFuncSetAttribute(k_pairs_columns<GRID_TILE, LV, PR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)bytes(128));
    CK(attr);
    prof_begin(PK_COLUMN_PAIRS, stream);
    k_pairs_columns<GRID_TILE, LV, PR><<<dim3((unsigned)nblk, (unsigned)nslice), 128, bytes(cols), stream>>>(a);
    note_launch();
    prof_end(PK_COLUMN_PAIRS, stream);
    CK(cudaGetLastError());
    return OK;
}

// u, v, w (pressure: and p) sums of the columns at their levels, out [nf][ncol nl]
int launch_column_pairs(const DevSea &sea, long ncol, int nl, const float2 *ph, const float *rr,
                        const float *z0, float *out, cudaStream_t stream, float *split_buf, long split_cap,
                        bool pressure) {
    constexpr int LV = 8;
    int nlg = 1;
    while (nlg * LV < nl) nlg *= 2;
    if (nlg > 16) return E_TOO_LARGE;
    if (pressure && !sea.d_tab_gp) return E_NOT_INITIALIZED;
    const int nf = pressure ? 4 : 3;
    PairArgs a{};
    a.ncol = ncol; a.nl = nl; a.nlg = nlg; a.ntile = sea.ntile_g; a.tab = sea.d_tab_grid;
    a.tabp = reinterpret_cast<const float2 *>(sea.d_tab_gp);
    a.ph = ph; a.rr = rr; a.rs = sea.trivial_ramp ? 0 : ncol; a.cf = sea.d_cf; a.cstride = sea.npad_g; a.z0 = z0;
    a.depth = (float)sea.depth; a.out = out; a.first = 1;
    int cols = 128 / nlg;
    // Few columns (a small grid, a column sample): split the tile-pair loop
    // over blockIdx.y so that the launch still fills the GPU, and sum the
    // slices in a fixed order afterwards.
    const long nblk = (ncol + cols - 1) / cols;
    const int ntp = sea.ntile_g * (sea.ntile_g + 1) / 2;
    int nslice = 1;
    a.tp_per = ntp;
    if (split_buf && nblk < SPLIT_TARGET_BLOCKS) {
        int want = (int)std::min<long>(ntp, (SPLIT_TARGET_BLOCKS + nblk - 1) / nblk);
        int per = (ntp + want - 1) / want;
        int ns = (ntp + per - 1) / per;
        if ((long)ns * nf * ncol * nl <= split_cap && ns > 1) {
            nslice = ns;
            a.tp_per = per;
            a.out = split_buf;
        }
    }
    int rc = pressure ? column_pairs_t<true>(a, nblk, nslice, cols, stream)
                      : column_pairs_t<false>(a, nblk, nslice, cols, stream);
    if (rc) return rc;
    if (nslice > 1) {
        long n = (long)nf * ncol * nl;
        k_sum_slices<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(n, nslice, split_buf, out);
        note_launch();
        CK(cudaGetLastError());
    }
    return OK;
}

// ---------------------------------------------------------------------------
// Phase-free part of the s-grid pressure (uvw2, Irregular.cpp:1036-1037 and
// 1076-1077): at the evaluation height z0 in [-h, 0] and time t
//   K(z) = sum_pairs r_i [X px_i(z) px_m(z) + Z pz_i(z) pz_m(z)]
//        + sum_diag  r_i [X px_i(z) + Z pz_i(z)],
// px = cosh(k(z+h))/cosh(kh), pz = sinh(k(z+h))/cosh(kh), rho folded into X, Z.
// K does not depend on the column, so one ring step needs one table of K and
// dK/dz on nz uniform heights (read by cubic Hermite interpolation) instead
// of a second pass over the pairs per node.
// ---------------------------------------------------------------------------
struct KinArgs {
    const float2 *tabk;        // grid-mask pair tiles (X, Z)
    int tt, ntile;             // the table's tiles
    int ncomp, npad, trivial_ramp, zb;
    const double *phase;       // [7][npad]: ramp parameters in rows 4..6
    const float *cf;           // [NCF][npad]
    double t, depth, h, dz;    // heights -h + dz j
    int nz;
    double *kin;               // [nz][2]: K, dK/dz
    const float *tpk;          // point-API products (point_at layout; the diagonal terms are CF_X1, CF_Z1), all
                               // ramps 1, instead of tabk
};

constexpr int KIN_ZB = 4;      // heights per block (upper bound)

__global__ void __launch_bounds__(256) k_pressure_kin(KinArgs a) {
    extern __shared__ float smk[];
    const int np = a.npad, zb = a.zb;
    float *s_k = smk, *s_r = smk + np, *s_px = smk + 2 * np, *s_pz = s_px + (long)zb * np;
    const int j0 = blockIdx.x * zb;
    for (int i = threadIdx.x; i < np; i += blockDim.x) {
        double k = 0.0, r = 0.0;
        if (i < a.ncomp) {
            k = a.cf[CF_K * np + i];
            const int ir = a.trivial_ramp ? 0 : i;
            r = a.tpk ? 1.0 : d_freq_ramp(a.t, a.phase[4 * np + ir], a.phase[5 * np + ir], a.phase[6 * np + ir]);
        }
        s_k[i] = (float)k;
        s_r[i] = (float)r;
        for (int q = 0; q < zb; q++) {
            const double z = fmin(0.0, -a.h + a.dz * min(j0 + q, a.nz - 1));
            // cosh(k(z+h))/cosh(kh) and sinh(k(z+h))/cosh(kh), both bounded by 1
            const double qn = 1.0 / (1.0 + exp(-2.0 * k * a.depth));
            const double E = exp(k * z), Y = exp(-k * (z + 2.0 * a.depth));
            s_px[q * np + i] = (float)(qn * (E + Y));
            s_pz[q * np + i] = (float)(qn * (E - Y));
        }
    }
    __syncthreads();
    float sK[KIN_ZB], cK[KIN_ZB], sD[KIN_ZB], cD[KIN_ZB];
#pragma unroll
    for (int q = 0; q < KIN_ZB; q++) sK[q] = cK[q] = sD[q] = cD[q] = 0.f;
    const int TT = a.tt;
    int I = 0, M = 0;
    const long ntiles = tile_index(a.ntile - 1, a.ntile - 1, a.ntile) + 1;
    for (long t = 0; t < ntiles; t++) {
        for (int e = threadIdx.x; e < TT * TT; e += blockDim.x) {
            const long g = t * (long)TT * TT + e;
            const int i = I * TT + e / TT, m = M * TT + e % TT;
            float2 c;
            if (!a.tpk) c = a.tabk[g];
            else if (i == m) c = make_float2(a.cf[CF_X1 * np + i], a.cf[CF_Z1 * np + i]);
            else c = make_float2(a.tpk[point_at(g, POINTK_NC, 0)], a.tpk[point_at(g, POINTK_NC, 1)]);
            if (c.x == 0.f && c.y == 0.f) continue;     // filtered pair or padding
            const float ri = s_r[i], ki = s_k[i], km = s_k[m];
#pragma unroll
            for (int q = 0; q < KIN_ZB; q++) {
                if (q >= zb) break;
                const float pxi = s_px[q * np + i], pzi = s_pz[q * np + i];
                float v, dv;
                if (i == m) {
                    v = c.x * pxi + c.y * pzi;
                    dv = ki * (c.x * pzi + c.y * pxi);
                } else {
                    const float pxm = s_px[q * np + m], pzm = s_pz[q * np + m];
                    v = c.x * pxi * pxm + c.y * pzi * pzm;
                    dv = c.x * (ki * pzi * pxm + km * pxi * pzm) + c.y * (ki * pxi * pzm + km * pzi * pxm);
                }
                kahan(sK[q], cK[q], ri * v);
                kahan(sD[q], cD[q], ri * dv);
            }
        }
        if (++M == a.ntile) { ++I; M = I; }
    }
    // block reduction in FP64, in a fixed order
    __shared__ double red[2][256];
    for (int q = 0; q < zb; q++) {
        __syncthreads();
        red[0][threadIdx.x] = (double)sK[q] - (double)cK[q];
        red[1][threadIdx.x] = (double)sD[q] - (double)cD[q];
        __syncthreads();
        for (int w = blockDim.x / 2; w > 0; w >>= 1) {
            if ((int)threadIdx.x < w) {
                red[0][threadIdx.x] += red[0][threadIdx.x + w];
                red[1][threadIdx.x] += red[1][threadIdx.x + w];
            }
            __syncthreads();
        }
        if (threadIdx.x == 0 && j0 + q < a.nz) {
            a.kin[2 * (j0 + q)] = red[0][0];
            a.kin[2 * (j0 + q) + 1] = red[1][0];
        }
    }
}

static int pressure_kin(const DevSea &sea, double t, bool point, double h, int nz, double *kin, cudaStream_t stream) {
    const int np = sea.npad_g;
    // shared memory: k, ramp and zb rows of px, pz per component
    const size_t cap = 200 * 1024;
    int zb = KIN_ZB;
    while (zb > 1 && sizeof(float) * (size_t)np * (2 + 2 * zb) > cap) zb--;
    const size_t smem = sizeof(float) * (size_t)np * (2 + 2 * zb);
    if (smem > cap) return E_TOO_LARGE;
    // set once per process (thread-safe static initialisation)
    static const cudaError_t attr = cudaFuncSetAttribute(k_pressure_kin, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap);
    CK(attr);
    KinArgs a;
    a.tabk = reinterpret_cast<const float2 *>(sea.d_tab_gk);
    a.tt = point ? POINT_TILE : GRID_TILE; a.ntile = point ? sea.ntile_p : sea.ntile_g;
    a.ncomp = sea.n; a.npad = np; a.trivial_ramp = sea.trivial_ramp ? 1 : 0; a.zb = zb;
    a.phase = sea.d_phase; a.cf = sea.d_cf;
    a.t = t; a.depth = sea.depth; a.h = h; a.dz = h / (nz - 1); a.nz = nz; a.kin = kin;
    a.tpk = point ? sea.d_tab_pk : nullptr;
    k_pressure_kin<<<(unsigned)((nz + zb - 1) / zb), 256, smem, stream>>>(a);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

int launch_pressure_kin(const DevSea &sea, double t, int nz, double *kin, cudaStream_t stream) {
    if (!sea.d_tab_gk || nz < 2) return E_NOT_INITIALIZED;
    return pressure_kin(sea, t, false, sea.depth, nz, kin, stream);
}

// The height table of the point API's phase-free pressure terms, built with
// the sea where every component has the same ramp (which then multiplies the
// whole sum): over [-h - max(0, swl), 0], the heights that the seabed clamp
// leaves.  The finest wavenumber is 2 kmax; at 2 kmax dz = 0.014 the Hermite
// interpolation's error is (2 kmax dz)^4 / 384 = 1e-10 of a term.  A sea too
// deep for 16385 heights or with too many components for the kernel has no
// table; its products are summed per point.
static int point_kin_build(DevSea &sea, cudaStream_t stream) {
    const double h = sea.depth + std::max(0.0, sea.swl);
    const double want = 2.0 * sea.kmax * h / 0.014 + 1.0;
    if (!sea.trivial_ramp || sea.n < 1 || !(h > 0.0) || !(want <= 16385.0)) return OK;
    const int nz = std::max(2049, (int)std::ceil(want));
    CK(cudaMalloc(&sea.d_kin, sizeof(double) * 2 * nz));
    const int rc = pressure_kin(sea, 0.0, true, h, nz, sea.d_kin, stream);
    if (rc) {
        cudaFree(sea.d_kin);
        sea.d_kin = nullptr;
        return rc == E_TOO_LARGE ? OK : rc;
    }
    sea.kin_nz = nz;
    sea.kin_h = h;
    return OK;
}

// One group of rows (velocity or pressure): the tile-pair walk split into
// slices where the points alone do not fill whole waves of the resident
// blocks, the slices summed in order into out.
template <bool VEL, bool PR, bool KIN>
static int point_pairs_t(PairArgs a, long n, int ntp, float *out, float *split_buf, long split_cap,
                         cudaStream_t stream) {
    using ST = PointStage<VEL, PR, KIN>;
    // set and queried once per process (thread-safe static initialisation)
    static const cudaError_t attr = cudaFuncSetAttribute(k_pairs_points<VEL, PR, KIN>,
                                                         cudaFuncAttributeMaxDynamicSharedMemorySize, ST::SMEM);
    CK(attr);
    static const long slots = [] {
        const long v = resident_slots(k_pairs_points<VEL, PR, KIN>, 128, ST::SMEM);
        return v > 0 ? v : SPLIT_TARGET_BLOCKS;
    }();
    const long nblk = (n + 127) / 128;
    a.tp_per = slice_plan(nblk, ntp, slots, split_buf ? split_cap / (ST::ROWS * n) : 1);
    const int nslice = (ntp + a.tp_per - 1) / a.tp_per;
    a.out = nslice > 1 ? split_buf : out;
    prof_begin(PK_POINT_PAIRS, stream);
    k_pairs_points<VEL, PR, KIN><<<dim3((unsigned)nblk, (unsigned)nslice), 128, ST::SMEM, stream>>>(a);
    note_launch();
    prof_end(PK_POINT_PAIRS, stream);
    CK(cudaGetLastError());
    if (nslice > 1) {
        const long m = ST::ROWS * n;
        k_sum_slices<<<(unsigned)((m + 255) / 256), 256, 0, stream>>>(m, nslice, split_buf, out);
        note_launch();
        CK(cudaGetLastError());
    }
    return OK;
}

// Rows u, v, w (mask bits 2, 4, 8) and p (16) of out [4][n]; rows not asked
// for are not written.  kin: the pressure's phase-free products summed here.
static int launch_point_pairs(const DevSea &sea, long n, const float2 *ph, const float *rr,
                              const double *z, bool clamp, float *out, int pairs, int mask, bool kin, cudaStream_t stream,
                              float *split_buf, long split_cap) {
    PairArgs a{};
    a.ncol = n; a.nl = 1; a.nlg = 1; a.ntile = sea.ntile_p; a.tab = sea.d_tab_point;
    a.tpp = reinterpret_cast<const float4 *>(sea.d_tab_pp);
    a.tpk = reinterpret_cast<const float4 *>(sea.d_tab_pk);
    a.ph = ph; a.rr = rr; a.rs = sea.trivial_ramp ? 0 : n; a.cf = sea.d_cf; a.cstride = sea.npad_g;
    a.z = z; a.swl = sea.swl; a.h = sea.depth; a.order = sea.order; a.clamp = clamp ? 1 : 0;
    a.pairs = pairs; a.first = 1; a.one = 1.f;
    const int ntp = pairs ? sea.ntile_p * (sea.ntile_p + 1) / 2 : sea.ntile_p;
    int rc = OK;
    if (mask & 14) rc = point_pairs_t<true, false, false>(a, n, ntp, out, split_buf, split_cap, stream);
    if (rc == OK && (mask & 16))
        rc = kin && pairs ? point_pairs_t<false, true, true>(a, n, ntp, out + 3 * n, split_buf, split_cap, stream)
                          : point_pairs_t<false, true, false>(a, n, ntp, out + 3 * n, split_buf, split_cap, stream);
    return rc;
}

// The whole evaluation of a few_points() batch.
static int launch_point_few(const DevSea &sea, long n, const double *x, const double *y, const double *z,
                            const double *t, int mask, double *out, bool table, const WsLayout &L,
                            cudaStream_t stream, const ApiRows *api) {
    FewArgs a{};
    a.n = n; a.ldo = n; a.x = x; a.y = y; a.z = z; a.t = t;
    a.swl = sea.swl; a.depth = sea.depth;
    ff_split(-sea.fx, a.ox.x, a.ox.y);
    ff_split(-sea.fy, a.oy.x, a.oy.y);
    a.ncomp = sea.n; a.npad = sea.npad_g; a.cstride = sea.npad_g; a.trivial_ramp = sea.trivial_ramp ? 1 : 0;
    a.order = sea.order; a.clamp = api ? 1 : 0; a.mask = mask;
    a.rec = sea.d_phrec; a.cf = sea.d_cf; a.cfp = sea.d_cfp; a.phase = sea.d_phase;
    a.ntp = sea.ntile_p; a.ntg = sea.ntile_g;
    a.tabv = sea.d_tab_point; a.tpp = sea.d_tab_pp; a.tpk = sea.d_tab_pk; a.tabe = sea.d_tab_eta;
    const bool pairs = sea.order == 2;
    a.kin = pairs && (mask & 16) && !table ? 1 : 0;
    const long tp = (long)sea.ntile_p * (sea.ntile_p + 1) / 2, tg = (long)sea.ntile_g * (sea.ntile_g + 1) / 2;
    const long ip = tp * POINT_TILE * POINT_TILE / FEW_E;
    a.nv = pairs && (mask & 14) ? ip : 0;
    a.np = pairs && (mask & 16) ? ip : 0;
    a.ne = pairs && (mask & 1) ? tg * GRID_TILE * GRID_TILE / FEW_E : 0;
    a.part = reinterpret_cast<float2 *>(L.split); a.out = out;
    if (api) a.api = *api;
    if (table) a.kt = KinTab{sea.d_kin, sea.kin_nz, sea.kin_h, sea.depth, nullptr};
    // as many slices as give every thread one item or component, up to about eight blocks an SM in all
    const long want = std::max<long>(1, (a.nv + a.np + a.ne + a.ncomp + FEW_T - 1) / FEW_T);
    const long cap = std::max<long>(1, 2 * SPLIT_TARGET_BLOCKS / n);
    const long ns = std::min(std::min(want, cap), std::max<long>(1, L.split_cap / (2 * FEW_Q * n)));
    const size_t smem = sizeof(float2) * (size_t)a.npad * (a.kin ? 2 : 1) + (sea.trivial_ramp ? 0 : sizeof(float) * a.npad);
    // set once per process (thread-safe static initialisation)
    static const cudaError_t attr = cudaFuncSetAttribute(k_point_few, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                         FEW_MAX_NPAD * 20);
    CK(attr);
    prof_begin(PK_POINT_PAIRS, stream);
    k_point_few<<<dim3((unsigned)n, (unsigned)ns), FEW_T, smem, stream>>>(a);
    note_launch();
    CK(cudaGetLastError());
    if (ns > 1) {
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3((unsigned)n);
        c.blockDim = dim3(FEW_T);
        c.stream = stream;
        c.attrs = &at;
        c.numAttrs = 1;
        CK(cudaLaunchKernelEx(&c, k_few_finish, a, (int)ns));
        note_launch();
    }
    prof_end(PK_POINT_PAIRS, stream);
    return OK;
}

// Phasor layout used by the pair kernels: the point kernel reads tiles of
// POINT_TILE, the grid kernels tiles of GRID_TILE; the workspace is sized for
// npad_g >= npad_p so both fit.
int irregular_eval(const DevSea &sea, long n, const double *x, const double *y, const double *z,
                   const double *t, int mask, double *out, Workspace &ws, void *stream_, const ApiRows *api) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (n <= 0) return OK;
    const long chunk = 1L << 18;
    const int npad = sea.npad_g;
    // the phase-free part of the pressure from the height table: the wave_*
    // calls clamp z to the range it covers
    const bool table = api && sea.d_kin && sea.order == 2;
    WsLayout L0 = layout(std::min(n, chunk), npad, nullptr);
    int rc = workspace_reserve(ws, L0.bytes);
    if (rc) return rc;
    if (few_points(n, npad) && !(sea.smit && (mask & 30)))
        return launch_point_few(sea, n, x, y, z, t, mask, out, table, layout(n, npad, ws.base), stream, api);
    for (long b = 0; b < n; b += chunk) {
        long m = std::min(chunk, n - b);
        WsLayout L = layout(m, npad, ws.base);
        // vertical_theory smit: u, v, w, dp need eta at the point first
        const bool smit = sea.smit && (mask & 30);
        // the first-order sums behind the rows asked for (the mask's bits are
        // those of first)
        rc = launch_phasors(sea, m, x + b, y + b, t + b, 1, 1, 1, npad, L.ph, L.rr, L.first, stream,
                            smit ? 1 : mask & 31);
        if (rc) return rc;
        float *eta2 = nullptr;
        if (((mask & 1) || smit) && sea.order == 2) {
            eta2 = L.sec + 4 * m;
            rc = launch_eta_pairs(sea, m, L.ph, L.rr, eta2, stream, L.split, L.split_cap);
            if (rc) return rc;
        }
        if (smit) {
            rc = smit_eval(sea, m, z + b, L.ph, L.rr, L.first, eta2, L.sec, L.split, L.split_cap, n, out + b,
                           mask, stream);
            if (rc) return rc;
        } else if (mask & 30) {
            // the point table is padded to POINT_TILE; the phasor rows beyond
            // npad_p are never read by the point kernel
            rc = launch_point_pairs(sea, m, L.ph, L.rr, z + b, api != nullptr, L.sec, sea.order != 0 ? 1 : 0, mask, !table, stream,
                                    L.split, L.split_cap);
            if (rc) return rc;
        }
        ApiRows ar{};
        if (api && !smit) {
            ar = *api;
            ar.x = api->x + b; ar.y = api->y + b; ar.t = api->t + b;
            for (int q = 0; q < 6; q++) ar.row[q] = api->row[q] ? api->row[q] + b : nullptr;
            ar.kin = api->kin ? api->kin + 4 * b : nullptr;
        }
        k_combine<<<(unsigned)((m + 255) / 256), 256, 0, stream>>>(m, n, sea.order, sea.swl, z + b,
                                                                   L.first, L.sec, eta2, smit ? (mask & 1) : mask,
                                                                   out ? out + b : nullptr, ar,
                                                                   KinTab{table && !smit ? sea.d_kin : nullptr,
                                                                          sea.kin_nz, sea.kin_h, sea.depth, L.rr});
        note_launch();
        CK(cudaGetLastError());
    }
    return OK;
}

size_t irregular_eval_scratch_bytes(const DevSea &sea, long n) {
    const long chunk = 1L << 18;
    return layout(std::min(n, chunk), sea.npad_g, nullptr).bytes;
}

}  // namespace cfdwm
