// Lagrangian stretched s-grid with 4-D cubic-Hermite query, on the GPU.
//
// Behaviour follows the reference's lsGridSpline (oystelan/CFDwavemaker
// v3.1.0, src/lsgrid_spline.cpp):
//   storage and ring of 4 time slots     :35-61, 847-931
//   sigma maps z2s/s2z/cart2sigmaS/...   :91-122
//   column body (eta, levels, uvw2)      :695-720, 880-903
//   finite-difference gradients          :124-366
//   spline query                         :368-605
//
// GB300 design: the whole grid lives in one device allocation (FP32 fields in
// the reference's [slot][i][j][m] layout), so the reference's MPI column
// partition and MPI_Allgatherv disappear.  A ring step is
//   phasors of the active columns  ->  eta2 pair sums  ->  level heights
//   ->  column pair sums (u, v, w at all levels of a column in registers)
//   ->  scatter into the slot  ->  one fused finite-difference pass.
// The query kernel gathers the 2x2(x2) stencils of the two bracketing slots
// and reduces x -> y -> s -> t exactly in the reference's order.
#include "cfdwm.h"
#include "sgrid_geom.cuh"
#include "ffmath.cuh"
#include "ramp.cuh"

#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstdio>
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

// launchers shared with irregular.cu
int launch_eta_pairs(const DevSea &sea, long n, const float2 *ph, const float *rr, float *out,
                     cudaStream_t stream, float *split_buf, long split_cap);
int launch_column_pairs(const DevSea &sea, long ncol, int nl, const float2 *ph, const float *rr,
                        const float *z0, float *out, cudaStream_t stream, float *split_buf, long split_cap,
                        bool pressure);
long column_pairs_split_floats(int nl);
int launch_pressure_kin(const DevSea &sea, double t, int nz, double *kin, cudaStream_t stream);

// heights of the table of the phase-free pressure terms over [-h, 0]
constexpr int KIN_NZ = 2049;
int launch_phasors_public(const DevSea &sea, long n, const double *x, const double *y,
                          const double *t, long sx, long sy, long st, int npad, float2 *ph,
                          float *rr, double *first, cudaStream_t stream);

__global__ void k_column_coords(GridGeom g, long nact, const int *act, double *xy) {
    long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (q >= nact) return;
    int c = act[q], i = c / g.ny, j = c % g.ny;
    xy[q] = g.d0 + g.dx * i;
    xy[nact + q] = g.d2 + g.dy * j;
}

// ETA of the slot, the level heights and the level offsets above swl.
// blockDim 128; the stretched coordinate of each level (which depends on the
// level only) is formed once per block
__global__ void k_levels(GridGeom g, long nact, const int *act, const double *sig, const double *first,
                         const float *eta2, int slot, float *ETA, float *zmin, float *zmax) {
    long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (q >= nact) return;
    int c = act[q];
    double e = first[q] + (double)eta2[q] + g.swl;     // eta1 + eta2 + swl
    float ef = (float)e;
    ETA[(long)slot * g.nx * g.ny + c] = ef;
    for (int m = 0; m < g.nl; m++) {
        // the reference evaluates the levels from the stored value; the FP32
        // store is the value the query sees, so use it here too
        double z = d_s2z(g, sig[m], (double)ef);
        zmin[q * g.nl + m] = (float)fmin(0.0, z);
        zmax[q * g.nl + m] = (float)fmax(0.0, z - g.swl);
    }
}

// The level sums into the slot, with the Taylor terms above swl
// (lsgrid_spline.cpp:892-897).  With UP: the dynamic pressure
//   dp1(z0) + rho uvw2.p(z0) + dp1_dz max(0, z - swl),
// the phase-free part of uvw2.p from the height table kin (cubic Hermite).
__global__ void k_scatter_levels(GridGeom g, long nact, const int *act, const double *first,
                                 const float *sec, const float *zmin, const float *zmax, int slot,
                                 float *UX, float *UY, float *UZ, float *UP, const double *kin, int nkz) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    long tot = nact * g.nl;
    if (e >= tot) return;
    long q = e / g.nl;
    int m = (int)(e % g.nl);
    long c = act[q];
    float za = zmax[e];
    long o = (long)slot * g.nx * g.ny * g.nl + c * g.nl + m;
    UX[o] = sec[0 * tot + e] + (float)first[1 * nact + q] * za;
    UY[o] = sec[1 * tot + e] + (float)first[2 * nact + q] * za;
    UZ[o] = sec[2 * tot + e] + (float)first[3 * nact + q] * za;
    if (UP) {
        const double dz = g.depth / (nkz - 1);
        double t = ((double)zmin[e] + g.depth) / dz;
        t = fmin(fmax(t, 0.0), (double)(nkz - 1));
        int i = min((int)t, nkz - 2);
        double r = t - i;
        double f0 = kin[2 * i], f1 = kin[2 * i + 2], d0 = kin[2 * i + 1], d1 = kin[2 * i + 3];
        double a = dz * d0 - (f1 - f0), b = -dz * d1 + (f1 - f0);
        double K = f0 * (1.0 - r) + f1 * r + r * (1.0 - r) * (a * (1.0 - r) + b * r);
        UP[o] = (float)((double)sec[3 * tot + e] + K) + (float)first[4 * nact + q] * za;
    }
}

// Floats of a query-image record: U, U_t, U_x, U_y, U_s of a node, each over
// the fields; 15 values in 64 bytes with three fields, 20 in 80 with the
// pressure.
template <int NF> struct QRec { static constexpr int F = NF == 3 ? 16 : 20, F4 = F / 4; };

// All finite differences of lsgrid_spline.cpp:124-366 and the query image in
// one pass over the nodes: x/y/s gradients of slots (tstep+1)%4, (tstep+2)%4
// into gradient slots 0/1, the time gradient of the slot(s) the reference
// writes, and, per node of those two slots, the record that the queries read
// (per column the elevation's: eta, eta_t, eta_x, eta_y).  The records are
// staged in shared memory so that they are written whole and coalesced; the
// image kernel that came after this one read all the gradients back (256 x 256
// x 16 ring: 49 + 61 us as two kernels).
struct GradArgs {
    GridGeom g;
    int tstep;
    const float *F[5];      // ETA, UX, UY, UZ (and the pressure)
    float *Fx[5], *Fy[5], *Fs[5], *Ft[5];
    float rdx, rdy, rds, rdt;   // reciprocal spacings
    float4 *img;            // [2][nodes] records
    float4 *eimg;           // [2][columns] elevation records
};

constexpr int GRAD_B = 128;

// FP32 differences of the FP32 node values times the reciprocal spacings
// (one-sided at the boundaries, central inside)
__device__ __forceinline__ float fd(const float *d, long e, long s, int i, int n, float r) {
    if (n == 1) return 0.f;
    if (i == 0) return (d[e + s] - d[e]) * r;
    if (i == n - 1) return (d[e] - d[e - s]) * r;
    return (d[e + s] - d[e - s]) * (0.5f * r);
}

// time gradients of element e of one field (stride S between slots); returns
// those of the two slots the image holds
__device__ __forceinline__ float2 fd_time(const GradArgs &a, const float *D, float *T, long S, long e) {
    if (a.tstep > 0) {
        const int tid = (a.tstep + 2) % 4, tid1 = (a.tstep + 3) % 4, tid0 = (a.tstep + 1) % 4;
        const float v = (D[tid1 * S + e] - D[tid0 * S + e]) * (0.5f * a.rdt);
        T[tid * S + e] = v;
        return make_float2(T[tid0 * S + e], v);
    }
    const float v1 = (D[2 * S + e] - D[1 * S + e]) * a.rdt;
    const float v2 = (D[3 * S + e] - D[1 * S + e]) * (0.5f * a.rdt);
    T[1 * S + e] = v1;
    T[2 * S + e] = v2;
    return make_float2(v1, v2);
}

template <int NF>
__global__ void __launch_bounds__(GRAD_B) k_gradients(GradArgs a) {
    constexpr int RF = QRec<NF>::F, R4 = QRec<NF>::F4;
    __shared__ float s_rec[GRAD_B][RF + 1];
    const GridGeom &g = a.g;
    const long S = (long)g.nx * g.ny * g.nl, cols = (long)g.nx * g.ny;
    const long e0 = blockIdx.x * (long)GRAD_B, e = e0 + threadIdx.x;
    const bool on = e < S;
    const long ec = on ? e : 0;
    const int m = (int)(ec % g.nl);
    const long c = ec / g.nl;
    const int i = (int)(c / g.ny), j = (int)(c % g.ny);
    const long sx = (long)g.ny * g.nl, sy = g.nl;
    const int slot[2] = {(a.tstep + 1) % 4, (a.tstep + 2) % 4};
    if (on && m == 0) {
        const float2 t = fd_time(a, a.F[0], a.Ft[0], cols, c);
        for (int q = 0; q < 2; q++) {
            const float *d = a.F[0] + slot[q] * cols;
            const float gx = fd(d, c, g.ny, i, g.nx, a.rdx), gy = fd(d, c, 1, j, g.ny, a.rdy);
            a.Fx[0][q * cols + c] = gx;
            a.Fy[0][q * cols + c] = gy;
            a.eimg[q * cols + c] = make_float4(d[c], q == 0 ? t.x : t.y, gx, gy);
        }
    }
    float2 t[NF];
    if (on)
#pragma unroll
        for (int f = 0; f < NF; f++) t[f] = fd_time(a, a.F[f + 1], a.Ft[f + 1], S, e);
    for (int q = 0; q < 2; q++) {
        if (on) {
            float *r = s_rec[threadIdx.x];
#pragma unroll
            for (int f = 0; f < NF; f++) {
                const float *d = a.F[f + 1] + slot[q] * S;
                const float gx = fd(d, e, sx, i, g.nx, a.rdx), gy = fd(d, e, sy, j, g.ny, a.rdy);
                const float gs = fd(d, e, 1, m, g.nl, a.rds);
                a.Fx[f + 1][q * S + e] = gx;
                a.Fy[f + 1][q * S + e] = gy;
                a.Fs[f + 1][q * S + e] = gs;
                r[f] = d[e];
                r[NF + f] = q == 0 ? t[f].x : t[f].y;
                r[2 * NF + f] = gx;
                r[3 * NF + f] = gy;
                r[4 * NF + f] = gs;
            }
            if (NF == 3) r[15] = 0.f;
        }
        __syncthreads();
        const long nrec = S - e0 < GRAD_B ? S - e0 : GRAD_B;
        float4 *o = a.img + ((long)q * S + e0) * R4;
        for (int k = threadIdx.x; k < nrec * R4; k += GRAD_B) {
            const float *r = s_rec[k / R4] + 4 * (k % R4);
            o[k] = make_float4(r[0], r[1], r[2], r[3]);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Query
// ---------------------------------------------------------------------------
struct QueryArgs {
    GridGeom g;
    double t0;
    const float4 *eimg;     // [2][columns]: eta, eta_t, eta_x, eta_y
    const float4 *img;      // [2][nodes] records (QRec)
    long n;
    const double *z;
    ApiRows api;    // x, y, t of the queries and the rows and records to write
    double inv_dx, inv_dy, inv_dt;   // reciprocals of the spacings (host-computed)
    float tanab;                     // tan(a)^b of the stretching
};

__device__ __forceinline__ float herm(float f0, float f1, float d0, float d1, float h, float r) {
    float a = h * d0 - (f1 - f0), b = -h * d1 + (f1 - f0);
    return f0 * (1.f - r) + f1 * r + r * (1.f - r) * (a * (1.f - r) + b * r);
}
__device__ __forceinline__ float lin(float f0, float f1, float r) { return f0 * (1.f - r) + f1 * r; }

// cart2sigmaS (lsgrid_spline.cpp:109-113).  The reference takes pow() of a
// negative base (NaN, then an out-of-range index) for eta - swl < z <= eta
// when swl != 0; here the base is clamped at zero, i.e. such points are
// evaluated at the surface level.
__device__ __forceinline__ float cart2sigmaS(const GridGeom &g, float tanab, float zpt, float e) {
    float z = fminf(zpt, e);
    float es = e - (float)g.swl;
    float sigma = fmaxf((z - es) / ((float)g.depth + es), -1.f);
    float base = fmaxf(-sigma * tanab, 0.f);
    return 1.f - atanf(powf(base, 1.f / (float)g.tan_b)) / (float)g.tan_a;
}

__device__ __forceinline__ int iclamp(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ void q_cp16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void q_cp_wait() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// A query reads, in each of the two bracketing slots and at each of the four
// columns around it, the records of two neighbouring levels: 128 (with the
// pressure 160) contiguous bytes.  A warp fetches these blocks for its 32
// queries together, 16 bytes a lane and neighbouring lanes on neighbouring
// addresses, into shared memory, two columns (the x pair) at a time; each
// lane then reads its own from there.  With every lane loading its own
// records 16 bytes at a time each load instruction touched 32 cache lines, and
// the L1's line lookups were the bound (88 % busy).  1e6 random queries of the
// 256 x 256 x 16 ring, the whole wave_Kinematics call: 0.35 ms then, 0.19 ms
// with the warp's fetch and 64-byte records (and the seabed clamp, the ramp
// and the rows in this kernel).  Registers are held to four blocks an SM: 0.20
// ms without the limit (144 registers), 0.22 with five, 0.28 with six.
constexpr int QB = 128;      // threads of a query block
template <int NF> struct QStage {
    static constexpr int PAIR = 4 * QRec<NF>::F4;     // float4 of the x pair's two blocks
    static constexpr int STRIDE = PAIR + 1;           // per query: lanes' 16-byte reads fall on distinct banks
};

template <int NF>
__global__ void __launch_bounds__(QB, NF == 3 ? 4 : 3) k_query(QueryArgs a) {
    constexpr int RF = QRec<NF>::F, R4 = QRec<NF>::F4, PAIR = QStage<NF>::PAIR, STRIDE = QStage<NF>::STRIDE;
    extern __shared__ float4 s_q[];
    const int lane = threadIdx.x & 31;
    float4 *sw = s_q + (threadIdx.x >> 5) * 32 * STRIDE;     // this warp's stage
    const long p0 = blockIdx.x * (long)QB + threadIdx.x;
    const long p = p0 < a.n ? p0 : a.n - 1;                  // (idle lanes help with the loads)
    const GridGeom &g = a.g;
    const double xpt = a.api.x[p], ypt = a.api.y[p], tpt = a.api.t[p];
    // std::modf with a float* argument selects the float overload in the
    // reference (lsgrid_spline.cpp:515-520): the fractions are float.
    float xi, yi;
    // (FP64 divisions per query replaced by products with the reciprocals:
    // FP64 runs at a small fraction of the FP32 rate on this GPU)
    float xd = modff((float)fmax(0.0, fmin((xpt - g.d0) * a.inv_dx, g.nx - 1.0)), &xi);
    float yd = modff((float)fmax(0.0, fmin((ypt - g.d2) * a.inv_dy, g.ny - 1.0)), &yi);
    float td = (float)fmin(1.0, fmax(0.0, (tpt - a.t0) * a.inv_dt));
    int xp = (int)xi, yp = (int)yi;
    const long nc = (long)g.nx * g.ny;
    const int x1 = iclamp(xp + 1, 0, g.nx - 1), y1 = iclamp(yp + 1, 0, g.ny - 1);
    const long cid[4] = {(long)xp * g.ny + yp, (long)xp * g.ny + y1, (long)x1 * g.ny + yp, (long)x1 * g.ny + y1};
    float4 C[4], D[4];       // eta, eta_t, eta_x, eta_y of the two slots
#pragma unroll
    for (int k = 0; k < 4; k++) {
        C[k] = __ldg(a.eimg + cid[k]);
        D[k] = __ldg(a.eimg + nc + cid[k]);
    }
    const float dx = (float)g.dx, dy = (float)g.dy;
    float C0 = herm(C[0].x, C[2].x, C[0].z, C[2].z, dx, xd), C1 = herm(C[1].x, C[3].x, C[1].z, C[3].z, dx, xd);
    float D0 = herm(D[0].x, D[2].x, D[0].z, D[2].z, dx, xd), D1 = herm(D[1].x, D[3].x, D[1].z, D[3].z, dx, xd);
    float C0y = lin(C[0].w, C[2].w, xd), C1y = lin(C[1].w, C[3].w, xd);
    float D0y = lin(D[0].w, D[2].w, xd), D1y = lin(D[1].w, D[3].w, xd);
    float C0t = lin(C[0].y, C[2].y, xd), C1t = lin(C[1].y, C[3].y, xd);
    float D0t = lin(D[0].y, D[2].y, xd), D1t = lin(D[1].y, D[3].y, xd);
    float e0 = herm(C0, C1, C0y, C1y, dy, yd), e1 = herm(D0, D1, D0y, D1y, dy, yd);
    float CCt = lin(C0t, C1t, yd), DDt = lin(D0t, D1t, yd);
    float eta = herm(e0, e1, CCt, DDt, (float)g.dt, td);
    // get_kinematics_at_point forms eta before it looks at z
    // (lsgrid_spline.cpp:505-571): one query serves wave_SurfElev (queried at
    // z = 0) and the velocities (queried at z clamped to the seabed).  Without
    // a pressure field rows 4 and 5 are the reference's 0.0
    // (CFDwavemaker.cpp:1808-1812, 1815-1891); with one, the irregular sea's
    // forms (:1807-1808, 1826-1830) on the grid.
    const ApiRows &A = a.api;
    double v[6] = {d_from_float(eta), 0.0, 0.0, 0.0, 0.0, 0.0};
    if (A.row[1] || A.row[2] || A.row[3] || A.kin || (NF == 4 && (A.row[4] || A.row[5]))) {
        // spline_interp_velo (lsgrid_spline.cpp:386-502) of every field, the
        // reductions x -> y -> s -> t in the reference's order
        const float zpt = (float)fmax(-g.depth, a.z[p]);
        float s0i, s1i;
        const float sd0 = modff(cart2sigmaS(g, a.tanab, zpt, e0) / (float)g.ds, &s0i);
        const float sd1 = modff(cart2sigmaS(g, a.tanab, zpt, e1) / (float)g.ds, &s1i);
        const int ls[2] = {iclamp((int)s0i, 0, g.nl - 1), iclamp((int)s1i, 0, g.nl - 1)};
        const unsigned nn = (unsigned)(nc * g.nl);
        const float ds = (float)g.ds;
        float red[2][NF], redt[2][NF];
#pragma unroll
        for (int q = 0; q < 2; q++) {        // q = 0: slot (tstep+1)%4 at s0; q = 1: slot (tstep+2)%4 at s1
            // the block's first level, and the two levels' records within it
            const int lb = g.nl > 1 ? min(ls[q], g.nl - 2) : 0;
            const int i0 = ls[q] - lb, i1 = iclamp(ls[q] + 1, 0, g.nl - 1) - lb;
            const float4 *img = a.img + (long)q * nn * R4;
            float vv[2][NF], yv[2][NF], tv[2][NF], sv[2][NF];    // [level]: at yp, then reduced in y
#pragma unroll
            for (int yy = 0; yy < 2; yy++) {
                const unsigned nb0 = (unsigned)(cid[yy] * g.nl) + lb, nb1 = (unsigned)(cid[2 + yy] * g.nl) + lb;
                __syncwarp();                                    // the stage has been read
#pragma unroll
                for (int it = 0; it < PAIR; it++) {
                    const int e = it * 32 + lane, qq = e / PAIR, r = e % PAIR;
                    const unsigned a0 = __shfl_sync(0xffffffffu, nb0, qq), a1 = __shfl_sync(0xffffffffu, nb1, qq);
                    int k = r < PAIR / 2 ? r : r - PAIR / 2;
                    if (g.nl == 1 && k >= R4) k -= R4;           // one level: its record twice
                    q_cp16(sw + qq * STRIDE + r, img + (long)(r < PAIR / 2 ? a0 : a1) * R4 + k);
                }
                q_cp_wait();
                __syncwarp();
                const float4 *mine = sw + lane * STRIDE;
#pragma unroll
                for (int l = 0; l < 2; l++) {
                    const float4 *ra = mine + (l == 0 ? i0 : i1) * R4, *rb = ra + PAIR / 2;
                    float fa[RF], fb[RF];
#pragma unroll
                    for (int k = 0; k < R4; k++) {
                        const float4 u = ra[k], w = rb[k];
                        fa[4 * k] = u.x; fa[4 * k + 1] = u.y; fa[4 * k + 2] = u.z; fa[4 * k + 3] = u.w;
                        fb[4 * k] = w.x; fb[4 * k + 1] = w.y; fb[4 * k + 2] = w.z; fb[4 * k + 3] = w.w;
                    }
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        const float hv = herm(fa[f], fb[f], fa[2 * NF + f], fb[2 * NF + f], dx, xd);
                        const float ht = lin(fa[NF + f], fb[NF + f], xd);
                        const float hy = lin(fa[3 * NF + f], fb[3 * NF + f], xd);
                        const float hs = lin(fa[4 * NF + f], fb[4 * NF + f], xd);
                        if (yy == 0) {
                            vv[l][f] = hv; tv[l][f] = ht; yv[l][f] = hy; sv[l][f] = hs;
                        } else {
                            vv[l][f] = herm(vv[l][f], hv, yv[l][f], hy, dy, yd);
                            sv[l][f] = lin(sv[l][f], hs, yd);
                            tv[l][f] = lin(tv[l][f], ht, yd);
                        }
                    }
                }
            }
            const float sd = q == 0 ? sd0 : sd1;
#pragma unroll
            for (int f = 0; f < NF; f++) {
                red[q][f] = herm(vv[0][f], vv[1][f], sv[0][f], sv[1][f], ds, sd);
                redt[q][f] = lin(tv[0][f], tv[1][f], sd);
            }
        }
#pragma unroll
        for (int f = 0; f < NF; f++)
            v[1 + f] = d_from_float(herm(red[0][f], red[1][f], redt[0][f], redt[1][f], (float)g.dt, td));
        if (NF == 4 && A.row[5]) v[5] = v[4] - A.rho * A.g * v[0];
    }
    if (p0 < a.n) api_store(A, p, v);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static GridGeom geom(const DevGrid &g) {
    GridGeom G;
    G.nx = g.nx; G.ny = g.ny; G.nl = g.nl;
    G.d0 = g.cfg.domain[0]; G.d2 = g.cfg.domain[2];
    G.dx = g.dx; G.dy = g.dy; G.ds = g.ds; G.depth = g.depth; G.swl = g.swl;
    G.tan_a = g.cfg.tan_a; G.tan_b = g.cfg.tan_b; G.dt = g.dt;
    return G;
}

// Extra per-grid device scratch kept alongside DevGrid (keyed by the grid).
struct GridExtra {
    int *act_all = nullptr, *act_live = nullptr;
    long n_all = 0, n_live = 0;
    double *xy = nullptr;      // [2][ncol]
    float *zmin = nullptr, *zmax = nullptr, *sec = nullptr;
    float *eta2 = nullptr;
    double *sig = nullptr;     // stretched coordinate of each level
    double *tdev = nullptr;    // the slot time, read with stride 0 by the phasor pass
    float *split = nullptr;    // slices of a split column-pair launch
    long split_cap = 0;
    double *kin = nullptr;     // [KIN_NZ][2] phase-free pressure terms of the slot being written
    // the table depends on t only through the component ramps: the ramps it
    // was built with, and the ramp parameters (ramptime, starttime, duration)
    std::vector<double> kin_r, ramp_par;
    bool kin_valid = false;
    DepthForm df;              // tensor-core form of the column sums (method 1)
    // live columns before row i (act_live is ascending in i ny + j):
    // the live columns of rows [i0, i1) are act_live[row_live[i0] .. row_live[i1])
    std::vector<long> row_live;
};
static std::vector<std::pair<const DevGrid *, GridExtra>> g_extra;
static GridExtra *extra(const DevGrid &g) {
    for (auto &e : g_extra) if (e.first == &g) return &e.second;
    g_extra.push_back({&g, GridExtra{}});
    return &g_extra.back().second;
}

int grid_create(const Config &cfg, DevGrid &g, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    grid_free(g);
    g.cfg = cfg.lsgrid;
    g.nx = cfg.lsgrid.nx; g.ny = cfg.lsgrid.ny; g.nl = cfg.lsgrid.nl;
    if (g.nx < 1 || g.ny < 1 || g.nl < 1) return E_BAD_ARGUMENT;
    if (g.nl > 128) return E_TOO_LARGE;
    // initialize_kinematics (lsgrid_spline.cpp:673-677) and set_ignore (:1406)
    g.dx = (g.cfg.domain[1] - g.cfg.domain[0]) / std::max(1., double(g.nx - 1));
    g.dy = (g.cfg.domain[3] - g.cfg.domain[2]) / std::max(1., double(g.ny - 1));
    g.ds = 1. / std::max(1., double(g.nl - 1));
    g.t0 = g.cfg.t0; g.dt = g.cfg.dt; g.depth = cfg.depth; g.swl = cfg.swl; g.tstep = 0;
    long c = (long)g.nx * g.ny, v = c * g.nl;
    CK(cudaMalloc(&g.ETA, sizeof(float) * 4 * c));
    CK(cudaMalloc(&g.ETAdt, sizeof(float) * 4 * c));
    CK(cudaMalloc(&g.ETAdx, sizeof(float) * 2 * c));
    CK(cudaMalloc(&g.ETAdy, sizeof(float) * 2 * c));
    CK(cudaMemsetAsync(g.ETA, 0, sizeof(float) * 4 * c, stream));
    CK(cudaMemsetAsync(g.ETAdt, 0, sizeof(float) * 4 * c, stream));
    for (int f = 0; f < 3; f++) {
        CK(cudaMalloc(&g.U[f], sizeof(float) * 4 * v));
        CK(cudaMalloc(&g.Ut[f], sizeof(float) * 4 * v));
        CK(cudaMalloc(&g.Ux[f], sizeof(float) * 2 * v));
        CK(cudaMalloc(&g.Uy[f], sizeof(float) * 2 * v));
        CK(cudaMalloc(&g.Us[f], sizeof(float) * 2 * v));
        CK(cudaMemsetAsync(g.U[f], 0, sizeof(float) * 4 * v, stream));
        CK(cudaMemsetAsync(g.Ut[f], 0, sizeof(float) * 4 * v, stream));
    }
    std::vector<int> ign(c), all, live;
    GridExtra *xr = extra(g);
    xr->row_live.assign(g.nx + 1, 0);
    for (int i = 0; i < g.nx; i++) {
        xr->row_live[i] = (long)live.size();
        double xp = g.cfg.domain[0] + g.dx * i;
        for (int j = 0; j < g.ny; j++) {
            double yp = g.cfg.domain[2] + g.dy * j;
            const double *di = g.cfg.domain_ignore;
            int ig = (xp >= di[0] && xp <= di[1] && yp >= di[2] && yp <= di[3]) ? 1 : 0;
            ign[(long)i * g.ny + j] = ig;
            all.push_back(i * g.ny + j);
            if (!ig) live.push_back(i * g.ny + j);
        }
    }
    xr->row_live[g.nx] = (long)live.size();
    CK(cudaMalloc(&g.IGNORE, sizeof(int) * c));
    CK(cudaMemcpyAsync(g.IGNORE, ign.data(), sizeof(int) * c, cudaMemcpyHostToDevice, stream));
    GridExtra *x = extra(g);
    x->n_all = (long)all.size();
    x->n_live = (long)live.size();
    CK(cudaMalloc(&x->act_all, sizeof(int) * std::max<long>(1, x->n_all)));
    CK(cudaMalloc(&x->act_live, sizeof(int) * std::max<long>(1, x->n_live)));
    CK(cudaMemcpyAsync(x->act_all, all.data(), sizeof(int) * x->n_all, cudaMemcpyHostToDevice, stream));
    if (x->n_live)
        CK(cudaMemcpyAsync(x->act_live, live.data(), sizeof(int) * x->n_live, cudaMemcpyHostToDevice, stream));
    CK(cudaMalloc(&x->xy, sizeof(double) * 2 * c));
    CK(cudaMalloc(&x->zmin, sizeof(float) * v));
    CK(cudaMalloc(&x->zmax, sizeof(float) * v));
    CK(cudaMalloc(&x->sec, sizeof(float) * 4 * v));
    CK(cudaMalloc(&x->eta2, sizeof(float) * c));
    CK(cudaMalloc(&x->tdev, sizeof(double)));
    CK(cudaMalloc(&x->sig, sizeof(double) * g.nl));
    int rc = grid_sigma_table(geom(g), x->sig, stream);
    if (!rc) rc = first_order_load();
    if (rc) return rc;
    x->split_cap = column_pairs_split_floats(g.nl);
    CK(cudaMalloc(&x->split, sizeof(float) * x->split_cap));
    CK(cudaMalloc(&g.QIMG, sizeof(float4) * 10 * v));
    CK(cudaMalloc(&g.EIMG, sizeof(float4) * 2 * c));
    CK(cudaStreamSynchronize(stream));
    return OK;
}

void grid_free(DevGrid &g) {
    float *ptrs[] = {g.ETA, g.ETAdx, g.ETAdy, g.ETAdt};
    for (float *p : ptrs) if (p) cudaFree(p);
    for (int f = 0; f < 4; f++) {
        float *q[] = {g.U[f], g.Ut[f], g.Ux[f], g.Uy[f], g.Us[f]};
        for (float *p : q) if (p) cudaFree(p);
        g.U[f] = g.Ut[f] = g.Ux[f] = g.Uy[f] = g.Us[f] = nullptr;
    }
    g.nf = 3;
    if (g.IGNORE) cudaFree(g.IGNORE);
    if (g.QIMG) cudaFree(g.QIMG);
    if (g.EIMG) cudaFree(g.EIMG);
    g.ETA = g.ETAdx = g.ETAdy = g.ETAdt = nullptr;
    g.IGNORE = nullptr;
    g.QIMG = nullptr;
    g.EIMG = nullptr;
    for (auto it = g_extra.begin(); it != g_extra.end(); ++it)
        if (it->first == &g) {
            GridExtra &x = it->second;
            void *q[] = {x.act_all, x.act_live, x.xy, x.zmin, x.zmax, x.sec, x.eta2, x.sig, x.tdev, x.split, x.kin};
            for (void *p : q) if (p) cudaFree(p);
            depthform_free(x.df);
            g_extra.erase(it);
            break;
        }
}

// Workspace of a fill.  Plain: phasors [npad][nact], ramps [npad][nact],
// first-order sums [5][nact]; tensor-core: phasor tables and the first-order sums.
struct FillBytes {
    size_t ph, rr, all;
};
static FillBytes fill_bytes(DevGrid &g, const DevSea &sea, long nact) {
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const bool tc = g.method == 1 && extra(g)->df.built;
    FillBytes b;
    b.ph = up(tc ? grid_tab_bytes(sea, g.nx, g.ny) : sizeof(float2) * (size_t)sea.npad_g * nact);
    b.rr = tc ? 0 : up(sizeof(float) * (size_t)sea.npad_g * nact);
    b.all = b.ph + b.rr + sizeof(double) * 5 * nact;
    return b;
}
size_t grid_fill_bytes(DevGrid &g, const DevSea &sea, long nact) { return fill_bytes(g, sea, nact).all; }

// Plain second-order fill of the columns act[0..nact) at time t into ring
// slot `slot` of the arrays ETA ([slot][nx*ny]) and U[f] ([slot][nx*ny*nl]);
// P (or null): the pressure field, when the grid holds one.
static int fill_cols(DevGrid &g, const DevSea &sea, Workspace &ws, const int *act, long nact, double t,
                     float *ETA, float *const U[3], float *P, int slot, cudaStream_t stream) {
    GridExtra *x = extra(g);
    if (nact == 0) return OK;
    const bool pres = P != nullptr && g.nf == 4;
    GridGeom G = geom(g);
    const int npad = sea.npad_g;
    const bool tc = g.method == 1 && x->df.built;
    const FillBytes fb = fill_bytes(g, sea, nact);
    int rc = workspace_reserve(ws, fb.all);
    if (rc) return rc;
    char *b = (char *)ws.base;
    double *first = (double *)(b + fb.ph + fb.rr);
    // the grid's own list of all columns (ascending) needs no look-up
    const bool all = (act == x->act_all || act == x->act_live) && nact == x->n_all;
    const GridCols cols = {G.d0, G.d2, G.dx, G.dy, g.nx, g.ny, 0, all ? nullptr : act, nact};
    GridTab tab;
    if (tc) {
        // eta1 and the Taylor gradients, then eta2 and the 3R depth-separated
        // quadratic forms of every column in one GEMM
        rc = grid_tab(sea, cols, t, b, true, &tab, stream);
        if (!rc) rc = first_surface(tab, cols, first, stream);
        if (!rc) rc = depthform_columns(x->df, sea, tab, cols, x->eta2, stream);
    } else {
        float2 *ph = (float2 *)b;
        float *rr = (float *)(b + fb.ph);
        k_column_coords<<<(unsigned)((nact + 255) / 256), 256, 0, stream>>>(G, nact, act, x->xy);
        note_launch();
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(x->tdev, &t, sizeof(double), cudaMemcpyHostToDevice, stream));
        rc = launch_phasors_public(sea, nact, x->xy, x->xy + nact, x->tdev, 1, 1, 0, npad, ph, rr, first, stream);
        if (!rc) rc = launch_eta_pairs(sea, nact, ph, rr, x->eta2, stream, x->split, x->split_cap);
    }
    if (rc) return rc;
    k_levels<<<(unsigned)((nact + 127) / 128), 128, 0, stream>>>(G, nact, act, x->sig, first, x->eta2, slot, ETA,
                                                                 x->zmin, x->zmax);
    note_launch();
    CK(cudaGetLastError());
    if (tc) {
        // first order at the level heights, then the second order from the R
        // basis functions of the level heights
        // (the form holds the pressure blocks when the grid holds pressure;
        // a fill without P leaves them unused)
        if (pres && x->df.nf != 4) return E_NOT_INITIALIZED;
        rc = first_levels(tab, cols, g.nl, x->df.nf, sea.depth, x->zmin, x->sec, stream);
        if (!rc) rc = depthform_combine(x->df, nact, g.nl, x->zmin, x->sec, stream);
    } else {
        // first and second order per (pair, level)
        rc = launch_column_pairs(sea, nact, g.nl, (float2 *)b, (float *)(b + fb.ph), x->zmin, x->sec, stream, x->split,
                                 x->split_cap, pres);
    }
    if (rc) return rc;
    if (pres) {
        // rebuild the height table only when a component ramp changed (once
        // every ramp has reached 1, the table stays valid)
        const size_t nc = x->ramp_par.size() / 3;
        std::vector<double> r(nc);
        for (size_t i = 0; i < nc; i++) {
            const double rt = x->ramp_par[3 * i], ts = x->ramp_par[3 * i + 1], du = x->ramp_par[3 * i + 2];
            const double down = std::max(std::min(1. - ((t - ts - du + rt) / (rt + SMALL)), 1.), 0.);
            const double up = std::max(std::min((t - ts) / (rt + SMALL), 1.), 0.);
            r[i] = up * down;
        }
        if (!x->kin_valid || r != x->kin_r) {
            rc = launch_pressure_kin(sea, t, KIN_NZ, x->kin, stream);
            if (rc) return rc;
            x->kin_r = r;
            x->kin_valid = true;
        }
    }
    long tot = nact * g.nl;
    k_scatter_levels<<<(unsigned)((tot + 255) / 256), 256, 0, stream>>>(
        G, nact, act, first, x->sec, x->zmin, x->zmax, slot, U[0], U[1], U[2], pres ? P : nullptr, x->kin, KIN_NZ);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

// Fill one ring slot at time t for the given column set.
static int fill_slot(DevGrid &g, const DevSea &sea, Workspace &ws, int slot, double t, bool live_only,
                     cudaStream_t stream) {
    GridExtra *x = extra(g);
    long nact = live_only ? x->n_live : x->n_all;
    const int *act = live_only ? x->act_live : x->act_all;
    return fill_cols(g, sea, ws, act, nact, t, g.ETA, g.U, g.nf == 4 ? g.U[3] : nullptr, slot, stream);
}

int grid_fill_columns(DevGrid &g, const DevSea &sea, Workspace &ws, const int *act, long nact, double t,
                      float *ETA, float *const U[3], int slot, void *stream) {
    if (nact < 0 || nact > (long)g.nx * g.ny) return E_BAD_ARGUMENT;
    return fill_cols(g, sea, ws, act, nact, t, ETA, U, nullptr, slot, (cudaStream_t)stream);
}

int grid_fill_slot(DevGrid &g, const DevSea &sea, Workspace &ws, int slot, double t, void *stream) {
    return fill_slot(g, sea, ws, slot, t, true, (cudaStream_t)stream);
}

void grid_live_columns(DevGrid &g, const int **act, long *n) {
    GridExtra *x = extra(g);
    *act = x->act_live;
    *n = x->n_live;
}

GridGeom grid_geom(const DevGrid &g) { return geom(g); }
const double *grid_sigma(const DevGrid &g) { return extra(g)->sig; }

static int gradients(DevGrid &g, cudaStream_t stream) {
    GradArgs a;
    a.g = geom(g);
    a.tstep = g.tstep;
    a.rdx = (float)(1.0 / g.dx); a.rdy = (float)(1.0 / g.dy); a.rds = (float)(1.0 / g.ds); a.rdt = (float)(1.0 / g.dt);
    a.F[0] = g.ETA; a.Fx[0] = g.ETAdx; a.Fy[0] = g.ETAdy; a.Fs[0] = nullptr; a.Ft[0] = g.ETAdt;
    for (int f = 0; f < 4; f++) {
        a.F[f + 1] = g.U[f]; a.Fx[f + 1] = g.Ux[f]; a.Fy[f + 1] = g.Uy[f];
        a.Fs[f + 1] = g.Us[f]; a.Ft[f + 1] = g.Ut[f];
    }
    a.img = reinterpret_cast<float4 *>(g.QIMG);
    a.eimg = reinterpret_cast<float4 *>(g.EIMG);
    const long nodes = (long)g.nx * g.ny * g.nl;
    const unsigned nb = (unsigned)((nodes + GRAD_B - 1) / GRAD_B);
    prof_begin(PK_GRADIENTS, stream);
    if (g.nf == 4) k_gradients<4><<<nb, GRAD_B, 0, stream>>>(a);
    else k_gradients<3><<<nb, GRAD_B, 0, stream>>>(a);
    note_launch();
    prof_end(PK_GRADIENTS, stream);
    CK(cudaGetLastError());
    return OK;
}

int grid_initialize(DevGrid &g, const DevSea &sea, Workspace &ws, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    bool wi = g.cfg.ignore_at_init;
    // initialize_kinematics[_with_ignore] (lsgrid_spline.cpp:679, 758)
    double tt0[4] = {wi ? g.t0 : g.t0 - g.dt, g.t0, g.t0 + g.dt, g.t0 + 2 * g.dt};
    g.tstep = 0;
    for (int tt = 0; tt < 4; tt++) {
        int rc = fill_slot(g, sea, ws, tt, tt0[tt], wi, stream);
        if (rc) return rc;
    }
    int rc = gradients(g, stream);
    if (rc) return rc;
    CK(cudaStreamSynchronize(stream));
    return OK;
}

int grid_gradients(DevGrid &g, void *stream) { return gradients(g, (cudaStream_t)stream); }

int grid_set_method(DevGrid &g, const Config &cfg, const DevSea &sea, int method, void *stream) {
    if (method != 0 && method != 1) return E_BAD_ARGUMENT;
    GridExtra *x = extra(g);
    if (method == 1 && (!x->df.built || x->df.nf != g.nf)) {
        int rc = depthform_build(cfg, sea, x->df, g.nf, stream);
        if (rc) return rc;
    }
    g.method = method;
    return OK;
}

int grid_set_pressure(DevGrid &g, const Config &cfg, const DevSea &sea, bool on, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    GridExtra *x = extra(g);
    const int nf = on ? 4 : 3;
    if (on && (!sea.d_tab_gp || !sea.d_tab_gk)) return E_UNSUPPORTED;   // first-order sea
    if (nf == g.nf) return OK;
    long v = (long)g.nx * g.ny * g.nl;
    if (on) {
        CK(cudaMalloc(&g.U[3], sizeof(float) * 4 * v));
        CK(cudaMalloc(&g.Ut[3], sizeof(float) * 4 * v));
        CK(cudaMalloc(&g.Ux[3], sizeof(float) * 2 * v));
        CK(cudaMalloc(&g.Uy[3], sizeof(float) * 2 * v));
        CK(cudaMalloc(&g.Us[3], sizeof(float) * 2 * v));
        CK(cudaMemsetAsync(g.U[3], 0, sizeof(float) * 4 * v, stream));
        CK(cudaMemsetAsync(g.Ut[3], 0, sizeof(float) * 4 * v, stream));
        if (!x->kin) CK(cudaMalloc(&x->kin, sizeof(double) * 2 * KIN_NZ));
        x->ramp_par.resize(3 * cfg.omega.size());
        for (size_t i = 0; i < cfg.omega.size(); i++) {
            x->ramp_par[3 * i] = cfg.ramptime[i];
            x->ramp_par[3 * i + 1] = cfg.starttime[i];
            x->ramp_par[3 * i + 2] = cfg.duration[i];
        }
        x->kin_valid = false;
    } else {
        float *q[] = {g.U[3], g.Ut[3], g.Ux[3], g.Uy[3], g.Us[3]};
        for (float *p : q) if (p) cudaFree(p);
        g.U[3] = g.Ut[3] = g.Ux[3] = g.Uy[3] = g.Us[3] = nullptr;
    }
    g.nf = nf;
    // the tensor-core form carries the pressure blocks only when asked to
    if (g.method == 1) {
        int rc = depthform_build(cfg, sea, x->df, nf, stream);
        if (rc) return rc;
    } else if (x->df.built) {
        depthform_free(x->df);
    }
    CK(cudaStreamSynchronize(stream));
    return OK;
}

int grid_tc_error(DevGrid &g, void *stream) { return depthform_error(extra(g)->df, stream); }

int depthform_rank(DevGrid &g) { return extra(g)->df.built ? extra(g)->df.R : 0; }

int grid_update(DevGrid &g, const DevSea &sea, Workspace &ws, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    // update (lsgrid_spline.cpp:847-931)
    g.tstep++;
    g.t0 += g.dt;
    double t2 = g.t0 + 2 * g.dt;
    int slot = (g.tstep + 3) % 4;
    int rc = fill_slot(g, sea, ws, slot, t2, true, stream);
    if (rc) return rc;
    return gradients(g, stream);
}

bool grid_check_time(const DevGrid &g, double t) { return t > g.t0 + g.dt; }

// ---------------------------------------------------------------------------
// Column shard.  The reference's MPI build splits the grid's rows of columns
// (index i) over the ranks by a work-balanced contiguous partition weighted
// by the live columns of each row (lsgrid_spline.cpp:652-664,
// mpi_utils.h:46-64); each rank fills its rows of the new slot and the slot's
// ETA, UX, UY, UZ are all-gathered (lsgrid_spline.cpp:907-910) before every
// rank recomputes the gradients.  A rank's rows [i0, i1) of a slot are
// contiguous in every field ([slot][i][j] and [slot][i][j][m]), so a block is
// one copy per field.
// ---------------------------------------------------------------------------
void grid_row_weights(const DevGrid &g, std::vector<long> &w) {
    GridExtra *x = extra(g);
    w.resize(g.nx);
    for (int i = 0; i < g.nx; i++) w[i] = x->row_live[i + 1] - x->row_live[i];
}

int grid_step_block(DevGrid &g, const DevSea &sea, Workspace &ws, int i0, int i1, void *stream_) {
    if (i0 < 0 || i1 > g.nx || i0 > i1) return E_BAD_ARGUMENT;
    cudaStream_t stream = (cudaStream_t)stream_;
    g.tstep++;
    g.t0 += g.dt;
    const double t2 = g.t0 + 2 * g.dt;
    const int slot = (g.tstep + 3) % 4;
    GridExtra *x = extra(g);
    const long a = x->row_live[i0], b = x->row_live[i1];
    return fill_cols(g, sea, ws, x->act_live + a, b - a, t2, g.ETA, g.U, g.nf == 4 ? g.U[3] : nullptr, slot, stream);
}

// rows [i0, i1) of field f (0 ETA, 1 + q the velocity / pressure field q) of
// the newest slot to or from buf (device or host memory); returns the count
long grid_block_elems(const DevGrid &g, int f, int i0, int i1) {
    return (long)(i1 - i0) * g.ny * (f == 0 ? 1 : g.nl);
}

int grid_block_copy(DevGrid &g, int f, int i0, int i1, float *buf, bool into_grid, void *stream_) {
    if (i0 < 0 || i1 > g.nx || i0 > i1 || f < 0 || f > g.nf || !buf) return E_BAD_ARGUMENT;
    cudaStream_t stream = (cudaStream_t)stream_;
    const int slot = (g.tstep + 3) % 4;
    const long c = (long)g.nx * g.ny;
    float *base = f == 0 ? g.ETA + (long)slot * c + (long)i0 * g.ny
                         : g.U[f - 1] + ((long)slot * c + (long)i0 * g.ny) * g.nl;
    const size_t bytes = sizeof(float) * grid_block_elems(g, f, i0, i1);
    if (bytes == 0) return OK;
    CK(cudaMemcpyAsync(into_grid ? base : buf, into_grid ? buf : base, bytes, cudaMemcpyDefault, stream));
    return OK;
}

int grid_query(const DevGrid &g, long n, const double *z, const ApiRows &rows, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (n <= 0) return OK;
    QueryArgs a;
    a.g = geom(g);
    a.t0 = g.t0;
    a.eimg = reinterpret_cast<const float4 *>(g.EIMG);
    a.img = reinterpret_cast<const float4 *>(g.QIMG);
    a.n = n; a.z = z; a.api = rows;
    a.inv_dx = 1.0 / a.g.dx; a.inv_dy = 1.0 / a.g.dy; a.inv_dt = 1.0 / a.g.dt;
    a.tanab = powf(tanf((float)a.g.tan_a), (float)a.g.tan_b);
    prof_begin(PK_QUERY, stream);
    const unsigned nb = (unsigned)((n + QB - 1) / QB);
    constexpr int SM3 = QB * QStage<3>::STRIDE * 16, SM4 = QB * QStage<4>::STRIDE * 16;
    static_assert(SM3 <= 48 * 1024 && SM4 <= 48 * 1024, "no shared-memory opt-in needed");
    if (g.nf == 4) k_query<4><<<nb, QB, SM4, stream>>>(a);
    else k_query<3><<<nb, QB, SM3, stream>>>(a);
    note_launch();
    prof_end(PK_QUERY, stream);
    CK(cudaGetLastError());
    return OK;
}

int grid_download(const DevGrid &g, int which, double *dst, long cap, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    long c = (long)g.nx * g.ny, v = c * g.nl;
    const float *src = nullptr;
    long n = 0;
    switch (which) {
    case 0: src = g.ETA; n = 4 * c; break;
    case 1: case 2: case 3: src = g.U[which - 1]; n = 4 * v; break;
    case 4: src = g.ETAdx; n = 2 * c; break;
    case 5: src = g.ETAdy; n = 2 * c; break;
    case 6: src = g.ETAdt; n = 4 * c; break;
    case 23:
        if (g.nf != 4) return E_UNSUPPORTED;
        src = g.U[3]; n = 4 * v; break;
    default:
        if (which >= 19 && which <= 22 && g.nf != 4) return E_UNSUPPORTED;
        if (which >= 7 && which <= 22) {
            int f = (which - 7) / 4, k = (which - 7) % 4;
            const float *arr[4] = {g.Ut[f], g.Ux[f], g.Uy[f], g.Us[f]};
            src = arr[k];
            n = (k == 0 ? 4 : 2) * v;
        } else {
            return E_BAD_ARGUMENT;
        }
    }
    if (!dst) return (int)std::min<long>(n, 0x7fffffff);
    if (cap < n) return E_TOO_LARGE;
    std::vector<float> h(n);
    CK(cudaMemcpyAsync(h.data(), src, sizeof(float) * n, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    for (long i = 0; i < n; i++) dst[i] = h[i];
    return (int)n;
}

}  // namespace cfdwm
