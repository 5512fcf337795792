// Learned s-grid update: a small convolutional operator over the grid's
// columns that predicts the second-order part of a ring slot from first-order
// channels, with the plain second-order method as its fallback and judge.
//
// The plain ring update (lsgrid_spline.cpp:847-931, columns :880-903) fills a
// slot with eta = eta1 + eta2 + swl and, at 16 stretched levels placed under
// that eta, U = first order + second order (uvw2, Irregular.cpp:975-1102) +
// the Taylor term above swl.  Its cost is the second-order pair sum
// (P ~ N^2 / 2 pairs per node).  This file replaces that sum, between full
// plain updates, by
//
//   features  first-order channels of every column on a grid extended by a
//             4-column halo: at the 16 levels placed under eta1 alone,
//             u, v, w and the hydrodynamic pressure head, each as the in-phase
//             sum (cos of the component phase) and its quadrature (the phase
//             shifted by -pi/2), scaled by the sea's first-order scales.
//             Products of in-phase and quadrature channels give exactly the
//             cos(phi_i +- phi_m) terms of the Sharma-Dean sums.
//   network   4 valid 3x3 convolutions (8 nl -> 32 -> 32 -> 32 -> 1 + 3 nl),
//             SiLU between them, BF16 weights, FP32 accumulation; the halo
//             makes the output exactly the grid's nx x ny columns.
//   output    eta2 and U - U1(levels under eta1) per level, scaled by the
//             second-order scales k sigma^2 and k sigma^2 omega.
//
// Training (forward, backward, Adam) runs on these kernels too; the training
// pairs are ring slots that the plain method filled.  Every surrogate step can
// be checked against the plain method on a sample of columns; when the
// sampled error exceeds the tolerance the plain method fills the slot.
//
// GB300 notes: the convolutions (forward, data and weight gradients) run as
// implicit GEMMs on the tcgen05 tensor cores (convtc.cu), with the FP32
// activations split into BF16 hi + lo parts and FP32 accumulation in TMEM.
// The features (firstorder.cu) leave in the convolutions' operand format.
#include "cfdwm.h"
#include "convtc.h"
#include "sgrid_geom.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
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

GridGeom grid_geom(const DevGrid &g);
const double *grid_sigma(const DevGrid &g);

namespace {

constexpr int SH = 4;        // halo columns per side: 4 valid 3x3 convolutions
constexpr int NQ = 8;        // first-order channels per level
constexpr int HID = CONV_HID;   // hidden channels
__global__ void k_adam(long n, float lr, float b1, float b2, float eps, float c1, float c2, const float *g,
                       float *w, float *m, float *v) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= n) return;
    float gg = g[e];
    float mm = b1 * m[e] + (1.f - b1) * gg;
    float vv = b2 * v[e] + (1.f - b2) * gg * gg;
    m[e] = mm;
    v[e] = vv;
    w[e] -= lr * (mm * c1) / (sqrtf(vv * c2) + eps);
}

// ---------------------------------------------------------------------------
// Slot-side kernels
// ---------------------------------------------------------------------------
// Normalised training targets of ring slot `slot` (all columns):
//   t[0][c] = (ETA - swl - eta1) / s_eta,  t[1 + f nl + m][c] = (U_f - base_f) / s_u
__global__ void k_surr_targets(int nx, int ny, int nl, int slot, float swl, const float *ETA, const float *U0,
                               const float *U1, const float *U2, const float *eta1, const float *base,
                               float inv_eta, float inv_u, float *tg) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    long nxy = (long)nx * ny, n = nxy * nl;
    if (e >= n) return;
    long c = e / nl;
    int m = (int)(e % nl);
    const float *U[3] = {U0, U1, U2};
    for (int f = 0; f < 3; f++) {
        float v = U[f][(long)slot * n + e] - base[(long)f * n + e];
        tg[(long)(1 + f * nl + m) * nxy + c] = v * inv_u;
    }
    if (m == 0) tg[c] = (ETA[(long)slot * nxy + c] - swl - eta1[c]) * inv_eta;
}

// Writes the predicted slot for the live columns.
// Writes the predicted slot for the live columns: first order + (network
// output + carried residual R of the last plain slot, when given).
__global__ void k_surr_apply(long nlive, const int *live, int nx, int ny, int nl, int slot, float swl,
                             const float *eta1, const float *base, const float *pred, const float *R,
                             float s_eta, float s_u, float *ETA, float *U0, float *U1, float *U2) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= nlive * nl) return;
    long q = e / nl;
    int m = (int)(e % nl);
    long c = live[q];
    long nxy = (long)nx * ny, n = nxy * nl;
    float *U[3] = {U0, U1, U2};
    for (int f = 0; f < 3; f++) {
        long o = (long)(1 + f * nl + m) * nxy + c;
        float v = pred[o] + (R ? R[o] : 0.f);
        U[f][(long)slot * n + c * nl + m] = base[(long)f * n + c * nl + m] + v * s_u;
    }
    if (m == 0) ETA[(long)slot * nxy + c] = eta1[c] + swl + (pred[c] + (R ? R[c] : 0.f)) * s_eta;
}

// Gaussian low-pass along one grid direction (dir 0: i, 1: j) of [C][nx][ny]
// planes, weights renormalised at the grid edges.
__global__ void k_blur(int C, int nx, int ny, int dir, float inv2s2, int rad, const float *in, float *out) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    long nxy = (long)nx * ny;
    if (e >= (long)C * nxy) return;
    long ch = e / nxy, c = e % nxy;
    int i = (int)(c / ny), j = (int)(c % ny);
    const float *pl = in + ch * nxy;
    float acc = 0.f, wsum = 0.f;
    for (int d = -rad; d <= rad; d++) {
        int ii = dir == 0 ? i + d : i, jj = dir == 0 ? j : j + d;
        if (ii < 0 || ii >= nx || jj < 0 || jj >= ny) continue;
        float w = __expf(-(float)(d * d) * inv2s2);
        acc += w * pl[(long)ii * ny + jj];
        wsum += w;
    }
    out[e] = acc / wsum;
}

__global__ void k_sub(long n, const float *b, float *a) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e < n) a[e] -= b[e];
}

__device__ __forceinline__ void atomic_max_pos(unsigned *p, float v) {
    if (!(v >= 0.f)) v = 3.0e38f;   // NaN counts as a failed check
    atomicMax(p, __float_as_uint(v));
}

// Max |slot - reference| over the columns col[0..n) (reference: slot 0 of the
// scratch arrays), eta and each velocity field, normalised.  err: [4] uint.
__global__ void k_surr_compare(long n, const int *col, int nx, int ny, int nl, int slot, const float *ETA,
                               const float *U0, const float *U1, const float *U2, const float *rETA,
                               const float *rU0, const float *rU1, const float *rU2, float inv_eta, float inv_u,
                               unsigned *err) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (e >= n * nl) return;
    long q = e / nl;
    int m = (int)(e % nl);
    long c = col ? col[q] : q;
    long nxy = (long)nx * ny, nn = nxy * nl;
    const float *U[3] = {U0, U1, U2}, *R[3] = {rU0, rU1, rU2};
    for (int f = 0; f < 3; f++)
        atomic_max_pos(err + 1 + f, fabsf(U[f][(long)slot * nn + c * nl + m] - R[f][c * nl + m]) * inv_u);
    if (m == 0) atomic_max_pos(err, fabsf(ETA[(long)slot * nxy + c] - rETA[c]) * inv_eta);
}

// max |ETA - swl| and max |U| over one slot (or slot-0 scratch arrays)
__global__ void k_slot_max(long nxy, int nl, float swl, const float *ETA, const float *U0, const float *U1,
                           const float *U2, unsigned *mx) {
    long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
    long n = nxy * nl;
    if (e >= n) return;
    float u = fmaxf(fabsf(U0[e]), fmaxf(fabsf(U1[e]), fabsf(U2[e])));
    atomic_max_pos(mx + 1, u);
    if (e < nxy) atomic_max_pos(mx, fabsf(ETA[e] - swl));
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct Surrogate {
    bool ready = false;
    int nl = 0, cin = 0, cout = 0;
    int ch[5] = {0, 0, 0, 0, 0};
    long off_w[4] = {0, 0, 0, 0}, off_b[4] = {0, 0, 0, 0}, nparams = 0;
    float *w32 = nullptr, *m1 = nullptr, *m2 = nullptr, *grad = nullptr;
    // BF16 weights as the convolutions read them, laid out anew when w32
    // changes: forward [0, 4) and data gradient [1, 4) of each layer
    __nv_bfloat16 *wp = nullptr;
    long off_f[4] = {0, 0, 0, 0}, off_d[4] = {0, 0, 0, 0};
    ConvPack pack[7];
    long adam_step = 0;
    // training / gradient scratch
    void *tr = nullptr;
    size_t tr_bytes = 0;
    int *d_idx = nullptr;
    int idx_cap = 0;
    float *h_loss = nullptr;   // pinned: the loss's block sums
    long loss_cap = 0;
    // grid-side buffers
    int gnx = 0, gny = 0, gnl = 0;
    const float *g_eta = nullptr;      // identity of the attached grid
    double g_dx = 0, g_dy = 0, g_dom[4] = {0, 0, 0, 0}, g_ign[4] = {0, 0, 0, 0};
    void *xs = nullptr;        // first-order channels, split (convtc.h)
    float *base = nullptr, *eta1 = nullptr, *pred = nullptr;
    float *R = nullptr;        // residual (plain - network) of the last plain slot, [cout][nx ny]
    float *Rtmp = nullptr;
    bool have_res = false;
    double carry_lw = 0.0;     // low-pass scale of the carried residual, in mean wavelengths (0: none)
    float *rETA = nullptr, *rU[3] = {nullptr, nullptr, nullptr};
    int *d_sample = nullptr;
    unsigned *d_err = nullptr;
    // the checked columns' plain fill runs beside the prediction
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    std::vector<int> live;
    float fmax_eta = 0.f, fmax_u = 0.f;
    unsigned long long rng = 0x2545F4914F6CDD1DULL;
    long steps = 0, fallbacks = 0, plain_steps = 0;
};

static Surrogate g_s;

static void free_grid_side(Surrogate &s) {
    void *q[] = {s.xs, s.base, s.eta1, s.pred, s.rETA, s.rU[0], s.rU[1], s.rU[2],
                 s.d_sample, s.d_err, s.R, s.Rtmp};
    for (void *p : q) if (p) cudaFree(p);
    s.xs = nullptr; s.base = s.eta1 = s.pred = s.rETA = s.R = nullptr;
    s.Rtmp = nullptr;
    s.have_res = false;
    s.rU[0] = s.rU[1] = s.rU[2] = nullptr;
    s.d_sample = nullptr; s.d_err = nullptr;
    s.gnx = s.gny = s.gnl = 0;
    s.g_eta = nullptr;
    s.live.clear();
}

static void free_all(Surrogate &s) {
    free_grid_side(s);
    void *q[] = {s.w32, s.m1, s.m2, s.grad, s.wp, s.tr, s.d_idx};
    for (void *p : q) if (p) cudaFree(p);
    if (s.h_loss) cudaFreeHost(s.h_loss);
    if (s.fork) cudaEventDestroy(s.fork);
    if (s.join) cudaEventDestroy(s.join);
    if (s.side) cudaStreamDestroy(s.side);
    s = Surrogate();
}

// splitmix64 + Box-Muller: the same initial weights on every host
static double rnd_unit(unsigned long long &st) {
    st += 0x9E3779B97F4A7C15ULL;
    unsigned long long z = st;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    return ((z >> 11) + 0.5) * (1.0 / 9007199254740992.0);
}

static int pack_weights(const Surrogate &s, cudaStream_t st) { return conv_pack(s.pack, 7, s.w32, s.wp, st); }

int surrogate_create(int nl, unsigned long long seed, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (nl < 1 || nl > 32) return E_BAD_ARGUMENT;
    free_all(g_s);
    Surrogate &s = g_s;
    s.nl = nl;
    s.cin = NQ * nl;
    s.cout = 1 + 3 * nl;
    int ch[5] = {s.cin, HID, HID, HID, s.cout};
    std::memcpy(s.ch, ch, sizeof(ch));
    long off = 0;
    // all weight blocks first, then the biases
    for (int l = 0; l < 4; l++) { s.off_w[l] = off; off += (long)ch[l + 1] * ch[l] * 9; }
    for (int l = 0; l < 4; l++) { s.off_b[l] = off; off += ch[l + 1]; }
    s.nparams = off;
    long op = 0;
    for (int q = 0; q < 7; q++) {
        const bool data = q >= 4;
        const int l = data ? q - 3 : q;
        s.pack[q] = {s.off_w[l], ch[l], ch[l + 1], data};
        (data ? s.off_d : s.off_f)[l] = op;
        op += data ? conv_pack_elems(ch[l + 1], ch[l]) : conv_pack_elems(ch[l], ch[l + 1]);
    }
    std::vector<float> w(off, 0.f);
    unsigned long long st = seed;
    for (int l = 0; l < 4; l++) {
        double sd = std::sqrt(2.0 / (ch[l] * 9.0)) * (l == 3 ? 0.1 : 1.0);
        for (long e = 0; e < (long)ch[l + 1] * ch[l] * 9; e++) {
            double u1 = rnd_unit(st), u2 = rnd_unit(st);
            w[s.off_w[l] + e] = (float)(sd * std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
        }
    }
    int low = 0, high = 0;
    CK(cudaDeviceGetStreamPriorityRange(&low, &high));
    CK(cudaStreamCreateWithPriority(&s.side, cudaStreamNonBlocking, high));
    CK(cudaEventCreateWithFlags(&s.fork, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&s.join, cudaEventDisableTiming));
    CK(cudaMalloc(&s.w32, sizeof(float) * off));
    CK(cudaMalloc(&s.m1, sizeof(float) * off));
    CK(cudaMalloc(&s.m2, sizeof(float) * off));
    CK(cudaMalloc(&s.grad, sizeof(float) * off));
    CK(cudaMalloc(&s.wp, sizeof(__nv_bfloat16) * op));
    CK(cudaMemcpyAsync(s.w32, w.data(), sizeof(float) * off, cudaMemcpyHostToDevice, stream));
    CK(cudaMemsetAsync(s.m1, 0, sizeof(float) * off, stream));
    CK(cudaMemsetAsync(s.m2, 0, sizeof(float) * off, stream));
    int rc = conv_load();
    if (!rc) rc = pack_weights(s, stream);
    if (rc) return rc;
    CK(cudaStreamSynchronize(stream));
    s.ready = true;
    return OK;
}

void surrogate_destroy() { free_all(g_s); }

long surrogate_nparams() { return g_s.ready ? g_s.nparams : 0; }
int surrogate_levels() { return g_s.ready ? g_s.nl : 0; }

int surrogate_get_params(float *dst, long n, void *stream) {
    if (!g_s.ready) return E_NOT_INITIALIZED;
    if (n < g_s.nparams || !dst) return E_BAD_ARGUMENT;
    CK(cudaMemcpyAsync(dst, g_s.w32, sizeof(float) * g_s.nparams, cudaMemcpyDefault, (cudaStream_t)stream));
    CK(cudaStreamSynchronize((cudaStream_t)stream));
    return OK;
}

int surrogate_set_params(const float *src, long n, void *stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    if (!g_s.ready) return E_NOT_INITIALIZED;
    if (n != g_s.nparams || !src) return E_BAD_ARGUMENT;
    CK(cudaMemcpyAsync(g_s.w32, src, sizeof(float) * n, cudaMemcpyDefault, stream));
    CK(cudaMemsetAsync(g_s.m1, 0, sizeof(float) * n, stream));
    CK(cudaMemsetAsync(g_s.m2, 0, sizeof(float) * n, stream));
    g_s.adam_step = 0;
    int rc = pack_weights(g_s, stream);
    if (rc) return rc;
    CK(cudaStreamSynchronize(stream));
    return OK;
}

// ---- layers ---------------------------------------------------------------
// The convolutions run as implicit GEMMs on the tcgen05 tensor cores
// (convtc.cu); the error word of their bounded waits is read where a call
// synchronises anyway.
static int conv_check(cudaStream_t st) {
    int e = conv_error(st);
    if (e == 0) return OK;
    std::fprintf(stderr, "cfdwm: a bounded wait of the tensor-core convolutions expired (code %d)\n", e);
    return E_CUDA;
}

static int reserve_tr(Surrogate &s, size_t bytes) {
    if (s.tr_bytes >= bytes) return OK;
    if (s.tr) cudaFree(s.tr);
    s.tr = nullptr;
    s.tr_bytes = 0;
    CK(cudaMalloc(&s.tr, bytes));
    s.tr_bytes = bytes;
    return OK;
}

static size_t up256(size_t b) { return (b + 255) / 256 * 256; }

// The hidden layers over split inputs h[0]: activations h[1..3] (split) and,
// for the backward pass, silu' of their pre-activations ds[1..3] (null: not
// kept).
static int net_hidden(const Surrogate &s, int B, int H, int W, void *const *h, void *const *ds, cudaStream_t st) {
    for (int l = 0; l < 3; l++) {
        int rc = conv_hidden(h[l], s.wp + s.off_f[l], s.w32 + s.off_b[l], B, s.ch[l], H - 2 * l, W - 2 * l, h[l + 1],
                             ds ? ds[l + 1] : nullptr, st);
        if (rc) return rc;
    }
    return OK;
}

// Forward + loss + backward into s.grad.  x: [*][cin][H][W], tg: [*][cout][H-8][W-8],
// batch entries idx[0..B) (device) or 0..B-1.  The loss's nloss block sums
// come to s.h_loss when want_loss is set (finish_loss).
static int loss_grad(Surrogate &s, const float *x, const float *tg, const int *idx, int B, int H, int W,
                     bool want_loss, long *nloss, cudaStream_t st) {
    if (H < 9 || W < 9 || B < 1 || s.cout > 64) return E_BAD_ARGUMENT;
    const long P4 = (long)(H - 8) * (W - 8);
    const int nl4 = conv_bias_parts(B, H - 8, W - 8), npo = s.cout <= 32 ? 32 : 64;
    // split input, h ds da of the hidden layers, dys, partial sums
    size_t bytes = 0;
    auto take = [&](size_t n) { size_t o = bytes; bytes += up256(n); return o; };
    const size_t o_x = take(conv_split_bytes(B, s.cin, H, W));
    size_t o_h[4] = {}, o_s[4] = {}, o_a[4] = {}, o_p[4] = {}, o_b[4] = {};
    ConvWgt wg[4] = {};
    for (int l = 0; l < 4; l++) {
        wg[l].C = s.ch[l]; wg[l].O = s.ch[l + 1]; wg[l].H = H - 2 * l; wg[l].W = W - 2 * l;
    }
    int rc = conv_wgt_plan(wg, 4, B);
    if (rc) return rc;
    for (int l = 0; l < 4; l++) {
        const int h = H - 2 * l, w = W - 2 * l;
        o_p[l] = take(sizeof(float) * 9 * s.ch[l] * s.ch[l + 1] * wg[l].nslab);
        if (l == 0) continue;
        const size_t n = conv_split_bytes(B, HID, h, w);
        o_h[l] = take(n);
        o_s[l] = take(n);
        o_a[l] = take(n);
        o_b[l] = take(sizeof(float) * HID * conv_bias_parts(B, h, w));
    }
    const size_t o_dy = take(conv_split_bytes(B, s.cout, H - 8, W - 8));
    const size_t o_l = take(sizeof(float) * nl4), o_bo = take(sizeof(float) * nl4 * npo);
    rc = reserve_tr(s, bytes);
    if (rc) return rc;
    char *base = (char *)s.tr;
    void *h[4], *ds[4], *da[5];
    for (int l = 1; l < 4; l++) { h[l] = base + o_h[l]; ds[l] = base + o_s[l]; da[l] = base + o_a[l]; }
    h[0] = base + o_x;
    da[4] = base + o_dy;
    float *lpart = (float *)(base + o_l), *bout = (float *)(base + o_bo);
    const long tbs = (long)s.cout * P4;
    if ((rc = conv_split(x, (long)s.cin * H * W, idx, B, s.cin, H, W, h[0], st))) return rc;
    if ((rc = net_hidden(s, B, H, W, h, ds, st))) return rc;
    // L = sum_{b,o,p} w_o (y - t)^2 / (B P sum_o w_o), w_0 = nl (the elevation), 1 else
    ConvLoss cl = {tg, tbs, idx, (float)s.nl, 0.f};
    cl.inv_norm = (float)(1.0 / ((double)B * P4 * (cl.w0 + (s.cout - 1))));
    if ((rc = conv_loss(h[3], s.wp + s.off_f[3], s.w32 + s.off_b[3], B, HID, s.cout, H - 6, W - 6, cl, da[4], bout,
                        lpart, st)))
        return rc;
    ConvSum sums[8];
    for (int l = 3; l >= 1; l--) {
        const int hh = H - 2 * l, ww = W - 2 * l;
        float *bp = (float *)(base + o_b[l]);
        if ((rc = conv_data_grad(da[l + 1], s.wp + s.off_d[l], ds[l], B, s.ch[l + 1], hh, ww, da[l], bp, st))) return rc;
        sums[4 + l] = {bp, s.grad + s.off_b[l - 1], HID, HID, conv_bias_parts(B, hh, ww), nullptr};
    }
    sums[4] = {bout, s.grad + s.off_b[3], s.cout, npo, nl4, nullptr};
    for (int l = 0; l < 4; l++) {
        const long n = 9L * s.ch[l] * s.ch[l + 1];
        wg[l].xs = h[l];
        wg[l].dys = da[l + 1];
        wg[l].part = (float *)(base + o_p[l]);
        sums[l] = {wg[l].part, s.grad + s.off_w[l], n, n, wg[l].nslab, &wg[l]};
    }
    if ((rc = conv_weight_grads(wg, 4, B, st))) return rc;
    if ((rc = conv_sums(sums, 8, st))) return rc;
    *nloss = nl4;
    if (want_loss) {
        if (s.loss_cap < nl4) {
            if (s.h_loss) cudaFreeHost(s.h_loss);
            s.h_loss = nullptr;
            s.loss_cap = 0;
            CK(cudaMallocHost(&s.h_loss, sizeof(float) * nl4));
            s.loss_cap = nl4;
        }
        CK(cudaMemcpyAsync(s.h_loss, lpart, sizeof(float) * nl4, cudaMemcpyDeviceToHost, st));
    }
    return OK;
}

// Synchronises; the loss from its block sums.
static int finish_loss(const Surrogate &s, long nloss, double *loss, cudaStream_t st) {
    int rc = conv_check(st);
    if (rc) return rc;
    double L = 0.0;
    for (long k = 0; k < nloss; k++) L += s.h_loss[k];
    *loss = L;
    return OK;
}

static int put_idx(Surrogate &s, const int *idx_host, int B, cudaStream_t st) {
    if (s.idx_cap < B) {
        if (s.d_idx) cudaFree(s.d_idx);
        s.d_idx = nullptr;
        CK(cudaMalloc(&s.d_idx, sizeof(int) * B));
        s.idx_cap = B;
    }
    CK(cudaMemcpyAsync(s.d_idx, idx_host, sizeof(int) * B, cudaMemcpyHostToDevice, st));
    return OK;
}

int surrogate_loss_grad(const float *x, const float *tg, int B, int H, int W, double *loss, float *grad,
                        void *stream_) {
    cudaStream_t st = (cudaStream_t)stream_;
    if (!g_s.ready) return E_NOT_INITIALIZED;
    long nloss;
    int rc = loss_grad(g_s, x, tg, nullptr, B, H, W, loss != nullptr, &nloss, st);
    if (rc) return rc;
    if (grad) CK(cudaMemcpyAsync(grad, g_s.grad, sizeof(float) * g_s.nparams, cudaMemcpyDefault, st));
    if (loss) return finish_loss(g_s, nloss, loss, st);
    CK(cudaStreamSynchronize(st));
    return OK;
}

int surrogate_train_step(const float *xs, const float *ts, long nsamples, const int *idx_host, int B, int H, int W,
                         float lr, double *loss, void *stream_) {
    cudaStream_t st = (cudaStream_t)stream_;
    Surrogate &s = g_s;
    if (!s.ready) return E_NOT_INITIALIZED;
    if (!idx_host || B < 1) return E_BAD_ARGUMENT;
    for (int b = 0; b < B; b++)
        if (idx_host[b] < 0 || idx_host[b] >= nsamples) return E_BAD_ARGUMENT;
    int rc = put_idx(s, idx_host, B, st);
    if (rc) return rc;
    long nloss;
    rc = loss_grad(s, xs, ts, s.d_idx, B, H, W, loss != nullptr, &nloss, st);
    if (!rc && loss) rc = finish_loss(s, nloss, loss, st);
    if (rc) return rc;
    s.adam_step++;
    const double b1 = 0.9, b2 = 0.999;
    float c1 = (float)(1.0 / (1.0 - std::pow(b1, (double)s.adam_step)));
    float c2 = (float)(1.0 / (1.0 - std::pow(b2, (double)s.adam_step)));
    k_adam<<<(unsigned)((s.nparams + 255) / 256), 256, 0, st>>>(s.nparams, lr, (float)b1, (float)b2, 1e-8f, c1, c2,
                                                                s.grad, s.w32, s.m1, s.m2);
    note_launch();
    CK(cudaGetLastError());
    return pack_weights(s, st);
}

int surrogate_check(void *stream) { return conv_check((cudaStream_t)stream); }

// The network over planes x or split inputs xs.
static int forward(Surrogate &s, const float *x, void *xs, int B, int H, int W, float *y, cudaStream_t st) {
    if (H < 9 || W < 9 || B < 1 || s.cout > 64) return E_BAD_ARGUMENT;
    size_t off[5] = {};
    for (int l = 0; l < 4; l++)
        off[l + 1] = off[l] + (l == 0 && xs ? 0 : up256(conv_split_bytes(B, s.ch[l], H - 2 * l, W - 2 * l)));
    int rc = reserve_tr(s, off[4]);
    if (rc) return rc;
    void *h[4];
    for (int l = 0; l < 4; l++) h[l] = (char *)s.tr + off[l];
    if (xs) h[0] = xs;
    prof_begin(PK_SURR_NET, st);
    if (!xs) rc = conv_split(x, (long)s.cin * H * W, nullptr, B, s.cin, H, W, h[0], st);
    if (!rc) rc = net_hidden(s, B, H, W, h, nullptr, st);
    if (!rc) rc = conv_output(h[3], s.wp + s.off_f[3], s.w32 + s.off_b[3], B, HID, s.cout, H - 6, W - 6, y, st);
    prof_end(PK_SURR_NET, st);
    return rc;
}

int surrogate_forward(const float *x, int B, int H, int W, float *y, void *stream) {
    if (!g_s.ready) return E_NOT_INITIALIZED;
    return forward(g_s, x, nullptr, B, H, W, y, (cudaStream_t)stream);
}

// ---- grid side ------------------------------------------------------------
// Sea-state scales: sigma^2 = sum A^2 / 2, omega_m and k_m the A^2-weighted means.
static void sea_scales(const Config &cfg, double &sigma, double &om, double &km) {
    double s2 = 0, so = 0, sk = 0;
    for (size_t i = 0; i < cfg.A.size(); i++) {
        double a2 = cfg.A[i] * cfg.A[i];
        s2 += a2;
        so += a2 * cfg.omega[i];
        sk += a2 * cfg.k[i];
    }
    sigma = std::sqrt(0.5 * s2);
    om = s2 > 0 ? so / s2 : 1.0;
    km = s2 > 0 ? sk / s2 : 1.0;
    if (sigma <= 0) sigma = 1.0;
}

// The grid-side buffers follow the grid: their sizes its dimensions, the
// halo coordinates and the live-column list its placement and ignore area.
static bool same_grid(const Surrogate &s, const DevGrid &g) {
    if (!(s.gnx == g.nx && s.gny == g.ny && s.gnl == g.nl && s.xs)) return false;
    if (s.g_eta != g.ETA || s.g_dx != g.dx || s.g_dy != g.dy) return false;
    for (int q = 0; q < 4; q++)
        if (s.g_dom[q] != g.cfg.domain[q] || s.g_ign[q] != g.cfg.domain_ignore[q]) return false;
    return true;
}

static int attach_grid(Surrogate &s, DevGrid &g, cudaStream_t st) {
    if (g.nl != s.nl) return E_BAD_ARGUMENT;
    if (same_grid(s, g)) return OK;
    free_grid_side(s);
    const int nxh = g.nx + 2 * SH, nyh = g.ny + 2 * SH;
    const long nxy = (long)g.nx * g.ny, n = nxy * g.nl;
    CK(cudaMalloc(&s.xs, conv_split_bytes(1, s.cin, nxh, nyh)));
    CK(cudaMalloc(&s.base, sizeof(float) * 3 * n));
    CK(cudaMalloc(&s.eta1, sizeof(float) * nxy));
    CK(cudaMalloc(&s.pred, sizeof(float) * s.cout * nxy));
    CK(cudaMalloc(&s.R, sizeof(float) * s.cout * nxy));
    CK(cudaMalloc(&s.Rtmp, sizeof(float) * s.cout * nxy));
    CK(cudaMalloc(&s.rETA, sizeof(float) * nxy));
    for (int f = 0; f < 3; f++) CK(cudaMalloc(&s.rU[f], sizeof(float) * n));
    CK(cudaMalloc(&s.d_err, sizeof(unsigned) * 8));
    CK(cudaMalloc(&s.d_sample, sizeof(int) * 4096));
    const int *act;
    long nlive;
    grid_live_columns(g, &act, &nlive);
    s.live.resize(nlive);
    if (nlive) CK(cudaMemcpyAsync(s.live.data(), act, sizeof(int) * nlive, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    s.gnx = g.nx; s.gny = g.ny; s.gnl = g.nl;
    s.g_eta = g.ETA; s.g_dx = g.dx; s.g_dy = g.dy;
    for (int q = 0; q < 4; q++) { s.g_dom[q] = g.cfg.domain[q]; s.g_ign[q] = g.cfg.domain_ignore[q]; }
    s.fmax_eta = s.fmax_u = 0.f;
    s.have_res = false;
    return OK;
}

static size_t features_bytes(const DevSea &sea, const DevGrid &g) {
    const int nxh = g.nx + 2 * SH, nyh = g.ny + 2 * SH;
    return up256(grid_tab_bytes(sea, nxh, nyh)) + up256(sizeof(double) * 5 * nxh * nyh);
}

// First-order channels of the attached grid at time t into planes feat and / or
// the split format xs (null: not wanted), base and eta1.
static int features(const Config &cfg, const DevSea &sea, DevGrid &g, Workspace &ws, double t, float *feat, void *xs,
                    float *base, float *eta1, cudaStream_t st) {
    const int nxh = g.nx + 2 * SH, nyh = g.ny + 2 * SH;
    const long nh = (long)nxh * nyh;
    int rc = workspace_reserve(ws, features_bytes(sea, g));
    if (rc) return rc;
    double *first = (double *)((char *)ws.base + up256(grid_tab_bytes(sea, nxh, nyh)));
    const GridGeom G = grid_geom(g);
    const GridCols cols = {G.d0, G.d2, G.dx, G.dy, nxh, nyh, SH, nullptr, nh};
    GridTab tab;
    prof_begin(PK_SURR_FEATURES, st);
    rc = grid_tab(sea, cols, t, ws.base, false, &tab, st);
    // eta1 and the Taylor gradients of the halo columns
    if (!rc) rc = first_surface(tab, cols, first, st);
    double sigma, om, km;
    sea_scales(cfg, sigma, om, km);
    if (!rc)
        rc = first_features(tab, cols, G, SH, grid_sigma(g), first, (float)(1.0 / (sigma * om)), (float)(1.0 / sigma),
                            feat, xs, base, eta1, st);
    prof_end(PK_SURR_FEATURES, st);
    return rc;
}

int surrogate_features(const Config &cfg, const DevSea &sea, DevGrid &g, Workspace &ws, double t, float *feat,
                       float *base, float *eta1, void *stream_) {
    cudaStream_t st = (cudaStream_t)stream_;
    Surrogate &s = g_s;
    if (!s.ready) return E_NOT_INITIALIZED;
    int rc = attach_grid(s, g, st);
    if (rc) return rc;
    return features(cfg, sea, g, ws, t, feat, feat ? nullptr : s.xs, base ? base : s.base, eta1 ? eta1 : s.eta1, st);
}

int surrogate_targets(const Config &cfg, DevGrid &g, int slot, const float *base, const float *eta1, float *tg,
                      void *stream_) {
    cudaStream_t st = (cudaStream_t)stream_;
    Surrogate &s = g_s;
    if (!s.ready) return E_NOT_INITIALIZED;
    if (slot < 0 || slot > 3 || g.nl != s.nl) return E_BAD_ARGUMENT;
    double sigma, om, km;
    sea_scales(cfg, sigma, om, km);
    const double s_eta = km * sigma * sigma, s_u = s_eta * om;
    long n = (long)g.nx * g.ny * g.nl;
    k_surr_targets<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        g.nx, g.ny, g.nl, slot, (float)g.swl, g.ETA, g.U[0], g.U[1], g.U[2], eta1 ? eta1 : s.eta1,
        base ? base : s.base, (float)(1.0 / s_eta), (float)(1.0 / s_u), tg);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

static int slot_max(Surrogate &s, DevGrid &g, const float *ETA, float *const U[3], cudaStream_t st, float *me,
                    float *mu) {
    long nxy = (long)g.nx * g.ny;
    CK(cudaMemsetAsync(s.d_err, 0, sizeof(unsigned) * 8, st));
    k_slot_max<<<(unsigned)((nxy * g.nl + 255) / 256), 256, 0, st>>>(nxy, g.nl, (float)g.swl, ETA, U[0], U[1], U[2],
                                                                      s.d_err + 4);
    note_launch();
    CK(cudaGetLastError());
    unsigned h[2];
    CK(cudaMemcpyAsync(h, s.d_err + 4, sizeof(h), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    std::memcpy(me, &h[0], 4);
    std::memcpy(mu, &h[1], 4);
    return OK;
}

// s.base, s.eta1 and the network's output s.pred at time t.
static int predict(Surrogate &s, const Config &cfg, const DevSea &sea, DevGrid &g, Workspace &ws, double t,
                   cudaStream_t st) {
    int rc = features(cfg, sea, g, ws, t, nullptr, s.xs, s.base, s.eta1, st);
    return rc ? rc : forward(s, nullptr, s.xs, 1, g.nx + 2 * SH, g.ny + 2 * SH, s.pred, st);
}

// Predicts slot `slot` at time t for the live columns.
static int predict_slot(Surrogate &s, const Config &cfg, const DevSea &sea, DevGrid &g, Workspace &ws, int slot,
                        double t, bool carry, cudaStream_t st) {
    int rc = predict(s, cfg, sea, g, ws, t, st);
    if (rc) return rc;
    double sigma, om, km;
    sea_scales(cfg, sigma, om, km);
    const double s_eta = km * sigma * sigma, s_u = s_eta * om;
    long nlive = (long)s.live.size();
    if (nlive == 0) return OK;
    const int *act;
    long nl2;
    grid_live_columns(g, &act, &nl2);
    k_surr_apply<<<(unsigned)((nlive * g.nl + 255) / 256), 256, 0, st>>>(
        nlive, act, g.nx, g.ny, g.nl, slot, (float)g.swl, s.eta1, s.base, s.pred, (carry && s.have_res) ? s.R : nullptr,
        (float)s_eta, (float)s_u, g.ETA, g.U[0], g.U[1], g.U[2]);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

// err[0..3]: max |eta - eta_ref| / max|eta_ref - swl|, and the same for u, v, w
// against max |U_ref| (the plain reference of the compared columns comes from
// the scratch arrays; col null: all columns).
static int compare(Surrogate &s, DevGrid &g, int slot, const int *col, long n, float inv_eta, float inv_u,
                   double err[4], cudaStream_t st) {
    CK(cudaMemsetAsync(s.d_err, 0, sizeof(unsigned) * 4, st));
    k_surr_compare<<<(unsigned)((n * g.nl + 255) / 256), 256, 0, st>>>(
        n, col, g.nx, g.ny, g.nl, slot, g.ETA, g.U[0], g.U[1], g.U[2], s.rETA, s.rU[0], s.rU[1], s.rU[2], inv_eta,
        inv_u, s.d_err);
    note_launch();
    CK(cudaGetLastError());
    unsigned h[4];
    CK(cudaMemcpyAsync(h, s.d_err, sizeof(h), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    int rc = conv_check(st);
    if (rc) return rc;
    for (int q = 0; q < 4; q++) {
        float v;
        std::memcpy(&v, &h[q], 4);
        err[q] = v;
    }
    return OK;
}

// R = (plain slot - first order) - network, normalised, for a slot the plain
// method filled at time t.  have_pred: s.pred/s.base/s.eta1 already hold the
// network's output and the first order at t.
static int refresh_residual(Surrogate &s, const Config &cfg, const DevSea &sea, DevGrid &g, Workspace &ws,
                            int slot, double t, bool have_pred, cudaStream_t st) {
    int rc;
    if (!have_pred) {
        rc = predict(s, cfg, sea, g, ws, t, st);
        if (rc) return rc;
    }
    rc = surrogate_targets(cfg, g, slot, s.base, s.eta1, s.R, st);
    if (rc) return rc;
    long n = (long)s.cout * g.nx * g.ny;
    k_sub<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, s.pred, s.R);
    note_launch();
    CK(cudaGetLastError());
    // keep the slowly varying part: a Gaussian of carry_lw mean wavelengths
    // (the sum-frequency part of the residual oscillates on half a wavelength
    // and in time at twice the wave frequency; the long-wave part persists)
    double sigma, om, km;
    sea_scales(cfg, sigma, om, km);
    const double lam = 2.0 * 3.141592653589793 / std::max(km, 1e-12);
    if (s.carry_lw > 0) {
        for (int dir = 0; dir < 2; dir++) {
            double sd = s.carry_lw * lam / (dir == 0 ? g.dx : g.dy);
            int rad = (int)std::min(3.0 * sd, (double)(dir == 0 ? g.nx : g.ny));
            float inv2s2 = (float)(0.5 / std::max(sd * sd, 1e-12));
            const float *src = dir == 0 ? s.R : s.Rtmp;
            float *dst = dir == 0 ? s.Rtmp : s.R;
            k_blur<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s.cout, g.nx, g.ny, dir, inv2s2, rad, src, dst);
            note_launch();
            CK(cudaGetLastError());
        }
    } else {
        CK(cudaMemsetAsync(s.R, 0, sizeof(float) * n, st));
    }
    s.have_res = true;
    return OK;
}

void surrogate_set_carry(double wavelengths) {
    g_s.carry_lw = wavelengths;
    g_s.have_res = false;
}

static unsigned long long lcg(unsigned long long &st) {
    st = st * 6364136223846793005ULL + 1442695040888963407ULL;
    return st >> 33;
}

// One ring step of the grid (lsgrid_spline.cpp:847-931 order: advance, fill
// the newest slot, gradients).  mode 0 plain; 1 surrogate with a check of
// nsample plain columns (fallback to plain above tol); 2 surrogate unchecked.
int surrogate_step(const Config &cfg, const DevSea &sea, DevGrid &g, Workspace &ws, int mode, double tol,
                   int nsample, int *fell_back, double *err_out, void *stream_) {
    cudaStream_t st = (cudaStream_t)stream_;
    Surrogate &s = g_s;
    const bool carry = (mode & 4) == 0;
    mode &= 3;
    if (mode != 0 && !s.ready) return E_NOT_INITIALIZED;
    if (mode > 2 || nsample < 0 || nsample > 4096) return E_BAD_ARGUMENT;
    if (mode != 0 && g.nf != 3) return E_UNSUPPORTED;   // the network predicts no pressure
    if (mode != 0) {
        int rc = attach_grid(s, g, st);
        if (rc) return rc;
        if (carry && !s.have_res) {
            // the newest slot is a plain one (initialisation or a plain step)
            rc = refresh_residual(s, cfg, sea, g, ws, (g.tstep + 3) % 4, g.t0 + 2 * g.dt, false, st);
            if (rc) return rc;
        }
    }
    g.tstep++;
    g.t0 += g.dt;
    const double t2 = g.t0 + 2 * g.dt;
    const int slot = (g.tstep + 3) % 4;
    int fb = 0;
    double err[4] = {0, 0, 0, 0};
    int rc = OK;
    if (mode == 0) {
        rc = grid_fill_slot(g, sea, ws, slot, t2, st);
        if (rc) return rc;
        s.plain_steps++;
        if (s.ready && same_grid(s, g)) {
            long nxy = (long)g.nx * g.ny;
            float *U[3] = {g.U[0] + (long)slot * nxy * g.nl, g.U[1] + (long)slot * nxy * g.nl,
                           g.U[2] + (long)slot * nxy * g.nl};
            rc = slot_max(s, g, g.ETA + (long)slot * nxy, U, st, &s.fmax_eta, &s.fmax_u);
            if (rc) return rc;
            if (carry) {
                rc = refresh_residual(s, cfg, sea, g, ws, slot, t2, false, st);
                if (rc) return rc;
            }
        }
    } else {
        if (s.fmax_eta <= 0.f || s.fmax_u <= 0.f) {
            // scales of the check: the slot the plain method filled last
            long nxy = (long)g.nx * g.ny;
            int prev = (g.tstep + 2) % 4;
            float *U[3] = {g.U[0] + (long)prev * nxy * g.nl, g.U[1] + (long)prev * nxy * g.nl,
                           g.U[2] + (long)prev * nxy * g.nl};
            rc = slot_max(s, g, g.ETA + (long)prev * nxy, U, st, &s.fmax_eta, &s.fmax_u);
            if (rc) return rc;
        }
        long ns = std::min<long>(nsample, (long)s.live.size());
        // the plain fill of a few columns leaves most of the GPU idle (64
        // columns: 190 us of latency and one read of the GEMM's weights), so it
        // runs on a stream and a part of the workspace of its own beside the
        // prediction, which shares no buffer with it.  The stream's blocks go
        // first: its GEMM needs whole SMs, and comes late otherwise (706 us a
        // step in one stream, 606 with the priority, 680 to 720 without)
        const bool check = mode == 1 && ns > 0;
        if (check) {
            std::vector<int> pick(ns);
            for (long q = 0; q < ns; q++) pick[q] = s.live[lcg(s.rng) % s.live.size()];
            CK(cudaMemcpyAsync(s.d_sample, pick.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, st));
            CK(cudaEventRecord(s.fork, st));
            CK(cudaStreamWaitEvent(s.side, s.fork, 0));
            float *rU[3] = {s.rU[0], s.rU[1], s.rU[2]};
            const size_t own = features_bytes(sea, g), part = grid_fill_bytes(g, sea, ns);
            rc = workspace_reserve(ws, own + part);
            Workspace side;
            side.bytes = part;
            side.base = (char *)ws.base + own;
            if (!rc) rc = grid_fill_columns(g, sea, side, s.d_sample, ns, t2, s.rETA, rU, 0, s.side);
        }
        const int rp = rc ? rc : predict_slot(s, cfg, sea, g, ws, slot, t2, carry, st);
        if (check) {
            CK(cudaEventRecord(s.join, s.side));
            CK(cudaStreamWaitEvent(st, s.join, 0));
        }
        if (rc || rp) return rc ? rc : rp;
        s.steps++;
        if (mode == 1 && ns > 0) {
            rc = compare(s, g, slot, s.d_sample, ns, 1.f / std::max(s.fmax_eta, 1e-30f),
                         1.f / std::max(s.fmax_u, 1e-30f), err, st);
            if (rc) return rc;
            double e = std::max(std::max(err[0], err[1]), std::max(err[2], err[3]));
            if (!(e <= tol)) {
                rc = grid_fill_slot(g, sea, ws, slot, t2, st);
                if (rc) return rc;
                fb = 1;
                s.fallbacks++;
                if (carry) {
                    rc = refresh_residual(s, cfg, sea, g, ws, slot, t2, true, st);
                    if (rc) return rc;
                }
            }
        }
    }
    if (fell_back) *fell_back = fb;
    if (err_out) for (int q = 0; q < 4; q++) err_out[q] = err[q];
    return grid_gradients(g, st);
}

// Plain fill of the newest slot's time into the scratch arrays and the
// normalised max errors of the grid's newest slot against it (all columns).
int surrogate_compare_newest(const Config &cfg, const DevSea &sea, DevGrid &g, Workspace &ws, double *err,
                             void *stream_) {
    (void)cfg;
    cudaStream_t st = (cudaStream_t)stream_;
    Surrogate &s = g_s;
    if (!s.ready) return E_NOT_INITIALIZED;
    int rc = attach_grid(s, g, st);
    if (rc) return rc;
    const int slot = (g.tstep + 3) % 4;
    const double t2 = g.t0 + 2 * g.dt;
    float *rU[3] = {s.rU[0], s.rU[1], s.rU[2]};
    const int *act;
    long nlive;
    grid_live_columns(g, &act, &nlive);
    const long nxy = (long)g.nx * g.ny;
    CK(cudaMemsetAsync(s.rETA, 0, sizeof(float) * nxy, st));
    for (int f = 0; f < 3; f++) CK(cudaMemsetAsync(s.rU[f], 0, sizeof(float) * nxy * g.nl, st));
    rc = grid_fill_columns(g, sea, ws, act, nlive, t2, s.rETA, rU, 0, st);
    if (rc) return rc;
    float me, mu;
    rc = slot_max(s, g, s.rETA, rU, st, &me, &mu);
    if (rc) return rc;
    return compare(s, g, slot, act, nlive, 1.f / std::max(me, 1e-30f), 1.f / std::max(mu, 1e-30f), err, st);
}

void surrogate_stats(long *steps, long *fallbacks, long *plain_steps) {
    if (steps) *steps = g_s.steps;
    if (fallbacks) *fallbacks = g_s.fallbacks;
    if (plain_steps) *plain_steps = g_s.plain_steps;
}

void surrogate_reset_stats() {
    g_s.steps = g_s.fallbacks = g_s.plain_steps = 0;
    g_s.fmax_eta = g_s.fmax_u = 0.f;
}

}  // namespace cfdwm
