// Valid 3x3 convolutions of the learned s-grid update as implicit GEMMs on
// the tcgen05 tensor cores (forward, data gradient and weight gradient).
//
//   forward      D[pixel][o]    = sum_{tap, c} x[c][pixel + tap] w[o][c][tap]
//   data grad    D[pixel][c]    = sum_{tap, o} dy[o][pixel - tap] w[o][c][tap]
//   weight grad  D[dy, c][o]    = sum_{pixel}  x[c][pixel + tap] dy[o][pixel], per dx
//
// Operand format.  Activations and gradients are kept split into BF16 hi + lo
// parts (16 significant bits, error <= 2^-17 of the value), eight channels to
// 16 bytes: [b][part][C / 8][H][W][8].  A tile of pixels with its halo is then
// one TMA box, and in shared memory every group of 8 pixels x 8 channels is a
// core matrix of the unswizzled operand layouts, whose strides the descriptors
// give: K-major (K = channels) for the forward and data-gradient GEMMs,
// MN-major (K = pixels) for the weight gradient.  A tap moves the operand by
// whole pixels, 16 bytes each, so the taps are start addresses in one copy of
// the tile: nothing is gathered, and nothing is split twice.  Zero padding
// (ragged tiles, the data gradient's border, channels past the last) is the
// boxes' out-of-range fill.
//
// The weights are BF16, so the forward and data-gradient GEMMs take two MMAs
// per K step (hi, lo) and the weight gradient, whose two operands are both
// split, three (hi hi, lo hi, hi lo); sums in FP32 in TMEM.  The first form
// of these kernels gathered each operand tile from FP32 planes with the CUDA
// cores, nine times over (issue-bound).  Network of 16 levels over a 264 x 264
// grid, the whole call: 356 us then, 61 now (11 of them the split of the input
// planes, at the memory's rate; 10 of them launch overlap).  Loss and gradient
// of eight 72 x 72 patches: 975 and 133 us.
//
// Every mbarrier wait is bounded and sets the error word when it gives up.
#include "cfdwm.h"
#include "convtc.h"
#include "tc05.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <mutex>
#include <utility>

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

constexpr int HID = CONV_HID;             // hidden channels: N of the forward and data-gradient GEMMs
constexpr int SMS = 152;
constexpr int SMEM_SM = 227 * 1024, SMEM_HALF = 112 * 1024;   // a CTA's shared memory, one or two on an SM

__device__ __forceinline__ float ct_sigmoid(float a) { return 1.f / (1.f + expf(-a)); }

// operand descriptor without swizzle: core matrices (8 rows of 16 bytes,
// contiguous) lbo bytes apart along K and sbo bytes apart along M or N
__device__ __forceinline__ uint64_t cdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr & 0x3FFFF) >> 4) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 |
           (uint64_t)1 << 46;
}

__device__ __forceinline__ void tma_4d(void *dst, const CUtensorMap *m, uint64_t *bar, int x, int y, int z, int w) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0],"
                 " [%1, {%3, %4, %5, %6}], [%2];"
                 ::"r"(su32(dst)), "l"(m), "r"(su32(bar)), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void tma_prefetch(const CUtensorMap *m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(su32(dst)), "l"(src), "r"(bytes), "r"(su32(bar)) : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(slot)), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
}

// A launch may start while the one before it in the stream drains: what
// precedes pdl_wait touches nothing that the earlier kernels write, and every
// kernel of the chain waits, so that all earlier ones are complete after it.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// FP32 planes [idx b][C][plane] to the split format; a thread per (pixel, chunk).
__global__ void __launch_bounds__(256) k_ct_split(const float *x, long xbs, const int *idx, int C, long plane,
                                                  uint4 *out) {
    pdl_next();
    pdl_wait();
    const long p = blockIdx.x * 256L + threadIdx.x;
    if (p >= plane) return;
    const int ch = blockIdx.y, nch = gridDim.y, b = blockIdx.z;
    const float *src = x + (long)(idx ? idx[b] : b) * xbs + (long)ch * 8 * plane + p;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] = ch * 8 + e < C ? src[e * plane] : 0.f;
    uint4 hi, lo;
    conv_split8(v, hi, lo);
    out[((long)(b * 2) * nch + ch) * plane + p] = hi;
    out[((long)(b * 2 + 1) * nch + ch) * plane + p] = lo;
}

// ---------------------------------------------------------------------------
// Weights: the B operands of the forward and data-gradient GEMMs,
// [16 input channels][dy][2 chunks][dx][NP][8] BF16; zero past the channels.
// ---------------------------------------------------------------------------
struct PackJobs {
    struct Job {
        long w, out, end;        // first weight and output element; end of the job's elements
        int K, N, NP, sk, sn;    // channels along K and N, padded N, their weight strides
        int flip;                // data gradient: the taps run backwards
    } j[CONV_MAX_PACK];
    int n;
};

__global__ void __launch_bounds__(256) k_ct_pack(PackJobs jobs, const float *w, __nv_bfloat16 *out) {
    const long e = blockIdx.x * 256L + threadIdx.x;
    int q = 0;
    while (q < jobs.n && e >= jobs.j[q].end) q++;
    if (q == jobs.n) return;
    const PackJobs::Job &j = jobs.j[q];
    const long i = e - j.out;
    const int c8 = (int)(i & 7), n = (int)(i / 8 % j.NP), dx = (int)(i / (8L * j.NP) % 3);
    const int kc = (int)(i / (24L * j.NP) % 2), dy = (int)(i / (48L * j.NP) % 3), st = (int)(i / (144L * j.NP));
    const int k = (st * 2 + kc) * 8 + c8, tap = dy * 3 + dx;
    float v = 0.f;
    if (k < j.K && n < j.N) v = w[j.w + (long)k * j.sk + (long)n * j.sn + (j.flip ? 8 - tap : tap)];
    out[e] = __float2bfloat16_rn(v);
}

// ---------------------------------------------------------------------------
// Forward and data gradient
// ---------------------------------------------------------------------------
enum { CT_HIDDEN = 0, CT_OUTPUT = 1, CT_DATA = 2, CT_LOSS = 3 };

// M = 128: 8 rows of 16 pixels, or 4 of 32.  An MMA costs about 33 + N / 2 cycles
// here (its 4 KB of A from shared memory, measured with N = 32 and 64), so the
// three dx of a kernel row share one MMA with N = 3 NP on the unshifted pixels,
// and the epilogue adds the neighbouring pixels' columns: 81 cycles for what
// takes 3 x 49 with a shifted operand per tap, less the two columns of a row
// that give no output.
template <int FW> struct Tile {
    static constexpr int W = FW, X = FW - 2, Y = 128 / FW;           // patch width, output tile
    static constexpr int CHUNK = (Y + 2) * W * 16;                   // bytes of 8 channels' patch
    static constexpr int PART = 2 * CHUNK, STAGE = 2 * PART;         // 16 channels, hi and lo
};
constexpr int FRING = 6;                             // stages in flight at most
constexpr int F_THREADS = 320;
constexpr int FHEAD = 256 + 4 * 64 * 4 + 32;         // barriers and flags, bias and loss sums

struct ConvArgs {
    const uint8_t *w;            // packed weights
    const float *bias;           // HIDDEN, OUTPUT, LOSS
    const float4 *ds;            // DATA: silu' of the layer's pre-activation [b][HID / 4][Ho][Wo]
    float4 *ds_out;              // HIDDEN: the same, or null
    uint4 *ys;                   // HIDDEN: activations, DATA, LOSS: gradient, split format
    float *y;                    // OUTPUT: planes [b][O][Ho][Wo]
    float *bpart;                // DATA, LOSS: sums of the CTA's gradients [CTA][NP]
    const float *tg;             // LOSS: targets, their batch stride and samples (ConvLoss)
    long tbs;
    const int *idx;
    float w0, inv_norm;
    float *lpart;                // LOSS: the CTA's share
    int nst, ring;               // K stages of 16 channels; stage buffers
    int origin;                  // of the patch relative to the tile: 0, data gradient -2
    int O, Ho, Wo, tiles_x, tiles_img, ntiles;
    int *err;
};

template <int NP> struct CtCfg {
    static constexpr int N = 3 * NP;
    static constexpr int WSTAGE = 3 * 2 * N * 16;    // weights of a K stage
    static constexpr int NACC = NP == 32 ? 2 : 1;    // accumulators, so that two CTAs fit an SM's TMEM
    static constexpr uint32_t ACOLS = NP == 32 ? 128 : 256, TCOLS = NACC * ACOLS;
};

// A persistent CTA, two on an SM: the weights stay in shared memory, warp 0
// copies patches through a ring of stages, warp 1 issues the MMAs, warps 2 to 9
// (two to a lane quarter, half of the channels each) make the epilogue of one
// tile while the next one accumulates.
template <int NP, int EPI, int FW>
__global__ void __launch_bounds__(F_THREADS, 2) k_conv(const __grid_constant__ CUtensorMap xm, ConvArgs a) {
    using CF = CtCfg<NP>;
    using T = Tile<FW>;
    extern __shared__ __align__(128) uint8_t ct_raw[];
    uint8_t *wsm = (uint8_t *)(((uintptr_t)ct_raw + 127) & ~(uintptr_t)127);
    uint8_t *asm_ = wsm + a.nst * CF::WSTAGE;
    uint64_t *full = (uint64_t *)(asm_ + a.ring * T::STAGE), *empty = full + FRING, *wfull = empty + FRING;
    uint64_t *afull = wfull + 1, *aempty = afull + 2;
    uint32_t *tslot = (uint32_t *)(aempty + 2);
    volatile int *fail = (volatile int *)(tslot + 1);
    float *red = (float *)(full + 32);                // DATA, LOSS: [4][NP], then [8]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int q = 0; q < 2 * FRING + 3; q++) mbar_init(full + q, 1);
        for (int q = 0; q < 2; q++) mbar_init(aempty + q, 8);
        *fail = 0;
        tma_prefetch(&xm);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(tslot, CF::TCOLS);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;
    pdl_next();
    float bs[NP / 32] = {}, ls = 0.f;

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(wfull, a.nst * CF::WSTAGE);
            for (int s = 0; s < a.nst; s++)
                bulk_load(wsm + s * CF::WSTAGE, a.w + (long)s * CF::WSTAGE, CF::WSTAGE, wfull);
            pdl_wait();
            int k = 0, buf = 0;                       // stages copied
            uint32_t par = 1;                         // of the stage buffer's last release
            bool ok = true;
            for (int t = blockIdx.x; ok && t < a.ntiles; t += gridDim.x) {
                const int b = t / a.tiles_img, r = t - b * a.tiles_img, ty = r / a.tiles_x;
                const int x0 = (r - ty * a.tiles_x) * T::X + a.origin, y0 = ty * T::Y + a.origin;
                for (int s = 0; s < a.nst; s++, k++) {
                    if (k >= a.ring && !mbar_wait(empty + buf, par, a.err, 11)) { ok = false; break; }
                    mbar_expect_tx(full + buf, T::STAGE);
                    tma_4d(asm_ + buf * T::STAGE, &xm, full + buf, x0 * 8, y0, s * 2, b * 2);
                    if (++buf == a.ring) { buf = 0; par ^= 1; }
                }
            }
            if (!ok) {
                *fail = 1;                            // let the copies in flight land
                for (int q = max(0, k - a.ring); q < k; q++)
                    mbar_wait(full + q % a.ring, (uint32_t)((q / a.ring) & 1), a.err, 11);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(CF::N >> 3) << 17) | (8u << 24);
            const uint32_t W = su32(wsm);
            bool ok = mbar_wait(wfull, 0u, a.err, 12);
            int buf = 0, acc = 0, i = 0;              // stage buffer, accumulator, tiles
            uint32_t par = 0, apar = 1;
            for (int t = blockIdx.x; ok && t < a.ntiles; t += gridDim.x, i++) {
                if (i >= CF::NACC && !mbar_wait(aempty + acc, apar, a.err, 13)) { ok = false; break; }
                const uint32_t d = tmem + acc * CF::ACOLS;
                for (int s = 0; s < a.nst; s++) {
                    if (!mbar_wait(full + buf, par, a.err, 14)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t da = cdesc(su32(asm_ + buf * T::STAGE), T::CHUNK, 128);
                    const uint64_t db = cdesc(W + s * CF::WSTAGE, CF::N * 16, 128);
#pragma unroll
                    for (int dy = 0; dy < 3; dy++) {
                        const uint64_t oa = (uint64_t)((dy * FW * 16) >> 4), ob = (uint64_t)((dy * 2 * CF::N * 16) >> 4);
                        umma(d, da + oa, db + ob, idesc, (s | dy) ? 1u : 0u);
                        umma(d, da + oa + (T::PART >> 4), db + ob, idesc, 1u);
                    }
                    umma_commit(empty + buf);
                    if (++buf == a.ring) { buf = 0; par ^= 1; }
                }
                if (ok) umma_commit(afull + acc);
                if (++acc == CF::NACC) { acc = 0; apar ^= 1; }
            }
            if (!ok) *fail = 1;
        }
    } else {
        pdl_wait();
        const int q = warp & 3, hf = (warp - 2) >> 2; // TMEM lane quarter, half of the channels
        const int m = q * 32 + lane;                  // row of D
        const int col = m & (FW - 1);
        const long plane = (long)a.Ho * a.Wo;
        int acc = 0;
        uint32_t par = 0;
        for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
            bool ok = mbar_wait(afull + acc, par, a.err, 15);
            if (!__all_sync(0xffffffffu, ok)) { *fail = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + acc * CF::ACOLS;
            const int b = t / a.tiles_img, r = t % a.tiles_img;
            const int oy = (r / a.tiles_x) * T::Y + (m / FW), ox = (r % a.tiles_x) * T::X + col;
            const long pix = (long)oy * a.Wo + ox;
            const bool live = col < T::X && oy < a.Ho && ox < a.Wo;
#pragma unroll
            for (int k = 0; k < NP / 32; k++) {
                const int h = hf * (NP / 32) + k;
                // the epilogue's inputs first, all in flight
                float in[16];
                if (EPI == CT_DATA) {
#pragma unroll
                    for (int f = 0; f < 4; f++) {
                        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (live) w = a.ds[((long)b * (HID / 4) + h * 4 + f) * plane + pix];
                        in[f * 4] = w.x; in[f * 4 + 1] = w.y; in[f * 4 + 2] = w.z; in[f * 4 + 3] = w.w;
                    }
                } else if (EPI == CT_LOSS) {
                    const float *tg = a.tg + (long)(live && a.idx ? a.idx[b] : b) * a.tbs + pix;
#pragma unroll
                    for (int n = 0; n < 16; n++) in[n] = live && h * 16 + n < a.O ? tg[(h * 16 + n) * plane] : 0.f;
                }
                float d[16], e1[16], e2[16];
                tmem_ld16x3(ta + h * 16, NP, d, e1, e2);
                if (k == NP / 32 - 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(aempty + acc);
                    if (++acc == CF::NACC) { acc = 0; par ^= 1; }
                }
#pragma unroll
                for (int n = 0; n < 16; n++)
                    d[n] += __shfl_down_sync(0xffffffffu, e1[n], 1) + __shfl_down_sync(0xffffffffu, e2[n], 2);
                if (EPI == CT_LOSS) {
                    // L = sum w_o (y - t)^2 inv_norm, dy = 2 w_o (y - t) inv_norm
#pragma unroll
                    for (int n = 0; n < 16; n++) {
                        const int o = h * 16 + n;
                        const float wo = o == 0 ? a.w0 : 1.f;
                        const float df = live && o < a.O ? d[n] + a.bias[o] - in[n] : 0.f;
                        ls += wo * df * df * a.inv_norm;
                        d[n] = 2.f * wo * df * a.inv_norm;
                    }
                    const int nco = (a.O + 7) / 8;
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        if (!live || h * 2 + c >= nco) break;
                        uint4 hi, lo;
                        conv_split8(d + c * 8, hi, lo);
                        a.ys[((long)(b * 2) * nco + h * 2 + c) * plane + pix] = hi;
                        a.ys[((long)(b * 2 + 1) * nco + h * 2 + c) * plane + pix] = lo;
                    }
                }
                if (EPI == CT_OUTPUT) {
                    if (live)
#pragma unroll
                        for (int n = 0; n < 16; n++)
                            if (h * 16 + n < a.O)
                                a.y[((long)b * a.O + h * 16 + n) * plane + pix] = d[n] + a.bias[h * 16 + n];
                }
#pragma unroll
                for (int c = 0; c < (EPI == CT_OUTPUT || EPI == CT_LOSS ? 0 : 2); c++) {
                    float *v = d + c * 8, g[8];
                    const int ch = h * 2 + c;                     // channel chunk
                    if (EPI == CT_DATA) {
#pragma unroll
                        for (int e = 0; e < 8; e++) v[e] = live ? v[e] * in[c * 8 + e] : 0.f;
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            const float p = v[e] + a.bias[ch * 8 + e], sg = ct_sigmoid(p);
                            v[e] = p * sg;
                            g[e] = sg * (1.f + p * (1.f - sg));
                        }
                    }
                    if (!live) continue;
                    uint4 hi, lo;
                    conv_split8(v, hi, lo);
                    a.ys[((long)(b * 2) * (HID / 8) + ch) * plane + pix] = hi;
                    a.ys[((long)(b * 2 + 1) * (HID / 8) + ch) * plane + pix] = lo;
                    if (EPI == CT_HIDDEN && a.ds_out)
#pragma unroll
                        for (int f = 0; f < 2; f++)
                            a.ds_out[((long)b * (HID / 4) + ch * 2 + f) * plane + pix] =
                                make_float4(g[f * 4], g[f * 4 + 1], g[f * 4 + 2], g[f * 4 + 3]);
                }
                if (EPI == CT_DATA || EPI == CT_LOSS) {
                    // the bias gradient's share: lane n ends with channel n of the warp's pixels
#pragma unroll
                    for (int o = 8; o >= 1; o >>= 1) {
                        const bool up = lane & o;
#pragma unroll
                        for (int n = 0; n < o; n++) {
                            const float send = up ? d[n] : d[n + o], keep = up ? d[n + o] : d[n];
                            d[n] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                        }
                    }
                    bs[k] += d[0] + __shfl_xor_sync(0xffffffffu, d[0], 16);
                }
            }
        }
        if ((EPI == CT_DATA || EPI == CT_LOSS) && lane < 16)
#pragma unroll
            for (int k = 0; k < NP / 32; k++) red[q * NP + (hf * (NP / 32) + k) * 16 + lane] = bs[k];
        if (EPI == CT_LOSS) {
            for (int o = 16; o >= 1; o >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, o);
            if (lane == 0) red[4 * NP + warp - 2] = ls;
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if ((EPI == CT_DATA || EPI == CT_LOSS) && tid < NP && !*fail) {
        a.bpart[(long)blockIdx.x * NP + tid] = (red[tid] + red[NP + tid]) + (red[2 * NP + tid] + red[3 * NP + tid]);
        if (EPI == CT_LOSS && tid == 0) {
            float l = 0.f;
            for (int k = 0; k < 8; k++) l += red[4 * NP + k];
            a.lpart[blockIdx.x] = l;
        }
    }
    if (warp == 0) tmem_free(tmem, CF::TCOLS);
}

// ---------------------------------------------------------------------------
// Weight gradient
// ---------------------------------------------------------------------------
constexpr int TX = 8, TY = 16;            // pixel tile: K = 128, a core matrix per tile row
constexpr int PX = TX + 2;                // width of the patch
constexpr int QCHUNK = TX * TY * 16;      // bytes of 8 channels of the plain tile
constexpr int W_THREADS = 256;
constexpr int W_UNITS = 12;               // (layer, M tile, N block) triples of a launch at most
constexpr int WHEAD = 128;

struct WgtUnit {
    float *part;                 // [slab][dx][q][3 P]: the slabs' sums
    int layer;                   // tensor maps
    int nch, rows;               // P's chunks, patch rows copied
    int g0, q0, N, Q;            // first row group, first q chunk, N of the MMAs, q channels in all
    int origin;                  // of the patch relative to the tile: 0, or -2 (P is dy)
    int ntiles, tiles_x, tiles_img;
    int nslab, end;              // CTAs; end of the unit's blocks
};

struct WgtArgs {
    CUtensorMap p[4], q[4];
    WgtUnit u[W_UNITS];
    int *err;
};

// All layers in one launch, a CTA per SM.  D's rows are (t, p): with the patch
// of P copied as [row][chunk][pixel], the row groups of 8 channels over the
// three kernel rows t and the chunks are one arithmetic progression of
// addresses, so M = 128 holds 16 of them (the kernel rows of 32 channels, and
// a fourth that is not kept).  dx is a start address, with an accumulator of
// its own; N are Q's channels, K the tile's pixels, two tile rows per MMA.
// P is x and Q dy, or, where x has more channels, the other way round (taps
// then run backwards): the layer with 128 inputs needs one M tile instead of
// three, 97 cycles an MMA (33 + N / 2) instead of 3 x 49.
// A CTA sums its slab (every nslab-th tile) in TMEM; the slabs are summed in
// order afterwards, so the result is deterministic.  The CTAs are divided
// between the units by their MMA cycles.
__global__ void __launch_bounds__(W_THREADS) k_conv_wgt(const __grid_constant__ WgtArgs a) {
    extern __shared__ __align__(128) uint8_t ct_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)ct_raw + 127) & ~(uintptr_t)127);
    uint64_t *full = (uint64_t *)smem, *empty = full + 2, *done = full + 4;
    uint32_t *tslot = (uint32_t *)(full + 5);
    volatile int *fail = (volatile int *)(full + 6);
    smem += WHEAD;
    const int tid = threadIdx.x, warp = tid >> 5;
    int ui = 0;
    while ((int)blockIdx.x >= a.u[ui].end) ui++;
    const WgtUnit &u = a.u[ui];
    const int slab = (int)blockIdx.x - (u.end - u.nslab);
    const int r0 = u.g0 / u.nch, ppart = u.rows * u.nch * PX * 16, pbytes = (2 * ppart + 127) & ~127;
    const int qpart = (u.N / 8) * QCHUNK, stage = pbytes + 2 * qpart;
    if (tid == 0) {
        for (int k = 0; k < 5; k++) mbar_init(full + k, 1);
        *fail = 0;
        tma_prefetch(&a.p[u.layer]);
        tma_prefetch(&a.q[u.layer]);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(tslot, 512);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;
    pdl_next();
    pdl_wait();

    if (tid == 0) {
        const CUtensorMap *pm = &a.p[u.layer], *qm = &a.q[u.layer];
        int k = 0;
        bool ok = true;
        for (int t = slab; t < u.ntiles; t += u.nslab, k++) {
            const int buf = k & 1;
            if (k > 1 && !mbar_wait(empty + buf, (uint32_t)(((k >> 1) - 1) & 1), a.err, 21)) { ok = false; break; }
            const int b = t / u.tiles_img, r = t % u.tiles_img;
            const int x0 = (r % u.tiles_x) * TX, y0 = (r / u.tiles_x) * TY;
            uint8_t *st = smem + buf * stage;
            mbar_expect_tx(full + buf, 2 * ppart + 2 * qpart);
            tma_4d(st, pm, full + buf, (x0 + u.origin) * 8, 0, y0 + u.origin + r0, b * 2);
            tma_4d(st + pbytes, qm, full + buf, x0 * 8, y0, u.q0, b * 2);
        }
        if (!ok) {
            *fail = 1;                                // let the copies in flight land
            for (int j = max(0, k - 2); j < k; j++) mbar_wait(full + (j & 1), (uint32_t)((j >> 1) & 1), a.err, 21);
        }
    } else if (tid == 32) {
        // both operands MN-major (bits 15 and 16)
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                               ((uint32_t)(u.N >> 3) << 17) | (8u << 24);
        int k = 0;
        bool ok = true;
        for (int t = slab; t < u.ntiles; t += u.nslab, k++) {
            const int buf = k & 1;
            if (!mbar_wait(full + buf, (uint32_t)((k >> 1) & 1), a.err, 22)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t P = su32(smem + buf * stage), Q = P + pbytes, rowb = (uint32_t)u.nch * PX * 16;
            const uint64_t dp = cdesc(P + (uint32_t)(u.g0 - r0 * u.nch) * PX * 16, rowb, PX * 16);
            const uint64_t dq = cdesc(Q, TX * 16, QCHUNK);
            const uint64_t lp = (uint64_t)(ppart >> 4), lq = (uint64_t)(qpart >> 4);
            for (int y = 0; y < TY; y += 2)
                for (int dx = 0; dx < 3; dx++) {
                    const uint64_t op = (uint64_t)((y * rowb + dx * 16) >> 4), oq = (uint64_t)((y * TX * 16) >> 4);
                    const uint32_t d = tmem + dx * u.N;
                    umma(d, dp + op, dq + oq, idesc, (k | y) ? 1u : 0u);
                    umma(d, dp + op + lp, dq + oq, idesc, 1u);
                    umma(d, dp + op, dq + oq + lq, idesc, 1u);
                }
            umma_commit(empty + buf);
        }
        if (!ok) *fail = 1;
        umma_commit(done);
    }
    __syncwarp();
    bool ok = mbar_wait(done, 0u, a.err, 23);
    ok = !__syncthreads_or(!ok) && !*fail;
    if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // warp w reads lane quarter w % 4, every other 16 columns
        const int row = u.g0 * 8 + (tid & 127), nrow = 3 * u.nch * 8, nq = min(u.N, u.Q - u.q0 * 8);
        const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        for (int dx = 0; dx < 3; dx++) {
            float *out = u.part + (((long)slab * 3 + dx) * u.Q + u.q0 * 8) * nrow + row;
            for (int h = (warp >> 2) * 16; h < u.N; h += 32) {
                float d[16];
                tmem_ld16(ta + dx * u.N + h, d);
                if (row < nrow)
#pragma unroll
                    for (int n = 0; n < 16; n++)
                        if (h + n < nq) out[(h + n) * nrow] = d[n];
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 512);
}

// Sums of the slabs' partial results, all layers in one launch: 32 elements
// per block, 32 interleaved shares of the slabs, added in a fixed order.
struct SumJobs {
    struct Job {
        const float *part;
        float *out;
        long n, stride;          // elements, and the distance of two slabs
        int nslab, P, Q, swap;   // P > 0: [dx][q][t p] to [o][c][dy dx]
        unsigned end;            // end of the job's blocks
    } j[CONV_MAX_SUMS];
    int n;
};

__global__ void __launch_bounds__(256) k_ct_sum(SumJobs jobs) {
    __shared__ float4 part[32][8];
    __shared__ float red[8][32];
    pdl_next();
    pdl_wait();
    int q = 0;
    while (blockIdx.x >= jobs.j[q].end) q++;
    const SumJobs::Job &j = jobs.j[q];
    const long e0 = (long)(blockIdx.x - (q ? jobs.j[q - 1].end : 0)) * 32;
    {
        const int v = threadIdx.x & 7, w = threadIdx.x >> 3;     // four elements, share
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e0 + v * 4 < j.n) {
#pragma unroll 4
            for (int k = w; k < j.nslab; k += 32) {
                const float4 f = *reinterpret_cast<const float4 *>(j.part + k * j.stride + e0 + v * 4);
                s.x += f.x; s.y += f.y; s.z += f.z; s.w += f.w;
            }
        }
        part[w][v] = s;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long e = e0 + lane;
    const float *ps = reinterpret_cast<const float *>(&part[w * 4][0]) + lane;
    red[w][lane] = (ps[0] + ps[32]) + (ps[64] + ps[96]);
    __syncthreads();
    if (w || e >= j.n) return;
    float s = red[0][lane];
    for (int k = 1; k < 8; k++) s += red[k][lane];
    long o = e;
    if (j.P > 0) {
        const int i = (int)e, p = i % j.P, tc = i / j.P, t = tc % 3, cd = tc / 3, c = cd % j.Q, dx = cd / j.Q;
        o = j.swap ? ((long)p * j.Q + c) * 9 + (2 - t) * 3 + 2 - dx : ((long)c * j.P + p) * 9 + t * 3 + dx;
    }
    j.out[o] = s;
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled ct_encode() {
    static const EncodeTiled fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess || q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (EncodeTiled)p;
    }();
    return fn;
}

// The split activations [2 B][nch][H][W][8] as a 4-D map whose boxes are bx
// pixels wide.  chunk_inner: dimensions (pixel, chunk, row, part) instead of
// (pixel, row, chunk, part).
int ct_map(CUtensorMap *m, const void *base, int B, int nch, int H, int W, bool chunk_inner, int bx, int brows,
           int bch) {
    EncodeTiled enc = ct_encode();
    if (!enc) return E_CUDA;
    const cuuint64_t row = (cuuint64_t)W * 16, chunk = row * H;
    cuuint64_t dims[4] = {(cuuint64_t)W * 8, (cuuint64_t)H, (cuuint64_t)nch, (cuuint64_t)B * 2};
    cuuint64_t strides[3] = {row, chunk, chunk * nch};
    cuuint32_t box[4] = {(cuuint32_t)bx * 8, (cuuint32_t)brows, (cuuint32_t)bch, 2};
    cuuint32_t es[4] = {1, 1, 1, 1};
    if (chunk_inner) {
        std::swap(dims[1], dims[2]);
        std::swap(strides[0], strides[1]);
        std::swap(box[1], box[2]);
    }
    const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(base), dims, strides, box, es,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? OK : E_CUDA;
}

std::mutex g_ct_mtx;          // serialises the lazy allocation of the error word
int *g_ct_err = nullptr;      // error word of the bounded waits: mapped host memory, read after a
                              // synchronisation without a copy

int ct_err_word(int **p) {
    std::lock_guard<std::mutex> lk(g_ct_mtx);
    if (!g_ct_err) {
        CK(cudaHostAlloc(&g_ct_err, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
        *g_ct_err = 0;
    }
    CK(cudaHostGetDevicePointer(p, g_ct_err, 0));
    return OK;
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }

// a launch that may start while the kernel before it drains (pdl_wait)
template <class... P, class... A>
int launch_pdl(void (*kern)(P...), dim3 grid, int threads, int smem, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = (size_t)smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    CK(cudaLaunchKernelEx(&c, kern, std::forward<A>(args)...));
    note_launch();
    return OK;
}

int conv_ctas(int ntiles) { return std::min(ntiles, 2 * SMS); }

// Tiles of B output planes.  32 pixels wide where that takes fewer rounds of the
// resident CTAs: the network of 264 x 264 has 627 tiles of 14 x 8 outputs a layer, a
// third round for 19 of them, and 594 of 30 x 4: first layer 16.2 and 14.7 us, the
// next two 10.8 and 9.9.  Otherwise 16, whose halo is smaller and which suits small
// planes (70 pixels are 5 tiles of 14, 3 of 30).
struct ConvTiles {
    int fw, tx, img, n;
};
ConvTiles conv_tiles(int B, int Ho, int Wo) {
    auto make = [&](int fw) {
        ConvTiles t;
        t.fw = fw;
        t.tx = ceil_div(Wo, fw - 2);
        t.img = t.tx * ceil_div(Ho, 128 / fw);
        t.n = B * t.img;
        return t;
    };
    const ConvTiles a = make(16), b = make(32);
    return ceil_div(b.n, 2 * SMS) < ceil_div(a.n, 2 * SMS) ? b : a;
}

template <int NP, int EPI, int FW>
int launch_conv_t(const CUtensorMap &m, ConvArgs &a, cudaStream_t st) {
    constexpr int STAGE = Tile<FW>::STAGE;
    const int wbytes = a.nst * CtCfg<NP>::WSTAGE, head = wbytes + FHEAD + 128;
    // two CTAs on an SM where the weights leave room for three stages each
    const int room = head + 3 * STAGE <= SMEM_HALF ? SMEM_HALF : SMEM_SM;
    a.ring = std::min(FRING, (room - head) / STAGE);
    if (a.ring < 1) return E_UNSUPPORTED;
    static const cudaError_t attr =
        cudaFuncSetAttribute(k_conv<NP, EPI, FW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_SM);
    CK(attr);
    return launch_pdl(k_conv<NP, EPI, FW>, dim3((unsigned)conv_ctas(a.ntiles)), F_THREADS, head + a.ring * STAGE, st, m,
                      a);
}

// The convolution of split inputs xs (K channels, H x W) to Ho x Wo outputs.
template <int NP, int EPI>
int launch_conv(ConvArgs &a, const void *xs, int B, int K, int H, int W, cudaStream_t st) {
    const ConvTiles t = conv_tiles(B, a.Ho, a.Wo);
    a.nst = ceil_div(K, 16);
    a.tiles_x = t.tx;
    a.tiles_img = t.img;
    a.ntiles = t.n;
    int rc = ct_err_word(&a.err);
    if (rc) return rc;
    CUtensorMap m;
    if ((rc = ct_map(&m, xs, B, ceil_div(K, 8), H, W, false, t.fw, 128 / t.fw + 2, 2))) return rc;
    return t.fw == 32 ? launch_conv_t<NP, EPI, 32>(m, a, st) : launch_conv_t<NP, EPI, 16>(m, a, st);
}

}  // namespace

size_t conv_split_bytes(int B, int C, int H, int W) { return (size_t)B * 2 * ((C + 7) / 8) * H * W * 16; }

int conv_split(const float *x, long xbs, const int *idx, int B, int C, int H, int W, void *xs, void *stream) {
    const long plane = (long)H * W;
    const dim3 grid((unsigned)((plane + 255) / 256), (unsigned)((C + 7) / 8), (unsigned)B);
    // an ordinary launch: the kernels that may overlap it read the weights
    // before their pdl_wait, so everything earlier has to be complete
    k_ct_split<<<grid, 256, 0, (cudaStream_t)stream>>>(x, xbs, idx, C, plane, (uint4 *)xs);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

long conv_pack_elems(int K, int N) { return (long)ceil_div(K, 16) * 144 * (N <= 32 ? 32 : 64); }

int conv_pack(const ConvPack *jobs, int n, const float *w, void *out, void *stream) {
    PackJobs p = {};
    p.n = n;
    long end = 0;
    for (int q = 0; q < n; q++) {
        PackJobs::Job &j = p.j[q];
        const ConvPack &c = jobs[q];
        const int C = c.C, O = c.O;
        j.w = c.w;
        j.out = end;
        j.flip = c.data ? 1 : 0;
        j.K = c.data ? O : C;
        j.N = c.data ? C : O;
        j.NP = j.N <= 32 ? 32 : 64;
        j.sk = (c.data ? C : 1) * 9;
        j.sn = (c.data ? 1 : C) * 9;
        j.end = end += conv_pack_elems(j.K, j.N);
    }
    k_ct_pack<<<(unsigned)((end + 255) / 256), 256, 0, (cudaStream_t)stream>>>(p, w, (__nv_bfloat16 *)out);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

int conv_hidden(const void *xs, const void *wp, const float *bias, int B, int C, int H, int W, void *ys, void *ds,
                void *stream) {
    if (C < 1 || H < 3 || W < 3 || B < 1) return E_BAD_ARGUMENT;
    ConvArgs a = {};
    a.w = (const uint8_t *)wp; a.Ho = H - 2; a.Wo = W - 2;
    a.bias = bias; a.ys = (uint4 *)ys; a.ds_out = (float4 *)ds;
    return launch_conv<32, CT_HIDDEN>(a, xs, B, C, H, W, (cudaStream_t)stream);
}

int conv_output(const void *xs, const void *wp, const float *bias, int B, int C, int O, int H, int W, float *y,
                void *stream) {
    if (O < 1 || O > 64 || C < 1 || H < 3 || W < 3 || B < 1) return E_BAD_ARGUMENT;
    ConvArgs a = {};
    a.w = (const uint8_t *)wp; a.Ho = H - 2; a.Wo = W - 2;
    a.bias = bias; a.y = y; a.O = O;
    return O <= 32 ? launch_conv<32, CT_OUTPUT>(a, xs, B, C, H, W, (cudaStream_t)stream)
                   : launch_conv<64, CT_OUTPUT>(a, xs, B, C, H, W, (cudaStream_t)stream);
}

int conv_loss(const void *xs, const void *wp, const float *bias, int B, int C, int O, int H, int W,
              const ConvLoss &l, void *dys, float *bpart, float *lpart, void *stream) {
    if (O < 1 || O > 64 || C < 1 || H < 3 || W < 3 || B < 1) return E_BAD_ARGUMENT;
    ConvArgs a = {};
    a.w = (const uint8_t *)wp; a.Ho = H - 2; a.Wo = W - 2;
    a.bias = bias; a.O = O; a.ys = (uint4 *)dys; a.bpart = bpart; a.lpart = lpart;
    a.tg = l.tg; a.tbs = l.tbs; a.idx = l.idx; a.w0 = l.w0; a.inv_norm = l.inv_norm;
    return O <= 32 ? launch_conv<32, CT_LOSS>(a, xs, B, C, H, W, (cudaStream_t)stream)
                   : launch_conv<64, CT_LOSS>(a, xs, B, C, H, W, (cudaStream_t)stream);
}

int conv_bias_parts(int B, int H, int W) { return conv_ctas(conv_tiles(B, H, W).n); }

int conv_data_grad(const void *dys, const void *wp, const void *ds, int B, int O, int H, int W, void *dxs,
                   float *bpart, void *stream) {
    if (O < 1 || H < 3 || W < 3 || B < 1) return E_BAD_ARGUMENT;
    ConvArgs a = {};
    a.w = (const uint8_t *)wp; a.origin = -2; a.Ho = H; a.Wo = W;
    a.ds = (const float4 *)ds; a.ys = (uint4 *)dxs; a.bpart = bpart;
    return launch_conv<32, CT_DATA>(a, dys, B, O, H - 2, W - 2, (cudaStream_t)stream);
}

// The units of the layers' weight gradients and their CTAs.
static int wgt_units(ConvWgt *l, int n, int B, WgtUnit *u, int *smem) {
    int nu = 0;
    double cost[W_UNITS], total = 0.0;
    *smem = 0;
    for (int i = 0; i < n; i++) {
        if (l[i].O < 1 || l[i].O > 64 || l[i].C < 8 || l[i].C % 8) return E_BAD_ARGUMENT;
        l[i].swap = 3 * l[i].C > 128 && l[i].O == HID;      // more than one M tile otherwise
        const int P = l[i].swap ? l[i].O : l[i].C, Q = l[i].swap ? l[i].C : l[i].O, nch = P / 8;
        const int H = l[i].swap ? l[i].H : l[i].H - 2, W = l[i].swap ? l[i].W : l[i].W - 2;   // Q's planes
        int span = 0;
        for (int g = 0; g < 3 * nch; g += 16) span = std::max(span, (g + 15) / nch - g / nch);
        for (int g = 0; g < 3 * nch; g += 16)
            for (int q0 = 0; q0 < ceil_div(Q, 8); q0 += 16, nu++) {
                if (nu == W_UNITS) return E_UNSUPPORTED;
                WgtUnit &v = u[nu];
                v = {};
                v.layer = i;
                v.nch = nch;
                v.rows = TY + span;
                v.g0 = g;
                v.q0 = q0;
                v.N = std::min(128, ceil_div(Q, 16) * 16);
                v.Q = Q;
                v.origin = l[i].swap ? -2 : 0;
                v.tiles_x = ceil_div(W, TX);
                v.tiles_img = v.tiles_x * ceil_div(H, TY);
                v.ntiles = B * v.tiles_img;
                *smem = std::max(*smem, 2 * (((2 * v.rows * nch * PX * 16 + 127) & ~127) + 2 * (v.N / 8) * QCHUNK));
                total += cost[nu] = (33.0 + 0.5 * v.N) * v.ntiles;
            }
    }
    *smem += WHEAD + 128;
    int end = 0;
    for (int k = 0; k < nu; k++) {
        // the units of a layer have the same slabs
        u[k].nslab = k && u[k].layer == u[k - 1].layer
                         ? u[k - 1].nslab
                         : std::min(u[k].ntiles, std::max(1, (int)(SMS * cost[k] / total)));
        u[k].end = end += u[k].nslab;
        l[u[k].layer].nslab = u[k].nslab;
    }
    return *smem <= SMEM_SM ? nu : E_UNSUPPORTED;
}

int conv_wgt_plan(ConvWgt *l, int n, int B) {
    WgtUnit u[W_UNITS];
    int smem;
    const int nu = wgt_units(l, n, B, u, &smem);
    return nu < 0 ? nu : OK;
}

int conv_weight_grads(ConvWgt *l, int n, int B, void *stream) {
    if (n < 1 || n > 4) return E_BAD_ARGUMENT;
    WgtArgs a = {};
    int smem;
    const int nu = wgt_units(l, n, B, a.u, &smem);
    if (nu < 0) return nu;
    int rc = ct_err_word(&a.err);
    if (rc) return rc;
    for (int k = 0; k < nu; k++) a.u[k].part = l[a.u[k].layer].part;
    for (int i = 0; i < n; i++) {
        const ConvWgt &c = l[i];
        int k = 0;
        while (a.u[k].layer != i) k++;
        const WgtUnit &v = a.u[k];
        const int cc = c.C / 8, co = ceil_div(c.O, 8), H = c.H, W = c.W;
        rc = c.swap ? ct_map(&a.p[i], c.dys, B, co, H - 2, W - 2, true, PX, v.rows, co)
                    : ct_map(&a.p[i], c.xs, B, cc, H, W, true, PX, v.rows, cc);
        if (rc) return rc;
        rc = c.swap ? ct_map(&a.q[i], c.xs, B, cc, H, W, false, TX, TY, v.N / 8)
                    : ct_map(&a.q[i], c.dys, B, co, H - 2, W - 2, false, TX, TY, v.N / 8);
        if (rc) return rc;
    }
    static const cudaError_t attr =
        cudaFuncSetAttribute(k_conv_wgt, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_SM);
    CK(attr);
    return launch_pdl(k_conv_wgt, dim3((unsigned)a.u[nu - 1].end), W_THREADS, smem, (cudaStream_t)stream, a);
}

int conv_sums(const ConvSum *jobs, int n, void *stream) {
    SumJobs p = {};
    p.n = n;
    unsigned end = 0;
    for (int q = 0; q < n; q++) {
        const ConvSum &c = jobs[q];
        SumJobs::Job &j = p.j[q];
        j.part = c.part; j.out = c.out; j.n = c.n; j.stride = c.stride; j.nslab = c.nslab;
        if (c.wgt) {
            j.swap = c.wgt->swap;
            j.P = j.swap ? c.wgt->O : c.wgt->C;
            j.Q = j.swap ? c.wgt->C : c.wgt->O;
        }
        j.end = end += (unsigned)((c.n + 31) / 32);
    }
    return launch_pdl(k_ct_sum, dim3(end), 256, 0, (cudaStream_t)stream, p);
}

// Loads the kernels (the first launch of each would otherwise).
int conv_load() {
    static const cudaError_t rc = [] {
        const void *k[] = {(const void *)k_ct_split, (const void *)k_ct_pack, (const void *)k_ct_sum,
                           (const void *)k_conv_wgt, (const void *)k_conv<32, CT_HIDDEN, 16>,
                           (const void *)k_conv<32, CT_OUTPUT, 16>, (const void *)k_conv<64, CT_OUTPUT, 16>,
                           (const void *)k_conv<32, CT_LOSS, 16>, (const void *)k_conv<64, CT_LOSS, 16>,
                           (const void *)k_conv<32, CT_DATA, 16>, (const void *)k_conv<32, CT_HIDDEN, 32>,
                           (const void *)k_conv<32, CT_OUTPUT, 32>, (const void *)k_conv<64, CT_OUTPUT, 32>,
                           (const void *)k_conv<32, CT_LOSS, 32>, (const void *)k_conv<64, CT_LOSS, 32>,
                           (const void *)k_conv<32, CT_DATA, 32>};
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

// The error word of the bounded waits after the stream's work (0: none
// expired); reading clears it.
int conv_error(void *stream) {
    if (cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess) return -1;
    std::lock_guard<std::mutex> lk(g_ct_mtx);
    if (!g_ct_err) return 0;
    const int h = *(volatile int *)g_ct_err;
    *g_ct_err = 0;
    return h;
}

}  // namespace cfdwm
