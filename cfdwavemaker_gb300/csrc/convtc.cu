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
// whole pixels, 16 bytes each, so the nine taps are nine start addresses in
// one copy of the tile: nothing is gathered, and nothing is split twice.
// Zero padding (ragged tiles, the data gradient's border, channels past the
// last) is the boxes' out-of-range fill.
//
// The weights are BF16, so the forward and data-gradient GEMMs take two MMAs
// per K step (hi, lo) and the weight gradient, whose two operands are both
// split, three (hi hi, lo hi, hi lo); sums in FP32 in TMEM.  The first form
// of these kernels gathered each operand tile from FP32 planes with the CUDA
// cores, nine times over (issue-bound).  Network of 16 levels over a 264 x 264
// grid: 357 us then, CT_FWD_US us now; loss and gradient of 8 patches of 72 x 72: 981
// and CT_GRAD_US us.
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
constexpr int TX = 8, TY = 16;            // pixel tile: 128 rows of D, a core matrix per tile row
constexpr int PX = TX + 2, PY = TY + 2;   // the tile with its halo
constexpr int KC = 4;                     // channel chunks (of 8) per stage: two K steps of 16
constexpr int CHUNK = PX * PY * 16;       // bytes of a chunk's patch
constexpr int APART = KC * CHUNK;         // of one split part of a stage
constexpr int CT_THREADS = 128;           // a thread per TMEM lane
constexpr int CT_HEAD = 64 + 4 * HID * 4; // barriers and flags, bias partial sums

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

// FP32 planes [idx b][C][plane] to the split format; a thread per (pixel, chunk).
__global__ void __launch_bounds__(256) k_ct_split(const float *x, long xbs, const int *idx, int C, long plane,
                                                  uint4 *out) {
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
// [stage][tap][KC][NP][8] BF16, a stage one bulk copy; zero past the channels.
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
    const int c8 = (int)(i & 7), n = (int)(i / 8 % j.NP), kc = (int)(i / (8L * j.NP) % KC);
    const int tap = (int)(i / (8L * j.NP * KC) % 9), st = (int)(i / (8L * j.NP * KC * 9));
    const int k = (st * KC + kc) * 8 + c8;
    float v = 0.f;
    if (k < j.K && n < j.N) v = w[j.w + (long)k * j.sk + (long)n * j.sn + (j.flip ? 8 - tap : tap)];
    out[e] = __float2bfloat16_rn(v);
}

// ---------------------------------------------------------------------------
// Forward and data gradient
// ---------------------------------------------------------------------------
enum { CT_HIDDEN = 0, CT_OUTPUT = 1, CT_DATA = 2 };

struct ConvArgs {
    const uint8_t *w;            // packed weights
    const float *bias;           // HIDDEN, OUTPUT
    const float4 *ds;            // DATA: silu' of the layer's pre-activation [b][HID / 4][Ho][Wo]
    float4 *ds_out;              // HIDDEN: the same, or null
    uint4 *ys;                   // HIDDEN: activations, DATA: gradient, split format
    float *y;                    // OUTPUT: planes [b][O][Ho][Wo]
    float *bpart;                // DATA: sums of the tile's gradient [tile][HID]
    int nst, nch;                // stages; input chunks
    int origin;                  // of the patch relative to the tile: 0, data gradient -2
    int O, Ho, Wo, tiles_x;
    int *err;
};

template <int NP> struct CtCfg {
    static constexpr int BTILE = 9 * KC * NP * 16;
    static constexpr int STAGE = 2 * APART + BTILE;
};

// A CTA makes one tile of 16 x 8 output pixels: M = 128, N = NP (the hidden
// channels, or the output's padded), K = 32 channels x 9 taps per stage.
// Thread 0 copies (two stages in flight), thread 32 issues the MMAs, the four
// warps read their TMEM lanes.  The operand's 4 KB per MMA from shared memory
// bound the tensor cores at these N (32 cycles an MMA); up to five CTAs an SM
// overlap copies, MMAs and epilogues of different tiles.
template <int NP, int EPI>
__global__ void __launch_bounds__(CT_THREADS) k_conv(const __grid_constant__ CUtensorMap xm, ConvArgs a) {
    using CF = CtCfg<NP>;
    extern __shared__ __align__(128) uint8_t ct_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)ct_raw + 127) & ~(uintptr_t)127);
    const int nbuf = a.nst < 2 ? a.nst : 2;
    uint64_t *full = (uint64_t *)(smem + nbuf * CF::STAGE), *empty = full + 2, *done = full + 4;
    uint32_t *tslot = (uint32_t *)(full + 5);
    volatile int *fail = (volatile int *)(full + 6);
    float *red = (float *)(full + 8);                 // DATA: [4][HID]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.y;
    const int x0 = (blockIdx.x % a.tiles_x) * TX, y0 = (blockIdx.x / a.tiles_x) * TY;
    if (tid == 0) {
        for (int q = 0; q < 5; q++) mbar_init(full + q, 1);
        *fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(tslot, NP);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;

    if (tid == 0) {
        for (int s = 0; s < a.nst; s++) {
            const int buf = s & 1;
            if (s >= 2 && !mbar_wait(empty + buf, (uint32_t)(((s >> 1) - 1) & 1), a.err, 11)) { *fail = 1; break; }
            uint8_t *st = smem + buf * CF::STAGE;
            mbar_expect_tx(full + buf, CF::STAGE);
            tma_4d(st, &xm, full + buf, (x0 + a.origin) * 8, y0 + a.origin, s * KC, b * 2);
            bulk_load(st + 2 * APART, a.w + (long)s * CF::BTILE, CF::BTILE, full + buf);
        }
    } else if (tid == 32) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NP >> 3) << 17) |
                               ((uint32_t)((TX * TY) >> 4) << 24);
        for (int s = 0; s < a.nst; s++) {
            const int buf = s & 1;
            const uint32_t par = (uint32_t)((s >> 1) & 1);
            if (!mbar_wait(full + buf, par, a.err, 12)) {
                *fail = 1;
                mbar_wait(full + buf, par, a.err, 12);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t A = su32(smem + buf * CF::STAGE), B = A + 2 * APART;
            const uint64_t da = cdesc(A, CHUNK, PX * 16), db = cdesc(B, NP * 16, 128);
            const int nk = (min(KC, a.nch - s * KC) + 1) / 2;
            for (int tap = 0; tap < 9; tap++)
                for (int k = 0; k < nk; k++) {
                    const uint64_t oa = (uint64_t)((2 * k * CHUNK + ((tap / 3) * PX + tap % 3) * 16) >> 4);
                    const uint64_t ob = (uint64_t)(((tap * KC + 2 * k) * NP * 16) >> 4);
                    umma(tmem, da + oa, db + ob, idesc, (s | tap | k) ? 1u : 0u);
                    umma(tmem, da + oa + (APART >> 4), db + ob, idesc, 1u);
                }
            umma_commit(empty + buf);
        }
        umma_commit(done);
    }
    __syncwarp();
    bool ok = mbar_wait(done, 0u, a.err, 13);
    ok = !__syncthreads_or(!ok) && !*fail;
    if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16);
        const int oy = y0 + (tid >> 3), ox = x0 + (tid & 7);
        const long plane = (long)a.Ho * a.Wo, pix = (long)oy * a.Wo + ox;
        const bool live = oy < a.Ho && ox < a.Wo;
        if (EPI == CT_OUTPUT) {
#pragma unroll
            for (int h = 0; h < NP / 32; h++) {
                float d[32];
                tmem_ld32(ta + h * 32, d);
                if (live)
#pragma unroll
                    for (int n = 0; n < 32; n++) {
                        const int o = h * 32 + n;
                        if (o >= a.O) break;
                        a.y[((long)b * a.O + o) * plane + pix] = d[n] + a.bias[o];
                    }
            }
        } else {
            float d[32];
            tmem_ld32(ta, d);
#pragma unroll
            for (int c = 0; c < HID / 8; c++) {
                float v[8], g[8];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    if (EPI == CT_DATA) {
                        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (live) f = a.ds[((long)b * (HID / 4) + c * 2 + q) * plane + pix];
                        g[q * 4] = f.x; g[q * 4 + 1] = f.y; g[q * 4 + 2] = f.z; g[q * 4 + 3] = f.w;
                    }
                }
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    if (EPI == CT_DATA) {
                        v[e] = live ? d[c * 8 + e] * g[e] : 0.f;
                        d[c * 8 + e] = v[e];
                    } else {
                        const float p = d[c * 8 + e] + a.bias[c * 8 + e], sg = ct_sigmoid(p);
                        v[e] = p / (1.f + expf(-p));
                        g[e] = sg * (1.f + p * (1.f - sg));
                    }
                }
                if (!live) continue;
                uint4 hi, lo;
                conv_split8(v, hi, lo);
                a.ys[((long)(b * 2) * (HID / 8) + c) * plane + pix] = hi;
                a.ys[((long)(b * 2 + 1) * (HID / 8) + c) * plane + pix] = lo;
                if (EPI == CT_HIDDEN && a.ds_out)
#pragma unroll
                    for (int q = 0; q < 2; q++)
                        a.ds_out[((long)b * (HID / 4) + c * 2 + q) * plane + pix] =
                            make_float4(g[q * 4], g[q * 4 + 1], g[q * 4 + 2], g[q * 4 + 3]);
            }
            if (EPI == CT_DATA) {
                // the bias gradient's share of this tile: lane c ends with channel c of its warp's pixels
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) {
                    const bool up = lane & o;
#pragma unroll
                    for (int i = 0; i < o; i++) {
                        const float send = up ? d[i] : d[i + o], keep = up ? d[i + o] : d[i];
                        d[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
                red[warp * HID + lane] = d[0];
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (EPI == CT_DATA && ok && warp == 1)
        a.bpart[((long)b * gridDim.x + blockIdx.x) * HID + lane] =
            (red[lane] + red[HID + lane]) + (red[2 * HID + lane] + red[3 * HID + lane]);
    if (warp == 0) tmem_free(tmem, NP);
}

// ---------------------------------------------------------------------------
// Weight gradient
// ---------------------------------------------------------------------------
struct WgtArgs {
    float *part;                 // [slab][3 dx][O][3 dy C]
    int nch, rows;               // input chunks; patch rows copied
    int ntiles, tiles_x, tiles_img;
    int nbuf;
    int O;
    int *err;
};

// D's rows are (dy, c) pairs: with the patch copied as [row][chunk][pixel],
// the row groups of 8 channels over dy and the chunks are one arithmetic
// progression of addresses, so M = 128 holds 16 of them whatever C is (four
// taps' worth of 32 channels; blockIdx.y counts the M tiles).  dx is a start
// address, with an accumulator of its own.  K is the tile's pixels, two tile
// rows per MMA.  A CTA sums its slab (every gridDim.x-th tile) in TMEM; the
// slabs are summed in order afterwards, so the result is deterministic.
template <int NP>
__global__ void __launch_bounds__(CT_THREADS)
k_conv_wgt(const __grid_constant__ CUtensorMap xm, const __grid_constant__ CUtensorMap dm, WgtArgs a) {
    constexpr int BPART = (NP / 8) * TY * TX * 16;
    constexpr uint32_t TCOLS = NP == 32 ? 128 : 256;
    extern __shared__ __align__(128) uint8_t ct_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)ct_raw + 127) & ~(uintptr_t)127);
    const int apart = a.rows * a.nch * PX * 16, abytes = (2 * apart + 127) & ~127, stage = abytes + 2 * BPART;
    uint64_t *full = (uint64_t *)(smem + a.nbuf * stage), *empty = full + 2, *done = full + 4;
    uint32_t *tslot = (uint32_t *)(full + 5);
    volatile int *fail = (volatile int *)(full + 6);
    const int tid = threadIdx.x, warp = tid >> 5;
    const int g0 = blockIdx.y * 16, r0 = g0 / a.nch;          // first row group of this M tile, its dy
    if (tid == 0) {
        for (int q = 0; q < 5; q++) mbar_init(full + q, 1);
        *fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(tslot, TCOLS);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;

    if (tid == 0) {
        int s = 0;
        for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x, s++) {
            const int buf = s % a.nbuf, use = s / a.nbuf;
            if (use > 0 && !mbar_wait(empty + buf, (uint32_t)((use - 1) & 1), a.err, 14)) { *fail = 1; break; }
            const int b = t / a.tiles_img, r = t % a.tiles_img;
            const int x0 = (r % a.tiles_x) * TX, y0 = (r / a.tiles_x) * TY;
            uint8_t *st = smem + buf * stage;
            mbar_expect_tx(full + buf, 2 * apart + 2 * BPART);
            tma_4d(st, &xm, full + buf, x0 * 8, 0, y0 + r0, b * 2);
            tma_4d(st + abytes, &dm, full + buf, x0 * 8, y0, 0, b * 2);
        }
    } else if (tid == 32) {
        // both operands MN-major (bits 15 and 16)
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                               ((uint32_t)(NP >> 3) << 17) | (8u << 24);
        int s = 0;
        for (int t = blockIdx.x; t < a.ntiles; t += gridDim.x, s++) {
            const int buf = s % a.nbuf;
            const uint32_t par = (uint32_t)((s / a.nbuf) & 1);
            if (!mbar_wait(full + buf, par, a.err, 15)) {
                *fail = 1;
                mbar_wait(full + buf, par, a.err, 15);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t A = su32(smem + buf * stage), B = A + abytes;
            const uint32_t rowb = (uint32_t)a.nch * PX * 16;
            const uint64_t da = cdesc(A + (uint32_t)(g0 - r0 * a.nch) * PX * 16, rowb, PX * 16);
            const uint64_t db = cdesc(B, TX * 16, TY * TX * 16);
            const uint64_t pa = (uint64_t)(apart >> 4), pb = (uint64_t)(BPART >> 4);
            for (int k = 0; k < TY / 2; k++)
                for (int dx = 0; dx < 3; dx++) {
                    const uint64_t oa = (uint64_t)((2 * k * rowb + dx * 16) >> 4);
                    const uint64_t ob = (uint64_t)((2 * k * TX * 16) >> 4);
                    const uint32_t d = tmem + dx * NP;
                    umma(d, da + oa, db + ob, idesc, (s | k) ? 1u : 0u);
                    umma(d, da + oa + pa, db + ob, idesc, 1u);
                    umma(d, da + oa, db + ob + pb, idesc, 1u);
                }
            umma_commit(empty + buf);
        }
        umma_commit(done);
    }
    __syncwarp();
    bool ok = mbar_wait(done, 0u, a.err, 16);
    ok = !__syncthreads_or(!ok) && !*fail;
    if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int row = g0 * 8 + tid, nrow = 3 * a.nch * 8;
        for (int dx = 0; dx < 3; dx++)
#pragma unroll
            for (int h = 0; h < NP / 32; h++) {
                float d[32];
                tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + dx * NP + h * 32, d);
                if (row < nrow)
#pragma unroll
                    for (int n = 0; n < 32; n++) {
                        const int o = h * 32 + n;
                        if (o >= a.O) break;
                        a.part[(((long)blockIdx.x * 3 + dx) * a.O + o) * nrow + row] = d[n];
                    }
            }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) tmem_free(tmem, TCOLS);
}

// Sums of the slabs' partial results in slab order: 32 elements per block,
// eight interleaved shares of the slabs each, all layers in one launch.
struct SumJobs {
    struct Job {
        const float *part;
        float *out;
        long n, stride;          // elements, and the distance of two slabs
        int nslab, O, C;         // C > 0: [dx][O][dy C] to [O][C][dy dx]
        unsigned end;            // end of the job's blocks
    } j[CONV_MAX_SUMS];
    int n;
};

__global__ void __launch_bounds__(256) k_ct_sum(SumJobs jobs) {
    __shared__ float red[8][32];
    int q = 0;
    while (blockIdx.x >= jobs.j[q].end) q++;
    const SumJobs::Job &j = jobs.j[q];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long e = (long)(blockIdx.x - (q ? jobs.j[q - 1].end : 0)) * 32 + lane;
    float s = 0.f;
    if (e < j.n) {
#pragma unroll 8
        for (int k = w; k < j.nslab; k += 8) s += j.part[k * j.stride + e];
    }
    red[w][lane] = s;
    __syncthreads();
    if (w || e >= j.n) return;
    for (int k = 1; k < 8; k++) s += red[k][lane];
    long o = e;
    if (j.C > 0) {
        const int nrow = 3 * j.C, row = (int)(e % nrow), oc = (int)(e / nrow % j.O), dx = (int)(e / ((long)nrow * j.O));
        o = ((long)oc * j.C + row % j.C) * 9 + (row / j.C) * 3 + dx;
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

int ct_tiles_x(int Wo) { return (Wo + TX - 1) / TX; }
int ct_tiles(int Ho, int Wo) { return ct_tiles_x(Wo) * ((Ho + TY - 1) / TY); }

template <int NP, int EPI>
int launch_conv(const CUtensorMap &m, ConvArgs &a, int B, cudaStream_t st) {
    const int smem = std::min(a.nst, 2) * CtCfg<NP>::STAGE + CT_HEAD + 128;
    static const cudaError_t attr = cudaFuncSetAttribute(
        k_conv<NP, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * CtCfg<NP>::STAGE + CT_HEAD + 128);
    CK(attr);
    const dim3 grid((unsigned)ct_tiles(a.Ho, a.Wo), (unsigned)B);
    k_conv<NP, EPI><<<grid, CT_THREADS, smem, st>>>(m, a);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

int ct_rows(int nch) {
    int span = 0;
    for (int g = 0; g < 3 * nch; g += 16) span = std::max(span, (g + 15) / nch - g / nch);
    return TY + span;
}

int ct_slabs(int ntiles, int nch) { return std::min(ntiles, std::max(1, 152 / ((3 * nch + 15) / 16))); }

}  // namespace

size_t conv_split_bytes(int B, int C, int H, int W) { return (size_t)B * 2 * ((C + 7) / 8) * H * W * 16; }

int conv_split(const float *x, long xbs, const int *idx, int B, int C, int H, int W, void *xs, void *stream) {
    const long plane = (long)H * W;
    const dim3 grid((unsigned)((plane + 255) / 256), (unsigned)((C + 7) / 8), (unsigned)B);
    k_ct_split<<<grid, 256, 0, (cudaStream_t)stream>>>(x, xbs, idx, C, plane, (uint4 *)xs);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

long conv_pack_elems(int K, int N) { return (long)((K + 31) / 32) * 9 * KC * (N <= 32 ? 32 : 64) * 8; }

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

static int conv_args(ConvArgs &a, CUtensorMap &m, const void *xs, const void *wp, int B, int K, int H, int W,
                     int origin, int Ho, int Wo) {
    a = {};
    a.w = (const uint8_t *)wp;
    a.nch = (K + 7) / 8;
    a.nst = (a.nch + KC - 1) / KC;
    a.origin = origin;
    a.Ho = Ho; a.Wo = Wo;
    a.tiles_x = ct_tiles_x(Wo);
    int rc = ct_err_word(&a.err);
    if (rc) return rc;
    return ct_map(&m, xs, B, a.nch, H, W, false, PX, PY, KC);
}

int conv_hidden(const void *xs, const void *wp, const float *bias, int B, int C, int H, int W, void *ys, void *ds,
                void *stream) {
    if (C < 1 || H < 3 || W < 3 || B < 1) return E_BAD_ARGUMENT;
    ConvArgs a;
    CUtensorMap m;
    int rc = conv_args(a, m, xs, wp, B, C, H, W, 0, H - 2, W - 2);
    if (rc) return rc;
    a.bias = bias; a.ys = (uint4 *)ys; a.ds_out = (float4 *)ds;
    return launch_conv<32, CT_HIDDEN>(m, a, B, (cudaStream_t)stream);
}

int conv_output(const void *xs, const void *wp, const float *bias, int B, int C, int O, int H, int W, float *y,
                void *stream) {
    if (O < 1 || O > 64 || C < 1 || H < 3 || W < 3 || B < 1) return E_BAD_ARGUMENT;
    ConvArgs a;
    CUtensorMap m;
    int rc = conv_args(a, m, xs, wp, B, C, H, W, 0, H - 2, W - 2);
    if (rc) return rc;
    a.bias = bias; a.y = y; a.O = O;
    return O <= 32 ? launch_conv<32, CT_OUTPUT>(m, a, B, (cudaStream_t)stream)
                   : launch_conv<64, CT_OUTPUT>(m, a, B, (cudaStream_t)stream);
}

long conv_bias_parts(int B, int H, int W) { return (long)B * ct_tiles(H, W); }

int conv_data_grad(const void *dys, const void *wp, const void *ds, int B, int O, int H, int W, void *dxs,
                   float *bpart, void *stream) {
    if (O < 1 || H < 3 || W < 3 || B < 1) return E_BAD_ARGUMENT;
    ConvArgs a;
    CUtensorMap m;
    int rc = conv_args(a, m, dys, wp, B, O, H - 2, W - 2, -2, H, W);
    if (rc) return rc;
    a.ds = (const float4 *)ds; a.ys = (uint4 *)dxs; a.bpart = bpart;
    return launch_conv<32, CT_DATA>(m, a, B, (cudaStream_t)stream);
}

long conv_wgt_part(int B, int C, int O, int H, int W, int *nslab) {
    *nslab = ct_slabs(B * ct_tiles(H - 2, W - 2), (C + 7) / 8);
    return (long)*nslab * 9 * O * C;
}

int conv_weight_grad(const void *xs, const void *dys, int B, int C, int O, int H, int W, float *part, void *stream) {
    if (O < 1 || O > 64 || C < 8 || C % 8 || H < 3 || W < 3 || B < 1) return E_BAD_ARGUMENT;
    const int NP = O <= 32 ? 32 : 64;
    WgtArgs a = {};
    a.part = part; a.O = O;
    a.nch = C / 8;
    a.rows = ct_rows(a.nch);
    a.tiles_x = ct_tiles_x(W - 2);
    a.tiles_img = ct_tiles(H - 2, W - 2);
    a.ntiles = B * a.tiles_img;
    int rc = ct_err_word(&a.err);
    if (rc) return rc;
    CUtensorMap xm, dm;
    if ((rc = ct_map(&xm, xs, B, a.nch, H, W, true, PX, a.rows, a.nch))) return rc;
    if ((rc = ct_map(&dm, dys, B, (O + 7) / 8, H - 2, W - 2, false, TX, TY, NP / 8))) return rc;
    // two stages where they fit (C <= 128 with O <= 32)
    constexpr int LIMIT = 227 * 1024;
    const int stage = ((2 * a.rows * a.nch * PX * 16 + 127) & ~127) + NP * TY * TX * 4;
    a.nbuf = 2 * stage + CT_HEAD + 128 <= LIMIT ? 2 : 1;
    const int smem = a.nbuf * stage + CT_HEAD + 128;
    if (smem > LIMIT) return E_UNSUPPORTED;
    const dim3 grid((unsigned)ct_slabs(a.ntiles, a.nch), (unsigned)((3 * a.nch + 15) / 16));
    auto kern = NP == 32 ? k_conv_wgt<32> : k_conv_wgt<64>;
    static const cudaError_t a32 =
        cudaFuncSetAttribute(k_conv_wgt<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, LIMIT);
    static const cudaError_t a64 =
        cudaFuncSetAttribute(k_conv_wgt<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, LIMIT);
    CK(a32);
    CK(a64);
    kern<<<grid, CT_THREADS, smem, (cudaStream_t)stream>>>(xm, dm, a);
    note_launch();
    CK(cudaGetLastError());
    return OK;
}

int conv_sums(const ConvSum *jobs, int n, void *stream) {
    SumJobs p = {};
    p.n = n;
    unsigned end = 0;
    for (int q = 0; q < n; q++) {
        const ConvSum &c = jobs[q];
        SumJobs::Job &j = p.j[q];
        j.part = c.part; j.out = c.out; j.n = c.n; j.stride = c.stride; j.nslab = c.nslab; j.O = c.O; j.C = c.C;
        j.end = end += (unsigned)((c.n + 31) / 32);
    }
    k_ct_sum<<<end, 256, 0, (cudaStream_t)stream>>>(p);
    note_launch();
    CK(cudaGetLastError());
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
