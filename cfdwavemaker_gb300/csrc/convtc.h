// The learned update's valid 3x3 convolutions (convtc.cu).  Activations and
// gradients that the convolutions read are split into BF16 hi and lo parts,
// [b][part][C / 8][H][W][8] (conv_split_bytes); the weights are packed once per
// change (conv_pack).
#pragma once

#include <cuda_bf16.h>

#include <cstddef>
#include <cstdint>

namespace cfdwm {

constexpr int CONV_HID = 32;          // channels of a hidden layer
constexpr int CONV_MAX_PACK = 8, CONV_MAX_SUMS = 8;

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t conv_pack_bf16(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}

// eight values as their hi and lo parts
__device__ __forceinline__ void conv_split8(const float *v, uint4 &hi, uint4 &lo) {
    float h[8], l[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        h[e] = __bfloat162float(__float2bfloat16_rn(v[e]));
        l[e] = v[e] - h[e];
    }
    hi = make_uint4(conv_pack_bf16(h[0], h[1]), conv_pack_bf16(h[2], h[3]), conv_pack_bf16(h[4], h[5]),
                    conv_pack_bf16(h[6], h[7]));
    lo = make_uint4(conv_pack_bf16(l[0], l[1]), conv_pack_bf16(l[2], l[3]), conv_pack_bf16(l[4], l[5]),
                    conv_pack_bf16(l[6], l[7]));
}
#endif

int conv_load();
size_t conv_split_bytes(int B, int C, int H, int W);
// planes x[idx[b] or b][C][H][W] (batch stride xbs) to the split format
int conv_split(const float *x, long xbs, const int *idx, int B, int C, int H, int W, void *xs, void *stream);

// packed weights of layers w[O][C][9] (FP32, rounded to BF16): forward, or for the data gradient
struct ConvPack { long w; int C, O; bool data; };
long conv_pack_elems(int K, int N);   // BF16 elements of a layer with K channels in and N out (data gradient: N in, K out)
int conv_pack(const ConvPack *jobs, int n, const float *w, void *out, void *stream);

// ys = silu(conv(xs) + bias), HID channels; ds (may be null): silu' there, [b][HID / 4][H-2][W-2] float4
int conv_hidden(const void *xs, const void *wp, const float *bias, int B, int C, int H, int W, void *ys, void *ds,
                void *stream);
// y[b][O][H-2][W-2] = conv(xs) + bias, O <= 64
int conv_output(const void *xs, const void *wp, const float *bias, int B, int C, int O, int H, int W, float *y,
                void *stream);
// that output against targets tg[idx[b] or b][O] (batch stride tbs), channel 0 weighted by w0:
// loss = sum w (y - t)^2 inv_norm as conv_bias_parts shares lpart, dys its gradient in the split
// format, bpart[share][32 or 64] its sums per channel
struct ConvLoss {
    const float *tg;
    long tbs;
    const int *idx;
    float w0, inv_norm;
};
int conv_loss(const void *xs, const void *wp, const float *bias, int B, int C, int O, int H, int W,
              const ConvLoss &l, void *dys, float *bpart, float *lpart, void *stream);
// dxs[b][HID channels][H][W] = conv^T(dys) ds; bpart[conv_bias_parts(B, H, W)][HID]: sums of shares of it
int conv_bias_parts(int B, int H, int W);
int conv_data_grad(const void *dys, const void *wp, const void *ds, int B, int O, int H, int W, void *dxs,
                   float *bpart, void *stream);
// the weight gradients of up to four layers (C a multiple of 8, O <= 64), each
// as nslab partial sums of 9 O C elements; the plan sets nslab and swap
struct ConvWgt {
    const void *xs, *dys;
    int C, O, H, W;
    float *part;
    int nslab;
    bool swap;
};
int conv_wgt_plan(ConvWgt *l, int n, int B);
int conv_weight_grads(ConvWgt *l, int n, int B, void *stream);
// sums over nslab of part[slab * stride + e], e < n (16-byte aligned, stride a multiple of 4 >= n); wgt: a weight gradient's elements, put in [O][C][9] order
struct ConvSum { const float *part; float *out; long n, stride; int nslab; const ConvWgt *wgt; };
int conv_sums(const ConvSum *jobs, int n, void *stream);

int conv_error(void *stream);         // synchronises; error word of the bounded waits

}  // namespace cfdwm
