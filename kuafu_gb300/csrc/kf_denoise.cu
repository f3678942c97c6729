// kf_denoise.cu — the learned denoiser that replaces kuafu's OptiX pass
// (src/core/denoiser.cpp:257-316, context.cpp:651-670): a 5-level U-Net of 3x3
// convolutions (32 / 64 / 96 / 128 / 160 channels) over noisy radiance, albedo,
// normal and depth, trained on low-spp / high-spp pairs this tracer renders.
//
// Every convolution (forward, backward-data) and every weight gradient runs on the
// tcgen05 kernels of kf_conv.cu (BF16 operands, FP32 accumulation). Activations
// and activation gradients are BF16 NHWC; master weights, weight gradients and
// Adam moments are FP32. Skip connections are written by the encoder straight
// into the channel slice of the decoder's concatenation buffer.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "kf_conv.h"
#include "kf_denoise.h"
#include "kf_host.h"
#include "kf_tone.cuh"

namespace kf {

namespace {

using bf16 = __nv_bfloat16;

// ---------------------------------------------------------------------------
// Elementwise kernels (HBM-bound, NHWC with channel stride / offset). Channel counts,
// strides and offsets of pooled / upsampled tensors are multiples of 8, so each thread
// moves 8 channels (16 bytes) per access.
// ---------------------------------------------------------------------------
struct F8 {
    float v[8];
};
__device__ __forceinline__ F8 ld8(const bf16* p) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
    F8 f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 t = __bfloat1622float2(h[k]);
        f.v[2 * k] = t.x;
        f.v[2 * k + 1] = t.y;
    }
    return f;
}
__device__ __forceinline__ void st8(bf16* p, const F8& f) {
    uint4 q;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(f.v[2 * k], f.v[2 * k + 1]);
    *reinterpret_cast<uint4*>(p) = q;
}

// ReLU's backward mask on the BF16-rounded gradient: zero where the forward output y is not positive
__device__ __forceinline__ void mask8(F8& v, const bf16* y) {
    const F8 m = ld8(y);
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (!(m.v[k] > 0.0f)) v.v[k] = 0.0f;
}

// gx (dense, H x W) = broadcast(gy / 4) + gskip[slice], masked by the forward output y[slice]
__global__ void k_pool_bwd_add(const bf16* __restrict__ gy, const bf16* __restrict__ gskip, int ss, int so, int C,
                               int N, int H, int W, const bf16* __restrict__ y, int ys, int yo, bf16* gx) {
    grid_dependency_wait();
    const int G = C / 8;
    const size_t total = (size_t)N * H * W * G;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int g = (int)(i % G);
        const size_t pix = i / G;
        const int xw = (int)(pix % W);
        const size_t ny = pix / W; // n * H + y
        const size_t low = (ny / 2) * (W / 2) + xw / 2;
        F8 v = ld8(gy + low * C + 8 * g);
        const F8 sk = ld8(gskip + pix * ss + so + 8 * g);
#pragma unroll
        for (int k = 0; k < 8; ++k) v.v[k] = v.v[k] * 0.25f + sk.v[k];
        mask8(v, y + pix * ys + yo + 8 * g);
        st8(gx + pix * C + 8 * g, v);
    }
}

// gx (dense, H/2 x W/2) = sum of the 2x2 block of gy[slice] (H x W), masked by the forward
// output y (dense, H/2 x W/2)
__global__ void k_up_bwd(const bf16* __restrict__ gy, int gs, int go, int C, int N, int H, int W,
                         const bf16* __restrict__ y, bf16* gx) {
    grid_dependency_wait();
    const int Ho = H / 2, Wo = W / 2, G = C / 8;
    const size_t total = (size_t)N * Ho * Wo * G;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int g = (int)(i % G);
        const size_t pix = i / G;
        const int xw = (int)(pix % Wo);
        const size_t ny = pix / Wo;
        const size_t row0 = (2 * ny) * W + 2 * xw;
        F8 a = ld8(gy + row0 * gs + go + 8 * g), b = ld8(gy + (row0 + 1) * gs + go + 8 * g);
        const F8 c = ld8(gy + (row0 + W) * gs + go + 8 * g), d = ld8(gy + (row0 + W + 1) * gs + go + 8 * g);
#pragma unroll
        for (int k = 0; k < 8; ++k) a.v[k] = ((a.v[k] + b.v[k]) + c.v[k]) + d.v[k];
        mask8(a, y + pix * C + 8 * g);
        st8(gx + pix * C + 8 * g, a);
    }
}

// Where each layer's parameters and packed weights lie, for k_update (a kernel parameter).
struct UpdateTable {
    int first[20]; // first block of each layer: a block per tap and 32 x 32 weights
    int cin[19], cout[19], rows[19], cout_k[19];
    uint32_t w_off[19], b_off[19], wf_off[19], wb_off[19];
};

// One pass over all parameters: Adam on the FP32 master weights (Kingma & Ba 2015; skipped when
// !step) and the BF16 weights the convolutions read: forward wf[tap][co][ci], backward-data
// wb[8 - tap][ci][co], and the first layer's input channels 0..15 alone (wf16: the inference path
// feeds it 16-channel features). Rows and columns of the padding stay zero from their allocation.
// A block holds 32 x 32 weights of one tap, transposed through shared memory so that both layouts
// are written in whole lines. Bound by HBM (36 bytes a parameter): 21 us for the 1.8 M
// parameters (cold cache); Adam and 20 packing launches took 92 us.
constexpr int kUpdateThreads = 256;
__global__ void __launch_bounds__(kUpdateThreads) k_update(UpdateTable tab, float* __restrict__ w,
                                                           const float* __restrict__ grad, float* __restrict__ m,
                                                           float* __restrict__ v, bf16* __restrict__ wf,
                                                           bf16* __restrict__ wb, bf16* __restrict__ wf16, int step,
                                                           float lr, float b1, float b2, float eps, float bc1,
                                                           float bc2) {
    __shared__ bf16 tile[32][34];
    int l = 0;
    while ((int)blockIdx.x >= tab.first[l + 1]) ++l;
    const int cin = tab.cin[l], cout = tab.cout[l], rows = tab.rows[l], cout_k = tab.cout_k[l];
    const int nci = cin / 32, k = (int)blockIdx.x - tab.first[l];
    const int ci0 = (k % nci) * 32, co0 = (k / nci) % (cout_k / 32) * 32, tap = k / (nci * (cout_k / 32));
    auto adam = [&](size_t i) {
        float x = w[i];
        if (step) {
            const float gi = grad[i];
            const float mi = b1 * m[i] + (1.0f - b1) * gi;
            const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
            m[i] = mi;
            v[i] = vi;
            x -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
            w[i] = x;
        }
        return x;
    };
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < 32; r += kUpdateThreads / 32) {
        const int co = co0 + r, ci = ci0 + lane;
        bf16 q = __float2bfloat16_rn(0.0f);
        if (co < cout) {
            q = __float2bfloat16_rn(adam(tab.w_off[l] + ((size_t)tap * cout + co) * cin + ci));
            wf[tab.wf_off[l] + ((size_t)tap * rows + co) * cin + ci] = q;
            if (l == 0 && ci < 16) wf16[((size_t)tap * rows + co) * 16 + ci] = q;
        }
        tile[r][lane] = q;
    }
    if (tap == 0 && ci0 == 0 && threadIdx.x < 32 && co0 + lane < cout && step) adam(tab.b_off[l] + co0 + lane);
    __syncthreads();
    for (int r = threadIdx.x >> 5; r < 32; r += kUpdateThreads / 32)
        wb[tab.wb_off[l] + ((size_t)(8 - tap) * cin + ci0 + r) * cout_k + co0 + lane] = tile[lane][r];
}

// The network works on g(x) = tone(x) of linear radiance (kf_tone.cuh).

// Network input from render targets: g(radiance), albedo (base colour of the first hit of
// sample 0), normal, hit distance t / (1 + t), log2(samples) / 8; CH channels (32, or 16
// for the inference path whose first convolution takes 16), the rest zero. base (optional)
// receives g(radiance) in FP32: the residual the network corrects. Pixels of the padded
// tensor outside (H, W) are zero.
template <int CH>
__global__ void k_pack_features(const float4* __restrict__ rad, const float4* __restrict__ alb,
                                const float4* __restrict__ nrm, const float* __restrict__ dep, float spp_feature,
                                int H, int W, int Hp, int Wp, bf16* out, float4* base) {
    const size_t total = (size_t)Hp * Wp;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % Wp), y = (int)(i / Wp);
        float f[32];
        for (int c = 0; c < 32; ++c) f[c] = 0.0f;
        if (x < W && y < H) {
            const size_t s = (size_t)y * W + x;
            const float4 r = rad[s], a = alb[s], n = nrm[s];
            const float d = dep[s];
            f[0] = tone(r.x);
            f[1] = tone(r.y);
            f[2] = tone(r.z);
            f[3] = a.x;
            f[4] = a.y;
            f[5] = a.z;
            f[6] = n.x;
            f[7] = n.y;
            f[8] = n.z;
            f[9] = d / (1.0f + d);
            f[10] = spp_feature;
        }
        bf16* o = out + i * CH;
#pragma unroll
        for (int g = 0; g < CH / 8; ++g) {
            F8 q;
#pragma unroll
            for (int k = 0; k < 8; ++k) q.v[k] = f[8 * g + k];
            st8(o + 8 * g, q);
        }
        if (base) base[i] = make_float4(f[0], f[1], f[2], 0.0f);
    }
}

// denoised linear radiance = g^-1(prediction + g(radiance)) for the (H, W) window: the
// residual add and the unpack in one pass, g(radiance) recomputed from the render target
// (the same function of the same value the feature pass applies, so the same bits)
__global__ void k_unpack_residual(const float4* __restrict__ pred, const float4* __restrict__ rad, int H, int W,
                                  int Wp, float4* out) {
    const size_t total = (size_t)H * W;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % W), y = (int)(i / W);
        const float4 p = pred[(size_t)y * Wp + x], r = rad[i];
        out[i] = make_float4(untone(p.x + tone(r.x)), untone(p.y + tone(r.y)), untone(p.z + tone(r.z)), 1.0f);
    }
}


// L = mean|p - t| + lambda * mean(|dx p - dx t| + |dy p - dy t|) in g space, p the FP32
// prediction [P][4] (+ base, the residual, where given), t = g(target); writes dL/dp as the BF16
// [P][32] gradient of the head. A block takes 32 x 8 pixels and brings predictions and g(target)
// with a border of one pixel to shared memory once, so that g is evaluated 1.3 times a pixel
// (with every neighbour read and mapped in place 5 times, and the 64-byte gradient written in
// 2-byte pieces, 16 x 128 x 128 pixels took 63 us; this form 11).
constexpr int kLossW = 32, kLossH = 8;
__global__ void __launch_bounds__(kLossW * kLossH) k_loss(const float4* __restrict__ pred,
                                                          const float4* __restrict__ base,
                                                          const float4* __restrict__ target, int N, int H, int W,
                                                          float lambda, float* loss, bf16* gpred) {
    __shared__ float sp[3][kLossH + 2][kLossW + 2], st[3][kLossH + 2][kLossW + 2];
    __shared__ float s_acc[kLossW * kLossH / 32];
    const int tx = (W + kLossW - 1) / kLossW, ty = (H + kLossH - 1) / kLossH;
    const int n = blockIdx.x / (tx * ty), r = blockIdx.x % (tx * ty);
    const int x0 = r % tx * kLossW, y0 = r / tx * kLossH;
    for (int i = threadIdx.x; i < (kLossH + 2) * (kLossW + 2); i += kLossW * kLossH) {
        const int lx = i % (kLossW + 2), ly = i / (kLossW + 2), x = x0 + lx - 1, y = y0 + ly - 1;
        if (x < 0 || x >= W || y < 0 || y >= H) continue;
        const size_t j = ((size_t)n * H + y) * W + x;
        float4 p = pred[j];
        const float4 t = target[j];
        if (base) {
            const float4 b = base[j];
            p.x += b.x;
            p.y += b.y;
            p.z += b.z;
        }
        sp[0][ly][lx] = p.x; sp[1][ly][lx] = p.y; sp[2][ly][lx] = p.z;
        st[0][ly][lx] = tone(t.x); st[1][ly][lx] = tone(t.y); st[2][ly][lx] = tone(t.z);
    }
    __syncthreads();
    const size_t total = (size_t)N * H * W;
    const float inv = 1.0f / (float)(total * 3);
    const int lx = (int)threadIdx.x % kLossW + 1, ly = (int)threadIdx.x / kLossW + 1;
    const int x = x0 + lx - 1, y = y0 + ly - 1;
    float acc = 0.0f;
    if (x < W && y < H) {
        F8 g;
#pragma unroll
        for (int c = 0; c < 8; ++c) g.v[c] = 0.0f;
        auto sign = [](float e) { return e > 0.0f ? 1.0f : (e < 0.0f ? -1.0f : 0.0f); };
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float p = sp[c][ly][lx], tv = st[c][ly][lx];
            const float d = p - tv;
            acc += fabsf(d);
            float gr = sign(d);
            // forward differences touching the pixel: (i, i+1) and (i-1, i) in x, same in y
            if (x + 1 < W) {
                const float e = (sp[c][ly][lx + 1] - p) - (st[c][ly][lx + 1] - tv);
                acc += lambda * fabsf(e);
                gr -= lambda * sign(e);
            }
            if (x > 0) gr += lambda * sign((p - sp[c][ly][lx - 1]) - (tv - st[c][ly][lx - 1]));
            if (y + 1 < H) {
                const float e = (sp[c][ly + 1][lx] - p) - (st[c][ly + 1][lx] - tv);
                acc += lambda * fabsf(e);
                gr -= lambda * sign(e);
            }
            if (y > 0) gr += lambda * sign((p - sp[c][ly - 1][lx]) - (tv - st[c][ly - 1][lx]));
            g.v[c] = gr * inv;
        }
        bf16* o = gpred + (((size_t)n * H + y) * W + x) * 32;
        st8(o, g);
        const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int q = 1; q < 4; ++q) reinterpret_cast<uint4*>(o)[q] = zero;
    }
    for (int off = 16; off; off >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, off);
    if ((threadIdx.x & 31) == 0) s_acc[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float a = 0.0f;
        for (int k = 0; k < kLossW * kLossH / 32; ++k) a += s_acc[k];
        atomicAdd(loss, a * inv);
    }
}

// A training target from the FP64 accumulation: sum of the frames' pixel means / frames.
__global__ void k_target_from_sum64(const dbl4* __restrict__ sum, size_t n, float4* out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const dbl4 v = sum[i];
        const double inv = v.w > 0.0 ? 1.0 / v.w : 0.0;
        out[i] = make_float4((float)(v.x * inv), (float)(v.y * inv), (float)(v.z * inv), 1.0f);
    }
}

// crop gather: features [n][H][W][32], residual bases and targets -> batch [b][c][c]
__global__ void k_gather_crops(const bf16* __restrict__ feat, const float4* __restrict__ base,
                               const float4* __restrict__ tgt, int H, int W, const int4* __restrict__ crops, int B,
                               int c, bf16* bf, float4* bb, float4* bt) {
    const size_t total = (size_t)B * c * c;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % c);
        const int y = (int)((i / c) % c);
        const int b = (int)(i / ((size_t)c * c));
        const int4 cr = crops[b]; // {input, y0, x0, target}
        const size_t src = ((size_t)cr.x * H + cr.y + y) * W + cr.z + x;
        const size_t src_t = ((size_t)cr.w * H + cr.y + y) * W + cr.z + x;
        const uint4* s = reinterpret_cast<const uint4*>(feat + src * 32);
        uint4* d = reinterpret_cast<uint4*>(bf + i * 32);
        for (int k = 0; k < 4; ++k) d[k] = s[k];
        bb[i] = base[src];
        bt[i] = tgt[src_t];
    }
}

inline unsigned grid_for(size_t n) { return (unsigned)std::min<size_t>((n + 255) / 256, 152 * 32); }
inline int pad32(int c) { return (c + 31) / 32 * 32; }
inline int pad16(int c) { return (c + 15) / 16 * 16; }

} // namespace

// ---------------------------------------------------------------------------
// Network
// ---------------------------------------------------------------------------
struct TRef {
    bf16* p;
    int cs, co, c; // channel stride, offset, count
};

struct Layer {
    int cin, cout, rows, cout_k;
    bool relu;
    size_t w_off, b_off;   // offsets in the FP32 parameter vector
    size_t wf_off, wb_off; // offsets in the BF16 packed weight buffers
};

struct Acts {
    int n = 0, h = 0, w = 0;
    DeviceBuffer<bf16> buf; // one arena for every activation and activation gradient
    DeviceBuffer<float> head; // FP32 network output [P][4] (log1p radiance, 0)
    std::vector<size_t> off;
    bf16* at(int k) { return buf.ptr + off[k]; }
};

// tensor ids in Acts
enum {
    T_IN, T_E0A, T_CAT0, T_P0, T_E1A, T_CAT1, T_P1, T_E2A, T_CAT2, T_P2, T_E3A, T_CAT3, T_P3, T_E4A, T_E4B, T_D3A, T_D3B,
    T_D2A, T_D2B, T_D1A, T_D1B, T_D0A, T_D0B, T_OUT,
    // gradients
    G_OUT, G_D0B, G_D0A, G_CAT0, G_D1B, G_D1A, G_CAT1, G_D2B, G_D2A, G_CAT2, G_D3B, G_D3A, G_CAT3, G_E4B, G_E4A, G_P3,
    G_E3B, G_E3A, G_P2, G_E2B, G_E2A, G_P1, G_E1B, G_E1A, G_P0, G_E0B, G_E0A,
    T_COUNT
};

} // namespace kf

// The object behind the C-ABI's kf_denoiser handle.
struct kf_denoiser_s {
    kf_renderer_s* r = nullptr;
    std::vector<kf::Layer> L;
    size_t nparams = 0, nwf = 0, nwb = 0;
    kf::DeviceBuffer<float> params, grads, m, v;
    kf::DeviceBuffer<__nv_bfloat16> wf, wb;
    kf::DeviceBuffer<__nv_bfloat16> wf0_16; // first layer, input channels 0..15 (inference)
    kf::DeviceBuffer<float> loss;
    int step = 0;
    bool packed = false;
    kf::Acts acts;
    // dataset: ds_n inputs (features + residual base), ds_targets targets; input k is
    // paired with target ds_tgt_of[k]. Capacities grow by doubling.
    int ds_h = 0, ds_w = 0, ds_n = 0, ds_targets = 0;
    size_t ds_cap_in = 0, ds_cap_tgt = 0;
    std::vector<int> ds_tgt_of;
    kf::DeviceBuffer<__nv_bfloat16> ds_feat;
    kf::DeviceBuffer<float4> ds_base, ds_tgt;
    kf::DeviceBuffer<__nv_bfloat16> batch_feat;
    kf::DeviceBuffer<float4> batch_base, batch_tgt;
    kf::DeviceBuffer<int4> crops;
    std::mt19937 rng{1234};
};

namespace kf {

namespace {

// (cin, cout, relu) of the 19 convolutions in order (encoder, bottleneck, decoder, head)
const int kLayers[19][3] = {{32, 32, 1},   {32, 32, 1},   {32, 64, 1},   {64, 64, 1},   {64, 96, 1},
                            {96, 96, 1},   {96, 128, 1},  {128, 128, 1}, {128, 160, 1}, {160, 160, 1},
                            {288, 128, 1}, {128, 128, 1}, {224, 96, 1},  {96, 96, 1},   {160, 64, 1},
                            {64, 64, 1},   {96, 32, 1},   {32, 32, 1},   {32, 3, 0}};

void build_layers(kf_denoiser_impl& d) {
    d.L.clear();
    size_t po = 0, fo = 0, bo = 0;
    for (const auto& l : kLayers) {
        Layer x;
        x.cin = l[0];
        x.cout = l[1];
        x.relu = l[2] != 0;
        x.rows = pad16(x.cout);
        x.cout_k = pad32(x.cout);
        x.w_off = po;
        po += (size_t)9 * x.cout * x.cin;
        x.b_off = po;
        po += (size_t)x.cout;
        x.wf_off = fo;
        fo += ((size_t)9 * x.rows * x.cin + 7) / 8 * 8;
        x.wb_off = bo;
        bo += ((size_t)9 * x.cin * x.cout_k + 7) / 8 * 8;
        d.L.push_back(x);
    }
    d.nparams = po;
    d.nwf = fo;
    d.nwb = bo;
}

void init_params(kf_denoiser_impl& d, uint32_t seed, cudaStream_t st) {
    std::vector<float> h(d.nparams, 0.0f);
    std::mt19937 g(seed);
    for (const Layer& l : d.L) {
        std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / (9.0f * (float)l.cin)));
        const float scale = l.relu ? 1.0f : 0.1f;
        for (size_t i = 0; i < (size_t)9 * l.cout * l.cin; ++i) h[l.w_off + i] = nd(g) * scale;
    }
    d.params.upload(h.data(), h.size(), st);
    d.grads.resize(d.nparams, st);
    d.m.resize(d.nparams, st);
    d.v.resize(d.nparams, st);
    KF_CUDA_CHECK(cudaMemsetAsync(d.m.ptr, 0, d.m.bytes(), st));
    KF_CUDA_CHECK(cudaMemsetAsync(d.v.ptr, 0, d.v.bytes(), st));
    d.wf.resize(d.nwf, st);
    d.wb.resize(d.nwb, st);
    d.wf0_16.resize((size_t)9 * d.L[0].rows * 16, st);
    KF_CUDA_CHECK(cudaMemsetAsync(d.wf.ptr, 0, d.wf.bytes(), st));
    KF_CUDA_CHECK(cudaMemsetAsync(d.wf0_16.ptr, 0, d.wf0_16.bytes(), st));
    KF_CUDA_CHECK(cudaMemsetAsync(d.wb.ptr, 0, d.wb.bytes(), st));
    d.loss.resize(4, st);
    d.packed = false;
    d.step = 0;
}

// The BF16 weights from the master weights, after an Adam step on them when `step` is its number
// (0: no step).
void update(kf_denoiser_impl& d, int step, float lr, cudaStream_t st) {
    UpdateTable t{};
    int blocks = 0;
    for (size_t k = 0; k < d.L.size(); ++k) {
        const Layer& l = d.L[k];
        t.first[k] = blocks;
        blocks += 9 * (l.cin / 32) * (l.cout_k / 32);
        t.cin[k] = l.cin;
        t.cout[k] = l.cout;
        t.rows[k] = l.rows;
        t.cout_k[k] = l.cout_k;
        t.w_off[k] = (uint32_t)l.w_off;
        t.b_off[k] = (uint32_t)l.b_off;
        t.wf_off[k] = (uint32_t)l.wf_off;
        t.wb_off[k] = (uint32_t)l.wb_off;
    }
    t.first[d.L.size()] = blocks;
    const float b1 = 0.9f, b2 = 0.999f;
    const float bc1 = 1.0f - std::pow(b1, (float)step), bc2 = 1.0f - std::pow(b2, (float)step);
    k_update<<<blocks, kUpdateThreads, 0, st>>>(t, d.params.ptr, d.grads.ptr, d.m.ptr, d.v.ptr, d.wf.ptr, d.wb.ptr,
                                                d.wf0_16.ptr, step, lr, b1, b2, 1e-8f, bc1, bc2);
    KF_CUDA_CHECK(cudaGetLastError());
    d.packed = true;
}
void pack(kf_denoiser_impl& d, cudaStream_t st) { update(d, 0, 0.0f, st); }

// channel counts and spatial level of every tensor
struct TDesc {
    int c, level;
};
const TDesc kT[T_COUNT] = {
    {32, 0}, {32, 0}, {96, 0}, {32, 1}, {64, 1}, {160, 1}, {64, 2}, {96, 2}, {224, 2}, {96, 3}, {128, 3}, {288, 3},
    {128, 4}, {160, 4}, {160, 4}, {128, 3}, {128, 3}, {96, 2}, {96, 2}, {64, 1}, {64, 1}, {32, 0}, {32, 0}, {32, 0},
    // gradients
    {32, 0}, {32, 0}, {32, 0}, {96, 0}, {64, 1}, {64, 1}, {160, 1}, {96, 2}, {96, 2}, {224, 2}, {128, 3}, {128, 3},
    {288, 3}, {160, 4}, {160, 4}, {128, 4}, {128, 3}, {128, 3}, {96, 3}, {96, 2}, {96, 2}, {64, 2}, {64, 1}, {64, 1},
    {32, 1}, {32, 0}, {32, 0}};

void ensure_acts(kf_denoiser_impl& d, int n, int h, int w, cudaStream_t st) {
    Acts& a = d.acts;
    if (a.n == n && a.h == h && a.w == w) return;
    KF_REQUIRE(h % 16 == 0 && w % 16 == 0, KF_ERR_INVALID_ARGUMENT, "denoiser tensors need H and W divisible by 16");
    a.off.assign(T_COUNT, 0);
    size_t total = 0;
    const size_t P0 = (size_t)n * h * w;
    for (int k = 0; k < T_COUNT; ++k) {
        a.off[k] = total;
        total += (P0 >> (2 * kT[k].level)) * kT[k].c;
        total = (total + 127) / 128 * 128;
    }
    a.buf.resize(total, st);
    KF_CUDA_CHECK(cudaMemsetAsync(a.buf.ptr, 0, a.buf.bytes(), st));
    a.head.resize(P0 * 4, st);
    KF_CUDA_CHECK(cudaMemsetAsync(a.head.ptr, 0, a.head.bytes(), st));
    a.n = n;
    a.h = h;
    a.w = w;
}

struct Ctx {
    kf_denoiser_impl& d;
    cudaStream_t st;
    int n, h, w;
    TRef in;           // the 32-channel input (16 channels when the first convolution takes those)
    bool keep = false; // a backward pass follows
    int H(int level) const { return h >> level; }
    int W(int level) const { return w >> level; }
    size_t P(int level) const { return (size_t)n * H(level) * W(level); }
};

// The convolution, with what `f` asks its epilogue to do besides; true: it pooled as well.
bool conv_fwd(Ctx& c, int li, int level, TRef x, TRef y, ConvFuse f = ConvFuse()) {
    const Layer& l = c.d.L[li];
    f.settled = li > 0; // behind the first convolution, whatever wrote the weights is complete
    return conv3x3_bf16(x.p, c.n, c.H(level), c.W(level), x.cs, c.d.wf.ptr + l.wf_off, l.rows,
                        c.d.params.ptr + l.b_off, l.cout, l.relu, y.p, y.cs, y.co, c.st, nullptr, &f);
}

// The weight gradients run on the renderer's second stream, beside the backward-data chain: both
// are rows of small kernels that leave most of the GPU idle (a step of 16 crops of 128 x 128
// 904 -> 838 us; a tensor's gradient buffer is written once per step, so nothing is shared but dz).
// Backward of z = conv(x) + b from dz = dL/dz (dense, the layer's channels padded to 32): adds dW
// and db; with gx.p, gx = dL/dx, masked by x > 0 where x is a ReLU's output that nothing else
// reads (mask: gx is then the dL/dz of the layer before).
void conv_bwd(Ctx& c, int li, int level, TRef x, TRef dz, TRef gx, bool mask) {
    const Layer& l = c.d.L[li];
    kf_renderer_s* r = c.d.r;
    KF_CUDA_CHECK(cudaEventRecord(r->ev_fork, c.st)); // dz is queued
    KF_CUDA_CHECK(cudaStreamWaitEvent(r->stream2, r->ev_fork, 0));
    conv3x3_wgrad_bf16(x.p + x.co, x.cs, c.n, c.H(level), c.W(level), l.cin, dz.p, l.cout_k, l.cout,
                       c.d.grads.ptr + l.w_off, c.d.grads.ptr + l.b_off, r->stream2);
    if (gx.p) {
        ConvFuse f;
        f.settled = true; // the weights were packed before the forward pass
        if (mask) {
            f.mask = x.p;
            f.mask_cs = x.cs;
            f.mask_co = x.co;
        }
        conv3x3_bf16(dz.p, c.n, c.H(level), c.W(level), l.cout_k, c.d.wb.ptr + l.wb_off, l.cin, nullptr, l.cin, false,
                     gx.p, gx.cs, gx.co, c.st, nullptr, &f);
    }
    KF_CUDA_CHECK(cudaGetLastError());
}

TRef T(Acts& a, int k) { return TRef{a.at(k), kT[k].c, 0, kT[k].c}; }
TRef S(Acts& a, int k, int off, int cnt) { return TRef{a.at(k), kT[k].c, off, cnt}; }

// conv into y, and 2x2 pooling of y into `pooled` (at level + 1) in the convolution's epilogue: for the
// network's layers (at most 128 channels at even sizes) both convolution kernels do it
void conv_pool(Ctx& c, int li, int level, TRef x, TRef y, TRef pooled) {
    ConvFuse f;
    f.pool_out = pooled.p;
    KF_REQUIRE(conv_fwd(c, li, level, x, y, f), KF_ERR_INTERNAL, "a convolution did not pool its output");
}
// conv, then nearest 2x upsampling of its output into the channel slice `up` (at level - 1), both
// in the convolution's epilogue; the output itself goes to y where a backward pass will read it.
// The four copies are what HBM has to take; a pass of its own read the output again and added its
// length to the multiplication's, which now hides most of the stores. At 1920 x 1088, convolution
// and pass: 92 -> 82 us into the full resolution, 43 -> 35 and 21 -> 20 below; the network 801 -> 777.
void conv_up(Ctx& c, int li, int level, TRef x, TRef y, TRef up) {
    ConvFuse f;
    f.up_out = up.p;
    f.up_cs = up.cs;
    f.up_co = up.co;
    f.up_only = !c.keep;
    conv_fwd(c, li, level, x, y, f);
}

// out (float4 pixels; the activations' head buffer or the caller's) = network(c.in) + base (FP32
// residual, optional), channel 3 zero. in16: c.in holds 16-channel features (the first convolution
// then reads half the bytes and does half the MMAs; channels 16..31 of the 32-channel input are
// zero, so the values are the same).
void forward(Ctx& c, const float* base, float* out, bool in16 = false) {
    Acts& a = c.d.acts;
    if (in16) {
        const Layer& l = c.d.L[0];
        conv3x3_bf16(c.in.p, c.n, c.h, c.w, 16, c.d.wf0_16.ptr, l.rows, c.d.params.ptr + l.b_off, l.cout, l.relu,
                     a.at(T_E0A), 32, 0, c.st);
    } else {
        conv_fwd(c, 0, 0, c.in, T(a, T_E0A));
    }
    conv_pool(c, 1, 0, T(a, T_E0A), S(a, T_CAT0, 64, 32), T(a, T_P0));
    conv_fwd(c, 2, 1, T(a, T_P0), T(a, T_E1A));
    conv_pool(c, 3, 1, T(a, T_E1A), S(a, T_CAT1, 96, 64), T(a, T_P1));
    conv_fwd(c, 4, 2, T(a, T_P1), T(a, T_E2A));
    conv_pool(c, 5, 2, T(a, T_E2A), S(a, T_CAT2, 128, 96), T(a, T_P2));
    conv_fwd(c, 6, 3, T(a, T_P2), T(a, T_E3A));
    conv_pool(c, 7, 3, T(a, T_E3A), S(a, T_CAT3, 160, 128), T(a, T_P3));
    conv_fwd(c, 8, 4, T(a, T_P3), T(a, T_E4A));
    conv_up(c, 9, 4, T(a, T_E4A), T(a, T_E4B), S(a, T_CAT3, 0, 160));
    conv_fwd(c, 10, 3, T(a, T_CAT3), T(a, T_D3A));
    conv_up(c, 11, 3, T(a, T_D3A), T(a, T_D3B), S(a, T_CAT2, 0, 128));
    conv_fwd(c, 12, 2, T(a, T_CAT2), T(a, T_D2A));
    conv_up(c, 13, 2, T(a, T_D2A), T(a, T_D2B), S(a, T_CAT1, 0, 96));
    conv_fwd(c, 14, 1, T(a, T_CAT1), T(a, T_D1A));
    conv_up(c, 15, 1, T(a, T_D1A), T(a, T_D1B), S(a, T_CAT0, 0, 64));
    conv_fwd(c, 16, 0, T(a, T_CAT0), T(a, T_D0A));
    conv_fwd(c, 17, 0, T(a, T_D0A), T(a, T_D0B));
    {
        const Layer& l = c.d.L[18];
        ConvFuse f;
        f.settled = true;
        f.head4 = true;
        f.base = base;
        conv3x3_bf16(a.at(T_D0B), c.n, c.h, c.w, 32, c.d.wf.ptr + l.wf_off, l.rows, c.d.params.ptr + l.b_off, l.cout,
                     false, nullptr, 4, 0, c.st, out, &f);
    }
    KF_CUDA_CHECK(cudaGetLastError());
}

void pool_bwd_add(Ctx& c, TRef gy_low, TRef gskip, int level_hi, TRef y, TRef gx) {
    const size_t n = c.P(level_hi) * gx.c / 8;
    launch_overlapped(k_pool_bwd_add, dim3(grid_for(n)), dim3(256), 0, c.st, gy_low.p, gskip.p, gskip.cs, gskip.co,
                      gx.c, c.n, c.H(level_hi), c.W(level_hi), y.p, y.cs, y.co, gx.p);
}
void up_bwd(Ctx& c, TRef gy_slice, int level_hi, TRef y, TRef gx_low) {
    const size_t n = c.P(level_hi + 1) * gx_low.c / 8;
    launch_overlapped(k_up_bwd, dim3(grid_for(n)), dim3(256), 0, c.st, gy_slice.p, gy_slice.cs, gy_slice.co, gx_low.c,
                      c.n, c.H(level_hi), c.W(level_hi), y.p, gx_low.p);
}

// Every gradient tensor G_* of a ReLU layer's output holds dL/dz: the ReLU's mask is applied by
// whatever writes it (the backward-data convolution's epilogue, the upsampling and pooling
// passes), with the rounded values a separate pass over gradient and output would mask.
void backward(Ctx& c) {
    Acts& a = c.d.acts;
    TRef none{nullptr, 0, 0, 0};
    conv_bwd(c, 18, 0, T(a, T_D0B), T(a, G_OUT), T(a, G_D0B), true);
    conv_bwd(c, 17, 0, T(a, T_D0A), T(a, G_D0B), T(a, G_D0A), true);
    conv_bwd(c, 16, 0, T(a, T_CAT0), T(a, G_D0A), T(a, G_CAT0), false);
    up_bwd(c, S(a, G_CAT0, 0, 64), 0, T(a, T_D1B), T(a, G_D1B));
    conv_bwd(c, 15, 1, T(a, T_D1A), T(a, G_D1B), T(a, G_D1A), true);
    conv_bwd(c, 14, 1, T(a, T_CAT1), T(a, G_D1A), T(a, G_CAT1), false);
    up_bwd(c, S(a, G_CAT1, 0, 96), 1, T(a, T_D2B), T(a, G_D2B));
    conv_bwd(c, 13, 2, T(a, T_D2A), T(a, G_D2B), T(a, G_D2A), true);
    conv_bwd(c, 12, 2, T(a, T_CAT2), T(a, G_D2A), T(a, G_CAT2), false);
    up_bwd(c, S(a, G_CAT2, 0, 128), 2, T(a, T_D3B), T(a, G_D3B));
    conv_bwd(c, 11, 3, T(a, T_D3A), T(a, G_D3B), T(a, G_D3A), true);
    conv_bwd(c, 10, 3, T(a, T_CAT3), T(a, G_D3A), T(a, G_CAT3), false);
    up_bwd(c, S(a, G_CAT3, 0, 160), 3, T(a, T_E4B), T(a, G_E4B));
    conv_bwd(c, 9, 4, T(a, T_E4A), T(a, G_E4B), T(a, G_E4A), true);
    conv_bwd(c, 8, 4, T(a, T_P3), T(a, G_E4A), T(a, G_P3), false);
    pool_bwd_add(c, T(a, G_P3), S(a, G_CAT3, 160, 128), 3, S(a, T_CAT3, 160, 128), T(a, G_E3B));
    conv_bwd(c, 7, 3, T(a, T_E3A), T(a, G_E3B), T(a, G_E3A), true);
    conv_bwd(c, 6, 3, T(a, T_P2), T(a, G_E3A), T(a, G_P2), false);
    pool_bwd_add(c, T(a, G_P2), S(a, G_CAT2, 128, 96), 2, S(a, T_CAT2, 128, 96), T(a, G_E2B));
    conv_bwd(c, 5, 2, T(a, T_E2A), T(a, G_E2B), T(a, G_E2A), true);
    conv_bwd(c, 4, 2, T(a, T_P1), T(a, G_E2A), T(a, G_P1), false);
    pool_bwd_add(c, T(a, G_P1), S(a, G_CAT1, 96, 64), 1, S(a, T_CAT1, 96, 64), T(a, G_E1B));
    conv_bwd(c, 3, 1, T(a, T_E1A), T(a, G_E1B), T(a, G_E1A), true);
    conv_bwd(c, 2, 1, T(a, T_P0), T(a, G_E1A), T(a, G_P0), false);
    pool_bwd_add(c, T(a, G_P0), S(a, G_CAT0, 64, 32), 0, S(a, T_CAT0, 64, 32), T(a, G_E0B));
    conv_bwd(c, 1, 0, T(a, T_E0A), T(a, G_E0B), T(a, G_E0A), true);
    conv_bwd(c, 0, 0, c.in, T(a, G_E0A), none, false);
    KF_CUDA_CHECK(cudaEventRecord(c.d.r->ev_join, c.d.r->stream2));
    KF_CUDA_CHECK(cudaStreamWaitEvent(c.st, c.d.r->ev_join, 0));
}

} // namespace

// ---------------------------------------------------------------------------
// Public operations
// ---------------------------------------------------------------------------
kf_denoiser_impl* denoiser_create(kf_renderer_s* r, uint32_t seed) {
    auto d = new kf_denoiser_impl();
    d->r = r;
    build_layers(*d);
    init_params(*d, seed, r->stream);
    d->rng.seed(seed ^ 0x5bd1e995u);
    return d;
}
void denoiser_destroy(kf_denoiser_impl* d) { delete d; }
size_t denoiser_num_params(const kf_denoiser_impl* d) { return d->nparams; }
uint32_t denoiser_num_views(const kf_denoiser_impl* d) { return (uint32_t)d->ds_n; }
kf_renderer_s* denoiser_renderer(const kf_denoiser_impl* d) { return d->r; }

void denoiser_get_params(kf_denoiser_impl* d, float* out, size_t n) {
    KF_REQUIRE(n >= d->nparams, KF_ERR_OUT_OF_RANGE, "parameter buffer too small");
    KF_CUDA_CHECK(cudaMemcpyAsync(out, d->params.ptr, d->nparams * 4, cudaMemcpyDeviceToHost, d->r->stream));
    KF_CUDA_CHECK(cudaStreamSynchronize(d->r->stream));
}
void denoiser_set_params(kf_denoiser_impl* d, const float* in, size_t n) {
    KF_REQUIRE(n == d->nparams, KF_ERR_INVALID_ARGUMENT, "parameter count mismatch");
    KF_CUDA_CHECK(cudaMemcpyAsync(d->params.ptr, in, d->nparams * 4, cudaMemcpyHostToDevice, d->r->stream));
    KF_CUDA_CHECK(cudaMemsetAsync(d->m.ptr, 0, d->m.bytes(), d->r->stream));
    KF_CUDA_CHECK(cudaMemsetAsync(d->v.ptr, 0, d->v.bytes(), d->r->stream));
    KF_CUDA_CHECK(cudaStreamSynchronize(d->r->stream));
    d->packed = false;
    d->step = 0;
}

namespace {

// The network over the caller's tensors. They are read and written in place where the kernels can
// (this device's memory at 16-byte boundaries), else through the activations' buffers. At
// 1920 x 1088 the copy of the input costs 41 us and that of the output 10 (778 us without both);
// the residual is added in the last convolution's epilogue, a pass of 12 us before. The API calls
// return when the stream is done, so nothing outlives the caller's tensors.
Ctx run_forward(kf_denoiser_impl* d, const void* feat, const void* base, int n, int h, int w, void* out, bool keep) {
    cudaStream_t st = d->r->stream;
    ensure_acts(*d, n, h, w, st);
    if (!d->packed) pack(*d, st);
    const auto in_place = [](const void* p) {
        cudaPointerAttributes at{};
        int dev = -1;
        if (((uintptr_t)p & 15) != 0) return false;
        if (cudaPointerGetAttributes(&at, p) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return at.type == cudaMemoryTypeDevice && at.device == dev;
    };
    Acts& a = d->acts;
    Ctx c{*d, st, n, h, w, T(a, T_IN), keep};
    if (in_place(feat))
        c.in.p = static_cast<bf16*>(const_cast<void*>(feat));
    else
        KF_CUDA_CHECK(cudaMemcpyAsync(c.in.p, feat, (size_t)n * h * w * 32 * 2, cudaMemcpyDeviceToDevice, st));
    // the head is written pixel by pixel while the residual is read: the same tensor, or one apart
    const uintptr_t ob = (uintptr_t)out, bb = (uintptr_t)base, bytes = (uintptr_t)n * h * w * 16;
    const bool apart = !base || ob == bb || ob + bytes <= bb || bb + bytes <= ob;
    const bool direct = out && apart && in_place(out);
    forward(c, static_cast<const float*>(base), direct ? static_cast<float*>(out) : a.head.ptr);
    if (out && !direct)
        KF_CUDA_CHECK(cudaMemcpyAsync(out, a.head.ptr, (size_t)n * h * w * 16, cudaMemcpyDeviceToDevice, st));
    return c;
}

} // namespace

// out: [n, h, w, 4] FP32 device buffer (channels 0..2 = prediction in g space, 3 = 0);
// base: optional FP32 residual [n, h, w] float4 added to the network output.
void denoiser_forward(kf_denoiser_impl* d, const void* feat, const void* base, int n, int h, int w, void* out) {
    run_forward(d, feat, base, n, h, w, out, false);
}

float denoiser_train_step(kf_denoiser_impl* d, const void* feat, const void* base, const float* tgt, int n, int h,
                          int w, float lr, float* grads_out, bool apply_update) {
    cudaStream_t st = d->r->stream;
    Ctx c = run_forward(d, feat, nullptr, n, h, w, nullptr, true); // the loss adds the residual
    Acts& a = d->acts;
    KF_CUDA_CHECK(cudaMemsetAsync(d->loss.ptr, 0, sizeof(float), st));
    const unsigned tiles = (unsigned)n * (unsigned)((w + kLossW - 1) / kLossW) * (unsigned)((h + kLossH - 1) / kLossH);
    k_loss<<<tiles, kLossW * kLossH, 0, st>>>(reinterpret_cast<const float4*>(a.head.ptr),
                                              static_cast<const float4*>(base), reinterpret_cast<const float4*>(tgt), n,
                                              h, w, 0.5f, d->loss.ptr, a.at(G_OUT));
    KF_CUDA_CHECK(cudaGetLastError());
    KF_CUDA_CHECK(cudaMemsetAsync(d->grads.ptr, 0, d->grads.bytes(), st));
    backward(c);
    if (grads_out)
        KF_CUDA_CHECK(cudaMemcpyAsync(grads_out, d->grads.ptr, d->nparams * 4, cudaMemcpyDeviceToDevice, st));
    if (apply_update) {
        update(*d, ++d->step, lr, st);
    }
    float loss = 0.0f;
    KF_CUDA_CHECK(cudaMemcpyAsync(&loss, d->loss.ptr, sizeof(float), cudaMemcpyDeviceToHost, st));
    KF_CUDA_CHECK(cudaStreamSynchronize(st));
    return loss;
}

// Features (and residual base) of a camera's current render targets, padded to [1][Hp][Wp].
static void camera_features(kf_camera_s* c, uint32_t samples, bf16* out, float4* base, int Hp, int Wp,
                            cudaStream_t st, bool ch16 = false) {
    const float spp_feature = std::log2((float)std::max(samples, 1u)) / 8.0f;
    const unsigned grid = grid_for((size_t)Hp * Wp);
    if (ch16)
        k_pack_features<16><<<grid, 256, 0, st>>>(c->accum.ptr, c->albedo.ptr, c->normal.ptr, c->depth.ptr,
                                                  spp_feature, c->target_h, c->target_w, Hp, Wp, out, base);
    else
        k_pack_features<32><<<grid, 256, 0, st>>>(c->accum.ptr, c->albedo.ptr, c->normal.ptr, c->depth.ptr,
                                                  spp_feature, c->target_h, c->target_w, Hp, Wp, out, base);
    KF_CUDA_CHECK(cudaGetLastError());
}

namespace {
// kuafu's frame state, restored when a training render leaves its scope
struct FrameStateGuard {
    kf_renderer_s* r;
    uint32_t accumulate;
    explicit FrameStateGuard(kf_renderer_s* rr) : r(rr), accumulate(rr->cfg.accumulate_frames) {}
    ~FrameStateGuard() {
        r->frame_count = -1;
        r->cfg.accumulate_frames = accumulate;
    }
};

template <class T> void grow(DeviceBuffer<T>& b, size_t old_n, size_t new_n, cudaStream_t st) {
    DeviceBuffer<T> nb;
    nb.resize(new_n, st);
    if (old_n) KF_CUDA_CHECK(cudaMemcpyAsync(nb.ptr, b.ptr, old_n * sizeof(T), cudaMemcpyDeviceToDevice, st));
    KF_CUDA_CHECK(cudaStreamSynchronize(st));
    b = std::move(nb);
}
} // namespace

void denoiser_add_view(kf_denoiser_impl* d, kf_scene_s* s, kf_camera_s* c, const uint32_t* low_spp,
                       uint32_t num_inputs, uint32_t high_spp, uint32_t high_frames) {
    kf_renderer_s* r = d->r;
    cudaStream_t st = r->stream;
    KF_REQUIRE(c->width % 16 == 0 && c->height % 16 == 0, KF_ERR_INVALID_ARGUMENT,
               "training views need width and height divisible by 16");
    if (d->ds_n == 0) {
        d->ds_h = c->height;
        d->ds_w = c->width;
    }
    KF_REQUIRE(c->width == d->ds_w && c->height == d->ds_h, KF_ERR_INVALID_ARGUMENT,
               "all training views must have the same size");
    const size_t npix = (size_t)c->width * c->height;
    const size_t k = (size_t)d->ds_n, t = (size_t)d->ds_targets;
    if (k + num_inputs > d->ds_cap_in) {
        const size_t cap = std::max<size_t>({k + num_inputs, 2 * d->ds_cap_in, 8});
        grow(d->ds_feat, npix * 32 * k, npix * 32 * cap, st);
        grow(d->ds_base, npix * k, npix * cap, st);
        d->ds_cap_in = cap;
    }
    if (t + 1 > d->ds_cap_tgt) {
        const size_t cap = std::max<size_t>({t + 1, 2 * d->ds_cap_tgt, 8});
        grow(d->ds_tgt, npix * t, npix * cap, st);
        d->ds_cap_tgt = cap;
    }
    FrameStateGuard guard(r);
    r->cfg.accumulate_frames = 1;
    // noisy inputs: one frame of low_spp[i] samples each (every render takes a new frame
    // index, so the inputs' random streams and the target's are independent)
    for (uint32_t i = 0; i < num_inputs; ++i) {
        r->frame_count = -1;
        render_frame(r, s, c, low_spp[i]);
        camera_features(c, low_spp[i], d->ds_feat.ptr + npix * 32 * (k + i), d->ds_base.ptr + npix * (k + i),
                        c->height, c->width, st);
    }
    // target: high_frames frames of high_spp samples, averaged from the FP64 accumulation
    r->frame_count = -1;
    for (uint32_t f = 0; f < high_frames; ++f) render_frame(r, s, c, high_spp);
    k_target_from_sum64<<<grid_for(npix), 256, 0, st>>>(c->sum64.ptr, npix, d->ds_tgt.ptr + npix * t);
    KF_CUDA_CHECK(cudaGetLastError());
    KF_CUDA_CHECK(cudaStreamSynchronize(st));
    for (uint32_t i = 0; i < num_inputs; ++i) d->ds_tgt_of.push_back((int)t);
    d->ds_n += (int)num_inputs;
    ++d->ds_targets;
}

float denoiser_train(kf_denoiser_impl* d, uint32_t iters, uint32_t batch, uint32_t crop, float lr) {
    KF_REQUIRE(d->ds_n > 0, KF_ERR_STATE, "the denoiser has no training views");
    KF_REQUIRE(crop % 16 == 0 && (int)crop <= d->ds_h && (int)crop <= d->ds_w && batch > 0, KF_ERR_INVALID_ARGUMENT,
               "crop must be a multiple of 16 no larger than the training views");
    cudaStream_t st = d->r->stream;
    const size_t per = (size_t)crop * crop;
    d->batch_feat.resize(per * 32 * batch, st);
    d->batch_base.resize(per * batch, st);
    d->batch_tgt.resize(per * batch, st);
    d->crops.resize(batch, st);
    std::vector<int4> cr(batch);
    double acc = 0.0;
    for (uint32_t it = 0; it < iters; ++it) {
        for (uint32_t b = 0; b < batch; ++b) {
            cr[b].x = (int)(d->rng() % (uint32_t)d->ds_n);
            cr[b].y = (int)(d->rng() % (uint32_t)(d->ds_h - crop + 1));
            cr[b].z = (int)(d->rng() % (uint32_t)(d->ds_w - crop + 1));
            cr[b].w = d->ds_tgt_of[(size_t)cr[b].x];
        }
        d->crops.upload(cr.data(), batch, st);
        k_gather_crops<<<grid_for(per * batch), 256, 0, st>>>(d->ds_feat.ptr, d->ds_base.ptr, d->ds_tgt.ptr, d->ds_h,
                                                              d->ds_w, d->crops.ptr, (int)batch, (int)crop,
                                                              d->batch_feat.ptr, d->batch_base.ptr, d->batch_tgt.ptr);
        acc += denoiser_train_step(d, d->batch_feat.ptr, d->batch_base.ptr,
                                   reinterpret_cast<const float*>(d->batch_tgt.ptr), (int)batch, (int)crop, (int)crop,
                                   lr, nullptr, true);
    }
    return iters ? (float)(acc / iters) : 0.0f;
}

void denoiser_camera_features(kf_denoiser_impl* d, kf_camera_s* c, void* feat, float* base) {
    kf_renderer_s* r = d->r;
    const int Hp = (c->target_h + 15) / 16 * 16, Wp = (c->target_w + 15) / 16 * 16;
    const uint32_t frames = (r->cfg.accumulate_frames && r->frame_count >= 0) ? (uint32_t)r->frame_count + 1u : 1u;
    camera_features(c, frames * std::max(r->stats.last_spp, 1u), static_cast<bf16*>(feat),
                    reinterpret_cast<float4*>(base), Hp, Wp, r->stream);
}

void denoiser_apply(kf_denoiser_impl* d, kf_camera_s* c) {
    kf_renderer_s* r = d->r;
    cudaStream_t st = r->stream;
    KF_REQUIRE(c->has_frame, KF_ERR_STATE, "the camera has no frame to denoise");
    const int Hp = (c->target_h + 15) / 16 * 16, Wp = (c->target_w + 15) / 16 * 16;
    ensure_acts(*d, 1, Hp, Wp, st);
    if (!d->packed) pack(*d, st);
    const uint32_t frames = (r->cfg.accumulate_frames && r->frame_count >= 0) ? (uint32_t)r->frame_count + 1u : 1u;
    // frames the halo convolution takes (at least 96 wide) use the 16-channel input
    const bool in16 = Wp >= 96;
    camera_features(c, frames * std::max(r->stats.last_spp, 1u), d->acts.at(T_IN), nullptr, Hp, Wp, st, in16);
    Ctx cx{*d, st, 1, Hp, Wp, T(d->acts, T_IN)};
    forward(cx, nullptr, d->acts.head.ptr, in16);
    const size_t npix = (size_t)c->target_w * c->target_h;
    if (c->denoised.count != npix) c->denoised.resize(npix, st);
    k_unpack_residual<<<grid_for(npix), 256, 0, st>>>(reinterpret_cast<const float4*>(d->acts.head.ptr),
                                                      c->accum.ptr, c->target_h, c->target_w, Wp, c->denoised.ptr);
    KF_CUDA_CHECK(cudaGetLastError());
}

} // namespace kf

namespace kf {

void present_denoised(kf_renderer_s* r, kf_camera_s* c) {
    denoiser_apply(r->denoiser, c);
    launch_srgb(c->denoised.ptr, (uint32_t)c->denoised.count, c->bgra.ptr, r->stream);
    KF_CUDA_CHECK(cudaGetLastError());
}

} // namespace kf
