// kf_conv.cu — tcgen05 tensor-core kernels of the learned denoiser:
//
//   * 3x3 convolutions (forward and backward-data) of NHWC BF16 activations, FP32 accumulation
//     in TMEM, bias / ReLU / pooling / ReLU-mask epilogues into a channel slice (so skip
//     concatenation costs nothing): k_conv_halo for wide images, k_conv_tile for narrow ones,
//     and k_tc for more input channels than k_conv_tile holds (one TMA box of 128 output pixels
//     x 32 input channels per filter tap);
//   * weight and bias gradients (k_wgrad);
//   * K-major GEMM D += A * B^T (k_tc): 2D TMA, 128-byte swizzle, split-K with FP32 atomics.
//
// In each, one thread issues TMA into mbarrier-guarded shared memory, another the MMAs, and
// other warps drain TMEM. A kernel lets the next one of the stream start only when it holds its own
// TMEM: the next one may take its columns before it waits for this one to end, and an allocation
// waits without a bound. Every wait is bounded (~1 s of SM clock); on expiry the kernel records
// an error code, drains its own copies and frees its TMEM. A warp that goes on to warp-wide
// instructions (TMEM loads, shuffles, votes) waits and gives up as one (mbar_wait_warp): lanes
// that decide for themselves could leave the others alone in them. Only single-lane roles
// (the producers) wait by themselves.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "kf_conv.h"
#include "kf_tc.cuh"
#include "kf_util.h"

namespace kf {

__device__ uint32_t g_tc_error;

namespace {

constexpr long long kWaitBudget = 2000000000ll; // SM cycles (~1 s)

struct TcParams {
    int N, H, W, Cin; // conv: A tensor NHWC
    int Cout;         // valid output channels
    int bw, bh;       // conv output tile (bw * bh = 128)
    int tiles_x, tiles_y;
    int n_tile;       // N columns per CTA
    int kchunks;      // conv: Cin / CK
    const float* bias;
    int relu;
    __nv_bfloat16* out;
    int out_cstride, out_coff;
    float* outf;      // gemm output (atomic add); conv: FP32 output instead of BF16 when set
    int ldo, M_valid, N_valid;
    int k_iters, k_per_split;
    uint32_t tmem_cols;
};

__device__ __forceinline__ void set_error(uint32_t code) { atomicCAS(&g_tc_error, 0u, code); }

// MODE 0: implicit conv3x3 (4D A, 3D B); MODE 1: GEMM (2D A, 2D B).
template <int MODE, int SWZ, int kStages>
__global__ void __launch_bounds__(128, 1) k_tc(const __grid_constant__ CUtensorMap tmA,
                                               const __grid_constant__ CUtensorMap tmB, const TcParams p) {
    constexpr int CK = SWZ / 2;                     // BF16 elements per K chunk (one swizzle row)
    constexpr uint32_t LAYOUT = SWZ == 128 ? 2u : (SWZ == 64 ? 4u : 6u);
    constexpr uint32_t SBO = 8u * SWZ;              // 8 rows of SWZ bytes
    constexpr uint32_t A_BYTES = 128u * SWZ;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t B_BYTES = ((uint32_t)p.n_tile * SWZ + 1023u) & ~1023u;
    uint8_t* sA = smem;
    uint8_t* sB = smem + kStages * A_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(sB + kStages * B_BYTES);
    uint64_t* empty = full + kStages;
    uint64_t* done = empty + kStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    float* sbias = reinterpret_cast<float*>(tmem_slot + 4); // the tile's bias (0 where none)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // ---- tile coordinates ----
    int n_img = 0, x0 = 0, y0 = 0, m0 = 0;
    const int n0 = blockIdx.y * p.n_tile;
    int k_begin = 0, k_end = p.k_iters;
    if (MODE == 0) {
        const int t = blockIdx.x;
        const int per_img = p.tiles_x * p.tiles_y;
        n_img = t / per_img;
        const int r = t % per_img;
        y0 = (r / p.tiles_x) * p.bh;
        x0 = (r % p.tiles_x) * p.bw;
    } else {
        m0 = blockIdx.x * 128;
        k_begin = blockIdx.z * p.k_per_split;
        k_end = min(p.k_iters, k_begin + p.k_per_split);
    }
    const int nk = max(0, k_end - k_begin);

    if (warp == 0) tc::tmem_alloc(tmem_slot, p.tmem_cols);
    if (MODE == 0)
        for (int i = threadIdx.x; i < p.n_tile; i += blockDim.x)
            sbias[i] = (p.bias && n0 + i < p.Cout) ? p.bias[n0 + i] : 0.0f;
    if (threadIdx.x == 32) {
        for (int s = 0; s < kStages; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        tc::mbar_init(done, 1);
        tc::fence_barrier_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0) {
        // ---- producer: TMA ----
        bool ok = true;
        for (int i = 0; i < nk && ok; ++i) {
            const int s = i % kStages;
            if (i >= kStages && !tc::mbar_wait(&empty[s], ((i / kStages) - 1) & 1, kWaitBudget)) {
                set_error(1);
                ok = false;
                break;
            }
            const uint32_t b_bytes = (uint32_t)p.n_tile * SWZ;
            tc::mbar_arrive_expect_tx(&full[s], A_BYTES + b_bytes);
            const int k = k_begin + i;
            if (MODE == 0) {
                const int tap = k / p.kchunks, ch = (k % p.kchunks) * CK;
                const int dy = tap / 3 - 1, dx = tap % 3 - 1;
                tc::tma_load_4d(sA + s * A_BYTES, &tmA, &full[s], ch, x0 + dx, y0 + dy, n_img);
                tc::tma_load_3d(sB + s * B_BYTES, &tmB, &full[s], ch, n0, tap);
            } else {
                tc::tma_load_2d(sA + s * A_BYTES, &tmA, &full[s], k * CK, m0);
                tc::tma_load_2d(sB + s * B_BYTES, &tmB, &full[s], k * CK, n0);
            }
        }
        // drain: the last use of every stage must have landed before the CTA may exit
        for (int s = 0; s < kStages && s < nk; ++s) {
            const int last = ((nk - 1 - s) / kStages) * kStages + s;
            if (!tc::mbar_wait(&full[s], (last / kStages) & 1, kWaitBudget)) set_error(2);
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the warp stays converged, one elected lane issues ----
        const uint32_t elected = tc::elect_one();
        const uint32_t idesc = tc::idesc_bf16(128, (uint32_t)p.n_tile);
        for (int i = 0; i < nk; ++i) {
            const int s = i % kStages;
            if (!tc::mbar_wait_warp(&full[s], (i / kStages) & 1, kWaitBudget)) {
                set_error(3);
                break;
            }
            tc::fence_after_sync();
            const uint32_t a_addr = tc::smem_u32(sA + s * A_BYTES);
            const uint32_t b_addr = tc::smem_u32(sB + s * B_BYTES);
#pragma unroll
            for (int kk = 0; kk < CK / 16; ++kk) {
                const uint64_t ad = tc::smem_desc(a_addr + kk * 32, SBO, LAYOUT);
                const uint64_t bd = tc::smem_desc(b_addr + kk * 32, SBO, LAYOUT);
                tc::mma_bf16(tmem, ad, bd, idesc, (i > 0 || kk > 0) ? 1u : 0u, elected);
            }
            if (elected) tc::mma_commit(&empty[s]);
        }
        if (elected) tc::mma_commit(done);
    }

    // ---- epilogue: all 4 warps, warp w owns TMEM lanes [32w, 32w + 32) ----
    __syncwarp(); // warp 0: its producer lane
    const bool ready = nk == 0 || tc::mbar_wait_warp(done, 0, kWaitBudget);
    if (!ready) set_error(4);
    __syncwarp();
    tc::fence_after_sync();
    const int row = warp * 32 + lane;
    if (MODE == 0) {
        const int px = x0 + (row % p.bw), py = y0 + (row / p.bw);
        const bool valid = ready && nk > 0 && px < p.W && py < p.H;
        const size_t base = ((size_t)((size_t)n_img * p.H + py) * p.W + px) * p.out_cstride + p.out_coff;
        // 16 columns per TMEM wait: two loads in flight; bias from shared memory
        auto emit8 = [&](const uint32_t(&r)[8], int c) {
            const int co = n0 + c;
            if (!valid || co >= p.Cout) return;
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] = __uint_as_float(r[j]);
                if (p.bias && co + j < p.Cout) v[j] += sbias[c + j];
                if (p.relu) v[j] = fmaxf(v[j], 0.0f);
            }
            if (p.outf) { // FP32 output (a network head)
                for (int j = 0; j < 8 && co + j < p.Cout; ++j) p.outf[base + co + j] = v[j];
                return;
            }
            __nv_bfloat16* dst = p.out + base;
            if (co + 8 <= p.Cout && ((p.out_coff + co) & 7) == 0 && (p.out_cstride & 7) == 0) {
                __nv_bfloat162 q[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) q[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                *reinterpret_cast<uint4*>(dst + co) = *reinterpret_cast<const uint4*>(q);
            } else {
                for (int j = 0; j < 8 && co + j < p.Cout; ++j) dst[co + j] = __float2bfloat16_rn(v[j]);
            }
        };
        for (int c = 0; c < p.n_tile; c += 16) {
            uint32_t r0[8], r1[8];
            tc::tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, r0);
            tc::tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c + 8), r1);
            tc::tmem_ld_wait();
            emit8(r0, c);
            emit8(r1, c + 8);
        }
    } else {
        const int m = m0 + row;
        const bool valid = ready && nk > 0 && m < p.M_valid;
        for (int c = 0; c < p.n_tile; c += 8) {
            uint32_t r[8];
            tc::tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, r);
            tc::tmem_ld_wait();
            if (!valid) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int n = n0 + c + j;
                if (n < p.N_valid) atomicAdd(p.outf + (size_t)m * p.ldo + n, __uint_as_float(r[j]));
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, p.tmem_cols);
}

// ---------------------------------------------------------------------------
// Halo convolution: persistent, warp-specialised, for images at least 96 pixels wide.
//
// A tile is R output rows x 128 pixels x n_tile output channels: R accumulators of
// n_tile TMEM columns, double-buffered so the epilogue of one tile overlaps the MMAs of
// the next. Per chunk of CK input channels one 4D TMA box brings the tile's input halo,
// (R + 2) rows x 130 pixels, into shared memory as [row][pixel][CK channels]: one swizzled
// K-major row of CK x 2 bytes (32- or 64-byte swizzle) per pixel, so TMA moves 32- or
// 64-byte pieces of the NHWC input (16-byte pieces deliver half the bytes per second).
// The A operand of tap (dy, dx) for output row r is that buffer viewed from row r + dy,
// pixel dx on: the descriptor's start address moves by whole rows. The tensor cores apply
// the swizzle to the absolute shared-memory address, as TMA does when it writes a box at
// a 1024-byte aligned address, so a view starting at any row reads the rows TMA wrote
// (the descriptor's base-offset field stays 0). The halo is read from L2 once per chunk
// and used by all 9 taps (the per-tap kernel above reads 9 shifted boxes). The weights of a
// chunk (9 blocks of n_tile rows of CK channels, swizzled, ordered [dx][dy = 2, 1, 0] so
// that one MMA covers up to STACK output rows: halo_chunk_mmas) stream with the halo by TMA,
// or, when one chunk covers all input channels, are loaded once per CTA.
//
// The epilogue writes 16 channels of a pixel with one 32-byte store and can also do the
// 2x2 average pooling that follows some layers (rows are paired inside a tile, the right
// neighbour is the next lane), saving the pass that would read the layer's output again.
//
// Warp 0 lane 0: TMA producer (a ring of STAGES stages). Warp 1: MMA issuer.
// Warps 2-9: epilogue, warp w owning TMEM lanes [32 (w % 4), +32) = tile pixels, warps 2-5
// the first half of the channels and warps 6-9 the second.
// Every wait is bounded; on expiry the kernel records an error code, lets its own
// copies and MMAs finish and frees its TMEM.
// ---------------------------------------------------------------------------
constexpr int kHaloW = 130;     // 128 output pixels + 2 halo pixels
// Halo stages in flight (STAGES): 3, or 2 where a third does not fit 227 KB (8-row
// tiles, or 32-channel chunks with streamed weights).
constexpr int kHaloThreads = 320;  // producer warp, MMA warp, 8 epilogue warps

// ---- epilogue pieces of the two persistent kernels: a lane holds 16 output channels of a pixel ----
// The epilogue warps run a few instructions deep in each other's results, so its length is what
// the narrow layers (16 and 32 input channels) wait for: bias in registers for all rows of a
// channel group, two groups of accumulators per TMEM wait, and pooling neighbours exchanged as
// packed BF16 pairs. Measured before and after: the 1920 x 1088 network 928 -> 842 us (its
// 32 -> 32 layer 56 -> 49), 16 x 64 x 64 pixels 64 -> 64 channels 15.8 -> 10.8 us, 64 -> 160
// 29.7 -> 15.3. The arrays stay in registers only while no call takes their address.
struct Bias16 {
    float v[16];
    __device__ __forceinline__ void load(const float* s) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 b = *reinterpret_cast<const float4*>(s + 4 * q);
            v[4 * q] = b.x; v[4 * q + 1] = b.y; v[4 * q + 2] = b.z; v[4 * q + 3] = b.w;
        }
    }
};
__device__ __forceinline__ void activate(const uint32_t (&raw)[16], const Bias16& b, int relu, float (&v)[16]) {
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(raw[q]) + b.v[q];
    if (relu) {
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = fmaxf(v[q], 0.0f);
    }
}
__device__ __forceinline__ void pack16(const float (&v)[16], uint32_t (&w)[8]) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
        w[q] = *reinterpret_cast<const uint32_t*>(&h);
    }
}
// 16 BF16 channels with one 32-byte store (dst 32-byte aligned)
__device__ __forceinline__ void store16(__nv_bfloat16* dst, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}
// a pixel of the network's head, with the residual added
__device__ __forceinline__ void store_head(float* dst, const float* base, const float (&v)[16]) {
    float4 o = make_float4(v[0], v[1], v[2], 0.0f);
    if (base) {
        const float4 b = *reinterpret_cast<const float4*>(base);
        o.x += b.x;
        o.y += b.y;
        o.z += b.z;
    }
    *reinterpret_cast<float4*>(dst) = o;
}
// the four copies of a pixel in an upsampled image
__device__ __forceinline__ void store16_up(__nv_bfloat16* dst, int px_step, size_t row_step, const uint32_t (&w)[8]) {
    store16(dst, w);
    store16(dst + px_step, w);
    store16(dst + row_step, w);
    store16(dst + row_step + px_step, w);
}
// the first n of 16 channels, at any alignment (16-byte stores where they fit)
__device__ __forceinline__ void store16_any(__nv_bfloat16* dst, const uint32_t (&w)[8], int n) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int m = n - 8 * h;
        if (m >= 8 && ((uintptr_t)(dst + 8 * h) & 15) == 0) {
            *reinterpret_cast<uint4*>(dst + 8 * h) = make_uint4(w[4 * h], w[4 * h + 1], w[4 * h + 2], w[4 * h + 3]);
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q < m) reinterpret_cast<uint16_t*>(dst)[8 * h + q] = (uint16_t)(w[4 * h + q / 2] >> (16 * (q & 1)));
        }
    }
}
// A ReLU's backward mask on the packed channels of one pixel: zero where the forward output is
// not positive. m: 16 channels, 16-byte aligned.
__device__ __forceinline__ void mask16(const __nv_bfloat16* m, uint32_t (&w)[8]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(m) + h);
        const uint32_t y[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float lo = __uint_as_float(y[k] << 16), hi = __uint_as_float(y[k] & 0xFFFF0000u);
            w[4 * h + k] &= (lo > 0.0f ? 0x0000FFFFu : 0u) | (hi > 0.0f ? 0xFFFF0000u : 0u);
        }
    }
}
// ((a + b) + c) + d in FP32, quartered, of packed BF16 pairs: the order the pooled values are defined by
__device__ __forceinline__ uint32_t pool_pair(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const float lo = 0.25f * (((__uint_as_float(a << 16) + __uint_as_float(b << 16)) + __uint_as_float(c << 16)) +
                              __uint_as_float(d << 16));
    const float hi = 0.25f * (((__uint_as_float(a & 0xFFFF0000u) + __uint_as_float(b & 0xFFFF0000u)) +
                               __uint_as_float(c & 0xFFFF0000u)) +
                              __uint_as_float(d & 0xFFFF0000u));
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

struct HaloParams {
    int N, H, W, Cin, Cout;
    int n_tile, R, kchunks;
    int tiles_x, tiles_y, num_tiles;
    int w_resident;          // 1: the weights of all input channels are one chunk, loaded once
    int stack;               // output rows one MMA covers (1..3, stack x n_tile <= 256)
    uint32_t halo_bytes;     // bytes of one halo box
    uint32_t halo_stride;    // its slot in shared memory (1024-aligned)
    uint32_t w_bytes;        // bytes of one chunk of weights (9 x n_tile x CK)
    uint32_t w_stride;
    uint32_t tmem_cols;
    const float* bias;
    int relu;
    __nv_bfloat16* out;
    int out_cstride, out_coff;
    float* outf;
    __nv_bfloat16* pool_out;   // fused 2x2 average pooling into a dense [N][H/2][W/2][Cout] tensor, or null
    union {                    // what the epilogue does besides (one at most; null: nothing)
        const __nv_bfloat16* mask; // ReLU backward mask: channel stride aux_cs, slice at aux_co
        __nv_bfloat16* up_out;     // EXTRA, BF16: 2x upsampling into a slice of [N][2H][2W][aux_cs]; out may be null
        const float* base;         // EXTRA, FP32: the residual of a head of 3 channels in float4 pixels
    };
    int aux_cs, aux_co;
    int settled;               // weights and bias may be read before the kernel before this one ends
};

// Constants of the MMA sequence that depend on n_tile: weight block offsets (in
// descriptor units of 16 bytes), instruction descriptors for 1..3 stacked rows, and the
// TMEM column of each output row.
struct HaloMmaConsts {
    uint32_t boff[9];
    uint32_t idesc[3];
    uint32_t dcol[8];
};

// The MMAs of one chunk, unrolled at compile time (the single issuing warp then spends a
// few instructions per MMA; built from a table at run time they took half again as long).
// Halo row hr with shift dx feeds output rows hr - 2 .. hr (tap dy = hr - r); their
// accumulators are adjacent TMEM columns and their weight blocks ([dx][dy = 2, 1, 0])
// adjacent rows, so one MMA of N = rows x n_tile covers up to STACK of them and the A
// operand is read once per (hr, dx, kk) instead of once per output row. The loop runs
// over halo rows outermost, so consecutive MMAs accumulate into the same columns. In a
// tile's first chunk the row a halo row reaches first (r = hr, at dx = 0, kk = 0) starts
// its accumulator with a non-accumulating MMA of its own.
template <int CK, int R, int STACK, bool FIRST>
__device__ __forceinline__ void halo_chunk_mmas(uint64_t ad0, uint64_t bd0, uint32_t acc, const HaloMmaConsts& k,
                                                uint32_t elected) {
    constexpr uint32_t W_ROW = CK * 2, HALO_ROW = kHaloW * W_ROW;
#pragma unroll
    for (int hr = 0; hr < R + 2; ++hr) {
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
#pragma unroll
            for (int kk = 0; kk < CK / 16; ++kk) {
                const uint64_t ad = ad0 + (((uint32_t)hr * HALO_ROW + (uint32_t)dx * W_ROW + kk * 32) >> 4);
                const int lo = hr - 2 > 0 ? hr - 2 : 0;
                int hi = hr < R - 1 ? hr : R - 1;
                if (FIRST && dx == 0 && kk == 0 && hi == hr) {
                    tc::mma_bf16(acc + k.dcol[hr], ad, bd0 + k.boff[dx * 3 + 2] + kk * 2, k.idesc[0], 0u, elected);
                    --hi;
                }
#pragma unroll
                for (int r0 = lo; r0 <= hi; r0 += STACK) {
                    const int r1 = r0 + STACK - 1 < hi ? r0 + STACK - 1 : hi;
                    tc::mma_bf16(acc + k.dcol[r0], ad, bd0 + k.boff[dx * 3 + 2 - (hr - r0)] + kk * 2,
                                 k.idesc[r1 - r0], 1u, elected);
                }
            }
        }
    }
}

template <int CK, int R, int STACK, int STAGES, bool EXTRA>
__global__ void __launch_bounds__(kHaloThreads, 1) k_conv_halo(const __grid_constant__ CUtensorMap tmX,
                                                                 const __grid_constant__ CUtensorMap tmW,
                                                                 const HaloParams p) {
    constexpr uint32_t W_ROW = CK * 2;                 // bytes per pixel row and weight row (the swizzle width)
    constexpr uint32_t W_LAYOUT = CK == 32 ? 4u : 6u;  // 64 B / 32 B swizzle
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* halo = smem;
    uint8_t* wst = halo + STAGES * p.halo_stride;
    const int w_slots = p.w_resident ? 1 : STAGES;
    uint64_t* full = reinterpret_cast<uint64_t*>(wst + w_slots * p.w_stride);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* wbar = acc_empty + 2;
    uint64_t* mma_done = wbar + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
    float* sbias = reinterpret_cast<float*>(tmem_slot + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.y * p.n_tile;
    const int acc_cols = p.R * p.n_tile;

    if (threadIdx.x == 32) {
        tc::prefetch_map(&tmX);
        tc::prefetch_map(&tmW);
    }
    if (!p.settled) grid_wait();
    if (warp == 0) tc::tmem_alloc(tmem_slot, p.tmem_cols);
    for (int i = threadIdx.x; i < p.n_tile; i += blockDim.x)
        sbias[i] = (p.bias && n0 + i < p.Cout) ? p.bias[n0 + i] : 0.0f;
    if (threadIdx.x == 32) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&acc_full[b], 1);
            tc::mbar_init(&acc_empty[b], 8);
        }
        tc::mbar_init(wbar, 1);
        tc::mbar_init(mma_done, 1);
        tc::fence_barrier_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    if (!p.settled) grid_launch_dependents();

    auto tile_origin = [&](int t, int& n_img, int& y0, int& x0) {
        const int per_img = p.tiles_x * p.tiles_y;
        n_img = t / per_img;
        const int r = t % per_img;
        y0 = (r / p.tiles_x) * p.R;
        x0 = (r % p.tiles_x) * 128;
    };

    if (warp == 0 && lane == 0) {
        // ---- producer ----
        bool ok = true;
        // the weights of a chunk in shared memory as 9 blocks of n_tile rows in the order
        // [dx][dy = 2, 1, 0]: the blocks of the taps one halo row and shift give the
        // output rows r, r + 1, r + 2 (dy = j - r) are adjacent, one stacked B operand
        auto load_weights = [&](uint8_t* dst, uint64_t* bar, int c) {
#pragma unroll 1
            for (int tap = 0; tap < 9; ++tap) {
                const int blk = (tap % 3) * 3 + (2 - tap / 3);
                tc::tma_load_3d(dst + (uint32_t)blk * p.n_tile * W_ROW, &tmW, bar, c * CK, n0, tap);
            }
        };
        if (p.w_resident) {
            tc::mbar_arrive_expect_tx(wbar, p.w_bytes);
            load_weights(wst, wbar, 0);
        }
        if (p.settled) grid_dependency_wait();
        uint32_t it = 0;
        for (int t = blockIdx.x; t < p.num_tiles && ok; t += gridDim.x) {
            int n_img, y0, x0;
            tile_origin(t, n_img, y0, x0);
            for (int c = 0; c < p.kchunks; ++c, ++it) {
                const uint32_t s = it % STAGES;
                if (it >= (uint32_t)STAGES &&
                    !tc::mbar_wait(&empty[s], ((it / STAGES) - 1) & 1, kWaitBudget)) {
                    set_error(11);
                    ok = false;
                    break;
                }
                tc::mbar_arrive_expect_tx(&full[s], p.halo_bytes + (p.w_resident ? 0u : p.w_bytes));
                tc::tma_load_4d(halo + s * p.halo_stride, &tmX, &full[s], c * CK, x0 - 1, y0 - 1, n_img);
                if (!p.w_resident) load_weights(wst + s * p.w_stride, &full[s], c);
            }
        }
        // drain: every issued copy must have landed before the CTA may exit
        for (uint32_t s = 0; s < (uint32_t)STAGES && s < it; ++s) {
            const uint32_t last = ((it - 1 - s) / STAGES) * STAGES + s;
            if (!tc::mbar_wait(&full[s], (last / STAGES) & 1, kWaitBudget)) set_error(12);
        }
        if (p.w_resident && !tc::mbar_wait(wbar, 0, kWaitBudget)) set_error(13);
    } else if (warp == 1) {
        // ---- MMA issuer: the warp stays converged, one elected lane issues ----
        const uint32_t elected = tc::elect_one();
        const uint32_t halo0 = tc::smem_u32(halo), w0 = tc::smem_u32(wst);
        // per-CTA constants of the unrolled MMA sequence (halo_chunk_mmas)
        HaloMmaConsts k;
#pragma unroll
        for (int b = 0; b < 9; ++b) k.boff[b] = (uint32_t)(b * p.n_tile) * W_ROW >> 4;
#pragma unroll
        for (int q = 0; q < 3; ++q) k.idesc[q] = tc::idesc_bf16(128, (uint32_t)((q + 1) * p.n_tile));
#pragma unroll
        for (int r = 0; r < R; ++r) k.dcol[r] = (uint32_t)(r * p.n_tile);
        bool ok = !p.w_resident || tc::mbar_wait_warp(wbar, 0, kWaitBudget);
        if (!ok) set_error(14);
        uint32_t it = 0, j = 0;
        for (int t = blockIdx.x; t < p.num_tiles && ok; t += gridDim.x, ++j) {
            const uint32_t b = j & 1;
            if (j >= 2 && !tc::mbar_wait_warp(&acc_empty[b], ((j / 2) - 1) & 1, kWaitBudget)) {
                set_error(15);
                break;
            }
            tc::fence_after_sync();
            const uint32_t acc = tmem + b * (uint32_t)acc_cols;
            for (int c = 0; c < p.kchunks; ++c, ++it) {
                const uint32_t s = it % STAGES;
                if (!tc::mbar_wait_warp(&full[s], (it / STAGES) & 1, kWaitBudget)) {
                    set_error(16);
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                const uint32_t ha = halo0 + s * p.halo_stride;
                const uint32_t wa = w0 + (p.w_resident ? 0u : s * p.w_stride);
                const uint64_t ad0 = tc::smem_desc(ha, 8u * W_ROW, W_LAYOUT);
                const uint64_t bd0 = tc::smem_desc(wa, 8u * W_ROW, W_LAYOUT);
                if (c == 0)
                    halo_chunk_mmas<CK, R, STACK, true>(ad0, bd0, acc, k, elected);
                else
                    halo_chunk_mmas<CK, R, STACK, false>(ad0, bd0, acc, k, elected);
                if (elected) tc::mma_commit(&empty[s]);
            }
            if (!ok) break;
            if (elected) tc::mma_commit(&acc_full[b]);
        }
        // every MMA of this CTA completes before the TMEM is freed
        if (elected) tc::mma_commit(mma_done);
        if (!tc::mbar_wait_warp(mma_done, 0, kWaitBudget)) set_error(17);
    } else if (warp >= 2) {
        // ---- epilogue: 8 warps, two per TMEM lane group, each taking half of the channel groups ----
        const int lg = warp & 3;                 // TMEM lane group of this warp
        const int px_in_tile = lg * 32 + lane;
        const int ng = p.n_tile >> 4;            // groups of 16 channels
        const int g0 = warp < 6 ? 0 : (ng + 1) / 2, g1 = warp < 6 ? (ng + 1) / 2 : ng;
        // whole 32-byte stores: the tensor, the channel stride and the slice are aligned to them
        const bool fast = !p.outf && p.out && ((uintptr_t)p.out & 31) == 0 && (p.out_cstride & 15) == 0 &&
                          ((p.out_coff + n0) & 15) == 0 && n0 + p.n_tile <= p.Cout;
        const bool pool_fast = p.pool_out && ((uintptr_t)p.pool_out & 31) == 0 && (p.Cout & 15) == 0;
        const uint32_t lanes = (uint32_t)(lg * 32) << 16;
        if (p.settled) grid_dependency_wait();
        uint32_t j = 0;
        for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x, ++j) {
            const uint32_t b = j & 1;
            // the residual's rows, while the tile is still multiplied (the network 796 -> 777 us)
            if (EXTRA && p.outf && p.base && g0 == 0) {
                int n_img, y0, x0;
                tile_origin(t, n_img, y0, x0);
                const int px = x0 + px_in_tile;
                if (px < p.W)
                    for (int r = 0; r < min(R, p.H - y0); ++r)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(
                            p.base + (((size_t)n_img * p.H + y0 + r) * p.W + px) * 4));
            }
            const bool ready = tc::mbar_wait_warp(&acc_full[b], (j / 2) & 1, kWaitBudget);
            __syncwarp();
            if (!ready) {
                set_error(18);
                break;
            }
            tc::fence_after_sync();
            int n_img, y0, x0;
            tile_origin(t, n_img, y0, x0);
            const int px = x0 + px_in_tile;
            const int rows = px < p.W ? min(R, p.H - y0) : 0; // this pixel column's rows inside the image
            const size_t pix = ((size_t)n_img * p.H + y0) * p.W + px;
            const size_t row_step = (size_t)p.W * p.out_cstride;
            // one row's 16 channels of this pixel
            auto emit = [&](int r, int g, const float(&v)[16], uint32_t(&w)[8]) {
                const int co = n0 + 16 * g;
                if (r >= rows || co >= p.Cout) return;
                const size_t at = pix * p.out_cstride + p.out_coff + co + r * row_step;
                if (EXTRA && p.outf) {
                    if (co == 0) store_head(p.outf + at, p.base ? p.base + at : nullptr, v);
                    return;
                }
                if (p.outf) { // FP32 output (a network head)
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        if (co + q < p.Cout) p.outf[at + q] = v[q];
                    return;
                }
                if (!EXTRA && p.mask) mask16(p.mask + (pix + (size_t)r * p.W) * p.aux_cs + p.aux_co + co, w);
                if (EXTRA) {
                    store16_up(p.up_out + (((size_t)n_img * p.H + y0 + r) * 4 * p.W + 2 * px) * p.aux_cs + p.aux_co + co,
                               p.aux_cs, (size_t)(2 * p.W) * p.aux_cs, w);
                    if (!p.out) return;
                }
                if (fast) store16(p.out + at, w);
                else store16_any(p.out + at, w, p.Cout - co);
            };
            for (int g = g0; g < g1; ++g) {
                Bias16 bias;
                bias.load(sbias + 16 * g);
                const uint32_t col0 = tmem + lanes + b * (uint32_t)acc_cols + 16u * (uint32_t)g;
#pragma unroll 1
                for (int r = 0; r < R; r += 2) { // two rows per TMEM wait (R = 1: one)
                    uint32_t r0[16], r1[16], w0[8], w1[8];
                    float v0[16], v1[16];
                    tc::tmem_ld16(col0 + (uint32_t)(r * p.n_tile), r0);
                    if (R > 1) tc::tmem_ld16(col0 + (uint32_t)((r + 1) * p.n_tile), r1);
                    tc::tmem_ld_wait();
                    activate(r0, bias, p.relu, v0);
                    pack16(v0, w0);
                    if (R > 1) {
                        activate(r1, bias, p.relu, v1);
                        pack16(v1, w1);
                        if (p.pool_out) {
                            // R and y0 are even: the 2x2 average of the BF16 outputs over (2y, 2x),
                            // (2y, 2x+1), (2y+1, 2x), (2y+1, 2x+1); the right neighbour is the next lane
                            uint32_t pw[8];
#pragma unroll
                            for (int q = 0; q < 8; ++q)
                                pw[q] = pool_pair(w0[q], __shfl_xor_sync(0xFFFFFFFFu, w0[q], 1), w1[q],
                                                  __shfl_xor_sync(0xFFFFFFFFu, w1[q], 1));
                            const int co = n0 + 16 * g;
                            if (!(lane & 1) && px + 1 < p.W && r + 1 < rows && co < p.Cout) {
                                __nv_bfloat16* dst = p.pool_out +
                                    (((size_t)n_img * (p.H / 2) + (y0 + r) / 2) * (p.W / 2) + px / 2) * p.Cout + co;
                                if (pool_fast) store16(dst, pw);
                                else store16_any(dst, pw, p.Cout - co);
                            }
                        }
                    }
                    emit(r, g, v0, w0);
                    if (R > 1) emit(r + 1, g, v1, w1);
                }
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&acc_empty[b]);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, p.tmem_cols);
}

// ---------------------------------------------------------------------------
// Tile convolution, for images that are narrow for the halo kernel above (training crops, the
// deep levels of small frames): persistent, with all weights of its output channels resident.
//
// A tile is 8 x 16 output pixels x n_tile channels. Per 32 input channels one TMA box brings the
// tile's halo (10 x 18 pixels) into shared memory as K-major rows of 64 bytes; the 128 rows of
// the A operand are 16 groups of 8 pixels, one per image row, so their stride is the halo's row
// (10 pixels) and a tap's view starts (dy * 10 + dx) rows further. The weights of the CTA's n_tile
// output channels (9 taps x all input channels) are loaded once; the halo of the next tile loads
// (two buffers where they fit) while this one multiplies, and the epilogue of the tile before
// drains the other accumulator. Sums run over taps, then channels: the order of the per-tap kernel
// k_tc, and so its bits.
//
// Bound: the tensor core's operand fetch (128 x 16 of A feed n_tile columns), and for a few tiles
// the latency of one load, one multiplication and one epilogue. k_tc loads 9 shifted boxes per 32
// channels through a ring of 2 or 3 stages, a round trip to L2 every few steps. 16 images, before
// and after: 160 -> 160 channels at 8 x 8 26 -> 12 us, 288 -> 128 at 16 x 16 36 -> 19, 96 -> 96 at
// 32 x 32 17 -> 10, 64 -> 160 at 64 x 64 38 -> 15, 160 -> 64 there 28 -> 23 (32 output channels per
// CTA are all that fit beside its halos, and an MMA costs 40 to 48 cycles of operand fetch with
// 32 columns as with 64); a 256 x 256 frame's whole network 391 -> 190 us (with the weights loaded
// while the kernel before drains).
//
// Warp 0 lane 0: TMA, warp 1: MMAs, warps 2-9: epilogue, two to a TMEM lane group (4 tile
// rows), each taking half of the channel groups. Every wait is bounded as in the kernels above.
// ---------------------------------------------------------------------------
constexpr int kTileThreads = 320;
constexpr int kTileW = 8, kTileH = 16, kTileHaloW = kTileW + 2, kTileHaloH = kTileH + 2;
constexpr uint32_t kTileHaloBytes = kTileHaloW * kTileHaloH * 64; // 32 channels
constexpr uint32_t kTileHaloSlot = (kTileHaloBytes + 1023u) & ~1023u;

struct TileParams {
    int H, W, Cout;
    int n_tile, bufs;
    int tiles_x, tiles_y, num_tiles;
    uint32_t tmem_cols;
    const float* bias;
    int relu;
    __nv_bfloat16* out;
    int out_cstride, out_coff;
    float* outf;
    __nv_bfloat16* pool_out; // fused 2x2 average pooling into a dense [N][H/2][W/2][Cout] tensor, or null
    union {                    // what the epilogue does besides (one at most; null: nothing)
        const __nv_bfloat16* mask; // ReLU backward mask: channel stride aux_cs, slice at aux_co
        __nv_bfloat16* up_out;     // EXTRA, BF16: 2x upsampling into a slice of [N][2H][2W][aux_cs]; out may be null
        const float* base;         // EXTRA, FP32: the residual of a head of 3 channels in float4 pixels
    };
    int aux_cs, aux_co;
    int settled; // weights and bias may be read before the kernel before this one ends
};

// The MMAs of a tile over KC chunks of 32 input channels, unrolled at compile time: the one
// issuing thread then spends a few instructions on each (in a loop over run-time chunks the
// 160 -> 64 layer of 16 x 64 x 64 pixels took 34.9 us, bound by their issue; now 23).
template <int KC>
__device__ __forceinline__ void tile_mmas(uint32_t acc, uint64_t ad0, uint64_t bd0, uint32_t tap_units, uint32_t idesc,
                                          uint32_t elected) {
#pragma unroll 1
    for (int dy = 0; dy < 3; ++dy) { // a filter row at a time: all 9 taps at once spill from 160 channels on
        const uint64_t ar = ad0 + (uint32_t)(dy * kTileHaloW * 4), br = bd0 + (uint32_t)dy * 3u * tap_units;
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
#pragma unroll
            for (int c = 0; c < KC; ++c) {
                const uint64_t ad = ar + (uint32_t)(dx * 4 + c * (kTileHaloSlot >> 4));
                const uint64_t bd = br + (uint32_t)(c * 9 + dx) * tap_units;
                tc::mma_bf16(acc, ad, bd, idesc, (dy > 0 || dx > 0 || c > 0) ? 1u : 0u, elected);
                tc::mma_bf16(acc, ad + 2, bd + 2, idesc, 1u, elected);
            }
        }
    }
}

template <int KC, bool EXTRA>
__global__ void __launch_bounds__(kTileThreads) k_conv_tile(const __grid_constant__ CUtensorMap tmX,
                                                               const __grid_constant__ CUtensorMap tmW,
                                                               const TileParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t tap_bytes = (uint32_t)p.n_tile * 64u;           // one tap, 32 channels
    const uint32_t buf_bytes = (uint32_t)KC * kTileHaloSlot;
    uint8_t* wst = smem + (uint32_t)p.bufs * buf_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(wst + (uint32_t)KC * 9u * tap_bytes);
    uint64_t* empty = full + 2;
    uint64_t* acc_full = empty + 2;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* wbar = acc_empty + 2;
    uint64_t* mma_done = wbar + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
    float* sbias = reinterpret_cast<float*>(tmem_slot + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.y * p.n_tile;

    if (threadIdx.x == 32) {
        tc::prefetch_map(&tmX);
        tc::prefetch_map(&tmW);
    }
    if (!p.settled) grid_wait();
    if (warp == 0) tc::tmem_alloc(tmem_slot, p.tmem_cols);
    for (int i = threadIdx.x; i < p.n_tile; i += blockDim.x)
        sbias[i] = (p.bias && n0 + i < p.Cout) ? p.bias[n0 + i] : 0.0f;
    if (threadIdx.x == 32) {
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&full[b], 1);
            tc::mbar_init(&empty[b], 1);
            tc::mbar_init(&acc_full[b], 1);
            tc::mbar_init(&acc_empty[b], 8);
        }
        tc::mbar_init(wbar, 1);
        tc::mbar_init(mma_done, 1);
        tc::fence_barrier_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    if (!p.settled) grid_launch_dependents();

    auto tile_origin = [&](int t, int& n_img, int& y0, int& x0) {
        const int per_img = p.tiles_x * p.tiles_y;
        n_img = t / per_img;
        const int r = t % per_img;
        y0 = (r / p.tiles_x) * kTileH;
        x0 = (r % p.tiles_x) * kTileW;
    };

    if (warp == 0 && lane == 0) {
        // ---- producer: the weights first, while the kernel before this one may still run ----
        const bool any = (int)blockIdx.x < p.num_tiles;
        if (any) {
            tc::mbar_arrive_expect_tx(wbar, (uint32_t)KC * 9u * tap_bytes);
            for (int c = 0; c < KC; ++c)
                tc::tma_load_3d(wst + (uint32_t)c * 9u * tap_bytes, &tmW, wbar, c * 32, n0, 0);
        }
        if (p.settled) grid_dependency_wait();
        uint32_t it = 0;
        for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x, ++it) {
            const uint32_t b = p.bufs == 2 ? (it & 1) : 0, use = p.bufs == 2 ? it >> 1 : it;
            if (use > 0 && !tc::mbar_wait(&empty[b], (use - 1) & 1, kWaitBudget)) {
                set_error(31);
                break;
            }
            int n_img, y0, x0;
            tile_origin(t, n_img, y0, x0);
            tc::mbar_arrive_expect_tx(&full[b], (uint32_t)KC * kTileHaloBytes);
            for (int c = 0; c < KC; ++c)
                tc::tma_load_4d(smem + b * buf_bytes + c * kTileHaloSlot, &tmX, &full[b], c * 32, x0 - 1, y0 - 1, n_img);
        }
        // drain: every issued copy must have landed before the CTA may exit
        for (uint32_t b = 0; b < (uint32_t)p.bufs && b < it; ++b) {
            const uint32_t uses = p.bufs == 2 ? (it - b + 1) / 2 : it;
            if (!tc::mbar_wait(&full[b], (uses - 1) & 1, kWaitBudget)) set_error(32);
        }
        if (any && !tc::mbar_wait(wbar, 0, kWaitBudget)) set_error(33);
    } else if (warp == 1) {
        // ---- MMA issuer: the warp stays converged, one elected lane issues ----
        const uint32_t elected = tc::elect_one();
        const uint32_t idesc = tc::idesc_bf16(128, (uint32_t)p.n_tile);
        const uint32_t halo0 = tc::smem_u32(smem);
        const uint64_t bd0 = tc::smem_desc(tc::smem_u32(wst), 512u, 4u);
        bool ok = (int)blockIdx.x >= p.num_tiles || tc::mbar_wait_warp(wbar, 0, kWaitBudget);
        if (!ok) set_error(34);
        uint32_t it = 0;
        for (int t = blockIdx.x; t < p.num_tiles && ok; t += gridDim.x, ++it) {
            const uint32_t b = p.bufs == 2 ? (it & 1) : 0, use = p.bufs == 2 ? it >> 1 : it, a = it & 1;
            if (it >= 2 && !tc::mbar_wait_warp(&acc_empty[a], ((it / 2) - 1) & 1, kWaitBudget)) {
                set_error(35);
                break;
            }
            if (!tc::mbar_wait_warp(&full[b], use & 1, kWaitBudget)) {
                set_error(36);
                break;
            }
            tc::fence_after_sync();
            const uint32_t acc = tmem + a * (uint32_t)p.n_tile;
            const uint64_t ad0 = tc::smem_desc(halo0 + b * buf_bytes, kTileHaloW * 64u, 4u);
            tile_mmas<KC>(acc, ad0, bd0, tap_bytes >> 4, idesc, elected);
            if (elected) {
                tc::mma_commit(&empty[b]);
                tc::mma_commit(&acc_full[a]);
            }
        }
        // every MMA of this CTA completes before the TMEM is freed
        if (elected) tc::mma_commit(mma_done);
        if (!tc::mbar_wait_warp(mma_done, 0, kWaitBudget)) set_error(37);
    } else if (warp >= 2) {
        // ---- epilogue: lane = pixel (4 rows of 8 per lane group) ----
        const int lg = warp & 3, m = lg * 32 + lane;
        const int ng = p.n_tile >> 4;
        const int g0 = warp < 6 ? 0 : (ng + 1) / 2, g1 = warp < 6 ? (ng + 1) / 2 : ng;
        const bool fast = !p.outf && ((uintptr_t)p.out & 31) == 0 && (p.out_cstride & 15) == 0 &&
                          ((p.out_coff + n0) & 15) == 0 && n0 + p.n_tile <= p.Cout;
        const bool pool_fast = p.pool_out && ((uintptr_t)p.pool_out & 31) == 0 && (p.Cout & 15) == 0;
        if (p.settled) grid_dependency_wait();
        uint32_t it = 0;
        for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x, ++it) {
            const uint32_t a = it & 1;
            const bool ready = tc::mbar_wait_warp(&acc_full[a], (it / 2) & 1, kWaitBudget);
            __syncwarp();
            if (!ready) {
                set_error(38);
                break;
            }
            tc::fence_after_sync();
            int n_img, y0, x0;
            tile_origin(t, n_img, y0, x0);
            const int px = x0 + (m & 7), py = y0 + (m >> 3);
            const bool valid = px < p.W && py < p.H;
            const size_t pix = ((size_t)n_img * p.H + py) * p.W + px;
            const uint32_t col0 = tmem + ((uint32_t)(lg * 32) << 16) + a * (uint32_t)p.n_tile;
            auto finish = [&](int g, const uint32_t(&raw)[16]) {
                Bias16 bias;
                bias.load(sbias + 16 * g);
                float v[16];
                uint32_t w[8];
                activate(raw, bias, p.relu, v);
                pack16(v, w);
                const int co = n0 + 16 * g;
                if (p.pool_out) {
                    // the 2x2 average of the BF16 outputs: the neighbours are lanes 1, 8 and 9 further
                    uint32_t pw[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        pw[q] = pool_pair(w[q], __shfl_xor_sync(0xFFFFFFFFu, w[q], 1),
                                          __shfl_xor_sync(0xFFFFFFFFu, w[q], 8), __shfl_xor_sync(0xFFFFFFFFu, w[q], 9));
                    if (valid && !(lane & 9) && co < p.Cout) {
                        __nv_bfloat16* dst =
                            p.pool_out + (((size_t)n_img * (p.H / 2) + py / 2) * (p.W / 2) + px / 2) * p.Cout + co;
                        if (pool_fast) store16(dst, pw);
                        else store16_any(dst, pw, p.Cout - co);
                    }
                }
                if (!valid || co >= p.Cout) return;
                const size_t at = pix * p.out_cstride + p.out_coff + co;
                if (EXTRA && p.outf) {
                    if (co == 0) store_head(p.outf + at, p.base ? p.base + at : nullptr, v);
                    return;
                }
                if (p.outf) { // FP32 output (a network head)
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        if (co + q < p.Cout) p.outf[at + q] = v[q];
                    return;
                }
                if (!EXTRA && p.mask) mask16(p.mask + pix * p.aux_cs + p.aux_co + co, w);
                if (EXTRA) {
                    store16_up(p.up_out + (((size_t)n_img * p.H + py) * 4 * p.W + 2 * px) * p.aux_cs + p.aux_co + co,
                               p.aux_cs, (size_t)(2 * p.W) * p.aux_cs, w);
                    if (!p.out) return;
                }
                if (fast) store16(p.out + at, w);
                else store16_any(p.out + at, w, p.Cout - co);
            };
#pragma unroll 1
            for (int g = g0; g < g1; g += 2) { // two groups per TMEM wait
                uint32_t r0[16], r1[16];
                tc::tmem_ld16(col0 + 16u * (uint32_t)g, r0);
                if (g + 1 < g1) tc::tmem_ld16(col0 + 16u * (uint32_t)(g + 1), r1);
                tc::tmem_ld_wait();
                finish(g, r0);
                if (g + 1 < g1) finish(g + 1, r1);
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&acc_empty[a]);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, p.tmem_cols);
}

// ---------------------------------------------------------------------------
// Weight gradients of a 3x3 convolution: dW[dy][dx][co][ci] += sum over pixels p of
// dZ[p][co] * X[p + (dy - 1, dx - 1)][ci], as one tcgen05 contraction over pixels.
//
// Both operands are read as the NHWC tensors store them (MN-major: channels contiguous, one
// pixel = one K row), so nothing is transposed in memory. A tile is kWgRows x bw pixels of X
// with one halo column on each side, and the (kWgRows + 2) x bw pixels of dZ around it, both
// by one TMA box (zero fill outside the image = zero padding). All 9 taps of 16 pixels are one
// MMA: the operands' 32-channel groups lie a leading offset apart in shared memory, and that
// offset is one pixel for A (M = 128: X shifted by dx = 0, 1, 2 and a fourth, unused shift) and
// one image row for B (N = 3 x co_block: dZ rows y - 1, y, y + 1, that is dy = 2, 1, 0). The
// shifted views start at any pixel: swizzling works on absolute shared-memory addresses.
//
// A CTA owns 32 input channels and one block of output channels, walks its share of the tiles and
// adds its FP32 sums to dW by atomics (lane = input channel, so a warp's add is one 128-byte
// line). It keeps to 110 KB of shared memory where two stages fit them, so that a convolution of
// the backward-data chain fits beside it. (Up to 5 blocks of input channels per CTA share dZ tiles,
// but leave fewer, larger CTAs: 904 against 892 us a step by itself, 877 against 838 beside the chain.)
//
// Bound: the TMA's rate of 64-byte rows at full resolution (with a quarter of the MMAs, no bias
// sums and no atomics the 96 -> 32 layer still takes 28 of 33 us), launch and first-tile latency at
// the deep levels. On a batch of 16 crops of 128 x 128 the 19 layers of the denoiser's backward
// pass take 0.29 ms in this form (8 to 33 us each); as 9 shifted transposes and 9 GEMMs a layer,
// each reading its operands from HBM again, they took 12.8 ms.
//
// One CTA of 192 threads: warp 0 lane 0 issues TMA, warp 1 the MMAs, warps 2 to 5 sum the bias
// gradient from the dZ tiles in shared memory (a pass over dZ of its own before), warps 0-2 (one
// per dx) drain TMEM. A stage is free when it is summed: with 2 warps the sums held the loads up
// (0.32 ms, a step 762 us; with 4 735, 6 739, 8 752, which leave less room for the other chain).
// Every wait is bounded as in the kernels above.
// ---------------------------------------------------------------------------
constexpr int kWgRows = 8;     // X rows of a tile
constexpr int kWgMaxStages = 4;
constexpr int kWgSumWarps = 4; // warps that sum the bias gradient
constexpr int kWgThreads = 64 + 32 * kWgSumWarps;

struct WgradParams {
    int tiles_x, tiles_y, num_tiles;
    int bw;                   // tile width: 8, 16 or 32
    int co_block;             // 32 or 64 output channels
    int stages;
    uint32_t x_stride;        // bytes of one 32-channel X tile (1024-aligned slot)
    uint32_t stage_stride;
    uint32_t x_bytes, z_bytes;
    uint32_t tmem_cols;
    int Cin, Cout;
    float* dw;
    float* db;
};

__global__ void __launch_bounds__(kWgThreads, 1) k_wgrad(const __grid_constant__ CUtensorMap tmX,
                                                  const __grid_constant__ CUtensorMap tmZ, const WgradParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)p.stages * p.stage_stride);
    uint64_t* empty = full + kWgMaxStages;
    uint64_t* done = empty + kWgMaxStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    float* s_db = reinterpret_cast<float*>(tmem_slot + 4); // bias sums of the CTA's channels
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int co0 = blockIdx.y * p.co_block;
    const bool bias = blockIdx.z == 0; // one CTA of a dZ tile's readers also sums it
    const int ci0 = blockIdx.z * 32;

    if (threadIdx.x == 32) {
        tc::prefetch_map(&tmX);
        tc::prefetch_map(&tmZ);
    }
    if (warp == 0) tc::tmem_alloc(tmem_slot, p.tmem_cols);
    if (threadIdx.x == 32) {
        for (int s = 0; s < p.stages; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], bias ? 1 + kWgSumWarps : 1); // the MMAs, and the warps that sum dZ
        }
        tc::mbar_init(done, 1);
        tc::fence_barrier_init();
    }
    if (threadIdx.x < 64) s_db[threadIdx.x] = 0.0f;
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    grid_dependency_wait();
    if (warp >= 2 && bias) {
        // ---- bias sums: thread = 8 channels of every `per`-th pixel of the tile's own rows
        const uint32_t groups = (uint32_t)p.co_block / 8, zrow = 2u * (uint32_t)p.co_block;
        const uint32_t tid = threadIdx.x - 64, g = tid % groups, pl = tid / groups, per = 32 * kWgSumWarps / groups;
        float sum[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) sum[q] = 0.0f;
        uint32_t it = 0, s = 0;
        for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x, ++it) {
            const bool ready = tc::mbar_wait_warp(&full[s], (it / p.stages) & 1, kWaitBudget);
            __syncwarp();
            if (!ready) {
                set_error(25);
                break;
            }
            // rows past the image are zero; the halo rows above and below are other tiles' own
            const uint8_t* z = smem + s * p.stage_stride;
            for (uint32_t r = (uint32_t)p.bw + pl; r < (uint32_t)p.bw * (kWgRows + 1); r += per) {
                const uint32_t piece = p.co_block == 64 ? (g ^ (r & 7)) : (g ^ ((r >> 1) & 3)); // TMA's swizzle
                const uint4 v = *reinterpret_cast<const uint4*>(z + r * zrow + piece * 16);
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 f = __bfloat1622float2(h[q]);
                    sum[2 * q] += f.x;
                    sum[2 * q + 1] += f.y;
                }
            }
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&empty[s]);
            if (++s == (uint32_t)p.stages) s = 0;
        }
        // lanes of the same channels first, then one shared add per warp and channel
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            for (uint32_t o = groups; o < 32; o <<= 1) sum[q] += __shfl_xor_sync(0xFFFFFFFFu, sum[q], o);
            if ((uint32_t)lane < groups) atomicAdd(&s_db[8 * g + q], sum[q]);
        }
    }
    if (warp == 0 && lane == 0) {
        uint32_t it = 0, s = 0;
        for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x, ++it) {
            if (it >= (uint32_t)p.stages && !tc::mbar_wait(&empty[s], ((it / p.stages) - 1) & 1, kWaitBudget)) {
                set_error(21);
                break;
            }
            const int per_img = p.tiles_x * p.tiles_y;
            const int n_img = t / per_img, r = t % per_img;
            const int y0 = (r / p.tiles_x) * kWgRows, x0 = (r % p.tiles_x) * p.bw;
            uint8_t* st = smem + s * p.stage_stride;
            tc::mbar_arrive_expect_tx(&full[s], p.x_bytes + p.z_bytes);
            tc::tma_load_4d(st, &tmZ, &full[s], co0, x0, y0 - 1, n_img);
            tc::tma_load_4d(st + p.stage_stride - p.x_stride, &tmX, &full[s], ci0, x0 - 1, y0, n_img);
            if (++s == (uint32_t)p.stages) s = 0;
        }
        // drain: every issued copy must have landed before the CTA may exit
        for (uint32_t q = 0; q < (uint32_t)p.stages && q < it; ++q) {
            const uint32_t last = ((it - 1 - q) / p.stages) * p.stages + q;
            if (!tc::mbar_wait(&full[q], (last / p.stages) & 1, kWaitBudget)) set_error(22);
        }
    } else if (warp == 1) { // converged; one elected lane issues
        const uint32_t elected = tc::elect_one();
        const uint32_t zrow = 2u * (uint32_t)p.co_block;     // bytes of one dZ pixel (its swizzle width)
        const uint32_t xrow = 64u;
        const uint32_t ximg = (uint32_t)(p.bw + 2) * xrow;   // one image row of the X tile
        // K = 16 pixels: two groups of 8, of one image row or, for 8-wide tiles, of two
        const uint32_t segs = p.bw >= 16 ? (uint32_t)p.bw / 16 : 1, row_step = p.bw >= 16 ? 1 : 2;
        const uint64_t ax = tc::smem_desc_mn(0, xrow, p.bw >= 16 ? 8u * xrow : ximg, 4u);
        const uint64_t bz = tc::smem_desc_mn(0, (uint32_t)p.bw * zrow, 8u * zrow, p.co_block == 64 ? 2u : 4u);
        const uint32_t idesc = tc::idesc_bf16(128, 3u * (uint32_t)p.co_block) | tc::kIdescMnMajorAB;
        uint32_t it = 0, s = 0;
        for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x, ++it) {
            if (!tc::mbar_wait_warp(&full[s], (it / p.stages) & 1, kWaitBudget)) {
                set_error(23);
                break;
            }
            tc::fence_after_sync();
            const uint32_t z = tc::smem_u32(smem + s * p.stage_stride);
            const uint32_t x = z + p.stage_stride - p.x_stride;
            for (uint32_t r = 0; r < (uint32_t)kWgRows; r += row_step)
                for (uint32_t q = 0; q < segs; ++q) {
                    const uint64_t ad = ax + ((x + r * ximg + q * 16 * xrow) >> 4);
                    const uint64_t bd = bz + ((z + (r * p.bw + q * 16) * zrow) >> 4);
                    tc::mma_bf16(tmem, ad, bd, idesc, (it > 0 || r > 0 || q > 0) ? 1u : 0u, elected);
                }
            if (elected) tc::mma_commit(&empty[s]);
            if (++s == (uint32_t)p.stages) s = 0;
        }
        if (elected) tc::mma_commit(done);
    }

    const bool any = (int)blockIdx.x < p.num_tiles;
    __syncwarp(); // warp 0: its producer lane
    const bool ready = any && tc::mbar_wait_warp(done, 0, kWaitBudget);
    if (any && !ready) set_error(24);
    __syncwarp();
    tc::fence_after_sync();
    if (ready && warp < 3) {
        const int ci = ci0 + lane;
        for (int j = 0; j < 3; ++j) {
            const int tap = (2 - j) * 3 + warp;
            for (int k = 0; k < p.co_block; k += 16) {
                uint32_t r0[16];
                tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(j * p.co_block + k), r0);
                tc::tmem_ld_wait();
                float* dst = p.dw + ((size_t)tap * p.Cout + co0 + k) * p.Cin + ci;
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    if (co0 + k + q < p.Cout) atomicAdd(dst + (size_t)q * p.Cin, __uint_as_float(r0[q]));
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (bias && threadIdx.x < (unsigned)p.co_block && co0 + (int)threadIdx.x < p.Cout)
        atomicAdd(p.db + co0 + threadIdx.x, s_db[threadIdx.x]);
    if (warp == 0) tc::tmem_dealloc(tmem, p.tmem_cols);
}

// ---- host: tensor maps ----
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    KF_REQUIRE(fn, KF_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    return fn;
}

CUtensorMap make_map(const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                     const uint32_t* box, CUtensorMapSwizzle swz) {
    CUtensorMap m;
    std::memset(&m, 0, sizeof(m));
    uint32_t estr[5] = {1, 1, 1, 1, 1};
    const CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base),
                                   reinterpret_cast<const cuuint64_t*>(dims),
                                   reinterpret_cast<const cuuint64_t*>(strides_bytes),
                                   reinterpret_cast<const cuuint32_t*>(box), estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        char msg[256];
        std::snprintf(msg, sizeof(msg),
                      "cuTensorMapEncodeTiled rejected a tensor layout (CUresult %d, rank %d, dims %llu x %llu, "
                      "box %u x %u)",
                      (int)r, rank, (unsigned long long)dims[0], (unsigned long long)dims[1], box[0], box[1]);
        throw KfError(KF_ERR_INVALID_ARGUMENT, msg);
    }
    return m;
}

uint32_t pow2_at_least(uint32_t v) {
    uint32_t c = 32;
    while (c < v) c <<= 1;
    return c;
}

template <int MODE, int SWZ, int kStages> size_t smem_bytes(int n_tile) {
    const size_t a = 128u * SWZ, b = (((size_t)n_tile * SWZ) + 1023) & ~size_t(1023);
    return 1024 + kStages * (a + b) + 256 + 4u * (size_t)n_tile;
}

template <int MODE, int SWZ, int kStages>
void launch_tc(dim3 grid, const CUtensorMap& a, const CUtensorMap& b, const TcParams& p, cudaStream_t st) {
    const size_t sm = smem_bytes<MODE, SWZ, kStages>(p.n_tile);
    static bool configured = false;
    if (!configured) {
        KF_CUDA_CHECK(cudaFuncSetAttribute(k_tc<MODE, SWZ, kStages>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem_bytes<MODE, SWZ, kStages>(256)));
        configured = true;
    }
    k_tc<MODE, SWZ, kStages><<<grid, 128, sm, st>>>(a, b, p);
    KF_CUDA_CHECK(cudaGetLastError());
}

// Shape of a halo-convolution launch: rows per tile R, channels per chunk CK, and the
// shared memory it takes. Larger R first (less halo per output row, fewer weight
// reloads per pixel), then larger CK; both accumulators must fit the 512 TMEM columns.
struct HaloShape {
    int R = 0, CK = 0, stages = 3;
    bool w_resident = false;
    uint32_t halo_bytes = 0, halo_stride = 0, w_bytes = 0, w_stride = 0;
    size_t smem = 0;
};

int halo_stack(int n_tile) { return std::min(3, 256 / n_tile); }

bool halo_shape(int Cin, int n_tile, HaloShape& out) {
    for (int R : {8, 4, 2, 1}) {
        if (2 * R * n_tile > 512) continue;
        const int S = halo_stack(n_tile);
        if (!((R >= 4 && S == 3) || (R == 2 && S >= 2) || (R == 1 && S == 1))) continue;
        // 32-channel chunks first (64-byte TMA pieces, half the chunk round trips), with three
        // stages or, where those do not fit, two; then 16-channel chunks
        for (const auto& [CK, stages] : {std::pair{32, 3}, std::pair{32, 2}, std::pair{16, 3}, std::pair{16, 2}}) {
            if (Cin % CK) continue;
            if (R == 8 && stages == 3) continue; // an 8-row halo leaves room for two
            HaloShape h;
            h.R = R;
            h.CK = CK;
            h.stages = stages;
            h.w_resident = Cin == CK;
            h.halo_bytes = (uint32_t)((R + 2) * kHaloW * CK * 2);
            h.halo_stride = (h.halo_bytes + 1023u) & ~1023u;
            h.w_bytes = (uint32_t)(9 * n_tile * CK * 2);
            h.w_stride = (h.w_bytes + 1023u) & ~1023u;
            h.smem = 1024 + (size_t)stages * h.halo_stride +
                     (size_t)(h.w_resident ? 1 : stages) * h.w_stride + 256 + 4u * (size_t)n_tile;
            if (h.smem <= 227u * 1024u) {
                out = h;
                return true;
            }
        }
    }
    return false;
}

int num_sms() {
    int dev = 0, n = 0;
    KF_CUDA_CHECK(cudaGetDevice(&dev));
    KF_CUDA_CHECK(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    return std::max(1, n);
}

template <int CK, int R, int STACK, int STAGES, bool EXTRA>
void launch_halo_kernel(dim3 grid, const CUtensorMap& x, const CUtensorMap& w, const HaloParams& p, size_t smem,
                 cudaStream_t st) {
    static bool configured = false;
    if (!configured) {
        KF_CUDA_CHECK(cudaFuncSetAttribute(k_conv_halo<CK, R, STACK, STAGES, EXTRA>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        configured = true;
    }
    launch_overlapped(k_conv_halo<CK, R, STACK, STAGES, EXTRA>, grid, dim3(kHaloThreads), smem, st, x, w, p);
}
// EXTRA: with an upsampled or a head output, in an instantiation of its own (its branches cost the
// layers without them 3 to 6 %: 96 -> 32 at 1920 x 1088 104 and 110 us).
template <int CK, int R, int STACK, int STAGES>
void launch_halo(dim3 grid, const CUtensorMap& x, const CUtensorMap& w, const HaloParams& p, size_t smem,
                 cudaStream_t st, bool extra) {
    if (extra) launch_halo_kernel<CK, R, STACK, STAGES, true>(grid, x, w, p, smem, st);
    else launch_halo_kernel<CK, R, STACK, STAGES, false>(grid, x, w, p, smem, st);
}

// One instantiation per (rows per tile, stacked rows, stages): R = 8 comes with n_tile <= 32
// and R = 4 with n_tile <= 64, so STACK = 3; R = 2 with n_tile <= 128 (STACK 2 or 3); R = 1
// with n_tile > 128 (STACK 1). halo_shape takes no other pair.
template <int CK, int STAGES>
bool launch_halo_stages(dim3 grid, const CUtensorMap& x, const CUtensorMap& w, const HaloParams& p, size_t smem,
                        cudaStream_t st, bool extra) {
    if (p.R == 8 && p.stack == 3 && STAGES == 2) launch_halo<CK, 8, 3, 2>(grid, x, w, p, smem, st, extra);
    else if (p.R == 4 && p.stack == 3) launch_halo<CK, 4, 3, STAGES>(grid, x, w, p, smem, st, extra);
    else if (p.R == 2 && p.stack == 2) launch_halo<CK, 2, 2, STAGES>(grid, x, w, p, smem, st, extra);
    else if (p.R == 2 && p.stack == 3) launch_halo<CK, 2, 3, STAGES>(grid, x, w, p, smem, st, extra);
    else if (p.R == 1 && p.stack == 1) launch_halo<CK, 1, 1, STAGES>(grid, x, w, p, smem, st, extra);
    else return false;
    return true;
}
template <int CK> void launch_halo_ck(dim3 grid, const CUtensorMap& x, const CUtensorMap& w, const HaloParams& p,
                                      int stages, size_t smem, cudaStream_t st, bool extra) {
    const bool ok = stages == 2 ? launch_halo_stages<CK, 2>(grid, x, w, p, smem, st, extra)
                                : launch_halo_stages<CK, 3>(grid, x, w, p, smem, st, extra);
    if (!ok) throw KfError(KF_ERR_INTERNAL, "conv3x3: no halo kernel for this tile shape");
}

// The halo kernel for images at least 96 pixels wide. Returns 0 when no shape
// fits (the caller takes the per-tile kernel), 1 when it ran, 2 when it also did the fused work.
int conv3x3_halo(const __nv_bfloat16* x, int N, int H, int W, int Cin, const __nv_bfloat16* w, int Cout_rows,
                 const float* bias, int Cout, bool relu, __nv_bfloat16* y, int y_cstride, int y_coff,
                 cudaStream_t st, float* y_f32, const ConvFuse* fuse) {
    const int n_tile = Cout_rows <= 256 ? Cout_rows : 128;
    HaloShape h;
    // a tile is 128 pixels of one row: from 96 pixels wide on, at most a quarter of its
    // rows are padding (the per-tile kernel takes narrower images)
    if (W < 96 || !halo_shape(Cin, n_tile, h)) return 0;
    // input NHWC: dims (Cin, W, H, N), a box of CK channels x 130 pixels x (R + 2) rows,
    // swizzled like the weights (CK x 2 bytes per row)
    const uint64_t xdims[4] = {(uint64_t)Cin, (uint64_t)W, (uint64_t)H, (uint64_t)N};
    const uint64_t xstr[3] = {(uint64_t)Cin * 2, (uint64_t)W * Cin * 2, (uint64_t)H * W * Cin * 2};
    const uint32_t xbox[4] = {(uint32_t)h.CK, (uint32_t)kHaloW, (uint32_t)h.R + 2, 1};
    const CUtensorMap mx = make_map(x, 4, xdims, xstr, xbox,
                                    h.CK == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    const uint64_t wdims[3] = {(uint64_t)Cin, (uint64_t)Cout_rows, 9};
    const uint64_t wstr[2] = {(uint64_t)Cin * 2, (uint64_t)Cout_rows * Cin * 2};
    const uint32_t wbox[3] = {(uint32_t)h.CK, (uint32_t)n_tile, 1};  // one tap per copy
    const CUtensorMap mw = make_map(w, 3, wdims, wstr, wbox,
                                    h.CK == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    HaloParams p{};
    p.N = N; p.H = H; p.W = W; p.Cin = Cin; p.Cout = Cout;
    p.n_tile = n_tile;
    p.R = h.R;
    p.kchunks = Cin / h.CK;
    p.tiles_x = (W + 127) / 128;
    p.tiles_y = (H + h.R - 1) / h.R;
    p.num_tiles = p.tiles_x * p.tiles_y * N;
    p.w_resident = h.w_resident ? 1 : 0;
    p.stack = halo_stack(n_tile);
    p.halo_bytes = h.halo_bytes;
    p.halo_stride = h.halo_stride;
    p.w_bytes = h.w_bytes;
    p.w_stride = h.w_stride;
    p.tmem_cols = pow2_at_least((uint32_t)(2 * h.R * n_tile));
    p.bias = bias;
    p.relu = relu ? 1 : 0;
    p.out = y;
    p.outf = y_f32;
    p.out_cstride = y_cstride;
    p.out_coff = y_coff;
    p.settled = fuse && fuse->settled ? 1 : 0;
    if (fuse && fuse->mask) {
        p.mask = fuse->mask;
        p.aux_cs = fuse->mask_cs;
        p.aux_co = fuse->mask_co;
    }
    bool fused = false;
    // pooling pairs rows inside a tile (R even) and reads the right neighbour's lane
    if (fuse && fuse->pool_out && y && !y_f32 && Cout % 8 == 0 && n_tile % 8 == 0 && h.R % 2 == 0 && H % 2 == 0 &&
        W % 2 == 0) {
        p.pool_out = fuse->pool_out;
        fused = true;
    }
    const bool extra = fuse && (fuse->up_out || fuse->head4);
    if (fuse && fuse->up_out) {
        p.up_out = fuse->up_out;
        p.aux_cs = fuse->up_cs;
        p.aux_co = fuse->up_co;
        if (fuse->up_only) p.out = nullptr;
    }
    if (fuse && fuse->head4) p.base = fuse->base;
    const int slices = (Cout_rows + n_tile - 1) / n_tile;
    const int per_slice = std::max(1, num_sms() / slices);
    const dim3 grid((unsigned)std::min(p.num_tiles, per_slice), (unsigned)slices, 1);
    if (h.CK == 32)
        launch_halo_ck<32>(grid, mx, mw, p, h.stages, h.smem, st, extra);
    else
        launch_halo_ck<16>(grid, mx, mw, p, h.stages, h.smem, st, extra);
    return fused ? 2 : 1;
}

template <int KC, bool EXTRA>
void launch_tile_kernel(dim3 grid, const CUtensorMap& x, const CUtensorMap& w, const TileParams& p, size_t smem,
                        cudaStream_t st) {
    static bool configured = false;
    if (!configured) {
        KF_CUDA_CHECK(
            cudaFuncSetAttribute(k_conv_tile<KC, EXTRA>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        configured = true;
    }
    launch_overlapped(k_conv_tile<KC, EXTRA>, grid, dim3(kTileThreads), smem, st, x, w, p);
}
template <int KC>
void launch_tile(dim3 grid, const CUtensorMap& x, const CUtensorMap& w, const TileParams& p, size_t smem,
                 cudaStream_t st, bool extra) {
    if (extra) launch_tile_kernel<KC, true>(grid, x, w, p, smem, st);
    else launch_tile_kernel<KC, false>(grid, x, w, p, smem, st);
}

// The tile kernel, for up to 288 input channels (one instantiation per 32; with more, the weights
// of 32 output channels and a halo no longer fit). Returns 0 for more (the caller takes k_tc), 1
// when it ran, 2 when it also did the fused work.
int conv3x3_tile(const __nv_bfloat16* x, int N, int H, int W, int Cin, const __nv_bfloat16* w, int Cout_rows,
                 const float* bias, int Cout, bool relu, __nv_bfloat16* y, int y_cstride, int y_coff,
                 cudaStream_t st, float* y_f32, const ConvFuse* fuse) {
    if (Cin % 32 || Cin > 288) return 0;
    TileParams p{};
    const int kchunks = Cin / 32;
    p.tiles_x = (W + kTileW - 1) / kTileW;
    p.tiles_y = (H + kTileH - 1) / kTileH;
    const int64_t tiles = (int64_t)p.tiles_x * p.tiles_y * N;
    if (tiles > (1 << 30)) return 0;
    p.num_tiles = (int)tiles;
    const int sms = num_sms();
    const size_t limit = 227 * 1024, halo = (size_t)kchunks * kTileHaloSlot;
    auto bytes = [&](int n, int bufs) {
        return 1024 + (size_t)bufs * halo + (size_t)kchunks * 9 * n * 64 + 256 + 4u * (size_t)n;
    };
    // Output channels per CTA: as many as fit (fewer reads of the halo, more columns per operand
    // fetch) while every SM still gets a tile; fewer, down to 16, where there are few tiles.
    int best = 0;
    for (int n = 16; n <= std::min(256, Cout_rows); n += 16) {
        const int slices = (Cout_rows + n - 1) / n;
        if (n > 16 && slices == (Cout_rows + n - 17) / (n - 16)) continue; // no fewer slices than n - 16
        if (bytes(n, 1) > limit) break;
        if (best && tiles * slices < sms) break;
        best = n;
    }
    if (!best) return 0;
    p.n_tile = best;
    const int slices = (Cout_rows + best - 1) / best;
    p.bufs = bytes(best, 2) <= limit && tiles * slices > sms ? 2 : 1;
    const size_t smem = bytes(best, p.bufs);
    const int per_sm = std::max<int>(1, std::min<int>((int)(limit / (smem + 1024)), 512 / (int)pow2_at_least(2u * best)));
    const uint64_t xdims[4] = {(uint64_t)Cin, (uint64_t)W, (uint64_t)H, (uint64_t)N};
    const uint64_t xstr[3] = {(uint64_t)Cin * 2, (uint64_t)W * Cin * 2, (uint64_t)H * W * Cin * 2};
    const uint32_t xbox[4] = {32, kTileHaloW, kTileHaloH, 1};
    const CUtensorMap mx = make_map(x, 4, xdims, xstr, xbox, CU_TENSOR_MAP_SWIZZLE_64B);
    const uint64_t wdims[3] = {(uint64_t)Cin, (uint64_t)Cout_rows, 9};
    const uint64_t wstr[2] = {(uint64_t)Cin * 2, (uint64_t)Cout_rows * Cin * 2};
    const uint32_t wbox[3] = {32, (uint32_t)best, 9};
    const CUtensorMap mw = make_map(w, 3, wdims, wstr, wbox, CU_TENSOR_MAP_SWIZZLE_64B);
    p.H = H; p.W = W; p.Cout = Cout;
    p.tmem_cols = pow2_at_least((uint32_t)(2 * best));
    p.bias = bias;
    p.relu = relu ? 1 : 0;
    p.out = y;
    p.outf = y_f32;
    p.out_cstride = y_cstride;
    p.out_coff = y_coff;
    p.settled = fuse && fuse->settled ? 1 : 0;
    if (fuse && fuse->mask) {
        p.mask = fuse->mask;
        p.aux_cs = fuse->mask_cs;
        p.aux_co = fuse->mask_co;
    }
    bool fused = false;
    if (fuse && fuse->pool_out && y && !y_f32 && Cout % 8 == 0 && H % 2 == 0 && W % 2 == 0) {
        p.pool_out = fuse->pool_out;
        fused = true;
    }
    const bool extra = fuse && (fuse->up_out || fuse->head4);
    if (fuse && fuse->up_out) {
        p.up_out = fuse->up_out;
        p.aux_cs = fuse->up_cs;
        p.aux_co = fuse->up_co;
        if (fuse->up_only) p.out = nullptr;
    }
    if (fuse && fuse->head4) p.base = fuse->base;
    const dim3 grid((unsigned)std::min<int64_t>(tiles, std::max(1, sms * per_sm / slices)), (unsigned)slices, 1);
    switch (kchunks) {
        case 1: launch_tile<1>(grid, mx, mw, p, smem, st, extra); break;
        case 2: launch_tile<2>(grid, mx, mw, p, smem, st, extra); break;
        case 3: launch_tile<3>(grid, mx, mw, p, smem, st, extra); break;
        case 4: launch_tile<4>(grid, mx, mw, p, smem, st, extra); break;
        case 5: launch_tile<5>(grid, mx, mw, p, smem, st, extra); break;
        case 6: launch_tile<6>(grid, mx, mw, p, smem, st, extra); break;
        case 7: launch_tile<7>(grid, mx, mw, p, smem, st, extra); break;
        case 8: launch_tile<8>(grid, mx, mw, p, smem, st, extra); break;
        default: launch_tile<9>(grid, mx, mw, p, smem, st, extra); break;
    }
    return fused ? 2 : 1;
}

} // namespace

bool conv3x3_bf16(const __nv_bfloat16* x, int N, int H, int W, int Cin, const __nv_bfloat16* w, int Cout_rows,
                  const float* bias, int Cout, bool relu, __nv_bfloat16* y, int y_cstride, int y_coff,
                  cudaStream_t st, float* y_f32, const ConvFuse* fuse) {
    KF_REQUIRE(N > 0 && H > 0 && W > 0, KF_ERR_INVALID_ARGUMENT, "conv3x3: empty tensor");
    KF_REQUIRE(y || y_f32, KF_ERR_INVALID_ARGUMENT, "conv3x3: no output tensor");
    KF_REQUIRE((Cin % 32 == 0 && Cin > 0) || Cin == 16, KF_ERR_INVALID_ARGUMENT,
               "conv3x3: input channels must be 16 or a multiple of 32");
    KF_REQUIRE(Cout > 0 && Cout <= Cout_rows && Cout_rows % 16 == 0, KF_ERR_INVALID_ARGUMENT,
               "conv3x3: weight rows must be a multiple of 16 covering the output channels");
    KF_REQUIRE(y_coff >= 0 && y_coff + Cout <= y_cstride, KF_ERR_INVALID_ARGUMENT, "conv3x3: output slice");
    // the epilogue stores 8 BF16 channels as one 16-byte word where the slice allows it
    KF_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0 && ((uintptr_t)y & 15) == 0 &&
                   ((uintptr_t)y_f32 & 3) == 0,
               KF_ERR_INVALID_ARGUMENT, "conv3x3: tensors must be 16-byte aligned (FP32 output: 4-byte)");
    KF_REQUIRE(!fuse || !fuse->pool_out || (((uintptr_t)fuse->pool_out & 15) == 0 && Cout % 8 == 0),
               KF_ERR_INVALID_ARGUMENT, "conv3x3: pooled output must be 16-byte aligned with Cout % 8 == 0");
    KF_REQUIRE(!fuse || !fuse->mask || (((uintptr_t)fuse->mask & 15) == 0 && Cout % 16 == 0 && fuse->mask_cs % 8 == 0 &&
                                        fuse->mask_co % 8 == 0 && Cin <= 288 && y && !fuse->pool_out),
               KF_ERR_INVALID_ARGUMENT, "conv3x3: mask layout");
    KF_REQUIRE(!fuse || !fuse->up_out ||
                   (((uintptr_t)fuse->up_out & 31) == 0 && Cout % 16 == 0 && fuse->up_cs % 16 == 0 &&
                    fuse->up_co % 16 == 0 && !fuse->pool_out && !fuse->mask && y && !y_f32 && Cin <= 288),
               KF_ERR_INVALID_ARGUMENT, "conv3x3: upsampled output layout");
    KF_REQUIRE(!fuse || !fuse->head4 ||
                   (y_f32 && ((uintptr_t)y_f32 & 15) == 0 && ((uintptr_t)fuse->base & 15) == 0 && Cout == 3 &&
                    y_cstride == 4 && y_coff == 0 && !fuse->mask && !fuse->up_out && Cin <= 288),
               KF_ERR_INVALID_ARGUMENT, "conv3x3: head layout");
    const int halo = conv3x3_halo(x, N, H, W, Cin, w, Cout_rows, bias, Cout, relu, y, y_cstride, y_coff, st, y_f32,
                                  fuse);
    if (halo) return halo == 2;
    KF_REQUIRE(Cin % 32 == 0, KF_ERR_INVALID_ARGUMENT,
               "conv3x3: 16 input channels need an image the halo kernel takes (at least 96 wide)");
    const int tile = conv3x3_tile(x, N, H, W, Cin, w, Cout_rows, bias, Cout, relu, y, y_cstride, y_coff, st, y_f32, fuse);
    if (tile) return tile == 2;
    // more input channels than the tile kernel holds: one CTA per tile of bw x bh = 128 pixels,
    // 9 tap-shifted boxes per chunk
    int bw = 128;
    while (bw > W && bw > 8) bw >>= 1;
    const int bh = 128 / bw;
    const uint64_t adims[4] = {(uint64_t)Cin, (uint64_t)W, (uint64_t)H, (uint64_t)N};
    const uint64_t astr[3] = {(uint64_t)Cin * 2, (uint64_t)W * Cin * 2, (uint64_t)H * W * Cin * 2};
    const uint32_t abox[4] = {32, (uint32_t)bw, (uint32_t)bh, 1};
    const CUtensorMap ma = make_map(x, 4, adims, astr, abox, CU_TENSOR_MAP_SWIZZLE_64B);
    const int n_tile = Cout_rows <= 256 ? Cout_rows : 128;
    const uint64_t bdims[3] = {(uint64_t)Cin, (uint64_t)Cout_rows, 9};
    const uint64_t bstr[2] = {(uint64_t)Cin * 2, (uint64_t)Cout_rows * Cin * 2};
    const uint32_t bbox[3] = {32, (uint32_t)n_tile, 1};
    const CUtensorMap mb = make_map(w, 3, bdims, bstr, bbox, CU_TENSOR_MAP_SWIZZLE_64B);
    TcParams p{};
    p.N = N; p.H = H; p.W = W; p.Cin = Cin; p.Cout = Cout;
    p.bw = bw; p.bh = bh;
    p.tiles_x = (W + bw - 1) / bw;
    p.tiles_y = (H + bh - 1) / bh;
    p.n_tile = n_tile;
    p.kchunks = Cin / 32;
    p.k_iters = 9 * p.kchunks;
    p.k_per_split = p.k_iters;
    p.bias = bias;
    p.relu = relu ? 1 : 0;
    p.out = y;
    p.outf = y_f32;
    p.out_cstride = y_cstride;
    p.out_coff = y_coff;
    p.tmem_cols = pow2_at_least((uint32_t)n_tile);
    const dim3 grid((unsigned)(p.tiles_x * p.tiles_y * N), (unsigned)((Cout_rows + n_tile - 1) / n_tile), 1);
    launch_tc<0, 64, 3>(grid, ma, mb, p, st);
    return false;
}

void gemm_bf16_tn(const __nv_bfloat16* a, int M, const __nv_bfloat16* b, int N, int K, float* d, int ldd, int splits,
                  cudaStream_t st) {
    KF_REQUIRE(M > 0 && N > 0 && K > 0, KF_ERR_INVALID_ARGUMENT, "gemm: empty operand");
    KF_REQUIRE(K % 8 == 0, KF_ERR_INVALID_ARGUMENT, "gemm: K must be a multiple of 8 (16-byte rows)");
    KF_REQUIRE(((uintptr_t)a & 15) == 0 && ((uintptr_t)b & 15) == 0, KF_ERR_INVALID_ARGUMENT,
               "gemm: operands must be 16-byte aligned");
    KF_REQUIRE(d && ((uintptr_t)d & 3) == 0 && ldd >= N, KF_ERR_INVALID_ARGUMENT,
               "gemm: output must be 4-byte aligned with ldd >= n");
    const int n_tile = N <= 256 ? ((N + 15) / 16) * 16 : 128;
    const uint64_t adims[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t astr[1] = {(uint64_t)K * 2};
    const uint32_t abox[2] = {64, 128};
    const CUtensorMap ma = make_map(a, 2, adims, astr, abox, CU_TENSOR_MAP_SWIZZLE_128B);
    const uint64_t bdims[2] = {(uint64_t)K, (uint64_t)N};
    const uint64_t bstr[1] = {(uint64_t)K * 2};
    const uint32_t bbox[2] = {64, (uint32_t)n_tile};
    const CUtensorMap mb = make_map(b, 2, bdims, bstr, bbox, CU_TENSOR_MAP_SWIZZLE_128B);
    TcParams p{};
    p.n_tile = n_tile;
    p.outf = d;
    p.ldo = ldd;
    p.M_valid = M;
    p.N_valid = N;
    p.k_iters = (K + 63) / 64;
    const int sp = std::max(1, std::min(splits, p.k_iters));
    p.k_per_split = (p.k_iters + sp - 1) / sp;
    p.tmem_cols = pow2_at_least((uint32_t)n_tile);
    const dim3 grid((unsigned)((M + 127) / 128), (unsigned)((N + n_tile - 1) / n_tile),
                    (unsigned)((p.k_iters + p.k_per_split - 1) / p.k_per_split));
    launch_tc<1, 128, 4>(grid, ma, mb, p, st);
}

void conv3x3_wgrad_bf16(const __nv_bfloat16* x, int x_cstride, int N, int H, int W, int Cin, const __nv_bfloat16* dz,
                        int dz_channels, int Cout, float* dw, float* db, cudaStream_t st) {
    KF_REQUIRE(N > 0 && H > 0 && W > 0, KF_ERR_INVALID_ARGUMENT, "wgrad: empty tensor");
    KF_REQUIRE(Cin > 0 && Cin % 32 == 0 && dz_channels % 32 == 0 && Cout > 0 && Cout <= dz_channels,
               KF_ERR_INVALID_ARGUMENT, "wgrad: channels must be multiples of 32");
    KF_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)dz & 15) == 0 && x_cstride % 8 == 0, KF_ERR_INVALID_ARGUMENT,
               "wgrad: tensors must be 16-byte aligned");
    KF_REQUIRE(x_cstride >= Cin, KF_ERR_INVALID_ARGUMENT, "wgrad: channel stride below the input channels");
    KF_REQUIRE(((uintptr_t)dw & 3) == 0 && ((uintptr_t)db & 3) == 0, KF_ERR_INVALID_ARGUMENT,
               "wgrad: gradients must be 4-byte aligned");
    KF_REQUIRE((int64_t)((W + 7) / 8) * ((H + kWgRows - 1) / kWgRows) * N <= (1 << 30), KF_ERR_LIMIT,
               "wgrad: too many pixels in one call");
    WgradParams p{};
    // K steps are 16 pixels of a row, or two rows of 8 where the image is that narrow; 32-pixel
    // tiles halve the halo columns where they leave no more padding than 16-pixel ones
    p.bw = W <= 8 ? 8 : ((W - 1) / 16 % 2 == 0 ? 16 : 32);
    p.tiles_x = (W + p.bw - 1) / p.bw;
    p.tiles_y = (H + kWgRows - 1) / kWgRows;
    p.num_tiles = p.tiles_x * p.tiles_y * N;
    p.co_block = dz_channels % 64 == 0 ? 64 : 32;
    p.Cin = Cin;
    p.Cout = Cout;
    p.dw = dw;
    p.db = db;
    p.x_bytes = (uint32_t)(kWgRows * (p.bw + 2) * 64);
    p.x_stride = (p.x_bytes + 64 + 1023u) & ~1023u; // the unused fourth shift reads one pixel past the tile
    p.z_bytes = (uint32_t)((kWgRows + 2) * p.bw * 2 * p.co_block);
    const uint32_t z_stride = (p.z_bytes + 1023u) & ~1023u;
    const int ci_blocks = Cin / 32, co_blocks = dz_channels / p.co_block, sms = num_sms();
    p.stage_stride = p.x_stride + z_stride;
    p.stages = std::max(2, std::min<int>(kWgMaxStages, (int)(110u * 1024u / p.stage_stride)));
    p.tmem_cols = pow2_at_least((uint32_t)(3 * p.co_block));
    const size_t smem = 1024 + (size_t)p.stages * p.stage_stride + 128 + 256;
    const uint64_t xdims[4] = {(uint64_t)Cin, (uint64_t)W, (uint64_t)H, (uint64_t)N};
    const uint64_t xstr[3] = {(uint64_t)x_cstride * 2, (uint64_t)W * x_cstride * 2, (uint64_t)H * W * x_cstride * 2};
    const uint32_t xbox[4] = {32, (uint32_t)p.bw + 2, kWgRows, 1};
    const CUtensorMap mx = make_map(x, 4, xdims, xstr, xbox, CU_TENSOR_MAP_SWIZZLE_64B);
    const uint64_t zdims[4] = {(uint64_t)dz_channels, (uint64_t)W, (uint64_t)H, (uint64_t)N};
    const uint64_t zstr[3] = {(uint64_t)dz_channels * 2, (uint64_t)W * dz_channels * 2,
                              (uint64_t)H * W * dz_channels * 2};
    const uint32_t zbox[4] = {(uint32_t)p.co_block, (uint32_t)p.bw, kWgRows + 2, 1};
    const CUtensorMap mz = make_map(dz, 4, zdims, zstr, zbox,
                                    p.co_block == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
    static bool configured = false;
    if (!configured) {
        KF_CUDA_CHECK(cudaFuncSetAttribute(k_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        configured = true;
    }
    const int blocks = co_blocks * ci_blocks;
    const int splits = std::max(1, std::min(p.num_tiles, sms / std::max(1, blocks)));
    const dim3 grid((unsigned)splits, (unsigned)co_blocks, (unsigned)ci_blocks);
    launch_overlapped(k_wgrad, grid, dim3(kWgThreads), smem, st, mx, mz, p);
}

namespace {
// One thread waits on an mbarrier that nothing arrives on, through the same bounded wait the
// tensor-core kernels use: it gives up after `budget` SM cycles and records `code`.
__global__ void k_wait_probe(long long budget, uint32_t code) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_barrier_init();
        if (!tc::mbar_wait(&bar, 0, budget)) set_error(code);
    }
}
} // namespace

void tc_wait_probe(long long budget_cycles, cudaStream_t st) {
    KF_REQUIRE(budget_cycles > 0 && budget_cycles <= kWaitBudget, KF_ERR_INVALID_ARGUMENT,
               "wait probe: budget must be in (0, 2e9] cycles");
    k_wait_probe<<<1, 32, 0, st>>>(budget_cycles, kWaitProbeError);
    KF_CUDA_CHECK(cudaGetLastError());
}

uint32_t tc_take_error() {
    uint32_t e = 0, z = 0;
    KF_CUDA_CHECK(cudaMemcpyFromSymbol(&e, g_tc_error, sizeof(e)));
    KF_CUDA_CHECK(cudaMemcpyToSymbol(g_tc_error, &z, sizeof(z)));
    return e;
}

} // namespace kf
