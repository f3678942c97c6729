// kf_conv.h — tensor-core convolution / GEMM launchers (kf_conv.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace kf {

// Work a convolution can take over from what follows it: 2x2 average pooling of its BF16 output into
// a dense [N][H/2][W/2][Cout] tensor (FP32 averages of the rounded outputs, rounded to BF16).
// And a ReLU's backward mask: outputs whose place in `mask` (NHWC, channel stride mask_cs, slice
// starting at mask_co, both multiples of 8) is not positive become zero.
// And nearest 2x upsampling of the BF16 output into the channel slice up_co of an NHWC tensor
// [N][2H][2W][up_cs] (up_out 32-byte aligned, up_cs, up_co and Cout multiples of 16); with
// up_only the output itself is not written. Always done (at most 288 input channels then).
// head4: the FP32 output has 3 channels at stride 4 (y_f32 16-byte aligned): the fourth becomes
// zero, and `base`, if any, is added to the three (same layout, may be y_f32 itself).
// settled: the weights and bias were complete before the kernel that precedes this one in the
// stream started (the previous launch is one of a chain that waited): they may be loaded while
// that kernel still runs.
struct ConvFuse {
    bool settled = false;
    __nv_bfloat16* pool_out = nullptr;
    const __nv_bfloat16* mask = nullptr;
    int mask_cs = 0, mask_co = 0;
    __nv_bfloat16* up_out = nullptr;
    int up_cs = 0, up_co = 0;
    bool up_only = false;
    bool head4 = false;
    const float* base = nullptr;
};

// y[n, y, x, y_coff + co] = act(bias[co] + sum_{tap, ci} x[n, y+dy, x+dx, ci] * w[tap][co][ci])
// NHWC BF16, zero padding, FP32 accumulation on tcgen05. w is [9][Cout_rows][Cin] with
// Cout_rows a multiple of 16 (rows >= Cout are computed and dropped); Cin % 32 == 0, or
// Cin == 16 for images at least 96 wide.
// With y_f32 set, the output is written there in FP32 (same strides) and y is unused.
// Returns true when it also did the pooling asked for in `fuse` (the persistent kernels do it for even
// sizes and, from 96 pixels wide on, up to 128 output channels). A mask is always applied (at
// most 288 input channels then).
bool conv3x3_bf16(const __nv_bfloat16* x, int N, int H, int W, int Cin, const __nv_bfloat16* w, int Cout_rows,
                  const float* bias, int Cout, bool relu, __nv_bfloat16* y, int y_cstride, int y_coff,
                  cudaStream_t st, float* y_f32 = nullptr, const ConvFuse* fuse = nullptr);

// d[m][n] += sum_k a[m][k] * b[n][k]   (BF16 K-major operands, FP32 atomics; split-K over `splits`)
void gemm_bf16_tn(const __nv_bfloat16* a, int M, const __nv_bfloat16* b, int N, int K, float* d, int ldd, int splits,
                  cudaStream_t st);

// dw[tap][co][ci] += sum over pixels of dz[p][co] * x[p shifted by tap][ci] and db[co] += sum
// over pixels of dz[p][co], for co < Cout (FP32 atomics; x NHWC with channel stride x_cstride, dz
// dense [N][H][W][dz_channels], Cin and dz_channels multiples of 32).
void conv3x3_wgrad_bf16(const __nv_bfloat16* x, int x_cstride, int N, int H, int W, int Cin, const __nv_bfloat16* dz,
                        int dz_channels, int Cout, float* dw, float* db, cudaStream_t st);

// Reads and clears the error word the tensor-core kernels set when a bounded wait expires.
uint32_t tc_take_error();
// Error word a wait probe leaves when its wait gives up.
constexpr uint32_t kWaitProbeError = 99;
// Launches a kernel whose wait on a barrier that nothing arrives on gives up after
// budget_cycles SM cycles and sets the error word to kWaitProbeError (no fault: the
// context stays usable).
void tc_wait_probe(long long budget_cycles, cudaStream_t st);

} // namespace kf
