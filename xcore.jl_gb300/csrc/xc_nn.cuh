// Internal declarations of the learned preconditioner's network (the U-Net
// and its BF16 tensor-core convolutions).
#pragma once

#include <cuda_runtime.h>

// the flag a kernel raises when one of its bounded waits runs out: `dev` for
// the kernels, check() waits for the stream and reports it as XC_TIMEOUT.  One
// flag serves any number of launches on any streams; it must outlive them.
struct ErrFlag {
  int* dev = nullptr;
  int* host = nullptr;
  bool* used = nullptr;      // its place in the context's page (null: allocated for itself)
  ErrFlag() = default;
  ErrFlag(const ErrFlag&) = delete;
  ErrFlag& operator=(const ErrFlag&) = delete;
  int init();
  int check(cudaStream_t s, const char* what);
  ~ErrFlag();
};

// y (NHWC BF16, or y_f32 FP32, either may be null) = relu?(conv3x3(x, w) + bias)
// x: NHWC BF16 [B][H][W][Cin]; w: BF16 [Cout][9][Cin]; bias: FP32 [Cout] or null.
// Cin, Cout in {16, 32, 64, 128}; W a multiple of 128 or a power of two below
// 128 with H divisible by 128 / W.  mask (NHWC BF16 like y, or null): y is
// zero where mask <= 0.  err: ErrFlag::dev.
int nn_conv3x3_fwd(const void* x, const void* w, const float* bias, void* y, float* y_f32, int B, int H, int W,
                   int Cin, int Cout, int relu, int* err, cudaStream_t s, const void* mask = nullptr);
// dw (FP32 [Cout][9][Cin]) = scale * sum_p dy[p] (x) x[p + off] and, unless
// null, db (FP32 [Cout]) = scale * sum_p dy[p] (each + its old value when
// accumulate); partial: FP32 scratch of nn_wgrad_scratch values
long long nn_wgrad_scratch(int B, int H, int W, int Cin, int Cout);
int nn_conv3x3_wgrad(const void* x, const void* dy, float* dw, float* db, float* partial, int B, int H, int W,
                     int Cin, int Cout, float scale, int accumulate, int* err, cudaStream_t s);

// the network on the stream without synchronising (graph capture allowed):
// the FP32 result [npix][16] (first out_ch channels used) is nn_out16(n)
struct xc_nn;
int nn_forward_async(xc_nn* n, const float* in, cudaStream_t s);
const float* nn_out16(const xc_nn* n);
// wait for the stream and report a bounded wait that ran out inside a
// convolution as XC_TIMEOUT
int nn_check(xc_nn* n, cudaStream_t s);
