// 3x3 convolutions of the learned preconditioner's U-Net on the 5th-generation
// tensor cores (tcgen05), BF16 operands with FP32 accumulation in TMEM.
//
// Activations are NHWC BF16 (channels contiguous), weights [Cout][9][Cin]
// BF16 (tap t = 3 * (dy + 1) + (dx + 1)).  Zero padding at the image edge.
//
// Forward (and the data gradient, which is the forward convolution of dY with
// the flipped, transposed weights): an implicit GEMM with M = 128 pixels of
// one tile, N = Cout, K = 9 taps x Cin.  The tile's pixels shifted by each tap
// (zeros outside the image, which is the padding) come into the K-major
// swizzled layout the tensor core reads by TMA (64 channels) or 16-byte copies
// (16, 32), the weights by TMA; an mbarrier ring overlaps them with the MMAs,
// which one thread issues; the
// accumulator (128 lanes x Cout FP32 columns of TMEM, two of them) is read back
// by four warps for the epilogue (bias, ReLU, mask, BF16 and/or FP32 store)
// while the next tile's MMAs run.
//
// Weight gradient: dW[co][t][ci] = sum_p dY[p][co] X[p + off(t)][ci], a GEMM
// over the pixels.  Both operands are channel-contiguous in memory, MN-major
// for the tensor core, so tiles of 128 pixels are operands as they lie in
// memory.  M holds several taps at once: 128 / Cin tiles of Cin channels each
// (they lie one after another, the descriptor's leading offset steps from one
// to the next), N is Cout.  The bias gradient sum_p dY is added in FP32 by warps
// of its own from the same tiles.  FP32 partial sums per CTA, reduced over CTAs
// in a fixed order (deterministic).
#include <algorithm>
#include <cstring>
#include <mutex>

#include <cuda_bf16.h>

// A grid may be scheduled as soon as the one before it is past its wait
// (U-Net gradient at 8 x 256^2: 1187 -> 1177 us).  The tensor-core kernels wait after they have allocated their
// tensor memory: a block that arrives early can then only wait for memory whose
// owner already has all it needs.
#define XC_PDL_EARLY
#include "xc_internal.cuh"
#include "xc_nn.cuh"
#include "xc_once.h"
#include "xc_nn_tc.cuh"

using namespace xcnn;

namespace {

// ---------------------------------------------------------------------------
// tensor maps (driver entry point looked up through the runtime)
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

CUtensorMapSwizzle swizzle_for(int row_bytes) {
  return row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                          : (row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

// NHWC BF16 activations as (C, W, H, B), box (64, bw, bh, 1)
int make_act_map(CUtensorMap* tm, const void* p, int B, int H, int W, int C, int bw, int bh) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) { xc_set_error("cuTensorMapEncodeTiled is not available from the driver"); return XC_CUDA; }
  cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)bw, (cuuint32_t)bh, 1};
  cuuint32_t es[4] = {1, 1, 1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p), dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { xc_set_error("cuTensorMapEncodeTiled (activations) failed: %d", (int)r); return XC_CUDA; }
  return XC_OK;
}

// weights [Cout][9][Cin] BF16 as (Cin, 9, Cout), box (kc, 1, Cout)
int make_weight_map(CUtensorMap* tm, const void* p, int Cin, int Cout, int kc) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) { xc_set_error("cuTensorMapEncodeTiled is not available from the driver"); return XC_CUDA; }
  if (((uintptr_t)p & 15u) != 0) { xc_set_error("conv3x3: weight pointer not 16-byte aligned"); return XC_BAD_ARG; }
  cuuint64_t dims[3] = {(cuuint64_t)Cin, 9, (cuuint64_t)Cout};
  cuuint64_t strides[2] = {(cuuint64_t)Cin * 2, (cuuint64_t)9 * Cin * 2};
  cuuint32_t box[3] = {(cuuint32_t)kc, 1, (cuuint32_t)Cout};
  cuuint32_t es[3] = {1, 1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(p), dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(kc * 2), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { xc_set_error("cuTensorMapEncodeTiled (weights) failed: %d", (int)r); return XC_CUDA; }
  return XC_OK;
}

struct ConvArgs {
  int B, H, W, Cin, nkc, bw, bh;
  const __nv_bfloat16* x;   // NHWC [.., Cin]
  const float* bias;        // [Cout] or null
  int relu;                 // 1: max(v, 0) after the bias
  const __nv_bfloat16* mask;   // NHWC [.., Cout] or null: zero where mask <= 0 (a ReLU's backward)
  int tiles;
  __nv_bfloat16* out;       // NHWC [.., Cout] or null
  float* out_f32;           // NHWC [.., Cout] or null
  int* err;                 // set to a nonzero code when a bounded wait ran out
};

__device__ __forceinline__ void flag_error(int* err, int code) {
  if (err) {
    *(volatile int*)err = code;       // pinned host memory: read after the stream has been waited for
    __threadfence_system();
  }
}

// Tiles of 128 pixels (bw x bh from (x0, y0) of image b, shifted by (dx, dy),
// zeros outside the image) x KC channels in the swizzled layout the tensor core
// reads.  64 channels come by TMA: a row of 128 bytes per pixel.  A TMA box
// moves at a row per 2 to 3 clocks whatever its width, so 16 and 32 channels
// (rows of 32 and 64 bytes) are copied by 128 threads in 16-byte asynchronous
// copies instead, repeated reads of neighbouring taps hitting L1: 16 x 16
// channels at 8 x 256 x 256 pixels by TMA 52 us, by copies 28 us; 64 x 64 at
// 8 x 64 x 64 12 and 18 us.  A thread's places in the tile are the same for
// every tile and are formed once.
struct ImageTile { int b, y0, x0; };
__device__ __forceinline__ ImageTile tile_at(int t, int W, int H, int bw, int bh) {
  const int tx = W / bw, per = tx * (H / bh), b = t / per, rem = t - b * per, ry = rem / tx;
  return ImageTile{b, ry * bh, (rem - ry * tx) * bw};
}
template <int KC>
struct PixelCopies {
  static constexpr uint32_t RB = KC * 2u;
  static constexpr int CH = KC / 8;         // copies per thread and tile
  int my[CH], mx[CH], off[CH];              // pixel in the tile, element offset from the tile's first pixel
  uint32_t to[CH];                          // byte offset in shared memory
  __device__ __forceinline__ PixelCopies(int tid, int W, int bw) {
    const int shift = 31 - __clz(bw);
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      const int idx = tid + k * 128, m = idx / CH, c = idx % CH;
      my[k] = m >> shift;
      mx[k] = m & (bw - 1);
      off[k] = (my[k] * W + mx[k]) * KC + c * 8;
      to[k] = swz_chunk<RB>((uint32_t)m, (uint32_t)c);
    }
  }
  // the taps dx0 .. dx0 + N - 1 of row dy, one tile after another
  template <int N>
  __device__ __forceinline__ void load(uint32_t dst, const __nv_bfloat16* src, int H, int W, const ImageTile& t, int dy,
                                       int dx0) const {
    const int y = t.y0 + dy, x = t.x0 + dx0;
    const __nv_bfloat16* first = src + (((long long)t.b * H + y) * W + x) * KC;
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      const bool iny = (unsigned)(y + my[k]) < (unsigned)H;
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const bool in = iny && (unsigned)(x + j + mx[k]) < (unsigned)W;
        cp_async16(dst + j * (128u * RB) + to[k], in ? first + off[k] + j * KC : src, in);
      }
    }
  }
};
// Persistent kernel: one CTA per SM (two where shared memory allows) walks the
// tiles.  Warps 0-3 bring the pixels, warp 4 issues the MMAs, warps 5-8 read the
// accumulator back and store, on one of two accumulators while the MMAs of the
// next tile fill the other.  A step is the three taps of a row (16 and 32
// channels) or one tap's 64 channels.  Weights that leave room for the ring
// (up to 64 x 64 channels) are loaded once and stay; of larger ones each
// step's block travels in the ring beside the pixels.
template <int KC, int NOUT>
struct FwdCfg {
  static constexpr int kTaps = KC == 64 ? 1 : 3;               // taps per step
  static constexpr uint32_t kRowBytes = KC * 2;
  static constexpr uint32_t kABytes = 128u * KC * 2;           // one tap's pixels
  static constexpr uint32_t kBBytes = NOUT * KC * 2;           // one tap's weights
  static constexpr uint32_t kBStride = (kBBytes + 1023u) & ~1023u;
  static constexpr uint32_t kStage(bool res) { return kTaps * (kABytes + (res ? 0u : kBStride)); }
  static constexpr uint32_t kTmemCols = tmem_cols_for(2 * NOUT);
};

constexpr int kFwdThreads = 288;
constexpr int kMaxStages = 12;

// RES: all weight blocks resident, else in the ring
template <int KC, int NOUT, bool RES>
__global__ void __launch_bounds__(kFwdThreads) conv3x3_fwd_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                  const __grid_constant__ CUtensorMap tmB, ConvArgs a,
                                                                  int nstages) {
  using Cfg = FwdCfg<KC, NOUT>;
  constexpr bool TMA_A = KC == 64;
  constexpr int TAPS = Cfg::kTaps;
  constexpr uint32_t SBO = 8u * Cfg::kRowBytes;
  constexpr uint32_t LAYOUT = layout_for_row_bytes(Cfg::kRowBytes);
  constexpr uint32_t IDESC = idesc_bf16(128, NOUT);
  constexpr uint32_t STAGE = Cfg::kStage(RES);
  extern __shared__ uint8_t dsm[];
  __shared__ __align__(8) uint64_t bar_full[kMaxStages], bar_empty[kMaxStages];
  __shared__ __align__(8) uint64_t bar_w, bar_acc[2], bar_free[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int s_fail;
  const uint32_t base = (smem_u32(dsm) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nsteps = 9 / TAPS * a.nkc;               // per tile: (tap row or tap, channel chunk), chunk innermost
  const uint32_t ring = base + (RES ? 9u * (uint32_t)a.nkc * Cfg::kBStride : 0u);

  if (threadIdx.x == 0) {
    for (int s = 0; s < nstages; ++s) {
      mbar_init(smem_u32(&bar_full[s]), (TMA_A ? 0 : 128) + (TMA_A || !RES ? 1 : 0));
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    mbar_init(smem_u32(&bar_w), 1);
    for (int q = 0; q < 2; ++q) {
      mbar_init(smem_u32(&bar_acc[q]), 1);
      mbar_init(smem_u32(&bar_free[q]), 4);
    }
    s_fail = 0;
    mbar_fence_init();
  }
  if (warp == 4) {
    tmem_alloc(smem_u32(&tmem_slot), Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  XC_PDL_WAIT();     // (all of the above touches nothing an earlier grid writes)

  if (warp < 4) {
    const int tid = threadIdx.x;
    if (RES && tid == 0) {
      mbar_expect_tx(smem_u32(&bar_w), 9u * (uint32_t)a.nkc * Cfg::kBBytes);
      for (int kk = 0; kk < 9 * a.nkc; ++kk)
        tma_load_3d(base + (uint32_t)kk * Cfg::kBStride, &tmB, (kk % a.nkc) * KC, kk / a.nkc, 0, smem_u32(&bar_w));
    }
    const PixelCopies<TMA_A ? 16 : KC> px(tid, a.W, a.bw);
    int it = 0;
    bool ok = true;
    if (!TMA_A || tid == 0)
      for (int t = blockIdx.x; t < a.tiles && ok; t += gridDim.x) {
        const ImageTile tile = tile_at(t, a.W, a.H, a.bw, a.bh);
        for (int st = 0; st < nsteps; ++st, ++it) {
          const int s = it % nstages;
          // the slot is refilled once the MMAs that read it completed
          if (it >= nstages && !mbar_wait(smem_u32(&bar_empty[s]), ((it / nstages) - 1) & 1)) {
            flag_error(a.err, 1);
            s_fail = 1;
            ok = false;
            break;
          }
          const int row = st / a.nkc, kc = st - row * a.nkc;   // first tap TAPS * row
          const uint32_t sa = ring + s * STAGE, full = smem_u32(&bar_full[s]);
          if (tid == 0 && (TMA_A || !RES)) {
            mbar_expect_tx(full, (TMA_A ? Cfg::kABytes : 0u) + (RES ? 0u : TAPS * Cfg::kBBytes));
            if (TMA_A) tma_load_4d(sa, &tmA, kc * KC, tile.x0 + row % 3 - 1, tile.y0 + row / 3 - 1, tile.b, full);
            if (!RES) {
#pragma unroll
              for (int j = 0; j < TAPS; ++j)
                tma_load_3d(sa + TAPS * Cfg::kABytes + j * Cfg::kBStride, &tmB, kc * KC, TAPS * row + j, 0, full);
            }
          }
          if constexpr (!TMA_A) {
            px.template load<TAPS>(sa, a.x, a.H, a.W, tile, row - 1, -1);
            cp_async_arrive(full);
          }
        }
      }
    // after a wait that ran out, whatever is in flight ends before the CTA does
    if constexpr (!TMA_A) cp_async_wait_all();
    if (tid == 0) {
      if (RES) mbar_wait(smem_u32(&bar_w), 0);
      if (TMA_A || !RES)
        for (int q = it - nstages > 0 ? it - nstages : 0; q < it; ++q)
          mbar_wait(smem_u32(&bar_full[q % nstages]), (q / nstages) & 1);
    }
  } else if (warp == 4 && lane == 0) {
    // MMA issuer: taps in order, the channel chunks of a tap in order
    bool ok = true;
    int it = 0, n = 0;
    if (RES && !mbar_wait(smem_u32(&bar_w), 0)) {
      flag_error(a.err, 5);
      s_fail = 1;
      ok = false;
    }
    for (int t = blockIdx.x; t < a.tiles && ok; t += gridDim.x, ++n) {
      const int q = n & 1;
      if (n >= 2 && !mbar_wait(smem_u32(&bar_free[q]), ((n >> 1) - 1) & 1)) {
        flag_error(a.err, 6);
        s_fail = 1;
        break;
      }
      tc_fence_after();
      const uint32_t acc = tmem + (uint32_t)(q * NOUT);
      for (int st = 0; st < nsteps; ++st, ++it) {
        const int s = it % nstages;
        if (!mbar_wait(smem_u32(&bar_full[s]), (it / nstages) & 1)) {
          flag_error(a.err, 2);
          s_fail = 1;
          ok = false;
          break;
        }
        if (!TMA_A) fence_async_shared();
        tc_fence_after();
        const uint32_t sa = ring + s * STAGE;
        const uint32_t sb = RES ? base + (uint32_t)(TAPS * st) * Cfg::kBStride : sa + TAPS * Cfg::kABytes;
#pragma unroll
        for (int j = 0; j < TAPS; ++j)
#pragma unroll
          for (int k = 0; k < KC / 16; ++k)
            umma_bf16(acc, smem_desc(sa + j * Cfg::kABytes + k * 32, SBO, LAYOUT),
                      smem_desc(sb + j * Cfg::kBStride + k * 32, SBO, LAYOUT), IDESC, (st | j | k) != 0 ? 1u : 0u);
        umma_commit(smem_u32(&bar_empty[s]));
      }
      if (ok) umma_commit(smem_u32(&bar_acc[q]));
    }
  } else if (warp >= 5) {
    // epilogue: warp w reads the TMEM lanes (tile rows) of its quarter
    const int quarter = warp & 3;
    const int m = quarter * 32 + lane;
    int n = 0;
    for (int t = blockIdx.x; t < a.tiles; t += gridDim.x, ++n) {
      const int q = n & 1;
      bool ready = false;
      // one wait may outlast a failure elsewhere by its own limit only
      if (!s_fail) ready = mbar_wait(smem_u32(&bar_acc[q]), (n >> 1) & 1);
      ready = __all_sync(0xffffffffu, ready);
      if (!ready) {
        if (lane == 0) flag_error(a.err, 3);
        s_fail = 1;
        break;
      }
      tc_fence_after();
      const ImageTile tile = tile_at(t, a.W, a.H, a.bw, a.bh);
      const size_t pix = ((size_t)tile.b * a.H + tile.y0 + m / a.bw) * a.W + tile.x0 + m % a.bw;
      const uint32_t acc = tmem + (uint32_t)(q * NOUT) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
      for (int c0 = 0; c0 < NOUT; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(acc + (uint32_t)c0, r);
        tmem_ld_wait();
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float x = __uint_as_float(r[j]) + (a.bias ? a.bias[c0 + j] : 0.0f);
          v[j] = a.relu ? fmaxf(x, 0.0f) : x;
        }
        if (a.out_f32) {
          float4* o = reinterpret_cast<float4*>(a.out_f32 + pix * NOUT + c0);
#pragma unroll
          for (int j = 0; j < 4; ++j) o[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        if (a.out) {
          uint32_t pk[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
            pk[j] = *reinterpret_cast<uint32_t*>(&h);
          }
          if (a.mask) {
            const uint4* y = reinterpret_cast<const uint4*>(a.mask + pix * NOUT + c0);
            const uint4 y0 = y[0], y1 = y[1];
            const uint32_t yy[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&yy[j]);
              pk[j] &= (__low2float(h) > 0.0f ? 0x0000ffffu : 0u) | (__high2float(h) > 0.0f ? 0xffff0000u : 0u);
            }
          }
          uint4* o = reinterpret_cast<uint4*>(a.out + pix * NOUT + c0);
          o[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          o[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_free[q]));
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::kTmemCols);
  }
}

// the shared memory a kernel opts into, once per context
int opt_in_smem(xc::PerKey<char>& done, const void* kernel, size_t bytes) {
  unsigned long long id = 0;
  XC_TRY(xc_context_id(&id));
  char* set = nullptr;
  return done.get(id, &set, [&](char*) -> int {
    XC_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return XC_OK;
  });
}

template <int KC, int NOUT, bool RES>
int launch_fwd_res(const CUtensorMap& ta, const CUtensorMap& tb, const ConvArgs& a, cudaStream_t s) {
  using Cfg = FwdCfg<KC, NOUT>;
  constexpr uint32_t kMost = 200u * 1024u;
  const uint32_t w = RES ? 9u * a.nkc * Cfg::kBStride : 0u;
  // two CTAs per SM where a ring of at least four steps fits half of its shared memory, and TMEM
  const int per_sm = w + 4u * Cfg::kStage(RES) + 1024u <= kMost / 2 && Cfg::kTmemCols <= 256 ? 2 : 1;
  int stages = (int)((kMost / per_sm - 1024u - w) / Cfg::kStage(RES));
  if (stages > kMaxStages) stages = kMaxStages;
  static xc::PerKey<char> smem;
  XC_TRY(opt_in_smem(smem, (const void*)conv3x3_fwd_kernel<KC, NOUT, RES>, kMost));
  const int grid = a.tiles < per_sm * kNumSMs ? a.tiles : per_sm * kNumSMs;
  xc_launch(conv3x3_fwd_kernel<KC, NOUT, RES>, grid, kFwdThreads, w + stages * Cfg::kStage(RES) + 1024u, s, ta, tb,
            a, stages);
  XC_LAUNCH_CHECK();
  return XC_OK;
}
template <int KC, int NOUT>
int launch_fwd(const CUtensorMap& ta, const CUtensorMap& tb, const ConvArgs& a, cudaStream_t s) {
  // the weights stay where they leave room for a ring of at least four steps
  if (9u * a.nkc * FwdCfg<KC, NOUT>::kBStride <= 100u * 1024u) return launch_fwd_res<KC, NOUT, true>(ta, tb, a, s);
  return launch_fwd_res<KC, NOUT, false>(ta, tb, a, s);
}

template <int KC>
int launch_fwd_n(int Cout, const CUtensorMap& ta, const CUtensorMap& tb, const ConvArgs& a, cudaStream_t s) {
  switch (Cout) {
    case 16: return launch_fwd<KC, 16>(ta, tb, a, s);
    case 32: return launch_fwd<KC, 32>(ta, tb, a, s);
    case 64: return launch_fwd<KC, 64>(ta, tb, a, s);
    case 128: return launch_fwd<KC, 128>(ta, tb, a, s);
    default: xc_set_error("conv3x3: Cout must be 16, 32, 64 or 128 (got %d)", Cout); return XC_BAD_ARG;
  }
}

bool tile_shape(int H, int W, int* bw, int* bh) {
  if (W <= 0 || H <= 0) return false;
  *bw = W >= 128 ? 128 : W;
  if (128 % *bw != 0 || W % *bw != 0) return false;
  *bh = 128 / *bw;
  return H % *bh == 0;
}

// ---------------------------------------------------------------------------
// weight gradient
// ---------------------------------------------------------------------------
// A CTA takes one row of taps (blockIdx.y: dy) over the tiles blockIdx.x,
// + gridDim.x, ...  A step is one tile: the three taps' X tiles, a tile of zeros
// behind them where 128 rows of A reach beyond the third, and dY's tile.  The rows
// of A are 128 / Cin of these tiles at a time (16 and 32 channels: all of them,
// 64: two and two, 128: one by one), so one pass over A serves several taps; rows
// beyond the fourth tile (16 channels) read what lies behind, and no row but
// the taps' is stored.  Operands come in as the forward's pixels do.  It was bound
// by two-byte transposing stores and by nine passes over dY with M mostly zero
// rows: 16 x 16 channels at 8 x 256 x 256 pixels 154 us, with the bias gradient's
// own two kernels 220; now 62 and 3 for the reduction.  What bounds it is the rate
// of the MMAs themselves (eight per tile and CTA, about 110 clocks each; a second
// accumulator for every other tile changes nothing).
struct WgradArgs {
  const __nv_bfloat16* x;    // NHWC [B][H][W][Cin]
  const __nv_bfloat16* dy;   // NHWC [B][H][W][Cout]
  float* partial;            // [gridDim.x][9][Cin][Cout], then [gridDim.x][kBiasWarps][Cout]
  int bias;                  // 1: the bias gradient's partial sums too
  int B, H, W, bw, bh, tiles;
  int* err;
};

constexpr int kBiasWarps = 2;
constexpr int kWgThreads = 160 + 32 * kBiasWarps;   // four loading warps, one issuing, those of the bias gradient
constexpr int kWgMaxStages = 8;

template <int CIN, int COUT>
struct WgCfg {
  static constexpr uint32_t kX = 128u * CIN * 2u, kY = 128u * COUT * 2u;
  static constexpr uint32_t kZeros = CIN == 128 ? 0u : kX;        // the fourth tile of A's rows
  static constexpr uint32_t kStage = 3u * kX + kZeros + kY;
  static constexpr uint32_t kRoom = 200u * 1024u;
  static constexpr int kStages = kRoom / kStage > kWgMaxStages ? kWgMaxStages : (int)(kRoom / kStage);
  // rows beyond the fourth tile (16 channels: four more tiles' worth) stay inside the allocation
  static constexpr uint32_t kTail = CIN == 16 ? 4u * kX : 0u;
  static constexpr uint32_t kSmem = kStages * kStage + kTail + 1024u;
  static constexpr int kSlots = 128 / CIN;                       // tiles per group of A rows
  static constexpr int kGroups = CIN == 16 || CIN == 32 ? 1 : (CIN == 64 ? 2 : 3);
  static constexpr uint32_t kTmemCols = tmem_cols_for(kGroups * COUT);
};

// sum over the 128 pixels of a dY tile by the kBiasWarps warps, thread t of
// them the 8 channels of chunk t % (COUT / 8) of every (32 kBiasWarps / CH)th
// pixel, added to acc
template <int COUT>
__device__ __forceinline__ void bias_add_tile(const uint8_t* tile, int t, float (&acc)[8]) {
  constexpr int CH = COUT / 8, STEP = 32 * kBiasWarps / CH, KY = COUT < 64 ? COUT : 64;
  constexpr uint32_t RB = KY * 2u;
  const int c = t % CH;
  const uint8_t* part = tile + (uint32_t)(c / (KY / 8)) * 128u * RB;
  float sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int m = t / CH; m < 128; m += STEP) {
    const uint4 q = *reinterpret_cast<const uint4*>(part + swz_chunk<RB>((uint32_t)m, (uint32_t)(c % (KY / 8))));
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sum[2 * j] += __uint_as_float(w[j] << 16);
      sum[2 * j + 1] += __uint_as_float(w[j] & 0xffff0000u);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] += sum[j];
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(kWgThreads, 1) conv3x3_wgrad_kernel(const __grid_constant__ CUtensorMap tmX,
                                                                      const __grid_constant__ CUtensorMap tmY,
                                                                      WgradArgs a) {
  using Cfg = WgCfg<CIN, COUT>;
  constexpr bool TX = CIN >= 64, TY = COUT >= 64;                                // by TMA
  constexpr int KX = CIN < 64 ? CIN : 64, KY = COUT < 64 ? COUT : 64;            // channels per row
  constexpr uint32_t RBX = KX * 2u, RBY = KY * 2u;
  constexpr uint32_t LX = layout_for_row_bytes(RBX), LY = layout_for_row_bytes(RBY);
  constexpr uint32_t TILEX = 128u * RBX, TILEY = 128u * RBY;                      // 128 pixels of one row width
  constexpr uint32_t IDESC = idesc_bf16(128, COUT, 1);
  constexpr int NS = Cfg::kStages;
  extern __shared__ uint8_t dsm[];
  __shared__ __align__(8) uint64_t bar_full[NS], bar_empty[NS], bar_done;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int s_fail;
  const uint32_t base = (smem_u32(dsm) + 1023u) & ~1023u;
  uint8_t* gbase = dsm + (base - smem_u32(dsm));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int dy = (int)blockIdx.y - 1;

  // The bias gradient's own warps in one row of CTAs: added in FP32, a tile's
  // sum apart from the running one.  As a row of ones in the MMAs it comes at no
  // cost, but the tensor core truncates its running sum: up to 2e-5 of sum |dY|
  // off (4 x 512^2 pixels), here up to 1.2e-7, in launches of its own 6e-7.  U-Net
  // gradient at 8 x 256^2 with ones 1181 us, two warps 1187, one 1210, four 1209.
  const bool bias = a.bias != 0 && dy == 0;

  for (int s = 0; s < NS; ++s)
    for (uint32_t o = tid * 16u; o < Cfg::kZeros; o += kWgThreads * 16u)
      *reinterpret_cast<uint4*>(gbase + s * Cfg::kStage + 3u * Cfg::kX + o) = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(smem_u32(&bar_full[s]), (TX && TY ? 0 : 128) + (TX || TY ? 1 : 0));
      mbar_init(smem_u32(&bar_empty[s]), bias ? 1 + kBiasWarps : 1);
    }
    mbar_init(smem_u32(&bar_done), 1);
    s_fail = 0;
    mbar_fence_init();
  }
  if (warp == 4) {
    tmem_alloc(smem_u32(&tmem_slot), Cfg::kTmemCols);
    tmem_relinquish();
  }
  fence_async_shared();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  XC_PDL_WAIT();

  if (warp < 4) {
    const PixelCopies<TX ? 16 : KX> px(tid, a.W, a.bw);
    const PixelCopies<TY ? 16 : KY> py(tid, a.W, a.bw);
    int it = 0;
    if (!(TX && TY) || tid == 0)
      for (int t = blockIdx.x; t < a.tiles; t += gridDim.x, ++it) {
        const int s = it % NS;
        if (it >= NS && !mbar_wait(smem_u32(&bar_empty[s]), ((it / NS) - 1) & 1)) {
          flag_error(a.err, 8);
          s_fail = 1;
          break;
        }
        const ImageTile tile = tile_at(t, a.W, a.H, a.bw, a.bh);
        const uint32_t sx = base + s * Cfg::kStage, sy = sx + 3u * Cfg::kX + Cfg::kZeros, full = smem_u32(&bar_full[s]);
        if (tid == 0 && (TX || TY)) {
          mbar_expect_tx(full, (TX ? 3u * Cfg::kX : 0u) + (TY ? Cfg::kY : 0u));
          if (TX) {
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
              for (int c = 0; c < CIN; c += 64)
                tma_load_4d(sx + j * Cfg::kX + (c / 64) * TILEX, &tmX, c, tile.x0 + j - 1, tile.y0 + dy, tile.b, full);
          }
          if (TY) {
#pragma unroll
            for (int c = 0; c < COUT; c += 64) tma_load_4d(sy + (c / 64) * TILEY, &tmY, c, tile.x0, tile.y0, tile.b, full);
          }
        }
        if constexpr (!(TX && TY)) {
          if constexpr (!TX) px.template load<3>(sx, a.x, a.H, a.W, tile, dy, -1);
          if constexpr (!TY) py.template load<1>(sy, a.dy, a.H, a.W, tile, 0, 0);
          cp_async_arrive(full);
        }
      }
    if constexpr (!(TX && TY)) cp_async_wait_all();
    // TMA loads still in flight (only after a wait ran out) end before the CTA does
    if (tid == 0 && (TX || TY))
      for (int q = it - NS > 0 ? it - NS : 0; q < it; ++q) mbar_wait(smem_u32(&bar_full[q % NS]), (q / NS) & 1);
  } else if (warp >= 5) {
    if (bias) {
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      bool ok = true;
      int it = 0;
      for (int t = blockIdx.x; t < a.tiles; t += gridDim.x, ++it) {
        const int s = it % NS;
        ok = true;
        if (lane == 0) ok = mbar_wait(smem_u32(&bar_full[s]), (it / NS) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) flag_error(a.err, 11);
          s_fail = 1;
          break;
        }
        bias_add_tile<COUT>(gbase + s * Cfg::kStage + 3u * Cfg::kX + Cfg::kZeros, tid - 160, acc);
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_empty[s]));
      }
      constexpr int CH = COUT / 8;
#pragma unroll
      for (int o = CH; o < 32; o <<= 1)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
      float* dst = a.partial + (size_t)gridDim.x * 9 * CIN * COUT + ((size_t)blockIdx.x * kBiasWarps + (warp - 5)) * COUT;
      if (ok && lane < CH)
#pragma unroll
        for (int j = 0; j < 8; ++j) dst[lane * 8 + j] = acc[j];
    }
  } else if (lane == 0) {
    int it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < a.tiles; t += gridDim.x, ++it) {
      const int s = it % NS;
      if (!mbar_wait(smem_u32(&bar_full[s]), (it / NS) & 1)) {
        flag_error(a.err, 10);
        s_fail = 1;
        ok = false;
        break;
      }
      if (!(TX && TY)) fence_async_shared();
      tc_fence_after();
      const uint32_t sx = base + s * Cfg::kStage, sy = sx + 3u * Cfg::kX + Cfg::kZeros;
#pragma unroll
      for (int g = 0; g < Cfg::kGroups; ++g)
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16(tmem + (uint32_t)(g * COUT),
                    smem_desc_mn(sx + g * Cfg::kSlots * Cfg::kX + k * 16 * RBX, TILEX, 8u * RBX, LX),
                    smem_desc_mn(sy + k * 16 * RBY, TILEY, 8u * RBY, LY), IDESC, (it | k) != 0 ? 1u : 0u);
      umma_commit(smem_u32(&bar_empty[s]));
    }
    if (ok) umma_commit(smem_u32(&bar_done));
  }
  __syncwarp();
  __syncthreads();      // loaders and issuer are through (each of their waits is bounded)
  bool ready = false;
  if (!s_fail) ready = mbar_wait(smem_u32(&bar_done), 0);
  ready = __syncthreads_and(ready);
  if (!ready && tid == 0) flag_error(a.err, 4);
  tc_fence_after();
  if (ready && warp < 4) {
    // TMEM lane = (tile of the group, input channel), column = output channel
    const int m = warp * 32 + lane;
#pragma unroll
    for (int g = 0; g < Cfg::kGroups; ++g) {
      const int slot = g * Cfg::kSlots + m / CIN;              // 0..2 taps
      const bool live = slot < 3;
      float* dst = a.partial + (((size_t)blockIdx.x * 9 + 3 * blockIdx.y + (live ? slot : 0)) * CIN + m % CIN) * COUT;
#pragma unroll
      for (int c0 = 0; c0 < COUT; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(g * COUT + c0), r);
        tmem_ld_wait();
        if (live) {
          float4* o = reinterpret_cast<float4*>(dst + c0);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            o[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]),
                               __uint_as_float(r[4 * j + 3]));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::kTmemCols);
  }
}

// dW = sum over CTAs of the partials in a fixed order (eight threads per value
// add every eighth CTA's, one adds the eight), transposed to [Cout][9][Cin],
// scaled, optionally accumulated; db (may be null) likewise from the bias
// partials
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float* __restrict__ partial, int nblk, int Cin,
                                                           int Cout, float* dw, float scale, int accumulate,
                                                           float* db) {
  XC_PDL_WAIT();
  __shared__ float sh[8][32];
  const int n = 9 * Cin * Cout;
  const int q = threadIdx.x >> 5, i = blockIdx.x * 32 + (threadIdx.x & 31);
  float v = 0.0f;
  if (i < n || (db && i < n + Cout)) {
    const float* p = i < n ? partial + i : partial + (size_t)nblk * n + (i - n);
    const size_t st = i < n ? n : Cout;
    const int nb = i < n ? nblk : nblk * kBiasWarps;
#pragma unroll 4
    for (int k = q; k < nb; k += 8) v += p[(size_t)k * st];
  }
  sh[q][threadIdx.x & 31] = v;
  __syncthreads();
  if (q != 0 || i >= n + Cout || (i >= n && !db)) return;
  const int l = threadIdx.x;
  v = ((sh[0][l] + sh[1][l]) + (sh[2][l] + sh[3][l])) + ((sh[4][l] + sh[5][l]) + (sh[6][l] + sh[7][l]));
  if (i < n) {
    const int co = i % Cout, ci = (i / Cout) % Cin, t = i / (Cout * Cin);
    float* d = dw + ((size_t)co * 9 + t) * Cin + ci;
    *d = accumulate ? *d + scale * v : scale * v;
  } else {
    db[i - n] = accumulate ? db[i - n] + scale * v : scale * v;
  }
}

template <int CIN, int COUT>
int launch_wgrad(const CUtensorMap& tx, const CUtensorMap& ty, const WgradArgs& a, int nx, cudaStream_t s) {
  using Cfg = WgCfg<CIN, COUT>;
  static xc::PerKey<char> smem;
  XC_TRY(opt_in_smem(smem, (const void*)conv3x3_wgrad_kernel<CIN, COUT>, Cfg::kSmem));
  xc_launch(conv3x3_wgrad_kernel<CIN, COUT>, dim3(nx, 3), kWgThreads, Cfg::kSmem, s, tx, ty, a);
  XC_LAUNCH_CHECK();
  return XC_OK;
}
template <int CIN>
int launch_wgrad_n(int Cout, const CUtensorMap& tx, const CUtensorMap& ty, const WgradArgs& a, int nx,
                   cudaStream_t s) {
  switch (Cout) {
    case 16: return launch_wgrad<CIN, 16>(tx, ty, a, nx, s);
    case 32: return launch_wgrad<CIN, 32>(tx, ty, a, nx, s);
    case 64: return launch_wgrad<CIN, 64>(tx, ty, a, nx, s);
    default: return launch_wgrad<CIN, 128>(tx, ty, a, nx, s);
  }
}

// CTAs along the tiles, times three rows of taps.  They set how many sums the
// tensor core chains in FP32, so with 34, the number before this kernel, the
// gradients keep their digits (3e-7).  More CTAs are nearer to 64 bits and, up to
// 50 (as many SMs as there are), faster: 16 x 16 channels at 8 x 256^2 pixels with
// 34, 50 and 152 are 1.7e-5, 1.2e-5 and 3.6e-6 of the gradient's norm off, a call
// takes 80, 62 and 66 us, the U-Net gradient there 1181, 1091 and 1178 us; 128 x
// 128 channels at 8 x 32^2 lose (37, 40 and 165 us).
constexpr int kWgBlocks = 34;

}  // namespace

// ---------------------------------------------------------------------------
// internal entry points (xc_nn.cuh)
// ---------------------------------------------------------------------------
int nn_conv3x3_fwd(const void* x, const void* w, const float* bias, void* y, float* y_f32, int B, int H, int W,
                   int Cin, int Cout, int relu, int* err, cudaStream_t s, const void* mask) {
  int bw = 0, bh = 0;
  if (!tile_shape(H, W, &bw, &bh) || B < 1) {
    xc_set_error("conv3x3: image %dx%d does not tile into 128-pixel tiles (W a multiple of 128, or a power of two "
                 "below it dividing H's tiling)", H, W);
    return XC_BAD_ARG;
  }
  if (Cin != 16 && Cin != 32 && Cin != 64 && Cin != 128) {
    xc_set_error("conv3x3: Cin must be 16, 32, 64 or 128 (got %d)", Cin);
    return XC_BAD_ARG;
  }
  if (!y && !y_f32) { xc_set_error("conv3x3: no output"); return XC_BAD_ARG; }
  const int kc = Cin >= 64 ? 64 : Cin;
  if (((uintptr_t)x & 15u) != 0) { xc_set_error("conv3x3: activation pointer not 16-byte aligned"); return XC_BAD_ARG; }
  CUtensorMap ta, tb;
  std::memset(&ta, 0, sizeof(ta));
  if (kc == 64) XC_TRY(make_act_map(&ta, x, B, H, W, Cin, bw, bh));
  XC_TRY(make_weight_map(&tb, w, Cin, Cout, kc));
  const int tiles = B * (H / bh) * (W / bw);
  ConvArgs a{B, H, W, Cin, Cin / kc, bw, bh, (const __nv_bfloat16*)x, bias, relu, (const __nv_bfloat16*)mask, tiles, (__nv_bfloat16*)y, y_f32,
             err};
  switch (kc) {
    case 16: return launch_fwd_n<16>(Cout, ta, tb, a, s);
    case 32: return launch_fwd_n<32>(Cout, ta, tb, a, s);
    default: return launch_fwd_n<64>(Cout, ta, tb, a, s);
  }
}

long long nn_wgrad_scratch(int B, int H, int W, int Cin, int Cout) {
  return std::min<long long>((long long)B * H * W / 128, kWgBlocks) * (9 * Cin + kBiasWarps) * Cout;
}

int nn_conv3x3_wgrad(const void* x, const void* dy, float* dw, float* db, float* partial, int B, int H, int W,
                     int Cin, int Cout, float scale, int accumulate, int* err, cudaStream_t s) {
  int bw = 0, bh = 0;
  if (!tile_shape(H, W, &bw, &bh) || B < 1) {
    xc_set_error("conv3x3 wgrad: image %dx%d does not tile into 128-pixel tiles", H, W);
    return XC_BAD_ARG;
  }
  if ((Cout != 16 && Cout != 32 && Cout != 64 && Cout != 128) ||
      (Cin != 16 && Cin != 32 && Cin != 64 && Cin != 128)) {
    xc_set_error("conv3x3 wgrad: channels must be 16, 32, 64 or 128 (Cin %d, Cout %d)", Cin, Cout);
    return XC_BAD_ARG;
  }
  if ((((uintptr_t)x | (uintptr_t)dy) & 15u) != 0) {
    xc_set_error("conv3x3 wgrad: activation pointer not 16-byte aligned");
    return XC_BAD_ARG;
  }
  const int tiles = B * (H / bh) * (W / bw);
  const int nx = tiles < kWgBlocks ? tiles : kWgBlocks;
  CUtensorMap tx, ty;
  std::memset(&tx, 0, sizeof(tx));
  std::memset(&ty, 0, sizeof(ty));
  if (Cin >= 64) XC_TRY(make_act_map(&tx, x, B, H, W, Cin, bw, bh));
  if (Cout >= 64) XC_TRY(make_act_map(&ty, dy, B, H, W, Cout, bw, bh));
  WgradArgs a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, partial, db ? 1 : 0, B, H, W, bw, bh, tiles, err};
  switch (Cin) {
    case 16: XC_TRY(launch_wgrad_n<16>(Cout, tx, ty, a, nx, s)); break;
    case 32: XC_TRY(launch_wgrad_n<32>(Cout, tx, ty, a, nx, s)); break;
    case 64: XC_TRY(launch_wgrad_n<64>(Cout, tx, ty, a, nx, s)); break;
    default: XC_TRY(launch_wgrad_n<128>(Cout, tx, ty, a, nx, s)); break;
  }
  const int n = 9 * Cout * Cin + Cout;
  xc_launch(wgrad_reduce_kernel, (n + 31) / 32, 256, 0, s, (const float*)partial, nx, Cin, Cout, dw, scale,
            accumulate, db);
  XC_LAUNCH_CHECK();
  return XC_OK;
}

// Error flags of the kernels' bounded waits: ints of one page of pinned host
// memory per context, taken for the length of a call (or of a network's life).
// Nothing is allocated, cleared or copied per call: a kernel writes its flag only
// when a wait ran out, and the host reads it after it has waited for the stream.
// A page is allocated on first use and kept; with all kFlagSlots taken a flag is
// allocated for itself.
namespace {
constexpr int kFlagSlots = 256;
struct FlagPage {
  int* host = nullptr;
  bool used[kFlagSlots] = {};
};
std::mutex g_flag_mu;                                       // of the pages' `used`
auto& g_flag_pages = *new xc::PerKey<FlagPage>();           // (outlives every flag)
}  // namespace

int ErrFlag::init() {
  unsigned long long id = 0;
  XC_TRY(xc_context_id(&id));
  FlagPage* p = nullptr;
  XC_TRY(g_flag_pages.get(id, &p, [](FlagPage* f) -> int {
    XC_CUDA_TRY(cudaHostAlloc((void**)&f->host, sizeof(int) * kFlagSlots, cudaHostAllocMapped));
    return XC_OK;
  }));
  {
    std::lock_guard<std::mutex> lock(g_flag_mu);
    for (int q = 0; q < kFlagSlots && !used; ++q)
      if (!p->used[q]) {
        used = &p->used[q];
        *used = true;
        host = p->host + q;
      }
  }
  if (!used) XC_CUDA_TRY(cudaHostAlloc((void**)&host, sizeof(int), cudaHostAllocMapped));
  *host = 0;
  XC_CUDA_TRY(cudaHostGetDevicePointer((void**)&dev, host, 0));
  return XC_OK;
}
int ErrFlag::check(cudaStream_t s, const char* what) {
  XC_CUDA_TRY(cudaStreamSynchronize(s));
  const int h = *(volatile int*)host;
  if (h != 0) {
    xc_set_error("%s: a bounded wait inside a convolution kernel ran out (code %d)", what, h);
    return XC_TIMEOUT;
  }
  return XC_OK;
}
ErrFlag::~ErrFlag() {
  if (used) {
    std::lock_guard<std::mutex> lock(g_flag_mu);
    *used = false;
  } else if (host) {
    cudaFreeHost(host);
  }
}

namespace {
// stream-ordered scratch of one call from a pool that keeps up to 32 MB (with
// the default pool every call that waits for its stream gives the memory back
// to the system and maps it again)
int scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  static xc::PerKey<cudaMemPool_t> pools;
  unsigned long long id = 0;
  XC_TRY(xc_context_id(&id));
  cudaMemPool_t* pool = nullptr;
  XC_TRY(pools.get(id, &pool, [](cudaMemPool_t* q) -> int {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    XC_CUDA_TRY(cudaGetDevice(&props.location.id));
    XC_CUDA_TRY(cudaMemPoolCreate(q, &props));
    unsigned long long keep = 32ull << 20;
    cudaMemPoolSetAttribute(*q, cudaMemPoolAttrReleaseThreshold, &keep);
    return XC_OK;
  }));
  XC_CUDA_TRY(cudaMallocFromPoolAsync(p, bytes, *pool, s));
  return XC_OK;
}
}  // namespace

extern "C" int xc_nn_conv3x3(const void* x, const void* w, const float* bias, void* y, float* y_f32, int B, int H,
                             int W, int Cin, int Cout, int relu, void* stream) {
  if (!x || !w) { xc_set_error("xc_nn_conv3x3: null pointer"); return XC_BAD_ARG; }
  cudaStream_t s = (cudaStream_t)stream;
  ErrFlag e;
  XC_TRY(e.init());
  const int st = nn_conv3x3_fwd(x, w, bias, y, y_f32, B, H, W, Cin, Cout, relu, e.dev, s);
  if (st == XC_BAD_ARG) return st;          // nothing was launched
  const int ck = e.check(s, "xc_nn_conv3x3");
  return st != XC_OK ? st : ck;
}

extern "C" int xc_nn_conv3x3_wgrad(const void* x, const void* dy, float* dw, int B, int H, int W, int Cin,
                                   int Cout, void* stream) {
  if (!x || !dy || !dw) { xc_set_error("xc_nn_conv3x3_wgrad: null pointer"); return XC_BAD_ARG; }
  cudaStream_t s = (cudaStream_t)stream;
  ErrFlag e;
  XC_TRY(e.init());
  float* partial = nullptr;
  if (Cin >= 16 && Cin <= 128 && Cout >= 16 && Cout <= 128 && B > 0 && H > 0 && W > 0)
    XC_TRY(scratch_alloc((void**)&partial, sizeof(float) * (size_t)nn_wgrad_scratch(B, H, W, Cin, Cout), s));
  const int st = nn_conv3x3_wgrad(x, dy, dw, nullptr, partial, B, H, W, Cin, Cout, 1.0f, 0, e.dev, s);
  if (partial) cudaFreeAsync(partial, s);
  if (st == XC_BAD_ARG) return st;
  const int ck = e.check(s, "xc_nn_conv3x3_wgrad");
  return st != XC_OK ? st : ck;
}
