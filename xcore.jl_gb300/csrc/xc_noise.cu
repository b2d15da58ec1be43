// noise! on the GPU: Ornstein-Uhlenbeck update, FFT Gaussian filter,
// re-standardisation, staggered differences, tapers and speed magnitudes.
//
// Reference: src/noise.jl:138-270 (and the NoiseState precompute 61-107).
//
// The filter.  compute_fft_filter (noise.jl:244-270) zero-pads psi by `pad`
// rows, applies exp(-s^2 (kz^2 + kx^2)) in 2-D Fourier space and unpads.  That
// spectrum is a product exp(-s^2 kz^2) * exp(-s^2 kx^2), so the operator is a
// z-direction circular convolution (period Nz+pad) followed by an x-direction
// circular convolution (period Nx), each with a real, even kernel c[d].  Only
// the Nz unpadded rows are kept and the input is zero outside them, so the
// z-pass is a linear convolution of the Nz-long column with c over lags
// |d| < Nz; it is evaluated exactly with a power-of-two FFT of length
// M >= 2 Nz - 1 (no wrap-around can reach the kept rows).  The x-pass uses a
// length-Nx FFT directly when Nx is a power of two (then the multiplier IS the
// reference's exp(-s^2 kx^2)), otherwise the same linear-convolution form.
// Two real lines are packed into one complex FFT (real kernel => the real and
// imaginary parts stay separate).  Mathematically this is the reference
// operator; the FFTs are hand-written radix-2 shared-memory transforms.
//
// Where the filter is well resolved its kernel is short: for s >= 2 h the
// spectrum falls below 2^-56 before the Nyquist wavenumber, so c[d] is the
// Gaussian exp(-(d h / 2 s)^2) itself (to that accuracy), and beyond R = 24
// (s = 2 h, the correlation length of three cells of every configuration) all
// its values together are below 2^-54 of its sum.  Both passes are then direct
// sums of 2 R + 1 terms: 49 FP64 instructions per cell and pass on a
// processor bound by its FP64 unit, against 60 (x, power of two) and 90 (z) of
// the FFTs, and up to three times that where the padding to a power of two
// doubles a line (a pass of 1024^2 in 94 us instead of 228 and 124, one of
// 300 x 231 in 7 instead of 105).  Longer kernels (R > 32) and unresolved ones take the FFT.
#include <cmath>
#include <complex>
#include <mutex>
#include <vector>

#include "xc_internal.cuh"

namespace {

bool is_pow2(int n) { return n > 0 && (n & (n - 1)) == 0; }
int next_pow2(int n) { int m = 1; while (m < n) m <<= 1; return m; }

// host radix-2 FFT (precompute only)
void host_fft(std::vector<std::complex<double>>& a) {
  const int n = (int)a.size();
  for (int i = 1, j = 0; i < n; ++i) {
    int bit = n >> 1;
    for (; j & bit; bit >>= 1) j ^= bit;
    j ^= bit;
    if (i < j) std::swap(a[i], a[j]);
  }
  for (int len = 2; len <= n; len <<= 1) {
    for (int k = 0; k < len / 2; ++k) {
      double ang = -2.0 * M_PI * (double)k / (double)len;
      std::complex<double> w(std::cos(ang), std::sin(ang));
      for (int i = 0; i < n; i += len) {
        std::complex<double> u = a[i + k], v = a[i + k + len / 2] * w;
        a[i + k] = u + v;
        a[i + k + len / 2] = u - v;
      }
    }
  }
}

// wavenumbers 2*pi*fftfreq(n, 1/h) (noise.jl:100-101, AbstractFFTs arithmetic)
std::vector<double> wavenumbers(int n, double h) {
  std::vector<double> k(n);
  int nn = (n + 1) >> 1;
  double mult = 2.0 * M_PI * ((1.0 / h) / (double)n);
  for (int i = 0; i < n; ++i) k[i] = (double)(i < nn ? i : i - n) * mult;
  return k;
}

}  // namespace

struct LineFilter {      // one 1-D convolution pass
  int L;                 // line length (input and output)
  int M;                 // FFT length
  int logM;
  double* khat;          // device, M real multipliers (already divided by M)
  double2* tw;           // device, M/2 twiddles exp(-2 pi i k / M)
};

constexpr int kMaxRadius = 32;
struct DirectFilter {    // one 1-D convolution pass as a direct sum
  int R;                 // largest lag (0: none, the FFT serves this pass)
  int period;            // lags wrap around at this length; cells beyond the line's end are zero
  double tap[kMaxRadius + 1];
};

struct NoisePlan {
  int padL0, padl0;
  double fL, fl;
  LineFilter ze, xe, zs, xs;   // e: sigma = L0h, pad = padL0; s: sigma = l0h, pad = padl0
  DirectFilter dz[2], dx[2];   // e, s
  bool direct;                 // all four passes are short: no FFT plans are built
};

namespace {

int build_line_filter(LineFilter& lf, int L, int period, double h, double sigma, bool direct_ok) {
  std::vector<double> kk = wavenumbers(period, h);
  std::vector<double> G(period);
  for (int k = 0; k < period; ++k) G[k] = std::exp(-(sigma * sigma) * (kk[k] * kk[k]));
  std::vector<double> khat;
  if (direct_ok && period == L && is_pow2(L)) {
    lf.M = L;
    khat = G;
  } else {
    lf.M = next_pow2(2 * L - 1);
    // circular kernel c[d] = (1/n) sum_k G(k) cos(2 pi k d / n), real and even
    std::vector<double> cd(L);
    for (int d = 0; d < L; ++d) {
      long double acc = 0.0L;
      for (int k = 0; k < period; ++k) {
        long long kd = ((long long)k * d) % period;
        acc += (long double)G[k] * std::cos(2.0L * (long double)M_PI * (long double)kd / (long double)period);
      }
      cd[d] = (double)(acc / (long double)period);
    }
    std::vector<std::complex<double>> kb(lf.M, 0.0);
    for (int d = 0; d < L; ++d) kb[d] = cd[d % period];
    for (int d = 1; d < L; ++d) kb[lf.M - d] = cd[d % period];
    host_fft(kb);
    khat.resize(lf.M);
    for (int k = 0; k < lf.M; ++k) khat[k] = kb[k].real();
  }
  lf.L = L;
  lf.logM = 0;
  while ((1 << lf.logM) < lf.M) ++lf.logM;
  for (auto& v : khat) v /= (double)lf.M;       // fold the inverse transform's 1/M
  std::vector<double2> tw(lf.M / 2 > 0 ? lf.M / 2 : 1);
  for (int k = 0; k < lf.M / 2; ++k) {
    long double ang = -2.0L * (long double)M_PI * (long double)k / (long double)lf.M;
    tw[k] = make_double2((double)std::cos(ang), (double)std::sin(ang));
  }
  XC_CUDA_TRY(cudaMalloc(&lf.khat, sizeof(double) * lf.M));
  XC_CUDA_TRY(cudaMalloc(&lf.tw, sizeof(double2) * tw.size()));
  XC_CUDA_TRY(cudaMemcpy(lf.khat, khat.data(), sizeof(double) * lf.M, cudaMemcpyHostToDevice));
  XC_CUDA_TRY(cudaMemcpy(lf.tw, tw.data(), sizeof(double2) * tw.size(), cudaMemcpyHostToDevice));
  return XC_OK;
}

// the direct form of a pass over lines of period n, or R = 0
void build_direct(DirectFilter& f, int n, double h, double sigma) {
  f.R = 0;
  f.period = n;
  const double s = sigma / h;
  if (!(s >= 1.99 && s <= 4.0)) return;
  auto gauss = [&](int d) { return std::exp(-(double)d * d / (4.0 * s * s)) / (2.0 * s * std::sqrt(M_PI)); };
  int R = 1;
  for (; R <= kMaxRadius; ++R) {
    double tail = 0.0;
    for (int d = R + 1; d < R + 64; ++d) tail += 2.0 * gauss(d);
    if (tail <= 0x1p-54) break;
  }
  if (R > kMaxRadius || 2 * R + 1 > n) return;
  f.R = R;
  for (int d = 0; d <= R; ++d) f.tap[d] = gauss(d);
}

void free_line_filter(LineFilter& lf) {
  if (lf.khat) cudaFree(lf.khat);
  if (lf.tw) cudaFree(lf.tw);
  lf.khat = nullptr;
  lf.tw = nullptr;
}

// complex product with two of its four products fused into FMAs (four FP64
// instructions instead of six; this file is otherwise compiled without FMA
// contraction, and the FFT's results are a different rounding of the
// reference's FFTW transform in any case)
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(__fma_rn(a.x, b.x, -(a.y * b.y)), __fma_rn(a.x, b.y, a.y * b.x));
}

// in-place radix-2 DIT FFT of P transforms of length M stored back to back in
// shared memory (input in bit-reversed order); inverse = conjugated twiddles
__device__ void smem_fft(double2* buf, int P, int M, int logM, const double2* __restrict__ tw,
                         bool inverse) {
  const int nb = P * (M >> 1);
  for (int s = 1; s <= logM; ++s) {
    const int half = 1 << (s - 1);
    const int stride = M >> s;       // twiddle index step
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
      int t = b / (M >> 1), r = b % (M >> 1);
      int grp = r / half, k = r % half;
      int i0 = t * M + grp * 2 * half + k;
      double2 w = tw[k * stride];
      if (inverse) w.y = -w.y;
      double2 u = buf[i0], v = cmul(buf[i0 + half], w);
      buf[i0] = make_double2(u.x + v.x, u.y + v.y);
      buf[i0 + half] = make_double2(u.x - v.x, u.y - v.y);
    }
    __syncthreads();
  }
}

__device__ __forceinline__ int bitrev(int i, int logM) { return __brev(i) >> (32 - logM); }

// Filter lines of a column-major (rows x cols) array along `axis` (0: lines
// are columns of length rows; 1: lines are rows of length cols).  Each CTA
// takes P line pairs.  in and out may not alias.
__global__ void line_filter_kernel(CView in, DView out, int rows, int cols, int axis, int M,
                                   int logM, const double* __restrict__ khat,
                                   const double2* __restrict__ tw, int P) {
  XC_PDL_WAIT();
  extern __shared__ double2 buf[];
  const int L = axis == 0 ? rows : cols;
  const int nlines = axis == 0 ? cols : rows;
  const int pair0 = blockIdx.x * P;
  // load: line pair (2q, 2q+1) -> complex, bit-reversed positions
  for (int e = threadIdx.x; e < P * M; e += blockDim.x) {
    int t = e / M, k = e % M;
    int la = 2 * (pair0 + t), lb = la + 1;
    double re = 0.0, im = 0.0;
    if (k < L) {
      if (axis == 0) {
        if (la < nlines) re = AT(in, k, la);
        if (lb < nlines) im = AT(in, k, lb);
      } else {
        if (la < nlines) re = AT(in, la, k);
        if (lb < nlines) im = AT(in, lb, k);
      }
    }
    buf[t * M + bitrev(k, logM)] = make_double2(re, im);
  }
  __syncthreads();
  smem_fft(buf, P, M, logM, tw, false);
  // multiply by the real spectrum, then bit-reverse in place for the inverse
  for (int e = threadIdx.x; e < P * M; e += blockDim.x) {
    int k = e % M;
    double g = khat[k];
    buf[e].x *= g;
    buf[e].y *= g;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < P * M; e += blockDim.x) {
    int t = e / M, k = e % M, r = bitrev(k, logM);
    if (k < r) {
      double2 a = buf[t * M + k];
      buf[t * M + k] = buf[t * M + r];
      buf[t * M + r] = a;
    }
  }
  __syncthreads();
  smem_fft(buf, P, M, logM, tw, true);
  for (int e = threadIdx.x; e < P * L; e += blockDim.x) {
    int t = e / L, k = e % L;
    int la = 2 * (pair0 + t), lb = la + 1;
    double2 v = buf[t * M + k];
    if (axis == 0) {
      if (la < nlines) AT(out, k, la) = v.x;
      if (lb < nlines) AT(out, k, lb) = v.y;
    } else {
      if (la < nlines) AT(out, la, k) = v.x;
      if (lb < nlines) AT(out, lb, k) = v.y;
    }
  }
}

int run_line_filter(const LineFilter& lf, CView in, DView out, int rows, int cols, int axis,
                    cudaStream_t s) {
  const int nlines = axis == 0 ? cols : rows;
  const int npairs = (nlines + 1) / 2;
  int P = 1;
  while (P * 2 * lf.M * (int)sizeof(double2) <= 64 * 1024 && P * 2 <= 8) P *= 2;
  size_t smem = (size_t)P * lf.M * sizeof(double2);
  if (smem > 48 * 1024) {
    // set to the largest need seen so far, never lowered: a graph may hold
    // launches of several filter lengths, captured in any order
    static std::mutex mu;
    static size_t limit = 0;
    std::lock_guard<std::mutex> lock(mu);
    if (smem > limit) limit = smem;
    XC_CUDA_TRY(cudaFuncSetAttribute(line_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
  }
  int threads = lf.M * P >= 1024 ? 512 : 256;
  xc_launch(line_filter_kernel, (npairs + P - 1) / P, threads, smem, s, in, out, rows, cols, axis, lf.M,
                                                                 lf.logM, lf.khat, lf.tw, P);
  XC_LAUNCH_CHECK();
  return XC_OK;
}

// Direct passes over the three noise fields side by side (blockIdx.z), an
// output per thread: a tile of 64 x 4 cells along z or 32 x 8 across x, with
// its 2 R neighbours on the line in shared memory.  The FP64 unit bounds it
// (2 R + 1 instructions of 64 cycles a warp and sub-partition); the tile's
// repeated reads come from L2.
struct DirectPass {
  CView in[3];
  DView out[3];
  DirectFilter f[2];       // of fields 0, 1 and of field 2
};
template <int AXIS>
__global__ void __launch_bounds__(256) direct_filter_kernel(const __grid_constant__ DirectPass p, int Nz, int Nx) {
  XC_PDL_WAIT();
  constexpr int BZ = AXIS == 0 ? 64 : 32, BX = AXIS == 0 ? 4 : 8;
  constexpr int LZ = AXIS == 0 ? BZ + 2 * kMaxRadius : BZ, LX = AXIS == 0 ? BX : BX + 2 * kMaxRadius;
  __shared__ double x[LX][LZ];
  const DirectFilter& f = p.f[blockIdx.z == 2 ? 1 : 0];
  const CView in = p.in[blockIdx.z];
  const int R = f.R, n = f.period;
  const int j0 = blockIdx.x * BZ, i0 = blockIdx.y * BX;
  const int nz = AXIS == 0 ? BZ + 2 * R : BZ, nx = AXIS == 0 ? BX : BX + 2 * R;
  for (int k = threadIdx.x; k < nz * nx; k += 256) {
    const int ii = k / nz, jj = k - ii * nz;
    int j = j0 + jj - (AXIS == 0 ? R : 0), i = i0 + ii - (AXIS == 1 ? R : 0);
    int& q = AXIS == 0 ? j : i;
    if (q < 0) q += n;
    else if (q >= n) q -= n;               // beyond n + R only in front of cells outside the grid
    x[ii][jj] = j < Nz && i < Nx ? AT(in, j, i) : 0.0;
  }
  __syncthreads();
  const int jj = threadIdx.x % BZ, ii = threadIdx.x / BZ, j = j0 + jj, i = i0 + ii;
  if (j >= Nz || i >= Nx) return;
  const double* c = AXIS == 0 ? &x[ii][jj + R] : &x[ii + R][jj];
  constexpr int st = AXIS == 0 ? 1 : LZ;
  double acc = 0.0;                        // from the smallest terms inwards
#pragma unroll 4
  for (int d = R; d > 0; --d) acc = __fma_rn(f.tap[d], c[-d * st] + c[d * st], acc);
  AT(p.out[blockIdx.z], j, i) = __fma_rn(f.tap[0], c[0], acc);
}

// OU update (noise.jl:160-183), one thread per cell
__global__ void ou_kernel(int Nz, int Nx, double Xi, double L0h, double i2L0h, double i2l0h, double txi0,
                          double dt, double cdt, double fL, double fl, CView V, CView vx, CView fReL, CView ke, CView chi,
                          CView ks, CView psieo, CView psixo, CView psiso, CView re, CView rs,
                          DView psie, DView psix, DView psis) {
  XC_PDL_WAIT();
  for_tiles(Nz, Nx, [&](int j, int i) {
    if (j >= Nz || i >= Nx) return;
    // The reference's twelve divisions (noise.jl:160-176) folded to five with
    // the same values up to rounding (these fields carry the 1e-12 tolerance):
    // 1/tau_e = 2 (V + eps) / L0h and 1/tau_s = 2 (vx + eps) / l0h as
    // products, and tau' = 1 / (1/tau + c) + dt with c = 1 / (100 dt) entering
    // only as -dt / tau' = -dt u / (1 + dt u), u = 1/tau + c.  Those five, the
    // roots and the exponentials run on the integer pipe: 45 FP64 instructions
    // per cell are left of 183 (bound by the FP64 unit, 375 -> 105 us at 1024^2).
    const double ve = AT(V, j, i) + XC_EPS, vs = AT(vx, j, i) + XC_EPS;
    const double taue = xc_div(L0h, xc_scale2<1>(ve));
    const double itaue = ve * i2L0h, itaus = vs * i2l0h;   // i2L0h = 2 / L0h, i2l0h = 2 / l0h
    double St = xc_div(txi0, taue + XC_EPS);
    double fr = AT(fReL, j, i), k = AT(ke, j, i), ch = AT(chi, j, i);
    double sge = Xi * xc_sqrt(xc_max0((fr * k) * itaue));
    double sgx = Xi * xc_sqrt(xc_max0(xc_div((((ch * fr) * k) * itaue) * St, 1.0 + St * St)));
    double sgs = Xi * xc_sqrt(xc_max0((ch * AT(ks, j, i)) * itaus));
    const double due = dt * (itaue + cdt), dus = dt * (itaus + cdt);   // cdt = 1 / (100 dt)
    double Fte = xc_exp(xc_div(-due, 1.0 + due)), Fts = xc_exp(xc_div(-dus, 1.0 + dus));
    double ae = xc_sqrt(xc_max0(1.0 - Fte * Fte)), as = xc_sqrt(xc_max0(1.0 - Fts * Fts));
    const double re1 = (ae * fL) * AT(re, j, i), rs1 = (as * fl) * AT(rs, j, i);
    AT(psie, j, i) = Fte * AT(psieo, j, i) + sge * re1;
    AT(psix, j, i) = Fte * AT(psixo, j, i) + sgx * re1;
    AT(psis, j, i) = Fts * AT(psiso, j, i) + sgs * rs1;
  });
}

// The filtered fields are re-standardised to the raw mean and std
// (noise.jl:261-267; st = {raw mean, raw sum sq dev, filtered mean, filtered
// sum sq dev} per field) where the staggered differences below read them:
// the ratio raw std / filtered std, the same for every cell, is formed once
// per block, and (v - mean) raw / flt becomes a product, within the 1e-12
// tolerance of these fields.
struct Standard {
  double mean[3], ratio[3], raw[3];
  int use[3];
};
__device__ __forceinline__ double standardised(const Standard& n, int q, double v) {
  return n.use[q] ? (v - n.mean[q]) * n.ratio[q] + n.raw[q] : v;
}

// grid.icz / grid.icx extension (closed z, periodic x: noise.jl:143-144)
__device__ __forceinline__ int icz_c(int j, int Nz) { return j == 0 ? 0 : (j == Nz + 1 ? Nz - 1 : j - 1); }
__device__ __forceinline__ int icx_p(int i, int Nx) { return i == 0 ? Nx - 1 : (i == Nx + 1 ? 0 : i - 1); }

// exp(y) where only 1 - exp(y) is used: below y = -38, exp(y) < 3.2e-17 is
// under half an ulp of 1 (2^-54), so 1 - exp(y) rounds to exactly 1.0 and
// the exponential is skipped without changing a bit (the crystal-fraction
// taper, a / 1e-4 with a >= 0.004)
__device__ __forceinline__ double exp_tail(double y) { return y < -38.0 ? 0.0 : xc_exp(y); }
__device__ __forceinline__ double taper(double a, double b) {
  return (1.0 - exp_tail(xc_div(-a, 1e-4))) * (1.0 - exp_tail(xc_div(-xc_max0(b - 0.4), 0.05)));
}

// staggered noise fluxes (noise.jl:195-220), one thread per (j, i) of
// (Nz+2, Nx+2), in tiles of 32 x 8.  The standardised fields of the extended
// grid (cells j, j+1 by i, i+1; corners need one more on the low side for the
// ghost rows and columns, which repeat and wrap) are formed once per tile in
// shared memory, and so is each corner's average.  22 FP64 instructions per
// cell instead of 106, and no pass of its own for the re-standardisation:
// 214 + 74 -> 100 us at 1024^2.
constexpr int SZ = 32, SX = 8;
__global__ void __launch_bounds__(256) stagger_kernel(int Nz, int Nx, CView pe, CView px, CView ps, const double* st,
                                                      CView chiw, CView muw, CView chiu, CView muu, DView xieu,
                                                      DView xiew, DView xixu, DView xixw, DView xisu, DView xisw) {
  XC_PDL_WAIT();
  __shared__ Standard norm;
  // e: psi_e on the extended rows j0-2 .. j0+32 and columns i0-1 .. i0+8; c: the
  // averages of the corners there; sx, ss: psi_x, psi_s from row j0, column i0
  __shared__ double e[SX + 2][SZ + 3], c[SX + 1][SZ + 2], sx[SX + 1][SZ + 1], ss[SX + 1][SZ + 1];
  const int tid = threadIdx.y * 32 + threadIdx.x;
  if (tid < 3) {
    const double nm1 = (double)Nz * (double)Nx - 1.0;
    const double* s = st + 4 * tid;
    const double raw_std = sqrt(s[1] / nm1), flt_std = sqrt(s[3] / nm1);
    norm.use[tid] = !(flt_std <= XC_EPS);   // a NaN anywhere makes the whole field NaN, as the 2-D FFT does
    norm.ratio[tid] = raw_std / flt_std;
    norm.mean[tid] = s[2];
    norm.raw[tid] = s[0];
  }
  __syncthreads();
  const int nbx = (Nz + 2 + SZ - 1) / SZ, nt = nbx * ((Nx + 2 + SX - 1) / SX);
  for (int t = blockIdx.x; t < nt; t += gridDim.x) {
    const int j0 = (t % nbx) * SZ, i0 = (t / nbx) * SX;
    // the extended index a stands for cell icz(a) / icx(a); the corner (b, d)
    // averages the cells b, b+1 by d, d+1.  Ghost row j of xieu takes the
    // corners of cell row icz(j): Nz-1 for row Nz+1, two before it, which may
    // be the tile's first.
    for (int k = tid; k < (SX + 2) * (SZ + 3); k += 256) {
      const int ii = k / (SZ + 3), jj = k - ii * (SZ + 3);
      const int a = j0 - 2 + jj, b = i0 - 1 + ii;
      if (a >= 0 && a <= Nz + 1 && b >= 0 && b <= Nx + 1) {
        const int cj = icz_c(a, Nz), ci = icx_p(b, Nx);
        e[ii][jj] = standardised(norm, 0, AT(pe, cj, ci));
        if (ii >= 1 && jj >= 2) {
          sx[ii - 1][jj - 2] = standardised(norm, 1, AT(px, cj, ci));
          ss[ii - 1][jj - 2] = standardised(norm, 2, AT(ps, cj, ci));
        }
      }
    }
    __syncthreads();
    for (int k = tid; k < (SX + 1) * (SZ + 2); k += 256) {
      const int ii = k / (SZ + 2), jj = k - ii * (SZ + 2);
      const int a = j0 - 2 + jj, b = i0 - 1 + ii;
      if (a >= 0 && a <= Nz && b >= 0 && b <= Nx)
        c[ii][jj] = xc_scale2<-2>(((e[ii][jj] + e[ii + 1][jj]) + e[ii][jj + 1]) + e[ii + 1][jj + 1]);
    }
    __syncthreads();
    const int jj = threadIdx.x, ii = threadIdx.y, j = j0 + jj, i = i0 + ii;
    if (j <= Nz + 1 && i <= Nx + 1) {
      if (i <= Nx) {   // (Nz+2, Nx+1): xieu = xieu_int[icz, :], xixu, xisu
        const int r = icz_c(j, Nz) - j0 + 2;       // corner rows r, r + 1 of the tile
        AT(xieu, j, i) = c[ii + 1][r + 1] - c[ii + 1][r];
        const double tap = taper(AT(chiu, j, i), AT(muu, j, i));
        AT(xixu, j, i) = (-(sx[ii + 1][jj] - sx[ii][jj])) * tap;
        AT(xisu, j, i) = (-(ss[ii + 1][jj] - ss[ii][jj])) * tap;
      }
      if (j <= Nz) {   // (Nz+1, Nx+2): xiew = xiew_int[:, icx], xixw, xisw
        const int d = icx_p(i, Nx) - i0 + 1;
        double hi, lo;
        if (d >= 0 && d < SX) {
          hi = c[d + 1][jj + 2];
          lo = c[d][jj + 2];
        } else {       // the wrapped ghost columns: another tile's corners
          const int ix = icx_p(i, Nx);
          auto corner = [&](int b) {
            auto ex = [&](int a, int q) { return standardised(norm, 0, AT(pe, icz_c(a, Nz), icx_p(q, Nx))); };
            return xc_scale2<-2>(((ex(j, b) + ex(j, b + 1)) + ex(j + 1, b)) + ex(j + 1, b + 1));
          };
          hi = corner(ix + 1);
          lo = corner(ix);
        }
        AT(xiew, j, i) = -(hi - lo);
        const double tap = taper(AT(chiw, j, i), AT(muw, j, i));
        AT(xixw, j, i) = (-(sx[ii][jj + 1] - sx[ii][jj])) * tap;
        AT(xisw, j, i) = (-(ss[ii][jj + 1] - ss[ii][jj])) * tap;
      }
    }
    __syncthreads();
  }
}

// speed magnitudes (noise.jl:223-236)
__global__ void speeds_kernel(int Nz, int Nx, CView xisw, CView xisu, CView xixw, CView xixu,
                              CView xiew, CView xieu, DView xis, DView xix, DView xie) {
  XC_PDL_WAIT();
  for_tiles(Nz, Nx, [&](int j, int i) {
    if (j >= Nz || i >= Nx) return;
    double wz = xc_half(AT(xisw, j, i + 1) + AT(xisw, j + 1, i + 1));
    double wx = xc_half(AT(xisu, j + 1, i) + AT(xisu, j + 1, i + 1));
    AT(xis, j, i) = xc_sqrt(wz * wz + wx * wx);
    wz = xc_half(AT(xixw, j, i + 1) + AT(xixw, j + 1, i + 1));
    wx = xc_half(AT(xixu, j + 1, i) + AT(xixu, j + 1, i + 1));
    AT(xix, j, i) = xc_sqrt(wz * wz + wx * wx);
    wz = xc_half(AT(xiew, j, i + 1) + AT(xiew, j + 1, i + 1));
    wx = xc_half(AT(xieu, j + 1, i) + AT(xieu, j + 1, i + 1));
    AT(xie, j, i) = xc_sqrt(wz * wz + wx * wx);
  });
}

}  // namespace

int noise_plan_create(xc_ctx* c) {
  NoisePlan* np = new NoisePlan();
  c->noise = np;
  const double h = c->p.h, L0h = c->p.L0h, l0h = c->p.l0h;
  np->padL0 = 4 * (int)std::ceil(L0h / h);
  np->padl0 = 4 * (int)std::ceil(l0h / h);
  np->fL = 2.0 / std::sqrt(1.0 - std::exp(-(h * h) / (2.0 * (L0h * L0h))));
  np->fl = 2.0 / std::sqrt(1.0 - std::exp(-(h * h) / (2.0 * (l0h * l0h))));
  const int Nz = c->Nz, Nx = c->Nx;
  build_direct(np->dz[0], Nz + np->padL0, h, L0h);
  build_direct(np->dx[0], Nx, h, L0h);
  build_direct(np->dz[1], Nz + np->padl0, h, l0h);
  build_direct(np->dx[1], Nx, h, l0h);
  np->direct = np->dz[0].R && np->dx[0].R && np->dz[1].R && np->dx[1].R;
  if (np->direct) return XC_OK;
  XC_TRY(build_line_filter(np->ze, Nz, Nz + np->padL0, h, L0h, false));
  XC_TRY(build_line_filter(np->xe, Nx, Nx, h, L0h, true));
  XC_TRY(build_line_filter(np->zs, Nz, Nz + np->padl0, h, l0h, false));
  XC_TRY(build_line_filter(np->xs, Nx, Nx, h, l0h, true));
  return XC_OK;
}

void noise_plan_destroy(xc_ctx* c) {
  if (!c->noise) return;
  free_line_filter(c->noise->ze);
  free_line_filter(c->noise->xe);
  free_line_filter(c->noise->zs);
  free_line_filter(c->noise->xs);
  delete c->noise;
  c->noise = nullptr;
}

int noise_impl(xc_ctx* c, double dt, int first_iter, const double* re, const double* rs, cudaStream_t s_in,
               double* partials) {
  const int Nz = c->Nz, Nx = c->Nx;
  const xc_params& p = c->p;
  cudaStream_t s = s_in ? s_in : c->stream;
  NoisePlan* np = c->noise;
  const size_t nb = sizeof(double) * (size_t)Nz * Nx;
  if (first_iter) {
    if (re) XC_CUDA_TRY(cudaMemcpyAsync(c->field[FLD_re], re, nb, cudaMemcpyHostToDevice, s));
    if (rs) XC_CUDA_TRY(cudaMemcpyAsync(c->field[FLD_rs], rs, nb, cudaMemcpyHostToDevice, s));
  }
  dim3 blk(32, 8);
  xc_launch(ou_kernel, dim3(persistent_grid((const void*)ou_kernel, Nz, Nx)), blk, 0, s, Nz, Nx, p.Xi, p.L0h,
      2.0 / p.L0h, 2.0 / p.l0h, p.txi0, dt,
      1.0 / (1e2 * dt), np->fL, np->fl, CF(c, FLD_V),
      CF(c, FLD_vx),
      CF(c, FLD_fReL), CF(c, FLD_ke), CF(c, FLD_chi), CF(c, FLD_ks), CF(c, FLD_psieo),
      CF(c, FLD_psixo), CF(c, FLD_psiso), CF(c, FLD_re), CF(c, FLD_rs), F(c, FLD_psie),
      F(c, FLD_psix), F(c, FLD_psis));
  XC_LAUNCH_CHECK();
  // filtered fields in tmp[2..4], z-pass intermediate in tmp[5]
  DView flt[3] = {DView{c->tmp[2], Nz}, DView{c->tmp[3], Nz}, DView{c->tmp[4], Nz}};
  DView mid{c->tmp[5], Nz};
  const int src[3] = {FLD_psie, FLD_psix, FLD_psis};
  const LineFilter* zf[3] = {&np->ze, &np->ze, &np->zs};
  const LineFilter* xf[3] = {&np->xe, &np->xe, &np->xs};
  double* st = c->dscal + SC_NOISE_STATS;
  const double n = (double)Nz * (double)Nx;
  if (np->direct) {
    // the z passes go to the speed fields, which the last kernel overwrites
    DirectPass pz, px;
    const int mids[3] = {FLD_xie, FLD_xix, FLD_xis};
    for (int q = 0; q < 3; ++q) {
      pz.in[q] = CF(c, src[q]);
      pz.out[q] = F(c, mids[q]);
      px.in[q] = CF(c, mids[q]);
      px.out[q] = flt[q];
    }
    for (int q = 0; q < 2; ++q) {
      pz.f[q] = np->dz[q];
      px.f[q] = np->dx[q];
    }
    xc_launch(direct_filter_kernel<0>, dim3((Nz + 63) / 64, (Nx + 3) / 4, 3), 256, 0, s, pz, Nz, Nx);
    xc_launch(direct_filter_kernel<1>, dim3((Nz + 31) / 32, (Nx + 7) / 8, 3), 256, 0, s, px, Nz, Nx);
    XC_LAUNCH_CHECK();
  } else {
    for (int q = 0; q < 3; ++q) {
      XC_TRY(run_line_filter(*zf[q], CF(c, src[q]), mid, Nz, Nx, 0, s));
      XC_TRY(run_line_filter(*xf[q], CView{mid.p, Nz}, flt[q], Nz, Nx, 1, s));
    }
  }
  // the six means in one launch, then the six centred sums of squares
  // (mean and corrected std of noise.jl:261-264)
  RedJob means[6], devs[6];
  for (int q = 0; q < 3; ++q) {
    CView raw = CF(c, src[q]), fv{flt[q].p, Nz};
    means[2 * q] = red_job(RED_SUM, raw, CView{nullptr, 0}, nullptr, Nz, Nx, st + 4 * q + 0, n);
    means[2 * q + 1] = red_job(RED_SUM, fv, CView{nullptr, 0}, nullptr, Nz, Nx, st + 4 * q + 2, n);
    devs[2 * q] = red_job(RED_SUM, raw, CView{nullptr, 0}, st + 4 * q + 0, Nz, Nx, st + 4 * q + 1);
    devs[2 * q + 1] = red_job(RED_SUM, fv, CView{nullptr, 0}, st + 4 * q + 2, Nz, Nx, st + 4 * q + 3);
  }
  XC_TRY(reduce_batch(c, means, 6, s, partials));
  XC_TRY(reduce_batch(c, devs, 6, s, partials));
  xc_launch(stagger_kernel, dim3(persistent_grid((const void*)stagger_kernel, Nz + 2, Nx + 2)), blk, 0, s, Nz, Nx,
      CView{flt[0].p, Nz},
      CView{flt[1].p, Nz}, CView{flt[2].p, Nz}, st, CF(c, FLD_chiw),
      CF(c, FLD_muw), CF(c, FLD_chiu), CF(c, FLD_muu), F(c, FLD_xieu), F(c, FLD_xiew),
      F(c, FLD_xixu), F(c, FLD_xixw), F(c, FLD_xisu), F(c, FLD_xisw));
  XC_LAUNCH_CHECK();
  xc_launch(speeds_kernel, dim3(persistent_grid((const void*)speeds_kernel, Nz, Nx)), blk, 0, s, Nz, Nx,
      CF(c, FLD_xisw), CF(c, FLD_xisu),
      CF(c, FLD_xixw), CF(c, FLD_xixu), CF(c, FLD_xiew),
      CF(c, FLD_xieu), F(c, FLD_xis), F(c, FLD_xix), F(c, FLD_xie));
  XC_LAUNCH_CHECK();
  return XC_OK;
}

// time the FFT line filter (z pass of psie) with CUDA events on the context stream
int noise_bench_zpass(xc_ctx* c, int iters, double out[4]) {
  const int Nz = c->Nz, Nx = c->Nx;
  NoisePlan* np = c->noise;
  cudaEvent_t e0, e1;
  XC_CUDA_TRY(cudaEventCreate(&e0));
  XC_CUDA_TRY(cudaEventCreate(&e1));
  int st = XC_OK;
  for (int it = -1; it < iters && st == XC_OK; ++it) {
    if (it == 0) cudaEventRecord(e0, c->stream);
    if (np->direct) {
      DirectPass p;
      for (int q = 0; q < 3; ++q) {
        p.in[q] = CF(c, FLD_psie);
        p.out[q] = DView{c->tmp[5], Nz};
      }
      p.f[0] = p.f[1] = np->dz[0];
      xc_launch(direct_filter_kernel<0>, dim3((Nz + 63) / 64, (Nx + 3) / 4, 1), 256, 0, c->stream, p, Nz, Nx);
      XC_LAUNCH_CHECK();
    } else {
      st = run_line_filter(np->ze, CF(c, FLD_psie), DView{c->tmp[5], Nz}, Nz, Nx, 0, c->stream);
    }
  }
  cudaEventRecord(e1, c->stream);
  cudaEventSynchronize(e1);
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (st != XC_OK) return st;
  const double M = np->ze.M, logM = np->ze.logM;
  out[0] = ms / iters;
  out[1] = 16.0 * Nz * (double)Nx;                   // read psi, write the filtered field
  // 2 R + 1 multiply-adds per cell, or forward + inverse complex FFT per line pair
  out[2] = np->direct ? 2.0 * (2 * np->dz[0].R + 1) * Nz * (double)Nx : (double)((Nx + 1) / 2) * 2.0 * 5.0 * M * logM;
  out[3] = (double)Nz * Nx;
  return XC_OK;
}
