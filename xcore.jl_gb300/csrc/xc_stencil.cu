// Advection and diffusion stencils, halo fill and phsevo! on the GPU.
//
// Reference: src/kernels/advect.jl, src/kernels/diffus.jl, src/kernels/ghosts.jl,
// src/phsevo.jl.  The reference evaluates every face value twice (once for each
// neighbouring cell, advect.jl:57-96) and then a third time in the per-face
// flux kernels (advect.jl:603-637).  Those three evaluations are bitwise
// identical (advect.jl:428-432), so here each CTA computes every face flux of
// its tile ONCE into shared memory and takes the cell divergence from there,
// in the reference's operation order: adv = (qxr - qxl + qzb - qzt) * invh.
// Compiled with -fmad=false so no multiply-add is contracted (Julia does not
// contract either); with identical inputs the results are bitwise equal to
// the reference arithmetic.
//
// What bounds it: sm_103a's FP64 unit takes one warp instruction per 64 cycles
// and sub-partition, so the stencils cost their FP64 instructions and little
// else.  Products by 2, 4 and 1/4 are exact and go into the following sum as an
// FMA (the same rounding, one instruction instead of two; WENO5's quarters of
// squares, where a subnormal one is far below the sum), quotients and most
// other products run on the integer pipe (xc_fp64.cuh), signs are tested on
// the bits: what is left for the FP64 unit are the sums.  WENO5 in the
// reference's form takes 27 FP64 instructions per face, and some 1400 integer
// ones beside them that issue in about their time.  One 1024^2 field with its
// fluxes: 443 us with everything on the FP64 unit, 237 us with the quotients
// taken off it, 156 us with the products off it too.
#include "xc_internal.cuh"

namespace {

// Tiles: TZ rows (z, contiguous in memory) x TX columns (x), NT threads.  One
// thread evaluates one face at a time and the x and z faces of a tile are one
// index space, so that a small tile's faces (280 of 16 x 8) are one round of
// its threads: the time of a small grid is that round.  The larger tile
// evaluates 2.09 faces per cell instead of 2.19 and reads less halo, but its
// last wave is emptier.  Measured, small against large tile, WENO5: 6.9 / 23.3
// us at 100^2, 29 / 40 at 400^2, 77 / 84 at 700^2, 111 / 117 at 850^2, 156 /
// 160 at 1024^2, 334 / 330 at 1500^2; diffusion, which is read and write: 6.6
// / 8.6 at 400^2, 8.6 / 9.9 at 512^2, 14.2 / 14.6 at 700^2, 27.0 / 24.5 at
// 1024^2.  The lines lie at 18 and at 7 waves of the larger tile (152 of 512
// cells each).
template <int Z, int X, int T> struct TileShape {
  static constexpr int TZ = Z, TX = X, NT = T;
};
using SmallTile = TileShape<16, 8, 288>;
using LargeTile = TileShape<32, 16, 256>;
constexpr long long kSmallAdvect = 18LL * kNumSMs * 512, kSmallDiffus = 7LL * kNumSMs * 512;
// (a grid has at most 65535 blocks along x: rows of more than 8 times as many
// columns, fields one or two cells high, take the larger tile's 16 columns too)
inline bool small_tile(long long most, int Nz, int Nx) {
  return (long long)Nz * Nx <= most && (Nx + SmallTile::TX - 1) / SmallTile::TX <= 65535;
}

// ---------------------------------------------------------------------------
// face reconstructions (advect.jl:35-53, 216-229, 275-283)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double weno5_poly(double fmm, double fm, double fc, double fp,
                                             double fpp) {
  const double sixth = 1.0 / 6.0, quarter = 0.25, c1312 = 13.0 / 12.0;
  const double eps_val = XC_EPS;
  const double p1 = xc_mul(__fma_rn(2.0, fmm, -xc_mul_small<7>(fm)) + xc_mul_small<11>(fc), sixth);
  const double p2 = xc_mul(__fma_rn(2.0, fp, xc_mul_small<5>(fc) - fm), sixth);
  const double p3 = xc_mul(__fma_rn(2.0, fc, xc_mul_small<5>(fp)) - fpp, sixth);
  const double fc3 = xc_mul_small<3>(fc);
  double t = __fma_rn(-2.0, fm, fmm) + fc, s = __fma_rn(-4.0, fm, fmm) + fc3;
  const double b1 = __fma_rn(quarter, xc_sqr(s), xc_mul(xc_sqr(t), c1312));
  t = __fma_rn(-2.0, fc, fm) + fp;
  s = fm - fp;
  const double b2 = __fma_rn(quarter, xc_sqr(s), xc_mul(xc_sqr(t), c1312));
  t = __fma_rn(-2.0, fp, fc) + fpp;
  s = __fma_rn(-4.0, fp, fc3) + fpp;
  const double b3 = __fma_rn(quarter, xc_sqr(s), xc_mul(xc_sqr(t), c1312));
  const double e1 = b1 + eps_val, e2 = b2 + eps_val, e3 = b3 + eps_val;
  const double w1 = xc_div(0.1, xc_sqr(e1));
  const double w2 = xc_div(0.6, xc_sqr(e2));
  const double w3 = xc_div(0.3, xc_sqr(e3));
  return xc_div((xc_mul(w1, p1) + xc_mul(w2, p2)) + xc_mul(w3, p3), (w1 + w2) + w3);
}

// The same reconstruction with the weights over a common denominator: with
// q_k = (eps + b_k)^2 the weights d_k / q_k are proportional to
// n_1 = q_2 q_3, n_2 = 6 q_1 q_3, n_3 = 3 q_1 q_2, so the weighted mean needs
// one division instead of four.  The smoothness indicators are formed four
// times as large and the q_k a sixteenth of their size (powers of two, which
// leave the weights as they are), and the common factor 1/6 of the three
// polynomials is applied once (within a few ulps).  The products n_k p_k grow as
// the ninth power of the field and are finite up to some 1e34; each q_k is at
// least (4 eps)^2 / 256, far from underflow.  27 FP64 instructions per
// reconstruction, as many as the reference's form takes: the products and the
// quotients are integer ones.
__device__ __forceinline__ double weno5_poly_onediv(double fmm, double fm, double fc, double fp,
                                                    double fpp) {
  const double c133 = 4.0 * (13.0 / 12.0), eps4 = 4.0 * XC_EPS;
  const double p1 = __fma_rn(11.0, fc, __fma_rn(-7.0, fm, xc_scale2<1>(fmm)));
  const double p2 = __fma_rn(2.0, fp, __fma_rn(5.0, fc, -fm));
  const double p3 = __fma_rn(2.0, fc, __fma_rn(5.0, fp, -fpp));
  double t = __fma_rn(-2.0, fm, fmm) + fc, s = __fma_rn(3.0, fc, __fma_rn(-4.0, fm, fmm));
  const double e1 = __fma_rn(xc_mul(t, c133), t, xc_sqr(s)) + eps4;
  t = __fma_rn(-2.0, fc, fm) + fp;
  s = fm - fp;
  const double e2 = __fma_rn(xc_mul(t, c133), t, xc_sqr(s)) + eps4;
  t = __fma_rn(-2.0, fp, fc) + fpp;
  s = __fma_rn(3.0, fc, __fma_rn(-4.0, fp, fpp));
  const double e3 = __fma_rn(xc_mul(t, c133), t, xc_sqr(s)) + eps4;
  const double q1 = xc_sqr<8>(e1), q2 = xc_sqr<8>(e2), q3 = xc_sqr<8>(e3);
  const double n1 = xc_mul(q2, q3), n2 = xc_mul_small<6>(xc_mul(q1, q3)), n3 = xc_mul_small<3>(xc_mul(q1, q2));
  return xc_mul(xc_div(__fma_rn(n1, p1, __fma_rn(n2, p2, xc_mul(n3, p3))), (n1 + n2) + n3), 1.0 / 6.0);
}

__device__ __forceinline__ double weno3_poly(double fm, double fc, double fp) {
  const double eps_val = 1e-6;
  double p1 = xc_half(fc + fp);
  double p2 = xc_half(xc_mul_small<3>(fc) - fm);
  double d1 = fp - fc, d2 = fc - fm;
  double w1 = xc_div(1.0 / 3.0, xc_sqr(d1) + eps_val);
  double w2 = xc_div(2.0 / 3.0, xc_sqr(d2) + eps_val);
  return xc_div(xc_mul(w1, p1) + xc_mul(w2, p2), w1 + w2);
}

__device__ __forceinline__ double tvd_flux(double fm, double fc, double fp, double vm, double vp) {
  double num = vm * (fc - fm);
  double den = vp * (fp - fc);
  double R = num / (den + copysign(XC_EPS, den));
  double l = jmax(0.0, jmax(jmin(1.0, 2.0 * R), jmin(2.0, R)));
  return fc + (0.5 * l) * (fp - fc);
}

__device__ __forceinline__ double vpos(double v) { return (v + fabs(v)) * 0.5; }
__device__ __forceinline__ double vneg(double v) { return (v - fabs(v)) * 0.5; }
__device__ __forceinline__ bool sign_bit(double v) { return __double2hiint(v) < 0; }
__device__ __forceinline__ bool zero_bits(double v) {
  return ((__double2hiint(v) & 0x7fffffff) | __double2loint(v)) == 0;
}
__device__ __forceinline__ bool finite_bits(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }

// Flux through the face between cells s2 and s3 of the six-cell window
// s0..s5, with face velocity v (and the neighbouring faces' vl, vr for TVD).
// Per-face formulas of advect.jl:444-695.
template <int S>
__device__ __forceinline__ double face_flux(double s0, double s1, double s2, double s3, double s4,
                                            double s5, double v, double vl, double vr) {
  if (S == XC_CENTR) {
    return v * (s2 + s3) * 0.5;
  } else if (S == XC_UPWD1) {
    return vpos(v) * s2 + vneg(v) * s3;
  } else if (S == XC_QUICK || S == XC_FROMM) {
    // vpos(v) pos + vneg(v) neg with only the upwind value formed: the other
    // term is a zero, which changes no value -- unless its factor is not
    // finite, so a window with an infinity or NaN takes the whole formula.
    const double sixth = 1.0 / 6.0;
    if (finite_bits(s1) && finite_bits(s2) && finite_bits(s3) && finite_bits(s4) && finite_bits(v)) {
      const bool up = !sign_bit(v);
      const double a1 = up ? s1 : s4, a2 = up ? s2 : s3, a3 = up ? s3 : s2;
      return xc_mul(v, S == XC_QUICK ? xc_mul(__fma_rn(2.0, a3, xc_mul_small<5>(a2)) - a1, sixth)
                                     : a2 + xc_scale2<-2>(a3 - a1));   // (a quarter of a subnormal rounds)
    }
    double pos, neg;
    if (S == XC_QUICK) {
      pos = sixth * ((2.0 * s3 + 5.0 * s2) - s1);
      neg = sixth * ((2.0 * s2 + 5.0 * s3) - s4);
    } else {
      pos = s2 + 0.25 * (s3 - s1);
      neg = s3 + 0.25 * (s2 - s4);
    }
    return vpos(v) * pos + vneg(v) * neg;
  } else if (S == XC_WENO3 || S == XC_WENO5 || S == kWeno5OneDiv) {
    // vpos(v) pos + vneg(v) neg has one weight exactly zero: only the upwind
    // reconstruction is evaluated.  The dropped term is (+0) x (finite) = +-0,
    // which changes no value (at most the sign of a zero result); v = +-0
    // gives 0 and a NaN v stays NaN, as in the full formula.  The other weight
    // is v itself.
    // The mirrored stencil is selected first, so a warp with faces of both
    // signs still evaluates one polynomial per face.
    const bool up = !sign_bit(v);
    const double a0 = up ? s0 : s5, a1 = up ? s1 : s4, a2 = up ? s2 : s3, a3 = up ? s3 : s2,
                 a4 = up ? s4 : s1;
    const double p = S == XC_WENO5        ? weno5_poly(a0, a1, a2, a3, a4)
                     : S == kWeno5OneDiv ? weno5_poly_onediv(a0, a1, a2, a3, a4)
                                         : weno3_poly(a1, a2, a3);
    return zero_bits(v) ? v : xc_mul(v, p);
  } else {  // XC_TVDIM
    double cpos = vpos(v), cneg = vneg(v);
    double pos = tvd_flux(s1, s2, s3, vpos(vl), cpos);
    double neg = tvd_flux(s4, s3, s2, vneg(vr), cneg);
    return cpos * pos + cneg * neg;
  }
}

template <int S> struct Halo {
  static constexpr int G = (S == XC_WENO5 || S == kWeno5OneDiv) ? 3 : (S == XC_CENTR || S == XC_UPWD1) ? 1 : 2;
};

__device__ __forceinline__ int map_bc(int k, int n, int bc) {
  if (bc == XC_PERIODIC) {
    k %= n;
    return k < 0 ? k + n : k;
  }
  return k < 0 ? 0 : (k >= n ? n - 1 : k);
}

// velocity at face index k (0..n) of an axis with n cells, extended by one
// face on each side for TVD exactly as the reference pads u/w (phsevo.jl:34-53)
__device__ __forceinline__ int map_face(int k, int n, int bc) {
  if (k >= 0 && k <= n) return k;
  if (bc == XC_PERIODIC) return k < 0 ? k + n : k - n;
  return k < 0 ? 0 : n;
}

// ---------------------------------------------------------------------------
// face-flux arrays with the reference's padding: qx is (Nz+2, Nx+1) and its
// rows 0 and Nz+1 copy the last and first interior row (periodic z) or the
// neighbouring one (closed); qz is (Nz+1, Nx+2), its columns 0 and Nx+1
// likewise in x (advect.jl:779-795, diffus.jl:194-208).  `qx`, `qz` view the
// unpadded faces; the thread that has a face's flux writes its copies too.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void put_qx(DView qx, int j, int i, double q, int Nz, int zBC, bool pad) {
  double* p = qx.p + (size_t)i * (size_t)qx.ld + j;
  *p = q;
  if (pad) {
    const bool per = zBC == XC_PERIODIC && Nz > 1;
    if (j == (per ? Nz - 1 : 0)) *(p - j - 1) = q;
    if (j == (per ? 0 : Nz - 1)) *(p - j + Nz) = q;
  }
}
__device__ __forceinline__ void put_qz(DView qz, int j, int i, double q, int Nx, int xBC, bool pad) {
  double* p = qz.p + (size_t)i * (size_t)qz.ld + j;
  *p = q;
  if (pad) {
    const bool per = xBC == XC_PERIODIC && Nx > 1;
    if (i == (per ? Nx - 1 : 0)) *(qz.p + j - qz.ld) = q;
    if (i == (per ? 0 : Nx - 1)) *(qz.p + j + (size_t)Nx * (size_t)qz.ld) = q;
  }
}

// One field's advection or diffusion: f the interior (Nz, Nx) field read
// through the BC map or, halo'd, the caller's (Nz+2G, Nx+2G) array.  u
// (Nz, Nx+1) x-face velocities, w (Nz+1, Nx) z-face velocities (halo'd tvdim:
// the padded (Nz, Nx+3) / (Nz+3, Nx)); k1 (times k2 when given) diffusivity.
// Outputs (any may be null): out (Nz, Nx), qx (Nz, Nx+1), qz (Nz+1, Nx).
struct FluxArgs {
  const double* f;
  int ld;
  CView u, w;
  const double *k1, *k2;
  DView out, qx, qz;
};

template <class T, int G> struct TileSmem {
  static constexpr int HZ = T::TZ + 2 * G, HX = T::TX + 2 * G;
  static constexpr int NXF = T::TZ * (T::TX + 1), NZF = (T::TZ + 1) * T::TX;   // x faces, then z faces
  double f[HX * HZ];
  double q[NXF + NZF];
};

// ---------------------------------------------------------------------------
// advection of one tile
// ---------------------------------------------------------------------------
template <class T, int S, bool HALOD>
__device__ __forceinline__ void advect_tile(TileSmem<T, Halo<S>::G>& sm, const FluxArgs& a, int Nz, int Nx, int xBC,
                                            int zBC, double invh, bool pad) {
  constexpr int G = Halo<S>::G, TZ = T::TZ, TX = T::TX, NT = T::NT;
  using M = TileSmem<T, G>;
  constexpr int HZ = M::HZ, HX = M::HX;
  const int j0 = blockIdx.x * TZ, i0 = blockIdx.y * TX;
  const int tid = threadIdx.x;

  for (int idx = tid; idx < HZ * HX; idx += NT) {
    int jj = idx % HZ, ii = idx / HZ;
    int j = j0 - G + jj, i = i0 - G + ii;
    double v = 0.0;
    if (HALOD) {
      int hj = j + G, hi = i + G;
      if (hj < Nz + 2 * G && hi < Nx + 2 * G) v = a.f[(size_t)hi * a.ld + hj];
    } else {
      v = a.f[(size_t)map_bc(i, Nx, xBC) * a.ld + map_bc(j, Nz, zBC)];
    }
    sm.f[idx] = v;
  }
  __syncthreads();

  for (int idx = tid; idx < M::NXF + M::NZF; idx += NT) {
    const bool xf = idx < M::NXF;
    const int k = xf ? idx : idx - M::NXF;
    const int ii = xf ? k / TZ : k / (TZ + 1), jj = k - ii * (xf ? TZ : TZ + 1);
    const int j = j0 + jj, i = i0 + ii;
    double q = 0.0;
    // x face i sits between cells i-1 and i, z face j between j-1 and j
    if (xf ? (j < Nz && i <= Nx) : (j <= Nz && i < Nx)) {
      double v, vl = 0.0, vr = 0.0;
      if (S == XC_TVDIM) {
        if (xf) {
          v = AT(a.u, j, HALOD ? i + 1 : i);
          vl = AT(a.u, j, HALOD ? i : map_face(i - 1, Nx, xBC));
          vr = AT(a.u, j, HALOD ? i + 2 : map_face(i + 1, Nx, xBC));
        } else {
          v = AT(a.w, HALOD ? j + 1 : j, i);
          vl = AT(a.w, HALOD ? j : map_face(j - 1, Nz, zBC), i);
          vr = AT(a.w, HALOD ? j + 2 : map_face(j + 1, Nz, zBC), i);
        }
      } else {
        v = xf ? AT(a.u, j, i) : AT(a.w, j, i);
      }
      const int st = xf ? HZ : 1;
      const double* c = sm.f + (ii + G) * HZ + jj + G;
      const double s0 = (G >= 3) ? c[-3 * st] : 0.0;
      const double s1 = (G >= 2) ? c[-2 * st] : 0.0;
      const double s4 = (G >= 2) ? c[st] : 0.0;
      const double s5 = (G >= 3) ? c[2 * st] : 0.0;
      q = face_flux<S>(s0, s1, c[-st], c[0], s4, s5, v, vl, vr);
      // the last tile of each axis also writes the closing face
      if (xf) {
        if (a.qx.p && (ii < TX || i == Nx)) put_qx(a.qx, j, i, q, Nz, zBC, pad);
      } else {
        if (a.qz.p && (jj < TZ || j == Nz)) put_qz(a.qz, j, i, q, Nx, xBC, pad);
      }
    }
    sm.q[idx] = q;
  }
  if (!a.out.p) return;
  __syncthreads();
  const double* qz = sm.q + M::NXF;
  for (int idx = tid; idx < TZ * TX; idx += NT) {
    int jj = idx % TZ, ii = idx / TZ;
    int j = j0 + jj, i = i0 + ii;
    if (j < Nz && i < Nx)
      AT(a.out, j, i) =
          xc_mul(((sm.q[idx + TZ] - sm.q[idx]) + qz[ii * (TZ + 1) + jj + 1]) - qz[ii * (TZ + 1) + jj], invh);
  }
}

template <class T, int S, bool HALOD>
__global__ void __launch_bounds__(T::NT) advect_tile_kernel(FluxArgs a, int Nz, int Nx, int xBC, int zBC, double invh,
                                                            bool pad) {
  XC_PDL_WAIT();
  __shared__ TileSmem<T, Halo<S>::G> sm;
  advect_tile<T, S, HALOD>(sm, a, Nz, Nx, xBC, zBC, invh, pad);
}

// ---------------------------------------------------------------------------
// diffusion of one tile (diffus.jl:9-31, 68-91).  A face's product
// (k_L + k_R)(f_R - f_L) is formed once: the divergence takes it from both
// sides, and the face flux -(k_L + k_R)/2 (f_R - f_L)/h is the same product
// halved and negated, which is exact but for subnormal products.  7 FP64
// instructions per cell instead of 28.
// ---------------------------------------------------------------------------
__device__ __noinline__ double diffus_flux_any(double k, double df, double invh) { return (((-k) * 0.5) * df) * invh; }
__device__ __forceinline__ double diffus_flux(double q, double mhalf_invh, double k, double df, double invh) {
  const uint64_t u = xc_bits(q) << 1;
  if (u - 1 < (3ull << 53) - 1) return diffus_flux_any(k, df, invh);     // not zero, below 2^-1020
  return xc_mul(q, mhalf_invh);
}
template <class T, bool HALOD>
__device__ __forceinline__ void diffus_tile(TileSmem<T, 1>& sm, double* sk, const FluxArgs& a, int Nz, int Nx, int xBC,
                                            int zBC, double invh, bool pad) {
  constexpr int TZ = T::TZ, TX = T::TX, NT = T::NT;
  using M = TileSmem<T, 1>;
  constexpr int HZ = M::HZ, HX = M::HX;
  const int j0 = blockIdx.x * TZ, i0 = blockIdx.y * TX;
  const int tid = threadIdx.x;
  for (int idx = tid; idx < HZ * HX; idx += NT) {
    int jj = idx % HZ, ii = idx / HZ;
    int j = j0 - 1 + jj, i = i0 - 1 + ii;
    double fv = 0.0, kv = 0.0;
    size_t o = (size_t)(i + 1) * a.ld + (j + 1);
    bool in = i <= Nx && j <= Nz;
    if (!HALOD) {
      o = (size_t)map_bc(i, Nx, xBC) * a.ld + map_bc(j, Nz, zBC);
      in = true;
    }
    if (in) {
      fv = a.f[o];
      kv = a.k1[o];
      if (a.k2) kv = xc_mul(kv, a.k2[o]);
    }
    sm.f[idx] = fv;
    sk[idx] = kv;
  }
  __syncthreads();
  const double mhalf_invh = -0.5 * invh;
  for (int idx = tid; idx < M::NXF + M::NZF; idx += NT) {
    const bool xf = idx < M::NXF;
    const int k = xf ? idx : idx - M::NXF;
    const int ii = xf ? k / TZ : k / (TZ + 1), jj = k - ii * (xf ? TZ : TZ + 1);
    const int j = j0 + jj, i = i0 + ii;
    const int c = (ii + 1) * HZ + jj + 1, b = c - (xf ? HZ : 1);
    const double ks = sk[c] + sk[b], df = sm.f[c] - sm.f[b], q = xc_mul(ks, df);
    sm.q[idx] = q;
    if (xf) {
      if (a.qx.p && j < Nz && i <= Nx && (ii < TX || i == Nx))
        put_qx(a.qx, j, i, diffus_flux(q, mhalf_invh, ks, df, invh), Nz, zBC, pad);
    } else {
      if (a.qz.p && j <= Nz && i < Nx && (jj < TZ || j == Nz))
        put_qz(a.qz, j, i, diffus_flux(q, mhalf_invh, ks, df, invh), Nx, xBC, pad);
    }
  }
  if (!a.out.p) return;
  __syncthreads();
  const double* qz = sm.q + M::NXF;
  const double hih2 = 0.5 * (invh * invh);
  for (int idx = tid; idx < TZ * TX; idx += NT) {
    int jj = idx % TZ, ii = idx / TZ;
    int j = j0 + jj, i = i0 + ii;
    if (j < Nz && i < Nx)
      AT(a.out, j, i) =
          xc_mul(((sm.q[idx + TZ] - sm.q[idx]) + qz[ii * (TZ + 1) + jj + 1]) - qz[ii * (TZ + 1) + jj], hih2);
  }
}

template <class T, bool HALOD>
__global__ void __launch_bounds__(T::NT) diffus_tile_kernel(FluxArgs a, int Nz, int Nx, int xBC, int zBC, double invh,
                                                            bool pad) {
  XC_PDL_WAIT();
  __shared__ TileSmem<T, 1> sm;
  __shared__ double sk[TileSmem<T, 1>::HX * TileSmem<T, 1>::HZ];
  diffus_tile<T, HALOD>(sm, sk, a, Nz, Nx, xBC, zBC, invh, pad);
}

// the three stencils of phsevo! side by side in one launch (blockIdx.z: the
// advection of X, of M, the diffusion of chi): they are independent, and a
// small grid's tiles of all three fill the GPU better than one after another
struct PhsevoFluxes { FluxArgs a[3]; };
template <class T, int S>
__global__ void __launch_bounds__(T::NT) phsevo_flux_kernel(PhsevoFluxes p, int Nz, int Nx, int xBC, int zBC,
                                                            double invh) {
  XC_PDL_WAIT();
  constexpr int G = Halo<S>::G;
  struct Diff { TileSmem<T, 1> t; double sk[TileSmem<T, 1>::HX * TileSmem<T, 1>::HZ]; };
  union Smem { TileSmem<T, G> adv; Diff dif; };
  __shared__ Smem sm;
  if (blockIdx.z < 2) advect_tile<T, S, false>(sm.adv, p.a[blockIdx.z], Nz, Nx, xBC, zBC, invh, true);
  else diffus_tile<T, false>(sm.dif.t, sm.dif.sk, p.a[2], Nz, Nx, xBC, zBC, invh, true);
}

// ghost ring of a halo'd array (ghosts.jl:18-51; for N >= halo the x-then-z
// fill equals reading the BC-mapped interior cell, corners included)
__global__ void fill_ghosts_kernel(double* f, int Nz, int Nx, int g, int zBC, int xBC) {
  XC_PDL_WAIT();
  const int rows = Nz + 2 * g, cols = Nx + 2 * g;
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)rows * cols) return;
  int hj = (int)(t % rows), hi = (int)(t / rows);
  int j = hj - g, i = hi - g;
  if (j >= 0 && j < Nz && i >= 0 && i < Nx) return;
  int sj = map_bc(j, Nz, zBC) + g, si = map_bc(i, Nx, xBC) + g;
  f[(size_t)hi * rows + hj] = f[(size_t)si * rows + sj];
}

// phsevo! tail (phsevo.jl:189, 197-211), one thread per cell
__global__ void phsevo_tail_kernel(int Nz, int Nx, double a1, double a2, double a3, double b1,
                                   double b2, double b3, double dt, double alpha, double G0,
                                   DView X, CView Xo, CView Xoo, DView M, DView x, DView m,
                                   CView rho, CView advn_X, CView advn_M, DView advn_rho,
                                   CView dffn_X, CView bndshape, DView Gx, DView dXdt,
                                   CView dXdto, CView dXdtoo) {
  XC_PDL_WAIT();
  for_tiles(Nz, Nx, [&](int j, int i) {
    if (j >= Nz || i >= Nx) return;
    double aX = AT(advn_X, j, i);
    AT(advn_rho, j, i) = aX + AT(advn_M, j, i);
    double gx = xc_mul(xc_mul(1.0 - AT(x, j, i), G0), AT(bndshape, j, i));
    AT(Gx, j, i) = gx;
    double dxdt = (-aX + AT(dffn_X, j, i)) + gx;
    AT(dXdt, j, i) = dxdt;
    double Xc = AT(X, j, i);
    double res = ((xc_mul(Xc, a1) - xc_mul(AT(Xo, j, i), a2)) - xc_mul(AT(Xoo, j, i), a3)) -
                 xc_mul((xc_mul(dxdt, b1) + xc_mul(AT(dXdto, j, i), b2)) + xc_mul(AT(dXdtoo, j, i), b3), dt);
    double upd = xc_div(xc_mul(res, -alpha), a1);
    double Xn = Xc + upd;
    double r = AT(rho, j, i);
    double lo = xc_mul(r, XC_EPS), hi = xc_mul(r, 1.0 - XC_EPS);
    Xn = Xn > hi ? hi : (Xn < lo ? lo : Xn);
    AT(X, j, i) = Xn;
    double Mn = r - Xn;
    AT(M, j, i) = Mn;
    AT(x, j, i) = xc_div(Xn, r);
    AT(m, j, i) = xc_div(Mn, r);
  });
}

template <class T>
dim3 tile_grid(int Nz, int Nx, int nz = 1) {
  return dim3((Nz + T::TZ - 1) / T::TZ, (Nx + T::TX - 1) / T::TX, nz);
}

template <class T, int S>
void launch_advect_tile(const FluxArgs& a, bool halod, int Nz, int Nx, int xBC, int zBC, double invh, bool pad,
                        cudaStream_t s) {
  if (halod)
    xc_launch(advect_tile_kernel<T, S, true>, tile_grid<T>(Nz, Nx), T::NT, 0, s, a, Nz, Nx, xBC, zBC, invh, pad);
  else
    xc_launch(advect_tile_kernel<T, S, false>, tile_grid<T>(Nz, Nx), T::NT, 0, s, a, Nz, Nx, xBC, zBC, invh, pad);
}

template <int S>
int launch_advect(const FluxArgs& a, bool halod, int Nz, int Nx, int xBC, int zBC, double invh, bool pad,
                  cudaStream_t s) {
  if (small_tile(kSmallAdvect, Nz, Nx))
    launch_advect_tile<SmallTile, S>(a, halod, Nz, Nx, xBC, zBC, invh, pad, s);
  else
    launch_advect_tile<LargeTile, S>(a, halod, Nz, Nx, xBC, zBC, invh, pad, s);
  XC_LAUNCH_CHECK();
  return XC_OK;
}

template <int S>
int launch_phsevo_fluxes(const PhsevoFluxes& p, int Nz, int Nx, int xBC, int zBC, double invh, cudaStream_t s) {
  if (small_tile(kSmallAdvect, Nz, Nx))
    xc_launch(phsevo_flux_kernel<SmallTile, S>, tile_grid<SmallTile>(Nz, Nx, 3), SmallTile::NT, 0, s, p, Nz, Nx, xBC,
              zBC, invh);
  else
    xc_launch(phsevo_flux_kernel<LargeTile, S>, tile_grid<LargeTile>(Nz, Nx, 3), LargeTile::NT, 0, s, p, Nz, Nx, xBC,
              zBC, invh);
  XC_LAUNCH_CHECK();
  return XC_OK;
}

int check_advect(int scheme, int Nz, int Nx) {
  int g = scheme_halo(scheme);
  if (g < 0) { xc_set_error("advect: unsupported scheme %d", scheme); return XC_BAD_ARG; }
  if (Nz < g || Nx < g) {
    xc_set_error("advect: grid %dx%d smaller than the scheme halo %d", Nz, Nx, g);
    return XC_BAD_ARG;
  }
  return XC_OK;
}

}  // namespace

int scheme_halo(int scheme) {
  switch (scheme) {
    case XC_CENTR: case XC_UPWD1: return 1;
    case XC_QUICK: case XC_FROMM: case XC_WENO3: case XC_TVDIM: return 2;
    case XC_WENO5: case kWeno5OneDiv: return 3;
    default: return -1;
  }
}

int stencil_advect_flux(const double* f, int ldf, bool halod, int Nz, int Nx, int scheme, int xBC,
                        int zBC, CView u, CView w, double h, DView adv, DView qx_int,
                        DView qz_int, cudaStream_t s, bool pad) {
  XC_TRY(check_advect(scheme, Nz, Nx));
  double invh = 1.0 / h;
  const FluxArgs a{f, ldf, u, w, nullptr, nullptr, adv, qx_int, qz_int};
  switch (scheme) {
    case XC_CENTR: return launch_advect<XC_CENTR>(a, halod, Nz, Nx, xBC, zBC, invh, pad, s);
    case XC_UPWD1: return launch_advect<XC_UPWD1>(a, halod, Nz, Nx, xBC, zBC, invh, pad, s);
    case XC_QUICK: return launch_advect<XC_QUICK>(a, halod, Nz, Nx, xBC, zBC, invh, pad, s);
    case XC_FROMM: return launch_advect<XC_FROMM>(a, halod, Nz, Nx, xBC, zBC, invh, pad, s);
    case XC_WENO3: return launch_advect<XC_WENO3>(a, halod, Nz, Nx, xBC, zBC, invh, pad, s);
    case XC_WENO5: return launch_advect<XC_WENO5>(a, halod, Nz, Nx, xBC, zBC, invh, pad, s);
    case kWeno5OneDiv: return launch_advect<kWeno5OneDiv>(a, halod, Nz, Nx, xBC, zBC, invh, pad, s);
    default: return launch_advect<XC_TVDIM>(a, halod, Nz, Nx, xBC, zBC, invh, pad, s);
  }
}

// diffusion of a halo'd field
static int diffus_launch(const double* f, const double* k, int ld, int Nz, int Nx, int xBC, int zBC, double h,
                         DView dff, DView qx, DView qz, bool pad, cudaStream_t s) {
  const FluxArgs a{f, ld, CView{nullptr, 0}, CView{nullptr, 0}, k, nullptr, dff, qx, qz};
  const double invh = 1.0 / h;
  if (small_tile(kSmallDiffus, Nz, Nx))
    xc_launch(diffus_tile_kernel<SmallTile, true>, tile_grid<SmallTile>(Nz, Nx), SmallTile::NT, 0, s, a, Nz, Nx, xBC,
              zBC, invh, pad);
  else
    xc_launch(diffus_tile_kernel<LargeTile, true>, tile_grid<LargeTile>(Nz, Nx), LargeTile::NT, 0, s, a, Nz, Nx, xBC,
              zBC, invh, pad);
  XC_LAUNCH_CHECK();
  return XC_OK;
}

// phsevo! (src/phsevo.jl:164-214)
int phsevo_impl(xc_ctx* c, int scheme, const double coefs[6], double dt, double alpha) {
  const int Nz = c->Nz, Nx = c->Nx, xBC = c->p.xBC, zBC = c->p.zBC;
  const double h = c->p.h;
  cudaStream_t s = c->stream;
  // face-velocity views: Wx[:, 2:end-1] (Nz+1, Nx), Ux[2:end-1, :] (Nz, Nx+1)
  DView Wx = F(c, FLD_Wx), Wm = F(c, FLD_Wm), Ux = F(c, FLD_Ux), Um = F(c, FLD_Um);
  CView Wx_face{Wx.p + Wx.ld, Wx.ld}, Wm_face{Wm.p + Wm.ld, Wm.ld};
  CView Ux_face{Ux.p + 1, Ux.ld}, Um_face{Um.p + 1, Um.ld};
  auto qx_int = [&](int id) { DView q = F(c, id); return DView{q.p + 1, q.ld}; };
  auto qz_int = [&](int id) { DView q = F(c, id); return DView{q.p + q.ld, q.ld}; };
  DView X = F(c, FLD_X), M = F(c, FLD_M);
  scheme = advect_scheme(scheme, c->p);
  XC_TRY(check_advect(scheme, Nz, Nx));
  const CView none{nullptr, 0};
  PhsevoFluxes pf{{{X.p, X.ld, Ux_face, Wx_face, nullptr, nullptr, F(c, FLD_advn_X), qx_int(FLD_qx_advn_X),
                    qz_int(FLD_qz_advn_X)},
                   {M.p, M.ld, Um_face, Wm_face, nullptr, nullptr, F(c, FLD_advn_M), qx_int(FLD_qx_advn_M),
                    qz_int(FLD_qz_advn_M)},
                   // diffusion of chi with k = X .* kx (phsevo.jl:192-194)
                   {F(c, FLD_chi).p, Nz, none, none, X.p, F(c, FLD_kx).p, F(c, FLD_dffn_X), qx_int(FLD_qx_dffn_X),
                    qz_int(FLD_qz_dffn_X)}}};
  const double invh = 1.0 / h;
  switch (scheme) {
    case XC_CENTR: XC_TRY(launch_phsevo_fluxes<XC_CENTR>(pf, Nz, Nx, xBC, zBC, invh, s)); break;
    case XC_UPWD1: XC_TRY(launch_phsevo_fluxes<XC_UPWD1>(pf, Nz, Nx, xBC, zBC, invh, s)); break;
    case XC_QUICK: XC_TRY(launch_phsevo_fluxes<XC_QUICK>(pf, Nz, Nx, xBC, zBC, invh, s)); break;
    case XC_FROMM: XC_TRY(launch_phsevo_fluxes<XC_FROMM>(pf, Nz, Nx, xBC, zBC, invh, s)); break;
    case XC_WENO3: XC_TRY(launch_phsevo_fluxes<XC_WENO3>(pf, Nz, Nx, xBC, zBC, invh, s)); break;
    case XC_WENO5: XC_TRY(launch_phsevo_fluxes<XC_WENO5>(pf, Nz, Nx, xBC, zBC, invh, s)); break;
    case kWeno5OneDiv: XC_TRY(launch_phsevo_fluxes<kWeno5OneDiv>(pf, Nz, Nx, xBC, zBC, invh, s)); break;
    default: XC_TRY(launch_phsevo_fluxes<XC_TVDIM>(pf, Nz, Nx, xBC, zBC, invh, s));
  }
  dim3 blk(32, 8);
  xc_launch(phsevo_tail_kernel, dim3(persistent_grid((const void*)phsevo_tail_kernel, Nz, Nx)), blk, 0, s, Nz, Nx,
      coefs[0], coefs[1], coefs[2], coefs[3],
      coefs[4], coefs[5], dt, alpha, c->p.G0,
      X, CF(c, FLD_Xo), CF(c, FLD_Xoo), M, F(c, FLD_x), F(c, FLD_m), CF(c, FLD_rho),
      CF(c, FLD_advn_X), CF(c, FLD_advn_M), F(c, FLD_advn_rho), CF(c, FLD_dffn_X),
      CF(c, FLD_bndshape), F(c, FLD_Gx), F(c, FLD_dXdt), CF(c, FLD_dXdto), CF(c, FLD_dXdtoo));
  XC_LAUNCH_CHECK();
  return XC_OK;
}

// ---------------------------------------------------------------------------
// C ABI: stencil-level entry points on caller device pointers
// ---------------------------------------------------------------------------
static bool bc_ok(int b) { return b == XC_PERIODIC || b == XC_CLOSED; }

extern "C" int xc_fill_ghosts(double* f, int Nz, int Nx, int halo, int zBC, int xBC, void* stream) {
  if (!f || Nz < halo || Nx < halo || halo < 1 || !bc_ok(zBC) || !bc_ok(xBC)) {
    xc_set_error("xc_fill_ghosts: bad arguments (Nz=%d Nx=%d halo=%d)", Nz, Nx, halo);
    return XC_BAD_ARG;
  }
  long long n = (long long)(Nz + 2 * halo) * (Nx + 2 * halo);
  xc_launch(fill_ghosts_kernel, (unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream, f, Nz, Nx, halo, zBC, xBC);
  XC_LAUNCH_CHECK();
  return XC_OK;
}

extern "C" int xc_advect(double* adv, const double* f_halo, const double* u, const double* w,
                         int Nz, int Nx, double h, int scheme, void* stream) {
  int g = scheme <= XC_TVDIM ? scheme_halo(scheme) : -1;   // the public scheme codes
  if (!adv || !f_halo || !u || !w || g < 0 || Nz < g || Nx < g) {
    xc_set_error("xc_advect: bad arguments (scheme=%d Nz=%d Nx=%d)", scheme, Nz, Nx);
    return XC_BAD_ARG;
  }
  CView uv{u, Nz}, wv{w, scheme == XC_TVDIM ? Nz + 3 : Nz + 1};
  return stencil_advect_flux(f_halo, Nz + 2 * g, true, Nz, Nx, scheme, XC_PERIODIC, XC_CLOSED, uv,
                             wv, h, DView{adv, Nz}, DView{nullptr, 0}, DView{nullptr, 0},
                             (cudaStream_t)stream);
}

extern "C" int xc_advect_with_flux(double* adv, double* qx, double* qz, const double* f_halo,
                                   const double* u, const double* w, int Nz, int Nx, double h,
                                   int scheme, int xBC, int zBC, void* stream) {
  int g = scheme <= XC_TVDIM ? scheme_halo(scheme) : -1;   // the public scheme codes
  if (!adv || !qx || !qz || !f_halo || !u || !w || g < 0 || Nz < g || Nx < g || !bc_ok(xBC) ||
      !bc_ok(zBC)) {
    xc_set_error("xc_advect_with_flux: bad arguments (scheme=%d Nz=%d Nx=%d)", scheme, Nz, Nx);
    return XC_BAD_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  CView uv{u, Nz}, wv{w, scheme == XC_TVDIM ? Nz + 3 : Nz + 1};
  return stencil_advect_flux(f_halo, Nz + 2 * g, true, Nz, Nx, scheme, xBC, zBC, uv, wv, h, DView{adv, Nz},
                             DView{qx + 1, Nz + 2}, DView{qz + (Nz + 1), Nz + 1}, s, true);
}

extern "C" int xc_advect_centered_with_flux(double* adv, double* qx, double* qz, const double* f,
                                            const double* u, const double* w, int Nz, int Nx,
                                            double h, int scheme, int xBC, int zBC, void* stream) {
  int g = scheme <= XC_TVDIM ? scheme_halo(scheme) : -1;   // the public scheme codes
  if (!adv || !f || !u || !w || g < 0 || Nz < g || Nx < g || !bc_ok(xBC) || !bc_ok(zBC) ||
      ((qx == nullptr) != (qz == nullptr))) {
    xc_set_error("xc_advect_centered_with_flux: bad arguments (scheme=%d Nz=%d Nx=%d)", scheme, Nz, Nx);
    return XC_BAD_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  CView uv{u, Nz}, wv{w, Nz + 1};
  DView qxi{qx ? qx + 1 : nullptr, Nz + 2}, qzi{qz ? qz + (Nz + 1) : nullptr, Nz + 1};
  return stencil_advect_flux(f, Nz, false, Nz, Nx, scheme, xBC, zBC, uv, wv, h, DView{adv, Nz}, qxi, qzi, s, true);
}

extern "C" int xc_diffus(double* dff, const double* f_halo, const double* k_halo, int Nz, int Nx,
                         double h, void* stream) {
  if (!dff || !f_halo || !k_halo || Nz < 1 || Nx < 1) {
    xc_set_error("xc_diffus: bad arguments");
    return XC_BAD_ARG;
  }
  return diffus_launch(f_halo, k_halo, Nz + 2, Nz, Nx, XC_PERIODIC, XC_CLOSED, h, DView{dff, Nz}, DView{nullptr, 0},
                       DView{nullptr, 0}, false, (cudaStream_t)stream);
}

extern "C" int xc_diffus_with_flux(double* dff, double* qx, double* qz, const double* f_halo,
                                   const double* k_halo, int Nz, int Nx, double h, int xBC,
                                   int zBC, void* stream) {
  if (!dff || !qx || !qz || !f_halo || !k_halo || Nz < 1 || Nx < 1 || !bc_ok(xBC) || !bc_ok(zBC)) {
    xc_set_error("xc_diffus_with_flux: bad arguments");
    return XC_BAD_ARG;
  }
  return diffus_launch(f_halo, k_halo, Nz + 2, Nz, Nx, xBC, zBC, h, DView{dff, Nz}, DView{qx + 1, Nz + 2},
                       DView{qz + (Nz + 1), Nz + 1}, true, (cudaStream_t)stream);
}
