// FP64 elementwise kernels (standalone real pass, line copy, size-1 real
// transform) and the FP64 kernel lookup.  Same algebra and thread mapping as
// the FP32 ones in real_pass.cu (afft's real_pass, onedim.hpp:1031-1108,
// multi.hpp:343-414): thread (q, k), k in [0, L/2], owns the pair (k, L-k)
// of line q, so the pass may run in place.
#include "kernels64.h"
#include "line_fx64.cuh"

namespace agb {

namespace {

__device__ __forceinline__ double2 post_one64(double2 s0, double2 s1, double2 w) {
  const double2 a = make_double2(0.5 * (s0.x + s1.x), 0.5 * (s0.y - s1.y));
  const double2 d = make_double2(0.5 * (s0.x - s1.x), 0.5 * (s0.y + s1.y));
  return zadd(a, zmul_negi(zmul(d, w)));
}

__device__ __forceinline__ double2 pre_one64(double2 s0, double2 s1, double2 w) {
  const double2 a = zadd(s0, zconj(s1));
  const double2 b = zmul(zsub(zconj(s1), s0), zconj(w));
  return zadd(a, zmul_negi(b));
}

__device__ __forceinline__ double ld64(const float* base, long long off) {
  return reinterpret_cast<const double*>(base)[off];
}

}  // namespace

// The pair (line q, bin k in [0, L/2]) of thread idx of a real pass.  64-bit
// division only where the index needs it (the FP32 pass, bound by its loads,
// gains nothing from this).
__device__ __forceinline__ void real_pass_index(const RealPassParams& p, long long idx, long long* q, long long* k) {
  const long long half = p.L / 2 + 1;
  const long long n = p.lines_fastest ? p.nlines : half;
  long long a, b;   // idx = a * n + b
  if (p.nlines * half < 0xffff0000LL) {
    const unsigned m = (unsigned)idx / (unsigned)n;
    a = m;
    b = (unsigned)idx - m * (unsigned)n;
  } else {
    a = idx / n;
    b = idx - a * n;
  }
  *q = p.lines_fastest ? b : a;
  *k = p.lines_fastest ? a : b;
}

// One pair of bins in block fixed point (line_fx64.cuh), its four values
// sharing an exponent: FP64 instructions bound this pass on the FP64 pipe (32
// x 2^19 complex points 437 us of a 2^20-point real forward's 951).  One
// product serves both bins: bin L-k's a and b are the conjugates of bin k's
// (2^20 x 32 r2c 952 -> 610 us, c2r 918 -> 618, 2^15 x 512 r2c 419 -> 248).
// The values the fixed-point form leaves out take the FP64 form.
template <bool INVERSE>
__device__ __forceinline__ void pair64(double2 s0, double2 s1, const int4* rtw, long long k, long long L, double2* xk,
                                       double2* xl) {
  const int top = max(max(d_hi(s0.x) & 0x7fffffff, d_hi(s0.y) & 0x7fffffff),
                      max(d_hi(s1.x) & 0x7fffffff, d_hi(s1.y) & 0x7fffffff));
  const int emax = top >> 20;
  if (emax < FX_EXP_MIN || emax > FX_EXP_MAX) {
    *xk = INVERSE ? pre_one64(s0, s1, ldz(rtw + k)) : post_one64(s0, s1, ldz(rtw + k));
    *xl = INVERSE ? pre_one64(s1, s0, ldz(rtw + (L - k))) : post_one64(s1, s0, ldz(rtw + (L - k)));
    return;
  }
  constexpr int TOP = 59;   // components < 2^60: sums < 2^61, products < 2^62, results < 2^62.6
  int4 w = __ldg(rtw + k);
  const fxc u0 = {fx_from<TOP>(s0.x, emax), fx_from<TOP>(s0.y, emax)};
  const fxc u1 = {fx_from<TOP>(s1.x, emax), fx_from<TOP>(s1.y, emax)};
  const fxc a = {u0.x + u1.x, u0.y - u1.y};
  fxc b;
  int sc20;
  if constexpr (INVERSE) {
    w.z = -w.z;
    w.w = -w.w;
    b = fx_cmul<true>({u1.x - u0.x, -u1.y - u0.y}, w);
    sc20 = (emax - 1023 - TOP) * (1 << 20);
  } else {   // a and b are twice the pass's: the exponent has the 1/2
    b = fx_cmul<true>({u0.x - u1.x, u0.y + u1.y}, w);
    sc20 = (emax - 1023 - TOP - 1) * (1 << 20);
  }
  const fxc x = csub_i(a, b), y = cadd_i(a, b);   // a - i b; conj(a + i b)
  *xk = make_double2(fx_to(x.x, sc20), fx_to(x.y, sc20));
  *xl = make_double2(fx_to(y.x, sc20), fx_to(-y.y, sc20));
}

__global__ void real_pass_kernel64(const RealPassParams p) {
  pdl_enter();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long half = p.L / 2 + 1;
  long long q, k;
  real_pass_index(p, idx, &q, &k);
  if (q >= p.nlines || k >= half) return;
  const long long L = p.L;
  const int4* rtw = reinterpret_cast<const int4*>(p.rtw);
  const long long bi = line_off(p.in, q), bo = line_off(p.out, q);
  const long long ik = bi + k * p.in.es, iL = bi + (L - k) * p.in.es;
  const long long ok = bo + k * p.out.es, oL = bo + (L - k) * p.out.es;
  double* ore = reinterpret_cast<double*>(p.out.re);
  double* oim = reinterpret_cast<double*>(p.out.im);
  if (k == 0) {
    if (!p.inverse) {
      const double2 s0 = make_double2(ld64(p.in.re, ik), ld64(p.in.im, ik));
      ore[ok] = s0.x + s0.y;
      oim[ok] = 0.0;
      ore[oL] = s0.x - s0.y;
      oim[oL] = 0.0;
    } else {
      const double x0 = ld64(p.in.re, ik), xL = ld64(p.in.re, iL);
      ore[ok] = x0 + xL;
      oim[ok] = x0 - xL;
    }
    return;
  }
  const double2 s0 = make_double2(ld64(p.in.re, ik), ld64(p.in.im, ik));
  const double2 s1 = make_double2(ld64(p.in.re, iL), ld64(p.in.im, iL));
  double2 xk, xl;
  if (p.inverse) pair64<true>(s0, s1, rtw, k, L, &xk, &xl);
  else pair64<false>(s0, s1, rtw, k, L, &xk, &xl);
  ore[ok] = xk.x;
  oim[ok] = xk.y;
  if (L - k != k) {
    ore[oL] = xl.x;
    oim[oL] = xl.y;
  }
}

__global__ void copy_lines_kernel64(const CopyParams p) {
  pdl_enter();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= p.nlines * p.len) return;
  const long long q = idx / p.len, i = idx - q * p.len;
  const long long a = line_off(p.in, q) + i * p.in.es;
  const long long b = line_off(p.out, q) + i * p.out.es;
  reinterpret_cast<double*>(p.out.re)[b] = ld64(p.in.re, a);
  reinterpret_cast<double*>(p.out.im)[b] = ld64(p.in.im, a);
}

__global__ void real1_kernel64(const RealPassParams p) {
  pdl_enter();
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= p.nlines) return;
  const long long i = line_off(p.in, q), o = line_off(p.out, q);
  reinterpret_cast<double*>(p.out.re)[o] = ld64(p.in.re, i);
  if (!p.inverse) reinterpret_cast<double*>(p.out.im)[o] = 0.0;
}

bool get_line_kernel64(int logl, bool cols, int kind, bool tstore, LineKernel* out) {
  if (kind != LK_C2C && kind != LK_R2C && kind != LK_C2R) return false;
  if (!cols) return !tstore && get_rows64(logl, kind, out);
  return get_cols64(logl, kind, tstore, out);
}

}  // namespace agb
