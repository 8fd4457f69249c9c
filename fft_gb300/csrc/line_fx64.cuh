// FP64 lines computed in 64-bit block fixed point on the integer pipes.
//
// GB300 has two FP64 lanes per SM and clock against 64 lanes each of 64-bit
// integer adds and of 32x32+64-bit multiply-adds (measured: add.s64 59,
// mad.wide.s32 60, DADD 1.7, cvt to and from f64 2.0 results per SM and
// clock).  An FP64 transform that runs on the FP64 pipe is bound by it at
// about a tenth of what HBM allows.  Here a line's doubles become 64-bit
// integers that share one exponent, the stages run on those, and the results
// are rounded to double once at the end.
//
// Precision.  A line's values are held with the largest one's top bit at
// bit 59 or 60 (57 to 60 before the first stage, by what it may grow), so the
// unit is at most 2^-59 of the line's largest value (2^-57),
// against 2^-53 relative roundoff per FP64 operation.  Between two stages the
// line is shifted (by the largest magnitude, so no headroom is spent that
// the data do not need) to keep it that way.  Products by a twiddle use its
// 62-bit fixed-point value; the low x low partial product, at most a quarter
// unit, is dropped.  The error is therefore relative to the line's norm, as
// that of the FP64 butterflies is, and smaller.  Relative L2 error in 1e-16
// against extended-precision FFTs (FP64 butterflies in brackets): 4096 points
// normal 0.9 (2.3), uniform(0,1) 0.7 (2.1), the same with one 1e5 1.0 (2.2);
// real inverses of the spectra of 8192 and 16384 reals 10 + normal 1.1 and
// 1.6 (1.9).
// What it does not have is the luck of values that FP64 never adds to larger
// ones: a value 2^-k of its line's largest is held in 60 - k bits, so of a
// line whose large values cancel exactly (even elements 1, odd ones 1e-12),
// bins that only the small ones reach carry the line's error, not their own.
//
// Range.  Lines with a non-finite value, one above 2^977, or nonzero data
// below 2^-823 throughout are left to the FP64 body of the same kernel, so
// infinities, NaNs, overflow and subnormals behave as there; the other lines
// of their tile are not, so no line's result depends on its neighbours.
// (Zeros come out as +0, whatever the signs of the zeros that went in.)
//
// Bounds, in bits (component magnitudes; |z| is the complex magnitude): first
// stage's output |z| < 2^62.5, every intermediate < 2^63; before a twiddle
// product the line's top bit is bit 59 or 60 (59 before the last stage of a
// real forward pass; components < 2^61, |z| < 2^61.5); the product is scaled
// by 1/4: |z| < 2^59.5, and < 2^62.5 after the next radix-8 stage.
#pragma once

#include "line_fft64.cuh"

namespace agb {

typedef long long fx;

struct fxc {
  fx x, y;
};

// bit of the largest input component's leading one: as high as the first
// stage's growth allows (output |z| < 2^62.5; a lone radix-8 stage, whose
// output the real post-pass adds in pairs, one lower)
template <int LOGL>
constexpr int fx_top() {
  using Sc = Sched64<LOGL>;
  return Sc::FIRST == 2 ? 60 : Sc::FIRST == 4 ? 59 : Sc::NSTAGES > 1 ? 58 : 57;
}
constexpr int FX_TOP_MIN = 59, FX_TOP_MAX = 60;   // the same where a twiddle product follows; MIN before the last
                                                  // stage of a pass that adds its output in pairs, the real forward
constexpr int FX_TOP_C2R = 59;    // and of a real inverse's bins, before its pre-pass (which may grow them fourfold)
constexpr int FX_EXP_MIN = 200;   // biased exponents the fixed-point form takes: below, subnormal results are
constexpr int FX_EXP_MAX = 2000;  // possible; above, overflow (14 bits of growth) and non-finite values

__device__ __forceinline__ int fx_hi(fx a) { return (int)(a >> 32); }
__device__ __forceinline__ int fx_lo(fx a) { return (int)a; }
// a = fx_s1(a) * 2^32 + (signed) fx_lo(a)
__device__ __forceinline__ int fx_s1(fx a) { return fx_hi(a) + (int)((unsigned)fx_lo(a) >> 31); }
__device__ __forceinline__ fx mw(int a, int b) { return (fx)a * (fx)b; }
// a / 2^n to nearest, ties away from zero, or to even: a mean of half a tie
// would add up over a line to an error in bin 0.  Away where it is input 0 of
// a butterfly: of the products by 1 beside it those of inputs 1, 2 and 5 round
// ties away from zero and the others towards it (split62 in plan.cu), so that
// on data of one sign the eight have no mean, nor one large harmonic (the
// sign's DFT is 0, 2.8, 4, 2.8, 0; alternating signs put 1.3e-15 of 16384
// positive reals with a spike into one bin, these 0.9e-15, FP64 0.8e-15).
__device__ __forceinline__ fx fx_sar(fx a, int n) { return (a + (1LL << (n - 1)) + (a >> 63)) >> n; }
__device__ __forceinline__ fx fx_sar_even(fx a, int n) { return (a + ((1LL << (n - 1)) - 1) + ((a >> n) & 1)) >> n; }

__device__ __forceinline__ fxc cadd(fxc a, fxc b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ fxc csub(fxc a, fxc b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ fxc csub_i(fxc a, fxc b) { return {a.x + b.y, a.y - b.x}; }   // a - i b
__device__ __forceinline__ fxc cadd_i(fxc a, fxc b) { return {a.x - b.y, a.y + b.x}; }   // a + i b

// z * w / 4 (FULL: z * w), w = (int4){re high, re low, im high, im low} of the
// 62-bit fixed-point root: low words signed, never -2^31
template <bool FULL = false>
__device__ __forceinline__ fxc fx_cmul(fxc z, int4 w) {
  const int r1 = fx_s1(z.x), r0 = fx_lo(z.x), i1 = fx_s1(z.y), i0 = fx_lo(z.y);
  const int nz = -w.z, nw = -w.w;
  constexpr fx half = FULL ? 1LL << 29 : 1LL << 31;
  const fx m = half + mw(r1, w.y) + mw(r0, w.x) + mw(i1, nw) + mw(i0, nz);
  const fx n = half + mw(r1, w.w) + mw(r0, w.z) + mw(i1, w.y) + mw(i0, w.x);
  if constexpr (FULL)
    return {((mw(r1, w.x) + mw(i1, nz)) << 2) + (m >> 30), ((mw(r1, w.z) + mw(i1, w.x)) << 2) + (n >> 30)};
  else
    return {(fx)fx_hi(m) + mw(r1, w.x) + mw(i1, nz), (fx)fx_hi(n) + mw(r1, w.z) + mw(i1, w.x)};
}

// a * sqrt(1/2) as a - a * (1 - sqrt(1/2)), the factor's 64-bit fraction in two signed words
__device__ __forceinline__ fx fx_rsqrt2(fx a) {
  constexpr int c1 = 1257966796, c0 = 102865788;
  const int a1 = fx_s1(a), a0 = fx_lo(a);
  const fx m = (1LL << 31) + mw(a1, -c0) + mw(a0, -c1);
  return a + mw(a1, -c1) + (fx)fx_hi(m);
}

__device__ __forceinline__ void fx_dft4(fxc& a0, fxc& a1, fxc& a2, fxc& a3) {
  const fxc s02 = cadd(a0, a2), d02 = csub(a0, a2), s13 = cadd(a1, a3), d13 = csub(a1, a3);
  a0 = cadd(s02, s13);
  a2 = csub(s02, s13);
  a1 = csub_i(d02, d13);
  a3 = cadd_i(d02, d13);
}

template <int R>
__device__ __forceinline__ void fx_dft(fxc (&x)[R]) {
  if constexpr (R == 2) {
    const fxc t = x[0];
    x[0] = cadd(t, x[1]);
    x[1] = csub(t, x[1]);
  } else if constexpr (R == 4) {
    fx_dft4(x[0], x[1], x[2], x[3]);
  } else if constexpr (R == 8) {
    fx_dft4(x[0], x[2], x[4], x[6]);
    fx_dft4(x[1], x[3], x[5], x[7]);
    const fxc w1 = {fx_rsqrt2(x[3].x + x[3].y), fx_rsqrt2(x[3].y - x[3].x)};   // W8 x[3]
    const fxc w3 = {fx_rsqrt2(x[7].y - x[7].x), fx_rsqrt2(x[7].x + x[7].y)};   // conj(W8^3 x[7])
    const fxc y0 = cadd(x[0], x[1]), y4 = csub(x[0], x[1]);
    const fxc y1 = cadd(x[2], w1), y5 = csub(x[2], w1);
    const fxc y2 = csub_i(x[4], x[5]), y6 = cadd_i(x[4], x[5]);
    const fxc y3 = {x[6].x + w3.x, x[6].y - w3.y}, y7 = {x[6].x - w3.x, x[6].y + w3.y};
    x[0] = y0, x[1] = y1, x[2] = y2, x[3] = y3, x[4] = y4, x[5] = y5, x[6] = y6, x[7] = y7;
  }
}

__device__ __forceinline__ int d_hi(double v) { return __double2hiint(v); }

// The double's value in units of 2^(emax - 1023 - TOP), rounded to nearest
// (half a unit lost by each small value would add up in bin 0 of a positive
// line); emax: the line's largest biased exponent field
template <int TOP>
__device__ __forceinline__ fx fx_from(double v, int emax) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned m = (hi & 0xfffffu) | 0x100000u;
  const int sh = (int)(((unsigned)(emax + 62 - TOP) << 20) + 0xfffffu - (hi & 0x7fffffffu)) >> 20;
  unsigned long long u = ((unsigned long long)__funnelshift_l(lo, m, 11) << 32) | (lo << 11);
  asm("shr.u64 %0, %0, %1;" : "+l"(u) : "r"(sh));   // PTX clamps the amount: zeros and tiny values give 0
  const fx s = (fx)((int)hi >> 31);
  return (((fx)u ^ s) + 1) >> 1;   // u: twice the magnitude; -u = ~u + 1
}

// a * 2^sc as the nearest double (sc << 20 given; no subnormal or overflowing result in the range this form takes)
__device__ __forceinline__ double fx_to(fx a, int sc20) {
  const double d = (double)a;
  const int hi = __double2hiint(d);
  return __hiloint2double(hi ? hi + sc20 : 0, __double2loint(d));
}

// The values seen, for their largest magnitude: the largest and the smallest
// high word, two three-way instructions per value (against an OR of x ^ 2x,
// four: 4096-point rows x 4096 239.0 -> 237.0 us, 512 x 32768 165.7 -> 162.8,
// 2^20 r2c x 32 610 -> 600, 256^3 502.5 -> 498.2).  word(): its top bit is one
// above that magnitude's, also in an OR of several.
struct FxMag {
  int hi = 0, lo = 0;
  __device__ __forceinline__ void add(fxc z) {
    const int a = fx_hi(z.x), b = fx_hi(z.y);
    hi = __vimax3_s32(hi, a, b);
    lo = __vimin3_s32(lo, a, b);
  }
  __device__ __forceinline__ int word() const { return max(hi, ~lo) << 1; }
};

// One value per line reduced over the line's threads.  Lines inside one warp
// in rows mode (and one-thread lines) reduce in registers; others through a
// shared-memory word per line that the caller zeroed: publish(), a barrier
// the stages need anyway, read().
template <int T, int C, bool COLS>
struct FxLine {
  static constexpr bool REG = T == 1 || (!COLS && T <= 32);
  static __device__ __forceinline__ int in_regs_or(int v) {
    if constexpr (T == 32) return (int)__reduce_or_sync(0xffffffffu, (unsigned)v);
#pragma unroll
    for (int o = 1; o < T; o <<= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  static __device__ __forceinline__ int in_regs_max(int v) {
    if constexpr (T == 32) return __reduce_max_sync(0xffffffffu, v);
#pragma unroll
    for (int o = 1; o < T; o <<= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  }
  static __device__ __forceinline__ void publish_or(int v, int* slot, int c) {
    if constexpr (!COLS) {   // one line per warp
      v = (int)__reduce_or_sync(0xffffffffu, (unsigned)v);
      if ((threadIdx.x & 31) == 0) atomicOr(slot + c, v);
    } else {
      if constexpr (T * C >= 32) {
#pragma unroll
        for (int o = C; o < 32; o <<= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
        if (C >= 32 || (threadIdx.x & 31) < C) atomicOr(slot + c, v);
      } else {
        atomicOr(slot + c, v);
      }
    }
  }
  static __device__ __forceinline__ void publish_max(int v, int* slot, int c) {
    if constexpr (!COLS) {
      v = __reduce_max_sync(0xffffffffu, v);
      if ((threadIdx.x & 31) == 0) atomicMax(slot + c, v);
    } else {
      if constexpr (T * C >= 32) {
#pragma unroll
        for (int o = C; o < 32; o <<= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (C >= 32 || (threadIdx.x & 31) < C) atomicMax(slot + c, v);
      } else {
        atomicMax(slot + c, v);
      }
    }
  }
};

// the shared-memory exchange of line_fft64, its 16-byte elements as integer pairs
template <int L, int C, bool COLS>
struct FxSmem {
  Smem64<L, C, COLS> s;
  __device__ __forceinline__ void put(int c, int j, fxc v) const {
    *reinterpret_cast<longlong2*>(s.s + s.idx(c, j)) = make_longlong2(v.x, v.y);
  }
  __device__ __forceinline__ fxc get(int c, int j) const {
    const longlong2 v = *reinterpret_cast<const longlong2*>(s.s + s.idx(c, j));
    return {v.x, v.y};
  }
};

// bit of the largest magnitude of a line whose FxMag word is m
__device__ __forceinline__ int fx_top_of(int m) { return 62 - __clz(m); }

// Shift a line whose FxMag word is m to top bit MAX, the exponent following,
// unless it is near enough (normal data mostly stays within the range by
// itself: a radix-8 stage grows it by 1.5 bits, the product takes 2; a line
// that one value dominates does not grow)
template <int MAX, int E>
__device__ __forceinline__ void fx_level(fxc (&v)[E], int m, int& sc) {
  const int top = fx_top_of(m);
  if (top >= FX_TOP_MIN && top <= MAX) return;
  const int n = MAX - top;
  sc -= n;
  if (n > 0) {
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = {v[e].x << n, v[e].y << n};
  } else {
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = {fx_sar_even(v[e].x, -n), fx_sar_even(v[e].y, -n)};
  }
}

// the Stockham stages of run_stages64, with the line's exponent carried along
template <int LOGL, int C, bool COLS, bool WARP_ONLY, bool PAIRS, int S, class SM>
__device__ __forceinline__ void fx_stages(fxc (&v)[Sched64<LOGL>::E], int t, int c, const int4* tw, const SM& sm,
                                          int* slots, int& sc) {
  using Sc = Sched64<LOGL>;
  if constexpr (S < Sc::NSTAGES) {
    constexpr int R = Sc::radix(S), NS = Sc::ns(S), E = Sc::E, T = Sc::T, B = E / R;
    constexpr bool LAST = S == Sc::NSTAGES - 1;
    using Ln = FxLine<T, C, COLS>;
    FxMag seen;
#pragma unroll
    for (int u = 0; u < B; u++) {
      const int b = t + T * u;
      fxc x[R];
#pragma unroll
      for (int r = 0; r < R; r++) x[r] = v[u + B * r];
      if constexpr (NS > 1) {
        const int k = b & (NS - 1);
        x[0] = {fx_sar(x[0].x, 2), fx_sar(x[0].y, 2)};   // the same 1/4 as the products
#pragma unroll
        for (int r = 1; r < R; r++) x[r] = fx_cmul(x[r], __ldg(tw + Sc::twoff(S) + (r - 1) * NS + k));
      }
      fx_dft<R>(x);
      if constexpr (LAST) {
#pragma unroll
        for (int r = 0; r < R; r++) v[u + B * r] = x[r];
      } else {
        const int base = (b / NS) * NS * R + (b & (NS - 1));
#pragma unroll
        for (int r = 0; r < R; r++) {
          seen.add(x[r]);
          sm.put(c, base + r * NS, x[r]);
        }
      }
    }
    if constexpr (NS > 1) sc += 2;
    if constexpr (!LAST) {
      int mag = seen.word();
      if constexpr (Ln::REG) mag = Ln::in_regs_or(mag);
      else Ln::publish_or(mag, slots + (S + 1) * C, c);
      line_sync<WARP_ONLY>();   // this stage's scatter (and the line's magnitudes) are complete
#pragma unroll
      for (int e = 0; e < E; e++) v[e] = sm.get(c, t + T * e);
      if constexpr (!Ln::REG) mag = slots[(S + 1) * C + c];
      if constexpr (S + 1 < Sc::NSTAGES - 1) line_sync<WARP_ONLY>();   // every gather is done before the next scatter
      fx_level<PAIRS && S + 1 == Sc::NSTAGES - 1 ? FX_TOP_MIN : FX_TOP_MAX>(v, mag, sc);
      fx_stages<LOGL, C, COLS, WARP_ONLY, PAIRS, S + 1>(v, t, c, tw, sm, slots, sc);
    }
  }
}

// the FP64 body, for the lines the fixed-point form leaves to it
template <int LOGL, int C, bool COLS, int KIND, bool TSTORE>
__device__ __noinline__ void line_fft64_general(const LineParams& p, long long cta, const int* only) {
  line_fft64_body<LOGL, C, COLS, KIND, TSTORE>(p, cta, only);
}

// whether a line whose largest high word (sign off) is top goes there; 1: all zeros and subnormals
__device__ __forceinline__ bool fx_out_of_range(int top) {
  return (top >> 20) > FX_EXP_MAX || (top > 0 && (top >> 20) < FX_EXP_MIN);
}

// The kernel body for one CTA (C lines), arguments as line_fft64_body.
template <int LOGL, int C, bool COLS, int KIND, bool TSTORE>
__device__ __forceinline__ void line_fx64_body(const LineParams& p, long long cta) {
  using Sc = Sched64<LOGL>;
  constexpr int L = Sc::L, E = Sc::E, T = Sc::T;
  constexpr bool WARP_ONLY = (!COLS && T <= 32) || (T * C <= 32);
  using Ln = FxLine<T, C, COLS>;
  extern __shared__ __align__(1024) double2 smem64[];
  // row 0: largest exponents (then the lines' scales), rows 1..: ORs of the magnitudes after each stage but the
  // last, whose row has those of the real inverse's pre-pass
  __shared__ int slots[(Sc::NSTAGES + 1) * C];
  __shared__ int odd_of[C];   // lines left to the FP64 body
  FxSmem<L, C, COLS> sm{{smem64}};
  const int4* tw = reinterpret_cast<const int4*>(p.tw);
  const int4* rtw = reinterpret_cast<const int4*>(p.rtw);

  const int tid = threadIdx.x;
  const int c = COLS ? (tid % C) : (tid / T);
  const int t = T == 1 ? 0 : COLS ? (tid / C) : (tid % T);   // (one thread per line: bins 0 and L known to the compiler)
  const long long q = cta * C + c;
  const bool active = q < p.nlines;
  const long long base = active ? line_off(p.in, q) : 0;
  // inverse: the forward transform with re and im exchanged on both sides
  // (not for the C2R loads, whose pre-pass needs them in order)
  const bool swap = KIND == LK_C2R || (KIND == LK_C2C && p.inverse);
  const float* in_re = KIND != LK_C2R && swap ? p.in.im : p.in.re;
  const float* in_im = KIND != LK_C2R && swap ? p.in.re : p.in.im;
  float* out_re = swap ? p.out.im : p.out.re;
  float* out_im = swap ? p.out.re : p.out.im;

  double2 d[E];
#pragma unroll
  for (int e = 0; e < E; e++) d[e] = make_double2(0.0, 0.0);
  double dL = 0.0;   // C2R: the real part of bin L (thread 0 of the line)
  if (active) {
#pragma unroll
    for (int e = 0; e < E; e++) {
      const long long a = base + (long long)(t + T * e) * p.in.es;
      d[e] = make_double2(ldd(in_re, a), ldd(in_im, a));
    }
    if constexpr (KIND == LK_C2R) {
      if (t == 0) {
        d[0].y = 0.0;   // bins 0 and L count with their real parts only
        dL = ldd(p.in.re, base + (long long)L * p.in.es);
      }
    }
  }
  if constexpr (!Ln::REG) {
    for (int i = tid; i < (Sc::NSTAGES + 1) * C; i += T * C) slots[i] = 0;
    line_sync<WARP_ONLY>();
  }
  int top = KIND == LK_C2R ? d_hi(dL) & 0x7fffffff : 0;
#pragma unroll
  for (int e = 0; e < E; e++) top = max(top, max(d_hi(d[e].x) & 0x7fffffff, d_hi(d[e].y) & 0x7fffffff));
  if (top == 0) {   // subnormals too small to show in a high word
    int low = KIND == LK_C2R ? __double2loint(dL) : 0;
#pragma unroll
    for (int e = 0; e < E; e++) low |= __double2loint(d[e].x) | __double2loint(d[e].y);
    top = low != 0;
  }
  // a line goes by its largest value; the thread that holds it says so first
  const bool maybe = fx_out_of_range(top);
  if constexpr (Ln::REG) top = Ln::in_regs_max(top);
  else Ln::publish_max(top, slots, c);
  const bool rare = __syncthreads_or(maybe);
  if (rare) {
    const bool odd = fx_out_of_range(Ln::REG ? top : slots[c]);
    if (__syncthreads_and(odd || !active)) {   // no line is left to the fixed-point form
      line_fft64_general<LOGL, C, COLS, KIND, TSTORE>(p, cta, nullptr);
      return;
    }
    if (t == 0) odd_of[c] = odd;
  }
  if constexpr (!Ln::REG) top = slots[c];
  constexpr int TOP = fx_top<LOGL>();
  const int emax = max(top >> 20, FX_EXP_MIN);   // (a line of zeros: every element shifts out)
  int sc = emax - 1023 - TOP;

  fxc v[E];
  if constexpr (KIND == LK_C2R) {
    // Z'[i] = a - i*b as line_fft64_body, |Z'| up to four times the bins (<
    // 2^62.5), so the line is shifted to what the first stage takes only then,
    // when its magnitudes are known: where bin 0 dominates (data with a mean)
    // nothing grows, and two bits fewer from the start would cost it twice
    // the error of FP64 (8192 reals 10 + normal 9.0e-16, now 1.1e-16).
    // A pair of bins at a time, i from the lower half of the line
    // and L - i, whose a and b are the conjugates: Z'[L-i] = conj(a + i b).
    // The upper half's bins go through shared memory and its Z' come back the
    // same way (element L - i is this thread's alone in between).
    constexpr int IN = FX_TOP_C2R;
    sc += TOP - IN;
    FxMag seen;
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = {fx_from<IN>(d[e].x, emax), fx_from<IN>(d[e].y, emax)};
#pragma unroll
    for (int e = E / 2; e < E; e++) sm.put(c, t + T * e, v[e]);
    line_sync<WARP_ONLY>();
#pragma unroll
    for (int e = 0; e < E / 2; e++) {
      const int i = t + T * e;
      fxc z, zl;
      if (i == 0) {   // from the real parts of X[0] and X[L]; Z'[L/2] = 2 conj(X[L/2])
        const fx r1 = fx_from<IN>(dL, emax);
        z = {v[0].x + r1, v[0].x - r1};
        zl = {2 * v[E / 2].x, -2 * v[E / 2].y};
      } else {
        const fxc s0 = v[e], s1 = sm.get(c, L - i);
        int4 w = __ldg(rtw + i);
        w.z = -w.z;
        w.w = -w.w;
        const fxc a = {s0.x + s1.x, s0.y - s1.y};
        const fxc b = fx_cmul<true>({s1.x - s0.x, -s1.y - s0.y}, w);
        z = csub_i(a, b);
        zl = cadd_i(a, b);
        zl.y = -zl.y;
      }
      seen.add(z);
      seen.add(zl);
      v[e] = {z.y, z.x};
      sm.put(c, i == 0 ? L / 2 : L - i, {zl.y, zl.x});
    }
    int mag = seen.word();
    if constexpr (Ln::REG) mag = Ln::in_regs_or(mag);
    else Ln::publish_or(mag, slots + Sc::NSTAGES * C, c);
    line_sync<WARP_ONLY>();
#pragma unroll
    for (int e = E / 2; e < E; e++) v[e] = sm.get(c, t + T * e);
    if constexpr (!Ln::REG) mag = slots[Sc::NSTAGES * C + c];
    line_sync<WARP_ONLY>();   // before the stages write the buffer
    const int n = fx_top_of(mag) - TOP;
    if (n > 0) {
      sc += n;
#pragma unroll
      for (int e = 0; e < E; e++) v[e] = {fx_sar_even(v[e].x, n), fx_sar_even(v[e].y, n)};
    }
  } else {
#pragma unroll
    for (int e = 0; e < E; e++) {
      v[e] = {fx_from<TOP>(d[e].x, emax), fx_from<TOP>(d[e].y, emax)};
    }
  }

  fx_stages<LOGL, C, COLS, WARP_ONLY, KIND == LK_R2C, 0>(v, t, c, tw, sm, slots, sc);

  if constexpr (KIND == LK_C2C && TSTORE) {
    if constexpr (Sc::NSTAGES > 1) __syncthreads();
#pragma unroll
    for (int e = 0; e < E; e++) sm.put(c, t + T * e, v[e]);
    if (t == 0) slots[c] = sc;
    __syncthreads();
    const int c2 = tid / T, t2 = tid % T;
    const long long q2 = cta * C + c2;
    if (q2 < p.nlines && !(rare && odd_of[c2])) {
      const long long ob = line_off(p.out, q2);
      const int4* twf = reinterpret_cast<const int4*>(p.tw_full);
      const int r2 = (int)((q2 >> p.tw_qshift) & p.tw_qmask);
      const int sc20 = (slots[c2] + (p.tw_n ? 2 : 0)) * (1 << 20);
#pragma unroll
      for (int e = 0; e < E; e++) {
        const int k = t2 + T * e;
        fxc x = sm.get(c2, k);
        if (p.tw_n) x = fx_cmul(x, __ldg(twf + (long long)r2 * L + k));
        const long long a = ob + (long long)k * p.out.es;
        std_(out_re, a, fx_to(x.x, sc20));
        std_(out_im, a, fx_to(x.y, sc20));
      }
    }
  } else if constexpr (KIND == LK_R2C) {
    // real forward post-pass as line_fft64_body, a pair of bins at a time (k
    // from the lower half of the line, and L - k: X[L-k] = conj(h + i b))
    if constexpr (Sc::NSTAGES > 1) line_sync<WARP_ONLY>();
#pragma unroll
    for (int e = E / 2; e < E; e++) sm.put(c, t + T * e, v[e]);
    line_sync<WARP_ONLY>();
    if (active && !(rare && odd_of[c])) {
      const long long ob = line_off(p.out, q);
      const int sc20 = sc * (1 << 20);
      auto emit = [&](int k, fxc x) {
        const long long a = ob + (long long)k * p.out.es;
        std_(p.out.re, a, fx_to(x.x, sc20));
        std_(p.out.im, a, fx_to(x.y, sc20));
      };
#pragma unroll
      for (int e = 0; e < E / 2; e++) {
        const int k = t + T * e;
        const fxc s0 = v[e];
        if (k == 0) {   // X[0] and X[L] from Z[0]; X[L/2] = conj(Z[L/2])
          emit(0, {s0.x + s0.y, 0});
          emit(L, {s0.x - s0.y, 0});
          emit(L / 2, {v[E / 2].x, -v[E / 2].y});
        } else {
          const fxc s1 = sm.get(c, L - k);
          const fxc h = {fx_sar(s0.x + s1.x, 1), fx_sar(s0.y - s1.y, 1)};
          const fxc g = {fx_sar(s0.x - s1.x, 1), fx_sar(s0.y + s1.y, 1)};
          const fxc b = fx_cmul<true>(g, __ldg(rtw + k));
          const fxc y = cadd_i(h, b);
          emit(k, csub_i(h, b));
          emit(L - k, {y.x, -y.y});
        }
      }
    }
  } else {
    if constexpr (KIND == LK_C2C && COLS) {
      if (p.tw_n) {
        const int4* twf = reinterpret_cast<const int4*>(p.tw_full);
        const int r2 = (int)((q >> p.tw_qshift) & p.tw_qmask);
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = fx_cmul(v[e], __ldg(twf + (long long)r2 * L + t + T * e));
        sc += 2;
      }
    }
    if (active && !(rare && odd_of[c])) {
      const long long ob = line_off(p.out, q);
      const int sc20 = sc * (1 << 20);
#pragma unroll
      for (int e = 0; e < E; e++) {
        const long long a = ob + (long long)(t + T * e) * p.out.es;
        std_(out_re, a, fx_to(v[e].x, sc20));
        std_(out_im, a, fx_to(v[e].y, sc20));
      }
    }
  }
  // (after the others' stores, which go to other lines: a call before them
  // would cost every kernel 100 to 200 bytes of spills)
  if (rare && __syncthreads_or(odd_of[c])) line_fft64_general<LOGL, C, COLS, KIND, TSTORE>(p, cta, odd_of);
}

// 1024 resident threads (64 registers each): at the 80 to 120 registers the
// compiler takes on its own, 4096-point lines have one CTA per SM and no
// other's work under its barriers (4096 x 4096 c2c 0.346 vs 0.259 ms, 512^3-
// point real volumes 3% slower); 1280 threads spill (256-point lines 0.156 vs 0.171 ms)
template <int LOGL, int C, bool COLS, int KIND, bool TSTORE>
__global__ void __launch_bounds__(Sched64<LOGL>::T * C, 1024 / (Sched64<LOGL>::T * C)) line_fx64(const LineParams p) {
  pdl_enter();
  line_fx64_body<LOGL, C, COLS, KIND, TSTORE>(p, blockIdx.x);
}

}  // namespace agb
