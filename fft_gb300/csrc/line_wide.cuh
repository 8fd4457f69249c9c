// Passes of 512 and 1024 points with 32 points per thread and two stages
// (16 or 32, then 32 points) instead of 16 per thread and three, and rows of
// 8192 and 16384 points with three stages (8 or 16, 32, 32) instead of four.  Included by
// line_fft.cuh, whose kernels (and those of line_fft_pipe.cuh) take this
// schedule where is_wide says so.
//
// The three-stage kernels move every value through shared memory twice: the
// L1 / shared-memory pipe ran at 72 to 84% of its peak there while HBM ran at
// 36 to 55%.  One exchange halves that traffic and its barriers.  A thread
// holds 32 values (128 registers in all), so 512 threads fill an SM's
// registers, each with 32 loads in flight.
//
// Layout of the exchange: element j of line c at (j + j / R1) * C + c (8
// lines), so that the two rows a half-warp touches differ in parity in the
// scatter (rows R1 apart) and in the gather (neighbouring rows); 16 lines are
// one row per half-warp and need no padding.  With the transposing store the
// column is XORed with j / 2 (8 lines) or j (16), so that 16 elements along
// one line spread over all banks.
#pragma once

namespace agb {

template <int LOGL>
struct Wide {
  static_assert(LOGL == 9 || LOGL == 10 || LOGL == 13 || LOGL == 14,
                "16 x 32, 32 x 32, 8 x 32 x 32 or 16 x 32 x 32 points");
  static constexpr int L = 1 << LOGL, E = 32, T = L / E, NSTAGES = LOGL <= 10 ? 2 : 3;
  static constexpr int R1 = LOGL <= 10 ? L / 32 : L / 1024;   // first stage's radix; the others are 32
  static constexpr int radix(int s) { return s == 0 ? R1 : 32; }
  static constexpr int ns(int s) { return s == 0 ? 1 : s == 1 ? R1 : 32 * R1; }
  // stage twiddles as Sched's: W_{NS R}^{r k} at [twoff(s) + (r - 1) * NS + k]
  static constexpr int twoff(int s) { return s <= 1 ? 0 : 31 * R1; }
  static constexpr int twsize() { return NSTAGES == 2 ? 31 * R1 : 31 * R1 * 33; }
};

template <int LOGL, int C, bool XOR>
struct WideSmem {
  static_assert(C == 8 || C == 16, "8 or 16 lines");
  static constexpr int R1 = Wide<LOGL>::R1;
  static constexpr int ROWS = Wide<LOGL>::L + (C == 8 ? 32 : 0);
  static constexpr int FLOAT2S = ROWS * C;
  float2* s;
  __device__ __forceinline__ int idx(int c, int j) const {
    const int row = C == 8 ? j + j / R1 : j;
    const int col = !XOR ? c : C == 8 ? c ^ ((j >> 1) & 7) : c ^ (j & 15);
    return row * C + col;
  }
  __device__ __forceinline__ void put(int c, int j, float2 v) const { s[idx(c, j)] = v; }
  __device__ __forceinline__ float2 get(int c, int j) const { return s[idx(c, j)]; }
};

// Rows mode: line c at c * LP.  Two stages: element j at j + j / R1, a
// half-warp's 16 consecutive threads of one line scatter R1 + 1 apart and gather
// side by side.  Three stages: j + j / 16 + 8 (j / 256), conflict-free for the
// first stage's scatter (stride 8 or 16), the second's (8 or 16 neighbours,
// groups of 8 going 256 apart) and the gather.
template <int LOGL, int C>
struct WideRowSmem {
  static constexpr int R1 = Wide<LOGL>::R1, L = Wide<LOGL>::L;
  static constexpr int LP = LOGL <= 10 ? L + 32 : L + L / 16 + 8 * (L / 256), FLOAT2S = C * LP;
  float2* s;
  __device__ __forceinline__ int idx(int c, int j) const {
    if constexpr (LOGL <= 10) return c * LP + j + j / R1;
    else return c * LP + j + (j >> 4) + ((j >> 8) << 3);
  }
  __device__ __forceinline__ void put(int c, int j, float2 v) const { s[idx(c, j)] = v; }
  __device__ __forceinline__ float2 get(int c, int j) const { return s[idx(c, j)]; }
};

// W32^K a, K = n1 k2 of the DFT-32's 4 x 8 split
template <int K>
__device__ __forceinline__ float2 w32(float2 a) {
  // cos(pi k / 16), k = 0 .. 8
  constexpr float cs[9] = {1.f, 0.98078528040323044f, AFFT_C8, 0.83146961230254524f, AFFT_R2, 0.55557023301960218f,
                           AFFT_S8, 0.19509032201612825f, 0.f};
  static_assert(K <= 21, "n1 < 4, k2 < 8");
  static_assert(K != 4 && K != 12, "these go by w8s");
  if constexpr (K % 8 == 0 && K < 16) return w16<K / 2>(a);
  else {
    constexpr float x = K < 8 ? cs[K] : K < 16 ? -cs[16 - K] : -cs[K - 16];
    constexpr float y = K < 8 ? -cs[8 - K] : K < 16 ? -cs[K - 8] : cs[24 - K];
    return cmulc<(x * x >= y * y)>(a, x, y);
  }
}

// The DFT-32's second half for one k2: twiddles W32^(n1 k2) and a DFT-4 over n1
template <bool PK, int K2>
__device__ __forceinline__ void dft32_col(float2 (&x)[32], const float2 (&a)[4][8]) {
  if constexpr (K2 < 8) {
    x[K2] = a[0][K2];
    if constexpr (K2 == 4) {
      x[K2 + 8] = w8s<1>(a[1][K2]);
      x[K2 + 24] = w8s<3>(a[3][K2]);
    } else {
      x[K2 + 8] = w32<K2>(a[1][K2]);
      x[K2 + 24] = w32<3 * K2>(a[3][K2]);
    }
    if constexpr (K2 == 2 || K2 == 6) x[K2 + 16] = w8s<K2 / 2>(a[2][K2]);
    else x[K2 + 16] = w32<2 * K2>(a[2][K2]);
    dft4_8<PK, K2 == 2 || K2 == 6, K2 == 4>(x[K2], x[K2 + 8], x[K2 + 16], x[K2 + 24]);
    dft32_col<PK, K2 + 1>(x, a);
  }
}

// in-place DFT-32, natural order in and out: n = n1 + 4 n2, k = k2 + 8 k1, 16
// full products and 12 by W8.  (As two DFT-16 and a last radix-2 step, 20
// full products and 10 by W8, each rounded by itself: 1024-point lines were
// off by 1.16e-7 of their norm instead of 1.09e-7, 1.11e-7 in three stages of 4,
// 16 and 16.)
template <bool PK>
__device__ __forceinline__ void dft32(float2 (&x)[32]) {
  float2 a[4][8];
#pragma unroll
  for (int i = 0; i < 32; i++) a[i & 3][i >> 2] = x[i];
#pragma unroll
  for (int n1 = 0; n1 < 4; n1++) dft<8, PK>(a[n1]);
  dft32_col<PK, 0>(x, a);
}

// Stage 1 in registers: output r of butterfly b = t + T u (u < 32 / R1) of
// the canonical values, element b * R1 + r, in v[u + (32 / R1) r].
template <int LOGL, bool PK>
__device__ __forceinline__ void wide_stage1(float2 (&v)[32]) {
  constexpr int R1 = Wide<LOGL>::R1, B1 = 32 / R1;
#pragma unroll
  for (int u = 0; u < B1; u++) {
    float2 x[R1];
#pragma unroll
    for (int r = 0; r < R1; r++) x[r] = v[u + B1 * r];
    if constexpr (R1 == 32) dft32<PK>(x);
    else dft<R1, PK>(x);
#pragma unroll
    for (int r = 0; r < R1; r++) v[u + B1 * r] = x[r];
  }
}

// The last stage on the gathered canonical values (butterfly t, k = t: T = NS)
template <int LOGL, bool PK>
__device__ __forceinline__ void wide_last(float2 (&v)[32], int t, const float2* tw) {
  constexpr int T = Wide<LOGL>::T;
  static_assert(T == Wide<LOGL>::ns(Wide<LOGL>::NSTAGES - 1), "one last-stage butterfly per thread");
#pragma unroll
  for (int r = 1; r < 32; r++) v[r] = cmul(v[r], ldg2(tw + (r - 1) * T + t));
  dft32<PK>(v);
}

// All stages, canonical layout in and out (as run_stages)
template <int LOGL, bool PK, bool WARP_ONLY, class SM>
__device__ __forceinline__ void wide_stages(float2 (&v)[32], int t, int c, const float2* tw, const SM& sm) {
  constexpr int R1 = Wide<LOGL>::R1, B1 = 32 / R1, T = Wide<LOGL>::T;
  wide_stage1<LOGL, PK>(v);
#pragma unroll
  for (int u = 0; u < B1; u++)
#pragma unroll
    for (int r = 0; r < R1; r++) sm.put(c, (t + T * u) * R1 + r, v[u + B1 * r]);
  line_sync<WARP_ONLY>();
#pragma unroll
  for (int e = 0; e < 32; e++) v[e] = sm.get(c, t + T * e);
  if constexpr (Wide<LOGL>::NSTAGES == 3) {
    line_sync<WARP_ONLY>();   // every gather is done before the next scatter
    const int k = t & (R1 - 1);
#pragma unroll
    for (int r = 1; r < 32; r++) v[r] = cmul(v[r], ldg2(tw + (r - 1) * R1 + k));
    dft32<PK>(v);
    const int base = (t / R1) * (32 * R1) + k;
#pragma unroll
    for (int r = 0; r < 32; r++) sm.put(c, base + r * R1, v[r]);
    line_sync<WARP_ONLY>();
#pragma unroll
    for (int e = 0; e < 32; e++) v[e] = sm.get(c, t + T * e);
  }
  wide_last<LOGL, PK>(v, t, tw + Wide<LOGL>::twoff(Wide<LOGL>::NSTAGES - 1));
}

}  // namespace agb
