// cols-mode complex line FFTs over interleaved pairs whose input tile is
// loaded by TMA: input pairs (one tensor map over the interleaved array),
// plain and with the transposing store, 2^8 to 2^10 points, and split input
// with output pairs (pass B of an interleaved or a long real inverse axis).
// Measured on GB300: interleaved 65536 x 4096 c2c 1.344 -> 1.318 ms, x 1001
// with the 256-point output pairs 0.335 -> 0.327 ms;
// interleaved 2^19 x 32 c2c 0.122 -> 0.108 ms, 2^20 x 64 c2r 0.315 -> 0.297
// ms with the 1024-point passes and the output pairs.
#include "kernels.h"
namespace agb {
template <int LOGL>
static bool tma_pairs_one(bool tstore, int pairs, LineKernel* out) {
  if (tstore && pairs == 1) *out = make_tma_kernel<LOGL, LK_C2C, 0, true, 1>();
  else if (tstore && pairs == 3) *out = make_tma_kernel<LOGL, LK_C2C, 0, true, 3>();
  else if (!tstore && pairs == 2) *out = make_tma_kernel<LOGL, LK_C2C, 0, false, 2>();
  else if (!tstore && pairs == 1) *out = make_tma_kernel<LOGL, LK_C2C, 0, false, 1>();
  else if (!tstore && pairs == 3) *out = make_tma_kernel<LOGL, LK_C2C, 0, false, 3>();
  else return false;
  return true;
}
bool get_cols_tma_pairs(int logl, bool tstore, int pairs, LineKernel* out) {
  switch (logl) {
    case 8: return tma_pairs_one<8>(tstore, pairs, out);
    case 9: return tma_pairs_one<9>(tstore, pairs, out);
    case 10: return tma_pairs_one<10>(tstore, pairs, out);
  }
  return false;
}
}  // namespace agb
