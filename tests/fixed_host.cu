// Prints "R fx_bits in_dit pad" for every radix that a plan can be built of: the
// bits of the inputs of a pass without and, in a DIT pass, before its twiddles,
// and those of the first pass over a padded line.
#include <cstdio>

#include "pal_fx_kernels.cuh"

template <int R>
void line() {
  using PL = pal::FxPlan<pal::Plan<12 * R, R, 12>>;
  std::printf("%d %d %d %d\n", R, pal::fx_bits(R), pal::fx_in_bits<PL, 0, true>(), pal::fx_pad_bits(R));
}

int main() {
  line<2>();
  line<3>();
  line<4>();
  line<6>();
  line<8>();
  line<12>();
  line<16>();
  line<24>();
  line<32>();
}
