// Reads lines of hexadecimal bit patterns and runs pal_sums.cuh on the host:
//   g <16 floats>      add_squares of eight points on an empty sum
//   p <n> <2 doubles>  add_point of n equal points on an empty sum
// and prints the bits of the running sum and of its compensation.
#include <cinttypes>
#include <cmath>
#include <cstdio>

#include "pal_sums.cuh"

int main() {
  char kind;
  while (std::scanf(" %c", &kind) == 1) {
    double acc = 0.0, comp = 0.0;
    if (kind == 'g') {
      float2 x[8];
      for (float2& p : x) {
        unsigned a, b;
        if (std::scanf("%x %x", &a, &b) != 2) return 1;
        p = float2{pal::bits_as<float>(a), pal::bits_as<float>(b)};
      }
      pal::add_squares(x, acc, comp);
    } else if (kind == 'p') {
      int n;
      uint64_t u, v;
      if (std::scanf("%d %" SCNx64 " %" SCNx64, &n, &u, &v) != 3) return 1;
      for (int i = 0; i < n; ++i) pal::add_point(pal::bits_as<double>(u), pal::bits_as<double>(v), acc, comp);
    } else {
      return 1;
    }
    std::printf("%016" PRIx64 " %016" PRIx64 "\n", pal::bits_as<uint64_t>(acc), pal::bits_as<uint64_t>(comp));
  }
}
