// Reads lines "nsteps ckpt_every plane_bytes"; prints the segment's length and the bytes of its planes.
#include <cstdio>

#include "pal_segments.h"

int main() {
  int n, c;
  unsigned long long b;
  while (std::scanf("%d %d %llu", &n, &c, &b) == 3) {
    const int seg = pal::adjoint_segment(n, c, b);
    std::printf("%d %llu\n", seg, (unsigned long long)pal::adjoint_planes(n, seg) * b);
  }
}
