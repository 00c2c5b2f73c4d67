// Segments of the adjoint's sweeps (pal_adjoint_palinstrophy).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>

namespace pal {

// Padded planes that a call holds for segments of `seg` steps: om and fnm1 at the
// start of every segment but the last, and the two velocity planes of each of the
// three stages of every step of one segment.
inline std::size_t adjoint_planes(std::size_t nsteps, std::size_t seg) {
  return 2 * ((nsteps + seg - 1) / seg - 1) + 6 * seg;
}

// Steps of a segment: ckpt_every while the planes stay below 1 GiB.  Beyond
// that sqrt(nsteps / 3), which needs the least memory: a segment is run forward
// once more whatever its length, so the length costs no time.  (50000 steps of
// N=512 FP64 with a checkpoint at every one would hold 315 GB; the least is 5.)
inline int adjoint_segment(int nsteps, int ckpt_every, std::size_t plane_bytes) {
  const std::size_t n = nsteps, seg = std::min(nsteps, ckpt_every);
  if (adjoint_planes(n, seg) * plane_bytes <= (std::size_t(1) << 30)) return (int)seg;
  const std::size_t least = std::max<std::size_t>(1, std::llround(std::sqrt(n / 3.0)));
  return (int)(adjoint_planes(n, least) < adjoint_planes(n, seg) ? least : seg);
}

}  // namespace pal
