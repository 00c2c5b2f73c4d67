// FP64 candidates, N = 2048 and 3072, with fixed-point transforms
// (pal_fx_kernels.cuh).  us per launch, first and second of a list, GB300: rows
// N=2048 296 and 295, 3072 757 and 755; columns 2048 271 and 288.
#include "pal_launch.cuh"

using namespace pal;

namespace {
using P3072 = Plan<3072, 8, 6, 8, 8>;
using P3072b = Plan<3072, 8, 4, 8, 12>;
using P4608 = Plan<4608, 12, 6, 8, 8>;
using P4608b = Plan<4608, 8, 6, 8, 12>;

const RowKernels r2048[] = {RowFxOf<P3072, 2, 256, 2>::make("8.6.8.8 V2x256 fx occ"),
                           RowFxOf<P3072b, 2, 256, 2>::make("8.4.8.12 V2x256 fx occ")};
const ColKernels c2048[] = {ColFxOf<P3072b, 256, 2>::make("8.4.8.12 x256 fx occ"),
                           ColFxOf<P3072b, 384, 2>::make("8.4.8.12 x384 fx occ")};
const RowKernels r3072[] = {RowFxOf<P4608, 2, 384>::make("12.6.8.8 V2x384 fx"),
                           RowFxOf<P4608b, 2, 384>::make("8.6.8.12 V2x384 fx")};
const ColKernels c3072[] = {ColFxOf<P4608b, 384>::make("8.6.8.12 x384 fx")};

PAL_KERNEL_SET(double, 1, 2048, r2048, c2048)
PAL_KERNEL_SET(double, 1, 3072, r3072, c3072)
}  // namespace

const KernelSet* pal_kernels_f64_c(int N) {
  switch (N) {
    case 2048: return &kSet2048;
    case 3072: return &kSet3072;
    default: return nullptr;
  }
}
