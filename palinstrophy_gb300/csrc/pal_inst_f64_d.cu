// FP64 candidates, N = 4096, with fixed-point transforms
// (pal_fx_kernels.cuh).  us per launch, first and second of a list, GB300: rows
// 1243 and 1230, columns 1268 and 1302.
#include "pal_launch.cuh"

using namespace pal;

namespace {
using P6144 = Plan<6144, 8, 8, 8, 12>;
using P6144b = Plan<6144, 12, 8, 8, 8>;

const RowKernels r4096[] = {RowFxOf<P6144, 2, 512>::make("8.8.8.12 V2x512 fx"),
                           RowFxOf<P6144b, 2, 512>::make("12.8.8.8 V2x512 fx")};
const ColKernels c4096[] = {ColFxOf<P6144, 512>::make("8.8.8.12 x512 fx"),
                           ColFxOf<P6144, 384>::make("8.8.8.12 x384 fx")};

PAL_KERNEL_SET(double, 1, 4096, r4096, c4096)
}  // namespace

const KernelSet* pal_kernels_f64_d(int N) {
  switch (N) {
    case 4096: return &kSet4096;
    default: return nullptr;
  }
}
