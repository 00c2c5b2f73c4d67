// FP64 candidates, N = 768 .. 1536, with fixed-point transforms
// (pal_fx_kernels.cuh).  us per launch, first and second of a list, GB300: rows
// N=768 41.1 and 39.8, 1024 72.2 and 72.9; columns 1024 91.3 and 81.0, 1536
// 192 and 188.
#include "pal_launch.cuh"

using namespace pal;

namespace {
using P1152 = Plan<1152, 12, 12, 8>;
using P1152b = Plan<1152, 8, 12, 12>;
using P1536 = Plan<1536, 12, 16, 8>;
using P1536b = Plan<1536, 3, 8, 8, 8>;
using P1536c = Plan<1536, 8, 16, 12>;
using P1536d = Plan<1536, 8, 4, 4, 12>;
using P2304 = Plan<2304, 16, 12, 12>;
using P2304b = Plan<2304, 4, 6, 8, 12>;

const RowKernels r768[] = {RowFxOf<P1152, 2, 192>::make("12.12.8 V2x192 fx"),
                           RowFxOf<P1152b, 2, 192>::make("8.12.12 V2x192 fx")};
const ColKernels c768[] = {ColFxOf<P1152b, 192>::make("8.12.12 x192 fx")};
const RowKernels r1024[] = {RowFxOf<P1536, 1, 128>::make("12.16.8 V1x128 fx"),
                           RowFxOf<P1536b, 1, 192>::make("3.8.8.8 V1x192 fx")};
const ColKernels c1024[] = {ColFxOf<P1536c, 192>::make("8.16.12 x192 fx"),
                           ColFxOf<P1536d, 256>::make("8.4.4.12 x256 fx")};
const RowKernels r1536[] = {RowFxOf<P2304b, 1, 192>::make("4.6.8.12 V1x192 fx")};
const ColKernels c1536[] = {ColFxOf<P2304, 192>::make("16.12.12 x192 fx"),
                           ColFxOf<P2304b, 192>::make("4.6.8.12 x192 fx")};

PAL_KERNEL_SET(double, 1, 768, r768, c768)
PAL_KERNEL_SET(double, 1, 1024, r1024, c1024)
PAL_KERNEL_SET(double, 1, 1536, r1536, c1536)
}  // namespace

const KernelSet* pal_kernels_f64_b(int N) {
  switch (N) {
    case 768: return &kSet768;
    case 1024: return &kSet1024;
    case 1536: return &kSet1536;
    default: return nullptr;
  }
}
