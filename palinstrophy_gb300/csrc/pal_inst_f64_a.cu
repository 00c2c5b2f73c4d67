// FP64 candidates, N = 32 .. 512, with fixed-point transforms
// (pal_fx_kernels.cuh, pal_fx_adjoint.cuh).  us per launch with the launch
// itself, first and second of a list, GB300: columns N=32 16.17 and 16.25, 256
// 20.1 and 21.9; rows 512 22.6 and 22.7.  The second ones are near enough to
// trade places on a shared GPU.
#include "pal_launch.cuh"

using namespace pal;

namespace {
using P48b = Plan<48, 6, 8>;
using P48c = Plan<48, 4, 12>;
using P96 = Plan<96, 6, 16>;
using P96c = Plan<96, 8, 12>;
using P192d = Plan<192, 4, 4, 12>;
using P384b = Plan<384, 6, 8, 8>;
using P384d = Plan<384, 4, 8, 12>;
using P576 = Plan<576, 6, 6, 16>;
using P576c = Plan<576, 6, 8, 12>;
using P768c = Plan<768, 12, 8, 8>;
using P768d = Plan<768, 8, 8, 12>;

const RowKernels r32[] = {RowFxOf<P48b, 2, 32>::make("6.8 V2x32 fx")};
const ColKernels c32[] = {ColFxOf<P48b, 32>::make("6.8 x32 fx"),
                           ColFxOf<P48c, 32>::make("4.12 x32 fx")};
const RowKernels r64[] = {RowFxOf<P96, 2, 64>::make("6.16 V2x64 fx")};
const ColKernels c64[] = {ColFxOf<P96c, 64>::make("8.12 x64 fx")};
const RowKernels r128[] = {RowFxOf<P192d, 2, 96>::make("4.4.12 V2x96 fx")};
const ColKernels c128[] = {ColFxOf<P192d, 96>::make("4.4.12 x96 fx")};
const RowKernels r256[] = {RowFxOf<P384b, 2, 128>::make("6.8.8 V2x128 fx")};
const ColKernels c256[] = {ColFxOf<P384b, 128>::make("6.8.8 x128 fx"),
                           ColFxOf<P384d, 96>::make("4.8.12 x96 fx")};
const RowKernels r384[] = {RowFxOf<P576, 2, 128>::make("6.6.16 V2x128 fx")};
const ColKernels c384[] = {ColFxOf<P576c, 192>::make("6.8.12 x192 fx")};
const RowKernels r512[] = {RowFxOf<P768d, 2, 192>::make("8.8.12 V2x192 fx"),
                           RowFxOf<P768c, 2, 192>::make("12.8.8 V2x192 fx")};
const ColKernels c512[] = {ColFxOf<P768d, 192>::make("8.8.12 x192 fx")};

PAL_KERNEL_SET_ADJ(double, 1, 32, r32, c32, (AdjOf<double, P48b, 2, 32, P48c, 32>::get()))
PAL_KERNEL_SET_ADJ(double, 1, 64, r64, c64, (AdjOf<double, P96, 2, 64, P96c, 64>::get()))
PAL_KERNEL_SET_ADJ(double, 1, 128, r128, c128, (AdjOf<double, P192d, 2, 96, P192d, 96>::get()))
PAL_KERNEL_SET_ADJ(double, 1, 256, r256, c256, (AdjOf<double, P384b, 2, 128, P384b, 128>::get()))
PAL_KERNEL_SET(double, 1, 384, r384, c384)
PAL_KERNEL_SET_ADJ(double, 1, 512, r512, c512, (AdjOf<double, P768d, 2, 192, P768d, 192>::get()))
}  // namespace

const KernelSet* pal_kernels_f64_a(int N) {
  switch (N) {
    case 32: return &kSet32;
    case 64: return &kSet64;
    case 128: return &kSet128;
    case 256: return &kSet256;
    case 384: return &kSet384;
    case 512: return &kSet512;
    default: return nullptr;
  }
}
