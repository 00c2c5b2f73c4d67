// Launch wrappers and the autotuning candidates.
//
// For each (precision, N) the library compiles several row-pass and column-pass
// candidates that differ in radix order (the Plan), rows per tile (V, row pass
// only) and threads per block.  The two passes only share the data layout of
// the work planes, so they are chosen independently; each carries its own
// twiddle tables.  pal_create times every candidate on the handle's own state
// and keeps the fastest (pal_autotune in pal_api.cu).
#pragma once
#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "pal_fx_adjoint.cuh"

namespace pal {

struct RowKernels {
  const char* name;
  int V, NT;
  bool tma;  // stores through TMA: the launch needs StepArgs::tmaps
  size_t smem;
  int tw_elems;
  cudaError_t (*configure)();
  void (*row)(const StepArgs&, cudaStream_t);
  void (*phys)(const StepArgs&, cudaStream_t);
  void (*twiddles)(void* tw, cudaStream_t);
  int (*blocks_per_sm)();  // resident k_row blocks per SM (occupancy calculator)
  bool multicast = false;  // loads by TMA cluster multicast (tma_multicast_allowed)
};

struct ColKernels {
  const char* name;
  int NT;
  size_t smem;
  int tw_elems;
  cudaError_t (*configure)();
  void (*col)(const StepArgs&, cudaStream_t);
  void (*col_inv)(const StepArgs&, cudaStream_t);
  void (*twiddles)(void* tw, cudaStream_t);
  // the same pass on butterfly-major om / fnm1 (a.om_p, a.fm_p), and the
  // conversions between that order and the natural columns (om alone under
  // F_NO_FM_IN)
  void (*col_perm)(const StepArgs&, cudaStream_t);
  void (*to_perm)(const StepArgs&, cudaStream_t);
  void (*from_perm)(const StepArgs&, cudaStream_t);
  int (*blocks_per_sm)();  // resident k_col blocks per SM (occupancy calculator)
  bool tma;                // the butterfly-major pass moves its planes by TMA: the launch needs StepArgs::cmaps
  int rp;                  // last radix of the plan (pad groups of the TMA column tile)
};

// Adjoint of LS-IMEX-RK3 stages (pal_adjoint.cuh, pal_fx_adjoint.cuh), on fixed
// plans.  a.tw is the row or the column table as the kernel needs.
struct AdjKernels {
  int tw_row_elems, tw_col_elems;
  cudaError_t (*configure)();
  void (*vel)(const StepArgs&, cudaStream_t);      // om_p -> velocity planes y0, y1
  void (*fwd_row)(const StepArgs&, cudaStream_t);  // y0, y1 -> product planes w0, w1
  void (*fwd_col)(const StepArgs&, cudaStream_t);  // w0, w1, om_p, fm_p -> om_p, fm_p, y0, y1
  void (*col)(const StepArgs&, cudaStream_t);      // F_ADJ_OUT / F_ADJ_IN on om_p = lam_om, fm_p = lam_f, w0, w1
  void (*row)(const StepArgs&, cudaStream_t);      // lam planes w0, w1 with the velocity planes y0, y1
  void (*tw_row)(void* tw, cudaStream_t);
  void (*tw_col)(void* tw, cudaStream_t);
  void (*seed)(const void* om, void* lom, void* lf, double* loss_part, cudaStream_t);  // N/2 partials
  // columns between the natural and the adjoint plan's butterfly-major order (as ColKernels)
  void (*to_perm)(const StepArgs&, cudaStream_t);
  void (*from_perm)(const StepArgs&, cudaStream_t);
};

struct KernelSet {
  int N, M, precision;
  const RowKernels* rows;
  int n_rows;
  const ColKernels* cols;
  int n_cols;
  void (*spectral)(const StepArgs&, cudaStream_t, int blocks);
  void (*transpose)(const void* in, void* out, int rows, int cols, int batch, cudaStream_t);
  void (*spectrum)(const void* om, int N, int nbins, double r_max, double k_nyq, double scale2, double* esum, int* cnt,
                   int* edge, cudaStream_t);  // edge: nbins + 1 ints of scratch
  // display: |u| into plane 2 of `phys`, and min/max -> 8-bit pixels of one plane
  void (*speed)(void* phys, long long plane, cudaStream_t);
  void (*pixels)(const void* plane, long long n, double* part, unsigned int* counter, double* mm, unsigned char* pix,
                 cudaStream_t);
  const AdjKernels* adj;  // nullptr where no adjoint is compiled
};

// Whether this process is a run on one GPU alone: it sees one device, and no
// launcher says that it is one of several processes (a job on several GPUs
// usually gives each process one of them).
inline bool single_gpu_run() {
  for (const char* name : {"WORLD_SIZE", "LOCAL_WORLD_SIZE", "OMPI_COMM_WORLD_SIZE", "PMI_SIZE", "SLURM_NTASKS"}) {
    const char* v = std::getenv(name);
    if (v && std::atoi(v) > 1) return false;
  }
  int devices = 0;
  return cudaGetDeviceCount(&devices) == cudaSuccess && devices == 1;
}
// Row candidates that load by TMA cluster multicast are for such runs only: a
// job on several GPUs neither tunes to one nor may set one (pal_set_variant).
// PAL_TMA_MULTICAST=0 keeps the autotuners off them on one GPU too.
inline bool tma_multicast_allowed() {
  const char* e = std::getenv("PAL_TMA_MULTICAST");
  return !(e && e[0] == '0') && single_gpu_run();
}

constexpr int kSpectralThreads = 256;
constexpr size_t kSmemLimit = 227 * 1024;
constexpr size_t kLargeTile = 64 * 1024;  // tiles from this size on ask for the max shared carveout
// Bytes allocated after each work plane: the column pass's bulk tensor boxes
// reach 16 bytes past the last group of a row (ColPlanar), and this keeps
// every such byte inside the allocation.
constexpr size_t kPlaneSlack = 256;

// TMA descriptors of the planes w0 / w1 (members x N/2 rows x M complex FP32)
// for a row candidate with tile height V; false if the driver call is missing
// or refuses the layout.
bool encode_row_maps(TmaMaps* out, void* w0, void* w1, int N, int V, int members);
// Descriptors of w0 / w1 for k_col_tma: each a 3D view (2 RP floats, M / RP
// groups, N/2 x members rows) with a (2 RP + 4 floats, min(256, M / RP), 1)
// box, so one box row is a padded group of ColPlanar.
bool encode_col_maps(TmaMaps* out, void* w0, void* w1, int N, int RP, int members);

// Launch of a kernel that begins with pdl_wait() where EARLY is set: with
// EARLY the stream may bring its blocks onto the GPU while the previous kernel's
// last ones run, which saves the launch between two kernels (about 1.5 us).  The
// blocks that wait hold their SM's registers and shared memory, though, and
// where several streams share the GPU with small kernels that costs more: three
// N=256 FP64 fields side by side took 372 us a call with it and 293 without.  So
// early launches are for
// - FP32 passes of several waves (kEarlyM: N=4096 RK3 3.50 ms for four steps,
//   3.55 without; one N=1536 field alone 1.77 ms for ten, 1.92 without);
// - the adjoint's short dependent launches, but for FP64 from N=256 on (AdjOf).
//   ms for 20 steps, one gradient alone / three side by side in threads, with
//   early launches and without: FP32 N=32 1.02 / 1.09 and 1.67 / 1.98, N=128
//   1.39 / 1.51 and 2.19 / 2.37, N=256 1.75 / 2.18 and 2.27 / 2.91, N=512 2.61 /
//   3.60 and 3.21 / 3.89; FP64 N=32 2.77 / 2.85 and 3.24 / 3.73, N=128 3.48 /
//   4.44 and 3.88 / 4.65, N=256 4.38 / 6.62 and 4.38 / 6.02, N=512 9.78 / 14.5
//   and 8.32 / 14.1.
template <bool EARLY, class... P, class... A>
inline void launch_pdl(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = EARLY ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, args...);  // an error stays for the caller's cudaGetLastError
}

template <typename T, class PL>
void launch_twiddles(void* tw, cudaStream_t s) {
  k_twiddles<T, PL><<<(PL::TW_TOTAL + 255) / 256, 256, 0, s>>>(static_cast<cplx<T>*>(tw));
}

// Blocks of one kernel resident on the whole device at once (one wave).
template <class K>
inline int wave_blocks(K kernel, int nt, size_t smem) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, nt, smem) != cudaSuccess) return 0;
  return sms * per_sm;
}

// Blocks per member of a pass that loops over `tiles` tiles: at most one wave
// over all members, and tile counts that differ by at most one between blocks
// (0: the wave is not known).
inline int phys_blocks(int tiles, int wave, int members) {
  const int most = wave / members > 0 ? wave / members : tiles;
  if (most >= tiles) return tiles;
  const int rounds = (tiles + most - 1) / most;
  return (tiles + rounds - 1) / rounds;
}

// Column-pass flags of LS-IMEX-RK3 stage s (0..2) on butterfly-major om /
// fnm1: the first stage reads no fnm1, the first two hand the next stage its
// combined q in om (k_col F_Q_OUT / F_Q_IN), the last stores om and fn.
// `beta` is the stage table of beta coefficients.
__host__ __device__ inline void rk3_stage_flags(StepArgs& a, int s, const double* beta) {
  a.flags |= (s == 0 ? F_NO_FM_IN : F_Q_IN) | (s < 2 ? F_Q_OUT : 0);
  a.beta_next = s < 2 ? beta[s + 1] : 0.0;
}

template <typename T, class PL, int V, int NT, int PF = 0>
struct RowOf {
  static constexpr bool EARLY = early_plan<PL>();
  static constexpr size_t smem = std::max(size_t(PL::PADM) * V * sizeof(cplx<T>), size_t(2) * NT * sizeof(double));
  static_assert(smem <= kSmemLimit, "row tile does not fit in shared memory");
  static_assert(PL::M % V == 0, "row tile must divide M");
  static inline int ahead = 0;
  static cudaError_t configure() {
    cudaError_t e =
        cudaFuncSetAttribute(k_row<T, PL, V, NT, PF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    // tiles of 64 KB and more ask for the largest shared-memory carveout, so that
    // two of them are resident per SM whatever ran before; smaller tiles leave
    // the split to the driver (their L1 holds the twiddle tables and planes)
    if (smem >= kLargeTile) {
      e = cudaFuncSetAttribute(k_row<T, PL, V, NT, PF>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return e;
    }
    if (PF & 1) ahead = ((PF & 32) ? 2 : 1) * wave_blocks(k_row<T, PL, V, NT, PF>, NT, smem);
    return cudaFuncSetAttribute(k_phys<T, PL, V, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  }
  static void row(const StepArgs& a, cudaStream_t s) {
    StepArgs b = a;
    b.ahead = ahead;
    static const TmaMaps none{};
    launch_pdl<EARLY>(k_row<T, PL, V, NT, PF>, dim3(PL::M / V, a.members > 1 ? a.members : 1), NT, smem, s, b, ((PF & 12) != 0 && a.tmaps) ? *a.tmaps : none);
  }
  // k_phys: one wave of blocks shared by the members, each looping over its
  // member's tiles
  static void phys(const StepArgs& a, cudaStream_t s) {
    static std::atomic<int> wave{0};
    const int m = a.members > 1 ? a.members : 1;
    if (wave == 0) wave = wave_blocks(k_phys<T, PL, V, NT>, NT, smem);
    launch_pdl<EARLY>(k_phys<T, PL, V, NT>, dim3(phys_blocks(PL::M / V, wave, m), m), NT, smem, s, a);
  }
  static int blocks_per_sm() {
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_row<T, PL, V, NT, PF>, NT, smem) == cudaSuccess ? n : -1;
  }
  static constexpr RowKernels make(const char* name) {
    return RowKernels{name, V,   NT, (PF & 12) != 0, smem, PL::TW_TOTAL, configure, row, phys, launch_twiddles<T, PL>,
                      blocks_per_sm};
  }
};

template <typename T, class PL, int NT, int PREF = 0>
struct ColOf {
  static constexpr bool EARLY = early_plan<PL>();
  // PREF 4: the butterfly-major pass is k_col_tma (planar tile, TMA bulk
  // copies of the planes); the natural-order pass is the plain k_col.
  // PREF 5 / 6: the same with registers capped for three / two blocks per SM.
  // PREF 8: PREF 4 with the passes around the middle taking two butterflies
  // per thread at a time.
  static constexpr bool TMA = PREF == 4 || PREF == 5 || PREF == 6 || PREF == 8;
  static constexpr bool DUAL = PREF == 8;
  static constexpr int BASE = TMA ? 0 : PREF;
  static constexpr size_t smem_inv = size_t(PL::PADM) * 2 * sizeof(cplx<T>);
  static constexpr size_t smem = smem_inv + (BASE == 1 ? size_t(2) * (2 * PL::M / 3) * sizeof(cplx<T>) : 0);
  // the butterfly-major variant has no shared-memory om staging (PREF 1)
  static constexpr int PERM_PREF = BASE == 1 ? 0 : BASE;
  static constexpr size_t smem_tma = TMA ? size_t(2) * ColPlanar<PL>::PB * sizeof(cplx<T>) : 0;
  static constexpr int MINB = PREF == 5 ? 3 : PREF == 6 ? 2 : 0;
  static_assert(MINB * (smem_tma + 1024 + 256) <= size_t(228 * 1024), "the capped block count fits in shared memory");
  static_assert(smem <= kSmemLimit && smem_tma <= kSmemLimit, "column tile does not fit in shared memory");
  static cudaError_t configure() {
    cudaError_t e =
        cudaFuncSetAttribute(k_col<T, PL, NT, BASE, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if constexpr (TMA) {
      e = cudaFuncSetAttribute(k_col_tma<T, PL, NT, true, MINB, DUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_tma);
      if (e != cudaSuccess) return e;
      e = cudaFuncSetAttribute(k_col_tma<T, PL, NT, false, MINB, DUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_tma);
      if (e != cudaSuccess) return e;
      e = cudaFuncSetAttribute(k_col_tma<T, PL, NT, true, MINB, DUAL>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return e;
      e = cudaFuncSetAttribute(k_col_tma<T, PL, NT, false, MINB, DUAL>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return e;
    }
    e = cudaFuncSetAttribute(k_col<T, PL, NT, PERM_PREF, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_inv);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_col<T, PL, NT, PERM_PREF, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_inv);
    if (e != cudaSuccess) return e;
    if (smem_inv >= kLargeTile) {
      e = cudaFuncSetAttribute(k_col<T, PL, NT, PERM_PREF, true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               (int)cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return e;
      e = cudaFuncSetAttribute(k_col<T, PL, NT, PERM_PREF, true, false>,
                               cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return e;
    }
    e = cudaFuncSetAttribute(k_om_perm<T, PL, true, EARLY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_perm);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_om_perm<T, PL, false, EARLY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_perm);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_col_inv<T, PL, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_inv);
  }
  static dim3 grid(const StepArgs& a) { return dim3(a.N / 2, a.members > 1 ? a.members : 1); }
  static void col(const StepArgs& a, cudaStream_t s) { launch_pdl<EARLY>(k_col<T, PL, NT, BASE, false>, grid(a), NT, smem, s, a); }
  // RK3 stages carrying the combined term run the flag-aware instantiation;
  // every other butterfly-major column pass runs the plain update
  static void col_perm(const StepArgs& a, cudaStream_t s) {
    if constexpr (TMA) {
      static const TmaMaps none{};
      const TmaMaps& m = a.cmaps ? *a.cmaps : none;
      if (a.flags & (F_Q_IN | F_Q_OUT | F_NO_FM_IN))
        launch_pdl<EARLY>(k_col_tma<T, PL, NT, true, MINB, DUAL>, grid(a), NT, smem_tma, s, a, m);
      else
        launch_pdl<EARLY>(k_col_tma<T, PL, NT, false, MINB, DUAL>, grid(a), NT, smem_tma, s, a, m);
      return;
    }
    if (a.flags & (F_Q_IN | F_Q_OUT | F_NO_FM_IN))
      launch_pdl<EARLY>(k_col<T, PL, NT, PERM_PREF, true, true>, grid(a), NT, smem_inv, s, a);
    else
      launch_pdl<EARLY>(k_col<T, PL, NT, PERM_PREF, true, false>, grid(a), NT, smem_inv, s, a);
  }
  static constexpr size_t smem_perm = PermTile<T, PL>::smem;  // one om or fnm1 column
  static_assert(smem_perm <= kSmemLimit, "om / fnm1 column does not fit in shared memory");
  static dim3 grid_perm(const StepArgs& a) {
    const dim3 g = grid(a);
    return dim3(g.x, g.y, (a.flags & F_NO_FM_IN) ? 1 : 2);
  }
  static void to_perm(const StepArgs& a, cudaStream_t s) {
    launch_pdl<EARLY>(k_om_perm<T, PL, true, EARLY>, grid_perm(a), 256, smem_perm, s, a);
  }
  static void from_perm(const StepArgs& a, cudaStream_t s) {
    launch_pdl<EARLY>(k_om_perm<T, PL, false, EARLY>, grid_perm(a), 256, smem_perm, s, a);
  }
  static void col_inv(const StepArgs& a, cudaStream_t s) {
    launch_pdl<EARLY>(k_col_inv<T, PL, NT>, dim3(a.N / 2, a.members > 1 ? a.members : 1), NT, smem_inv, s, a);
  }
  static int blocks_per_sm() {
    int n = 0;
    cudaError_t e;
    if constexpr (TMA)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_col_tma<T, PL, NT, false, MINB, DUAL>, NT, smem_tma);
    else
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_col<T, PL, NT, PERM_PREF, true, false>, NT, smem_inv);
    return e == cudaSuccess ? n : -1;
  }
  static constexpr ColKernels make(const char* name) {
    return ColKernels{name,    NT,     smem,     PL::TW_TOTAL,          configure, col,
                      col_inv, launch_twiddles<T, PL>, col_perm, to_perm, from_perm, blocks_per_sm, TMA, PL::RP};
  }
};

// FP64 passes with fixed-point transforms (pal_fx_kernels.cuh).  MINB > 0 caps
// the registers so that MINB blocks share an SM.
template <class PL>
void launch_twiddles_fx(void* tw, cudaStream_t s) {
  using FP = FxPlan<PL>;
  if (FP::TW_TOTAL > 0) k_twiddles_fx<FP><<<(FP::TW_TOTAL + 127) / 128, 128, 0, s>>>(static_cast<int4*>(tw));
}

template <class K>
cudaError_t set_tile_smem(K kernel, size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess && smem >= kLargeTile)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  return e;
}

template <class PL, int V, int NT, int MINB = 0>
struct RowFxOf {
  using FP = FxPlan<PL>;
  static constexpr size_t smem = size_t(PL::PADM) * V * sizeof(fxc);
  static_assert(smem <= kSmemLimit && PL::M % V == 0 && NT % 32 == 0, "row tile, whole warps");
  static cudaError_t configure() {
    cudaError_t e = set_tile_smem(k_row_fx<FP, V, NT, MINB>, smem);
    return e == cudaSuccess ? set_tile_smem(k_phys_fx<FP, V, NT>, smem) : e;
  }
  static dim3 grid(const StepArgs& a) { return dim3(PL::M / V, a.members > 1 ? a.members : 1); }
  static void row(const StepArgs& a, cudaStream_t s) { k_row_fx<FP, V, NT, MINB><<<grid(a), NT, smem, s>>>(a); }
  static void phys(const StepArgs& a, cudaStream_t s) {
    static std::atomic<int> wave{0};
    const dim3 g = grid(a);
    if (wave == 0) wave = wave_blocks(k_phys_fx<FP, V, NT>, NT, smem);
    k_phys_fx<FP, V, NT><<<dim3(phys_blocks(g.x, wave, g.y), g.y), NT, smem, s>>>(a);
  }
  static int blocks_per_sm() {
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_row_fx<FP, V, NT, MINB>, NT, smem) == cudaSuccess ? n : -1;
  }
  static constexpr RowKernels make(const char* name) {
    return RowKernels{name, V, NT, false, smem, FP::TW_TOTAL, configure, row, phys, launch_twiddles_fx<PL>, blocks_per_sm};
  }
};

template <class PL, int NT, int MINB = 0>
struct ColFxOf {
  using FP = FxPlan<PL>;
  static constexpr size_t smem = size_t(PL::PADM) * 2 * sizeof(fxc);
  static constexpr size_t smem_perm = PermTile<double, PL>::smem;
  static_assert(smem <= kSmemLimit && smem_perm <= kSmemLimit && NT % 32 == 0, "column tile, whole warps");
  static cudaError_t configure() {
    cudaError_t e = set_tile_smem(k_col_fx<FP, NT, false, MINB>, smem);
    if (e == cudaSuccess) e = set_tile_smem(k_col_fx<FP, NT, true, MINB>, smem);
    if (e == cudaSuccess) e = set_tile_smem(k_col_inv_fx<FP, NT>, smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_om_perm<double, PL, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_perm);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_om_perm<double, PL, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_perm);
    return e;
  }
  static dim3 grid(const StepArgs& a) { return dim3(a.N / 2, a.members > 1 ? a.members : 1); }
  static dim3 grid_perm(const StepArgs& a) {
    const dim3 g = grid(a);
    return dim3(g.x, g.y, (a.flags & F_NO_FM_IN) ? 1 : 2);
  }
  static void col(const StepArgs& a, cudaStream_t s) { k_col_fx<FP, NT, false, MINB><<<grid(a), NT, smem, s>>>(a); }
  static void col_perm(const StepArgs& a, cudaStream_t s) { k_col_fx<FP, NT, true, MINB><<<grid(a), NT, smem, s>>>(a); }
  static void col_inv(const StepArgs& a, cudaStream_t s) { k_col_inv_fx<FP, NT><<<grid(a), NT, smem, s>>>(a); }
  static void to_perm(const StepArgs& a, cudaStream_t s) {
    k_om_perm<double, PL, true, false><<<grid_perm(a), 256, smem_perm, s>>>(a);
  }
  static void from_perm(const StepArgs& a, cudaStream_t s) {
    k_om_perm<double, PL, false, false><<<grid_perm(a), 256, smem_perm, s>>>(a);
  }
  static int blocks_per_sm() {
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_col_fx<FP, NT, true, MINB>, NT, smem) == cudaSuccess ? n : -1;
  }
  static constexpr ColKernels make(const char* name) {
    return ColKernels{name,     NT,      smem,      FP::TW_TOTAL,  configure, col, col_inv, launch_twiddles_fx<PL>,
                      col_perm, to_perm, from_perm, blocks_per_sm, false,     PL::RP};
  }
};

template <typename T, class PLR, int V, int NTR, class PLC, int NTC>
struct AdjOf {
  static constexpr bool FX = std::is_same_v<T, double>;
  static constexpr bool EARLY = !FX || PLC::M < 384;
  static constexpr size_t smem_fwd = size_t(PLR::PADM) * V * sizeof(cplx<T>);
  static constexpr size_t smem_row = 2 * smem_fwd;  // the lam and the velocity tile
  static constexpr size_t smem_col = size_t(PLC::PADM) * 2 * sizeof(cplx<T>);
  static constexpr size_t smem_perm = PermTile<T, PLC>::smem;
  static_assert(smem_row <= kSmemLimit && smem_col <= kSmemLimit, "adjoint tiles do not fit");
  static constexpr int N = 2 * PLC::M / 3;
  static cudaError_t configure() {
    cudaError_t e;
    if constexpr (FX) {
      e = set_tile_smem(k_adj_row_fx<FxPlan<PLR>, V, NTR>, smem_row);
      if (e == cudaSuccess) e = set_tile_smem(k_adj_fwd_row_fx<FxPlan<PLR>, V, NTR>, smem_fwd);
      if (e == cudaSuccess) e = set_tile_smem(k_adj_col_fx<FxPlan<PLC>, NTC>, smem_col);
      if (e == cudaSuccess) e = set_tile_smem(k_adj_fwd_col_fx<FxPlan<PLC>, NTC>, smem_col);
      if (e == cudaSuccess) e = set_tile_smem(k_adj_vel_fx<FxPlan<PLC>, NTC>, smem_col);
    } else {
      e = set_tile_smem(k_adj_row<T, PLR, V, NTR>, smem_row);
      if (e == cudaSuccess) e = set_tile_smem(k_adj_fwd_row<T, PLR, V, NTR>, smem_fwd);
      if (e == cudaSuccess) e = set_tile_smem(k_adj_col<T, PLC, NTC>, smem_col);
      if (e == cudaSuccess) e = set_tile_smem(k_adj_fwd_col<T, PLC, NTC>, smem_col);
      if (e == cudaSuccess) e = set_tile_smem(k_adj_vel<T, PLC, NTC>, smem_col);
    }
    if (e == cudaSuccess) e = set_tile_smem(k_om_perm<T, PLC, true, true>, smem_perm);
    if (e == cudaSuccess) e = set_tile_smem(k_om_perm<T, PLC, false, true>, smem_perm);
    return e;
  }
  static void vel(const StepArgs& a, cudaStream_t s) {
    if constexpr (FX)
      launch_pdl<EARLY>(k_adj_vel_fx<FxPlan<PLC>, NTC>, N / 2, NTC, smem_col, s, a);
    else
      launch_pdl<EARLY>(k_adj_vel<T, PLC, NTC>, N / 2, NTC, smem_col, s, a);
  }
  static void fwd_row(const StepArgs& a, cudaStream_t s) {
    if constexpr (FX)
      launch_pdl<EARLY>(k_adj_fwd_row_fx<FxPlan<PLR>, V, NTR>, PLR::M / V, NTR, smem_fwd, s, a);
    else
      launch_pdl<EARLY>(k_adj_fwd_row<T, PLR, V, NTR>, PLR::M / V, NTR, smem_fwd, s, a);
  }
  static void fwd_col(const StepArgs& a, cudaStream_t s) {
    if constexpr (FX)
      launch_pdl<EARLY>(k_adj_fwd_col_fx<FxPlan<PLC>, NTC>, N / 2, NTC, smem_col, s, a);
    else
      launch_pdl<EARLY>(k_adj_fwd_col<T, PLC, NTC>, N / 2, NTC, smem_col, s, a);
  }
  static void col(const StepArgs& a, cudaStream_t s) {
    if constexpr (FX)
      launch_pdl<EARLY>(k_adj_col_fx<FxPlan<PLC>, NTC>, N / 2, NTC, smem_col, s, a);
    else
      launch_pdl<EARLY>(k_adj_col<T, PLC, NTC>, N / 2, NTC, smem_col, s, a);
  }
  static void row(const StepArgs& a, cudaStream_t s) {
    if constexpr (FX)
      launch_pdl<EARLY>(k_adj_row_fx<FxPlan<PLR>, V, NTR>, PLR::M / V, NTR, smem_row, s, a);
    else
      launch_pdl<EARLY>(k_adj_row<T, PLR, V, NTR>, PLR::M / V, NTR, smem_row, s, a);
  }
  static void seed(const void* om, void* lom, void* lf, double* loss_part, cudaStream_t s) {
    k_adj_seed<T, PLC, 128><<<N / 2, 128, 0, s>>>(static_cast<const cplx<T>*>(om), static_cast<cplx<T>*>(lom),
                                                  static_cast<cplx<T>*>(lf), loss_part);
  }
  static dim3 grid_perm(const StepArgs& a) { return dim3(N / 2, 1, (a.flags & F_NO_FM_IN) ? 1 : 2); }
  static void to_perm(const StepArgs& a, cudaStream_t s) { launch_pdl<EARLY>(k_om_perm<T, PLC, true, true>, grid_perm(a), 256, smem_perm, s, a); }
  static void from_perm(const StepArgs& a, cudaStream_t s) {
    launch_pdl<EARLY>(k_om_perm<T, PLC, false, true>, grid_perm(a), 256, smem_perm, s, a);
  }
  static const AdjKernels* get() {
    if constexpr (FX) {
      static const AdjKernels k = {FxPlan<PLR>::TW_TOTAL, FxPlan<PLC>::TW_TOTAL, configure, vel, fwd_row, fwd_col, col, row,
                                   launch_twiddles_fx<PLR>, launch_twiddles_fx<PLC>, seed, to_perm, from_perm};
      return &k;
    } else {
      static const AdjKernels k = {PLR::TW_TOTAL, PLC::TW_TOTAL, configure, vel, fwd_row, fwd_col, col, row,
                                   launch_twiddles<T, PLR>, launch_twiddles<T, PLC>, seed, to_perm, from_perm};
      return &k;
    }
  }
};

template <typename T>
void launch_spectral(const StepArgs& a, cudaStream_t s, int blocks) {
  k_spectral<T, kSpectralThreads><<<dim3(blocks, a.members > 1 ? a.members : 1), kSpectralThreads, 0, s>>>(a);
}

template <typename T>
void launch_transpose(const void* in, void* out, int rows, int cols, int batch, cudaStream_t s) {
  dim3 grid((cols + 31) / 32, (rows + 31) / 32, batch);
  k_transpose<T><<<grid, dim3(32, 8), 0, s>>>(static_cast<const cplx<T>*>(in), static_cast<cplx<T>*>(out), rows,
                                              cols);
}

template <typename T>
void launch_spectrum(const void* om, int N, int nbins, double r_max, double k_nyq, double scale2, double* esum,
                     int* cnt, int* edge, cudaStream_t s) {
  const int nh = N / 2, kmax2 = (nh - 1) * (nh - 1) + nh * nh;
  k_spectrum_edges<32><<<nbins / 32 + 1, 32, 0, s>>>(edge, nbins, r_max, k_nyq, kmax2);
  k_spectrum<T, 128><<<nbins, 128, 0, s>>>(static_cast<const cplx<T>*>(om), N, edge, scale2, esum, cnt);
}

template <typename T>
void launch_speed(void* phys, long long plane, cudaStream_t s) {
  k_speed<T><<<1024, 256, 0, s>>>(static_cast<T*>(phys), plane);
}

template <typename T>
void launch_pixels(const void* plane, long long n, double* part, unsigned int* counter, double* mm, unsigned char* pix,
                   cudaStream_t s) {
  k_minmax<T, 256><<<512, 256, 0, s>>>(static_cast<const T*>(plane), n, part, counter, mm);
  k_pixels<T><<<1024, 256, 0, s>>>(static_cast<const T*>(plane), n, mm, pix);
}

#define PAL_KERNEL_SET(T, PREC, N, ROWS, COLS) PAL_KERNEL_SET_ADJ(T, PREC, N, ROWS, COLS, nullptr)
#define PAL_KERNEL_SET_ADJ(T, PREC, N, ROWS, COLS, ADJ)                                                 \
  static const ::pal::KernelSet kSet##N = {N,                                                           \
                                           3 * (N) / 2,                                                 \
                                           PREC,                                                        \
                                           ROWS,                                                        \
                                           (int)(sizeof(ROWS) / sizeof(ROWS[0])),                       \
                                           COLS,                                                        \
                                           (int)(sizeof(COLS) / sizeof(COLS[0])),                       \
                                           ::pal::launch_spectral<T>,                                   \
                                           ::pal::launch_transpose<T>,                                  \
                                           ::pal::launch_spectrum<T>,                                   \
                                           ::pal::launch_speed<T>,                                      \
                                           ::pal::launch_pixels<T>,                                     \
                                           ADJ};

// One launch per pass for an ensemble of several sizes (pal_ens_fused.cu).  The
// blocks of a pass are laid out group by group, member by member: group g's
// blocks start at `first`, `per_member` of them per member; every block
// decodes its (group, member, index) and runs that size's kernel body.
constexpr int kFusedMax = 4;
struct FusedGroupArgs {
  StepArgs a;      // the group's arguments (all of its members)
  int slot;        // which compiled size of the fused set this group is
  int first;       // first block of the group in the launch
  int per_member;  // blocks per member in this pass
};
struct FusedArgs {  // aligned as CUtensorMap
  TmaMaps maps[kFusedMax];  // row-tile TMA descriptors of each group
  FusedGroupArgs g[kFusedMax];
  int ngroups;
};
// A compiled set of sizes with fixed kernel candidates of one block size.
struct FusedSet {
  int nsizes;
  int N[kFusedMax];
  const char* row_name[kFusedMax];  // the KernelSet candidates whose twiddle tables (same plan)
  const char* col_name[kFusedMax];  // and TMA row layout (same tile height) the fused bodies use
  int V[kFusedMax];                 // row tile height of each size
  int NT;  // row-pass block size (the column passes may use another)
  size_t smem_row, smem_col, smem_perm;
  cudaError_t (*configure)();
  void (*row)(const FusedArgs&, int blocks, cudaStream_t);
  void (*col)(const FusedArgs&, int blocks, bool qm, cudaStream_t);  // qm: RK3 stages (ColOf::col_perm)
  void (*phys)(const FusedArgs&, int blocks, cudaStream_t);
  void (*to_perm)(const FusedArgs&, int blocks, cudaStream_t);
  void (*from_perm)(const FusedArgs&, int blocks, cudaStream_t);
};

}  // namespace pal

// The fused set holding every size in Ns (FP32), or nullptr.
const pal::FusedSet* pal_fused_set_f32(int n, const int* Ns);

// Per-precision lookup (pal_inst_f32.cu / pal_inst_f64.cu); nullptr if unsupported.
const pal::KernelSet* pal_kernels_f32(int N);
const pal::KernelSet* pal_kernels_f64(int N);
