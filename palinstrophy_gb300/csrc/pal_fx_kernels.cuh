// The passes of the FP64 form with their transforms in 64-bit block fixed point
// (pal_fixed.cuh): the same tiles, plans and work planes as the kernels of
// pal_kernels.cuh, FP64 in HBM on both sides.  The spectral update, the
// statistics and the diagnostics stay FP64.
//
// A tile in shared memory holds either FP64 values ("raw", before a scaled
// pass) or integers with one exponent for the tile.  A pass reads its inputs
// shifted below 2^fx_bits(R), runs the butterfly, and notes the largest word of
// its outputs; the next pass shifts by it.  A tile with a NaN or an
// infinity runs on zeros and stores NaN everywhere, as an FP64 transform does.
#pragma once
#include "pal_kernels.cuh"

namespace pal {

// The plan with its tables in fixed point: pass p < NP - 1 holds
// W_{L_p}^(i k), 1 <= k < R_p, as [k - 1][i], so that the lanes of a warp, which
// hold consecutive butterflies i, read consecutive 16-byte entries.
template <class PL>
struct FxPlan : PL {
  static constexpr int tw_off(int p) {
    int o = 0;
    for (int q = 0; q < p; ++q) o += PL::stride(q) > 1 ? PL::stride(q) * (PL::R[q] - 1) : 0;
    return o;
  }
  static constexpr int TW_TOTAL = tw_off(PL::NP);
  static constexpr bool radices_fit() {
    for (int q = 0; q < PL::NP; ++q)
      if (PL::R[q] > 32) return false;  // fx_bits
    return true;
  }
  static_assert(radices_fit(), "fixed-point passes have radices up to 32");
};

template <class PL, int Q>
__device__ __forceinline__ int fx_tw_index(int e) {  // a of table entry e: exp(-2 pi i a / M)
  if constexpr (Q < PL::NP) {
    constexpr int off = PL::tw_off(Q), S = PL::stride(Q), n = S > 1 ? S * (PL::R[Q] - 1) : 0;
    if (e < off + n) {
      const int k = (e - off) / S + 1, i = (e - off) - (k - 1) * S;
      return (PL::M / PL::span(Q)) * i * k;
    }
    return fx_tw_index<PL, Q + 1>(e);
  }
  return 0;
}
template <class PL>
__global__ void k_twiddles_fx(int4* tw) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < PL::TW_TOTAL) tw[e] = fx_root(fx_tw_index<PL, 0>(e), PL::M);
}

// The twiddles of butterfly i, with the factor 1/4 of fx_cmul4.
template <class PL, int P, int SIGN, int R>
__device__ __forceinline__ void fx_pass_tw(fxc (&x)[R], const int4* __restrict__ tw, int i) {
  constexpr int S = PL::stride(P);
  const int4* __restrict__ t = tw + PL::tw_off(P) + i;
  x[0] = fxc{(x[0].x + 2) >> 2, (x[0].y + 2) >> 2};
#pragma unroll
  for (int k = 1; k < R; ++k) x[k] = fx_cmul4<(SIGN > 0)>(x[k], __ldg(t + (k - 1) * S));
}
// Bits of a pass's inputs: a DIT pass with twiddles divides them by 4 first, but
// multiplies them before it does, which has room for 62 bits (fx_cmul).
template <class PL, int P, bool DIT>
constexpr int fx_in_bits() {
  const int b = fx_bits(PL::R[P]);
  return !(DIT && PL::stride(P) > 1) ? b : b + 2 < 62 ? b + 2 : 62;
}
template <class PL, int P>
constexpr int fx_gain() {  // the pass's factor 2^-gain
  return PL::stride(P) > 1 ? 2 : 0;
}

// Per-tile words in shared memory: the largest word of each pass's outputs, and
// the largest FP64 high word of each raw tile.
struct FxWords {
  unsigned bits[16];
  unsigned top[2];
};
template <int NT>
__device__ __forceinline__ void fx_words_clear(FxWords* s, int tid) {
  if (tid < 18) (tid < 16 ? s->bits[tid] : s->top[tid - 16]) = 0u;
}
__device__ __forceinline__ unsigned fx_top(double d) {
  return (unsigned)((unsigned long long)__double_as_longlong(d) >> 32) & 0x7fffffffu;
}
__device__ __forceinline__ void fx_note(unsigned t, unsigned* slot, int tid) {
  t = __reduce_max_sync(0xffffffffu, t);
  if ((tid & 31) == 0) atomicMax(slot, t);
}

// FP64 values held in an integer tile until the tile's scale is known.
__device__ __forceinline__ fxc fx_raw(double2 d) { return fxc{__double_as_longlong(d.x), __double_as_longlong(d.y)}; }
__device__ __forceinline__ double2 fx_unraw(fxc q) {
  return make_double2(__longlong_as_double(q.x), __longlong_as_double(q.y));
}

// The tile's scale: value = q 2^E; bad: a non-finite value came in.
struct FxScale {
  int E;
  bool bad;
};
__device__ __forceinline__ int fx_emax(unsigned top) { return max((int)(top >> 20), 1); }
__device__ __forceinline__ double fx_value(long long q, const FxScale& sc) {
  if (sc.bad) return __longlong_as_double(0x7ff8000000000000LL);
  return fx_normal(sc.E) ? fx_to_double(q, sc.E) : fx_scalbn(q, sc.E);
}

// |u| + |v| of a point, and the FP64 value of a tile's largest: the row pass and
// k_phys take it from the same integers, so that both give the same CFLM.
__device__ __forceinline__ unsigned long long fx_speed(fxc x) {
  return (unsigned long long)(x.x < 0 ? -x.x : x.x) + (unsigned long long)(x.y < 0 ? -x.y : x.y);
}
__device__ __forceinline__ double fx_speed_value(unsigned long long top, FxScale sc) {
  if (sc.bad) return 0.0;
  if (top >> 63) {
    top = (top >> 1) | (top & 1);
    sc.E += 1;
  }
  return fx_value((long long)top, sc);
}

// One pass over a [slot][v] tile.  RAW: the tile is FP64 with the largest
// exponent `s`, taken to K bits, else integers to be shifted by `s`.  PAD:
// positions N/2 .. M - N/2 of the lines are zero (the 3/2 pad): whole segments
// are not read.  Returns the largest word of the outputs.
template <class PL, int V, int NT, int P, int SIGN, bool DIT, bool RAW, bool PAD = false, int K = fx_bits(PL::R[P])>
__device__ __forceinline__ unsigned fx_pass(fxc* sm, const int4* __restrict__ tw, int tid, int s, bool bad) {
  constexpr int R = PL::R[P];
  constexpr int L = PL::span(P);
  constexpr int S = L / R;
  constexpr int SP = PL::pstride(P);
  constexpr int NB = V * (PL::M / R);
  constexpr int Nh = PL::M / 3;
  FxRange rg;
  for (int w = tid; w < NB; w += NT) {
    const int v = w % V;
    const int b = w / V;
    const int blk = b / S;
    const int i = b - blk * S;
    fxc* p = sm + PL::phys(blk * L + i) * V + v;
    fxc x[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      if (PAD && k * S >= Nh && k * S + S - 1 <= PL::M - Nh) {
        x[k] = fxc{0, 0};
      } else if constexpr (RAW) {
        const double2 d = fx_unraw(p[k * SP * V]);
        x[k] = bad ? fxc{0, 0} : fxc{fx_from_double<K>(d.x, s), fx_from_double<K>(d.y, s)};
      } else {
        x[k] = p[k * SP * V];
      }
    }
    if constexpr (!RAW) fx_rescale<R>(x, s);
    if constexpr (DIT && S > 1) fx_pass_tw<PL, P, SIGN>(x, tw, i);
    Dft<R, SIGN, fxc>::run(x);
    if constexpr (!DIT && S > 1) fx_pass_tw<PL, P, SIGN>(x, tw, i);
#pragma unroll
    for (int k = 0; k < R; ++k) {
      p[k * SP * V] = x[k];
      rg.add(x[k]);
    }
  }
  return rg.word();
}

// Integer passes P .. TO - 1 (DIF) or P down to TO (DIT), a barrier after each;
// pass q notes its magnitudes in bits[BASE + q].  The first one reads what was
// noted in `from`.
template <class PL, int V, int NT, int SIGN, int P, int TO, int BASE>
__device__ __forceinline__ void fx_dif(fxc* sm, const int4* __restrict__ tw, int tid, FxWords* ws, FxScale& sc) {
  if constexpr (P < TO) {
    const int s = fx_shift(ws->bits[BASE + P - 1], fx_in_bits<PL, P, false>());
    sc.E += fx_gain<PL, P>() - s;
    fx_note(fx_pass<PL, V, NT, P, SIGN, false, false>(sm, tw, tid, s, false), &ws->bits[BASE + P], tid);
    __syncthreads();
    fx_dif<PL, V, NT, SIGN, P + 1, TO, BASE>(sm, tw, tid, ws, sc);
  }
}
template <class PL, int V, int NT, int SIGN, int P, int TO, int BASE>
__device__ __forceinline__ void fx_dit(fxc* sm, const int4* __restrict__ tw, int tid, FxWords* ws, FxScale& sc) {
  if constexpr (P >= TO) {
    const int s = fx_shift(ws->bits[BASE + P + 1], fx_in_bits<PL, P, true>());
    sc.E += fx_gain<PL, P>() - s;
    fx_note(fx_pass<PL, V, NT, P, SIGN, true, false>(sm, tw, tid, s, false), &ws->bits[BASE + P], tid);
    __syncthreads();
    fx_dit<PL, V, NT, SIGN, P - 1, TO, BASE>(sm, tw, tid, ws, sc);
  }
}

// Rows z0 .. z0 + V - 1 of the U planes through the inverse x-transform: Z[k] =
// u^[k] + i v^[k] (k < N/2; real parts only at k = 0), Z[M - k] = conj(u^[k]) + i
// conj(v^[k]), zeros between (the 3/2 pad).  A thread keeps its rows' values in
// registers until the tile's largest exponent is known.  Leaves the integers u +
// i v in digit-reversed order, their largest word in bits[NP - 1].
template <class PL, int V, int NT>
__device__ __forceinline__ void fx_rows_inverse(const void* p0, const void* p1, fxc* sm, const int4* __restrict__ tw,
                                                int z0, int tid, FxWords* ws, FxScale& sc) {
  constexpr int M = PL::M, Nh = M / 3;
  constexpr int CNT = (Nh * V + NT - 1) / NT;
  // Z is a sum of two, of values taken to half units and rounded to nearest: a
  // row with a few large values and many small ones loses most here, at the
  // tile's unit.  With values truncated at fx_bits - 1 a velocity of spectrum
  // k^-2 was 3.0, 3.1 and 3.8 to 6.1e-16 off at N = 1024, 2048 and 4096, where
  // FP64 transforms are 2.4, 2.8 and 3.3e-16 off and this is 1.4, 2.3 and 2.7.
  constexpr int K = fx_pad_bits(PL::R[0]);
  const double2* __restrict__ w0 = static_cast<const double2*>(p0);
  const double2* __restrict__ w1 = static_cast<const double2*>(p1);
  fx_words_clear<NT>(ws, tid);
  double2 u[CNT], q[CNT];
  unsigned top = 0;
#pragma unroll
  for (int c = 0; c < CNT; ++c) {
    const int w = tid + c * NT;
    u[c] = q[c] = make_double2(0.0, 0.0);
    if (Nh * V % NT == 0 || w < Nh * V) {
      const size_t at = (size_t)(w / V) * M + z0 + w % V;
      u[c] = w0[at];
      q[c] = w1[at];
    }
    top = max(max(top, max(fx_top(u[c].x), fx_top(u[c].y))), max(fx_top(q[c].x), fx_top(q[c].y)));
  }
  __syncthreads();
  fx_note(top, &ws->top[0], tid);
  for (int w = tid; w < V * (M - 2 * Nh + 1); w += NT) sm[PL::phys(Nh + w / V) * V + w % V] = fxc{0, 0};
  __syncthreads();
  const int emax = fx_emax(ws->top[0]);
  sc = FxScale{fx_exponent(emax, K) + 1, emax == 0x7ff};
#pragma unroll
  for (int c = 0; c < CNT; ++c) {
    const int w = tid + c * NT;
    if (Nh * V % NT == 0 || w < Nh * V) {
      const int v = w % V, k = w / V;
      long long ux = 0, uy = 0, qx = 0, qy = 0;
      if (!sc.bad) {
        ux = fx_from_double<K>(u[c].x, emax);
        uy = fx_from_double<K>(u[c].y, emax);
        qx = fx_from_double<K>(q[c].x, emax);
        qy = fx_from_double<K>(q[c].y, emax);
      }
      if (k == 0) uy = qy = 0;
      sm[PL::phys(k) * V + v] = fxc{(ux - qy + 1) >> 1, (uy + qx + 1) >> 1};
      if (k > 0) sm[PL::phys(M - k) * V + v] = fxc{(ux + qy + 1) >> 1, (qx - uy + 1) >> 1};
    }
  }
  __syncthreads();
  fx_note(fx_pass<PL, V, NT, 0, +1, false, false, true>(sm, tw, tid, 0, false), &ws->bits[0], tid);
  sc.E += fx_gain<PL, 0>();
  __syncthreads();
  fx_dif<PL, V, NT, +1, 1, PL::NP, 0>(sm, tw, tid, ws, sc);
}

// Unpack P = FFT(a + i b) (natural order, largest word in bits[NP]) into A =
// F(a), B = F(b) for kx < N/2.
template <class PL, int V, int NT>
__device__ __forceinline__ void fx_rows_unpack(void* p0, void* p1, const fxc* sm, int z0, int tid, const FxWords* ws,
                                               const FxScale& sc) {
  constexpr int M = PL::M, Nh = M / 3, NP = PL::NP;
  double2* __restrict__ w0 = static_cast<double2*>(p0);
  double2* __restrict__ w1 = static_cast<double2*>(p1);
  const int s = min(fx_shift_exact(ws->bits[NP], 62), 0);  // room for the sums
  const FxScale out{sc.E - s - 1, sc.bad};
  for (int w = tid; w < V * Nh; w += NT) {
    const int v = w % V;
    const int k = w / V;
    fxc p[2] = {sm[PL::phys(k) * V + v], sm[PL::phys(k == 0 ? 0 : M - k) * V + v]};
    fx_rescale<2>(p, s);
    const size_t at = (size_t)k * M + z0 + v;
    w0[at] = make_double2(fx_value(p[0].x + p[1].x, out), fx_value(p[0].y - p[1].y, out));
    w1[at] = make_double2(fx_value(p[0].y + p[1].y, out), fx_value(p[1].x - p[0].x, out));
  }
}

// k_row in fixed point: U-state rows -> products -> P-state rows, optional CFL
// statistics.  No pipe is full (ncu, N=4096: issue 46 %, integer ALU 50 %, the
// FMA pipe that runs the widening multiply-adds 24 %): with one or two tiles per
// SM the latency of loads, passes and barriers in turn bounds it.  N=4096 1191 us
// (FP64 transforms: 6120, the FP64 pipe 83 % busy), N=1024 72 us (352).
template <class PL, int V, int NT>
__device__ __forceinline__ void row_fx_body(const StepArgs& a, const void* u0, const void* u1, const Blk bk) {
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ FxWords ws;
  fxc* sm = reinterpret_cast<fxc*>(smraw);
  constexpr int M = PL::M, NP = PL::NP;
  const int tid = threadIdx.x;
  const int z0 = bk.x * V;
  const int4* __restrict__ tw = static_cast<const int4*>(a.tw);
  FxScale sc;
  fx_rows_inverse<PL, V, NT>(u0, u1, sm, tw, z0, tid, &ws, sc);

  // products u^2 - v^2, u v of the inverse transform's points, divided by 2^64,
  // and the first forward pass on them: u, v are brought below 2^KU
  const bool stats = (a.flags & F_STATS) != 0;
  double mx = 0.0, acc = 0.0;
  {
    constexpr int R = PL::RP;
    constexpr int KU = (fx_bits(R) + 64) / 2;
    static_assert(KU <= 61, "u + v stays below 2^62");
    constexpr int NB = V * (M / R);
    const int s = fx_shift_exact(ws.bits[NP - 1], KU);
    unsigned long long top = 0;
    FxRange rg;
    for (int w = tid; w < NB; w += NT) {
      const int v = w % V;
      const int b = w / V;
      fxc* p = sm + b * (R + 1) * V + v;
      fxc x[R];
#pragma unroll
      for (int j = 0; j < R; ++j) x[j] = p[j * V];
      if (stats) {
#pragma unroll
        for (int j = 0; j < R; ++j) top = max(top, fx_speed(x[j]));
      }
      fx_rescale<R>(x, s);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const long long u = x[j].x, q = x[j].y;
        x[j] = fxc{fx_mul(u - q, u + q), fx_mul(u, q)};
      }
      Dft<R, -1, fxc>::run(x);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        p[j * V] = x[j];
        rg.add(x[j]);
      }
    }
    fx_note(rg.word(), &ws.bits[2 * NP - 1], tid);
    if (stats) {
      mx = fx_speed_value(top, sc);
      acc = sc.bad ? fx_value(0, sc) : mx * mx;  // finiteness of u^2 + v^2
    }
    sc.E = 2 * (sc.E - s) + 64;
    __syncthreads();
  }
  fx_dit<PL, V, NT, -1, NP - 2, 0, NP>(sm, tw, tid, &ws, sc);

  fx_rows_unpack<PL, V, NT>(a.w0, a.w1, sm, z0, tid, &ws, sc);
  if (stats) finish_stats<NT, false>(a, mx, acc, 0.0, M, tid, bk);
}
template <class PL, int V, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_row_fx(StepArgs a0) {
  const Blk bk = hw_blk();
  const StepArgs a = member_args(a0, sizeof(double2), bk.y);
  row_fx_body<PL, V, NT>(a, a.w0, a.w1, bk);
}

// k_phys in fixed point: U-state rows -> physical u, v (statistics, optional
// plane store), tiles and statistics as phys_body.
template <class PL, int V, int NT>
__global__ void __launch_bounds__(NT) k_phys_fx(StepArgs a0) {
  const Blk bk = hw_blk();
  const StepArgs a = member_args(a0, sizeof(double2), bk.y);
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ FxWords ws;
  fxc* sm = reinterpret_cast<fxc*>(smraw);
  constexpr int M = PL::M;
  static_assert(size_t(PL::PADM) * V * sizeof(fxc) >= size_t(2) * NT * sizeof(double), "finish_stats' sums fit in the tile");
  const int tid = threadIdx.x;
  double mx = 0.0, acc = 0.0, comp = 0.0;
  double* __restrict__ ph = static_cast<double*>(a.phys);
  const bool store = (a.flags & F_PHYS) != 0;
  const bool diag = (a.flags & F_DIAG) != 0;
  for (int tile = bk.x; tile < M / V; tile += bk.nx) {
    const int z0 = tile * V;
    FxScale sc;
    fx_rows_inverse<PL, V, NT>(a.w0, a.w1, sm, static_cast<const int4*>(a.tw), z0, tid, &ws, sc);
    unsigned long long top = 0;
    for (int w = tid; w < V * M; w += NT) {
      const int v = w % V;
      const int pos = w / V;
      const fxc q = sm[PL::phys(pos) * V + v];
      const double x = fx_value(q.x, sc), y = fx_value(q.y, sc);
      top = max(top, fx_speed(q));
      if (diag)
        add_point(x, y, acc, comp);
      else
        acc = fma(x, x, fma(y, y, acc));  // finiteness check only
      if (store) {
        const int n = PL::freq(pos);
        ph[(size_t)(z0 + v) * M + n] = x;
        ph[(size_t)M * M + (size_t)(z0 + v) * M + n] = y;
      }
    }
    mx = fmax(mx, fx_speed_value(top, sc));
    __syncthreads();  // the tile and its words are free
  }
  if (diag) {
    finish_stats<NT, true>(a, mx, acc, comp, M, tid, bk, reinterpret_cast<double*>(smraw));
  } else {
    finish_stats<NT, false>(a, mx, acc, 0.0, M, tid, bk);
  }
}

// Column kx of two planes into a raw tile, its largest high word in top[0].
template <class PL, int NT>
__device__ __forceinline__ void fx_column_load(fxc* sm, const void* p0, const void* p1, int kx, int tid, FxWords* ws) {
  constexpr int M = PL::M, V = 2;
  const double2* __restrict__ w0 = static_cast<const double2*>(p0) + (size_t)kx * M;
  const double2* __restrict__ w1 = static_cast<const double2*>(p1) + (size_t)kx * M;
  fx_words_clear<NT>(ws, tid);
  __syncthreads();
  unsigned top = 0;
  constexpr int U = 8;  // loads in flight per thread
  for (int w = tid; w < V * M; w += U * NT) {
    double2 d[U];
#pragma unroll
    for (int c = 0; c < U; ++c)
      if (w + c * NT < V * M) d[c] = (((w + c * NT) & 1) == 0 ? w0 : w1)[(w + c * NT) >> 1];
#pragma unroll
    for (int c = 0; c < U; ++c)
      if (w + c * NT < V * M) {
        sm[PL::phys((w + c * NT) >> 1) * V + ((w + c * NT) & 1)] = fx_raw(d[c]);
        top = max(top, max(fx_top(d[c].x), fx_top(d[c].y)));
      }
  }
  fx_note(top, &ws->top[0], tid);
  __syncthreads();
}
// Forward passes 0 .. TO - 1 of a raw column tile (largest high word in top[0]).
template <class PL, int NT, int TO>
__device__ __forceinline__ FxScale fx_column_forward(fxc* sm, const int4* __restrict__ tw, int tid, FxWords* ws) {
  const int emax = fx_emax(ws->top[0]);
  FxScale sc{fx_exponent(emax, fx_bits(PL::R[0])), emax == 0x7ff};
  fx_note(fx_pass<PL, 2, NT, 0, -1, false, true>(sm, tw, tid, emax, sc.bad), &ws->bits[0], tid);
  sc.E += fx_gain<PL, 0>();
  __syncthreads();
  fx_dif<PL, 2, NT, -1, 1, TO, 0>(sm, tw, tid, ws, sc);
  return sc;
}

// The inverse z-transform of a raw column tile (A tile of two lines in
// digit-reversed order, its largest high word in top[SLOT]) into the U planes.
// Its first pass is over the lines' pad: with RP divisible by 3 the middle third
// of every butterfly's inputs is zero (fx_pad_bits).
template <class PL, int NT, int SLOT>
__device__ __forceinline__ void fx_column_inverse(fxc* sm, const int4* __restrict__ tw, double2* __restrict__ w0,
                                                  double2* __restrict__ w1, int kx, int tid, FxWords* ws) {
  constexpr int M = PL::M, V = 2, NP = PL::NP;
  const int emax = fx_emax(ws->top[SLOT]);
  constexpr int K = fx_pad_bits(PL::RP);
  FxScale sc{fx_exponent(emax, K), emax == 0x7ff};
  fx_note(fx_pass<PL, V, NT, NP - 1, +1, true, true, false, K>(sm, tw, tid, emax, sc.bad), &ws->bits[2 * NP - 1], tid);
  __syncthreads();
  fx_dit<PL, V, NT, +1, NP - 2, 1, NP>(sm, tw, tid, ws, sc);
  // the last pass straight into the planes
  constexpr int R = PL::R[0];
  constexpr int S = M / R;
  const int s = fx_shift(ws->bits[NP + 1], fx_in_bits<PL, 0, true>());
  sc.E += fx_gain<PL, 0>() - s;
  for (int w = tid; w < V * S; w += NT) {
    const int v = w & 1;
    const int i = w >> 1;
    double2* __restrict__ dst = (v == 0 ? w0 : w1) + (size_t)kx * M;
    const fxc* p = sm + PL::phys(i) * V + v;
    fxc x[R];
#pragma unroll
    for (int k = 0; k < R; ++k) x[k] = p[k * PL::pstride(0) * V];
    fx_rescale<R>(x, s);
    fx_pass_tw<PL, 0, +1>(x, tw, i);
    Dft<R, +1, fxc>::run(x);
#pragma unroll
    for (int j = 0; j < R; ++j) dst[i + j * S] = make_double2(fx_value(x[j].x, sc), fx_value(x[j].y, sc));
  }
}

// k_col in fixed point: P-state column -> (om, fnm1 update) -> U-state column.
// The update between the transforms is FP64, 28 to 32 FP64 instructions a mode:
// reciprocals in four, the scale 1 / M^2 in the stage's weights, wave-number
// products in integers (exact: N is at most 4096).  PERM and the stage flags as
// k_col.  N=4096 1225 us (FP64 transforms: 4300), N=1024 81 us (317).
template <class PL, int NT, bool PERM>
__device__ __forceinline__ void col_fx_body(const StepArgs& a, void* d0, void* d1, const Blk bk) {
  static_assert(PL::M <= 6144, "K2 within 24 bits (fx_small)");
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ FxWords ws;
  fxc* sm = reinterpret_cast<fxc*>(smraw);
  constexpr int M = PL::M, V = 2, NP = PL::NP, N = 2 * M / 3, Nh = M / 3;
  const int tid = threadIdx.x;
  const int kx = bk.x;
  const int4* __restrict__ tw = static_cast<const int4*>(a.tw);
  double2* __restrict__ om =
      PERM ? static_cast<double2*>(a.om_p) + (size_t)kx * M : static_cast<double2*>(a.om) + (size_t)kx * N;
  double2* __restrict__ fm =
      PERM ? static_cast<double2*>(a.fm_p) + (size_t)kx * M : static_cast<double2*>(a.fnm1) + (size_t)kx * N;
  fx_column_load<PL, NT>(sm, a.w0, a.w1, kx, tid, &ws);
  const ModeCoef<double> cf = col_coef<double>(a, N);
  FxScale sc = fx_column_forward<PL, NT, NP - 1>(sm, tw, tid, &ws);

  // last forward pass -> nonlinear term, update, inversion -> raw (u^, v^)
  {
    constexpr int R = PL::RP;
    constexpr int NB = V * (M / R);
    constexpr int FSTEP = M / R;
    constexpr bool BAND_CT = (R % 3 == 0) && ((R / 3) % 2 == 0);
    const bool q_in = (a.flags & F_Q_IN) != 0;
    const bool fm_in = (a.flags & (F_Q_IN | F_NO_FM_IN)) == 0;
    const bool q_out = (a.flags & F_Q_OUT) != 0;
    const double ax = fx_small(kx), c2d = cf.c2 * cf.divxz, c3nd = cf.c3n * cf.divxz;
    const int s = fx_shift(ws.bits[NP - 2], fx_in_bits<PL, NP - 1, false>());
    sc.E -= s;
    unsigned top = 0;
    for (int w0i = 0; w0i < NB; w0i += NT) {
      const int w = w0i + tid;
      const bool act = w < NB;
      const int v = w & 1;
      const int b = act ? (w >> 1) : 0;
      fxc* p = sm + b * (R + 1) * V + v;
      const int fb = PL::freq(b * R);
      fxc x[R];
#pragma unroll
      for (int j = 0; j < R; ++j) x[j] = act ? p[j * V] : fxc{0, 0};
      fx_rescale<R>(x, s);
      Dft<R, -1, fxc>::run(x);
#pragma unroll
      for (int j = 0; j < R; j += 2) {
        if (BAND_CT && j >= R / 3 && j < 2 * R / 3) {
          if (act) p[j * V] = p[(j + 1) * V] = fxc{0, 0};
          continue;
        }
        // lane 0 takes position j, lane 1 position j+1
        const fxc keep = v == 0 ? x[j] : x[j + 1], send = v == 0 ? x[j + 1] : x[j];
        fxc recv;
        recv.x = __shfl_xor_sync(0xffffffffu, send.x, 1);
        recv.y = __shfl_xor_sync(0xffffffffu, send.y, 1);
        const fxc Aq = v == 0 ? keep : recv, Bq = v == 0 ? recv : keep;
        const int f = fb + (j + v) * FSTEP;
        const bool inband = act && (BAND_CT || f < Nh || f >= N);
        const int z = f < Nh ? f : f - Nh;
        double2 uh = {0.0, 0.0}, vh = {0.0, 0.0};
        if (inband) {
          const int zi = PERM ? (j + v) * FSTEP + b : z;
          const double2 o = om[zi];
          double2 fo = {0.0, 0.0};
          if (fm_in) fo = fm[zi];
          const int iz = z < Nh ? z : z - N;
          const int ik2 = kx * kx + iz * iz;
          const double gz = fx_small(iz), K2 = fx_small(ik2), k2s = ik2 > 0 ? K2 : 1.0;
          double2 F = {0.0, 0.0};  // fn = divxz F
          if (z != Nh) {
            const double2 Az = {fx_value(Aq.x, sc), fx_value(Aq.y, sc)}, Bz = {fx_value(Bq.x, sc), fx_value(Bq.y, sc)};
            const double ga = fx_small(kx * iz), g2 = fx_small(iz * iz - kx * kx);
            F.x = fma(Az.x, ga, Bz.x * g2);
            F.y = fma(Az.y, ga, Bz.y * g2);
          }
          double2 num;
          if (q_in) {
            num.x = fma(c2d, F.x, o.x);
            num.y = fma(c2d, F.y, o.y);
          } else {
            const double c1 = fma(-K2, cf.h1, 1.0);
            num.x = fma(c1, o.x, c2d * F.x);
            num.y = fma(c1, o.y, c2d * F.y);
            if (fm_in) {
              num.x = fma(cf.c3, fo.x, num.x);
              num.y = fma(cf.c3, fo.y, num.y);
            }
          }
          const double rden = newton_rcp(fma(K2, cf.h2, 1.0)), ik = newton_rcp(k2s);
          const double2 on = {num.x * rden, num.y * rden};
          const double2 t = {on.x * ik, on.y * ik};
          if (q_out) {
            const double c1n = fma(-K2, cf.h1n, 1.0);
            om[zi] = make_double2(fma(c1n, on.x, c3nd * F.x), fma(c1n, on.y, c3nd * F.y));
          } else {
            om[zi] = on;
            fm[zi] = make_double2(F.x * cf.divxz, F.y * cf.divxz);
          }
          // -i kz om' / K2, i kx om' / K2 (zero at K2 = 0, where both wave numbers are)
          uh = make_double2(t.y * gz, -t.x * gz);
          vh = make_double2(-t.y * ax, t.x * ax);
        }
        // lane 0 keeps u^ of position j and receives u^ of j+1; lane 1 the v^ pair
        const double2 mine = v == 0 ? uh : vh, send2 = v == 0 ? vh : uh;
        double2 other;
        other.x = __shfl_xor_sync(0xffffffffu, send2.x, 1);
        other.y = __shfl_xor_sync(0xffffffffu, send2.y, 1);
        top = max(max(top, max(fx_top(mine.x), fx_top(mine.y))), max(fx_top(other.x), fx_top(other.y)));
        if (act) {
          p[j * V] = fx_raw(v == 0 ? mine : other);
          p[(j + 1) * V] = fx_raw(v == 0 ? other : mine);
        }
      }
    }
    fx_note(top, &ws.top[1], tid);
    __syncthreads();
  }
  fx_column_inverse<PL, NT, 1>(sm, tw, static_cast<double2*>(d0), static_cast<double2*>(d1), kx, tid, &ws);
  col_finish<NT>(a, tid, bk.nx);
}
template <class PL, int NT, bool PERM, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_col_fx(StepArgs a0) {
  const Blk bk = hw_blk();
  const StepArgs a = member_args(a0, sizeof(double2), bk.y);
  col_fx_body<PL, NT, PERM>(a, a.w0, a.w1, bk);
}

// k_col_inv in fixed point: velocity low band (src, the om inversion, or a
// display scalar) -> pad -> inverse z-transform -> U planes.
template <class PL, int NT>
__global__ void __launch_bounds__(NT) k_col_inv_fx(StepArgs a0) {
  const StepArgs a = member_args(a0, sizeof(double2));
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ FxWords ws;
  fxc* sm = reinterpret_cast<fxc*>(smraw);
  constexpr int M = PL::M, V = 2;
  const int tid = threadIdx.x;
  const int kx = blockIdx.x;
  fx_words_clear<NT>(&ws, tid);
  __syncthreads();
  unsigned top = 0;
  for (int w = tid; w < V * M; w += NT) {
    const double2 val = col_inv_value<double, PL>(a, kx, w & 1, w >> 1);
    sm[PL::phys(w >> 1) * V + (w & 1)] = fx_raw(val);
    top = max(top, max(fx_top(val.x), fx_top(val.y)));
  }
  fx_note(top, &ws.top[0], tid);
  __syncthreads();
  fx_column_inverse<PL, NT, 0>(sm, static_cast<const int4*>(a.tw), static_cast<double2*>(a.w0),
                               static_cast<double2*>(a.w1), kx, tid, &ws);
}

}  // namespace pal
