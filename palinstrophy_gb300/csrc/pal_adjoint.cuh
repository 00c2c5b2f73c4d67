// Discrete adjoint of one LS-IMEX-RK3 stage at fixed dt.
//
// Forward stage (see k_col): U = Inv(om_in); (u, v) = P(U) = C2R2(pad U);
// a = u^2 - v^2, b = u v; (A, B) = Q(a, b) = gather(R2C2 a, R2C2 b);
// fn = divxz (GA A + (G^2 - A^2) B) (row N/2 zero);
// om_out = D (c1 om_in + c2 fn + c3 f_in), f_out = fn, D = 1/(1 + K2 h2).
//
// With the real inner product <x, y> = Re sum conj(x) y the transposes are
//   P^T(lam) = w' R2C2(lam) at the kept modes,  Q^T(lam) = C2R2(pad(lam / w')),
// w' = 1 for kx = 0 and 2 otherwise (C2R2 counts each kx >= 1 mode twice),
// and for the complex scalings (Inv, GA, c1 D, ...) the conjugate scaling.
//
// Both sweeps run on these kernels.  A segment of steps runs forward, keeping
// every stage's velocity planes (k_adj_vel for the first, then k_adj_fwd_row and
// k_adj_fwd_col per stage), and then backward, two launches a stage:
//   k_adj_col : the end of stage q (forward z-FFT of the adjoint velocity,
//               lam_om += conj(Inv) (w' lam_U, w' lam_V)) and the start of stage
//               q - 1 on the same column (lam_fn = c2 D lam_om + lam_f;
//               lam_om <- c1 D lam_om, lam_f <- c3 D lam_om; (lam_A, lam_B)/w'
//               padded, inverse z-FFT)
//   k_adj_row : inverse x of the lam planes and of the stage's velocity planes,
//               lam_u = 2u lam_a + v lam_b, lam_v = -2v lam_a + u lam_b, forward
//               x, unpack
// om, fnm1 and the adjoints lam_om, lam_f are columns in the adjoint column
// plan's butterfly-major order throughout, so every kernel reads and writes
// them in consecutive order.  The FP64 form runs the same passes with
// fixed-point transforms (pal_fx_adjoint.cuh).
//
// Small grids are bound by the latency of the passes and launches: N=512 FP32,
// 200 steps 40.2 ms before (natural-order columns, the stage inputs copied, the
// velocity transformed again, seven launches a stage), 23.9 ms now; FP64 20
// steps 37.1 and 8.3 ms.
#pragma once
#include "pal_kernels.cuh"

namespace pal {

enum : int {
  F_ADJ_OUT = 1 << 16,  // k_adj_col: end a stage
  F_ADJ_IN = 1 << 17,   // k_adj_col: start a stage (weights a.alpha, a.beta)
};

template <typename T>
struct StageCoef {
  T h1, h2, c2, c3, divxz;
};

template <typename T, int M>
__device__ __forceinline__ StageCoef<T> stage_coef(const StepArgs& a) {
  const double dt = a.sc->dt, visc = a.sc->visc;
  StageCoef<T> c;
  c.h1 = T((a.beta * dt) * visc);
  c.h2 = T((a.alpha * dt) * visc);
  c.c2 = T(a.alpha * dt);
  c.c3 = T(a.beta * dt);
  const T m32 = T(M);
  c.divxz = T(1) / (m32 * m32);
  return c;
}

__device__ __forceinline__ float adj_rcp(float x) { return 1.0f / x; }
__device__ __forceinline__ double adj_rcp(double x) { return newton_rcp(x); }

// One mode of the column pass: lam_om += the adjoint velocity (lu, lv) of the
// stage that ends, then the start of the next one; returns its (lam_A, lam_B) /
// w' (zero without F_ADJ_IN).
template <typename T>
struct AdjPair {
  cplx<T> a, b;
};
template <typename T>
__device__ __forceinline__ AdjPair<T> adj_mode(int flags, cplx<T> lu, cplx<T> lv, cplx<T>& lw_io, cplx<T>& lf_io,
                                               const StageCoef<T>& cf, int kx, int z, int N) {
  using C = cplx<T>;
  const int Nh = N >> 1;
  const T ax = T(kx), gz = T(z < Nh ? z : z - N);
  const T K2 = ax * ax + gz * gz;
  constexpr T half = sizeof(T) == 4 ? T(0.5) : T(1);  // the FP32 row pass leaves twice the transforms
  C lw = lw_io;
  if (flags & F_ADJ_OUT) {
    if (kx >= 1) {
      // conj(-i gz/K2) w' lu + conj(i ax/K2) w' lv = i (gz w'/K2) lu - i (ax w'/K2) lv
      const T ik = T(2) * half * adj_rcp(K2);
      const T su = gz * ik, sv = ax * ik;
      lw = C{lw.x - su * lu.y + sv * lv.y, lw.y + su * lu.x - sv * lv.x};
    } else if (z >= 1) {
      const T ig = half / gz;  // conj(-i/gz) = i/gz
      lw = C{lw.x - ig * lu.y, lw.y + ig * lu.x};
    }
  }
  AdjPair<T> r = {{T(0), T(0)}, {T(0), T(0)}};
  if (flags & F_ADJ_IN) {
    const T D = adj_rcp(T(1) + K2 * cf.h2);
    const T c1 = T(1) - K2 * cf.h1;
    const C lff = lf_io;
    const C lfn = {cf.c2 * D * lw.x + lff.x, cf.c2 * D * lw.y + lff.y};
    lf_io = C{cf.c3 * D * lw.x, cf.c3 * D * lw.y};
    lw = C{c1 * D * lw.x, c1 * D * lw.y};
    if (z != Nh) {
      const T w = kx == 0 ? cf.divxz : T(0.5) * cf.divxz;
      const T sa = w * (gz * ax), sb = w * (gz * gz - ax * ax);
      r.a = C{sa * lfn.x, sa * lfn.y};
      r.b = C{sb * lfn.x, sb * lfn.y};
    }
  }
  lw_io = lw;
  return r;
}

// The in-band entries of a butterfly-major column, consecutive threads on
// consecutive entries: f(index, digit-reversed position, z).
template <class PL, int NT, class F>
__device__ __forceinline__ void for_column(int tid, F&& f) {
  constexpr int M = PL::M, N = 2 * M / 3, Nh = M / 3, FSTEP = PL::FSTEP;
  for (int p = tid; p < M; p += NT) {
    const int j = p / FSTEP, b = p - j * FSTEP;
    const int fr = PL::freq(b * PL::RP) + j * FSTEP;
    const bool in = fr < Nh || fr >= N;
    f(p, b * PL::RP + j, in, fr < Nh ? fr : fr - Nh);
  }
}

template <typename T, class PL, int NT>
__global__ void __launch_bounds__(NT) k_adj_col(StepArgs a) {
  pdl_wait();
  using C = cplx<T>;
  extern __shared__ __align__(128) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  constexpr int M = PL::M, V = 2, N = 2 * M / 3;
  const int tid = threadIdx.x, kx = blockIdx.x;
  const C* __restrict__ tw = static_cast<const C*>(a.tw);
  C* __restrict__ lom = static_cast<C*>(a.om_p) + (size_t)kx * M;
  C* __restrict__ lf = static_cast<C*>(a.fm_p) + (size_t)kx * M;
  C* __restrict__ x0 = static_cast<C*>(a.w0) + (size_t)kx * M;
  C* __restrict__ x1 = static_cast<C*>(a.w1) + (size_t)kx * M;
  const StageCoef<T> cf = stage_coef<T, M>(a);
  if (a.flags & F_ADJ_OUT) {
    for (int w = tid; w < V * M; w += NT) sm[PL::phys(w >> 1) * V + (w & 1)] = ((w & 1) == 0 ? x0 : x1)[w >> 1];
    __syncthreads();
    dif_range<T, PL, V, NT, -1, 0, PL::NP>(sm, tw, tid);
  }
  for_column<PL, NT>(tid, [&](int p, int pos, bool in, int z) {
    C* s = sm + PL::phys(pos) * V;
    AdjPair<T> r = {{T(0), T(0)}, {T(0), T(0)}};
    if (in) {
      C lw = lom[p], lff = {T(0), T(0)};
      if (a.flags & F_ADJ_IN) lff = lf[p];
      r = adj_mode<T>(a.flags, s[0], s[1], lw, lff, cf, kx, z, N);
      lom[p] = lw;
      if (a.flags & F_ADJ_IN) lf[p] = lff;
    }
    s[0] = r.a;
    s[1] = r.b;
  });
  if (!(a.flags & F_ADJ_IN)) return;
  __syncthreads();
  dit_range<T, PL, V, NT, +1, PL::NP - 1, 1>(sm, tw, tid);
  col_last_pass<T, PL, NT>(sm, static_cast<C*>(a.w0), static_cast<C*>(a.w1), tw, kx, tid);
}

// The lam planes and the stage's velocity planes (y0, y1) share a thread's
// butterflies in the last inverse pass, where the pointwise step happens.
template <typename T, class PL, int V, int NT>
__global__ void __launch_bounds__(NT) k_adj_row(StepArgs a) {
  pdl_wait();
  using C = cplx<T>;
  extern __shared__ __align__(128) unsigned char smraw[];
  C* lam = reinterpret_cast<C*>(smraw);
  C* vel = lam + PL::PADM * V;
  constexpr int M = PL::M;
  const int tid = threadIdx.x, z0 = blockIdx.x * V;
  const C* __restrict__ tw = static_cast<const C*>(a.tw);
  StepArgs b = a;
  b.w0 = const_cast<void*>(a.y0);
  b.w1 = const_cast<void*>(a.y1);
  {
    // half of the block transforms each of the two tiles
    constexpr int NH = NT / 2;
    const bool second = tid >= NH;
    const int t = second ? tid - NH : tid;
    row_first_pass_paired<T, PL, V, NH>(second ? b : a, second ? vel : lam, z0, t);
    dif_range<T, PL, V, NH, +1, 1, PL::NP - 1>(second ? vel : lam, tw, t);
  }
  {
    constexpr int R = PL::RP;
    for (int w = tid; w < V * (M / R); w += NT) {
      const int at = (w / V) * (R + 1) * V + w % V;
      C l[R], q[R];
#pragma unroll
      for (int j = 0; j < R; ++j) l[j] = lam[at + j * V];
      Dft<R, +1, C>::run(l);
#pragma unroll
      for (int j = 0; j < R; ++j) q[j] = vel[at + j * V];
      Dft<R, +1, C>::run(q);
      // l = (lam_a, lam_b), q = (u, v) at each physical point
#pragma unroll
      for (int j = 0; j < R; ++j)
        l[j] = C{T(2) * q[j].x * l[j].x + q[j].y * l[j].y, -T(2) * q[j].y * l[j].x + q[j].x * l[j].y};
      Dft<R, -1, C>::run(l);
#pragma unroll
      for (int j = 0; j < R; ++j) lam[at + j * V] = l[j];
    }
    __syncthreads();
  }
  dit_range<T, PL, V, NT, -1, PL::NP - 2, 1>(lam, tw, tid);
  row_last_pass_paired<T, PL, V, NT>(a, lam, z0, tid);
}

// Forward stage of a kept segment, out of place: velocity planes (y0, y1) ->
// product planes (w0, w1) ...
template <typename T, class PL, int V, int NT>
__global__ void __launch_bounds__(NT) k_adj_fwd_row(StepArgs a) {
  pdl_wait();
  extern __shared__ __align__(128) unsigned char smraw[];
  cplx<T>* sm = reinterpret_cast<cplx<T>*>(smraw);
  const int tid = threadIdx.x, z0 = blockIdx.x * V;
  const cplx<T>* __restrict__ tw = static_cast<const cplx<T>*>(a.tw);
  StepArgs b = a;
  b.w0 = const_cast<void*>(a.y0);
  b.w1 = const_cast<void*>(a.y1);
  row_first_pass_paired<T, PL, V, NT>(b, sm, z0, tid);
  dif_range<T, PL, V, NT, +1, 1, PL::NP - 1>(sm, tw, tid);
  T mx = T(0), acc = T(0);
  row_products<T, PL, V, NT>(sm, tid, false, mx, acc);
  dit_range<T, PL, V, NT, -1, PL::NP - 2, 1>(sm, tw, tid);
  row_last_pass_paired<T, PL, V, NT>(a, sm, z0, tid);
}

// ... and product planes, om and fnm1 -> the next stage's om, fnm1 and velocity
// planes (y0, y1).
template <typename T, class PL, int NT>
__global__ void __launch_bounds__(NT) k_adj_fwd_col(StepArgs a) {
  pdl_wait();
  using C = cplx<T>;
  extern __shared__ __align__(128) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  constexpr int M = PL::M, V = 2, N = 2 * M / 3;
  const int tid = threadIdx.x, kx = blockIdx.x;
  const C* __restrict__ tw = static_cast<const C*>(a.tw);
  const C* __restrict__ w0 = static_cast<const C*>(a.w0);
  const C* __restrict__ w1 = static_cast<const C*>(a.w1);
  {
    constexpr int R = PL::R[0];
    constexpr int S = M / R;
    for (int w = tid; w < V * S; w += NT) {
      const int v = w & 1, i = w >> 1;
      const C* __restrict__ src = (v == 0 ? w0 : w1) + (size_t)kx * M;
      C x[R];
#pragma unroll
      for (int j = 0; j < R; ++j) x[j] = src[i + j * S];
      Dft<R, -1, C>::run(x);
      pass_tw<PL, 0, -1>(x, tw, i);
      C* p = sm + PL::phys(i) * V + v;
#pragma unroll
      for (int k = 0; k < R; ++k) p[k * PL::pstride(0) * V] = x[k];
    }
    __syncthreads();
  }
  dif_range<T, PL, V, NT, -1, 1, PL::NP - 1>(sm, tw, tid);
  const ModeCoef<T> cf = col_coef<T>(a, N);
  col_middle<T, PL, NT, false, true, true>(sm, nullptr, nullptr, static_cast<C*>(a.om_p) + (size_t)kx * M,
                                           static_cast<C*>(a.fm_p) + (size_t)kx * M, cf, kx, tid, a.flags);
  dit_range<T, PL, V, NT, +1, PL::NP - 2, 1>(sm, tw, tid);
  col_last_pass<T, PL, NT>(sm, static_cast<C*>(const_cast<void*>(a.y0)), static_cast<C*>(const_cast<void*>(a.y1)), tw,
                           kx, tid);
  col_finish<NT>(a, tid, (int)gridDim.x);
}

// The value of k_adj_vel at an in-band entry of line v of column kx: u^ or v^
// of om.
template <typename T>
__device__ __forceinline__ cplx<T> adj_velocity(cplx<T> o, int kx, int z, int N, int v) {
  using C = cplx<T>;
  const T gz = T(z < (N >> 1) ? z : z - N), ax = T(kx);
  if (kx >= 1) {
    const T ik = T(1) / (ax * ax + gz * gz);
    const C t = {o.x * ik, o.y * ik};
    return v == 0 ? C{t.y * gz, -t.x * gz} : C{-t.y * ax, t.x * ax};
  }
  if (v == 0 && z >= 1) {
    const T ig = T(1) / gz;
    return C{o.y * ig, -o.x * ig};
  }
  return C{T(0), T(0)};
}
// om -> velocity planes (y0, y1).
template <typename T, class PL, int NT>
__global__ void __launch_bounds__(NT) k_adj_vel(StepArgs a) {
  pdl_wait();
  using C = cplx<T>;
  extern __shared__ __align__(128) unsigned char smraw[];
  C* sm = reinterpret_cast<C*>(smraw);
  constexpr int M = PL::M, V = 2, N = 2 * M / 3;
  const int tid = threadIdx.x, kx = blockIdx.x;
  const C* __restrict__ tw = static_cast<const C*>(a.tw);
  const C* __restrict__ om = static_cast<const C*>(a.om_p) + (size_t)kx * M;
  for_column<PL, NT>(tid, [&](int p, int pos, bool in, int z) {
    C* s = sm + PL::phys(pos) * V;
    const C o = in ? om[p] : C{T(0), T(0)};
    s[0] = in ? adj_velocity<T>(o, kx, z, N, 0) : o;
    s[1] = in ? adj_velocity<T>(o, kx, z, N, 1) : o;
  });
  __syncthreads();
  dit_range<T, PL, V, NT, +1, PL::NP - 1, 1>(sm, tw, tid);
  col_last_pass<T, PL, NT>(sm, static_cast<C*>(const_cast<void*>(a.y0)), static_cast<C*>(const_cast<void*>(a.y1)), tw,
                           kx, tid);
}

// Loss gradient seed: lam_om = w' K2 om (L = 1/2 sum w' K2 |om|^2), lam_f = 0;
// om (natural columns), lam_om and lam_f (butterfly-major).  One partial of the
// loss per column.
template <typename T, class PL, int NT>
__global__ void __launch_bounds__(NT) k_adj_seed(const cplx<T>* __restrict__ om, cplx<T>* __restrict__ lom,
                                                 cplx<T>* __restrict__ lf, double* __restrict__ loss_part) {
  using C = cplx<T>;
  constexpr int M = PL::M, N = 2 * M / 3, Nh = M / 3;
  const int kx = blockIdx.x;
  double acc = 0.0;
  for_column<PL, NT>(threadIdx.x, [&](int p, int, bool in, int z) {
    if (!in) return;
    const T gz = T(z < Nh ? z : z - N);
    const T K2 = T(kx) * T(kx) + gz * gz;
    const T w = kx == 0 ? T(1) : T(2);
    const C o = om[(size_t)kx * N + z];
    lom[(size_t)kx * M + p] = C{w * K2 * o.x, w * K2 * o.y};
    lf[(size_t)kx * M + p] = C{T(0), T(0)};
    acc += 0.5 * (double)w * (double)K2 * ((double)o.x * (double)o.x + (double)o.y * (double)o.y);
  });
  __shared__ double red[NT / 32];
  double v[1] = {acc};
  block_sum<NT, 1>(v, red, threadIdx.x);
  if (threadIdx.x == 0) loss_part[kx] = v[0];
}

}  // namespace pal
