// The adjoint passes of the FP64 form (pal_adjoint.cuh) with fixed-point
// transforms: the same tiles, orders and per-mode arithmetic.
#pragma once
#include "pal_adjoint.cuh"
#include "pal_fx_kernels.cuh"

namespace pal {

template <class PL, int NT>
__global__ void __launch_bounds__(NT) k_adj_col_fx(StepArgs a) {
  pdl_wait();
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ FxWords ws;
  fxc* sm = reinterpret_cast<fxc*>(smraw);
  constexpr int M = PL::M, V = 2, N = 2 * M / 3;
  const int tid = threadIdx.x, kx = blockIdx.x;
  const int4* __restrict__ tw = static_cast<const int4*>(a.tw);
  double2* __restrict__ lom = static_cast<double2*>(a.om_p) + (size_t)kx * M;
  double2* __restrict__ lf = static_cast<double2*>(a.fm_p) + (size_t)kx * M;
  const StageCoef<double> cf = stage_coef<double, M>(a);
  FxScale sc{0, false};
  if (a.flags & F_ADJ_OUT) {
    fx_column_load<PL, NT>(sm, a.w0, a.w1, kx, tid, &ws);
    sc = fx_column_forward<PL, NT, PL::NP>(sm, tw, tid, &ws);
  } else {
    fx_words_clear<NT>(&ws, tid);
    __syncthreads();
  }
  unsigned top = 0;
  for_column<PL, NT>(tid, [&](int p, int pos, bool in, int z) {
    fxc* s = sm + PL::phys(pos) * V;
    AdjPair<double> r = {{0.0, 0.0}, {0.0, 0.0}};
    if (in) {
      double2 lw = lom[p], lff = {0.0, 0.0}, lu = {0.0, 0.0}, lv = {0.0, 0.0};
      if (a.flags & F_ADJ_IN) lff = lf[p];
      if (a.flags & F_ADJ_OUT) {
        lu = make_double2(fx_value(s[0].x, sc), fx_value(s[0].y, sc));
        lv = make_double2(fx_value(s[1].x, sc), fx_value(s[1].y, sc));
      }
      r = adj_mode<double>(a.flags, lu, lv, lw, lff, cf, kx, z, N);
      lom[p] = lw;
      if (a.flags & F_ADJ_IN) lf[p] = lff;
    }
    s[0] = fx_raw(r.a);
    s[1] = fx_raw(r.b);
    top = max(max(top, max(fx_top(r.a.x), fx_top(r.a.y))), max(fx_top(r.b.x), fx_top(r.b.y)));
  });
  if (!(a.flags & F_ADJ_IN)) return;
  fx_note(top, &ws.top[1], tid);
  __syncthreads();
  fx_column_inverse<PL, NT, 1>(sm, tw, static_cast<double2*>(a.w0), static_cast<double2*>(a.w1), kx, tid, &ws);
}

template <class PL, int V, int NT>
__global__ void __launch_bounds__(NT) k_adj_row_fx(StepArgs a) {
  pdl_wait();
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ FxWords wl, wv;
  fxc* lam = reinterpret_cast<fxc*>(smraw);
  fxc* vel = lam + PL::PADM * V;
  constexpr int M = PL::M, NP = PL::NP, R = PL::RP;
  const int tid = threadIdx.x, z0 = blockIdx.x * V;
  const int4* __restrict__ tw = static_cast<const int4*>(a.tw);
  FxScale sl, sv;
  fx_rows_inverse<PL, V, NT>(a.w0, a.w1, lam, tw, z0, tid, &wl, sl);
  fx_rows_inverse<PL, V, NT>(a.y0, a.y1, vel, tw, z0, tid, &wv, sv);
  // pointwise on values below 2^60: three products below 2^56 each stay below
  // the next pass's 2^58
  static_assert(fx_bits(R) >= 58, "three products of 2^56");
  const int dl = fx_shift_exact(wl.bits[NP - 1], 60), dv = fx_shift_exact(wv.bits[NP - 1], 60);
  FxRange rg;
  for (int w = tid; w < V * (M / R); w += NT) {
    const int at = (w / V) * (R + 1) * V + w % V;
    fxc l[R], q[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      l[j] = lam[at + j * V];
      q[j] = vel[at + j * V];
    }
    fx_rescale<R>(l, dl);
    fx_rescale<R>(q, dv);
#pragma unroll
    for (int j = 0; j < R; ++j)
      l[j] = fxc{fx_mul(2 * q[j].x, l[j].x) + fx_mul(q[j].y, l[j].y), fx_mul(q[j].x, l[j].y) - fx_mul(2 * q[j].y, l[j].x)};
    Dft<R, -1, fxc>::run(l);
#pragma unroll
    for (int j = 0; j < R; ++j) {
      lam[at + j * V] = l[j];
      rg.add(l[j]);
    }
  }
  fx_note(rg.word(), &wl.bits[2 * NP - 1], tid);
  FxScale sc{(sl.E - dl) + (sv.E - dv) + 64, sl.bad || sv.bad};
  __syncthreads();
  fx_dit<PL, V, NT, -1, NP - 2, 0, NP>(lam, tw, tid, &wl, sc);
  fx_rows_unpack<PL, V, NT>(a.w0, a.w1, lam, z0, tid, &wl, sc);
}

template <class PL, int V, int NT>
__global__ void __launch_bounds__(NT) k_adj_fwd_row_fx(StepArgs a) {
  pdl_wait();
  row_fx_body<PL, V, NT>(a, a.y0, a.y1, hw_blk());
}

template <class PL, int NT>
__global__ void __launch_bounds__(NT) k_adj_fwd_col_fx(StepArgs a) {
  pdl_wait();
  col_fx_body<PL, NT, true>(a, const_cast<void*>(a.y0), const_cast<void*>(a.y1), hw_blk());
}

template <class PL, int NT>
__global__ void __launch_bounds__(NT) k_adj_vel_fx(StepArgs a) {
  pdl_wait();
  extern __shared__ __align__(128) unsigned char smraw[];
  __shared__ FxWords ws;
  fxc* sm = reinterpret_cast<fxc*>(smraw);
  constexpr int M = PL::M, V = 2, N = 2 * M / 3;
  const int tid = threadIdx.x, kx = blockIdx.x;
  const double2* __restrict__ om = static_cast<const double2*>(a.om_p) + (size_t)kx * M;
  fx_words_clear<NT>(&ws, tid);
  __syncthreads();
  unsigned top = 0;
  for_column<PL, NT>(tid, [&](int p, int pos, bool in, int z) {
    fxc* s = sm + PL::phys(pos) * V;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const double2 x = in ? adj_velocity<double>(om[p], kx, z, N, v) : make_double2(0.0, 0.0);
      s[v] = fx_raw(x);
      top = max(top, max(fx_top(x.x), fx_top(x.y)));
    }
  });
  fx_note(top, &ws.top[1], tid);
  __syncthreads();
  fx_column_inverse<PL, NT, 1>(sm, static_cast<const int4*>(a.tw), static_cast<double2*>(const_cast<void*>(a.y0)),
                               static_cast<double2*>(const_cast<void*>(a.y1)), kx, tid, &ws);
}

}  // namespace pal
