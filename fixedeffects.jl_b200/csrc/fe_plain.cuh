// fe_plain.cuh -- the plain FP64 LSMR loop of narrow tiles (one problem, two
// to four fixed effects, at most 8 columns) as one cooperative kernel: the
// iterations of src/utils/lsmr.jl:101-219 with u formed row by row, the same
// recurrences and tests as the launched loop (fe_lsmr.cuh; the norms are summed
// in another order, so a count may differ by one), two passes and
// two grid barriers an iteration instead of six launches:
//   rows:    u <- s A v + c u, ||u||^2, and the primary FE's sums A_p'u, which
//            lie in row order;
//   levels:  the other FEs' sums over gathered rows of u, each followed at once
//            by its level's update of v, h, hbar and x; the primary levels'.
// Taken for small problems (plain_takes), which the barriers and the scalar
// step bound; large ones are as fast launched.  Measured per solve, launched
// loop -> this: 1M rows x 1, two effects, 0.68 -> 0.55 ms; the loop's kernel
// takes 0.24 ms there, 0.41 ms with three effects.
#pragma once

#include "fe_coef.cuh"

namespace fe {

// u <- s (A v) + c u over the positions of the primary FE's levels; s += c_p u
template <int C, int NG, int W>
struct PlainRowU {
  static constexpr int kGathers = NG + 1, kI = NG, kD = W == 2 ? NG + 1 : W;
  const PlainArgs& a;
  const CoefSmem<C>& sm;
  double (&nrm)[CoefShape<C>::VEC];
  int jl;
  CoefRow<C> tp;  // the level's own table row
  struct Val {
    CoefRow<C> u, t[NG];
  };
  __device__ __forceinline__ void level(int l) {
    if (l >= 0) tp.load(a.vs + (a.s.p.base + l) * C + coef_col0<C>(jl));
  }
  __device__ __forceinline__ const int32_t* idx_array(int i) const { return a.s.p.gi[i]; }
  __device__ __forceinline__ const double* dbl_array(int i) const { return a.s.p.d[i]; }
  template <int P>
  __device__ __forceinline__ void load(const int32_t* si, uint32_t i, uint32_t qa, Val& v) const {
    v.u.load(a.u + (int64_t)(qa + i) * C + coef_col0<C>(jl));
#pragma unroll
    for (int g = 0; g < NG; ++g)
      v.t[g].load(a.vs + (a.s.p.gb[g] + si[g * P + i]) * C + coef_col0<C>(jl));
  }
  template <int P>
  __device__ __forceinline__ void add(const double* sw, uint32_t i, uint32_t qa, const Val& v,
                                      CoefRow<C>& acc) const {
    const double cp = W == 1 ? sw[i] : W == 2 && a.s.p.d[0] ? sw[i] : 1.0;
    CoefRow<C> n;
#pragma unroll
    for (int e = 0; e < CoefShape<C>::VEC; ++e) {
      double x = W == 2 ? cp * tp.v[e] : tp.v[e];
#pragma unroll
      for (int g = 0; g < NG; ++g)
        x += (W == 2 && a.s.p.d[1 + g] ? sw[(1 + g) * P + i] * v.t[g].v[e] : v.t[g].v[e]);
      if (W == 1) x *= cp;
      const int j = coef_col<C>(jl, e);
      n.v[e] = sm.sc[0][j] * x + sm.sc[1][j] * v.u.v[e];
      nrm[e] += n.v[e] * n.v[e];
      acc.v[e] += W ? cp * n.v[e] : n.v[e];
    }
    n.store(a.u + (int64_t)(qa + i) * C + coef_col0<C>(jl));
  }
};
// s += c_k u over the positions of another FE's levels
template <int C, int W>
struct PlainRowS {
  static constexpr int kGathers = 1, kI = 1, kD = W ? 1 : 0;
  const double* u;
  const CoefSide& sd;
  using Val = CoefRow<C>;
  __device__ __forceinline__ void level(int) {}
  __device__ __forceinline__ const int32_t* idx_array(int) const { return sd.perm; }
  __device__ __forceinline__ const double* dbl_array(int) const { return sd.dw; }
  template <int P>
  __device__ __forceinline__ void load(const int32_t* si, uint32_t i, uint32_t qa, Val& v) const {
    v.load(u + (sd.perm ? (int64_t)si[i] : (int64_t)(qa + i)) * C);
  }
  template <int P>
  __device__ __forceinline__ void add(const double* sw, uint32_t i, uint32_t, const Val& v,
                                      CoefRow<C>& acc) const {
    const double c = W && sd.dw ? sw[i] : 1.0;
#pragma unroll
    for (int e = 0; e < CoefShape<C>::VEC; ++e)
      acc.v[e] = W ? fma(c, v.v[e], acc.v[e]) : acc.v[e] + v.v[e];
  }
};

// The update of one level's columns (as PEpiLsmr of the launched loop): s its
// sum A'u, sc its scale; na, nb: ||v||^2 and ||x||^2.
template <int C>
__device__ __forceinline__ void plain_update(const PlainArgs& a, const CoefSmem<C>& sm, int64_t row,
                                             double sc, const CoefRow<C>& s, int jl,
                                             double (&na)[CoefShape<C>::VEC],
                                             double (&nb)[CoefShape<C>::VEC]) {
  const int64_t o = row * C + coef_col0<C>(jl);
  CoefRow<C> v, h, hb, x, vs;
  v.load(a.v + o);
  h.load(a.h + o);
  hb.load(a.hb + o);
  x.load(a.x + o);
#pragma unroll
  for (int e = 0; e < CoefShape<C>::VEC; ++e) {
    const int j = coef_col<C>(jl, e), m = sm.mode[j];
    const double vo = sm.sc[6][j] * v.v[e];
    if (m == 2) {
      const double hbn = h.v[e] + sm.sc[3][j] * hb.v[e];
      hb.v[e] = hbn;
      x.v[e] += sm.sc[4][j] * hbn;
      h.v[e] = vo + sm.sc[5][j] * h.v[e];
    } else if (m) {
      h.v[e] = vo;
      hb.v[e] = 0.0;
      if (m == 3) x.v[e] = 0.0;
    }
    if (m) nb[e] += x.v[e] * x.v[e];
    if (sm.vact[j]) {
      const double vn = s.v[e] * sc * sm.sc[2][j] - sm.svp[j] * v.v[e];
      v.v[e] = vn;
      na[e] += vn * vn;
    }
    vs.v[e] = v.v[e] * sc;
  }
  v.store(a.v + o);
  h.store(a.h + o);
  hb.store(a.hb + o);
  x.store(a.x + o);
  vs.store(a.vs + o);
}

template <int C, int NG, int W>
__device__ __noinline__ void plain_pass_u(const PlainArgs& a, CoefSmem<C>& sm, int par) {
  const int jl = (threadIdx.x & 31) % CoefShape<C>::CL;
  double nrm[1][CoefShape<C>::VEC];
  coef_clear<C>(nrm);
  const CoefSide& sd = a.s.p;
  coef_sweep<C, NG, W>(a.s, sd, PlainRowU<C, NG, W>{a, sm, nrm[0], jl, {}}, nrm,
                       coef_epi<1>(sd.lev, [&](int l, const auto&, CoefRow<C>& s, int jl, auto&) {
                         s.store(a.sp + (int64_t)l * C + coef_col0<C>(jl));
                       }));
  coef_publish<C, 1>(nrm, sm, a.s.part, par);
}

template <int C, int NG, int W>
__device__ __noinline__ void plain_pass_v(const PlainArgs& a, CoefSmem<C>& sm, int par) {
  using Sh = CoefShape<C>;
  const int lane = threadIdx.x & 31, jl = lane % Sh::CL;
  double nrm[2][Sh::VEC];
  coef_clear<C>(nrm);
#pragma unroll 1
  for (int f = 0; f < NG; ++f) {
    const CoefSide& sd = a.s.f[f];
    coef_sweep<C, NG, W>(a.s, sd, PlainRowS<C, W>{a.u + coef_col0<C>(jl), sd}, nrm,
                         coef_epi<1>(sd.lev, [&](int l, const auto& k, CoefRow<C>& s, int jl, auto& nr) {
                           plain_update<C>(a, sm, sd.base + l, k.v[0], s, jl, nr[0], nr[1]);
                         }));
  }
  const int64_t r0 =
      ((int64_t)blockIdx.x * kCoefWarps + (threadIdx.x >> 5)) * Sh::R + lane / Sh::CL;
  for (int64_t r = r0; r < a.s.p.n; r += (int64_t)gridDim.x * kCoefWarps * Sh::R) {
    CoefRow<C> s;
    s.load(a.sp + r * C + coef_col0<C>(jl));
    plain_update<C>(a, sm, a.s.p.base + r, __ldg(a.s.p.lev + r), s, jl, nrm[0], nrm[1]);
  }
  coef_publish<C, 2>(nrm, sm, a.s.part, par);
}

template <int C, int NG, int W>
__global__ void __launch_bounds__(kCoefThreads, 1) k_plain(const PlainArgs args) {
  __shared__ PlainArgs a;
  CoefSmem<C>& sm = *reinterpret_cast<CoefSmem<C>*>(coef_dyn);
  const int tid = threadIdx.x;
  if (tid == 0) a = args;
  uint32_t gen = 0;
  int par = 0;
  if (tid < C) sm.inst[tid] = args.s.inst[tid];
  __syncthreads();
  // the instances' coefficients (the launched loop reads them from Inst)
  auto set = [&](int j) {
    const Inst& s = sm.inst[j];
    sm.sc[0][j] = s.ex_av;
    sm.sc[1][j] = s.ex_au;
    sm.sc[3][j] = s.c1;
    sm.sc[4][j] = s.c2;
    sm.sc[5][j] = s.c3;
    sm.sc[6][j] = s.s_v;
    sm.mode[j] = s.active ? s.upd_mode : 0;
  };
  if (tid < C) set(tid);
  // the prescaled table of the first v
  {
    using Sh = CoefShape<C>;
    const int lane = tid & 31, jl = lane % Sh::CL;
    for (int f = 0; f <= NG; ++f) {
      const CoefSide& sd = f < NG ? a.s.f[f] : a.s.p;
      const int64_t r0 = ((int64_t)blockIdx.x * kCoefWarps + (tid >> 5)) * Sh::R + lane / Sh::CL;
      for (int64_t r = r0; r < sd.n; r += (int64_t)gridDim.x * kCoefWarps * Sh::R) {
        const int64_t o = (sd.base + r) * C + coef_col0<C>(jl);
        CoefRow<C> v;
        v.load(a.v + o);
        const double sc = __ldg(sd.lev + r);
#pragma unroll
        for (int e = 0; e < Sh::VEC; ++e) v.v[e] *= sc;
        v.store(a.vs + o);
      }
    }
  }
  bool alive = coef_barrier(a.s, gen, &sm.ok);
  bool any = __syncthreads_or(tid < C && sm.inst[tid].active);
  while (alive && any) {
    plain_pass_u<C, NG, W>(a, sm, par);
    alive = coef_barrier(a.s, gen, &sm.ok);
    if (!alive) break;
    coef_totals<C, 1>(sm, a.s, par, a.s.multi_p, a.s.nmulti);
    par ^= 1;
    if (tid < C) {
      // beta = ||u||; if beta > 0: u /= beta, v = A'u - beta v  (lsmr.jl:104-108)
      Inst& s = sm.inst[tid];
      sm.vact[tid] = 0;
      if (s.active) {
        s.beta = sqrt(sm.tot[0][tid]);
        s.do_v = s.beta > 0 ? 1 : 0;
        s.u_scale = s.do_v ? 1.0 / s.beta : 1.0;
        sm.sc[2][tid] = s.u_scale;
        sm.svp[tid] = s.beta * s.s_v;
        sm.vact[tid] = s.do_v;
      }
    }
    __syncthreads();
    plain_pass_v<C, NG, W>(a, sm, par);
    alive = coef_barrier(a.s, gen, &sm.ok);
    if (!alive) break;
    coef_totals<C, 2>(sm, a.s, par, 0, a.s.multi_p);
    par ^= 1;
    if (tid < C) {
      Inst& s = sm.inst[tid];
      if (s.active) {
        if (s.pending) {
          s.normx = sqrt(sm.tot[1][tid]);
          lsmr_test(s);
          s.pending = 0;
          if (s.istop) deactivate(s);
        }
        if (s.active) {
          s.iter += 1;
          if (s.do_v) {
            s.alpha = sqrt(sm.tot[0][tid]);
            s.s_v = s.alpha > 0 ? 1.0 / s.alpha : 1.0;
          }
          lsmr_rotate(s);
          s.upd_mode = 2;
          s.pending = 1;
          s.ex_av = s.s_v;
          s.ex_au = -s.alpha * s.u_scale;
        }
      }
      set(tid);
    }
    any = __syncthreads_or(tid < C && sm.inst[tid].active);
  }
  if (blockIdx.x == 0 && tid < C) a.s.inst[tid] = sm.inst[tid];
}

template <int C>
const void* plain_kernel(int nf, int w) {
  switch (nf * 3 + w) {
    case 3: return (const void*)k_plain<C, 1, 0>;
    case 4: return (const void*)k_plain<C, 1, 1>;
    case 5: return (const void*)k_plain<C, 1, 2>;
    case 6: return (const void*)k_plain<C, 2, 0>;
    case 7: return (const void*)k_plain<C, 2, 1>;
    case 8: return (const void*)k_plain<C, 2, 2>;
    case 9: return (const void*)k_plain<C, 3, 0>;
    case 10: return (const void*)k_plain<C, 3, 1>;
    default: return (const void*)k_plain<C, 3, 2>;
  }
}

}  // namespace fe
