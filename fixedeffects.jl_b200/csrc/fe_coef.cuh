// fe_coef.cuh -- the coefficient-side solve (fe_coef.h) as one cooperative
// kernel: every pass over the data, the FP64 scalar recurrences and the
// stopping tests of a tile run in a single launch, with grid-wide barriers
// between the passes.  Included by one translation unit per tile width.
//
// What bounds it: the row-side loop reads and writes the N x C rows and reads
// them again for the sums of the other FEs, four launches an iteration; here
// an iteration reads the level ids (and weights) once in every FE's order and
// gathers one row of a coefficient table per entry, from L1 or L2 unless the
// primary FE's table outgrows them, in two passes.  Large problems are bound
// by the passes' instructions and the latency of their gathers (0.8 warp
// instructions per SM and cycle, 4 to 5 per row and pass), small ones by the
// chain of loads of a pass (of 23.6 us an iteration at 800k rows and two
// effects the two passes take 14.1 us, averaged over the CTAs, the waits for
// the slowest CTA and the barriers 6.0, the sums of the norms 2.4, the scalar
// steps 1.1; in one CTA, 2k rows, 7.5, 0.2, 2.4 and 1.5 of 11.6 us).  Measured
// per solve, against the row-side loop: 100M rows x 8 weighted columns 84.0 ->
// 38.9 ms, 10M x 1 with three effects, one interacted, 3.4 -> 3.0 ms, 150k x 5
// 0.91 -> 0.41 ms, 2k x 1 0.41 -> 0.14 ms, 800k x 1 of 5184 iterations 268 ->
// 122 ms (FP64 throughout needs one inner solve where FP32 took three).
#pragma once

#include <algorithm>

#include "fe_coef.h"
#include "fe_lsmr.cuh"

namespace fe {

extern __shared__ __align__(16) unsigned char coef_dyn[];  // CoefSmem, then the warps' windows

// Lane layout of a C-column row: CL lanes of NCH two-column chunks each, so
// that a chunk of the row is one contiguous load of the lanes; R rows side by
// side in a warp.  A lane holds up to four columns: the index and weight of a
// row are then read by few lanes.
template <int C>
struct CoefShape {
  static constexpr int CW = C >= 2 ? 2 : 1;
  static constexpr int NCH = C >= 4 ? 2 : 1;
  static constexpr int VEC = CW * NCH;
  static constexpr int CL = C / VEC;
  static constexpr int R = 32 / CL;
};
// resident CTAs per SM: 16 warps of up to 128 registers, which keeps the walk
// free of spills (at 64 registers their reloads took half of L1's cycles), or
// 32 warps of 64 where the passes wait for the gathers of a large table.
// Measured, pair of passes: 800k x 1 28 us with 32 warps, 19 us with 16; 2M x
// 3 weighted 106 and 95 us; 100M x 8 weighted 3.39 and 3.49 ms.
template <int C, int NG, int W>
constexpr int kCoefCtas() {
  return C == 8 && NG == 1 && W < 2 ? 2 : 1;
}
// rows in flight per lane of a pass with G gathers per row
template <int C, int NG, int W>
constexpr int coef_unroll(int G) {
  return G * CoefShape<C>::VEC * kCoefCtas<C, NG, W>() <= 4 ? 4 : 2;
}

template <int C>
struct CoefRow {
  using Sh = CoefShape<C>;
  double v[Sh::VEC];
  __device__ __forceinline__ void load(const double* row) {  // row: at the lane's first column
    if constexpr (Sh::CW == 1) {
      v[0] = row[0];
    } else {
#pragma unroll
      for (int c = 0; c < Sh::NCH; ++c) {
        const double2 t = *reinterpret_cast<const double2*>(row + c * Sh::CL * 2);
        v[2 * c] = t.x;
        v[2 * c + 1] = t.y;
      }
    }
  }
  __device__ __forceinline__ void load(const float* row) {
    if constexpr (Sh::CW == 1) {
      v[0] = (double)row[0];
    } else {
#pragma unroll
      for (int c = 0; c < Sh::NCH; ++c) {
        const float2 t = *reinterpret_cast<const float2*>(row + c * Sh::CL * 2);
        v[2 * c] = (double)t.x;
        v[2 * c + 1] = (double)t.y;
      }
    }
  }
  __device__ __forceinline__ void store(double* row) const {
    if constexpr (Sh::CW == 1) {
      row[0] = v[0];
    } else {
#pragma unroll
      for (int c = 0; c < Sh::NCH; ++c)
        *reinterpret_cast<double2*>(row + c * Sh::CL * 2) = make_double2(v[2 * c], v[2 * c + 1]);
    }
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < Sh::VEC; ++i) v[i] = 0.0;
  }
};
// the lane's first column, and the column of element i of its row
template <int C>
__device__ __forceinline__ int coef_col0(int jl) {
  return CoefShape<C>::CW * jl;
}
template <int C>
__device__ __forceinline__ int coef_col(int jl, int i) {
  using Sh = CoefShape<C>;
  return Sh::CW == 1 ? 0 : ((i / 2) * Sh::CL + jl) * 2 + (i & 1);
}

// Grid-wide barrier of the co-resident CTAs of a cooperative launch.  A wait
// is bounded: a CTA that gives up sets bar[1], which ends every other wait.
// (It may be seen by that CTA alone, the last one may have arrived since, so
// bar[1] decides whether the launch counts, not what one CTA saw.)
__device__ __forceinline__ bool coef_barrier(const CoefArgs& a, uint32_t& gen, int* sm_ok) {
  uint32_t* const bar = a.bar;
  __syncthreads();
  if (gridDim.x == 1) return true;
  if (threadIdx.x == 0) {
    gen += gridDim.x;
    __threadfence();
    atomicAdd(bar, 1u);
    int ok = 1;
    uint32_t spins = 0;
    while ((int32_t)(*(volatile uint32_t*)bar - gen) < 0) {
      if (++spins > a.spins || ((spins & 255u) == 0 && *(volatile uint32_t*)(bar + 1) != 0)) {
        atomicExch(bar + 1, 1u);
        ok = 0;
        break;
      }
    }
    __threadfence();
    *sm_ok = ok;
  }
  __syncthreads();
  return *sm_ok != 0;
}

template <int C>
struct alignas(16) CoefSmem {
  double red[3][kCoefWarps][C];
  double tot[3][C];
  // per column: cS, cV, cP (v update), c1, c2, c3 (deferred update), s_v
  double sc[7][C];
  double svp[C], irr[C], nb2[C], nall[C], dt2[C];
  int vact[C], mode[C];
  Inst inst[C];
  int ok;
};

// norms of this CTA -> its slot of the partial buffer (`par` alternates, so a
// CTA that is still reading the previous totals is not overtaken)
template <int C, int NQ>
__device__ __forceinline__ void coef_publish(const double (&nrm)[NQ][CoefShape<C>::VEC],
                                             CoefSmem<C>& sm, double* part, int par) {
  using Sh = CoefShape<C>;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, jl = lane % Sh::CL;
#pragma unroll
  for (int k = 0; k < NQ; ++k)
#pragma unroll
    for (int v = 0; v < Sh::VEC; ++v) {
      double t = nrm[k][v];
#pragma unroll
      for (int o = Sh::CL; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane < Sh::CL) sm.red[k][wib][coef_col<C>(jl, v)] = t;
    }
  __syncthreads();
  for (int t = threadIdx.x; t < NQ * C; t += kCoefThreads) {
    const int k = t / C, j = t - k * C;
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < kCoefWarps; ++w) s += sm.red[k][w][j];
    part[((int64_t)(par * 3 + k) * gridDim.x + blockIdx.x) * C + j] = s;
  }
}
// after the barrier: every CTA sums all slots in the same order (m0..m1: the
// pass's levels with slots of their own)
template <int C, int NQ>
__device__ __forceinline__ void coef_totals(CoefSmem<C>& sm, const CoefArgs& a, int par, int m0,
                                            int m1) {
  constexpr int PER = kCoefThreads / C;  // threads per column
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int j = threadIdx.x % C, p0 = threadIdx.x / C;
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    const double* pk = a.part + (int64_t)(par * 3 + k) * gridDim.x * C + j;
    const double* mk = a.mnrm + (int64_t)k * a.nmulti * C + j;
    double s = 0.0;
#pragma unroll 8
    for (int b = p0; b < (int)gridDim.x; b += PER) s += __ldcg(pk + (int64_t)b * C);
#pragma unroll 16
    for (int b = m0 + p0; b < m1; b += PER) s += __ldcg(mk + (int64_t)b * C);
#pragma unroll
    for (int o = C; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane < C) sm.red[k][wib][j] = s;
  }
  __syncthreads();
  // 16 lanes per column add the warps' sums
  if (threadIdx.x < (16 * C < 32 ? 32 : 16 * C)) {
    const int col = threadIdx.x / 16, w = threadIdx.x % 16;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      double s = 0.0;
      for (int q = w; q < kCoefWarps && col < C; q += 16) s += sm.red[k][q][col];
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (w == 0 && col < C) sm.tot[k][col] = s;
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void coef_copy16(void* smem, const void* gmem, int bytes) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}

// Sums `row` over the positions of every level of a side and hands each sum
// to `epi` on the lanes that own the level's columns.
//
// A warp walks its items (whole levels of at most T positions together, or a
// piece of a longer level) window by window: the next window's indices and
// weights are copied to shared memory while the current one's rows are
// gathered, so a row costs one shared-memory read per index and weight, its
// gathers, and its arithmetic.  A window starts at a multiple of 4 positions
// (every copy is 16 aligned bytes) and is at most P = T + 4 positions long.
// In an item of whole levels a team of CL << rlog lanes takes a level; rlog
// and the levels per item are chosen so that the teams of a warp take whole
// rounds of levels (coef_items).  The warp that finishes a level of several
// pieces last adds them in order: the order of every sum is fixed by the plan
// and the grid.
//
// epi.pre loads a level's constants (before its rows); epi adds its norms to
// nrm; those of a level finished by whichever warp came last go to the level's
// own slot (coef_totals adds them in order).
template <int C, int NG, int W, class Row, int NQ, class Epi>
__device__ __forceinline__ void coef_sweep(const CoefArgs& a, const CoefSide& sd, Row row,
                                           double (&nrm)[NQ][CoefShape<C>::VEC], const Epi& epi) {
  using Sh = CoefShape<C>;
  constexpr int CL = Sh::CL, VEC = Sh::VEC;
  constexpr int T = coef_window(NG, W), P = T + 4;
  constexpr int kIBytes = Row::kI * P * 4, kBytes = kIBytes + Row::kD * P * 8;
  constexpr int U = coef_unroll<C, NG, W>(Row::kGathers);
  constexpr uint32_t kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, jl = lane % CL, wib = threadIdx.x >> 5;
  const uint32_t nw = gridDim.x * kCoefWarps, nitems = sd.nitems;
  uint32_t it = blockIdx.x * kCoefWarps + wib;
  if (it >= nitems) return;
  unsigned char* const ring = coef_dyn + sizeof(CoefSmem<C>) + wib * 2 * kBytes;
  const int4* __restrict__ items = reinterpret_cast<const int4*>(sd.items);
  const int32_t* __restrict__ off = sd.off;
  const uint32_t npos = sd.npos;
  const int rlog = sd.rlog, tl = CL << rlog, nt = 32 / tl, team = lane / tl;
  const uint32_t rr = (uint32_t)(lane % tl) / CL;
  // item: {first position, end, first level, levels} or {.., level, -1 - piece}
  auto item = [&](uint32_t i) {
    return i < nitems ? __ldg(items + i) : make_int4(0, 0, 0, 0);
  };
  auto begin_of = [&](const int4& d) -> uint32_t {  // the lane's level of a whole-level item
    return lane < d.w ? (uint32_t)__ldg(off + d.z + lane) : (uint32_t)d.y;
  };
  const int32_t* ia[Row::kI > 0 ? Row::kI : 1];
  const double* da[Row::kD > 0 ? Row::kD : 1];
#pragma unroll
  for (int i = 0; i < Row::kI; ++i) ia[i] = row.idx_array(i);
#pragma unroll
  for (int i = 0; i < Row::kD; ++i) da[i] = row.dbl_array(i);
  int4 cur = item(it), nxt = item(it + nw), nn = item(it + 2 * nw);
  uint32_t lb = begin_of(cur), lbn = begin_of(nxt);
  // the single constant of the lane's level, ahead of its rows
  auto ahead_of = [&](const int4& d) -> double {
    return Epi::kAhead && lane < d.w ? __ldg(epi.lev + d.z + lane) : 0.0;
  };
  double ah = ahead_of(cur), ahn = ahead_of(nxt);
  auto issue = [&](uint32_t q0, uint32_t q1, int stage) {
    unsigned char* const st = ring + stage * kBytes;
    const uint32_t qa = q0 & ~3u, n = q1 - qa, left = npos - qa;
#pragma unroll
    for (int i = 0; i < Row::kI; ++i) {
      const int32_t* const src = ia[i];
      if (!src) continue;
      const uint32_t c = lane * 4;
      if (c < n)
        coef_copy16(st + (i * P + c) * 4, src + qa + c, left - c < 4 ? (int)(left - c) * 4 : 16);
    }
#pragma unroll
    for (int i = 0; i < Row::kD; ++i) {
      const double* const src = da[i];
      if (!src) continue;
#pragma unroll
      for (int h = 0; h < P; h += 64) {
        const uint32_t c = lane * 2 + h;
        if (c < n)
          coef_copy16(st + kIBytes + (i * P + c) * 8, src + qa + c, left - c < 2 ? 8 : 16);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  static_assert(P <= 128, "one 16-byte copy of indices per lane");
  int stage = 0;
  uint32_t q0 = cur.x, q1 = min((uint32_t)cur.x + T, (uint32_t)cur.y);
  issue(q0, q1, 0);
  CoefRow<C> acc;
  acc.zero();
  for (;;) {
    const bool same = q1 < (uint32_t)cur.y;  // the item goes on in another window
    const uint32_t n0 = same ? q1 : (uint32_t)nxt.x;
    const uint32_t n1 = min(n0 + T, same ? (uint32_t)cur.y : (uint32_t)nxt.y);
    issue(n0, n1, stage ^ 1);
    asm volatile("cp.async.wait_group 1;\n" ::);
    __syncwarp();
    const uint32_t qa = q0 & ~3u;
    const int32_t* const si = reinterpret_cast<const int32_t*>(ring + stage * kBytes);
    const double* const sw = reinterpret_cast<const double*>(ring + stage * kBytes + kIBytes);
    auto walk = [&](uint32_t i, uint32_t e, uint32_t stride) {  // local positions
      typename Row::Val val[U];
      for (; i + (U - 1) * stride < e; i += U * stride) {
#pragma unroll
        for (int u = 0; u < U; ++u) row.template load<P>(si, i + u * stride, qa, val[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) row.template add<P>(sw, i + u * stride, qa, val[u], acc);
      }
      if (i < e) {
#pragma unroll
        for (int u = 0; u < U - 1; ++u)
          if (i + u * stride < e) row.template load<P>(si, i + u * stride, qa, val[u]);
#pragma unroll
        for (int u = 0; u < U - 1; ++u)
          if (i + u * stride < e) row.template add<P>(sw, i + u * stride, qa, val[u], acc);
      }
    };
    if (cur.w >= 0) {
      uint32_t le = __shfl_down_sync(kAll, lb, 1);
      if (lane == 31) le = cur.y;
      for (int i0 = 0; i0 < cur.w; i0 += nt) {
        const int i = i0 + team;
        const uint32_t b = __shfl_sync(kAll, lb, i & 31) - qa;
        const uint32_t e = __shfl_sync(kAll, le, i & 31) - qa;
        const bool own = i < cur.w;
        typename Epi::Pre pre;
        if constexpr (Epi::kAhead) pre.v[0] = __shfl_sync(kAll, ah, i & 31);
        else pre = epi.pre(own ? cur.z + i : -1);
        acc.zero();
        row.level(own ? cur.z + i : -1);
        walk(b + rr, own ? e : 0, 1u << rlog);
        __syncwarp();
        for (int o = CL; o < tl; o <<= 1)
#pragma unroll
          for (int v = 0; v < VEC; ++v) acc.v[v] += __shfl_xor_sync(kAll, acc.v[v], o);
        if (own && rr == 0) epi(cur.z + i, pre, acc, jl, nrm);
      }
    } else {
      row.level(cur.z);
      walk(q0 - qa + lane / CL, q1 - qa, Sh::R);
      __syncwarp();
      if (!same) {
#pragma unroll
        for (int o = CL; o < 32; o <<= 1)
#pragma unroll
          for (int v = 0; v < VEC; ++v) acc.v[v] += __shfl_xor_sync(kAll, acc.v[v], o);
        const CoefPiece pc = sd.pieces[-1 - cur.w];
        if (pc.np == 1) {
          if (lane < CL) epi(cur.z, epi.pre(cur.z), acc, jl, nrm);
        } else {
          if (lane < CL)
            acc.store(a.ppart + (int64_t)(sd.piece0 - 1 - cur.w) * C + coef_col0<C>(jl));
          __threadfence();
          __syncwarp();
          int last = 0;
          if (lane == 0) last = atomicAdd(a.pcnt + pc.cnt, 1) == pc.np - 1 ? 1 : 0;
          last = __shfl_sync(kAll, last, 0);
          if (last) {
            __threadfence();
            acc.zero();
            const double* pp = a.ppart + (int64_t)(sd.piece0 + pc.first) * C;
#pragma unroll 4
            for (int j = lane / CL; j < pc.np; j += Sh::R) {
#pragma unroll
              for (int v = 0; v < VEC; ++v)
                acc.v[v] += __ldcg(pp + (int64_t)j * C + coef_col<C>(jl, v));
            }
#pragma unroll
            for (int o = CL; o < 32; o <<= 1)
#pragma unroll
              for (int v = 0; v < VEC; ++v) acc.v[v] += __shfl_xor_sync(kAll, acc.v[v], o);
            if (lane == 0) a.pcnt[pc.cnt] = 0;
            if (lane < CL) {
              double own[NQ][VEC];
#pragma unroll
              for (int k = 0; k < NQ; ++k)
#pragma unroll
                for (int v = 0; v < VEC; ++v) own[k][v] = 0.0;
              epi(cur.z, epi.pre(cur.z), acc, jl, own);
#pragma unroll
              for (int k = 0; k < NQ; ++k)
#pragma unroll
                for (int v = 0; v < VEC; ++v)
                  a.mnrm[((int64_t)k * a.nmulti + pc.cnt) * C + coef_col<C>(jl, v)] = own[k][v];
            }
          }
        }
        acc.zero();
      }
    }
    __syncwarp();  // the stage is refilled by the next issue
    if (!same) {
      it += nw;
      if (it >= nitems) break;
      cur = nxt;
      lb = lbn;
      nxt = nn;
      nn = item(it + 2 * nw);
      lbn = begin_of(nxt);
      ah = ahn;
      ahn = ahead_of(nxt);
    }
    q0 = n0;
    q1 = n1;
    stage ^= 1;
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
}

// ---------------------------------------------------------------------------
// row functors (see coef_sweep): kI index arrays and kD weight arrays are
// staged; load gathers the rows of local position i, add sums them up.  W: 0
// no weights, 1 weights alone (one array for every entry), 2 interactions: the
// entries' products of weights and interactions, slot 0.. of the distinct
// arrays or -1 for 1.  level announces the team's level before its rows.
// ---------------------------------------------------------------------------
template <int W, int P>
__device__ __forceinline__ double coef_weight(const double* sw, int slot, uint32_t i) {
  if (W == 0) return 1.0;
  if (W == 1) return sw[i];
  return slot >= 0 ? sw[slot * P + i] : 1.0;
}
// s += sum_g c_g t_g[level]: the primary side of A_r t.  With several other
// FEs also nrm += w tau^2, tau the observation's sum (with one, that norm is
// a sum over its levels, see coef_pass_f).
template <int C, int NG, int W>
struct CoefRowP {
  static constexpr int kGathers = NG, kI = NG;
  static constexpr int kD = W == 2 && NG > 1 ? NG + 2 : W > 0 ? 1 : 0;
  const double* t[NG];
  double (&nrm)[CoefShape<C>::VEC];
  const CoefSide& sd;
  int slot[NG], sx, sn;
  struct Val {
    CoefRow<C> t[NG];
  };
  __device__ __forceinline__ CoefRowP(const CoefSide& s, const double* tab, int jl,
                                      double (&n)[CoefShape<C>::VEC])
      : nrm(n), sd(s), sx(s.slot_w), sn(s.slot_n) {
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      t[g] = tab + s.gb[g] * C + coef_col0<C>(jl);
      slot[g] = s.slot_g[g];
    }
  }
  __device__ __forceinline__ void level(int) {}
  __device__ __forceinline__ const int32_t* idx_array(int i) const { return sd.gi[i]; }
  __device__ __forceinline__ const double* dbl_array(int i) const { return sd.d[i]; }
  template <int P>
  __device__ __forceinline__ void load(const int32_t* si, uint32_t i, uint32_t, Val& v) const {
#pragma unroll
    for (int g = 0; g < NG; ++g) v.t[g].load(t[g] + (int64_t)si[g * P + i] * C);
  }
  template <int P>
  __device__ __forceinline__ void add(const double* sw, uint32_t i, uint32_t, const Val& v,
                                      CoefRow<C>& acc) const {
    if constexpr (NG == 1) {
      const double c = coef_weight<W, P>(sw, slot[0], i);
#pragma unroll
      for (int e = 0; e < CoefShape<C>::VEC; ++e)
        acc.v[e] = W ? fma(c, v.t[0].v[e], acc.v[e]) : acc.v[e] + v.t[0].v[e];
    } else {
      // W = 2: c_g = x_g, then w x_p (slot_w) and w (slot_n) times the sum
      double c[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) c[g] = W == 2 ? coef_weight<2, P>(sw, slot[g], i) : 1.0;
      const double w = W == 2 ? coef_weight<2, P>(sw, sn, i) : coef_weight<W, P>(sw, 0, i);
      const double wx = W == 2 ? coef_weight<2, P>(sw, sx, i) : w;
#pragma unroll
      for (int e = 0; e < CoefShape<C>::VEC; ++e) {
        double tau = W == 2 ? c[0] * v.t[0].v[e] : v.t[0].v[e];
#pragma unroll
        for (int g = 1; g < NG; ++g)
          tau = W == 2 ? fma(c[g], v.t[g].v[e], tau) : tau + v.t[g].v[e];
        acc.v[e] = W ? fma(wx, tau, acc.v[e]) : acc.v[e] + tau;
        nrm[e] = fma(W ? w * tau : tau, tau, nrm[e]);
      }
    }
  }
};
// s += sum over the other FEs of c_g t_g - c_z z: another FE's side, without
// its own table rows (added by the caller, one product per level)
template <int C, int NO, int W>
struct CoefRowF {
  static constexpr int NA = NO > 0 ? NO : 1;
  static constexpr int kGathers = NO + 1, kI = NO + 1, kD = W == 2 ? NO + 1 : W;
  const double* z;
  const double* t[NA];
  const CoefSide& sd;
  int sz, slot[NA];
  struct Val {
    CoefRow<C> z, t[NA];
  };
  __device__ __forceinline__ CoefRowF(const CoefSide& s, const double* tab, const double* zz, int jl)
      : z(zz + coef_col0<C>(jl)), sd(s), sz(s.slot_w) {
#pragma unroll
    for (int g = 0; g < NO; ++g) {
      t[g] = tab + s.gb[g] * C + coef_col0<C>(jl);
      slot[g] = s.slot_g[g];
    }
  }
  __device__ __forceinline__ void level(int) {}
  __device__ __forceinline__ const int32_t* idx_array(int i) const {
    return i == 0 ? sd.zi : sd.gi[i - 1];
  }
  __device__ __forceinline__ const double* dbl_array(int i) const { return sd.d[i]; }
  template <int P>
  __device__ __forceinline__ void load(const int32_t* si, uint32_t i, uint32_t, Val& v) const {
    v.z.load(z + (int64_t)si[i] * C);
#pragma unroll
    for (int g = 0; g < NO; ++g) v.t[g].load(t[g] + (int64_t)si[(1 + g) * P + i] * C);
  }
  template <int P>
  __device__ __forceinline__ void add(const double* sw, uint32_t i, uint32_t, const Val& v,
                                      CoefRow<C>& acc) const {
    const double cz = coef_weight<W, P>(sw, sz, i);
    double c[NA];
#pragma unroll
    for (int g = 0; g < NO; ++g) c[g] = W == 2 ? coef_weight<2, P>(sw, slot[g], i) : cz;
#pragma unroll
    for (int e = 0; e < CoefShape<C>::VEC; ++e) {
      if (W == 2) {
        acc.v[e] = fma(-cz, v.z.v[e], acc.v[e]);
#pragma unroll
        for (int g = 0; g < NO; ++g) acc.v[e] = fma(c[g], v.t[g].v[e], acc.v[e]);
      } else {
        double tau = NO > 0 ? v.t[0].v[e] - v.z.v[e] : -v.z.v[e];
#pragma unroll
        for (int g = 1; g < NO; ++g) tau += v.t[g].v[e];
        acc.v[e] = W ? fma(cz, tau, acc.v[e]) : acc.v[e] + tau;
      }
    }
  }
};
// the primary side of b: s += w x_p y, nrm += w y^2
template <int C, int W>
struct CoefRowYP {
  static constexpr int kGathers = 1, kI = 0, kD = W;
  const float* y;
  const CoefSide& sd;
  double (&nrm)[CoefShape<C>::VEC];
  using Val = CoefRow<C>;
  __device__ __forceinline__ void level(int) {}
  __device__ __forceinline__ const int32_t* idx_array(int) const { return nullptr; }
  __device__ __forceinline__ const double* dbl_array(int i) const { return i ? sd.dwx : sd.dw; }
  template <int P>
  __device__ __forceinline__ void load(const int32_t*, uint32_t i, uint32_t qa, Val& v) const {
    v.load(y + (int64_t)(qa + i) * C);
  }
  template <int P>
  __device__ __forceinline__ void add(const double* sw, uint32_t i, uint32_t, const Val& v,
                                      CoefRow<C>& acc) const {
    const double w = coef_weight<W, P>(sw, sd.dw ? 0 : -1, i);
    const double wx = W == 2 ? coef_weight<2, P>(sw, sd.dwx ? 1 : -1, i) : w;
#pragma unroll
    for (int e = 0; e < CoefShape<C>::VEC; ++e) {
      acc.v[e] = W ? fma(wx, v.v[e], acc.v[e]) : acc.v[e] + v.v[e];
      nrm[e] = fma(W ? w * v.v[e] : v.v[e], v.v[e], nrm[e]);
    }
  }
};
// ||M b||^2 from the projected rows: nrm += w (y - x_p zb)^2
template <int C, int W>
struct CoefRowB {
  static constexpr int kGathers = 1, kI = 0, kD = W;
  const float* y;
  const double* zb;
  const CoefSide& sd;
  double (&nrm)[CoefShape<C>::VEC];
  CoefRow<C> z;  // the level's
  using Val = CoefRow<C>;
  __device__ __forceinline__ void level(int l) {
    if (l >= 0) z.load(zb + (int64_t)l * C);
  }
  __device__ __forceinline__ const int32_t* idx_array(int) const { return nullptr; }
  __device__ __forceinline__ const double* dbl_array(int i) const { return i ? sd.dwx : sd.dw; }
  template <int P>
  __device__ __forceinline__ void load(const int32_t*, uint32_t i, uint32_t qa, Val& v) const {
    v.load(y + (int64_t)(qa + i) * C);
  }
  template <int P>
  __device__ __forceinline__ void add(const double* sw, uint32_t i, uint32_t, const Val& v,
                                      CoefRow<C>&) const {
    const double w = coef_weight<W, P>(sw, sd.dw ? 0 : -1, i);
    const double xp = W == 2 && w != 0.0 ? coef_weight<2, P>(sw, sd.dwx ? 1 : -1, i) / w : 1.0;
#pragma unroll
    for (int e = 0; e < CoefShape<C>::VEC; ++e) {
      const double u = v.v[e] - xp * z.v[e];
      nrm[e] = fma(W ? w * u : u, u, nrm[e]);
    }
  }
};
// another FE's side of M b: s += c_y y - c_z zb
template <int C, int W>
struct CoefRowYF {
  static constexpr int kGathers = 2, kI = 2, kD = W;
  const float* y;
  const double* zb;
  const CoefSide& sd;
  struct Val {
    CoefRow<C> y, z;
  };
  __device__ __forceinline__ void level(int) {}
  __device__ __forceinline__ const int32_t* idx_array(int i) const {
    return i == 0 ? sd.zi : sd.perm;
  }
  __device__ __forceinline__ const double* dbl_array(int i) const {
    return W == 1 ? sd.dw : i ? sd.dwx : (sd.slot_w >= 0 ? sd.d[sd.slot_w] : nullptr);
  }
  template <int P>
  __device__ __forceinline__ void load(const int32_t* si, uint32_t i, uint32_t qa, Val& v) const {
    v.y.load(y + (sd.perm ? (int64_t)si[P + i] : (int64_t)(qa + i)) * C);
    v.z.load(zb + (int64_t)si[i] * C);
  }
  template <int P>
  __device__ __forceinline__ void add(const double* sw, uint32_t i, uint32_t, const Val& v,
                                      CoefRow<C>& acc) const {
    if (W == 2) {  // c_z, then c_y = w x_k
      const double cz = coef_weight<2, P>(sw, sd.slot_w >= 0 ? 0 : -1, i);
      const double cy = coef_weight<2, P>(sw, sd.dwx ? 1 : -1, i);
#pragma unroll
      for (int e = 0; e < CoefShape<C>::VEC; ++e)
        acc.v[e] += cy * v.y.v[e] - cz * v.z.v[e];
    } else {
      const double w = coef_weight<W, P>(sw, 0, i);
#pragma unroll
      for (int e = 0; e < CoefShape<C>::VEC; ++e) {
        const double u = v.y.v[e] - v.z.v[e];
        acc.v[e] = W ? fma(w, u, acc.v[e]) : acc.v[e] + u;
      }
    }
  }
};

// ---------------------------------------------------------------------------
// scalar steps of one column (every CTA runs them on its own copy)
// ---------------------------------------------------------------------------
// The scalar step of lsmr.jl:113-186 (lambda = 0) with one reciprocal per
// rotation, and the tests of the iteration: an inner solve ends when the outer
// test is expected to pass, when the bidiagonalisation is exhausted, or at the
// limit of iterations.  (The reference's atol and btol are 0 here; of its tests
// on ||r|| the one against ||b|| is kept, for fits that are exact.)
template <int C>
__device__ __forceinline__ bool coef_rotate(CoefSmem<C>& sm, int j) {
  Inst& s = sm.inst[j];
  const double rho2 = s.alphabar * s.alphabar + s.beta * s.beta;
  const double ir = rsqrt(rho2), rho = rho2 * ir;
  const double c = s.alphabar * ir, sn = s.beta * ir;
  const double thetanew = sn * s.alpha;
  const double thetabar = s.sbar * rho, rhotemp = s.cbar * rho;
  const double rhobar2 = rhotemp * rhotemp + thetanew * thetanew;
  const double irb = rsqrt(rhobar2), rhobar = rhobar2 * irb;
  const double zetaold = s.zeta;
  s.alphabar = c * s.alpha;
  s.cbar = rhotemp * irb;
  s.sbar = thetanew * irb;
  s.zeta = s.cbar * s.zetabar;
  s.zetabar = -s.sbar * s.zetabar;
  // the (deferred) vector update, lsmr.jl:138-142
  sm.sc[3][j] = -thetabar * rho * sm.irr[j];
  sm.sc[4][j] = s.zeta * ir * irb;
  sm.sc[5][j] = -thetanew * ir;
  sm.irr[j] = ir * irb;
  // the estimate of ||r||
  const double betahat = c * s.betadd;
  s.betadd = -sn * s.betadd;
  const double it = rsqrt(s.rhodold * s.rhodold + thetabar * thetabar);
  const double ct = s.rhodold * it, st = thetabar * it;
  s.tautildeold = (zetaold - s.thetatilde * s.tautildeold) * it;
  s.thetatilde = st * rhobar;
  s.rhodold = ct * rhobar;
  s.betad = -st * s.betad + ct * betahat;
  const double taud = (s.zeta - s.thetatilde * s.tautildeold) / s.rhodold;
  const double dr = s.betad - taud;
  const double normr2 = dr * dr + s.betadd * s.betadd;
  // ||A|| and cond(A)
  s.normA2 += s.beta * s.beta;
  const double normA2 = s.normA2;
  s.normA2 += s.alpha * s.alpha;
  s.maxrbar = fmax(s.maxrbar, s.rhobar);
  if (s.iter > 1) s.minrbar = fmin(s.minrbar, s.rhobar);
  s.rho = rho;
  s.rhobar = rhobar;
  s.normA = normA2;  // squares; coef_outer adds them up
  s.normAr = fabs(s.zetabar);
  const double mx = fmax(s.maxrbar, rhotemp), mn = fmin(s.minrbar, rhotemp);
  const double nar2 = s.normAr * s.normAr;
  const double th = s.inner_theta_tol * s.inner_theta_tol;
  return s.iter >= s.maxiter || !(mn > s.ctol * mx) ||
         !(nar2 > th * (s.normA2_prev + normA2) * normr2) ||
         !(s.normAr > s.inner_rho * s.normAr0) || !(normr2 > 1e-32 * s.normb * s.normb) ||
         !(normr2 > th * s.normb0 * s.normb0);
}

// beta_{k+1} from T = v_k'N v_k (see fe_coef.h)
template <int C>
__device__ void coef_beta(CoefSmem<C>& sm, int j) {
  Inst& s = sm.inst[j];
  sm.vact[j] = 0;
  if (!s.active) return;
  const double T = sm.tot[0][j] * s.s_v * s.s_v;
  const double b2 = T - s.alpha * s.alpha;
  // below the rounding of T the residual space is exhausted: beta = 0
  const double ib = b2 > 4e-15 * T ? rsqrt(b2) : 0.0, beta = b2 * ib;
  if (ib > 0.0) {
    sm.sc[0][j] = s.s_v * ib;
    sm.sc[1][j] = T * s.s_v * ib;
    sm.sc[2][j] = s.iter > 0 ? s.alpha * s.beta * sm.svp[j] * ib : 0.0;
    sm.vact[j] = 1;
  }
  s.beta = ib > 0.0 ? beta : 0.0;
}

template <int C>
__device__ void coef_alpha(CoefSmem<C>& sm, int j) {
  Inst& s = sm.inst[j];
  sm.mode[j] = 0;
  if (!s.active) return;
  s.iter += 1;
  if (sm.vact[j]) {
    sm.svp[j] = s.s_v;
    const double a2 = sm.tot[0][j];
    s.s_v = a2 > 0 ? rsqrt(a2) : 1.0;
    s.alpha = a2 > 0 ? a2 * s.s_v : 0.0;
    sm.dt2[j] = sm.tot[1][j];
  }
  const bool last = coef_rotate<C>(sm, j);
  sm.mode[j] = 2;
  sm.sc[6][j] = s.s_v;
  if (last) s.active = 0;  // x_k is completed before the outer test
}

// The outer test on FP64 norms (nr2 = ||r||^2, ng = ||B'r||, nx = ||x||), and
// the start of the next inner solve on the correction problem.  True: the
// column is beyond what this side can tell, and the tile goes to the row side,
// which forms r and confirms x, or solves it from the start (at once where
// outer_rounds is left 0):
//   ||r||^2 = ||M b||^2 - x'(c + g) cancels when the fit is nearly exact;
//   g = c - N x is rounding when the tolerance lies near it (another round
//   gained less than a digit);
//   c itself is rounding, or x has grown along a direction that the data do
//   not determine (an FE nested in another), until r would lose its digits.
template <int C>
__device__ bool coef_outer(CoefSmem<C>& sm, int j, double nr2, double ng, double nx,
                           double rho_more, int64_t cap) {
  Inst& s = sm.inst[j];
  sm.mode[j] = 0;
  sm.vact[j] = 0;
  s.active = 0;
  if (!s.outer_active) return false;
  const double nr = sqrt(nr2);
  if (s.outer_rounds == 0) {
    s.normb0 = nr;
    s.normA2_prev = 0.0;
    s.iter_total = 0;
    sm.nb2[j] = nr2;
  } else {
    s.iter_total += s.iter;
    if (s.iter > 0) s.normA2_prev += s.normA;  // (a square, see coef_rotate)
    s.inner_rho = rho_more;
  }
  const double nAt = sqrt(s.normA2_prev);
  if (!isfinite(ng) || !isfinite(sm.nall[j])) {
    if (s.outer_rounds > 0) {
      s.outer_rounds = 0;
      return true;
    }
    // a NaN or infinite right-hand side stops at once, not converged
    s.last_test2 = nr * ng;
    s.converged = 0;
    s.outer_active = 0;
    return false;
  }
  s.normx = nx;
  if (s.outer_rounds > 0) {
    if (!(nx <= 1e6 * s.normb0)) {
      s.outer_rounds = 0;
      return true;
    }
    if (!(nr2 > 1e-9 * sm.nb2[j])) return true;
  } else if (ng > s.tol_a * nr && !(ng > 1e-13 * sqrt(sm.nall[j]))) {
    return true;
  }
  bool conv = false;
  s.last_test2 = (nAt > 0 && nr > 0) ? ng / (nAt * nr) : (ng == 0.0 ? 0.0 : 1.0);
  if (ng == 0.0 || nr == 0.0) {
    conv = true;
  } else if (s.outer_rounds == 0) {
    // the columns of B have norm 1 (or all but vanish), so ||B|| >= 1
    conv = ng <= s.tol_a * nr;
    if (conv) s.last_test2 = ng / nr;
  } else if (nAt > 0) {
    const double rtol = s.tol_b + s.tol_a * nAt * nx / s.normb0;
    conv = s.last_test2 <= s.tol_a || nr / s.normb0 <= rtol;
  }
  if (conv || s.iter_total >= s.maxiter_total) {
    s.converged = conv ? 1 : 0;
    s.outer_active = 0;
    return false;
  }
  if (s.outer_rounds >= s.max_rounds || (s.outer_rounds > 0 && s.last_test2 < 1e-15) ||
      (s.outer_rounds > 1 && s.last_test2 > 0.1 * s.rd_v))
    return true;
  s.rd_v = s.last_test2;  // (of the row side's kernels, free here)
  s.outer_rounds += 1;
  s.mode_inner = 1;
  s.maxiter = s.maxiter_total - s.iter_total < cap ? s.maxiter_total - s.iter_total : cap;
  s.beta = nr;
  s.u_scale = 1.0 / nr;
  s.alpha = ng / nr;
  s.s_v = 1.0 / ng;
  lsmr_init(s, 1);
  s.normAr0 = s.normAr;
  if (s.active) sm.mode[j] = 1;  // h <- v, hbar <- 0; x goes on from its value
  sm.sc[6][j] = s.s_v;
  sm.svp[j] = 0.0;
  sm.irr[j] = 1.0;
  return false;
}

// ---------------------------------------------------------------------------
// the passes of a solve; each ends with its norms in the CTA's slots.  They
// are not inlined, so that each has the registers of its own gathers only.
// ---------------------------------------------------------------------------
template <int C, int NQ>
__device__ __forceinline__ void coef_clear(double (&n)[NQ][CoefShape<C>::VEC]) {
#pragma unroll
  for (int k = 0; k < NQ; ++k)
#pragma unroll
    for (int v = 0; v < CoefShape<C>::VEC; ++v) n[k][v] = 0.0;
}

// an epilogue of coef_sweep: NL constants per level, loaded ahead, and the body
template <int NL, class Body>
struct CoefEpi {
  static constexpr bool kAhead = NL == 1;
  const double* lev;
  Body body;
  struct Pre {
    double v[NL];
  };
  __device__ __forceinline__ Pre pre(int l) const {
    Pre p;
    if (l >= 0) {
      if constexpr (NL == 1) {
        p.v[0] = __ldg(lev + l);
      } else {
        const double2 t = __ldg(reinterpret_cast<const double2*>(lev + (int64_t)l * 4));
        p.v[0] = t.x;
        p.v[1] = t.y;
        p.v[2] = __ldg(lev + (int64_t)l * 4 + 2);
      }
    }
    return p;
  }
  template <class Acc, class Nrm>
  __device__ __forceinline__ void operator()(int l, const Pre& p, Acc& s, int jl, Nrm& nr) const {
    body(l, p, s, jl, nr);
  }
};
template <int NL, class Body>
__device__ __forceinline__ CoefEpi<NL, Body> coef_epi(const double* lev, const Body& b) {
  return CoefEpi<NL, Body>{lev, b};
}

// zb = (A_p'A_p)^-1 A_p'b; norms: ||M b||^2, ||b||^2
template <int C, int NG, int W>
__device__ __noinline__ void coef_pass_yp(const CoefArgs& a, CoefSmem<C>& sm, int par) {
  constexpr int VEC = CoefShape<C>::VEC;
  const int jl = (threadIdx.x & 31) % CoefShape<C>::CL;
  const CoefSide& sd = a.p;
  double nrm[2][VEC];
  coef_clear<C>(nrm);
  coef_sweep<C, NG, W>(a, sd, CoefRowYP<C, W>{a.y + coef_col0<C>(jl), sd, nrm[1]}, nrm,
                   coef_epi<1>(sd.lev, [&](int l, const auto& k, CoefRow<C>& s, int jl, auto& nr) {
#pragma unroll
                     for (int v = 0; v < VEC; ++v) {
                       const double z = s.v[v] * k.v[0];
                       nr[0][v] -= s.v[v] * z;
                       s.v[v] = z;
                     }
                     s.store(a.zb + (int64_t)l * C + coef_col0<C>(jl));
                   }));
#pragma unroll
  for (int v = 0; v < VEC; ++v) nrm[0][v] += nrm[1][v];
  coef_publish<C, 2>(nrm, sm, a.part, par);
}

// ||M b||^2 as a sum over the projected rows
template <int C, int NG, int W>
__device__ __noinline__ void coef_pass_b(const CoefArgs& a, CoefSmem<C>& sm, int par) {
  const int jl = (threadIdx.x & 31) % CoefShape<C>::CL;
  const CoefSide& sd = a.p;
  double nrm[1][CoefShape<C>::VEC];
  coef_clear<C>(nrm);
  coef_sweep<C, NG, W>(
      a, sd, CoefRowB<C, W>{a.y + coef_col0<C>(jl), a.zb + coef_col0<C>(jl), sd, nrm[0], {}}, nrm,
      coef_epi<1>(sd.lev, [](int, const auto&, CoefRow<C>&, int, auto&) {}));
  coef_publish<C, 1>(nrm, sm, a.part, par);
}

// c = A_r'M b, the first v (into t), x = 0; norms: ||v||^2, and of two-FE
// plans sum D t^2 = ||A_r t||^2
template <int C, int NG, int W>
__device__ __noinline__ void coef_pass_yf(const CoefArgs& a, CoefSmem<C>& sm, double* t, int par) {
  constexpr int VEC = CoefShape<C>::VEC;
  const int jl = (threadIdx.x & 31) % CoefShape<C>::CL;
  double nrm[2][VEC];
  coef_clear<C>(nrm);
#pragma unroll 1
  for (int f = 0; f < NG; ++f) {
    const CoefSide& sd = a.f[f];
    coef_sweep<C, NG, W>(
        a, sd, CoefRowYF<C, W>{a.y + coef_col0<C>(jl), a.zb + coef_col0<C>(jl), sd}, nrm,
        coef_epi<3>(sd.lev, [&](int l, const auto& k, CoefRow<C>& s, int jl, auto& nr) {
          const int64_t o = (sd.base + l) * C + coef_col0<C>(jl);
          s.store(a.c + o);
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            const double n = k.v[1] * s.v[v];
            nr[0][v] += n * s.v[v];
            nr[1][v] += k.v[0] * n * n;
            s.v[v] = n;
          }
          s.store(t + o);
          s.zero();
          s.store(a.x + o);
        }));
  }
  coef_publish<C, 2>(nrm, sm, a.part, par);
}

// z = (A_p'A_p)^-1 A_p'A_r t; norm: ||M A_r t||^2 (of two-FE plans without the
// part ||A_r t||^2, which is known)
template <int C, int NG, int W>
__device__ __noinline__ void coef_pass_p(const CoefArgs& a, CoefSmem<C>& sm, const double* t,
                                         int par) {
  constexpr int VEC = CoefShape<C>::VEC;
  const int jl = (threadIdx.x & 31) % CoefShape<C>::CL;
  double nrm[1][VEC];
  coef_clear<C>(nrm);
  const CoefSide& sd = a.p;
  coef_sweep<C, NG, W>(a, sd, CoefRowP<C, NG, W>(sd, t, jl, nrm[0]), nrm,
                   coef_epi<1>(sd.lev, [&](int l, const auto& k, CoefRow<C>& s, int jl, auto& nr) {
#pragma unroll
                     for (int v = 0; v < VEC; ++v) {
                       const double z = s.v[v] * k.v[0];
                       nr[0][v] -= s.v[v] * z;
                       s.v[v] = z;
                     }
                     s.store(a.z + (int64_t)l * C + coef_col0<C>(jl));
                   }));
  coef_publish<C, 1>(nrm, sm, a.part, par);
}

// v_{k+1} (into tp) and the deferred update of h, hbar, x; norms:
// ||alpha v_{k+1}||^2, and of two-FE plans ||A_r D v_{k+1}||^2 = sum D t^2
template <int C, int NG, int W>
__device__ __noinline__ void coef_pass_f(const CoefArgs& a, CoefSmem<C>& sm, const double* t,
                                         double* tp, int par) {
  constexpr int VEC = CoefShape<C>::VEC;
  const int jl = (threadIdx.x & 31) % CoefShape<C>::CL;
  constexpr int NQ = NG == 1 ? 2 : 1;
  double nrm[NQ][VEC];
  coef_clear<C>(nrm);
#pragma unroll 1
  for (int f = 0; f < NG; ++f) {
    const CoefSide& sd = a.f[f];
    coef_sweep<C, NG, W>(
        a, sd, CoefRowF<C, NG - 1, W>(sd, t, a.z, jl), nrm,
        coef_epi<3>(sd.lev, [&](int l, const auto& k, CoefRow<C>& s, int jl, auto& nr) {
          const int64_t o = (sd.base + l) * C + coef_col0<C>(jl);
          CoefRow<C> tc, tn, h, hb, x;
          tc.load(t + o);
          tn.load(tp + o);
          h.load(a.h + o);
          hb.load(a.hb + o);
          x.load(a.x + o);
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            const int j = coef_col<C>(jl, v);
            const double vo = sm.sc[6][j] * tc.v[v];
            const int m = sm.mode[j];
            if (m == 2) {
              const double hbn = h.v[v] + sm.sc[3][j] * hb.v[v];
              hb.v[v] = hbn;
              x.v[v] += sm.sc[4][j] * hbn;
              h.v[v] = vo + sm.sc[5][j] * h.v[v];
            } else if (m == 1) {
              h.v[v] = vo;
              hb.v[v] = 0.0;
            }
            if (sm.vact[j]) {
              const double S = k.v[0] * tc.v[v] + s.v[v];
              double n = sm.sc[0][j] * k.v[1] * S - sm.sc[1][j] * tc.v[v];
              if (sm.sc[2][j] != 0.0) n -= sm.sc[2][j] * tn.v[v];
              tn.v[v] = n;
              nr[0][v] += n * n * k.v[2];
              if constexpr (NQ == 2) nr[1][v] += n * n * k.v[0];
            }
          }
          tn.store(tp + o);
          h.store(a.h + o);
          hb.store(a.hb + o);
          x.store(a.x + o);
        }));
  }
  coef_publish<C, NQ>(nrm, sm, a.part, par);
}

// the last x update of the columns whose inner solve has just ended
template <int C, int NG>
__device__ __noinline__ void coef_pass_x(const CoefArgs& a, const CoefSmem<C>& sm) {
  using Sh = CoefShape<C>;
  const int lane = threadIdx.x & 31, jl = lane % Sh::CL;
  const int64_t rows = a.f[NG - 1].base + a.f[NG - 1].n;
  const int64_t r0 =
      ((int64_t)blockIdx.x * kCoefWarps + (threadIdx.x >> 5)) * Sh::R + lane / Sh::CL;
  for (int64_t r = r0; r < rows; r += (int64_t)gridDim.x * kCoefWarps * Sh::R) {
    const int64_t o = r * C + coef_col0<C>(jl);
    CoefRow<C> h, hb, x;
    h.load(a.h + o);
    hb.load(a.hb + o);
    x.load(a.x + o);
#pragma unroll
    for (int v = 0; v < Sh::VEC; ++v) {
      const int j = coef_col<C>(jl, v);
      if (sm.mode[j] == 2) x.v[v] += sm.sc[4][j] * (h.v[v] + sm.sc[3][j] * hb.v[v]);
    }
    x.store(a.x + o);
  }
}

// g = c - N x (t <- D^2 g, the next v); norms: ||D g||^2, ||x||^2, x'(c + g)
template <int C, int NG, int W>
__device__ __noinline__ void coef_pass_g(const CoefArgs& a, CoefSmem<C>& sm, double* t, int par) {
  constexpr int VEC = CoefShape<C>::VEC;
  const int jl = (threadIdx.x & 31) % CoefShape<C>::CL;
  double nrm[3][VEC];
  coef_clear<C>(nrm);
#pragma unroll 1
  for (int f = 0; f < NG; ++f) {
    const CoefSide& sd = a.f[f];
    coef_sweep<C, NG, W>(
        a, sd, CoefRowF<C, NG - 1, W>(sd, a.x, a.z, jl), nrm,
        coef_epi<3>(sd.lev, [&](int l, const auto& k, CoefRow<C>& s, int jl, auto& nr) {
          const int64_t o = (sd.base + l) * C + coef_col0<C>(jl);
          CoefRow<C> x, c;
          x.load(a.x + o);
          c.load(a.c + o);
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            const double g = c.v[v] - (k.v[0] * x.v[v] + s.v[v]);
            nr[0][v] += k.v[1] * g * g;
            nr[1][v] += x.v[v] * x.v[v] * k.v[2];
            nr[2][v] += x.v[v] * (c.v[v] + g);
            s.v[v] = k.v[1] * g;
          }
          s.store(t + o);
        }));
  }
  coef_publish<C, 3>(nrm, sm, a.part, par);
}

// ---------------------------------------------------------------------------
// the solve of one tile
// ---------------------------------------------------------------------------
template <int C, int NG, int W>
__global__ void __launch_bounds__(kCoefThreads, kCoefCtas<C, NG, W>()) k_coef(const CoefArgs args) {
  __shared__ CoefArgs a;
  CoefSmem<C>& sm = *reinterpret_cast<CoefSmem<C>*>(coef_dyn);
  const int tid = threadIdx.x;
  if (tid == 0) a = args;
  uint32_t gen = 0;
  int par = 0;
  if (tid < C) {
    Inst& s = sm.inst[tid];
    memset(&s, 0, sizeof(s));
    s.ctol = 1e-8;
    s.tol_a = s.tol_b = args.tol;
    s.maxiter_total = s.maxiter = args.maxiter;
    s.inner_theta_tol = args.theta * args.tol;
    s.inner_rho = args.rho;
    s.outer_active = tid < args.ncols ? 1 : 0;
    s.converged = tid < args.ncols ? 0 : 1;
    s.max_rounds = args.max_rounds;
    sm.vact[tid] = sm.mode[tid] = 0;
  }
  __syncthreads();
  double* t = a.ta;
  double* tp = a.tb;
  double nr2 = 0.0;  // thread j < C: ||M b_j||^2
  bool handed = false;  // the row side goes on with the tile
  coef_pass_yp<C, NG, W>(a, sm, par);
  bool alive = coef_barrier(a, gen, &sm.ok);
  if (alive) {
    coef_totals<C, 2>(sm, a, par, a.multi_p, a.nmulti);
    par ^= 1;
    // ||M b||^2 = ||b||^2 - ... loses digits where the primary FE explains most
    // of b (a large mean): the projected rows are summed instead.  What is left
    // of a column that is constant within the levels is rounding.
    bool small = false;
    if (tid < C) {
      nr2 = sm.tot[0][tid];
      const double nall = sm.nall[tid] = sm.tot[1][tid];
      small = isfinite(nall) && nall > 0.0 && !(nr2 > 1e-4 * nall);
    }
    if (__syncthreads_or(small)) {
      coef_pass_b<C, NG, W>(a, sm, par);
      alive = coef_barrier(a, gen, &sm.ok);
      if (alive) coef_totals<C, 1>(sm, a, par, a.multi_p, a.nmulti);
      par ^= 1;
      if (alive && small) nr2 = sm.tot[0][tid];
      handed = __syncthreads_or(alive && small && !(nr2 > 1e-24 * sm.nall[tid]));
    }
  }
  if (alive && !handed) {
    coef_pass_yf<C, NG, W>(a, sm, t, par);
    alive = coef_barrier(a, gen, &sm.ok);
    if (alive) coef_totals<C, 2>(sm, a, par, 0, a.multi_p);
  }
  // LSMR ends after as many iterations as there are unknowns, but for rounding;
  // one that goes on far beyond is tested and started again
  const int64_t cap = 4 * (a.f[NG - 1].base + a.f[NG - 1].n) + 50;
  bool have_z = false;
  while (alive && !handed) {
    // outer test
    par ^= 1;
    bool hand = false;
    if (tid < C) {
      if (!have_z) {
        hand = coef_outer<C>(sm, tid, nr2, sqrt(sm.tot[0][tid]), 0.0, a.rho_more, cap);
        sm.dt2[tid] = sm.tot[1][tid];
      } else {
        hand = coef_outer<C>(sm, tid, sm.nb2[tid] - sm.tot[2][tid], sqrt(sm.tot[0][tid]),
                             sqrt(sm.tot[1][tid]), a.rho_more, cap);
      }
    }
    handed = __syncthreads_or(hand);
    if (handed) break;
    const bool outer = __syncthreads_or(tid < C && sm.inst[tid].outer_active);
    if (!outer && have_z) break;
    bool any = __syncthreads_or(tid < C && sm.inst[tid].active);
    if (NG == 1 && any && have_z) {
      // a second inner solve starts from pass_g's t, whose sum D t^2 is not known
      double nrm[2][CoefShape<C>::VEC];
      coef_clear<C>(nrm);
      const int lane = tid & 31, jl = lane % CoefShape<C>::CL;
      const int64_t r0 = ((int64_t)blockIdx.x * kCoefWarps + (tid >> 5)) * CoefShape<C>::R +
                         lane / CoefShape<C>::CL;
      for (int64_t r = r0; r < a.f[0].n; r += (int64_t)gridDim.x * kCoefWarps * CoefShape<C>::R) {
        CoefRow<C> v;
        v.load(t + r * C + coef_col0<C>(jl));
        const double d = __ldg(a.f[0].lev + r * 4);
#pragma unroll
        for (int i = 0; i < CoefShape<C>::VEC; ++i) nrm[1][i] += d * v.v[i] * v.v[i];
      }
      coef_publish<C, 2>(nrm, sm, a.part, par);
      alive = coef_barrier(a, gen, &sm.ok);
      if (!alive) break;
      coef_totals<C, 2>(sm, a, par, 0, 0);
      par ^= 1;
      if (tid < C) sm.dt2[tid] = sm.tot[1][tid];
      __syncthreads();
    }
    // inner LSMR
    while (any) {
      coef_pass_p<C, NG, W>(a, sm, t, par);
      alive = coef_barrier(a, gen, &sm.ok);
      if (!alive) break;
      coef_totals<C, 1>(sm, a, par, a.multi_p, a.nmulti);
      par ^= 1;
      if (tid < C) {
        if (NG == 1) sm.tot[0][tid] += sm.dt2[tid];
        coef_beta<C>(sm, tid);
      }
      __syncthreads();
      coef_pass_f<C, NG, W>(a, sm, t, tp, par);
      alive = coef_barrier(a, gen, &sm.ok);
      if (!alive) break;
      coef_totals<C, NG == 1 ? 2 : 1>(sm, a, par, 0, a.multi_p);
      par ^= 1;
      if (tid < C) coef_alpha<C>(sm, tid);
      double* sw = t;
      t = tp;
      tp = sw;
      any = __syncthreads_or(tid < C && sm.inst[tid].active);
    }
    if (!alive) break;
    if (__syncthreads_or(tid < C && sm.mode[tid] == 2)) {
      coef_pass_x<C, NG>(a, sm);
      alive = coef_barrier(a, gen, &sm.ok);
      if (!alive) break;
    }
    coef_pass_p<C, NG, W>(a, sm, a.x, par);
    have_z = true;
    if (!outer) break;  // every column stopped at once: z of x = 0
    alive = coef_barrier(a, gen, &sm.ok);
    if (!alive) break;
    par ^= 1;
    coef_pass_g<C, NG, W>(a, sm, t, par);
    alive = coef_barrier(a, gen, &sm.ok);
    if (alive) coef_totals<C, 3>(sm, a, par, 0, a.multi_p);
  }
  if (blockIdx.x == 0) {
    if (tid < C) a.inst[tid] = sm.inst[tid];
    if (tid == 0 && handed) a.bar[2] = kCoefHandOver;
  }
}

template <int C>
const void* coef_kernel(int nf, int w) {
  switch (nf * 3 + w) {
    case 3: return (const void*)k_coef<C, 1, 0>;
    case 4: return (const void*)k_coef<C, 1, 1>;
    case 5: return (const void*)k_coef<C, 1, 2>;
    case 6: return (const void*)k_coef<C, 2, 0>;
    case 7: return (const void*)k_coef<C, 2, 1>;
    case 8: return (const void*)k_coef<C, 2, 2>;
    case 9: return (const void*)k_coef<C, 3, 0>;
    case 10: return (const void*)k_coef<C, 3, 1>;
    default: return (const void*)k_coef<C, 3, 2>;
  }
}
// shared memory: CoefSmem and two windows per warp, of the pass that stages most
template <int C>
size_t coef_smem_bytes(int nf, int w) {
  const int pos = coef_window(nf, w) + 4;
  const int ni = std::max(nf, 2), nd = w == 2 ? nf + 2 : w;
  return sizeof(CoefSmem<C>) + (size_t)kCoefWarps * 2 * (ni * pos * 4 + nd * pos * 8);
}

}  // namespace fe
