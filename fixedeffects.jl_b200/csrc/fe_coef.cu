// fe_coef.cu -- plan data, row kernels and driver of the coefficient-side
// solve (fe_coef.h; the solve kernel itself is fe_coef.cuh).
#include "fe_coef.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "fe_prof.h"

namespace fe {

static inline unsigned grid1(int64_t n, int b = 256) { return (unsigned)((n + b - 1) / b); }

// ---------------------------------------------------------------------------
// plan data
// ---------------------------------------------------------------------------
static __global__ void k_take_i(const int32_t* __restrict__ src, const int32_t* __restrict__ perm,
                                int32_t* __restrict__ dst, int64_t n) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) dst[q] = src[perm ? perm[q] : q];
}
// out[q] = product of sw^2 and of up to four interactions, at position q
struct CoefProduct {
  const double* sw;
  const double* x[kCoefMaxFE + 1];
};
static __global__ void k_product(const CoefProduct a, const int32_t* __restrict__ perm,
                                 double* __restrict__ dst, int64_t n) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int64_t i = perm ? perm[q] : q;
  double v = 1.0;
  if (a.sw) v = a.sw[i] * a.sw[i];
#pragma unroll
  for (int g = 0; g <= kCoefMaxFE; ++g)
    if (a.x[g]) v *= a.x[g][i];
  dst[q] = v;
}
static __global__ void k_lev_primary(const double* __restrict__ scale, double* __restrict__ lev,
                                     int64_t n) {
  const int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (l < n) lev[l] = scale[l] * scale[l];
}
static __global__ void k_lev_other(const double* __restrict__ scale,
                                   const double* __restrict__ abs_scale, double* __restrict__ lev,
                                   int64_t n) {
  const int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= n) return;
  const double j = scale[l], s = abs_scale[l];
  lev[4 * l] = j > 0 ? 1.0 / (j * j) : 0.0;
  lev[4 * l + 1] = s * s;
  lev[4 * l + 2] = s > 0 ? 1.0 / (s * s) : 0.0;
  lev[4 * l + 3] = 0.0;
}

// the other FEs and their table rows
static CoefPlan& coef_layout(fe_plan* pl) {
  if (!pl->coef) pl->coef = std::make_shared<CoefPlan>();
  CoefPlan& cp = *pl->coef;
  if (cp.laid_out) return cp;
  for (int k = 0; k < pl->K; ++k)
    if (k != pl->primary) {
      cp.fe[cp.nf] = k;
      cp.base[cp.nf] = cp.rows;
      cp.rows += pl->nlev[k];
      ++cp.nf;
    }
  cp.laid_out = true;
  return cp;
}

static int coef_plan(fe_plan* pl) {
  CoefPlan& cp = coef_layout(pl);
  cudaStream_t s = pl->stream;
  const int kp = pl->primary;
  const int64_t N = pl->N;
  int st = 0;
  if (!cp.built) {
    for (int f = 0; f < cp.nf; ++f) {
      const int32_t* perm = pl->dev.perm[cp.fe[f]];
      if ((st = cp.zi[f].ensure((size_t)N * 4))) return st;
      k_take_i<<<grid1(N), 256, 0, s>>>(pl->dev.refs[kp], perm, cp.zi[f].as<int32_t>(), N);
      for (int g = 0; g < cp.nf; ++g) {
        if (g == f) continue;
        if ((st = cp.gi[f][g].ensure((size_t)N * 4))) return st;
        k_take_i<<<grid1(N), 256, 0, s>>>(pl->dev.refs[cp.fe[g]], perm, cp.gi[f][g].as<int32_t>(), N);
      }
      FE_CK(cudaGetLastError());
    }
    cp.built = true;
  }
  if (!cp.weights_built) {
    for (auto& w : cp.wt) w.second.filled = false;
    for (int f = 0; f <= cp.nf; ++f) {
      const int k = f < cp.nf ? cp.fe[f] : kp;
      const int64_t n = pl->nlev[k];
      if ((st = cp.lev[f].ensure((size_t)std::max<int64_t>(n, 1) * (f < cp.nf ? 32 : 8)))) return st;
      if (n > 0) {
        if (f < cp.nf)
          k_lev_other<<<grid1(n), 256, 0, s>>>(pl->d_scale_d[k].as<double>(),
                                               pl->d_abs_scale_d[k].as<double>(),
                                               cp.lev[f].as<double>(), n);
        else
          k_lev_primary<<<grid1(n), 256, 0, s>>>(pl->d_scale_d[k].as<double>(),
                                                 cp.lev[f].as<double>(), n);
      }
      FE_CK(cudaGetLastError());
    }
    cp.weights_built = true;
  }
  return 0;
}

// The product of w (bit 0) and of the interactions of the FE slots whose bit
// 1 + slot is set, in the order of FE slot f; null: all 1.
static int coef_weights(fe_plan* pl, int f, int mask, const double** out) {
  CoefPlan& cp = *pl->coef;
  CoefProduct p;
  memset(&p, 0, sizeof(p));
  int m = 0, eff = 0;
  if ((mask & 1) && pl->weighted) {
    p.sw = pl->d_sw_sorted.as<double>();
    eff |= 1;
  }
  for (int g = 0; g <= cp.nf; ++g) {
    const int k = g < cp.nf ? cp.fe[g] : pl->primary;
    if (!((mask >> (1 + g)) & 1) || !pl->interacted[k]) continue;
    p.x[m++] = pl->d_inter_sorted[k].as<double>();
    eff |= 2 << g;
  }
  *out = nullptr;
  if (!eff) return 0;
  CoefPlan::Weights& w = cp.wt[{f, eff}];
  const int st = w.buf.ensure((size_t)pl->N * 8);
  if (st) return st;
  if (!w.filled) {
    const int k = f < cp.nf ? cp.fe[f] : pl->primary;
    k_product<<<grid1(pl->N), 256, 0, pl->stream>>>(p, pl->dev.perm[k], w.buf.as<double>(), pl->N);
    FE_CK(cudaGetLastError());
    w.filled = true;
  }
  *out = w.buf.as<double>();
  return 0;
}

// Work items: consecutive levels packed into windows, longer levels cut into
// pieces.  A warp has 32 / (CL << rlog) teams that take a level each.  Levels longer than a
// quarter of a warp's share of the positions are cut, so that few long levels
// still fill the GPU evenly, but to no less than 1024 positions where the share
// is more (a piece costs a handshake of about 1.5 us) and no less than 4 steps
// of a warp.
static int coef_items(fe_plan* pl, int C, int window, CoefPlan::Items** out) {
  CoefPlan& cp = *pl->coef;
  std::unique_ptr<CoefPlan::Items>& slot = cp.items[{C, window}];
  if (slot) {
    *out = slot.get();
    return 0;
  }
  std::unique_ptr<CoefPlan::Items> its(new CoefPlan::Items());
  int sms = 148;
  FE_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, pl->device));
  const int cl = C >= 4 ? C / 4 : 1;
  const int64_t share = pl->N / std::max<int64_t>(1, (int64_t)sms * kCoefWarps);
  const int64_t psz = std::max<int64_t>(
      4 * (32 / cl), std::min<int64_t>(16384, std::min(share, std::max<int64_t>(1024, share / 4))));
  std::vector<CoefItem> whole, items;
  std::vector<CoefPiece> pcs;
  for (int f = 0; f <= cp.nf; ++f) {
    const int k = f < cp.nf ? cp.fe[f] : pl->primary;
    const std::vector<int64_t>& off = pl->seg_off[k];
    const int64_t nl = pl->nlev[k];
    const double avg = nl > 0 ? std::max(1.0, (double)pl->seg_len[k] / (double)nl) : 1.0;
    // the cheapest team size by the instructions of a pass, counted in its
    // source: a window, a round of its teams, a step of a round (a level is about
    // two standard deviations longer than the mean where it decides the round's
    // length).  On ten shapes (levels of 3 to 300 rows, 1 to 8 columns) its choice
    // was within 1.5 % of the best of all sizes, the worst 1.2 to 2.8 times slower.
    const int fit = std::max(1, std::min(32, (int)(window / avg)));
    int rlog = 0, cap = fit;
    double best = 1e300;
    for (int r = 0; (cl << r) <= 32; ++r) {
      const int nt = 32 / (cl << r);
      const double steps = std::ceil((avg + 2.0 * std::sqrt(avg)) / (1 << r));
      for (const int n : {fit, fit / nt * nt}) {
        if (n < 1) continue;
        const double cost = (150.0 + (n + nt - 1) / nt * (60.0 + 12.0 * r + 12.0 * steps)) / (n * avg);
        if (cost < best) {
          best = cost;
          rlog = r;
          cap = n;
        }
      }
    }
    its->rlog[f] = rlog;
    if (f == cp.nf) its->multi_p = its->nmulti;
    its->piece0[f] = its->pieces;
    whole.clear();
    items.clear();
    pcs.clear();
    int64_t l0 = 0;  // first level of the open item
    auto close = [&](int64_t l) {
      if (l > l0)
        whole.push_back({(uint32_t)off[(size_t)l0], (uint32_t)off[(size_t)l], (int32_t)l0,
                         (int32_t)(l - l0)});
      l0 = l;
    };
    for (int64_t l = 0; l < nl; ++l) {
      const int64_t b = off[(size_t)l], e = off[(size_t)l + 1], n = e - b;
      if (n > window) {
        close(l);
        l0 = l + 1;
        const int64_t np = (n + psz - 1) / psz, sz = (n + np - 1) / np;
        const int32_t first = (int32_t)pcs.size();
        for (int64_t i = 0; i < np; ++i) {
          items.push_back({(uint32_t)(b + i * sz), (uint32_t)std::min(b + (i + 1) * sz, e),
                           (int32_t)l, -1 - (int32_t)pcs.size()});
          pcs.push_back({first, (int32_t)np, its->nmulti, 0});
        }
        if (np > 1) ++its->nmulti;
        continue;
      }
      if (l - l0 == cap || e - off[(size_t)l0] > window) close(l);
    }
    close(nl);
    items.insert(items.end(), whole.begin(), whole.end());
    its->n[f] = (int64_t)items.size();
    its->pieces += (int32_t)pcs.size();
    int st = its->dev[f].ensure(std::max<size_t>(items.size(), 1) * sizeof(CoefItem));
    if (!st) st = its->piece[f].ensure(std::max<size_t>(pcs.size(), 1) * sizeof(CoefPiece));
    if (st) return st;
    if (!items.empty())
      FE_CK(cudaMemcpyAsync(its->dev[f].p, items.data(), items.size() * sizeof(CoefItem),
                            cudaMemcpyHostToDevice, pl->stream));
    if (!pcs.empty())
      FE_CK(cudaMemcpyAsync(its->piece[f].p, pcs.data(), pcs.size() * sizeof(CoefPiece),
                            cudaMemcpyHostToDevice, pl->stream));
    FE_CK(cudaStreamSynchronize(pl->stream));  // the host lists are reused
  }
  const int st = its->cnt.ensure((size_t)std::max(its->nmulti, 1) * 4);
  if (st) return st;
  slot = std::move(its);
  *out = slot.get();
  return 0;
}

// ---------------------------------------------------------------------------
// rows: host layout <-> sorted [N][C] rows
// ---------------------------------------------------------------------------
// As k_load / k_unload of fe_solve_impl.cuh, without weights and in FP32, the
// caller's type: half the bytes of an FP64 row copy.
constexpr int kRowElems = 2048;  // elements per CTA
template <int C>
__global__ void __launch_bounds__(256) k_rows_in(const float* __restrict__ Y, int64_t ld, int64_t col0,
                                                 int ncols, const int32_t* __restrict__ dst,
                                                 float* __restrict__ B, int64_t N) {
  constexpr int R = kRowElems / C, PER = kRowElems / 256;
  __shared__ float tile[R][C + 1];
  const int64_t i0 = (int64_t)blockIdx.x * R;
  float v[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int e = threadIdx.x + u * 256;
    const int j = e / R, r = e % R;
    v[u] = (i0 + r < N && j < ncols) ? Y[i0 + r + (col0 + j) * ld] : 0.f;
  }
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int e = threadIdx.x + u * 256;
    tile[e % R][e / R] = v[u];
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int e = threadIdx.x + u * 256;
    const int r = e / C, j = e % C;
    if (i0 + r < N) B[(int64_t)__ldg(dst + i0 + r) * C + j] = tile[r][j];
  }
}
// tiles of 1 or 2 columns: gathered through the inverse permutation, so that
// the rows, shorter than a sector, are written in order
template <int C>
__global__ void __launch_bounds__(256) k_rows_gather(const float* __restrict__ Y, int64_t ld,
                                                     int64_t col0, int ncols,
                                                     const int32_t* __restrict__ src,
                                                     float* __restrict__ B, int64_t N) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= N) return;
  const int64_t i = src[q];
#pragma unroll
  for (int j = 0; j < C; ++j) B[q * C + j] = j < ncols ? Y[i + (col0 + j) * ld] : 0.f;
}
template <int C>
__global__ void __launch_bounds__(256) k_rows_out(const float* __restrict__ B, int64_t ld, int64_t col0,
                                                  int ncols, const int32_t* __restrict__ dst,
                                                  float* __restrict__ Y, int64_t N,
                                                  const uint32_t* __restrict__ bar) {
  constexpr int R = kRowElems / C, PER = kRowElems / 256;
  __shared__ float tile[R][C + 1];
  if (bar[1] | bar[2]) return;  // the caller takes the row-side path
  const int64_t i0 = (int64_t)blockIdx.x * R;
  float v[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int e = threadIdx.x + u * 256;
    const int r = e / C, j = e % C;
    v[u] = i0 + r < N ? B[(int64_t)__ldg(dst + i0 + r) * C + j] : 0.f;
  }
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int e = threadIdx.x + u * 256;
    tile[e / C][e % C] = v[u];
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int e = threadIdx.x + u * 256;
    const int j = e / R, r = e % R;
    if (i0 + r < N && j < ncols) Y[i0 + r + (col0 + j) * ld] = tile[r][j];
  }
}

// r = y - A_r x - A_p (zb - z), in place on the sorted rows.  An observation
// of weight 0 gets NaN, as dividing its weighted residual by sqrt(w) does
// (src/AbstractFixedEffectSolver.jl:62-66).
struct CoefResid {
  const int32_t* refp;
  const int32_t* gi[kCoefMaxFE];
  const double* tab[kCoefMaxFE];
  const double* xg[kCoefMaxFE];
  const double *xp, *w, *zb, *z;
  int nf;
};
template <int C>
__global__ void __launch_bounds__(256) k_rows_resid(const CoefResid a, float* __restrict__ B, int64_t N,
                                                    const uint32_t* __restrict__ bar) {
  constexpr int VEC = C >= 2 ? 2 : 1, CL = C / VEC;
  if (bar[1] | bar[2]) return;
  const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int64_t q = e / CL;
  if (q >= N) return;
  const int j0 = (int)(e % CL) * VEC;
  const int64_t lp = __ldg(a.refp + q);
  const double xp = a.xp ? __ldg(a.xp + q) : 1.0;
  double fit[VEC], y[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    fit[v] = xp * (__ldg(a.zb + lp * C + j0 + v) - __ldg(a.z + lp * C + j0 + v));
    y[v] = (double)B[q * C + j0 + v];
  }
#pragma unroll
  for (int g = 0; g < kCoefMaxFE; ++g) {
    if (g >= a.nf) break;
    const double xg = a.xg[g] ? __ldg(a.xg[g] + q) : 1.0;
    const double* t = a.tab[g] + (int64_t)__ldg(a.gi[g] + q) * C + j0;
#pragma unroll
    for (int v = 0; v < VEC; ++v) fit[v] += xg * __ldg(t + v);
  }
  const bool zero = a.w && __ldg(a.w + q) == 0.0;
#pragma unroll
  for (int v = 0; v < VEC; ++v)
    B[q * C + j0 + v] = zero ? (float)nan("") : (float)(y[v] - fit[v]);
}

template <int C>
static int rows_in(fe_plan* pl, const SolveReq& rq, int64_t col0, int ncols, float* B) {
  if (C <= 2)
    k_rows_gather<C><<<grid1(pl->N), 256, 0, pl->stream>>>(
        (const float*)rq.Y, rq.ld, col0, ncols, pl->d_obs_src.as<int32_t>(), B, pl->N);
  else
    k_rows_in<C><<<grid1(pl->N, kRowElems / C), 256, 0, pl->stream>>>(
        (const float*)rq.Y, rq.ld, col0, ncols, pl->d_obs_dst.as<int32_t>(), B, pl->N);
  FE_CK(cudaGetLastError());
  return 0;
}
template <int C>
static int rows_out(fe_plan* pl, const SolveReq& rq, int64_t col0, int ncols, float* B,
                    const CoefResid& r, const uint32_t* bar, double rbytes, double ubytes) {
  constexpr int CL = C >= 2 ? C / 2 : 1;
  {
    ProfScope ps(pl, "resid", rbytes);
    k_rows_resid<C><<<grid1(pl->N * CL), 256, 0, pl->stream>>>(r, B, pl->N, bar);
    FE_CK(cudaGetLastError());
  }
  ProfScope ps(pl, "unload", ubytes);
  k_rows_out<C><<<grid1(pl->N, kRowElems / C), 256, 0, pl->stream>>>(
      B, rq.ld, col0, ncols, pl->d_obs_dst.as<int32_t>(), (float*)rq.Y, pl->N, bar);
  FE_CK(cudaGetLastError());
  return 0;
}

// ---------------------------------------------------------------------------
// driver
// ---------------------------------------------------------------------------
// 0: no weights or interactions, 1: weights alone, 2: interactions
static int entry_kind(const fe_plan* pl) {
  int kind = pl->weighted ? 1 : 0;
  for (int k = 0; k < pl->K; ++k)
    if (pl->interacted[k]) kind = 2;
  return kind;
}

// Whether the passes' gathers pay.  Every further FE adds a gather per position
// to every other FE's pass, so their cost grows with the square of the FEs'
// number, while the row-side loop's grows with it; interactions add staged
// arrays in the same way; and where levels hold two or three rows, the tables
// (FP64, several per level) are as large as the rows they replace.  Small
// problems gain all the same, as the row-side loop is then bound by launches.
// The lines lie between measured ratios, solve of the row-side loop / of this
// one, over 30k to 10M rows (to 60M for the short levels of two FEs), 1 to 8
// columns, levels of 2 to 60 rows and FEs of few levels.  "Short" levels: fewer
// than 2.5 (two FEs) or 3 rows per level, and 12 per level of the other FEs;
// "long" ones: 20 rows, where the other FEs' tables do not fit L1.
//   two FEs: 1.1 to 3.1, and below 1 for short levels of many elements only:
//     1 column 10M 1.14, 40M 0.93, 8 columns 1M 1.13, 3M 0.94, 2 columns 40M
//     1.16; weighted: 1 column 3M 1.24, 10M 0.96, 2 columns 10M 1.03, 4 columns 3M
//     1.10, 10M 0.83; interacted: 1M x 4 1.03, 1M x 8 0.99, and 4 columns with
//     long levels 1M 1.4, 3M 0.87
//   three: 1M x 1 to x 8 1.15 to 1.6, 3M x 1 1.06 to 1.4; short levels 2M x 2
//     1.01, 4M x 2 0.89, 3M x 4 0.93, 1M x 8 1.15, 3M x 8 0.79; 10M x 1 0.88,
//     1.2 where the other FEs' tables fit L1; long levels 3M x 2 0.96, in L1 16M x 2 1.35;
//     interacted: 1M x 1 1.05 to 1.36, 3M x 1 0.79 to 1.07, 300k x 2 1.11 to
//     1.43, 1M x 2 0.76 to 0.97, 1M x 4 1.03 to 1.27, 3M x 4 0.80 to 1.03, 8
//     columns short 300k 1.27, 1M 0.95, else 3M 1.03 to 1.08, 10M 0.93 to 1.11
//   four: 1 column 300k 1.34 to 1.96, 1M short 0.93, else 1.0 to 1.2, 1.5M 0.98; 2
//     columns 1M 1.07 to 1.36, 8 columns 300k 1.13 to 1.92; interacted: 1 column
//     300k 1.23 to 1.36, 1M 0.6 to 0.8, 2 columns 300k 1.24 to 1.6, 4 columns 100k
//     1.21 to 1.58, 8 columns 100k 1.24 to 1.42
// "Hard" problems, of more levels than rows, or interacted with short levels in
// three FEs, belong here whatever an iteration costs: the row side's FP32 inner
// solves stall on them (median of 20 to 24 columns: 4M x 2 3000 iterations and
// more against 74 here, 2M x 2 1147 against 67, 3M x 4 850 against 56, 1M x 1 of
// four FEs 769 against 54).
static bool coef_pays(const fe_plan* pl, int C) {
  const int nf = pl->K - 1, kind = entry_kind(pl);
  const int64_t N = pl->N, elems = N * C, levels = pl->P - pl->K;
  int64_t largest = 0;  // of the other FEs
  for (int k = 0; k < pl->K; ++k)
    if (k != pl->primary) largest = std::max(largest, pl->nlev[k]);
  const int64_t others = levels - pl->nlev[pl->primary];
  const bool in_l1 = others <= 16'384;
  const bool is_short = 2 * N < (nf == 1 ? 5 : 6) * levels && N < 12 * others;
  const bool is_long = N > 20 * levels && !in_l1;
  if (nf == 1) {
    if (!is_short) return !(kind == 2 && C == 4 && is_long) || elems <= 6'000'000;
    if (kind == 0) return C == 2 || elems <= 12'000'000;
    if (kind == 1) return elems <= (C == 2 ? 24'000'000 : C == 4 ? 12'000'000 : 8'000'000);
    return elems <= 6'000'000;
  }
  const bool hard =
      levels >= N || (kind == 2 && N < 2 * levels && N < 100 * (others - largest));
  if (nf == 2) {
    if (C <= 2 && N > 4'000'000 && !in_l1) return false;
    if (hard) return true;
    if (kind < 2) {
      if (is_short && elems > (C == 8 ? 8'000'000 : 5'000'000)) return false;
      return !(C == 2 && is_long && N > 2'000'000);
    }
    if (C == 1) return N <= 1'500'000 || in_l1;
    if (C == 2) return N <= 400'000;
    if (C == 4) return N <= 1'500'000 || in_l1;
    return N <= 400'000 || (!is_short && (N <= 4'000'000 || in_l1));
  }
  if (elems > (kind == 2 ? 1'000'000 : 2'500'000)) return false;
  if (hard) return true;
  if (kind < 2) return C > 1 || N <= (is_short ? 800'000 : 1'200'000);
  return elems <= (C == 1 ? 400'000 : C == 8 ? 1'000'000 : 600'000);
}

// Both cooperative kernels follow a row to its level in every FE, so every row
// has to have one: an FE that the problem lacks (no levels, level ids 0) leaves
// its rows outside the level order, on the slab's null row, which only the
// launched loops hold.
static bool every_row_has_levels(const fe_plan* pl) {
  for (int k = 0; k < pl->K; ++k)
    if (pl->seg_len[k] != pl->N) return false;
  return true;
}

// An option that names a kernel of the launched loops selects those.
static bool options_allow(const fe_plan* pl) {
  return pl->opt_ex_variant < 0 && pl->opt_seg_variant < 0 && pl->opt_rowsum_variant < 0;
}

// Mixed-precision residual solves of FP32 columns on plans whose primary FE is
// absorbed, with at most kCoefMaxFE other FEs, unless an option names a kernel
// of the row-side loop.  (FP64 columns keep the row-side iteration: theirs are
// returned unrounded, so another iteration would show in them at the level of
// the tolerance.  Tiles of 16 and 32 columns keep the row-side loop's FP32
// rows: at 10M x 32, three FEs, an FP64 iteration here takes 2.5 ms against
// 1.3 ms there.)
bool coef_takes(const fe_plan* pl, const SolveReq& rq, int C) {
  return C <= kCoefMaxCols && rq.precision == 1 && rq.dtype == 1 && rq.residuals && pl->absorbable && pl->opt_absorb != 0 &&
         pl->opt_abs_scale != 0 && pl->nprob == 1 && !pl->xchg && pl->N > 0 &&
         pl->K - 1 <= kCoefMaxFE && pl->perm_identity[pl->primary] && pl->opt_exdm != 0 &&
         pl->opt_exdm_pipe < 0 && pl->opt_firm_atomic == 0 && pl->opt_fused_resid < 0 &&
         options_allow(pl) && every_row_has_levels(pl) &&
         coef_pays(pl, C);
}

static const void* kernel_of(int C, int nf, int w, bool plain, size_t* smem) {
  switch (C) {
    case 1:
      *smem = coef_smem_bytes<1>(nf, w);
      return plain ? plain_kernel<1>(nf, w) : coef_kernel<1>(nf, w);
    case 2:
      *smem = coef_smem_bytes<2>(nf, w);
      return plain ? plain_kernel<2>(nf, w) : coef_kernel<2>(nf, w);
    case 4:
      *smem = coef_smem_bytes<4>(nf, w);
      return plain ? plain_kernel<4>(nf, w) : coef_kernel<4>(nf, w);
    default:
      *smem = coef_smem_bytes<8>(nf, w);
      return plain ? plain_kernel<8>(nf, w) : coef_kernel<8>(nf, w);
  }
}

// Polls of a grid barrier before a wait gives up: tens of seconds, or
// FE_B200_SPIN_LIMIT (read on every launch, so that a test can let waits run
// out; the solve then takes the launched loops).
static uint32_t spin_limit() {
  const char* v = getenv("FE_B200_SPIN_LIMIT");
  const unsigned long n = v ? strtoul(v, nullptr, 10) : 0;
  return n > 0 && n < (1ul << 25) ? (uint32_t)n : 1u << 25;
}

// What both cooperative kernels of a tile need: work items, kernel, grid,
// buffers of partial sums and the zeroed barrier.  *grid = 0: it does not fit.
struct CoefLaunch {
  CoefPlan::Items* its = nullptr;
  const void* kern = nullptr;
  size_t smem = 0;
  int64_t grid = 0;
  int weights = 0;
};
static int coef_prepare(fe_plan* pl, int C, bool plain, CoefLaunch* l, CoefArgs* a) {
  CoefPlan& cp = *pl->coef;
  const int nf = cp.nf;
  l->weights = entry_kind(pl);
  int st = coef_items(pl, C, coef_window(nf, l->weights), &l->its);
  if (st) return st;
  CoefPlan::Items* its = l->its;
  l->kern = kernel_of(C, nf, l->weights, plain, &l->smem);
  int sms = 148;
  FE_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, pl->device));
  // opt-in shared memory, once per kernel and device
  static PerDeviceOnce attr_set[2][4][9];
  const int ci = C == 1 ? 0 : C == 2 ? 1 : C == 4 ? 2 : 3;
  PerDeviceOnce& once = attr_set[plain][ci][(nf - 1) * 3 + l->weights];
  if (once.needed(pl->device)) {
    FE_CK(cudaFuncSetAttribute(l->kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)l->smem));
    once.done(pl->device);
  }
  if (!its->occ[plain] || its->occ_w[plain] != l->weights) {
    int o = 0;
    FE_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, l->kern, kCoefThreads, l->smem));
    if (o < 1) return 0;
    its->occ[plain] = o;
    its->occ_w[plain] = l->weights;
  }
  // a CTA per 512 rows of up to 4 columns, one for the smallest problems, which
  // then need no grid barrier (2k x 1: 148 us in one CTA, 159 in four; 20k x 1:
  // 184 us at 512 rows a CTA, 210 at 2048)
  const int64_t rows = pl->N * ((C + 3) / 4);
  const int64_t grid =
      rows <= 2048 ? 1 : std::min<int64_t>((int64_t)its->occ[plain] * sms, (rows + 511) / 512);
  const size_t rc = (size_t)C * 8;
  if ((st = cp.part.ensure((size_t)2 * 3 * grid * rc))) return st;
  if ((st = cp.ppart.ensure((size_t)std::max(its->pieces, 1) * rc))) return st;
  if ((st = cp.mnrm.ensure((size_t)3 * std::max(its->nmulti, 1) * rc))) return st;
  if ((st = cp.bar.ensure(64 + (size_t)C * sizeof(Inst)))) return st;
  a->part = cp.part.as<double>();
  a->ppart = cp.ppart.as<double>();
  a->mnrm = cp.mnrm.as<double>();
  a->nmulti = its->nmulti;
  a->multi_p = its->multi_p;
  a->pcnt = its->cnt.as<int32_t>();
  a->bar = cp.bar.as<uint32_t>();
  a->spins = spin_limit();
  for (int f = 0; f <= nf; ++f) {
    CoefSide& sd = f < nf ? a->f[f] : a->p;
    const int k = f < nf ? cp.fe[f] : pl->primary;
    sd.off = pl->d_off[k].as<int32_t>();
    sd.perm = pl->dev.perm[k];
    sd.items = its->dev[f].as<CoefItem>();
    sd.pieces = its->piece[f].as<CoefPiece>();
    sd.nitems = (int32_t)its->n[f];
    sd.piece0 = its->piece0[f];
    sd.n = (int32_t)pl->nlev[k];
    sd.rlog = its->rlog[f];
    sd.npos = (uint32_t)pl->N;
  }
  FE_CK(cudaMemsetAsync(cp.bar.p, 0, 64, pl->stream));
  FE_CK(cudaMemsetAsync(its->cnt.p, 0, its->cnt.bytes, pl->stream));
  l->grid = grid;
  return 0;
}

// *fits = false: the stream's share of the GPU (a partition of its SMs) does not
// hold the grid at once, the caller takes the launched loops.  (Host-side
// injection, read on every launch: FE_B200_FAIL_COOPERATIVE=1 makes launches
// fail like that.)
static int launch_cooperative(fe_plan* pl, const CoefLaunch& l, void** params, bool* fits) {
  const char* v = getenv("FE_B200_FAIL_COOPERATIVE");
  const cudaError_t e =
      v && *v == '1' ? cudaErrorCooperativeLaunchTooLarge
                     : cudaLaunchCooperativeKernel(l.kern, dim3((unsigned)l.grid),
                                                   dim3(kCoefThreads), params, l.smem, pl->stream);
  *fits = e != cudaErrorCooperativeLaunchTooLarge;
  if (!*fits) {
    (void)cudaGetLastError();
    return 0;
  }
  FE_CK(e);
  return 0;
}

#define FE_COEF_C(C, CALL)          \
  switch (C) {                      \
    case 1: { constexpr int W = 1; CALL; break; }   \
    case 2: { constexpr int W = 2; CALL; break; }   \
    case 4: { constexpr int W = 4; CALL; break; }   \
    default: { constexpr int W = 8; CALL; break; }  \
  }

static int coef_solve(fe_plan* pl, const SolveReq& rq, int C, int64_t col0, int ncols,
                      std::vector<Inst>& out, std::vector<Inst>& start, int* done) {
  NvtxRange nv("fe: tile (coefficient side)");
  *done = 0;
  int st = coef_plan(pl);
  if (st) return st;
  CoefPlan& cp = *pl->coef;
  const int kp = pl->primary, nf = cp.nf;
  const int64_t N = pl->N;
  const size_t es = 4, rc = (size_t)C * 8;
  const size_t pn = (size_t)std::max<int64_t>(pl->nlev[kp], 1), rn = (size_t)std::max<int64_t>(cp.rows, 1);
  if ((st = cp.y.ensure((size_t)N * C * es))) return st;
  if ((st = cp.zb.ensure(pn * rc))) return st;
  if ((st = cp.z.ensure(pn * rc))) return st;
  for (DevBuf* b : {&cp.ta, &cp.tb, &cp.h, &cp.hb, &cp.xx, &cp.c})
    if ((st = b->ensure(rn * rc))) return st;
  CoefArgs a;
  memset(&a, 0, sizeof(a));
  for (int f = 0; f <= nf; ++f) {
    CoefSide& sd = f < nf ? a.f[f] : a.p;
    // the weight arrays of this order, each distinct one staged once
    int nd = 0;
    const auto slot = [&](int mask, int32_t* out) -> int {
      const double* p = nullptr;
      const int e = coef_weights(pl, f, mask, &p);
      if (e) return e;
      *out = -1;
      for (int i = 0; i < nd && p; ++i)
        if (sd.d[i] == p) *out = i;
      if (p && *out < 0) {
        *out = nd;
        sd.d[nd++] = p;
      }
      return 0;
    };
    const int own = 2 << f, prim = 2 << nf;
    int m = 0;
    for (int g = 0; g < nf; ++g) {
      if (g == f) continue;
      sd.gi[m] = f < nf ? cp.gi[f][g].as<int32_t>() : pl->dev.refs[cp.fe[g]];
      sd.gb[m] = cp.base[g];
      const int mask = f < nf ? 1 | own | (2 << g) : nf == 1 ? 1 | prim | (2 << g) : 2 << g;
      if ((st = slot(mask, &sd.slot_g[m]))) return st;
      ++m;
    }
    sd.slot_w = sd.slot_n = -1;
    if ((f < nf || nf > 1) && (st = slot(f < nf ? 1 | own | prim : 1 | prim, &sd.slot_w))) return st;
    if (f == nf && nf > 1 && (st = slot(1, &sd.slot_n))) return st;
    if ((st = coef_weights(pl, f, 1, &sd.dw))) return st;
    if ((st = coef_weights(pl, f, f < nf ? 1 | own : 1 | prim, &sd.dwx))) return st;
    if (f < nf) {
      sd.zi = cp.zi[f].as<int32_t>();
      sd.base = cp.base[f];
    }
    sd.lev = cp.lev[f].as<double>();
  }
  CoefLaunch cl;
  if ((st = coef_prepare(pl, C, false, &cl, &a))) return st;
  if (!cl.grid) return 0;
  a.y = cp.y.as<float>();
  a.ncols = ncols;
  a.zb = cp.zb.as<double>();
  a.z = cp.z.as<double>();
  a.ta = cp.ta.as<double>();
  a.tb = cp.tb.as<double>();
  a.h = cp.h.as<double>();
  a.hb = cp.hb.as<double>();
  a.x = cp.xx.as<double>();
  a.c = cp.c.as<double>();
  a.inst = reinterpret_cast<Inst*>(static_cast<char*>(cp.bar.p) + 64);
  a.tol = rq.tol;
  a.theta = pl->opt_inner_theta;
  a.rho = pl->opt_coef_rho;
  a.rho_more = (float)pl->opt_inner_rho;
  a.maxiter = rq.maxiter - 1;
  a.max_rounds = pl->opt_max_rounds;
  {
    ProfScope ps(pl, "load", (double)N * (ncols + C) * es);
    FE_COEF_C(C, (st = rows_in<W>(pl, rq, col0, ncols, cp.y.as<float>())));
    if (st) return st;
  }
  bool fits = false;
  {
    ProfScope ps(pl, "coef_solve", 0.0);
    void* params[] = {&a};
    if ((st = launch_cooperative(pl, cl, params, &fits))) return st;
  }
  if (!fits) return 0;
  CoefResid r;
  memset(&r, 0, sizeof(r));
  r.refp = pl->dev.refs[kp];
  r.xp = pl->interacted[kp] ? pl->d_inter_sorted[kp].as<double>() : nullptr;
  r.w = pl->weighted ? pl->d_sw_sorted.as<double>() : nullptr;
  r.zb = a.zb;
  r.z = a.z;
  r.nf = nf;
  for (int g = 0; g < nf; ++g) {
    r.gi[g] = a.p.gi[g];
    r.xg[g] = pl->interacted[cp.fe[g]] ? pl->d_inter_sorted[cp.fe[g]].as<double>() : nullptr;
    r.tab[g] = a.x + cp.base[g] * C;
  }
  const double meta = (double)N * (4.0 * pl->K + (pl->weighted ? 8 : 0));
  const double rbytes = meta + (double)N * C * 2 * es + (double)pn * rc * 2 + (double)rn * rc;
  const double ubytes = (double)N * (ncols + C) * es;
  FE_COEF_C(C, (st = rows_out<W>(pl, rq, col0, ncols, cp.y.as<float>(), r, a.bar, rbytes, ubytes)));
  if (st) return st;
  std::vector<char> res(64 + (size_t)C * sizeof(Inst));
  FE_CK(cudaMemcpyAsync(res.data(), cp.bar.p, res.size(), cudaMemcpyDeviceToHost, pl->stream));
  FE_CK(cudaStreamSynchronize(pl->stream));
  uint32_t bar[3];
  memcpy(bar, res.data(), sizeof(bar));
  if (bar[1]) return prof_flush(pl);
  out.resize((size_t)C);
  memcpy(out.data(), res.data() + 64, (size_t)C * sizeof(Inst));
  // bytes of the solve kernel: per iteration (the longest column's) the index
  // and weight arrays of every order, one gathered z row per position of the
  // other FEs, the z rows written, the coefficient vectors
  int64_t iters = 0, rounds = 0;
  for (const Inst& s : out) {
    iters = std::max(iters, s.iter_total);
    rounds = std::max<int64_t>(rounds, s.outer_rounds);
  }
  double per = 0.0;
  for (int f = 0; f <= nf; ++f) {
    const CoefSide& sd = f < nf ? a.f[f] : a.p;
    per += (double)N * 4.0 * nf + (f < nf ? (double)N * rc : (double)pn * rc);
    for (const double* d : sd.d) per += d ? (double)N * 8.0 : 0.0;
  }
  pl->prof.bytes_per_launch["coef_solve"] =
      (per + 9.0 * rn * rc) * (double)(iters + rounds) + (double)N * C * es * (1 + nf) + (double)N * rc * nf;
  if (bar[2] == 0) {
    *done = 1;
    return prof_flush(pl);
  }
  // worth confirming if every column has been solved here, with an x that keeps
  // r's digits, or stopped at its first test
  bool all = true;
  for (int j = 0; j < ncols; ++j) {
    const Inst& s = out[(size_t)j];
    all = all && (s.outer_rounds > 0 ? s.normx <= 1e3 * s.normb0 : !s.outer_active);
  }
  if (all && rounds > 0) start = out;
  return prof_flush(pl);
}

// Without room for its arrays a solve takes the launched loops, which need
// fewer; they are given back, whole.
static bool no_room(fe_plan* pl, int st) {
  if (st != 3) return false;  // FE_ERR_ALLOC
  pl->coef.reset();
  return true;
}

int coef_solve_tile(fe_plan* pl, const SolveReq& rq, int C, int64_t col0, int ncols,
                    std::vector<Inst>& out, std::vector<Inst>& start, int* done) {
  const int st = coef_solve(pl, rq, C, col0, ncols, out, start, done);
  return no_room(pl, st) ? 0 : st;
}

// X64 of one FE: the table's coefficients in the scaled unknowns of the
// absorbed operator, for the columns of the mask
static __global__ void k_start(const double* __restrict__ tab, const double* __restrict__ scale,
                               double* __restrict__ x, int64_t n, int C, uint32_t mask) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * C) return;
  const double s = scale[e / C];
  if ((mask >> (e % C)) & 1u) x[e] = s > 0 ? tab[e] / s : 0.0;
}

int coef_start(fe_plan* pl, int C, const std::vector<Inst>& start, double* X64,
               std::vector<Inst>& h) {
  const CoefPlan& cp = *pl->coef;
  uint32_t mask = 0;
  for (int j = 0; j < C; ++j) {
    const Inst& s = start[(size_t)j];
    if (s.outer_rounds < 1) continue;
    mask |= 1u << j;
    h[(size_t)j].confirm = 1;
    h[(size_t)j].outer_rounds = s.outer_rounds;
    h[(size_t)j].iter_total = s.iter_total;
    h[(size_t)j].normA2_prev = s.normA2_prev;
    h[(size_t)j].normb0 = s.normb0;
  }
  for (int f = 0; f < cp.nf; ++f) {
    const int k = cp.fe[f];
    const int64_t n = pl->nlev[k];
    if (n == 0) continue;
    k_start<<<grid1(n * C), 256, 0, pl->stream>>>(cp.xx.as<double>() + cp.base[f] * C,
                                                  pl->d_abs_scale_d[k].as<double>(),
                                                  X64 + pl->lev_base[k] * C, n, C, mask);
    FE_CK(cudaGetLastError());
  }
  return 0;
}

// ---------------------------------------------------------------------------
// the plain FP64 loop
// ---------------------------------------------------------------------------
// Whether the loop gains by running in one kernel, which saves launches but
// sweeps one FE after the other, each a chain of loads (and, for an FE of few
// levels, of pieces), where a launch sums all of them side by side.  Measured,
// launched loop / this one, 1k to 2.4M rows, levels of 2 to 20 rows; "few": FEs of
// few levels, 6 to 30 of them:
//   two FEs: 1.0 to 2.0; interacted: 4 columns 10k and 30k 0.92 to 1.13, 1 column
//     1M 1.24 to 1.39, 2.4M 0.93 to 1.18
//   three: 1 column 1.05 to 1.7, interacted to 1M 0.99 to 1.6, 2.4M 0.86 to 1.08; 2
//     columns 1.02 to 1.8, interacted 1.05 to 1.5, with two few 100k 1.03; 4 columns
//     100k and more 1.2 to 1.36, with two few 100k 0.93, 300k 1.08, weighted with one
//     few 30k 0.92, 100k 1.17; 8 columns 1.2 to 1.5, with two few 0.98, weighted 300k
//     0.88; interacted 4 and 8 columns 0.82 to 1.19
//   four: 1 and 2 columns 1.04 to 1.7, interacted to 300k 1.02 to 1.46, 1M 0.75 to
//     0.97; with few 100k 0.87 to 1.1, 300k 1.12 to 1.18, 1M x 1 1.0, 1M x 2 0.97; 4
//     and 8 columns 100k 1.19 to 1.27, 300k 1.32 to 1.52, weighted 0.93 to 1.44
//   up to 32k rows these hold for two FEs and for 1 and 2 columns; 4 and 8 columns
//     of three or four FEs stay here too, at 0.72 to 1.5 (up to 0.2 ms a call
//     slower, as fast or faster below 2k rows, where one CTA runs the loop)
// and 4M x 1 0.96, 1M x 8 0.97, 10M x 1 0.79: the bound on all of them.
static bool plain_pays(const fe_plan* pl, int C) {
  const int nf = pl->K - 1, kind = entry_kind(pl);
  const int64_t N = pl->N;
  if (N * C > 2'500'000) return false;
  if (N <= 32'768) return true;
  if (nf == 1) return kind < 2 || N <= 1'500'000;
  int few = 0;
  for (int k = 0; k < pl->K; ++k) few += k != pl->primary && 256 * pl->nlev[k] < N;
  if (nf == 2) {
    const bool many = few < 2 || N >= 200'000;
    if (C == 1) return kind < 2 || N <= 1'500'000;
    if (C == 2) return kind < 2 || many;
    if (C == 4) return many && (kind == 0 || (kind == 1 && N >= 48'000));
    return kind == 0 || (kind == 1 && few < 2);
  }
  if (few) return kind < 2 && C <= 2 && N >= 200'000 && N * C <= 1'200'000;
  if (C <= 2) return kind < 2 || N <= 400'000;
  return kind == 0 && N >= 80'000;
}

// One problem of two to four FEs that is bound by launches, unless an option
// names a launched kernel of the loop.
bool plain_takes(const fe_plan* pl, const SolveReq& rq, int C) {
  return C <= kCoefMaxCols && rq.precision == 0 && pl->nprob == 1 && !pl->xchg && pl->N > 0 &&
         pl->K >= 2 && pl->K - 1 <= kCoefMaxFE && pl->perm_identity[pl->primary] &&
         options_allow(pl) && every_row_has_levels(pl) && plain_pays(pl, C);
}

int plain_loop(fe_plan* pl, int C, Inst* inst, double* U, double* V, double* H, double* Hb,
               double* X, int* done) {
  NvtxRange nv("fe: LSMR loop");
  *done = 0;
  CoefPlan& cp = coef_layout(pl);
  const int kp = pl->primary, nf = cp.nf;
  PlainArgs a;
  memset(&a, 0, sizeof(a));
  CoefLaunch cl;
  int st = coef_prepare(pl, C, true, &cl, &a.s);
  if (!st && !cl.grid) return 0;
  if (!st) st = cp.vs.ensure((size_t)pl->P * C * 8);
  if (!st) st = cp.sp.ensure((size_t)std::max<int64_t>(pl->nlev[kp], 1) * C * 8);
  if (st) return no_room(pl, st) ? 0 : st;
  for (int f = 0; f <= nf; ++f) {
    CoefSide& sd = f < nf ? a.s.f[f] : a.s.p;
    const int k = f < nf ? cp.fe[f] : kp;
    sd.lev = pl->d_scale_d[k].as<double>();
    sd.base = pl->lev_base[k];
    if (f < nf) {
      sd.dw = pl->dev.cwp_d[k];
      continue;
    }
    sd.d[0] = pl->dev.cw_d[kp];
    for (int g = 0; g < nf; ++g) {
      sd.gi[g] = pl->dev.refs[cp.fe[g]];
      sd.gb[g] = pl->lev_base[cp.fe[g]];
      sd.d[1 + g] = pl->dev.cw_d[cp.fe[g]];
    }
  }
  a.s.inst = inst;
  a.u = U;
  a.v = V;
  a.vs = cp.vs.as<double>();
  a.h = H;
  a.hb = Hb;
  a.x = X;
  a.sp = cp.sp.as<double>();
  void* params[] = {&a};
  ProfScope ps(pl, "plain_loop", 0.0);  // its bytes are known after the solve
  bool fits = false;
  if ((st = launch_cooperative(pl, cl, params, &fits))) return st;
  *done = fits ? 1 : 0;
  return 0;
}

const uint32_t* plain_gave_up(const fe_plan* pl) { return pl->coef->bar.as<uint32_t>() + 1; }

}  // namespace fe
