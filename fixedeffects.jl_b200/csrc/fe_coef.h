// fe_coef.h -- the coefficient-side solve of mixed-precision residual calls
// (fe_coef.cuh, fe_coef.cu).  Internal.
//
// The absorbed problem min || M (b - A_r x) || (M projects the primary FE
// out) has normal equations over the non-primary levels alone, and
//   A_r' M A_r t = A_r' (tau - A_p z),  tau = A_r t,  z = (A_p'A_p)^-1 A_p' tau,
// needs the observations' level ids and weights but no N x C vector: z is one
// sum per primary level over gathered rows of t, the product one sum per
// other level over gathered rows of z.  LSMR's bidiagonalisation
// (src/utils/lsmr.jl:104-109) follows from this product alone: with N = B'B,
//   beta_{k+1}^2 = v_k'N v_k - alpha_k^2,
//   alpha_{k+1} beta_{k+1} v_{k+1} = N v_k - (v_k'N v_k) v_k - alpha_k beta_k v_{k-1},
// so u is never formed.  All of it runs in FP64.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fe_plan.h"
#include "fe_solve.h"

namespace fe {

constexpr int kCoefThreads = 512;
constexpr int kCoefWarps = kCoefThreads / 32;
constexpr int kCoefMaxCols = 8;  // widest tile of this path
constexpr int kCoefMaxFE = 3;  // non-primary FEs of a plan that takes this path

// positions per staged window (and per item of whole levels): one 16-byte copy
// of indices per lane, or half where five weight arrays are staged (nf, w as
// coef_kernel).  Measured on 10M rows in levels of 10, three effects, one
// interacted: 124 positions 136 + 242 us a pair of passes, 92 positions 278 +
// 299 us (fewer levels a window, idle teams); windows as long as shared memory
// allows (up to 768 positions) took 100M x 8 from 38.6 to 45.4 ms a solve.
constexpr int coef_window(int nf, int w) { return w == 2 && nf == 3 ? 60 : 124; }

// Work item of a warp, one 16-byte load: levels [level, level + levels) at
// positions [q0, q1), at most 32 of them and coef_window positions; or, with
// levels = -1 - p, piece p of a longer level.
struct alignas(16) CoefItem {
  uint32_t q0, q1;
  int32_t level, levels;
};
// A piece of a level: the level's pieces are first..first + np - 1; cnt: the
// level's counter and norm slot, when np > 1.
struct alignas(16) CoefPiece {
  int32_t first, np, cnt, pad;
};

// One FE's level order.  zi/gi: per position, the primary level and the level
// of each gathered FE.  The entries of A_r and A_p are weights times
// interactions; their products per position are the distinct arrays d[0..],
// and a slot names the one of a term (-1: all 1):
//   primary FE: slot_g of the gathered FEs' interactions, slot_w of w x_p,
//     slot_n of w; with one gathered FE slot_g[0] holds w x_p x_g
//   other FEs: slot_w of w x_k x_p (the z term), slot_g of w x_k x_g
// dw, dwx: w and w x_p of the primary FE; dwx: w x_k of another (null: 1).
struct CoefSide {
  const int32_t* off;
  const int32_t* perm;  // position -> sorted row (null: identity)
  const int32_t* zi;
  const int32_t* gi[kCoefMaxFE];
  const double* d[kCoefMaxFE + 2];
  const double *dw, *dwx;
  // per level: primary FE {1 / ||a_l||^2}; others {||a_l||^2, s^2, 1 / s^2, 0}
  // with s the column scale of the absorbed operator
  const double* lev;
  const CoefItem* items;
  const CoefPiece* pieces;
  int64_t gb[kCoefMaxFE];  // first table row of each gathered FE
  int64_t base;            // first table row of this FE
  int32_t slot_w, slot_n, slot_g[kCoefMaxFE];
  int32_t n;               // levels
  int32_t nitems;
  int32_t piece0;          // index of its first piece in the partial buffers
  int32_t rlog;            // log2 of the rows a team reads at a time
  uint32_t npos;           // positions
};

struct CoefArgs {
  CoefSide p, f[kCoefMaxFE];
  const float* y;  // sorted rows [N][C] of the right-hand sides, unweighted
  int32_t ncols;
  uint32_t spins;            // polls of a grid barrier before a wait gives up
  double *zb, *z;            // [primary levels][C]: of b, of the current table
  double *ta, *tb;           // [levels][C]: D v_k and D v_{k-1}, unnormalised
  double *h, *hb, *x, *c;    // [levels][C]: h, hbar, x (times D); A_r'M b
  double* part;              // [2][3][grid][C] norm partials
  double* ppart;             // [pieces][C]
  double* mnrm;              // [3][nmulti][C] norms of the levels of several pieces
  int32_t nmulti, multi_p;   // such levels; the primary FE's start at multi_p
  int32_t* pcnt;
  uint32_t* bar;             // [0] arrivals, [1] a wait gave up, [2] status
  Inst* inst;
  double tol, theta, rho;    // rho: drop of ||A'r|| that ends the first inner solve
  int64_t maxiter;
  int32_t max_rounds;
  float rho_more;            // ... a later one
};

// The plain FP64 loop (fe_plain.cuh): the sides' items and scales (lev), index
// and entry arrays (primary: gi, and d[0] = its entries, d[1 + g] those of the
// gathered FEs; with weights alone d[0] = sqrt(w) for all; others: perm, dw);
// base, gb: slab rows.
struct PlainArgs {
  CoefArgs s;
  double* u;                 // [N][C] rows
  double *v, *vs, *h, *hb, *x;  // [P][C]; vs: scale times v
  double* sp;                // [primary levels][C]: A_p'u
};

// status word of a solve that came to its end (bar[1] == 0): bar[2]
constexpr uint32_t kCoefHandOver = 1;  // the row side confirms x, or starts again

// Per-plan data of the path: index and weight arrays in every FE's level
// order, built on the first solve that takes it, weights again after
// fe_plan_update_weights.
struct CoefPlan {
  bool laid_out = false, built = false, weights_built = false;
  int nf = 0;
  int fe[kCoefMaxFE] = {};       // non-primary FEs
  int64_t base[kCoefMaxFE] = {};  // first table row of each
  int64_t rows = 0;              // table rows
  DevBuf zi[kCoefMaxFE], gi[kCoefMaxFE][kCoefMaxFE];
  // weight arrays in every FE's order (last: primary), built on demand: the
  // product of w (bit 0) and of the interactions of the FE slots in the mask
  struct Weights {
    DevBuf buf;
    bool filled = false;
  };
  std::map<std::pair<int, int>, Weights> wt;
  DevBuf lev[kCoefMaxFE + 1];
  // work items and pieces of every side (last: primary), by (C, window)
  struct Items {
    int64_t n[kCoefMaxFE + 1] = {};
    int32_t rlog[kCoefMaxFE + 1] = {}, piece0[kCoefMaxFE + 1] = {};
    int32_t pieces = 0, nmulti = 0, multi_p = 0;
    DevBuf dev[kCoefMaxFE + 1], piece[kCoefMaxFE + 1], cnt;
    int occ[2] = {}, occ_w[2] = {-1, -1};  // resident CTAs per SM of the kernels with weights occ_w
  };
  std::map<std::pair<int, int>, std::unique_ptr<Items>> items;
  DevBuf vs, sp;  // plain loop
  DevBuf y, zb, z, ta, tb, h, hb, xx, c, part, ppart, mnrm, bar;
};

// whether the request takes the coefficient-side path
bool coef_takes(const fe_plan* pl, const SolveReq& rq, int C);
// one tile; *done = 0: the caller runs the row-side path (the columns are
// untouched), to confirm the state in `start` if there is one
int coef_solve_tile(fe_plan* pl, const SolveReq& rq, int C, int64_t col0, int ncols,
                    std::vector<Inst>& out, std::vector<Inst>& start, int* done);
// Makes `start` the row side's state of a tile: X64 ([P][C], zero) and the
// counts and norms of the instances h.  Columns without a finished round start
// from zero.
int coef_start(fe_plan* pl, int C, const std::vector<Inst>& start, double* X64,
               std::vector<Inst>& h);

// Whether a plain FP64 solve of C columns runs its loop in one kernel, and the
// loop: the instances at `inst` (device) hold the state after the first
// bidiagonalisation step, U the rows, V, H, Hb, X the [P][C] slabs.  *done = 0:
// it does not fit, the caller launches the loop.  plain_gave_up: device address
// of a word that is not 0 after the loop's kernel if one of its waits gave up;
// U, V, H, Hb and X are then unfinished.
bool plain_takes(const fe_plan* pl, const SolveReq& rq, int C);
int plain_loop(fe_plan* pl, int C, Inst* inst, double* U, double* V, double* H, double* Hb,
               double* X, int* done);
const uint32_t* plain_gave_up(const fe_plan* pl);

// the kernels of a tile width (fe_coef_c*.cu)
template <int C>
const void* coef_kernel(int nf, int w);  // w: 0 none, 1 weights, 2 interactions too
template <int C>
const void* plain_kernel(int nf, int w);
template <int C>
size_t coef_smem_bytes(int nf, int w);

}  // namespace fe
