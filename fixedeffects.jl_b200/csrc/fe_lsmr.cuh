// fe_lsmr.cuh -- the LSMR scalar recurrences of one instance, in FP64
// (src/utils/lsmr.jl:46-222, lambda = 0), shared by the scalar kernel of the
// row-side solves (fe_scalar.cu) and the one-kernel solves (fe_plain.cuh,
// fe_coef.cuh).  Every multiply and add rounds separately, as in the
// reference's scalar code, in whichever kernel they are compiled.
#pragma once

#include <cuda_runtime.h>

#include "fe_internal.h"

namespace fe {

// A double whose products and sums are rounded one by one (the compiler does
// not contract them to fused multiply-adds).
struct Rn {
  double v;
  __device__ __forceinline__ Rn(double x) : v(x) {}
};
__device__ __forceinline__ Rn operator*(Rn a, Rn b) { return __dmul_rn(a.v, b.v); }
__device__ __forceinline__ Rn operator+(Rn a, Rn b) { return __dadd_rn(a.v, b.v); }
__device__ __forceinline__ Rn operator-(Rn a, Rn b) { return __dadd_rn(a.v, -b.v); }
__device__ __forceinline__ Rn operator-(Rn a) { return -a.v; }
__device__ __forceinline__ Rn operator/(Rn a, Rn b) { return __ddiv_rn(a.v, b.v); }
__device__ __forceinline__ Rn root(Rn a) { return __dsqrt_rn(a.v); }

// Kernel coefficients of a stopped instance: the expand keeps U
// (U <- 0*(A v) + 1*U) and the P-side update is skipped (upd_mode 0, no v).
__device__ static void deactivate(Inst& s) {
  s.active = 0;
  s.ex_av = 0.0;
  s.ex_au = 1.0;
  s.upd_mode = 0;
  s.do_v = 0;
}

__device__ static void lsmr_test(Inst& s) {
  // src/utils/lsmr.jl:188-215
  const Rn normA = s.normA, normr = s.normr, normAr = s.normAr, normb = s.normb, normx = s.normx;
  const double test1 = (normr / normb).v;
  const double test2 = (normAr / (normA * normr)).v;
  const double test3 = (Rn(1.0) / s.condA).v;
  const double t1 = (Rn(test1) / (Rn(1.0) + normA * normx / normb)).v;
  const double rtol = (Rn(s.btol) + Rn(s.atol) * normA * normx / normb).v;
  int istop = 0;
  if (s.iter >= s.maxiter) istop = 7;
  else if (1.0 + test3 <= 1.0) istop = 6;
  else if (1.0 + test2 <= 1.0) istop = 5;
  else if (1.0 + t1 <= 1.0) istop = 4;
  else if (test3 <= s.ctol) istop = 3;
  else if (test2 <= s.atol) istop = 2;
  else if (test1 <= rtol) istop = 1;
  if (!istop && s.mode_inner) {
    // inner solve of the mixed mode: stop once the FP64 outer test is
    // expected to pass, or once normAr fell by inner_rho (the FP32 floor)
    const Rn nAt = root(Rn(s.normA2_prev) + normA * normA);
    if (s.normAr <= (Rn(s.inner_theta_tol) * nAt * normr).v ||
        s.normAr <= (Rn(s.inner_rho) * s.normAr0).v)
      istop = 2;
  }
  s.istop = istop;
}

__device__ static void lsmr_rotate(Inst& s) {
  // src/utils/lsmr.jl:113-186, lambda = 0
  const Rn alpha = s.alpha, beta = s.beta, alphabar = s.alphabar, lambda = 0.0;
  const Rn alphahat = root(alphabar * alphabar + lambda * lambda);
  const Rn chat = alphabar / alphahat;
  const Rn shat = lambda / alphahat;
  const Rn rhoold = s.rho;
  const Rn rho = root(alphahat * alphahat + beta * beta);
  const Rn c = alphahat / rho;
  const Rn sn = beta / rho;
  const Rn thetanew = sn * alpha;
  s.alphabar = (c * alpha).v;
  const Rn rhobarold = s.rhobar;
  const Rn zetaold = s.zeta;
  const Rn thetabar = Rn(s.sbar) * rho;
  const Rn rhotemp = Rn(s.cbar) * rho;
  const Rn rhobar = root(rhotemp * rhotemp + thetanew * thetanew);
  const Rn cbar = rhotemp / rhobar;
  const Rn sbar = thetanew / rhobar;
  const Rn zeta = cbar * s.zetabar;
  s.zetabar = (-sbar * s.zetabar).v;
  s.rho = rho.v;
  s.rhobar = rhobar.v;
  s.cbar = cbar.v;
  s.sbar = sbar.v;
  s.zeta = zeta.v;
  // coefficients of the (deferred) vector update, lsmr.jl:138-142
  s.c1 = (-thetabar * rho / (rhoold * rhobarold)).v;
  s.c2 = (zeta / (rho * rhobar)).v;
  s.c3 = (-thetanew / rho).v;
  // estimate of ||r||
  const Rn betaacute = chat * s.betadd;
  const Rn betacheck = -shat * s.betadd;
  const Rn betahat = c * betaacute;
  const Rn betadd = -sn * betaacute;
  const Rn thetatildeold = s.thetatilde;
  const Rn rhotildeold = root(Rn(s.rhodold) * s.rhodold + thetabar * thetabar);
  const Rn ctildeold = Rn(s.rhodold) / rhotildeold;
  const Rn stildeold = thetabar / rhotildeold;
  const Rn thetatilde = stildeold * rhobar;
  const Rn rhodold = ctildeold * rhobar;
  const Rn betad = -stildeold * s.betad + ctildeold * betahat;
  const Rn tautildeold = (zetaold - thetatildeold * s.tautildeold) / rhotildeold;
  const Rn taud = (zeta - thetatilde * tautildeold) / rhodold;
  const Rn d = Rn(s.d) + betacheck * betacheck;
  s.betadd = betadd.v;
  s.thetatilde = thetatilde.v;
  s.rhodold = rhodold.v;
  s.betad = betad.v;
  s.tautildeold = tautildeold.v;
  s.d = d.v;
  s.normr = root(d + (betad - taud) * (betad - taud) + betadd * betadd).v;
  // estimate of ||A|| and cond(A)
  const Rn normA2 = Rn(s.normA2) + beta * beta;
  s.normA = root(normA2).v;
  s.normA2 = (normA2 + alpha * alpha).v;
  s.maxrbar = s.maxrbar > rhobarold.v ? s.maxrbar : rhobarold.v;
  if (s.iter > 1) s.minrbar = s.minrbar < rhobarold.v ? s.minrbar : rhobarold.v;
  const double mx = s.maxrbar > rhotemp.v ? s.maxrbar : rhotemp.v;
  const double mn = s.minrbar < rhotemp.v ? s.minrbar : rhotemp.v;
  s.condA = (Rn(mx) / mn).v;
  s.normAr = fabs(s.zetabar);
}

// Initial values of src/utils/lsmr.jl:68-100 given alpha, beta.
__device__ static void lsmr_init(Inst& s, int init_mode) {
  s.zetabar = s.alpha * s.beta;
  s.alphabar = s.alpha;
  s.rho = 1.0;
  s.rhobar = 1.0;
  s.cbar = 1.0;
  s.sbar = 0.0;
  s.betadd = s.beta;
  s.betad = 0.0;
  s.rhodold = 1.0;
  s.tautildeold = 0.0;
  s.thetatilde = 0.0;
  s.zeta = 0.0;
  s.d = 0.0;
  s.normA = -1.0;
  s.condA = -1.0;
  s.normx = -1.0;
  s.normA2 = s.alpha * s.alpha;
  s.maxrbar = 0.0;
  s.minrbar = 1e100;
  s.normb = s.beta;
  s.istop = 0;
  s.normr = s.beta;
  s.normAr = s.alpha * s.beta;
  s.iter = 0;
  s.pending = 0;
  s.upd_mode = init_mode;  // h <- v, hbar <- 0 (and x <- 0) at the next reduce
  s.do_v = 1;
  s.active = (s.normAr != 0.0 && s.maxiter > 0 && !s.skip_lsmr) ? 1 : 0;
  // a NaN or infinite right-hand side: the reference runs maxiter iterations
  // on NaN norms (no test can pass) and reports istop = 7, not converged;
  // here the instance stops at once with the same verdict
  if (!isfinite(s.normAr)) {
    s.active = 0;
    s.istop = 7;
  }
  s.ex_av = s.s_v;
  s.ex_au = -s.alpha * s.u_scale;
  if (!s.active) deactivate(s);
}

}  // namespace fe
