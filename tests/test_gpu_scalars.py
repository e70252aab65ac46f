"""The LSMR scalar recurrences as the one-kernel solves compile them: bit for
bit those of separately rounded arithmetic (src/utils/lsmr.jl:113-186), and
the FP64 loop in one kernel against the oracle in every column."""
import ctypes
import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent


def _steps(alpha, beta):
    """lsmr.jl:68-100 and 113-186 in Python floats, lambda = 0."""
    alphabar, zetabar = alpha[0], alpha[0] * beta[0]
    rho = rhobar = cbar = rhodold = 1.0
    sbar = betad = tautildeold = thetatilde = zeta = d = 0.0
    betadd, normA2, maxrbar, minrbar = beta[0], alpha[0] * alpha[0], 0.0, 1e100
    out = []
    for k in range(1, len(alpha)):
        a, b = alpha[k], beta[k]
        alphahat = math.sqrt(alphabar * alphabar + 0.0)
        chat, shat = alphabar / alphahat, 0.0 / alphahat
        rhoold, rho = rho, math.sqrt(alphahat * alphahat + b * b)
        c, s = alphahat / rho, b / rho
        thetanew, alphabar = s * a, c * a
        rhobarold, zetaold = rhobar, zeta
        thetabar, rhotemp = sbar * rho, cbar * rho
        rhobar = math.sqrt((cbar * rho) * (cbar * rho) + thetanew * thetanew)
        cbar, sbar = cbar * rho / rhobar, thetanew / rhobar
        zeta, zetabar = cbar * zetabar, -sbar * zetabar
        c1 = -thetabar * rho / (rhoold * rhobarold)
        c2, c3 = zeta / (rho * rhobar), -thetanew / rho
        betaacute, betacheck = chat * betadd, -shat * betadd
        betahat, betadd = c * betaacute, -s * betaacute
        thetatildeold = thetatilde
        rhotildeold = math.sqrt(rhodold * rhodold + thetabar * thetabar)
        ct, st = rhodold / rhotildeold, thetabar / rhotildeold
        thetatilde, rhodold = st * rhobar, ct * rhobar
        betad = -st * betad + ct * betahat
        tautildeold = (zetaold - thetatildeold * tautildeold) / rhotildeold
        taud = (zeta - thetatilde * tautildeold) / rhodold
        d = d + betacheck * betacheck
        normr = math.sqrt(d + (betad - taud) * (betad - taud) + betadd * betadd)
        normA2 = normA2 + b * b
        normA = math.sqrt(normA2)
        normA2 = normA2 + a * a
        maxrbar = max(maxrbar, rhobarold)
        if k > 1:
            minrbar = min(minrbar, rhobarold)
        condA = max(maxrbar, rhotemp) / min(minrbar, rhotemp)
        out.append((normr, normA, condA, abs(zetabar), c1, c2, c3))
    return np.array(out)


def test_recurrences_round_every_operation(fe, tmp_path):
    from fe_b200 import build
    so = tmp_path / "lsmr_steps.so"
    src = ROOT / "tests" / "native" / "lsmr_steps.cu"
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "-shared", "-o", str(so), str(src)],
                   check=True, capture_output=True)
    lib = ctypes.CDLL(str(so))
    rng = np.random.default_rng(12)
    n, p = 40, ctypes.POINTER(ctypes.c_double)
    for _ in range(8):
        alpha, beta = rng.uniform(0.3, 1.2, n + 1), rng.uniform(0.3, 1.2, n + 1)
        out = np.zeros((n, 7))
        assert lib.lsmr_steps(alpha.ctypes.data_as(p), beta.ctypes.data_as(p), n,
                              out.ctypes.data_as(p)) == 0
        assert np.array_equal(out, _steps(list(map(float, alpha)), list(map(float, beta))))


@pytest.mark.parametrize("weighted,cols", [(False, 3), (True, 8)])
def test_plain_loop_matches_the_oracle_in_every_column(fe, oracle, weighted, cols):
    rng = np.random.default_rng(8)
    n, nlev = 20_011, [2000, 200, 30]
    refs = [rng.integers(1, m + 1, n) for m in nlev]
    w = rng.uniform(0.5, 1.5, n) if weighted else None
    Y = np.asfortranarray(rng.standard_normal((n, cols)) + (refs[0] % 7)[:, None] * 0.4)
    feM = fe.AbstractFixedEffectSolver([fe.FixedEffect.from_refs(r, m) for r, m in zip(refs, nlev)],
                                       w, "CUDA", np.float64)
    feM.set_option(fe._lib.FE_OPT_PROFILE, 1)
    R, its, cv = feM.solve_residuals(Y.copy(order="F"), tol=1e-8)
    assert "plain_loop" in feM.kernel_stats() and cv.all()
    feM.close()
    R_o, it_o, _ = oracle.solve_residuals_cols(Y, refs, nlev, [None] * 3, w, tol=1e-8)
    for j in range(cols):
        assert abs(int(its[j]) - int(it_o[j])) <= 1
        assert np.linalg.norm(R[:, j] - R_o[:, j]) < 1e-6 * np.linalg.norm(R_o[:, j])
