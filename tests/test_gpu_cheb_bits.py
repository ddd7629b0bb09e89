"""The accuracy of the Chebyshev mass solves, beside the same recurrence in FP64 (numpy): with u = 0, α = 0, the
central flux and reflecting walls the right-hand side of the mass systems is the data array PiCdiv as it
stands, so that the solves alone are seen."""
import math

import numpy as np
import pytest

import edg_westervelt_gb300 as W
from oracle import coefficients as oc
from oracle.precompute import precompute as opre

pytestmark = pytest.mark.gpu

# (lowest, highest) 2βv: ε = δ/θ of 0.025, 0.58, 0.80, 0.959, 0.9678, 0.9692, 0.9656, 0.958, 0.9676, 0.9685, 0.995; θ
# of 0.126 and 0.124; a matrix far from and one close to zero everywhere; a spread of three orders
SPANS = [(-0.02, 0.03), (-0.58, 0.58), (-6.0, 0.2), (-0.9, 0.96), (-0.9, 0.969), (-0.9, 0.9703), (-3.0, 0.93),
         (-6.0, 0.85), (-6.9, 0.87), (-7.1, 0.87), (-1.0, 0.995), (0.868, 0.88), (0.87, 0.882), (-40.0, -3.0),
         (0.999, 0.9995), (-300.0, 0.9)]


def _operators(po):
    """P_h and W_h P_h as the workspace holds them: the second half of the points is the first half's mirror image."""
    P, w = po["P_h_v"].copy(), np.sqrt(np.diag(po["W2d_h"]))
    n = len(w)
    for i in range(n // 2):
        w[n - 1 - i] = w[i]
        P[n - 1 - i] = P[i] * (-1.0) ** np.arange(P.shape[1])
    if n % 2:
        P[n // 2, 1::2] = 0.0
    return P, w[:, None] * P


def _chebyshev(P, PW, G, R, th, de, n, T):
    """Saad's Algorithm 12.1 with n steps an element on M = I - Pᵀ W G P, in arithmetic T."""
    P, PW, G, th, de = (x.astype(T) for x in (P, PW, G, th, de))
    r, s1 = R.astype(T), th / de
    X, d, rho = np.zeros_like(r), r / th[:, None, None], 1 / s1
    for step in range(1, int(n.max()) + 1):
        X = np.where((step <= n)[:, None, None], X + d, X)
        y = (P @ d @ P.T) * G
        r = r - d + PW.T @ y @ PW
        rhon = 1 / (2 * s1 - rho)
        d = (rhon * rho)[:, None, None] * d + (2 * rhon / de)[:, None, None] * r
        rho = rhon
    return X


@pytest.mark.parametrize("equal", [False, True])
@pytest.mark.parametrize("q,mixed", [(1, False), (2, False), (4, False), (6, True), (7, False)])
def test_solves_carry_the_bits_of_fp64(gpu, q, mixed, equal):
    """The rounding errors of the solves (against the recurrence with more bits), over the elements, are no larger
    than those of FP64, to the half unit 1.1e-16 of a result. Right-hand sides: entries of unlike and of
    nearly the same size (the largest Euclidean norm)."""
    N = 4
    po, _ = opre(q, N, coefficients=oc.constant_coefficients(c=1.0, alpha=0.0, beta=0.5), mixed=mixed, flux="central",
                 mode="initial_value", boundary="wall", kappa=0.5)
    for side in ("bcB_spy", "bcT_spy", "bcL_spx", "bcR_spx"):
        po[side] = np.zeros_like(po[side])
    nu, nv = po["qu1"], po["qv1"]
    P, PW = _operators(po)
    rng = np.random.default_rng(100 * q + mixed)
    U = np.zeros((N, N, nu, nu), order="F")
    for lo, hi in SPANS:
        R = rng.standard_normal((N * N, nv, nv))
        if equal:
            R = 1.0 + 1e-3 * R
        po["PiCdiv"] = np.asfortranarray(R.reshape(N, N, nv, nv).transpose(2, 3, 0, 1))
        X = rng.standard_normal((N * N, nv, nv)) * np.exp(-0.5 * np.add.outer(np.arange(nv), np.arange(nv)))
        X[:, 0, 0] = 0.0
        g = P @ X @ P.T
        X *= ((hi - lo) / np.ptp(g, axis=(1, 2)))[:, None, None]
        X[:, 0, 0] = 2.0 * (hi - (P @ X @ P.T).max(axis=(1, 2)))          # the constant mode is 1/2; 2β = 1
        V = np.asfortranarray(X.reshape(N, N, nv, nv))
        vt = W.Workspace(po, N).rhs(U, V, 0.0)[1].reshape(N * N, nv, nv)

        LD = np.longdouble
        G = P.astype(LD) @ X.astype(LD) @ P.T.astype(LD)
        amin, amax = 1 - G.max(axis=(1, 2)), 1 - G.min(axis=(1, 2))
        th = (amax + amin) / 2
        de = np.maximum((amax - amin) / 2, 1e-15 * th)
        steps = math.acosh(1.0 / po["mass_tol"]) / np.arccosh((th / de).astype(np.float64))
        assert np.abs(steps - np.rint(steps)).min() > 1e-9 * steps.max()  # the count is not in doubt
        n = np.ceil(steps)
        exact = _chebyshev(P, PW, G, R, th, de, n, LD)
        fp64 = _chebyshev(P, PW, P @ X @ P.T, R, th, de, n, np.float64)
        size = np.abs(exact).max(axis=(1, 2))
        err = [float(np.sqrt(((np.abs(x - exact).max(axis=(1, 2)) / size) ** 2).mean())) for x in (vt, fp64)]
        assert err[0] <= err[1] + 1.1e-16, (lo, hi, int(n.max()), err)
