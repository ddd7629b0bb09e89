"""The fixed-point contractions of the stage kernels where they can go wrong: every range of the
Chebyshev solves (equal counts of one, tiny and wide spectra, the FP64 form beyond the fixed-point
one's limits), states of extreme size, zeros and numbers that are not finite."""
import numpy as np
import pytest

import edg_westervelt_gb300 as W
from conftest import rel_max
from oracle.precompute import precompute as opre

pytestmark = pytest.mark.gpu


def _problem(q, N, mixed, **kw):
    co = W.constant_coefficients(c=1.0, alpha=1e-3, beta=0.5)
    from oracle import coefficients as oc
    kw = dict(mixed=mixed, flux="upwind", mode="initial_value", boundary="wall", kappa=0.5, **kw)
    po, _ = opre(q, N, coefficients=oc.constant_coefficients(c=1.0, alpha=1e-3, beta=0.5), **kw)
    return W.precompute(q, N, coefficients=co, **kw)[0], po


# (lowest, highest) 2βv of an element: constant, nearly constant, a wave's, a front's, close to the limit of
# the mass matrix (κ = 60 and 400) and far below zero
SPANS = [(0.0, 0.0), (0.3, 0.3 + 1e-12), (-1e-7, 1e-7), (-0.02, 0.03), (-0.58, 0.58), (-0.9, 0.97), (-1.0, 0.995),
         (-6.0, 0.2), (-40.0, -3.0)]


@pytest.mark.parametrize("q,mixed", [(1, True), (1, False), (2, False), (3, True), (4, False), (5, False), (6, True),
                                     (6, False), (7, True), (7, False)])
def test_mass_solves_over_the_spectra(gpu, q, mixed):
    """One element per span of 2βv against the dense reference (LU). The solve's residual is 1e-14 of R,
    so the error is at most κ 1e-14 in the Euclidean norm of an element (NV times the largest entry);
    twice that for the rounding of the steps."""
    from oracle.reference_rhs import dense_volume, edg_rhs_reference, reference_pre
    N = 3
    pp, po = _problem(q, N, mixed)
    nu, nv = pp["qu1"], pp["qv1"]
    rng = np.random.default_rng(q)
    Ph = po["P_h_v"]
    w = np.sqrt(np.diag(po["W2d_h"]))
    U = np.asfortranarray(rng.standard_normal((N, N, nu, nu)))
    dense = dense_volume(reference_pre(po))
    ws = W.Workspace(pp, N)
    assert ws.stats()["fast_path"] == 1
    for lo, hi in SPANS:
        V = np.zeros((N, N, nv, nv), order="F")
        for j in range(N):
            for k in range(N):
                X = rng.standard_normal((nv, nv)) * np.exp(-0.5 * np.add.outer(np.arange(nv), np.arange(nv)))
                X[0, 0] = 0.0
                g = Ph @ X @ Ph.T
                span = g.max() - g.min()
                X = X * ((hi - lo) / span) if span > 0 else X * 0.0
                g = Ph @ X @ Ph.T
                X[0, 0] = 2.0 * (hi - g.max())      # the constant mode is 1/2
                V[j, k] = X                          # 2β = 1
        a = edg_rhs_reference(U, V, 0.0, N, 1.0 / N, dense)
        b = ws.rhs(U, V, 0.0)
        g = np.einsum("ra,jkab,sb->jkrs", Ph, V, Ph)
        kappa = float(((1 - g).max(axis=(2, 3)) / (1 - g).min(axis=(2, 3))).max())
        tol = 2e-14 * kappa * nv + 1e-13
        assert rel_max(a, b) < tol, (lo, hi, kappa, rel_max(a, b), tol)
    assert w.size == Ph.shape[0]


@pytest.mark.parametrize("q,mixed", [(1, True), (1, False), (4, True), (6, False), (7, False)])
def test_cg_solves_over_the_spectra(gpu, q, mixed):
    """The conjugate gradient solves of the same spans. They end at |r| <= 1e-14 |R|, an error of at most
    κ 1e-14 in the Euclidean norm (NV times the largest entry); twice that, and κ NV² roundings of 1e-16
    of the recurrence's r against the true one."""
    from oracle.reference_rhs import dense_volume, edg_rhs_reference, reference_pre
    N = 2
    pp, po = _problem(q, N, mixed, mass_solver="cg")
    nu, nv = pp["qu1"], pp["qv1"]
    rng = np.random.default_rng(10 + q)
    Ph = po["P_h_v"]
    U = np.asfortranarray(rng.standard_normal((N, N, nu, nu)))
    dense = dense_volume(reference_pre(po))
    ws = W.Workspace(pp, N)
    for lo, hi in SPANS[:6]:
        V = np.zeros((N, N, nv, nv), order="F")
        for j in range(N):
            for k in range(N):
                X = rng.standard_normal((nv, nv)) * np.exp(-0.5 * np.add.outer(np.arange(nv), np.arange(nv)))
                X[0, 0] = 0.0
                span = np.ptp(Ph @ X @ Ph.T)
                X = X * ((hi - lo) / span) if span > 0 else X * 0.0
                X[0, 0] = 2.0 * (hi - (Ph @ X @ Ph.T).max())
                V[j, k] = X
        a = edg_rhs_reference(U, V, 0.0, N, 1.0 / N, dense)
        b = ws.rhs(U, V, 0.0)
        g = np.einsum("ra,jkab,sb->jkrs", Ph, V, Ph)
        kappa = float(((1 - g).max(axis=(2, 3)) / (1 - g).min(axis=(2, 3))).max())
        tol = kappa * (2e-14 * nv + 1e-16 * nv * nv) + 1e-13
        assert rel_max(a, b) < tol, (lo, hi, kappa, rel_max(a, b), tol)


@pytest.mark.parametrize("q,mixed", [(2, True), (4, False), (7, False)])
def test_rhs_scales_with_the_state(gpu, q, mixed):
    """With β = 0 and no data the right-hand side is linear: a state scaled by a power of two, as far as
    the exponents go, gives the same bits scaled."""
    N = 4
    co = W.constant_coefficients(c=1.25, alpha=2e-3, beta=0.0)
    pp, _ = W.precompute(q, N, coefficients=co, mixed=mixed, flux="central", mode="source", boundary="wall", kappa=0.5)
    rng = np.random.default_rng(3)
    u = np.asfortranarray(rng.standard_normal((N, N, pp["qu1"], pp["qu1"])))
    v = np.asfortranarray(rng.standard_normal((N, N, pp["qv1"], pp["qv1"])))
    ws = W.Workspace(pp, N)
    t = 2.0                                          # past the source
    a = [x.copy() for x in ws.rhs(u, v, t)]
    for k in (-700, -300, -1, 1, 300, 900):
        f = 2.0 ** k
        b = ws.rhs(u * f, v * f, t)
        assert all(np.array_equal(x * f, y) for x, y in zip(a, b)), k
    z = ws.rhs(u * 0.0, v * 0.0, t)
    assert all(np.array_equal(x, np.zeros_like(x)) for x in z)


def test_numbers_that_are_not_finite(gpu):
    """An infinity or NaN in u leaves its element and the neighbours that share a face with it not
    finite, the others untouched; in v, there or in the second stage of a step, it is refused as a mass
    matrix that is not positive definite."""
    N, q = 5, 4
    pp, _ = _problem(q, N, False)
    rng = np.random.default_rng(4)
    u = np.asfortranarray(rng.standard_normal((N, N, q + 1, q + 1)))
    v = np.asfortranarray(0.02 * rng.standard_normal((N, N, q + 1, q + 1)))
    ws = W.Workspace(pp, N)
    a = [x.copy() for x in ws.rhs(u, v, 0.0)]
    for bad in (np.nan, np.inf, -np.inf):
        u1 = u.copy(order="F")
        u1[2, 2, 1, 2] = bad
        b = ws.rhs(u1, v, 0.0)
        for x, y in zip(a, b):
            assert not np.isfinite(y[2, 2]).all()
            far = np.ones((N, N), bool)
            for j, k in ((2, 2), (1, 2), (3, 2), (2, 1), (2, 3)):
                far[j, k] = False
            assert np.array_equal(x[far], y[far])
        u2, v2 = u1.copy(order="F"), v.copy(order="F")
        with pytest.raises(W.ErrorException, match="mass matrix not positive definite"):
            ws.rk4_steps(u2, v2, 0.0, 1e-6, 1)
    v1 = v.copy(order="F")
    v1[1, 3, 0, 1] = np.nan
    with pytest.raises(W.ErrorException, match="mass matrix not positive definite"):
        ws.rhs(u, v1, 0.0)
