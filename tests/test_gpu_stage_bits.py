"""The accuracy of the u-equation's solve in the constant-coefficient kernels, beside the same right-hand side in FP64
(numpy), where the 1D operators and their eigenbasis are exact to a rounding or two (q_u up to 3)."""
import numpy as np
import pytest

import edg_westervelt_gb300 as W
from oracle import coefficients as oc
from oracle.precompute import precompute as opre

pytestmark = pytest.mark.gpu


def _mirrored(A, sg):
    """A with the second half of its points the first half's mirror image times sg, as the workspace holds it."""
    A, n = A.copy(), A.shape[0]
    for i in range(n // 2):
        A[n - 1 - i] = A[i] * sg
    if n % 2:
        A[n // 2, sg < 0] = 0.0
    return A


def _ut(po, U, V, N, al, kap, T):
    """ut of src/rhs.jl with c = 1, α = al constant and reflecting walls without data, in arithmetic T."""
    nu = po["qu1"]
    sg = (-1.0) ** np.arange(nu)
    S, w = _mirrored(po["S_u"], -sg).astype(T), _mirrored(po["w"][:, None], np.ones(1))[:, 0].astype(T)
    El, E1 = po["Ebl_u"][0].astype(T), po["E1bl_u"][0].astype(T)
    El, E1 = (El, sg * El), (E1, -sg * E1)                      # low and high end
    K1 = S.T @ (w[:, None] * S)
    K1[(np.add.outer(np.arange(nu), np.arange(nu)) % 2) == 1] = 0
    K1[0] = K1[:, 0] = 0
    U, Vp = U.astype(T), np.zeros(U.shape, T)
    Vp[:, :, :V.shape[2], :V.shape[3]] = V
    th, tau, lu, lv, al = (T(x) for x in (po["theta"], po["tau"], po["lambda_u"], po["lambda_v"], al))
    two = 2 * T(N)
    b = K1 @ Vp + Vp @ K1
    b[:, :, 0, 0] += Vp[:, :, 0, 0]
    for axis, sub in ((0, "a,jkab->jkb"), (1, "b,jkab->jka")):
        du, dv = ([np.einsum(sub, E1[end], X) for end in (0, 1)] for X in (U, Vp))
        v = [np.einsum(sub, El[end], Vp) for end in (0, 1)]
        du, dv, v = ([np.moveaxis(x, axis, 0) for x in y] for y in (du, dv, v))
        F = [np.zeros_like(du[0]) for _ in (0, 1)]
        dum, vm, dvm, dup, vp, dvp = du[1][:-1], v[1][:-1], dv[1][:-1], du[0][1:], v[0][1:], dv[0][1:]
        J = two * (dum - dup) + al * two * (dvm - dvp)
        F[0][1:] = th * (vm - vp) - tau * J
        F[1][:-1] = -((1 - th) * (vp - vm) - tau * J)
        for end, i, s in ((0, 0, -1), (1, -1, 1)):              # a wall: F = -sgn c² dv
            F[end][i] = s * T(kap) * (s * two * (du[end][i] + al * dv[end][i]))
        F = [np.moveaxis(x, 0, axis) for x in F]
        for end in (0, 1):
            b = b - np.einsum("a,jkb->jkab" if axis == 0 else "b,jka->jkab", E1[end], F[end])
    n2 = nu * nu
    eye = np.eye(nu, dtype=T)
    A = np.kron(K1, eye) + np.kron(eye, K1)
    A[0, 0] += 1
    Ai, B = np.linalg.inv(A.astype(np.float64)).astype(T), b.reshape(N * N, n2).T
    x = Ai @ B
    for _ in range(4):
        x = x + Ai @ (B - A @ x)
    return x.T.reshape(N, N, nu, nu)


@pytest.mark.parametrize("flux", ["central", "upwind", "alternating"])
@pytest.mark.parametrize("q,mixed", [(1, False), (1, True), (2, False), (2, True), (3, False), (3, True)])
def test_u_solve_carries_the_bits_of_fp64(gpu, q, mixed, flux):
    """On smooth states (entries falling by 10 from mode to mode) the errors of ut, the largest of each element over
    its largest entry, are on average no larger than FP64's, to the half unit 1.1e-16 of a result."""
    N, al, kap = 6, 1e-2, 0.5
    po, _ = opre(q, N, coefficients=oc.constant_coefficients(c=1.0, alpha=al, beta=0.0), mixed=mixed, flux=flux,
                 mode="initial_value", boundary="wall", kappa=kap)
    for k in ("bcB_spy", "bcT_spy", "bcL_spx", "bcR_spx"):
        po[k] = np.zeros_like(po[k])
    rng = np.random.default_rng(q)
    U, V = (np.asfortranarray(rng.standard_normal((N, N, n, n)) * 10.0 ** -np.add.outer(np.arange(n), np.arange(n)))
            for n in (po["qu1"], po["qv1"]))
    ut = W.Workspace(po, N).rhs(U, V, 0.0)[0]
    exact = _ut(po, U, V, N, al, kap, np.longdouble)
    size = np.abs(exact).max(axis=(2, 3))
    err = [float((np.abs(x - exact).max(axis=(2, 3)) / size).mean()) for x in (ut, _ut(po, U, V, N, al, kap, np.float64))]
    assert err[0] <= err[1] + 1.1e-16, err
