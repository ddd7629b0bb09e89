"""Which error a right-hand side reports where several elements fail and the mesh takes many waves of
blocks: the boundary weights before the mass matrices, and the first failing point or element, whatever
the order in which blocks run."""
import numpy as np
import pytest

import edg_westervelt_gb300 as W

pytestmark = pytest.mark.gpu

SIDES = dict(bot="absorbing_2beta", top="wall", lft="absorbing", rgt="dirichlet")


@pytest.mark.parametrize("solver", ["chebyshev", "cg"])
def test_first_error_over_many_blocks(gpu, solver):
    """N = 512: element j + N k, its blocks in this order. The constant mode is 1/2, so an entry of 3 makes
    2βv = 1.5 on its element."""
    import torch
    N = 512
    co = W.constant_coefficients(c=1.0, alpha=1e-6, beta=0.5)
    pre, _ = W.precompute(2, N, coefficients=co, mixed=False, flux="upwind", mode="source", boundary=SIDES,
                          mass_solver=solver)
    nu, nq = pre["qu1"], pre["qu1"]
    ws = W.Workspace(pre, N)
    u = torch.zeros(nu * nu * N * N, dtype=torch.float64, device=gpu)
    ut, vt = torch.empty_like(u), torch.empty_like(u)

    def error(*elements):
        v = torch.zeros_like(u)                          # [e + E (a + n b)]
        for j, k in elements:
            v[j + N * k] = 3.0
        with pytest.raises(W.ErrorException) as ei:
            ws.rhs(u, v, 10.0, ut, vt)                   # past the source
        return str(ei.value), ws.error_key

    def bnd(kind, s, m):
        kk = "2" if kind == "absorbing_2beta" else ""
        return f"boundary weight 1 - {kk}βv_h ≤ 0 at a face point ({kind} side)", 2 * (s * nq * N + m * nq) + 1

    def mass(j, k):
        where = j + N * k + 1 if solver == "chebyshev" else f"({j + 1}, {k + 1})"
        return f"mass matrix not positive definite on element {where}: 1 - 2βv_h ≤ 0", j + N * k + 1

    for _ in range(5):
        # an element that is not definite in the first blocks, a failing weight in the last ones
        # (absorbing kinds: 1 - kβv with k = 2 at the bottom, 1 on the left)
        assert error((5, 1), (0, N - 2)) == bnd("absorbing_2beta", 0, N - 2)
        # weights in the second and the last column of elements; the later one has the smaller key
        assert error((0, 1), (0, N - 1)) == bnd("absorbing_2beta", 0, 1)
        v = (0, N - 1), (200, 0)
        assert error(*v, (7, 1)) == bnd("absorbing_2beta", 0, N - 1)
        # elements alone, in blocks far from each other
        assert error((300, 300), (3, 2), (4, N - 2)) == mass(3, 2)
    ws.rhs(u, torch.zeros_like(u), 10.0, ut, vt)         # and the workspace goes on
    assert bool(torch.isfinite(ut).all()) and bool(torch.isfinite(vt).all())


def test_errors_of_one_stage_only(gpu):
    """An error ends the call: steps after it change neither the state nor the error."""
    N = 16
    co = W.constant_coefficients(c=1.0, alpha=1e-6, beta=0.5)
    for solver in ("chebyshev", "cg"):
        pre, _ = W.precompute(3, N, coefficients=co, mixed=False, flux="upwind", mode="source", boundary=SIDES,
                              mass_solver=solver)
        ws = W.Workspace(pre, N)
        u = np.zeros((N, N, 4, 4), order="F")
        v = np.zeros_like(u, order="F")
        v[9, 9, 0, 0] = 3.0
        v[9, 3, 0, 0] = 3.0
        u0, v0 = u.copy(order="F"), v.copy(order="F")
        for n in (1, 2, 5):
            with pytest.raises(W.ErrorException, match="mass matrix"):
                ws.rk4_steps(u, v, 10.0, 1e-4, n)
            assert ws.error_key == 9 + N * 3 + 1
            assert np.array_equal(u, u0) and np.array_equal(v, v0)


def test_a_matrix_singular_to_rounding_is_refused(gpu):
    """1 - 2βv from some 0.1 to 1e18: θ and δ of the Chebyshev interval are the same double, and no number of steps is
    enough (the reference's ceil(Int, Inf) throws)."""
    N = 3
    co = W.constant_coefficients(c=1.0, alpha=1e-6, beta=0.5)
    pre, _ = W.precompute(3, N, coefficients=co, mixed=False, flux="upwind", mode="source", boundary="wall", kappa=0.5)
    P = np.asarray(pre["P_h_v"])
    u = np.zeros((N, N, 4, 4), order="F")
    v = np.zeros_like(u, order="F")
    X = np.zeros((4, 4))
    X[1, 0] = 1.0
    g = P @ X @ P.T
    X *= 1e18 / np.ptp(g)
    X[0, 0] = 2.0 * (0.9 - (P @ X @ P.T).max())
    v[1, 1] = X
    ws = W.Workspace(pre, N)
    with pytest.raises(W.ErrorException, match="mass matrix not positive definite on element 5"):
        ws.rhs(u, v, 10.0)
