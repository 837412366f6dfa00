"""Spectral bounds of the Chebyshev expansion: Lanczos runs whose Krylov space ends
early, and the mean error over many chains.

Errors: the double-float recursion rounds at 2^-48 = 3.6e-15 of ||H|| a step; with
scalars rounded as FP64 results the mean over random f stays below that (2.8e-15
measured, 2.9e-15 with FP64 scalars, 3.5e-15 with scalars good to 1e-14).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f", ["stripe", "checkerboard", "empty"])
def test_exhausted_krylov_space(cuda_ok, fkg_lib, f):
    """cubic2d L = 4 with an ordered f has at most 8 distinct eigenvalues that the start vector reaches: the run ends
    there instead of at the first check of longer runs (32 steps and two more)."""
    import fk_mc_gb300
    from fk_mc_gb300.lattice import dense
    pos = np.stack(np.unravel_index(np.arange(16), (4, 4)), axis=1)
    f = {"stripe": pos[:, 0] % 4 < 2, "checkerboard": pos.sum(1) % 2, "empty": np.zeros(16)}[f]
    d = 4.0 * (f - 0.5)
    s = fk_mc_gb300.Solver(max_n=16, max_batch=1, precision="f64")
    s.set_lattice(0, "cubic2d", 4)
    s.set_chebyshev(6, 12)
    r = s.chebyshev_logz([0], d, 4.0)
    s.close()
    w = np.linalg.eigvalsh(dense("cubic2d", 4) + np.diag(d))
    assert r["lanczos_steps"][0] <= 16
    assert max(abs(r["e_min"][0] - w[0]), abs(r["e_max"][0] - w[-1])) <= 1e-13 * np.abs(w).max()


def test_mean_error_of_the_bounds(cuda_ok, fkg_lib):
    import fk_mc_gb300
    from fk_mc_gb300.lattice import dense
    means, B = [], 150
    for kind, L, n in (("cubic1d", 200, 200), ("cubic2d", 8, 64), ("cubic2d", 13, 169), ("cubic3d", 5, 125)):
        s = fk_mc_gb300.Solver(max_n=n, max_batch=B, precision="f64")
        s.set_lattice(0, kind, L)
        s.set_chebyshev(10, 20)
        H = dense(kind, L)
        for U in (1.0, 4.0):
            d = U * (np.random.default_rng(L).integers(0, 2, (B, n)) - 0.5)
            r = s.chebyshev_logz(np.zeros(B, np.int32), d.ravel(), 5.0)
            w = np.array([np.linalg.eigvalsh(H + np.diag(x))[[0, -1]] for x in d])
            e = np.maximum(np.abs(r["e_min"] - w[:, 0]), np.abs(r["e_max"] - w[:, 1])) / np.abs(w).max(1)
            means.append(e.mean())
        s.close()
    assert np.exp(np.mean(np.log(means))) <= 2.0 ** -48, means


def test_bounds_of_converged_spectra(cuda_ok, fkg_lib):
    """The Krylov space of cubic2d L = 8 is exhausted long after its ends have converged; copies of them come up, whose
    distance is the scalars' rounding. Bound: two roundings of a pair; a twice rounded 1 / beta left 1.3e-14."""
    import fk_mc_gb300
    from fk_mc_gb300.lattice import dense
    B, n = 25, 64
    s = fk_mc_gb300.Solver(max_n=n, max_batch=B, precision="f64")
    s.set_lattice(0, "cubic2d", 8)
    s.set_chebyshev(10, 20)
    d = 0.5 * (np.random.default_rng(0).integers(0, 2, (B, n)) - 0.5)
    r = s.chebyshev_logz(np.zeros(B, np.int32), d.ravel(), 5.0)
    s.close()
    w = np.array([np.linalg.eigvalsh(dense("cubic2d", 8) + np.diag(x))[[0, -1]] for x in d])
    assert np.mean(np.abs(r["e_min"] - w[:, 0]) / np.abs(w).max(1)) <= 2.0 * 2.0 ** -48
    assert np.mean(np.abs(r["e_max"] - w[:, 1]) / np.abs(w).max(1)) <= 2.0 * 2.0 ** -48
