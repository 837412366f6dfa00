"""FP64 eigenvalues that lie close together, to the last bits: open disordered
chains, U = 4, whose localised states have neighbours down to 1e-6 ||T|| and less.

The chain's matrix is tridiagonal already and its entries (+-2, -1) are exact in the
reduction's fixed-point numbers, so the eigenvalue stage works on T = H and its
error is all there is. Reference: bisection with Sturm counts in long double.
Bound 4 eps ||T||: the rounding of FP64 recurrences is a perturbation of T's entries
by 3 eps of themselves at most (three operations an entry), and bisection stops at
2 eps |lambda| + eps ||T|| / 2.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _reference(d, near):
    """Eigenvalues of the tridiagonal (d, -1) in long double; near: to 1e-12."""
    d = d.astype(np.longdouble)
    lo, hi = near.astype(np.longdouble) - 1e-12, near.astype(np.longdouble) + 1e-12
    j = np.arange(d.size)
    for _ in range(24):  # 2e-12 / 2^24 = 1e-19
        x = (lo + hi) / 2
        q = d[0] - x
        c = (q < 0).astype(int)
        for i in range(1, d.size):
            q = np.where(q == 0, np.longdouble(1e-40), q)
            q = d[i] - x - 1 / q
            c += q < 0
        hi = np.where(c > j, x, hi)
        lo = np.where(c > j, lo, x)
    return (lo + hi) / 2


@pytest.mark.parametrize("n,seed", [(33, 0), (128, 1), (129, 2), (343, 0), (343, 2), (900, 0)])
def test_close_eigenvalues_to_four_ulps_of_the_norm(cuda_ok, fkg_lib, n, seed):
    import fk_mc_gb300
    d = 4.0 * (np.random.default_rng(seed).integers(0, 2, n) - 0.5)
    i = np.arange(n)
    rows = np.concatenate([i[1:], i[:-1]])
    cols = np.concatenate([i[:-1], i[1:]])
    order = np.lexsort((cols, rows))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    s = fk_mc_gb300.Solver(max_n=n, max_batch=1, precision="f64")
    s.set_hopping(0, rowptr, cols[order].astype(np.int32), np.full(2 * (n - 1), -1.0))
    w = s.eigh_logz([0], d, 5.0)["evals"]
    s.close()
    T = np.diag(d) - np.diag(np.ones(n - 1), 1) - np.diag(np.ones(n - 1), -1)
    ref = _reference(d, np.linalg.eigvalsh(T))
    assert np.abs(w - ref).max() <= 4 * EPS * np.abs(T).sum(1).max()
