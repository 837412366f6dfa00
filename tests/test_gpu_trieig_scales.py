"""FP64 eigenvalues of Hamiltonians in other units of energy: the double-float
recurrences of trieig.cu work on T scaled to norm 1 .. 2.

Bound against LAPACK: 8 n eps ||H||_inf (both sides leave errors below O(n) eps
||H||). A scale by a power of two changes no digit of H, so the eigenvalue stage
has the same work at every scale: at most twice the time leaves room for noise,
where the FP64 list that takes what leaves FP32's range costs 30 times as much.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _hopping(kind, L, t):
    from fk_mc_gb300.lattice import dense
    H = dense(kind, L) * t
    nz = H != 0
    return H, (np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32), np.nonzero(nz)[1].astype(np.int32), H[nz])


@pytest.mark.parametrize("scale", [1e-12, 1e-6, 1e-4, 0.3, 3e3, 11604.5, 1e5, 1e6, 1e7, 1e12])
@pytest.mark.parametrize("kind,L", [("cubic1d", 97), ("cubic1d", 100), ("cubic2d", 17)])
def test_values_at_scales(cuda_ok, fkg_lib, kind, L, scale):
    import fk_mc_gb300
    H, csr = _hopping(kind, L, scale)
    n, B = H.shape[0], 3
    s = fk_mc_gb300.Solver(max_n=n, max_batch=B, precision="f64")
    s.set_hopping(0, *csr)
    d = scale * 4.0 * (np.random.default_rng(L).integers(0, 2, (B, n)) - 0.5)
    w = s.eigh_logz(np.zeros(B, np.int32), d.ravel(), 1.0 / scale)["evals"].reshape(B, n)
    s.close()
    for c in range(B):
        A = H + np.diag(d[c])
        assert np.abs(w[c] - np.linalg.eigvalsh(A)).max() <= 8 * n * EPS * np.abs(A).sum(1).max()


def test_time_does_not_depend_on_the_scale(cuda_ok, fkg_lib):
    import fk_mc_gb300
    B, L = 304, 16
    n = L * L
    s = fk_mc_gb300.Solver(max_n=n, max_batch=B, precision="f64")
    f = np.random.default_rng(1).integers(0, 2, (B, n)) - 0.5
    ms = []
    for scale in (1.0, 2.0 ** -13, 2.0 ** 14, 2.0 ** 20):
        s.set_hopping(0, *_hopping("cubic2d", L, scale)[1])
        ids, d = np.zeros(B, np.int32), (2.0 * scale * f).ravel()
        s.eigh_logz(ids, d, 1.0 / scale)
        s.profile(True)
        for _ in range(3):
            s.eigh_logz(ids, d, 1.0 / scale)
        ms.append(s.stage_time("trieig")[0])
        s.profile(False)
    s.close()
    assert max(ms) <= 2 * ms[0], ms


@pytest.mark.parametrize("n,small", [(96, 2.0 ** -20), (300, 2.0 ** -20), (300, 2.0 ** -45)])
def test_uncoupled_blocks_of_different_scale(cuda_ok, fkg_lib, n, small):
    """Values to 8 n eps ||H||, residuals of the vectors to the same, and vectors orthonormal to 1e-9 (clusters, into which
    the small block's values may fall, are orthogonalised)."""
    import fk_mc_gb300
    A = np.zeros((n, n))
    i = np.arange(n // 2 - 1)
    for o, t in ((0, 1.0), (n // 2, small)):
        A[o + i, o + i + 1] = A[o + i + 1, o + i] = -t
    nz = A != 0
    s = fk_mc_gb300.Solver(max_n=n, max_batch=1, precision="f64")
    s.set_hopping(0, np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32), np.nonzero(nz)[1].astype(np.int32),
                  A[nz])
    d = np.random.default_rng(n).uniform(-2, 2, n) * np.where(np.arange(n) < n // 2, 1.0, small)
    out = s.eigh_logz([0], d, 3.0, vectors=True)
    s.close()
    A += np.diag(d)
    w, X, bound = out["evals"], out["evecs"][0], 8 * n * EPS * np.abs(A).sum(1).max()
    assert np.abs(w - np.linalg.eigvalsh(A)).max() <= bound
    assert np.abs(A @ X - X * w).max() <= bound
    assert np.abs(X.T @ X - np.eye(n)).max() <= 1e-9
