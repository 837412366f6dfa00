"""Ordered configurations: spectra of exact and near multiplets, the states that a
low-temperature chain settles in.

Every eigenvalue of such a block is finished by the FP64 list of trieig.cu.
Values of the FP64 path against LAPACK: both sides leave errors below O(n) eps
||H|| (bound 8 n eps ||H||_inf). The list holds 0 .. 128 eigenvalues a block:
defects in the checkerboard lift part of the multiplets.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps
NDIM = {"cubic1d": 1, "cubic2d": 2, "cubic3d": 3}


def _checkerboard(kind, L):
    pos = np.stack(np.unravel_index(np.arange(L ** NDIM[kind]), (L,) * NDIM[kind]), axis=1)
    return pos.sum(1) % 2


@pytest.mark.parametrize("kind,L", [("cubic2d", 4), ("cubic2d", 8), ("cubic3d", 6), ("cubic2d", 18), ("cubic1d", 300),
                                    ("cubic3d", 8), ("cubic2d", 30)])
def test_multiplets_by_value(cuda_ok, fkg_lib, kind, L):
    import fk_mc_gb300
    from fk_mc_gb300.lattice import dense
    n = L ** NDIM[kind]
    rng = np.random.default_rng(n)
    cb = _checkerboard(kind, L)
    fs = [cb, np.zeros(n, int), np.ones(n, int)]
    for share in (1, 2, n // 100, n // 20, n // 5):  # defects
        g = cb.copy()
        g[rng.choice(n, max(1, share), replace=False)] ^= 1
        fs.append(g)
    U, H0 = 4.0, dense(kind, L)
    s = fk_mc_gb300.Solver(max_n=n, max_batch=len(fs), precision="f64")
    s.set_lattice(0, kind, L)
    w = s.eigh_logz(np.zeros(len(fs), np.int32), np.concatenate([U * (f - 0.5) for f in fs]), 8.0)["evals"]
    s.close()
    w = w.reshape(len(fs), n)
    assert np.all(np.diff(w, axis=1) >= 0)
    for x, f in zip(w, fs):
        A = H0 + np.diag(U * (f - 0.5))
        assert np.abs(x - np.linalg.eigvalsh(A)).max() <= 8 * n * EPS * np.abs(A).sum(1).max()


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_multiplets_cost_no_warp_each(cuda_ok, fkg_lib, precision):
    """An eigenvalue of a multiplet takes ~37 FP64 Sturm counts by bisection (width 4e-6 ||T|| to 1e-16), three FP64
    operations a row, where an isolated one takes ~5 evaluations of 40-70 FP32 ones: ~10 times the time of random f,
    if a warp's counts serve 32 eigenvalues (a warp for each: 70 to 150 times)."""
    import fk_mc_gb300
    L, B = 16, 304
    n = L * L
    s = fk_mc_gb300.Solver(max_n=n, max_batch=B, precision=precision)
    s.set_lattice(0, "cubic2d", L)
    ms = []
    for f in (np.random.default_rng(1).integers(0, 2, (B, n)), np.tile(_checkerboard("cubic2d", L), (B, 1))):
        ids, d = np.zeros(B, np.int32), (4.0 * (f - 0.5)).ravel()
        s.eigh_logz(ids, d, 4.0)
        s.profile(True)
        s.eigh_logz(ids, d, 4.0)
        ms.append(s.stage_time("trieig")[0])
        s.profile(False)
    s.close()
    assert ms[1] <= 35 * ms[0], ms


@pytest.mark.parametrize("kind,L", [("cubic2d", 4), ("cubic2d", 8), ("cubic3d", 6), ("cubic2d", 24)])
def test_vectors_of_multiplets(cuda_ok, fkg_lib, kind, L):
    """Inverse iteration with the members of a multiplet orthogonalised against each other: residual below
    8 n eps ||H||, orthogonal to 1e-10 (the FP64 path's stated accuracy)."""
    import fk_mc_gb300
    from fk_mc_gb300.lattice import dense
    n = L ** NDIM[kind]
    cb = _checkerboard(kind, L)
    one = cb.copy()
    one[n // 3] ^= 1
    fs = [cb, np.zeros(n, int), one]
    s = fk_mc_gb300.Solver(max_n=n, max_batch=len(fs), precision="f64")
    s.set_lattice(0, kind, L)
    out = s.eigh_logz(np.zeros(len(fs), np.int32), np.concatenate([4.0 * (f - 0.5) for f in fs]), 8.0, vectors=True)
    s.close()
    for c, f in enumerate(fs):
        A, X, w = dense(kind, L) + np.diag(4.0 * (f - 0.5)), out["evecs"][c], out["evals"][c * n:(c + 1) * n]
        assert np.abs(A @ X - X * w).max() <= 8 * n * EPS * np.abs(A).sum(1).max()
        assert np.abs(X.T @ X - np.eye(n)).max() <= 1e-10


def test_vectors_of_multiplets_use_whole_warps(cuda_ok, fkg_lib):
    """The N = 576 lattice without f: multiplets of 4, 8 and 46. Members are solved one after the other (a lane at
    work: ~4 times the time of single eigenvalues); their orthogonalisation, n multiply-adds for every pair, must not
    take a lane's time each as well (then 40 times)."""
    import time
    import fk_mc_gb300
    L, B = 24, 16
    n = L * L
    s = fk_mc_gb300.Solver(max_n=n, max_batch=B, precision="f64")
    s.set_lattice(0, "cubic2d", L)
    ms = []
    for f in (np.random.default_rng(1).integers(0, 2, (B, n)), np.zeros((B, n))):
        ids, d = np.zeros(B, np.int32), (4.0 * (f - 0.5)).ravel()
        s.measure_ipr(ids, d, 4.0)
        t = time.perf_counter()
        s.measure_ipr(ids, d, 4.0)
        ms.append(time.perf_counter() - t)
    s.close()
    assert ms[1] <= 18 * ms[0], ms
