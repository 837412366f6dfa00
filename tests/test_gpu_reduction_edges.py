"""The cluster reduction of the FP64 path (sytrd_cluster.cuh) at its edges: orders
around the tile and warp sizes, every cluster size (the batch decides it),
tiles beyond shared memory, flat columns, scales far from 1, and errors.

Tolerance: a backward-stable reduction and LAPACK's both leave eigenvalue errors
below p(n) eps ||H|| with p(n) = O(n); 8 n eps ||H||_inf bounds their difference.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _random_csr(n, rng, density=4, scale=1.0):
    H = np.zeros((n, n))
    for _ in range(density):
        p = rng.permutation(n)
        v = rng.uniform(-1, 1, n) * scale
        H[np.arange(n), p] += v
        H[p, np.arange(n)] += v
    return H


def _set(s, lid, H):
    n = H.shape[0]
    nz = H != 0
    rowptr = np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32)
    s.set_hopping(lid, rowptr, np.nonzero(nz)[1].astype(np.int32), H[nz])


def _check(s, H, diags):
    n, B = H.shape[0], len(diags)
    out = s.eigh_logz(np.zeros(B, np.int32), np.concatenate(diags), 1.5)
    w = out["evals"].reshape(B, n)
    for c in sorted({0, B // 2, B - 1}):
        A = H + np.diag(diags[c])
        ref = np.linalg.eigvalsh(A)
        bound = 8 * n * EPS * np.abs(A).sum(1).max()
        assert np.abs(w[c] - ref).max() <= bound, (n, B, c)


@pytest.fixture()
def solver(cuda_ok, fkg_lib):
    import fk_mc_gb300
    s = fk_mc_gb300.Solver(max_n=1024, max_batch=170, precision="f64")
    yield s
    s.close()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 32, 33, 34, 63, 64, 65, 95, 97, 128, 129, 160, 193, 255, 257, 321])
def test_orders_around_tiles(solver, n):
    rng = np.random.default_rng(n)
    H = _random_csr(n, rng)
    _set(solver, 0, H)
    _check(solver, H, [rng.uniform(-2, 2, n) for _ in range(3)])


@pytest.mark.parametrize("n,B", [(353, 1), (353, 20), (353, 60), (353, 160), (200, 170), (384, 170), (385, 153), (700, 1), (700, 40), (1000, 2), (1024, 17), (400, 40), (576, 25), (784, 40), (1000, 22), (1024, 28)])
def test_cluster_sizes_and_spilled_tiles(solver, n, B):
    rng = np.random.default_rng(n + B)
    H = _random_csr(n, rng)
    _set(solver, 0, H)
    _check(solver, H, [rng.uniform(-2, 2, n) for _ in range(B)])


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("n", [3, 66, 131, 290])
def test_panel_widths(solver, n, variant):
    rng = np.random.default_rng(n)
    H = _random_csr(n, rng)
    _set(solver, 0, H)
    solver.set_tuning("f64", n, variant)
    _check(solver, H, [rng.uniform(-2, 2, n) for _ in range(2)])


@pytest.mark.parametrize("n", [40, 200])
def test_flat_columns(solver, n):
    """Diagonal, block-diagonal and already tridiagonal matrices: columns whose reflector is the identity."""
    rng = np.random.default_rng(n)
    d = [rng.uniform(-2, 2, n)]
    Z = np.zeros((n, n))
    _set(solver, 0, Z)
    _check(solver, Z, d)
    # the zero matrix: exact up to the eigenvalue stage's pivot floor (a few DBL_MIN)
    assert np.abs(solver.eigh_logz([0], np.zeros(n), 1.5)["evals"]).max() <= 16 * np.finfo(float).tiny
    T = np.diag(np.ones(n - 1), 1)
    T[n // 2, n // 2 + 1] = 0.0
    T = T + T.T
    _set(solver, 0, T)
    _check(solver, T, d)
    K = _random_csr(n // 2, rng)
    Bk = np.kron(np.eye(2), K)
    _set(solver, 0, Bk)
    _check(solver, Bk, [rng.uniform(-2, 2, 2 * (n // 2))])


@pytest.mark.parametrize("scale", [1e-8, 1e8])  # the eigenvalue stage squares e in FP32
def test_scales(solver, scale):
    n = 150
    rng = np.random.default_rng(7)
    H = _random_csr(n, rng, scale=scale)
    _set(solver, 0, H)
    _check(solver, H, [rng.uniform(-2, 2, n) * scale])


@pytest.mark.parametrize("kind,L", [("triangular", 6), ("cubic2d", 8), ("cubic3d", 4)])
def test_degenerate_spectrum_is_ascending(solver, kind, L):
    """Ordered configurations on symmetric lattices: exact multiplets, eigenvalues still ascending."""
    n = solver.set_lattice(0, kind, L)
    i = np.arange(n)
    fs = [np.zeros(n), np.ones(n), i % 2, (i // L + i) % 2, (i % 3 == 0) * 1.0]
    w = solver.eigh_logz(np.zeros(len(fs), np.int32), np.concatenate([4.0 * (f - 0.5) for f in fs]), 8.0)["evals"]
    assert np.all(np.diff(w.reshape(len(fs), n), axis=1) >= 0)


def test_uneven_batch_of_small_and_large(solver):
    rng = np.random.default_rng(3)
    Hs = [_random_csr(n, rng) for n in (1, 2, 33, 96, 500, 130)]
    for i, H in enumerate(Hs):
        _set(solver, i, H)
    ids = np.array([4, 0, 1, 2, 3, 5, 2, 4, 1], np.int32)
    ds = [rng.uniform(-1, 1, Hs[i].shape[0]) for i in ids]
    w = solver.eigh_logz(ids, np.concatenate(ds), 2.0)["evals"]
    off = 0
    for i, d in zip(ids, ds):
        A = Hs[i] + np.diag(d)
        n = A.shape[0]
        assert np.abs(w[off:off + n] - np.linalg.eigvalsh(A)).max() <= 8 * n * EPS * np.abs(A).sum(1).max()
        off += n


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_not_finite_is_an_error(solver, bad):
    from fk_mc_gb300._lib import FkgError
    solver.set_lattice(0, "cubic2d", 6)
    d = np.zeros((2, 36))
    d[1, 7] = bad
    with pytest.raises(FkgError, match="FKG_ERR_NUMERIC"):
        solver.eigh_logz([0, 0], d, 1.0)
    assert np.all(np.isfinite(solver.eigh_logz([0], np.zeros(36), 1.0)["evals"]))


@pytest.mark.parametrize("n", [33, 150, 401])
def test_vectors_from_stored_reflectors(solver, n):
    rng = np.random.default_rng(n)
    H = _random_csr(n, rng)
    _set(solver, 0, H)
    d = rng.uniform(-2, 2, n)
    out = solver.eigh_logz([0], d, 1.0, vectors=True)
    V, w, A = out["evecs"][0], out["evals"], H + np.diag(d)
    nrm = np.abs(A).sum(1).max()
    assert np.abs(V.T @ V - np.eye(n)).max() < 1e-10        # the FP64 path's stated accuracy
    assert np.abs(A @ V - V * w).max() < 1e-10 * nrm
