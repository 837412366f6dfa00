"""FP64 eigenvectors (inverse iteration, then the fixed-point back-transformation) at the orders where the
kernels' tiles end: rows a lane holds, columns a CTA takes, reflectors to a block; one chain of the order and a
smaller one in the same call.

Tolerances: the residual of a backward-stable solver is below p(n) eps ||H|| with p(n) = O(n), taken as 8 n; vectors
whose eigenvalues are further apart than 1e-5 ||T|| are orthogonal to eps / 1e-5 times a small factor, closer ones are
orthogonalised: 1e-10.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _random_csr(n, rng, density=4):
    H = np.zeros((n, n))
    for _ in range(density):
        p = rng.permutation(n)
        v = rng.uniform(-1, 1, n)
        H[np.arange(n), p] += v
        H[p, np.arange(n)] += v
    return H


def _set(s, lid, H):
    nz = H != 0
    rowptr = np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32)
    s.set_hopping(lid, rowptr, np.nonzero(nz)[1].astype(np.int32), H[nz])


@pytest.fixture(scope="module")
def solver(cuda_ok, fkg_lib):
    import fk_mc_gb300
    s = fk_mc_gb300.Solver(max_n=1024, max_batch=4, precision="f64")
    yield s
    s.close()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 15, 16, 17, 31, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 384, 385,
                               576, 577, 768, 769, 1023, 1024])
def test_vectors_at_the_edges(solver, n):
    rng = np.random.default_rng(n)
    small = max(1, n // 3)
    Hs = [_random_csr(n, rng), _random_csr(small, rng)]
    for lid, H in enumerate(Hs):
        _set(solver, lid, H)
    ids = [0, 1, 0]
    diags = [rng.uniform(-2, 2, Hs[i].shape[0]) for i in ids]
    out = solver.eigh_logz(ids, np.concatenate(diags), 1.5, vectors=True)
    off = 0
    for i, d, X in zip(ids, diags, out["evecs"]):
        A = Hs[i] + np.diag(d)
        m = len(d)
        w = out["evals"][off:off + m]
        off += m
        assert np.abs(A @ X - X * w).max() <= 8 * m * EPS * np.abs(A).sum(1).max()
        assert np.abs(X.T @ X - np.eye(m)).max() <= 1e-10
