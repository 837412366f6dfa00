"""The cluster reduction of the mixed path (sytrd_cluster.cuh in FP32) at its
edges: orders around the tile size, both warp counts and panel widths, every
cluster size (the batch decides it), tiles beyond shared memory.

The mixed path's eigenvalues are Rayleigh quotients with H, second order in the
FP32 eigenvectors' error; the bound is the path's stated 1e-9 ||H|| for lattices
with random f (a disordered chain of hundreds of sites has gaps small enough to
exceed it with any reduction)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solver(cuda_ok, fkg_lib):
    import fk_mc_gb300
    s = fk_mc_gb300.Solver(max_n=1024, max_batch=320, precision="mixed", tuning=None)
    yield s
    s.close()


def _grid(n):
    """Periodic lx x ly lattice of n sites (a ring if n is prime), hopping -1."""
    lx = max(k for k in range(1, int(n ** 0.5) + 1) if n % k == 0)
    H = np.zeros((n, n))
    x, y = np.arange(n) % lx, np.arange(n) // lx
    for dx, dy in ((1, 0), (0, 1)):
        j = (x + dx) % lx + lx * ((y + dy) % (n // lx))
        far = j != np.arange(n)
        np.add.at(H, (np.arange(n)[far], j[far]), -1.0)
        np.add.at(H, (j[far], np.arange(n)[far]), -1.0)
    return H


def _run(s, n, B, seed):
    rng = np.random.default_rng(seed)
    H = _grid(n)
    nz = H != 0
    s.set_hopping(0, np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32),
                  np.nonzero(nz)[1].astype(np.int32), H[nz])
    d = rng.integers(0, 2, (B, n)) * 2.0 - 1.0 + 0.1 * rng.uniform(-1, 1, (B, n))
    w = s.eigh_logz(np.zeros(B, np.int32), d.ravel(), 1.5)["evals"].reshape(B, n)
    for c in sorted({0, B // 2, B - 1}):
        ref = np.linalg.eigvalsh(H + np.diag(d[c]))
        assert np.abs(w[c] - ref).max() <= 1e-9 * np.abs(ref).max(), (n, B, c)


@pytest.mark.parametrize("n", [3, 4, 5, 31, 32, 33, 63, 65, 96, 97, 129, 255, 257, 321])
def test_orders_around_tiles(solver, n):
    _run(solver, n, 3, n)


@pytest.mark.parametrize("n,B", [(200, 310), (256, 305), (130, 306), (256, 153), (350, 1), (350, 160), (480, 160), (481, 160), (600, 20),
                                 (700, 60), (1000, 2), (1024, 17), (800, 100), (400, 40), (576, 25), (784, 40), (1024, 22)])
def test_cluster_sizes_and_warp_counts(solver, n, B):
    _run(solver, n, B, n + B)


@pytest.mark.parametrize("sizes,variant", [((31, 32), 3), ((32, 12), 1)])
def test_vector_solves_above_960(cuda_ok, fkg_lib, sizes, variant):
    """Solves whose FP32 eigenvectors leave the library: with the shipped table they are, bit for bit, the two-stage
    reduction's where every chain is above 960, and the width-8 one-stage reduction's in a batch of other orders."""
    import fk_mc_gb300
    res = []
    for explicit in (False, True):
        s = fk_mc_gb300.Solver(max_n=1024, max_batch=2, precision="mixed")
        if explicit:
            for n_max in (192, 1024):
                s.set_tuning("mixed", n_max, variant)
        f = np.concatenate([np.random.default_rng(L).integers(0, 2, s.set_lattice(i, "cubic2d", L))
                            for i, L in enumerate(sizes)])
        res.append(s.free_energy_grad(np.arange(2, dtype=np.int32), f, 2.0, 1.0, 1.0, 4.0))
        s.close()
    for k in ("F", "dU", "dt", "dmu", "dbeta"):
        assert np.array_equal(res[0][k], res[1][k]), k
