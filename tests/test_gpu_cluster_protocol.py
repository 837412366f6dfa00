"""The cluster reduction's exchanges between CTAs (sytrd_cluster.cuh): the work
list's items reach every CTA of a cluster after it has started, and rejected
chains leave the cluster's CTAs in step with each other.

Results are compared bit for bit with those of a solve of the same inputs on an
idle GPU (the fixed-point sums do not depend on the schedule) and with LAPACK
within 8 n eps ||H||_inf (a backward-stable reduction and LAPACK's both leave
eigenvalue errors below O(n) eps ||H||).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.fixture()
def solver(cuda_ok, fkg_lib):
    import fk_mc_gb300
    s = fk_mc_gb300.Solver(max_n=1024, max_batch=64, precision="f64")
    yield s
    s.close()


@pytest.mark.parametrize("kind,L,B", [("cubic3d", 7, 1), ("cubic3d", 7, 60), ("cubic2d", 24, 40)])
def test_clusters_start_on_a_busy_gpu(solver, kind, L, B):
    import torch
    n = solver.set_lattice(0, kind, L)
    d = np.random.default_rng(B).uniform(-2, 2, B * n)
    ids = np.zeros(B, np.int32)
    quiet = solver.eigh_logz(ids, d, 1.5)["evals"]
    a = torch.ones((4096, 4096), device="cuda")
    other = torch.cuda.Stream()
    for _ in range(3):
        with torch.cuda.stream(other):  # kernels that come and go on every SM meanwhile
            for _ in range(20):
                a = a * 1.0
        assert np.array_equal(solver.eigh_logz(ids, d, 1.5)["evals"], quiet)
    torch.cuda.synchronize()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("n,B", [(353, 9), (353, 40), (1024, 17)])
def test_rejected_chains_between_good_ones(solver, n, B, bad):
    """Chains with an entry that is not finite among good ones: an error, and the next call's results are right."""
    from fk_mc_gb300._lib import FkgError
    rng = np.random.default_rng(n + B)
    i = np.arange(n)
    H = np.zeros((n, n))
    for step in (1, 19):
        H[i, (i + step) % n] += -1.0
        H[(i + step) % n, i] += -1.0
    nz = H != 0
    solver.set_hopping(0, np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32),
                       np.nonzero(nz)[1].astype(np.int32), H[nz])
    d = rng.uniform(-2, 2, (B, n))
    ids = np.zeros(B, np.int32)
    for rows in ([0], [B - 1], list(range(0, B, 2)), list(range(B))):
        x = d.copy()
        x[rows, rng.integers(0, n, len(rows))] = bad
        with pytest.raises(FkgError, match="FKG_ERR_NUMERIC"):
            solver.eigh_logz(ids, x.ravel(), 1.5)
    w = solver.eigh_logz(ids, d.ravel(), 1.5)["evals"].reshape(B, n)
    for c in sorted({0, B // 2, B - 1}):
        A = H + np.diag(d[c])
        assert np.abs(w[c] - np.linalg.eigvalsh(A)).max() <= 8 * n * EPS * np.abs(A).sum(1).max(), c


@pytest.mark.parametrize("kind,L,B", [("cubic2d", 15, 320), ("cubic2d", 19, 5), ("cubic2d", 31, 20)])
def test_fp32_products_do_not_depend_on_timing(cuda_ok, fkg_lib, kind, L, B):
    """Partial products that different lanes of a warp add to one entry: the FP32 sums have one order."""
    import fk_mc_gb300
    s = fk_mc_gb300.Solver(max_n=1024, max_batch=B, precision="mixed", tuning=None)
    n = s.set_lattice(0, kind, L)
    f = np.random.default_rng(L).integers(0, 2, (B, n))
    runs = [s.eigh_logz(np.zeros(B, np.int32), (2.0 * f - 1.0).ravel(), 3.0)["evals"] for _ in range(4)]
    s.close()
    for w in runs[1:]:
        assert np.array_equal(w, runs[0])


@pytest.mark.parametrize("n,B", [(200, 1), (353, 1), (600, 20)])
def test_scale_at_a_rounding_edge(solver, n, B):
    """A row whose absolute sum lies on either side of a power of two's threshold, as the order of its additions
    has it: all CTAs of a cluster still work in one scale."""
    a, b, c = 0.6870830067379103, 0.23316528022862978, 1.0797517111708146
    assert {((a + b) + c) * (1 + 2.0 ** -30) >= 2.0, ((a + c) + b) * (1 + 2.0 ** -30) >= 2.0} == {True, False}
    H = np.zeros((n, n))
    i = np.arange(3, n - 1)
    H[i, i + 1] = H[i + 1, i] = 0.1
    H[0, 1] = H[1, 0] = b
    H[0, 2] = H[2, 0] = c
    H[2, 3] = H[3, 2] = 0.05
    nz = H != 0
    solver.set_hopping(0, np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32),
                       np.nonzero(nz)[1].astype(np.int32), H[nz])
    d = np.zeros(n)
    d[0] = a
    ref = np.linalg.eigvalsh(H + np.diag(d))
    for _ in range(10):
        w = solver.eigh_logz(np.zeros(B, np.int32), np.tile(d, B), 1.5)["evals"].reshape(B, n)
        assert np.abs(w - ref).max() <= 8 * n * EPS * np.abs(H + np.diag(d)).sum(1).max()


def test_two_threads_with_contexts_of_different_size(cuda_ok, fkg_lib):
    """Launches of one kernel with different shared memory from two threads: neither changes the other's limit."""
    import threading
    import fk_mc_gb300
    errors = []

    def work(L, B, seed):
        try:
            s = fk_mc_gb300.Solver(max_n=L * L, max_batch=B, precision="f64")
            n = s.set_lattice(0, "cubic2d", L)
            d = np.random.default_rng(seed).uniform(-2, 2, B * n)
            first = s.eigh_logz(np.zeros(B, np.int32), d, 2.0)["evals"]
            for _ in range(60):
                assert np.array_equal(s.eigh_logz(np.zeros(B, np.int32), d, 2.0)["evals"], first)
            s.close()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in ((12, 1, 1), (23, 2, 2), (15, 9, 3))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
