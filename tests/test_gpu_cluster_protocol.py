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
