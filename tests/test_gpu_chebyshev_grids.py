"""The Chebyshev logZ's coefficient sums on coarse and fine grids (a thread per
moment, a warp from 64 points on; the table of T_m on the grid in blocks of
moments that fit 64 KB) against the numpy restatement of calc_chebyshev.

logZ = sum of M coefficients times moments; bounds and moments are good to a few
1e-14 (double-float) and a moment's condition grows with m^2: 1e-10 relative up
to M = 200.
"""
import numpy as np
import pytest

from oracle import chebyshev as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,G", [(2, 2), (4, 63), (4, 64), (4, 65), (32, 33), (34, 257), (130, 64), (200, 400), (10, 4096),
                                 (2, 4096)])
def test_logz_on_grids(cuda_ok, fkg_lib, oracle, M, G):
    import fk_mc_gb300
    L, U, beta, B = 8, 2.0, 4.0, 2
    s = fk_mc_gb300.Solver(max_n=64, max_batch=B, precision="f64")
    s.set_lattice(0, "cubic2d", L)
    s.set_chebyshev(M, G)
    f = np.random.default_rng(M + G).integers(0, 2, (B, L * L))
    logz = s.chebyshev_logz(np.zeros(B, np.int32), (U * (f - 0.5)).ravel(), beta)["logz"]
    s.close()
    csr = oracle.lattice_csr("cubic2d", L, -1.0)
    for c in range(B):
        ref = C.calc_chebyshev(C.dense_h(csr, f[c], U, U / 2), beta, M, G)["logZ"]
        assert abs(logz[c] - ref) <= 1e-10 * abs(ref)


def test_time_on_the_finest_grid(cuda_ok, fkg_lib):
    """M G is 64 times larger on the finest grid than at M = 64, G = 1024, and so is the work: at most 1.5 times that
    in time (few threads on few moments at a time: 180 times)."""
    import fk_mc_gb300
    s = fk_mc_gb300.Solver(max_n=64, max_batch=1, precision="f64")
    s.set_lattice(0, "cubic2d", 8)
    d = 2.0 * (np.random.default_rng(1).integers(0, 2, 64) - 0.5)
    ms = []
    for M, G in ((64, 1024), (1024, 4096)):
        s.set_chebyshev(M, G)
        s.chebyshev_logz([0], d, 4.0)
        s.profile(True)
        s.chebyshev_logz([0], d, 4.0)
        ms.append(s.stage_time("logz")[0])
        s.profile(False)
    s.close()
    assert ms[1] <= 96 * ms[0], ms
