"""A proposal whose Hamiltonian is out of the FP64 reduction's range (entries from
2^900 on): the call fails, the proposal is not accepted and the chain stays as it
was, the other chains take their steps.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,L", [("cubic2d", 6), ("cubic2d", 13), ("cubic3d", 7)])
def test_rejected_proposal_leaves_the_chain(cuda_ok, fkg_lib, kind, L):
    import fk_mc_gb300
    from fk_mc_gb300._lib import FkgError
    s = fk_mc_gb300.Solver(max_n=1024, max_batch=2, precision="f64")
    n = s.set_lattice(0, kind, L)
    s.chains_init([0, 0], np.zeros(2 * n, np.int32), [1e280, 1.0], 0.0, 0.0, 1.0)
    f0, logz0, w0 = s.chains_get()
    with pytest.raises(FkgError, match="FKG_ERR_NUMERIC"):
        s.propose_accept(np.array([[3, 5]], np.int32), np.zeros((1, 2)))  # u = 0: whatever has a weight is accepted
    f, logz, w = s.chains_get()
    s.close()
    assert np.array_equal(f[:n], f0[:n]) and logz[0] == logz0[0] and np.array_equal(w[:n], w0[:n])
    assert f[n:].sum() == 1 and f[n + 5] == 1 and np.isfinite(logz[1])
