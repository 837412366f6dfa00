"""Which reduction the mixed path takes: the caller's settings per size bucket, for
solves and for resident chains, by the number of launches (a two-stage solve has
two more than a one-stage one) and by results.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def solver(cuda_ok, fkg_lib):
    import fk_mc_gb300
    s = fk_mc_gb300.Solver(max_n=1024, max_batch=2, precision="mixed", tuning=None)
    s.set_graphs(False)
    yield s
    s.close()


def _launches(s, call):
    call()  # workspaces
    n0 = s.launch_count()
    call()
    return s.launch_count() - n0


def _lattices(s, *sizes):
    return [s.set_lattice(i, "cubic2d", L) for i, L in enumerate(sizes)]


def _diag(ns, seed=3):
    return np.random.default_rng(seed).integers(0, 2, sum(ns)) * 2.0 - 1.0


def test_chains_can_be_set_apart(solver):
    s = solver
    ns = _lattices(s, 9, 9)
    ids, rng = [0, 1], np.random.default_rng(1)
    f, site, u = rng.integers(0, 2, sum(ns)), rng.integers(0, 81, (1, 2)), np.full((1, 2), 2.0)  # u = 2: none accepted
    solve = lambda: s.eigh_logz(ids, _diag(ns), 4.0)
    step = lambda: s.propose_accept(site, u)
    init = lambda: s.chains_init(ids, f, 2.0, 1.0, 1.0, 4.0)
    init()
    one_solve, one_step, one_init, dl = _launches(s, solve), _launches(s, step), _launches(s, init), step()[1]
    for solves, chains, more_solve, more_step in [(3, None, 2, 2), (3, 2, 2, 0), (3, 1, 2, 2), (3, -1, 2, 2),
                                                  (1, None, 0, 0), (1, 0, 0, 2), (1, 100, 0, 0), (3, None, 2, 2),
                                                  (-1, None, 0, 0)]:  # two chains
        s.set_tuning("mixed", 81, solves)  # takes the chains' bucket back to its own choice
        if chains is not None:
            s.set_tuning_chains(81, chains)
        case = (solves, chains)
        assert _launches(s, solve) == one_solve + more_solve, case
        assert _launches(s, init) == one_init + more_step, case
        assert _launches(s, step) == one_step + more_step, case
        assert np.abs(step()[1] - dl).max() < 1e-8, case


def test_chains_setting_rejects_what_it_does_not_know(solver):
    from fk_mc_gb300._lib import FkgError
    for n_max, v in [(0, 0), (1025, 0), (64, -2)]:
        with pytest.raises(FkgError, match="FKG_ERR_ARG"):
            solver.set_tuning_chains(n_max, v)


def test_shipped_table_by_size_and_kind(cuda_ok, fkg_lib):
    """With the shipped table: solves of chains that are all above 960 take two stages, with eigenvectors or without;
    solves of an uneven batch one; two resident chains of N = 1024 one (their entry's number of chains is above two)."""
    import fk_mc_gb300
    s = fk_mc_gb300.Solver(max_n=1024, max_batch=2, precision="mixed")
    s.set_graphs(False)
    launches = {}
    for name, sizes in (("uniform", (32, 32)), ("uneven", (32, 12))):
        ns = _lattices(s, *sizes)
        f = np.random.default_rng(1).integers(0, 2, sum(ns))
        launches["values", name] = _launches(s, lambda: s.eigh_logz([0, 1], _diag(ns), 4.0))
        launches["vectors", name] = _launches(s, lambda: s.free_energy_grad([0, 1], f, 2.0, 1.0, 1.0, 4.0))
        launches["chains", name] = _launches(s, lambda: s.chains_init([0, 1], f, 2.0, 1.0, 1.0, 4.0))
    s.close()
    assert launches["values", "uniform"] == launches["values", "uneven"] + 2, launches
    assert launches["vectors", "uniform"] == launches["vectors", "uneven"] + 2, launches
    assert launches["chains", "uniform"] == launches["chains", "uneven"], launches


@pytest.mark.parametrize("sizes", [(32, 32), (32, 12)])
def test_settings_hold_for_vector_solves_above_960(solver, sizes):
    """Every setting of the bucket above 960 reaches solves with eigenvectors: the two-stage reduction by its
    launches, the panel widths by their different roundings, all by the free energy's derivative."""
    s = solver
    ns = _lattices(s, *sizes)
    f = np.random.default_rng(2).integers(0, 2, sum(ns))
    grad = lambda: s.free_energy_grad([0, 1], f, 2.0, 1.0, 1.0, 4.0)
    two_stage = sizes[0] == sizes[1]
    res, launches = {}, {}
    for v in (0, 1, 2, 3):
        s.set_tuning("mixed", 1024, v)
        launches[v] = _launches(s, grad)
        res[v] = grad()["dU"]
    assert launches[0] == launches[1] == launches[2] == launches[3] - 2 * two_stage, launches
    for a in range(4):
        for b in range(a):
            if two_stage or a < 3:  # width 8 where two stages are not for every chain
                assert not np.array_equal(res[a], res[b]), (a, b)
            assert np.allclose(res[a], res[b], rtol=1e-5, atol=0), (a, b)
    if not two_stage:
        assert np.array_equal(res[3], res[1])


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("L", [5, 10, 20, 31])
def test_every_variant_of_a_solve_with_vectors(solver, L, variant):
    """Eigenvalues to 1e-9 ||H||, residuals to 1e-5 ||H|| (the mixed path's stated accuracy) with every panel width and
    the two-stage reduction."""
    from fk_mc_gb300.lattice import dense
    s = solver
    ns = _lattices(s, L, L)
    n = ns[0]
    s.set_tuning("mixed", n, variant)
    d = _diag(ns, L)
    out = s.eigh_logz([0, 1], d, 4.0, vectors=True)
    for c in range(2):
        A = dense("cubic2d", L) + np.diag(d[c * n:(c + 1) * n])
        w, X = out["evals"][c * n:(c + 1) * n], out["evecs"][c]
        norm = np.abs(A).sum(1).max()
        assert np.abs(w - np.linalg.eigvalsh(A)).max() <= 1e-9 * norm
        assert np.abs(A @ X - X * w).max() <= 1e-5 * norm


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("n,B", [(129, 153), (200, 165), (353, 170), (384, 153), (385, 3)])
def test_both_panel_widths_in_large_fp64_batches(cuda_ok, fkg_lib, n, B, variant):
    """More chains than SMs take the kernel of 4 warps up to n = 384. Bound 8 n eps ||H||_inf, as a backward-stable
    reduction and LAPACK's leave together."""
    import fk_mc_gb300
    s = fk_mc_gb300.Solver(max_n=n, max_batch=B, precision="f64", tuning=None)
    i = np.arange(n)
    H = np.zeros((n, n))
    for step in (1, 11):
        H[i, (i + step) % n] -= 1.0
        H[(i + step) % n, i] -= 1.0
    nz = H != 0
    s.set_hopping(0, np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32), np.nonzero(nz)[1].astype(np.int32),
                  H[nz])
    s.set_tuning("f64", n, variant)
    d = np.random.default_rng(n).uniform(-2, 2, (B, n))
    w = s.eigh_logz(np.zeros(B, np.int32), d.ravel(), 1.5)["evals"].reshape(B, n)
    s.close()
    for c in sorted({0, B // 2, B - 1}):
        A = H + np.diag(d[c])
        assert np.abs(w[c] - np.linalg.eigvalsh(A)).max() <= 8 * n * np.finfo(float).eps * np.abs(A).sum(1).max(), c


@pytest.mark.parametrize("n,B", [(200, 24), (216, 32), (240, 100), (256, 24), (256, 48), (256, 152)])
def test_values_reduce_no_slower_than_vectors(cuda_ok, fkg_lib, n, B):
    """The cluster kernel's size per chain is chosen by a fitted time: at every order and number of chains it must not
    be slower than the one-CTA kernel that solves with vectors keep (5 % for the clock's noise)."""
    import fk_mc_gb300
    s = fk_mc_gb300.Solver(max_n=n, max_batch=B, precision="mixed", tuning=None)
    s.set_lattice(0, "cubic1d", n)
    f, ids = np.random.default_rng(n).integers(0, 2, (B, n)), np.zeros(B, np.int32)
    ms = []
    for call in (lambda: s.eigh_logz(ids, (2.0 * f - 1.0).ravel(), 4.0),
                 lambda: s.free_energy_grad(ids, f.ravel(), 2.0, 1.0, 1.0, 4.0)):
        call()
        s.profile(True)
        for _ in range(5):
            call()
        ms.append(s.stage_time("reduce")[0])
        s.profile(False)
    s.close()
    assert ms[0] <= 1.05 * ms[1], ms
