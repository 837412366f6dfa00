"""Contexts of different size in several threads: a kernel's shared-memory limit belongs to the process, and no
thread's launches may lower it for another's."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(op, size, seed):
    import fk_mc_gb300
    rng = np.random.default_rng(seed)
    B = 2
    L = {"chebyshev": 12, "two-stage": (10, 24)[size]}.get(op, (6, 24)[size])
    s = fk_mc_gb300.Solver(max_n=L * L, max_batch=B, precision="mixed" if op in ("gradients", "two-stage") else "f64")
    n = s.set_lattice(0, "cubic2d", L)
    f, ids = rng.integers(0, 2, B * n), np.zeros(B, np.int32)
    d = 2.0 * f - 1.0
    if op == "chebyshev":  # the final kernel's table: 3 KB and 72 KB
        s.set_chebyshev(*((8, 16), (64, 128))[size])
        return s, lambda: s.chebyshev_logz(ids, d, 3.0)["logz"]
    if op == "two-stage":
        s.set_tuning("mixed", n, 3)
    if op in ("gradients", "two-stage"):
        return s, lambda: s.free_energy_grad(ids, f, 2.0, 1.0, 1.0, 3.0)["dU"]
    if op == "rank-one":
        w, V = np.linalg.eigh(rng.standard_normal((n, n)) + 4 * np.eye(n))
        w = np.sort(w)
        return s, lambda: s.rank1_logz(np.tile(w, (B, 1)), V[:B], np.full(B, 1.0), np.full(B, 2.0))
    return s, lambda: s.eigh_logz(ids, d, 3.0, vectors=op == "vectors")["evals"]


@pytest.mark.parametrize("op", ["chebyshev", "values", "vectors", "gradients", "two-stage", "rank-one"])
def test_other_threads_launches(cuda_ok, fkg_lib, op):
    errors = []

    def work(size, seed):
        try:
            s, call = _call(op, size, seed)
            first = np.array(call())
            for _ in range(300):
                assert np.array_equal(call(), first)
            s.close()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in ((0, 1), (1, 2), (0, 3))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
