"""Device memory of FP64 solves with eigenvectors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_memory_of_a_solve_with_vectors(cuda_ok, fkg_lib):
    """Matrix-sized buffers of an FP64 solve with eigenvectors: the reflectors, the vectors, six of inverse iteration.
    The reduction's tiles beyond shared memory take no ninth one."""
    import torch
    import fk_mc_gb300
    n, B = 1024, 32
    s = fk_mc_gb300.Solver(max_n=n, max_batch=B, precision="f64")
    s.set_lattice(0, "cubic2d", 32)
    d = np.random.default_rng(1).uniform(-2, 2, B * n)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    s.measure_ipr(np.zeros(B, np.int32), d, 2.0)
    used = free - torch.cuda.mem_get_info()[0]
    s.close()
    assert used <= 8.5 * 8 * B * n * n, used / (8 * B * n * n)
