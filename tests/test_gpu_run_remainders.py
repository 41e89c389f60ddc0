"""Runs whose number of attempts is no multiple of a graph's: the left-over attempts run as
plain kernels the first time and from a graph of one attempt afterwards, with the same bits."""
import numpy as np
import pytest

from helpers import GAMMA, case, gpu_solver

pytestmark = pytest.mark.gpu

ARGS = (2, 1e-5, 0.8, 1e-19, 2e-13)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("chunks", [(1, 1, 1, 8, 3, 7), (11, 10), (21,), (3, 5, 9, 4)])
def test_chunked_run_equals_single_steps(orc, gpu, chunks, prec):
    c = case(32, 24)
    m = orc.init_uniform_with_noise(32 * 24, (1, 0, 0), 0.1, 5)
    a, b = gpu_solver(gpu, c, prec), gpu_solver(gpu, c, prec)
    pa, pb = (gpu.LLGParams(GAMMA, 0.02, 1e-13, (0.02, 0.0, 0.0)) for _ in range(2))
    a.set_state(m)
    b.set_state(m)
    for n in chunks:
        acc, _, _ = a.run_rk45(pa, *ARGS, n_accepted=n)
        assert acc == n
    done = 0
    while done < sum(chunks):
        done += b.step_rk45(pb, *ARGS)[1]
    assert np.array_equal(a.get_state(), b.get_state()) and pa.dt == pb.dt
