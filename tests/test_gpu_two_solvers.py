"""Several live solvers: the shared-memory limits of the kernels are state of the process,
so creating a solver of shorter films must leave the ones of longer films usable."""
import numpy as np
import pytest

from helpers import GAMMA, case, gpu_solver, oracle_solver, random_m, rel_err

pytestmark = pytest.mark.gpu

BEXT = (0.01, 0.0, -0.02)


# (long film, short film): generic row and column kernels above the default 48 KiB of shared
# memory (12 buffers of the length) beside generic ones below it, and beside power-of-two films
# that set no generic size at all; FP64 from 229 cells on, FP32 from 483
@pytest.mark.parametrize("long_shape,short_shape,prec", [((250, 9), (24, 10), 1), ((9, 250), (16, 16), 1),
                                                         ((500, 6), (24, 10), 0), ((6, 520), (32, 32), 0),
                                                         ((1000, 3), (250, 125), 0)])
def test_longer_film_first(orc, gpu, long_shape, short_shape, prec):
    c = case(*long_shape)
    o, a = oracle_solver(orc, c), gpu_solver(gpu, c, prec)
    b = gpu_solver(gpu, case(*short_shape), prec)
    m = random_m(orc, long_shape[0] * long_shape[1], 3)
    a.set_state(m)
    b.set_state(random_m(orc, short_shape[0] * short_shape[1], 4))
    p = gpu.LLGParams(GAMMA, 0.1, 1e-14, BEXT)
    b.step_rk45(p, 2, 1e-5, 0.8, 1e-19, 1e-11)
    # the field of the step tests' tolerance, then steps (the fused row pass)
    assert rel_err(a.build_h_eff(gpu.LLGParams(GAMMA, 0.1, 1e-14, BEXT), 2), o.build_h_eff(m, BEXT, 2)) <= (
        1e-9 if prec else 2e-5)
    po = orc.make_params(GAMMA, 0.1, 1e-14, BEXT)
    pg = gpu.LLGParams(GAMMA, 0.1, 1e-14, BEXT)
    for _ in range(2):
        ro = o.step_rk45(m, po, 2, 1e-5, 0.8, 1e-19, 1e-11)
        rg = a.step_rk45(pg, 2, 1e-5, 0.8, 1e-19, 1e-11)
        assert ro[1] == rg[1]
        pg.dt = po.dt
    assert np.abs(a.get_state() - m).max() <= (1e-12 if prec else 1e-6)
    a.close()
    b.close()


def test_demag_operators_of_two_lengths(gpu):
    """The strided transforms of the demag operator: the longer operator, used after a shorter one."""
    mat_ms = 8e5
    big, small = gpu.Grid2D(700, 3, 4e-9, 4e-9, 3e-9), gpu.Grid2D(20, 5, 4e-9, 4e-9, 3e-9)
    rng = np.random.default_rng(3)
    m = rng.standard_normal((2100, 3))
    a = gpu.DemagOp(big, 1, 0)
    first = a.field(mat_ms, m)
    b = gpu.DemagOp(small, 1, 0)
    b.field(mat_ms, rng.standard_normal((100, 3)))
    assert np.array_equal(a.field(mat_ms, m), first)
