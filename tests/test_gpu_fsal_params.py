"""FSAL reuse when the caller changes gamma or alpha between attempts.

The reference keeps the torque of an accepted step as the next k1 whatever gamma and
alpha become (llg.rs:854-867) and evaluates k1 anew after a rejected attempt; the FP64
oracle does the same.  Tolerances are those of the step tests with constant parameters:
states to 1e-12 (FP64) / 1e-6 (FP32), error norms to 1e-9 / 1e-2 relative, but not
below their rounding: four units in the last place of a unit state (RK23, a difference of
two states) or of a torque times dt (RK45).  A k1 of the wrong alpha misses by 1e-5 or more."""
import numpy as np
import pytest

from helpers import GAMMA, case, gpu_solver, oracle_solver

pytestmark = pytest.mark.gpu

ACCEPT, REJECT = 1e3, 1e-30   # error bounds that decide an attempt
BEXT = (0.01, 0.015, 0.0)
# (gamma factor, alpha, bound)
SEQUENCE = [(1.0, 0.02, ACCEPT), (1.0, 0.4, ACCEPT), (1.0, 0.9, REJECT), (1.0, 0.9, ACCEPT), (1.0, 0.1, REJECT),
            (1.0, 0.5, ACCEPT), (0.5, 0.5, REJECT), (0.25, 0.5, REJECT), (1.0, 0.5, ACCEPT), (1.0, 0.3, REJECT),
            (1.0, 0.3, REJECT), (1.0, 0.3, ACCEPT)]


def _states_agree(g, mo, prec):
    assert np.abs(g - mo).max() <= (1e-12 if prec else 1e-6)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("stepper", ["step_rk45", "step_rk23_relax"])
@pytest.mark.parametrize("nx,ny", [(20, 12), (32, 16)])
def test_single_steps(orc, gpu, nx, ny, stepper, prec):
    c = case(nx, ny, dmi=1e-3)
    o, g = oracle_solver(orc, c), gpu_solver(gpu, c, prec)
    mo = orc.init_uniform_with_noise(nx * ny, (1, 0, 0), 0.3, 8)
    g.set_state(mo)
    ulp4 = 4 * 2.0 ** (-53 if prec else -24) * (1.0 if stepper == "step_rk23_relax" else
                             GAMMA * np.linalg.norm(o.build_h_eff(mo, BEXT, 2), axis=1).max() * 1e-13)
    for i, (gam, alpha, bound) in enumerate(SEQUENCE):
        po = orc.make_params(gam * GAMMA, alpha, 1e-13, BEXT)
        pg = gpu.LLGParams(gam * GAMMA, alpha, 1e-13, BEXT)
        args = (2, bound, 0.8, 1e-19, 1e-11)
        ro = getattr(o, stepper)(mo, po, *args)
        rg = getattr(g, stepper)(pg, *args)
        assert ro[1] == rg[1] == (bound == ACCEPT), i
        assert rg[0] == pytest.approx(ro[0], rel=1e-9 if prec else 1e-2, abs=ulp4), i
        _states_agree(g.get_state(), mo, prec)


def _oracle_run(o, m, p, n, args):
    acc = rej = 0
    while acc < n:
        _, ok, _ = o.step_rk45(m, p, *args)
        acc += ok
        rej += not ok
    return acc, rej


@pytest.mark.parametrize("prec", [0, 1])
def test_run_rejects_its_first_attempts(orc, gpu, prec):
    """A run with another alpha than the run before, whose first attempts are rejected."""
    c = case(20, 12)
    o, g = oracle_solver(orc, c), gpu_solver(gpu, c, prec)
    mo = orc.init_uniform_with_noise(240, (1, 0, 0), 0.3, 9)
    g.set_state(mo)
    args = (2, 1e-6, 0.8, 1e-19, 1e-11)
    for alpha, dt, n, rejected in ((0.02, 1e-13, 4, False), (0.8, 8e-12, 12, True), (0.1, 8e-12, 3, True)):
        po = orc.make_params(GAMMA, alpha, dt, BEXT)
        pg = gpu.LLGParams(GAMMA, alpha, dt, BEXT)
        want = _oracle_run(o, mo, po, n, args)
        got = g.run_rk45(pg, *args, n_accepted=n)
        assert tuple(got[:2]) == want and (want[1] > 0) == rejected
        # the step size follows the error norm (to 1e-2 in FP32) to the power 1/5
        assert pg.dt == pytest.approx(po.dt, rel=1e-9 if prec else 1e-2)


def test_batch_run_changes_one_films_alpha(orc, gpu):
    shapes = [(20, 12), (16, 16), (9, 7)]
    cs = [case(nx, ny) for nx, ny in shapes]
    os_ = [oracle_solver(orc, c) for c in cs]
    b = gpu.Batch([gpu.Grid2D(c["nx"], c["ny"], c["dx"], c["dy"], c["dz"]) for c in cs],
                  [gpu.Material(c["ms"], c["a_ex"], c["k_u"], c["easy"], c["dmi"], c["demag"]) for c in cs], gpu.FP64)
    ms = [orc.init_uniform_with_noise(nx * ny, (1, 0, 0), 0.3, 20 + i) for i, (nx, ny) in enumerate(shapes)]
    for i, m in enumerate(ms):
        b.set_state(i, m)
    args = (2, 1e-6, 0.8, 1e-19, 1e-11)
    for alphas, dt in (((0.02, 0.02, 0.02), 1e-13), ((0.02, 0.9, 0.02), 8e-12), ((0.3, 0.9, 0.02), 8e-12)):
        pg = [gpu.LLGParams(GAMMA, a, dt, BEXT) for a in alphas]
        acc, rej, _ = b.run_rk45(pg, *args, n_accepted=5)
        for i, o in enumerate(os_):
            po = orc.make_params(GAMMA, alphas[i], dt, BEXT)
            assert (acc[i], rej[i]) == _oracle_run(o, ms[i], po, 5, args), i
            assert np.abs(b.get_state(i) - ms[i]).max() <= 1e-10, i
