"""Relaxation with each field mask.  With the full mask energy and torque requests share one
evaluation; with the others the torque has a pass of its own (local terms only) beside the
energy's, which always includes the demag field of a film that has one."""
import numpy as np
import pytest

from helpers import GAMMA, case, gpu_solver, holes_mask, oracle_solver, random_m

pytestmark = pytest.mark.gpu

BEXT = (0.03, 0.0, 0.01)


def _settings(mod, orc_side, **kw):
    kw = dict(dict(torque_threshold=1e-3, max_accepted_steps=400), **kw)
    return mod.default_relax_settings(**kw) if orc_side else mod.RelaxSettings.default(**kw)


def _pair(orc, gpu, fmask, prec, **kw):
    c = case(20, 12, dmi=1e-3, k_u=2e4)
    o, g = oracle_solver(orc, c), gpu_solver(gpu, c, prec)
    mo = orc.init_uniform_with_noise(240, (1, 0, 0.2), 0.2, 4)
    g.set_state(mo)
    ro = o.relax(mo, orc.make_params(GAMMA, 0.5, 1e-13, BEXT), fmask, _settings(orc, True, **kw))
    rg = g.relax(gpu.LLGParams(GAMMA, 0.5, 1e-13, BEXT), fmask, _settings(gpu, False, **kw))
    return ro, rg, np.abs(g.get_state() - mo).max()


@pytest.mark.parametrize("fmask", [0, 1, 2])
def test_single_film_matches_oracle(orc, gpu, fmask):
    ro, rg, err = _pair(orc, gpu, fmask, gpu.FP64)
    assert rg.stop_reason == ro.stop_reason
    # round-off may flip one decision near a bound; the counts then differ by a little
    same = (rg.accepted_steps, rg.rejected_steps) == (ro.accepted_steps, ro.rejected_steps)
    assert abs(rg.accepted_steps - ro.accepted_steps) <= max(3, ro.accepted_steps // 100)
    assert abs(rg.rejected_steps - ro.rejected_steps) <= 2
    assert abs(rg.torque_checks - ro.torque_checks) <= 2
    assert err < (1e-9 if same else 1e-3)


@pytest.mark.parametrize("fmask", [0, 1, 2])
def test_first_steps_in_fp32_match_oracle(orc, gpu, fmask):
    """12 steps with an energy every 5 and a torque every 3: the error norms agree to 1e-2 and
    so the step sizes (to the power 1/3) to some 1e-3, of a way of about 1e-2 per step."""
    ro, rg, err = _pair(orc, gpu, fmask, gpu.FP32, max_accepted_steps=12, energy_stride=5, torque_check_stride=3)
    assert (rg.accepted_steps, rg.rejected_steps) == (ro.accepted_steps, ro.rejected_steps)
    assert (rg.stop_reason, rg.torque_checks) == (ro.stop_reason, ro.torque_checks)
    assert err <= 1e-3


@pytest.mark.parametrize("prec", [1, 0])
@pytest.mark.parametrize("fmask", [0, 1])
def test_batch_with_both_requests_in_an_iteration(orc, gpu, fmask, prec):
    """Films of different strides and histories, some of which ask for an energy while others
    ask for a torque, relax as they do alone."""
    cases = [case(20, 12, dmi=1e-3), case(32, 16, k_u=5e4), case(20, 12, demag=False),
             case(16, 16, mask=holes_mask(16, 16, [(3, 2, 3)]))]
    gs = [gpu.Grid2D(c["nx"], c["ny"], c["dx"], c["dy"], c["dz"]) for c in cases]
    ma = [gpu.Material(c["ms"], c["a_ex"], c["k_u"], c["easy"], c["dmi"], c["demag"]) for c in cases]
    b = gpu.Batch(gs, ma, prec, masks=[c["mask"] for c in cases])
    ms = [random_m(orc, c["nx"] * c["ny"], 60 + i, c["mask"]) for i, c in enumerate(cases)]
    for i, m in enumerate(ms):
        b.set_state(i, m)
    p = lambda: gpu.LLGParams(GAMMA, 0.5, 1e-13, BEXT)  # noqa: E731
    kw = dict(max_accepted_steps=150, energy_stride=5, torque_check_stride=3)
    reps = b.relax([p() for _ in cases], fmask, _settings(gpu, False, **kw))
    for i, c in enumerate(cases):
        s = gpu_solver(gpu, c, prec)
        s.set_state(ms[i])
        r = s.relax(p(), fmask, _settings(gpu, False, **kw))
        assert (r.stop_reason, r.accepted_steps, r.rejected_steps, r.torque_checks) == (
            reps[i].stop_reason, reps[i].accepted_steps, reps[i].rejected_steps, reps[i].torque_checks), i
        assert np.array_equal(s.get_state(), b.get_state(i)), i
        s.close()
    b.close()


def test_largest_step_limit(gpu, orc):
    """max_accepted_steps of the largest integer relaxes as a large limit does."""
    c = case(16, 12)
    m = orc.init_uniform_with_noise(192, (1, 0, 0), 0.1, 3)
    out = []
    for limit in (10 ** 6, 2 ** 63 - 1):
        g = gpu_solver(gpu, c, gpu.FP64)
        g.set_state(m)
        r = g.relax(gpu.LLGParams(GAMMA, 0.5, 1e-13, BEXT), 2, _settings(gpu, False, max_accepted_steps=limit))
        out.append(((r.stop_reason, r.accepted_steps, r.rejected_steps, r.torque_checks), g.get_state()))
        g.close()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
