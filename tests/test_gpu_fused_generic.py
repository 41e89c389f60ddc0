"""The fused row pass of films whose width has no register FFT gives the bits of the
unfused passes (LLG_B200_NO_FUSE=1): RK45 runs, masked relaxations, one-row films."""
import numpy as np
import pytest

from helpers import GAMMA, case, gpu_solver, holes_mask, random_m

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nx,ny,demag,holes", [(96, 20, True, False), (50, 33, True, True), (7, 5, True, False),
                                               (60, 1, True, False), (300, 16, True, True), (30, 9, False, False),
                                               (30, 320, True, False)])   # more row blocks than SMs
def test_fused_generic_rows_equal_unfused(orc, gpu, monkeypatch, nx, ny, demag, holes, prec):
    mask = holes_mask(nx, ny, [(0.1 * nx, 0.0, 0.2 * ny)]) if holes else None
    c = case(nx, ny, dmi=1e-3, k_u=5e4, demag=demag, mask=mask)
    m = random_m(orc, nx * ny, nx + ny, mask)
    out = []
    for env in (None, "LLG_B200_NO_FUSE"):
        if env:
            monkeypatch.setenv(env, "1")
        s = gpu_solver(gpu, c, prec)
        if env:
            monkeypatch.delenv(env)
        s.set_state(m)
        p = gpu.LLGParams(GAMMA, 0.1, 1e-14, (0.01, 0.0, 0.02))
        counts = s.run_rk45(p, 2, 1e-5, 0.8, 1e-19, 1e-11, n_accepted=5)
        a = s.get_state()
        s.set_state(m)
        p = gpu.LLGParams(GAMMA, 0.5, 1e-14, (0.0, 0.01, 0.0))
        rep = s.relax(p, 2, gpu.RelaxSettings.default(torque_threshold=1e-2, max_accepted_steps=20))
        out.append((counts, a, rep.accepted_steps, rep.rejected_steps, s.get_state()))
        s.close()
    assert out[0][0] == out[1][0] and out[0][2:4] == out[1][2:4]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][4], out[1][4])
