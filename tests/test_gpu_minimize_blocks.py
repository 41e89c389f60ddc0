"""The minimiser's row pass has two forms: blocks of twice the threads in launches with at
most one block per SM, else plain ones.  Both do the same operations on every cell."""
import numpy as np
import pytest

from helpers import GAMMA, case, gpu_solver, holes_mask, random_m

pytestmark = pytest.mark.gpu


def _settings(gpu):
    return gpu.MinimizeSettings.default(max_iters=24, torque_threshold=0.0, dm_stop=None, lambda0=2e-4,
                                        lambda_min=1e-5, lambda_max=1e-3, stall_iters=10 ** 9)


# rows per block: 4 at 256 cells, 8 at 128, 16 at 64; a batch of `n` films crosses 148 blocks
@pytest.mark.parametrize("nx,ny,n,masked", [(256, 256, 3, False), (128, 124, 12, True), (64, 64, 40, False)])
def test_batch_beyond_one_block_per_sm_equals_single_films(orc, gpu, nx, ny, n, masked):
    msk = holes_mask(nx, ny, [(nx // 5, ny // 6, ny // 5)]) if masked else None
    c = case(nx, ny, dmi=1e-3, k_u=2e4, mask=msk)
    b = gpu.Batch([gpu.Grid2D(nx, ny, c["dx"], c["dy"], c["dz"])] * n,
                  [gpu.Material(c["ms"], c["a_ex"], c["k_u"], c["easy"], c["dmi"], c["demag"])] * n, gpu.FP32,
                  masks=[msk] * n if masked else None)
    ms = [random_m(orc, nx * ny, 40 + i, msk) for i in range(n)]
    for i, m in enumerate(ms):
        b.set_state(i, m)
    p = gpu.LLGParams(GAMMA, 0.5, 1e-13, (0.01, 0.0, 0.02))
    reports = b.minimize([p] * n, 2, _settings(gpu))
    one = gpu_solver(gpu, c, gpu.FP32)
    for i in (0, n // 2, n - 1):
        one.set_state(ms[i])
        r = one.minimize(p, 2, _settings(gpu))
        assert r.iters == reports[i].iters
        assert np.array_equal(one.get_state(), b.get_state(i)), i
    one.close()
    b.close()


@pytest.mark.parametrize("nx,ny", [(256, 592), (256, 596), (64, 2368 // 2)])
def test_blocks_around_the_number_of_sms(orc, gpu, nx, ny):
    """148 and 149 row blocks of 4 rows, 74 of 16: the same film alone and beside a tiny one."""
    c = case(nx, ny, dmi=1e-3)
    m = random_m(orc, nx * ny, 7)
    p = gpu.LLGParams(GAMMA, 0.5, 1e-13, (0.01, 0.0, 0.02))
    one = gpu_solver(gpu, c, gpu.FP32)
    one.set_state(m)
    one.minimize(p, 2, _settings(gpu))
    g, mat = gpu.Grid2D(nx, ny, c["dx"], c["dy"], c["dz"]), gpu.Material(c["ms"], c["a_ex"], 0.0, c["easy"], c["dmi"],
                                                                         True)
    b = gpu.Batch([g, g], [mat, mat], gpu.FP32)
    b.set_state(0, m)
    b.set_state(1, m)
    b.minimize([p, p], 2, _settings(gpu))
    assert np.array_equal(one.get_state(), b.get_state(0)) and np.array_equal(b.get_state(0), b.get_state(1))
    one.close()
    b.close()
