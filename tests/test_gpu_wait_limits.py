"""Bounded waits of the tensor-core kernels: with any limit a call either reports the
timeout or returns the bits of an unlimited call.  Limits between the ones that always and
never suffice let some threads of a block give up on a copy or an MMA that others see
complete; the decision is the block's, so no result of half-built operands gets out."""
import numpy as np
import pytest

import warmstart_ref as ref

pytestmark = pytest.mark.gpu

LIMITS = [0, 1, 2, 3] + [int(4 * 1.6 ** i) for i in range(24)]
UNLIMITED = 1 << 26


def _inputs(nimg, ny, nx, seed):
    rng = np.random.default_rng(seed)
    m = rng.standard_normal((nimg, ny * nx, 3))
    m /= np.linalg.norm(m, axis=2, keepdims=True)
    t = rng.standard_normal((nimg, ny * nx, 3))
    t /= np.linalg.norm(t, axis=2, keepdims=True)
    return m, t, rng.uniform(-0.02, 0.02, (nimg, 3))


def _same_or_timeout(gpu, call, want):
    try:
        got = call()
    except gpu.LLGError as e:
        assert e.code == -3
        return False
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    return True


# several 128-cell tiles per block (pipelined form, up to 256 cells wide), few tiles, and the
# one-shot form beyond 256 cells
@pytest.mark.parametrize("nimg,ny,nx", [(2, 200, 160), (1, 9, 20), (1, 40, 300)])
def test_any_limit_reports_or_gives_the_same_bits(gpu, nimg, ny, nx):
    torch = pytest.importorskip("torch")
    params = ref.random_params(2)
    m, t, b = _inputs(nimg, ny, nx, 5)
    dev = [torch.from_numpy(np.ascontiguousarray(a.transpose(0, 2, 1), dtype=np.float32)).cuda() for a in (m, t)]
    mask = torch.ones(nimg, ny * nx, dtype=torch.uint8, device="cuda")
    bext = torch.from_numpy(b).cuda()
    tr = gpu.WarmStartTrainer(params, nimg * ny * nx)
    net = gpu.WarmStartNet(params)
    calls = [(tr, lambda: tr.gradients(nimg, ny, nx, dev[0].data_ptr(), mask.data_ptr(), bext.data_ptr(),
                                       dev[1].data_ptr())),
             (net, lambda: (net.forward(m.reshape(-1, 3), None, b, ny, nx),))]
    for obj, call in calls:
        want = call()
        done = []
        for limit in LIMITS:
            obj.set_spin_limit(limit)
            done += [_same_or_timeout(gpu, call, want) for _ in range(3)]
        assert not any(done[:3])
        obj.set_spin_limit(UNLIMITED)
        assert _same_or_timeout(gpu, call, want)
    tr.close()
    net.close()
