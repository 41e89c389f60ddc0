"""Periodic demag field against numpy FFTs of the operator's own planes, at sizes that take
every number of signals per block (1, 2, 4, 8) with full and partly filled last blocks, the
few-block form, and lengths with and without register butterflies.  An FP64 transform of
length up to 2000 errs by a few ulp times log2 of its length: 1e-13 of the largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (nx, ny): rows are 3 ny signals of length nx, columns 3 nx of length ny
SHAPES = [(1, 3), (16, 16), (97, 101), (301, 251), (130, 509), (40, 1001), (1999, 7), (512, 384)]


@pytest.mark.parametrize("pbc", [(1, 1), (0, 2)])
@pytest.mark.parametrize("nx,ny", SHAPES)
def test_field_equals_numpy_convolution(gpu, nx, ny, pbc):
    op = gpu.DemagOp(gpu.Grid2D(nx, ny, 4e-9, 4e-9, 3e-9), *pbc)
    k = op.kspace()   # [4][py][px] complex: xx, xy, yy, zz
    py, px = k.shape[1:]
    m = np.random.default_rng(nx + ny).standard_normal((ny, nx, 3))
    ms = 8e5
    M = np.fft.fft2(np.pad(ms * m, ((0, py - ny), (0, px - nx), (0, 0))), axes=(0, 1))
    B = np.stack([k[0] * M[..., 0] + k[1] * M[..., 1], k[1] * M[..., 0] + k[2] * M[..., 1], k[3] * M[..., 2]], axis=-1)
    want = np.fft.ifft2(B, axes=(0, 1)).real[:ny, :nx]
    got = op.field(ms, m.reshape(-1, 3)).reshape(ny, nx, 3)
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
    op.close()
