"""The pruned path of the open-boundary demag operator against the general path
(full complex transforms) and the oracle.  A kernel file whose planes are not real and
even keeps the general path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DX, DY, DZ, MS = 1e-9, 1.5e-9, 0.5e-9, 8e5


def _convolve(k, ms, m, nx, ny):
    f = np.fft.fft2(ms * m.reshape(ny, nx, 3).transpose(2, 0, 1), s=(2 * ny, 2 * nx))
    b = np.stack([k[0] * f[0] + k[1] * f[1], k[1] * f[0] + k[2] * f[1], k[3] * f[2]])
    return np.fft.ifft2(b).real[:, :ny, :nx].transpose(1, 2, 0).reshape(-1, 3)


@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 6), (5, 1), (9, 7), (20, 8), (33, 20), (48, 31), (130, 3)])
def test_open_path_equals_general_path_and_oracle(gpu, orc, tmp_path, nx, ny):
    g, og = gpu.Grid2D(nx, ny, DX, DY, DZ), orc.make_grid(nx, ny, DX, DY, DZ)
    m = orc.init_random(nx * ny, 17 + nx)
    f = tmp_path / "k.bin"
    op = gpu.DemagOp(g, 0, 0, cache_path=f)
    b, k = op.field(MS, m), op.kspace()
    op.close()
    bo = orc.demag_field_pbc(og, MS, 0, 0, m)
    scale = np.abs(bo).max()
    assert np.abs(b - bo).max() <= 1e-10 * scale
    # the same planes from the file take the same path
    op = gpu.DemagOp(g, 0, 0, cache_path=f)
    assert op.loaded and np.array_equal(op.field(MS, m), b) and np.array_equal(op.kspace(), k)
    op.close()
    # one imaginary part far above round-off: the planes are used as they are
    raw = bytearray(f.read_bytes())
    data = np.frombuffer(bytes(raw[68:]), "<f8").copy()
    data[1] += 1e-3 * np.abs(data).max()
    f.write_bytes(bytes(raw[:68]) + data.tobytes())
    op = gpu.DemagOp(g, 0, 0, cache_path=f)
    assert op.loaded
    k2 = data.view(np.complex128).reshape(4, 2 * ny, 2 * nx)
    bg, want = op.field(MS, m), _convolve(k2, MS, m, nx, ny)
    assert np.abs(bg - want).max() <= 1e-10 * np.abs(want).max()
    op.close()


def test_asymmetric_real_planes_keep_the_general_path(gpu, orc, tmp_path):
    nx, ny = 12, 10
    g = gpu.Grid2D(nx, ny, DX, DY, DZ)
    f = tmp_path / "k.bin"
    gpu.DemagOp(g, 0, 0, cache_path=f).close()
    raw = f.read_bytes()
    data = np.frombuffer(raw[68:], "<f8").copy()
    k = data.view(np.complex128).reshape(4, 2 * ny, 2 * nx)
    k[0, 3, 4] *= 1.5
    f.write_bytes(raw[:68] + data.tobytes())
    m = orc.init_random(nx * ny, 2)
    op = gpu.DemagOp(g, 0, 0, cache_path=f)
    want = _convolve(k, MS, m, nx, ny)
    assert np.abs(op.field(MS, m) - want).max() <= 1e-10 * np.abs(want).max()
    op.close()


@pytest.mark.parametrize("nx,ny", [(3, 300), (2, 1536), (5, 2048), (600, 7), (2048, 2)])
def test_open_path_long_columns_and_rows(gpu, orc, nx, ny):
    """Column blocks of 128 to 512 threads, rows of several rounds of the grouped loads."""
    m = orc.init_random(nx * ny, 5 + nx)
    op = gpu.DemagOp(gpu.Grid2D(nx, ny, DX, DY, DZ), 0, 0)
    want = _convolve(op.kspace().reshape(4, 2 * ny, 2 * nx), MS, m, nx, ny)
    assert np.abs(op.field(MS, m) - want).max() <= 1e-10 * np.abs(want).max()
    op.close()
