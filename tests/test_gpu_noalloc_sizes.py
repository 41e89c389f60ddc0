"""The allocation-free demag field at the sizes where its launches change: lengths up to 64
and beyond, as many blocks as SMs (148) and one more in either pass, buffers on either side of
the thresholds for 256 and 384 threads, primes, the longest sides."""
import numpy as np
import pytest

from helpers import case, gpu_solver, rel_err

pytestmark = pytest.mark.gpu


# row blocks: ceil(ny / 2), columns: nx + 1
@pytest.mark.parametrize("nx,ny", [(1, 1), (64, 64), (65, 63), (147, 12), (148, 12), (12, 296), (20, 297), (151, 480),
                                   (480, 301), (300, 797), (797, 300), (2048, 40), (40, 2048), (509, 131)])
def test_field_equals_fp64_convolution(gpu, nx, ny):
    torch = pytest.importorskip("torch")
    c = case(nx, ny)
    s = gpu_solver(gpu, c, gpu.FP32)
    k = s.kernel_kspace()   # [4][ny+1][nx+1]: xx, xy, yy, zz, real
    s.close()
    m = np.random.default_rng(nx + ny).standard_normal((3, ny, nx)).astype(np.float32)
    dm, dk = torch.from_numpy(m).cuda(), torch.from_numpy(k).cuda()
    out = torch.full_like(dm, float("nan"))
    for _ in range(2):
        gpu.demag_field_noalloc(nx, ny, c["ms"], dm.data_ptr(), dk.data_ptr(), out.data_ptr(),
                                torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    M = np.fft.rfft2(c["ms"] * m.astype(np.float64), s=(2 * ny, 2 * nx))
    full = np.concatenate([k, k[:, ny - 1:0:-1] * np.array([1, -1, 1, 1])[:, None, None]], axis=1)   # Kxy odd in ky
    B = np.stack([full[0] * M[0] + full[1] * M[1], full[1] * M[0] + full[2] * M[1], full[3] * M[2]])
    want = np.fft.irfft2(B, s=(2 * ny, 2 * nx))[:, :ny, :nx]
    assert rel_err(out.cpu().numpy(), want) <= 2e-5   # FP32 transforms, as in the field tests
