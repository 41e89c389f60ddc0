"""The generic shared-memory transforms (films whose sides have no register FFT) at
the edges of their plans: every radix, one to several passes, prime factors, padded
and unpadded signals; and the column groups of the allocation-free entry point."""
import numpy as np
import pytest

from helpers import case, gpu_solver, oracle_solver, random_m, rel_err

pytestmark = pytest.mark.gpu
TOL = {0: 2e-5, 1: 1e-9}   # the parity tests' bounds for demag fields

# radices 2..16 alone and combined; 7 and 13 as passes of their own; 1152 in FP64 is
# too long for padded signals
SHAPES = [(6, 10), (12, 5), (48, 60), (80, 36), (144, 15), (240, 14), (7, 26), (192, 20), (250, 9)]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nx,ny", SHAPES)
def test_demag_field_of_generic_lengths(orc, gpu, nx, ny, prec):
    c = case(nx, ny)
    o, g = oracle_solver(orc, c), gpu_solver(gpu, c, prec)
    m = random_m(orc, nx * ny, 7 * nx + ny)
    g.set_state(m)
    assert rel_err(g.compute_demag_field(), o.demag_field(m)) <= TOL[prec]
    g.close()


def test_longest_double_precision_rows(orc, gpu):
    nx, ny = 1152, 2
    c = case(nx, ny)
    o, g = oracle_solver(orc, c), gpu_solver(gpu, c, 1)
    m = random_m(orc, nx * ny, 5)
    g.set_state(m)
    assert rel_err(g.compute_demag_field(), o.demag_field(m)) <= TOL[1]
    g.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (5, 9), (30, 200), (33, 300), (6, 1024)])
def test_noalloc_column_groups(orc, gpu, nx, ny):
    """nx + 1 columns in groups of 4, 2 or 1 (by ny), with every remainder."""
    import torch

    c = case(nx, ny)
    o, g = oracle_solver(orc, c), gpu_solver(gpu, c, 1)
    m = random_m(orc, nx * ny, 3)
    planes = torch.from_numpy(g.kernel_kspace()).cuda()
    md = torch.from_numpy(np.ascontiguousarray(m.T)).float().cuda()
    b = torch.zeros_like(md)
    gpu.demag_field_noalloc(nx, ny, c["ms"], md.data_ptr(), planes.data_ptr(), b.data_ptr())
    torch.cuda.synchronize()
    assert rel_err(b.double().cpu().numpy().T, o.demag_field(m)) <= TOL[0]
    g.close()
