"""Line lengths without compiled kernels (products of 2, 3, 5 and 7): the
run-time radix plans on every axis, against the FP64 oracle."""
import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# user (nx, ny, nz); Z lines of nx points, Y of 2 ny, X of 2 nz:
# one, two and three stages, radices 5 to 25, odd lines, one-point Z lines
# (periodic), a tile wider than the columns, rows that end inside a tile
GRIDS = [((10, 5, 1), (0, 0, 0)), ((25, 10, 5), (0, 0, 0)), ((250, 50, 10), (0, 0, 0)), ((49, 45, 7), (0, 0, 0)),
         ((2, 15, 2), (1, 0, 0)), ((70, 20, 9), (1, 1, 0)), ((40, 98, 1), (0, 1, 0)), ((360, 105, 1), (0, 0, 0)),
         ((9, 250, 1), (0, 0, 0)), ((14, 6, 30), (0, 0, 1)), ((1029, 4, 1), (0, 0, 0)), ((20, 540, 1), (0, 0, 0))]


def config(grid, per):
    return dict(grid=grid, periodic=per, cell=(4e-9, 4e-9, 4e-9), msat=1.1e6, aexch=1.5e-11, alpha=0.5, anis=1, k1=5e5,
                axis=(0, 0, 1), bext=(0.01, -0.02, 0.03))


@pytest.mark.parametrize("grid,per", GRIDS)
def test_field(eng, cuda, grid, per):
    """float32 transforms of a few stages: 2e-6 of the field's norm, as for
    the compiled lengths."""
    import torch
    c = config(grid, per)
    m = O.seeded_m(grid, 3, "random")
    s = eng.Solver(eng.mmx_params(**c))
    d, h = torch.from_numpy(m).cuda(), torch.empty(m.shape, device="cuda")
    s.field(d.data_ptr(), h.data_ptr())
    want = O.OracleSim(O.make_cfg(**c), m, bits=64).heff(m)
    got = h.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - want) < 2e-6 * np.linalg.norm(want)
    s.close()


@pytest.mark.parametrize("size,padded", [((3, 5, 10), (6, 10, 20)), ((4, 9, 49), (8, 18, 98)), ((1, 7, 50), (1, 14, 50)),
                                         ((5, 125, 6), (5, 250, 12)), ((2, 3, 1500), (4, 6, 3000)),
                                         ((1, 4, 8), (1, 6000, 16))])
def test_plan_round_trip(eng, cuda, size, padded):
    """The drop-in plan against numpy, forward and back."""
    import torch
    L = eng.lib()
    g = np.random.default_rng(4)
    a = g.standard_normal(size).astype(np.float32)
    s3, p3 = (ctypes.c_int * 3)(*size), (ctypes.c_int * 3)(*padded)
    plan = L.new_gpuFFT3dPlan_padded(s3, p3)
    x = torch.from_numpy(a).cuda()
    spec = torch.zeros((padded[0], padded[1], padded[2] + 2), device="cuda")
    back = torch.zeros(size, device="cuda")
    torch.cuda.synchronize()
    L.gpuFFT3dPlan_forward(plan, x.data_ptr(), spec.data_ptr())
    torch.cuda.synchronize()
    got = spec.cpu().numpy().astype(np.float64).view(np.complex128)[..., :padded[2] // 2 + 1]
    want = np.fft.rfftn(a.astype(np.float64), s=padded)
    assert np.linalg.norm(got - want) < 2e-6 * np.linalg.norm(want)
    L.gpuFFT3dPlan_inverse(plan, spec.data_ptr(), back.data_ptr())
    torch.cuda.synchronize()
    n = float(np.prod(padded))
    assert np.linalg.norm(back.cpu().numpy() / n - a) < 2e-6 * np.linalg.norm(a)
    L.delete_gpuFFT3dPlan(plan)
