"""The longest compiled lines on every axis, whose tile and twiddle table
together pass 48 KB of shared memory (columns of 2048 and 4096 points, forward
rows of 3072 and 4096, inverse rows of 1536 and more), against the FP64
oracle."""
import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def config(grid, solver="heun"):
    return dict(grid=grid, cell=(4e-9, 4e-9, 4e-9), msat=1.1e6, aexch=1.5e-11, alpha=0.5, anis=1, k1=5e5, axis=(0, 0, 1),
                bext=(0.01, -0.02, 0.03), solver=solver, dt=1e-14)


# user (nx, ny, nz): Z lines of nx points, Y of 2 ny, X of 2 nz
@pytest.mark.parametrize("grid", [(4, 1024, 1), (4, 1024, 2), (4, 2048, 1), (4, 2048, 2), (1536, 4, 1), (3072, 2, 1),
                                  (4096, 2, 1), (2, 2, 1024), (2, 2, 1536), (2, 2, 2048)])
def test_field_and_steps(eng, cuda, grid):
    """The field within 2e-6 of its norm, as for every transform of a few
    stages; Heun and RK4 steps within 1e-5."""
    import torch
    m = O.seeded_m(grid, 41, "random")
    s = eng.Solver(eng.mmx_params(**config(grid)))
    d, h = torch.from_numpy(m).cuda(), torch.empty(m.shape, device="cuda")
    s.field(d.data_ptr(), h.data_ptr())
    want = O.OracleSim(O.make_cfg(**config(grid)), m, bits=64).heff(m)
    got = h.cpu().numpy().astype(np.float64)
    s.close()
    assert np.linalg.norm(got - want) < 2e-6 * np.linalg.norm(want)
    for solver in ("heun", "rk4"):
        s = eng.Solver(eng.mmx_params(**config(grid, solver)))
        s.set_m(m)
        s.step(2)
        o = O.OracleSim(O.make_cfg(**config(grid, solver)), m, bits=64)
        o.steps(2)
        assert np.abs(s.get_m() - o.m()).max() < 1e-5, solver
        s.close()


def test_batch(eng, cuda):
    """The batch's passes of the same lines: each instance as alone."""
    cfgs = [config(g, "rk4") for g in [(4, 1024, 2), (4, 2048, 2), (1536, 4, 1), (3072, 2, 1), (4096, 2, 1),
                                       (2, 2, 2048), (4, 2048, 1)]]
    b = eng.Batch([eng.mmx_params(**c) for c in cfgs])
    for i, c in enumerate(cfgs):
        b.instances[i].set_m(O.seeded_m(c["grid"], 50 + i, "random"))
    b.step(2)
    for i, c in enumerate(cfgs):
        s = eng.Solver(eng.mmx_params(**c))
        s.set_m(O.seeded_m(c["grid"], 50 + i, "random"))
        s.step(2)
        assert np.array_equal(s.get_m(), b.instances[i].get_m()), c["grid"]
        s.close()
    b.close()


@pytest.mark.parametrize("size,padded", [((1, 1024, 4), (1, 2048, 8)), ((1, 2048, 4), (1, 4096, 8)),
                                         ((2048, 2, 4), (4096, 4, 8)), ((1, 2, 3072), (1, 4, 6144)),
                                         ((1, 2, 4096), (1, 4, 8192))])
def test_plan_round_trip(eng, cuda, size, padded):
    """The drop-in plan of the same lines against numpy, forward and back."""
    import torch
    L = eng.lib()
    a = np.random.default_rng(6).standard_normal(size).astype(np.float32)
    plan = L.new_gpuFFT3dPlan_padded((ctypes.c_int * 3)(*size), (ctypes.c_int * 3)(*padded))
    x = torch.from_numpy(a).cuda()
    spec = torch.zeros((padded[0], padded[1], padded[2] + 2), device="cuda")
    back = torch.zeros(size, device="cuda")
    torch.cuda.synchronize()
    L.gpuFFT3dPlan_forward(plan, x.data_ptr(), spec.data_ptr())
    torch.cuda.synchronize()
    got = spec.cpu().numpy().astype(np.float64).view(np.complex128)[..., :padded[2] // 2 + 1]
    want = np.fft.rfftn(a.astype(np.float64), s=padded, axes=(0, 1, 2))
    assert np.linalg.norm(got - want) < 2e-6 * np.linalg.norm(want)
    L.gpuFFT3dPlan_inverse(plan, spec.data_ptr(), back.data_ptr())
    torch.cuda.synchronize()
    assert np.linalg.norm(back.cpu().numpy() / float(np.prod(padded)) - a) < 2e-6 * np.linalg.norm(a)
    L.delete_gpuFFT3dPlan(plan)
