"""Steps that go on from each inverse Z to the next evaluation's forward Z:
several steps in one call (which hand the transform of m from step to step)
give bit for bit what single-step calls give, in a graph and without, alone
and in a batch, and track the FP64 oracle."""
import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# one row tile and less, tiles that end inside the last row, a periodic Z
# line (not chained), an odd line, the shortest line
GRIDS = [((64, 16, 1), (0, 0, 0)), ((48, 20, 3), (0, 0, 0)), ((256, 6, 2), (0, 0, 0)), ((32, 16, 1), (1, 0, 0)),
         ((25, 12, 2), (0, 0, 0)), ((50, 14, 1), (0, 0, 0)), ((2, 4, 2), (0, 0, 0))]


def config(grid, per, solver):
    return dict(grid=grid, periodic=per, cell=(4e-9, 4e-9, 4e-9), msat=1.1e6, aexch=1.5e-11, alpha=0.5, anis=1, k1=5e5,
                axis=(0, 0, 1), bext=(0.01, -0.02, 0.03), solver=solver, dt=1e-14)


@pytest.mark.parametrize("solver", ["heun", "rk4", "rk2"])
@pytest.mark.parametrize("grid,per", GRIDS)
def test_steps_in_one_call(eng, cuda, grid, per, solver):
    c = config(grid, per, solver)
    m = O.seeded_m(grid, 11, "random")
    got = {}
    for how in ("graph", "graph single", "plain", "plain single"):
        s = eng.Solver(eng.mmx_params(**c))
        s.set_m(m)
        s.use_graph("graph" in how)
        for n in [1] * 5 if "single" in how else [3, 2]:
            s.step(n)
        got[how] = s.get_m()
        s.close()
    for how in got:
        assert np.array_equal(got[how], got["plain"]), (how, np.abs(got[how] - got["plain"]).max())
    o = O.OracleSim(O.make_cfg(**c), m, bits=64)
    o.steps(5)
    assert np.abs(got["plain"] - o.m()).max() < 1e-5


@pytest.mark.parametrize("solver", ["rk23", "rkdp", "rk12", "rkck"])
@pytest.mark.parametrize("grid", [(48, 20, 3), (50, 14, 1), (25, 12, 2)])
def test_adaptive_host_and_device(eng, cuda, grid, solver):
    """Host and device controllers take the same trials; both with dt bounds
    (stage 0 is not chained) and without."""
    for max_dt in (0.0, 1e-14):
        m = O.seeded_m(grid, 12, "random")
        got = []
        for dev in (False, True):
            p = eng.mmx_params(**config(grid, (0, 0, 0), solver), maxerror=1e-2)
            p.max_dt = max_dt
            s = eng.Solver(p)
            s.set_m(m)
            s.device_control(dev)
            s.step(4)
            st = s.state()
            got.append((s.get_m(), st["time"], st["steps"]))
            s.close()
        assert got[0][2] == got[1][2] == 4
        assert abs(got[0][1] - got[1][1]) <= 1e-6 * got[0][1]
        assert np.abs(got[0][0] - got[1][0]).max() < 1e-6


def test_m_written_between_calls(eng, cuda):
    """A Runge-Kutta call starts from m itself, also when a program has
    written it through its device address since the last call."""
    import torch
    c = config((48, 20, 3), (0, 0, 0), "rk4")
    m1, m2 = O.seeded_m(c["grid"], 13, "random"), O.seeded_m(c["grid"], 14, "random")
    a, b = eng.Solver(eng.mmx_params(**c)), eng.Solver(eng.mmx_params(**c))
    a.use_graph(True)
    a.set_m(m1)
    a.step(3)
    buf = torch.from_numpy(m2).cuda()
    torch.cuda.synchronize()
    b.set_m(m2)
    # m of solver a takes m2 through its device pointer
    eng.lib().memcpy_on_gpu(ctypes.c_void_p(buf.data_ptr()), ctypes.c_void_p(a.m_device()), m2.size)
    for s in (a, b):
        s.step(2)
    assert np.array_equal(a.get_m(), b.get_m())
    a.close()
    b.close()


@pytest.mark.parametrize("solver", ["rk4", "heun"])
def test_batch_steps_in_one_call(eng, cuda, solver):
    cfgs = [config(g, p, solver) for g, p in GRIDS if g[0] in (64, 256, 32, 2)]
    cfgs.append(config((48, 24, 3), (0, 0, 0), solver))
    got = {}
    for how in ("graph", "graph single", "plain", "plain single"):
        b = eng.Batch([eng.mmx_params(**c) for c in cfgs])
        b.use_graph("graph" in how)
        for i, c in enumerate(cfgs):
            b.instances[i].set_m(O.seeded_m(c["grid"], 20 + i, "random"))
        for n in [1] * 4 if "single" in how else [3, 1]:
            b.step(n)
        got[how] = [v.get_m() for v in b.instances]
        b.close()
    for how in got:
        for x, y in zip(got[how], got["plain"]):
            assert np.array_equal(x, y), how


@pytest.mark.parametrize("how", ["graph", "plain", "profile"])
@pytest.mark.parametrize("n", [1, 2])
def test_heun_m_written_between_calls(eng, cuda, how, n):
    """A Heun call, too, starts from m itself once the program holds its
    device address; the steps of solvers whose address nobody took stay the
    same."""
    import torch
    c = config((48, 20, 3), (0, 0, 0), "heun")
    m1, m2 = O.seeded_m(c["grid"], 15, "random"), O.seeded_m(c["grid"], 16, "random")

    def solver():
        s = eng.Solver(eng.mmx_params(**c))
        s.use_graph(how == "graph")
        s.profile(2 if how == "profile" else 0)
        return s

    a, b, other = solver(), solver(), solver()
    a.set_m(m1)
    a.step(3)
    buf = torch.from_numpy(m2).cuda()
    torch.cuda.synchronize()
    for s in (b, other):
        s.set_m(m2)
    for k in range(3):
        # m of solver a takes what the program has, the state of the others at first
        if k:
            buf = torch.from_numpy(b.get_m()).cuda()
            torch.cuda.synchronize()
        eng.lib().memcpy_on_gpu(ctypes.c_void_p(buf.data_ptr()), ctypes.c_void_p(a.m_device()), buf.numel())
        for s in (a, b, other):
            s.step(n)
        if k == 0:
            assert b.m_device()  # taken after its first steps
        assert np.array_equal(a.get_m(), b.get_m())
        assert np.array_equal(a.get_m(), other.get_m())
    for s in (a, b, other):
        s.close()
