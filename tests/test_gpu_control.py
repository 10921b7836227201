"""The device dt controller against the host one where the two meet: host
steps before the switch, torque-based dt bounds, rejected trials, a field
changed between trials."""
import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

GRID = (48, 20, 3)


def params(eng, solver, dt=1e-14, maxerror=1e-2, faithful=1, **set_):
    p = eng.mmx_params(grid=GRID, cell=(4e-9, 4e-9, 4e-9), msat=1.1e6, aexch=1.5e-11, alpha=0.5, anis=1, k1=5e5,
                       axis=(0, 0, 1), bext=(0.01, -0.02, 0.03), solver=solver, dt=dt, maxerror=maxerror,
                       faithful=faithful)
    for k, v in set_.items():
        setattr(p, k, v)
    return p


@pytest.mark.parametrize("max_dt", [0.0, 1e-14])
@pytest.mark.parametrize("solver", ["rk23", "rkdp", "rk12", "rkck"])
def test_switch_after_host_steps(eng, cuda, solver, max_dt):
    """Host steps, then a run: the controllers write the same rows, the first
    one with the torque of the last host step, and take the same steps; the
    switch keeps the torque and the error."""
    out = []
    for dev in (False, True):
        s = eng.Solver(params(eng, solver, max_dt=max_dt))
        s.set_m(O.seeded_m(GRID, 31, "random"))
        s.step(3)
        before = s.state()
        assert before["torque"] > 0
        if dev:
            # on, off and on again: nothing is lost on the way
            for on in (True, False, True) if solver in ("rk12", "rkck") else (True,):
                s.device_control(on)
                assert s.state() == before
        rows = s.run(4.5e-14, 1e-15)
        assert rows[0, 4] == np.float32(before["torque"])
        out.append((rows, s.state(), s.get_m()))
        s.close()
    (ra, sa, ma), (rb, sb, mb) = out
    assert sa["steps"] == sb["steps"] and ra.shape == rb.shape and len(ra) >= (4 if max_dt else 1)
    assert np.abs(ra - rb).max() <= 1e-6 * np.abs(ra).max()
    assert abs(sa["time"] - sb["time"]) <= 1e-6 * sa["time"]
    assert np.abs(ma - mb).max() < 1e-6


# a step's largest change dm = dt max|k0| is some 0.01 at dt = 1e-14 s here
@pytest.mark.parametrize("bounds", [dict(max_dm=2e-3), dict(min_dm=3e-2), dict(min_dt=1.5e-14), dict(max_dt=4e-15),
                                    dict(min_dm=1e-3, max_dm=4e-3, min_dt=1e-17, max_dt=5e-15)])
@pytest.mark.parametrize("solver", ["rk23", "rkdp", "rk12", "rkck"])
def test_dt_bounds(eng, cuda, solver, bounds):
    """min_dm, max_dm, min_dt and max_dt give both controllers the same dt,
    another one than without them."""
    out = []
    for dev, b in ((False, {}), (False, bounds), (True, bounds)):
        s = eng.Solver(params(eng, solver, **b))
        s.set_m(O.seeded_m(GRID, 32, "random"))
        s.device_control(dev)
        s.step(3)
        out.append((s.state(), s.get_m()))
        s.close()
    (free, _), (h, mh), (d, md) = out
    assert h["steps"] == d["steps"] == 3
    assert abs(h["time"] - free["time"]) > 1e-2 * free["time"]
    for k in ("time", "dt", "torque"):
        assert abs(h[k] - d[k]) <= 1e-6 * abs(h[k]), k
    assert np.abs(mh - md).max() < 1e-6


@pytest.mark.parametrize("max_dm", [0.0, 0.8])
@pytest.mark.parametrize("faithful", [0, 1])
@pytest.mark.parametrize("solver", ["rk23", "rkdp", "rk12", "rkck"])
def test_rejected_trials(eng, cuda, solver, faithful, max_dm):
    """A start dt that is far too large: the first trials are rejected, m
    stays, and both controllers end at the same accepted steps.  faithful
    restarts an FSAL trial from the rejected one's last torque."""
    kw = dict(dt=8e-13, maxerror=1e-5, faithful=faithful, max_dm=max_dm)
    m0 = O.seeded_m(GRID, 33, "random")
    h = eng.Solver(params(eng, solver, **kw))
    h.set_m(m0)
    h.step(3)
    d = eng.Solver(params(eng, solver, **kw))
    d.set_m(m0)
    d.device_control(True)
    trials = 0
    while d.state()["steps"] < 3 and trials < 40:
        d.step(1)
        trials += 1
        if d.state()["steps"] == 0:
            assert np.array_equal(d.get_m(), m0)
    sh, sd = h.state(), d.state()
    assert sh["steps"] == sd["steps"] == 3 and trials > 3
    for k in ("time", "dt", "torque"):
        assert abs(sh[k] - sd[k]) <= 1e-5 * abs(sh[k]), k
    assert np.abs(h.get_m() - d.get_m()).max() < 1e-6
    h.close()
    d.close()


def test_field_changed_between_trials(eng, cuda):
    """set_hext holds for the trials, the run and the profiled steps that
    follow it, whatever graph was captured before it."""
    h2 = (ctypes.c_float * 3)(0.4, -0.3, 0.2)
    m0 = O.seeded_m(GRID, 34, "random")

    def pair(solver, prepare, advance, change=True, **kw):
        s = eng.Solver(params(eng, solver, **kw))
        s.set_m(m0)
        prepare(s)
        advance(s)
        if change:
            assert eng.lib().mmx_solver_set_hext(s.h, h2) == 0
        advance(s)
        m = s.get_m()
        # and from a new m (an FSAL solver's first trial)
        s.set_m(m0)
        advance(s)
        m = np.concatenate([m, s.get_m()])
        s.close()
        return m

    def trials(s):
        s.step(3)

    def run(s):
        s.run(2.5e-14, 1e-15)

    for solver in ("rk23", "rk12"):
        for adv in (trials, run):
            want = pair(solver, lambda s: s.device_control(False), adv, max_dt=1e-14)
            got = pair(solver, lambda s: s.device_control(True), adv, max_dt=1e-14)
            old = pair(solver, lambda s: s.device_control(False), adv, change=False, max_dt=1e-14)
            assert np.abs(want - old).max() > 1e-4
            assert np.abs(got - want).max() < 1e-6, (solver, adv.__name__)
    for solver in ("heun", "rk4"):
        want = pair(solver, lambda s: None, trials, maxerror=0.0)
        for prepare in (lambda s: s.use_graph(True), lambda s: s.profile(2)):
            assert np.array_equal(pair(solver, prepare, trials, maxerror=0.0), want), solver
