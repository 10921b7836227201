"""The calls that a program using the LLG engine spends its time in, with the
inputs such a program has in hand before each.

Every case is a pass through the package's public entry points:

  step     Solver.step (one CUDA graph per step) and Solver.avg_m, the loop of a
           simulation with a fixed time step that logs <m>
  trials   the adaptive RK solvers with the dt controller on the device
           (Solver.device_control), n trials and <m>
  run      Solver.run: a stretch of simulated time with a table row every period
  field    Solver.field: one effective-field evaluation of a device array
  batch    Batch.step: many uneven instances advanced together
  serve    Server: requests submitted, pumped to completion and read back
  dropin   DriverSim: the call sequence of the unchanged Go front end over the
           libgpukern primitives, the magnetisation read back at the end

The adaptive cases set max_dt, as a program does that wants evenly spaced rows:
the controller then ends at the same dt whatever the last bits of the error
estimate are, so that two builds stay comparable.

Axes: a case's nx, ny, nz are the user's; arrays are internal, [3][nz][ny][nx].
"""
import ctypes
import importlib
import math

import numpy as np
import torch

# Materials of the standard configurations: a permalloy film, a cube with
# uniaxial anisotropy along the user's z, and the film of the vortex problem.
MATERIALS = {
    "film": dict(cell=(3.90625e-9, 3.90625e-9, 3e-9), msat=8.0e5, aexch=1.3e-11, alpha=0.02,
                 bext=(-24.6e-3, 4.3e-3, 0.0)),
    "cube": dict(cell=(4e-9, 4e-9, 4e-9), msat=1.1e6, aexch=1.5e-11, alpha=0.5, anis=1, k1=5e5, axis=(0, 0, 1)),
    "vortex": dict(cell=(2e-9, 2e-9, 2e-9), msat=8.6e5, aexch=1.3e-11, alpha=0.1),
}


def listed():
    return [
        # the smallest film anyone runs: launches and their gaps are the time
        dict(name="film-64x16-heun", kind="step", nx=64, ny=16, nz=1, material="film", solver="heun", dt=2e-14, n=1),
        # the standard switching problem, 25 table rows in one call
        dict(name="film-128x32-rk23-run", kind="run", nx=128, ny=32, nz=1, material="film", solver="rk23", dt=1e-13,
             maxerror=1e-5, n=50),
        # the vortex film with FP32 transforms and with the tensor-core form
        dict(name="film-512x512-rk23", kind="trials", nx=512, ny=512, nz=1, material="vortex", solver="rk23", dt=1e-14,
             maxerror=1e-4, n=8),
        dict(name="film-512x512-rk23-bf16x3", kind="trials", nx=512, ny=512, nz=1, material="vortex", solver="rk23",
             dt=1e-14, maxerror=1e-4, n=8, precision=1),
        # a large film, the upper end of the published table's sizes
        dict(name="film-2048x1536-heun", kind="step", nx=2048, ny=1536, nz=1, material="film", solver="heun", dt=2e-14,
             n=4),
        # a cube of the same table with the classical fourth-order solver
        dict(name="cube-64-rk4", kind="step", nx=64, ny=64, nz=64, material="cube", solver="rk4", dt=1e-14, n=4),
        # the headline grid
        dict(name="grid-256x256x32-heun", kind="step", nx=256, ny=256, nz=32, material="cube", solver="heun", dt=1e-14,
             n=8),
        # sizes that are no power of two, with the seven-stage solver
        dict(name="grid-250x100x10-rkdp", kind="trials", nx=250, ny=100, nz=10, material="cube", solver="rkdp",
             dt=1e-14, maxerror=1e-4, n=4),
        # one field evaluation, periodic along the user's y
        dict(name="field-192x128x24-periodic", kind="field", nx=192, ny=128, nz=24, material="cube", per=1),
        # many small uneven solves at once
        dict(name="batch-24-rk4", kind="batch", count=24, draw_seed=4, n=4),
        # the serving loop: relaxations and sweeps, admission to result
        dict(name="serve-10", kind="serve", count=10, draw_seed=5, points=3, cap=60),
        # the Go front end's call sequence
        dict(name="dropin-128x128x16-heun", kind="dropin", nx=128, ny=128, nz=16, material="cube", solver="heun",
             dt=1e-14, n=10),
    ]


def smooth(rng, lo, hi, odd=0.5):
    """A grid size in [lo, hi], spread over its logarithm: 2^a or 3*2^a, or
    (with probability 'odd') any even product of 2, 3, 5 and 7."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    anysize = rng.random() < odd
    best = None
    for s in range(lo, hi + 1):
        m = s
        for p in (2, 3) + ((5, 7) if anysize else ()):
            while m % p == 0:
                m //= p
        if m != 1 or (not anysize and s % 9 == 0) or (anysize and s % 2):
            continue
        if best is None or abs(math.log(s / v)) < abs(math.log(best / v)):
            best = s
    return best or lo


def draw(rng):
    kind = rng.choice(["step", "step", "step", "trials", "trials", "run", "field", "field", "batch", "serve",
                       "dropin", "precision"])
    if kind == "precision":
        return dict(kind="trials", nx=smooth(rng, 16, 512), ny=512, nz=1, material="vortex", solver="rk23", dt=1e-14,
                    maxerror=1e-4, n=rng.randint(2, 8), precision=1)
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(3, 24), draw_seed=rng.randint(0, 10 ** 6), n=rng.randint(1, 4))
    if kind == "serve":
        return dict(kind="serve", count=rng.randint(2, 4), draw_seed=rng.randint(0, 10 ** 6),
                    points=rng.randint(2, 3), cap=20 * rng.randint(1, 2))
    flat = kind == "run" or rng.random() < 0.5
    c = dict(kind=kind)
    if flat:
        # above 512 cells: 2^k and 3*2^k
        hi = 256 if kind == "run" else 512
        c.update(nx=smooth(rng, 16, hi), ny=smooth(rng, 16, hi), nz=1, material=rng.choice(["film", "vortex"]))
        if kind in ("step", "field") and rng.random() < 0.4:
            c.update(nx=rng.choice([256, 384, 512, 768, 1024, 2048]), ny=rng.choice([256, 384, 512, 768, 1536]))
    else:
        c.update(nz=smooth(rng, 2, 32), ny=smooth(rng, 16, 256 if kind != "dropin" else 128),
                 nx=smooth(rng, 16, 256 if kind != "dropin" else 128), material="cube")
    if kind == "field":
        c["per"] = rng.choice([0, 0, 1])
        return c
    if kind in ("trials", "run"):
        # the second-order pair needs the smooth state to hold its error at this dt
        film = c["material"] == "film"
        c.update(solver=rng.choice(["rk23", "rkck", "rkdp"] + ["rk12"] * film), dt=3e-14 if film else 1e-14,
                 maxerror=1e-4, n=rng.randint(2, 6) if kind == "trials" else rng.randint(8, 50))
    else:
        c.update(solver=rng.choice(["heun", "rk4"]) if kind == "step" else "heun", dt=1e-14, n=rng.randint(1, 4))
    return c


# ---------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------
def engine():
    return importlib.import_module("1_b200")


def physical(case):
    """The user-level description of a single-grid case (SI units, user axes)."""
    return dict(grid=(case["nx"], case["ny"], case["nz"]), periodic=(0, case.get("per", 0), 0),
                **MATERIALS[case["material"]])


def magnetisation(case, seed):
    """The initial state, internal [3][nz][ny][nx] on the GPU: a tilted
    uniform state with 1% noise (film), independent unit vectors (cube), an
    in-plane curl with a core along +z, tilted by a field, and 2% noise
    (vortex)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    u = torch.randn((3, nz, ny, nx), generator=g, device="cuda", dtype=torch.float64)
    if case["material"] == "film":
        u = 1.0 + 0.01 * u
    elif case["material"] == "vortex":
        y = torch.arange(ny, device="cuda", dtype=torch.float64)[:, None] - (ny - 1) / 2.0
        x = torch.arange(nx, device="cuda", dtype=torch.float64)[None, :] - (nx - 1) / 2.0
        r = torch.sqrt(x * x + y * y)
        core = r <= 2.5
        v = torch.zeros_like(u)
        v[0] = torch.where(core, torch.zeros_like(r), -y / r.clamp_min(1e-12))
        v[1] = torch.where(core, torch.zeros_like(r), x / r.clamp_min(1e-12))
        v[2] = core.to(torch.float64)
        u = v + 0.3 + 0.02 * u
    u = u / u.square().sum(0, keepdim=True).sqrt()
    return u.flip(0).to(torch.float32).contiguous()


class DeviceArray:
    """A float32 device buffer of the engine, for torch.as_tensor; keeps the
    buffer's owner alive as long as the tensor is."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f4", data=(ptr, False), version=3)


def resident(solver, owner=None):
    """The solver's magnetisation as a torch tensor on its own memory."""
    return torch.as_tensor(DeviceArray(owner or solver, solver.m_device(), (3,) + tuple(solver.N)), device="cuda")


def params(case):
    eng = engine()
    p = eng.mmx_params(**physical(case), solver=case.get("solver", "heun"), dt=case.get("dt", 1e-14),
                       maxerror=case.get("maxerror", 0.0), precision=case.get("precision", 0))
    if case["kind"] in ("trials", "run"):
        p.max_dt = case["dt"]
    return p


def prepare(case, seed):
    eng = engine()
    kind = case["kind"]
    st = dict(case=case, kind=kind)
    if kind == "batch":
        cfgs = eng.batch_config(case["count"], case["draw_seed"])
        b = eng.Batch([eng.mmx_params(**c) for c in cfgs])
        b.use_graph(True)
        for i, c in enumerate(cfgs):
            nx, ny, nz = c["grid"]
            m = magnetisation(dict(nx=nx, ny=ny, nz=nz, material="cube"), seed * 1000 + i)
            b.instances[i].set_m_device(m.data_ptr())
        st.update(batch=b, m=[resident(v, b) for v in b.instances])
        return st
    if kind == "serve":
        # sweeps and relaxations from a nearly saturated state
        reqs = eng.serve_stream(case["count"], seed=case["draw_seed"], sweep_points=case["points"])
        st["requests"] = []
        for i, r in enumerate(reqs):
            nx, ny, nz = r["cfg"]["grid"]
            m = magnetisation(dict(nx=nx, ny=ny, nz=nz, material="film"), seed * 1000 + i).cpu().numpy()
            st["requests"].append((eng.mmx_params(**r["cfg"]), m, r["fields"]))
        st["server"] = eng.Server(batched=True, check_every=20, keep_m=True)
        return st
    m = magnetisation(case, seed)
    if kind == "dropin":
        p = eng.mmx_params(**physical(case), solver=case["solver"], dt=case["dt"])
        N, per = tuple(p.size), tuple(p.periodic)
        P = tuple(2 * n if n > 1 and q == 0 else n for n, q in zip(N, per))
        k6 = torch.zeros((6,) + P, device="cuda")
        eng.face_kernel6_device(P, per, [p.cellsize[d] for d in range(3)],
                                out_ptr=ctypes.c_void_p(k6.data_ptr()))
        torch.cuda.synchronize()
        cfg = eng.driver_config(**physical(case), solver=case["solver"], dt=case["dt"])
        st["sim"] = eng.DriverSim(cfg, m.cpu().numpy(), k6.cpu().numpy())
        return st
    s = eng.Solver(params(case))
    st["solver"] = s
    if kind == "field":
        st.update(m=m, h=torch.empty_like(m))
        return st
    s.set_m_device(m.data_ptr())
    st["m"] = resident(s)
    st["avg"] = torch.zeros(3).pin_memory()
    if kind == "step":
        s.use_graph(True)
    else:
        s.device_control(True)
    return st


# ---------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------
def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "field":
        st["solver"].field(st["m"].data_ptr(), st["h"].data_ptr())
        return st["h"]
    if kind in ("step", "trials"):
        s = st["solver"]
        s.step(case["n"])
        s.avg_m(st["avg"].data_ptr())
        return {"m": st["m"], "avg": st["avg"]}
    if kind == "run":
        rows = st["solver"].run((case["n"] - 0.5) * case["dt"], 1.99 * case["dt"], max_rows=case["n"] + 1)
        # column 4, the last maximum torque, is returned with the others
        return {"m": st["m"], "rows": rows}
    if kind == "batch":
        st["batch"].step(case["n"])
        return st["m"]
    if kind == "dropin":
        st["sim"].steps(case["n"])
        return {"m": st["sim"].m(), "avg": st["sim"].avg_m()}
    sv = st["server"]
    ids = [sv.submit(p, m, f, 1e-4, case["cap"]) for p, m, f in st["requests"]]
    while any(sv.pump()):
        pass
    out = []
    for i in ids:
        r = sv.result(i)
        out.append({"m": sv.result_m(i), "avg": r["avg_m"], "steps": int(r["steps"])})
        sv.release(i)
    return out


# ---------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------
STAGES = {"heun": 2, "rk2": 2, "rk12": 2, "rk23": 3, "rk4": 4, "rkck": 6, "rkdp": 6}


def one_field(nx, ny, nz, per=0):
    """Bytes and operations of one field evaluation: m read and h written
    once, the real kernel spectrum (one octant a component) read once; the
    transforms of the rows that hold data, and the product."""
    N = (nz, ny, nx)
    P = (2 * nz if nz > 1 else 1, ny if per else 2 * ny, 2 * nx)
    hz = P[2] // 2 + 1
    n = N[0] * N[1] * N[2]
    comps = 6 if P[0] > 1 else 4
    octant = (P[0] // 2 + 1) * (P[1] // 2 + 1) * hz
    b = 24.0 * n + 4.0 * comps * octant
    fl = 6 * (2.5 * N[0] * N[1] * P[2] * math.log2(max(2, P[2])) + 5.0 * N[0] * hz * P[1] * math.log2(max(2, P[1])))
    if P[0] > 1:
        fl += 6 * 5.0 * P[1] * hz * P[0] * math.log2(P[0])
    return b, fl + (30.0 if comps == 6 else 14.0) * P[0] * P[1] * hz


def one_step(nx, ny, nz, solver, per=0):
    """A step: its field evaluations, m and the stage torques (12 bytes a cell
    each) written once and read once where a later stage needs them."""
    b, f = one_field(nx, ny, nz, per)
    k = STAGES[solver]
    n = nx * ny * nz
    return k * b + 24.0 * n * (k - 1), k * f + 60.0 * n * k


def work(case):
    kind = case["kind"]
    if kind == "field":
        b, f = one_field(case["nx"], case["ny"], case["nz"], case["per"])
        return {"bytes": b, "flops": f}
    eng = engine()
    if kind == "batch":
        w = [one_step(*c["grid"], "rk4") for c in eng.batch_config(case["count"], case["draw_seed"])]
        k = case["n"]
    elif kind == "serve":
        w = [[v * (1 if r["fields"] is None else len(r["fields"])) for v in one_step(*r["cfg"]["grid"], "rk4")]
             for r in eng.serve_stream(case["count"], seed=case["draw_seed"], sweep_points=case["points"])]
        k = case["cap"]
    else:
        w = [one_step(case["nx"], case["ny"], case["nz"], case["solver"])]
        k = case["n"]
    return {"bytes": k * sum(x[0] for x in w), "flops": k * sum(x[1] for x in w)}


# ---------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------
def f32(x):
    return np.float32(x)


def internal(phys, dt):
    """Internal parameters, each rounded to float32 where the front end
    rounds it (lengths in exchange lengths, times in 1 / (gamma0 Ms), fields
    in mu0 Ms), axes reversed."""
    mu0, gamma0 = f32(4.0e-7 * np.pi), f32(2.211e5)
    ms, a = f32(phys["msat"]), f32(phys["aexch"])
    length = f32(np.sqrt(2.0 * np.float64(f32(a / f32(f32(mu0 * ms) * ms)))))
    time, field = f32(f32(1.0) / f32(gamma0 * ms)), f32(mu0 * ms)
    energy = f32(f32(a * length) / f32(f32(length * length) * length))
    rev = (2, 1, 0)
    p = dict(cell=[float(f32(f32(phys["cell"][d]) / length)) for d in rev],
             hext=[float(f32(f32(phys.get("bext", (0, 0, 0))[d]) / field)) for d in rev],
             alpha=float(f32(phys["alpha"])), dt=float(f32(f32(dt) / time)), unit_time=float(time), K=0.0, u=[0, 0, 0])
    if phys.get("anis"):
        p["K"] = float(f32(f32(phys["k1"]) / energy))
        ax = np.array([phys["axis"][d] for d in rev], np.float32)
        p["u"] = [float(v) for v in ax / f32(np.sqrt(np.float64((ax * ax).sum())))]
    return p


class Exact:
    """One grid in float64: the field by transforms of the whole padded box,
    the torque, and the solvers' steps."""

    def __init__(self, phys, dt):
        nx, ny, nz = phys["grid"]
        self.N = (nz, ny, nx)
        per = tuple(phys.get("periodic", (0, 0, 0))[d] for d in (2, 1, 0))
        self.P = tuple(2 * n if n > 1 and q == 0 else n for n, q in zip(self.N, per))
        self.p = internal(phys, dt)
        self.kern = self.kernel(per)

    def kernel(self, per):
        """Spectra of the six demag + exchange components (XX, YY, ZZ, YZ, XZ,
        XY): 8 x 8 point charges on the two faces of a cell along its
        magnetisation, at every displacement in the box, images summed."""
        P, cs, n = self.P, self.p["cell"], 8
        rng = []
        for d in range(3):
            lo, hi = -((P[d] - 1) // 2), P[d] // 2 - 1
            if P[d] == 1 and per[d] == 0:
                hi = 0
            rng.append(torch.arange(lo * (per[d] + 1), hi * (per[d] + 1) + 1, device="cuda"))
        comp = {(0, 0): 0, (1, 1): 1, (2, 2): 2, (1, 2): 3, (0, 2): 4, (0, 1): 5}
        k = torch.zeros((6,) + P, dtype=torch.float64, device="cuda")
        ax = [r.to(torch.float64) * c for r, c in zip(rng, cs)]
        for s in range(3):
            v, w = (s + 1) % 3, (s + 2) % 3
            acc = [torch.zeros([len(r) for r in rng], dtype=torch.float64, device="cuda") for _ in range(3 - s)]
            for i in range(n):
                for j in range(n):
                    for side in (1.0, -1.0):
                        at = [0.0, 0.0, 0.0]
                        at[s] = side * cs[s] / 2
                        at[v] = -cs[v] / 2 + cs[v] / (2 * n) + i * cs[v] / n
                        at[w] = -cs[w] / 2 + cs[w] / (2 * n) + j * cs[w] / n
                        r = [(ax[d] - at[d]).reshape([-1 if e == d else 1 for e in range(3)]) for d in range(3)]
                        inv = (r[0] * r[0] + r[1] * r[1] + r[2] * r[2]).pow_(-1.5)
                        for d in range(s, 3):
                            acc[d - s].addcmul_(inv, r[d].expand_as(inv), value=side)
            for d in range(s, 3):
                b = acc[d - s] * (cs[v] * cs[w] / (4 * math.pi * n * n))
                for e in range(3):  # wrap the displacements (and images) onto the box
                    shape = list(b.shape)
                    shape[e] = P[e]
                    b = torch.zeros(shape, dtype=torch.float64, device="cuda").index_add_(e, rng[e] % P[e], b)
                k[comp[(s, d)]] += b
        # six-neighbour exchange; where two of the seven cells wrap onto one, the last counts
        inv = [1.0 / (c * c) for c in cs]
        cells = {(0, 0, 0): -2.0 * sum(inv)}
        for d in range(3):
            for step in (1, -1):
                c = [0, 0, 0]
                c[d] = step % P[d]
                cells[tuple(c)] = inv[d]
        for c, val in cells.items():
            for e in range(3):
                k[(e,) + c] += val
        out = []
        for c in range(6):
            out.append(None if P[0] == 1 and c > 3 else torch.fft.rfftn(k[c]).real.contiguous())
        return out

    def field(self, m):
        P, N, K = self.P, self.N, self.kern
        f = [torch.fft.rfftn(m[c], s=P) for c in range(3)]
        h = torch.empty_like(m)
        rows = ((K[0], K[5], K[4]), (K[5], K[1], K[3]), (K[4], K[3], K[2]))
        for c in range(3):
            t = None
            for d in range(3):
                if rows[c][d] is not None:
                    t = f[d] * rows[c][d] if t is None else t.addcmul_(f[d], rows[c][d].to(f[d].dtype))
            h[c] = torch.fft.irfftn(t, s=P)[: N[0], : N[1], : N[2]]
        mu = sum(m[c] * self.p["u"][c] for c in range(3))
        for c in range(3):
            h[c] += self.p["hext"][c] + self.p["K"] * self.p["u"][c] * mu
        return h

    def torque(self, m):
        h = self.field(m)
        t = torch.linalg.cross(m, h, dim=0)
        return (t - self.p["alpha"] * torch.linalg.cross(m, t, dim=0)) / (1.0 + self.p["alpha"] ** 2)

    @staticmethod
    def unit(m):
        return m / m.square().sum(0, keepdim=True).sqrt()

    def step(self, m, solver, k_last=None):
        """One step of the fixed dt; returns (m, last stage torque, first stage torque)."""
        dt = self.p["dt"]
        if solver == "heun":
            t0 = self.torque(m)
            t1 = self.torque(self.unit(m + dt * t0))
            return self.unit(m + 0.5 * dt * (t0 + t1)), None, t0
        a, b, fsal = TABLEAUX[solver]
        k = []
        for i, row in enumerate(a):
            if i == 0 and fsal and k_last is not None:
                k.append(k_last)
                continue
            x = m
            for c, kj in zip(row, k):
                if c:
                    x = x + dt * c * kj
            k.append(self.torque(x))
        x = m
        for c, kj in zip(b, k):
            if c:
                x = x + dt * c * kj
        return self.unit(x), k[-1], k[0]


TABLEAUX = {
    "rk12": ([(), (1.0,)], (0.5, 0.5), False),
    "rk4": ([(), (0.5,), (0.0, 0.5), (0.0, 0.0, 1.0)], (1 / 6, 1 / 3, 1 / 3, 1 / 6), False),
    "rk23": ([(), (0.5,), (0.0, 0.75), (2 / 9, 1 / 3, 4 / 9)], (2 / 9, 1 / 3, 4 / 9, 0.0), True),
    "rkck": ([(), (1 / 5,), (3 / 40, 9 / 40), (3 / 10, -9 / 10, 6 / 5), (-11 / 54, 5 / 2, -70 / 27, 35 / 27),
              (1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096)],
             (37 / 378, 0.0, 250 / 621, 125 / 594, 0.0, 512 / 1771), False),
    "rkdp": ([(), (1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
              (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
              (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
              (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84)],
             (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84, 0.0), True),
}


def averages(m):
    return m.mean((1, 2, 3))


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return None  # thousands of steps
    if kind == "batch":
        out = []
        for i, c in enumerate(engine().batch_config(case["count"], case["draw_seed"])):
            nx, ny, nz = c["grid"]
            e = Exact(c, c["dt"])
            m = magnetisation(dict(nx=nx, ny=ny, nz=nz, material="cube"), seed * 1000 + i).double()
            for _ in range(case["n"]):
                m = e.step(m, "rk4")[0]
            out.append(m)
        return out
    e = Exact(physical(case), case.get("dt", 1e-14))
    m = magnetisation(case, seed).double()
    if kind == "field":
        return e.field(m)
    k = None
    if kind != "run":
        for _ in range(case["n"]):
            m, k, _t = e.step(m, case["solver"], k)
        return {"m": m, "avg": averages(m)}
    # rows: time, <m> in user order, the torque of the step before, min and max of the user's m_z
    m = e.unit(m)
    rows, since, t, torque = [], np.float32(0), 0.0, 0.0
    ut, period = np.float32(e.p["unit_time"]), np.float32(1.99 * case["dt"])
    stop = (case["n"] - 0.5) * case["dt"] / float(ut)
    while t < stop:
        now = np.float32(np.float32(t) * ut)
        if now == 0 or np.float32(now - since) >= period:
            since = now
            a = averages(m).tolist()
            rows.append([float(now), a[2], a[1], a[0], torque, float(m[0].min()), float(m[0].max())])
        m, k, k0 = e.step(m, case["solver"], k)
        torque = float(k0.abs().max())
        t += e.p["dt"]
    return {"m": m, "rows": np.array(rows)}
