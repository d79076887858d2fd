"""The work a user of this framework has it do, as cases that can be timed.

Five kinds of calls, each through the package's public entry points:

  solve    one stirred-tank run: start from rest, then per time step rotate the
           impeller (on the device, or blades generated by the host), collide
           and stream, force, queue the impeller load; at the end the XZ plane
           through the impeller (moments and force). The bench's workload.
  dropin   the reference's own main loop (main.cpp:409-454): every step hands
           forcing() the whole marker list of the geometry from host memory;
           at the end density, velocity and force of every cell.
  fields   a dump of a developed run: density, velocity, force, eddy viscosity
           of every cell.
  batch    many tanks of uneven size advanced together (Batch), each tank's
           impeller load and plane at the end.
  serve    requests handed to a running Server and their results collected.

Sizes run from the 24^3 tank of the smoke test to the bench's 400^3 tank.
A run starts again from rest on every pass, so passes do not depend on one
another, and stays within the step counts that the Simple scheme's wall rule
keeps finite. The oracle in exact() restates the step in 64-bit torch.
"""
import math
import random

import numpy as np
import torch

import tdlbcpp_b200 as tb

ALPHA, BETA = 0.97, 1.9   # FlowParams defaults, bench.py
CS0, G3 = 0.1, 0.8        # bench.py


def listed():
    return [
        # the smallest tank (smoke test's size): launches and latency
        dict(name="solve24_simple", kind="solve", x=24, y=24, z=24, streaming="Simple", storage="fp32", les=True,
             steps=60, blades="device"),
        # odd, ragged extents, blades generated by the host each step (bench's end-to-end leg)
        dict(name="solve101_ragged_hostblades", kind="solve", x=101, y=83, z=97, streaming="Simple", storage="fp32",
             les=True, steps=60, blades="host"),
        # an ordinary tank in half precision
        dict(name="solve160_simple_fp16", kind="solve", x=160, y=160, z=160, streaming="Simple", storage="fp16",
             les=True, steps=60, blades="device"),
        # an ordinary tank on the single-buffer scheme, without the turbulence model
        dict(name="solve192_esotwist_nolesbf16", kind="solve", x=192, y=192, z=192, streaming="Esotwist",
             storage="bf16", les=False, steps=60, blades="device"),
        # a large single-buffer tank
        dict(name="solve256_esotwist", kind="solve", x=256, y=256, z=256, streaming="Esotwist", storage="fp32",
             les=True, steps=40, blades="device"),
        # the bench's headline tank
        dict(name="solve400_simple", kind="solve", x=400, y=400, z=400, streaming="Simple", storage="fp32", les=True,
             steps=40, blades="device"),
        # the same tank in half precision on the single-buffer scheme
        dict(name="solve400_esotwist_fp16", kind="solve", x=400, y=400, z=400, streaming="Esotwist", storage="fp16",
             les=True, steps=40, blades="device"),
        # the reference's shipped debug input (60^3, Esotwist, rho 8, no LES) driven as its main loop does
        dict(name="dropin60", kind="dropin", x=60, y=60, z=60, streaming="Esotwist", storage="fp32", les=False, steps=20),
        # the same loop on an ordinary tank
        dict(name="dropin144_simple", kind="dropin", x=144, y=144, z=144, streaming="Simple", storage="fp32", les=True,
             steps=4),
        # a dump of every field
        dict(name="fields128", kind="fields", x=128, y=128, z=128, streaming="Simple", storage="fp32", les=True, steps=30),
        # the batched bench's tank sizes
        dict(name="batch12", kind="batch", count=12, lo=32, hi=128, streaming="Esotwist", storage="fp32", les=True,
             steps=48),
        # a handful of small requests to a resident server
        dict(name="serve6", kind="serve", count=6, lo=24, hi=56, streaming="Esotwist", storage="fp32", les=True,
             steps=100),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "dropin", "fields", "batch", "serve"])
    streaming, les = rng.choice(["Simple", "Esotwist"]), rng.random() < 0.75
    storage = rng.choice(["fp32", "fp32", "fp16", "bf16"])
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    if kind in ("batch", "serve"):
        lo = rng.randrange(24, 41)
        return dict(kind=kind, count=rng.randrange(3, 11), lo=lo, hi=lo + rng.randrange(8, 24 if kind == "serve" else 72),
                    streaming=streaming, storage=storage, les=les, steps=rng.randrange(30, 100))
    edge = log(24, 384 if kind == "solve" else 150)
    x = edge
    z = max(24, edge - rng.randrange(0, 1 + edge // 8))
    y = max(24, min(int(edge * rng.uniform(0.6, 1.25)), 400))
    if kind == "solve":
        return dict(kind=kind, x=x, y=y, z=z, streaming=streaming, storage=storage, les=les,
                    steps=rng.randrange(20, 41) if edge > 160 else rng.randrange(30, 81),
                    blades=rng.choice(["device", "device", "host"]))
    return dict(kind=kind, x=x, y=y, z=z, streaming=streaming, storage="fp32" if kind == "dropin" else storage, les=les,
                steps=rng.randrange(2, 5) if edge > 80 else rng.randrange(4, 16))


# ---------------------------------------------------------------- inputs

def _edges(case):
    """Tank edges of a batch or of the requests: spread evenly over [lo, hi], largest first."""
    n = case["count"]
    return [int(round(case["hi"] - (case["hi"] - case["lo"]) * q / max(1, n - 1))) for q in range(n)]


def _flow(rng):
    """Tip speed, Reynolds number and first impeller angle of one tank."""
    return rng.uniform(0.05, 0.1), math.exp(rng.uniform(math.log(2e3), math.log(2e4))), rng.uniform(0.0, 1.0)


def _turbine(x, y, z, tip):
    return tb.RushtonTurbine(x, y, z, tip_speed=tip, startup_steps=0, tank_diameter=float(min(x, z)))


def _tank(case, tip, re):
    rt = _turbine(case["x"], case["y"], case["z"], tip)
    nu = tb.nu_from_reynolds(re, tip, rt.blade_outer_radius())
    rho = 8.0 if case["kind"] == "dropin" else 1.0
    cfg = dict(x=case["x"], y=case["y"], z=case["z"], nu=nu, cs0=CS0, g3=G3, useLES=int(case["les"]), initialRho=rho,
               streaming=case["streaming"], storage=case["storage"])
    return rt, nu, rho, cfg


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "serve":
        flows = [_flow(rng)[:2] for _ in range(case["count"])]
        return dict(case=case, flows=flows, server=tb.Server(max_active=case["count"]), next_id=0)
    if kind == "batch":
        tanks = []
        for edge in _edges(case):
            tip, re, angle = _flow(rng)
            rt, _, _, cfg = _tank(dict(case, x=edge, y=edge, z=edge), tip, re)
            tanks.append((rt, cfg, angle))
        b = tb.Batch([cfg for _, cfg, _ in tanks])
        for cu, (rt, _, angle) in zip(b.tanks, tanks):
            d = rt.increment(1)
            cu.attach_rushton(rt, d, angle, d)
        return dict(case=case, batch=b, tanks=tanks)
    tip, re, angle = _flow(rng)
    rt, nu, rho, cfg = _tank(case, tip, re)
    d = rt.increment(1)
    s = dict(case=case, rt=rt, rho=rho, angle=angle, d=d, cu=tb.ComputeUnit(**cfg), plane=_impeller_plane(case))
    if kind == "dropin":
        # the host's list: the part that stays, then the blades, written anew each step
        still = np.concatenate([rt.fixed(), rt.rotating_nonupdating(d)])
        s["markers"] = np.concatenate([still, rt.rotating(angle, d)])
        s["n_still"] = len(still)
        return s
    s["cu"].attach_rushton(rt, d, angle, d)
    if kind == "solve":
        s["loads"] = torch.empty((case["steps"], 5), dtype=torch.float64, pin_memory=True)
    else:
        _solve(s, None)
        s["cu"].synchronize()
    return s


def _impeller_plane(case):
    return min(case["y"] - 1, int(round(min(case["x"], case["z"]) / 3.0)))


# ---------------------------------------------------------------- one pass

def _solve(s, loads):
    cu, rt, d, case = s["cu"], s["rt"], s["d"], s["case"]
    angle = s["angle"]
    host = case.get("blades") == "host"
    if host:
        cu.set_rotating_markers(rt.rotating(angle, d))
    else:
        cu.rotate_impeller(angle, d)
    cu.initialise(s["rho"])
    cu.forcing_resident(ALPHA, BETA)
    for q in range(case["steps"]):
        angle += d
        if host:
            cu.set_rotating_markers(rt.rotating(angle, d))
        else:
            cu.rotate_impeller(angle, d)
        cu.collision()
        cu.forcing_resident(ALPHA, BETA)
        if loads is not None:
            cu.impeller_load_async(loads[q].data_ptr())


def _plane(cu, j):
    """The plane dump as dense arrays: moments (or raw Esotwist slots) and force."""
    q, f = cu.plane_xz(j)
    m = np.zeros((cu.x, cu.z, 4), np.float32)
    m[q["iGrid"], q["kGrid"]] = q["q"]
    force = np.zeros((cu.x, cu.z, 3), np.float32)
    force[f["iGrid"], f["kGrid"]] = f["q"]
    return m, force


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "solve":
        _solve(s, s["loads"])
        m, force = _plane(s["cu"], s["plane"])
        s["cu"].synchronize()
        return dict(loads=s["loads"].numpy()[:, :4].astype(np.float32), moments=m, force=force)
    if kind == "dropin":
        cu, rt, d, mk, n0 = s["cu"], s["rt"], s["d"], s["markers"], s["n_still"]
        angle = s["angle"]
        mk[n0:] = rt.rotating(angle, d)
        cu.initialise(s["rho"])
        cu.forcing(mk, ALPHA, BETA)
        for _ in range(case["steps"]):
            angle += d
            mk[n0:] = rt.rotating(angle, d)
            cu.collision()
            cu.bounceBackBoundary()
            cu.streamingPush()
            cu.moments()
            cu.forcing(mk, ALPHA, BETA)
        rho, u = cu.read_velocity_density()
        return dict(rho=rho, u=u, force=cu.read_force())
    if kind == "fields":
        cu = s["cu"]
        rho, u = cu.read_velocity_density()
        return dict(rho=rho, u=u, force=cu.read_force(), nu=cu.read_nu())
    if kind == "batch":
        b = s["batch"]
        for cu, (rt, cfg, angle) in zip(b.tanks, s["tanks"]):
            cu.rotate_impeller(angle, rt.increment(1))
            cu.initialise(1.0)
            cu.forcing_resident(ALPHA, BETA)
        b.run(case["steps"], ALPHA, BETA)
        out = []
        for cu in b.tanks:
            load = cu.impeller_load()
            m, force = _plane(cu, _impeller_plane(dict(x=cu.x, y=cu.y, z=cu.z)))
            out.append(dict(load=load[:4].astype(np.float32), moments=m, force=force))
        return out
    server = s["server"]
    first = s["next_id"]
    for q, (edge, (tip, re)) in enumerate(zip(_edges(case), s["flows"])):
        server.submit(first + q, edge, tip, re, case["steps"], storage=case["storage"], streaming=case["streaming"],
                      les=case["les"], fields=True)
    s["next_id"] = first + case["count"]
    server.wait_idle(600.0)
    got = []
    while len(got) < case["count"]:
        got += server.poll()
    out = []
    for r in sorted(got, key=lambda r: r["id"]):
        f = r["fields"]
        out.append(dict(status=r["status"], diag=np.array(r["force"] + [r["torque"], r["mass"]], np.float32), rho=f["rho"],
                        u=np.stack([f["ux"], f["uy"], f["uz"]], axis=-1)))
    return out


def work(case):
    """Bytes: per step each population read and written once, the eddy viscosity read and written with LES; the
    fields handed back once. Operations: about 400 per cell and step."""
    cells = sum(e ** 3 for e in _edges(case)) if case["kind"] in ("batch", "serve") else case["x"] * case["y"] * case["z"]
    size = 4 if case["storage"] == "fp32" else 2
    step = 36 * size + (8 if case["les"] else 0)
    kind = case["kind"]
    if kind == "fields":   # populations, force and viscosity read, 8 floats written
        return dict(bytes=cells * (18 * size + 16 + 32.0), flops=cells * 80.0)
    out = {"solve": 0, "dropin": 28, "batch": 0, "serve": 16}[kind]
    return dict(bytes=float(cells * (step * case["steps"] + out)), flops=float(cells * 400 * case["steps"]))


# ---------------------------------------------------------------- 64-bit oracle

_CX = (1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0)
_CY = (0, 0, 1, -1, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 1, -1)
_CZ = (0, 0, 0, 0, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, -1, 1, -1, 1)


def _moments(q):
    """The 18 moments M01..M18 (CollisionEgglesSomers.hpp:186-256) of 18 population arrays."""
    def s(f):
        out = None
        for d in range(18):
            w = f(_CX[d], _CY[d], _CZ[d], d < 6)
            if w:
                out = (q[d] * w) if out is None else out.add_(q[d], alpha=w)
        return out
    return [
        s(lambda x, y, z, f: 1.0),
        s(lambda x, y, z, f: x), s(lambda x, y, z, f: y), s(lambda x, y, z, f: z),
        s(lambda x, y, z, f: x * x - 1 if f else 1 - y * y * z * z),
        s(lambda x, y, z, f: x * y),
        s(lambda x, y, z, f: y * y - 1 if f else 1 - x * x * z * z),
        s(lambda x, y, z, f: x * z), s(lambda x, y, z, f: y * z),
        s(lambda x, y, z, f: z * z - 1 if f else 1 - x * x * y * y),
        s(lambda x, y, z, f: -x if f else x * (2 if y else -1)),
        s(lambda x, y, z, f: -y if f else y * (2 if x else -1)),
        s(lambda x, y, z, f: -3 * x if f else (3 * x if z else 0)),
        s(lambda x, y, z, f: -3 * y if f else (3 * y if z else 0)),
        s(lambda x, y, z, f: -2 * z if f else z),
        s(lambda x, y, z, f: 0 if f else (3 * z if y else -3 * z)),
        s(lambda x, y, z, f: (-1 if z else 0.5) if f else (0.5 if z else -1)),
        s(lambda x, y, z, f: 1.5 * (x * x - y * y) if f else (0 if not z else (1.5 if y else -1.5))),
    ]


class _Exact:
    """One tank in 64 bits: moments, force, eddy viscosity as (x, y, z) arrays, stepped as the reference steps them."""

    def __init__(self, x, y, z, nu, rho, les, simple):
        self.shape, self.simple, self.les, self.nu0, self.even = (x, y, z), simple, les, nu, True
        zero = lambda: torch.zeros(self.shape, dtype=torch.float64, device="cuda")  # noqa: E731
        self.m = [zero() for _ in range(18)]
        self.m[0] += rho
        self.F = [zero() for _ in range(3)]
        self.nu = zero()

    def step(self):
        m, F = self.m, self.F
        rho = m[0]
        j = [m[1 + a] + 0.5 * F[a] for a in range(3)]
        u = [v / rho for v in j]
        if self.les:
            fct = 3.0 / (rho * (1.0 + 6.0 * (self.nu + self.nu0)))
            dx, dy, dz = (fct * (m[1 + a] + 0.5 * F[a] * u[a] - m[i]) for a, i in ((0, 4), (1, 6), (2, 9)))
            sh = 2.0 * (dx * dx + dy * dy + dz * dz) - (2.0 / 3.0) * (dx + dy + dz) ** 2
            del dx, dy, dz
            for a, b, i in ((1, 0, 5), (2, 0, 7), (2, 1, 8)):
                sh += (2.0 * fct * (m[1 + a] + 0.5 * F[a] * u[b] - m[i])) ** 2
            self.nu = CS0 * CS0 * sh.abs_().sqrt_()
            del fct, sh
            nut = self.nu + self.nu0
        else:
            nut = self.nu0
        b, c = 1.0 / (1.0 + 6.0 * nut), 1.0 - 6.0 * nut
        a = [rho / 24.0] + [(m[1 + k] + F[k]) / 24.0 for k in range(3)]
        for i, (p, q) in zip(range(4, 10), ((0, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2))):
            a.append((2.0 * j[p] * u[q] - m[i] * c) * b / 24.0)
        a += [m[i] * (-G3 / 24.0) for i in range(10, 16)]
        del j, u, b, c
        self.m = m = None
        f = [None] * 18
        for d in range(18):
            x, y, z = _CX[d], _CY[d], _CZ[d]
            if d < 6:
                v = 2.0 * a[0] + 3.0 * ((2 * x * x - 1) * a[4] + (2 * y * y - 1) * a[6] + (2 * z * z - 1) * a[9])
                if x:
                    v += x * (4.0 * a[1] - 2.0 * (a[10] + a[12]))
                elif y:
                    v += y * (4.0 * a[2] - 2.0 * (a[11] + a[13]))
                else:
                    v += z * 4.0 * (a[3] - a[14])
            else:
                v = a[0] + 1.5 * ((1 if x else -1) * a[4] + (1 if y else -1) * a[6] + (1 if z else -1) * a[9])
                if not z:
                    v += 2.0 * x * (a[1] + a[10]) + 2.0 * y * (a[2] + a[11]) + 6.0 * x * y * a[5]
                elif not y:
                    v += x * (2.0 * a[1] - a[10] + a[12]) + z * (2.0 * a[3] + a[14] - a[15]) + 6.0 * x * z * a[7]
                else:
                    v += y * (2.0 * a[2] - a[11] + a[13]) + z * (2.0 * a[3] + a[14] + a[15]) + 6.0 * y * z * a[8]
            f[d] = self._move(v, (x, y, z))
        del a
        self.m = _moments(f)
        self.even = not self.even

    def _move(self, v, c):
        """f(x - c); off the lattice the cell's own value (Simple) or the periodic one (Esotwist)."""
        w = torch.roll(v, c, (0, 1, 2))
        if self.simple:
            for axis, s in enumerate(c):
                if s:
                    edge = 0 if s > 0 else self.shape[axis] - 1
                    w.select(axis, edge).copy_(v.select(axis, edge))
        return w

    def load_markers(self, mk):
        """The stencil cells, weights, velocities and levels of a marker list: a marker's level is one above the
        highest of the earlier markers it shares a cell with."""
        x, y, z = self.shape
        g = lambda name: torch.from_numpy(np.ascontiguousarray(mk[name])).cuda()  # noqa: E731
        i, j, k, fi, fk = g("i"), g("j"), g("k"), g("iCartFraction").double(), g("kCartFraction").double()
        o1 = torch.arange(-1, 2, device="cuda")
        cell = (((i[:, None, None] + o1[None, None, :]) % x * y + j[:, None, None]) * z
                + (k[:, None, None] + o1[None, :, None]) % z).reshape(-1, 9)

        def phi(r):
            r = r.abs()
            near = (1.0 + (1.0 - 3.0 * r * r).clamp(min=0).sqrt()) / 3.0
            far = (5.0 - 3.0 * r - (1.0 - 3.0 * (1.0 - r) ** 2).clamp(min=0).sqrt()) / 6.0
            return torch.where(r <= 0.5, near, torch.where(r <= 1.5, far, torch.zeros_like(r)))
        w = (phi(o1[None, None, :] - fi[:, None, None]) * phi(o1[None, :, None] - fk[:, None, None])).reshape(-1, 9)
        vel = torch.stack([g("uDelta"), g("vDelta"), g("wDelta")]).double()
        known, local = torch.unique(cell, return_inverse=True)
        n = cell.shape[0]
        owner = torch.full((known.numel(),), n, dtype=torch.int64, device="cuda")
        left, levels = torch.arange(n, device="cuda"), []
        while left.numel():
            c = local[left]
            owner.fill_(n)
            owner.scatter_reduce_(0, c.reshape(-1), left[:, None].expand(-1, 9).reshape(-1), "amin")
            ready = (owner[c] == left[:, None]).all(1)
            levels.append(left[ready])
            left = left[~ready]
        arm = torch.stack([i + fi - (x - 1.0) / 2.0, k + fk - (z - 1.0) / 2.0])
        return dict(cell=cell, w=w, vel=vel, levels=levels, arm=arm)

    def force(self, lists, load_from):
        """One forcing pass over marker lists in order; (Fx, Fy, Fz, torque) on the markers of list q from load_from[q] on."""
        rho, jj = self.m[0].view(-1), [self.m[1 + a].view(-1) for a in range(3)]
        F = [v.view(-1) for v in self.F]
        touched = torch.zeros(rho.shape, dtype=torch.bool, device="cuda")
        load = torch.zeros(4, dtype=torch.float64, device="cuda")
        for mk, begin in zip(lists, load_from):
            total = torch.zeros_like(mk["vel"])
            for lev in mk["levels"]:
                c, w = mk["cell"][lev], mk["w"][lev]
                r = (w * rho[c]).sum(1)
                for a in range(3):
                    s = (w * (jj[a][c] + 0.5 * F[a][c])).sum(1) - r * mk["vel"][a][lev]
                    total[a][lev] = s
                    F[a][c] = ALPHA * F[a][c] - BETA * w * s[:, None]
            touched[mk["cell"].view(-1)] = True
            t = -BETA * total[:, begin:]
            arm = mk["arm"][:, begin:]
            load += torch.stack([t[0].sum(), t[1].sum(), t[2].sum(), (arm[1] * t[0] - arm[0] * t[2]).sum()])
        for v in F:
            v.mul_(touched)
        return load

    def fields(self):
        return self.m[0], torch.stack([(self.m[1 + a] + 0.5 * self.F[a]) / self.m[0] for a in range(3)], -1)

    def plane(self, j):
        out = []
        for s in range(4):
            if self.simple:
                out.append(self.m[s][:, j])
            else:   # the raw slots: moment d of the cell the write map takes slot s from
                d = s if self.even else s ^ 1
                back = tuple(1 if c[d] < 0 else 0 for c in (_CX, _CY, _CZ))
                out.append(torch.roll(self.m[d], back, (0, 1, 2))[:, j])
        return torch.stack(out, -1), torch.stack([v[:, j] for v in self.F], -1)


def _exact_run(case, x, y, z, rt, nu, rho, angle, steps):
    """The tank after `steps` steps from rest and the load of every step."""
    d = rt.increment(1)
    nu = float(np.float32(nu))
    t = _Exact(x, y, z, nu, rho, case["les"], case["streaming"] == "Simple")
    fixed = rt.fixed()
    still = t.load_markers(np.concatenate([fixed, rt.rotating_nonupdating(d)]))
    blades = lambda: t.load_markers(rt.rotating(angle, d))  # noqa: E731
    load = t.force([still, blades()], [len(fixed), 0])
    loads = []
    for _ in range(steps):
        angle += d
        t.step()
        load = t.force([still, blades()], [len(fixed), 0])
        loads.append(load)
    return t, (torch.stack(loads) if loads else load[None])


def exact(case, seed):
    rng = random.Random(seed)
    kind, steps = case["kind"], case["steps"]
    if kind in ("batch", "serve"):
        out, rngs = [], [_flow(rng) for _ in range(case["count"])]
        for edge, (tip, re, angle) in zip(_edges(case), rngs):
            if kind == "batch":
                rt = _turbine(edge, edge, edge, tip)
            else:
                rt = tb.RushtonTurbine(edge, edge, edge, tip_speed=tip, startup_steps=0)
                angle = rt.increment(1)
            nu = tb.nu_from_reynolds(re, tip, rt.blade_outer_radius())
            t, loads = _exact_run(case, edge, edge, edge, rt, nu, 1.0, angle, steps)
            if kind == "batch":
                m, force = t.plane(_impeller_plane(dict(x=edge, y=edge, z=edge)))
                out.append(dict(load=loads[-1], moments=m, force=force))
            else:
                r, u = t.fields()
                out.append(dict(status=0, diag=torch.cat([loads[-1], t.m[0].sum()[None]]), rho=r, u=u))
        return out
    tip, re, angle = _flow(rng)
    rt, nu, rho, _ = _tank(case, tip, re)
    t, loads = _exact_run(case, case["x"], case["y"], case["z"], rt, nu, rho, angle, steps)
    if kind == "solve":
        m, force = t.plane(_impeller_plane(case))
        return dict(loads=loads, moments=m, force=force)
    r, u = t.fields()
    out = dict(rho=r, u=u, force=torch.stack(t.F, -1))
    if kind == "fields":
        out["nu"] = t.nu
    return out
