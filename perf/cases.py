"""Timed cases of the FSI step: the calls a simulation makes, over the sizes it makes them at.

A case is a dict of plain values.  `kind` says which call sequence it times:

* "steps": one scene, already set up and past its first steps, advanced by
  `steps` steps (Scene.step_forward for one, Scene.run for several) and its
  velocity and pressure read into pinned host memory
  (Scene.snapshot / snapshot_wait), as a run that hands its fields on does.
  With `tracers` the scene also carries passive tracers, read back too.
* "batch": several independent scenes advanced together (Batch.step), their
  fields read the same way.
* "frame": the diagnostics and slices of one output frame (Scene.macro,
  Scene.slice), as the stepper collects them for macro.dat and its slices.
* "serve": a request stream through the serving loop (serve), scene creation,
  set-up, stepping and results included.

Grids are nx x ny x nz cells of equal spacing, the shortest side of length 1;
`walls` 1 is the lid-driven cavity (no-slip walls, moving lid at the top), 0 a
periodic box.  `spheres` neo-Hookean spheres are placed, sized and given their
stiffness, density, stretch and spin from the seed, as are the lid speed and
the viscosity.  `form` is the arithmetic form, `var_den` the variable-density
build, `v_down` / `v_up` the multigrid smoothing counts.
"""
import ctypes
import math
import os
import random
import tempfile

import numpy as np
import torch

import rmt3d_b200 as R

FORMS = {"fp64": R.FP64, "mixed": R.MIXED, "mixed_bulk32": R.MIXED_BULK32}
FIELDS = ["u", "v", "w", "p"]
WARM = 24  # steps taken in prepare(): the flow has left its start from rest
FRAMES = 100000


def _case(name, kind="steps", nx=64, ny=0, nz=0, walls=1, spheres=1, form="mixed", var_den=0, steps=1, v_down=2,
          v_up=2, tracers=0, scenes=0):
    c = {"kind": kind, "nx": nx, "ny": ny or nx, "nz": nz or nx, "walls": walls, "spheres": spheres, "form": form,
         "var_den": var_den, "steps": steps, "v_down": v_down, "v_up": v_up, "tracers": tracers, "scenes": scenes}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest calls: a coarse fluid-only cavity advanced one step at a time (parameter studies, coupling to
        # a host program that sets dt every step)
        _case("cavity16_fp64", nx=16, spheres=0, form="fp64"),
        # a mid-size fluid run without solids, several steps between reads
        _case("cavity64_mixed", nx=64, spheres=0, steps=4),
        # the smallest size of the batched and served streams, alone on the GPU
        _case("sphere32_mixed", nx=32, steps=2),
        # the headline workload's size, in the plain and the mixed form, with the smoothing counts the autotuner
        # picks for each
        _case("sphere64_fp64", form="fp64", v_down=1, v_up=1),
        _case("sphere64_mixed", steps=2, v_down=2, v_up=1),
        # an uneven, non-cubic channel with a few spheres and tracers, default smoothing counts
        _case("box48x40x88_tracers", nx=48, ny=40, nz=88, spheres=3, form="fp64", steps=2, tracers=20000),
        # several spheres of differing density (the largest scenes of the batched stream)
        _case("spheres96_mixed_vd", nx=96, spheres=5, var_den=1, steps=2),
        # a periodic box with a pre-stretched spinning sphere, FP32 advection
        _case("periodic128_bulk32", nx=128, walls=0, form="mixed_bulk32", steps=2),
        # the largest size of the served stream
        _case("sphere192_mixed", nx=192, steps=4),
        # sixteen scenes of 32^3 to 96^3 stepped together
        _case("batch16_mixed_vd", "batch", nx=96, spheres=4, var_den=1, steps=2, scenes=16),
        # one output frame: diagnostics and slices
        _case("frame64", "frame", spheres=2, form="fp64"),
        # a burst of small requests through the serving loop
        _case("serve6", "serve", nx=64, steps=6, scenes=6),
    ]


def _levels(nodes):
    """Multigrid level sizes of a wall-bounded (nodal: odd counts halve to
    (n-1)/2+1, cells: even counts halve) hierarchy, as the solver coarsens."""
    out = [tuple(nodes)]
    while out[-1][0] * out[-1][1] * out[-1][2] > 1000:
        n = out[-1]
        if all(v % 2 == 0 and v >= 4 for v in n):
            out.append(tuple(v // 2 for v in n))
        elif all(v % 2 == 1 and v >= 3 for v in n):
            out.append(tuple((v - 1) // 2 + 1 for v in n))
        else:
            break
    return out


def _coarsens(n, walls, var_den):
    mac = _levels(n)
    fem = _levels([v + 1 for v in n]) if walls else mac
    small = all(math.prod(h[-1]) <= 1000 for h in (mac, fem))
    return small and (not var_den or (len(fem) <= len(mac)))


def draw(rng):
    """One more case: grids of 16 to 160 cells a side (spread over the
    logarithm, cubic or not), every form and option."""
    kind = rng.choice(["steps"] * 6 + ["batch", "frame", "serve"])
    form = rng.choice(["fp64", "mixed", "mixed", "mixed_bulk32"])
    var_den = int(rng.random() < 0.4)
    walls = int(rng.random() < 0.75)
    v_down, v_up = rng.choice([(2, 2), (2, 1), (1, 1), (1, 2)])
    if kind == "batch":
        return _case(None, "batch", nx=rng.choice([48, 64, 96]), spheres=rng.randint(1, 5), form=form,
                     var_den=var_den, steps=rng.randint(1, 3), v_down=v_down, v_up=v_up, scenes=rng.randint(3, 14))
    if kind == "serve":
        return _case(None, "serve", nx=rng.choice([32, 64]), form=form, steps=rng.randint(2, 6), v_down=2, v_up=2,
                     scenes=rng.randint(2, 3 if form == "fp64" else 5))
    while True:
        if kind == "frame":
            walls = 1
        a = math.exp(rng.uniform(math.log(16), math.log(160)))
        n = []
        for _ in range(3):
            v = a * rng.choice([1, 1, 1, rng.uniform(0.8, 1.6)])
            q = 4 if v < 40 else 8 if v < 100 else 16
            n.append(max(16, int(v / q + 0.5) * q))
        spheres = rng.randint(0, 3 if min(n) >= 40 else 1) if min(n) >= 24 else 0
        if not walls:
            spheres = max(spheres, 1)
        if math.prod(n) <= 170**3 and min(n) >= (24 if spheres else 16) and _coarsens(n, walls, var_den):
            break
    if kind == "frame":
        return _case(None, "frame", n[0], n[1], n[2], spheres=max(spheres, 1) if min(n) >= 24 else 0, form=form,
                     var_den=var_den)
    # a pass no dearer than the largest listed one (192^3, four mixed steps; the plain form takes about twice as long)
    most = int(4 * 192**3 / (math.prod(n) * (2.2 if form == "fp64" else 1.1)))
    return _case(None, "steps", n[0], n[1], n[2], walls, spheres, form, var_den, min(rng.randint(1, 4), most), v_down,
                 v_up, rng.choice([0, 0, 0, int(math.exp(rng.uniform(math.log(100), math.log(50000))))]))


def _cfg(case, rng, n):
    """The reference-format .cfg of one scene: walls or periodic box, seeded spheres."""
    h = 1.0 / min(n)
    side = [v * h for v in n]
    t = "suppress 1\ndump_code %d\nntracers %d\n" % (1 if case["tracers"] else 0, case["tracers"])
    t += "frames %d\nstop_short -1\nsys_size %d %d %d\n" % (FRAMES, n[0], n[1], n[2])
    box = "0 %r 0 %r 0 %r" % tuple(side)
    t += "xyz_bounds %s\nwall_pos %s\ndt 10\nT %d\nsim_type objects\nfmu %r\n" % (
        box, box, FRAMES, rng.uniform(0.008, 0.012))
    # a lid that moves obliquely: a lid along x over a centred flow would leave the y velocity at rounding level
    lid, angle = rng.uniform(0.7, 1.2), rng.uniform(0.2, 1.3)
    if case["walls"]:
        for f in ("xl", "xh", "yl", "yh", "zl", "zh"):
            uv = (lid * math.cos(angle), lid * math.sin(angle)) if f == "zh" else (0.0, 0.0)
            t += "bc_%s 1 1 1 %r %r 0\n" % (f, uv[0], uv[1])
    placed = []
    r0, r1 = (0.16, 0.22) if case["spheres"] == 1 else (0.11, 0.15)
    r0 = max(r0, 4.2 * h)
    r1 = max(r1, r0 + 0.01)
    for _ in range(5000):
        if len(placed) >= case["spheres"]:
            break
        r = rng.uniform(r0, r1)
        gap = r + (6 * h if min(n) >= 40 else 3 * h)
        if any(s <= 2 * gap for s in side):
            r = r0
            gap = r + 3 * h
        c = [rng.uniform(gap, s - gap) for s in side]
        if all(math.dist(c, q[0]) >= r + q[1] + 8 * h for q in placed):
            placed.append((c, r))
    if placed:
        t += "wt_n 1.5\nnlayers 5\nn_obj %d\n" % len(placed)
    for i, (c, r) in enumerate(placed):
        t += "object_list %d %d\nbasic_specs %d %r %r %r %r\n" % (i, 0 if case["walls"] else 1, i, c[0], c[1], c[2], r)
        if not case["walls"]:
            t += "extra_specs %d %d %r %r %r %r 0 0 0 0 0\n" % (
                i, rng.randrange(3), math.sqrt(rng.uniform(1.1, 1.25)), rng.uniform(-1, 1), rng.uniform(-1, 1),
                rng.uniform(-1, 1))
        rho = rng.uniform(0.85, 1.2) if case["var_den"] else 1.0
        t += "shear_mod %d %r\nsrho %d %r\n" % (i, 10 ** rng.uniform(-0.5, 0.5), i, rho)
    return t


def _desc(case, rng, n=None):
    n = n or [case["nx"], case["ny"], case["nz"]]
    fd, path = tempfile.mkstemp(suffix=".cfg")
    with os.fdopen(fd, "w") as f:
        f.write(_cfg(case, rng, n))
    d = R.desc_from_cfg(path)
    os.unlink(path)
    d.precision = FORMS[case["form"]]
    d.var_den = case["var_den"]
    return d


def _pinned(cells):
    return [torch.empty(cells, dtype=torch.float64).pin_memory() for _ in FIELDS]


def _ok(status):
    if any(status):
        raise RuntimeError("step status %r" % (status,))


def prepare(case, seed):
    rng = random.Random("%d" % seed)
    kind = case["kind"]
    if kind == "serve":
        sizes = [32] if case["nx"] < 64 else [32, 32, 64]
        reqs = []
        for i in range(case["scenes"]):
            n = rng.choice(sizes) if i else max(sizes)
            reqs.append((0.0, case["steps"], _desc(case, rng, [n] * 3)))
        return {"case": case, "requests": reqs}
    if kind == "batch":
        sizes = [s for s in (32, 48, 64, 96) if s <= case["nx"]]
        # the same mix of sizes for every seed, so that passes cost alike
        descs = [_desc(case, rng, [sizes[-1 - i % len(sizes)]] * 3) for i in range(case["scenes"])]
        b = R.Batch(descs)
        hosts, reads = [], []
        which = (ctypes.c_int * len(FIELDS))(*[R.FIELD_INDEX[f] for f in FIELDS])
        for i, d in enumerate(descs):
            h = b.scene_handle(i)
            R._lib.check(R.lib().rmt3d_scene_set_schedule(h, case["v_down"], case["v_up"], -1))
            bufs = _pinned((d.sys_size[0] + 4) * (d.sys_size[1] + 4) * (d.sys_size[2] + 4))
            hosts.append(bufs)
            reads.append((h, (ctypes.c_void_p * len(FIELDS))(*[t.data_ptr() for t in bufs])))
        b.prepare()
        _ok(b.step(WARM))
        return {"case": case, "batch": b, "which": which, "reads": reads, "hosts": hosts}
    sc = R.Scene(_desc(case, rng))
    sc.set_schedule(case["v_down"], case["v_up"])
    sc.prepare()
    _ok([sc.run(WARM)])
    return {"case": case, "scene": sc, "hosts": _pinned(sc.ncell)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "steps":
        sc, hosts = state["scene"], state["hosts"]
        _ok([sc.step_forward(0) if case["steps"] == 1 else sc.run(case["steps"])])
        sc.snapshot(FIELDS, hosts)
        out = {"fields": hosts}
        if case["tracers"]:
            out["tracers"] = sc.tracers()
        sc.snapshot_wait()
        return out
    if kind == "batch":
        L = R.lib()
        _ok(state["batch"].step(case["steps"]))
        for h, dst in state["reads"]:
            R._lib.check(L.rmt3d_snapshot_fields(h, state["which"], len(FIELDS), dst))
        for h, _ in state["reads"]:
            R._lib.check(L.rmt3d_snapshot_wait(h))
        return state["hosts"]
    if kind == "frame":
        sc = state["scene"]
        m = sc.macro()
        vals = [m.div_u_l2, *m.momentum, m.energy, m.kinetic, m.elastic, m.potential]
        out = {"macro": np.array(vals)}
        if m.n_obj:
            out["centroid"] = np.array([tuple(m.centroid[o]) for o in range(m.n_obj)])
            out["velocity"] = np.array([tuple(m.velocity[o]) for o in range(m.n_obj)])
        mid = case["nz"] // 2
        for otype in (0, 2, 7, 5) + ((8, 9) if m.n_obj else ()):
            out["slice_" + R.OUTPUT_NAMES[otype]] = sc.slice(otype, 2, mid)
        return out
    res, _summary = R.serve(state["requests"], 64 << 30, 16)
    _ok([r["status"] for r in res])
    return {"checksum": np.array([r["checksum"] for r in res]), "steps": np.array([r["steps_done"] for r in res])}


def _cells(case):
    if case["kind"] == "batch":
        sizes = [s for s in (32, 48, 64, 96) if s <= case["nx"]]
        return sum(sizes[-1 - i % len(sizes)] ** 3 for i in range(case["scenes"]))
    if case["kind"] == "serve":
        return case["scenes"] * 32**3
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """What a step cannot do without: the state that goes from one step to the
    next read and written once (velocity and pressure, with solids the maps of
    their cells, about 1/6 of the box: x in and out), and the operations of
    the stencils; a frame reads the velocity, the pressure and the maps once."""
    cells = _cells(case)
    maps = min(1.0, 0.06 * case["spheres"])
    state = 8 * (4 + 3 * maps)
    if case["kind"] == "frame":
        return {"bytes": state * cells, "flops": 60 * cells}
    steps = case["steps"]
    # two Poisson solves: at least one V-cycle each (8/7 of a fine-level pass: 30 and 60 operations a point)
    flops = (900 + 8 / 7 * (case["v_down"] + case["v_up"] + 1) * 90 + 3000 * maps) * cells * steps
    read_out = 8 * 4 * cells
    return {"bytes": 2 * state * cells * steps + read_out, "flops": flops}


# --- the fluid-only cavity in 64 bits --------------------------------------
# The step of the lid-driven cavity without solids, in plain torch: Godunov
# slopes and half-step states, upwinding, the marker-and-cell projection, the
# explicit momentum update and the Q1 finite-element projection, with both
# Poisson problems solved exactly in their cosine eigenbasis.


def _shift(a, d, s):
    return torch.roll(a, -s, 2 - d)  # a[cell + s along axis d]; arrays are (z, y, x)


def _slope(u, d):
    m2, m1, p1, p2 = (_shift(u, d, s) for s in (-2, -1, 1, 2))

    def lim(a, b, c):
        t1, t2 = 2 * (b - a), 2 * (c - b)
        return torch.where(t1 * t2 > 0, torch.minimum(t1.abs(), t2.abs()), torch.zeros_like(t1))

    def sgn(a):
        return torch.where(a >= 0, 1.0, -1.0).to(a.dtype)

    def delf(a, b, c):
        cen = 0.5 * (c - a)
        return sgn(cen) * torch.minimum(cen.abs(), lim(a, b, c))

    cen = 0.5 * (p1 - m1)
    near = (delf(m2, m1, u) + delf(u, p1, p2)) / 6.0
    return sgn(cen) * torch.minimum(lim(m1, u, p1), (4.0 / 3.0 * cen - near).abs())


class _Cavity:
    def __init__(self, desc, device):
        self.n = list(desc.sys_size)
        self.h = (desc.bounds[1] - desc.bounds[0]) / self.n[0]
        self.mu, self.lid = desc.fmu, [desc.bcv[c][5] for c in range(3)]
        self.dt_reg = min(0.5 * desc.frho / (desc.fmu * 3 / self.h**2) * desc.fdt_pad, desc.dt)
        frame = desc.T / (desc.frames - 1)
        steps = int(frame / self.dt_reg)
        rem = frame - steps * self.dt_reg
        self.dt_fit = self.dt_reg - (self.dt_reg - rem) / (steps + 1) if rem > 0 else self.dt_reg
        shape = [v + 4 for v in reversed(self.n)]
        new = lambda: torch.zeros(shape, dtype=torch.float64, device=device)  # noqa: E731
        self.vel, self.p, self.new = [new() for _ in range(3)], new(), new
        ar = lambda m: torch.arange(m, dtype=torch.float64, device=device)  # noqa: E731
        self.mac, self.fem = [], []
        for N in self.n:
            k = ar(N)
            V = torch.cos(math.pi * k[None, :] * (k[:, None] + 0.5) / N)
            self.mac.append((V, torch.linalg.inv(V), 2 * torch.cos(math.pi * k / N) - 2))
            k = ar(N + 1)
            V = torch.cos(math.pi * k[None, :] * k[:, None] / N)
            c = torch.cos(math.pi * k / N)
            half = torch.ones_like(k)
            half[0] = half[-1] = 0.5
            self.fem.append((V, torch.linalg.inv(V), 2 - 2 * c, (4 + 2 * c) / 6, half))

    @staticmethod
    def _apply(mats, a):
        x, y, z = mats
        a = torch.einsum("ia,cba->cbi", x, a)
        a = torch.einsum("jb,cbi->cji", y, a)
        return torch.einsum("kc,cji->kji", z, a)

    def solve_mac(self, r):
        e = self.mac
        lam = e[0][2][None, None, :] + e[1][2][None, :, None] + e[2][2][:, None, None]
        c = self._apply([v[1] for v in e], r)
        lam[0, 0, 0] = 1
        c = c / lam
        c[0, 0, 0] = 0
        return self._apply([v[0] for v in e], c)

    def solve_fem(self, r):
        e = self.fem
        kx, ky, kz = e[0][2][None, None, :], e[1][2][None, :, None], e[2][2][:, None, None]
        mx, my, mz = e[0][3][None, None, :], e[1][3][None, :, None], e[2][3][:, None, None]
        lam = 12 * (kx * my * mz + mx * ky * mz + mx * my * kz)
        half = e[0][4][None, None, :] * e[1][4][None, :, None] * e[2][4][:, None, None]
        c = self._apply([v[1] for v in e], r / half)
        lam[0, 0, 0] = 1
        c = c / lam
        c[0, 0, 0] = 0
        return self._apply([v[0] for v in e], c)

    def ghosts(self):
        # both ghost layers of every wall face by reflection, axis by axis
        for d in range(3):
            ax, N = 2 - d, self.n[d]
            for side in (0, 1):
                for layer in (1, 2):
                    gh, mi = (2 - layer, 1 + layer) if side == 0 else (1 + N + layer, 2 + N - layer)
                    for c in range(3):
                        bc = self.lid[c] if (d, side) == (2, 1) else 0.0
                        self.vel[c].select(ax, gh).copy_(2 * bc - self.vel[c].select(ax, mi))

    def walls(self, fv):
        for d in range(3):
            ax, N = 2 - d, self.n[d]
            for side in (0, 1):
                face, inner = 2 * d + side, 2 * d + 1 - side
                for c in range(3):
                    bc = self.lid[c] if (d, side) == (2, 1) else 0.0
                    fv[face][c].select(ax, 2 if side == 0 else 1 + N).fill_(bc)
                    fv[inner][c].select(ax, 1 if side == 0 else 2 + N).fill_(bc)

    def accel(self):
        h = self.h
        acc = []
        grad = self.node_gradient(self.p)
        for c in range(3):
            a = torch.zeros_like(self.p)
            for d in range(3):
                s = self.mu / h * (self.vel[c] - _shift(self.vel[c], d, -1))
                a = a + (_shift(s, d, 1) - s) / h
            acc.append(a - grad[c])
        return acc

    def node_gradient(self, p):
        out = []
        for c in range(3):
            o = [d for d in range(3) if d != c]
            t = _shift(p, c, 1) - p
            t = t + _shift(t, o[0], 1)
            out.append(0.25 / self.h * (t + _shift(t, o[1], 1)))
        return out

    def inner(self, a):
        return a[2:-2, 2:-2, 2:-2]

    def divergence_rhs(self, dvel):
        # Q1 right-hand side: every cell adds its increment times the basis gradients at its eight nodes
        fac = 3 * self.h / self.dt_reg
        r = torch.zeros([v + 1 for v in reversed(self.n)], dtype=torch.float64, device=self.p.device)
        d = [self.inner(a) for a in dvel]
        for m in range(8):
            a, b, c = m % 2, m // 2 % 2, m // 4
            t = fac * ((2 * a - 1) * d[0] + (2 * b - 1) * d[1] + (2 * c - 1) * d[2])
            r[c : c + self.n[2], b : b + self.n[1], a : a + self.n[0]] += t
        return r

    def step(self, dt):
        h = self.h
        nv = [[_slope(self.vel[c], d) / h for c in range(3)] for d in range(3)]
        acc = self.accel()
        fv = [[None] * 3 for _ in range(6)]
        for c in range(3):
            adv = -0.5 * dt * sum(self.vel[b] * nv[b][c] for b in range(3))
            base = self.vel[c] + adv + 0.5 * dt * acc[c]
            for f in range(6):
                fv[f][c] = base + 0.5 * h * (2 * (f % 2) - 1) * nv[f // 2][c]
        self.walls(fv)
        for d in range(3):
            lo, hi = 2 * d, 2 * d + 1
            left = list(fv[hi])
            right = [_shift(fv[lo][c], d, 1) for c in range(3)]
            nl, nr = left[d], right[d]
            up, dn = (nl + nr > 0) & (nl > 0), (nl + nr < 0) & (nr < 0)
            for c in range(3):
                mid = torch.zeros_like(nl) if c == d else 0.5 * (left[c] + right[c])
                f = torch.where(up, left[c], torch.where(dn, right[c], mid))
                fv[hi][c], fv[lo][c] = f.clone(), _shift(f, d, -1)
        self.walls(fv)
        q = self.new()
        div = sum(self.inner(fv[2 * d + 1][d] - fv[2 * d][d]) for d in range(3))
        self.inner(q).copy_(self.solve_mac(h / (2 * dt) * div))
        for d in range(3):
            fv[2 * d][d] = fv[2 * d][d] - 2 * dt / h * (q - _shift(q, d, -1))
            fv[2 * d + 1][d] = fv[2 * d + 1][d] - 2 * dt / h * (_shift(q, d, 1) - q)
        self.walls(fv)
        adv = [-0.5 * dt * (fv[2 * d][d] + fv[2 * d + 1][d]) / h for d in range(3)]
        dvel = []
        for c in range(3):
            dv = sum(adv[d] * (fv[2 * d + 1][c] - fv[2 * d][c]) for d in range(3)) + dt * acc[c]
            dvel.append(dv)
            self.inner(self.vel[c]).add_(self.inner(dv))
        self.ghosts()
        x = self.solve_fem(self.divergence_rhs(dvel))
        x = x - x.mean()
        dp = self.new()
        dp[2:-1, 2:-1, 2:-1] = x
        self.p[2:-1, 2:-1, 2:-1] += x
        g = self.node_gradient(dp)
        for c in range(3):
            self.inner(self.vel[c]).sub_(dt * self.inner(g[c]))
            dvel[c] = dvel[c] - dt * g[c]
        self.ghosts()
        return dvel

    def set_up(self, num_iters):
        # pressure pre-iterations: a step whose pressure is kept and whose velocity is thrown away
        dt = self.dt_fit
        for _ in range(num_iters):
            self.ghosts()
            dvel = self.step(dt)
            r = self.divergence_rhs(dvel)
            half = self.fem[0][4][None, None, :] * self.fem[1][4][None, :, None] * self.fem[2][4][:, None, None]
            divu = float(((half * r * r).sum() / r.numel()).sqrt())
            for v in self.vel:
                v.zero_()
            dt = self.dt_reg
            if divu < 1e-4:
                break


def exact(case, seed):
    """The fields of a fluid-only cavity after the same steps.  None for the
    scenes with solids: their reference maps are advected, extrapolated and
    redrawn by data-dependent rules that have no value of their own outside
    the scheme, so there is nothing plainer to compare them with."""
    if case["kind"] != "steps" or case["spheres"] or not case["walls"] or case["var_den"] or case["tracers"]:
        return None
    if _cells(case) > 80**3:
        return None
    d = _desc(case, random.Random("%d" % seed))
    c = _Cavity(d, "cuda" if torch.cuda.is_available() else "cpu")
    c.set_up(d.num_iters)  # leaves the ghost layers at rest too: the lid acts from the first step's momentum update
    for _ in range(WARM + case["steps"]):
        c.step(c.dt_fit)
    return {"fields": [a.reshape(-1).cpu() for a in c.vel + [c.p]]}
