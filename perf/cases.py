"""Performance cases of the voxel-physics step: what a program that simulates soft robots asks of it.

A program builds a batch of robots (one context), advances it by some number of time steps
and reads the state and the centres of mass back into page-locked buffers; or, to
differentiate, records some steps and runs the adjoint backwards over them.  One pass is one
such call sequence on a batch that is already built; a further pass goes on from where the
last one ended, as a simulation does.

The cases span the sizes that a batch takes (one robot of a hundred voxels to a thousand
robots or one body of 64^3 cells), both precisions, self-collision on and off, the cilia
option, forward runs and gradients, and step counts that do and do not fill a graph chunk.

`exact` restates the step in 64-bit torch: the beam links, the voxel integration with floor
contact and friction, the actuation, self-collision by exact pair tests, cilia; gradients come
from torch's own reverse mode over that restatement.
"""

import math
import zlib

import numpy as np
import torch

from __graft_entry__ import load_package

load_package()
from vx3g import abi, workloads as wl  # noqa: E402

AMPLITUDE, PERIOD = 39.0, 0.2  # degrees C and seconds: the actuation of every workload here


def _case(name, robots, lo, hi, fill, materials, precision, steps, **kw):
    """One case.  lo, hi: the range of a robot's extents in cells (the same text "x,y,z" fixes
    them); fill: Bernoulli fill of the box (the largest connected part is kept); materials: how
    many (a population's moduli are log-uniform in [1e5, 1e7] Pa); phases: every voxel an actuation
    phase of its own, or all in step; drop: cells above the floor; checkpoint: of a gradient."""
    c = dict(name=name, robots=robots, lo=lo, hi=hi, fill=fill, materials=materials, precision=precision, steps=steps,
             kind="forward", collision=False, cilia=False, actuated=True, phases=True, drop=0, checkpoint=0)
    c.update(kw)
    return c


def listed():
    return [
        # one small robot: what a designer drags about, or one evaluation of a serial search; the smallest call
        _case("robot_6x5x4_mixed", 1, "6,5,4", "6,5,4", 0.8, 2, "mixed", 100),
        # the plain reference-method workload: a solid block dropped on the floor, FP64
        _case("block_10x10x10_fp64", 1, "10,10,10", "10,10,10", 1.0, 1, "fp64", 100, actuated=False, phases=False, drop=2),
        # a control loop: a few steps at a time (fewer than a graph chunk, and odd), the state read in between
        _case("control_12x12x6_mixed", 1, "12,12,6", "12,12,6", 1.0, 2, "mixed", 25),
        # an evolutionary search's population, the batched workload at its configured size
        _case("population_1024_mixed", 1024, "4,4,4", "16,16,16", 0.7, 4, "mixed", 200),
        # the same kind of population in the reference's arithmetic, a count that divides nothing
        _case("population_203_fp64", 203, "4,4,4", "16,16,16", 0.7, 4, "fp64", 40),
        # one large self-colliding body that contracts in step and folds, the 64^3 workload, in both precisions
        _case("body_64_mixed", 1, "64,64,64", "64,64,64", 0.6, 2, "mixed", 200, collision=True, phases=False),
        _case("body_64_fp64", 1, "64,64,64", "64,64,64", 0.6, 2, "fp64", 20, collision=True, phases=False),
        # the collision-heavy population at its configured size, and a smaller one in FP64 with an odd step count
        _case("colliding_256_mixed", 256, "8,8,8", "20,20,20", 0.65, 4, "mixed", 200, collision=True),
        _case("colliding_37_fp64", 37, "8,8,8", "20,20,20", 0.65, 4, "fp64", 33, collision=True),
        # robots that swim by cilia (the option that drives cell-based robots), self-colliding
        _case("cilia_64_mixed", 64, "5,5,4", "9,9,7", 0.85, 2, "mixed", 100, collision=True, cilia=True, actuated=False,
              phases=False),
        # optimisation by gradient: one robot's phases and moduli, and a colliding batch
        _case("gradient_12x12x6", 1, "12,12,6", "12,12,6", 1.0, 1, "fp64", 200, kind="gradient", checkpoint=100),
        _case("gradient_colliding_12", 12, "8,8,8", "14,14,14", 0.65, 4, "fp64", 60, kind="gradient", checkpoint=25,
              collision=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# voxel-steps of one drawn pass at most: below the largest listed case of its precision and kind
_BUDGET = {"mixed": 1.2e8, "fp64": 5e6, "gradient": 6e5}


def draw(rng):
    kind = rng.choice(["population", "population", "population", "body", "gradient"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    fill = round(rng.uniform(0.55, 1.0), 3)
    if kind == "body":
        dims = [_log_int(rng, 12, 60) for _ in range(3)]
        text = "%d,%d,%d" % tuple(dims)
        cells, robots, lo, hi = dims[0] * dims[1] * dims[2] * fill, 1, text, text
        if precision == "fp64" and cells > 60000:
            precision = "mixed"
    else:
        a = rng.randint(3, 8)
        b = a + rng.randint(1, 12)
        robots = _log_int(rng, 1, 24 if kind == "gradient" else 900 if precision == "mixed" else 200)
        cells, lo, hi = robots * ((a + b) / 2.0) ** 3 * fill, "%d,%d,%d" % (a, a, a), "%d,%d,%d" % (b, b, b)
    if kind == "gradient":
        precision = "fp64"
    most = _BUDGET["gradient" if kind == "gradient" else precision] / cells
    steps = max(1, min(_log_int(rng, 20, 200), int(most)))
    kw = dict(collision=rng.random() < 0.5, phases=rng.random() < 0.7, drop=rng.choice([0, 0, 1]))
    if kind == "gradient":
        kw.update(kind="gradient", checkpoint=rng.choice([10, 25, 50, 100]))
    elif kind == "population" and rng.random() < 0.2:
        kw.update(cilia=True, collision=True, actuated=False, phases=False)
    c = _case("", robots, lo, hi, fill, rng.randint(1, 4), precision, steps, **kw)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs from the seed
def _largest_parts(masks):
    """The largest 6-connected part of every box of a [R, Z, Y, X] stack of masks."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = torch.from_numpy(masks).to(dev)
    cells = m[0].numel()
    lab = torch.arange(1, cells + 1, device=dev, dtype=torch.int32).view(m.shape[1:]).expand(m.shape) * m
    while True:
        before = lab
        for _ in range(8):
            new = lab.clone()
            for d in (1, 2, 3):
                n = lab.shape[d]
                a, b = new.narrow(d, 0, n - 1), new.narrow(d, 1, n - 1)
                x, y = lab.narrow(d, 0, n - 1), lab.narrow(d, 1, n - 1)
                torch.maximum(a, y, out=a)
                torch.maximum(b, x, out=b)
            lab = new * m
        if torch.equal(lab, before):
            break
    flat = lab.view(lab.shape[0], -1).long()
    count = torch.zeros(flat.shape[0], cells + 1, dtype=torch.int32, device=dev)
    count.scatter_add_(1, flat, torch.ones_like(flat, dtype=torch.int32))
    count[:, 0] = 0
    best = count.argmax(1, keepdim=True)
    return ((flat == best) & (best > 0)).view(m.shape).cpu().numpy()


def _robots(case, seed):
    """The case's robots.  Their shapes belong to the case (a search varies what is in a set of
    bodies, and outputs of one case have one shape); palettes, moduli, densities, phases, cilia
    and weights come from the seed."""
    shape = repr([case[k] for k in ("robots", "lo", "hi", "fill", "materials")])
    shapes, rng = np.random.default_rng(zlib.crc32(shape.encode())), np.random.default_rng([int(seed), 20240911])
    lo = [int(x) for x in case["lo"].split(",")]
    hi = [int(x) for x in case["hi"].split(",")]
    R = case["robots"]
    dims = np.stack([shapes.integers(a, b + 1, size=R) for a, b in zip(lo, hi)], 1)
    big = dims.max(0)
    masks = shapes.random((R, big[2], big[1], big[0])) < case["fill"]
    for r in range(R):  # a robot's own box
        masks[r, dims[r, 2]:], masks[r, :, dims[r, 1]:], masks[r, :, :, dims[r, 0]:] = False, False, False
        masks[r, 0, 0, 0] = True
    masks = _largest_parts(masks)
    palette = rng.integers(1, case["materials"] + 1, size=masks.shape).astype(np.uint8)
    out = []
    for r in range(R):
        X, Y, Z = (int(x) for x in dims[r])
        grid = np.ascontiguousarray(masks[r, :Z, :Y, :X] * palette[r, :Z, :Y, :X])
        mats = []
        for k in range(case["materials"]):
            E = float(10 ** rng.uniform(5, 7)) if R > 1 else 1e6
            cte = 0.01 if case["actuated"] and (R > 1 or k > 0 or case["materials"] == 1) else 0.0
            mats.append(wl.Material(E=E, nu=0.35, rho=1e3, cte=cte, cilia=1.0 if case["cilia"] else 0.0))
        kw = dict(z_offset=case["drop"], enable_collision=case["collision"])
        if case["actuated"]:
            kw.update(temp_vary=True, temp_amplitude=AMPLITUDE, temp_period=PERIOD)
        if case["phases"]:
            kw["phase"] = rng.random((Z, Y, X))
        elif case["actuated"]:  # in step, about to contract (half a period in)
            kw["phase"] = np.full((Z, Y, X), rng.uniform(0.5, 0.55))
        if case["kind"] == "gradient":
            kw["log10E"] = rng.uniform(5, 7, size=(Z, Y, X))
        if case["cilia"]:
            kw.update(enable_cilia=True, cilia_base=rng.uniform(-0.02, 0.02, size=(Z, Y, X, 3)))
        if R == 1 and not case["phases"] and not case["actuated"]:
            # a lone passive block falls at a speed of its own
            kw["grav_acc"] = -9.81 * float(rng.uniform(0.8, 1.2))
            mats = [wl.Material(**{**m.__dict__, "rho": 1e3 * float(rng.uniform(0.8, 1.2))}) for m in mats]
        out.append(wl.Robot(grid=grid, materials=mats, **kw))
    return out


def _weights(case, seed):
    """dL/d(centre of mass at the end), per robot."""
    return np.random.default_rng([int(seed), 77]).normal(size=(case["robots"], 3))


def prepare(case, seed):
    robots = _robots(case, seed)
    b = abi.Batch(robots, abi.PRECISION_FP64 if case["precision"] == "fp64" else abi.PRECISION_MIXED)
    comps = (("pos", 3), ("orient", 4), ("linmom", 3), ("angmom", 3))
    pinned = {k: torch.zeros((b.nv, n), dtype=torch.float64, pin_memory=True) for k, n in comps}
    return dict(batch=b, case=case, pinned=pinned, out={k: t.numpy() for k, t in pinned.items()},
                weights=_weights(case, seed))


def run(state):
    b, case = state["batch"], state["case"]
    if case["kind"] == "gradient":
        b.record(case["steps"], case["checkpoint"])
        dphase, dlog10E = b.backward(state["weights"])
        return dict(dphase=dphase, dlog10E=dlog10E, **b.state(out=state["out"]))
    b.step(case["steps"])
    return dict(com=b.com(), **b.state(out=state["out"]))


def work(case):
    """The state read once and written once a pass (13 doubles a voxel; 9 values of local state,
    two strains and the flags a link), the constants read once, and the arithmetic of every step:
    about 400 operations a link, 260 a voxel, 30 a candidate pair of a surface voxel (some 12
    each) and, for a gradient, three times the step again."""
    lo = [int(x) for x in case["lo"].split(",")]
    hi = [int(x) for x in case["hi"].split(",")]
    cells = case["robots"] * math.prod((a + b) / 2.0 for a, b in zip(lo, hi))
    voxels = cells * case["fill"]
    links = 3 * cells * case["fill"] ** 2 * 0.92
    real = 8 if case["precision"] == "fp64" else 4
    bytes_ = voxels * (2 * 13 * 8 + 13 * 8 + 24) + links * (2 * 9 * real + 2 * 8 + 24)
    flops = case["steps"] * (400 * links + 260 * voxels + (360 * voxels if case["collision"] else 0))
    if case["kind"] == "gradient":
        bytes_ += 2 * 8 * voxels
        flops *= 4
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------ the step in 64-bit torch
# toAxisX: the bond's own frame, whose +x points along the bond (axis 0, 1, 2)
_PERM = [[0, 1, 2], [1, 0, 2], [2, 1, 0]]
_SIGN = [[1, 1, 1], [1, -1, 1], [1, 1, -1]]


def _conj(q):
    return torch.cat([q[:, :1], -q[:, 1:]], 1)


def _mul(a, b):
    w1, v1, w2, v2 = a[:, :1], a[:, 1:], b[:, :1], b[:, 1:]
    return torch.cat([w1 * w2 - (v1 * v2).sum(1, keepdim=True), w1 * v2 + w2 * v1 + torch.linalg.cross(v1, v2)], 1)


def _turn(q, v):
    """q v q* of a unit quaternion, in the product form (no assumption that |q| is exactly 1)."""
    return _mul(_mul(q, torch.cat([torch.zeros_like(v[:, :1]), v], 1)), _conj(q))[:, 1:]


def _rotation_vector(q):
    w, v = q[:, :1], q[:, 1:]
    sq = 1 - w * w
    near = sq < 2.4e-3  # the model's own small-angle form
    ws = torch.where(near, w, torch.ones_like(w))
    wl_ = torch.where(near, torch.zeros_like(w), w)
    g = torch.where(near, 2 * torch.sqrt(2 / (1 + ws)), 2 * torch.acos(wl_) / torch.sqrt(1 - wl_ * wl_))
    return v * g


def _from_rotation_vector(r):
    th = r / 2
    m2 = (th * th).sum(1, keepdim=True)
    tiny = m2 * m2 < 5.328e-15
    m = torch.sqrt(torch.where(tiny, torch.ones_like(m2), m2))
    w = torch.where(tiny, 1 - 0.5 * m2, torch.cos(m))
    s = torch.where(tiny, 1 - m2 / 6, torch.sin(m) / m)
    return torch.cat([w, th * s], 1)


def _to_pos_x(p):
    """The rotation that takes p to +x."""
    x, y, z = p[:, :1], p[:, 1:2], p[:, 2:]
    yx, zx = y / x, z / x
    small = (yx.abs() < 1.732e-2) & (zx.abs() < 1.732e-2)
    qy, qz = 0.5 * zx, -0.5 * yx
    q1 = torch.cat([1 - 0.5 * (qy * qy + qz * qz), torch.zeros_like(x), qy, qz], 1)
    n = p / p.norm(dim=1, keepdim=True)
    one = torch.ones_like(x)
    nx = torch.where(small, torch.zeros_like(x), n[:, :1]).clamp(-1, 1)
    h = 0.5 * torch.acos(nx)
    ai = 1 / torch.where(small, one, torch.sqrt(n[:, 1:2] ** 2 + n[:, 2:] ** 2).clamp_min(1e-300))
    s = torch.sin(h) * ai
    q2 = torch.cat([torch.cos(h), torch.zeros_like(x), n[:, 2:] * s, -n[:, 1:2] * s], 1)
    back = torch.tensor([0.0, 0.0, 1.0, 0.0], dtype=p.dtype, device=p.device)
    q2 = torch.where(2 * h > 3.14159265358979 - 1e-7, back, q2)
    return torch.where(small, q1, q2)


def _f32(x):
    """x rounded to 32 bits where the model stores 32 bits; the derivative passes through."""
    return x + (x.float().double() - x).detach()


class _Model:
    """The batch in 64 bits: topology and constants of every voxel and link."""

    def __init__(self, robots, dev, differentiate):
        f = np.float64
        pos, mat, phase, le, cil, robot, ends, axis, ijk = [], [], [], [], [], [], [], [], []
        base = 0
        self.nr = len(robots)
        for r, R in enumerate(robots):
            Z, Y, X = R.grid.shape
            g = R.grid > 0
            idx = np.full(g.shape, -1, np.int64)
            idx[g] = base + np.arange(g.sum())
            z, y, x = np.nonzero(g)
            n = len(z)
            ijk.append(np.stack([x, y, z + R.z_offset], 1))
            pos.append(ijk[-1].astype(f) * R.vox_size)
            robot.append(np.full(n, r))
            mat.append(np.array([(m.E, m.cte, m.rho, m.cilia) for m in R.materials], f)[R.grid[g] - 1])
            phase.append(R.phase[g] if R.phase is not None else np.zeros(n))
            le.append(R.log10E[g] if R.log10E is not None else np.zeros(n))
            cil.append(R.cilia_base[g] if R.cilia_base is not None else np.zeros((n, 3)))
            for a, d in ((0, 2), (1, 1), (2, 0)):
                lo, hi = np.moveaxis(idx, d, 0)[:-1], np.moveaxis(idx, d, 0)[1:]
                k = (lo >= 0) & (hi >= 0)
                ends.append(np.stack([lo[k], hi[k]], 1))
                axis.append(np.full(int(k.sum()), a))
            base += n
        t = lambda a, dt=torch.float64: torch.as_tensor(np.concatenate(a), device=dev).to(dt)  # noqa: E731
        self.pos0, self.robot, self.ends, self.axis = t(pos), t(robot, torch.int64), t(ends, torch.int64), t(axis, torch.int64)
        self.ijk = t(ijk, torch.int64)
        m = t(mat)
        R0 = robots[0]
        self.R0, self.dev = R0, dev
        self.nv, self.nl = self.pos0.shape[0], self.ends.shape[0]
        self.phase, self.log10E = t(phase), t(le)
        if differentiate:
            self.phase.requires_grad_(True)
            self.log10E.requires_grad_(True)
        E = _f32(10.0 ** self.log10E) if R0.log10E is not None else _f32(m[:, 0])
        self.E, self.cte, rho = E, _f32(m[:, 1]), _f32(m[:, 2])
        self.cilia, self.cil = m[:, 3:4], t(cil)
        L = R0.vox_size
        nu0 = float(np.float32(0.35))
        ehat = lambda e, n: e / ((1 - 2 * n) * (1 + n))  # noqa: E731
        self.mass = _f32(L ** 3 * rho)
        self.mom = _f32(self.mass * L * L / 6)
        zc, zi, zg = R0.col_damping, R0.bond_damping, R0.slow_damping
        self.c_glob = _f32(zg * 2 * torch.sqrt(_f32(self.mass * E) * L))
        self.c_rot = _f32(zg * 2 * torch.sqrt(_f32(self.mom * E) * L ** 3))
        self.c_col = _f32(zc * 2 * torch.sqrt(_f32(self.mass * E) * L))
        grav = torch.tensor([float(np.float32(-np.float32(r.grav_acc) / 9.80665)) for r in robots], dtype=torch.float64,
                            device=dev)
        self.weight = _f32(-self.mass * float(np.float32(9.80665)) * grav[self.robot])
        self.stiff = _f32(2 * E * L)
        self.dmc = _f32(2 * torch.sqrt(self.mass) * zi)
        e0, e1 = self.ends[:, 0], self.ends[:, 1]
        En, Ep = E[e0], E[e1]
        El = _f32(2 * En * Ep / (En + Ep))
        hn, hp = ehat(En, nu0), ehat(Ep, nu0)
        hl = 2 * hn * hp / (hn + hp)
        nu = _f32(torch.sqrt((hl - El) / (2 * hl) + 0.0625) - 0.25).detach()  # both ends' ratio is one and the same
        Lf = float(np.float32(L))
        self.nu, self.eHat = nu, _f32(ehat(El, nu))
        self.a2 = _f32(El * Lf ** 3 / (12 * (1 + nu)))
        self.b1, self.b2, self.b3 = _f32(El * Lf), _f32(El * Lf ** 2 / 2), _f32(El * Lf ** 3 / 6)
        self.sqA1, self.sqB1 = torch.sqrt(El * Lf), torch.sqrt(self.b1)
        self.sqA2, self.sqB2 = torch.sqrt(self.a2 * Lf * Lf / 6), torch.sqrt(self.b2 * Lf / 2)
        self.sqB3 = torch.sqrt(self.b3 * Lf * Lf / 6)
        self.area = float(np.float32(Lf) ** 2)
        self.perm = torch.tensor(_PERM, device=dev)[self.axis]
        self.sign = torch.tensor(_SIGN, device=dev, dtype=torch.float64)[self.axis]
        # the voxel's link in each of its six directions, nl for none
        self.slot = torch.full((self.nv, 6), self.nl, dtype=torch.int64, device=dev)
        ln = torch.arange(self.nl, device=dev)
        self.slot[e0, 2 * self.axis] = ln
        self.slot[e1, 2 * self.axis + 1] = ln
        self.surface = (self.slot == self.nl).any(1)
        # the stable time step of every robot, then its stored 32 bits
        self.bs0 = self.base_size(torch.zeros(self.nr, dtype=torch.float64, device=dev))
        rest = 0.5 * (self.bs0[e0] + self.bs0[e1])
        k = (self.eHat * self.area / rest).float().double()
        f2 = torch.zeros(self.nr, dtype=torch.float64, device=dev)
        f2.scatter_reduce_(0, self.robot[e0], (k / torch.minimum(self.mass[e0], self.mass[e1])).detach(), "amax")
        lone = torch.zeros_like(f2).scatter_reduce_(0, self.robot, (E * L / self.mass).detach(), "amax")
        f2 = torch.where(f2 > 0, f2, lone)
        self.dt = (R0.dt_frac / (float(np.float32(6.283185)) * torch.sqrt(f2))).float().double()

    def base_size(self, t):
        R = self.R0
        if not R.temp_vary:
            return torch.full((self.nv,), R.vox_size, dtype=torch.float64, device=self.dev)
        T = R.temp_amplitude * torch.sin(float(np.float32(2 * np.float32(3.1415926))) * (t[self.robot] / R.temp_period + self.phase))
        T = torch.minimum(T, torch.zeros_like(T)) if not R.enable_expansion else T
        return R.vox_size * _f32(1 + _f32(T) * self.cte)

    def to_x(self, v):
        return v.gather(1, self.perm) * self.sign

    def from_x(self, v):
        return (v * self.sign).gather(1, self.perm)

    def quat_x(self, q):
        return torch.cat([q[:, :1], self.to_x(q[:, 1:])], 1)


def _pairs(m, pos, reach):
    """Pairs (later, earlier) of unlinked surface voxels of one robot within `reach` of each other."""
    s = torch.nonzero(m.surface)[:, 0]
    p = pos[s].detach()
    c = torch.floor((p - p.min(0).values) / reach).long() + 1
    n = c.max(0).values + 2
    key = ((m.robot[s] * n[0] + c[:, 0]) * n[1] + c[:, 1]) * n[2] + c[:, 2]
    key, order = torch.sort(key)
    s, p = s[order], p[order]
    found = []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                k = key + (dx * n[1] + dy) * n[2] + dz
                a, b = torch.searchsorted(key, k), torch.searchsorted(key, k, right=True)
                count = b - a
                i = torch.repeat_interleave(torch.arange(len(s), device=s.device), count)
                first = torch.cumsum(count, 0) - count
                j = a[i] + torch.arange(len(i), device=s.device) - first[i]
                ok = (s[i] > s[j]) & ((p[i] - p[j]).norm(dim=1) <= reach) & (m.robot[s[i]] == m.robot[s[j]])
                found.append(torch.stack([s[i[ok]], s[j[ok]]], 1))
    pr = torch.cat(found)
    d = (m.ijk[pr[:, 0]] - m.ijk[pr[:, 1]]).abs().sum(1)
    return pr[d != 1]  # face neighbours are linked


def _steps(m, n):
    """n steps from rest; the state after them."""
    R, dev = m.R0, m.dev
    z3 = torch.zeros(m.nv, 3, dtype=torch.float64, device=dev)
    pos, lin, ang = m.pos0.clone(), z3, z3
    q = torch.cat([torch.ones_like(z3[:, :1]), z3], 1)
    bs = m.bs0
    lz = torch.zeros(m.nl, 3, dtype=torch.float64, device=dev)
    old, oldA1, oldA2 = lz, lz, lz
    small = torch.ones(m.nl, dtype=torch.bool, device=dev)
    valid = torch.zeros(m.nl, dtype=torch.bool, device=dev)
    stat = torch.ones(m.nv, dtype=torch.bool, device=dev)
    t = torch.zeros(m.nr, dtype=torch.float64, device=dev)
    e0, e1 = m.ends[:, 0], m.ends[:, 1]
    dt = m.dt[m.robot][:, None]
    minv, iinv = (1 / m.mass).float().double()[:, None], (1 / m.mom).float().double()[:, None]
    mu_s, mu_k = (float(np.float32(x)) for x in (R.materials[0].mu_static, R.materials[0].mu_kinetic))
    L = R.vox_size
    cutoff, margin = 1.25 * L * 1.0001, 0.5 * L
    pairs, built = None, None
    X, Y, Z = 0, 1, 2
    for _ in range(n):
        # the beam links
        p = m.to_x(pos[e1] - pos[e0])
        c = _conj(m.quat_x(q[e0]))
        rest = 0.5 * (bs[e0] + bs[e1])
        p = _turn(c, p)
        A = _mul(c, m.quat_x(q[e1]))
        turn = (p[:, Z].abs() + p[:, Y].abs()) / p[:, X]
        ext = (1 - p[:, X] / rest).abs()
        get = ~small & (turn < 0.05) & (ext < 0.5)
        lose = small & ((turn > 0.06) | (ext > 0.6))
        small = (small | get) & ~lose
        valid = valid & ~get & ~lose
        sm = small[:, None]
        ident = torch.zeros_like(A)
        ident[:, 0] = 1
        if bool(small.all()):
            B1, B2 = ident, A
            pos2 = torch.cat([p[:, :1] - rest[:, None], p[:, 1:]], 1)
        else:
            B1 = torch.where(sm, ident, _to_pos_x(torch.where(sm, torch.tensor([1.0, 0.5, 0.0], dtype=p.dtype, device=dev), p)))
            B2 = torch.where(sm, A, _mul(B1, A))
            far = torch.cat([p.norm(dim=1, keepdim=True) - rest[:, None], torch.zeros_like(p[:, 1:])], 1)
            pos2 = torch.where(sm, torch.cat([p[:, :1] - rest[:, None], p[:, 1:]], 1), far)
        a1 = torch.zeros_like(p) if bool(small.all()) else torch.where(sm, torch.zeros_like(p), _rotation_vector(B1))
        a2 = _rotation_vector(B2)
        dP, d1, d2 = 0.5 * (pos2 - old), 0.5 * (a1 - oldA1), 0.5 * (a2 - oldA2)
        old, oldA1, oldA2 = pos2, a1, a2
        eps = pos2[:, X] / rest
        f0 = m.eHat * (1 - m.nu) * eps * m.area
        fN = torch.stack([f0, m.b1 * pos2[:, Y] - m.b2 * (a1[:, Z] + a2[:, Z]), m.b1 * pos2[:, Z] + m.b2 * (a1[:, Y] + a2[:, Y])], 1)
        fP = -fN
        mN = torch.stack([m.a2 * (a2[:, X] - a1[:, X]), -m.b2 * pos2[:, Z] - m.b3 * (2 * a1[:, Y] + a2[:, Y]),
                          m.b2 * pos2[:, Y] - m.b3 * (2 * a1[:, Z] + a2[:, Z])], 1)
        mP = torch.stack([m.a2 * (a1[:, X] - a2[:, X]), -m.b2 * pos2[:, Z] - m.b3 * (a1[:, Y] + 2 * a2[:, Y]),
                          m.b2 * pos2[:, Y] - m.b3 * (a1[:, Z] + 2 * a2[:, Z])], 1)
        k = valid.double()[:, None] / m.dt[m.robot[e0]][:, None]
        kN, kP = k * m.dmc[e0][:, None], k * m.dmc[e1][:, None]
        pc = torch.stack([m.sqA1 * dP[:, X], m.sqB1 * dP[:, Y] - m.sqB2 * (d1[:, Z] + d2[:, Z]),
                          m.sqB1 * dP[:, Z] + m.sqB2 * (d1[:, Y] + d2[:, Y])], 1)
        uN = torch.stack([-m.sqA2 * (d2[:, X] - d1[:, X]), m.sqB2 * dP[:, Z] + m.sqB3 * (2 * d1[:, Y] + d2[:, Y]),
                          -m.sqB2 * dP[:, Y] + m.sqB3 * (2 * d1[:, Z] + d2[:, Z])], 1)
        uP = torch.stack([m.sqA2 * (d2[:, X] - d1[:, X]), m.sqB2 * dP[:, Z] + m.sqB3 * (d1[:, Y] + 2 * d2[:, Y]),
                          -m.sqB2 * dP[:, Y] + m.sqB3 * (d1[:, Z] + 2 * d2[:, Z])], 1)
        fN, fP = fN + kN * pc, fP - kP * pc
        mN, mP = mN - 0.5 * kN * uN, mP - 0.5 * kP * uP
        valid = torch.ones_like(valid)
        iB1, iB2 = _conj(B1), _conj(B2)
        if not bool(small.all()):
            fN, mN = _turn(iB1, fN), _turn(iB1, mN)
        fP, mP = _turn(iB2, fP), _turn(iB2, mP)
        sN = torch.cat([m.from_x(fN), m.from_x(mN)], 1)
        sP = torch.cat([m.from_x(fP), m.from_x(mP)], 1)
        none = torch.zeros(1, 6, dtype=torch.float64, device=dev)
        sN, sP = torch.cat([sN, none]), torch.cat([sP, none])
        S = sum(sN[m.slot[:, 2 * a]] + sP[m.slot[:, 2 * a + 1]] for a in range(3))
        # contacts of the state the step starts with
        contact = z3
        vel = lin * minv
        if R.enable_collision:
            if pairs is None or float((pos.detach() - built).norm(dim=1).max()) > 0.49 * margin:
                pairs, built = _pairs(m, pos, cutoff + margin), pos.detach().clone()
            with torch.no_grad():
                reach = 0.625 * (bs[pairs[:, 0]] + bs[pairs[:, 1]])
                hit = pairs[(pos[pairs[:, 1]] - pos[pairs[:, 0]]).norm(dim=1) < reach]
            u, v = hit[:, 0], hit[:, 1]
            off = pos[v] - pos[u]
            dist = off.norm(dim=1, keepdim=True)
            un = off / dist
            rel = 0.625 * (bs[u] + bs[v])[:, None] - dist
            ks = (2 / (1 / m.stiff[u] + 1 / m.stiff[v]))[:, None]
            cs = (0.5 * (m.c_col[u] + m.c_col[v]))[:, None]
            f = un * (ks * rel + cs * ((vel[u] - vel[v]) * un).sum(1, keepdim=True))
            contact = z3.index_add(0, u, f).index_add(0, v, -f)
        # the voxels
        F = _turn(q, S[:, :3]) - vel * m.c_glob[:, None]
        F = F + torch.stack([torch.zeros_like(m.weight), torch.zeros_like(m.weight), m.weight], 1) - contact
        if R.enable_cilia:
            F = F + torch.where(m.surface[:, None], _turn(q, m.cil) * m.cilia, z3)
        pen = bs / 2 - L / 2 - pos[:, Z]
        on = pen >= 0
        normal = m.stiff * pen * on
        Fz = torch.where(on, normal - m.c_col * vel[:, Z], torch.zeros_like(pen))
        free = F
        F = F + torch.stack([torch.zeros_like(Fz), torch.zeros_like(Fz), Fz], 1)
        slip = on & stat & ((F[:, X] ** 2 + F[:, Y] ** 2).detach() > (mu_s * normal.detach()) ** 2)
        kin = on & ~stat
        h2 = vel[:, X] ** 2 + vel[:, Y] ** 2
        moving = h2 > 0
        h = torch.sqrt(torch.where(moving, h2, torch.ones_like(h2)))
        drag = torch.where((kin & moving)[:, None], vel[:, :2] / h[:, None], torch.zeros_like(vel[:, :2]))
        F = F - torch.cat([drag * (mu_k * normal)[:, None], torch.zeros_like(Fz)[:, None]], 1)
        stat = on & stat & ~slip
        fric = (F - free).detach()
        lin = lin + F * dt
        tr = lin * (dt * minv)
        with torch.no_grad():
            wk = fric[:, X] * tr[:, X] + fric[:, Y] * tr[:, Y]
            ke = 0.5 * minv[:, 0] * (lin[:, X] ** 2 + lin[:, Y] ** 2)
            stat = on & (stat | (ke + wk <= 0))
            # resting without a normal force or momentum: any push frees it (the gradient's side of the kink)
            held = stat & ~((normal == 0) & (lin[:, X] == 0) & (lin[:, Y] == 0))
        keep = torch.stack([~held, ~held, torch.ones_like(held)], 1).double()
        lin, tr = lin * keep, tr * keep
        pos = pos + tr
        M = _turn(q, S[:, 3:]) - ang * iinv * m.c_rot[:, None]
        ang = ang + M * dt
        q = _mul(_from_rotation_vector(ang * (dt * iinv)), q)
        still = stat & ((bs / 2 - L / 2 - pos[:, Z]).detach() >= 0)
        still_g = held & still
        ang = ang * (~still_g).double()[:, None]
        ang = torch.where((still & ~still_g)[:, None], ang - ang.detach(), ang)
        t = t + m.dt
        bs = m.base_size(t)
    return pos, q, lin, ang


def exact(case, seed):
    """The outputs of a first pass on these inputs."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    robots = _robots(case, seed)
    grad = case["kind"] == "gradient"
    m = _Model(robots, dev, grad)
    with torch.set_grad_enabled(grad):
        pos, q, lin, ang = _steps(m, case["steps"])
        mass = m.mass.detach()[:, None]
        total = torch.zeros(m.nr, 1, dtype=torch.float64, device=dev).index_add(0, m.robot, mass)
        com = torch.zeros(m.nr, 3, dtype=torch.float64, device=dev).index_add(0, m.robot, pos * mass) / total
    out = dict(pos=pos.detach(), orient=q.detach(), linmom=lin.detach(), angmom=ang.detach())
    if grad:
        w = torch.as_tensor(_weights(case, seed), device=dev)
        gp, ge = torch.autograd.grad((w * com).sum(), [m.phase, m.log10E], allow_unused=True)
        zero = torch.zeros(m.nv, dtype=torch.float64, device=dev)
        out.update(dphase=zero if gp is None else gp, dlog10E=zero if ge is None else ge)
    else:
        out["com"] = com.detach()
    return out
