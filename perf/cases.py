"""What a program does with this package, as cases of one size each: a substep of one cloth, of self-contacting
cloth, of batches of cloths and of soft bodies, and a differentiated rollout.

A pass is one substep as a simulation loop calls it (``CollisionPipeline.collide`` and ``SolverVBD.step``) from
start positions that the program writes into the state, or one gradient of a short rollout
(``DifferentiableVBD.rollout`` and ``backward``). A model (topology, materials, pins, shapes) belongs to its case;
positions, velocities, moduli and targets come from the seed. ``exact`` is the same substep in 64 bits, written
with torch operations over whole color groups from the model's arrays.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

import newton_chysx_b200 as nb
from newton_chysx_b200.adjoint import DifferentiableVBD

DT = 1.0 / 600.0  # ten substeps of a 60 Hz frame
MARGIN = 0.01  # particle-shape contact margin
SOFT = (1.0e4, 1.0e-4, 0.5)  # contact stiffness, damping and friction of the models and of their shapes
SC_RADIUS, SC_MARGIN = 2.0e-3, 3.5e-3


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest program: one 32 x 32 cloth, where launches and latency count
        _sheet("cloth_32", 32, 32),
        # an ordinary prop: an odd-sized cloth lying over four kinds of shapes
        _sheet("cloth_161x97_shapes", 161, 97, shapes="four"),
        # one fine cloth over a sphere, twenty iterations, no self-contact
        _sheet("cloth_256_sphere", 256, 256, iterations=20, shapes="sphere"),
        # a stiff sheet with a stiffness ratio of 1e3, FP64 solves where the FP32 block is ill-conditioned
        _sheet("cloth_512_mixed", 512, 512, iterations=30, precision="mixed", stiff=True),
        # all-FP64 runs, as used to check a scene
        _sheet("cloth_96_fp64", 96, 96, precision="fp64", shapes="sphere"),
        # two layers of cloth in self-contact, one model (garment layers)
        _self_contact("layers_176", 1, 176),
        # many small layered cloths with self-contact
        _self_contact("layers_16_x512", 512, 16),
        # a small batch with the default options, hinges and membranes damped
        _batch("batch_60_damped", 60, 16, 40, damped=True),
        # a large batch of uneven sizes with the launch shape that the autotuner picks for it
        _batch("batch_512", 512, 16, 128, tuned=True),
        # a batch of soft blocks hung on springs over the ground
        _soft("blocks_x1024", 1024, 8, 4, 4),
        # one large soft block
        _soft("block_28x16x16", 1, 28, 16, 16),
        # a gradient through two substeps: moduli of every triangle and initial velocities of a curtain
        _gradient("gradient_64", 64, 64, substeps=2),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("sheet", "sheet", "sheet", "self_contact", "batch", "batch", "soft", "gradient"))
    if kind == "sheet":
        precision = rng.choice(("fp32", "fp32", "fp32", "mixed", "fp64"))
        return _sheet(None, log(16, 300), log(16, 300), iterations=rng.choice((5, 10, 20)), precision=precision,
                      shapes=rng.choice(("ground", "sphere", "four")), damped=rng.random() < 0.3,
                      stiff=rng.random() < 0.3)  # fmt: skip
    if kind == "self_contact":
        worlds = rng.choice((1, log(2, 400)))
        return _self_contact(None, worlds, log(16, 160) if worlds == 1 else log(8, min(40, int(360 / worlds**0.5))),
                             iterations=rng.choice((5, 10, 20)))  # fmt: skip
    if kind == "batch":
        lo = log(8, 60)
        hi = log(lo, 128)
        return _batch(None, log(2, 300), lo, hi, tuned=rng.random() < 0.4, damped=rng.random() < 0.3)
    if kind == "soft":
        worlds = rng.choice((1, log(2, 800)))
        most = 20 if worlds == 1 else 7
        return _soft(None, worlds, log(2, most), log(2, most), log(2, most))
    return _gradient(None, log(12, 64), log(12, 64), substeps=rng.choice((1, 2)))


def _named(name, case):
    return case if name is None else dict(name=name, **case)


def _sheet(name, nx, ny, iterations=10, precision="fp32", shapes="ground", damped=False, stiff=False):
    return _named(name, dict(kind="sheet", nx=nx, ny=ny, iterations=iterations, precision=precision, shapes=shapes,
                             damped=damped, stiff=stiff))  # fmt: skip


def _self_contact(name, worlds, n, iterations=20):
    return _named(name, dict(kind="self_contact", worlds=worlds, n=n, iterations=iterations, precision="fp32"))


def _batch(name, worlds, lo, hi, tuned=False, damped=False):
    return _named(name, dict(kind="batch", worlds=worlds, lo=lo, hi=hi, iterations=10, precision="fp32", tuned=tuned,
                             damped=damped))  # fmt: skip


def _soft(name, worlds, cx, cy, cz):
    return _named(name, dict(kind="soft", worlds=worlds, cx=cx, cy=cy, cz=cz, iterations=10, precision="fp32"))


def _gradient(name, nx, ny, substeps):
    return _named(name, dict(kind="gradient", nx=nx, ny=ny, iterations=10, precision="fp32", substeps=substeps))


# ------------------------------------------------------------------------------------------------ the models
def _cfg():
    return nb.ModelBuilder.ShapeConfig(ke=SOFT[0], kd=SOFT[1], mu=SOFT[2])


def _grid(nx, ny, pos=(0.0, 0.0, 0.0), rot=None, longest=1.0, damped=False, bend=1.0e-4, E=1.0e4):
    """A builder with one nx x ny cloth, its longer side `longest` m: E = 1e4 Pa, nu = 0.3, 1 mm, 0.2 kg/m^2."""
    nu, h, cell = 0.3, 1.0e-3, longest / (max(nx, ny) - 1)
    b = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
    b.add_cloth_grid(pos=pos, rot=rot or nb.quat_identity(), vel=(0.0, 0.0, 0.0), dim_x=nx - 1, dim_y=ny - 1,
                     cell_x=cell, cell_y=cell, mass=0.2 * cell * cell, tri_ke=E * h / (2.0 * (1.0 + nu)),
                     tri_ka=E * h * nu / (1.0 - nu * nu), tri_kd=1.0e-3 if damped else 0.0, edge_ke=bend,
                     edge_kd=1.0e-3 if damped else 0.0, particle_radius=2.0e-3)  # fmt: skip
    return b


def _pin(b, vertices):
    flags = b.particle_flags
    flags[np.asarray(vertices, dtype=np.int64)] = 0
    b.set_particle_flags(flags)


def _shapes(case):
    """The shapes of a sheet: (kind, centre, quaternion, sizes)."""
    ident = (0.0, 0.0, 0.0, 1.0)
    q = nb.quat_from_axis_angle((0.2, 1.0, 0.3), 0.6)
    ground, sphere = ("plane", (0.0, 0.0, 0.0), ident, ()), ("sphere", (0.0, 0.0, 0.1), ident, (0.3,))
    if case.get("shapes") == "sphere":
        return [ground, sphere]
    if case.get("shapes") == "four":
        return [ground, ("sphere", (0.2, 0.1, 0.055), ident, (0.15,)), ("box", (-0.2, -0.1, 0.08), q, (0.12, 0.1, 0.06)),
                ("capsule", (-0.15, 0.18, 0.07), q, (0.05, 0.1))]  # fmt: skip
    return [ground]


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


def _builder(case):
    return _cached_builder(_key(case))


@functools.lru_cache(maxsize=24)
def _cached_builder(key):
    case = dict(key)
    rng = np.random.default_rng(7)
    kind = case["kind"]
    if kind == "sheet":
        nx, ny = case["nx"], case["ny"]
        cell = 1.0 / (max(nx, ny) - 1)
        b = _grid(nx, ny, (-0.5 * cell * (nx - 1), -0.5 * cell * (ny - 1), 0.0), damped=case["damped"])
        if case["stiff"]:
            mats = b.tri_materials
            mats[:, :2] *= (10.0 ** rng.uniform(1.0, 4.0, len(mats)))[:, None]  # E log-uniform in [1e5, 1e8] Pa
            b._tri_mat = [mats]
        _pin(b, [nx * (ny - 1), nx * ny - 1])
        for what, p, q, size in _shapes(case):
            if what == "plane":
                b.add_ground_plane(cfg=_cfg())
            elif what == "sphere":
                b.add_shape_sphere(xform=(p, q), radius=size[0], cfg=_cfg())
            elif what == "box":
                b.add_shape_box(xform=(p, q), hx=size[0], hy=size[1], hz=size[2], cfg=_cfg())
            else:
                b.add_shape_capsule(xform=(p, q), radius=size[0], half_height=size[1], cfg=_cfg())
        b.color(include_bending=True)
        return b
    if kind == "self_contact":
        n, worlds = case["n"], case["worlds"]
        side = 176 / 256 if worlds == 1 else 0.25
        cloth = _grid(n, n, (-0.5 * side, -0.5 * side, 0.0), longest=side)
        turned = _grid(n, n, (-0.5 * side, -0.5 * side, 0.0), longest=side)
        two = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
        c, s = math.cos(math.radians(17.0)), math.sin(math.radians(17.0))
        for k, one in enumerate((cloth, turned)):
            q = one.particle_q
            if k:
                q = np.stack([c * q[:, 0] - s * q[:, 1] + 0.4 * side, s * q[:, 0] + c * q[:, 1] + 0.3 * side, q[:, 2]], 1)
            start = two.add_particles(q, (0.0, 0.0, 0.0), one.particle_mass, radius=2.0e-3)
            t = one.tri_indices + start
            m = one.tri_materials
            two.add_triangles(t[:, 0], t[:, 1], t[:, 2], m[:, 0], m[:, 1], m[:, 2])
            e, p = one.edge_indices + np.where(one.edge_indices >= 0, start, 0), one.edge_bending_properties
            two.add_edges(e[:, 0], e[:, 1], e[:, 2], e[:, 3], edge_ke=p[:, 0], edge_kd=p[:, 1])
        two.color(include_bending=True)
        if worlds == 1:
            two.add_ground_plane(cfg=_cfg())
            return two
        b = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
        k = int(math.ceil(math.sqrt(worlds)))
        for w in range(worlds):  # worlds 0.5 m apart around the origin
            b.add_world(two)
            b._q[-1] = b._q[-1] + np.array([0.5 * (w % k - 0.5 * k), 0.5 * (w // k - 0.5 * k), 0.0])
        b.add_ground_plane(cfg=_cfg())
        return b
    if kind == "batch":
        b = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
        templates = {}
        for n in rng.integers(case["lo"], case["hi"] + 1, size=case["worlds"]):
            n = int(n)
            if n not in templates:
                templates[n] = _grid(n, n, damped=case["damped"])
                templates[n].color(include_bending=True)
            one = templates[n]
            b.add_world(one)
            E, bend = 10.0 ** rng.uniform(3.0, 6.0), 10.0 ** rng.uniform(-5.0, -3.0)
            b._tri_mat[-1] = b._tri_mat[-1] * np.array([E / 1e4, E / 1e4, 1.0, 1.0, 1.0])
            b._edge_prop[-1] = b._edge_prop[-1] * np.array([bend / 1e-4, 1.0])
            flags = b._flags[-1].copy()
            flags[rng.choice((0, n - 1, n * (n - 1), n * n - 1), size=int(rng.integers(1, 5)), replace=False)] = 0
            b._flags[-1] = flags
        b.add_ground_plane(cfg=_cfg())
        return b
    if kind == "soft":
        nx, ny, nz = case["cx"] + 1, case["cy"] + 1, case["cz"] + 1
        one = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
        one.add_soft_grid(pos=(0.0, 0.0, 0.0), rot=nb.quat_identity(), vel=(0.0, 0.0, 0.0), dim_x=nx - 1, dim_y=ny - 1,
                          dim_z=nz - 1, cell_x=0.02, cell_y=0.02, cell_z=0.02, density=500.0, k_mu=2.0e4,
                          k_lambda=3.0e4, k_damp=1.0e-3, particle_radius=2.0e-3)  # fmt: skip
        top = nx * ny * (nz - 1)
        anchor = one.add_particle((0.01 * nx, 0.01 * ny, 0.02 * nz + 0.4), (0.0, 0.0, 0.0), 0.0, 2.0e-3)
        for corner in (top, top + nx - 1, top + nx * (ny - 1), top + nx * ny - 1):
            one.add_spring(anchor, corner, 50.0, 1.0e-2, 0.0)
        one.color()
        if case["worlds"] == 1:
            one.add_ground_plane(cfg=_cfg())
            return one
        b = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
        for _ in range(case["worlds"]):
            b.add_world(one)
        b.add_ground_plane(cfg=_cfg())
        return b
    # gradient: a curtain, its top row pinned
    nx, ny = case["nx"], case["ny"]
    b = _grid(nx, ny, rot=nb.quat_from_axis_angle((1.0, 0.0, 0.0), math.pi * 0.5), bend=1.0e-2)
    _pin(b, range(nx * (ny - 1), nx * ny))
    b.color(include_bending=True)
    return b


def _model(case, device="cuda"):
    m = _builder(case).finalize(device)
    m.soft_contact_ke, m.soft_contact_kd, m.soft_contact_mu = SOFT
    return m


# ------------------------------------------------------------------------------------------------ the inputs
def _waves(gen, uv, group, groups, amplitude, count=4):
    """Smooth random displacements of points uv ([N, 2], in units of the cloth's side): per group `count` plane waves
    of 1 to 3 periods."""
    dev = uv.device
    out = torch.zeros((len(uv), 3), dtype=torch.float64, device=dev)
    for _ in range(count):
        k = torch.randint(-3, 4, (groups, 2), generator=gen, device=dev).double()
        phase = torch.rand((groups, 1), generator=gen, device=dev, dtype=torch.float64) * (2.0 * math.pi)
        a = torch.randn((groups, 3), generator=gen, device=dev, dtype=torch.float64)
        arg = 2.0 * math.pi * (uv * k[group]).sum(1, keepdim=True) + phase[group]
        out += torch.sin(arg) * a[group]
    return out * torch.tensor(amplitude, dtype=torch.float64, device=dev) / math.sqrt(count)


def _sdf(shape, x):
    """Signed distance and outward normal of points x to a shape (kind, centre, quaternion, sizes)."""
    kind, p, q, size = shape
    if kind == "plane":
        return x[:, 2] - p[2], torch.tensor([0.0, 0.0, 1.0], dtype=x.dtype, device=x.device).expand(len(x), 3)
    R = torch.as_tensor(nb.sim.quat_to_matrix(q), dtype=x.dtype, device=x.device)
    y = (x - torch.tensor(p, dtype=x.dtype, device=x.device)) @ R
    if kind == "box":
        h = torch.tensor(size, dtype=x.dtype, device=x.device)
        a = y.abs() - h
        out = a.clamp(min=0.0)
        dist = out.norm(dim=1)
        inside = a.max(dim=1)
        face = torch.nn.functional.one_hot(inside.indices, 3).to(x.dtype) * torch.where(y < 0, -1.0, 1.0)
        far = y - torch.minimum(torch.maximum(y, -h), h)
        n = torch.where((dist > 0)[:, None], far / dist.clamp(min=1e-300)[:, None], face)
        return torch.where(dist > 0, dist, inside.values), n @ R.T
    if kind == "capsule":
        y = torch.cat([y[:, :2], (y[:, 2] - y[:, 2].clamp(-size[1], size[1]))[:, None]], 1)
    l = y.norm(dim=1).clamp(min=1e-12)
    return l - size[0], (y / l[:, None]) @ R.T


def _inputs(case, seed):
    """Start positions and velocities (float32 values, as float64) of one pass."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    b = _builder(case)
    q = torch.as_tensor(b.particle_q, device=dev)
    n = len(q)
    starts = list(b.world_particle_start) or [0]
    world = torch.zeros(n, dtype=torch.long, device=dev)
    world[torch.tensor(starts[1:], dtype=torch.long, device=dev)] = 1
    world = world.cumsum(0)
    W = len(starts)
    local = q - q[torch.tensor(starts, device=dev)][world]
    kind = case["kind"]
    v = _waves(gen, local[:, :2], world, W, (0.3, 0.3, 0.5)) + torch.tensor([0.0, 0.0, -0.5], dtype=q.dtype, device=dev)
    if kind == "gradient":
        q = q + _waves(gen, local[:, [0, 2]], world, W, (2e-3, 1e-2, 2e-3))
        v = _waves(gen, local[:, [0, 2]], world, W, (0.1, 0.1, 0.1))
    elif kind == "soft":
        lift = 1.5e-3 + 2.0e-3 * torch.rand((W, 1), generator=gen, device=dev, dtype=q.dtype)
        heavy = (torch.as_tensor(b.particle_mass, device=dev) > 0)[:, None]
        scale = torch.tensor((8.0, 8.0), dtype=q.dtype, device=dev)
        q = torch.where(heavy, q + lift[world] + _waves(gen, local[:, :2] * scale, world, W, (8e-4, 8e-4, 4e-4)), q)
        v = torch.where(heavy, v, torch.zeros_like(v))
    elif kind == "self_contact":
        # a lower cloth near the ground and an upper one settling on it: gaps from just under the contact radius up
        side = 176 / 256 if W == 1 else 0.25
        per = n // W // 2
        upper = (torch.arange(n, device=dev) % (2 * per) >= per)[:, None]
        uv = local[:, :2] / side
        h = 5.0e-3 + 1.0e-3 * side * _waves(gen, uv, world, W, (0.0, 0.0, 1.0))[:, 2]
        gap = 3.2e-3 + 1.2e-3 * torch.sin(_waves(gen, uv, world, W, (0.0, 0.0, 2.0))[:, 2])
        z = h.clamp(min=1.99e-3) + torch.where(upper[:, 0], gap, torch.zeros_like(gap))
        flat = _waves(gen, uv, world * 2 + upper[:, 0].long(), 2 * W, (3.0e-5 * side, 3.0e-5 * side, 0.0))
        q = q + flat + torch.stack([torch.zeros_like(z), torch.zeros_like(z), z], 1)
        q = q + 1.0e-6 * torch.randn(q.shape, generator=gen, device=dev, dtype=q.dtype)
        v = 0.01 * v + torch.tensor([0.5, 0.0, 0.0], dtype=q.dtype, device=dev)
        v[:, 2] -= 0.02 * upper[:, 0]
    else:
        # a sheet under slight tension with wrinkles, just above its shapes
        amplitude = 2e-5 if case.get("stiff") else 5e-5
        q = q + 1e-2 * local + _waves(gen, local[:, :2], world, W, (amplitude, amplitude, 2e-3))
        q[:, 2] += {"sphere": 0.401, "four": 0.201}.get(case.get("shapes"), 4.0e-3)
        for shape in _shapes(case):  # pushed out of the shapes up to a small penetration
            d, nrm = _sdf(shape, q)
            depth = 3.0e-4 * torch.rand(n, generator=gen, device=dev, dtype=q.dtype)
            q = q + (2.0e-3 - depth - d).clamp(min=0.0)[:, None] * nrm
    return q.float().double(), v.float().double()


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    m = _model(case)
    q, v = _inputs(case, seed)
    if s.kind == "gradient":
        s.sim = DifferentiableVBD(m, iterations=case["iterations"])
        s.q0, s.v0 = q.float(), v.float()
        s.mu, s.lam, s.target = _gradient_inputs(m.tri_count, q, seed)
        s.substeps = case["substeps"]
        return s
    kw = {}
    if s.kind == "self_contact":
        kw = dict(particle_enable_self_contact=True, particle_self_contact_radius=SC_RADIUS,
                  particle_self_contact_margin=SC_MARGIN)  # fmt: skip
    elif case.get("tuned"):
        kw = dict(layout="ell16", lanes_per_vertex=1, positions_in_shared="off", min_blocks_per_sm=3,
                  schedule="persistent")  # fmt: skip
    s.solver = nb.SolverVBD(m, iterations=case["iterations"], precision=case["precision"], **kw)
    s.pipe = nb.CollisionPipeline(m, soft_contact_margin=MARGIN)
    s.contacts = s.pipe.contacts()
    s.a, s.b, s.seen = m.state(), m.state(), m.state()
    for st in (s.a, s.b):
        if case["precision"] == "fp64":
            st.particle_f = None
            st.particle_q, st.particle_qd = st.particle_q.double(), st.particle_qd.double()
    s.f64 = case["precision"] == "fp64"
    s.q = q if s.f64 else q.float()
    s.a.particle_qd.copy_(v)
    return s


def _gradient_inputs(tri_count, q, seed):
    gen = torch.Generator(device=q.device)
    gen.manual_seed(int(seed) + 1)
    E = 10.0 ** (3.5 + torch.rand(tri_count, generator=gen, device=q.device, dtype=torch.float64))
    nu, h = 0.3, 1.0e-3
    target = q + 0.05 * torch.randn(q.shape, generator=gen, device=q.device, dtype=torch.float64)
    return (E * (h / (2.0 * (1.0 + nu)))).float(), (E * (h * nu / (1.0 - nu * nu))).float(), target.float()


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    if s.kind == "gradient":
        mu, lam = s.mu.detach().requires_grad_(), s.lam.detach().requires_grad_()
        v0 = s.v0.detach().requires_grad_()
        q, qd = s.sim.rollout(s.q0, v0, mu, lam, DT, s.substeps)
        loss = ((q - s.target) ** 2).sum(dim=1).mean()
        g = torch.autograd.grad(loss, (mu, lam, v0))
        return {"q": q.detach(), "qd": qd.detach(), "loss": loss.detach(), "mu": g[0], "lambda": g[1], "v0": g[2]}
    s.a.particle_q.copy_(s.q)
    view = s.a
    if s.f64:  # contact generation reads FP32 positions
        s.seen.particle_q.copy_(s.a.particle_q)
        view = s.seen
    s.pipe.collide(view, s.contacts)
    s.solver.step(s.a, s.b, None, s.contacts, DT)
    return {"q": s.b.particle_q, "qd": s.b.particle_qd}


def work(case):
    """Bytes: the model's arrays and the start state read once, positions and velocities written once. Operations: the
    element terms of every vertex in every iteration (a membrane term of one vertex 130, a hinge 150, a tetrahedron
    220, a block solve 90; a gradient does each term again for the state and about three times over for its
    derivatives)."""
    b = _builder(case)
    V, T, E, NT, NS = b.particle_count, b.tri_count, b.edge_count, b.tet_count, b.spring_count
    live = 0 if case["kind"] == "soft" else 1  # a soft block's surface has no stiffness of its own
    real = 8 if case["precision"] == "fp64" else 4
    size = V * (16 + 15 * real) + live * (T * 44 + E * 32) + NT * 64 + NS * 20
    flops = case["iterations"] * (live * (3 * T * 130 + 4 * E * 150) + 4 * NT * 220 + 2 * NS * 40 + V * 90)
    if case["kind"] == "gradient":
        flops *= 5 * case["substeps"]
        size += V * 12 * 4 + T * 16
    return {"bytes": size, "flops": flops}


def tolerance(case):
    # velocities are differences of positions over dt: FP32 rounding of a position is 1e-5 to 1e-4 of them
    if case["precision"] == "fp64":
        return {"rel": 1e-9, "max": 1e-6}
    if case["kind"] == "self_contact":  # a plane or a contact that just cuts in moves single vertices by some 0.1 mm
        return {"rel": 1e-2, "max": 0.95}
    if case["kind"] in ("soft", "gradient"):
        return {"rel": 3e-4, "max": 2e-3}
    # a vertex that comes out of or into contact, or buckles, amplifies rounding: 6e-3 measured at worst on a sphere
    return {"rel": 2e-2, "max": 0.95}


# ------------------------------------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    m = _model(case)
    q, v = _inputs(case, seed)
    sim = _Exact(case, m)
    if case["kind"] == "gradient":
        mu, lam, target = (x.double() for x in _gradient_inputs(m.tri_count, q, seed))
        mu.requires_grad_(), lam.requires_grad_()
        v.requires_grad_()
        x, u = q, v
        for _ in range(case["substeps"]):
            x, u = sim.step(x, u, mu, lam)
        loss = ((x - target) ** 2).sum(dim=1).mean()
        g = torch.autograd.grad(loss, (mu, lam, v))
        return {"q": x.detach(), "qd": u.detach(), "loss": loss.detach(), "mu": g[0], "lambda": g[1], "v0": g[2]}
    with torch.no_grad():
        x, u = sim.step(q, v, sim.mu, sim.lam)
    return {"q": x, "qd": u}


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _outer(a, s=None):
    return (a[..., :, None] if s is None else (a * s)[..., :, None]) * a[..., None, :]


class _Exact:
    """The vertex block descent substep over color groups: all vertices of a color from the positions at its start."""

    def __init__(self, case, m):
        self.case = case
        self.iterations = case["iterations"]
        d = lambda t: t.to(torch.float64)  # noqa: E731
        self.V = V = m.particle_count
        self.mass, self.flags, self.radius = d(m.particle_mass), m.particle_flags, d(m.particle_radius)
        self.moves = ((self.flags & 1) != 0) & (self.mass > 0)
        self.g = d(m.gravity)[0]
        self.tri, self.pose = m.tri_indices.long(), d(m.tri_poses)
        self.mu, self.lam, self.tri_kd = (d(m.tri_materials[:, k]) for k in range(3))
        self.area = d(m.tri_areas)
        self.edge = m.edge_indices.long()
        self.rest = d(m.edge_rest_angle)
        prop = d(m.edge_bending_properties)
        self.ke, self.ekd = prop[:, 0] * d(m.edge_rest_length), prop[:, 1]
        self.tet, self.dm, self.tet_mat = m.tet_indices.long(), d(m.tet_poses), d(m.tet_materials)
        self.spring = m.spring_indices.long().reshape(-1, 2)
        self.spring_prop = torch.stack([d(m.spring_rest_length), d(m.spring_stiffness), d(m.spring_damping)], 1)
        live = self._rows(V, self.tri, (self.mu > 0) | (self.lam > 0))
        hinges = self._rows(V, self.edge, (self.ke > 0) & (self.edge[:, 0] >= 0) & (self.edge[:, 1] >= 0))
        tets = self._rows(V, self.tet, (self.tet_mat[:, 0] > 0) | (self.tet_mat[:, 1] > 0))
        springs = self._rows(V, self.spring, torch.ones(len(self.spring), dtype=torch.bool, device=self.tri.device))
        self.colors = []
        for group in m.particle_color_groups:
            verts = group.long()
            place = torch.full((V,), -1, dtype=torch.long, device=verts.device)
            place[verts] = torch.arange(len(verts), device=verts.device)
            self.colors.append((verts, place, *(tuple(x[place[r[0]] >= 0] for x in r) for r in (live, hinges, tets, springs))))
        self.shapes = _shapes(case) if case["kind"] != "gradient" else []

    @staticmethod
    def _rows(V, elements, keep):
        """(vertex, element, order) of every vertex of the kept elements."""
        e = keep.nonzero()[:, 0]
        k = elements.shape[1]
        return elements[e].reshape(-1), e.repeat_interleave(k), torch.arange(k, device=e.device).repeat(len(e))

    # -- element terms of one vertex each: (force, Hessian)
    def membrane(self, x, xp, t, order, mu, lam):
        p, pp = x[self.tri[t]], xp[self.tri[t]]
        D = self.pose[t]
        F = torch.stack([p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]], 2) @ D  # columns f0, f1
        f0, f1 = F[:, :, 0], F[:, :, 1]
        mu, lam, A = mu[t][:, None], lam[t][:, None], self.area[t][:, None]
        f00, f11, f01 = _dot(f0, f0), _dot(f1, f1), _dot(f0, f1)
        J = (f00 * f11 - f01 * f01).clamp(min=1e-20).sqrt()
        lnh = lam + mu
        s = lnh * (J - (1.0 + mu / lnh))
        sel = torch.tensor([[-1.0, -1.0], [1.0, 0.0], [0.0, 1.0]], dtype=x.dtype, device=x.device)[order]
        dd = (sel[:, None, :] @ D)[:, 0]
        d0, d1 = dd[:, :1], dd[:, 1:]
        g0, g1 = (f11 * f0 - f01 * f1) / J, (f00 * f1 - f01 * f0) / J  # dJ/df0, dJ/df1
        dJ = g0 * d0 + g1 * d1
        force = -A * ((mu * f0 + s * g0) * d0 + (mu * f1 + s * g1) * d1)
        w = f1 * d0 - f0 * d1
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        r = (A * s.clamp(min=0.0) / J)[..., None]
        H = (A * mu * (d0 * d0 + d1 * d1))[..., None] * eye + (A * lnh)[..., None] * _outer(dJ)
        H = H + r * (_dot(w, w)[..., None] * eye - _outer(w) - _outer(dJ))
        if bool((self.tri_kd > 0).any()):
            kd = self.tri_kd[t][:, None]
            G00, G11, G01 = 0.5 * (f00 - 1.0), 0.5 * (f11 - 1.0), 0.5 * f01
            Gsq = G00 * G00 + G11 * G11 + 2.0 * G01 * G01
            on = (Gsq >= 1e-20).to(x.dtype)
            u = p - pp
            dF = torch.stack([u[:, 1] - u[:, 0], u[:, 2] - u[:, 0]], 2) @ D / DT
            e0, e1 = dF[:, :, 0], dF[:, :, 1]
            C = Gsq.clamp(min=1e-30).sqrt()
            n00, n01, n11 = G00 / C, G01 / C, G11 / C
            r00, r11, r01 = _dot(f0, e0), _dot(f1, e1), 0.5 * (_dot(f0, e1) + _dot(f1, e0))
            c = d0 * (n00 * f0 + n01 * f1) + d1 * (n01 * f0 + n11 * f1)
            l = d0 * f0 + d1 * f1
            km, kl = on * A * mu * kd, on * A * lam * kd
            force = force - km * (n00 * r00 + n11 * r11 + 2.0 * n01 * r01) * c - kl * (r00 + r11) * l
            H = H + _outer(c, km / DT) + _outer(l, kl / DT)
        return force, H

    def hinge(self, x, xp, e, order):
        p = x[self.edge[e]]
        x02, x03, x13, x12 = p[:, 2] - p[:, 0], p[:, 3] - p[:, 0], p[:, 3] - p[:, 1], p[:, 2] - p[:, 1]
        ed = p[:, 3] - p[:, 2]
        N1, N2, le = _cross(x02, x03), _cross(x13, x12), ed.norm(dim=1, keepdim=True)
        l1, l2 = N1.norm(dim=1, keepdim=True), N2.norm(dim=1, keepdim=True)
        on = ((l1 > 1e-6) & (l2 > 1e-6) & (le > 1e-6)).to(x.dtype)
        n1, n2, eh = N1 / l1.clamp(min=1e-12), N2 / l2.clamp(min=1e-12), ed / le.clamp(min=1e-12)
        theta = torch.atan2(_dot(_cross(n1, n2), eh), _dot(n1, n2))
        a1, a2 = 1.0 / l1.clamp(min=1e-12), 1.0 / l2.clamp(min=1e-12)
        grads = torch.stack([-le * a1 * n1, -le * a2 * n2, _dot(x03, eh) * a1 * n1 + _dot(x13, eh) * a2 * n2,
                             -_dot(x02, eh) * a1 * n1 - _dot(x12, eh) * a2 * n2], 1)  # fmt: skip
        dt = grads[torch.arange(len(e), device=e.device), order]
        k = on * self.ke[e][:, None]
        force = -k * (theta - self.rest[e][:, None]) * dt
        hk = k
        if bool((self.ekd > 0).any()):
            rate = (grads * (p - xp[self.edge[e]])).sum((1, 2))[:, None] / DT
            c = k * self.ekd[e][:, None]
            force = force - c * rate * dt
            hk = k + c / DT
        return force, _outer(dt, hk)

    def tetrahedron(self, x, xp, t, order):
        p, pp, D = x[self.tet[t]], xp[self.tet[t]], self.dm[t]
        mu, lam, kd = (self.tet_mat[t][:, k : k + 1] for k in range(3))
        vol = (1.0 / (6.0 * torch.linalg.det(D)))[:, None]
        F = torch.stack([p[:, k] - p[:, 0] for k in (1, 2, 3)], 2) @ D
        F0, F1, F2 = F.unbind(2)
        cof = torch.stack([_cross(F1, F2), _cross(F2, F0), _cross(F0, F1)], 2)
        J = _dot(F0, cof[:, :, 0])
        lnh = lam + mu
        s = lnh * (J - (1.0 + mu / lnh))
        rows = torch.cat([-D.sum(1, keepdim=True), D], 1)
        mrow = rows[torch.arange(len(t), device=t.device), order]
        Fm, gg = (F @ mrow[..., None])[..., 0], (cof @ mrow[..., None])[..., 0]
        force = -vol * (mu * Fm + s * gg)
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        H = (vol * mu * _dot(mrow, mrow))[..., None] * eye + _outer(gg, vol * lnh)
        u = p - pp
        dF = torch.stack([u[:, k] - u[:, 0] for k in (1, 2, 3)], 2) @ D / DT
        rate = (cof * dF).sum((1, 2))[:, None]
        force = force - kd * vol * (mu * (dF @ mrow[..., None])[..., 0] + lnh * rate * gg)
        return force, (1.0 + kd / DT)[..., None] * H

    def spring_term(self, x, xp, k, end):
        a, b = self.spring[k, 0], self.spring[k, 1]
        rest, ke, kd = (self.spring_prop[k][:, j : j + 1] for j in range(3))
        diff = x[a] - x[b]
        l = diff.norm(dim=1, keepdim=True).clamp(min=1e-8)
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        H = (ke * (1.0 - rest / l))[..., None] * eye + _outer(diff, ke * rest / l**3)
        sign = torch.where(end == 0, 1.0, -1.0)[:, None].to(x.dtype)
        own = torch.where(end == 0, a, b)
        force = sign * (ke * (rest - l) / l) * diff + (kd / DT) * (H @ (xp[own] - x[own])[..., None])[..., 0]
        return force, (1.0 + kd / DT)[..., None] * H

    def contact_terms(self, x, xp, contacts, f, H, place):
        """Penalty, damping and friction of the particle-shape contacts found at the substep's start."""
        for p, point, nrm in contacts:
            j = place[p]
            on = j >= 0
            p, point, nrm, j = p[on], point[on], nrm[on], j[on]
            pen = self.radius[p][:, None] - _dot(nrm, x[p] - point)
            on = (pen > 0).to(x.dtype)
            rel = x[p] - xp[p]
            rn = _dot(nrm, rel)
            fn = pen * SOFT[0]
            damp = torch.where(rn < 0, SOFT[1] * SOFT[0] / DT, 0.0)
            ut = rel - nrm * rn
            un = ut.norm(dim=1, keepdim=True)
            eps = 1e-2 * DT
            f1 = torch.where(un > eps, 1.0 / un.clamp(min=1e-300), (2.0 - un / eps) / eps)
            fr = SOFT[2] * fn * f1 * (un > 0)
            eye = torch.eye(3, dtype=x.dtype, device=x.device)
            f.index_add_(0, j, on * (nrm * (fn - damp * rn) - fr * ut))
            H.index_add_(0, j, on[..., None] * (_outer(nrm, SOFT[0] + damp - fr) + fr[..., None] * eye))

    def find_contacts(self, q):
        found = []
        for shape in self.shapes:
            d, nrm = _sdf(shape, q)
            p = ((d < MARGIN + self.radius) & ((self.flags & 1) != 0)).nonzero()[:, 0]
            found.append((p, q[p] - nrm[p] * d[p][:, None], nrm[p]))
        return found

    def block(self, color, x, xp, y, mu, lam, contacts, extra=None):
        """The moves H^-1 f of the color's vertices."""
        verts, place, tris, hinges, tets, springs = color
        md = torch.where(self.moves, self.mass, 0.0)[verts][:, None] / (DT * DT)
        f = md * (y[verts] - x[verts])
        H = md[..., None] * torch.eye(3, dtype=x.dtype, device=x.device)
        terms = []
        if len(tris[0]):
            terms.append((tris[0], self.membrane(x, xp, tris[1], tris[2], mu, lam)))
        if len(hinges[0]):
            terms.append((hinges[0], self.hinge(x, xp, hinges[1], hinges[2])))
        if len(tets[0]):
            terms.append((tets[0], self.tetrahedron(x, xp, tets[1], tets[2])))
        if len(springs[0]):
            terms.append((springs[0], self.spring_term(x, xp, springs[1], springs[2])))
        for v, (df, dH) in terms:
            f, H = f.index_add(0, place[v], df), H.index_add(0, place[v], dH)
        if contacts:
            self.contact_terms(x, xp, contacts, f, H, place)
        if extra is not None:
            extra(x, xp, f, H, place)
        on = self.moves[verts] & (torch.linalg.det(H).abs() > 1e-8)
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        move = torch.linalg.solve(torch.where(on[:, None, None], H, eye), f[..., None])[..., 0]
        return torch.where(on[:, None], move, torch.zeros_like(move))

    def step(self, q, v, mu, lam):
        if self.case["kind"] == "self_contact":
            return self.step_self_contact(q, v, mu, lam)
        contacts = self.find_contacts(q) if self.shapes else []
        u = (v + self.g * DT) * DT
        y = x = torch.where(self.moves[:, None], q + u, q)
        for _ in range(self.iterations):
            for color in self.colors:
                x = x.index_add(0, color[0], self.block(color, x, q, y, mu, lam, contacts))
        return x, (x - q) / DT

    # -- self-contact
    def step_self_contact(self, q, v, mu, lam):
        contacts = self.find_contacts(q)
        u = torch.where(self.moves[:, None], (v + self.g * DT) * DT, torch.zeros_like(v))
        y = q + u
        pairs = self.find_pairs(q)
        d = self.truncated(q, u, pairs)
        base = q + d
        pairs = self.find_pairs(base)
        d = torch.zeros_like(d)
        for _ in range(self.iterations):
            for color in self.colors:
                x = base + d
                extra = functools.partial(self.pair_terms, pairs)
                d = d.index_add(0, color[0], self.block(color, x, q, y, mu, lam, contacts, extra))
                d = self.truncated(base, d, pairs)
        x = base + d
        return x, (x - q) / DT

    def near(self, points, others, reach):
        """Index pairs (i, j) of points and others closer than `reach` (at least)."""
        lo = torch.minimum(points.min(0).values, others.min(0).values) - 2 * reach
        a, b = ((points - lo) / reach).long(), ((others - lo) / reach).long()
        span = torch.maximum(a.max(0).values, b.max(0).values) + 2
        key = lambda c: (c[:, 0] * span[1] + c[:, 1]) * span[2] + c[:, 2]  # noqa: E731
        sorted_keys, order = key(b).sort()
        got = []
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dz in (-1, 0, 1):
                    k = key(a + torch.tensor([dx, dy, dz], device=a.device))
                    first = torch.searchsorted(sorted_keys, k)
                    count = torch.searchsorted(sorted_keys, k, right=True) - first
                    i = torch.arange(len(k), device=k.device).repeat_interleave(count)
                    within = torch.arange(len(i), device=k.device) - (count.cumsum(0) - count)[i]
                    j = order[first[i] + within]
                    on = (points[i] - others[j]).square().sum(1) <= reach * reach
                    got.append(torch.stack([i[on], j[on]], 1))
        return torch.cat(got)

    def close_ids(self, a, b):
        """Whether vertices a and b are the same or the ends of one edge of the mesh."""
        if not hasattr(self, "links"):
            e = self.edge[:, 2:]
            self.links = torch.cat([e[:, 0] * self.V + e[:, 1], e[:, 1] * self.V + e[:, 0]]).unique()
        key = a * self.V + b
        at = torch.searchsorted(self.links, key).clamp(max=len(self.links) - 1)
        return (a == b) | (self.links[at] == key)

    def find_pairs(self, x):
        """Vertex ids of the vertex-triangle pairs (t0, t1, t2, v) and edge-edge pairs (a0, a1, b0, b1) within the
        margin, neighbours over one edge left out; at most 32 and 64 per vertex and edge, those of lowest index."""
        t = x[self.tri]
        mid = t.mean(1)
        reach = SC_MARGIN + float((t - mid[:, None]).norm(dim=2).max())
        vt = self.near(x, mid, reach)
        tri = self.tri[vt[:, 1]]
        far = ~(self.close_ids(vt[:, 0], tri[:, 0]) | self.close_ids(vt[:, 0], tri[:, 1]) | self.close_ids(vt[:, 0], tri[:, 2]))
        vt, tri = vt[far], tri[far]
        p = x[vt[:, 0]]
        bary = _closest_on_triangle(x[tri[:, 0]], x[tri[:, 1]], x[tri[:, 2]], p)
        dist = ((x[tri] * bary[..., None]).sum(1) - p).norm(dim=1)
        on = self.lowest(vt, dist < SC_MARGIN, 32)
        vt_ids = torch.cat([tri[on], vt[on][:, :1]], 1)
        e = self.edge[:, 2:]
        p = x[e]
        mid = p.mean(1)
        reach = SC_MARGIN + float((p[:, 0] - p[:, 1]).norm(dim=1).max())
        ee = self.near(mid, mid, reach)
        ids = torch.cat([e[ee[:, 0]], e[ee[:, 1]]], 1)
        far = torch.ones(len(ee), dtype=torch.bool, device=x.device)
        for i in (0, 1):
            for j in (2, 3):
                far &= ~self.close_ids(ids[:, i], ids[:, j])
        ee, ids = ee[far], ids[far]
        s, r = _closest_on_segments(*(x[ids[:, k]] for k in range(4)), 1e-5)
        c1, c2 = _mix(x, ids[:, 0], ids[:, 1], s), _mix(x, ids[:, 2], ids[:, 3], r)
        on = self.lowest(ee, (c1 - c2).norm(dim=1) < SC_MARGIN, 64)
        return vt_ids, ids[on]

    def lowest(self, pairs, on, most):
        """Indices of the pairs that are `on`, at most `most` per first index, lowest second index first."""
        k = on.nonzero()[:, 0]
        k = k[(pairs[k, 0] * (pairs.max() + 1) + pairs[k, 1]).argsort()]
        i = pairs[k, 0]
        first = torch.searchsorted(i, i)
        return k[torch.arange(len(k), device=k.device) - first < most]

    def pair_terms(self, pairs, x, xp, f, H, place):
        vt, ee = pairs
        on = (place[vt] >= 0).any(1)
        vt = vt[on]
        p, pp = x[vt], xp[vt]
        bary = _closest_on_triangle(p[:, 0], p[:, 1], p[:, 2], p[:, 3])
        weight = torch.cat([-bary, torch.ones_like(bary[:, :1])], 1)
        sign = torch.tensor([-1.0, -1.0, -1.0, 1.0], dtype=x.dtype, device=x.device)
        self.barrier(vt, p, pp, weight, sign, 4, f, H, place)
        ee = ee[(place[ee[:, :2]] >= 0).any(1)]
        p, pp = x[ee], xp[ee]
        s, r = _closest_on_segments(p[:, 0], p[:, 1], p[:, 2], p[:, 3], 1e-5)
        weight = torch.cat([1.0 - s, s, r - 1.0, -r], 1)
        sign = torch.ones(4, dtype=x.dtype, device=x.device)
        self.barrier(ee, p, pp, weight, sign, 2, f, H, place)

    def barrier(self, ids, p, pp, weight, sign, slots, f, H, place):
        diff = (weight[..., None] * p).sum(1)
        dist = diff.norm(dim=1, keepdim=True)
        on = ((dist > 0) & (dist < SC_RADIUS)).to(p.dtype)
        n = diff / dist.clamp(min=1e-300)
        ke, kd, fmu = SOFT
        tau, small = 0.5 * SC_RADIUS, 1.0e-5
        k2 = tau * tau * ke
        g = torch.where(dist < tau, -k2 / dist.clamp(min=small), -ke * (SC_RADIUS - dist))
        h = torch.where(dist < tau, k2 / dist.clamp(min=small) ** 2, torch.full_like(dist, ke))
        g = torch.where(dist <= small, k2 * (dist - 2 * small) / small**2, g)
        u = (weight[..., None] * (p - pp)).sum(1)
        ut = u - n * _dot(n, u)
        un = ut.norm(dim=1, keepdim=True)
        eps = 1e-2 * DT
        f1 = torch.where(un > eps, 1.0 / un.clamp(min=1e-300), (2.0 - un / eps) / eps)
        fr = -fmu * g * f1 * (un > 0)
        eye = torch.eye(3, dtype=p.dtype, device=p.device)
        for k in range(slots):
            j = place[ids[:, k]]
            mine = (j >= 0) & (on[:, 0] > 0)
            w, nn = weight[mine, k : k + 1], n[mine]
            back = (pp - p)[mine, k]
            hn = h[mine] * w * w
            nb_ = _dot(nn, back)
            damp = torch.where(nb_ * sign[k] > 0, kd / DT, 0.0) * hn
            f.index_add_(0, j[mine], -g[mine] * w * nn + damp * nb_ * nn - w * fr[mine] * ut[mine])
            tangent = fr[mine][..., None] * (eye - _outer(nn))
            H.index_add_(0, j[mine], _outer(nn, hn + damp) + (w * w)[..., None] * tangent)

    def truncated(self, base, d, pairs):
        """Displacements cut at the planes that divide every pair, and at half the margin."""
        gamma = 0.85
        ts = torch.ones(self.V, dtype=d.dtype, device=d.device)
        vt, ee = pairs
        for ids, kind in ((vt[:, [3, 0, 1, 2]], "vt"), (ee, "ee")):
            if not len(ids):
                continue
            x, u = base[ids], d[ids]
            if kind == "vt":
                bary = _closest_on_triangle(x[:, 1], x[:, 2], x[:, 3], x[:, 0])
                c2 = (bary[..., None] * x[:, 1:]).sum(1)
                c1, one = x[:, 0], (0,)
            else:
                s, r = _closest_on_segments(x[:, 0], x[:, 1], x[:, 2], x[:, 3], 1e-6)
                c1, c2, one = x[:, 0] + (x[:, 1] - x[:, 0]) * s, x[:, 2] + (x[:, 3] - x[:, 2]) * r, (0, 1)
            two = tuple(k for k in range(4) if k not in one)
            nh = c1 - c2
            n = nh / nh.norm(dim=1, keepdim=True).clamp(min=1e-12)
            a1 = torch.stack([-_dot(n, u[:, k]) for k in one]).amax(0).clamp(min=0.0)
            a2 = torch.stack([_dot(n, u[:, k]) for k in two]).amax(0).clamp(min=0.0)
            l = torch.where(a1 + a2 == 0, 0.5, (a2 / (a1 + a2).clamp(min=1e-300)).clamp(0.05, 0.95))
            at = c2 + l * nh
            late = 1e-8 if kind == "vt" else 1e-6
            for k in range(4):
                speed = _dot(n, u[:, k])
                t = _dot(n, at - x[:, k]) / torch.where(speed == 0, 1.0, speed)
                cut = ((a1 if k in one else a2) > 0) & (speed.abs() >= 1e-6) & (t >= -1e-8) & (t <= 1.0 + late)
                cut &= speed.abs() >= 1e-5
                part = torch.where(t < 0, 1.0, torch.minimum(t * gamma, t - 1e-3).clamp(0.0, 1.0))
                ts.scatter_reduce_(0, ids[:, k][cut[:, 0]], part[cut], "amin")
        d = d * ts[:, None]
        most = SC_MARGIN * gamma * 0.5
        length = d.norm(dim=1, keepdim=True)
        return torch.where(length > most, d * most / length.clamp(min=1e-300), d)


def _mix(x, a, b, s):
    return x[a] + (x[b] - x[a]) * s


def _closest_on_triangle(a, b, c, p):
    """Barycentric weights of the point of triangle abc that is closest to p."""
    ab, ac = b - a, c - a
    d1, d2 = _dot(ab, p - a), _dot(ac, p - a)
    d3, d4 = _dot(ab, p - b), _dot(ac, p - b)
    d5, d6 = _dot(ab, p - c), _dot(ac, p - c)
    va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
    zero, one = torch.zeros_like(va), torch.ones_like(va)
    div = lambda u, w: u / torch.where(w == 0, one, w)  # noqa: E731
    total = va + vb + vc
    v, w = div(vb, total), div(vc, total)
    out = torch.cat([1 - v - w, v, w], 1)
    v = div(d4 - d3, (d4 - d3) + (d5 - d6))
    out = torch.where((va <= 0) & (d4 >= d3) & (d5 >= d6), torch.cat([zero, 1 - v, v], 1), out)
    v = div(d2, d2 - d6)
    out = torch.where((vb <= 0) & (d2 >= 0) & (d6 <= 0), torch.cat([1 - v, zero, v], 1), out)
    v = div(d1, d1 - d3)
    out = torch.where((vc <= 0) & (d1 >= 0) & (d3 <= 0), torch.cat([1 - v, v, zero], 1), out)
    out = torch.where((d6 >= 0) & (d5 <= d6), torch.cat([zero, zero, one], 1), out)
    out = torch.where((d3 >= 0) & (d4 <= d3), torch.cat([zero, one, zero], 1), out)
    return torch.where((d1 <= 0) & (d2 <= 0), torch.cat([one, zero, zero], 1), out)


def _closest_on_segments(p1, q1, p2, q2, eps):
    """Parameters of the closest points of segments p1 q1 and p2 q2. Squared lengths of at most eps count as points."""
    d1, d2, r = q1 - p1, q2 - p2, p1 - p2
    a, e, f, c, b = _dot(d1, d1), _dot(d2, d2), _dot(d2, r), _dot(d1, r), _dot(d1, d2)
    one = torch.ones_like(a)
    div = lambda u, w: u / torch.where(w == 0, one, w)  # noqa: E731
    den = a * e - b * b
    s = torch.where(den != 0, div(b * f - c * e, den).clamp(0, 1), torch.zeros_like(a))
    t = div(b * s + f, e)
    s = torch.where(t < 0, div(-c, a).clamp(0, 1), torch.where(t > 1, div(b - c, a).clamp(0, 1), s))
    t = t.clamp(0, 1)
    point1, point2 = a <= eps, e <= eps
    s = torch.where(point2, div(-c, a).clamp(0, 1), s)
    t = torch.where(point2, torch.zeros_like(t), t)
    t = torch.where(point1, torch.where(point2, torch.zeros_like(t), div(f, e).clamp(0, 1)), t)
    return torch.where(point1, torch.zeros_like(s), s), t
