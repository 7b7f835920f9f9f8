"""Instances split over several CTAs (vbd_parts.cu) against the FP64 oracle and against the kernels they replace, at the
edges of the rules that choose the split: one cluster and a grid, runs of one and two rounds, one to eight lanes per
vertex, pinned ghosts, damping, several contacts per particle, worlds merged into jobs, refreshed materials, capture.

Tolerances. FP64 sums in another order: 1e-9 m per substep, as the other FP64 kernels are held to. FP32 against FP64
over one substep: 1e-4 m per m, the bound of every FP32 kernel here; on the finest sheets (2.4 mm cells under
compression) the per-color FP32 kernel itself is 1.6e-4 m off, and the split one is held to twice that kernel's own
distance, the factor for another order of the same sums."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import newton_chysx_b200 as nb  # noqa: E402
from newton_chysx_b200 import CollisionPipeline, SolverVBD, _lib  # noqa: E402
from tests.helpers import cloth_grid_builder  # noqa: E402

DT = 1.0 / 600.0


def _sheet(nx, ny, kd=0.0, shapes=1):
    b = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
    cell = 1.0 / max(nx - 1, ny - 1)
    b.add_cloth_grid(pos=(0.0, 0.0, 4e-3), rot=nb.quat_identity(), vel=(0.0, 0.0, 0.0), dim_x=nx - 1, dim_y=ny - 1,
                     cell_x=cell, cell_y=cell, mass=0.2 * cell * cell, tri_ke=4.0, tri_ka=3.0, tri_kd=kd,
                     edge_ke=1e-4, edge_kd=kd, particle_radius=5e-3)  # fmt: skip
    flags = b.particle_flags
    flags[:: max(7, len(flags) // 9)] = 0  # pinned particles all over, so that some are ghosts
    b.set_particle_flags(flags)
    b.color(include_bending=True)
    cfg = nb.ModelBuilder.ShapeConfig(ke=1e4, kd=1e-4, mu=0.5)
    for k in range(shapes):
        b.add_ground_plane(height=-1e-4 * k, cfg=cfg)
    return b


def _start(model, seed):
    rng = np.random.default_rng(seed)
    q = model.particle_q.cpu().numpy().astype(np.float64)
    q = q * np.array([1.003, 1.002, 1.0]) + 2e-3 * np.sin(9.0 * q[:, [1, 0, 1]] + rng.uniform(0, 6, 3))
    qd = np.array([0.2, -0.1, -0.4]) + 0.1 * np.sin(7.0 * q[:, [1, 0, 0]])
    return q.astype(np.float32), qd.astype(np.float32)


def _run(model, q, qd, substeps=2, **kw):
    kw = dict(dict(iterations=6), **kw)
    solver = SolverVBD(model, **kw)
    f64 = kw.get("precision") == "fp64"
    pipe = CollisionPipeline(model, soft_contact_margin=0.01)
    contacts = pipe.contacts()
    s0, s1, seen = model.state(), model.state(), model.state()
    for s in (s0, s1):
        if f64:
            s.particle_f = None
            s.particle_q, s.particle_qd = s.particle_q.double(), s.particle_qd.double()
    s0.particle_q.copy_(torch.as_tensor(q))
    s0.particle_qd.copy_(torch.as_tensor(qd))
    for _ in range(substeps):
        seen.particle_q.copy_(s0.particle_q)
        pipe.collide(seen, contacts)
        solver.step(s0, s1, None, contacts, DT)
        s0, s1 = s1, s0
    torch.cuda.synchronize()
    assert solver.device_errors() == 0
    return s0.particle_q.double().cpu().numpy(), s0.particle_qd.double().cpu().numpy()


# 9 x 7: less than two CTAs' worth; 32 x 32: the largest cluster; 41 x 27: the first grid; 300 x 60: 148 CTAs with
# eight lanes; 320 x 160 and 411 x 260: four and two lanes; 700 x 801: one lane, runs longer than a CTA's threads
@pytest.mark.parametrize("nx,ny,kd,shapes,parts,lanes,grid", [
    (9, 7, 0.0, 1, 2, 8, False), (32, 32, 1e-3, 3, 16, 8, False), (41, 27, 0.0, 2, 18, 8, True),
    (300, 60, 1e-3, 1, 148, 8, True), (320, 160, 0.0, 1, 148, 4, True), (411, 260, 0.0, 1, 148, 2, True),
    (700, 801, 0.0, 1, 148, 1, True)])  # fmt: skip
def test_split_sheet_matches_the_per_color_kernels(nx, ny, kd, shapes, parts, lanes, grid):
    model = _sheet(nx, ny, kd, shapes).finalize("cuda:0")
    chosen = SolverVBD(model, iterations=6).split
    assert (chosen["parts"], chosen["lanes"], chosen["grid"], chosen["jobs"]) == (parts, lanes, grid, 1)
    model.soft_contact_ke, model.soft_contact_kd, model.soft_contact_mu = 1e4, 1e-4, 0.5
    q, qd = _start(model, nx)
    ref, ref_d = _run(model, q, qd, precision="fp64", schedule="per_color")
    got, got_d = _run(model, q, qd, precision="fp64")
    assert np.abs(got - ref).max() <= 1e-9 and np.abs(got_d - ref_d).max() <= 1e-9 / DT
    for precision in ("fp32", "mixed"):
        got, _ = _run(model, q, qd, substeps=1, precision=precision)
        old, _ = _run(model, q, qd, substeps=1, precision=precision, schedule="per_color")
        one, _ = _run(model, q, qd, substeps=1, precision="fp64", schedule="per_color")
        assert np.abs(got - one).max() <= max(1e-4, 2.0 * np.abs(old - one).max())


@pytest.mark.parametrize("sides", [(5, 6), (17, 30, 8, 9, 21), (40,) * 30, (100, 128, 16, 90) * 6])
def test_split_worlds_match_the_one_cta_kernel(sides):
    top = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
    for n in sides:
        top.add_world(_sheet(n, n, 1e-3 if n == 17 else 0.0, shapes=0))
    top.add_ground_plane(cfg=nb.ModelBuilder.ShapeConfig(ke=1e4, kd=1e-4, mu=0.5))
    model = top.finalize("cuda:0")
    model.soft_contact_ke, model.soft_contact_kd, model.soft_contact_mu = 1e4, 1e-4, 0.5
    q, qd = _start(model, len(sides))
    ref, _ = _run(model, q, qd, precision="fp64", schedule="persistent", layout="ell")
    chosen = SolverVBD(model, iterations=6, schedule="persistent", layout="ell16", min_blocks_per_sm=3).split
    assert chosen["grid"] == (len(q) > 1024)
    got, _ = _run(model, q, qd, precision="fp64", schedule="persistent", layout="ell16")
    assert np.abs(got - ref).max() <= 1e-9
    got, _ = _run(model, q, qd, substeps=1, schedule="persistent", layout="ell16", min_blocks_per_sm=3)
    ref, _ = _run(model, q, qd, substeps=1, precision="fp64", schedule="persistent", layout="ell")
    assert np.abs(got - ref).max() <= 1e-4


@pytest.mark.parametrize("nx,ny,kd", [(32, 32, 0.0), (64, 64, 0.0), (41, 27, 1e-3), (90, 80, 0.0)])
def test_split_fp64_holds_elements_as_the_csr_kernel_does(nx, ny, kd):
    """One FP64 substep split and by csr launches differ by the order of the sums alone: some roundings (1.1e-16) of
    positions of 1 m, 2e-15 m. Products rounded to FP32 in the records are 1e-14 to 3e-12 m off here."""
    model = _sheet(nx, ny, kd).finalize("cuda:0")
    q, qd = _start(model, nx)
    ref, ref_d = _run(model, q, qd, substeps=1, precision="fp64", schedule="per_color", layout="csr")
    got, got_d = _run(model, q, qd, substeps=1, precision="fp64")
    assert SolverVBD(model, precision="fp64").split is not None
    assert np.abs(got - ref).max() <= 2e-15 and np.abs(got_d - ref_d).max() <= 2e-15 / DT


@pytest.mark.parametrize("shared", ["on", "off"])
@pytest.mark.parametrize("kd", [0.0, 1e-3])
@pytest.mark.parametrize("precision", ["fp32", "mixed"])
def test_unsplit_ell16_worlds_match_fp64(precision, kd, shared):
    """The kernel of large batches, one CTA per world on 16-bit records, with and without hinge damping (two kernels) and
    positions in shared memory: FP32 sums against FP64 over one substep, 1e-4 m per m as every FP32 kernel here."""
    top = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
    for n in (17, 30, 9, 64):
        top.add_world(_sheet(n, n, kd, shapes=0))
    top.add_ground_plane(cfg=nb.ModelBuilder.ShapeConfig(ke=1e4, kd=1e-4, mu=0.5))
    model = top.finalize("cuda:0")
    model.soft_contact_ke, model.soft_contact_kd, model.soft_contact_mu = 1e4, 1e-4, 0.5
    q, qd = _start(model, 4)
    kw = dict(schedule="persistent", layout="ell16", split="off")
    assert SolverVBD(model, precision=precision, positions_in_shared=shared, **kw).split is None
    got, _ = _run(model, q, qd, substeps=1, precision=precision, positions_in_shared=shared, **kw)
    ref, _ = _run(model, q, qd, substeps=1, precision="fp64", schedule="persistent", layout="csr")
    assert np.abs(got - ref).max() <= 1e-4


def _damp(model, faces, hinges):
    model.tri_materials[:, 2] = faces
    model.edge_bending_properties[:, 1] = hinges


# the damping (membranes, hinges) at the capture and after the refresh; 20 x 20 is one cluster, 64 x 64 a grid
@pytest.mark.parametrize("n", [20, 64])
@pytest.mark.parametrize("before,after", [((0.0, 0.0), (0.0, 0.0)), ((0.0, 0.0), (0.0, 2e-3)), ((0.0, 2e-3), (0.0, 0.0)),
                                          ((0.0, 0.0), (2e-3, 0.0)), ((2e-3, 2e-3), (0.0, 0.0))])  # fmt: skip
def test_split_refresh_and_capture(n, before, after):
    """A graph captured before a refresh steps with the new materials, damping that came or went among them, and agrees
    bit for bit with an eager step and with a new solver; a state stepped in place keeps working."""
    model = _sheet(n, n).finalize("cuda:0")
    _damp(model, *before)
    q, qd = _start(model, n)
    solver = SolverVBD(model, iterations=5)
    pipe = CollisionPipeline(model, soft_contact_margin=0.01)
    contacts = pipe.contacts()
    s0, s1 = model.state(), model.state()

    def reset():
        s0.particle_q.copy_(torch.as_tensor(q))
        s0.particle_qd.copy_(torch.as_tensor(qd))

    reset()
    pipe.collide(s0, contacts)
    solver.step(s0, s1, None, contacts, DT)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
        pipe.collide(s0, contacts)
        solver.step(s0, s1, None, contacts, DT)
    torch.cuda.synchronize()
    reset()
    graph.replay()
    torch.cuda.synchronize()
    old = s1.particle_q.clone()
    model.tri_materials[:, :2] *= 3.0 if before == after else 1.0
    _damp(model, *after)
    solver.notify_model_changed()
    reset()
    graph.replay()
    torch.cuda.synchronize()
    captured = s1.particle_q.clone()
    assert not torch.equal(captured, old)
    reset()
    pipe.collide(s0, contacts)
    solver.step(s0, s1, None, contacts, DT)
    torch.cuda.synchronize()
    assert torch.equal(captured, s1.particle_q)
    fresh = SolverVBD(model, iterations=5)
    assert solver.split is not None and fresh.split == solver.split
    reset()
    pipe.collide(s0, contacts)
    fresh.step(s0, s0, None, contacts, DT)
    torch.cuda.synchronize()
    assert torch.equal(captured, s0.particle_q)
    del graph


@pytest.mark.parametrize("n", [20, 41])
def test_split_refresh_inside_a_capture(n):
    """A refresh of a default cloth launches kernels only: captured with the step, a replay takes the materials that the
    model holds by then. The same kernels on the same data as an eager refresh and step: bit for bit."""
    model = _sheet(n, n).finalize("cuda:0")
    q, qd = (torch.as_tensor(x, device="cuda") for x in _start(model, n))
    solver = SolverVBD(model, iterations=5)
    assert solver.split is not None and solver.layout == "csr"
    s0, s1 = model.state(), model.state()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
        s0.particle_q.copy_(q)
        s0.particle_qd.copy_(qd)
        solver.notify_model_changed()
        solver.step(s0, s1, None, None, DT)
    out = []
    for scale, hinges in ((1.0, 0.0), (3.0, 2e-3)):
        model.tri_materials[:, :2] *= scale
        _damp(model, 0.0, hinges)
        graph.replay()
        torch.cuda.synchronize()
        out.append(s1.particle_q.clone())
        s0.particle_q.copy_(q)
        s0.particle_qd.copy_(qd)
        SolverVBD(model, iterations=5).step(s0, s1, None, None, DT)
        torch.cuda.synchronize()
        assert torch.equal(out[-1], s1.particle_q)
    assert not torch.equal(*out)
    del graph


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_split_refresh_takes_materials_under_the_floor(precision):
    """A refresh to triangles with |lambda + mu| < 1e-6 needs the reference's floor on the material values: a default cloth
    takes it, as its csr layout does unsplit; a named ell16 layout refuses it and keeps the materials it had."""
    model = _sheet(24, 24).finalize("cuda:0")
    q, qd = (torch.as_tensor(x, device="cuda") for x in _start(model, 3))
    solvers = [SolverVBD(model, iterations=5, precision=precision, **kw)
               for kw in ({}, dict(layout="csr", schedule="persistent", lanes_per_vertex=1), dict(layout="ell16", schedule="persistent"))]  # fmt: skip
    assert [s.split is not None for s in solvers] == [True, False, True]

    def step(solver):
        a, b = model.state(), model.state()
        if precision == "fp64":
            for s in (a, b):
                s.particle_f = None
                s.particle_q, s.particle_qd = s.particle_q.double(), s.particle_qd.double()
        a.particle_q.copy_(q)
        a.particle_qd.copy_(qd)
        solver.step(a, b, None, None, DT)
        torch.cuda.synchronize()
        assert solver.device_errors() == 0
        return b.particle_q.double()

    before = step(solvers[2])
    model.tri_materials[::3, 0], model.tri_materials[::3, 1] = 4.0e-7, 1.0e-7
    model.tri_materials[1::7, 0], model.tri_materials[1::7, 1] = 2.0, -2.0
    for solver in solvers[:2]:
        solver.notify_model_changed()
    with pytest.raises(_lib.VbdError, match="unsupported"):
        solvers[2].notify_model_changed()
    assert torch.equal(step(solvers[2]), before)
    got, ref = step(solvers[0]), step(solvers[1])
    assert not torch.equal(got, before)
    assert (got - ref).abs().max().item() <= (1e-9 if precision == "fp64" else 1e-5)


def test_a_particle_without_a_color_is_not_solved():
    """Colors that list one particle twice and another never: the latter takes its inertial target, on every schedule, and
    the recorded substep, whose checkpoints could not hold the states between the colors, refuses the model."""
    from newton_chysx_b200.adjoint import DifferentiableVBD

    b = cloth_grid_builder(n=12, hanging=False, height=1.0)
    groups = [np.sort(np.int32(g)) for g in b.particle_color_groups]
    left_out, groups[1] = int(groups[1][3]), np.concatenate([groups[1][:3], groups[1][4:], groups[0][5:6]])
    b.set_coloring(groups)
    model = b.finalize("cuda:0")
    q, qd = _start(model, 1)
    target = q[left_out] + DT * (qd[left_out] + DT * np.float32([0.0, 0.0, -9.81]))
    for kw in ({}, dict(schedule="per_color", layout="csr"), dict(schedule="persistent", layout="ell")):
        assert SolverVBD(model, **kw).split is None
        got, _ = _run(model, q, qd, substeps=1, **kw)
        assert np.abs(got[left_out] - target).max() <= 1e-6  # FP32 positions of up to 1.1 m
    sim = DifferentiableVBD(model, iterations=3)
    mu, lam = model.tri_materials[:, 0].clone(), model.tri_materials[:, 1].clone()
    with pytest.raises(_lib.VbdError, match="invalid argument"):
        sim.rollout(torch.as_tensor(q, device="cuda"), torch.as_tensor(qd, device="cuda"), mu, lam, DT, 1)


def test_what_steps_split_and_what_does_not():
    """The split is reported, taken with the default options and with ell16 whatever its launch shape, and left where an
    option names another kernel, split="off" asks for it, there is nothing to split or enough worlds fill the GPU."""
    model = cloth_grid_builder(n=12).finalize("cuda:0")
    small = dict(parts=3, jobs=1, lanes=8, grid=False)
    for kw in ({}, dict(schedule="persistent"), dict(precision="mixed"), dict(precision="fp64"), dict(layout="ell16", schedule="persistent"),
               dict(layout="ell16", schedule="persistent", lanes_per_vertex=1, block_size=128, min_blocks_per_sm=3,
                    positions_in_shared="off")):  # fmt: skip
        got = SolverVBD(model, iterations=4, **kw).split
        assert got is not None and {k: got[k] for k in small} == small and got["threads"] >= 64
    ell16 = dict(layout="ell16", schedule="persistent")
    for kw in (dict(split="off"), dict(ell16, split="off"), dict(schedule="per_color"), dict(layout="csr"), dict(layout="ell"),
               dict(layout="ring", schedule="persistent"), dict(block_size=128), dict(lanes_per_vertex=4),
               dict(positions_in_shared="on"), dict(ell16, pair_vertices=True), dict(iterations=0),
               dict(particle_enable_self_contact=True, particle_self_contact_radius=1e-3, particle_self_contact_margin=2e-3),
               dict(layout="csr", schedule="persistent", lanes_per_vertex=4, instance_per_warp=True)):  # fmt: skip
        assert SolverVBD(model, **dict(dict(iterations=4), **kw)).split is None, kw
    # vertices of an element in one color: opposite vertices of a hinge with the default coloring, and of a triangle
    # without stiffness, which a refresh can switch on
    for triangles in (False, True):
        b = cloth_grid_builder(n=12)
        if triangles:
            free = int(b.tri_indices[-1][0])
            groups = [[int(v) for v in g if int(v) != free] for g in b.particle_color_groups]
            other = int(b.tri_indices[-1][1])
            next(g for g in groups if other in g).append(free)
            mats = b.tri_materials
            mats[(b.tri_indices == free).any(axis=1), :2] = 0.0
            b._tri_mat = [mats]
            b.set_coloring([np.sort(np.int32(g)) for g in groups])
        else:
            b.color()
        assert SolverVBD(b.finalize("cuda:0"), iterations=4).split is None
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for worlds in (6 * sms - 1, 6 * sms):
        top = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
        one = cloth_grid_builder(n=4)
        for _ in range(worlds):
            top.add_world(one)
        assert (SolverVBD(top.finalize("cuda:0"), iterations=4).split is not None) == (worlds < 6 * sms)
    with pytest.raises(KeyError):
        SolverVBD(model, split="on")


def test_the_autotuner_times_the_kernels_it_names(monkeypatch):
    """Every unsplit candidate steps the kernel that it names, the split is a candidate of its own, and what the tuner
    returns steps as what it timed; a winner that is split carries a launch shape for models too large to split."""
    from newton_chysx_b200 import autotune

    top = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
    for n in (9, 12, 16):
        top.add_world(cloth_grid_builder(n=n))
    model = top.finalize("cuda:0")
    built = []

    class Spy(SolverVBD):
        def __init__(self, *args, **kw):
            super().__init__(*args, **kw)
            built.append((kw.get("split"), kw["layout"], self.layout, self.split is not None))

    monkeypatch.setattr(autotune, "SolverVBD", Spy)
    best = autotune.tune(model, iterations=3, substeps=1)
    assert sum(is_split for *_, is_split in built) == 1
    for asked, layout, got, is_split in built:
        assert layout == got and is_split == (asked != "off")
    solver = SolverVBD(model, iterations=3, **best)
    assert (solver.split is None) == (best.get("split") == "off")
    one = [dict(layout="csr", lanes_per_vertex=2, split="off"), dict(layout="ell16", lanes_per_vertex=1, min_blocks_per_sm=3, split="off"),
           dict(layout="ell16", lanes_per_vertex=1)]  # fmt: skip
    for keep, want in ((one, dict(one[1], schedule="persistent")), (one[:2], None)):
        monkeypatch.setattr(autotune, "candidates", lambda *_: keep)
        got = autotune.tune(model, iterations=40, substeps=1)
        if want is not None and "split" not in got:
            want.pop("split")
            assert got == want
        elif want is None:
            assert got["split"] == "off"
