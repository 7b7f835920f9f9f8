"""Soft bodies whose surface has no stiffness skip its triangles and hinges, and colors without springs inside them skip
the pre-pass: both have to follow a refresh of the model. FP64 schedules agree to 1e-9 m (other orders of the same sums);
a refreshed solver and a new one run the same kernels on the same data, bit for bit."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import newton_chysx_b200 as nb  # noqa: E402
from newton_chysx_b200 import SolverVBD  # noqa: E402

DT = 1.0 / 600.0


def _block(surface, same_color_spring):
    b = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
    b.add_soft_grid(pos=(0.0, 0.0, 0.0), rot=nb.quat_identity(), vel=(0.0, 0.0, 0.0), dim_x=4, dim_y=3, dim_z=2,
                    cell_x=0.02, cell_y=0.02, cell_z=0.02, density=500.0, k_mu=2e4, k_lambda=3e4, k_damp=1e-3,
                    tri_ke=surface, tri_ka=surface, edge_ke=surface * 1e-3, particle_radius=2e-3)  # fmt: skip
    top = b.add_particle((0.04, 0.03, 0.2), (0.0, 0.0, 0.0), 0.0, 2e-3)
    b.add_spring(top, 59, 50.0, 1e-2, 0.0)
    b.color(include_bending=True)  # a coloring that holds with the surface's stiffness on
    if same_color_spring:
        group = [int(v) for v in b.particle_color_groups[1][:2]]
        b.add_spring(group[0], group[1], 40.0, 1e-2, 0.0)
    return b.finalize("cuda:0")


def _step(solver, model, q, qd):
    f64 = solver.precision == "fp64"
    a, b = model.state(), model.state()
    for s in (a, b):
        if f64:
            s.particle_f = None
            s.particle_q, s.particle_qd = s.particle_q.double(), s.particle_qd.double()
    a.particle_q.copy_(q)
    a.particle_qd.copy_(qd)
    solver.step(a, b, None, None, DT)
    torch.cuda.synchronize()
    return b.particle_q.clone()


@pytest.mark.parametrize("cells,worlds,schedule", [(6, 1, "persistent"), (8, 1, "per_color"), (8, 2, "per_color"),
                                                    (8, 30, "persistent")])  # fmt: skip
def test_automatic_schedule_of_soft_blocks(cells, worlds, schedule):
    """344 particles in one world stay on one CTA, 730 take per-color launches up to 16,384 in all; options that the
    per-color schedule does not take keep the persistent one. Either way the same step."""
    one = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
    one.add_soft_grid(pos=(0.0, 0.0, 0.0), rot=nb.quat_identity(), vel=(0.0, 0.0, 0.0), dim_x=cells, dim_y=cells,
                      dim_z=cells, cell_x=0.02, cell_y=0.02, cell_z=0.02, density=500.0, k_mu=2e4, k_lambda=3e4,
                      k_damp=1e-3, particle_radius=2e-3)  # fmt: skip
    one.color()
    b = one
    if worlds > 1:
        b = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
        for _ in range(worlds):
            b.add_world(one)
    model = b.finalize("cuda:0")
    rng = np.random.default_rng(cells)
    q = model.particle_q.double() + torch.as_tensor(1e-3 * rng.normal(size=(model.particle_count, 3)), device="cuda:0")
    qd = torch.zeros_like(q)
    solver = SolverVBD(model, iterations=3, precision="fp64")
    assert solver.schedule == schedule
    assert SolverVBD(model, iterations=3, block_size=256).schedule == "persistent"
    other = "per_color" if schedule == "persistent" else "persistent"
    ref = _step(SolverVBD(model, iterations=3, precision="fp64", schedule=other), model, q, qd)
    assert float((_step(solver, model, q, qd) - ref).abs().max()) <= 1e-9


@pytest.mark.parametrize("schedule", ["per_color", "persistent"])
@pytest.mark.parametrize("same_color_spring", [False, True])
def test_surface_stiffness_comes_and_goes(schedule, same_color_spring):
    model = _block(30.0, same_color_spring)
    rng = np.random.default_rng(3)
    q = model.particle_q.double() + torch.as_tensor(1e-3 * rng.normal(size=(model.particle_count, 3)), device="cuda:0")
    qd = torch.as_tensor(rng.normal(size=(model.particle_count, 3)), device="cuda:0")
    solver = SolverVBD(model, iterations=5, precision="fp64", schedule=schedule)
    other = "per_color" if schedule == "persistent" else "persistent"
    for mu, ke in ((0.0, 0.0), (30.0, 0.0), (0.0, 2e-2), (30.0, 2e-2), (0.0, 0.0)):
        model.tri_materials[:, :2] = mu
        model.edge_bending_properties[:, 0] = ke
        solver.notify_model_changed()
        got = _step(solver, model, q, qd)
        assert torch.equal(got, _step(SolverVBD(model, iterations=5, precision="fp64", schedule=schedule), model, q, qd))
        ref = _step(SolverVBD(model, iterations=5, precision="fp64", schedule=other, lanes_per_vertex=1), model, q, qd)
        assert float((got - ref).abs().max()) <= 1e-9
        if mu == 0.0 and ke == 0.0:
            bare = got
        else:
            assert float((got - bare).abs().max()) > 1e-9  # the surface takes part


@pytest.mark.parametrize("schedule", ["per_color", "persistent"])
def test_surface_stiffness_follows_a_captured_refresh(schedule):
    """A refresh launches kernels only: captured with the step, a replay takes the surface that the model has by then."""
    model = _block(0.0, False)
    rng = np.random.default_rng(5)
    q = model.particle_q + torch.as_tensor(1e-3 * rng.normal(size=(model.particle_count, 3)), device="cuda:0").float()
    qd = torch.zeros_like(q)
    solver = SolverVBD(model, iterations=5, schedule=schedule)
    a, b = model.state(), model.state()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
        a.particle_q.copy_(q)
        a.particle_qd.copy_(qd)
        solver.notify_model_changed()
        solver.step(a, b, None, None, DT)
    out = []
    for mu in (0.0, 30.0, 0.0):
        model.tri_materials[:, :2] = mu
        graph.replay()
        torch.cuda.synchronize()
        out.append(b.particle_q.clone())
        assert torch.equal(out[-1], _step(SolverVBD(model, iterations=5, schedule=schedule), model, q, qd))
    assert torch.equal(out[0], out[2]) and not torch.equal(out[0], out[1])
    del graph
