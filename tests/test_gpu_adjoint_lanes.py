"""The adjoint where a vertex has more elements than a round of its warp takes (eight elements at a time, and 16 lanes in
the recorded forward): fans of 3 to 21 triangles around one vertex, undamped and damped, against FP64 central
differences. Tolerance 1e-3 relative, that of the adjoint's other checks (h = 1e-5: truncation ~h^2, rounding ~1e-16 / h
of gradients of order 1)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import newton_chysx_b200 as nb  # noqa: E402
from newton_chysx_b200.adjoint import DifferentiableVBD  # noqa: E402

DT = 1.0 / 600.0


def _fan(spokes, kd):
    """A disc of `spokes` inner triangles around vertex 0 and a ring of quads around them."""
    a = np.linspace(0.0, 2.0 * np.pi, spokes, endpoint=False)
    ring = np.stack([np.cos(a), np.sin(a), 0.05 * np.sin(2.0 * a)], 1)
    verts = np.concatenate([np.zeros((1, 3)), 0.1 * ring, 0.2 * ring])
    tris = []
    for i in range(spokes):
        j = (i + 1) % spokes
        tris += [(0, 1 + i, 1 + j), (1 + i, 1 + spokes + i, 1 + spokes + j), (1 + i, 1 + spokes + j, 1 + j)]
    b = nb.ModelBuilder(up_axis="Z", gravity=-9.81)
    b.add_cloth_mesh((0.0, 0.0, 1.0), nb.quat_identity(), 1.0, (0.0, 0.0, 0.0), verts, np.array(tris).reshape(-1), 0.2,
                     tri_ke=8.0, tri_ka=6.0, tri_kd=kd, edge_ke=1e-2, edge_kd=kd, particle_radius=5e-3)  # fmt: skip
    flags = b.particle_flags
    flags[1 + spokes] = 0
    b.set_particle_flags(flags)
    b.color(include_bending=True)
    return b.finalize("cuda:0")


@pytest.mark.parametrize("spokes", [3, 8, 9, 21])
@pytest.mark.parametrize("kd", [0.0, 1e-3])
def test_adjoint_of_a_fan_matches_central_differences(spokes, kd):
    model = _fan(spokes, kd)
    sim = DifferentiableVBD(model, iterations=4, precision="fp64")
    rng = np.random.default_rng(spokes)
    dev, n = "cuda:0", model.particle_count

    def rand(*shape):
        return torch.as_tensor(rng.normal(size=shape), device=dev)

    q0 = model.particle_q.double() + 2e-3 * rand(n, 3)
    v0 = 0.2 * rand(n, 3)
    mu, lam = model.tri_materials[:, 0].double().clone(), model.tri_materials[:, 1].double().clone()
    wq, wv = rand(n, 3), 1e-2 * rand(n, 3)

    def loss(q, v):
        x, u = sim.rollout(q, v, mu, lam, DT, 2)
        return (wq * x).sum() + (wv * u).sum()

    q, v = q0.clone().requires_grad_(), v0.clone().requires_grad_()
    gq, gv = torch.autograd.grad(loss(q, v), (q, v))
    for _ in range(3):
        dq, dv = rand(n, 3), rand(n, 3)
        h = 1e-5 / float(dq.norm())
        with torch.no_grad():
            fd = float(loss(q0 + h * dq, v0 + h * dv) - loss(q0 - h * dq, v0 - h * dv)) / (2.0 * h)
        ad = float((gq * dq).sum() + (gv * dv).sum())
        assert abs(ad - fd) <= 1e-3 * max(abs(fd), float(gq.norm()))
