"""Several solvers that are alive at once: split instances of the same kernel with different amounts of shared memory, and
unsplit ones, stepped in turn. Each has to step as it does alone, bit for bit (the same kernel on the same data)."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from newton_chysx_b200 import CollisionPipeline, SolverVBD  # noqa: E402
from tests.test_gpu_split import DT, _sheet, _start  # noqa: E402


class _Program:
    def __init__(self, nx, ny, **kw):
        self.model = _sheet(nx, ny).finalize("cuda:0")
        self.solver = SolverVBD(self.model, iterations=3, **kw)
        self.pipe = CollisionPipeline(self.model, soft_contact_margin=0.01)
        self.contacts = self.pipe.contacts()
        self.q, self.qd = (torch.as_tensor(x) for x in _start(self.model, nx))

    def step(self):
        s0, s1 = self.model.state(), self.model.state()
        s0.particle_q.copy_(self.q)
        s0.particle_qd.copy_(self.qd)
        self.pipe.collide(s0, self.contacts)
        self.solver.step(s0, s1, None, self.contacts, DT)
        torch.cuda.synchronize()
        return s1.particle_q.clone()


# 700 x 801 and 520 x 520: one lane per vertex, 140 and 72 KB of shared memory; 161 x 97 and 32 x 32: eight lanes on a
# grid and on a cluster; one CTA per instance with its positions in shared memory (192 KB and 48 KB)
@pytest.mark.parametrize("kw,large,small", [({}, (700, 801), (520, 520)), ({}, (161, 97), (32, 32)),
                                            (dict(schedule="persistent", layout="ell", positions_in_shared="on"), (128, 128), (64, 64))])  # fmt: skip
def test_a_smaller_solver_leaves_a_larger_one_working(kw, large, small):
    a = _Program(*large, **kw)
    alone = a.step()
    b = _Program(*small, **kw)
    first = b.step()
    for _ in range(2):
        assert torch.equal(a.step(), alone)
        assert torch.equal(b.step(), first)
