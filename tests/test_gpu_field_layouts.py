"""Fsmooth and Fapply on fields of other layouts than the level's: boxes that are larger than the
level, and storage that begins off a 16-byte boundary.  Staging copies, direct writes and their
remainders must give what compact fields give, bit for bit, and leave the nodes around alone."""
import numpy as np
import pytest

from anisotropicfracture_gb300 import models
from anisotropicfracture_gb300.elastic import Elastic, Field, level_desc
from helpers import bc_random

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# one, and more than 152 * 8 blocks of 1024 nodes (four nodes a thread in the copies); grain maps take
# the split sweep, per-node tensors the per-node one
@pytest.mark.parametrize("cells", [(10, 6, 12), (110, 114, 112)])
@pytest.mark.parametrize("grains", [True, False])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("sweeps", [1, 2])
def test_other_layouts_give_the_compact_result(cells, grains, dtype, sweeps):
    rng = np.random.default_rng(5)
    shape = tuple(c + 1 for c in cells[::-1])
    op = Elastic([level_desc(cells)], models.MAJORMINOR)
    table = models.cubic(1.68, 1.21, 0.75, models.random_rotations(7, rng))
    gid = rng.integers(0, 7, size=shape)
    if grains:
        op.SetModelGrains(0, Field(np.ascontiguousarray(gid[None], dtype=np.int32)), table)
    else:
        op.SetModel(0, Field(np.ascontiguousarray(np.moveaxis(table[gid], -1, 0))))
    op.SetBC(bc_random(rng))
    op.SetUniform(False)
    op.prepareForSolve()
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x0 = torch.randn((3,) + shape, device="cuda", dtype=dtype, generator=g)
    b0 = torch.randn((3,) + shape, device="cuda", dtype=dtype, generator=g)

    def run(wrap):
        x, b, f = wrap(x0), wrap(b0), wrap(torch.full_like(x0, 7.0))
        op.Fapply(0, 0, f[0], x[0])
        op.Fsmooth(0, 0, x[0], b[0], sweeps)
        torch.cuda.synchronize()
        return [x, f]

    def compact(t):
        t = t.clone()
        return Field(t), t, None

    def padded(t):  # nodes (2, 1, 3) below and (1, 2, 1) above the level, storage off by one element
        s = (3, shape[0] + 4, shape[1] + 3, shape[2] + 3)
        mem = torch.full((s[0] * s[1] * s[2] * s[3] + 1,), -3.0, device="cuda", dtype=dtype)
        big = mem[1:].view(s)
        inner = big[:, 3:3 + shape[0], 1:1 + shape[1], 2:2 + shape[2]]
        inner.copy_(t)
        return Field(big, (-2, -1, -3)), inner, big

    for (_, ref, _), (_, got, big) in zip(run(compact), run(padded)):
        assert torch.equal(got, ref)
        got.fill_(-3.0)
        assert bool((big == -3.0).all())
