"""Split sweeps of grain maps whose tables fit shared memory in part or not at all.  A grain's row is 36
FP64 numbers and its stiffness 21: 40 KiB hold the rows of 142 grains, 44 KiB rows and stiffness of 98, and
the FP32 kernel keeps 24 KiB of padded stiffness, 256 grains.  The result is the one-pass sweep's, bit for
bit, at every count."""
import os

import numpy as np
import pytest

from anisotropicfracture_gb300 import models
from anisotropicfracture_gb300.elastic import Elastic, Field, level_desc
from helpers import bc_random

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CELLS = (34, 18, 22)


def _op(split, gid, table, bc):
    os.environ["AE_SPLIT"] = "1" if split else "0"
    try:
        op = Elastic([level_desc(CELLS)], models.MAJORMINOR)
    finally:
        os.environ.pop("AE_SPLIT", None)
    op.SetModelGrains(0, Field(gid), table)
    op.SetBC(bc)
    op.SetUniform(False)
    op.prepareForSolve()
    return op


@pytest.mark.parametrize("ngrains", [1, 98, 99, 142, 143, 256, 257])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_any_number_of_grains(ngrains, dtype):
    rng = np.random.default_rng(ngrains)
    shape = tuple(c + 1 for c in CELLS[::-1])
    gid = np.ascontiguousarray(rng.integers(0, ngrains, size=(1,) + shape), dtype=np.int32)
    table = models.cubic(1.68, 1.21, 0.75, models.random_rotations(ngrains, rng))
    bc = bc_random(rng)
    g = torch.Generator(device="cuda")
    g.manual_seed(ngrains)
    x = torch.randn((3,) + shape, device="cuda", dtype=dtype, generator=g)
    b = torch.randn((3,) + shape, device="cuda", dtype=dtype, generator=g)
    out = []
    for split in (True, False):
        op = _op(split, gid, table, bc)
        f, y = torch.zeros_like(x), x.clone()
        op.Fapply(0, 0, Field(f), Field(x))
        op.Fsmooth(0, 0, Field(y), Field(b), 2)
        torch.cuda.synchronize()
        out.append((f, y))
    assert torch.equal(out[0][0], out[1][0])
    assert torch.equal(out[0][1], out[1][1])
