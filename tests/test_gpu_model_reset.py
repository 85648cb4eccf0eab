"""A grain map given again to an operator that was prepared with another one: until it is prepared
again, an FP64 product (the one call that needs no preparation) takes rows, grad C columns and boundary
rows all from the new map and table.  Every route computes a node to the same bits, so it equals the
product of an operator that never had another model."""
import numpy as np
import pytest

from anisotropicfracture_gb300 import _lib, models
from anisotropicfracture_gb300._lib import AeError
from anisotropicfracture_gb300.elastic import Elastic, Field, level_desc
from helpers import bc_random, random_coeffs

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CELLS = (34, 18, 22)
SHAPE = tuple(c + 1 for c in CELLS[::-1])


def _table(model, n, rng):
    if model == models.MAJORMINOR:
        return models.cubic(1.68, 1.21, 0.75, models.random_rotations(n, rng))
    return 1.0 + rng.random((n, models.NCOEF[model]))


def _gid(n, rng):
    return np.ascontiguousarray(rng.integers(0, n, size=(1,) + SHAPE), dtype=np.int32)


def _op(model, bc):
    op = Elastic([level_desc(CELLS)], model)
    op.SetBC(bc)
    op.SetUniform(False)
    return op


def _apply(op, x):
    f = torch.zeros_like(x)
    op.Fapply(0, 0, Field(f), Field(x))
    torch.cuda.synchronize()
    return f


# grains before and after: the same map, fewer, more (past what the first preparation's arrays held)
@pytest.mark.parametrize("model", [models.MAJORMINOR, models.ISOTROPIC, models.DIAGONAL])
@pytest.mark.parametrize("before,after,same_map", [(40, 40, True), (40, 40, False), (40, 7, False), (7, 140, False),
                                                   (40, 300, False)])
def test_product_after_another_grain_map(model, before, after, same_map):
    rng = np.random.default_rng(before + after)
    bc = bc_random(rng)
    gid = _gid(before, rng)
    x = torch.from_numpy(rng.standard_normal((3,) + SHAPE)).cuda()
    op = _op(model, bc)
    op.SetModelGrains(0, Field(gid), _table(model, before, rng))
    op.prepareForSolve()
    _apply(op, x)
    gid2, table2 = (gid if same_map else _gid(after, rng)), _table(model, after, rng)
    op.SetModelGrains(0, Field(gid2), table2)
    f = _apply(op, x)
    fresh = _op(model, bc)
    fresh.SetModelGrains(0, Field(gid2), table2)
    assert torch.equal(f, _apply(fresh, x))
    for o in (op, fresh):
        o.prepareForSolve()
    assert torch.equal(_apply(op, x), f) and torch.equal(_apply(fresh, x), f)


def test_product_after_a_field_and_a_grain_map():
    """Prepared with a map, then a field (no map), then another map: still the last one's product."""
    rng = np.random.default_rng(8)
    bc = bc_random(rng)
    x = torch.from_numpy(rng.standard_normal((3,) + SHAPE)).cuda()
    op, fresh = _op(models.MAJORMINOR, bc), _op(models.MAJORMINOR, bc)
    op.SetModelGrains(0, Field(_gid(9, rng)), _table(models.MAJORMINOR, 9, rng))
    op.prepareForSolve()
    field = random_coeffs(models.MAJORMINOR, SHAPE, rng)
    gid, table = _gid(9, rng), _table(models.MAJORMINOR, 9, rng)
    for o in (op, fresh):
        o.SetModel(0, Field(field))
    assert torch.equal(_apply(op, x), _apply(fresh, x))
    for o in (op, fresh):
        o.SetModelGrains(0, Field(gid), table)
    assert torch.equal(_apply(op, x), _apply(fresh, x))


def test_product_after_a_refused_grain_map():
    """A map with an id outside its table is refused; the good one given next is the operator's."""
    rng = np.random.default_rng(9)
    bc = bc_random(rng)
    x = torch.from_numpy(rng.standard_normal((3,) + SHAPE)).cuda()
    op, fresh = _op(models.MAJORMINOR, bc), _op(models.MAJORMINOR, bc)
    op.SetModelGrains(0, Field(_gid(9, rng)), _table(models.MAJORMINOR, 9, rng))
    op.prepareForSolve()
    gid, table = _gid(9, rng), _table(models.MAJORMINOR, 9, rng)
    bad = gid.copy()
    bad[0, 3, 2, 1] = 9
    with pytest.raises(AeError) as e:
        op.SetModelGrains(0, Field(bad), table)
    assert e.value.code == _lib.AE_ERR_ARG
    for o in (op, fresh):
        o.SetModelGrains(0, Field(gid), table)
    assert torch.equal(_apply(op, x), _apply(fresh, x))
