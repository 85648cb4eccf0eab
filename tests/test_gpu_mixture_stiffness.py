"""The stiffness SetModelMixture writes, for every compiled phase count and beyond it and every kind of
table, seen through the operator it feeds: the product with the device's mixture against the oracle's product
with the oracle's, to 1e-12 of the field's max-norm (each slot is a weighted mean, off by at most (2 np + 10)
2^-53 of the largest entry on both sides; a row sums fewer than a hundred products of it, with differences of
O(1) values times 1 / dx^2 that set the field's scale)."""
import numpy as np
import pytest

from anisotropicfracture_gb300 import models
from anisotropicfracture_gb300.elastic import Elastic, Field, level_desc
from helpers import bc_random, normwise_err
from oracle import pyoracle as po

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phases", [1, 2, 3, 4, 5, 6, 7, 9])
@pytest.mark.parametrize("model", [models.MAJORMINOR, models.ISOTROPIC, models.DIAGONAL])
@pytest.mark.parametrize("eigenstrain", [True, False])
def test_mixed_stiffness_of_any_number_of_phases(phases, model, eigenstrain):
    cells = (7, 5, 9)
    rng = np.random.default_rng(511 + phases)
    L = po.level(cells)
    eta = rng.random((phases, cells[2] + 1, cells[1] + 2, cells[0] + 2))
    eta[0] += 0.05
    eta[1:][rng.random(eta[1:].shape) < 0.5] = 0.0  # most cells hold few of the phases
    if model == models.MAJORMINOR:
        table = models.cubic(1.68, 1.21, 0.75, models.random_rotations(phases, rng))
    else:
        table = 0.5 + rng.random((phases, models.NCOEF[model]))
    F0table = 0.01 * rng.standard_normal((phases, 9)) if eigenstrain else None
    C_ref, _ = po.model_mixture((0, 0, 0), cells, eta, (-1, -1, 0), table, F0table)
    op = Elastic([level_desc(cells, dx=tuple(L.dx))], model)
    op.SetModelMixture(0, Field(eta, (-1, -1, 0)), table, F0table, Field(np.zeros((9,) + L.shape)) if eigenstrain else None)
    bc = bc_random(rng)
    op.SetBC(bc)
    op.SetUniform(False)
    u = rng.standard_normal((3,) + L.shape)
    f = torch.zeros((3,) + L.shape, dtype=torch.float64, device="cuda")
    op.Fapply(0, 0, Field(f), Field(torch.from_numpy(u).cuda()))
    torch.cuda.synchronize()
    assert normwise_err(f.cpu().numpy(), po.fapply(L, model, np.ascontiguousarray(C_ref), bc.type, u)) <= 1e-12
