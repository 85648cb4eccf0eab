"""Set-up kernels at the edges of their dispatch: mixtures of every compiled phase count and beyond,
and a stiffness that is not finite in any one slot.

The mixed eigenstrain is a weighted mean of table entries: its error against the oracle is that of np
weights (four roundings each, on both sides) and of np products and sums, below (2 np + 10) 2^-53 of the
largest entry."""
import numpy as np
import pytest

from anisotropicfracture_gb300 import _lib, models
from anisotropicfracture_gb300._lib import AeError
from anisotropicfracture_gb300.elastic import Elastic, Field, level_desc
from helpers import bc_random, random_coeffs
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phases", [1, 2, 3, 4, 5, 6, 7, 9])
def test_mixture_of_any_number_of_phases(phases):
    cells = (5, 3, 7)
    rng = np.random.default_rng(411 + phases)
    L = po.level(cells)
    eta = rng.random((phases, cells[2] + 1, cells[1] + 2, cells[0] + 2))
    eta[0] += 0.05
    eta[1:][rng.random(eta[1:].shape) < 0.5] = 0.0  # most cells hold few of the phases
    table = models.cubic(1.68, 1.21, 0.75, models.random_rotations(phases, rng))
    F0table = 0.01 * rng.standard_normal((phases, 9))
    C_ref, F0_ref = po.model_mixture((0, 0, 0), cells, eta, (-1, -1, 0), table, F0table)
    op = Elastic([level_desc(cells, dx=tuple(L.dx))], models.MAJORMINOR)
    F0 = np.zeros((9,) + L.shape)
    op.SetModelMixture(0, Field(eta, (-1, -1, 0)), table, F0table, Field(F0))
    assert np.abs(F0 - F0_ref).max() <= (2 * phases + 10) * 2.0**-53 * np.abs(F0table).max()


@pytest.mark.parametrize("model", [models.MAJORMINOR, models.DIAGONAL, models.ISOTROPIC])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_a_slot_that_is_not_finite_is_refused(model, value):
    """A zero difference times a slot that is not finite is not a number: whichever slot of an
    interior node it is, the diagonal is refused."""
    n = 6
    rng = np.random.default_rng(420)
    C = random_coeffs(model, (n + 1,) * 3, rng)
    for q in range(C.shape[0]):
        Cn = C.copy()
        Cn[q, 4, 3, 2] = value
        op = Elastic([level_desc(n)], model)
        op.SetModel(0, Field(Cn))
        op.SetBC(bc_random(rng))
        with pytest.raises(AeError) as e:
            op.prepareForSolve()
        assert e.value.code == _lib.AE_ERR_NAN
