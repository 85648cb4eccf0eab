"""The coarsest level packed to CSR on the device, where it is too large for the four-warp solve or its long
rows do not fit there: 864, 1536 and 648 unknowns (rows of 2 and 21 slots, not a multiple of 32 or of a block's
four rows at a time among them).  The solve over it converges where a plain Krylov loop over the oracle's
operator does, with the bounds of test_gpu_bottom_converges.py, and the same again after another model."""
import numpy as np
import pytest

from anisotropicfracture_gb300 import models
from anisotropicfracture_gb300.elastic import BCElastic, Elastic, Field, Linear, level_desc
from oracle import pyoracle as po

BOXES = [(5, 5, 7), (7, 7, 7), (5, 5, 5), (4, 5, 6)]


def _problem(cells, model, seed):
    rng = np.random.default_rng(seed)
    L = po.level(cells)
    if model == models.ISOTROPIC:
        C = 1.0 + 0.1 * rng.random((2,) + L.shape)
    else:
        c = models.cubic(1.68, 1.21, 0.75, models.random_rotations(1, rng))[0]
        C = c[:, None, None, None] * (1.0 + 0.02 * rng.random(L.shape))
    b = np.zeros((3,) + L.shape)
    b[:, 1:-1, 1:-1, 1:-1] = rng.standard_normal(b[:, 1:-1, 1:-1, 1:-1].shape)
    return L, np.ascontiguousarray(C), BCElastic(), b


def _reference_converges(L, model, C, bc, b, tol=1e-5, maxiter=100):
    """BiCGStab to a tenth of the tolerance in half of the iterations."""
    def A(x):
        return po.fapply(L, model, C, bc.type, x.reshape(b.shape)).reshape(-1)

    r = b.reshape(-1).copy()
    stop = tol * np.abs(r).max()
    rh, p, rho = r.copy(), r.copy(), r @ r
    for _ in range(maxiter):
        v = A(p)
        a = rho / (rh @ v)
        s = r - a * v
        t = A(s)
        w = (t @ s) / (t @ t)
        r = s - w * t
        if min(np.abs(s).max(), np.abs(r).max()) < stop:
            return True
        rho, old = rh @ r, rho
        p = r + rho / old * a / w * (p - w * v)
    return False


@pytest.mark.parametrize("cells", BOXES)
@pytest.mark.parametrize("model", [models.ISOTROPIC, models.MAJORMINOR])
def test_reference_converges(cells, model):
    for seed in (31, 32):
        L, C, bc, b = _problem(cells, model, seed)
        assert _reference_converges(L, model, C, bc, b)


@pytest.mark.gpu
@pytest.mark.parametrize("cells", BOXES)
@pytest.mark.parametrize("model", [models.ISOTROPIC, models.MAJORMINOR])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solve_over_the_packed_level(cells, model, precision):
    op = None
    for seed in (31, 32):
        L, C, bc, b = _problem(cells, model, seed)
        if op is None:
            op = Elastic([level_desc(cells, dx=tuple(L.dx))], model)
            op.SetBC(bc)
            op.SetUniform(False)
        op.SetModel(0, Field(C))
        s = Linear(op)
        s.setMaxFmgIter(0)
        s.setPrecision(precision)
        s.setFixedIter(1)
        x = np.zeros_like(b)
        s.solve(Field(x), Field(b), 1e-10, 0.0)
        assert op.NMGLevels() == 1 and s.stats.bottom_fail == 0
        r = b - po.fapply(L, model, C, bc.type, x)
        assert np.abs(r).max() <= (1e-4 + (1e-12 if precision == "fp64" else 1e-5)) * np.abs(b).max()
    op.close()
