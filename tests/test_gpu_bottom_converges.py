"""The four-warp bottom solve converges where a Krylov loop does: on boxes too small to coarsen, one multigrid
iteration from zero is the bottom solve alone.  With a displacement on every face and no load there, the
iteration stays on the interior, whose operator is near symmetric and definite; a plain CG / BiCGStab in
numpy on the oracle's matrix reaches a tenth of the tolerance within half of the iterations, and the device's
has to reach the tolerance: no failure, and at most bottom_reltol = 1e-4 of the right-hand side left (mixed
precision: 1e-5 more, the FP32 rounding of b and x, 2^-24 times the operator's 1 / dx^2 scale, below 100, and
a few terms)."""
import numpy as np
import pytest

from anisotropicfracture_gb300 import models
from anisotropicfracture_gb300.elastic import BCElastic, Elastic, Field, Linear, level_desc
from oracle import pyoracle as po


def _problem(cells):
    rng = np.random.default_rng(23)
    L = po.level(cells)
    C = np.ascontiguousarray(1.0 + 0.1 * rng.random((2,) + L.shape))
    b = np.zeros((3,) + L.shape)
    b[:, 1:-1, 1:-1, 1:-1] = rng.standard_normal(b[:, 1:-1, 1:-1, 1:-1].shape)
    return L, C, BCElastic(), b


def _reference_converges(L, C, bc, b, bottom, tol=1e-5, maxiter=100):
    def A(x):
        return po.fapply(L, po.ORC_ISOTROPIC, C, bc.type, x.reshape(b.shape)).reshape(-1)

    r = b.reshape(-1).copy()
    stop = tol * np.abs(r).max()
    if bottom == "cg":
        p, rho = r.copy(), r @ r
        for _ in range(maxiter):
            q = A(p)
            a = rho / (p @ q)
            r = r - a * q
            if np.abs(r).max() < stop:
                return True
            rho, old = r @ r, rho
            p = r + rho / old * p
        return False
    rh, p, rho = r.copy(), r.copy(), r @ r
    for _ in range(maxiter):
        v = A(p)
        a = rho / (rh @ v)
        s = r - a * v
        if np.abs(s).max() < stop:
            return True
        t = A(s)
        w = (t @ s) / (t @ t)
        r = s - w * t
        if np.abs(r).max() < stop:
            return True
        rho, old = rh @ r, rho
        p = r + rho / old * a / w * (p - w * v)
    return False


# unknowns a thread: 1, 2, 3, 4 and 6 (the last two in the kernel of six)
BOXES = [(2, 2, 2), (3, 3, 3), (3, 3, 5), (5, 3, 5), (5, 5, 5)]


@pytest.mark.parametrize("cells", BOXES)
@pytest.mark.parametrize("bottom", ["cg", "bicgstab"])
def test_reference_converges(cells, bottom):
    assert _reference_converges(*_problem(cells), bottom)


@pytest.mark.gpu
@pytest.mark.parametrize("cells", BOXES)
@pytest.mark.parametrize("bottom", ["cg", "bicgstab"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_bottom_solve_converges(cells, bottom, precision):
    L, C, bc, b = _problem(cells)
    op = Elastic([level_desc(cells, dx=tuple(L.dx))], models.ISOTROPIC)
    op.SetModel(0, Field(C))
    op.SetBC(bc)
    op.SetUniform(False)
    assert op.NMGLevels() == 1
    s = Linear(op)
    s.setMaxFmgIter(0)
    s.setBottomSolver(bottom)
    s.setPrecision(precision)
    s.setFixedIter(1)
    x = np.zeros_like(b)
    s.solve(Field(x), Field(b), 1e-10, 0.0)
    assert s.stats.bottom_fail == 0
    r = b - po.fapply(L, po.ORC_ISOTROPIC, C, bc.type, x)
    assert np.abs(r).max() <= (1e-4 + (1e-12 if precision == "fp64" else 1e-5)) * np.abs(b).max()
    op.close()
