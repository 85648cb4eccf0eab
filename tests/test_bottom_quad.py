"""The four-warp bottom solve: its matrix layout (csrc/ae_bottom_ell.h) on the CPU, and solves over
it on the GPU, on boxes too small to coarsen: there one multigrid iteration from zero is the bottom
solve alone.

A Krylov iterate is not compared entry by entry: BiCGStab amplifies the rounding of its sums.  What
is checked is what the solve promises: when it succeeds, the oracle's residual of the result is at
most bottom_reltol = 1e-4 of the right-hand side (in mixed precision plus the FP32 rounding of b and
x, 1e-5 of it: 2^-24 times the operator's 1 / dx^2 scale, below 100, and a few terms); when it fails,
the result is eight smoother calls from zero, the oracle's to 1e-12 (FP32: 2e-5)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from anisotropicfracture_gb300 import models
from anisotropicfracture_gb300.elastic import Elastic, Field, Linear, level_desc
from helpers import bc_pull_z, random_coeffs
from oracle import pyoracle as po

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bottom_ell_layout(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "bottom_ell_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "anisotropicfracture_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "bottom_ell_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


# 81, 108, 192, 216, 432 unknowns (one, two, four a thread)
@pytest.mark.gpu
@pytest.mark.parametrize("cells", [(2, 2, 2), (2, 3, 2), (3, 3, 3), (3, 2, 5), (5, 2, 7)])
@pytest.mark.parametrize("bottom", ["cg", "bicgstab"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_bottom_solve_keeps_its_promise(cells, bottom, precision):
    rng = np.random.default_rng(11)
    L = po.level(cells)
    C = np.ascontiguousarray(1.0 + 0.1 * random_coeffs(models.ISOTROPIC, L.shape, rng))
    bc = bc_pull_z()
    b = po.fapply(L, po.ORC_ISOTROPIC, C, bc.type, rng.standard_normal((3,) + L.shape))
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
    if s.stats.bottom_fail:
        D = po.diagonal(L, po.ORC_ISOTROPIC, C, bc.type)
        ref = np.zeros_like(b)
        for _ in range(8):
            ref = po.fsmooth(L, po.ORC_ISOTROPIC, C, bc.type, D, ref, b)
        assert np.abs(x - ref).max() <= (1e-12 if precision == "fp64" else 2e-5) * np.abs(ref).max()
    else:
        r = b - po.fapply(L, po.ORC_ISOTROPIC, C, bc.type, x)
        assert np.abs(r).max() <= (1e-4 + (1e-12 if precision == "fp64" else 1e-5)) * np.abs(b).max()
    op.close()
