"""Finest-level sweeps of cells on a grain map (marching in FP32, two passes otherwise) at the edges of
their dispatch: planes smaller than a block, rows of any length, edges and grain counts past what fits
shared memory.  Each runs the arithmetic of the per-node sweeps on the equivalent field, so solutions
agree bit for bit with a cell given as that field."""
import numpy as np
import pytest

from anisotropicfracture_gb300 import cells

pytestmark = pytest.mark.gpu

OPTS = dict(max_fmg_iter=0, nu1=2, nu2=2, sweeps=2, bottom=1, bottom_max_iter=200, bottom_reltol=1e-4, nuf=8, max_iter=4)


# marching: 4 to 64 nodes an edge; 140 grains and 72 nodes an edge do not march; 60 grains
# do not fit the FP64 tables
@pytest.mark.parametrize("n,ngr", [(4, 3), (8, 1), (20, 7), (36, 60), (64, 96), (24, 140), (72, 20)])
@pytest.mark.parametrize("precision", [0, 1])
def test_grain_sweeps_equal_the_field_bit_for_bit(n, ngr, precision):
    seeds, table = cells.rve_grains(n, ngr, seed=50 + n)
    B = cells.CellBatch([(n, 2), (12, 1)])  # beside another cell
    F = cells.CellBatch([(n, 2)])
    B.set_grains(0, seeds, table)
    B.set_grains(1, *cells.rve_grains(12, 5, seed=9))
    F.set_model(0, cells.rve_stiffness(n, seeds, table))
    E = cells.unit_strains()
    for s, load in enumerate([E[0] + E[4], E[2], E[1]]):
        B.set_load(s, load)
        if s < 2:
            F.set_load(s, load)
    B.prepare()
    F.prepare()
    sb, _ = B.solve(precision=precision, inner_cycles=2, check=False, **OPTS)
    sf, _ = F.solve(precision=precision, inner_cycles=2, check=False, **OPTS)
    for s in range(2):
        assert sb[s]["iters"] == sf[s]["iters"]
        assert np.array_equal(B.solution(s), F.solution(s))
        assert np.array_equal(sb[s]["mean_stress"], sf[s]["mean_stress"])
