"""Finest-level sweeps of cells on a grain map over the rules that choose them.  FP32: cells of at most 96
grains march, with rows of up to 64 nodes once such cells hold 1.5 million nodes of solves (9 slots: 3
million), with rows of up to 128 from 5 million on; the others take one pass.  FP64: two passes from 300
thousand nodes of solves on, from 90 thousand if a grain holds 512 of them, else one.  A filler cell beside
the one under test sets the totals.  Every way runs the arithmetic of the per-node sweeps on the equivalent
field, so solutions agree bit for bit with a cell given as that field."""
import numpy as np
import pytest

from anisotropicfracture_gb300 import cells, models

pytestmark = pytest.mark.gpu

OPTS = dict(max_fmg_iter=0, nu1=2, nu2=2, sweeps=2, bottom=1, bottom_max_iter=20, bottom_reltol=1e-4, nuf=8, max_iter=2)
NONE, ROWS64, ROWS64D, ROWS128 = None, (64, 6), (64, 12), (128, 3)  # filler: nodes an edge, load cases


def _table(model, n, rng):
    if model == models.MAJORMINOR:
        return models.cubic(1.68, 1.21, 0.75, models.random_rotations(n, rng))
    return 1.0 + rng.random((n, models.NCOEF[model]))


def _nearest(n, seeds):
    """The grain of every node: the nearest seed over all periodic images (unit edges)."""
    z, y, x = np.meshgrid(*[np.arange(m) / m for m in n[::-1]], indexing="ij")
    best, gid = np.full(x.shape, np.inf), np.zeros(x.shape, dtype=np.int64)
    for g, s in enumerate(seeds):
        d2 = 0.0
        for c, p in zip((x, y, z), s):
            d = np.abs(c - p)
            d = np.minimum(d, 1.0 - d)
            d2 = d2 + d * d
        near = d2 < best
        gid[near], best[near] = g, d2[near]
    return gid


def _check(n, ngr, precision, filler, model):
    n = (n,) * 3 if np.isscalar(n) else n
    rng = np.random.default_rng(sum(n) + ngr)
    seeds, table = rng.random((ngr, 3)), _table(model, ngr, rng)
    B = cells.CellBatch([(n, 2)] + ([filler] if filler else []), model)
    F = cells.CellBatch([(n, 2)], model)
    B.set_grains(0, seeds, table)
    if filler:
        B.set_grains(1, rng.random((5, 3)), _table(model, 5, rng))
    F.set_model(0, np.ascontiguousarray(np.moveaxis(table[_nearest(n, seeds)], -1, 0)))
    E = cells.unit_strains()
    for s in range(B.nsolves):
        B.set_load(s, E[s % 6])
        if s < 2:
            F.set_load(s, E[s % 6])
    B.prepare()
    F.prepare()
    sb, _ = B.solve(precision=precision, inner_cycles=2, check=False, **OPTS)
    sf, _ = F.solve(precision=precision, inner_cycles=2, check=False, **OPTS)
    for s in range(2):
        assert sb[s]["iters"] == sf[s]["iters"]
        assert np.array_equal(B.solution(s), F.solution(s))
        assert np.array_equal(sb[s]["mean_stress"], sf[s]["mean_stress"])
    B.close()
    F.close()


# rows around both limits, planes smaller than a block, uneven boxes, grain counts around the limit
@pytest.mark.parametrize("n,ngr", [(4, 3), (20, 7), (62, 9), (64, 96), (66, 9), (72, 97), (104, 33), (128, 96), (130, 4),
                                   ((128, 6, 10), 6), ((6, 128, 10), 6), ((66, 4, 4), 2), ((126, 20, 4), 12)])
@pytest.mark.parametrize("filler", [ROWS64, ROWS128])
def test_fp32_sweeps_equal_the_field_bit_for_bit(n, ngr, filler):
    _check(n, ngr, 1, filler, models.MAJORMINOR)


@pytest.mark.parametrize("model", [models.ISOTROPIC, models.DIAGONAL])
@pytest.mark.parametrize("n,ngr", [(20, 7), (104, 20), ((128, 6, 10), 6)])
@pytest.mark.parametrize("filler", [NONE, ROWS64, ROWS64D, ROWS128])
def test_fp32_sweeps_of_the_other_kinds(model, n, ngr, filler):
    _check(n, ngr, 1, filler, model)


# 56 grains fill the FP64 tables, 57 do not
@pytest.mark.parametrize("model", [models.MAJORMINOR, models.ISOTROPIC, models.DIAGONAL])
@pytest.mark.parametrize("n,ngr", [(4, 2), (20, 57), ((12, 34, 6), 56), (48, 30)])
@pytest.mark.parametrize("filler", [NONE, ROWS64])
def test_fp64_sweeps_equal_the_field_bit_for_bit(model, n, ngr, filler):
    _check(n, ngr, 0, filler, model)
