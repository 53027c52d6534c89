"""FP64 quotients and powers of the plain path at the edges of their ranges.

The plain path takes the quotients that share a divisor from one reciprocal
(hydro_math.cuh div_y) and divides where that leaves the normal range: densities
whose square over- or underflows.  Its two-rarefaction star state uses fifth roots
(root5), from pow() outside the single-precision range of their estimate: pressures
above 1e37.  Every scale against the FP64 oracle, per cell <= 1e-12 (both evaluate
the same expressions; the bound is the one of the other parity tests), colliding and
receding streams so that all three star-pressure estimates are taken.
"""
import numpy as np
import pytest

import oracle
from emma_b200 import OctTree, PREC_FP64, ResidentHydro
from emma_b200._lib import ST_NAN
from helpers import per_cell_rel

pytestmark = pytest.mark.gpu


def box(level, dscale, pscale, uscale, seed=7):
    t = OctTree(level, level)
    rng = np.random.default_rng(seed)
    n = 8 * t.noct(level)
    d, p = (np.exp(rng.uniform(-1.5, 1.5, n)) for _ in range(2))
    u, v, w = (rng.uniform(-1.0, 1.0, n) for _ in range(3))
    t.set_fields(level, d * dscale, u * uscale, v * uscale, w * uscale, p * pscale)
    return t


@pytest.mark.parametrize("dscale,pscale,uscale", [
    (1.0, 1.0, 1.0),          # ordinary
    (1.0, 1e-6, 1e-3),        # pressures towards the floor
    (1e155, 1e149, 1e-3),     # d^2 overflows
    (1e-155, 1e-4, 1e75),     # d^2 underflows, 1/d^2 overflows
    (1.0, 1e40, 1e20),        # pressures beyond single precision
])
def test_fp64_quotients_and_roots_at_extreme_scales(gpu, dscale, pscale, uscale):
    level = 4
    t, to = box(level, dscale, pscale, uscale), box(level, dscale, pscale, uscale)
    r = ResidentHydro(t, precision=PREC_FP64, cfl=0.8)
    r.coarse_step()
    _, _, err = oracle.Restatement().run(to.firstoct, level, level, 1, 0.8)
    assert err == 0 and r.status() == 0
    o = to.get_fields(level)[:5]
    assert np.isfinite(o).all()
    assert per_cell_rel(r.state(level), o).max() <= 1e-12


def test_fp64_nan_cell_is_reported_and_contained(gpu):
    """A NaN cell raises EMMA_ST_NAN, and one step leaves every cell beyond its
    stencil (two cells) as the clean run has it."""
    level, n = 4, 16
    clean, dirty = box(level, 1.0, 1.0, 1.0), box(level, 1.0, 1.0, 1.0)
    f = dirty.get_fields(level)[:5]
    f[4, 100] = np.nan
    dirty.set_fields(level, *f)
    out = []
    for t in (clean, dirty):
        r = ResidentHydro(t, precision=PREC_FP64, cfl=0.8)
        r.advance_level(level, 1e-3)
        out.append((r.state(level), r.status()))
    assert out[0][1] == 0 and out[1][1] & ST_NAN
    c = np.floor(clean.cell_centres(level) * n).astype(int)
    away = np.abs((c - c[100] + n // 2) % n - n // 2).sum(1) > 3
    assert np.array_equal(out[0][0][:, away], out[1][0][:, away])
