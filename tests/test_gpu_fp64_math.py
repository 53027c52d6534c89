"""FP64 quotients and powers of the plain path at the edges of their ranges.

The plain path takes the quotients that share a divisor from one reciprocal
(hydro_math.cuh div_y) and computes with the operators again where a wave speed or a
flux is not finite: densities whose square over- or underflows, streams so fast that
u +- a rounds to u.  Its two-rarefaction star state uses fifth roots
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


SCALES = [(1.0, 1.0, 1.0), (1e155, 1e149, 1e-3), (1e-155, 1e-4, 1e75), (1.0, 1e40, 1e20),
          (1.0, 1.0, 1e20),    # hypersonic: u +- a rounds to u, zero divisors in the star state
          (1.0, 1.0, 1e70),    # ... and the two-rarefaction p* = r^5 of receding streams overflows
          (1.0, 1e-6, 1e62)]


def one_step_on(kernel, trees, oracle_lib, levels, **variant):
    """One coarse step on the brick (-1) or the column kernel and by the oracle: states, velocities
    relative to |v| + c_s, pressures to p + d |v|^2, the energy that a pressure is a difference of."""
    r = ResidentHydro(trees[0], precision=PREC_FP64, cfl=0.8, column=kernel, **variant)
    r.coarse_step()
    assert (r.column_tuning(levels)[0] > 0) == (kernel > 0)
    _, _, err = oracle_lib.run(trees[1].firstoct, levels, levels, 1, 0.8, **variant)
    assert err == 0 and r.status() == 0
    g, o = r.state(levels), trees[1].get_fields(levels)[:5]
    assert np.isfinite(o).all() and np.isfinite(g).all()
    v2 = (o[1:4] ** 2).sum(0)
    scale = [o[0]] + 3 * [np.sqrt(v2) + np.sqrt(5.0 / 3.0 * o[4] / o[0])] + [o[4] + o[0] * v2]
    return max(float((np.abs(g[k] - o[k]) / scale[k]).max()) for k in range(5)), r


@pytest.mark.parametrize("kernel", [-1, 4])
@pytest.mark.parametrize("variant", ["plain", "dual", "tracer"])
@pytest.mark.parametrize("scale", SCALES)
def test_fp64_extreme_scales_on_each_kernel(gpu, scale, variant, kernel):
    level = 4
    trees = [box(level, *scale) for _ in range(2)]
    if variant == "tracer":
        trees = [OctTree(level, level, rh=True) for _ in range(2)]
        for t in trees:
            f = box(level, *scale).get_fields(level)[:5]
            t.set_fields(level, *f)
            t.set_tracer(level, f[0] * np.random.default_rng(11).uniform(0.0, 1.0, f.shape[1]))
    worst, r = one_step_on(kernel, trees, oracle.Restatement(rh=variant == "tracer"), level,
                           **({"dual": True} if variant == "dual" else {}))
    assert worst <= 1e-12
    if variant == "tracer":
        r.download()
        x, o = (t.get_tracer(level) for t in trees)
        # at 1e155 the tracer flux (d u) dT / d overflows in the reference's order too
        assert np.array_equal(np.isnan(x), np.isnan(o)) and (np.isfinite(o).all() or scale[0] == 1e155)
        ok = ~np.isnan(o)
        assert (np.abs(x - o)[ok] <= 1e-12 * trees[1].get_fields(level)[0][ok]).all()


@pytest.mark.parametrize("kernel", [-1, 4])
@pytest.mark.parametrize("dual", [False, True])
@pytest.mark.parametrize("where", ["cell", "half"])
def test_fp64_cells_without_pressure(gpu, where, dual, kernel):
    """p = 0 cells (cold gas): a sound speed of 0 in the predictor, the floor on their faces."""
    level = 4
    trees = [box(level, 1.0, 1.0, 1.0) for _ in range(2)]
    for t in trees:
        f = t.get_fields(level)[:5]
        cold = t.cell_centres(level)[:, 0] < 0.5 if where == "half" else np.arange(f.shape[1]) == 100
        f[4, cold] = 0.0
        t.set_fields(level, *f)
    assert one_step_on(kernel, trees, oracle.Restatement(), level, **({"dual": True} if dual else {}))[0] <= 1e-12


@pytest.mark.parametrize("scale", [(1e45, 1e30, 1e-9), (1e38, 1e23, 1e-9), (1e-43, 1e-10, 1.0), (1e30, 1e40, 1e-3)])
def test_fp64_time_steps_outside_single_precision(gpu, scale):
    """From the second step on dt comes from the maximum that the level kernel leaves; the
    column kernel screens cells by an FP32 estimate, which these densities or pressures
    leave: the bricks' maximum, bit for bit, and the oracle's time."""
    level, steps, out = 5, 4, []
    for kernel in (-1, 2, 32):
        r = ResidentHydro(box(level, *scale), precision=PREC_FP64, cfl=0.8, column=kernel)
        for _ in range(steps):
            r.coarse_step()
        assert r.status() == 0
        out.append((r.tsim, r.state(level)))
    assert all(t == out[0][0] and np.array_equal(s, out[0][1]) for t, s in out[1:])
    to = box(level, *scale)
    t, _, err = oracle.Restatement().run(to.firstoct, level, level, steps, 0.8)
    assert err == 0 and abs(out[0][0] - t) <= 1e-12 * t
