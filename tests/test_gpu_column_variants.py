"""The column kernel's precisions, variants and transmissive x faces against the brick
kernel (emma_b200/csrc/column_kernel.cuh, level_kernel.cuh).

Both evaluate the same expressions per cell and face.  FP64: equal bits.  Mixed: the
FP32 contraction of the two kernels may differ, L1 <= 1e-6 of every field (the bar of
the plain variant's comparison).  Items of 2 planes (every plane a halo of another item), the
whole column, and balanced runs; levels of 1, 4 and 16 columns.
"""
import numpy as np
import pytest

from emma_b200 import OctTree, PREC_FP64, PREC_MIXED, ResidentHydro, TRANS_XM, TRANS_XP, TRANS_YM
from helpers import l1_rel

pytestmark = pytest.mark.gpu


def run(level, precision, variant, trans=0, steps=3, **kw):
    rng = np.random.default_rng(3)
    t = OctTree(level, level, rh=variant == "tracer")
    n = 8 * t.noct(level)
    d, p = (np.exp(rng.uniform(-1, 1, n)) for _ in range(2))
    t.set_fields(level, d, *(rng.uniform(-1, 1, n) for _ in range(3)), p)
    if variant == "tracer":
        x0 = d * rng.uniform(0, 1, n)
        t.set_tracer(level, x0)
    r = ResidentHydro(t, precision=precision, cfl=0.8, trans=trans, gravity=variant == "gravity",
                      dual=variant == "dual", **kw)
    if variant == "gravity":
        r.set_force(level, *(rng.uniform(-1, 1, n) for _ in range(3)))
    for _ in range(steps):
        r.coarse_step()
    assert r.status() == 0
    s = r.state(level)
    if variant == "tracer":
        r.download()
        s = np.vstack([s, t.get_tracer(level)[None]])
        assert l1_rel(s[5], x0) > 1e-3  # it was advected
    return s, r.tsim, r.column_tuning(level)[0]


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("variant,trans", [("plain", 0), ("plain", TRANS_XM), ("plain", TRANS_XP),
                                           ("plain", TRANS_XM | TRANS_XP), ("gravity", 0), ("dual", 0),
                                           ("dual", TRANS_XM | TRANS_XP), ("tracer", 0)])
@pytest.mark.parametrize("level", [4, 5, 6])
def test_column_equals_brick(gpu, level, variant, trans, precision):
    ref, t_ref, planes = run(level, precision, variant, trans, column=-1)
    assert planes == 0
    first = None
    for kw in ({"column": 2}, {"column": 2 ** level}, {"column": 4, "balanced": 1}):
        s, t, planes = run(level, precision, variant, trans, **kw)
        assert planes == kw["column"]
        if precision == PREC_FP64:
            assert np.array_equal(s, ref) and t == t_ref
        else:
            # every row: density, velocities (a tenth to one sound speed), pressure, tracer
            assert all(l1_rel(s[k], ref[k]) <= 1e-6 for k in range(len(ref))) and abs(t - t_ref) <= 1e-6 * t_ref
            first = s if first is None else first
            assert np.array_equal(s, first)  # the work split changes no bit


@pytest.mark.parametrize("kw", [{"trans": TRANS_YM}, {"tile_octs": 32}, {"tile_octs": 8}])
def test_fp64_keeps_the_brick_kernel(gpu, kw):
    """Other transmissive faces, whose ghosts are not copies of the boundary cells on every
    side, and a forced brick shape."""
    assert run(5, PREC_FP64, "plain", steps=1, **kw)[2] == 0


def test_captured_step_follows_a_forced_brick_shape(gpu):
    """tile_octs set between two steps of a resident tree decides the kernel (FP64: the bricks
    when it is forced): the captured step of the other kernel is not launched again."""
    rng = np.random.default_rng(3)
    t = OctTree(5, 5)
    n = 8 * t.noct(5)
    d, p = (np.exp(rng.uniform(-1, 1, n)) for _ in range(2))
    t.set_fields(5, d, *(rng.uniform(-1, 1, n) for _ in range(3)), p)
    r = ResidentHydro(t, precision=PREC_FP64, cfl=0.8, column=4)
    launches = []
    for octs in (0, 32, 0):
        r.tile_octs = octs
        r._apply()
        r.coarse_step()
        assert (r.column_tuning(5)[0] > 0) == (octs == 0)
        launches.append(r.graph_info()[3])
    # column kernel: its last CTA ends the step; bricks: CFL, begin, level, end
    assert launches == [2, 4, 2] and r.status() == 0
