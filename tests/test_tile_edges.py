"""The stage kernels where their tiles, lines and selection rules can go wrong:
grids around multiples of the 3D 8x8x8 tile and of the pieces its lines are cut
into, grids on both sides of the rule that gives the mixed form 32x16 tiles,
constant and extremely small fields in the viscosity ratios, and the CFL maxima
of grids with more tiles than run at once (a tile skips the cells that cannot
raise the maxima it saw when it started).

Tolerances: 1e-12 relative L2 against the FP64 oracle, as in the parity tests;
the mixed form stores floats (6e-8 relative per rounding) and takes a handful
of stages, each of which rounds a stage state once: 1e-6."""
import numpy as np
import pytest

from smaug_b200 import params as P
from tests.util import ot_rect, params3, params_for, rel_l2, state3d, with_background

pytestmark = pytest.mark.gpu


def run_both(engine_lib, oracle, w, pos, p, steps):
    e = engine_lib.Engine(p, w, pos)
    e.step(steps)
    got, cm = e.state(), e.cmax()
    e.close()
    return got, cm, oracle.OracleRun(p, w, pos).advance(steps)


@pytest.mark.parametrize("integ", [P.INT_EULER, P.INT_RK4])
@pytest.mark.parametrize("n", [(7, 8, 9), (8, 16, 8), (17, 15, 16), (24, 9, 5), (5, 25, 23)])
def test_3d_tile_edges(engine_lib, oracle, n, integ):
    w, pos, dx = state3d(*n, seed=n[0])
    p = params3(w, dx, integrator=integ, g=(-0.1, 0.05, 0.0),
                boundtype=(P.BC_CONTCD4, P.BC_PERIODIC, P.BC_SYMM))
    got, cm, ref = run_both(engine_lib, oracle, w, pos, p, 3)
    for f in range(8):
        assert rel_l2(got[f], ref.w[f]) <= 1e-12
    assert np.allclose(cm, oracle.cmax(p, got), rtol=1e-13, atol=0)


@pytest.mark.parametrize("bg", [False, True])
@pytest.mark.parametrize("nx,ny", [(1184, 64), (1184, 48), (1153, 50), (1152, 64)])
def test_mixed_tile_rule(engine_lib, oracle, nx, ny, bg):
    """37 x 4 tiles of 32x16 (the rule's smallest grid), fewer, and partial ones."""
    w, pos, dx = ot_rect(nx, ny, seed=nx + ny)
    if bg:
        w = with_background(w)
    p = params_for(w, dx, integrator=P.INT_RK4, precision=P.PREC_MIXED)
    got, cm, ref = run_both(engine_lib, oracle, w, pos, p, 2)
    for f in range(6):
        assert rel_l2(got[f], ref.w[f]) <= 1e-6
    assert np.allclose(cm, oracle.cmax(p, got), rtol=1e-6, atol=0)


@pytest.mark.parametrize("scale", [0.0, 1e-140, 1e140])
def test_ratio_range(engine_lib, oracle, scale):
    """A field that is constant (0 / 0 ratios everywhere), or so small or large
    that its squares leave the range of doubles while its differences do not."""
    w, pos, dx = ot_rect(67, 41, seed=4)
    if scale <= 1e-100:
        w[4:6] *= scale
    else:  # every field scaled so that pressures and speeds stay as they are
        w[4:6] *= 0.0
        w[0:4] *= scale
    p = params_for(w, dx, integrator=P.INT_RK4)
    got, _, ref = run_both(engine_lib, oracle, w, pos, p, 4)
    for f in range(6):
        assert rel_l2(got[f], ref.w[f]) <= 1e-12
    assert np.isfinite(got).all()


@pytest.mark.parametrize("prec", [P.PREC_FP64, P.PREC_MIXED])
@pytest.mark.parametrize("bg", [False, True])
def test_cfl_maxima_of_many_tiles(engine_lib, oracle, bg, prec):
    w, pos, dx = ot_rect(1000, 700, seed=6)
    if bg:
        w = with_background(w)
    p = params_for(w, dx, integrator=P.INT_RK4, precision=prec, boundtype=(P.BC_CONTCD4, P.BC_PERIODIC))
    e = engine_lib.Engine(p, w, pos)
    for _ in range(3):
        e.step(1)
        st = e.state()
        # the mixed form's maxima are those of the FP64 sums; its state keeps a
        # float pair (48 bits) of them
        assert np.allclose(e.cmax(), oracle.cmax(p, st), rtol=1e-13 if prec == P.PREC_FP64 else 1e-12, atol=0)
    e.close()
