"""The warp pipeline of the FP32 skewed passes at the sizes where it can go wrong: grids one
column short of, at and past the tile steps of 120 and 112 columns and the 128-column tile,
column ny-1 at every place of a lane's group, fewer rows than levels, odd row counts and
depths, chunks of the smallest height, and each compiled form of the update (every cell
written, masked cells, the general one with KAPPA and FLOOR) with mask and table coefficients.
Every FP32 stepper rounds each cell the same way, so the fields must equal the single
updates' bit for bit."""
import numpy as np
import pytest

from helpers import equalize_unwritten
from youtube_simulations_gb300 import params as P
from youtube_simulations_gb300 import scenes
from youtube_simulations_gb300 import wavegpu as W

pytestmark = pytest.mark.gpu

SIZES = [(3, 119), (5, 120), (9, 121), (13, 112), (14, 113), (41, 126), (40, 127), (61, 128), (60, 129), (97, 241),
         (130, 360), (257, 122)]


def scene(form, nx, ny):
    rng = np.random.default_rng(nx * 1000 + ny)
    kw = dict(masked=dict(b_cond=P.BC_DIRICHLET), every=dict(b_cond=P.BC_ABSORBING, twospeeds=1, courantb=0.07, gammab=2e-4),
              masked_absorbing=dict(b_cond=P.BC_ABSORBING),
              general=dict(b_cond=P.BC_DIRICHLET, kappa=1e-3, floor_clamp=1, vmax=0.4),
              osc=dict(b_cond=P.BC_ABSORBING, oscillate_left=1, omega=0.07))[form]
    p = P.make_params(nx, ny, courant=0.12, gamma=1e-4, **kw)
    xy = scenes.mask(p, scenes.D_CIRCLES, circles=[(-0.9, 0.2, 0.5), (1.1, -0.6, 0.4), (2.0, 1.1, 0.3)])
    if form == "every":
        p.src_on, p.src_i, p.src_j, p.src_amp, p.src_period = 1, nx // 2, min(ny - 1, 118), 0.05, 17.0
    phi = 0.3 * rng.standard_normal(nx * ny)
    if not p.twospeeds:
        phi = np.where(xy != 0, phi, 0.0)
    f = equalize_unwritten(p, dict(phi=phi, psi=0.98 * phi, tmp=np.zeros_like(phi)), xy)
    return p, xy, f["phi"], f["psi"], scenes.tables(p, xy)


def run(p, coef, xy, phi, psi, tab, blocking, n):
    with W.Scene(p, P.FP32, coef) as s:
        s.set_blocking(*blocking)
        s.upload(phi, psi, xy, *tab)
        s.step(n)
        return s.download()


@pytest.mark.parametrize("form", ["masked", "every", "masked_absorbing", "general", "osc"])
@pytest.mark.parametrize("coef", [P.COEF_MASK, P.COEF_TABLE])
def test_pipeline_equals_single_updates(form, coef):
    for nx, ny in SIZES:
        p, xy, phi, psi, tab = scene(form, nx, ny)
        n = 17
        want = run(p, coef, xy, phi, psi, tab, (1,), n)
        for k, rows in [(2, 8), (3, 8), (4, 8), (5, 8), (6, 8), (6, 64)]:
            got = run(p, coef, xy, phi, psi, tab, (k, rows, 1), n)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (nx, ny, k, rows)


@pytest.mark.parametrize("form", ["masked", "every", "masked_absorbing", "general", "osc"])
@pytest.mark.parametrize("coef", [P.COEF_MASK, P.COEF_TABLE])
def test_pipeline_near_the_stability_limit(form, coef):
    """The same at a Courant number where a wrong value at the far end of a halo is not lost in rounding."""
    for nx, ny in SIZES:
        p, xy, phi, psi, _ = scene(form, nx, ny)
        p.courant, p.courantb = 0.65, 0.5
        tab = scenes.tables(p, xy)
        n = 17
        want = run(p, coef, xy, phi, psi, tab, (1,), n)
        assert np.isfinite(want[0]).all()
        for k, rows in [(2, 8), (3, 8), (4, 8), (5, 8), (6, 8), (6, 64)]:
            got = run(p, coef, xy, phi, psi, tab, (k, rows, 1), n)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (nx, ny, k, rows)
