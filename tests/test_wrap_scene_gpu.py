"""Periodic FP32 scenes on skewed passes (ghost layout): the values of the scene on single updates,
for every coefficient form, at widths around a tile and grids smaller than the halo, with
everything between the steps that writes the fields, the mask or the tables: a pulse, new
fields, a new domain, single updates."""
import numpy as np
import pytest

from youtube_simulations_gb300 import params as P
from youtube_simulations_gb300 import scenes
from youtube_simulations_gb300 import wavegpu as W

pytestmark = pytest.mark.gpu

SIZES = [(3, 8), (5, 13), (9, 96), (40, 112), (33, 113), (64, 128), (130, 257)]


def drive(s, p, f, g, blocking):
    s.upload(*f)
    s.set_blocking(*blocking)
    s.step(7)
    s.step(5)
    s.add_circular_wave(0.1, -0.05, 0.7)
    s.step(6)
    s.set_blocking(1)
    s.step(2)
    s.set_blocking(*blocking)
    s.step(11)
    s.upload_state(*g)
    s.step(4)
    s.build_domain(scenes.D_ELLIPSE, lam=1.5)
    s.set_blocking(*blocking)
    s.step(9)
    return s.download(native=True)


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("coef", [P.COEF_MASK, P.COEF_TABLE])
@pytest.mark.parametrize("kw", [dict(), dict(twospeeds=1, courantb=0.06, gammab=1e-4), dict(floor_clamp=1, vmax=0.5),
                                dict(kappa=1e-3, twospeeds=1, courantb=0.06, gammab=1e-4)])
def test_passes_match_single_updates(nx, ny, coef, kw):
    rng = np.random.default_rng(nx * 1000 + ny)
    p = P.make_params(nx, ny, b_cond=P.BC_PERIODIC, courant=0.1, gamma=1e-4, **kw)
    n = nx * ny
    xy = (rng.random(n) < 0.7).astype(np.int16)
    tables = tuple(t * (1.0 + 0.2 * rng.random(n)) if k < 2 else t for k, t in enumerate(scenes.tables(p, xy)))
    f = (rng.standard_normal(n), rng.standard_normal(n), xy) + (tables if coef == P.COEF_TABLE else ())
    g = rng.standard_normal(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    with W.Scene(p, P.FP32, coef) as s:
        ref = drive(s, p, f, g, (1,))
    for blocking in [(2, 8, 1), (3, 8, 1), (4, 16, 1), (5, 8, 1), (6, 8, 1), (6, 64, 1), (0,)]:
        with W.Scene(p, P.FP32, coef) as s:
            got = drive(s, p, f, g, blocking)
            if blocking[0]:
                assert s.blocking() == blocking
        for a, b in zip(got, ref):
            assert np.array_equal(a, b), blocking
