"""Amplitude frames whose values lie on, next to and far from the palette's boundaries, where
the FP32 index must hand over to the FP64 one: fields at rest, signed values down to the
subnormals, every boundary of the 256 indices with offsets of 1e-12 to 1e-4, saturation,
infinities; frames one pixel short of, at and past the tiles, with and without fades.

The oracle's tanh and the GPU's are each within 2 ulp, so a pixel may differ only where the
oracle's 256-fold index lies within 256 * 8 * 2^-53 < 3e-13 of a whole number (1e-12 here), and
not where the argument is below 1e-6, whose tanh is exact to the last bit of 1 + amp."""
import numpy as np
import pytest

import oracle
from helpers import frame_lut
from youtube_simulations_gb300 import params as P
from youtube_simulations_gb300 import scenes
from youtube_simulations_gb300 import wavegpu as W

pytestmark = pytest.mark.gpu

SLOPE, SCALE, RANGE = 1.3, 0.9, 0.8


def boundary_field(n, rng, prec):
    """Arguments on the palette's boundaries and around them, zeros, tiny and huge values."""
    amp = (rng.integers(0, 257, n) / 128.0 - 1.0) / RANGE
    u = np.arctanh(np.clip(amp, -0.99999, 0.99999)) * SCALE / SLOPE
    u = u * (1.0 + rng.choice([0.0, 1e-12, 1e-9, 1e-7, 1e-5, 1e-4], n) * rng.choice([-1.0, 1.0], n))
    tiny = rng.choice([1e-3, 1e-7, 1e-14, 1e-15, 3e-16, 1e-16, 1e-17, 1e-18, 1e-30, 1e-44], n) * rng.choice([-1.0, 1.0], n)
    pick = rng.integers(0, 8, n)
    u = np.where(pick == 0, 0.0, np.where(pick == 1, -0.0, np.where(pick <= 4, tiny, u)))
    u = np.where(rng.random(n) < 0.02, rng.choice([1e30, -1e30, np.inf, -np.inf], n), u)
    return u.astype(np.float32).astype(np.float64) if prec == P.FP32 else u


@pytest.mark.parametrize("nx,ny", [(3, 3), (7, 31), (8, 32), (9, 33), (16, 64), (41, 97)])
@pytest.mark.parametrize("prec", [P.FP32, P.FP64])
@pytest.mark.parametrize("opts", [dict(), dict(fade=True, fade_value=0.7, fade_in_obstacle=True),
                                  dict(attenuation=0.02, time=3, fade=True, fade_value=-0.3)])
def test_amplitude_frames_at_the_palette_boundaries(nx, ny, prec, opts):
    rng = np.random.default_rng(nx * 1000 + ny + prec)
    p = P.make_params(nx, ny, b_cond=P.BC_DIRICHLET, courant=0.1, courantb=0.06, twospeeds=1)
    xy = (rng.random(nx * ny) < 0.6).astype(np.int16)
    tcc, tc, tg = scenes.tables(p, xy)
    phi = boundary_field(nx * ny, rng, prec)
    L = frame_lut(4)
    kw = dict(size=1, vshift=0.0, slope=SLOPE, scale=SCALE, color_range=RANGE, **opts)
    with W.Scene(p, prec, P.COEF_TABLE) as s:
        s.upload(phi, np.zeros_like(phi), xy, tcc, tc, tg)
        img = s.frame_rgb8(L, **kw)
    stored = tcc.astype(np.float32).astype(np.float64) if prec == P.FP32 else tcc
    ref = oracle.frame_rgb8(p, phi, xy, L, tcc=stored, **kw)
    u = phi.reshape(nx, ny).T * SLOPE / SCALE
    amp = RANGE * np.tanh(u) * np.exp(-opts.get("time", 0) * opts.get("attenuation", 0.0))
    hv = 128.0 * (1.0 + amp)
    may_differ = (np.abs(hv - np.round(hv)) < 1e-12) & (np.abs(u) > 1e-6)
    diff = np.any(img != ref, axis=-1)
    assert not np.any(diff & ~may_differ), np.argwhere(diff & ~may_differ)[:5]


@pytest.mark.parametrize("prec", [P.FP32, P.FP64])
@pytest.mark.parametrize("coef", [P.COEF_MASK, P.COEF_TABLE])
@pytest.mark.parametrize("plot", [0, 1])
def test_obstacle_fade_without_a_speed(prec, coef, plot):
    """COURANT = 0: the obstacle fade is (0/0)^0.1 inside, drawn black, as 0 outside with COURANTB = 0."""
    nx, ny = 17, 35
    n = nx * ny
    rng = np.random.default_rng(2)
    L = frame_lut(4)
    for courantb in (0.0, 0.1):
        p = P.make_params(nx, ny, b_cond=P.BC_DIRICHLET, courant=0.0, courantb=courantb, twospeeds=1)
        xy = (rng.random(n) < 0.6).astype(np.int16)
        phi = rng.standard_normal(n).astype(np.float32).astype(np.float64)
        tab = scenes.tables(p, xy)
        with W.Scene(p, prec, coef) as s:
            s.upload(phi, phi, xy, *(tab if coef == P.COEF_TABLE else ()))
            img = s.frame_rgb8(L, size=1, plot=plot, fade_in_obstacle=True)
        with np.errstate(all="ignore"):
            ref = oracle.frame_rgb8(p, phi, xy, L, size=1, plot=plot, psi=phi, fade_in_obstacle=True)
        assert np.array_equal(img[(xy.reshape(nx, ny) != 0).T], ref[(xy.reshape(nx, ny) != 0).T])
        assert not img[(xy.reshape(nx, ny) != 0).T].any()
        assert np.array_equal(img, ref)
