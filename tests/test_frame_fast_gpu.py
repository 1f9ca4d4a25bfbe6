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


SCALES = [  # plot, frame parameters, scene parameters, size of phi, size of psi/phi - 1
    (0, dict(vscale=1e30, slope=1e17, scale=1.0), dict(), 2e-47, 1.0),
    (0, dict(vscale=1e-40, slope=1e17, scale=1.0), dict(), 1e23, 1.0),
    (0, dict(slope=1.0, scale=1e46), dict(), 1e38, 1.0),
    (0, dict(slope=1e40, scale=1.0), dict(), 1e-40, 1.0),
    (1, dict(slope=1e30, scale=1.0), dict(e_scale=1e-25), 1e10, 1.0),
    (2, dict(slope=1e30, scale=1.0), dict(e_scale=1e-25), 1e10, 1.0),
    (3, dict(slope=1e30, scale=1.0), dict(e_scale=1e-25), 1e10, 1.0),
    (4, dict(slope=1e19, log_scale=1e-20, log_shift=0.0), dict(), 1.0, 0.5),
    (6, dict(flux_scale=1e38, slope=1e8, scale=1.0), dict(), 1e-23, 1.0),
    (8, dict(slope=1e30, scale=1.0), dict(e_scale=1e-25), 1e10, 1.0),
]


@pytest.mark.parametrize("plot,kw,prm,size,rate", SCALES)
def test_scales_beyond_fp32(plot, kw, prm, size, rate):
    """Parameters and fields whose products, but not whose factors, are of ordinary size in FP32: the index
    is the FP64 one.  The index of the log, mean and average modes follows from a logarithm or a
    sum rounded a few times, so a pixel may differ only within 1e-10 of a boundary."""
    nx, ny = 33, 70
    n = nx * ny
    rng = np.random.default_rng(9)
    p = P.make_params(nx, ny, b_cond=P.BC_DIRICHLET, courant=0.1, courantb=0.06, twospeeds=1, **prm)
    xy = (rng.random(n) < 0.6).astype(np.int16)
    phi = size * rng.standard_normal(n)
    psi = phi * (1.0 - rate * rng.standard_normal(n))
    L = frame_lut(4)
    kw = dict(dict(size=1, vshift=0.0), **kw)
    with W.Scene(p, P.FP64, P.COEF_MASK) as s:
        s.upload(phi, psi, xy)
        img = s.frame_rgb8(L, plot=plot, **kw)
    ref = oracle.frame_rgb8(p, phi, xy, L, plot=plot, psi=psi, **kw)
    near = np.zeros((ny, nx), bool)
    for shift in (-1e-10, 1e-10):  # where the palette index changes within 1e-10 of the amplitude
        moved = oracle.frame_rgb8(p, phi, xy, np.repeat(np.arange(256), 3).reshape(256, 3).astype(np.uint8), plot=plot, psi=psi,
                                  **dict(kw, color_range=0.8 * (1 + shift)))
        near |= np.any(moved != oracle.frame_rgb8(p, phi, xy, np.repeat(np.arange(256), 3).reshape(256, 3).astype(np.uint8),
                                                  plot=plot, psi=psi, **kw), axis=-1)
    assert len(np.unique(ref.reshape(-1, 3), axis=0)) > 1
    diff = np.any(img != ref, axis=-1)
    assert not np.any(diff & ~near), (int(diff.sum()), int(near.sum()))


@pytest.mark.parametrize("coef", [P.COEF_MASK, P.COEF_TABLE])
@pytest.mark.parametrize("courantb", [5.5e-23, 1e-21, 1e-19, 1e-15, 1e-12])
def test_obstacle_fade_of_tiny_speeds(coef, courantb):
    nx, ny = 33, 70
    n = nx * ny
    rng = np.random.default_rng(10)
    p = P.make_params(nx, ny, b_cond=P.BC_DIRICHLET, courant=0.1, courantb=courantb, twospeeds=1)
    xy = (rng.random(n) < 0.3).astype(np.int16)
    phi = rng.standard_normal(n)
    tcc, tc, tg = scenes.tables(p, xy)
    tcc = tcc * (1.0 + rng.random(n)) if coef == P.COEF_TABLE else tcc
    L = frame_lut(4)
    kw = dict(size=1, fade=True, fade_value=0.4 / (courantb / 0.1) ** 0.2, fade_in_obstacle=True)
    with W.Scene(p, P.FP64, coef) as s:
        s.upload(phi, phi, xy, *((tcc, tc, tg) if coef == P.COEF_TABLE else ()))
        img = s.frame_rgb8(L, **kw)
    ref = oracle.frame_rgb8(p, phi, xy, L, tcc=tcc, **kw)
    out = (xy.reshape(nx, ny) == 0).T  # (inside, the fade saturates every byte but 0)
    assert len(np.unique(ref[out].reshape(-1, 3), axis=0)) > 10
    assert np.array_equal(img, ref)
