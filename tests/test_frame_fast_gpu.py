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


def palette_position(p, plot, phi, psi, xy, kw):
    """The oracle's palette index before it is cut to a whole number (frames of size 1, drawn cells)."""
    energy, vel, gx, gy = oracle.frame_cells(p, phi, psi, xy, 1)
    x = phi.reshape(p.nx, p.ny).T
    t1 = float(kw.get("time", 0) + 1)
    with np.errstate(divide="ignore"):
        value = {1: energy, 2: np.where((np.arange(p.ny) > p.ny // 2)[:, None], x, energy), 3: energy / t1,
                 4: kw["log_shift"] + kw["log_scale"] * np.log(np.maximum(energy, 1e-20)),
                 5: kw["log_shift"] + kw["log_scale"] * np.log(np.where(energy == 0.0, 1e-20, energy) / t1),
                 6: vel * np.sqrt(gx * gx + gy * gy) * kw["flux_scale"], 8: 0.25 * energy,
                 9: np.where(energy == 0.0, kw["log_shift"] - 10.0 * kw["log_scale"],
                             kw["log_shift"] + kw["log_scale"] * np.log(np.where(energy == 0.0, 1.0, 0.25 * energy)))}[plot]
    amp = kw["color_range"] * np.tanh(kw["slope"] * value / kw["scale"])
    return 256.0 * amp if plot in (1, 3, 6, 8) else 128.0 * (1.0 + amp)


def boundary_energies(p, plot, phi, kw, rng):
    """A psi whose velocity puts each cell's value on a palette boundary, or 1e-12 to 1e-4 (relative) beside
    it, where the gradient alone does not exceed it; velocities down to far below an ulp of phi,
    and at rest, elsewhere."""
    n = phi.size
    z = np.zeros_like(phi)
    xy = np.ones(n, np.int16)
    grad, _, gx, gy = (a.T.reshape(-1) for a in oracle.frame_cells(p, phi, phi, xy, 1))  # the energy at rest
    asym = plot in (1, 3, 6, 8)
    hv = rng.integers(1, 200, n) if asym else rng.integers(30, 226, n)
    u = np.arctanh(np.clip((hv / 256.0 if asym else hv / 128.0 - 1.0) / kw["color_range"], -0.9999, 0.9999))
    value = u * kw["scale"] / kw["slope"]
    value = value * (1.0 + rng.choice([0.0, 1e-12, 1e-10, 1e-9, 1e-8, 1e-7, 1e-6, 1e-5, 1e-4], n) * rng.choice([-1.0, 1.0], n))
    t1 = float(kw.get("time", 0) + 1)
    if plot == 6:
        vel = value / np.maximum(np.sqrt(gx * gx + gy * gy) * kw["flux_scale"], 1e-30)
    else:
        if plot in (4, 5, 9):
            value = np.exp((value - kw["log_shift"]) / kw["log_scale"])
        value = value * (t1 if plot in (3, 5) else 4.0 if plot in (8, 9) else 1.0)
        vel = np.sqrt(np.maximum(value - grad, 0.0)) / p.e_scale
    tiny = np.abs(phi) * 10.0 ** rng.uniform(-20, -9, n)
    pick = rng.random(n)
    vel = np.where(pick < 0.1, tiny, np.where(pick < 0.15, z, vel)) * rng.choice([-1.0, 1.0], n)
    return phi - np.where(np.isfinite(vel), vel, 0.0)


MODES = {1: dict(slope=1.5, scale=40.0), 2: dict(slope=1.5, scale=40.0), 3: dict(slope=1.5, scale=40.0, time=3),
         4: dict(slope=1.0, scale=1.5, log_scale=0.25, log_shift=0.1), 5: dict(slope=1.0, scale=1.5, log_scale=0.25, log_shift=0.1, time=2),
         6: dict(slope=1.0, scale=1.0, flux_scale=3e4), 8: dict(slope=1.5, scale=40.0, avrg_e_factor=0.75),
         9: dict(slope=1.0, scale=1.5, log_scale=0.25, log_shift=0.1, avrg_e_factor=0.75)}


@pytest.mark.parametrize("plot", sorted(MODES))
@pytest.mark.parametrize("prec", [P.FP32, P.FP64])
@pytest.mark.parametrize("rough", [1e-3, 1e-6, 0.0])
def test_other_modes_at_the_palette_boundaries(plot, prec, rough):
    """Energies, fluxes and their logarithms, means and averages on, next to and between the palette's
    boundaries, over rough, smooth and flat fields.  The oracle's and the GPU's tanh and log are
    each within 2 ulp and the energies are rounded alike, so a pixel may differ only where the
    oracle's 256-fold index lies within 256 * 16 * 2^-53 * (1 + |log|) < 1e-11 of a whole number."""
    nx, ny = 65, 259
    n = nx * ny
    rng = np.random.default_rng(plot * 10 + prec)
    p = P.make_params(nx, ny, b_cond=P.BC_DIRICHLET, courant=0.1, courantb=0.06, twospeeds=1)
    kw = dict(dict(size=1, color_range=0.8, log_scale=1.0, log_shift=0.0, flux_scale=1.0), **MODES[plot])
    phi = (0.5 * rng.choice([1.0, -1.0]) + rough * rng.standard_normal(n)).astype(np.float32).astype(np.float64)
    if plot == 2:  # the half drawn by the field itself
        amp = (rng.integers(30, 226, n) / 128.0 - 1.0) / kw["color_range"]
        u = np.arctanh(amp) * kw["scale"] / kw["slope"] * (1.0 + rng.choice([0.0, 1e-9, 1e-7, 1e-6, 1e-4], n))
        phi = np.where(np.tile(np.arange(ny) > ny // 2 + 1, nx), u, phi)
        phi = phi.astype(np.float32).astype(np.float64) if prec == P.FP32 else phi
    psi = boundary_energies(p, plot, phi, kw, rng)
    xy = np.ones(n, np.int16)
    L = np.repeat(np.arange(256), 3).reshape(256, 3).astype(np.uint8)
    with W.Scene(p, prec, P.COEF_MASK) as s:
        s.upload(phi, psi, xy)
        img = s.frame_rgb8(L, plot=plot, **kw)
        phi, psi = s.download()
    ref = oracle.frame_rgb8(p, phi, xy, L, plot=plot, psi=psi, **kw)
    hv = palette_position(p, plot, phi, psi, xy, kw)
    near = np.abs(hv - np.round(hv)) < 1e-11
    diff = np.any(img != ref, axis=-1)
    assert len(np.unique(ref)) > 20 or (plot == 6 and rough == 0.0)  # (a flat field has no flux)
    assert not np.any(diff & ~near), (int(diff.sum()), np.argwhere(diff & ~near)[:5], hv[diff & ~near][:5])


@pytest.mark.parametrize("plot", [1, 4, 6])
@pytest.mark.parametrize("color_range", [0.8, 3.0])
def test_velocities_below_an_ulp_of_phi(plot, color_range):
    """FP32 fields far from zero whose velocity, after damped updates, is no multiple of phi's FP64 ulp:
    psi = phi - v, and the energy from it, lose all or part of v in the oracle."""
    nx, ny = 40, 96
    n = nx * ny
    rng = np.random.default_rng(3)
    p = P.make_params(nx, ny, b_cond=P.BC_DIRICHLET, courant=0.1, gamma=0.3)
    band = np.repeat(10.0 ** np.arange(0, 8), nx // 8)  # flat bands of 5 rows
    phi = np.repeat(band, ny)
    psi = phi - np.repeat(band * rng.choice([1, 2, 5, 40], nx) * 2.0 ** -53, ny)
    kw = dict(size=1, slope=1.0, scale=3.0, log_scale=0.25, log_shift=2.0, flux_scale=1e9, color_range=color_range)
    L = np.repeat(np.arange(256), 3).reshape(256, 3).astype(np.uint8)
    xy = np.ones(n, np.int16)
    with W.Scene(p, P.FP32, P.COEF_MASK) as s:
        s.set_blocking(1)
        s.upload(phi, psi, xy)
        for _ in range(4):
            s.step(1)
            img = s.frame_rgb8(L, plot=plot, **kw)
            x, y = s.download()
            ref = oracle.frame_rgb8(p, x, xy, L, plot=plot, psi=y, **kw)
            hv = palette_position(p, plot, x, y, xy, kw)
            diff = np.any(img != ref, axis=-1) & (np.abs(hv - np.round(hv)) >= 1e-11)
            assert not diff.any(), (int(diff.sum()), np.argwhere(diff)[:5])


def test_log_energy_of_a_velocity_that_psi_loses():
    """A flat FP32 field whose velocity is less than half an FP64 ulp of phi: the oracle's energy is 0, FP32's
    is not, and they differ by far more than their logarithm's first-order error."""
    nx, ny = 9, 40
    n = nx * ny
    p = P.make_params(nx, ny, b_cond=P.BC_DIRICHLET, courant=0.1, gamma=0.6, e_scale=1e6)
    phi = np.full(n, float(np.float32(1e26)))
    psi = phi - np.spacing(phi)
    kw = dict(size=1, slope=1.0, scale=1.0, log_scale=2e-4, log_shift=0.0328, color_range=30.0)
    L = np.repeat(np.arange(256), 3).reshape(256, 3).astype(np.uint8)
    with W.Scene(p, P.FP32, P.COEF_MASK) as s:
        s.set_blocking(1)
        s.upload(phi, psi, np.ones(n, np.int16))
        s.step(1)
        img = s.frame_rgb8(L, plot=4, **kw)
        x, y = s.download()
    assert np.array_equal(x, y)
    assert np.array_equal(img, oracle.frame_rgb8(p, x, np.ones(n), L, plot=4, psi=y, **kw))
