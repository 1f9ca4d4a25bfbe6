"""Periodic FP32 scenes on skewed passes (ghost layout): the values of the scene on single updates,
for every coefficient form, at widths around a tile and grids smaller than the halo, with
everything between the steps that writes the fields, the mask or the tables: a pulse, new
fields, a new domain, single updates."""
import numpy as np
import pytest
import torch

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


@pytest.mark.parametrize("ny", [109, 113, 114, 115, 117, 225, 241, 257, 717])
@pytest.mark.parametrize("courant", [0.3, 0.5, 0.65])
@pytest.mark.parametrize("coef,kw", [(P.COEF_MASK, dict()), (P.COEF_TABLE, dict(twospeeds=1, courantb=0.2, gammab=1e-4)),
                                     (P.COEF_MASK, dict(floor_clamp=1, vmax=2.0))])
def test_ghosts_of_the_last_group_of_columns(ny, courant, coef, kw):
    """Passes that read the ghosts another pass wrote, at Courant numbers near the stability limit, where
    a wrong value at the far end of a halo is not lost in rounding: widths that leave the last
    group of four columns one, two, three and four cells, in one tile and in several."""
    nx = 45
    rng = np.random.default_rng(ny)
    n = nx * ny
    p = P.make_params(nx, ny, b_cond=P.BC_PERIODIC, courant=courant, **kw)
    xy = (rng.random(n) < 0.9).astype(np.int16)
    f = (rng.standard_normal(n), rng.standard_normal(n), xy) + (scenes.tables(p, xy) if coef == P.COEF_TABLE else ())

    def run(blocking):
        out = []
        with W.Scene(p, P.FP32, coef) as s:
            s.upload(*f)
            s.set_blocking(*blocking)
            for steps in (6, 12, 18, 11):
                s.step(steps)
                out += s.download(native=True)
        return out
    ref = run((1,))
    assert all(np.isfinite(a).all() for a in ref)
    for blocking in [(5, 8, 1), (6, 8, 1), (6, 64, 1)]:
        for a, b in zip(run(blocking), ref):
            assert np.array_equal(a, b), blocking


def recorded(stream, call):
    """`call` recorded as a graph on the (torch) stream; it does not run."""
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        g.capture_begin()
        try:
            call()
        finally:
            g.capture_end()
    return g


def replay(stream, g):
    with torch.cuda.stream(stream):
        g.replay()


@pytest.mark.parametrize("blocking", [None, (6, 8, 1), (5, 64, 1)])
@pytest.mark.parametrize("steps", [6, 10])
def test_recorded_before_the_first_call(blocking, steps):
    """A call may be recorded on a periodic scene that has not been stepped, and so not tuned, yet."""
    nx, ny = 37, 131
    n = nx * ny
    rng = np.random.default_rng(5)
    p = P.make_params(nx, ny, b_cond=P.BC_PERIODIC, courant=0.5, twospeeds=1, courantb=0.3)
    f = rng.standard_normal(n), rng.standard_normal(n), (rng.random(n) < 0.9).astype(np.int16)
    with W.Scene(p, P.FP32, P.COEF_MASK) as s:
        s.set_blocking(1)
        s.upload(*f)
        s.step(2 * steps)
        want = s.download()
    st = torch.cuda.Stream()
    with W.Scene(p, P.FP32, P.COEF_MASK, stream=st.cuda_stream) as s:
        s.upload(*f)
        if blocking:
            s.set_blocking(*blocking)
        g = recorded(st, lambda: s.step(steps))
        for _ in range(2):
            replay(st, g)
        got = s.download()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind", ["step", "pulse", "state"])
def test_replays_between_calls(kind):
    """A replayed graph changes the fields without notice: the next call's ghosts are the new fields'."""
    nx, ny = 37, 131
    n = nx * ny
    rng = np.random.default_rng(6)
    p = P.make_params(nx, ny, b_cond=P.BC_PERIODIC, courant=0.5, twospeeds=1, courantb=0.3)
    f = rng.standard_normal(n), rng.standard_normal(n), (rng.random(n) < 0.9).astype(np.int16)
    rows = [torch.from_numpy(rng.standard_normal(n).astype(np.float32)).pin_memory() for _ in range(2)]
    st = torch.cuda.Stream()

    def call(s):
        if kind == "step":
            s.step(4)
        elif kind == "pulse":  # over a corner
            s.add_circular_wave(1.0, -1.98, 1.1, variance=0.05)
        else:
            W.check(W.lib().wg_scene_upload_state(s.h, rows[0].data_ptr(), rows[1].data_ptr(), P.FP32))

    def run(blocking, as_graph):
        with W.Scene(p, P.FP32, P.COEF_MASK, stream=st.cuda_stream) as s:
            s.upload(*f)
            s.set_blocking(*blocking)
            s.step(4)
            g = recorded(st, lambda: call(s)) if as_graph else None
            for _ in range(3):
                replay(st, g) if as_graph else call(s)
                s.step(4)
            return s.download(native=True)
    want = run((1,), False)
    for a, b in zip(run((2, 8, 1), True), want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("nx,ny,blocking", [(37, 131, (6, 8, 1)), (37, 131, (3, 16, 1)), (700, 45, None)])
@pytest.mark.parametrize("steps", [2, 4, 6, 10, 18])
@pytest.mark.parametrize("warm", [True, False])
def test_replays_advance_the_scene(nx, ny, blocking, steps, warm):
    """A graph of an even number of updates leaves the fields in the buffers that it holds, as single updates
    do, whether the scene was tuned and stepped before, and with other calls in between: steps of any
    even length, another blocking (the graph keeps its task lists), a first tuning."""
    n = nx * ny
    rng = np.random.default_rng(7)
    p = P.make_params(nx, ny, b_cond=P.BC_PERIODIC, courant=0.5, twospeeds=1, courantb=0.3)
    f = rng.standard_normal(n), rng.standard_normal(n), (rng.random(n) < 0.9).astype(np.int16)
    st = torch.cuda.Stream()

    def run(blk, as_graph):
        with W.Scene(p, P.FP32, P.COEF_MASK, stream=st.cuda_stream) as s:
            s.upload(*f)
            if blk:
                s.set_blocking(*blk)
            if warm:
                s.step(steps)
            g = recorded(st, lambda: s.step(steps)) if as_graph else None

            def again():
                replay(st, g) if as_graph else s.step(steps)
            again()
            again()
            s.step(6)
            again()
            if as_graph:
                s.set_blocking(6, 64, 1)
            s.step(12)
            again()
            return s.download(native=True)
    want = run((1,), False)
    for a, b in zip(run(blocking, True), want):
        assert np.array_equal(a, b)


def test_upload_that_fails_half_way():
    """An upload without the tables it needs is refused after the mask has changed: the next steps take that
    mask's ghosts too, as single updates take the mask."""
    nx, ny = 37, 131
    n = nx * ny
    rng = np.random.default_rng(8)
    p = P.make_params(nx, ny, b_cond=P.BC_PERIODIC, courant=0.5)
    xy, other = ((rng.random(n) < q).astype(np.int16) for q in (0.9, 0.5))
    f = rng.standard_normal(n), rng.standard_normal(n)
    out = []
    for blocking in [(1,), (6, 8, 1)]:
        with W.Scene(p, P.FP32, P.COEF_TABLE) as s:
            s.upload(*f, xy, *scenes.tables(p, np.ones_like(xy)))
            s.set_blocking(*blocking)
            s.step(12)
            with pytest.raises(W.WaveGpuError):
                s.upload(*f, other)
            s.step(12)
            out.append(s.download(native=True))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_calls_of_two_updates():
    """Calls of 2 updates take single updates, beside calls that take passes."""
    nx, ny = 45, 225
    n = nx * ny
    rng = np.random.default_rng(11)
    p = P.make_params(nx, ny, b_cond=P.BC_PERIODIC, courant=0.6)
    f = rng.standard_normal(n), rng.standard_normal(n), (rng.random(n) < 0.9).astype(np.int16)
    out = []
    for blocking in [(1,), (6, 8, 1), (2, 8, 1)]:
        with W.Scene(p, P.FP32, P.COEF_MASK) as s:
            s.upload(*f)
            s.set_blocking(*blocking)
            for k in (2, 6, 2, 2, 4, 3, 2, 1, 2, 12):
                s.step(k)
            out.append(s.download(native=True))
    for got in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got, out[0]))
