"""Downloads into page-locked rows, which the forming kernel writes in place in whole lines: rows
that start anywhere in a line, either row alone, grids of one lane to several blocks, both
precisions, scenes and batches; the same bits as through pageable rows, and nothing beside them."""
import ctypes

import numpy as np
import pytest
import torch

from youtube_simulations_gb300 import params as P
from youtube_simulations_gb300 import wavegpu as W

pytestmark = pytest.mark.gpu


def pinned(n, offset, dt):
    """An array of n cells, `offset` cells into page-locked memory, and the whole of it (filled with 7)."""
    whole = torch.empty((n + 2 * offset + 40,), dtype=dt, pin_memory=True).numpy()
    whole[:] = 7.0
    return whole[offset:offset + n], whole


@pytest.mark.parametrize("nx,ny", [(3, 3), (3, 8), (5, 33), (31, 64), (64, 131), (67, 257)])
@pytest.mark.parametrize("prec,native", [(P.FP32, True), (P.FP32, False), (P.FP64, False)])
@pytest.mark.parametrize("offsets", [(0, 0), (1, 3), (17, 30)])
def test_page_locked_rows(nx, ny, prec, native, offsets):
    rng = np.random.default_rng(nx + ny)
    n = nx * ny
    p = P.make_params(nx, ny, b_cond=P.BC_DIRICHLET, courant=0.1)
    xy = np.ones(n, np.int16)
    f = rng.standard_normal(n), rng.standard_normal(n)
    dt = torch.float32 if native else torch.float64
    code = P.FP32 if native else P.FP64
    with W.Scene(p, prec, P.COEF_MASK) as s, W.Batch(prec) as b:
        s.upload(*f, xy)
        s.step(1)
        slot = b.add(p, *f, xy)
        b.step(1)
        ref = s.download(native=native)
        calls = [lambda x, y: W.lib().wg_scene_download(s.h, x, y, code)]
        if not native:
            calls.append(lambda x, y: W.lib().wg_batch_download(b.h, slot, x, y))
        for call in calls:
            for use in ((True, True), (True, False), (False, True)):
                rows = [pinned(n, o, dt) for o in offsets]
                W.check(call(*(ctypes.c_void_p(r.ctypes.data) if u else None for (r, _), u in zip(rows, use))))
                for (r, whole), u, o, want in zip(rows, use, offsets, ref):
                    assert np.array_equal(r, want) if u else np.all(r == 7.0)
                    assert np.all(whole[:o] == 7.0) and np.all(whole[o + n:] == 7.0)
        both, _ = pinned(n, 1, dt)  # the same rows twice: psi's copy comes last
        W.check(calls[0](both.ctypes.data, both.ctypes.data))
        assert np.array_equal(both, ref[1])


@pytest.mark.parametrize("prec,native,shift", [(P.FP32, True, 1), (P.FP32, True, 2), (P.FP32, False, 1), (P.FP32, False, 4),
                                               (P.FP64, False, 2), (P.FP64, False, 4)])
def test_page_locked_rows_not_aligned_to_their_cells(prec, native, shift):
    """Rows at any byte address are copied, not accessed as cells in place: the same values, down and up."""
    nx, ny = 13, 37
    n = nx * ny
    dt = np.dtype(np.float32 if native else np.float64)
    code = P.FP32 if native else P.FP64
    rng = np.random.default_rng(shift)
    f = rng.standard_normal(n), rng.standard_normal(n)
    whole = [torch.zeros(n * dt.itemsize + 16, dtype=torch.uint8, pin_memory=True).numpy() for _ in range(2)]
    rows = [w[shift:shift + n * dt.itemsize] for w in whole]
    with W.Scene(P.make_params(nx, ny, courant=0.1), prec, P.COEF_MASK) as s, W.Batch(prec) as b:
        s.upload(*f, np.ones(n, np.int16))
        s.step(3)
        want = s.download(native=native)
        W.check(W.lib().wg_scene_download(s.h, rows[0].ctypes.data, rows[1].ctypes.data, code))
        got = [r.copy().view(dt) for r in rows]
        assert all(np.array_equal(g, w) for g, w in zip(got, want))
        W.check(W.lib().wg_scene_upload_state(s.h, rows[0].ctypes.data, rows[1].ctypes.data, code))
        up = s.download(native=native)
        s.upload_state(*want)
        assert all(np.array_equal(g, w) for g, w in zip(up, s.download(native=native)))
        if not native:
            slot = b.add(s.params, *f, np.ones(n, np.int16))
            b.step(3)
            W.check(W.lib().wg_batch_download(b.h, slot, rows[0].ctypes.data, rows[1].ctypes.data))
            assert all(np.array_equal(r.copy().view(dt), w) for r, w in zip(rows, b.download(slot)))


@pytest.mark.parametrize("nx,ny", [(2045, 2049), (2050, 2053)])
def test_fp64_rows_below_and_above_the_in_place_size(nx, ny):
    """FP64 rows of less than 32 MB are copied, larger page-locked ones written in place."""
    n = nx * ny
    f = np.random.default_rng(1).standard_normal(n)
    rows = [pinned(n, o, torch.float64) for o in (1, 3)]
    with W.Scene(P.make_params(nx, ny, courant=0.1), P.FP64, P.COEF_MASK) as s:
        s.upload(f, 0.5 * f, np.ones(n, np.int16))
        s.step(1)
        ref = s.download()
        W.check(W.lib().wg_scene_download(s.h, rows[0][0].ctypes.data, rows[1][0].ctypes.data, P.FP64))
    for (r, whole), o, want in zip(rows, (1, 3), ref):
        assert np.array_equal(r, want)
        assert np.all(whole[:o] == 7.0) and np.all(whole[o + n:] == 7.0)
