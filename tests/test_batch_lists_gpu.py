"""Task lists of a batch's skewed passes, from one small grid (less than a task per team, chunks
of 8 rows) to more tasks than teams fit on the GPU (taken by ticket after the first per block):
each scene bit for bit the scene alone on single updates, at odd depths and frame lengths."""
import numpy as np
import pytest

from youtube_simulations_gb300 import params as P
from youtube_simulations_gb300 import wavegpu as W

pytestmark = pytest.mark.gpu


def instance(k, nx, ny, bc):
    rng = np.random.default_rng(1000 + k)
    p = P.make_params(nx, ny, b_cond=bc, courant=float(rng.uniform(0.05, 0.15)), gamma=1e-4 * (k % 3))
    xy = (rng.random(nx * ny) < 0.8).astype(np.int16)
    if k % 5 == 1 and bc != P.BC_PERIODIC:
        p.src_on, p.src_i, p.src_j, p.src_amp, p.src_period = 1, nx // 2, ny // 2, 0.05, 23.0
        xy[(nx // 2) * ny + ny // 2] = 1
    phi = np.where(xy != 0, rng.standard_normal(nx * ny), 0.0)
    return p, phi, np.where(xy != 0, 0.9 * phi, 0.0), xy


@pytest.mark.parametrize("bc", [P.BC_DIRICHLET, P.BC_ABSORBING, P.BC_PERIODIC])
@pytest.mark.parametrize("count,nx,ny", [(2, 4, 9), (3, 6, 13), (1, 9, 40), (1, 131, 257), (3, 33, 240), (40, 70, 129), (420, 61, 250)])
@pytest.mark.parametrize("mode", [3, 6, -1])
def test_lists_of_every_length(bc, count, nx, ny, mode):
    with W.Batch(P.FP32) as b:
        b.set_skew(mode)
        inst = [instance(k, nx, ny, bc) for k in range(count)]
        slots = [b.add(*i) for i in inst]
        for n in (10, 7, 4):
            b.step(n)
        for k in range(0, count, max(1, count // 7)):
            p, phi, psi, xy = inst[k]
            with W.Scene(p, P.FP32, P.COEF_MASK) as s:
                s.set_blocking(1)
                s.upload(phi, psi, xy)
                s.step(21)
                ref = s.download()
            got = b.download(slots[k])
            for x, y in zip(got, ref):
                assert np.array_equal(np.asarray(x).view(np.int64), np.asarray(y).view(np.int64)), k


@pytest.mark.parametrize("bc", [P.BC_PERIODIC, P.BC_DIRICHLET, P.BC_ABSORBING])
@pytest.mark.parametrize("count,nx,ny", [(420, 61, 129), (420, 61, 241), (6, 131, 257), (3, 40, 113)])
@pytest.mark.parametrize("mode", [6, 5, -1])
def test_deep_passes_near_the_stability_limit(bc, count, nx, ny, mode):
    """Frames cut into passes of the greatest depth (6, 12 and 16 updates), each reading what the one before
    wrote, at Courant numbers where a wrong value at the far end of a halo is not lost in
    rounding; one column in the last group of four, lists with and without tickets."""
    with W.Batch(P.FP32) as b:
        b.set_skew(mode)
        inst = []
        for k in range(count):
            p, phi, psi, xy = instance(k, nx, ny, bc)
            p.courant = (0.65, 0.5, 0.3)[k % 3]
            inst.append((p, phi, psi, xy))
        slots = [b.add(*i) for i in inst]
        for n in (6, 12, 16):
            b.step(n)
        for k in range(0, count, max(1, count // 9)):
            p, phi, psi, xy = inst[k]
            with W.Scene(p, P.FP32, P.COEF_MASK) as s:
                s.set_blocking(1)
                s.upload(phi, psi, xy)
                s.step(34)
                ref = s.download()
            assert np.isfinite(ref[0]).all()
            for x, y in zip(b.download(slots[k]), ref):
                assert np.array_equal(np.asarray(x).view(np.int64), np.asarray(y).view(np.int64)), k
