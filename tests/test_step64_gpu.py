"""The FP64 update's strips (k_step64, k_batch_step64) at the sizes where they can go wrong:
grids one column short of, at and past the strip of 60 columns, one interior row, odd sizes;
every boundary rule, mask and table coefficients, and fields that the integer Laplacian takes,
refuses and mixes: noise, exponential tails over hundreds of binades, zeros of both signs,
subnormals, infinities.  Scenes and batches must hold the oracle's values, the drop-in the
oracle's bits."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import oracle
from helpers import equalize_unwritten
from youtube_simulations_gb300 import params as P
from youtube_simulations_gb300 import scenes
from youtube_simulations_gb300 import wavegpu as W

pytestmark = pytest.mark.gpu

SIZES = [(3, 3), (3, 59), (4, 60), (5, 61), (37, 62), (64, 119), (70, 121), (131, 180), (200, 301)]
BCS = [P.BC_DIRICHLET, P.BC_PERIODIC, P.BC_ABSORBING, P.BC_VPER_HABS]


def fields(kind, nx, ny, rng):
    n = nx * ny
    if kind == "noise":
        phi = rng.standard_normal(n)
    elif kind == "tail":
        x, y = np.meshgrid(np.linspace(-1, 1, nx), np.linspace(-1, 1, ny), indexing="ij")
        phi = (np.exp(-(x * x + y * y) * 900.0)).reshape(-1)
    elif kind == "zeros":
        phi = np.where(rng.random(n) < 0.5, 0.0, rng.standard_normal(n))
        phi = np.where(rng.random(n) < 0.1, -0.0, phi)
    else:
        phi = rng.standard_normal(n) * rng.choice([1.0, 1e-310, 1e300, 1e-3], n)
        phi[rng.integers(0, n)] = np.inf
    return phi


def setup(kind, nx, ny, bc, kappa, gamma, seed):
    rng = np.random.default_rng(seed)
    p = P.make_params(nx, ny, b_cond=bc, courant=0.1, kappa=kappa, gamma=gamma, gammab=gamma)
    xy = scenes.mask(p, scenes.D_CIRCLES, circles=[(-0.8, 0.3, 0.45), (1.2, -0.7, 0.3)])
    if bc == P.BC_ABSORBING:
        p.twospeeds, p.courantb = 1, 0.07
    phi = fields(kind, nx, ny, rng)
    psi = 0.97 * phi
    if not p.twospeeds:
        phi, psi = np.where(xy != 0, phi, 0.0), np.where(xy != 0, psi, 0.0)
    return p, xy, phi, psi, scenes.tables(p, xy)


@pytest.mark.parametrize("bc", BCS)
@pytest.mark.parametrize("kind", ["noise", "tail", "zeros", "special"])
@pytest.mark.parametrize("kappa,gamma", [(0.0, 0.0), (0.0, 1e-3), (1e-3, 2e-4)])
def test_scene_batch_and_dropin(bc, kind, kappa, gamma):
    n = 6
    for k, (nx, ny) in enumerate(SIZES):
        p, xy, phi, psi, tab = setup(kind, nx, ny, bc, kappa, gamma, 100 + k)
        f = equalize_unwritten(p, dict(phi=phi, psi=psi, tmp=np.zeros_like(phi)), xy)
        with np.errstate(all="ignore"):
            new, prev, third, _ = oracle.run(p, f["phi"], f["psi"], f["tmp"], xy, *tab, n)
        for coef in (P.COEF_MASK, P.COEF_TABLE):
            with W.Scene(p, P.FP64, coef) as s:
                s.upload(f["phi"], f["psi"], xy, *tab)
                s.step(n)
                a, b = s.download()
            assert np.array_equal(a, new, equal_nan=True) and np.array_equal(b, prev, equal_nan=True), (nx, ny, coef)
        with W.Batch(P.FP64) as bt:
            sl = bt.add(p, f["phi"], f["psi"], xy)
            bt.step(n)
            a, b = bt.download(sl)
        assert np.array_equal(a, new, equal_nan=True) and np.array_equal(b, prev, equal_nan=True), (nx, ny, "batch")
        W.configure(p)
        W.set_mode(True)
        rf = W.RowFields(p, f["phi"], f["psi"], f["tmp"], xy, *tab)
        for _ in range(n // 3):
            W.evolve_wave(rf)
        W.sync()
        W.set_mode(False)
        for got, w in ((rf.phi, new), (rf.psi, prev), (rf.tmp, third)):
            got, nan = got.reshape(-1), np.isnan(w)
            assert np.array_equal(np.isnan(got), nan)
            assert np.array_equal(got[~nan].view(np.uint64), w[~nan].view(np.uint64)), (nx, ny, "drop-in")


THREADS = """
import sys, threading
sys.path.insert(0, {tests!r})
import conftest  # noqa: F401  (loads the package)
import numpy as np
from youtube_simulations_gb300 import params as P
from youtube_simulations_gb300 import wavegpu as W

CASES = [(P.FP64, 0.0, P.BC_DIRICHLET), (P.FP64, 1e-3, P.BC_ABSORBING), (P.FP32, 0.0, P.BC_DIRICHLET), (P.FP32, 1e-3, P.BC_PERIODIC)]

def run(k, out):
    prec, kappa, bc = CASES[k % len(CASES)]
    p = P.make_params(150, 203, b_cond=bc, courant=0.3, kappa=kappa)
    f = np.random.default_rng(k % len(CASES)).standard_normal(150 * 203)
    with W.Scene(p, prec, P.COEF_MASK) as s:
        if prec == P.FP32:
            s.set_blocking(4, 16, 1)
        s.upload(f, 0.9 * f, np.ones(150 * 203, np.int16))
        for _ in range(5):
            s.step(4)
        out[k] = s.download()

got, want = {{}}, {{}}
threads = [threading.Thread(target=run, args=(k, got)) for k in range(12)]
[t.start() for t in threads]
[t.join() for t in threads]
[run(k, want) for k in range(12)]
assert all(np.array_equal(a, b) for k in range(12) for a, b in zip(got[k], want[k]))
print("same")
"""


def test_first_updates_from_several_threads():
    """A process whose first updates come from several threads at once: what the launches ask of the device
    and keep is the same whichever thread asks."""
    here = Path(__file__).resolve().parent
    r = subprocess.run([sys.executable, "-c", THREADS.format(tests=str(here))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
