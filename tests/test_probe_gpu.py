"""SAVE_TIME_SERIES probes (wave_billiard.c:667-672, 900-908) on the GPU: phi at the
probe cells after every update, against the oracle stepped one update at a time
(FP64 bit for bit, FP32 within 1e-5 of the field maximum); the buffer refuses to
overflow and partial reads keep the rest; the drop-in's resident cell read."""
import numpy as np
import pytest

import oracle
from helpers import variant_inputs
from youtube_simulations_gb300 import params as P
from youtube_simulations_gb300 import wavegpu as W

pytestmark = pytest.mark.gpu

CELLS = [(10, 20), (33, 22), (60, 40), (0, 5)]


def oracle_series(p, f, xy, n):
    phi, psi, tmp = f["phi"], f["psi"], f["tmp"]
    out = []
    for _ in range(n):
        phi, psi, tmp, _ = oracle.run(p, phi, psi, tmp, xy, f["tcc"], f["tc"], f["tgamma"], 1)
        out.append([phi.reshape(p.nx, p.ny)[i, j] for i, j in CELLS])
    return np.array(out), phi


@pytest.mark.parametrize("prec", [P.FP64, P.FP32])
def test_probes_match_oracle_every_update(prec):
    p, f, xy, _ = variant_inputs("s_abs", seed=8)
    n = 12
    ref, final = oracle_series(p, f, xy, n)
    with W.Scene(p, prec, P.COEF_TABLE) as s:
        s.upload(f["phi"], f["psi"], xy, f["tcc"], f["tc"], f["tgamma"])
        s.set_probes(CELLS, capacity=n)
        s.step(5)
        first = s.read_probes(max_updates=3)   # partial read: updates 1-3
        s.step(7)
        rest = s.read_probes()                  # updates 4-12
        got = np.vstack([first, rest])
        with pytest.raises(W.WaveGpuError):
            s.step(n + 1)                       # would overflow the buffer
    assert got.shape == (n, len(CELLS))
    if prec == P.FP64:
        assert np.array_equal(got, ref)
    else:
        assert np.max(np.abs(got - ref)) <= 1e-5 * np.max(np.abs(final))


def test_probe_out_of_grid_refused():
    p, f, xy, _ = variant_inputs("s_abs", seed=8)
    with W.Scene(p, P.FP64, P.COEF_TABLE) as s:
        s.upload(f["phi"], f["psi"], xy, f["tcc"], f["tc"], f["tgamma"])
        with pytest.raises(W.WaveGpuError):
            s.set_probes([(p.nx, 0)], capacity=4)


def test_dropin_resident_cell():
    p, f, xy, _ = variant_inputs("s_dir", seed=4)
    new, _, _, _ = oracle.run(p, f["phi"], f["psi"], f["tmp"], xy, f["tcc"], f["tc"], f["tgamma"], 9)
    W.configure(p)
    W.set_mode(True)
    rf = W.RowFields(p, f["phi"], f["psi"], f["tmp"], xy, f["tcc"], f["tc"], f["tgamma"])
    for _ in range(3):
        W.evolve_wave(rf)
    for i, j in [(5, 7), (30, 20), (66, 44)]:
        assert W.dropin_cell(rf, i, j) == new.reshape(p.nx, p.ny)[i, j]
    W.set_mode(False)


@pytest.mark.parametrize("bc", [P.BC_PERIODIC, P.BC_DIRICHLET])
def test_probes_set_before_the_first_step(bc):
    """The first step of a size class times candidate blockings; the probes sample none of those updates."""
    nx, ny = 1100, 9 if bc == P.BC_PERIODIC else 17
    n = nx * ny
    rng = np.random.default_rng(1)
    p = P.make_params(nx, ny, b_cond=bc, courant=0.3)
    phi, xy = rng.standard_normal(n), np.ones(n, np.int16)
    cells = [(0, 0), (5, 3), (nx - 1, ny - 1)]
    got = []
    for blocking in (0, 1):
        with W.Scene(p, P.FP32, P.COEF_MASK) as s:
            if blocking:
                s.set_blocking(1)
            s.upload(phi, 0.9 * phi, xy)
            s.set_probes(cells, capacity=4000)
            s.step(7)
            got.append(s.read_probes())
    assert got[0].shape == (7, len(cells)) and np.array_equal(*got)
