"""The last reduction of an energy at one block of columns, a warp's, a block's and more than a
block's share of partial sums: totals, columns and boxes of FP64 scenes and batches against the oracle's
compensated sums.  Cell energies are the oracle's bits and the sums compensated on both sides, so
they agree to a few last bits of the result: 1e-14 relative."""
import numpy as np
import pytest

import oracle
from youtube_simulations_gb300 import params as P
from youtube_simulations_gb300 import wavegpu as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [3, 8, 9, 255, 256, 257, 2047, 2048, 2049, 2100])
def test_energy_sums(nx):
    ny = 12
    rng = np.random.default_rng(nx)
    n = nx * ny
    p = P.make_params(nx, ny, b_cond=P.BC_DIRICHLET, courant=0.1, twospeeds=1, courantb=0.06)
    xy = (rng.random(n) < 0.7).astype(np.int16)
    phi, psi = rng.standard_normal(n), rng.standard_normal(n)
    il, ir = nx // 3, 2 * nx // 3
    with W.Scene(p, P.FP64, P.COEF_MASK) as s, W.Batch(P.FP64) as b:
        s.upload(phi, psi, xy)
        total, cols, boxes = s.energy(ileft=il, iright=ir)
        assert s.total_energy() == total
        assert b.energy(b.add(p, phi, psi, xy)) == total
    want = oracle.energy_total(p, phi, psi, xy)
    assert abs(total - want) <= 1e-14 * want
    ref = oracle.energy_x(p, phi, psi, xy)
    assert np.all(np.abs(cols - ref) <= 1e-14 * ref)
    # the oracle's boxes are plain sums of up to n terms: their own error is at most n 2^-53
    ref = oracle.energy_tblr(p, phi, psi, xy, il, ir)
    assert np.all(np.abs(boxes - ref) <= (1e-14 + n * 2.0 ** -53) * ref)
