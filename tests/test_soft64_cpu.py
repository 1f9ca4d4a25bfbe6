"""The integer form of the FP64 Laplacian (csrc/wg_soft64.h) against the machine's additions.

The header is host and device code; compiled here with g++, s64_laplacian must return the bits
of RN(RN(RN(RN(n + s) + e) + w) - 4x) (numpy float64, one rounding an operation) wherever it
accepts the operands, over random fields, nearly equal operands (deep cancellation), exponents
spread around the limit, significands at the ties of each rounding, zeros of both signs,
subnormals, infinities and NaN; it must accept what smooth fields hold and refuse the rest."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "youtube-simulations_gb300" / "csrc"
SRC = r"""
#include "wg_soft64.h"
extern "C" void lap(long n, const double *v, double *out, unsigned char *ok)
{
    for (long i = 0; i < n; i++) {
        bool k;
        const double *q = v + 5 * i;
        out[i] = wg::s64_laplacian(wg::s64_unpack(q[0]), wg::s64_unpack(q[1]), wg::s64_unpack(q[2]), wg::s64_unpack(q[3]),
                                   wg::s64_unpack(q[4]), k);
        ok[i] = k;
    }
}
"""


@pytest.fixture(scope="module")
def lap(tmp_path_factory):
    d = tmp_path_factory.mktemp("soft64")
    (d / "s.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-ffp-contract=off", f"-I{CSRC}", "-o", str(d / "s.so"), str(d / "s.cpp")],
                   check=True)
    L = ctypes.CDLL(str(d / "s.so"))

    def run(v):
        v = np.ascontiguousarray(v, np.float64)
        out, ok = np.empty(len(v)), np.empty(len(v), np.uint8)
        L.lap(ctypes.c_long(len(v)), v.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p),
              ok.ctypes.data_as(ctypes.c_void_p))
        return out, ok.astype(bool)
    return run


def want(v):
    with np.errstate(all="ignore"):
        return (((v[:, 0] + v[:, 1]) + v[:, 2]) + v[:, 3]) - 4.0 * v[:, 4]


def family(kind, n, rng):
    base = np.ldexp(rng.uniform(-1, 1, (n, 1)), rng.integers(-300, 300, (n, 1)))
    if kind == "uniform":
        return rng.uniform(-1, 1, (n, 5))
    if kind == "near":
        return base * (1 + 1e-3 * rng.standard_normal((n, 5)))
    if kind == "nearer":
        return base * (1 + 1e-14 * rng.integers(-30, 30, (n, 5)))
    if kind == "spread":
        return rng.uniform(-1, 1, (n, 5)) * np.ldexp(1.0, rng.integers(0, 10, (n, 5)))
    if kind == "ties":  # short and all-ones significands, exponents within the reach
        m = rng.choice([1.0, 1.5, 2 - 2.0 ** -52, 1 + 2.0 ** -52, 1 + 2.0 ** -51, 1 + 2.0 ** -50, 2 - 2.0 ** -51], (n, 5))
        return m * np.ldexp(1.0, rng.integers(0, 9, (n, 5))) * rng.choice([-1.0, 1.0], (n, 5))
    if kind == "zeros":
        v = rng.uniform(-1, 1, (n, 5))
        v[rng.random((n, 5)) < 0.5] = 0.0
        v[rng.random((n, 5)) < 0.1] = -0.0
        return v
    v = rng.uniform(-1, 1, (n, 5)) * rng.choice([1.0, 1e-310, 1e-320, 1e300, 1.7e308], (n, 5))
    v[rng.random((n, 5)) < 0.1] = rng.choice([np.inf, -np.inf, np.nan])
    return v


@pytest.mark.parametrize("kind", ["uniform", "near", "nearer", "spread", "ties", "zeros", "special"])
def test_laplacian_bits(lap, kind):
    rng = np.random.default_rng(11)
    v = family(kind, 300_000, rng)
    out, ok = lap(v)
    w = want(v)
    assert np.array_equal(out[ok].view(np.uint64), w[ok].view(np.uint64))
    if kind in ("uniform", "near", "ties"):
        assert ok.mean() > 0.8
    refused = ~np.isfinite(v).all(1) | (v.view(np.uint64) == np.uint64(1 << 63)).any(1) | \
        ((v != 0) & (np.abs(v) < 2.3e-308)).any(1)
    assert not ok[refused].any()


def test_all_zero_cell(lap):
    out, ok = lap(np.zeros((1, 5)))
    assert ok[0] and out.view(np.uint64)[0] == 0


SUB = r"""
#include "wg_soft64.h"
extern "C" void sub(long n, const double *v, double *out, unsigned char *ok)
{
    for (long i = 0; i < n; i++) {
        bool k;
        out[i] = wg::s64_sub(wg::s64_unpack(v[2 * i]), wg::s64_unpack(v[2 * i + 1]), k);
        ok[i] = k;
    }
}
"""


@pytest.mark.parametrize("kind", ["uniform", "near", "nearer", "spread", "ties", "zeros", "special"])
def test_difference_bits(tmp_path, kind):
    """s64_sub: the bits of x - y wherever it accepts them."""
    (tmp_path / "d.cpp").write_text(SUB)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-ffp-contract=off", f"-I{CSRC}", "-o", str(tmp_path / "d.so"), str(tmp_path / "d.cpp")],
                   check=True)
    rng = np.random.default_rng(12)
    v = np.ascontiguousarray(family(kind, 300_000, rng)[:, :2])
    if kind == "nearer":  # neighbours in the last bits, and equal
        v[:, 1] = v[:, 0] * (1.0 + 2.0 ** -52 * rng.integers(-6, 7, len(v)))
    out, ok = np.empty(len(v)), np.empty(len(v), np.uint8)
    ctypes.CDLL(str(tmp_path / "d.so")).sub(ctypes.c_long(len(v)), v.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p),
                                            ok.ctypes.data_as(ctypes.c_void_p))
    ok = ok.astype(bool)
    with np.errstate(all="ignore"):
        want = v[:, 0] - v[:, 1]
    assert np.array_equal(out[ok].view(np.uint64), want[ok].view(np.uint64))
    if kind in ("uniform", "near", "ties"):
        assert ok.mean() > 0.8
    refused = ~np.isfinite(v).all(1) | (v.view(np.uint64) == np.uint64(1 << 63)).any(1) | ((v != 0) & (np.abs(v) < 2.3e-308)).any(1)
    assert not ok[refused].any()
