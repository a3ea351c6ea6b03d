"""Arithmetic the kernels share with the host (csrc/ug_hd.h), compiled alone."""
import ctypes
import math
import re
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "unsupervised_growth_gb300" / "csrc"

SOURCE = r"""
#include "ug_hd.h"
#include <cmath>
extern "C" void div_known(const double* x, double d, double* out, int n)
{
    const double z = 1.0 / d;
    for (int k = 0; k < n; ++k) out[k] = ug::div_known(x[k], d, z);
}
extern "C" int list_start(int resume, int at, int cap) { return ug::list_start(resume != 0, at, cap); }
"""


@pytest.fixture(scope="module")
def hd(tmp_path_factory):
    d = tmp_path_factory.mktemp("hd")
    (d / "hd.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wall", "-Werror", "-shared", "-fPIC", "-I", str(CSRC),
                    str(d / "hd.cpp"), "-o", str(d / "hd.so")], check=True)
    return ctypes.CDLL(str(d / "hd.so"))


@pytest.mark.parametrize("cap", [2, 65, 315])
def test_resumed_event_lists_stay_inside(hd, cap):
    """A list of cap entries keeps the last for its mark, so the closing mark of a resumed list
    lies inside it even where the first segment filled it."""
    assert hd.list_start(0, 7, cap) == 0
    for listed in range(cap):   # a segment lists at most cap - 1 events, its mark behind them
        at = hd.list_start(1, listed, cap)
        assert at == (listed + 1 if listed + 1 < cap else cap - 1)
        assert at < cap


def divisors():
    """Every fixed divisor of the double-precision kernels with eight lanes per neuron: of the
    gates' exponentials, the areas, the update's 6 and 3, and the Dormand-Prince tableau."""
    src = (CSRC / "ug_neuron.cuh").read_text()
    tableau = re.findall(r"#define UG_DP_(?:B\d+|OUT) ((?:[^\n]*\\\n)*[^\n]*)", src)
    dens = {float(d) for row in tableau for d in re.findall(r"\{\d+, [-\d.]+, ([\d.]+)\}", row)}
    assert len(dens) > 40
    return sorted(dens | {18, 48, 32, 64, 80, 6, 3, 5000, 10000, 9.5, 10, 15, 5, 7, 20, 2.0 ** 50 - 1})


def test_division_by_a_known_divisor(hd):
    """div_known(x, d, 1 / d) is x / d to the bit: over the whole range of exponents, for x
    whose quotient lies next to the middle of two doubles, and on its rare path (quotients
    near both ends of the range, subnormal and zero x of either sign, infinities, NaN)."""
    hd.div_known.argtypes = [ctypes.c_void_p, ctypes.c_double, ctypes.c_void_p, ctypes.c_int]
    rng = np.random.default_rng(3)
    rare = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.0 ** -1022, -2.0 ** -1022, 2.0 ** -1023,
                     np.nextafter(np.inf, 0), -np.nextafter(np.inf, 0)])
    for d in divisors():
        m = rng.uniform(1.0, 2.0, 4000)
        x = np.ldexp(m * rng.choice([-1.0, 1.0], m.size), rng.integers(-1074, 1024, m.size))
        edges = np.concatenate([np.ldexp(m[:200], e) for e in range(-1000, -880, 3)] +
                               [np.ldexp(m[:200], e) for e in range(1000, 1024, 3)])
        # next to the middle of two doubles: d times (an odd multiple of half an ulp), rounded, and its neighbours
        half = [int(v) * 2 + 1 for v in rng.integers(2 ** 52, 2 ** 53, 2000)]
        num, den = (int(v) for v in float(d).as_integer_ratio())
        near = np.array([math.ldexp(h * num / (den << 60), 7) for h in half])
        near = np.concatenate([near, np.nextafter(near, 0), np.nextafter(near, np.inf)])
        x = np.ascontiguousarray(np.concatenate([x, edges, near, rare]))
        got = np.empty_like(x)
        hd.div_known(x.ctypes.data, d, got.ctypes.data, x.size)
        with np.errstate(all="ignore"):
            want = x / d
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64)), d
