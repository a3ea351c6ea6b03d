"""Arithmetic the kernels share with the host (csrc/ug_hd.h), compiled alone."""
import ctypes
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "unsupervised_growth_gb300" / "csrc"

SOURCE = r"""
#include "ug_hd.h"
extern "C" int list_start(int resume, int at, int cap) { return ug::list_start(resume != 0, at, cap); }
"""


@pytest.fixture(scope="module")
def hd(tmp_path_factory):
    d = tmp_path_factory.mktemp("hd")
    (d / "hd.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", str(CSRC),
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
