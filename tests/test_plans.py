"""The host arithmetic that chooses launch shapes (csrc/ug_plan.h), compiled alone."""
import ctypes
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "unsupervised_growth_gb300" / "csrc"

SOURCE = r"""
#include "ug_plan.h"
extern "C" int shape(int n_ra, int n_i, int req_ra, int req_i, int sms, int resident, int* out)
{
    const bool fits[2] = {(resident & 1) != 0, (resident & 2) != 0};
    const ug::UnitsShape u = ug::units_shape(n_ra, n_i, req_ra, req_i, sms, fits);
    if (!u.lanes) return 0;
    const int v[] = {u.lanes, u.ra_units, u.i_units, u.ra_per, u.i_per, u.nb_ra, u.nb_i, u.nb_sync, u.nb_row};
    for (int k = 0; k < 9; ++k) out[k] = v[k];
    return u.blocks();
}
"""


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    d = tmp_path_factory.mktemp("plans")
    (d / "plans.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), str(d / "plans.cpp"),
                    "-o", str(d / "plans.so")], check=True)
    return ctypes.CDLL(str(d / "plans.so"))


def units_shape(plans, n_ra, n_i, req=(0, 0), sms=152, resident=3):
    out = (ctypes.c_int * 9)()
    blocks = plans.shape(n_ra, n_i, *req, sms, resident, out)
    names = ("lanes", "ra_units", "i_units", "ra_per", "i_per", "nb_ra", "nb_i", "nb_sync", "nb_row")
    return blocks, dict(zip(names, out)) if blocks else {}


@pytest.mark.parametrize("n_ra", [1, 33, 300, 2000, 3600, 5000, 8000])
@pytest.mark.parametrize("ratio", [0.02, 0.25, 1.0])
def test_growth_trial_roles_cover_the_network(plans, n_ra, ratio):
    n_i = max(2, int(n_ra * ratio))
    blocks, u = units_shape(plans, n_ra, n_i)
    assert 0 < blocks <= 152 and u["nb_row"] >= 8
    assert blocks == u["nb_ra"] + u["nb_i"] + u["nb_sync"] + u["nb_row"]
    assert u["nb_ra"] * u["ra_per"] >= u["ra_units"] and u["ra_units"] * 32 * u["lanes"] >= n_ra
    assert u["nb_i"] * u["i_per"] >= u["i_units"] and u["i_units"] * 32 >= n_i


@pytest.mark.parametrize("n_ra", [8001, 10000, 18000, 25000, 60000])
@pytest.mark.parametrize("req", [(0, 0), (256, 256)])
def test_large_networks_take_the_interval_launches(plans, n_ra, req):
    """Their rows and LTP need the whole GPU: one launch leaves them a third of it or less, is
    slower there, and a busy interval outlasts its bounded waits."""
    assert units_shape(plans, n_ra, n_ra // 4, req)[0] == 0


def test_requested_widths(plans):
    assert units_shape(plans, 300, 75, (33, 32))[0] == 0           # not whole warps
    assert units_shape(plans, 300, 75, (288, 32))[0] == 0          # wider than a block
    assert units_shape(plans, 3600, 40, (32, 32))[1]["lanes"] == 1
    assert units_shape(plans, 4200, 40, (32, 32))[1]["lanes"] == 2   # 132 blocks with one neuron per thread
    assert units_shape(plans, 8000, 8000, (32, 32))[0] == 0        # no blocks left for the rows


@pytest.mark.parametrize("n_ra", [33, 2000, 8000])
def test_a_kernel_no_sm_can_hold_is_not_planned(plans, n_ra):
    """resident: bit 0 the form with one HVC(RA) neuron per thread, bit 1 the one with two."""
    assert units_shape(plans, n_ra, 40, resident=0)[0] == 0
    assert units_shape(plans, n_ra, 40, resident=1)[1]["lanes"] == 1
    assert units_shape(plans, n_ra, 40, resident=2)[1]["lanes"] == 2
