"""Cuts on grids whose num_cell + 1 buckets are a whole number of the scan's tiles of 2,048: the
contact queue's length, the word behind the buckets, starts each step at zero there as on every
other grid, and the fused step agrees with the CPU oracle as it does on those (test_gpu_parity)."""
import numpy as np
import pytest

from sph_fem_2d_cutting_gpu_gb300 import abi, setups, tune
from sph_fem_2d_cutting_gpu_gb300.solver import Solver
from test_gpu_parity import FUSED, compare, pair

pytestmark = pytest.mark.gpu


def small_cut_on(nx, ny):
    """The small cut on a grid of nx x ny cells."""
    c = setups.small_cut()
    g = c.grid
    for i, cells in enumerate((nx, ny)):
        g.bbmax[i] = g.bbmin[i] + (cells - 0.5) * g.h * g.cell_factor - 2e-6
    return c


def ordinary_cut():
    return setups.cutting("cut", setups.AISI1045, 245, 42, 5e-4, 1.7, 120.0, 0.008, 0.0, 6.0, 5e-4, 0.35, s_min=2e-4,
                          s_max=3e-3, tool_size=0.05)


@pytest.mark.parametrize("make,cells", [(lambda: small_cut_on(63, 65), 4095), (lambda: small_cut_on(89, 23), 2047),
                                        (ordinary_cut, 102_399)])
def test_fused_steps_match_oracle(lib, make, cells):
    c = make()
    s, o = pair(c, preload_dx=0.3)
    assert s.geometry().num_cell == cells
    for k in range(5):
        s.step()
        o.step()
        compare(s, o, FUSED, what=f"[{cells} cells, step {k}]")
    assert (s.download(["on_seg"])["on_seg"] >= 0).any(), "contact never became active"
    assert s.status() == 0


def test_fp32k_matches_persistent_form(lib):
    """The fast form on such a grid, bit for bit where the persistent form, which has no queue, ends."""
    c = setups.placed(small_cut_on(63, 65), preload_dx=0.3)
    out = []
    for form in (abi.SPH_STEP_LAUNCHES, abi.SPH_STEP_PERSISTENT):
        s = Solver(c, abi.SPH_PREC_FP32K, place_tool=False)
        tune.set_step_form(s, form)
        s.step(5)
        assert s.geometry().num_cell == 4095 and s.status() == 0
        out.append(s.download(["pos", "vel", "rho", "S", "T", "fc", "ft", "on_seg", "hash", "idx"]))
    assert (out[0]["on_seg"] >= 0).any(), "contact never became active"
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f], equal_nan=True), f
