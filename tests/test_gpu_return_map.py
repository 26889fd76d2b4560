"""FP64 return mapping: a case small enough for groups of four lanes (one wave of the sums'
blocks; with the registers of three blocks an SM up to 3 * 152 * 32 particles, of five up to
5 * 152 * 32) and the same case first in a batch too large for them, where each lane maps its
own particle.  They share their arithmetic rounding for rounding, so the case ends with the same
bits, yielding particles included."""
import numpy as np
import pytest

from sph_fem_2d_cutting_gpu_gb300 import abi, setups
from sph_fem_2d_cutting_gpu_gb300.solver import Batch

pytestmark = pytest.mark.gpu

FIELDS = ["pos", "vel", "rho", "S", "T", "eps_pl", "eps_pl_dot", "blanked", "fc", "hash"]


def cut(speed):
    c = setups.cutting("map", setups.AISI1045, 120, 50, 5e-4, 1.7, speed, 0.008, 0.0, 5.0, 5e-4, 0.35, s_min=2e-4,
                       s_max=2.5e-3, tool_size=0.02)
    return setups.placed(c, preload_dx=0.5)


@pytest.mark.parametrize("steps", [1, 40])
def test_lanes_and_groups_map_alike(lib, steps):
    out = []
    for n_cases in (1, 3, 5):
        b = Batch([cut(300.0)] + [cut(120.0 + 10 * k) for k in range(n_cases - 1)], abi.SPH_PREC_FP64)
        assert (b.N <= 3 * 152 * 32) == (n_cases == 1) and (b.N <= 5 * 152 * 32) == (n_cases <= 3)
        b.step(steps)
        out.append(b.download_cases(FIELDS)[0])
        b.close()
    for f in FIELDS:
        assert np.array_equal(out[0][f], out[1][f], equal_nan=True), f
        assert np.array_equal(out[0][f], out[2][f], equal_nan=True), f
    if steps == 40:
        assert np.count_nonzero(out[0]["eps_pl_dot"]) > 20   # particles on the yield surface
