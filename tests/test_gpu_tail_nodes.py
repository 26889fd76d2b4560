"""The tool nodes' thermal update in the launch of the step's tail (up to 8 * 152 * 256
particles) and in one of its own (more): on both sides of the line the step ends bit for bit
where the persistent form, which always runs it as a phase of its own, does."""
import numpy as np
import pytest

from sph_fem_2d_cutting_gpu_gb300 import abi, setups, tune
from sph_fem_2d_cutting_gpu_gb300.solver import Solver

pytestmark = pytest.mark.gpu

FIELDS = ["pos", "vel", "rho", "S", "T", "eps_pl", "fc", "ft", "hash"]


def run(case, form):
    s = Solver(case, abi.SPH_PREC_FP32K, place_tool=False)
    tune.set_step_form(s, form)
    s.step(2)
    n0 = s.launch_count()
    s.step(2)
    out = s.download(FIELDS)
    out["T_nodes"] = s.fem()["T"]
    launches = s.launch_count() - n0
    s.close()
    return out, launches


@pytest.mark.parametrize("ny", [405, 406])
def test_tool_nodes_with_or_before_the_tail(lib, ny):
    nx, dx = 768, 5e-4
    assert (nx * ny <= 8 * 152 * 256) == (ny == 405)
    case = setups.placed(setups.cutting("tail", setups.AISI1045, nx, ny, dx, 1.7, 300.0, 0.3 * ny * dx, 0.0, 6.0, 2 * dx,
                                        0.35, s_min=2e-4, s_max=3e-3, tool_size=0.05), preload_dx=0.3)
    a, n_a = run(case, abi.SPH_STEP_LAUNCHES)
    b, n_b = run(case, abi.SPH_STEP_PERSISTENT)
    assert n_b < n_a   # fewer launches: the persistent form ran
    for f in a:
        assert np.array_equal(a[f], b[f], equal_nan=True), f
    assert np.any(a["T_nodes"] != a["T_nodes"][0])   # the update did run
