"""Nearly hydrostatic states: the von Mises square of the return mapping (actions_gpu.cu:689-754)
is a difference of squares of the pressure's size, which cancels to a little above or below zero.
Below zero its root is NaN, the particle counts as yielding, and the reference maps it.  Which
particles these are hangs on how a compiler fuses the products; that it is a good part of them
does not.  The step in FP64, the step in FP32K and the CPU oracle treat such a block alike, and
the two in 64 bits map nothing where the deviator is large beside their rounding."""
import numpy as np
import pytest

from oracle.oracle import OracleSim
from sph_fem_2d_cutting_gpu_gb300 import abi, setups
from sph_fem_2d_cutting_gpu_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def block(deviator):
    """Uneven pressure (1 % of the bulk modulus), at rest; S: `deviator` times a small random stress."""
    c = setups.micro(n_side=64, seed=3)
    for f in ("vel", "pos_t", "vel_t", "rho_t", "S_t", "T_t"):
        c.particles[f][:] = 0.0
    c.particles["S"] *= deviator
    c.particles["rho"][:] = c.constants.phys.rho0 * (1.0 + np.random.default_rng(5).uniform(-1e-2, 1e-2, c.N))
    return c


def mapped_on_device(c, precision, staged):
    s = Solver(c, precision)
    (s.step_staged if staged else s.step)()
    G = s.download(["S", "eps_pl_dot"])
    s.close()
    return np.mean(G["eps_pl_dot"] != 0.0), np.mean(np.isnan(G["S"]).any(1))


@pytest.mark.parametrize("deviator", [0.0, 1e-12, 1e-9, 1e-3])
def test_mapped_as_in_the_reference(lib, deviator):
    c = block(deviator)
    o = OracleSim(c.constants, c.grid, {k: v.copy() for k, v in c.particles.items()}, c.dt)
    o.step()
    mapped = np.mean(o.P["eps_pl_dot"] != 0.0)
    assert (0.2 < mapped < 0.8) if deviator < 1e-6 else mapped == 0.0
    forms = [(abi.SPH_PREC_FP64, False), (abi.SPH_PREC_FP64, True), (abi.SPH_PREC_FP32K, False)]
    for precision, staged in forms if deviator < 1e-6 else forms[:2]:
        part, nan = mapped_on_device(c, precision, staged)
        assert (0.2 < part < 0.8) if deviator < 1e-6 else part == 0.0, (precision, staged)
        assert nan == (part if deviator == 0.0 else 0.0), (precision, staged)   # S / |S| of a zero stress
