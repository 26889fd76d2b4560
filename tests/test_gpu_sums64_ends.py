"""The FP64 neighbour sums (staged and fused) against the CPU oracle for velocities at which the
viscosity's products leave the doubles: a diverging state, whose infinities and NaN must come out
where the reference's do and blank the particles, and one nearly at rest, whose products are
subnormal.

Tolerance: as in test_gpu_sums64; and subnormal numbers are rounded by 2^-1075, under 20 times in
each of at most 60 terms, and the viscosity's are then divided by r^2 (above dx^2 / 2 on the
disturbed lattice) and multiplied by the gradient of W (below 0.5 / h^3) and the mass.  Between
speeds of 1e148 and 1e155 it depends on the order of the factors whether a product overflows."""
import numpy as np
import pytest

from oracle.oracle import OracleSim
from sph_fem_2d_cutting_gpu_gb300 import abi, setups
from sph_fem_2d_cutting_gpu_gb300.solver import Solver

pytestmark = pytest.mark.gpu

SUMS = ("S_der", "v_der", "pos_t", "vel_t", "T_t")


def lattice(speed):
    c = setups.micro(n_side=24, seed=3)
    rng = np.random.default_rng(4)
    c.particles["vel"][:] = rng.uniform(-1.0, 1.0, c.particles["vel"].shape) * speed
    if speed < 1.0:   # nothing but the velocities acts
        c.particles["S"][:] = 0.0
        c.particles["rho"][:] = c.constants.phys.rho0
        for f in ("pos_t", "vel_t", "rho_t", "S_t", "T_t"):
            c.particles[f][:] = 0.0
    return c


def agree(a, b, what, gain):
    finite = np.isfinite(b)
    assert np.array_equal(np.isfinite(a), finite), f"{what}: {np.count_nonzero(np.isfinite(a) != finite)} entries"
    if finite.any():
        a, b = a[finite], b[finite]
        scale = np.abs(b).max()
        assert np.abs(a / 2 - b / 2).max() <= 0.5e-12 * scale + 600 * gain * 2.0 ** -1074, what


@pytest.mark.parametrize("speed", [1e90, 1e145, 1e157, 1e170, 1e250, 1e-290, 1e-304, 1e-306, 1e-308, 1e-312])
def test_sums_match_oracle(lib, speed):
    c = lattice(speed)
    gain = max(1.0, 0.5 / c.grid.h ** 3 * c.constants.phys.mass) * 2.0 / c.info["dx"] ** 2
    s = Solver(c)
    o = OracleSim(c.constants, c.grid, s.download(), c.dt)
    for call in ("assign_hashes", "sort", "material_eos", "corrector_artificial_stress", "interactions_monaghan"):
        getattr(s, call)()
        with np.errstate(all="ignore"):
            getattr(o, call)()
    G = s.download()
    for f in SUMS:
        agree(G[f], o.P[f], f"{speed:g} {f}", gain)
    if speed > 1e155:
        assert not np.isfinite(G["vel_t"]).all()
    s.close()
    s = Solver(c)
    o = OracleSim(c.constants, c.grid, s.download(), c.dt)
    s.step()
    o.step()
    G = s.download()
    assert np.array_equal(G["blanked"], o.P["blanked"])
    assert bool(s.status() & abi.STATUS_BITS["nan_blanked"]) == (G["blanked"] == 1.0).any()
    if speed > 1e155:
        assert (G["blanked"] == 1.0).any()
    act = G["blanked"] != 1.0
    for f in ("vel", "vel_t", "pos_t", "rho_t"):
        agree(G[f][act], o.P[f][act], f"{speed:g} fused {f}", gain)
    s.close()
