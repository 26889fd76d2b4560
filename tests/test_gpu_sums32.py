"""The FP32K neighbour sums (staged and fused) against the CPU oracle where the candidate scan
can go wrong: particle counts around its groups of four and its blocks, lists longer than one
pass, every cell geometry, columns shorter than the frame of eight rows, and positions moved
out of their cells since the sort.

Tolerance: a pair term has under 25 FP32 roundings and the compensated sums add none that
counts, so an element is within 25 * 2^-24 = 1.5e-6 of the sum of its terms' magnitudes, of which
the random fields leave at least a tenth in the largest sums, which rel_err divides by: 1.5e-5,
and 2e-5 with the rounding of the inputs."""
import numpy as np
import pytest

from conftest import rel_err
from oracle.oracle import OracleSim
from sph_fem_2d_cutting_gpu_gb300 import abi, setups
from sph_fem_2d_cutting_gpu_gb300.solver import Solver

pytestmark = pytest.mark.gpu

SUMS = ("S_der", "v_der", "pos_t", "vel_t", "T_t")
CASES = {
    "25": dict(side=5), "121": dict(side=11), "1089": dict(side=33), "2h-cells": dict(side=31, cell=(2, 1)),
    "2h-cells-wide": dict(side=31, cell=(2, 2)), "seven-columns": dict(side=29, cell=(1, 3)),
    "two-passes": dict(side=30, hdx=2.1), "five-passes": dict(side=40, hdx=4.4, cell=(2, 1)),
    "one-cell": dict(side=9, cell=(30, 1)),
}


def lattice(side, hdx=1.7, cell=(1, 2), seed=4):
    c = setups.micro(n_side=side, hdx=hdx, seed=seed, cell_factor=cell[0], stencil=cell[1])
    rng = np.random.default_rng(seed + 1)
    c.particles["T"][:] = 300.0 + rng.uniform(0.0, 200.0, c.N)
    c.particles["eps_pl"][:] = rng.uniform(0.05, 0.3, c.N)
    c.particles["S"] *= 0.3
    return c


def sums(c, pos=None):
    """The staged sums and the oracle's, `pos` (if given) replacing the positions after the sort."""
    s = Solver(c, abi.SPH_PREC_FP32K)
    o = OracleSim(c.constants, c.grid, s.download(), c.dt)
    for call in ("assign_hashes", "sort"):
        getattr(s, call)()
        getattr(o, call)()
    if pos is not None:
        o.P["pos"][:] = pos(o.P["pos"])
        s.upload({"pos": o.P["pos"]})
    for call in ("init", "predict", "material_eos", "corrector_artificial_stress", "interactions_monaghan"):
        getattr(s, call)()
        getattr(o, call)()
    return s.download(), o.P


@pytest.mark.parametrize("name", list(CASES))
def test_sums_match_oracle(lib, name):
    c = lattice(**CASES[name])
    G, P = sums(c)
    for f in SUMS:
        e = rel_err(G[f], P[f])
        assert e <= 2e-5, f"{name} {f}: {e:.2e}"
    s = Solver(c, abi.SPH_PREC_FP32K)
    o = OracleSim(c.constants, c.grid, s.download(), c.dt)
    s.step()
    o.step()
    G = s.download()
    for f in ("pos_t", "vel_t", "rho_t", "S_t", "T_t"):
        e = rel_err(G[f], o.P[f])
        assert e <= 2e-5, f"{name} fused {f}: {e:.2e}"
    assert np.array_equal(G["idx"], o.P["idx"])


def test_positions_moved_since_the_sort(lib):
    """Some particles a little, some a cell and more out of the cells they are listed in."""
    c = lattice(side=24)
    rng = np.random.default_rng(9)

    def moved(pos):
        far = rng.random(len(pos)) < 0.1
        return pos + far[:, None] * rng.uniform(-1.5, 1.5, pos.shape) * c.grid.h

    G, P = sums(c, moved)
    for f in SUMS:
        e = rel_err(G[f], P[f])
        assert e <= 2e-5, f"{f}: {e:.2e}"
