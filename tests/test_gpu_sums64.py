"""The FP64 neighbour sums (staged and fused) against the CPU oracle where the kernel can go
wrong: particle counts around its blocks of 32, neighbour lists longer than one pass, pairs of
unequal smoothing length, cells that exceed the FP32 candidate test's premise, and values
outside the range of the mantissa arithmetic.

Tolerance: a sum of n <= 300 terms, each with under 20 roundings, has a relative error below
(n + 20) 2^-53 < 4e-14 of the sum of its terms' magnitudes; the random fields leave at least a
tenth of that in the largest sums, which rel_err divides by: 1e-12."""
import numpy as np
import pytest

from conftest import rel_err
from oracle.oracle import OracleSim
from sph_fem_2d_cutting_gpu_gb300 import abi, setups
from sph_fem_2d_cutting_gpu_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def lattice(side, hdx=1.7, cell=(1, 2), vary_h=0.0, scale=1.0, seed=3):
    c = setups.micro(n_side=side, dx=2.5e-4 * scale, hdx=hdx, seed=seed, cell_factor=cell[0], stencil=cell[1])
    rng = np.random.default_rng(seed + 1)
    c.particles["T"][:] = 300.0 + rng.uniform(0.0, 200.0, c.N)
    c.particles["eps_pl"][:] = rng.uniform(0.05, 0.3, c.N)
    c.particles["S"] *= 0.3
    if vary_h:
        c.particles["h"] *= 1.0 - rng.uniform(0.0, vary_h, c.N)
    return c


CASES = {
    "25": dict(side=5), "36": dict(side=6), "1024": dict(side=32), "1089": dict(side=33),
    "two-passes": dict(side=30, hdx=2.6), "five-passes": dict(side=40, hdx=4.6, cell=(2, 1)),
    "unequal-h": dict(side=24, vary_h=0.2), "wide-cells": dict(side=24, cell=(20, 1)),
    "outside-range": dict(side=12, scale=1e22),
}


@pytest.mark.parametrize("name", list(CASES))
def test_sums_match_oracle(lib, name):
    c = lattice(**CASES[name])
    s = Solver(c)
    o = OracleSim(c.constants, c.grid, s.download(), c.dt)
    for call in ("assign_hashes", "sort", "init", "predict", "material_eos", "corrector_artificial_stress",
                 "interactions_monaghan"):
        getattr(s, call)()
        getattr(o, call)()
    G = s.download()
    for f in ("S_der", "v_der", "pos_t", "vel_t", "T_t"):
        e = rel_err(G[f], o.P[f])
        assert e <= 1e-12, f"{name} {f}: {e:.2e}"
    s.close()
    s = Solver(c)   # the same sums with the fused epilogue
    o = OracleSim(c.constants, c.grid, s.download(), c.dt)
    s.step()
    o.step()
    G = s.download()
    for f in ("vel", "S", "rho", "T", "pos_t", "vel_t", "rho_t", "S_t", "T_t"):
        e = rel_err(G[f], o.P[f])
        assert e <= 1e-12, f"{name} fused {f}: {e:.2e}"
    assert np.array_equal(G["idx"], o.P["idx"])
