"""CPU property test of the FP32 candidate entries (csrc/state.cuh, cand_pack32): the distance
in y from two entries whose frame repeats every 8 cells, and the tests that blanked and
undecided entries fail and pass."""
import numpy as np
import pytest


@pytest.mark.parametrize("cell", [4.25e-4, 8.5e-4, 1.0, 3.7e3])
def test_wrapped_distance(cell):
    rng = np.random.default_rng(5)
    n = 200_000
    c = np.float32(cell)
    row_i, diff = rng.integers(0, 5000, n), rng.integers(-3, 4, n)
    row_j = np.maximum(row_i + diff, 0)
    # offsets in the cell, up to a quarter of a cell beyond its box (further ones are marked far)
    yr_i, yr_j = (rng.uniform(-0.25, 1.25, n).astype(np.float32) * c for _ in range(2))

    def y8(row, yr):
        return (np.float64(np.float32(row % 8)) * np.float64(c) + np.float64(yr)).astype(np.float32)   # one rounding (fma)

    d = y8(row_i, yr_i) - y8(row_j, yr_j)
    dy = np.abs(np.minimum(np.abs(d), np.float32(8) * c - np.abs(d)))   # squared in the test: |d| may pass 8 cells
    true = np.abs((row_i - row_j) * np.float64(c) + np.float64(yr_i) - np.float64(yr_j))
    near = true <= 4 * np.float64(c)
    assert np.abs(dy[near] - true[near]).max() <= 2.0 ** -19 * cell
    # beyond 4 cells the wrap shortens the distance, but never into a support (2h <= 2 cells)
    assert (~near).any() and dy[~near].min() >= 3.4 * cell


def test_special_entries():
    x = np.float32(0.3)
    for entry, passes in ((np.float32(np.inf), False), (np.float32(np.nan), True)):
        dx = x - entry
        rr2 = dx * dx + np.float32(0.1)
        assert (not (rr2 >= np.float32(4.0)) and not (rr2 < np.float32(1e-8))) is passes
