"""CPU check of the reset of the counting sort's counts (csrc/cells.cu): the stores of zero in
k_scan_down, with their own guards evaluated for every thread of the launch, clear exactly the
words 0..n -- the n = num_cell + 1 buckets and, behind them, the length of the contact queue --
on grids around whole tiles of the scan; and the clear before a first histogram takes all of
them, too."""
import re
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "sph_fem_2d_cutting_gpu_gb300" / "csrc"
SOURCE = (CSRC / "cells.cu").read_text()
CONSTANTS = {k: int(v) for k, v in re.findall(r"constexpr int (kScanThreads|kScanItems) = (\d+);",
                                              (CSRC / "cells.cuh").read_text())}
CONSTANTS["kScanTile"] = CONSTANTS["kScanThreads"] * CONSTANTS["kScanItems"]


def evaluate(expression, names):
    return eval(expression.replace("blockIdx.x", "block").replace("threadIdx.x", "thread"), {}, names)


def cleared(n):
    body = re.search(r"\n__global__[^{;]*k_scan_down\(.*?\n}\n", SOURCE, re.S).group(0)
    tiles = evaluate(re.search(r"int scan_blocks\(int num_cell\) \{ return div_up\((.*?)\); \}", SOURCE).group(1)
                     .replace(", kScanTile", ""), {"num_cell": n - 1})
    tiles = -(-tiles // CONSTANTS["kScanTile"])
    block, thread, k = np.meshgrid(np.arange(tiles), np.arange(CONSTANTS["kScanThreads"]),
                                   np.arange(CONSTANTS["kScanItems"]), indexing="ij")
    names = dict(CONSTANTS, n=n, block=block, thread=thread, k=k)
    names["base"] = evaluate(re.search(r"int base = (.*?);", body).group(1), names)
    out = np.zeros(n + 1 + CONSTANTS["kScanTile"], bool)
    stores = re.findall(r"if \(([^;{}]*)\) counts\[(.*?)\] = 0;", body)
    assert stores
    for guard, index in stores:
        on = np.all([np.broadcast_to(evaluate(g, names), block.shape) for g in guard.split("&&")], axis=0)
        out[np.broadcast_to(evaluate(index, names), block.shape)[on]] = True
    return out


@pytest.mark.parametrize("n", [2, 2047, 2048, 2049, 4095, 4096, 4097, 102_400])
def test_every_step_clears_buckets_and_queue_length(n):
    out = cleared(n)
    assert out[:n + 1].all() and not out[n + 1:].any()


def test_first_histogram_clears_buckets_and_queue_length():
    body = re.search(r"static void count\(.*?\n}\n", SOURCE, re.S).group(0)
    words = re.search(r"cudaMemsetAsync\(X\.counts, 0, sizeof\(int32_t\) \* \(\(size_t\)g\.num_cell \+ (\d+)\)", body)
    assert words and int(words.group(1)) == 2
