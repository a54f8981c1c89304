"""CPU: the window widths of batches without fixed-base tables."""
import numpy as np
import pytest

import gpu_msm_b200 as gm
from gpu_msm_b200 import workload as wl


def tuned(group, sizes):
    return [gm.tuned_window(group, s) for s in sizes]


def cost(sizes, widths):
    """Products of a batch, with 2e6 for every class after the first."""
    return (sum(10 * n * (299 // c + 1) + 60 * (320 // c + 1) * 2 ** (c - 1) for n, c in zip(sizes, widths)) +
            2e6 * (len(set(widths)) - 1))


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("sizes", [[1 << 17] + [16] * 2000, [250000] + [8] * 50, [1 << 15] + [64] * 100,
                                   [1 << 15] * 3 + [256] * 40])
def test_skewed_batches_keep_their_widths(group, sizes):
    """One width for a few large MSMs and many tiny ones costs up to twice the separate classes."""
    table = gm.ResidentBases.__new__(gm.ResidentBases)
    table.group, table.precomputed = group, []
    assert table.windows_for(sizes) == tuned(group, sizes)


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("lo,hi,count", [(6, 12, 20), (10, 14, 28), (8, 15, 8), (4, 10, 40)])
def test_small_even_batches_take_one(group, lo, hi, count):
    sizes = [int(s) for s in wl.mixed_sizes(count, lo, hi, seed=3)]
    widths = gm.batch_widths(group, sizes)
    each = tuned(group, sizes)
    assert len(set(widths)) == 1 < len(set(each)) and min(each) <= widths[0] <= max(each)


@pytest.mark.parametrize("seed", range(30))
def test_never_dearer_than_the_tuned_widths(seed):
    rng = np.random.default_rng(seed)
    group = 1 + seed % 2
    sizes = [int(2 ** u) for u in rng.uniform(2, rng.uniform(4, 17), size=int(2 ** rng.uniform(1, 9)))]
    widths = gm.batch_widths(group, sizes)
    assert len(widths) == len(sizes)
    assert cost(sizes, widths) <= cost(sizes, tuned(group, sizes))


def test_accepts_what_it_took():
    """Any sequence of sizes, as before there were batch-wide widths."""
    table = gm.ResidentBases.__new__(gm.ResidentBases)
    table.group, table.precomputed = 1, []
    want = table.windows_for([100, 3000])
    for sizes in ((100, 3000), np.array([100, 3000]), np.array([100, 3000], dtype=np.int32), iter([100, 3000])):
        assert table.windows_for(sizes) == want
    assert table.windows_for([]) == [] and table.windows_for([500]) == [gm.tuned_window(1, 500)]
