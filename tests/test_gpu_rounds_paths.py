"""GPU: every route of an MSM or a batch takes the rounds of affine additions
alike, so that results agree word for word, in the memory that it is given."""
import numpy as np
import pytest
import torch

import gpu_msm_b200 as gm
import oracle
from gpu_msm_b200 import workload as wl

pytestmark = pytest.mark.gpu


def dev(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).to(cuda)


def make_batch(cuda, group=1, count=80, widths=(9, 10), tabled=False, seed=5):
    """Each class has 40 MSMs of about 2000 points, 2.6 to 3 M entries: two rounds (G1)."""
    n = 1 << 12
    logs = wl.make_base_logs(n, seed=seed)
    table = gm.ResidentBases(gm.generator_mul_batch(dev(logs, cuda), group=group), group=group)
    if tabled:
        for c in widths:
            table.precompute(c)
    sizes = np.array([2000 + 7 * i % 90 for i in range(count)], dtype=np.int64)
    wins = np.array([widths[i % len(widths)] for i in range(count)], dtype=np.int32)
    sc = wl.make_scalars(int(sizes.sum()), seed=seed + 1)
    return table, sizes, wins, dev(sc, cuda), wl.expected_logs(sizes, sc, logs)


def check(out, want, group=1):
    res = oracle.proj_to_affine(gm.to_numpy_proj(out, group), group)
    for i in range(0, len(want), 9):
        assert oracle.same_point(res[i:i + 1], oracle.generator_multiple(want[i], group=group)), i


@pytest.mark.parametrize("tabled", [False, True])
def test_plan_modes_agree_word_for_word(cuda, tabled):
    table, sizes, wins, sc, want = make_batch(cuda, tabled=tabled)
    plan = gm.BatchPlan(table, sizes, window_bits=wins)
    assert len(plan.classes()) == 2
    queued = plan.run(sc)
    plan.set_queue(False)
    classes = plan.run(sc)
    again = plan.run(sc)
    torch.cuda.synchronize()
    check(classes, want)
    assert torch.equal(queued, classes) and torch.equal(classes, again)
    plan.close()
    table.close()
