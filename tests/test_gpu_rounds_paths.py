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


@pytest.mark.parametrize("group,tabled", [(1, False), (1, True), (2, False)])
def test_batch_in_workspaces_of_either_size(cuda, group, tabled):
    """In the reported size the batch runs as it does from the pool, word for
    word and launch for launch; in the least accepted size without the rounds,
    the same points; below that it is refused."""
    table, sizes, wins, sc, want = make_batch(cuda, group=group, tabled=tabled)
    least = gm.batch_workspace_min_bytes(table, sizes, window_bits=wins)
    full = gm.batch_workspace_bytes(table, sizes, window_bits=wins)
    assert full > least + (256 << 20)
    gm.launch_count_reset()
    pooled = gm.batch_run(table, sizes, sc, window_bits=wins)
    n_pooled = gm.launch_count_reset()
    guard = 1 << 20
    ws = torch.zeros(full + guard, dtype=torch.uint8, device=cuda)
    ws[full:] = 77
    outs = {}
    for name, size in (("full", full), ("least", least), ("short", full - (64 << 20))):
        if name == "least":
            ws[least:] = 77
        outs[name] = gm.batch_run(table, sizes, sc, window_bits=wins, workspace=ws[:size])
        outs[name + "_launches"] = gm.launch_count_reset()
        if name != "short":
            assert bool((ws[size:size + guard] == 77).all())
    torch.cuda.synchronize()
    assert torch.equal(outs["full"], pooled) and outs["full_launches"] == n_pooled
    check(outs["least"], want, group)
    assert outs["least_launches"] < n_pooled
    check(outs["short"], want, group)
    with pytest.raises(gm.MSMError):
        gm.batch_run(table, sizes, sc, window_bits=wins, workspace=ws[:least - 1])
    table.close()


def test_reported_size_covers_the_pooled_run(cuda):
    """gm_batch_run takes no more device memory than gm_batch_workspace_bytes reports."""
    table, sizes, wins, sc, want = make_batch(cuda)
    out = torch.empty((len(sizes), gm.G1P_WORDS), dtype=torch.int64, device=cuda)
    gm.batch_run(table, sizes[:4], sc[:int(sizes[:4].sum())], window_bits=wins[:4], out=out[:4])
    gm.trim_memory()
    before = torch.cuda.mem_get_info()[0]
    gm.batch_run(table, sizes, sc, window_bits=wins, out=out)
    torch.cuda.synchronize()
    taken = before - torch.cuda.mem_get_info()[0]
    check(out, want)
    full = gm.batch_workspace_bytes(table, sizes, window_bits=wins)
    assert taken <= full + (128 << 20)  # the pool grows by whole chunks
    table.close()


def test_server_slots_hold_the_rounds(cuda):
    """A server's full batch runs in its slot as it would from the pool."""
    from gpu_msm_b200 import serving
    table, sizes, wins, sc, want = make_batch(cuda)
    server = serving.MsmServer({1: table}, max_batch=64, max_points=1 << 18, slots=2)
    for _, t, sz in server._limit_shapes():
        assert gm.batch_workspace_bytes(t, sz) <= server.slot_bytes
    sz = [int(s) for s in sizes[:64]]
    rows = int(sum(sz))
    gm.launch_count_reset()
    pooled = gm.batch_run(table, sz, sc[:rows])
    n = gm.launch_count_reset()
    own = gm.batch_run(table, sz, sc[:rows], workspace=server.slots[0].ws)
    assert gm.launch_count_reset() == n
    torch.cuda.synchronize()
    assert torch.equal(own, pooled)
    table.close()


def test_tables_within_32_bit_offsets(cuda):
    """Two widths whose one class would hold more than 2^32 entries stay two: the batch is planned, not refused."""
    n = 1 << 12
    logs = wl.make_base_logs(n, seed=3)
    table = gm.ResidentBases(gm.generator_mul_batch(dev(logs, cuda)), group=1).precompute(4).precompute(16)
    # all but the last take width 16, 4 entries short of 2^32; the last one width 4
    sizes = np.array([n] * 49930 + [2991, 2991, 2990, 1], dtype=np.int64)
    assert int(sizes[:-1].sum()) * 21 == 2 ** 32 - 4
    assert gm.batch_workspace_min_bytes(table, sizes) > 0
    table.close()


def test_given_widths_do_not_sway_the_others(cuda):
    """MSMs with a width of their own are left out of the choice of a table for the rest."""
    n = 1 << 15
    logs = wl.make_base_logs(n, seed=4)
    table = gm.ResidentBases(gm.generator_mul_batch(dev(logs, cuda)), group=1).precompute(6).precompute(14)
    small, large = [300] * 8 + [2000] * 2, [n] * 12
    alone = gm.BatchPlan(table, small).classes()
    sizes = small + large
    wins = [0] * len(small) + [9] * len(large)
    plan = gm.BatchPlan(table, sizes, window_bits=wins)
    assert [c for c in plan.classes() if c[0] != 9] == alone
    sc = wl.make_scalars(sum(sizes), seed=5)
    out = plan.run(dev(sc, cuda))
    torch.cuda.synchronize()
    res = oracle.proj_to_affine(gm.to_numpy_proj(out))
    for i, w in enumerate(wl.expected_logs(sizes, sc, logs)):
        assert oracle.same_point(res[i:i + 1], oracle.generator_multiple(w)), i
    plan.close()
    table.close()


def test_large_msms_keep_their_table(cuda):
    """Two large MSMs beside tiny ones stay on the wider table: 1.5 ms against 2.0 on the tiny ones'."""
    n = 1 << 15
    logs = wl.make_base_logs(n, seed=6)
    table = gm.ResidentBases(gm.generator_mul_batch(dev(logs, cuda)), group=1).precompute(11).precompute(14)
    sizes = [31000] * 2 + [30] * 26
    plan = gm.BatchPlan(table, sizes)
    assert sorted(plan.classes()) == [(11, 26), (14, 2)]
    plan.close()
    table.close()
