"""GPU: the scratch blocks of the rounds of affine additions: shared by streams
and threads, bounded, given back, replaced by a graph's own memory under
capture, and done without where the device has no room.  Results agree word
for word wherever the rounds run."""
import threading

import numpy as np
import pytest
import torch

import gpu_msm_b200 as gm
import oracle
from gpu_msm_b200 import workload as wl

pytestmark = pytest.mark.gpu
N, C = 131072, 10  # 4.3 M entries, two rounds: 0.65 GB of scratch, 0.25 GB of workspace


def dev(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).to(cuda)


@pytest.fixture(scope="module")
def case():
    cuda = torch.device("cuda:0")
    logs, sc = wl.make_base_logs(N, seed=61), wl.make_scalars(N, seed=62)
    pts, scd = gm.generator_mul_batch(dev(logs, cuda)), dev(sc, cuda)
    out = gm.msm_device(pts, scd, window_bits=C)
    torch.cuda.synchronize()
    got = oracle.proj_to_affine(gm.to_numpy_proj(out))
    assert oracle.same_point(got, oracle.generator_multiple(wl.expected_log(sc, logs)))
    return pts, scd, out


def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def phases(pts, sc):
    gm.profile_enable(True)
    try:
        out = gm.msm_device(pts, sc, window_bits=C)
        return [name for name, _ in gm.profile_collect()], out
    finally:
        gm.profile_enable(False)


def test_streams_share_and_give_back(case):
    pts, sc, want = case
    streams = [torch.cuda.Stream() for _ in range(12)]
    outs = [torch.empty_like(want) for _ in streams]
    gm.trim_memory()
    start = free()
    gm.msm_device(pts, sc, window_bits=C, out=outs[0], stream=streams[0])
    one = start - free()
    for _ in range(3):
        for s, o in zip(streams, outs):
            o.zero_()
        torch.cuda.synchronize()
        for s, o in zip(streams, outs):
            gm.msm_device(pts, sc, window_bits=C, out=o, stream=s)
        torch.cuda.synchronize()
        assert all(torch.equal(o, want) for o in outs)
    assert start - free() < 0.6 * len(streams) * one
    gm.trim_memory()
    assert start - free() < one / 4


def test_threads(case):
    pts, sc, want = case
    outs = [[torch.empty_like(want) for _ in range(6)] for _ in range(5)]
    streams = [torch.cuda.Stream() for _ in outs]
    torch.cuda.synchronize()
    errors = []

    def work(s, os):
        try:
            for o in os:
                gm.msm_device(pts, sc, window_bits=C, out=o, stream=s)
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    ts = [threading.Thread(target=work, args=a) for a in zip(streams, outs)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    torch.cuda.synchronize()
    assert not errors
    assert all(torch.equal(o, want) for os in outs for o in os)


def test_larger_calls_replace_blocks(case):
    """Blocks too small for the next call; the smaller calls then share the larger block."""
    pts, sc, want = case
    gm.trim_memory()
    streams = [torch.cuda.Stream() for _ in range(5)]
    small = 60000  # 2 M entries: one round
    first = gm.msm_device(pts[:small], sc[:small], window_bits=C)
    torch.cuda.synchronize()
    for n, ref in ((small, first), (N, want), (small, first), (N, want)):
        outs = [gm.msm_device(pts[:n], sc[:n], window_bits=C, stream=s) for s in streams]
        torch.cuda.synchronize()
        assert all(torch.equal(o, ref) for o in outs), n


def test_capture(case):
    pts, sc, want = case
    out = torch.empty_like(want)
    static = sc.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        gm.msm_device(pts, static, window_bits=C, out=out)
    for _ in range(2):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    del g


def test_without_room(case):
    """Room for the workspace, not for twice the scratch: exact without the rounds, and with them again after."""
    pts, sc, want = case
    gm.trim_memory()
    torch.cuda.empty_cache()
    names, out = phases(pts, sc)
    assert "affine" in names and torch.equal(out, want)
    gm.trim_memory()
    fill = torch.empty(free() - (1400 << 20), dtype=torch.uint8, device=pts.device)
    names, out = phases(pts, sc)
    del fill
    torch.cuda.empty_cache()
    assert "affine" not in names and "accumulate" in names
    same = oracle.proj_to_affine(gm.to_numpy_proj(out))
    assert oracle.same_point(same, oracle.proj_to_affine(gm.to_numpy_proj(want)))
    names, out = phases(pts, sc)
    assert "affine" in names and torch.equal(out, want)


def test_plan_without_room(case):
    """A plan takes the rounds' memory where the device has four times as much free, else runs without: the same points."""
    pts, sc, _ = case
    table = gm.ResidentBases(pts[:4096].contiguous(), group=1)
    sizes = [2000 + i for i in range(60)]
    wins = [9] * 50 + [6] * 10
    rows = sum(sizes)
    gm.trim_memory()
    torch.cuda.empty_cache()
    outs, counts, taken = [], [], []
    for leave in (None, 2200 << 20):
        fill = torch.empty(free() - leave, dtype=torch.uint8, device=pts.device) if leave else None
        plan = gm.BatchPlan(table, sizes, window_bits=wins)
        taken.append(plan.workspace_bytes)
        gm.launch_count_reset()
        outs.append(plan.run(sc[:rows]))
        torch.cuda.synchronize()
        counts.append(gm.launch_count_reset())
        plan.close()
        del fill
        torch.cuda.empty_cache()
    assert counts[1] < counts[0] and taken[1] < taken[0]
    a, b = (oracle.proj_to_affine(gm.to_numpy_proj(o)) for o in outs)
    assert oracle.same_point(a, b)
    table.close()


def test_graph_memory_is_given_back(case):
    """A captured call's scratch is the graph's; destroyed and trimmed, the device has it again."""
    pts, sc, want = case
    out = torch.empty_like(want)
    gm.trim_memory()
    start = free()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        gm.msm_device(pts, sc, window_bits=C, out=out)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    held = start - free()
    assert held > 256 << 20
    g.reset()
    del g
    gm.trim_memory()
    assert start - free() < held / 4
