"""GPU: the rounds of affine additions in front of the bucket accumulation
(large MSMs and batch classes): exact results where every exceptional pair
occurs (equal points, opposite points, infinity, x = 0, points of order two),
for odd buckets, skewed buckets and batch classes, with and without fixed-base
tables.  The rounds run from about 1.8 M (G1) and 1.2 M (G2) entries up on a
148-SM GPU; every case here is above that."""
import numpy as np
import pytest
import torch

import gpu_msm_b200 as gm
import oracle
from gpu_msm_b200 import workload as wl

pytestmark = pytest.mark.gpu


def dev(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).to(cuda)


def run(pts, sc, group, cuda, c=0):
    out = gm.msm_device(pts, dev(sc, cuda), group=group, window_bits=c)
    torch.cuda.synchronize()
    return oracle.proj_to_affine(gm.to_numpy_proj(out, group), group)


@pytest.mark.parametrize("group,n,c", [(1, 70001, 10), (1, 150000, 9), (1, 131071, 14), (2, 50001, 10), (2, 70000, 13)])
def test_few_distinct_bases(cuda, group, n, c):
    """40 distinct logs, their negatives and infinity: buckets full of equal and opposite points."""
    rng = np.random.default_rng(n + c)
    few = wl.uniform_below_r(rng, 40)
    neg = np.stack([wl.int_to_limbs(wl.R_ORDER - t) for t in wl.limbs_to_ints(few)])
    pool = np.concatenate([few, neg, np.zeros((1, 5), dtype=np.uint64)])
    logs = pool[rng.integers(0, len(pool), size=n)]
    sc = wl.make_scalars(n, seed=n)
    pts = gm.generator_mul_batch(dev(logs, cuda), group=group)
    want = oracle.generator_multiple(wl.dot_log(wl.limbs16(sc), wl.limbs16(logs)), group=group)
    assert oracle.same_point(run(pts, sc, group, cuda, c), want)


@pytest.mark.parametrize("group,n,c", [(1, 140000, 12), (2, 70000, 11)])
def test_equal_scalars_and_bases(cuda, group, n, c):
    """A third of the scalars equal (one bucket per window holds a third of the points), a third of the bases equal."""
    rng = np.random.default_rng(c)
    logs = wl.make_base_logs(n, seed=c)
    logs[rng.integers(0, n, size=n // 3)] = logs[0]
    sc = wl.make_scalars(n, seed=c + 1)
    sc[rng.integers(0, n, size=n // 3)] = sc[1]
    pts = gm.generator_mul_batch(dev(logs, cuda), group=group)
    want = oracle.generator_multiple(wl.dot_log(wl.limbs16(sc), wl.limbs16(logs)), group=group)
    assert oracle.same_point(run(pts, sc, group, cuda, c), want)


@pytest.mark.parametrize("c", [8, 11])
def test_torsion_points(cuda, c):
    """Bases of order two and three, (-1, 0) and (0, +-1) on y^2 = x^3 + 1, and infinity."""
    n, p = 120000, wl.P_MODULUS
    one = (1 << 448) % p
    t2, t3, m3 = (p - one, 0), (0, one), (0, p - one)
    rng = np.random.default_rng(c)
    kind = rng.integers(0, 4, size=n)
    rows = np.zeros((4, gm.G1_WORDS), dtype=np.uint64)
    for k, (x, y) in enumerate((t2, t3, m3)):
        rows[k, :7], rows[k, 7:14] = wl.int_to_limbs(x, 7), wl.int_to_limbs(y, 7)
    rows[3, 14] = 1
    sc = rng.integers(0, 2 ** 64, size=(n, 3), dtype=np.uint64)
    got = run(dev(rows[kind], cuda), sc, 1, cuda, c)

    # multiples of T2 mod 2 and of T3 mod 3 (2^64 = 1 mod 3)
    a = int(np.bitwise_xor.reduce(sc[kind == 0, 0])) & 1
    m = (sc % np.uint64(3)).astype(np.int64).sum(axis=1)
    b = int(m[kind == 1].sum() - m[kind == 2].sum()) % 3
    if a == 0 and b == 0:
        assert bool(got["infinity"][0])
        return
    if a == 0:
        x, y = (t3, m3)[b - 1]
    elif b == 0:
        x, y = t2
    else:
        # (-1, 0) + (0, e): slope e, x = e^2 + 1 = 2, y = -e - 2 e
        e = 1 if b == 1 else -1
        x, y = 2 * one % p, (-3 * e * one) % p
    assert not bool(got["infinity"][0])
    assert np.array_equal(got["x"][0], wl.int_to_limbs(x, 7)) and np.array_equal(got["y"][0], wl.int_to_limbs(y, 7))


@pytest.mark.parametrize("group,count,lo,hi,tabled", [(1, 60, 10.0, 12.0, False), (1, 60, 10.0, 12.5, True),
                                                     (2, 40, 9.0, 12.0, False)])
def test_batch_class(cuda, group, count, lo, hi, tabled):
    """One class large enough for the rounds, and a small second class beside it."""
    n = 1 << 13
    logs = wl.make_base_logs(n, seed=5)
    logs[3] = 0
    table = gm.ResidentBases(gm.generator_mul_batch(dev(logs, cuda), group=group), group=group)
    sizes = wl.mixed_sizes(count, lo, hi, seed=3)
    wins = np.full(count, 9, dtype=np.int32)
    wins[:2] = 6
    if tabled:
        table.precompute(9)
    rng = np.random.default_rng(1)
    offs = np.array([rng.integers(0, n - s + 1) for s in sizes], dtype=np.int64)
    sc = wl.make_scalars(int(sizes.sum()), seed=9)
    want = wl.expected_logs(sizes, sc, logs, offs)
    sct = dev(sc, cuda)
    plan = gm.BatchPlan(table, sizes, offs, window_bits=wins)
    outs = [plan.run(sct), plan.run(sct)]
    plan.set_queue(False)
    outs.append(plan.run(sct))
    outs.append(gm.batch_run(table, sizes, sct, base_offsets=offs, window_bits=wins))
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1])
    for out in outs:
        res = oracle.proj_to_affine(gm.to_numpy_proj(out, group), group)
        for i, w in enumerate(want):
            assert oracle.same_point(res[i:i + 1], oracle.generator_multiple(w, group=group)), i
    plan.close()
    table.close()


def test_batch_over_runs_of_empty_buckets(cuda):
    """Scalars of 100 bits in 5 limbs: most windows of every MSM are empty, in the middle of the batch's keys."""
    n, count, group, c = 1 << 15, 9, 1, 12
    logs = wl.make_base_logs(n, seed=15)
    table = gm.ResidentBases(gm.generator_mul_batch(dev(logs, cuda), group=group), group=group)
    sizes = np.array([n - 7 * i for i in range(count)], dtype=np.int64)
    sc = wl.make_scalars(int(sizes.sum()), seed=16)
    sc[:, 2:] = 0
    sc[:, 1] &= np.uint64((1 << 36) - 1)
    sc[:: 1000, 4] = 1  # and a few full-width ones
    want = wl.expected_logs(sizes, sc, logs)
    out = gm.BatchPlan(table, sizes, window_bits=np.full(count, c, dtype=np.int32)).run(dev(sc, cuda))
    torch.cuda.synchronize()
    res = oracle.proj_to_affine(gm.to_numpy_proj(out, group), group)
    for i, w in enumerate(want):
        assert oracle.same_point(res[i:i + 1], oracle.generator_multiple(w, group=group)), i


@pytest.mark.parametrize("sizes,one", [([5, 300, 17, 4000], True), ([1 << 17, 1 << 17, 7], False)])
def test_small_batches_take_one_width(cuda, sizes, one):
    """A small batch is one class, exact; a large one keeps the tuned widths."""
    n = max(sizes)
    logs = wl.make_base_logs(n, seed=21)
    table = gm.ResidentBases(gm.generator_mul_batch(dev(logs, cuda), group=1), group=1)
    plan = gm.BatchPlan(table, sizes)
    assert (len(plan.classes()) == 1) == one
    sc = wl.make_scalars(sum(sizes), seed=22)
    out = plan.run(dev(sc, cuda))
    torch.cuda.synchronize()
    res = oracle.proj_to_affine(gm.to_numpy_proj(out, 1), 1)
    for i, w in enumerate(wl.expected_logs(sizes, sc, logs)):
        assert oracle.same_point(res[i:i + 1], oracle.generator_multiple(w)), i


def test_tables_of_small_and_mixed_batches(cuda):
    """Over two tables: the whole batch on one of them, or each MSM on its own best."""
    n = 1 << 16
    logs = wl.make_base_logs(n, seed=31)
    table = gm.ResidentBases(gm.generator_mul_batch(dev(logs, cuda), group=1), group=1).precompute(6).precompute(14)
    for sizes, classes in (([20, 30, 25], 1), ([60000, 50000], 1), ([60000] + [20] * 40, 2)):
        plan = gm.BatchPlan(table, sizes)
        assert len(plan.classes()) == classes, plan.classes()
        sc = wl.make_scalars(sum(sizes), seed=32)
        out = plan.run(dev(sc, cuda))
        torch.cuda.synchronize()
        res = oracle.proj_to_affine(gm.to_numpy_proj(out, 1), 1)
        for i, w in enumerate(wl.expected_logs(sizes, sc, logs)):
            assert oracle.same_point(res[i:i + 1], oracle.generator_multiple(w)), i
        plan.close()
