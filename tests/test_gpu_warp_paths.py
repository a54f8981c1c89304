"""GPU: the warp-cooperative point arithmetic behind the fix-up, the bucket
reduction and the window combination, at the sizes where its kernels change
shape: one and few windows, the most windows, segments that do not divide the
buckets, sums of one and of two stages, level 0 on warps and on threads; and
points of order 2, whose double is infinity.  Exact: results are compared as
canonical affine points."""
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


# (group, n, limbs, c): windows 64 limbs / c + 1, buckets 2^(c-1) per window
SHAPES = [(1, 1, 1, 20), (1, 40, 1, 16), (1, 70, 8, 2), (1, 300, 5, 7), (1, 500, 2, 13), (1, 2000, 1, 18),
          (1, 900, 5, 14), (2, 1, 1, 18), (2, 33, 8, 3), (2, 200, 5, 6), (2, 400, 1, 15), (2, 300, 5, 13)]


@pytest.mark.parametrize("group,n,limbs,c", SHAPES)
def test_reduction_shapes(cuda, group, n, limbs, c):
    rng = np.random.default_rng(n + c)
    logs = wl.make_base_logs(n, seed=n, dup_frac=0.1)
    sc = rng.integers(0, 2 ** 64, size=(n, limbs), dtype=np.uint64)
    sc[:: 5] = 0
    sc[1:: 5] = 1 if limbs == 1 else sc[1:: 5]
    pts = gm.generator_mul_batch(dev(logs, cuda), group=group)
    ks, ts = wl.limbs_to_ints(sc), wl.limbs_to_ints(logs)
    want = oracle.generator_multiple(sum(k * t for k, t in zip(ks, ts)), group=group)
    assert oracle.same_point(run(pts, sc, group, cuda, c), want)


@pytest.mark.parametrize("c", [2, 4, 9])
@pytest.mark.parametrize("odd", [False, True])
def test_points_of_order_two(cuda, c, odd):
    """(-1, 0) on y^2 = x^3 + 1: its multiples are itself and infinity."""
    n = 37
    minus_one = (wl.P_MODULUS - (1 << 448)) % wl.P_MODULUS  # -1 in Montgomery form
    pts = np.zeros((n, gm.G1_WORDS), dtype=np.uint64)
    pts[:, :7] = wl.int_to_limbs(minus_one, 7)
    sc = np.random.default_rng(c).integers(0, 2 ** 64, size=(n, 2), dtype=np.uint64)
    sc[0, 0] = (int(sc[0, 0]) & ~1) + (int(sc[1:, 0].sum(dtype=np.uint64)) + (1 if odd else 0)) % 2
    got = run(dev(pts, cuda), sc, 1, cuda, c)
    assert bool(got["infinity"][0]) == (not odd)
    if odd:
        assert np.array_equal(got["x"][0], pts[0, :7]) and not got["y"][0].any()


# entries n (64 limbs / c + 1) around the line between slices on warps and on threads of a 148-SM GPU
# (151552 entries), and far below it
@pytest.mark.parametrize("group,n,c", [(1, 1, 7), (1, 5, 7), (1, 101, 9), (1, 3294, 7), (1, 3295, 7), (2, 3295, 7)])
def test_slices_on_warps_and_threads(cuda, group, n, c):
    """Half of the scalars are equal, so one bucket per window spans many slices; bases repeat and lie at infinity."""
    logs = wl.make_base_logs(n, seed=n, dup_frac=0.2)
    logs[::7] = 0
    sc = wl.make_scalars(n, seed=n + 1)
    sc[: n // 2] = sc[0]
    pts = gm.generator_mul_batch(dev(logs, cuda), group=group)
    want = oracle.generator_multiple(wl.expected_log(sc, logs), group=group)
    assert oracle.same_point(run(pts, sc, group, cuda, c), want)


@pytest.mark.parametrize("group", [1, 2])
@pytest.mark.parametrize("n", [1, 2, 50, 0])
def test_affine_result(cuda, group, n):
    """The affine form of the result (an inversion on the device), infinity included."""
    logs = wl.make_base_logs(max(n, 1), seed=3 + n)[:n]
    sc = wl.make_scalars(max(n, 1), seed=4 + n)[:n]
    if n == 2:  # P - P
        logs[1] = logs[0]
        sc[0], sc[1] = wl.int_to_limbs(5), wl.int_to_limbs(wl.R_ORDER - 5)
    words = gm.G1_WORDS if group == 1 else gm.G2_WORDS
    pts = gm.generator_mul_batch(dev(logs, cuda), group=group) if n else torch.empty((0, words), dtype=torch.int64,
                                                                                    device=cuda)
    out = gm.msm_device_affine(pts, dev(sc, cuda), group=group)
    torch.cuda.synchronize()
    got = gm.to_numpy_points(out, group)
    if n in (0, 2):
        assert bool(got["infinity"][0]) and not got["x"].any() and not got["y"].any()
    else:
        assert oracle.same_point(got, oracle.generator_multiple(wl.expected_log(sc, logs), group=group))


@pytest.mark.parametrize("group", [1, 2])
def test_affine_results_of_many_values(cuda, group):
    """64 one-point MSMs: as many different values through the inversion."""
    logs = wl.make_base_logs(64, seed=77)
    pts = gm.generator_mul_batch(dev(logs, cuda), group=group)
    one = dev(np.array([[3]], dtype=np.uint64), cuda)
    words = gm.G1_WORDS if group == 1 else gm.G2_WORDS
    out = torch.zeros((64, words), dtype=torch.int64, device=cuda)
    for i in range(64):
        gm.msm_device_affine(pts[i:i + 1], one, group=group, out=out[i])
    torch.cuda.synchronize()
    got = gm.to_numpy_points(out, group)
    for i, t in enumerate(wl.limbs_to_ints(logs)):
        assert oracle.same_point(got[i:i + 1], oracle.generator_multiple(3 * t, group=group)), i
