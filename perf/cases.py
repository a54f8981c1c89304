"""Workloads of the MSM engine, from the smallest calls to the largest.

Each case is one call (or one batch) as a proving or verifying program makes
it, and ends with what such a program goes on with: affine points, or field
elements.  The sizes are those of the benchmark configurations, of the tests
and odd sizes between them.

Inputs are synthetic and seeded: scalars uniform in [0, r) with 1 % zeros and
1 % ones, bases P_i = t_i G with t_i uniform in [1, r) and 2 % of the bases
duplicated.  As every t_i is known, the exact result of an MSM is
(sum_i k_i t_i mod r) G, which `exact` computes with Python integers.
"""
import numpy as np
import torch

import gpu_msm_b200 as gm

# curve: base field, scalar field, generators (y^2 = x^3 + 1; y^2 = x^3 + 1 + i over i^2 = -1)
U = -0x6008204000000020001
R_ORDER = U ** 4 - U ** 2 + 1
P = (U - 1) ** 2 * R_ORDER // 3 + U
R = 1 << 448
R_INV = pow(R, -1, P)
G1_GEN_MONT = (
    (7917664463663687095, 1355176381348215757, 9309256319878456358, 16082309242814470913, 1457786988405400601,
     2532676885992645838, 4266797631218839278),
    (4868026731894891110, 12304408657332121882, 7441369506613370646, 10864257464733093146, 2875956116323242790,
     14896292406590517651, 878043436812691251))
G2_GEN_MONT = (
    ((4123490056514120819, 2888875260792682753, 17655201647264233221, 7157421936295224695, 15498584076058546935,
      15228297334835920, 4244443893027848071),
     (9689639818784850924, 1629246158933521251, 11423128445604303869, 16398231048073676806, 468062648903243987,
      14345089387303932758, 2855398789980915890)),
    ((11342985268414953941, 10459569641143299718, 17058451870372416372, 11935997349792929207, 1623745315435952156,
      10825731736850511142, 4331460898642949879),
     (16947683615433868223, 2484215721908895818, 6050651669238557934, 8875663977313421353, 1988428140903801186,
      2083688187386050035, 3129790274208079714)))

TABLE = 1 << 16   # entries of the resident base table of the batched cases


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a verifier's or a test's sum of a hundred points with machine-word scalars
        {"name": "g1_n100_u64", "kind": "device", "group": 1, "n": 100, "limbs": 1},
        # the plain configuration of 1024 points, full-width scalars
        {"name": "g1_n1024", "kind": "device", "group": 1, "n": 1024, "limbs": 5},
        # a middle-sized commitment of odd length
        {"name": "g1_n20011", "kind": "device", "group": 1, "n": 20011, "limbs": 5},
        # the headline G1 MSM
        {"name": "g1_n2p20", "kind": "device", "group": 1, "n": 1 << 20, "limbs": 5},
        # a small G2 MSM (the G2 query of a small circuit)
        {"name": "g2_n1500", "kind": "device", "group": 2, "n": 1500, "limbs": 5},
        # the headline G2 MSM
        {"name": "g2_n2p18", "kind": "device", "group": 2, "n": 1 << 18, "limbs": 5},
        # the drop-in host call: standard-form points and u64 scalars in host memory, copies included
        {"name": "g1_host_u64_n10007", "kind": "host_u64", "group": 1, "n": 10007, "limbs": 1},
        # full-width scalars through host buffers
        {"name": "g1_host_n100003", "kind": "host", "group": 1, "n": 100003, "limbs": 5},
        # 512 MSMs of 2^8..2^16 points over a shared resident table, planned once
        {"name": "batch_g1_512", "kind": "plan", "group": 1, "count": 512, "lo": 8.0, "hi": 16.0, "limbs": 5},
        # a ragged batch of small G2 MSMs over a resident table, planned once
        {"name": "batch_g2_20", "kind": "plan", "group": 2, "count": 20, "lo": 6.0, "hi": 12.0, "limbs": 5},
        # a server's batch: requests that arrived together, over a table with precomputed windows, shape new
        # on every call
        {"name": "serve_g1_24", "kind": "serve", "group": 1, "count": 24, "lo": 10.0, "hi": 16.0, "limbs": 5},
        # element-wise products in the extension field
        {"name": "fp2_mul_n500009", "kind": "field", "op": "fp2_mont_mul", "n": 500009},
    ]


def _log(rng, lo, hi):
    return int(round(float(lo) * (float(hi) / float(lo)) ** rng.random()))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "device", "host", "host_u64", "plan", "serve", "field"])
    if kind == "device":
        group = rng.choice([1, 1, 2])
        limbs = rng.choice([1, 5, 5, 5])
        return {"kind": kind, "group": group, "n": _log(rng, 100, (1 << 20) if group == 1 else (1 << 18)), "limbs": limbs}
    if kind == "host":
        group = rng.choice([1, 2])
        return {"kind": kind, "group": group, "n": _log(rng, 100, 300000 // group ** 2), "limbs": 5}
    if kind == "host_u64":
        return {"kind": kind, "group": 1, "n": _log(rng, 100, 300000), "limbs": 1}
    if kind == "plan":
        group = rng.choice([1, 2])
        count = _log(rng, 4, 256 if group == 1 else 48)
        hi = round(rng.uniform(8.5, 16.0 if group == 1 else 13.0), 2)
        return {"kind": kind, "group": group, "count": count, "lo": 6.0, "hi": hi, "limbs": 5}
    if kind == "serve":
        return {"kind": kind, "group": 1, "count": _log(rng, 1, 48), "lo": 8.0, "hi": round(rng.uniform(10.0, 16.0), 2),
                "limbs": 5}
    op = rng.choice(["fp_mont_mul", "fp2_mont_mul"])
    return {"kind": kind, "op": op, "n": _log(rng, 10000, 1500000 if op == "fp_mont_mul" else 500000)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
R_TOP = 1 << (R_ORDER.bit_length() - 256)
R_WORDS = np.array([(R_ORDER >> (64 * i)) & (2 ** 64 - 1) for i in range(5)], dtype=np.uint64)


def _below_r(rng, n):
    """n integers uniform in [0, r), as (n, 5) little-endian 64-bit limbs."""
    s = rng.integers(0, 2 ** 64, size=(n, 5), dtype=np.uint64)
    s[:, 4] &= np.uint64(R_TOP - 1)
    while True:
        lt, eq = np.zeros(n, dtype=bool), np.ones(n, dtype=bool)
        for i in range(4, -1, -1):
            lt |= eq & (s[:, i] < R_WORDS[i])
            eq &= s[:, i] == R_WORDS[i]
        bad = np.flatnonzero(~lt)
        if not len(bad):
            return s
        s[bad] = rng.integers(0, 2 ** 64, size=(len(bad), 5), dtype=np.uint64)
        s[bad, 4] &= np.uint64(R_TOP - 1)


def _scalars(rng, n, limbs):
    s = _below_r(rng, n) if limbs == 5 else rng.integers(0, 2 ** 64, size=(n, limbs), dtype=np.uint64)
    idx = rng.permutation(n)
    k = n // 100
    s[idx[:2 * k]] = 0
    s[idx[k:2 * k], 0] = 1
    return s


def _logs(rng, n):
    t = _below_r(rng, n)
    t[~t.any(axis=1), 0] = 1
    k = n // 50
    t[rng.permutation(n)[:k]] = t[rng.integers(0, n, size=k)]
    return t


def _sizes(case, rng):
    return np.minimum(np.floor(2.0 ** rng.uniform(case["lo"], case["hi"], size=case["count"])).astype(np.int64), TABLE)


def _inputs(case, seed):
    """(scalars, logs of the bases, sizes, offsets into the table) as numpy arrays."""
    rng = np.random.default_rng(1000 + seed)
    if case["kind"] in ("plan", "serve"):
        # the shape belongs to the case, the values to the seed
        shape = np.random.default_rng(7)
        sizes = _sizes(case, shape)
        offs = np.array([int(shape.integers(0, TABLE - s + 1)) for s in sizes], dtype=np.int64)
        return _scalars(rng, int(sizes.sum()), case["limbs"]), _logs(rng, TABLE), sizes, offs
    return _scalars(rng, case["n"], case["limbs"]), _logs(rng, case["n"]), None, None


def _field_inputs(case, seed):
    rng = np.random.default_rng(1000 + seed)
    cols = 7 if case["op"].startswith("fp_") else 14
    out = []
    for _ in range(2):
        a = rng.integers(0, 2 ** 64, size=(case["n"], cols), dtype=np.uint64)
        # top limbs below the modulus' own, so that every element is canonical
        a[:, 6::7] %= np.uint64(P >> 384)
        out.append(a)
    return out


def _dev(a):
    return torch.from_numpy(a.view(np.int64)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "field":
        a, b = _field_inputs(case, seed)
        a, b = _dev(a), _dev(b)
        return {"kind": kind, "op": case["op"], "a": a, "b": b, "out": torch.empty_like(a)}
    group = case["group"]
    sc, logs, sizes, offs = _inputs(case, seed)
    points = gm.generator_mul_batch(_dev(logs), group=group)
    state = {"kind": kind, "group": group}
    words = (gm.G1_WORDS, gm.G2_WORDS)[group - 1]
    if kind == "device":
        state.update(points=points, scalars=_dev(sc), out=torch.zeros(words, dtype=torch.int64, device="cuda"))
    elif kind == "host":
        state.update(points=gm.to_numpy_points(points, group), scalars=sc)
    elif kind == "host_u64":
        # this entry point takes standard-form points
        pts = gm.to_numpy_points(points, group)
        mont = points[:, :14].reshape(-1, 7).contiguous()
        one = torch.zeros_like(mont)
        one[:, 0] = 1
        std = gm.field_mul_array(mont, one, op="fp_mont_mul")
        std = std.reshape(-1, 14).cpu().numpy().view(np.uint64)
        pts["x"], pts["y"] = std[:, :7], std[:, 7:]
        state.update(points=pts, scalars=sc.reshape(-1))
    else:
        table = gm.ResidentBases(points, group=group)
        state.update(table=table, scalars=_dev(sc))
        if kind == "plan":
            state["plan"] = gm.BatchPlan(table, sizes, offs, scalar_limbs=case["limbs"])
        else:
            for c in (11, 14):
                table.precompute(c, case["limbs"])
            state.update(sizes=sizes, offs=offs)
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _affine(proj, group):
    """Projective results -> affine points (Montgomery form), as 64-bit words."""
    a = gm.projective_to_affine(proj, group)
    return a.view(np.int64).reshape(len(a), -1)


def run(state):
    kind = state["kind"]
    if kind == "field":
        return gm.field_mul_array(state["a"], state["b"], op=state["op"], out=state["out"])
    group = state["group"]
    if kind == "device":
        return gm.msm_device_affine(state["points"], state["scalars"], group=group, out=state["out"])
    if kind == "host":
        return _affine(gm.msm(state["points"], state["scalars"], group=group), group)
    if kind == "host_u64":
        return _affine(gm.g1_msm_wrapper(state["points"], state["scalars"]), 1)
    if kind == "plan":
        proj = state["plan"].run(state["scalars"])
    else:
        proj = gm.batch_run(state["table"], state["sizes"], state["scalars"], base_offsets=state["offs"])
    # the results are read back as the affine points that a proof is made of
    return _affine(gm.to_numpy_proj(proj, group), group)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _msm_muls(n, bits):
    """Field products of a bucket-method MSM: six per affine addition into a
    bucket (an inversion shared by many), two 14-product additions per bucket,
    at the window width where the sum is least."""
    best = None
    for c in range(2, 23):
        w = -(-(bits + 1) // c)
        v = 6 * n * w + 28 * 2 ** (c - 1) * w
        best = v if best is None else min(best, v)
    return best


def work(case):
    mul = 2 * 14 * 14 * 2   # 32-bit multiply-adds of one Montgomery product (product and reduction), two operations each
    if case["kind"] == "field":
        words, k = (7, 1) if case["op"].startswith("fp_") else (14, 3)
        return {"bytes": 3 * 8 * words * case["n"], "flops": k * mul * case["n"]}
    group, limbs = case["group"], case["limbs"]
    bits = min(64 * limbs, R_ORDER.bit_length())
    k = 1 if group == 1 else 3
    point = 112 * group
    if case["kind"] in ("plan", "serve"):
        _, _, sizes, offs = _shape(case)
        used = np.zeros(TABLE, dtype=bool)
        for s, o in zip(sizes, offs):
            used[o:o + s] = True
        n = int(sizes.sum())
        muls = sum(_msm_muls(int(s), bits) for s in sizes)
        return {"bytes": n * 8 * limbs + int(used.sum()) * point + len(sizes) * point, "flops": k * mul * muls}
    n = case["n"]
    return {"bytes": n * (8 * limbs + point) + point, "flops": k * mul * _msm_muls(n, bits)}


def _shape(case):
    shape = np.random.default_rng(7)
    sizes = _sizes(case, shape)
    return None, None, sizes, np.array([int(shape.integers(0, TABLE - s + 1)) for s in sizes], dtype=np.int64)


# ---------------------------------------------------------------------------
# exact results, with Python integers alone
# ---------------------------------------------------------------------------
def _int(words):
    return sum(int(w) << (64 * i) for i, w in enumerate(words))


class _F1:
    @staticmethod
    def mul(a, b):
        return a * b % P

    @staticmethod
    def sub(a, b):
        return (a - b) % P

    @staticmethod
    def add(a, b):
        return (a + b) % P

    @staticmethod
    def inv(a):
        return pow(a, -1, P)

    @staticmethod
    def zero(a):
        return a == 0
    ONE = 1


class _F2:
    @staticmethod
    def mul(a, b):
        t0, t1 = a[0] * b[0], a[1] * b[1]
        return ((t0 - t1) % P, ((a[0] + a[1]) * (b[0] + b[1]) - t0 - t1) % P)

    @staticmethod
    def sub(a, b):
        return ((a[0] - b[0]) % P, (a[1] - b[1]) % P)

    @staticmethod
    def add(a, b):
        return ((a[0] + b[0]) % P, (a[1] + b[1]) % P)

    @staticmethod
    def inv(a):
        n = pow(a[0] * a[0] + a[1] * a[1], -1, P)
        return (a[0] * n % P, -a[1] * n % P)

    @staticmethod
    def zero(a):
        return a[0] == 0 and a[1] == 0
    ONE = (1, 0)


def _gen(group):
    if group == 1:
        return tuple(_int(c) * R_INV % P for c in G1_GEN_MONT)
    return tuple(tuple(_int(c) * R_INV % P for c in xy) for xy in G2_GEN_MONT)


def _gen_doubles(group):
    """2^j G, j < 300, affine."""
    F = _F1 if group == 1 else _F2
    x, y = _gen(group)
    out = [(x, y)]
    for _ in range(299):
        xx = F.mul(x, x)
        lam = F.mul(F.add(F.add(xx, xx), xx), F.inv(F.add(y, y)))
        x3 = F.sub(F.mul(lam, lam), F.add(x, x))
        x, y = x3, F.sub(F.mul(lam, F.sub(x, x3)), y)
        out.append((x, y))
    return out


def _gen_times(k, doubles, F):
    """k G for 0 <= k < r, affine or None: mixed Jacobian additions of the
    2^j G at the set bits (a partial sum never meets +-2^j G below r)."""
    acc = None
    for j in range(k.bit_length()):
        if not (k >> j) & 1:
            continue
        x2, y2 = doubles[j]
        if acc is None:
            acc = (x2, y2, F.ONE)
            continue
        x1, y1, z1 = acc
        zz = F.mul(z1, z1)
        h = F.sub(F.mul(x2, zz), x1)
        r = F.sub(F.mul(y2, F.mul(zz, z1)), y1)
        hh = F.mul(h, h)
        hhh = F.mul(h, hh)
        v = F.mul(x1, hh)
        x3 = F.sub(F.sub(F.mul(r, r), hhh), F.add(v, v))
        acc = (x3, F.sub(F.mul(r, F.sub(v, x3)), F.mul(y1, hhh)), F.mul(z1, h))
    if acc is None:
        return None
    zi = F.inv(acc[2])
    z2 = F.mul(zi, zi)
    return F.mul(acc[0], z2), F.mul(acc[1], F.mul(z2, zi))


def _dot(k, t):
    """sum_i k_i t_i mod r from (n, limbs) 64-bit limbs, through exact sums of 16-bit limb products."""
    acc = 0
    for r0 in range(0, len(k), 1 << 18):
        a = k[r0:r0 + (1 << 18)].view(np.uint16).reshape(-1, 4 * k.shape[1]).astype(np.float64)
        b = t[r0:r0 + (1 << 18)].view(np.uint16).reshape(-1, 4 * t.shape[1]).astype(np.float64)
        m = (a.T @ b).astype(np.int64)
        for i in range(m.shape[0]):
            for j in range(m.shape[1]):
                acc += int(m[i, j]) << (16 * (i + j))
    return acc % R_ORDER


def _words(point, group):
    """Affine point -> the words of its struct (Montgomery form, infinity flag)."""
    if point is None:
        return [0] * (14 * group) + [1]
    vals = list(point) if group == 1 else [c for xy in point for c in xy]
    out = []
    for v in vals:
        m = v * R % P
        out += [(m >> (64 * i)) & (2 ** 64 - 1) for i in range(7)]
    return out + [0]


def exact(case, seed):
    if case["kind"] == "field":
        a, b = _field_inputs(case, seed)
        cols = a.shape[1]
        x = [int.from_bytes(a[i].tobytes()[s:s + 56], "little") for i in range(len(a)) for s in range(0, 8 * cols, 56)]
        y = [int.from_bytes(b[i].tobytes()[s:s + 56], "little") for i in range(len(b)) for s in range(0, 8 * cols, 56)]
        if cols == 7:
            z = [u * v * R_INV % P for u, v in zip(x, y)]
        else:
            z = []
            for u0, u1, v0, v1 in zip(x[0::2], x[1::2], y[0::2], y[1::2]):
                z.append((u0 * v0 - u1 * v1) * R_INV % P)
                z.append((u0 * v1 + u1 * v0) * R_INV % P)
        out = np.frombuffer(b"".join(v.to_bytes(56, "little") for v in z), dtype=np.int64)
        return torch.from_numpy(out.reshape(case["n"], cols).copy())
    group = case["group"]
    F = _F1 if group == 1 else _F2
    sc, logs, sizes, offs = _inputs(case, seed)
    doubles = _gen_doubles(group)
    if sizes is None:
        rows = [_words(_gen_times(_dot(sc, logs), doubles, F), group)]
    else:
        rows, at = [], 0
        for s, o in zip(sizes, offs):
            rows.append(_words(_gen_times(_dot(sc[at:at + s], logs[o:o + s]), doubles, F), group))
            at += s
    out = np.array(rows, dtype=np.uint64).view(np.int64)
    return torch.from_numpy(out[0].copy()) if case["kind"] == "device" else out
