"""Split windows at every window width and chunk length, against the oracle: chunks that are full, one term short and one
over, equal, opposite and identity points, scalars 0, 1 and r - 1, chunks whose digits share one bucket, and rows that are
rejected beside good ones."""
import random

import pytest

from helpers import R_MOD as R
from tests.test_gpu_parity import _on_curve_outside_g1

pytestmark = pytest.mark.gpu
LAMBDA = 0xAC45A4010001A4020000000100000000
INF = bytes([0xC0]) + bytes(47)


def be(k):
    return k.to_bytes(32, "big")


def expected(oracle, msm):
    """The sum with the scalars of equal points added first: a few terms whatever the length."""
    total = {}
    for p, k in zip(*msm):
        total[p] = (total.get(p, 0) + int.from_bytes(k, "big")) % R
    return oracle.g1_msm(list(total), [be(k) for k in total.values()])


@pytest.fixture(scope="module")
def base(oracle):
    p1, gens = oracle.generators(6)
    pts = [p1] + list(gens)
    return pts + [bytes([p[0] ^ 0x20]) + p[1:] for p in pts[:3]] + [INF]


@pytest.mark.parametrize("t", [8, 16, 32, 64, 120])
@pytest.mark.parametrize("c", [3, 4, 5])
def test_every_form(gpu, oracle, base, c, t):
    rng = random.Random(repr((c, t)))
    ks = [0, 1, R - 1] + [rng.randrange(R) for _ in range(40)]
    sizes = [0, 1, 2, t - 1, t, t + 1, 2 * t - 1, 2 * t, 2 * t + 1, 9 * t, 0, 7]
    msms = [([rng.choice(base) for _ in range(k)], [be(rng.choice(ks)) for _ in range(k)]) for k in sizes]
    # both halves of every scalar the same: x (LAMBDA + 1); the digits of each window all fall in one bucket
    windows = 127 // c
    for d in (1, (1 << (c - 1)) - 1, 1 << (c - 1), (1 << c) - 1):
        x = sum(d << (c * w) for w in range(windows))
        msms.append(([base[i % 7] for i in range(t)], [be(x * (LAMBDA + 1) % R)] * t))
    assert gpu.g1_msm_batch(msms, split=(c, t)) == [(0, expected(oracle, m)) for m in msms]


@pytest.mark.parametrize("split", [None, (3, 8), (5, 120)])
def test_rejected_rows(gpu, oracle, base, split):
    """A point outside G1, of order 3, off the curve, not reduced, with bad flags; a scalar r and one above it: the row is
    rejected wherever the bad term stands, and every other row is right."""
    off = next(bytes([0x80]) + x.to_bytes(47, "big") for x in range(1, 99)
               if pow(x ** 3 + 4, (oracle.P_MOD - 1) // 2, oracle.P_MOD) != 1)
    unreduced = bytearray((oracle.P_MOD + 1).to_bytes(48, "big"))
    unreduced[0] |= 0x80
    bad = [(_on_curve_outside_g1(oracle, b"split"), be(5)), (bytes([0x80]) + bytes(47), be(5)), (off, be(5)),
           (bytes(unreduced), be(5)), (bytes([base[0][0] & 0x7F]) + base[0][1:], be(5)), (bytes([0xE0]) + bytes(47), be(5)),
           (base[1], be(R)), (base[1], b"\xff" * 32), (INF, be(R)), (_on_curve_outside_g1(oracle, b"split"), be(0))]
    rng = random.Random(9)
    msms, rejected = [], {}
    for i in range(64):
        k = 8 + i % 30 if i % 16 else 250
        pts, scs = [rng.choice(base) for _ in range(k)], [be(rng.randrange(R)) for _ in range(k)]
        if i % 3 == 1:
            at = (0, k - 1, k // 2)[len(rejected) % 3]
            pts[at], scs[at] = bad[len(rejected) % len(bad)]
            rejected[i] = True
        msms.append((pts, scs))
    assert len(rejected) > 2 * len(bad)
    got = gpu.g1_msm_batch(msms, split=split)
    assert [code for code, _ in got] == [1 if i in rejected else 0 for i in range(64)]
    assert [p for i, (_, p) in enumerate(got) if i not in rejected] == \
        [expected(oracle, m) for i, m in enumerate(msms) if i not in rejected]
