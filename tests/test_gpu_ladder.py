"""The eight-lane G1 ladders: launches that leave lanes of a warp over, scalars at the edges of the signed 4-bit digits
and of the GLV split, the identity, and the membership test on points in and out of G1, of small order too."""
import pytest

from helpers import scalar
from tests.test_gpu_parity import _on_curve_outside_g1

pytestmark = pytest.mark.gpu
LAMBDA = 0xAC45A4010001A4020000000100000000
INF = bytes([0xC0]) + bytes(47)


@pytest.mark.parametrize("n", [1, 2, 3, 8])
def test_terms(gpu, oracle, n):
    p1, gens = oracle.generators(4)
    r = oracle.R_MOD
    ks = [0, 1, 2, 7, 8, 9, 15, 16, 17, 128, LAMBDA - 1, LAMBDA, LAMBDA + 1, 8 * LAMBDA + 8, (1 << 128) - 1, 1 << 128,
          int("88" * 16, 16), int("77" * 16, 16) * LAMBDA % r, r - 1, r - LAMBDA]
    ks += [int.from_bytes(scalar(b"ladder", b"k", i), "big") for i in range(4)]
    pts = [p1] + gens[:3]
    for at in range(0, len(ks), n):  # n one-term MSMs a call: fewer than the bucket engine takes
        msms = [([pts[(at + j) % 4]], [k.to_bytes(32, "big")]) for j, k in enumerate(ks[at:at + n])]
        assert gpu.g1_msm_batch(msms) == [(0, oracle.g1_mul(p[0], s[0])) for p, s in msms], at
    assert gpu.g1_msm_batch([([INF], [ks[3].to_bytes(32, "big")])] * n) == [(0, INF)] * n


@pytest.mark.parametrize("n", [608, 609])
def test_terms_shared_products(gpu, oracle, n):
    """The most terms whose products two warps share, and one more."""
    p1, gens = oracle.generators(4)
    pts = [p1] + gens[:3]
    ks = [scalar(b"shared", b"k", i) for i in range(n)]
    ks[5], ks[n - 1] = bytes(32), (oracle.R_MOD - 1).to_bytes(32, "big")
    got = gpu.g1_msm_batch([([pts[i % 4]], [ks[i]]) for i in range(n)])
    assert all(c == 0 for c, _ in got)
    for i in (0, 1, 5, 6, n // 2, n - 2, n - 1):
        assert got[i][1] == oracle.g1_mul(pts[i % 4], ks[i]), i


@pytest.mark.parametrize("n", [1, 3, 4, 6])
def test_membership(gpu, oracle, n):
    p1, gens = oracle.generators(4)
    order3 = [bytes([0x80 | sign]) + bytes(47) for sign in (0, 0x20)]  # (0, 2) and (0, -2)
    pts = [(p1, 0), (_on_curve_outside_g1(oracle, b"ladder"), 1), (order3[0], 1), (gens[0], 0), (order3[1], 1),
           (gens[1], 0)]
    got = gpu.g1_subgroup_for_test([p for p, _ in pts[:n]])
    assert got == [(0, bad) for _, bad in pts[:n]]
    assert gpu.g1_subgroup_for_test([INF] * n) == [(1, 0)] * n


@pytest.mark.parametrize("rows", [1, 3, 45, 700, 1400])
def test_fixed_rows(gpu, oracle, rows):
    """Fixed-base rows from one (a block of warps) to many (several rows a warp), with scalars whose windows sit on
    either side of half at every table width, zero and r - 1 rows among them."""
    p1, gens = oracle.generators(11)
    pts, r = [p1] + gens, oracle.R_MOD

    def edge(w, d):  # every window half + d
        return sum(((1 << (w - 1)) + d) << (w * k) for k in range(255 // w)) % r
    kinds = [0, r - 1, 1] + [edge(w, d) for w in (8, 14, 16, 19, 20) for d in (-1, 0, 1)]

    def row(i):
        if i % 97 == 1:
            return [bytes(32)] * 12
        return [(kinds[(i + k) % len(kinds)]).to_bytes(32, "big") if (i + k) % 3 == 0 else scalar(b"rows", b"%d" % i, k)
                for k in range(12)]
    scalars = [row(i) for i in range(rows)]
    got = gpu.g1_msm_common_points(pts, scalars)
    assert all(c == 0 for c, _, _ in got)
    for i in sorted({0, 1, 2, 7, 8, 15, 16, 31, 32, 98, rows // 2, rows - 2, rows - 1} & set(range(rows))):
        assert got[i][2] == oracle.g1_msm(pts, scalars[i]), i


@pytest.mark.parametrize("n", [1, 31, 33, 70])
def test_decode_pairs(gpu, oracle, n):
    """Points decoded on pairs of warps, spare lanes in the last block: both signs, the identity, an x off the curve, an
    x that is not reduced, bad flag bits, and points outside G1, through the checked MSM decode."""
    p1, gens = oracle.generators(4)
    neg = [bytes([p[0] ^ 0x20]) + p[1:] for p in (p1, gens[0])]
    off = next(bytes([0x80]) + x.to_bytes(47, "big") for x in range(1, 99)
               if pow(x ** 3 + 4, (oracle.P_MOD - 1) // 2, oracle.P_MOD) != 1)
    big = bytearray((oracle.P_MOD + 1).to_bytes(48, "big"))
    big[0] |= 0x80
    kinds = [(p1, 0), (neg[0], 0), (off, 1), (gens[1], 0), (INF, 0), (bytes(big), 1), (neg[1], 0),
             (bytes([p1[0] & 0x7F]) + p1[1:], 1), (_on_curve_outside_g1(oracle, b"pairs"), 1),
             (bytes([0xE0]) + bytes(47), 1), (bytes([0x80]) + bytes(47), 1)]
    one = (1).to_bytes(32, "big")
    want = [(p if not bad else None) for p, bad in (kinds[i % len(kinds)] for i in range(n))]
    got = gpu.g1_msm_batch([([kinds[i % len(kinds)][0]], [one]) for i in range(n)])
    assert [c for c, _ in got] == [0 if w is not None else 1 for w in want]
    assert [p for (_, p), w in zip(got, want) if w is not None] == [w for w in want if w is not None]


@pytest.mark.parametrize("n", [19456, 19457])
def test_membership_of_many(gpu, oracle, n):
    """A lane per point, in Jacobian coordinates, and the lane pairs just below: points in and out of G1, of order 3 and
    of order 11 or 121 (sums with equal and opposite points, and the identity, within the chain)."""
    p, q = oracle.P_MOD, oracle.R_MOD

    def add(a, b):
        if a is None or b is None:
            return a or b
        if a[0] == b[0]:
            if (a[1] + b[1]) % p == 0:
                return None
            m = 3 * a[0] * a[0] * pow(2 * a[1], -1, p)
        else:
            m = (b[1] - a[1]) * pow(b[0] - a[0], -1, p)
        x = (m * m - a[0] - b[0]) % p
        return x, (m * (a[0] - x) - a[1]) % p
    order = 0x396C8C005555E1568C00AAAB0000AAAB * q
    assert order % 121 == 0
    small, x = [], 0
    while len(small) < 2:
        x += 1
        y = pow(x ** 3 + 4, (p + 1) // 4, p)
        if (y * y - x ** 3 - 4) % p:
            continue
        r, k, b = None, order // 121, (x, y)
        while k:
            r, b, k = add(r, b) if k & 1 else r, add(b, b), k >> 1
        if r:
            small.append(bytes([r[0].to_bytes(48, "big")[0] | 0x80 | (0x20 if r[1] > p // 2 else 0)]) +
                         r[0].to_bytes(48, "big")[1:])
    p1, gens = oracle.generators(2)
    pts = [(p1, 0), (_on_curve_outside_g1(oracle, b"many"), 1), (bytes([0x80]) + bytes(47), 1), (small[0], 1),
           (gens[0], 0), (small[1], 1), (gens[1], 0)]
    assert gpu.g1_subgroup_for_test([pts[i % 7][0] for i in range(n)]) == [(0, pts[i % 7][1]) for i in range(n)]
