"""The phase tables of the four-warp pairing (pairing_quad_program.cuh), decoded the way pairing_quad.cuh reads them and
run on exact integers with the device's bounds, against the schoolbook Fp12 of gen_pairing_program.py."""
import pathlib
import random
import re
import sys

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "cubbs-cred_gb300" / "csrc"


@pytest.fixture(scope="module")
def gen():
    sys.path.insert(0, str(CSRC))
    try:
        import gen_pairing_quad
    finally:
        sys.path.remove(str(CSRC))
    return gen_pairing_quad


@pytest.fixture(scope="module")
def header():
    return (CSRC / "pairing_quad_program.cuh").read_text()


def _entries(text, name):
    start = text.index(name + "[")
    body = text[text.index("{", start):text.index("};", start)]
    w = [int(x, 16) for x in re.findall(r"0x([0-9a-f]{8})\b", body)]
    return [w[k:k + 4] for k in range(0, len(w), 4)]


def _slot(off):
    assert off % 48 == 0
    return off // 48


def _product(q, s, e):
    a, b = s[_slot(e[0] & 0xFFFF)], s[_slot(e[0] >> 16)]
    if e[3] & 0x10:
        a, b = a + s[_slot(e[1] & 0xFFFF)], b + s[_slot(e[1] >> 16)]
    r = q.mont(a, b << ((e[3] >> 5) & 1))
    assert r < 1.42 * q.P
    return r


def _lane_sum(q, s, plus, minus):
    return q.lane_sum(s, (_slot(plus & 0xFFFF), _slot(plus >> 16), _slot(minus & 0xFFFF), _slot(minus >> 16)))


def _run(q, header, s, prog):
    first = [int(x) for x in re.search(r"PQ_FIRST\[PQ_NPROG \+ 1\] = \{([^}]*)\}", header).group(1).split(",")]
    ent = _entries(header, "PQ_ENTRY")
    assert len(ent) == first[-1] * q.LANES
    for ph in range(first[prog], first[prog + 1]):
        rows, res = ent[ph * q.LANES:(ph + 1) * q.LANES], {}
        assert len({r[3] & 1 for r in rows}) == 1  # one type a phase
        if not rows[0][3] & 1:
            assert len({r[3] & 0x10 for r in rows}) == 1
            res = {_slot(r[2]): _product(q, s, r) for r in rows if r[2] != q.NONE}
        else:
            for w in range(4):
                lanes = rows[32 * w:32 * w + 32]
                assert len({r[3] for r in lanes}) == 1
                g = (lanes[0][3] >> 4) & 7
                if g == 7:
                    continue
                for k in range(0, 32, 1 << g):
                    outs = [r[2] for r in lanes[k:k + (1 << g)] if r[2] != q.NONE]
                    assert len(outs) <= 1 and (not outs or lanes[k][2] == outs[0])
                    if outs:
                        res[_slot(outs[0])] = q.reduce13(sum(_lane_sum(q, s, r[0], r[1]) for r in lanes[k:k + (1 << g)]))
        s.update(res)


def _cyclo(q, header, s):
    em, es = _entries(header, "PQ_CYCLO_M"), _entries(header, "PQ_CYCLO_S")
    s.update({_slot(e[2]): _product(q, s, e) for e in em if e[2] != q.NONE})
    v = [3 * _lane_sum(q, s, e[0], e[1]) + s[_slot(e[2] >> 16)] - s[_slot(e[3])] for e in es]
    assert min(v) > 0
    s.update({_slot(es[k][2] & 0xFFFF): q.reduce13(v[k] + v[k + 1]) for k in range(0, 32, 2)
              if es[k][2] & 0xFFFF != q.NONE})


@pytest.mark.parametrize("values", ["random", "extreme"])
def test_tables_match_schoolbook(gen, header, values):
    rng = random.Random(11)
    for prog, name in enumerate(list(gen.PROGRAMS) + ["CYCLO"]):
        if name == "LINE":
            continue
        v = gen.G.random_slots(rng, cyclo_regs=(gen.REG_R,) if name == "CYCLO" else ())
        v.update({gen.LB + k: rng.randrange(gen.P) for k in range(4)})
        v.update({gen.NORM2 + k: x for k, x in enumerate(gen.norm2())})
        if values == "extreme" and name != "CYCLO":
            v.update({k: rng.choice([0, 1, gen.P - 1, gen.P - 2]) for k in range(72)})
        s = {k: (x << 384) % gen.P for k, x in v.items()}
        s.update({k: rng.randrange(gen.P) for k in range(gen.TMP, gen.TMP + gen.LANES)})
        if name == "CYCLO":
            _cyclo(gen, header, s)
        else:
            _run(gen, header, s, prog)
        r, want = gen.expected(name, v)
        assert gen.G.to_w({k: x * gen.R_INV % gen.P for k, x in s.items()}, r) == want(), name


def test_quotient_estimate_bounds(gen):
    """Every multiple of p in the table, its neighbours, and random sums: the remainder is below 1.001 p."""
    rng = random.Random(3)
    for k in range(1, gen.QMAX):
        for d in (-2, -1, 0, 1, 1 << 359, -(1 << 359)):
            gen.reduce13(min(max(0, k * gen.P + d), gen.QMAX * gen.P - 1))
    for _ in range(2000):
        gen.reduce13(rng.randrange(gen.QMAX * gen.P))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 4, 153, 700])
def test_checks_by_launch_size(gpu, oracle, n):
    """One block per check, from one check to several per SM: e(sk2 P1, pk1) == e(sk1 P1, pk2) holds, a swapped key
    breaks it, and identity points drop one pair or both."""
    from helpers import keypair
    p1, _ = oracle.generators(1)
    (sk1, pk1), (sk2, pk2) = keypair(oracle, b"quad", 1), keypair(oracle, b"quad", 2)
    a, b, inf = oracle.g1_mul(p1, sk2), oracle.g1_mul(p1, sk1), bytes([0xC0]) + bytes(47)
    kinds = [((a, pk1, b, pk2), True), ((a, pk1, b, pk1), False), ((inf, pk1, inf, pk2), True),
             ((inf, pk1, b, pk2), False), ((a, pk1, inf, pk2), False)]
    reqs, want = zip(*(kinds[i % len(kinds)] for i in range(n)))
    assert gpu.pairing_eq_batch(list(reqs)) == [(0, w) for w in want]
