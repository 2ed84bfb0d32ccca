"""The inline PTX of the field products (field_ptx.cuh, fp_bipartite.cuh) and the slot programs of the eight-lane ladders
(g1_ladder.cuh), run on exact integers: results, stated bounds, and no carry out of an instruction that drops it."""
import pathlib
import random
import re

import pytest

from helpers import R_MOD

CSRC = pathlib.Path(__file__).resolve().parents[1] / "cubbs-cred_gb300" / "csrc"
P = 0x1A0111EA397FE69A4B1BA7B6434BACD764774B84F38512BF6730D2A0F6B0F6241EABFFFEB153FFFFB9FEFFFFFFFFAAAB
MASK = 0xFFFFFFFF
ALL = 1 << 384
EDGES = [0, 1, 2, P - 1, P, P + 1, 2 * P, ALL - 1, ALL - 2, (1 << 192) - 1, 1 << 192, ALL - (1 << 192), (1 << 352) - 1,
         ALL - (1 << 352), sum(MASK << (64 * k) for k in range(6)), sum(MASK << (64 * k + 32) for k in range(6))]


def _limbs(x, n):
    return [(x >> (32 * k)) & MASK for k in range(n)]


def _value(words):
    return sum(w << (32 * k) for k, w in enumerate(words))


def _body(header, name):
    text = (CSRC / header).read_text()
    text = text[text.index("void %s(" % name):]
    text = text[text.index('asm("') + 5:]
    return text[:text.index('" :')].split("\\n\\t")


def _run(lines, outputs, inputs):
    """The words that the asm text leaves in its operands %0 .. %(outputs - 1)."""
    regs = {"%%%d" % (outputs + k): v for k, v in enumerate(inputs)}
    carry = 0

    def val(x):
        return int(x, 16) if x.startswith("0x") else int(x) & MASK if x.isdigit() else regs[x]
    for line in lines:
        line = line.strip().rstrip(";")
        if line.startswith("{") or line == "}":
            continue
        op, rest = line.split(None, 1)
        a, mods = [x.strip() for x in rest.split(",")], op.split(".")
        base = mods[0]
        if base == "mov":
            regs[a[0]] = val(a[1])
        elif base == "shf":
            assert mods[1:] == ["l", "clamp", "b32"] and 0 < val(a[3]) < 32
            regs[a[0]] = (val(a[2]) << val(a[3]) | val(a[1]) >> (32 - val(a[3]))) & MASK
        elif base == "mul":
            regs[a[0]] = val(a[1]) * val(a[2]) >> (32 if "hi" in mods else 0) & MASK
        else:
            assert base in ("add", "addc", "mad", "madc"), line
            if base.startswith("mad"):
                t = (val(a[1]) * val(a[2]) >> (32 if "hi" in mods else 0) & MASK) + val(a[3])
            else:
                t = val(a[1]) + val(a[2])
            t += carry if base.endswith("c") else 0
            regs[a[0]] = t & MASK
            if "cc" in mods:
                carry = t >> 32
            else:
                assert t >> 32 == 0, line
    return [regs["%%%d" % k] for k in range(outputs)]


def _operands(rng, n, bound, count):
    edges = [x for x in EDGES if x < bound] + [bound - 1]
    for k in range(count):
        yield [rng.choice(edges) if rng.random() < 0.5 else rng.randrange(bound) for _ in range(n)]


def test_products_on_two_warps():
    """Any two 384-bit values: the halves' finish is a b / 2^256 mod p below p + 2^352; the square likewise."""
    body = {n: _body("fp_bipartite.cuh", "fp_bp_" + n) for n in ("mul_lo", "mul_hi", "sqr_lo", "sqr_hi", "finish")}
    r_inv, rng = pow(1 << 256, -1, P), random.Random(5)

    def finish(kind, words):
        r = _value(_run(body["finish"], 12, _run(body[kind + "_lo"], 13, words) + _run(body[kind + "_hi"], 13, words)))
        assert r < P + (1 << 352)
        return r
    pairs = [[x, y] for x in EDGES for y in EDGES] + list(_operands(rng, 2, ALL, 200))
    for a, b in pairs:
        assert (finish("mul", _limbs(a, 12) + _limbs(b, 12)) - a * b * r_inv) % P == 0, (a, b)
    for a in EDGES + [x for x, _ in pairs[-200:]]:
        assert (finish("sqr", _limbs(a, 12)) - a * a * r_inv) % P == 0, a


@pytest.mark.parametrize("name,mod,n,args,bound", [("fp_mont_mul", P, 12, 2, 6 * P), ("fp_mont_sqr", P, 12, 1, 4 * P),
                                                   ("fr_mont_mul", R_MOD, 8, 2, R_MOD)])
def test_products_on_one_lane(name, mod, n, args, bound):
    """Operands up to the largest factors in use: a b / 2^(32 n) mod p, below p + a b / 2^(32 n)."""
    body, rng = _body("field_ptx.cuh", name), random.Random(6)
    r_inv = pow(1 << (32 * n), -1, mod)
    for v in _operands(rng, args, bound, 300):
        want = v[0] * v[-1]
        r = _value(_run(body, n, [w for x in v for w in _limbs(x, n)]))
        assert (r - want * r_inv) % mod == 0 and r <= mod + (want >> (32 * n)), v


# ---- the ladders' operations
@pytest.fixture(scope="module")
def ladder():
    """The slot numbers and the three operations, from the header's text."""
    text = (CSRC / "g1_ladder.cuh").read_text()
    names = ["ZERO", "AX", "AY", "AZ"] + ["P%d" % k for k in range(8)] + ["E%d" % k for k in range(6)]
    ns = {n: k for k, n in enumerate(names)}
    ns.update(NONE=None, BY_TAB=0)

    def rows(op):
        body = text[text.index("__device__ const Op %s = " % op):]
        body = body[body.index("=") + 1:body.index(";")]
        body = body.replace("GL_IDLE_M", "{ZERO, ZERO, ZERO, ZERO, NONE, 1}")
        body = body.replace("GL_IDLE_S", "{ZERO, ZERO, ZERO, ZERO, NONE}")
        body = re.sub(r"BY_TAB \| (\d)", lambda m: '("tab", %s)' % m.group(1), body)
        groups = eval(body.replace("{", "[").replace("}", "]"), {}, ns)  # the header's own braces
        assert [len(g) for g in groups] == [8, 8, 8]
        return groups
    return ns, {op: rows(op) for op in ("DBL", "ADD", "ADD4")}


# bounds of the slots in units of p: the accumulator, the tables and the outputs are reduced sums
REDUCED = 1.001
QMAX = 72


def _bounds(ns, op):
    """Largest value of every slot and sum of an operation whose inputs are reduced, in units of p; checks that no
    lane_sum can be negative, no factor reaches 2^384 and every value that reduce13 takes is below QMAX p."""
    first, sums, second = op
    two384 = ALL / P
    hi = {ns["ZERO"]: 0.0, ns["AX"]: REDUCED, ns["AY"]: REDUCED, ns["AZ"]: REDUCED}
    lo = dict.fromkeys(hi, 0.0)
    get = lambda s: REDUCED if isinstance(s, tuple) else hi[s]  # noqa: E731

    def product(x, y):
        assert x < two384 and y < two384
        return x * y / two384 + 1
    out = {}
    for a, a2, b, b2, o, k in first:
        v = k * product(get(a) + get(a2), get(b) + get(b2))
        assert v < QMAX and k < 256
        if o is not None:
            out[o] = REDUCED
    hi.update(out)
    lo.update(dict.fromkeys(out, 0.0))
    out = {}
    for p0, p1, m0, m1, o in sums:
        top, low = 3 + hi[p0] + hi[p1], 3 - hi[m0] - hi[m1]
        assert low > 0 and top < two384
        if o is not None:
            out[o] = top
    hi.update(out)
    worst = 0.0
    v = [k * product(hi[a], hi[b]) for a, a2, b, b2, o, k in second]
    assert all(a2 == b2 == ns["ZERO"] for _, a2, _, b2, _, _ in second)
    for k, row in enumerate(second):
        pair = v[k] + v[k ^ 1]
        assert pair < QMAX
        worst = max(worst, pair)
        if row[4] is not None:
            assert k % 2 == 0 or second[k ^ 1][4] is None
    return worst


def test_ladder_bounds(ladder):
    ns, ops = ladder
    assert max(_bounds(ns, op) for op in ops.values()) < QMAX  # 53.7: 36 P0 E3 + E5 E4 of ADD4


def _apply(ns, op, acc, tab):
    """(X, Y, Z) that the operation leaves, on plain residues."""
    first, sums, second = op
    s = {ns["ZERO"]: 0, ns["AX"]: acc[0], ns["AY"]: acc[1], ns["AZ"]: acc[2]}
    get = lambda x: tab[{0: 0, 1: 1, 3: 2}[x[1]]] if isinstance(x, tuple) else s[x]  # noqa: E731
    out = {o: (get(a) + get(a2)) * (get(b) + get(b2)) * k % P for a, a2, b, b2, o, k in first if o is not None}
    s.update(out)
    out = {o: (s[p0] + s[p1] - s[m0] - s[m1]) % P for p0, p1, m0, m1, o in sums if o is not None}
    s.update(out)
    v = [k * s[a] * s[b] for a, _, b, _, _, k in second]
    s.update({row[4]: (v[k] + v[k ^ 1]) % P for k, row in enumerate(second) if row[4] is not None})
    return s[ns["AX"]], s[ns["AY"]], s[ns["AZ"]]


def test_ladder_operations_are_complete(ladder):
    """DBL, ADD on y^2 = x^3 + 2/3 and ADD4 on y^2 = x^3 + 4 equal the affine law for general, equal, opposite and
    identity points, the point of order 3 with x = 0 among them."""
    ns, ops = ladder
    rng = random.Random(7)

    def points(b):
        out = []
        while len(out) < 4:
            x = rng.randrange(P)
            y = pow(x ** 3 + b, (P + 1) // 4, P)
            if (y * y - x ** 3 - b) % P == 0:
                out.append((x, y))
        y = pow(b, (P + 1) // 4, P)
        return out + ([(0, y)] if y * y % P == b % P else [])

    def add(a, b):
        if a is None or b is None:
            return a or b
        if a[0] == b[0]:
            if (a[1] + b[1]) % P == 0:
                return None
            m = 3 * a[0] * a[0] * pow(2 * a[1], -1, P)
        else:
            m = (b[1] - a[1]) * pow(b[0] - a[0], -1, P)
        x = (m * m - a[0] - b[0]) % P
        return x, (m * (a[0] - x) - a[1]) % P

    def project(a):
        z = rng.randrange(1, P)
        return (0, z, 0) if a is None else (a[0] * z % P, a[1] * z % P, z)

    def affine(t):
        assert any(t)
        return None if t[2] == 0 else (t[0] * pow(t[2], -1, P) % P, t[1] * pow(t[2], -1, P) % P)
    for name, b in (("DBL", 2 * pow(3, -1, P) % P), ("ADD", 2 * pow(3, -1, P) % P), ("ADD4", 4)):
        pts = points(b)
        pts += [None] + [(x, P - y) for x, y in pts[:2]]
        for u in pts:
            if name == "DBL":
                assert affine(_apply(ns, ops[name], project(u), None)) == add(u, u)
                continue
            for w in pts:
                assert affine(_apply(ns, ops[name], project(u), project(w))) == add(u, w), name
