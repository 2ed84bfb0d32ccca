#!/usr/bin/env python3
"""Generates pairing_quad_program.cuh: the phase tables of the four-warp pairing.

One check runs on a block of 128 lanes over the slot array of
gen_pairing_program.py (same registers, lines, points and constants).  Its
programs alternate two kinds of phases:

  M phase : a lane computes slot[out] = (slot[a] + slot[a2]) * (slot[b] + slot[b2]) << dbl
            (one Montgomery product; the a2, b2 loads only in phases that have sums)
  S phase : 2^g neighbouring lanes compute one output, each lane
            3p + slot[p0] + slot[p1] - slot[m0] - slot[m1], added over the lanes and reduced
            by the multiple of p its top bits give

so every output of an Fp12 operation is one signed sum of products, whatever
its number of terms, and an operation is one M and one S phase: schoolbook Fp2
products (four, or three with operand sums for the full Fp12 product), 128 at
most.  The cyclotomic squaring (30 products, outputs on lane pairs) has a
table of its own for one warp; its outputs 3 A -+ 2 v are 3 (A -+ v) +- v.

Values in slots stay below 1.001 p (S outputs) or 1.41 p (products); the
check below runs every program on exact integers, follows the device's
quotient estimate in single precision and asserts each bound, and compares the
results with the schoolbook Fp12 of gen_pairing_program.py.

Usage: python gen_pairing_quad.py [--check-only]
"""
import pathlib
import random
import sys

import numpy as np

import gen_pairing_program as G
from gen_pairing_program import P, reg_slot, REG_F, REG_T, REG_A, REG_X, REG_R, REG_U

LANES = 128
NONE = 0xFFFF
ZERO = G.ZERO_SLOT
LINE, PT, GAMMA = G.LINE_BASE, G.PT_BASE, G.GAMMA_BASE
LB = G.TMP_BASE          # B xP of both lines (4 slots)
LAM = LB + 4             # the product of both lines: w^0, w^2, w^3, w^4, w^5 (10 slots)
NORM2 = LAM + 10         # gamma_e conj(gamma_e), e = 1..5: the factors of x -> x^(p^2) (5 slots)
TMP = NORM2 + 5          # products
QMAX = 72                # multiples of p in the table
K_OF_W = [0, 3, 1, 4, 2, 5]  # slot-order coefficient of w^e


def reg(r):
    """Fp2 coefficients of register r by power of w, as slot pairs."""
    return [(reg_slot(r, K_OF_W[e], 0), reg_slot(r, K_OF_W[e], 1)) for e in range(6)]


class M:
    """One M phase: products by operands, results in temporaries (or given slots)."""

    def __init__(self):
        self.ent, self.next = [], TMP

    def mul(self, a, b, dbl=0, out=None):
        """a, b: slot or (slot, slot) for a sum."""
        if out is None:
            out, self.next = self.next, self.next + 1
        self.ent.append((out, a, b, dbl))
        return out

    def f2(self, x, y):
        """Forms (re, im) of the Fp2 product x y: four products."""
        p = [[self.mul(x[i], y[j]) for j in range(2)] for i in range(2)]
        return {p[0][0]: 1, p[1][1]: -1}, add({p[0][1]: 1}, {p[1][0]: 1})

    def f2_twice(self, x, y):
        p = [[self.mul(x[i], y[j], 1) for j in range(2)] for i in range(2)]
        return {p[0][0]: 1, p[1][1]: -1}, add({p[0][1]: 1}, {p[1][0]: 1})

    def f2_kar(self, x, y):
        """The same from three products of which one has operand sums."""
        p0, p1, p2 = self.mul(x[0], y[0]), self.mul(x[1], y[1]), self.mul((x[0], x[1]), (y[0], y[1]))
        return {p0: 1, p1: -1}, {p2: 1, p0: -1, p1: -1}

    def f2_sqr(self, x):
        p0, p1, d = self.mul(x[0], x[0]), self.mul(x[1], x[1]), self.mul(x[0], x[1], 1)
        return {p0: 1, p1: -1}, {d: 1}


def add(*forms):
    r = {}
    for f in forms:
        for s, c in f.items():
            r[s] = r.get(s, 0) + c
    return {s: c for s, c in r.items() if c}


def neg(f):
    return {s: -c for s, c in f.items()}


def xi(v):
    return add(v[0], neg(v[1])), add(*v)


class Sum:
    """One S phase: outputs (slot, form) on 2^g lanes each; `warps`: [(g, outputs)], one entry per warp."""

    def __init__(self, outs, g=3):
        per = 32 >> g
        self.warps = [(g, outs[k:k + per]) for k in range(0, len(outs), per)]

    def then(self, outs, g):
        per = 32 >> g
        self.warps += [(g, outs[k:k + per]) for k in range(0, len(outs), per)]
        assert len(self.warps) <= 4
        return self


def outputs(r, coeffs, conj=False):
    """S outputs of the Fp12 value with forms coeffs[e] into register r, conjugated (odd powers negated) if asked."""
    out = []
    for e, (s0, s1) in enumerate(reg(r)):
        for s, f in zip((s0, s1), coeffs[e]):
            out.append((s, neg(f) if conj and e & 1 else f))
    return out


def product(m, x, y, prod, signs=lambda i, j: 1):
    """Forms of sum_ij x_i y_j w^(i+j), w^6 = xi; x, y: {power: slots}."""
    acc = [({}, {}) for _ in range(6)]
    for i, a in x.items():
        for j, b in y.items():
            v = prod(m, a, b)
            if signs(i, j) < 0:
                v = neg(v[0]), neg(v[1])
            if i + j >= 6:
                v = xi(v)
            k = (i + j) % 6
            acc[k] = add(acc[k][0], v[0]), add(acc[k][1], v[1])
    return acc


def d(r):
    return dict(enumerate(reg(r)))


def lam_slots():
    return {e: (LAM + 2 * k, LAM + 2 * k + 1) for k, e in enumerate((0, 2, 3, 4, 5))}


def lines(m):
    """S outputs of l_0 l_1 with l_p = A_p + (B_p xP_p) w^2 + yP_p w^3."""
    A = [(LINE + 4 * p, LINE + 4 * p + 1) for p in (0, 1)]
    B = [(LB + 2 * p, LB + 2 * p + 1) for p in (0, 1)]
    y = [PT + 2 * p + 1 for p in (0, 1)]

    def by_y(x, s):
        return {m.mul(x[0], s): 1}, {m.mul(x[1], s): 1}
    yy = m.mul(y[0], y[1])
    ab, ba = m.f2(A[0], B[1]), m.f2(A[1], B[0])
    ay, ya = by_y(A[0], y[1]), by_y(A[1], y[0])
    byv, yb = by_y(B[0], y[1]), by_y(B[1], y[0])
    aa = m.f2(A[0], A[1])
    co = {0: (add(aa[0], {yy: 1}), add(aa[1], {yy: 1})),  # xi y_0 y_1 = (y_0 y_1, y_0 y_1)
          2: (add(ab[0], ba[0]), add(ab[1], ba[1])), 3: (add(ay[0], ya[0]), add(ay[1], ya[1])),
          4: m.f2(B[0], B[1]), 5: (add(byv[0], yb[0]), add(byv[1], yb[1]))}
    return [(s, f) for e, sl in lam_slots().items() for s, f in zip(sl, co[e])]


def next_line(m):
    """B xP of the lines now in the line slots."""
    for p in (0, 1):
        for c in (0, 1):
            m.mul(LINE + 4 * p + 2 + c, PT + 2 * p, out=LB + 2 * p + c)


def prog_line():
    m = M()
    next_line(m)
    return [m]


def prog_dbl():
    m1 = M()
    f = reg(REG_F)
    co = [({}, {}) for _ in range(6)]
    for i in range(6):
        for j in range(i, 6):
            v = m1.f2_sqr(f[i]) if i == j else m1.f2_twice(f[i], f[j])
            if i + j >= 6:
                v = xi(v)
            k = (i + j) % 6
            co[k] = add(co[k][0], v[0]), add(co[k][1], v[1])
    lam = lines(m1)
    s1 = Sum(outputs(REG_U, co)).then(lam, 1)
    m2 = M()
    s2 = Sum(outputs(REG_F, product(m2, d(REG_U), lam_slots(), M.f2)))
    next_line(m2)
    return [m1, s1, m2, s2]


def prog_add():
    m1 = M()
    s1 = Sum(lines(m1), 1)
    m2 = M()
    s2 = Sum(outputs(REG_F, product(m2, d(REG_F), lam_slots(), M.f2)))
    next_line(m2)
    return [m1, s1, m2, s2]


def prog_mul(out, x, y, conj_y=False, conj_out=False):
    """out = x y, x conj(y) or conj(x y); x, y: registers or {power: slots}."""
    m = M()
    x, y = (v if isinstance(v, dict) else d(v) for v in (x, y))
    co = product(m, x, y, M.f2_kar, lambda i, j: -1 if conj_y and j & 1 else 1)
    return [m, Sum(outputs(out, co, conj_out))]


def frob2(m, r, out):
    """x^(p^2): the products of register r's powers 1..5 with their factors into register out's slots (power 0 stays)."""
    for e in range(1, 6):
        for j in range(2):
            m.mul(reg(r)[e][j], NORM2 + e - 1, out=reg(out)[e][j])
    return {e: reg(r if e == 0 else out)[e] for e in range(6)}


def prog_frob2_mul(out, r, other, via):
    m = M()
    x = frob2(m, r, via)
    return [m] + prog_mul(out, x, other)


def prog_frob(out, r):
    """x^p: conj(x_e) gamma_e."""
    m = M()
    co = [({reg(r)[0][0]: 1}, {reg(r)[0][1]: -1})]
    for e in range(1, 6):
        g = (GAMMA + 2 * (e - 1), GAMMA + 2 * (e - 1) + 1)
        x = reg(r)[e]
        p = [[m.mul(x[i], g[j]) for j in range(2)] for i in range(2)]
        co.append(({p[0][0]: 1, p[1][1]: 1}, {p[0][1]: 1, p[1][0]: -1}))
    return [m, Sum(outputs(out, co))]


PROGRAMS = {
    "LINE": prog_line,
    "DBL": prog_dbl,
    "ADD": prog_add,
    "T_F_CU": lambda: prog_mul(REG_T, REG_F, REG_U, conj_y=True),
    "T_T2_T": lambda: prog_frob2_mul(REG_T, REG_T, REG_T, REG_U),
    "R_R_T": lambda: prog_mul(REG_R, REG_R, REG_T),
    "R_R_A": lambda: prog_mul(REG_R, REG_R, REG_A),
    "R_R_X": lambda: prog_mul(REG_R, REG_R, REG_X),
    "A_CRT": lambda: prog_mul(REG_A, REG_R, REG_T, conj_out=True),
    "A_CRA": lambda: prog_mul(REG_A, REG_R, REG_A, conj_out=True),
    "X_FROB_A": lambda: prog_frob(REG_X, REG_A),
    "A_X_CR": lambda: prog_mul(REG_A, REG_X, REG_R, conj_y=True),
    "R_A2_R": lambda: prog_frob2_mul(REG_R, REG_A, REG_R, REG_U),
    "R_R_CA": lambda: prog_mul(REG_R, REG_R, REG_A, conj_y=True),
}


def cyclo():
    """The cyclotomic squaring of register R: (products, outputs); an output is (slot, form A', post form) with value
    3 A' + post."""
    S = [(reg_slot(REG_R, k, 0), reg_slot(REG_R, k, 1)) for k in range(6)]
    m, outs = M(), []

    def put(k, forms, sign):  # 3 form + 2 sign S_k = 3 (form + sign S_k) - sign S_k
        for s, f in zip(S[k], forms):
            outs.append((s, add(f, {s: sign}), {s: -sign}))
    for g, (a, b) in enumerate(((0, 4), (3, 2), (1, 5))):
        x, y = S[a], S[b]
        x2, y2, xy = m.f2_sqr(x), m.f2_sqr(y), m.f2_twice(x, y)
        yx = xi(y2)
        put((0, 1, 2)[g], (add(yx[0], x2[0]), add(yx[1], x2[1])), -1)
        put((4, 5, 3)[g], xi(xy) if g == 2 else xy, 1)
    return m, outs


# ----------------------------------------------------------------------------- lanes
def split_terms(form, lanes):
    """Distributes a form over `lanes` lanes of two added and two subtracted slots each."""
    plus = [s for s, c in sorted(form.items()) for _ in range(c)]
    minus = [s for s, c in sorted(form.items()) for _ in range(-c)]
    assert len(plus) <= 2 * lanes and len(minus) <= 2 * lanes, (len(plus), len(minus), lanes)
    plus += [ZERO] * (2 * lanes - len(plus))
    minus += [ZERO] * (2 * lanes - len(minus))
    return [(plus[k], plus[k + lanes], minus[k], minus[k + lanes]) for k in range(lanes)]


T_M, T_S = 0, 1


def off(s):
    return NONE if s == NONE else 48 * s


def words(u):
    return [off(u[0]) | off(u[1]) << 16, off(u[2]) | off(u[3]) << 16, off(u[4]), u[5]]


def m_lane(e):
    """x: a | b << 16, y: a2 | b2 << 16, z: out, w: type | sums << 4 | dbl << 5."""
    out, a, b, dbl = e
    a, a2 = a if isinstance(a, tuple) else (a, ZERO)
    b, b2 = b if isinstance(b, tuple) else (b, ZERO)
    return [a, b, a2, b2, out, dbl << 5 | T_M]


def phase_rows(ph):
    if isinstance(ph, M):
        assert len(ph.ent) <= LANES, len(ph.ent)
        sums = any(isinstance(v, tuple) for e in ph.ent for v in e[1:3])
        rows = [m_lane(e) for e in ph.ent] + [[ZERO, ZERO, ZERO, ZERO, NONE, T_M]] * (LANES - len(ph.ent))
        return [r[:5] + [r[5] | sums << 4] for r in rows]
    rows = []
    for g, outs in ph.warps:
        w = []
        for s, f in outs:
            for k, t in enumerate(split_terms(f, 1 << g)):
                w.append([t[0], t[1], t[2], t[3], s if k == 0 else NONE, T_S | g << 4])
        rows += w + [[ZERO] * 4 + [NONE, T_S | g << 4]] * (32 - len(w))
    # a warp without outputs: g = 7
    return rows + [[ZERO] * 4 + [NONE, T_S | 7 << 4]] * (LANES - len(rows))


def cyclo_rows():
    """Two uint4 per lane of one warp: the M entry; the S terms p0 | p1 << 16, m0 | m1 << 16, out | post+ << 16,
    post- of the lane pair 2k, 2k + 1 (the post terms on the odd lane)."""
    m, outs = cyclo()
    assert len(m.ent) <= 32 and len(outs) == 12
    a = [words(m_lane(e)) for e in m.ent] + [words([ZERO, ZERO, ZERO, ZERO, NONE, T_M])] * (32 - len(m.ent))
    b = []
    for s, f, post in outs:
        pp = [x for x, c in post.items() if c > 0] or [ZERO]
        pm = [x for x, c in post.items() if c < 0] or [ZERO]
        for k, t in enumerate(split_terms(f, 2)):
            b.append([off(t[0]) | off(t[1]) << 16, off(t[2]) | off(t[3]) << 16,
                      off(s if k == 0 else NONE) | off(pp[0] if k else ZERO) << 16, off(pm[0] if k else ZERO)])
    b += [[off(ZERO) * 0x10001, off(ZERO) * 0x10001, NONE | off(ZERO) << 16, off(ZERO)]] * (32 - len(b))
    return a, b


# ----------------------------------------------------------------------------- device arithmetic on integers
R_INV = pow(1 << 384, -1, P)
QK = np.float32(256.0 / 436277739.0 * (1 - 2.0 ** -20))  # 436277739 = floor(p / 2^352) + 1


def mont(a, b):
    """The Montgomery product without its last conditional subtraction."""
    assert a < (1 << 384) - 3 * P and b < 1 << 384
    t = a * b
    return (t + (-t * pow(P, -1, 1 << 384) % (1 << 384)) * P) >> 384


def reduce13(v):
    assert 0 <= v < QMAX * P
    top = (v >> 360) & 0xFFFFFFFF
    assert v >> 392 == 0
    q = int(np.float32(np.float32(top) * QK))  # the device converts towards zero: never larger than this by rounding up
    if np.float32(top) > top:
        q = int(np.float32(np.nextafter(np.float32(top), np.float32(0)) * QK))
    r = v - q * P
    assert 0 <= r < 1.001 * P and q < QMAX, (q, r / P)
    return r


def lane_sum(s, t):
    r = 3 * P + s[t[0]] + s[t[1]] - s[t[2]] - s[t[3]]
    assert 0 < r < 6 * P
    return r


def run_phase(ph, s):
    res = {}
    if isinstance(ph, M):
        for out, a, b, dbl in ph.ent:
            va = sum(s[x] for x in a) if isinstance(a, tuple) else s[a]
            vb = sum(s[x] for x in b) if isinstance(b, tuple) else s[b]
            assert out not in res
            res[out] = mont(va, vb << dbl)
            assert res[out] < 1.42 * P
    else:
        for g, outs in ph.warps:
            for o, f in outs:
                assert o not in res
                res[o] = reduce13(sum(lane_sum(s, t) for t in split_terms(f, 1 << g)))
    s.update(res)


def run_cyclo(s):
    m, outs = cyclo()
    run_phase(m, s)
    res = {}
    for o, f, post in outs:
        v = sum(3 * lane_sum(s, t) for t in split_terms(f, 2)) + sum(c * s[x] for x, c in post.items())
        res[o] = reduce13(v)
    s.update(res)


def expected(name, s):
    F, T, A, X, R, U = (G.to_w(s, r) for r in range(6))
    frob = lambda x: G.wpow(x, P)
    conj, mul = G.wconj, G.wmul

    def line(p):
        b = LINE + 4 * p
        l = [(0, 0)] * 6
        l[0] = (s[b], s[b + 1])
        l[2] = (s[LB + 2 * p], s[LB + 2 * p + 1])
        l[3] = (s[PT + 2 * p + 1], 0)
        return l
    lam = mul(line(0), line(1))
    return {
        "DBL": (REG_F, lambda: mul(mul(F, F), lam)), "ADD": (REG_F, lambda: mul(F, lam)),
        "T_F_CU": (REG_T, lambda: mul(F, conj(U))), "T_T2_T": (REG_T, lambda: mul(frob(frob(T)), T)),
        "R_R_T": (REG_R, lambda: mul(R, T)), "R_R_A": (REG_R, lambda: mul(R, A)), "R_R_X": (REG_R, lambda: mul(R, X)),
        "A_CRT": (REG_A, lambda: conj(mul(R, T))), "A_CRA": (REG_A, lambda: conj(mul(R, A))),
        "X_FROB_A": (REG_X, lambda: frob(A)), "A_X_CR": (REG_A, lambda: mul(X, conj(R))),
        "R_A2_R": (REG_R, lambda: mul(frob(frob(A)), R)), "R_R_CA": (REG_R, lambda: mul(R, conj(A))),
        "CYCLO": (REG_R, lambda: mul(R, R)),
    }[name]


def norm2():
    """gamma_e conj(gamma_e), e = 1..5."""
    return [(g[0] * g[0] + g[1] * g[1]) % P for g in (G.gammas()[e] for e in range(1, 6))]


def to_mont(x, rng):
    """A device value of x: its Montgomery residue, sometimes not fully reduced."""
    r = (x << 384) % P
    return r + P if r < P // 2000 and rng.random() < 0.5 else r


def check(rng):
    for name in list(PROGRAMS) + ["CYCLO"]:
        for trial in range(2):
            v = G.random_slots(rng, cyclo_regs=(REG_R,) if name == "CYCLO" else ())
            v.update({LB + k: rng.randrange(P) for k in range(4)})
            v.update({NORM2 + k: x for k, x in enumerate(norm2())})
            if trial:  # extreme values
                for k in range(72):
                    if name != "CYCLO":
                        v[k] = rng.choice([0, 1, P - 1, P - 2, rng.randrange(P)])
            s = {k: to_mont(x, rng) for k, x in v.items()}
            s.update({k: rng.randrange(P) for k in range(TMP, TMP + LANES)})
            old = dict(s)
            if name == "CYCLO":
                run_cyclo(s)
            else:
                for ph in PROGRAMS[name]():
                    run_phase(ph, s)
            back = {k: x * R_INV % P for k, x in s.items()}
            if name == "LINE":
                ok = all(back[LB + 2 * p + c] == v[LINE + 4 * p + 2 + c] * v[PT + 2 * p] % P
                         for p in (0, 1) for c in (0, 1))
                assert ok
                continue
            r, want = expected(name, v)
            assert G.to_w(back, r) == want(), name
            if name in ("DBL", "ADD"):
                assert all(back[LB + 2 * p + c] == v[LINE + 4 * p + 2 + c] * v[PT + 2 * p] % P
                           for p in (0, 1) for c in (0, 1)), name
            keep = {REG_F, REG_T, REG_A, REG_X, REG_R} - {r}
            for q in keep:
                assert all(s[12 * q + k] == old[12 * q + k] for k in range(12)), (name, q)


# ----------------------------------------------------------------------------- emission
def rows_text(rows):
    return "  " + ", ".join("{0x%08x, 0x%08x, 0x%08x, 0x%08x}" % tuple(r) for r in rows) + ","


def emit():
    progs = {n: f() for n, f in PROGRAMS.items()}
    first, phases, note = [], [], []
    for n, p in progs.items():
        first.append(len(phases))
        phases += p
        note.append("// %-8s %s" % (n, " ".join("M(%d)" % len(x.ent) if isinstance(x, M) else
                                               "S(%d)" % sum(len(o) for _, o in x.warps) for x in p)))
    first.append(len(phases))
    m, outs = cyclo()
    note.append("// CYCLO    M(%d) S(%d)" % (len(m.ent), len(outs)))
    top = max([x.next for x in phases if isinstance(x, M)] + [m.next])
    lim = lambda x: ", ".join("0x%08xu" % ((x >> (32 * j)) & 0xFFFFFFFF) for j in range(12))
    L = ["// GENERATED by gen_pairing_quad.py -- do not edit by hand.",
         "// Phase tables of the four-warp pairing (see pairing_quad.cuh): products per M phase, outputs per S phase."]
    L += note
    L += ["#pragma once", "#include <stdint.h>", "",
          "#define PQ_LANES %d" % LANES, "#define PQ_NONE 0x%04x" % NONE, "#define PQ_SLOTS %d" % max(top, 270),
          "#define PQ_NORM2_BASE %d" % NORM2, "#define PQ_QMAX %d  // multiples of p" % QMAX,
          "enum {" + ", ".join("PQ_" + n for n in progs) + ", PQ_NPROG };",
          "__device__ const uint16_t PQ_FIRST[PQ_NPROG + 1] = {%s};" % ", ".join(map(str, first)),
          "// One uint4 per (phase, lane); slots as byte offsets.  M: a | b << 16, a2 | b2 << 16, out, sums << 4 | dbl << 5.",
          "// S: p0 | p1 << 16, m0 | m1 << 16, out, 1 | g << 4 (g = 7: a warp without outputs).",
          "__device__ const uint4 PQ_ENTRY[%d * PQ_LANES] = {" % len(phases)]
    for ph in phases:
        L.append(rows_text([words(r) for r in phase_rows(ph)]))
    L.append("};")
    a, b = cyclo_rows()
    L += ["// The cyclotomic squaring on one warp: M entries; S entries p0 | p1 << 16, m0 | m1 << 16, out | post+ << 16, post-.",
          "__device__ const uint4 PQ_CYCLO_M[32] = {", rows_text(a), "};",
          "__device__ const uint4 PQ_CYCLO_S[32] = {", rows_text(b), "};",
          "// gamma_e conj(gamma_e), e = 1..5, Montgomery form",
          "__device__ const fp PQ_NORM2[5] = {"] + ["  {{%s}}," % lim((x << 384) % P) for x in norm2()] + ["};"]
    return "\n".join(L) + "\n"


def main():
    check(random.Random(20260101))
    if "--check-only" not in sys.argv:
        out = pathlib.Path(__file__).resolve().parent / "pairing_quad_program.cuh"
        out.write_text(emit())
        print("wrote", out)


if __name__ == "__main__":
    main()
