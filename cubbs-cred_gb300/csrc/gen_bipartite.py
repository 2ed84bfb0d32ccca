"""Generate fp_bipartite.cuh: a product mod p split over two warps.

bp(a, b) = a b / 2^256 mod p.  With a = a0 + a1 2^192 and b likewise, the product
divided by 2^192 is

    a0 b0 / 2^192  +  a0 b1 + a1 b0  +  a1 b1 2^192      (mod p)

The first warp takes a0 b0 through six Montgomery rows and adds a0 b1; the
second folds the high half of a1 b1 onto 2^(384 + 32 i) mod p, which needs no
quotient digits, and adds its low half and a1 b0 (M. Kaihara and N. Takagi,
"Bipartite modular multiplication method", IEEE Trans. Computers 57(2), 2008,
with a table fold for the upper part).  The two sums, below 2^416 together, are
exchanged and added, and two more Montgomery rows bring them below p + 2^352.
Each warp has 168 multiply-adds in its chain where the product on one lane has
288; a square 135 against 222.  Operands may be any 384-bit values.

Run:  python gen_bipartite.py   (rewrites fp_bipartite.cuh beside this file)
"""
import pathlib

from gen_field_ptx import P, limbs

PL = limbs(P, 12)
PINV = (-pow(P, -1, 1 << 32)) % (1 << 32)


class Asm:
    """Lines of one asm block; registers r0, r1, .. are allocated, operands are %n."""

    def __init__(self):
        self.lines, self.n = [], 0

    def regs(self, k):
        out = [f"r{self.n + j}" for j in range(k)]
        self.n += k
        return out

    def __call__(self, s):
        self.lines.append(s + ";")

    def fresh(self, acc, xs, y):
        for k, x in enumerate(xs):
            self(f"mul.lo.u32 {acc[2 * k]}, {x}, {y}")
            self(f"mul.hi.u32 {acc[2 * k + 1]}, {x}, {y}")

    def chain(self, acc, xs, y, carry_in=False, carry_out=True, zero_top=False):
        """acc += sum_k xs[k] y 2^(64 k) on one carry chain; zero_top: the top pair of acc counts as zero."""
        for k, x in enumerate(xs):
            c = "c" if k or carry_in else ""
            last = k == len(xs) - 1
            lo, hi = acc[2 * k], acc[2 * k + 1]
            z = zero_top and last
            self(f"mad{c}.lo.cc.u32 {lo}, {x}, {y}, {'0' if z else lo}")
            self(f"madc.hi{'.cc' if carry_out or not last else ''}.u32 {hi}, {x}, {y}, {'0' if z else hi}")

    def add(self, out, a, b):
        """out = a + b (equal lengths; None counts as zero), no carry out."""
        n = len(out)
        for j in range(n):
            x, y = a[j] or "0", b[j] or "0"
            self(f"add{'c' if j else ''}{'.cc' if j < n - 1 else ''}.u32 {out[j]}, {x}, {y}")

    def mul6(self, x, y):
        """12 words of x y, six limbs each: rows on an even and an odd chain, merged at the end."""
        n = 6
        lo, E, O = [], self.regs(n), self.regs(n)
        left = None
        for i in range(len(y)):
            if i == 0:
                self.fresh(O, x[1::2], y[i])
                self.fresh(E, x[0::2], y[i])
            else:
                self(f"add.cc.u32 {E[0]}, {E[0]}, {left}")
                self.chain(O, x[1::2], y[i], carry_in=True, carry_out=False, zero_top=True)
                self.chain(E, x[0::2], y[i])
                self(f"addc.u32 {O[n - 1]}, {O[n - 1]}, 0")
            r = self.regs(1)[0]
            self(f"mov.u32 {r}, {E[0]}")  # limb i is done
            lo.append(r)
            left = E[1]
            E, O = O, E[2:] + E[:2]
        hi = self.regs(n)
        self.add(hi, E, [left] + O[:n - 2] + [None])
        # (words n-2, n-1 of O are stale: the shift left them empty)
        return lo + hi

    def merge(self, E, O, left):
        """Words of E + O 2^32 + left after a shift of twelve-limb rows (no carry past word 11)."""
        out = self.regs(12)
        self(f"add.cc.u32 {out[0]}, {E[0]}, {left}")
        for j in range(1, 12):
            self(f"addc{'.cc' if j < 11 else ''}.u32 {out[j]}, {E[j]}, {O[j - 1] if j < 11 else '0'}")
        return out

    def rows(self, E, count, top=None):
        """`count` Montgomery rows on the words E (12; top: a word at limb 12); the 12 words of the quotient."""
        odd, even = [f"0x{v:08x}" for v in PL[1::2]], [f"0x{v:08x}" for v in PL[0::2]]
        O = self.regs(12)
        E = list(E)
        m = self.regs(1)[0]
        left = None
        for i in range(count):
            if i:
                self(f"add.cc.u32 {E[0]}, {E[0]}, {left}")
                # the carry must reach O's chain past the multiply, which leaves the flag alone
            self(f"mul.lo.u32 {m}, {E[0]}, 0x{PINV:08x}")
            if i == 0:
                self.fresh(O, odd, m)
                if top:
                    self(f"add.u32 {O[11]}, {O[11]}, {top}")
            else:
                self.chain(O, odd, m, carry_in=True, carry_out=False, zero_top=True)
            self.chain(E, even, m)
            self(f"addc.u32 {O[11]}, {O[11]}, 0")
            left = E[1]
            E, O = O, E[2:] + E[:2]
        return self.merge(E, O, left)

    def sqr6(self, x):
        """12 words of x^2."""
        n = 6
        t, u = self.regs(2 * n), self.regs(2 * n)
        live = {0: set(), 1: set()}
        acc = {0: t, 1: u}
        for i in range(n - 1):
            for par in (0, 1):
                R, L = acc[par], live[par]
                on = False
                js = [j for j in range(i + 1, n) if (i + j) % 2 == par]
                for j in js:
                    k = i + j
                    if k in L:
                        self(f"mad{'c' if on else ''}.lo.cc.u32 {R[k]}, {x[i]}, {x[j]}, {R[k]}")
                        self(f"madc.hi.cc.u32 {R[k + 1]}, {x[i]}, {x[j]}, {R[k + 1]}")
                        on = True
                    elif on:
                        self(f"madc.lo.cc.u32 {R[k]}, {x[i]}, {x[j]}, 0")
                        self(f"madc.hi.u32 {R[k + 1]}, {x[i]}, {x[j]}, 0")
                        on = False
                    else:
                        self(f"mul.lo.u32 {R[k]}, {x[i]}, {x[j]}")
                        self(f"mul.hi.u32 {R[k + 1]}, {x[i]}, {x[j]}")
                    L |= {k, k + 1}
                if on:
                    k = i + js[-1] + 2
                    if k in L:
                        self(f"addc.u32 {R[k]}, {R[k]}, 0")
                    else:
                        self(f"addc.u32 {R[k]}, 0, 0")
                        L.add(k)
                        if k + 1 < 2 * n:
                            self(f"mov.u32 {R[k + 1]}, 0")
                            L.add(k + 1)
        for k in range(1, 2 * n):
            a, b = (acc[p][k] if k in live[p] else "0" for p in (0, 1))
            self(f"add{'c' if k > 1 else ''}{'.cc' if k < 2 * n - 1 else ''}.u32 {t[k]}, {a}, {b}")
        self(f"shf.l.clamp.b32 {u[1]}, 0, {t[1]}, 1")
        for k in range(2, 2 * n):
            self(f"shf.l.clamp.b32 {u[k]}, {t[k - 1]}, {t[k]}, 1")
        self(f"mul.lo.u32 {t[0]}, {x[0]}, {x[0]}")
        self(f"mad.hi.cc.u32 {t[1]}, {x[0]}, {x[0]}, {u[1]}")
        for j in range(1, n):
            self(f"madc.lo.cc.u32 {t[2 * j]}, {x[j]}, {x[j]}, {u[2 * j]}")
            self(f"madc.hi{'.cc' if j < n - 1 else ''}.u32 {t[2 * j + 1]}, {x[j]}, {x[j]}, {u[2 * j + 1]}")
        return t

    def twice(self, w):
        """2 w, one word longer."""
        o = self.regs(len(w) + 1)
        self(f"shf.l.clamp.b32 {o[0]}, 0, {w[0]}, 1")
        for k in range(1, len(w)):
            self(f"shf.l.clamp.b32 {o[k]}, {w[k - 1]}, {w[k]}, 1")
        self(f"shf.l.clamp.b32 {o[-1]}, {w[-1]}, 0, 1")
        return o

    def fold(self, h):
        """13 words of sum_i h_i (2^(384 + 32 i) mod p)."""
        E, O = self.regs(12), self.regs(12)
        for i, y in enumerate(h):
            c = limbs((1 << (384 + 32 * i)) % P, 12)
            odd, even = [f"0x{v:08x}" for v in c[1::2]], [f"0x{v:08x}" for v in c[0::2]]
            if i == 0:
                self.fresh(O, odd, y)
                self.fresh(E, even, y)
            else:
                self.chain(O, odd, y, carry_out=False)
                self.chain(E, even, y)
                self(f"addc.u32 {O[11]}, {O[11]}, 0")
        out = self.regs(13)
        self(f"mov.u32 {out[0]}, {E[0]}")
        self.add(out[1:], E[1:] + [None], O)
        return out

    def text(self, n_out, n_in):
        body = "\\n\\t".join([f"{{ .reg .u32 r<{self.n}>;"] + self.lines + ["}"])
        return body


def fn(name, n_out, operands, build):
    """operands: [(name, words)]."""
    asm = Asm()
    at, ops = n_out, {}
    for v, k in operands:
        ops[v] = [f"%{at + j}" for j in range(k)]
        at += k
    res = build(asm, **ops)
    for j in range(n_out):
        asm(f"mov.u32 %{j}, {res[j]}")
    outs = ", ".join(f'"=&r"(o[{j}])' for j in range(n_out))
    ins = ", ".join(f'"r"({v}[{j}])' for v, k in operands for j in range(k))
    args = ", ".join(f"const uint32_t *{v}" for v, _ in operands)
    return (f"__device__ __forceinline__ void {name}(uint32_t *o, {args}) {{\n"
            f'  asm("{asm.text(n_out, at - n_out)}" : {outs} : {ins});\n}}\n')


def mul_lo(s, a, b):
    """First warp: (a0 b0 + m p) / 2^192 + a0 b1."""
    u = s.rows(s.mul6(a[:6], b[:6]), 6)
    x = s.mul6(a[:6], b[6:])
    out = s.regs(13)
    s.add(out, u + [None], x + [None])
    return out


def mul_hi(s, a, b):
    """Second warp: fold(high half of a1 b1) + its low half 2^192 + a1 b0."""
    p = s.mul6(a[6:], b[6:])
    f = s.fold(p[6:])
    x = s.mul6(a[6:], b[:6])
    t, out = s.regs(13), s.regs(13)
    s.add(t, f, [None] * 6 + p[:6] + [None])
    s.add(out, t, x + [None])
    return out


def sqr_lo(s, a):
    u = s.rows(s.sqr6(a[:6]), 6)
    x = s.twice(s.mul6(a[6:], a[:3]))  # 9 words, doubled
    out = s.regs(13)
    s.add(out, u + [None], x + [None] * (13 - len(x)))
    return out


def sqr_hi(s, a):
    p = s.sqr6(a[6:])
    f = s.fold(p[6:])
    x = s.twice(s.mul6(a[6:], a[3:6]))
    t, out = s.regs(13), s.regs(13)
    s.add(t, f, [None] * 6 + p[:6] + [None])
    s.add(out, t, [None] * 3 + x)
    return out


def finish(s, x, y):
    """(x + y + m p) / 2^64 for 13-word x, y."""
    t = s.regs(13)
    s.add(t, x, y)
    return s.rows(t[:12], 2, top=t[12])


FUNCTIONS = [
    ("fp_bp_mul_lo", 13, [("a", 12), ("b", 12)], mul_lo, "(a0 b0 + m p) / 2^192 + a0 b1"),
    ("fp_bp_mul_hi", 13, [("a", 12), ("b", 12)], mul_hi, "a1 b1 2^192 with its high half folded mod p, + a1 b0"),
    ("fp_bp_sqr_lo", 13, [("a", 12)], sqr_lo, "(a0^2 + m p) / 2^192 + 2 a1 (limbs 0..2 of a0)"),
    ("fp_bp_sqr_hi", 13, [("a", 12)], sqr_hi, "a1^2 2^192 with its high half folded mod p, + 2 a1 (limbs 3..5 of a0)"),
    ("fp_bp_finish", 12, [("x", 13), ("y", 13)], finish, "(x + y + m p) / 2^64, below p + 2^352"),
]


def sqrt_steps(width=4):
    """(p + 1) / 4 as sliding windows: [squarings, then the odd power to multiply by (0: a, 1: a^3, ..; none: 255)]; the
    first entry's power is the starting value."""
    bits = bin((P + 1) // 4)[2:]
    steps, i, run = [], 0, 0
    while i < len(bits):
        if bits[i] == "0":
            run, i = run + 1, i + 1
            continue
        j = min(i + width, len(bits))
        while bits[j - 1] == "0":
            j -= 1
        steps.append((run + j - i if steps else 0, int(bits[i:j], 2) >> 1))
        run, i = 0, j
    if run:
        steps.append((run, 255))
    e = 0  # check
    for k, (sq, idx) in enumerate(steps):
        e = (e << sq) + (2 * idx + 1 if idx != 255 else 0)
    assert e == (P + 1) // 4
    return steps


def main():
    out = ["// GENERATED by gen_bipartite.py -- do not edit by hand.",
           "// a b / 2^256 mod p split over two warps: each computes one of the lo / hi sums, and fp_bp_finish of both is",
           "// the product.", "#pragma once", "#include <stdint.h>", ""]
    for name, n, ops, build, what in FUNCTIONS:
        out += [f"// {what}", fn(name, n, ops, build)]
    steps = sqrt_steps()
    out += ["// The exponent (p + 1) / 4 in sliding windows: squarings, then the odd power a^(2 k + 1) to multiply by (255: none).",
            "#define FP_SQRT_STEPS %d" % len(steps), "#define FP_SQRT_POWERS %d" % (1 + max(k for _, k in steps if k != 255)),
            "__device__ const uint8_t FP_SQRT_STEP[FP_SQRT_STEPS][2] = {" +
            ", ".join("{%d, %d}" % x for x in steps) + "};",
            "#define C_FP_BP_IN {{%s}}   // 2^256 mod p: to the form x 2^256 from Montgomery form" %
            ", ".join("0x%08xu" % v for v in limbs((1 << 256) % P, 12)),
            "#define C_FP_BP_OUT {{%s}}  // 2^512 mod p: back" %
            ", ".join("0x%08xu" % v for v in limbs((1 << 512) % P, 12)), ""]
    path = pathlib.Path(__file__).with_name("fp_bipartite.cuh")
    path.write_text("\n".join(out))
    print("wrote", path)


if __name__ == "__main__":
    main()
