"""Generate field_ptx.cuh: Montgomery multiplication and modular add/sub for
the BLS12-381 base field (12 x 32-bit limbs) and scalar field (8 x 32-bit
limbs) as inline-PTX carry chains (mad.lo.cc / madc.hi.cc / addc / subc).

Run:  python gen_field_ptx.py   (rewrites field_ptx.cuh beside this file)

The product in use is gen_mont's: rows of 64-bit multiply-adds on an even and
an odd carry chain (gen_mont_sqr: the square).  The rows of operand-scanning
CIOS are kept for the tests: for each limb b_i of the second operand, one asm
block adds lo(a*b_i) and hi(a*b_i), computes the Montgomery quotient
m = t0 * (-p^-1 mod 2^32), and adds lo(m*p) and hi(m*p).  Each block keeps its
carry flag local, so no condition code crosses asm statements.  The modulus
words are embedded as immediates.  Intermediate values stay below 2^(32n+32).
"""
import pathlib

P = int("1a0111ea397fe69a4b1ba7b6434bacd764774b84f38512bf6730d2a0f6b0f6241eabfffeb153ffffb9feffffffffaaab", 16)
R = int("73eda753299d7d483339d80809a1d80553bda402fffe5bfeffffffff00000001", 16)


def limbs(x, n):
    return [(x >> (32 * i)) & 0xFFFFFFFF for i in range(n)]


def gen_field(name, mod, n, cios):
    ml = limbs(mod, n)
    pinv = (-pow(mod, -1, 1 << 32)) % (1 << 32)
    Rm = (1 << (32 * n)) % mod
    R2 = (Rm * Rm) % mod
    out = []
    w = out.append
    w(f"// ---- {name}: {n} x 32-bit limbs, modulus 0x{mod:x}")
    w(f"#define {name.upper()}_NLIMBS {n}")
    w(f"__device__ __constant__ static const uint32_t {name.upper()}_MOD[{n}] = {{{', '.join(f'0x{x:08x}u' for x in ml)}}};")
    w(f"static const uint32_t {name.upper()}_MOD_H[{n}] = {{{', '.join(f'0x{x:08x}u' for x in ml)}}};")
    w(f"static const uint32_t {name.upper()}_ONE_H[{n}] = {{{', '.join(f'0x{x:08x}u' for x in limbs(Rm, n))}}};")
    w(f"static const uint32_t {name.upper()}_R2_H[{n}] = {{{', '.join(f'0x{x:08x}u' for x in limbs(R2, n))}}};")
    w(f"#define {name.upper()}_PINV 0x{pinv:08x}u")
    w(f"#define {name.upper()}_MOD_INIT {{{{{', '.join(f'0x{x:08x}u' for x in ml)}}}}}")
    w(f"#define {name.upper()}_ONE_INIT {{{{{', '.join(f'0x{x:08x}u' for x in limbs(Rm, n))}}}}}")
    w(f"#define {name.upper()}_R2_INIT {{{{{', '.join(f'0x{x:08x}u' for x in limbs(R2, n))}}}}}")
    w("")
    # ---- one CIOS row: t[0..n] (n+1 words, t[n] == 0 on entry) += a*b ; += m*mod ; t[0] becomes 0.
    regs_t = [f"%{i}" for i in range(n + 1)]
    regs_a = [f"%{n + 1 + i}" for i in range(n)]
    reg_b = f"%{2 * n + 1}"
    body = []
    body.append("{ .reg .u32 m;")
    # pass A: lo(a*b)
    body.append(f"mad.lo.cc.u32 {regs_t[0]}, {regs_a[0]}, {reg_b}, {regs_t[0]};")
    for j in range(1, n):
        body.append(f"madc.lo.cc.u32 {regs_t[j]}, {regs_a[j]}, {reg_b}, {regs_t[j]};")
    body.append(f"addc.u32 {regs_t[n]}, 0, 0;")
    # pass B: hi(a*b) into t[1..n]
    body.append(f"mad.hi.cc.u32 {regs_t[1]}, {regs_a[0]}, {reg_b}, {regs_t[1]};")
    for j in range(1, n - 1):
        body.append(f"madc.hi.cc.u32 {regs_t[j + 1]}, {regs_a[j]}, {reg_b}, {regs_t[j + 1]};")
    body.append(f"madc.hi.u32 {regs_t[n]}, {regs_a[n - 1]}, {reg_b}, {regs_t[n]};")
    # quotient
    body.append(f"mul.lo.u32 m, {regs_t[0]}, 0x{pinv:08x};")
    # pass C: lo(m*mod)
    body.append(f"mad.lo.cc.u32 {regs_t[0]}, m, 0x{ml[0]:08x}, {regs_t[0]};")
    for j in range(1, n):
        body.append(f"madc.lo.cc.u32 {regs_t[j]}, m, 0x{ml[j]:08x}, {regs_t[j]};")
    body.append(f"addc.u32 {regs_t[n]}, {regs_t[n]}, 0;")
    # pass D: hi(m*mod) into t[1..n]
    body.append(f"mad.hi.cc.u32 {regs_t[1]}, m, 0x{ml[0]:08x}, {regs_t[1]};")
    for j in range(1, n - 1):
        body.append(f"madc.hi.cc.u32 {regs_t[j + 1]}, m, 0x{ml[j]:08x}, {regs_t[j + 1]};")
    body.append(f"madc.hi.u32 {regs_t[n]}, m, 0x{ml[n - 1]:08x}, {regs_t[n]};")
    body.append("}")
    asm_text = "\\n\\t".join(body)
    if cios:
        w(f"// t[0..{n}] += a*b + m*mod with m = t0*pinv; afterwards t0 == 0 and the value is t[1..{n}].")
        w(f"__device__ __forceinline__ void {name}_cios_row(uint32_t *t, const uint32_t *a, uint32_t b) {{")
        outs = ", ".join(f'"+&r"(t[{i}])' for i in range(n + 1))
        ins = ", ".join(f'"r"(a[{i}])' for i in range(n)) + ', "r"(b)'
        w(f'  asm volatile("{asm_text}" : {outs} : {ins});')
        w("}")
        w("")
    # ---- conditional subtract: r = t >= mod ? t - mod : t  (t < 2*mod)
    body = []
    body.append("{ .reg .u32 d<%d>; .reg .u32 bw; .reg .pred ge;" % n)
    body.append(f"sub.cc.u32 d0, %{n}, 0x{ml[0]:08x};")
    for j in range(1, n):
        body.append(f"subc.cc.u32 d{j}, %{n + j}, 0x{ml[j]:08x};")
    body.append("subc.u32 bw, 0, 0;")
    body.append("setp.eq.u32 ge, bw, 0;")
    for j in range(n):
        body.append(f"selp.u32 %{j}, d{j}, %{n + j}, ge;")
    body.append("}")
    asm_text = "\\n\\t".join(body)
    w(f"__device__ __forceinline__ void {name}_reduce_once(uint32_t *r, const uint32_t *t) {{")
    outs = ", ".join(f'"=&r"(r[{i}])' for i in range(n))
    ins = ", ".join(f'"r"(t[{i}])' for i in range(n))
    w(f'  asm("{asm_text}" : {outs} : {ins});')
    w("}")
    w("")
    # ---- add: r = a + b mod (a,b < mod; sum < 2^(32n) as mod < 2^(32n-1))
    body = []
    body.append("{ .reg .u32 s<%d>; .reg .u32 d<%d>; .reg .u32 bw; .reg .pred ge;" % (n, n))
    body.append(f"add.cc.u32 s0, %{n}, %{2 * n};")
    for j in range(1, n):
        body.append(f"addc.cc.u32 s{j}, %{n + j}, %{2 * n + j};")
    body.append(f"sub.cc.u32 d0, s0, 0x{ml[0]:08x};")
    for j in range(1, n):
        body.append(f"subc.cc.u32 d{j}, s{j}, 0x{ml[j]:08x};")
    body.append("subc.u32 bw, 0, 0;")
    body.append("setp.eq.u32 ge, bw, 0;")
    for j in range(n):
        body.append(f"selp.u32 %{j}, d{j}, s{j}, ge;")
    body.append("}")
    asm_text = "\\n\\t".join(body)
    w(f"__device__ __forceinline__ void {name}_add_raw(uint32_t *r, const uint32_t *a, const uint32_t *b) {{")
    outs = ", ".join(f'"=&r"(r[{i}])' for i in range(n))
    ins = ", ".join(f'"r"(a[{i}])' for i in range(n)) + ", " + ", ".join(f'"r"(b[{i}])' for i in range(n))
    w(f'  asm("{asm_text}" : {outs} : {ins});')
    w("}")
    w("")
    # ---- sub: r = a - b mod
    body = []
    body.append("{ .reg .u32 s<%d>; .reg .u32 bw;" % n)
    body.append(f"sub.cc.u32 s0, %{n}, %{2 * n};")
    for j in range(1, n):
        body.append(f"subc.cc.u32 s{j}, %{n + j}, %{2 * n + j};")
    body.append("subc.u32 bw, 0, 0;")
    # add (mod & bw)
    body.append("{ .reg .u32 k;")
    body.append(f"and.b32 k, bw, 0x{ml[0]:08x};")
    body.append("add.cc.u32 %0, s0, k;")
    for j in range(1, n):
        body.append(f"and.b32 k, bw, 0x{ml[j]:08x};")
        cc = ".cc" if j < n - 1 else ""
        body.append(f"addc{cc}.u32 %{j}, s{j}, k;")
    body.append("}}")
    asm_text = "\\n\\t".join(body)
    w(f"__device__ __forceinline__ void {name}_sub_raw(uint32_t *r, const uint32_t *a, const uint32_t *b) {{")
    w(f'  asm("{asm_text}" : {outs} : {ins});')
    w("}")
    w("")
    return "\n".join(out)


def gen_lazy(name, mod, n):
    """Unreduced sums for short signed sums of reduced values (at most 6 terms
    of [0, mod], so every partial sum stays below 6 mod < 2^(32n)):
    {name}_acc_add / _acc_sub (plain add and subtract; _x: of n + 1 words),
    {name}_acc_add_3mod (a + 3 mod), {name}_from_mod (mod - a) and {name}_csub{k}
    (subtract k*mod when the value is at least k*mod, k = 4, 2, 1), which bring
    a value below 8 mod back to [0, mod)."""
    assert 6 * mod < 1 << (32 * n)
    out = []
    w = out.append
    outs = ", ".join(f'"=&r"(r[{i}])' for i in range(n))
    ins2 = ", ".join(f'"r"(a[{i}])' for i in range(n)) + ", " + ", ".join(f'"r"(b[{i}])' for i in range(n))
    ins1 = ", ".join(f'"r"(a[{i}])' for i in range(n))
    body = [f"add.cc.u32 %0, %{n}, %{2 * n};"]
    for j in range(1, n):
        body.append(f"add{'c.cc' if j < n - 1 else 'c'}.u32 %{j}, %{n + j}, %{2 * n + j};")
    w(f"__device__ __forceinline__ void {name}_acc_add(uint32_t *r, const uint32_t *a, const uint32_t *b) {{")
    w(f'  asm("' + "\\n\\t".join(body) + f'" : {outs} : {ins2});')
    w("}")
    ml = limbs(mod, n)
    body = [f"sub.cc.u32 %0, %{n}, %{2 * n};"]
    for j in range(1, n):
        body.append(f"sub{'c.cc' if j < n - 1 else 'c'}.u32 %{j}, %{n + j}, %{2 * n + j};")
    w(f"__device__ __forceinline__ void {name}_acc_sub(uint32_t *r, const uint32_t *a, const uint32_t *b) {{")
    w(f'  asm("' + "\\n\\t".join(body) + f'" : {outs} : {ins2});')
    w("}")
    m3 = limbs(3 * mod, n)
    body = [f"add.cc.u32 %0, %{n}, 0x{m3[0]:08x};"]
    for j in range(1, n):
        body.append(f"add{'c.cc' if j < n - 1 else 'c'}.u32 %{j}, %{n + j}, 0x{m3[j]:08x};")
    w(f"__device__ __forceinline__ void {name}_acc_add_3mod(uint32_t *r, const uint32_t *a) {{")
    w(f'  asm("' + "\\n\\t".join(body) + f'" : {outs} : {ins1});')
    w("}")
    # sums of n + 1 words
    k = n + 1
    for nm, op in (("acc_add_x", "add"), ("acc_sub_x", "sub")):
        body = [f"{op}.cc.u32 %0, %{k}, %{2 * k};"]
        for j in range(1, k):
            body.append(f"{op}{'c.cc' if j < k - 1 else 'c'}.u32 %{j}, %{k + j}, %{2 * k + j};")
        outx = ", ".join(f'"=&r"(r[{i}])' for i in range(k))
        insx = ", ".join(f'"r"({v}[{i}])' for v in "ab" for i in range(k))
        w(f"__device__ __forceinline__ void {name}_{nm}(uint32_t *r, const uint32_t *a, const uint32_t *b) {{")
        w(f'  asm("' + "\\n\\t".join(body) + f'" : {outx} : {insx});')
        w("}")
    body = [f"sub.cc.u32 %0, 0x{ml[0]:08x}, %{n};"]
    for j in range(1, n):
        body.append(f"sub{'c.cc' if j < n - 1 else 'c'}.u32 %{j}, 0x{ml[j]:08x}, %{n + j};")
    w(f"__device__ __forceinline__ void {name}_from_mod(uint32_t *r, const uint32_t *a) {{")
    w(f'  asm("' + "\\n\\t".join(body) + f'" : {outs} : {ins1});')
    w("}")
    for k in (4, 2, 1):
        kl = limbs(k * mod, n)
        body = ["{ .reg .u32 d<%d>; .reg .u32 bw; .reg .pred ge;" % n, f"sub.cc.u32 d0, %{n}, 0x{kl[0]:08x};"]
        for j in range(1, n):
            body.append(f"subc.cc.u32 d{j}, %{n + j}, 0x{kl[j]:08x};")
        body.append("subc.u32 bw, 0, 0;")
        body.append("setp.eq.u32 ge, bw, 0;")
        for j in range(n):
            body.append(f"selp.u32 %{j}, d{j}, %{n + j}, ge;")
        body.append("}")
        w(f"__device__ __forceinline__ void {name}_csub{k}(uint32_t *r, const uint32_t *a) {{")
        w(f'  asm("' + "\\n\\t".join(body) + f'" : {outs} : {ins1});')
        w("}")
    w("")
    return "\n".join(out)


def asm_fn(name, n, body, operands):
    """An inline function `name`(r, operand arrays...) around one asm block; %0..%{n-1} are r."""
    outs = ", ".join(f'"=&r"(r[{i}])' for i in range(n))
    ins = ", ".join(f'"r"({v}[{i}])' for v in operands for i in range(n))
    args = ", ".join(f"const uint32_t *{v}" for v in operands)
    text = "\\n\\t".join(body)
    return (f"__device__ __forceinline__ void {name}(uint32_t *r, {args}) {{\n"
            f'  asm("{text}" : {outs} : {ins});\n}}\n')


def wide_chain(lines, acc, xs, y, first_carry=False, carry_out=True, fresh=False, fresh_top=False):
    """acc (2 len(xs) words) += sum_k xs[k] y 2^(64 k), one carry chain of 64-bit multiply-adds.
    first_carry: the chain starts from the carry flag; carry_out: it ends in it; fresh: acc is written, not added to
    (no carries at all); fresh_top: the top pair of acc counts as zero."""
    for k, x in enumerate(xs):
        lo, hi = acc[2 * k], acc[2 * k + 1]
        if fresh:
            lines.append(f"mul.lo.u32 {lo}, {x}, {y};")
            lines.append(f"mul.hi.u32 {hi}, {x}, {y};")
            continue
        c = "c" if k or first_carry else ""
        cc = ".cc" if carry_out or k < len(xs) - 1 else ""
        zero = fresh_top and k == len(xs) - 1
        lines.append(f"mad{c}.lo.cc.u32 {lo}, {x}, {y}, {'0' if zero else lo};")
        lines.append(f"madc.hi{cc}.u32 {hi}, {x}, {y}, {'0' if zero else hi};")


def gen_mont(name, mod, n):
    """{name}_mont_mul(r, a, b) = a b / 2^(32n) mod mod up to one mod too large.

    The running sum is kept in two arrays of n words: E at limbs 0..n-1 holds the products of even limb distance, O
    at limbs 1..n those of odd distance, so a row b_i adds its n products as two carry chains of n/2 64-bit
    multiply-adds whose words line up in pairs.  Then m = E_0 (-mod^-1), a row m mod in the same way, and E_0 is
    zero.  Dropping that limb turns O into the next E and E's words 2.. into the next O; the word E_1 left over is
    added to the next E_0 and its carry enters the next row's O chain.
    Bounds: the sum before a shift is below 2^32 (a + mod + the sum before), so operands with
    a < 2^(32n) - 3 mod never carry out of limb n, and the result is below mod + a b / 2^(32n)."""
    assert n % 2 == 0
    ml = limbs(mod, n)
    pinv = (-pow(mod, -1, 1 << 32)) % (1 << 32)
    odd = [f"0x{ml[j]:08x}" for j in range(1, n, 2)]
    even = [f"0x{ml[j]:08x}" for j in range(0, n, 2)]

    body = [f"{{ .reg .u32 x<{n}>; .reg .u32 y<{n}>; .reg .u32 m;"]
    a, b = [f"%{n + j}" for j in range(n)], [f"%{2 * n + j}" for j in range(n)]
    E, O = [f"x{j}" for j in range(n)], [f"y{j}" for j in range(n)]
    for i in range(n):
        if i == 0:
            wide_chain(body, O, a[1::2], b[i], fresh=True)
            wide_chain(body, E, a[0::2], b[i], fresh=True)
        else:
            body.append(f"add.cc.u32 {E[0]}, {E[0]}, {left};")
            wide_chain(body, O, a[1::2], b[i], first_carry=True, carry_out=False, fresh_top=True)
            wide_chain(body, E, a[0::2], b[i])
            body.append(f"addc.u32 {O[n - 1]}, {O[n - 1]}, 0;")
        body.append(f"mul.lo.u32 m, {E[0]}, 0x{pinv:08x};")
        wide_chain(body, O, odd, "m", carry_out=False)
        wide_chain(body, E, even, "m")
        body.append(f"addc.u32 {O[n - 1]}, {O[n - 1]}, 0;")
        left = E[1]
        E, O = O, E[2:] + E[:2]  # the two top words of the new O count as zero (fresh_top)
    body.append(f"add.cc.u32 %0, {E[0]}, {left};")
    for j in range(1, n):
        body.append(f"addc{'.cc' if j < n - 1 else ''}.u32 %{j}, {E[j]}, {O[j - 1] if j < n - 1 else '0'};")
    body.append("}")
    return (f"// r = a b / 2^{32 * n} mod p, up to one p too large (interleaved Montgomery rows on even / odd carry "
            f"chains).\n" + asm_fn(f"{name}_mont_mul", n, body, "ab"))


def gen_mont_sqr(name, mod, n):
    """{name}_mont_sqr(r, a) = a^2 / 2^(32n) mod mod up to one mod too large: the n(n-1)/2 cross products in an even
    (t) and an odd (u) array of carry chains, doubled by shifts, the n squares added in one chain, then n reduction
    rows on the low words as in {name}_mont_mul and the high words added at the end (222 multiply-adds for n = 12
    instead of 288)."""
    ml = limbs(mod, n)
    pinv = (-pow(mod, -1, 1 << 32)) % (1 << 32)
    odd = [f"0x{ml[j]:08x}" for j in range(1, n, 2)]
    even = [f"0x{ml[j]:08x}" for j in range(0, n, 2)]
    a = [f"%{n + j}" for j in range(n)]
    L = [f"{{ .reg .u32 t<{2 * n}>; .reg .u32 u<{2 * n}>; .reg .u32 m;"]
    live = {"t": set(), "u": set()}
    for i in range(n - 1):
        for par, R in ((0, "t"), (1, "u")):
            chain = False
            js = [j for j in range(i + 1, n) if (i + j) % 2 == par]
            for j in js:
                k = i + j
                if k in live[R]:
                    L.append(f"mad{'c' if chain else ''}.lo.cc.u32 {R}{k}, {a[i]}, {a[j]}, {R}{k};")
                    L.append(f"madc.hi.cc.u32 {R}{k + 1}, {a[i]}, {a[j]}, {R}{k + 1};")
                    chain = True
                elif chain:  # a fresh pair takes the chain's carry and cannot overflow
                    L.append(f"madc.lo.cc.u32 {R}{k}, {a[i]}, {a[j]}, 0;")
                    L.append(f"madc.hi.u32 {R}{k + 1}, {a[i]}, {a[j]}, 0;")
                    chain = False
                else:
                    L.append(f"mul.lo.u32 {R}{k}, {a[i]}, {a[j]};")
                    L.append(f"mul.hi.u32 {R}{k + 1}, {a[i]}, {a[j]};")
                live[R] |= {k, k + 1}
            if chain:  # the carry past the last pair: a word that holds nothing but such carries
                k = i + js[-1] + 2
                if k in live[R]:
                    L.append(f"addc.u32 {R}{k}, {R}{k}, 0;")
                else:
                    L.append(f"addc.u32 {R}{k}, 0, 0;")
                    live[R].add(k)
                    if k + 1 < 2 * n:
                        L.append(f"mov.u32 {R}{k + 1}, 0;")
                        live[R].add(k + 1)
    for k in range(1, 2 * n):  # t = t + u
        x, y = (f"{R}{k}" if k in live[R] else "0" for R in "tu")
        L.append(f"add{'c' if k > 1 else ''}{'.cc' if k < 2 * n - 1 else ''}.u32 t{k}, {x}, {y};")
    L.append("shf.l.clamp.b32 u1, 0, t1, 1;")  # u = 2 t
    for k in range(2, 2 * n):
        L.append(f"shf.l.clamp.b32 u{k}, t{k - 1}, t{k}, 1;")
    L.append(f"mul.lo.u32 t0, {a[0]}, {a[0]};")  # t = u + the squares
    L.append(f"mad.hi.cc.u32 t1, {a[0]}, {a[0]}, u1;")
    for j in range(1, n):
        L.append(f"madc.lo.cc.u32 t{2 * j}, {a[j]}, {a[j]}, u{2 * j};")
        L.append(f"madc.hi{'.cc' if j < n - 1 else ''}.u32 t{2 * j + 1}, {a[j]}, {a[j]}, u{2 * j + 1};")
    E, O = [f"t{j}" for j in range(n)], [f"u{j}" for j in range(n)]
    for i in range(n):
        L.append(f"mul.lo.u32 m, {E[0]}, 0x{pinv:08x};")
        wide_chain(L, O, odd, "m", first_carry=i > 0, carry_out=False, fresh=i == 0, fresh_top=True)
        wide_chain(L, E, even, "m")
        L.append(f"addc.u32 {O[n - 1]}, {O[n - 1]}, 0;")
        left = E[1]
        E, O = O, E[2:] + E[:2]
        L.append(f"add.cc.u32 {E[0]}, {E[0]}, {left};")  # its carry enters the next O chain
    for j in range(1, n):
        L.append(f"addc{'.cc' if j < n - 1 else ''}.u32 {E[j]}, {E[j]}, {O[j - 1] if j < n - 1 else '0'};")
    L.append(f"add.cc.u32 %0, {E[0]}, t{n};")
    for j in range(1, n):
        L.append(f"addc{'.cc' if j < n - 1 else ''}.u32 %{j}, {E[j]}, t{n + j};")
    L.append("}")
    return (f"// r = a^2 / 2^{32 * n} mod p, up to one p too large.\n" + asm_fn(f"{name}_mont_sqr", n, L, "a"))


def main():
    text = [
        "// GENERATED by gen_field_ptx.py -- do not edit by hand.",
        "// Inline-PTX carry chains for BLS12-381 Fp (12 limbs) and Fr (8 limbs).",
        "#pragma once",
        "#include <stdint.h>",
        "",
        gen_field("fp", P, 12, cios=True),
        gen_lazy("fp", P, 12),
        gen_mont("fp", P, 12),
        gen_mont_sqr("fp", P, 12),
        gen_field("fr", R, 8, cios=False),
        gen_mont("fr", R, 8),
    ]
    dst = pathlib.Path(__file__).with_name("field_ptx.cuh")
    dst.write_text("\n".join(text) + "\n")
    print("wrote", dst)


if __name__ == "__main__":
    main()
