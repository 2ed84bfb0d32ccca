// G1 scalar multiplication and the G1 membership test for launches too small to
// fill the GPU: a ladder runs on eight lanes (four ladders a warp) with its
// state in shared-memory slots.
//
// What bounds it: a lone warp's product (1730 cycles of multiply-adds,
// field.cuh) times the depth of the chain.  The point formulas are the
// complete addition law for curves with a = 0 (J. Renes, C. Costello, L.
// Batina, "Complete addition formulas for prime order elliptic curves",
// EUROCRYPT 2016, algorithms 7 and 9) in homogeneous coordinates: two products
// deep for a doubling (five and four products) and for an addition (seven and
// six), against three and four for XYZZ coordinates on a lane quad.  They hold
// for every pair of points of E(Fp) (its order is odd), so no lane ever
// branches, and a zero digit adds the identity.  The ladder runs on the
// isomorphic curve E': y^2 = x^3 + 2/3, where the constant 3b of the formulas
// is 2.
//
// A round: lane `role` multiplies two slots (or sums of two), scales the
// product by a small constant, adds its neighbour's where an output is a sum
// of two products, reduces by a multiple of p and stores.  Between the two
// rounds of an operation one sum per lane forms the factors of the second.
// Operands stay in slots, so nothing is kept in registers across a product:
// the quad formulas held four coordinates and eight products there, and
// spilling them around each out-of-line product made a round of 1900 cycles
// cost 4500.
#pragma once
#include "curve.cuh"
#include "fp_bipartite.cuh"
#include "slots.cuh"

namespace gl {

using namespace slots;

enum : uint32_t {
  ZERO = 0, AX, AY, AZ,          // accumulator
  P0, P1, P2, P3, P4, P5, P6, P7,  // products of the first round
  E0, E1, E2, E3, E4, E5,        // sums
  TAB,                           // entry k: X, Y, -Y, Z of (k + 1) P
  ONE = TAB + 32,
  NSLOT                          // odd: neighbouring ladders' slots fall on different banks
};
static_assert(NSLOT % 2 == 1, "bank spread");
constexpr uint32_t NONE = 0xff, BY_TAB = 0x80;  // BY_TAB | c: coordinate c of the chosen table entry
constexpr int LADDERS = 4;

struct Mem {
  fp slot[LADDERS][NSLOT];
  fp mul_p[QMAX];
};

// An operation: first-round products (a + a2)(b + b2) k -> out; sums p0 + p1 -
// m0 - m1 -> out; second-round products a b k, added in neighbouring pairs -> out.
struct alignas(8) Mul { uint8_t a, a2, b, b2, out, k; };  // one 8-byte load
struct alignas(8) Sum { uint8_t p0, p1, m0, m1, out; };
struct Op { Mul first[8]; Sum sum[8]; Mul second[8]; };
#define GL_IDLE_M {ZERO, ZERO, ZERO, ZERO, NONE, 1}
#define GL_IDLE_S {ZERO, ZERO, ZERO, ZERO, NONE}
// 2 (X, Y, Z): t0 = Y^2, w = 2 Z^2; X' = 2 (t0 - 3w) XY, Y' = (t0 - 3w)(t0 + w) + 8 t0 w, Z' = 8 t0 YZ
__device__ const Op DBL = {
    {{AY, ZERO, AY, ZERO, P0, 1}, {AY, ZERO, AZ, ZERO, P1, 1}, {AX, ZERO, AY, ZERO, P2, 1}, {AZ, ZERO, AZ, ZERO, P3, 2},
     {AZ, ZERO, AZ, ZERO, P4, 6}, GL_IDLE_M, GL_IDLE_M, GL_IDLE_M},
    {{P0, ZERO, P4, ZERO, E0}, {P0, P3, ZERO, ZERO, E1}, GL_IDLE_S, GL_IDLE_S, GL_IDLE_S, GL_IDLE_S, GL_IDLE_S, GL_IDLE_S},
    {{E0, ZERO, P2, ZERO, AX, 2}, GL_IDLE_M, {E0, ZERO, E1, ZERO, AY, 1}, {P0, ZERO, P3, ZERO, NONE, 8},
     {P0, ZERO, P1, ZERO, AZ, 8}, GL_IDLE_M, GL_IDLE_M, GL_IDLE_M}};
// (X1, Y1, Z1) + (X2, Y2, Z2): t3 = X1Y2 + X2Y1, t4 = Y1Z2 + Y2Z1, ty = X1Z2 + X2Z1, f1, f2 = Y1Y2 -+ 2 Z1Z2;
// X' = t3 f1 - 2 t4 ty, Y' = f2 f1 + 6 X1X2 ty, Z' = t4 f2 + 3 X1X2 t3
__device__ const Op ADD = {
    {{AX, ZERO, BY_TAB | 0, ZERO, P0, 1}, {AY, ZERO, BY_TAB | 1, ZERO, P1, 1}, {AZ, ZERO, BY_TAB | 3, ZERO, P2, 1},
     {AZ, ZERO, BY_TAB | 3, ZERO, P3, 2}, {AX, AY, BY_TAB | 0, BY_TAB | 1, P4, 1},
     {AY, AZ, BY_TAB | 1, BY_TAB | 3, P5, 1}, {AX, AZ, BY_TAB | 0, BY_TAB | 3, P6, 1}, GL_IDLE_M},
    {{P4, ZERO, P0, P1, E0}, {P1, P2, P5, ZERO, E1}, {P5, ZERO, P1, P2, E2}, {P6, ZERO, P0, P2, E3},
     {P1, ZERO, P3, ZERO, E4}, {P1, P3, ZERO, ZERO, E5}, GL_IDLE_S, GL_IDLE_S},
    {{E0, ZERO, E4, ZERO, AX, 1}, {E1, ZERO, E3, ZERO, NONE, 2}, {E5, ZERO, E4, ZERO, AY, 1}, {P0, ZERO, E3, ZERO, NONE, 6},
     {E2, ZERO, E5, ZERO, AZ, 1}, {P0, ZERO, E0, ZERO, NONE, 3}, GL_IDLE_M, GL_IDLE_M}};

// The addition on y^2 = x^3 + 4 itself (3b = 12), for sums of points given as
// projective triples (add_points).
__device__ const Op ADD4 = {
    {{AX, ZERO, BY_TAB | 0, ZERO, P0, 1}, {AY, ZERO, BY_TAB | 1, ZERO, P1, 1}, {AZ, ZERO, BY_TAB | 3, ZERO, P2, 1},
     {AZ, ZERO, BY_TAB | 3, ZERO, P3, 12}, {AX, AY, BY_TAB | 0, BY_TAB | 1, P4, 1},
     {AY, AZ, BY_TAB | 1, BY_TAB | 3, P5, 1}, {AX, AZ, BY_TAB | 0, BY_TAB | 3, P6, 1}, GL_IDLE_M},
    {{P4, ZERO, P0, P1, E0}, {P1, P2, P5, ZERO, E1}, {P5, ZERO, P1, P2, E2}, {P6, ZERO, P0, P2, E3},
     {P1, ZERO, P3, ZERO, E4}, {P1, P3, ZERO, ZERO, E5}, GL_IDLE_S, GL_IDLE_S},
    {{E0, ZERO, E4, ZERO, AX, 1}, {E1, ZERO, E3, ZERO, NONE, 12}, {E5, ZERO, E4, ZERO, AY, 1},
     {P0, ZERO, E3, ZERO, NONE, 36}, {E2, ZERO, E5, ZERO, AZ, 1}, {P0, ZERO, E0, ZERO, NONE, 3}, GL_IDLE_M, GL_IDLE_M}};

DEV uint32_t at(uint32_t slot) { return slot * (uint32_t)sizeof(fp); }

// One lane's part of an operation, as slot addresses (k: the constants; a
// negative out: nothing stored).
struct Role {
  uint32_t a, a2, b, b2, k1, p0, p1, m0, m1, c, d, k2;
  int32_t out1, sum, out2;
};
// acc, x, y, z: addresses of the accumulator's X and of the operand's
// coordinates; tmp: that of ZERO .. E5.
DEV Role role_of(const Op &op, uint32_t acc, uint32_t x, uint32_t y, uint32_t z, uint32_t tmp) {
  auto where = [&](uint32_t s) {
    return s & BY_TAB ? (s == (BY_TAB | 0) ? x : s == (BY_TAB | 1) ? y : z)
                      : s - AX < 3u ? acc + at(s - AX) : tmp + at(s);
  };
  auto to = [&](uint32_t s) { return s == NONE ? -1 : (int32_t)where(s); };
  const int r = threadIdx.x & 7;
  const Mul f = op.first[r], g = op.second[r];
  const Sum u = op.sum[r];
  return {where(f.a), where(f.a2), where(f.b), where(f.b2), f.k, where(u.p0), where(u.p1), where(u.m0), where(u.m1),
          where(g.a), where(g.b), g.k, to(f.out), to(u.out), to(g.out)};
}
// Where a lane's first-round operands b, b2 come from in an addition: 0 a fixed
// slot, 1, 2, 3 the operand's X, Y, Z.
struct Operand {
  uint32_t b, b2;
  DEV static uint32_t code(uint32_t s) { return !(s & BY_TAB) ? 0 : s == (BY_TAB | 0) ? 1 : s == (BY_TAB | 1) ? 2 : 3; }
  DEV static Operand of(const Op &op) {
    const Mul f = op.first[threadIdx.x & 7];
    return {code(f.b), code(f.b2)};
  }
  DEV void set(Role &r, uint32_t x, uint32_t y, uint32_t z) const {
    if (b) r.b = b == 1 ? x : b == 2 ? y : z;
    if (b2) r.b2 = b2 == 1 ? x : b2 == 2 ? y : z;
  }
};

// The second warp's halves of the products where two warps share a launch's
// ladders (HALVES): both compute half of each product (fp_bipartite.cuh), the
// first does the rest.  Slots then hold x 2^256 instead of x 2^384 (mod p).
struct Halves {
  uint4 v[3][32];
  uint32_t top[32];
};
DEV void pair_sync() { asm volatile("bar.sync 1, 64;" ::: "memory"); }
// t = x y on the first warp
DEV void halved(uint32_t halves, bool second, const fp &x, const fp &y, fp &t) {
  uint32_t m[13];
  const uint32_t at_v = halves + 16 * (threadIdx.x & 31), at_top = halves + 3 * 32 * 16 + 4 * (threadIdx.x & 31);
  if (second) {
    fp_bp_mul_hi(m, x.w, y.w);
#pragma unroll
    for (int k = 0; k < 3; k++)
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at_v + 512 * k), "r"(m[4 * k]), "r"(m[4 * k + 1]),
                   "r"(m[4 * k + 2]), "r"(m[4 * k + 3])
                   : "memory");
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(at_top), "r"(m[12]) : "memory");
  } else {
    fp_bp_mul_lo(m, x.w, y.w);
  }
  __syncwarp();
  pair_sync();
  if (!second) {
    uint32_t o[13];
#pragma unroll
    for (int k = 0; k < 3; k++)
      asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(o[4 * k]), "=r"(o[4 * k + 1]), "=r"(o[4 * k + 2]), "=r"(o[4 * k + 3])
                   : "r"(at_v + 512 * k)
                   : "memory");
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(o[12]) : "r"(at_top) : "memory");
    fp_bp_finish(t.w, m, o);
  }
}

// The operation on the slots of `r`; octets with `live` false compute and store
// nothing.  All lanes of the warp (of both warps, with HALVES) call it.
template <bool HALVES = false> DEV void apply(const Role &r, uint32_t mul_p, bool live, uint32_t halves = 0) {
  const bool second = HALVES && threadIdx.x >= 32;
  uint32_t v[13], w[12];
  if constexpr (HALVES) {
    __syncwarp();
    pair_sync();  // the first warp has written the operands
  }
  {
    fp x = ld(r.a), y = ld(r.b);
    const fp x2 = ld(r.a2), y2 = ld(r.b2);
    fp_acc_add(x.w, x.w, x2.w);
    fp_acc_add(y.w, y.w, y2.w);
    fp t;
    if constexpr (HALVES) halved(halves, second, x, y, t);
    else fp_mont_mul(t.w, x.w, y.w);
    if (!second) {
      scale(v, t.w, r.k1);
      reduce13(mul_p, v, w);
      __syncwarp();  // every lane has read its operands
      if (live && r.out1 >= 0) st((uint32_t)r.out1, w);
      __syncwarp();
    }
  }
  if (!second) {
    const fp t = lane_sum(r.p0, r.p1, r.m0, r.m1);
    if (live && r.sum >= 0) st((uint32_t)r.sum, t.w);
    __syncwarp();
  }
  if constexpr (HALVES) pair_sync();  // and the second round's
  {
    const fp x = ld(r.c), y = ld(r.d);
    fp t;
    if constexpr (HALVES) halved(halves, second, x, y, t);
    else fp_mont_mul(t.w, x.w, y.w);
    if (!second) {
      scale(v, t.w, r.k2);
      add_lane(v, 1);
      reduce13(mul_p, v, w);
      __syncwarp();
      if (live && r.out2 >= 0) st((uint32_t)r.out2, w);
      __syncwarp();
    }
  }
}

// table entry k = acc
DEV void store_entry(fp *sl, int role, int k) {
  if (role < 4) {
    fp v = sl[role == 0 ? AX : role == 3 ? AZ : AY];
    if (role == 2) {
      fp_csub1(v.w, v.w);
      fp_from_mod(v.w, v.w);
    }
    sl[TAB + 4 * k + role] = v;
  }
  __syncwarp();
}

// A warp's four ladders: the lanes' parts of a doubling and of an addition.
// With HALVES a second warp runs the same code for its half of the products;
// only the first (`first`) writes slots.
template <bool HALVES> struct LaddersOf {
  Role dbl, add;
  Operand operand;
  uint32_t tab, mul_p;  // addresses of table entry 0 and of the multiples of p
  fp *sl;
  int role;
  uint32_t halves;
  bool first;
  // acc *= 2, or acc += digit * P for digit in -8 .. 8 (entry |digit| - 1; 0
  // adds the identity).  One copy in the code: the loops select the operation.
  DEV void step(bool doubling, int digit) const {
    Role r = add;
    const uint32_t e = tab + at(4 * (uint32_t)(abs(digit) - 1)), zero = tab - at(TAB);
    operand.set(r, digit ? e : zero, digit ? e + at(digit < 0 ? 2 : 1) : tab + at(ONE - TAB), digit ? e + at(3) : zero);
    if (doubling) r = dbl;
    apply<HALVES>(r, mul_p, true, halves);
  }
  // table entry k = acc
  DEV void entry(int k) const {
    if (first) store_entry(sl, role, k);
  }
};
using Ladders = LaddersOf<false>;

// The constants, ladder state and base point: acc = entry 0 = the image on E'
// of (x, y), or of phi(x, y) = (beta x, -y).  All lanes of the warp (of both
// warps, with HALVES, where h is room for the halves) call it.
template <bool HALVES = false> DEV LaddersOf<HALVES> start(Mem *m, const g1a &p, bool phi, Halves *h = nullptr) {
  const int lane = threadIdx.x & 31, role = lane & 7;
  fp *sl = m->slot[lane >> 3];
  LaddersOf<HALVES> l;
  l.first = !HALVES || threadIdx.x < 32;
  l.halves = HALVES ? addr(h) : 0;
  if (l.first) {
    for (int k = lane; k < QMAX; k += 32) m->mul_p[k] = multiple_of_p((uint32_t)k);
    const fp form = C_FP_BP_IN;  // 2^256: a Montgomery product with it leaves x 2^256
    if (role == 0) {
      const fp s2 = C_B3_S2, bs2 = C_B3_BETA_S2;
      fp x = fp_mul(p.x, phi ? bs2 : s2);
      sl[AX] = HALVES ? fp_mul(x, form) : x;
      sl[ZERO] = fp_zero();
    } else if (role == 1) {
      const fp s3 = C_B3_S3;
      fp y = fp_mul(phi ? fp_neg(p.y) : p.y, s3);
      sl[AY] = HALVES ? fp_mul(y, form) : y;
      sl[ONE] = HALVES ? form : fp_one();
    } else if (role == 2) {
      sl[AZ] = HALVES ? form : fp_one();
    }
    __syncwarp();
    store_entry(sl, role, 0);
  }
  const uint32_t a = addr(sl);
  l.dbl = role_of(DBL, a + at(AX), a, a, a, a);
  l.add = role_of(ADD, a + at(AX), a, a, a, a);
  l.operand = Operand::of(ADD);
  l.tab = a + at(TAB);
  l.mul_p = addr(m->mul_p);
  l.sl = sl;
  l.role = role;
  return l;
}

// acc = k P on each of the four ladders (sh: k's 128-bit half of a GLV term),
// then acc += the point that `join` has stored as entry 0.
template <bool HALVES, class Join>
DEV void ladder128(const LaddersOf<HALVES> &l, const uint32_t sh[4], const Join &join) {
  // signed digits: nibbles of sh + 0x888...8, less 8
  uint32_t d[5];
  uint64_t c = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    c += (uint64_t)sh[k] + 0x88888888u;
    d[k] = (uint32_t)c;
    c >>= 32;
  }
  d[4] = (uint32_t)c;
  // steps 0..6: entries 2P .. 8P; 7: the top digit into the identity; then 32
  // times four doublings and a digit; last: the join
  constexpr int BUILD = 7, MAIN = BUILD + 1, END = MAIN + 5 * 32;
  int quint = 0;
#pragma unroll 1
  for (int i = 0; i <= END; i++) {
    bool doubling = i == 0;
    int digit = 1;
    if (i == BUILD) {
      digit = (int)d[4];
      if (l.first && l.role == 0) l.sl[AX] = fp_zero();
      if (l.first && l.role == 1) l.sl[AY] = l.sl[ONE];
      if (l.first && l.role == 2) l.sl[AZ] = fp_zero();
      __syncwarp();
    } else if (i == END) {
      if (l.first) join();
      __syncwarp();
    } else if (i >= MAIN) {
      doubling = quint < 4;
      digit = (int)(d[3] >> 28) - 8;
      quint = doubling ? quint + 1 : 0;
      if (!doubling) {
        d[3] = __funnelshift_l(d[2], d[3], 4);
        d[2] = __funnelshift_l(d[1], d[2], 4);
        d[1] = __funnelshift_l(d[0], d[1], 4);
        d[0] <<= 4;
      }
    }
    l.step(doubling, digit);
    if (i < BUILD) l.entry(i + 1);
  }
}

// acc = [z^2] acc for acc = entry 0 = P; entry 1 is P afterwards.
DEV void mul_z2(const Ladders &l) {
#pragma unroll 1
  for (int half = 0; half < 2; half++) {
    bool add = false;
#pragma unroll 1
    for (int i = 62; i >= 0;) {
      l.step(!add, 1);
      add = !add && zabs_bit(i);
      if (!add) i--;
    }
    if (half) break;
    store_entry(l.sl, l.role, 1);
    if (l.role < 4) {  // swap entries 0 and 1: the second half multiplies [|z|]P
      const fp t = l.sl[TAB + l.role];
      l.sl[TAB + l.role] = l.sl[TAB + 4 + l.role];
      l.sl[TAB + 4 + l.role] = t;
    }
    __syncwarp();
  }
}

// The accumulator, taken back from E' as an XYZZ point, by the ladder's lanes
// 0 and 1: (X Z, s^2 Z^2) and (Y Z^2, s^3 Z^3).
template <bool HALVES = false> DEV void leave(const fp *sl, int role, fp v[2]) {
  const fp s2 = C_B3_S2, s3 = C_B3_S3, form = C_FP_BP_OUT;
  fp z = sl[AZ], xy = sl[AX + role];
  if (HALVES) {  // to x 2^384
    z = fp_mul(z, form);
    xy = fp_mul(xy, form);
  }
  fp zz = z;
  if (role == 1) zz = fp_mul(z, z);
  v[0] = fp_mul(xy, zz);
  v[1] = fp_mul(fp_mul(zz, z), role ? s3 : s2);
}

// ---- sums of many points
// Projective triples (X, Y, Z) in shared memory, added in place by the lane
// octets of a warp: a level of a tree sum is one complete addition of two
// products' depth for up to four pairs, where every lane adding its neighbour's
// XYZZ point (g1_add and shuffles) is fourteen products deep for half of the
// lanes.
constexpr uint32_t TRIPLE = 3 * (uint32_t)sizeof(fp);       // an odd number of 16-byte units
constexpr uint32_t TMP_SLOTS = 19;                          // ZERO .. E5, one more to keep it odd
constexpr uint32_t TMP_BYTES = TMP_SLOTS * (uint32_t)sizeof(fp);

DEV void put_triple(fp *t, const g1 &p) {
  const bool inf = g1_is_inf(p);
  t[0] = fp_mul(p.X, p.ZZZ);
  t[1] = inf ? fp_one() : fp_mul(p.Y, p.ZZ);
  t[2] = fp_mul(p.ZZ, p.ZZZ);
}
// Per warp: the octets' scratch (TMP_BYTES each from `tmp`, zero slots set) and
// their parts of an addition.
struct Adder {
  Role add;
  Operand operand;
  uint32_t mul_p;
  bool acc_a, acc_a2, acc_out;  // which of the lane's slots lie in the accumulator
  DEV static Adder on(uint32_t tmp, uint32_t mul_p, const Op &op = ADD4) {
    const uint32_t oct = (threadIdx.x & 31) >> 3, t = tmp + oct * TMP_BYTES;
    const Mul f = op.first[threadIdx.x & 7], g = op.second[threadIdx.x & 7];
    return {role_of(op, 0, 0, 0, 0, t), Operand::of(op), mul_p, f.a - AX < 3u, f.a2 - AX < 3u, g.out != NONE};
  }
  // For e < count: the triple (e / d) stride + e % d (in steps of `step` bytes
  // from base) takes the one d further on.  One warp, all lanes.
  DEV void level(uint32_t base, uint32_t count, uint32_t d, uint32_t stride, uint32_t step) const {
    const uint32_t oct = (threadIdx.x & 31) >> 3;
#pragma unroll 1
    for (uint32_t e0 = 0; e0 < count; e0 += 4) {
      const uint32_t e = min(e0 + oct, count - 1), acc = base + ((e / d) * stride + e % d) * step, op = acc + d * step;
      Role r = add;
      if (acc_a) r.a += acc;
      if (acc_a2) r.a2 += acc;
      if (acc_out) r.out2 += acc;
      operand.set(r, op, op + at(1), op + at(2));
      apply(r, mul_p, e0 + oct < count);
    }
  }
};
// The triple at t as an XYZZ point, written by the octet's lanes 0..2.
DEV void get_triple(const fp *t, int role, g1 *out) {
  if (role > 2) return;
  const fp z = t[2];
  const fp zz = fp_mul(z, role == 0 ? t[0] : z);  // X Z, or Z^2
  if (role == 0) {
    out->X = zz;
  } else {
    const fp c = fp_mul(zz, role == 1 ? t[1] : z);  // Y Z^2, or Z^3
    if (role == 1) {
      out->Y = c;
    } else {
      out->ZZ = zz;
      out->ZZZ = c;
    }
  }
}

}  // namespace gl
