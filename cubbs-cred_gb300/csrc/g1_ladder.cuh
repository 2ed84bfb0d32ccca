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

DEV uint32_t at(uint32_t slot) { return slot * (uint32_t)sizeof(fp); }

// One product per lane; PAIR: an output is the sum of two neighbouring lanes'.
template <bool PAIR> DEV void mul_round(Mem *m, fp *sl, const Mul &e, uint32_t b, uint32_t b2) {
  fp x = ld(sl, at(e.a)), y = ld(sl, at(b));
  if (!PAIR) {
    const fp x2 = ld(sl, at(e.a2)), y2 = ld(sl, at(b2));
    fp_acc_add(x.w, x.w, x2.w);
    fp_acc_add(y.w, y.w, y2.w);
  }
  fp t;
  fp_mont_mul(t.w, x.w, y.w);
  uint32_t v[13], r[12];
  scale(v, t.w, e.k);
  if (PAIR) add_lane(v, 1);
  reduce13(m->mul_p, v, r);
  __syncwarp();  // every lane has read its operands
  if (e.out != NONE) st(sl, at(e.out), r);
  __syncwarp();
}

// acc = op(acc, table entry): x, y, z are the slots of the entry's coordinates
// (ignored by a doubling).  All lanes of the warp call it.
static __device__ __noinline__ void apply(Mem *m, const Op *op, uint32_t x, uint32_t y, uint32_t z) {
  const int role = threadIdx.x & 7;
  fp *sl = m->slot[(threadIdx.x & 31) >> 3];
  auto pick = [&](uint32_t s) { return !(s & BY_TAB) ? s : s == (BY_TAB | 0) ? x : s == (BY_TAB | 1) ? y : z; };
  const Mul f = op->first[role], s = op->second[role];
  const Sum u = op->sum[role];
  mul_round<false>(m, sl, f, pick(f.b), pick(f.b2));
  const fp t = lane_sum(sl, at(u.p0), at(u.p1), at(u.m0), at(u.m1));
  if (u.out != NONE) st(sl, at(u.out), t.w);
  __syncwarp();
  mul_round<true>(m, sl, s, s.b, ZERO);
}
DEV void dbl(Mem *m) { apply(m, &DBL, ZERO, ZERO, ZERO); }
// acc += digit * P for digit in -8 .. 8 (entry |digit| - 1; 0 adds the identity)
DEV void add_digit(Mem *m, int digit) {
  const uint32_t e = TAB + 4 * (uint32_t)(abs(digit) - 1);
  apply(m, &ADD, digit ? e : ZERO, digit ? e + (digit < 0 ? 2 : 1) : ONE, digit ? e + 3 : ZERO);
}
// table entry k = acc
DEV void store_entry(fp *sl, int role, int k) {
  if (role < 4) {
    fp v = ld(sl, at(role == 0 ? AX : role == 3 ? AZ : AY));
    if (role == 2) {
      fp_csub1(v.w, v.w);
      fp_from_mod(v.w, v.w);
    }
    st(sl, at(TAB + 4 * k + role), v.w);
  }
  __syncwarp();
}

// The constants, ladder state and base point: acc = entry 0 = the image on E'
// of (x, y), or of phi(x, y) = (beta x, -y).  All lanes of the warp call it.
DEV void start(Mem *m, const g1a &p, bool phi) {
  const int lane = threadIdx.x & 31, role = lane & 7;
  fp *sl = m->slot[lane >> 3];
  for (int k = lane; k < QMAX; k += 32) m->mul_p[k] = multiple_of_p((uint32_t)k);
  const fp s2 = C_B3_S2, bs2 = C_B3_BETA_S2, s3 = C_B3_S3;
  if (role == 0) sl[ZERO] = fp_zero();
  if (role == 1) sl[ONE] = fp_one();
  if (role == 2) sl[AX] = p.x;
  if (role == 3) sl[AY] = phi ? fp_neg(p.y) : p.y;
  if (role == 4) sl[AZ] = fp_one();
  if (role == 5) sl[E0] = phi ? bs2 : s2;
  if (role == 6) sl[E1] = s3;
  __syncwarp();
  const Mul e = {(uint8_t)(role ? AY : AX), ZERO, (uint8_t)(role ? E1 : E0), ZERO,
                 (uint8_t)(role == 0 ? AX : role == 1 ? AY : NONE), 1};
  mul_round<false>(m, sl, e, e.b, ZERO);
  store_entry(sl, role, 0);
}

// k P for four ladders: half 0 or 1 of a GLV term on each (sh: the half's 128-bit
// scalar).  Returns with the multiple in the accumulator.
DEV void ladder128(Mem *m, const uint32_t sh[4]) {
  const int lane = threadIdx.x & 31, role = lane & 7;
  fp *sl = m->slot[lane >> 3];
#pragma unroll 1
  for (int k = 1; k < 8; k++) {  // entries 2P .. 8P
    if (k == 1) dbl(m);
    else add_digit(m, 1);
    store_entry(sl, role, k);
  }
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
  if (role == 0) sl[AX] = fp_zero();
  if (role == 1) sl[AY] = fp_one();
  if (role == 2) sl[AZ] = fp_zero();
  __syncwarp();
  add_digit(m, (int)d[4]);
#pragma unroll 1
  for (int i = 31; i >= 0; i--) {
#pragma unroll 1
    for (int k = 0; k < 4; k++) dbl(m);
    add_digit(m, (int)(d[3] >> 28) - 8);
    d[3] = __funnelshift_l(d[2], d[3], 4);
    d[2] = __funnelshift_l(d[1], d[2], 4);
    d[1] = __funnelshift_l(d[0], d[1], 4);
    d[0] <<= 4;
  }
}

// acc = [|z|] acc, entry 0 being acc at the start
DEV void mul_zabs(Mem *m) {
#pragma unroll 1
  for (int i = 62; i >= 0; i--) {
    dbl(m);
    if (zabs_bit(i)) add_digit(m, 1);
  }
}

}  // namespace gl
