// Fp values in shared-memory slots: the vector loads, small signed sums and
// reductions that the four-warp pairing (pairing_quad.cuh) and the G1 ladders
// (g1_ladder.cuh) share.  Between rounds a slot holds a value below 1.42 p
// (products) or 1.001 p (reduced sums).
#pragma once
#include "field.cuh"

namespace slots {

constexpr int QMAX = 72;  // multiples of p in the table of reduce13

DEV fp ld(const fp *sl, uint32_t off) {  // off in bytes
  const uint4 *p = reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(sl) + off);
  const uint4 a = p[0], b = p[1], c = p[2];
  return {{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w}};
}
DEV void st(fp *sl, uint32_t off, const uint32_t *w) {
  uint4 *p = reinterpret_cast<uint4 *>(reinterpret_cast<uint8_t *>(sl) + off);
  p[0] = make_uint4(w[0], w[1], w[2], w[3]);
  p[1] = make_uint4(w[4], w[5], w[6], w[7]);
  p[2] = make_uint4(w[8], w[9], w[10], w[11]);
}

// k p for the table of reduce13
DEV fp multiple_of_p(uint32_t k) {
  const fp pm = FP_MOD_INIT;
  fp r;
  uint64_t c = 0;
#pragma unroll
  for (int j = 0; j < 12; j++) {
    c += (uint64_t)pm.w[j] * k;
    r.w[j] = (uint32_t)c;
    c >>= 32;
  }
  return r;
}

// 3p + slot[p0] + slot[p1] - slot[m0] - slot[m1], in (0, 6p)
DEV fp lane_sum(const fp *sl, uint32_t p0, uint32_t p1, uint32_t m0, uint32_t m1) {
  const fp a = ld(sl, p0), b = ld(sl, p1), c = ld(sl, m0), d = ld(sl, m1);
  fp t;
  fp_acc_add_3mod(t.w, a.w);
  fp_acc_add(t.w, t.w, b.w);
  fp_acc_sub(t.w, t.w, c.w);
  fp_acc_sub(t.w, t.w, d.w);
  return t;
}

// The 13-word value v < QMAX p brought below 1.001 p: the quotient from its top
// 32 bits (bits 360..391) in single precision, a little low so that it never
// exceeds v / p, and that multiple of p taken off.
DEV void reduce13(const fp *mul_p, const uint32_t *v, uint32_t *r) {
  constexpr float K = (float)(256.0 / 436277739.0 * (1.0 - 1.0 / 1048576.0));  // 436277739 = floor(p / 2^352) + 1
  const uint32_t q = (uint32_t)(__uint2float_rz(__funnelshift_l(v[11], v[12], 24)) * K);
  const fp m = ld(mul_p, q * (uint32_t)sizeof(fp));
  fp_acc_sub(r, v, m.w);
}

// v += v of the lane whose number differs by d (every lane of the warp calls it)
DEV void add_lane(uint32_t *v, int d) {
  uint32_t o[13];
#pragma unroll
  for (int j = 0; j < 13; j++) o[j] = __shfl_xor_sync(0xffffffffu, v[j], d);
  fp_acc_add_x(v, v, o);
}

// v = k a, 13 words (k < 2^8)
DEV void scale(uint32_t *v, const uint32_t *a, uint32_t k) {
  uint64_t c = 0;
#pragma unroll
  for (int j = 0; j < 12; j++) {
    c += (uint64_t)a[j] * k;
    v[j] = (uint32_t)c;
    c >>= 32;
  }
  v[12] = (uint32_t)c;
}

}  // namespace slots
