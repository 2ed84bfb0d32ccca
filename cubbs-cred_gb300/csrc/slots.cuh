// Fp values in shared-memory slots: the vector loads, small signed sums and
// reductions that the four-warp pairing (pairing_quad.cuh) and the G1 ladders
// (g1_ladder.cuh) share.  Between rounds a slot holds a value below 1.42 p
// (products of the pairing) or 1.001 p (reduced sums); the ladders also keep
// unreduced sums of four slots there (lane_sum, below 5.01 p) and multiply those,
// up to 53.7 p of the QMAX p that reduce13 takes.
#pragma once
#include "field.cuh"

namespace slots {

constexpr int QMAX = 72;  // multiples of p in the table of reduce13

// Slots are addressed by their 32-bit shared-memory addresses: a pointer that
// crosses an out-of-line call would be a generic one.
DEV uint32_t addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
DEV fp ld(uint32_t a) {
  fp r;
#pragma unroll
  for (int k = 0; k < 3; k++)
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.w[4 * k]), "=r"(r.w[4 * k + 1]), "=r"(r.w[4 * k + 2]), "=r"(r.w[4 * k + 3])
                 : "r"(a + 16 * k)
                 : "memory");
  return r;
}
DEV void st(uint32_t a, const uint32_t *w) {
#pragma unroll
  for (int k = 0; k < 3; k++)
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a + 16 * k), "r"(w[4 * k]), "r"(w[4 * k + 1]),
                 "r"(w[4 * k + 2]), "r"(w[4 * k + 3])
                 : "memory");
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

// 3p + [p0] + [p1] - [m0] - [m1], in (0, 6p)
DEV fp lane_sum(uint32_t p0, uint32_t p1, uint32_t m0, uint32_t m1) {
  const fp a = ld(p0), b = ld(p1), c = ld(m0), d = ld(m1);
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
DEV void reduce13(uint32_t mul_p, const uint32_t *v, uint32_t *r) {
  constexpr float K = (float)(256.0 / 436277739.0 * (1.0 - 1.0 / 1048576.0));  // 436277739 = floor(p / 2^352) + 1
  const uint32_t q = (uint32_t)(__uint2float_rz(__funnelshift_l(v[11], v[12], 24)) * K);
  const fp m = ld(mul_p + q * (uint32_t)sizeof(fp));
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
