// Products mod p split over two warps (fp_bipartite.cuh), for launches bound by
// one lane's chain of products: the lanes l of two warps on different SM
// sub-partitions hold the same values, each warp computes one half of the
// product's sum, and they exchange the halves through shared memory.
// What bounds it: a lone warp's multiply-adds at six cycles each (field.cuh):
// 168 per product and 135 per square instead of 300 and 234, plus about 130
// cycles for the exchange (14 stores, a barrier of the two warps, 14 loads).
// Values are x 2^256 mod p, below p + 2^352.
#pragma once
#include "field.cuh"
#include "fp_bipartite.cuh"

namespace bp {

// One exchange buffer per pair of warps; rounds alternate between two halves
// of it, so one barrier a round suffices.
struct Exchange {
  uint4 v[2][2][3][32];
  uint32_t top[2][2][32];
};
struct Pair {
  Exchange *ex;
  int half, lane, bar;  // warp of the pair, lane, named barrier (1..15)
  int turn;

  DEV fp finish(const uint32_t *mine) {
    Exchange &e = *ex;
#pragma unroll
    for (int k = 0; k < 3; k++)
      e.v[turn][half][k][lane] = make_uint4(mine[4 * k], mine[4 * k + 1], mine[4 * k + 2], mine[4 * k + 3]);
    e.top[turn][half][lane] = mine[12];
    asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
    uint32_t other[13];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const uint4 q = e.v[turn][half ^ 1][k][lane];
      other[4 * k] = q.x;
      other[4 * k + 1] = q.y;
      other[4 * k + 2] = q.z;
      other[4 * k + 3] = q.w;
    }
    other[12] = e.top[turn][half ^ 1][lane];
    turn ^= 1;
    fp r;
    fp_bp_finish(r.w, mine, other);
    return r;
  }
  DEV fp mul(const fp &a, const fp &b) {
    uint32_t m[13];
    if (half) fp_bp_mul_hi(m, a.w, b.w);
    else fp_bp_mul_lo(m, a.w, b.w);
    return finish(m);
  }
  DEV fp sqr(const fp &a) {
    uint32_t m[13];
    if (half) fp_bp_sqr_hi(m, a.w);
    else fp_bp_sqr_lo(m, a.w);
    return finish(m);
  }
};

// a^((p + 1) / 4) by sliding windows; `pow`: the odd powers of the pair's lanes.
struct Powers {
  uint4 v[FP_SQRT_POWERS][3][32];
};
DEV void put(Powers &p, int k, int lane, const fp &a) {
#pragma unroll
  for (int q = 0; q < 3; q++) p.v[k][q][lane] = make_uint4(a.w[4 * q], a.w[4 * q + 1], a.w[4 * q + 2], a.w[4 * q + 3]);
}
DEV fp get(const Powers &p, int k, int lane) {
  fp a;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const uint4 t = p.v[k][q][lane];
    a.w[4 * q] = t.x;
    a.w[4 * q + 1] = t.y;
    a.w[4 * q + 2] = t.z;
    a.w[4 * q + 3] = t.w;
  }
  return a;
}
DEV fp sqrt_power(Pair &w, Powers &pow, const fp &a) {
  const fp a2 = w.sqr(a);
  fp x = a;
  #pragma unroll 1
  for (int k = 0; k < FP_SQRT_POWERS; k++) {  // x = a^(2 k + 1)
    if (w.half == 0) put(pow, k, w.lane, x);
    x = w.mul(x, a2);
  }
  fp r = get(pow, FP_SQRT_STEP[0][1], w.lane);  // (stored before the last product's barrier)
  #pragma unroll 1
  for (int s = 1; s < FP_SQRT_STEPS; s++) {
    #pragma unroll 1
    for (int n = FP_SQRT_STEP[s][0]; n > 0; n--) r = w.sqr(r);
    const int k = FP_SQRT_STEP[s][1];
    if (k != 255) r = w.mul(r, get(pow, k, w.lane));
  }
  return r;
}

}  // namespace bp
