// Four-warp pairing check: one block of 128 lanes evaluates
//     e(P_a, Q_a) * e(P_b, Q_b) == 1
// for the launches whose latency is one check's: both lines share one Miller
// loop, and an Fp12 operation is one round of products and one round of signed
// sums (tables of gen_pairing_quad.py, checked there on exact integers).
//
// What bounds it: a lone warp's product, 1730 cycles of multiply-adds at six
// cycles each (field.cuh), in a chain of 315 cyclotomic squarings, 136 Miller
// rounds and about 40 others.  So every operation is cut to one product deep
// (two in a Miller step): schoolbook Fp2 products on up to 128 lanes, one warp
// per SM sub-partition, all outputs as sums of products.  The sums take
// 2^g lanes an output, four slots a lane, carry chains instead of
// weighted multiply-adds, and one reduction by a multiple of p from a table.
// The cyclotomic squaring is 30 products: they stay in one warp, but a second
// warp computes half of each (fp_bipartite.cuh: a b / 2^256 from both ends of
// a, 168 multiply-adds a warp instead of 300): the check takes 0.67 ms instead
// of 0.75.
// Such a product keeps the form x 2^256 (mod p), so the register that is squared
// holds x 2^256 and the one it is multiplied by in between x 2^384, whose
// Montgomery product is of the first form again.  Against the two-warp teams per pair that this replaces (LIN
// phases of at most 14 weighted terms, four to six a product): see
// k_pairing_check_team.
#pragma once
#include "fp_bipartite.cuh"
#include "pairing_team.cuh"
#include "slots.cuh"

#include "pairing_quad_program.cuh"

namespace pq {

static_assert(PQ_SLOTS >= PP_SLOTS, "the inverse runs on the same slots");
static_assert(PQ_QMAX == slots::QMAX, "the bounds checked by the generator");
struct Mem {
  fp slot[PQ_SLOTS];
  fp mul_p[PQ_QMAX];  // k p
  uint4 half[3][32];  // the second warp's halves of the products
  uint32_t half_top[32];
};
constexpr uint32_t HALF = (PQ_SLOTS + PQ_QMAX) * (uint32_t)sizeof(fp), HALF_TOP = HALF + 3 * 32 * 16;  // from the slots
constexpr uint32_t MUL_P = PQ_SLOTS * (uint32_t)sizeof(fp);  // from the slots

using namespace slots;
// slot[out] = (slot[a] [+ slot[a2]]) (slot[b] [+ slot[b2]]) << dbl, not fully
// reduced: operands below 2.1 p give a product below 1.42 p.  sl: address of
// the slots.
DEV void factors(uint32_t sl, const uint4 &e, fp &a, fp &b) {
  a = ld(sl + (e.x & 0xffffu));
  b = ld(sl + (e.x >> 16));
  if (e.w & 0x10u) {  // the same on every lane of a phase
    const fp a2 = ld(sl + (e.y & 0xffffu)), b2 = ld(sl + (e.y >> 16));
    fp_acc_add(a.w, a.w, a2.w);
    fp_acc_add(b.w, b.w, b2.w);
  }
  const uint32_t sh = (e.w >> 5) & 1u;
#pragma unroll
  for (int j = 11; j > 0; j--) b.w[j] = __funnelshift_l(b.w[j - 1], b.w[j], sh);
  b.w[0] <<= sh;
}
DEV void product(uint32_t sl, const uint4 &e) {
  fp a, b, r;
  factors(sl, e, a, b);
  fp_mont_mul(r.w, a.w, b.w);
  if ((e.z & 0xffffu) != PQ_NONE) st(sl + (e.z & 0xffffu), r.w);
}

// One output per 2^g lanes; every lane of the warp calls it.
DEV void sums(uint32_t sl, const uint4 &e) {
  const int g = (int)(e.w >> 4) & 7;
  if (g == 7) return;
  uint32_t v[13];
  const fp t = lane_sum(sl + (e.x & 0xffffu), sl + (e.x >> 16), sl + (e.y & 0xffffu), sl + (e.y >> 16));
#pragma unroll
  for (int j = 0; j < 12; j++) v[j] = t.w[j];
  v[12] = 0;
#pragma unroll 1
  for (int d = 1; d < (1 << g); d <<= 1) add_lane(v, d);
  if ((e.z & 0xffffu) != PQ_NONE) {
    uint32_t r[12];
    reduce13(sl + MUL_P, v, r);
    st(sl + (e.z & 0xffffu), r);
  }
}

// Runs program `prog`; every lane of the block calls it, and the block is in
// step before and after.
static __device__ __noinline__ void run(uint32_t sl, int prog) {
  const int lane = threadIdx.x;
  const int ph0 = PQ_FIRST[prog], ph1 = PQ_FIRST[prog + 1];
  uint4 e = __ldg(&PQ_ENTRY[ph0 * PQ_LANES + lane]);
#pragma unroll 1
  for (int ph = ph0; ph < ph1; ph++) {
    const uint4 nx = __ldg(&PQ_ENTRY[min(ph + 1, ph1 - 1) * PQ_LANES + lane]);
    if (e.w & 1u) sums(sl, e);
    else if ((e.z & 0xffffu) != PQ_NONE) product(sl, e);
    __syncthreads();
    e = nx;
  }
}

// Register R squared n times in the cyclotomic subgroup, on one warp, or on two
// (HALVES): both compute their half of every product, the first adds the halves
// and has the sums to itself.  An output is 3 A + post with A on a lane pair (two lane sums)
// and post one slot added or subtracted on the odd lane.
template <bool HALVES> static __device__ __noinline__ void cyclo(uint32_t sl, int n) {
  const int lane = threadIdx.x & 31;
  const bool second = threadIdx.x >= 32;
  const uint4 em = __ldg(&PQ_CYCLO_M[lane]), es = __ldg(&PQ_CYCLO_S[lane]);
  const uint32_t half = sl + HALF + 16 * lane, top = sl + HALF_TOP + 4 * lane;
#pragma unroll 1
  for (; n > 0; n--) {
    if constexpr (HALVES) {
      uint32_t m[13];
      {
        fp x, y;
        factors(sl, em, x, y);
        if (second) fp_bp_mul_hi(m, x.w, y.w);
        else fp_bp_mul_lo(m, x.w, y.w);
      }
      if (second) {
#pragma unroll
        for (int k = 0; k < 3; k++)
          asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(half + 512 * k), "r"(m[4 * k]), "r"(m[4 * k + 1]),
                       "r"(m[4 * k + 2]), "r"(m[4 * k + 3])
                       : "memory");
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(top), "r"(m[12]) : "memory");
      }
      __syncwarp();
      asm volatile("bar.sync 1, 64;" ::: "memory");  // the halves
      if (second) {
        asm volatile("bar.sync 1, 64;" ::: "memory");  // the outputs
        continue;
      }
      if ((em.z & 0xffffu) != PQ_NONE) {
        uint32_t o[13];
#pragma unroll
        for (int k = 0; k < 3; k++)
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(o[4 * k]), "=r"(o[4 * k + 1]), "=r"(o[4 * k + 2]), "=r"(o[4 * k + 3])
                       : "r"(half + 512 * k)
                       : "memory");
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(o[12]) : "r"(top) : "memory");
        fp r;
        fp_bp_finish(r.w, m, o);
        st(sl + (em.z & 0xffffu), r.w);
      }
    } else {
      product(sl, em);
    }
    __syncwarp();
    const fp t = lane_sum(sl + (es.x & 0xffffu), sl + (es.x >> 16), sl + (es.y & 0xffffu), sl + (es.y >> 16));
    const fp pp = ld(sl + (es.z >> 16)), pm = ld(sl + es.w);
    uint32_t a[13], v[13];
    v[0] = t.w[0] << 1;
#pragma unroll
    for (int j = 1; j < 12; j++) v[j] = __funnelshift_l(t.w[j - 1], t.w[j], 1);
    v[12] = t.w[11] >> 31;
#pragma unroll
    for (int j = 0; j < 12; j++) a[j] = t.w[j];
    a[12] = 0;
    fp_acc_add_x(v, v, a);  // 3 t
#pragma unroll
    for (int j = 0; j < 12; j++) a[j] = pp.w[j];
    fp_acc_add_x(v, v, a);
#pragma unroll
    for (int j = 0; j < 12; j++) a[j] = pm.w[j];
    fp_acc_sub_x(v, v, a);
    add_lane(v, 1);
    __syncwarp();  // every lane has read its slots
    if ((es.z & 0xffffu) != PQ_NONE) {
      uint32_t r[12];
      reduce13(sl + MUL_P, v, r);
      st(sl + (es.z & 0xffffu), r);
    }
    __syncwarp();
    if constexpr (HALVES) asm volatile("bar.sync 1, 64;" ::: "memory");
  }
}

// Register `dst` = register `src`.
DEV void copy_reg(Mem *m, int dst, int src) {
  const int t = threadIdx.x;
  if (t < 36) {
    const uint4 *s = reinterpret_cast<const uint4 *>(&m->slot[PP_REG(src)]);
    reinterpret_cast<uint4 *>(&m->slot[PP_REG(dst)])[t] = s[t];
  }
  __syncthreads();
}
// Register r between the forms x 2^384 and x 2^256 (to: 2^256 or 2^512).
template <bool HALVES> DEV void to_form(Mem *m, int r, const fp &to) {
  if constexpr (!HALVES) return;
  const int t = threadIdx.x;
  if (t < 12) {
    fp &v = m->slot[PP_REG(r) + t];
    fp x;
    fp_mont_mul(x.w, v.w, to.w);
    fp_csub1(x.w, x.w);
    v = x;
  }
  __syncthreads();
}
// R = R^|z|, of the form x 2^256 with HALVES, with R = the base that the register of mul_prog holds as x 2^384.
template <bool HALVES> DEV void exp_by_zabs(uint32_t sl, int mul_prog) {
#pragma unroll 1
  for (int k = 0; k < 6; k++) {
    // |z| = 2^63 + 2^62 + 2^60 + 2^57 + 2^48 + 2^16
    const int n = k < 3 ? k + 1 : k == 3 ? 9 : k == 4 ? 32 : 16;
    if (threadIdx.x < (HALVES ? 64 : 32)) cyclo<HALVES>(sl, n);
    __syncthreads();
    if (k < 5) run(sl, mul_prog);
  }
}

// Registers r's slots fully reduced (S outputs are below 1.001 p).
DEV void canonical(Mem *m, int r) {
  const int t = threadIdx.x;
  if (t < 12) {
    fp &v = m->slot[PP_REG(r) + t];
    fp_csub1(v.w, v.w);
  }
  __syncthreads();
}

// Component c (A.c0, A.c1, B.c0, B.c1) of a line; a skipped pair has the line 1.
DEV fp line_part(const line2 *L, bool skip, int idx, int c) {
  if (skip) return c == 0 ? fp_one() : fp_zero();
  const line2 &l = L[idx];
  return c == 0 ? l.a.c0 : c == 1 ? l.a.c1 : c == 2 ? l.b.c0 : l.b.c1;
}

// The whole check; true on every lane when the product of the pairings is 1.
// All 128 lanes of the block call it.
template <bool HALVES, class Job> DEV bool pairing_check(Mem *m, const Job &j, const line2 *lines) {
  const int t = threadIdx.x;
  const bool skip[2] = {(j.flags & 1) != 0, (j.flags & 2) != 0};
  const line2 *const L[2] = {lines + (size_t)j.slot_a * MILLER_LINES, lines + (size_t)j.slot_b * MILLER_LINES};
  fp *sl = m->slot;
  const uint32_t at = addr(sl);
  // constants, points, F = 1
  if (t < PQ_QMAX) {
    m->mul_p[t] = multiple_of_p((uint32_t)t);
  } else if (t < PQ_QMAX + 10) {
    const fp2 g[6] = C_FROB_GAMMA;
    const int k = t - PQ_QMAX;
    const fp2 &ge = g[1 + (k >> 1)];
    sl[PP_GAMMA_BASE + k] = (k & 1) ? ge.c1 : ge.c0;
  } else if (t < PQ_QMAX + 14) {
    const int k = t - PQ_QMAX - 10, p = k >> 1;
    const g1a &pt = p ? j.pb : j.pa;
    sl[PP_PT_BASE + k] = skip[p] ? fp_zero() : ((k & 1) ? pt.y : pt.x);
  } else if (t == PQ_QMAX + 14) {
    sl[PP_ZERO_SLOT] = fp_zero();
  } else if (t >= 96 && t < 108) {
    sl[PP_REG(PP_REG_F) + t - 96] = t == 96 ? fp_one() : fp_zero();
  } else if (t >= 112 && t < 120) {
    sl[PP_LINE_BASE + t - 112] = line_part(L[(t - 112) >> 2], skip[(t - 112) >> 2], 0, t & 3);
  }
  __syncthreads();
  run(at, PQ_LINE);
  // Miller loop: the lanes that no product of a step's first round uses fetch
  // the next step's lines, whose B xP the second round multiplies
  const int lp = (t >> 2) & 1;
  const bool fetch = t >= 120;
  int idx = 1;
#pragma unroll 1
  for (int i = 62; i >= 0; i--) {
#pragma unroll 1
    for (int add = 0; add <= (int)zabs_bit(i); add++) {
      const int ph = PQ_FIRST[add ? PQ_ADD : PQ_DBL];
      const uint4 *tab = &PQ_ENTRY[ph * PQ_LANES + t];
      uint4 e = __ldg(tab);
      fp next = fp_zero();
      if (fetch && idx < MILLER_LINES) next = line_part(L[lp], skip[lp], idx, t & 3);
      idx++;
      const uint4 e1 = __ldg(tab + PQ_LANES), e2 = __ldg(tab + 2 * PQ_LANES), e3 = __ldg(tab + 3 * PQ_LANES);
#pragma unroll 1
      for (int k = 0; k < 2; k++) {
        if ((e.z & 0xffffu) != PQ_NONE) product(at, e);
        __syncthreads();
        if (k == 0 && fetch) sl[PP_LINE_BASE + t - 120] = next;
        sums(at, k ? e3 : e1);
        __syncthreads();
        e = e2;
      }
    }
  }
  // F holds the conjugate of the Miller value f (z < 0), so f^(p^6 - 1) =
  // F conj(F)^-1 = F conj(F^-1); then the powers as in final_exponentiation of
  // pairing.cuh (b^(z^2) needs no conjugation: both signs cancel)
  canonical(m, PP_REG_F);
  if (t < 64) pp::run<64>(sl, t, PP_INV_U_F, 1);
  __syncthreads();
  if (t < 5) sl[PQ_NORM2_BASE + t] = PQ_NORM2[t];  // the inverse's temporaries lie over these slots
  __syncthreads();
  run(at, PQ_T_F_CU);
  run(at, PQ_T_T2_T);
  const fp one256 = C_FP_BP_IN, two512 = C_FP_BP_OUT;
  copy_reg(m, PP_REG_R, PP_REG_T);
  to_form<HALVES>(m, PP_REG_R, one256);
  exp_by_zabs<HALVES>(at, PQ_R_R_T);
  run(at, PQ_A_CRT);  // a = t^z conj(t), as x 2^256
  copy_reg(m, PP_REG_R, PP_REG_A);
  to_form<HALVES>(m, PP_REG_A, two512);
  exp_by_zabs<HALVES>(at, PQ_R_R_A);
  run(at, PQ_A_CRA);  // a = a^z conj(a)
  copy_reg(m, PP_REG_R, PP_REG_A);
  to_form<HALVES>(m, PP_REG_A, two512);
  exp_by_zabs<HALVES>(at, PQ_R_R_A);
  run(at, PQ_X_FROB_A);
  run(at, PQ_A_X_CR);  // b = a^z a^p
  copy_reg(m, PP_REG_R, PP_REG_A);
  to_form<HALVES>(m, PP_REG_A, two512);
  exp_by_zabs<HALVES>(at, PQ_R_R_A);
  copy_reg(m, PP_REG_X, PP_REG_R);
  to_form<HALVES>(m, PP_REG_X, two512);
  exp_by_zabs<HALVES>(at, PQ_R_R_X);  // b^(z^2)
  run(at, PQ_R_A2_R);         // b^(z^2) b^(p^2)
  run(at, PQ_R_R_CA);
  run(at, PQ_R_R_T);
  run(at, PQ_R_R_T);
  run(at, PQ_R_R_T);
  canonical(m, PP_REG_R);
  bool one = true;
  if (t < 12) {
    const fp v = sl[PP_REG(PP_REG_R) + t];
    one = t == 0 ? fp_eq(v, HALVES ? one256 : fp_one()) : fp_is_zero(v);
  }
  return __syncthreads_and(one);
}

}  // namespace pq
