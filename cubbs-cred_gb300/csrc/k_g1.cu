// G1 kernels: point decoding, the subgroup check, fixed-base window tables over
// the resident generators, the fixed-base MSM (4 to 512 lanes per MSM row,
// signed w-bit windows, affine table entries, mixed XYZZ additions, octet tree
// sums), GLV variable-base multiplication and point compression.
//
// Reference counterparts: comb tables and comb MSMs
// (native/cuda/src/kernels/comb_precompute.cuh:8-268, comb_msm.cuh:3-363),
// GLV variable base (kernels/variable_base_universal.cuh:25-331), BLST decode
// and compress on the host (native/cuda/src/g1_msm_blst.cpp:614-732).  Here
// decode and compress run on the device.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "bipartite.cuh"
#include "g1_ladder.cuh"
#include "runtime.cuh"

namespace cubbs {

__global__ void __launch_bounds__(64) k_g1_decode(const uint8_t *pts, uint32_t stride, uint32_t n, g1a *out,
                                                   int32_t *status) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint8_t b[48];
  for (int k = 0; k < 48; k++) b[k] = pts[(size_t)i * stride + k];
  g1a a;
  int st = g1_decompress(b, a, false);
  if (st != DEC_OK) {
    a.x = fp_zero();
    a.y = fp_zero();
  }
  out[i] = a;
  status[i] = st;
}

// The same on pairs of warps (bipartite.cuh): lane l of both warps of a block decodes point 32 blockIdx + l.  Bound by the chain of
// 376 squares and 86 products of one square root; 1 to 3072 points: 0.41 -> 0.26 ms.
__global__ void __launch_bounds__(64) k_g1_decode_pair(const uint8_t *pts, uint32_t stride, uint32_t n, g1a *out,
                                                       int32_t *status) {
  __shared__ __align__(16) bp::Exchange ex;
  __shared__ __align__(16) bp::Powers pow;
  const uint32_t lane = threadIdx.x & 31, i = 32 * blockIdx.x + lane;
  if (n == 0) return;
  uint8_t b[48];
  const uint8_t *src = pts + (size_t)min(i, n - 1) * stride;  // spare lanes repeat the last point
  for (int k = 0; k < 48; k++) b[k] = src[k];
  g1a a;
  fp rhs = fp_zero();
  bool sort;
  int st = g1_x(b, a.x, rhs, sort);
  const fp in = C_FP_BP_IN, back = C_FP_BP_OUT;
  __syncwarp();  // the rounds' barriers want whole warps
  bp::Pair w{&ex, (int)(threadIdx.x >> 5), (int)lane, 1, 0};
  const fp root = bp::sqrt_power(w, pow, fp_mul(rhs, in));
  if (w.half || i >= n) return;
  if (st == DEC_OK) {
    a.y = fp_mul(root, back);
    if (!fp_eq(fp_sqr(a.y), rhs)) st = DEC_BAD;
    else if (fp_lex_largest(a.y) != sort) a.y = fp_neg(a.y);
  }
  if (st != DEC_OK) a.x = a.y = fp_zero();
  out[i] = a;
  status[i] = st;
}

// Window bases of a table chunk: bases[(g - g0) * nwin + k] = 2^(w k) G_g in
// affine form, one thread per (generator, window).
__global__ void __launch_bounds__(64) k_table_bases(const g1a *gens, int g0, int g1n, FixedTable t, g1a *bases) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (g1n - g0) * t.nwin) return;
  const int g = g0 + tid / t.nwin, k = tid % t.nwin;
  g1 B = g1_from_aff(gens[g]);
  #pragma unroll 1
  for (int i = 0; i < t.w * k; i++) B = g1_dbl(B);
  g1_to_aff(B, bases[tid]);
}

// Table entries d * B for d = 1..half of every window base B, one thread per
// run of `run` consecutive entries: the thread reaches (d0 + 1) B by double-
// and-add from B, adds B for each further entry and normalises its run to
// affine with one batched inversion.  The runs keep the build parallel at
// wide windows (2^19 entries per window at w = 20).
__global__ void __launch_bounds__(64) k_table_build(const g1a *bases, int g0, int g1n, FixedTable t, int run,
                                                    g1 *scratch, fp *prod) {
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int runs = t.half / run;
  if (tid >= (size_t)(g1n - g0) * t.nwin * runs) return;
  const size_t base_i = tid / runs;
  const int d0 = (int)(tid % runs) * run;
  const g1a Ba = bases[base_i];
  g1 e = g1_from_aff(Ba);
  const uint32_t m = (uint32_t)d0 + 1;  // e = m * B
  #pragma unroll 1
  for (int b = 30 - __clz(m); b >= 0; b--) {
    e = g1_dbl(e);
    if ((m >> b) & 1) e = g1_add_aff(e, Ba);
  }
  g1 *E = scratch + tid * run;
  fp *Pp = prod + tid * run;
  fp acc = fp_one();
  #pragma unroll 1
  for (int j = 0; j < run; j++) {
    if (j > 0) e = g1_add_aff(e, Ba);
    E[j] = e;
    acc = fp_mul(acc, fp_mul(e.ZZ, e.ZZZ));
    Pp[j] = acc;
  }
  fp inv = fp_inv(acc);  // inverse of prod_j ZZ_j ZZZ_j
  g1a *dst = t.entries + ((size_t)g0 * t.nwin + base_i) * t.half + d0;
  #pragma unroll 1
  for (int j = run - 1; j >= 0; j--) {
    fp zinv = j > 0 ? fp_mul(inv, Pp[j - 1]) : inv;  // 1 / (ZZ_j ZZZ_j)
    g1 ej = E[j];
    inv = fp_mul(inv, fp_mul(ej.ZZ, ej.ZZZ));
    g1a a;
    a.x = fp_mul(ej.X, fp_mul(zinv, ej.ZZZ));
    a.y = fp_mul(ej.Y, fp_mul(zinv, ej.ZZ));
    dst[j] = a;
  }
}

// w-bit field of a raw 256-bit scalar in memory, starting at bit pos < 256
DEV uint32_t scalar_bits(const uint32_t *s, int pos, int w) {
  const int wi = pos >> 5;
  const uint32_t lo = s[wi], hi = wi + 1 < 8 ? s[wi + 1] : 0;
  return __funnelshift_r(lo, hi, pos & 31) & ((1u << w) - 1);
}

// Signed w-bit digit of window k of scalar s: digits in (-half, half], a digit
// above half becomes d - 2^w with a carry into the next window.  The carry
// into window k is 1 when the window below it is above half, 0 when it is
// less, and that window's own carry when it is half: one more window is read
// almost always.
DEV uint32_t fixed_digit(const uint32_t *s, int k, int w, uint32_t half, bool &neg) {
  uint32_t carry = 0;
  #pragma unroll 1
  for (int i = k - 1; i >= 0; i--) {
    const uint32_t v = scalar_bits(s, i * w, w);
    if (v != half) {
      carry = v > half ? 1u : 0u;
      break;
    }
  }
  const uint32_t d = scalar_bits(s, k * w, w) + carry;
  neg = d > half;
  return neg ? (1u << w) - d : d;  // 2^w - d is 0 for d = 2^w (the carry alone)
}

// Fixed-base MSM: row r = sum_g scalars[r*stride + g] * G_g, g < nterms[r].
// A row runs on a group of L lanes, L a power of two: 4 .. 32 (a block of
// one warp, 32 / L rows) or L / 32 warps (a block, one row).  Its (generator,
// window) units g * nwin + k are dealt round robin to the lanes, so every lane
// does the same number of mixed additions whatever the row's length (give or
// take one); each nonzero digit costs one table lookup and one mixed addition,
// and the next unit's table entry (a random 96-byte read from HBM) is fetched
// while the current one is added.  The lanes' sums are added as projective
// triples by the lane octets (g1_ladder.cuh, Adder::level): 9 levels of a 32-lane
// row take 41 thousand cycles where five rounds of shuffled full additions
// took 140 thousand, so that short rows can spread over many lanes.
// Dynamic shared memory: fixed_smem of the block's warps.
constexpr uint32_t fixed_smem(uint32_t warps) { return warps * (32 * gl::TRIPLE + 4 * gl::TMP_BYTES); }
// THREADS: the largest block.  Few rows spread over 256 or 512 lanes take the
// form with 128 registers, which spills (396 bytes stored, 508 loaded a thread);
// the other has 204 and spills nothing.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_fixed_msm(FixedTable t, const fr *scalars, uint32_t stride,
                                                   const uint32_t *nterms, uint32_t rows, uint32_t L, g1 *out) {
  extern __shared__ __align__(16) uint8_t fixed_mem[];
  __shared__ __align__(16) fp mul_p[slots::QMAX];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const uint32_t per_block = L < 32 ? 32 / L : 1, sub = threadIdx.x & (L - 1);
  const uint32_t row = blockIdx.x * per_block + threadIdx.x / L;
  const uint32_t half = (uint32_t)t.half, nwin = (uint32_t)t.nwin;
  fp *base = reinterpret_cast<fp *>(fixed_mem);
  for (uint32_t k = threadIdx.x; k < slots::QMAX; k += blockDim.x) mul_p[k] = slots::multiple_of_p(k);
  const uint32_t tmp = warps * 32 * gl::TRIPLE + warp * 4 * gl::TMP_BYTES;
  if ((lane & 7) == 0)
    *reinterpret_cast<fp *>(fixed_mem + tmp + (lane >> 3) * gl::TMP_BYTES + gl::at(gl::ZERO)) = fp_zero();

  const uint32_t units = row < rows ? nterms[row] * nwin : 0;
  g1 acc = g1_inf();
  g1a next;
  bool have = false, neg = false;
  auto fetch = [&](uint32_t u) {
    have = false;
    if (u >= units) return;
    const uint32_t g = u / nwin, k = u - g * nwin;
    const uint32_t d = fixed_digit(scalars[(size_t)row * stride + g].w, (int)k, t.w, half, neg);
    have = d != 0;
    if (have) next = t.entries[((size_t)g * nwin + k) * half + d - 1];
  };
  fetch(sub);
  #pragma unroll 1
  for (uint32_t u = sub; u < units; u += L) {
    g1a e = next;
    const bool use = have;
    if (neg) e.y = fp_neg(e.y);
    fetch(u + L);
    if (use) acc = g1_add_aff_inl(acc, e);  // inlined: no struct arguments through the stack
  }
  gl::put_triple(base + 3 * threadIdx.x, acc);
  __syncthreads();  // the triples, the multiples of p and the zero slots
  // each warp adds its own 32 triples (32 / L rows of L, or one part of a row),
  // then the first warp the warps' sums; one loop, one copy of the addition
  const uint32_t in_warp = L < 32 ? L : 32;
  const gl::Adder adder = gl::Adder::on(slots::addr(fixed_mem) + tmp, slots::addr(mul_p));
  const uint32_t groups = 32 / in_warp;
  uint32_t first = slots::addr(base + 3 * 32 * warp), span = in_warp, step = gl::TRIPLE, d = in_warp / 2;
  #pragma unroll 1
  for (bool across = false;; d >>= 1) {
    if (d == 0) {
      if (across || L <= 32) break;
      across = true;
      __syncthreads();
      if (warp != 0) return;
      first = slots::addr(base);
      step = 32 * gl::TRIPLE;
      d = warps / 2;
      span = warps;
    }
    adder.level(first, groups * d, d, span, step);
  }
  // one octet per row (up to four at a time) writes it
  #pragma unroll 1
  for (uint32_t k = lane >> 3; k < per_block; k += 4) {
    const uint32_t r = blockIdx.x * per_block + k;
    if (r < rows) gl::get_triple(base + 3 * k * in_warp, (int)(lane & 7), &out[r]);
  }
}

// One lane pair per job (g1_mul_glv_pair): the pair splits each point
// operation's products, halving the latency of a job.
__global__ void __launch_bounds__(128) k_var_mul_pair(const g1a *points, const VarJob *jobs, const fr *scalars,
                                                      uint32_t n, g1 *out) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t i = t >> 1;
  if (i >= n) return;  // both lanes of a pair leave together
  const LanePair lp = LanePair::here();
  const VarJob j = jobs[i];
  if (j.flags & 1) {
    if (lp.role == 0) out[i] = g1_inf();
    return;
  }
  const g1 r = g1_mul_glv_pair(lp, points[j.point], scalars[i]);
  if (lp.role == 0) out[i] = r;
}
// One lane quad per job (g1_mul_glv_quad).
__global__ void __launch_bounds__(128) k_var_mul_quad(const g1a *points, const VarJob *jobs, const fr *scalars,
                                                      uint32_t n, g1 *out) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t i = t >> 2;
  if (i >= n) return;  // the four lanes of a quad leave together
  const LaneQuad lq = LaneQuad::here();
  const VarJob j = jobs[i];
  if (j.flags & 1) {
    if (lq.role == 0) out[i] = g1_inf();
    return;
  }
  const g1 r = g1_mul_glv_quad(lq, points[j.point], scalars[i]);
  if (lq.role == 0) out[i] = r;
}
// Two ladders of eight lanes per job (g1_ladder.cuh), one per GLV half; two
// jobs a block of one warp, or of two that share the products (HALVES).
template <bool HALVES>
__global__ void __launch_bounds__(HALVES ? 64 : 32) k_var_mul_ladder(const g1a *points, const VarJob *jobs,
                                                                     const fr *scalars, uint32_t n, g1 *out) {
  __shared__ __align__(16) gl::Mem mem;
  __shared__ __align__(16) gl::Halves halves;
  if (n == 0) return;
  const int lane = threadIdx.x & 31, role = lane & 7, half = (lane >> 3) & 1;
  const uint32_t i = 2 * blockIdx.x + (lane >> 4);
  const uint32_t j = min(i, n - 1);  // a warp's spare ladders repeat the last job
  const VarJob job = jobs[j];
  const bool inf = job.flags & 1;
  g1a p;
  p.x = p.y = fp_one();
  if (!inf) p = points[job.point];
  const gl::LaddersOf<HALVES> l = gl::start<HALVES>(&mem, p, half != 0, &halves);
  uint32_t s[4], q[4];
  glv_split(scalars[j], s, q);
  fp *sl = l.sl;
  // the first ladder takes the second's sum as its entry 0, and leaves E'
  gl::ladder128(l, half ? q : s, [&] {
    if (!half && role < 3) sl[gl::TAB + (role == 2 ? 3 : role)] = mem.slot[(lane >> 3) + 1][gl::AX + role];
  });
  if (!l.first) return;
  if (!half && role < 2) {
    fp v[2];
    gl::leave<HALVES>(sl, role, v);
    if (i < n) {
      if (inf) {
        const g1 o = g1_inf();
        v[0] = role ? o.Y : o.X;
        v[1] = fp_zero();
      }
      (role ? out[i].Y : out[i].X) = v[0];
      (role ? out[i].ZZZ : out[i].ZZ) = v[1];
    }
  }
}
__global__ void __launch_bounds__(128) k_var_mul(const g1a *points, const VarJob *jobs, const fr *scalars,
                                                 uint32_t n, g1 *out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  VarJob j = jobs[i];
  if (j.flags & 1) {
    out[i] = g1_inf();
    return;
  }
  out[i] = g1_mul_glv(points[j.point], scalars[i]);
}

__global__ void __launch_bounds__(128) k_g1_compress(const g1 *pts, uint32_t n, uint8_t *out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint8_t b[48];
  g1_compress(pts[i], b);
  for (int k = 0; k < 48; k++) out[48 * (size_t)i + k] = b[k];
}

// Subgroup check of points decoded without it: bad[i] = 1 when point i
// decoded to an affine point outside G1 (status DEC_OK), else 0.  Without
// `bad` the point itself is marked as not decoded (DEC_BAD, zero coordinates).
DEV void subgroup_result(g1a *pts, int32_t *status, uint32_t i, int32_t *bad, bool outside) {
  if (bad) {
    bad[i] = outside ? 1 : 0;
  } else if (outside) {
    status[i] = DEC_BAD;
    pts[i].x = pts[i].y = fp_zero();
  }
}
// One lane per point: for launches that fill every SM sub-partition several
// times.  Bound by the products (126 doublings of two products and five
// squares); the base point waits in shared memory so that ten warps fit an SM
// (133 thousand points beside other kernels: 5.3 -> 4.7 ms; twelve or sixteen
// spill: 4.9, 5.0).
__global__ void __launch_bounds__(32, 10) k_g1_subgroup_lane(g1a *pts, int32_t *status, uint32_t n, int32_t *bad) {
  __shared__ g1j base[32];
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  subgroup_result(pts, status, i, bad, status[i] == DEC_OK && !g1_in_subgroup(pts[i], &base[threadIdx.x]));
}
// One lane pair per point.
__global__ void __launch_bounds__(32) k_g1_subgroup(g1a *pts, int32_t *status, uint32_t n, int32_t *bad) {
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 1;
  if (i >= n) return;  // both lanes of a pair leave together
  const LanePair lp = LanePair::here();
  const bool outside = status[i] == DEC_OK && !g1_in_subgroup_pair(lp, pts[i]);
  __syncwarp(lp.mask);  // the other lane has read the point
  if (lp.role == 0) subgroup_result(pts, status, i, bad, outside);
}
// One lane quad per point.
__global__ void __launch_bounds__(64) k_g1_subgroup_quad(g1a *pts, int32_t *status, uint32_t n, int32_t *bad) {
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  if (i >= n) return;  // the four lanes of a quad leave together
  const LaneQuad lq = LaneQuad::here();
  const bool outside = status[i] == DEC_OK && !g1_in_subgroup_quad(lq, pts[i]);
  __syncwarp(lq.mask);  // the other lanes have read the point
  if (lq.role == 0) subgroup_result(pts, status, i, bad, outside);
}

// One ladder of eight lanes per point (g1_ladder.cuh), four points a warp, one
// warp a block: phi(P) == -[z^2]P, that is [z^2]P == (beta x, -y).
__global__ void __launch_bounds__(32) k_g1_subgroup_ladder(g1a *pts, int32_t *status, uint32_t n, int32_t *bad) {
  __shared__ __align__(16) gl::Mem mem;
  if (n == 0) return;
  const int lane = threadIdx.x & 31, role = lane & 7;
  const uint32_t i = 4 * blockIdx.x + (lane >> 3), j = min(i, n - 1);
  const bool ok = status[j] == DEC_OK;
  g1a p;
  p.x = p.y = fp_one();
  if (ok) p = pts[j];
  const gl::Ladders l = gl::start(&mem, p, false);
  const fp *sl = l.sl;
  gl::mul_z2(l);
  if (role == 0 && i < n) {
    const fp beta = C_GLV_BETA;
    fp X = sl[gl::AX], Y = sl[gl::AY], Z = sl[gl::AZ], x = sl[gl::TAB + 4], y = sl[gl::TAB + 5];
    fp_csub1(X.w, X.w);
    fp_csub1(Y.w, Y.w);
    fp_csub1(Z.w, Z.w);
    fp_csub1(x.w, x.w);
    fp_csub1(y.w, y.w);
    const bool in = !fp_is_zero(Z) && fp_eq(X, fp_mul(fp_mul(x, beta), Z)) && fp_eq(Y, fp_mul(fp_neg(y), Z));
    subgroup_result(pts, status, i, bad, ok && !in);
  }
}

// CUBBS_BBS_VAR_LANES (1, 2, 4 or 8; else 0: chosen by launch size).
int var_lanes_setting() {
  static const int v = [] {
    const char *e = std::getenv("CUBBS_BBS_VAR_LANES");
    const int x = e && *e ? std::atoi(e) : 0;
    return (x == 1 || x == 2 || x == 4 || x == 8) ? x : 0;
  }();
  return v;
}
// Lanes per job for a launch of n jobs: the CUBBS_BBS_VAR_LANES setting, else
// by size.  Few jobs leave the GPU idle, so each takes ladders of eight lanes
// (g1_ladder.cuh); thousands fill it, where lane pairs spend fewer
// instructions a job.  Terms on GB300, 8 lanes against 2: 64 0.39 ms against
// 1.16, 1000 0.49 against 1.16, 7168 1.46 against 1.16; whole calls at 4096
// terms (ProofVerify of 1024 over 64 keys) were 3 % slower on 8 lanes, and
// lane quads at every size slower than one or the other; those are left for
// the setting.  The line counts the whole GPU's SMs, as do the other lines of
// this file; ProofVerify of a few keys makes these launches on partitions of 48
// and 88 SMs, where they would lie lower (run_pverify has one of its own).
static int lanes_for(uint32_t n) {
  const int l = var_lanes_setting();
  return l ? l : n <= 2048 ? 8 : 2;
}

// Above one warp per SM sub-partition (152 x 4) of points, one lane each: the
// Jacobian doublings there cost seven products' time, the pair's ten.
int subgroup_lanes(uint32_t n) { return n > 19456 && !var_lanes_setting() ? 1 : lanes_for(n); }

void launch_g1_subgroup(cudaStream_t s, g1a *pts, int32_t *status, uint32_t n, int32_t *bad, int lanes) {
  if (!n) return;
  if (lanes == 0) lanes = subgroup_lanes(n);
  if (lanes == 8) k_g1_subgroup_ladder<<<blocks_for(n, 4), 32, 0, s>>>(pts, status, n, bad);
  else if (lanes == 4) k_g1_subgroup_quad<<<blocks_for(4 * (size_t)n, 64), 64, 0, s>>>(pts, status, n, bad);
  else if (lanes == 2) k_g1_subgroup<<<blocks_for(2 * (size_t)n, 32), 32, 0, s>>>(pts, status, n, bad);
  else k_g1_subgroup_lane<<<blocks_for(n, 32), 32, 0, s>>>(pts, status, n, bad);
}
void launch_g1_decode(cudaStream_t s, const uint8_t *pts48, uint32_t stride, uint32_t n, g1a *out, int32_t *status,
                      bool check_subgroup) {
  if (!n) return;
  // Up to one warp per SM sub-partition (152 x 4, two warps per 32 points) the
  // launch is bound by one square root's chain, which pairs of warps shorten
  // (0.41 -> 0.26 ms); beyond that the one-lane form has fewer multiply-adds a
  // point.
  if (n > 9728) k_g1_decode<<<blocks_for(n, 64), 64, 0, s>>>(pts48, stride, n, out, status);
  else k_g1_decode_pair<<<blocks_for(n, 32), 64, 0, s>>>(pts48, stride, n, out, status);
  if (check_subgroup) launch_g1_subgroup(s, out, status, n, nullptr);
}
void launch_build_table(cudaStream_t s, const g1a *gens, int g0, int g1n, FixedTable t, g1a *bases, g1 *scratch,
                        fp *prod) {
  const int nb = (g1n - g0) * t.nwin;
  if (nb <= 0) return;
  k_table_bases<<<blocks_for(nb, 64), 64, 0, s>>>(gens, g0, g1n, t, bases);
  const int run = std::min(t.half, 256);
  k_table_build<<<blocks_for((size_t)nb * (t.half / run), 64), 64, 0, s>>>(bases, g0, g1n, t, run, scratch, prod);
}
// Lanes per row (CUBBS_BBS_FIXED_LANES forces 4, 8, 16 or 32): the power of two
// that a model of the launch finds fastest.  A lane does units / L mixed
// additions of ten products; the tree sum is `passes` additions of two
// products' depth; a product costs a lone warp of an SM sub-partition 1816
// cycles and each of several warps 1215.
static uint32_t fixed_lanes_for(uint32_t rows, uint32_t stride, int nwin) {
  static const uint32_t forced = [] {
    const char *e = std::getenv("CUBBS_BBS_FIXED_LANES");
    const int x = e && *e ? std::atoi(e) : 0;
    return (uint32_t)((x == 4 || x == 8 || x == 16 || x == 32) ? x : 0);
  }();
  if (forced) return forced;
  int dev = 0, sms = 152;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const double units = (double)stride * nwin;
  uint32_t best = 4;
  double best_cost = 0;
  for (uint32_t L = 4; L <= 512; L *= 2) {
    const uint32_t in_warp = L < 32 ? L : 32, warps = L < 32 ? 1 : L / 32;
    double passes = 0;
    for (uint32_t d = in_warp / 2; d > 0; d >>= 1) passes += (32 / in_warp * d + 3) / 4;
    for (uint32_t d = warps / 2; d > 0; d >>= 1) passes += (d + 3) / 4;
    const double products = std::ceil(units / L) * 10 + 3 + 2.4 * passes;
    const double total = (double)rows * L / 32, per = std::ceil(total / (4.0 * sms));
    const double cost = products * (per <= 1 ? 1816 : per * 1215);
    if (L == 4 || cost < best_cost) {
      best = L;
      best_cost = cost;
    }
  }
  return best;
}
void launch_fixed_msm(cudaStream_t s, const FixedTable &t, const fr *scalars, uint32_t stride,
                      const uint32_t *nterms, uint32_t rows, g1 *out) {
  if (!rows) return;
  const uint32_t L = fixed_lanes_for(rows, stride, t.nwin), threads = L < 32 ? 32 : L, per_block = L < 32 ? 32 / L : 1;
  static const bool attr = [] {
    CUBBS_CHECK(cudaFuncSetAttribute(k_fixed_msm<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fixed_smem(16)));
    return true;
  }();
  (void)attr;
  const unsigned blocks = (rows + per_block - 1) / per_block;
  const size_t smem = fixed_smem(threads / 32);
  if (threads <= 128) k_fixed_msm<128><<<blocks, threads, smem, s>>>(t, scalars, stride, nterms, rows, L, out);
  else k_fixed_msm<512><<<blocks, threads, smem, s>>>(t, scalars, stride, nterms, rows, L, out);
}
void launch_var_mul(cudaStream_t s, const g1a *points, const VarJob *jobs, const fr *scalars, uint32_t n, g1 *out,
                    int lanes) {
  if (!n) return;
  if (lanes == 0) lanes = lanes_for(n);
  // Products shared by two warps while those still find a sub-partition each
  // (152 x 4): 64 terms 0.39 -> 0.33 ms.
  if (lanes == 8 && n <= 608) k_var_mul_ladder<true><<<blocks_for(n, 2), 64, 0, s>>>(points, jobs, scalars, n, out);
  else if (lanes == 8) k_var_mul_ladder<false><<<blocks_for(n, 2), 32, 0, s>>>(points, jobs, scalars, n, out);
  else if (lanes == 4) k_var_mul_quad<<<blocks_for(4 * (size_t)n, 128), 128, 0, s>>>(points, jobs, scalars, n, out);
  else if (lanes == 2) k_var_mul_pair<<<blocks_for(2 * (size_t)n, 128), 128, 0, s>>>(points, jobs, scalars, n, out);
  else k_var_mul<<<blocks_for(n, 128), 128, 0, s>>>(points, jobs, scalars, n, out);
}
void share_carveout_g1() {
  share_carveout(k_g1_decode, k_g1_decode_pair, k_fixed_msm<128>, k_fixed_msm<512>, k_var_mul, k_var_mul_pair,
                 k_var_mul_quad, k_var_mul_ladder<true>, k_var_mul_ladder<false>, k_g1_subgroup_lane, k_g1_subgroup, k_g1_subgroup_quad,
                 k_g1_subgroup_ladder, k_g1_compress);
}
cudaError_t warm_decode_and_var_mul_kernels(uint8_t *any_device_buffer) {
  // n = 0: every thread returns before touching memory
  k_g1_decode<<<1, 64>>>(any_device_buffer, 48, 0, nullptr, nullptr);
  k_g1_decode_pair<<<1, 64>>>(any_device_buffer, 48, 0, nullptr, nullptr);
  k_g1_subgroup_lane<<<1, 32>>>(nullptr, nullptr, 0, nullptr);
  k_g1_subgroup<<<1, 32>>>(nullptr, nullptr, 0, nullptr);
  k_g1_subgroup_quad<<<1, 64>>>(nullptr, nullptr, 0, nullptr);
  k_g1_subgroup_ladder<<<1, 32>>>(nullptr, nullptr, 0, nullptr);
  k_var_mul<<<1, 128>>>(nullptr, nullptr, nullptr, 0, nullptr);
  k_var_mul_pair<<<1, 128>>>(nullptr, nullptr, nullptr, 0, nullptr);
  k_var_mul_quad<<<1, 128>>>(nullptr, nullptr, nullptr, 0, nullptr);
  k_var_mul_ladder<true><<<1, 64>>>(nullptr, nullptr, nullptr, 0, nullptr);
  k_var_mul_ladder<false><<<1, 32>>>(nullptr, nullptr, nullptr, 0, nullptr);
  return cudaGetLastError();
}
void launch_g1_compress(cudaStream_t s, const g1 *pts, uint32_t n, uint8_t *out48) {
  if (n) k_g1_compress<<<blocks_for(n, 128), 128, 0, s>>>(pts, n, out48);
}

}  // namespace cubbs
