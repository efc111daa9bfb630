// qb_tc2.cuh -- tensor-core form with two states per accumulator (tile pairs): one problem,
// or (16-bit form) the work items of a batch.
//
// Same decomposition as qb_tc.cuh (t: tile index in Gray order, y: the 128 MMA rows, u: the
// 256 MMA columns; E(t, y, u) = R_t(y) + C_t(u) + y^T V u), but the Gray-ordered tiles are
// taken in pairs (i, i + 1) with i even.  Their tile values t and t' = t ^ 1 differ in t
// bit 0 (variable n-16) alone, so
//   E(t', y, u) = R_t'(y) + D(y, u) + s * gamma(u),   D(y, u) = y^T V u + C_t(u)
//   gamma(u)    = sum_j W[n-16][n-1-j] u_j          (the couplings of variable n-16 with u)
//   s           = +1 if t bit 0 is 0, else -1       (bit 0 of gray(i) = (i >> 1) & 1)
// One MMA computes D for tile t; the epilogue reads each accumulator once and derives the
// partner tile's value from it.  Every TMEM accumulator thus stands for two states, which
// halves the MMAs, accumulator round trips and TMEM loads per state.  Measured on B200
// (n = 36 TSP QUBO, 2^36 states): fp32 pair form 3.83 ms, 16-bit pair form (below) 1.75 ms,
// against 3.8-3.95 ms for one state per accumulator; the 16-bit pair form is the default
// where it applies, and qb_autotune times both forms.
//
// fp32 pair form: roles, pipelines, records and bounded waits are those of
// tc_pass1_kernel<false> (qb_tc.cuh), with "tile" replaced by "pair" in the MMA, B-stage and
// accumulator pipelines: per pair the B producer writes the column-term digits of tile t and
// the row terms of both tiles.  acc_full takes two arrivals, the MMA's commit and the MMA
// thread's own arrive after it saw the pair's B stage full, so the epilogue's acquire of
// acc_full also orders the row terms and it needs no wait on the B stage.  Records (both
// forms): per block of 2^gl tiles (2^(gl-1) pairs, gl >= 5) 8 records, as in qb_tc.cuh
// (kGeomTC); a pair never straddles two blocks.
//
// Its epilogue (tc_pair_fp32_kernel): the partner's values by one fma per state (gamma of the 5
// low u bits as constant operands, the 3 high u bits added to each 32-column chunk's minimum)
// and 3-input fp32 minima.
//
// 16-bit pair form (tc_pair_kernel<kItems>: one problem, or the batch's work items;
// tc2_u16_eligible, tc2_u16_quantized).  As in the one-state 16-bit epilogue (qb_tc.cuh,
// tc_u16_eligible) the accumulator is an integer in [2^23, 2^24) whose fp32 pattern holds a
// 16-bit value in its low half, loaded two columns per register (.pack::16b).  Here the MMA
// computes F = D~ + 2^23 - Dlow_s with D~(y, u) = D(y, u) + s * X(u), X the gamma of the chunk
// bits u4, u5, u6 and Dlow_s = Dmin + min_u s * X(u): the column term carries s * X(u).  In a
// warp's 64 registers (u = 128 hh + 32 L + 2 j + half, register j of load L) the chunk
// c = (u4, u5, u6) = (j >> 3, L) and the position k = j & 7 (u1, u2, u3) with the half bit u0
// index an 8 x 8 grid, and
//   tile t:   D  - Dmin = (F mod 2^16) - s * X(c) + (Dlow_s - Dmin)       per-chunk correction
//   tile t':  D' - Dmin = (F mod 2^16) + s * (gamma - X)(k, u0, hh) + (Dlow_s - Dmin)
//                                                                      per-position correction
// so tile t takes the packed minimum over each chunk (8 registers) plus one add.u16x2 per
// chunk, and tile t' the packed minimum over the 8 chunks at each position plus one add.u16x2
// per position: 64 packed 3-input minimum inputs and 16 adds per 64 registers (8192 states),
// against 64 adds more when the partner's values are formed register by register.  Every
// corrected value is D - Dmin of a state, in [0, Dmax - Dmin]; the uncorrected ones lie in
// [0, Dmax - Dmin + sum_{b=4..6} |gamma_b|] < 2^16 (the eligibility condition), so packed
// 16-bit minima and mod-2^16 adds are exact.  Tile t of a pair is the one with t bit 0 clear
// (s = +1), whatever its Gray index, so one set of 16 corrections serves every pair.
//
// Exactness: for integer Q with sum|Q| <= 2^22, D + s*gamma(u) = y^T V u + C_t'(u) is an
// integer of magnitude at most sum|Q| (it is the accumulator tile t' would have had), so the
// fma is exact.  For float Q, gamma in fp32, its partial sums g5, the fma and the chunk
// offset add at most 8 roundings of 2^-24 relative to sum|Q| (scaled units) to the error
// bound of the digit contraction; tc2_error_bound() includes them.
#pragma once
#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "qb_tc.cuh"

namespace qb {

// per-state error bound of the float-digit pair form (unscaled units)
inline double tc2_error_bound(double abs_sum) { return 264.0 * abs_sum * 5.9604644775390625e-08 + 1e-300; }

// the 16-bit pair form's constants of one problem for either sign ([0] for s = +1, the one the
// kernel uses: tile t is the pair's tile with t bit 0 clear; [1] for s = -1), in the problem's
// units
struct Tc2Tab {
  float gx[3];               // gamma of the chunk bits u4, u5, u6
  float k0s[2];              // 2^23 - Dlow_s, the offset of the column term
  float dmin;                // lower bound of every accumulator value D
  uint32_t corr_t[2][8];     // tile t: correction of chunk c (u4 = c & 1, u5, u6 = c >> 1), both halves
  uint32_t corr_p[2][2][8];  // partner: correction of position k (u1..u3) in column half hh (u7)
};

struct Tc2Params {
  TcParams P;       // n, nt, gl, stall, exact, inv_scale, W, tile_begin, groups, groups_per_cta, rec, err
  alignas(8) float g5[32];     // fp32 form: gamma of register k of a 32-column chunk, sum_{j < 5} w_j k_j
  float whi[3];     // fp32 form: w_5, w_6, w_7, the gamma of u bits 5..7 (scaled W)
  Tc2Tab tab;       // 16-bit form, one problem (tc_pair_kernel<false>)
  const Tc2Tab* tabs;  // 16-bit form, work items: per item (tc_pair_kernel<true>)
};

// 16-bit pair kernel: t bits above the pair's that one B stage serves (kept in the A operand),
// epilogue warp groups (one 128-column TMEM accumulator each) and B stages
constexpr int kTc2Low = 3;
constexpr int kTc2Groups = 4;
constexpr int kTc2Threads = 128 + 128 * kTc2Groups;
constexpr int kTc2BStages = 4;
constexpr int kTc2EsRing = 8;  // blocks whose low-pattern energies are kept (a slot's readers are at most 5 blocks behind)
constexpr int kTc2LoCols = 8 + 7 + (kTc2Low + 1) + 1;
static_assert(kTc2Low == 3, "six K slots: two digits per low t bit; 2^4 tiles per block, at least 2^5 per record");

// K slots of low t bit m's digits d: 11 + 2 m + d, except that m = 2 has 15 and 7
__host__ __device__ constexpr int tc2_low_slot(int m, int d) { return m < 2 ? 11 + 2 * m + d : (d ? 7 : 15); }
__host__ __device__ constexpr int tc2_low_bit(int k) { return k == 7 || k == 15 ? 2 : (k - 11) >> 1; }
__host__ __device__ constexpr int tc2_low_digit(int k) { return k == 7 ? 1 : k == 15 ? 0 : (k - 11) & 1; }

// per-block parameters published by the block walk (the low t bits 0)
struct Tc2Slot {
  float f[8];             // (t^T W_TU)_j
  float g[7];             // (t^T W_TY)_i
  float c[kTc2Low + 1];  // couplings of the block's t with the low t bits
  float et;               // E_T(t)
};

struct Tc2Layout {
  uint32_t a_off, b_off, bar_off, slot_off, ct_off, wl_off, ll_off, eu_off, ey_off, rs_off, es_off, misc_off,
      lo_off, w_off, total;
};

__host__ __device__ inline Tc2Layout tc2_layout(int n) {
  Tc2Layout L;
  uint32_t o = 0;
  L.a_off = o;
  o += (1u << kTc2Low) * 128 * 32;  // A: 128 rows x 16 f16 per low pattern
  L.b_off = o;
  o += kTc2BStages * kTcN * 32;
  L.ct_off = o;
  o += 32 * 4;
  L.wl_off = o;
  o += (1u << kTc2Low) * 128 * 8;
  L.lo_off = o;
  o += 32 * kTc2LoCols * 8;
  L.w_off = o;
  o += (uint32_t)n * n * 8;
  L.bar_off = o;
  o += (2 * kTcParamSlots + 2 * kTc2BStages + 2 * kTc2Groups) * 8;
  L.slot_off = o;
  o += kTcParamSlots * sizeof(Tc2Slot);
  L.ll_off = o;
  o += 32 * 4;
  L.eu_off = o;
  o += kTcN * 4;
  L.ey_off = o;
  o += 128 * 4;  // E_Y(y) per row
  L.rs_off = o;
  o += kTc2BStages * 128 * 4;
  L.es_off = o;
  o += kTc2EsRing * 32 * 4;
  L.misc_off = o;
  o += 64;
  L.total = o;
  return L;
}

// dynamic shared memory of the kernel: at least 120 KB so that one CTA (and one 512-column
// TMEM allocation) runs per SM
inline size_t tc2_smem_bytes(int n) { return std::max<size_t>(tc2_layout(n).total, 120 * 1024) + 1024; }

// u bits that form the 16-bit pair epilogue's chunks (their gamma is folded into the MMA)
constexpr int kTc2ChunkBits[3] = {4, 5, 6};

// The 16-bit pair form applies (integer Q on the exact path; W unscaled, n x n FP64): the
// problems of the one-state 16-bit epilogue with room for the chunk offsets,
// Dmax - Dmin + sum over the chunk bits b of |gamma_b| < 2^16.
inline bool tc2_u16_eligible(int n, const double* W, float* dmin) {
  double span = 0.0;
  if (!tc_u16_eligible(n, W, dmin, &span)) return false;
  double gx = 0.0;
  for (int b : kTc2ChunkBits) gx += std::fabs(W[(size_t)(n - 16) * n + (n - 1 - b)]);
  return span + gx <= 65535.0;
}

// The 16-bit pair form off the exact path (float Q, or integer Q with sum|Q| > 2^22).  The
// kernel then works in units of 1/sigma, sigma a power of two applied to W: every MMA operand
// (the y coupling rows, T(u), the column term's constant part, the gammas of the corrections)
// is rounded to an integer in those units, so the accumulators are integers and the 16-bit
// epilogue stays exact on the rounded values.  The column term takes half of what the roundings
// of a column's seven y rows and three low t rows leave over before it is rounded itself, so that
// a row, in the state or not, adds at most a quarter unit: 2.5 units per state and 0.5 of the
// column term, for the partner 0.75 of the three chunk couplings of gamma, halved the same way,
// and 0.5 of their sum with the others.  Measured against FP64 (rms in units, n = 20 .. 24, float
// and wide integer Q): 0.55 for a pair's tile t and 0.66 for the partner; 0.86 and 0.96 with
// every row's rounding left where it falls.  fp32 rounding of the row terms and of the column
// term adds less than 2^-18 sum|Q| sigma.  eps = 10 / sigma + 2^-16 sum|Q| bounds it all
// (unscaled), and pass 2 re-walks every record within 2 eps of the minimum in FP64.  Applies
// when, at the largest such sigma, every y coupling row stays within +-2047 units, the value span
// with the chunk offsets and a 40-unit margin within 2^16 units, and the span covers at least
// 1024 units.  W: the unscaled n x n FP64 W.
// On success: sigma, dmin (the lower bound of the rounded values in units, an integer) and eps.
inline bool tc2_u16_quantized(int n, const double* W, double abs_sum, double* sigma, float* dmin, double* eps) {
  if (n < 20) return false;
  double lo = 0.0, hi = 0.0, rowmax = 0.0;
  auto add = [&](double w) {
    if (w < 0) lo += w;
    else hi += w;
  };
  for (int i = 0; i < 7; ++i) {
    double rp = 0.0, rn = 0.0;
    for (int j = 0; j < 8; ++j) {
      const double w = W[(size_t)(n - 9 - i) * n + (n - 1 - j)];
      if (w < 0) rn -= w;
      else rp += w;
      add(w);
    }
    rowmax = std::max(rowmax, std::max(rp, rn));
  }
  for (int j = 0; j < 8; ++j) {
    const int a = n - 1 - j;
    add(W[(size_t)a * n + a]);
    for (int j2 = 0; j2 < j; ++j2) add(W[(size_t)a * n + (n - 1 - j2)]);
    for (int t = 0; t < n - 15; ++t) add(W[(size_t)t * n + a]);
  }
  double gA = 0.0;
  for (int b : kTc2ChunkBits) gA += std::fabs(W[(size_t)(n - 16) * n + (n - 1 - b)]);
  const double span = hi - lo;
  if (!(span > 0.0) || !std::isfinite(span + gA)) return false;
  double lim = (65535.0 - 40.0) / (span + gA);
  if (rowmax > 0.0) lim = std::min(lim, 2047.0 / rowmax);
  double sg = std::ldexp(1.0, (int)std::floor(std::log2(lim)));
  while (sg * rowmax > 2047.0 || sg * (span + gA) + 40.0 > 65535.0) sg *= 0.5;
  if (sg * span < 1024.0) return false;  // too coarse: most records would become candidates
  *sigma = sg;
  *dmin = (float)(std::floor(sg * lo) - 12.0);
  *eps = 10.0 / sg + std::ldexp(abs_sum, -16);
  return true;
}


// the 16-bit pair form's constants from gamma (integers in the kernel's units, rounded here)
// and Dmin
inline void tc2_u16_tables(const float* gamma, float dmin, Tc2Tab* Q) {
  Q->dmin = dmin;
  int64_t g[8];
  for (int j = 0; j < 8; ++j) g[j] = (int64_t)std::llrint(gamma[j]);
  double left = 0.0;  // half of what rounding the chunk couplings leaves over
  for (int b : kTc2ChunkBits) left += 0.5 * ((double)gamma[b] - (double)g[b]);
  for (int b = 0; b < 3; ++b) Q->gx[b] = (float)g[kTc2ChunkBits[b]];
  for (int neg = 0; neg < 2; ++neg) {
    const int64_t s = neg ? -1 : 1;
    int64_t lo = 0;  // min over the chunk bits of s * X(u) = Dlow_s - Dmin
    for (int b = 0; b < 3; ++b) lo += std::min<int64_t>(0, s * g[kTc2ChunkBits[b]]);
    Q->k0s[neg] = (float)(8388608.0 - ((double)dmin + (double)lo));
    for (int c = 0; c < 8; ++c) {
      const int64_t x = ((c & 1) ? g[4] : 0) + ((c & 2) ? g[5] : 0) + ((c & 4) ? g[6] : 0);
      const uint32_t v = (uint32_t)((lo - s * x) & 0xffff);
      Q->corr_t[neg][c] = v | (v << 16);
    }
    for (int hh = 0; hh < 2; ++hh)
      for (int k = 0; k < 8; ++k) {
        uint32_t h[2];
        for (int d = 0; d < 2; ++d) {
          // rounded as one sum: half a unit off at most, whatever the number of couplings
          const double y = left + (d ? (double)gamma[0] : 0.0) + ((k & 1) ? (double)gamma[1] : 0.0) +
                           ((k & 2) ? (double)gamma[2] : 0.0) + ((k & 4) ? (double)gamma[3] : 0.0) +
                           (hh ? (double)gamma[7] : 0.0);
          const int64_t gp = (int64_t)std::llrint(y);
          h[d] = (uint32_t)((s * gp + lo) & 0xffff);
        }
        Q->corr_p[neg][hh][k] = h[0] | (h[1] << 16);
      }
  }
}

#ifdef __CUDACC__

// min over k of (D_k + s * g5[k]) for one 32-column chunk, two registers per packed fma
// (fma.rn.f32x2: the same rounding as two scalar fmas); g5 pairs are read from the parameter
// space with a constant index
__device__ __forceinline__ float min32_shift(const uint32_t* r, const Tc2Params& Q, float s) {
  float v[32];
  const uint64_t ss = ((uint64_t)__float_as_uint(s) << 32) | __float_as_uint(s);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const uint64_t g = *reinterpret_cast<const uint64_t*>(&Q.g5[2 * k]);
    const uint64_t d = ((uint64_t)r[2 * k + 1] << 32) | r[2 * k];
    uint64_t o;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(o) : "l"(g), "l"(ss), "l"(d));
    v[2 * k] = __uint_as_float((uint32_t)o);
    v[2 * k + 1] = __uint_as_float((uint32_t)(o >> 32));
  }
  float m0 = fmin3(v[0], v[1], v[2]);
  float m1 = fmin3(v[3], v[4], v[5]);
  float m2 = fmin3(v[6], v[7], v[8]);
  float m3 = fmin3(v[9], v[10], v[11]);
  float m4 = fmin3(v[12], v[13], v[14]);
  float m5 = fmin3(v[15], v[16], v[17]);
  float m6 = fmin3(v[18], v[19], v[20]);
  float m7 = fmin3(v[21], v[22], v[23]);
  float m8 = fmin3(v[24], v[25], v[26]);
  float m9 = fmin3(v[27], v[28], v[29]);
  float n0 = fmin3(m0, m1, m2);
  float n1 = fmin3(m3, m4, m5);
  float n2 = fmin3(m6, m7, m8);
  float n3 = fmin3(m9, v[30], v[31]);
  return fmin3(n0, n1, fminf(n2, n3));
}

// One N = 128 MMA, its commit on `full` issued by one elected
// lane of the (converged) calling warp: predicated instructions instead of a divergent branch,
// so the descriptors stay in uniform registers.
__device__ __forceinline__ void tc_issue_n128(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t full) {
  constexpr uint32_t idesc = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
  asm volatile(
      "{\n .reg .pred e, z;\n elect.sync _|e, 0xffffffff;\n setp.ne.b32 z, %4, %4;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, z;\n"
      " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%4];\n"
      "}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(full)
      : "memory");
}

// bounded wait of a role with slack (the tile walk and the B producer, up to 64 blocks and 4
// B stages ahead): sleeps between polls so that it leaves the issue slots to the epilogue,
// after a few polls without sleep (the pipeline's start, where nothing is ahead yet)
__device__ __forceinline__ bool mbar_wait_idle(uint64_t* b, uint32_t parity, volatile int* abort_flag) {
  for (int it = 0; it < 16; ++it)
    if (mbar_try_wait(b, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  for (;;) {
    __nanosleep(1000);
    if (mbar_try_wait(b, parity)) return true;
    if (*abort_flag) return false;
    if (globaltimer_ns() - t0 > kTcWaitLimitNs) return false;
  }
}

// bounded wait of the epilogue and the MMA issue, by a converged warp, as one statement without a
// result: a failed wait (the limit ran out, or another role gave up) sets fail, which the caller
// looks at once per block; with fail set, later waits return after one poll.  Every branch is on
// a vote, so that the warp stays together and fail is the same in all its lanes whatever the
// lanes' polls and clocks say.  The usual path is one try_wait, one vote and one branch.  The
// polls carry a 100 ns suspend hint (1.73 -> 1.72 ms per 2^36 states against the default; 1 us on
// the first try as well 1.78 ms).
__device__ __forceinline__ void mbar_wait_flag(uint32_t bar, uint32_t parity, uint32_t abort_addr, uint32_t& fail) {
  asm volatile(
      "{\n .reg .pred p, q;\n .reg .u64 t0, t1;\n .reg .u32 a;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n vote.sync.all.pred p, p, 0xffffffff;\n @p bra.uni DONE;\n"
      " setp.ne.u32 q, %0, 0;\n vote.sync.any.pred q, q, 0xffffffff;\n @q bra.uni DONE;\n mov.u64 t0, %%globaltimer;\n"
      "POLL:\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 100;\n vote.sync.all.pred p, p, 0xffffffff;\n"
      " @p bra.uni DONE;\n"
      " ld.volatile.shared.u32 a, [%3];\n mov.u64 t1, %%globaltimer;\n sub.u64 t1, t1, t0;\n"
      " setp.gt.u64 q, t1, %4;\n setp.ne.or.u32 q, a, 0, q;\n vote.sync.any.pred q, q, 0xffffffff;\n @!q bra.uni POLL;\n"
      " mov.u32 %0, 1;\n"
      "DONE:\n}\n"
      : "+r"(fail)
      : "r"(bar), "r"(parity), "r"(abort_addr), "n"(kTcWaitLimitNs)
      : "memory");
}

__device__ __forceinline__ void mbar_arrive_elect(uint32_t bar) {
  asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n @e mbarrier.arrive.shared::cta.b64 _, [%0];\n}\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ float u16lo_f(uint32_t v) {
  float f;
  asm("{\n .reg .u16 l, h;\n mov.b32 {l, h}, %1;\n cvt.rn.f32.u16 %0, l;\n}\n" : "=f"(f) : "r"(v));
  return f;
}
__device__ __forceinline__ float u16hi_f(uint32_t v) {
  float f;
  asm("{\n .reg .u16 l, h;\n mov.b32 {l, h}, %1;\n cvt.rn.f32.u16 %0, h;\n}\n" : "=f"(f) : "r"(v));
  return f;
}

__device__ __forceinline__ uint32_t uadd2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));  // per half, mod 2^16
  return d;
}

// packed unsigned 16-bit minimum of 8 registers (3-input minima)
__device__ __forceinline__ uint32_t umin8(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f,
                                          uint32_t g, uint32_t h) {
  return __vimin3_u16x2(__vimin3_u16x2(a, b, c), __vimin3_u16x2(d, e, f), umin2(g, h));
}

__global__ void __launch_bounds__(kTcThreads, 1) tc_pair_fp32_kernel(const __grid_constant__ Tc2Params Q) {
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  const TcParams& P = Q.P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const TcSmemLayout L = tc_layout(P.n);
  unsigned char* Asm = tc_smem + L.a_off;
  unsigned char* Bsm = tc_smem + L.b_off;
  uint64_t* bars = reinterpret_cast<uint64_t*>(tc_smem + L.bar_off);
  uint64_t* p_full = bars;
  uint64_t* p_empty = p_full + kTcParamSlots;
  uint64_t* b_full = p_empty + kTcParamSlots;
  uint64_t* b_empty = b_full + kTcBStages;
  uint64_t* acc_full = b_empty + kTcBStages;
  uint64_t* acc_empty = acc_full + kTcStages;
  TcSlot* slots = reinterpret_cast<TcSlot*>(tc_smem + L.slot_off);
  float* EU = reinterpret_cast<float*>(tc_smem + L.eu_off);
  float* EY = reinterpret_cast<float*>(tc_smem + L.ey_off);
  float* Rs = reinterpret_cast<float*>(tc_smem + L.rs_off);            // tile t of each pair
  float* Rs2 = reinterpret_cast<float*>(tc_smem + L.total);            // tile t' of each pair
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tc_smem + L.misc_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tc_smem + L.misc_off + 4);
  double* LO = reinterpret_cast<double*>(tc_smem + L.lo_off);
  double* Ws = reinterpret_cast<double*>(tc_smem + L.w_off);

  const uint64_t g0 = (uint64_t)blockIdx.x * P.groups_per_cta;
  if (g0 >= P.groups) return;  // uniform per CTA
  const uint64_t g1 = min(P.groups, g0 + P.groups_per_cta);
  const int n = P.n, nt = P.nt, gl = P.gl, exact = P.exact;
  const uint64_t i_begin = P.tile_begin + (g0 << gl), ntiles = (g1 - g0) << gl;
  float* rec = P.rec + (g0 << 3);
  const uint64_t t0 = gray64(i_begin);
  const float s1 = exact ? 2048.0f : 1.0f;

  if (tid == 0) {
    for (int s = 0; s < kTcParamSlots; ++s) {
      mbar_init(&p_full[s], 1);
      mbar_init(&p_empty[s], 1);
    }
    for (int s = 0; s < kTcBStages; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], 1);
    }
    for (int s = 0; s < kTcStages; ++s) {
      mbar_init(&acc_full[s], 2);  // the MMA's commit and the MMA thread (after it saw the B stage full)
      mbar_init(&acc_empty[s], kTcEpiWarps / 2);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  for (int i = tid; i < n * n; i += kTcThreads) Ws[i] = P.W[i] * P.scale;
  for (uint64_t r = (uint64_t)tid; r < ((ntiles >> gl) << 3); r += kTcThreads) rec[r] = __int_as_float(0x7f800000);
  __syncthreads();
  // A operand (constant)
  for (int e = tid; e < 128 * 16; e += kTcThreads) {
    int y = e >> 4, k = e & 15;
    float v;
    if (k < 14)
      v = ((y >> (k >> 1)) & 1) ? ((k & 1) ? s1 : 1.0f) : 0.0f;
    else
      v = (k & 1) ? s1 : 1.0f;
    *reinterpret_cast<__half*>(Asm + kmaj_off(y, k)) = __float2half_rn(v);
  }
  // B operand, coupling columns (same in every stage)
  for (int e = tid; e < kTcN * 7; e += kTcThreads) {
    int u = e / 7, i = e % 7;
    const double* row = Ws + (n - 9 - i) * n;
    double v = 0.0;
    for (int j = 0; j < 8; ++j)
      if ((u >> j) & 1) v += row[n - 1 - j];
    __half2 dg = digits((float)v, exact);
    for (int s = 0; s < kTcBStages; ++s)
      *reinterpret_cast<__half2*>(Bsm + s * kTcN * 32 + kmaj_off(u, 2 * i)) = dg;
  }
  for (int u = tid; u < kTcN; u += kTcThreads) {
    double e = 0.0;
    for (int j = 0; j < 8; ++j) {
      if (!((u >> j) & 1)) continue;
      const double* row = Ws + (n - 1 - j) * n;
      e += row[n - 1 - j];
      for (int j2 = 0; j2 < j; ++j2)
        if ((u >> j2) & 1) e += row[n - 1 - j2];
    }
    EU[u] = (float)e;
  }
  for (int y = tid; y < 128; y += kTcThreads) {
    double e = 0.0;
    for (int i = 0; i < 7; ++i) {
      if (!((y >> i) & 1)) continue;
      const double* row = Ws + (n - 9 - i) * n;
      e += row[n - 9 - i];
      for (int i2 = 0; i2 < i; ++i2)
        if ((y >> i2) & 1) e += row[n - 9 - i2];
    }
    EY[y] = (float)e;
  }
  for (int e = tid; e < 32 * 16; e += kTcThreads) {
    const int p = e >> 4, c = e & 15;
    double v = 0.0;
    if (c == 15) {
      for (int k = 0; k < 5; ++k) {
        if (!((p >> k) & 1)) continue;
        const double* row = Ws + (n - 16 - k) * n;
        v += row[n - 16 - k];
        for (int k2 = 0; k2 < k; ++k2)
          if ((p >> k2) & 1) v += row[n - 16 - k2];
      }
    } else {
      const int col = c < 8 ? n - 1 - c : n - 9 - (c - 8);
      for (int k = 0; k < 5; ++k)
        if ((p >> k) & 1) v += Ws[(n - 16 - k) * n + col];
    }
    LO[e] = v;
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t npairs = (uint32_t)(ntiles >> 1);

  bool ok = true;
  if (warp == 0 && P.stall) {
    // test hook (QB_FLAG_TEST_STALL): nothing is published, every other wait runs out
  } else if (warp == 0) {
    // ------------------------------------------------------------ tile walk (every tile)
    const int nh = nt - 5;
    double fh[8], gh[7], c[5], eh = 0.0, h0 = 0.0, h1 = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) fh[k] = 0.0;
#pragma unroll
    for (int k = 0; k < 7; ++k) gh[k] = 0.0;
#pragma unroll
    for (int k = 0; k < 5; ++k) c[k] = 0.0;
    const uint64_t th0 = t0 >> 5;
    for (int m = 0; m < nh; ++m) {
      if (!((th0 >> m) & 1)) continue;
      const double* row = Ws + (n - 21 - m) * n;
      eh += row[n - 21 - m];
      for (int m2 = 0; m2 < m; ++m2)
        if ((th0 >> m2) & 1) eh += row[n - 21 - m2];
      if (lane < nh && lane != m) h0 += row[n - 21 - lane];
      if (lane + 32 < nh && lane + 32 != m) h1 += row[n - 21 - lane - 32];
#pragma unroll
      for (int k = 0; k < 8; ++k) fh[k] += row[n - 1 - k];
#pragma unroll
      for (int k = 0; k < 7; ++k) gh[k] += row[n - 9 - k];
#pragma unroll
      for (int k = 0; k < 5; ++k) c[k] += row[n - 16 - k];
    }
    for (uint64_t j0 = 0; j0 < ntiles && ok; j0 += 32) {
      const uint64_t i0 = i_begin + j0;
      if (j0 > 0) {
        const int kb = __ffsll((long long)i0) - 1;
        const int m = kb - 5;
        const double sg = ((gray64(i0) >> kb) & 1) ? 1.0 : -1.0;
        const double hm = __shfl_sync(0xffffffffu, m < 32 ? h0 : h1, m & 31);
        const double* row = Ws + (n - 21 - m) * n;
        eh += sg * (row[n - 21 - m] + hm);
        if (lane < nh && lane != m) h0 += sg * row[n - 21 - lane];
        if (lane + 32 < nh && lane + 32 != m) h1 += sg * row[n - 21 - lane - 32];
#pragma unroll
        for (int k = 0; k < 8; ++k) fh[k] += sg * row[n - 1 - k];
#pragma unroll
        for (int k = 0; k < 7; ++k) gh[k] += sg * row[n - 9 - k];
#pragma unroll
        for (int k = 0; k < 5; ++k) c[k] += sg * row[n - 16 - k];
      }
      const uint64_t j = j0 + (uint64_t)lane;
      const int tl = (int)(gray64(i0 + (uint64_t)lane) & 31ull);
      const double* lo = LO + tl * 16;
      double et = eh + lo[15];
#pragma unroll
      for (int k = 0; k < 5; ++k)
        if ((tl >> k) & 1) et += c[k];
      const int s = (int)(j % kTcParamSlots);
      ok = mbar_wait(&p_empty[s], (uint32_t)(((j / kTcParamSlots) & 1) ^ 1), abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      TcSlot& sl = slots[s];
#pragma unroll
      for (int k = 0; k < 8; ++k) sl.f[k] = (float)(fh[k] + lo[k]);
#pragma unroll
      for (int k = 0; k < 7; ++k) sl.g[k] = (float)(gh[k] + lo[8 + k]);
      sl.et = (float)et;
      mbar_arrive(&p_full[s]);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issue (one per pair)
    if (lane == 0) {
      const uint64_t adesc = umma_desc(smem_u32(Asm), 128, 256);
      const uint64_t bdesc0 = umma_desc(smem_u32(Bsm), 128, 256);
      for (uint32_t p0 = 0; p0 < npairs && ok; p0 += kTcBStages) {
        const uint32_t pb = (p0 >> 3) & 1u;
#pragma unroll
        for (int k = 0; k < kTcBStages; ++k) {
          const uint32_t as = (uint32_t)k & 1u;
          ok = mbar_wait(&b_full[k], pb, abort_flag) &&
               mbar_wait_short(&acc_empty[as], (((uint32_t)k >> 1) & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (p0 + (uint32_t)k >= (uint32_t)kTcStages) mbar_arrive(&b_empty[(k + kTcBStages - kTcStages) % kTcBStages]);
          tc_mma(tmem + as * (uint32_t)kTcN, adesc, bdesc0 + (uint64_t)(k * (kTcN * 32 / 16)));
          tc_commit(&acc_full[as]);
          // the second arrival on acc_full: this thread has seen the B stage full, so the
          // epilogue's acquire of acc_full also orders the row terms written with the stage
          mbar_arrive(&acc_full[as]);
        }
      }
    }
    __syncwarp();
  } else if (warp < 4) {
    // ------------------------------------------------------------ B producers (per pair)
    // warp 2 + (p & 1) fills pair p: the C_t(u) digits of tile 2p (rows u = lane + 32 r) and
    // the row terms of tiles 2p and 2p + 1 (rows y = lane + 32 r)
    for (uint32_t p = (uint32_t)(warp - 2); p < npairs && ok; p += 2) {
      const uint32_t ja = 2 * p, jb = ja + 1;
      const uint32_t sa = ja & (uint32_t)(kTcParamSlots - 1), sb = jb & (uint32_t)(kTcParamSlots - 1);
      const uint32_t bs = p & (uint32_t)(kTcBStages - 1);
      ok = mbar_wait(&p_full[sa], (ja >> 6) & 1u, abort_flag) && mbar_wait(&p_full[sb], (jb >> 6) & 1u, abort_flag);
      if (!ok) break;
      __half2 dg[8];
      float ra[4], rb[4];
      {
        const TcSlot& sl = slots[sa];
        float s5 = 0.f;
#pragma unroll
        for (int jb5 = 0; jb5 < 5; ++jb5)
          if ((lane >> jb5) & 1) s5 += sl.f[jb5];
        const float f5 = sl.f[5], f6 = sl.f[6], f7 = sl.f[7];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          float cr = s5;
          if (r & 1) cr += f5;
          if (r & 2) cr += f6;
          if (r & 4) cr += f7;
          dg[r] = digits(EU[lane + 32 * r] + cr, exact);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const TcSlot& sl = slots[h ? sb : sa];
        float g5 = sl.et;
#pragma unroll
        for (int i = 0; i < 5; ++i)
          if ((lane >> i) & 1) g5 += sl.g[i];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          float v = g5;
          if (r & 1) v += sl.g[5];
          if (r & 2) v += sl.g[6];
          (h ? rb : ra)[r] = v + EY[lane + 32 * r];
        }
      }
      ok = mbar_wait(&b_empty[bs], ((p >> 3) & 1u) ^ 1u, abort_flag);
      if (!ok) break;
      unsigned char* Bst = Bsm + bs * kTcN * 32;
#pragma unroll
      for (int r = 0; r < 8; ++r) *reinterpret_cast<__half2*>(Bst + kmaj_off(lane + 32 * r, 14)) = dg[r];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        Rs[bs * 128 + lane + 32 * r] = ra[r];
        Rs2[bs * 128 + lane + 32 * r] = rb[r];
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&b_full[bs]);
        mbar_arrive(&p_empty[sa]);
        mbar_arrive(&p_empty[sb]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3;
    const int cq = (warp - 4) >> 2;
    const int y = q * 32 + lane;
    const float inf = __int_as_float(0x7f800000);
    float rmin = inf;
    const uint32_t sp = (uint32_t)cq >> 1;   // pair parity = accumulator stage
    const uint32_t hh = (uint32_t)cq & 1u;   // column half: u bit 7
    const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + sp * (uint32_t)kTcN + hh * 128u;
    // gamma of u bits 5..7 for the four 32-column chunks of this half
    float ghi[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) ghi[c] = ((c & 1) ? Q.whi[0] : 0.f) + ((c & 2) ? Q.whi[1] : 0.f) + (hh ? Q.whi[2] : 0.f);
    // records every 2^gl tiles = 2^(gl-1) pairs, 2^(gl-2) of this warp's parity
    uint32_t rec_left = 1u << (gl - 2);
    uint32_t Jrec = 0;
    for (uint32_t p = sp; p < npairs && ok; p += 2) {
      const uint32_t bs = p & (uint32_t)(kTcBStages - 1);
      // s = +1 when tile 2p has t bit 0 clear (its partner sets the bit); i_begin is even
      const float s = (((i_begin >> 1) + p) & 1ull) ? -1.0f : 1.0f;
      // acc_full completes after the MMA thread saw this pair's B stage full
      ok = mbar_wait(&acc_full[sp], (p >> 1) & 1u, abort_flag);
      if (!ok) break;
      const float R1 = Rs[bs * 128 + y];
      const float R2 = Rs2[bs * 128 + y];
      tc_fence_after();
      uint32_t ra[32], rb[32];
      QB_TC_LD32(tbase, ra);
      QB_TC_LD32(tbase + 32, rb);
      tc_wait_ld();
      reg_fence32(ra);
      reg_fence32(rb);
      float m1 = fminf(min32(ra), min32(rb));
      float m2 = fminf(fmaf(ghi[0], s, min32_shift(ra, Q, s)), fmaf(ghi[1], s, min32_shift(rb, Q, s)));
      QB_TC_LD32(tbase + 64, ra);
      QB_TC_LD32(tbase + 96, rb);
      tc_wait_ld();
      reg_fence32(ra);
      reg_fence32(rb);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[sp]);
      m1 = fminf(m1, fminf(min32(ra), min32(rb)));
      m2 = fmin3(m2, fmaf(ghi[2], s, min32_shift(ra, Q, s)), fmaf(ghi[3], s, min32_shift(rb, Q, s)));
      rmin = fmin3(rmin, m1 + R1, m2 + R2);
      if (--rec_left == 0) {
        const float wm = warp_min_f(rmin) * P.inv_scale;
        if (lane == 0) {
          float* dst = rec + (((uint64_t)Jrec << 3) | ((uint64_t)hh << 2) | (uint64_t)q);
          if (wm >= 0.f)
            atomicMin(reinterpret_cast<int*>(dst), __float_as_int(wm));
          else
            atomicMax(reinterpret_cast<unsigned*>(dst), __float_as_uint(wm));
        }
        ++Jrec;
        rec_left = 1u << (gl - 2);
        rmin = inf;
      }
    }
  }
  if (!ok) {
    *abort_flag = 1;
    atomicOr(P.err, kErrTimeout);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}


// The 16-bit pair form.  kItems = false: one problem, each CTA a contiguous run of its record
// blocks (one work item), its constants in Q.tab; kItems = true: the CTA's list of work items
// (runs of record blocks of the batch's problems, qb_batch.cuh), Q.tabs[it] the constants of
// item it's problem, as tc_pass1_kernel<true> does for one state per accumulator.
//
// A block is 2^(kTc2Low + 1) tiles that share every t bit above the lowest kTc2Low + 1 (block K:
// t >> (kTc2Low + 1) = gray(K)); its 2^kTc2Low pairs share one B stage, because t bits
// 1 .. kTc2Low are K slots of the MMA: B holds their couplings with u (two exact digits each,
// the same in every stage) and there is one constant A operand per setting of them.  The block
// walk and the B producer thus run once per 16 tiles.  A row's term of tile t is the block's
// (written with the stage) plus a constant table of the low t bits' couplings with y plus the
// low bits' energy in this block.  Every pair is two N = 128 MMAs, one per column half, into
// one of four 128-column accumulators, each owned by one group of four epilogue warps (group
// g: pairs of parity g >> 1, column half g & 1): an accumulator is released by its own four
// warps right after their loads, and its next MMA completes while they take the minima.
//
// Roles (20 warps): warp 0 block walk (FP64), warp 2 B producer, warps 1 and 3 MMA issue (even
// and odd pairs; elected lane, warp-uniform control flow so that descriptors and addresses stay
// in uniform registers), warps 4-19 the epilogue.  Between a batch's items all roles meet at a
// CTA barrier with the pipelines empty (every MMA has been waited for by its epilogue warps),
// so the per-item tables, B operand columns and constants can be rewritten; barrier slots, B
// stages and phases follow the CTA-wide block counter bbase.  W is taken in the
// problem's units (times scale as it is loaded: sigma off the exact path).
//
// What bounds it: the epilogue's ALU work.  Per warp and 8192 states 72 packed minima and 2
// float minima of 88 ALU instructions (half rate: 176 of the measured 225 cycles per scheduler,
// 0.78 busy); register reads (about 1.8 operands per cycle and scheduler) allow the 16
// corrections and the row terms beside them, but not one more add per register.  Measured
// (n = 36, 2^36 states, the kernel alone): 1.75 ms (1.72-1.77 between cards), against 2.36 ms with one B stage and one
// N = 256 MMA per pair, issued by one thread of a divergent warp.  On the way: the low t bits
// in the A operand with one MMA issuer 2.66; uniform MMA issue 2.33; two issuers and the
// epilogue's four pairs per block unrolled 2.03; waits without a result register, u16 -> f32
// conversions instead of byte permutes 1.97; corrections read from shared memory at their use
// instead of held in 16 registers 1.87; warp index by shuffle (uniform), elected arrivals 1.79;
// one x64 TMEM load instead of four x16 1.73.  Dropped: walking t bits 1.. in the epilogue by
// one packed add per register from a shared-memory table (2.18-2.31; each such step costs 262
// cycles against 196 from TMEM, the register read ports), each group issuing its own MMA
// behind a named barrier (2.37), three groups on a ring of four accumulators (2.33), one N =
// 256 MMA per pair (2.03 at the 2.00 stage), 3.5 instead of 4 minima per 8 inputs by moving
// the odd input behind the correction (1.80 against 1.75), corrections as constant operands
// (1.83-1.90), two groups of four warps with two accumulators each and the next unit's load in
// flight (12 warps, 165 registers: 2.01-2.09), row terms inside the MMA so that corrections and
// conversions run once per block (1.79: its second K slice costs what they save).
template <bool kItems>
__global__ void __launch_bounds__(kTc2Threads, 1) tc_pair_kernel(const __grid_constant__ Tc2Params Q) {
  constexpr int KW = kTc2Low, NS = 1 << KW;  // low t bits per block, pairs per block
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  const TcParams& P = Q.P;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform to the compiler
  const Tc2Layout L = tc2_layout(kItems ? P.n_max : P.n);  // only the W block grows with n
  unsigned char* Asm = tc_smem + L.a_off;
  unsigned char* Bsm = tc_smem + L.b_off;
  uint64_t* p_full = reinterpret_cast<uint64_t*>(tc_smem + L.bar_off);
  uint64_t* p_empty = p_full + kTcParamSlots;
  uint64_t* b_full = p_empty + kTcParamSlots;
  uint64_t* b_empty = b_full + kTc2BStages;
  uint64_t* acc_full = b_empty + kTc2BStages;
  uint64_t* acc_empty = acc_full + kTc2Groups;
  Tc2Slot* slots = reinterpret_cast<Tc2Slot*>(tc_smem + L.slot_off);
  uint32_t* Ct = reinterpret_cast<uint32_t*>(tc_smem + L.ct_off);    // corr_t[8], corr_p[hh][8]
  float2* WL = reinterpret_cast<float2*>(tc_smem + L.wl_off);        // [pair][row]: low t bits x y couplings
  float* LL = reinterpret_cast<float*>(tc_smem + L.ll_off);          // energies of the low t bits alone
  float* EU = reinterpret_cast<float*>(tc_smem + L.eu_off);
  float* EY = reinterpret_cast<float*>(tc_smem + L.ey_off);
  float* Rs = reinterpret_cast<float*>(tc_smem + L.rs_off);          // per B stage: row terms of the block
  float* Es = reinterpret_cast<float*>(tc_smem + L.es_off);          // ring of kTc2EsRing blocks: energy of low pattern 2 s + b
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tc_smem + L.misc_off);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tc_smem + L.misc_off + 4);
  double* LO = reinterpret_cast<double*>(tc_smem + L.lo_off);
  double* Ws = reinterpret_cast<double*>(tc_smem + L.w_off);

  // this CTA's work: one run of record blocks of one problem, or a list of items
  uint32_t it_lo = 0, it_hi = 1;
  TcItem one{};
  if (kItems) {
    it_lo = P.item_first[blockIdx.x];
    it_hi = P.item_first[blockIdx.x + 1];
    if (it_lo >= it_hi) return;  // uniform per CTA
  } else {
    const uint64_t g0 = (uint64_t)blockIdx.x * P.groups_per_cta;
    if (g0 >= P.groups) return;  // uniform per CTA
    const uint64_t g1 = min(P.groups, g0 + P.groups_per_cta);
    one = TcItem{P.W, P.rec + (g0 << 3), P.tile_begin + (g0 << P.gl), (g1 - g0) << P.gl, P.n, P.gl, P.exact,
                 P.inv_scale, P.scale};
  }

  // the item's W into shared memory, its records to +infinity, its corrections
  auto load_item = [&](uint32_t it) {
    const TcItem I = kItems ? P.items[it] : one;
    const Tc2Tab& Tb = kItems ? Q.tabs[it] : Q.tab;
    for (int i = tid; i < I.n * I.n; i += kTc2Threads) Ws[i] = I.W[i] * I.scale;
    for (uint64_t r = (uint64_t)tid; r < ((I.ntiles >> I.gl) << 3); r += kTc2Threads) I.rec[r] = __int_as_float(0x7f800000);
    if (tid < 24) Ct[tid] = tid < 8 ? Tb.corr_t[0][tid] : Tb.corr_p[0][(tid - 8) >> 3][tid & 7];
  };
  if (tid < kTcParamSlots) {
    mbar_init(&p_full[tid], 1);
    mbar_init(&p_empty[tid], 1);
    if (tid < kTc2BStages) {
      mbar_init(&b_full[tid], 1);
      mbar_init(&b_empty[tid], 4 * kTc2Groups);  // every epilogue warp
    }
    if (tid < kTc2Groups) {
      mbar_init(&acc_full[tid], 1);
      mbar_init(&acc_empty[tid], 4);
    }
    if (tid == 0) *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // A operands (constant, the same for every item), one per low pattern st: A[y][i] = y_i
  // (i < 7); the column term's digits (slots 8-10) 1, 2048, 32768; low t bit m (slots
  // tc2_low_slot(m, 0) and (m, 1)) bit m of st times 1, 2048
  load_item(it_lo);
  for (int e = tid; e < NS * 128 * 2; e += kTc2Threads) {  // 8 columns (16 bytes) at a time
    const int st = e >> 8, y = (e >> 1) & 127, kh = e & 1;
    constexpr uint32_t h1 = 0x3C00u, h2048 = 0x6800u, h32768 = 0x7800u;  // f16 1, 2048, 32768
    uint32_t w[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t h[2];
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        const int kl = 2 * c + d, kg = 8 + kl;  // column kl, or kg in the upper half
        const uint32_t lo = kl < 7 ? (((y >> kl) & 1) ? h1 : 0u) : (((st >> tc2_low_bit(7)) & 1) ? h2048 : 0u);
        const uint32_t hi = kg == 8 ? h1
                            : kg == 9 ? h2048
                            : kg == 10 ? h32768
                                       : (((st >> tc2_low_bit(kg)) & 1) ? (tc2_low_digit(kg) ? h2048 : h1) : 0u);
        h[d] = kh ? hi : lo;
      }
      w[c] = h[0] | (h[1] << 16);
    }
    *reinterpret_cast<uint4*>(Asm + st * 128 * 32 + kmaj_off(y, kh * 8)) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  uint32_t bnext = 0;  // CTA-wide block counter of the next item
  for (uint32_t it = it_lo; it < it_hi; ++it) {
    const TcItem I = kItems ? P.items[it] : one;
    const Tc2Tab& Tb = kItems ? Q.tabs[it] : Q.tab;
    const int n = I.n, gl = I.gl;
    const uint64_t k_begin = I.i_begin >> (KW + 1);             // first block
    const uint32_t nblk = (uint32_t)(I.ntiles >> (KW + 1));
    float* rec = I.rec;
    // the CTA-wide block counter at the item's start (a compile-time 0 for one problem)
    const uint32_t bbase = kItems ? bnext : 0u;

    // ------------------------------------------------------------ per-item set-up
    // Tables from W, FP64, without branches on the patterns' bits; different warps build
    // different ones.  (n = 20: the whole kernel 31 -> 18 thousand cycles.)
    const int kb0 = n - 17 - KW;  // variable of block bit 0 (block bit k: kb0 - k)
    if (warp < 8) {
      // column u = tid: E_U(u), and the B operand's constant rows -- the couplings of the y
      // variables (one exact fp16 integer each) and of the low t bits (two exact digits each);
      // half of what the rows' rounding leaves over goes to E_U
      const int u = tid;
      double e = 0.0, left = 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const double* row = Ws + (n - 1 - j) * n;
        double r = row[n - 1 - j];
#pragma unroll
        for (int j2 = 0; j2 < j; ++j2) r += ((u >> j2) & 1) ? row[n - 1 - j2] : 0.0;
        e += ((u >> j) & 1) ? r : 0.0;
      }
      unsigned char* Bu = Bsm + kmaj_off(u, 0);
#pragma unroll
      for (int i = 0; i < 10; ++i) {  // i < 7: y variable i; else low t bit i - 7
        const double* row = Ws + (i < 7 ? n - 9 - i : n - 17 - (i - 7)) * n;
        double v = 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) v += ((u >> j) & 1) ? row[n - 1 - j] : 0.0;
        const double w = rint(v);
        left += v - w;
        const float r = (float)w;
        const float d1 = i < 7 ? 0.f : floorf(r * (1.0f / 2048.0f));
        const __half h0 = __float2half_rn(fmaf(-2048.0f, d1, r)), h1 = __float2half_rn(d1);
#pragma unroll
        for (int s = 0; s < kTc2BStages; ++s) {
          unsigned char* Bs = Bu + s * kTcN * 32;
          *reinterpret_cast<__half*>(Bs + kmaj_off(0, i < 7 ? i : tc2_low_slot(i - 7, 0))) = h0;
          if (i >= 7) *reinterpret_cast<__half*>(Bs + kmaj_off(0, tc2_low_slot(i - 7, 1))) = h1;
        }
      }
      EU[u] = (float)(e + 0.5 * left);
    } else if (warp < 12) {
      // low t bits (pattern p = 2 st + b: bit 0 the pair's) x row couplings, y = tid - 256
      const int y = tid - 256;
      double r[KW + 1], v[2 * NS];
#pragma unroll
      for (int m = 0; m <= KW; ++m) {
        const double* row = Ws + (n - 16 - m) * n;
        r[m] = 0.0;
#pragma unroll
        for (int i = 0; i < 7; ++i) r[m] += ((y >> i) & 1) ? row[n - 9 - i] : 0.0;
      }
      v[0] = 0.0;
#pragma unroll
      for (int m = 0; m <= KW; ++m)
#pragma unroll
        for (int p = 0; p < (1 << m); ++p) v[(1 << m) + p] = v[p] + r[m];
#pragma unroll
      for (int st = 0; st < NS; ++st) WL[st * 128 + y] = make_float2((float)v[2 * st], (float)v[2 * st + 1]);
    } else if (warp < 16) {
      const int y = tid - 384;
      double e = 0.0;
#pragma unroll
      for (int i = 0; i < 7; ++i) {
        const double* row = Ws + (n - 9 - i) * n;
        double r = row[n - 9 - i];
#pragma unroll
        for (int i2 = 0; i2 < i; ++i2) r += ((y >> i2) & 1) ? row[n - 9 - i2] : 0.0;
        e += ((y >> i) & 1) ? r : 0.0;
      }
      EY[y] = (float)e;
      if (y < 2 * NS) {  // energy of the low t bits' pattern y alone
        double v = 0.0;
#pragma unroll
        for (int m = 0; m <= KW; ++m) {
          const double* row = Ws + (n - 16 - m) * n;
          double r = row[n - 16 - m];
#pragma unroll
          for (int m2 = 0; m2 < m; ++m2) r += ((y >> m2) & 1) ? row[n - 16 - m2] : 0.0;
          v += ((y >> m) & 1) ? r : 0.0;
        }
        LL[y] = (float)v;
      }
    } else {
      // LO[p]: the five lowest block bits' pattern p: couplings with u (8), y (7), the low t
      // bits (KW + 1) and their own energy (block bits beyond the problem's are never set)
      for (int e = tid - 512; e < 32 * kTc2LoCols; e += 128) {
        const int p = e & 31, c = e >> 5;
        double v = 0.0;
        if (c == kTc2LoCols - 1) {
#pragma unroll
          for (int b = 0; b < 5; ++b) {
            if (b > kb0) break;
            const double* row = Ws + (kb0 - b) * n;
            double r = row[kb0 - b];
#pragma unroll
            for (int b2 = 0; b2 < b; ++b2) r += ((p >> b2) & 1) ? row[kb0 - b2] : 0.0;
            v += ((p >> b) & 1) ? r : 0.0;
          }
        } else {
          const int col = c < 8 ? n - 1 - c : c < 15 ? n - 9 - (c - 8) : n - 16 - (c - 15);
#pragma unroll
          for (int b = 0; b < 5; ++b) {
            if (b > kb0) break;
            v += ((p >> b) & 1) ? Ws[(kb0 - b) * n + col] : 0.0;
          }
        }
        LO[p * kTc2LoCols + c] = v;
      }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    bool ok = true;
    const uint32_t abort_addr = smem_u32(tmem_slot) + 4u;
    uint32_t fail = 0u;
    if (warp == 0 && P.stall) {
      // test hook (QB_FLAG_TEST_STALL): nothing is published, every other wait runs out
    } else if (warp == 0) {
      // ---------------------------------------------------------- block walk (32 blocks at a time)
      // lane = the five lowest bits of the block index; the bits above are one Gray walk
      const int nh = kb0 + 1 - 5;  // block bits above the lanes' five: variables kb0 - 5 - m
      double fh[8], gh[7], ch[KW + 1], c[5], eh = 0.0, h0 = 0.0, h1 = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) fh[k] = 0.0;
#pragma unroll
      for (int k = 0; k < 7; ++k) gh[k] = 0.0;
#pragma unroll
      for (int k = 0; k <= KW; ++k) ch[k] = 0.0;
#pragma unroll
      for (int k = 0; k < 5; ++k) c[k] = 0.0;
      const uint64_t kc0 = k_begin >> 5, kc1 = (k_begin + nblk + 31) >> 5;
      const uint64_t th0 = gray64(kc0);
      for (int m = 0; m < nh; ++m) {
        if (!((th0 >> m) & 1)) continue;
        const int vm = kb0 - 5 - m;
        const double* row = Ws + vm * n;
        eh += row[vm];
        for (int m2 = 0; m2 < m; ++m2)
          if ((th0 >> m2) & 1) eh += row[kb0 - 5 - m2];
        if (lane < nh && lane != m) h0 += row[kb0 - 5 - lane];
        if (lane + 32 < nh && lane + 32 != m) h1 += row[kb0 - 5 - lane - 32];
#pragma unroll
        for (int k = 0; k < 8; ++k) fh[k] += row[n - 1 - k];
#pragma unroll
        for (int k = 0; k < 7; ++k) gh[k] += row[n - 9 - k];
#pragma unroll
        for (int k = 0; k <= KW; ++k) ch[k] += row[n - 16 - k];
#pragma unroll
        for (int k = 0; k < 5; ++k) c[k] += row[kb0 - k];
      }
      for (uint64_t kc = kc0; kc < kc1 && ok; ++kc) {
        if (kc > kc0) {
          const int m = __ffsll((long long)kc) - 1;
          const double sg = ((gray64(kc) >> m) & 1) ? 1.0 : -1.0;
          const double hm = __shfl_sync(0xffffffffu, m < 32 ? h0 : h1, m & 31);
          const int vm = kb0 - 5 - m;
          const double* row = Ws + vm * n;
          eh += sg * (row[vm] + hm);
          if (lane < nh && lane != m) h0 += sg * row[kb0 - 5 - lane];
          if (lane + 32 < nh && lane + 32 != m) h1 += sg * row[kb0 - 5 - lane - 32];
#pragma unroll
          for (int k = 0; k < 8; ++k) fh[k] += sg * row[n - 1 - k];
#pragma unroll
          for (int k = 0; k < 7; ++k) gh[k] += sg * row[n - 9 - k];
#pragma unroll
          for (int k = 0; k <= KW; ++k) ch[k] += sg * row[n - 16 - k];
#pragma unroll
          for (int k = 0; k < 5; ++k) c[k] += sg * row[kb0 - k];
        }
        const uint64_t K = (kc << 5) | (uint64_t)lane;
        const bool mine = K >= k_begin && K < k_begin + nblk;
        const uint32_t jg = bbase + (uint32_t)(K - k_begin);  // CTA-wide block counter
        const int tl = (int)(gray64(K) & 31ull);
        const double* lo = LO + tl * kTc2LoCols;
        double et = eh + lo[kTc2LoCols - 1];
#pragma unroll
        for (int k = 0; k < 5; ++k)
          if ((tl >> k) & 1) et += c[k];
        const int s = (int)(jg % kTcParamSlots);
        if (mine) ok = mbar_wait_idle(&p_empty[s], (uint32_t)(((jg / kTcParamSlots) & 1) ^ 1), abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (mine) {
          Tc2Slot& sl = slots[s];
#pragma unroll
          for (int k = 0; k < 8; ++k) sl.f[k] = (float)(fh[k] + lo[k]);
#pragma unroll
          for (int k = 0; k < 7; ++k) sl.g[k] = (float)(gh[k] + lo[8 + k]);
#pragma unroll
          for (int k = 0; k <= KW; ++k) sl.c[k] = (float)(ch[k] + lo[15 + k]);
          sl.et = (float)et;
          mbar_arrive(&p_full[s]);
        }
        __syncwarp();
      }
    } else if (warp == 1 || warp == 3) {
      // ---------------------------------------------------------- MMA issue: warp 1 the even, warp 3 the odd pairs
      const uint32_t par = (uint32_t)warp >> 1;
      const uint64_t adesc = umma_desc(smem_u32(Asm), 128, 256) + (uint64_t)(par * (128 * 32 / 16));
      const uint64_t bdesc0 = umma_desc(smem_u32(Bsm), 128, 256);
      const uint32_t d0 = tmem + par * 256u;
      const uint32_t full0 = smem_u32(&acc_full[2 * par]), empty0 = smem_u32(&acc_empty[2 * par]);
      for (uint32_t p = 0; p < nblk && !fail; ++p) {
        const uint32_t jg = bbase + p, bs = jg & (kTc2BStages - 1);
        mbar_wait_flag(smem_u32(&b_full[bs]), (jg / kTc2BStages) & 1u, abort_addr, fail);
        const uint64_t bd = bdesc0 + (uint64_t)(bs * (kTcN * 32 / 16));
#pragma unroll
        for (uint32_t v = 0; v < NS; ++v) {
          // pair 2 (v >> 1) + par, column half v & 1: use (NS / 2) jg + (v >> 1) of the accumulator
          mbar_wait_flag(empty0 + 8u * (v & 1u), ((v >> 1) & 1u) ^ 1u, abort_addr, fail);
          if (fail) break;
          tc_fence_after();
          tc_issue_n128(d0 + (v & 1u) * 128u, adesc + (uint64_t)((v >> 1) * (2 * 128 * 32 / 16)),
                        bd + (uint64_t)((v & 1u) * (128 * 32 / 16)), full0 + 8u * (v & 1u));
        }
      }
      ok = !fail;
    } else if (warp == 2) {
      // ---------------------------------------------------------- B producer (once per block)
      // X(u) + 2^23 - Dlow of the lane's columns u = lane + 32 r, by r & 3: u4 is lane bit 4
      float xk[4];
#pragma unroll
      for (int c = 0; c < 4; ++c)
        xk[c] = Tb.k0s[0] + ((lane >> 4) ? Tb.gx[0] : 0.f) + ((c & 1) ? Tb.gx[1] : 0.f) + ((c & 2) ? Tb.gx[2] : 0.f);
      for (uint32_t p = 0; p < nblk && ok; ++p) {
        const uint32_t jg = bbase + p;
        const uint32_t sa = jg & (uint32_t)(kTcParamSlots - 1), bs = jg & (uint32_t)(kTc2BStages - 1);
        // the lanes' waits end apart, at the limit with different results: all go on or none does
        ok = __all_sync(0xffffffffu, mbar_wait_idle(&p_full[sa], (jg / kTcParamSlots) & 1u, abort_flag));
        if (!ok) break;
        const Tc2Slot& sl = slots[sa];
        __half2 dg[8];
        __half dh[8];
        float ra[4], el;
        {
          float s5 = 0.f;
#pragma unroll
          for (int b = 0; b < 5; ++b)
            if ((lane >> b) & 1) s5 += sl.f[b];
          const float f5 = sl.f[5], f6 = sl.f[6], f7 = sl.f[7];
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            float cr = s5;
            if (r & 1) cr += f5;
            if (r & 2) cr += f6;
            if (r & 4) cr += f7;
            // the whole column term: an integer in (0, 2^24), three exact digits
            const float c = rintf(cr + EU[lane + 32 * r]) + xk[r & 3];
            const float d2 = floorf(c * (1.0f / 32768.0f)), rem = fmaf(-32768.0f, d2, c);
            const float d1 = floorf(rem * (1.0f / 2048.0f));
            dg[r] = __floats2half2_rn(fmaf(-2048.0f, d1, rem), d1);
            dh[r] = __float2half_rn(d2);
          }
          float g5 = sl.et;
#pragma unroll
          for (int i = 0; i < 5; ++i)
            if ((lane >> i) & 1) g5 += sl.g[i];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            float v = g5;
            if (r & 1) v += sl.g[5];
            if (r & 2) v += sl.g[6];
            ra[r] = v + EY[lane + 32 * r];
          }
          const int lp = lane & (2 * NS - 1);
          el = LL[lp];
#pragma unroll
          for (int m = 0; m <= KW; ++m)
            if ((lp >> m) & 1) el += sl.c[m];
        }
        ok = __all_sync(0xffffffffu, mbar_wait_idle(&b_empty[bs], ((jg / kTc2BStages) & 1u) ^ 1u, abort_flag));
        if (!ok) break;
        unsigned char* Bst = Bsm + bs * kTcN * 32;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          *reinterpret_cast<__half2*>(Bst + kmaj_off(lane + 32 * r, 8)) = dg[r];
          *reinterpret_cast<__half*>(Bst + kmaj_off(lane + 32 * r, 10)) = dh[r];
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) Rs[bs * 128 + lane + 32 * r] = ra[r];
        Es[(jg & (kTc2EsRing - 1)) * 32 + lane] = el;
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&b_full[bs]);
          mbar_arrive(&p_empty[sa]);
        }
      }
    } else {
      // ---------------------------------------------------------- epilogue (16-bit minima)
      const int q = warp & 3;                          // TMEM lane quarter
      const uint32_t grp = (uint32_t)(warp - 4) >> 2;  // accumulator: pairs of parity grp >> 1, column half grp & 1
      const uint32_t hh = grp & 1u;
      const int y = q * 32 + lane;
      const float inf = __int_as_float(0x7f800000);
      const float dmin = Tb.dmin, inv = I.inv_scale;
      const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + grp * 128u;
      const float2* wp = WL + (grp >> 1) * 128 + y;
      const uint2* ctp = reinterpret_cast<const uint2*>(Ct);
      const uint4* cpp = reinterpret_cast<const uint4*>(Ct + 8 + hh * 8);
      const int rsh = gl - KW - 1;  // blocks per record: 2^rsh
      float rmin = inf;
      uint32_t kmin = 0xffffffffu;  // smallest record value of this warp
      const uint32_t full = smem_u32(&acc_full[grp]);
      for (uint32_t p = 0; p < nblk && !fail; ++p) {
        const uint32_t jg = bbase + p, bs = jg & (uint32_t)(kTc2BStages - 1);
        // complete before the block's MMAs were issued; orders the row terms written with the stage
        mbar_wait_flag(smem_u32(&b_full[bs]), (jg / kTc2BStages) & 1u, abort_addr, fail);
        const float rb = Rs[bs * 128 + y] + dmin;
        const float2* ep = reinterpret_cast<const float2*>(Es + (jg & (kTc2EsRing - 1)) * 32) + (grp >> 1);
#pragma unroll
        for (uint32_t j = 0; j < NS / 2; ++j) {
          mbar_wait_flag(full, j & 1u, abort_addr, fail);
          tc_fence_after();
          uint32_t r[4][16];
          QB_TC_LD64P(tbase, r);
          tc_wait_ld();
#pragma unroll
          for (int c = 0; c < 4; ++c) reg_fence16(r[c]);
          tc_fence_before();
          __syncwarp();
          mbar_arrive_elect(smem_u32(&acc_empty[grp]));
          if (j == NS / 2 - 1) mbar_arrive_elect(smem_u32(&b_empty[bs]));  // the warp's last use of the B stage
          uint32_t m1 = 0u, v2[8];
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const uint32_t* a = r[b];
            const uint2 cc = ctp[b];
            const uint32_t t0 = uadd2(umin8(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]), cc.x);
            const uint32_t t1 = uadd2(umin8(a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15]), cc.y);
            m1 = b ? __vimin3_u16x2(m1, t0, t1) : umin2(t0, t1);
#pragma unroll
            for (int k = 0; k < 8; ++k) v2[k] = b ? __vimin3_u16x2(v2[k], a[k], a[k + 8]) : umin2(a[k], a[k + 8]);
          }
          const uint4 c0 = cpp[0], c1 = cpp[1];
          const uint32_t cp[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
          for (int k = 0; k < 8; ++k) v2[k] = uadd2(v2[k], cp[k]);
          const uint32_t m2 = umin8(v2[0], v2[1], v2[2], v2[3], v2[4], v2[5], v2[6], v2[7]);
          const float2 e2 = ep[2 * j], w2 = wp[2 * 128 * j];
          const float R1 = (rb + e2.x) + w2.x, R2 = (rb + e2.y) + w2.y;
          rmin = fmin3(rmin, u16lo_f(m1) + R1, u16hi_f(m1) + R1);
          rmin = fmin3(rmin, u16lo_f(m2) + R2, u16hi_f(m2) + R2);
        }
        if (((p + 1) >> rsh) != (p >> rsh)) {  // end of a record
          const float wm = warp_min_f(rmin) * inv;
          if (!kItems) kmin = min(kmin, f2key(wm));
          if (lane == 0) {
            float* dst = rec + (((uint64_t)(p >> rsh) << 3) | ((uint64_t)hh << 2) | (uint64_t)q);
            if (wm >= 0.f)
              atomicMin(reinterpret_cast<int*>(dst), __float_as_int(wm));
            else
              atomicMax(reinterpret_cast<unsigned*>(dst), __float_as_uint(wm));
          }
          rmin = inf;
        }
      }
      if (!kItems && lane == 0 && P.min_key) atomicMin(P.min_key, kmin);
      ok = !fail;
    }
    if (!ok) {
      *abort_flag = 1;
      atomicOr(P.err, kErrTimeout);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    bnext = bbase + nblk;
    if (*abort_flag) break;  // uniform: read after the barrier
    if (kItems && it + 1 < it_hi) {
      load_item(it + 1);
      __syncthreads();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}

// the pair-form search kernel (one persistent CTA per SM); gamma = couplings of variable
// n-16 with u bits 0..7, in the units of the scaled W
// W: n*n on the device; err: the error word (cleared); min_key: receives the smallest
// record value (16-bit form; initially 0xffffffff)
inline int tc2_launch(const TcPlan& p, const float* gamma, float* rec, const double* W, unsigned* err,
                      uint32_t* min_key, cudaStream_t st, int sms, int* kernels) {
  const uint64_t groups = (p.tile_end - p.tile_begin) >> p.gl;
  if (!groups) return 0;
  uint64_t ctas = std::min<uint64_t>((uint64_t)sms, groups);
  uint64_t gpc = (groups + ctas - 1) / ctas;
  ctas = (groups + gpc - 1) / gpc;
  if ((gpc << p.gl) >> 32) return 1;
  Tc2Params Q{};
  TcParams& P = Q.P;
  P.n = p.n;
  P.nt = p.nt;
  P.gl = p.gl;
  P.exact = p.exact ? 1 : 0;
  P.inv_scale = (float)(1.0 / p.scale);
  P.W = W;
  P.scale = p.scale;
  P.tile_begin = p.tile_begin;
  P.groups = groups;
  P.groups_per_cta = gpc;
  P.rec = rec;
  P.err = err;
  P.min_key = min_key;
  P.stall = p.stall ? 1 : 0;
  for (int k = 0; k < 32; ++k) {
    float g = 0.f;
    for (int j = 0; j < 5; ++j)
      if ((k >> j) & 1) g += gamma[j];
    Q.g5[k] = g;
  }
  Q.whi[0] = gamma[5];
  Q.whi[1] = gamma[6];
  Q.whi[2] = gamma[7];
  if (p.u16) tc2_u16_tables(gamma, p.dmin, &Q.tab);
  const TcSmemLayout L = tc_layout(p.n);
  const size_t smem = p.u16 ? tc2_smem_bytes(p.n) : std::max<size_t>(L.total + kTcBStages * 128 * 4, 120 * 1024) + 1024;
  auto* kern = p.u16 ? tc_pair_kernel<false> : tc_pair_fp32_kernel;
  kern<<<(unsigned)ctas, p.u16 ? kTc2Threads : kTcThreads, smem, st>>>(Q);
  ++*kernels;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
#endif

}  // namespace qb
