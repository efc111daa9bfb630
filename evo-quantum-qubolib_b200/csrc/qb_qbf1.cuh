// qb_qbf1.cuh -- QB_F1 with the reference's int16 arithmetic (opt-in).
//
// The reference's QB_F1 (src/qubo_lib/solvers/qbf1.py:86-133, 179-249, 253-289) keeps every
// energy in int16: the suffix table BB, the Gray-permuted prefix table AA, the cross table
// ABBA = (Q_0B + Q_1A^T) X_B^T and the running suffix sums all wrap modulo 2^16.  Where the
// partial sums of Q leave the int16 range its answer is not the true minimum.  This form
// reproduces that answer: because every int16 operation is exact modulo 2^16, each value the
// reference holds equals the exact integer quantity reduced modulo 2^16 to [-32768, 32767],
// so the tables are built from exact integers and the search repeats the reference's
// per-thread order (256 x 64 threads, 16 suffix columns each: column = block * 1024 +
// 64 * c + thread; Gray prefix steps; strict < keeps the earliest step; lowest thread wins;
// the suffix is then the first minimum of that prefix's int16 row).
//
// B = 18 suffix bits, A = n - 18 prefix bits (19 <= n <= 46).
#pragma once
#include "qb_common.cuh"

namespace qb {

constexpr int kQbf1B = 18;
constexpr int kQbf1Threads = 16384;  // the reference's grid: 256 blocks x 64 threads
constexpr int kQbf1MaxN = 46;

__device__ __forceinline__ int wrap16(int v) { return (int)(short)v; }

// The tables, one launch.  Blocks 0 .. 511: BB[s] and ABBA[k][s] (k < A) for every 18-bit suffix s
// (MSB-first: bit 17 - j of s is variable A + j), one block per value of the upper 9 suffix bits,
// whose sums (for BB, for every row k and for the fields of the lower 9 variables) its threads
// share; a thread adds the lower bits' for two neighbouring suffixes.  The other blocks: AA[i] =
// int16 of E_pre(gray(i)) (prefix bit A-1-k is variable k) in both halves of a word, 256 steps at
// a time, whose upper bits' sums are shared the same way.  Q: n x n int32 copy of the int16 matrix.
// A = 16: 11.7 us, against 11.7 + 9.4 us as two kernels with every prefix summed alone.
constexpr int kQbf1Lo = 9;
constexpr int kQbf1TableBlocks = 1 << (kQbf1B - kQbf1Lo);
inline size_t qbf1w_tables_smem(int n, int A) {
  return ((size_t)n * n + (size_t)A * (kQbf1Lo + 1) + kQbf1Lo * kQbf1Lo + kQbf1Lo + 1) * sizeof(int);
}
__device__ inline void qbf1w_prefix(const int* q, int n, int A, uint32_t* __restrict__ AA, int* sm) {
  int* lw = sm;        // [b][c]: couplings among the 8 lowest prefix bits, diagonal W_bb
  int* f = lw + 64;    // [b]: their fields from the upper bits; [8]: the upper bits' energy
  const int t = threadIdx.x, lane = t & 31;
  auto W = [&](int u, int v) { return u == v ? q[u * n + u] : q[u * n + v] + q[v * n + u]; };
  if (t < 64) lw[t] = (t >> 3) < A && (t & 7) < A ? W(A - 1 - (t >> 3), A - 1 - (t & 7)) : 0;
  const uint64_t steps = 1ull << A;
  const int nh = A - 8;  // upper bits: bit m is variable nh - 1 - m
  for (uint64_t g = blockIdx.x - kQbf1TableBlocks; (g << 8) < steps; g += gridDim.x - kQbf1TableBlocks) {
    const uint64_t hi = gray64(g);
    if (t < 64) {  // warp 0: the fields; warp 1: the energy, a bit per lane
      int v = 0;
      const int own = t < 32 ? (lane < 8 ? A - 1 - lane : -1) : (lane < nh && ((hi >> lane) & 1) ? nh - 1 - lane : -1);
      if (own >= 0) {
        if (t >= 32) v = W(own, own);
        for (int m = 0; m < (t < 32 ? nh : lane); ++m)
          if ((hi >> m) & 1) v += W(own, nh - 1 - m);
      }
      if (t >= 32) v = __reduce_add_sync(0xffffffffu, v);
      if (t < 8 || t == 32) f[t < 8 ? t : 8] = v;
    }
    __syncthreads();
    const uint64_t i = (g << 8) + (uint64_t)t;
    const int p = (int)(gray64(i) & 255ull);
    int e = f[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      int r = lw[b * 8 + b] + f[b];
#pragma unroll
      for (int c = 0; c < b; ++c) r += ((p >> c) & 1) ? lw[b * 8 + c] : 0;
      e += ((p >> b) & 1) ? r : 0;
    }
    if (i < steps) AA[i] = ((uint32_t)e & 0xffffu) * 0x10001u;
    __syncthreads();
  }
}
__global__ void __launch_bounds__(256) qbf1w_tables_kernel(const int* __restrict__ Q, int n, int A,
                                                           short* __restrict__ BB, short* __restrict__ ABBA,
                                                           uint32_t* __restrict__ AA) {
  extern __shared__ __align__(16) int q1_smem[];
  const int t = threadIdx.x;
  for (int i = t; i < n * n; i += blockDim.x) q1_smem[i] = Q[i];
  __syncthreads();
  if (blockIdx.x >= kQbf1TableBlocks) {  // uniform per block
    qbf1w_prefix(q1_smem, n, A, AA, q1_smem + n * n);
    return;
  }
  int* clo = q1_smem + n * n;            // [k][b]: couplings of row k with lower suffix bit b
  int* slo = clo + A * kQbf1Lo;          // [b][c]: couplings among the lower bits, diagonal W_bb
  int* chi = slo + kQbf1Lo * kQbf1Lo;    // [k]: row k's sum over the block's upper bits
  int* fhi = chi + A;                    // [b]: lower bit b's field from the upper bits; [9]: their energy
  const int hi = blockIdx.x;             // suffix bits 9 .. 17
  auto W = [&](int u, int v) { return u == v ? q1_smem[u * n + u] : q1_smem[u * n + v] + q1_smem[v * n + u]; };
  const int v0 = n - 1;                  // variable of suffix bit 0; bit b: v0 - b
  for (int i = t; i < A * kQbf1Lo; i += blockDim.x) clo[i] = W(i / kQbf1Lo, v0 - i % kQbf1Lo);
  for (int i = t; i < kQbf1Lo * kQbf1Lo; i += blockDim.x) slo[i] = W(v0 - i / kQbf1Lo, v0 - i % kQbf1Lo);
  for (int i = t; i < A + kQbf1Lo + 1; i += blockDim.x) {
    int s = 0;
    for (int b = 0; b < kQbf1Lo; ++b) {
      if (!((hi >> b) & 1)) continue;
      const int v = v0 - kQbf1Lo - b;
      if (i < A + kQbf1Lo)
        s += W(i < A ? i : v0 - (i - A), v);
      else
        for (int c = 0; c <= b; ++c)
          if ((hi >> c) & 1) s += W(v, v0 - kQbf1Lo - c);
    }
    chi[i] = s;
  }
  __syncthreads();
  const int lo = 2 * t;                  // this thread: suffixes (hi, lo) and (hi, lo + 1)
  int e0 = fhi[kQbf1Lo], d0 = slo[0] + fhi[0];
#pragma unroll
  for (int b = 1; b < kQbf1Lo; ++b) {
    if (!((lo >> b) & 1)) continue;
    e0 += slo[b * kQbf1Lo + b] + fhi[b];
    d0 += slo[b];
#pragma unroll
    for (int c = 1; c < b; ++c)
      if ((lo >> c) & 1) e0 += slo[b * kQbf1Lo + c];
  }
  const size_t at = (((size_t)hi << kQbf1Lo) + (size_t)lo) >> 1;
  reinterpret_cast<uint32_t*>(BB)[at] = ((uint32_t)e0 & 0xffffu) | ((uint32_t)(e0 + d0) << 16);
  for (int k = 0; k < A; ++k) {
    int c0 = chi[k];
    const int* ck = clo + k * kQbf1Lo;
#pragma unroll
    for (int b = 1; b < kQbf1Lo; ++b)
      if ((lo >> b) & 1) c0 += ck[b];
    reinterpret_cast<uint32_t*>(ABBA)[((size_t)k << (kQbf1B - 1)) + at] =
        ((uint32_t)c0 & 0xffffu) | ((uint32_t)(c0 + ck[0]) << 16);
  }
}

// packed int16 pairs: per-halfword add (wraps modulo 2^16) and signed minimum
__device__ __forceinline__ uint32_t add16x2(uint32_t x, uint32_t y) {
  uint32_t r;
  asm("add.u16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
  return r;
}
__device__ __forceinline__ uint32_t min16x2(uint32_t x, uint32_t y) {
  uint32_t r;
  asm("min.s16x2 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(y));
  return r;
}
// per halfword -x
__device__ __forceinline__ uint32_t neg16x2(uint32_t x) { return add16x2(~x, 0x00010001u); }

// signed minimum of 16 packed pairs
__device__ __forceinline__ uint32_t min16x2_16(const uint32_t* e) {
  const uint32_t a = __vimin3_s16x2(__vimin3_s16x2(e[0], e[1], e[2]), e[3], e[4]);
  const uint32_t b = __vimin3_s16x2(__vimin3_s16x2(e[5], e[6], e[7]), e[8], e[9]);
  const uint32_t c = __vimin3_s16x2(__vimin3_s16x2(e[10], e[11], e[12]), e[13], e[14]);
  return min16x2(__vimin3_s16x2(a, b, c), e[15]);
}

// signed minimum of 16 packed sums e + r, each wrapping modulo 2^16 (fused add-and-minimum)
__device__ __forceinline__ uint32_t addmin16x2_16(const uint32_t* e, const uint32_t* r) {
  uint32_t m = add16x2(e[0], r[0]);
#pragma unroll
  for (int c = 1; c < 16; ++c) m = __viaddmin_s16x2(e[c], r[c], m);
  return m;
}

// shared memory of the search kernel: +ABBA and -ABBA rows of the block's 1024 columns,
// two columns per 32-bit word
inline size_t qbf1w_search_smem(int A) { return (size_t)2 * A * 512 * sizeof(uint32_t); }

// steps a search key stands for: a chunk of at least 32 steps is walked in aligned groups of 32
// and reports the group of its best step, a shorter one the step itself
__host__ __device__ inline int qbf1w_group(uint64_t chunk_len) { return (chunk_len & 31) == 0 ? 32 : 1; }

// The search.  blockIdx.x = the reference block (64 threads, 1024 columns); a warp walks one chunk
// of Gray steps (8 per CTA, blockIdx.y) for all of the block's threads: lane l has the reference
// threads 2 l and 2 l + 1 in the halves of its words, word c their columns 64 c + t.  A step's
// minimum over the 16 columns is thus 16 packed values and needs no merging of halves before the
// AA entry is added.  Chunks of at least 32 steps are walked in aligned groups of 32, in which the
// flipped prefix bit and its direction are constants.  The words hold the state without prefix
// bits 0 and 1: four steps in a row share it, their minima are those of E, F = E + r0, F + r1 and
// E + r1 (rows in registers; a Gray group of four visits them in either direction), the last two
// by fused add-and-minimum without storing the sums, and only every fourth step updates the words
// (with the negated row where a variable is turned off).  All sums wrap like the reference's
// int16.  A group keeps only its minimum, and the exact step is found afterwards for the one
// thread that wins (qbf1w_final_kernel).  Each thread reports (best int16 value, its group) of
// its chunk into key[tid] by a 64-bit atomic min, which keeps the smallest value and, among equal
// values, the earliest group.
//
// What bounds it: the half-rate packed pipes (per step 13.8 ALU and 9.2 FMA-pipe instructions of 32
// states a lane: 72% and 48% of what they can take) with the register reads of the three-operand
// forms beside them.  2^34 states (n = 34): 565 us; all sums of two steps of four by fused
// add-and-minimum, F not stored, 575 us (80% of the ALU).  With a reference thread's column pairs
// in a word, every step's sums stored and the halves merged per step it was 722 us.
__global__ void __launch_bounds__(256, 2) qbf1w_search_kernel(int A, const short* __restrict__ BB,
                                                              const short* __restrict__ ABBA,
                                                              const uint32_t* __restrict__ AA, uint64_t chunk_len,
                                                              unsigned long long* __restrict__ key) {
  extern __shared__ __align__(16) uint32_t q1w_smem[];  // [2][A][16][32]: word (row k, column index c, lane)
  const int blk = blockIdx.x;
  for (int i = threadIdx.x; i < A * 128; i += blockDim.x) {
    const uint4 w = reinterpret_cast<const uint4*>(ABBA + ((size_t)(i >> 7) << kQbf1B) + (size_t)blk * 1024)[i & 127];
    reinterpret_cast<uint4*>(q1w_smem)[i] = w;
    reinterpret_cast<uint4*>(q1w_smem)[A * 128 + i] =
        make_uint4(neg16x2(w.x), neg16x2(w.y), neg16x2(w.z), neg16x2(w.w));
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint64_t chunk = (uint64_t)blockIdx.y * 8 + (threadIdx.x >> 5);
  const uint64_t steps = 1ull << A;
  const uint64_t i0 = chunk * chunk_len;
  if (i0 >= steps) return;
  const uint64_t i1 = min(steps, i0 + chunk_len);
  const uint32_t* pos = q1w_smem + lane;            // + row * 512 + c * 32
  const uint32_t* neg = q1w_smem + A * 512 + lane;
  uint32_t E2[16];
  {
    const uint64_t p0 = gray64(i0);
    const uint32_t* b = reinterpret_cast<const uint32_t*>(BB) + blk * 512 + lane;
#pragma unroll
    for (int c = 0; c < 16; ++c) E2[c] = b[c * 32];
    for (int k = 0; k < A; ++k)
      if ((p0 >> (A - 1 - k)) & 1) {
#pragma unroll
        for (int c = 0; c < 16; ++c) E2[c] = add16x2(E2[c], pos[k * 512 + c * 32]);
      }
  }
  int best[2];
  uint64_t bi[2] = {i0, i0};
  if ((chunk_len & 31) == 0) {
    best[0] = best[1] = 32768;  // above every int16
    uint32_t r0[16], r1[16];  // rows of prefix bits 0 and 1 (variables A-1, A-2)
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      r0[c] = pos[(A - 1) * 512 + c * 32];
      r1[c] = pos[(A - 2) * 512 + c * 32];
    }
    for (uint64_t ig = i0; ig < i1; ig += 32) {
      const uint4* aa = reinterpret_cast<const uint4*>(AA + ig);
      if (ig != i0) {  // the chunk's first step is its start state
        const int kb = __ffsll((long long)ig) - 1;  // >= 5
        const uint32_t* r = (((gray64(ig) >> kb) & 1) ? pos : neg) + (A - 1 - kb) * 512;
#pragma unroll
        for (int c = 0; c < 16; ++c) E2[c] = add16x2(E2[c], r[c * 32]);
      }
      const uint32_t* r4 = (((ig >> 5) & 1) ? neg : pos) + (A - 5) * 512;  // prefix bit 4: off in odd groups
      uint32_t gm = 0x7fff7fffu;
#pragma unroll
      for (int q = 0; q < 8; ++q) {  // four steps each
        const uint4 a = __ldg(aa + q);
        if (q) {
          const int kb = 2 + ctz5(q);
          const bool on = !((q >> (kb - 1)) & 1);
          const uint32_t* r = kb == 4 ? r4 : (on ? pos : neg) + (A - 1 - kb) * 512;
#pragma unroll
          for (int c = 0; c < 16; ++c) E2[c] = add16x2(E2[c], r[c * 32]);
        }
        // prefix bits (1, 0): 00, 01, 11, 10 where prefix bit 2 was last 0, else the reverse
        uint32_t F2[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) F2[c] = add16x2(E2[c], r0[c]);
        const uint32_t m00 = min16x2_16(E2), m01 = min16x2_16(F2), m11 = addmin16x2_16(F2, r1),
                       m10 = addmin16x2_16(E2, r1);
        gm = __vimin3_s16x2(gm, add16x2(m00, q & 1 ? a.w : a.x), add16x2(m01, q & 1 ? a.z : a.y));
        gm = __vimin3_s16x2(gm, add16x2(m11, q & 1 ? a.y : a.z), add16x2(m10, q & 1 ? a.x : a.w));
      }
      const int g[2] = {(int)(short)(gm & 0xffffu), (int)gm >> 16};
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (g[h] < best[h]) {  // strict: the earliest group keeps a tie
          best[h] = g[h];
          bi[h] = ig;
        }
    }
  } else {
    best[0] = best[1] = 32768;
    for (uint64_t i = i0; i < i1; ++i) {
      if (i != i0) {
        const int kb = __ffsll((long long)i) - 1;
        const uint32_t* r = (((gray64(i) >> kb) & 1) ? pos : neg) + (A - 1 - kb) * 512;
#pragma unroll
        for (int c = 0; c < 16; ++c) E2[c] = add16x2(E2[c], r[c * 32]);
      }
      const uint32_t tt = add16x2(min16x2_16(E2), AA[i]);
      const int g[2] = {(int)(short)(tt & 0xffffu), (int)tt >> 16};
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (g[h] < best[h]) {
          best[h] = g[h];
          bi[h] = i;
        }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
    atomicMin(key + blk * 64 + 2 * lane + h, ((unsigned long long)(best[h] + 32768) << 40) | (unsigned long long)bi[h]);
}

// The answer's parts, on the device: what the reference's host picks from the threads' results.
struct Qbf1Answer {
  unsigned long long row;  // (value + 32768) << 32 | suffix: first minimum of the winning prefix's row
  unsigned long long step; // the winning thread's best step
  int tid, best16;
  int found, pad;
};

// One block of 512 threads: the thread with the smallest value (the lowest among equals), then the
// first step of its reported group with that value: warp c evaluates the thread's column c at the
// group's 32 steps from the tables.
__global__ void __launch_bounds__(512) qbf1w_final_kernel(int A, const short* __restrict__ BB,
                                                          const short* __restrict__ ABBA, const uint32_t* __restrict__ AA,
                                                          const unsigned long long* __restrict__ key, int group,
                                                          Qbf1Answer* __restrict__ ans) {
  __shared__ unsigned long long red[16];
  __shared__ int val[16][32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  // (value << 14 | tid): tids have 14 bits, values 16
  unsigned long long b = ~0ull;
  for (int i = t; i < kQbf1Threads; i += 512) {
    const unsigned long long k = key[i];
    const unsigned long long c = k == ~0ull ? ~0ull : ((k >> 40) << 14) | (unsigned long long)i;
    b = c < b ? c : b;
  }
  for (int off = 16; off; off >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, b, off);
    b = o < b ? o : b;
  }
  if (lane == 0) red[warp] = b;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 16; ++w) b = red[w] < b ? red[w] : b;
  if (b == ~0ull) {  // uniform: no thread reported
    if (t == 0) ans->found = 0;
    return;
  }
  const int tid = (int)(b & 16383ull), best16 = (int)(b >> 14) - 32768;
  const uint64_t s0 = key[tid] & ((1ull << 40) - 1);
  const uint64_t st = s0 + (uint64_t)lane;
  const bool in = lane < group;
  int v = 32767;
  if (in) {
    const int col = (tid >> 6) * 1024 + 64 * warp + (tid & 63);
    const uint64_t p = gray64(st);
    v = BB[col];
#pragma unroll 8
    for (int k = 0; k < A; ++k) {
      const int w = ABBA[((size_t)k << kQbf1B) + col];
      v += ((p >> (A - 1 - k)) & 1) ? w : 0;
    }
    v = wrap16(v);
  }
  val[warp][lane] = v;
  __syncthreads();
  if (warp == 0) {
    for (int c = 1; c < 16; ++c) v = min(v, val[c][lane]);
    const bool hit = in && wrap16((int)(short)AA[in ? st : s0] + v) == best16;
    const unsigned h = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) {
      ans->step = s0 + (uint64_t)(h ? __ffs(h) - 1 : 0);
      ans->tid = tid;
      ans->best16 = best16;
      ans->found = h ? 1 : 0;
    }
  }
}

// int16 row of the winning prefix: first s with the smallest wrap16(BB[s] + sum of ABBA rows)
__global__ void __launch_bounds__(256) qbf1w_row_kernel(int A, const short* __restrict__ BB,
                                                        const short* __restrict__ ABBA, Qbf1Answer* __restrict__ ans) {
  __shared__ uint32_t red[8];
  const int s = blockIdx.x * 256 + threadIdx.x;  // the grid covers the 2^18 suffixes
  const uint64_t p = gray64(ans->step);
  int v = BB[s];
#pragma unroll 8
  for (int k = 0; k < A; ++k) {
    const int w = ABBA[(size_t)k * (1 << kQbf1B) + s];
    v += ((p >> (A - 1 - k)) & 1) ? w : 0;
  }
  // one atomic per block: (value, thread) in 24 bits
  uint32_t k = ((uint32_t)(wrap16(v) + 32768) << 8) | threadIdx.x;
  k = __reduce_min_sync(0xffffffffu, k);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = k;
  __syncthreads();
  if (threadIdx.x < 32) {
    k = __reduce_min_sync(0xffffffffu, threadIdx.x < 8 ? red[threadIdx.x] : 0xffffffffu);
    if (threadIdx.x == 0)
      atomicMin(&ans->row, ((unsigned long long)(k >> 8) << 32) | (unsigned long long)(blockIdx.x * 256 + (k & 255u)));
  }
}

}  // namespace qb
