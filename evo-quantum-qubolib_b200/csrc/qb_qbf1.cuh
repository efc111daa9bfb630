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

// BB[s] and ABBA[k][s] (k < A) for every 18-bit suffix s (MSB-first: bit 17 - j of s is
// variable A + j).  Q: n x n int32 copy of the int16 matrix.  One block per value of the upper 9
// suffix bits, whose sums (for BB, for every row k and for the fields of the lower 9 variables)
// its threads share; a thread adds the lower bits' for two neighbouring suffixes.  8 us at
// A = 16, against 32 us with every suffix summed alone.
constexpr int kQbf1Lo = 9;
inline size_t qbf1w_tables_smem(int n, int A) {
  return ((size_t)n * n + (size_t)A * (kQbf1Lo + 1) + kQbf1Lo * kQbf1Lo + kQbf1Lo + 1) * sizeof(int);
}
__global__ void __launch_bounds__(256) qbf1w_tables_kernel(const int* __restrict__ Q, int n, int A,
                                                           short* __restrict__ BB, short* __restrict__ ABBA) {
  extern __shared__ int q1_smem[];
  int* clo = q1_smem + n * n;            // [k][b]: couplings of row k with lower suffix bit b
  int* slo = clo + A * kQbf1Lo;          // [b][c]: couplings among the lower bits, diagonal W_bb
  int* chi = slo + kQbf1Lo * kQbf1Lo;    // [k]: row k's sum over the block's upper bits
  int* fhi = chi + A;                    // [b]: lower bit b's field from the upper bits; [9]: their energy
  const int t = threadIdx.x;
  const int hi = blockIdx.x;             // suffix bits 9 .. 17
  for (int i = t; i < n * n; i += blockDim.x) q1_smem[i] = Q[i];
  __syncthreads();
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

// AA[i] = int16 of E_pre(gray(i)) (prefix bit A-1-k is variable k)
__global__ void qbf1w_prefix_kernel(const int* __restrict__ Q, int n, int A, short* __restrict__ AA) {
  extern __shared__ int q1p_smem[];
  for (int i = threadIdx.x; i < A * A; i += blockDim.x) q1p_smem[i] = Q[(i / A) * n + (i % A)];
  __syncthreads();
  const uint64_t steps = 1ull << A;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < steps; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t p = gray64(i);
    int e = 0;
    for (int k = 0; k < A; ++k) {
      if (!((p >> (A - 1 - k)) & 1)) continue;
      for (int l = 0; l < A; ++l)
        if ((p >> (A - 1 - l)) & 1) e += q1p_smem[k * A + l];
    }
    AA[i] = (short)wrap16(e);
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
__device__ __forceinline__ uint32_t pack16(int lo, int hi) { return (uint32_t)(uint16_t)lo | ((uint32_t)(uint16_t)hi << 16); }

// shared memory of the search kernel: +ABBA and -ABBA rows of the block's 1024 columns,
// two columns per 32-bit word
inline size_t qbf1w_search_smem(int A) { return (size_t)2 * A * 512 * sizeof(uint32_t); }

// steps a search key stands for: a chunk of at least 32 steps is walked in aligned groups of 32
// and reports the group of its best step, a shorter one the step itself
__host__ __device__ inline int qbf1w_group(uint64_t chunk_len) { return (chunk_len & 31) == 0 ? 32 : 1; }

// signed minimum of 8 packed pairs
__device__ __forceinline__ uint32_t min16x2_8(const uint32_t* e) {
  return __vimin3_s16x2(__vimin3_s16x2(e[0], e[1], e[2]), __vimin3_s16x2(e[3], e[4], e[5]), min16x2(e[6], e[7]));
}

// The search.  blockIdx.x = the reference block (64 threads, 1024 columns), blockIdx.y picks
// 4 consecutive chunks of Gray steps; thread = (chunk lane, reference thread t).  Thread t's
// 16 columns 64 c + t are held as 8 int16 pairs (c = 2 c2, 2 c2 + 1), so one step costs 8
// packed adds and 4 three-input packed minima; a step that turns a prefix variable off adds the
// negated row.  Chunks of at least 32 steps are walked in aligned groups of 32 unrolled steps,
// in which the flipped prefix bit and its direction are constants; the rows of the two lowest
// prefix bits (three steps of four) stay in registers.  Two steps' minima over their columns are
// packed into one word (even step low), which one add.u16x2 with the packed AA entries turns
// into both steps' values, wrapping like the reference's int16; a group keeps only its minimum,
// and the exact step is found afterwards for the one thread that wins (qbf1w_final_kernel).
// Each thread reports (best int16 value, its group) of its chunk into key[tid] by a 64-bit
// atomic min, which keeps the smallest value and, among equal values, the earliest group.
//
// What bounds it: the register reads and the half-rate pipes of the 8 adds (FMA pipe) and 5.75
// minima and permutes (ALU) per step of 16 states.  2^34 states (n = 34): 727 us, against
// 1230 us with one step at a time (44 instructions per step: the halves extracted, added and
// compared as scalars, every row read from shared memory).
__global__ void __launch_bounds__(256, 3) qbf1w_search_kernel(int A, const short* __restrict__ BB,
                                                              const short* __restrict__ ABBA,
                                                              const short* __restrict__ AA, uint64_t chunk_len,
                                                              unsigned long long* __restrict__ key) {
  extern __shared__ uint32_t q1w_smem[];  // [2][A][8][64]: word (row k, pair c2, thread t)
  const int blk = blockIdx.x;
  for (int i = threadIdx.x; i < A * 512; i += blockDim.x) {
    const int k = i >> 9, c2 = (i >> 6) & 7, tt = i & 63;
    const size_t base = (size_t)k * (1 << kQbf1B) + (size_t)blk * 1024 + tt;
    const int lo = ABBA[base + 64 * (2 * c2)], hi = ABBA[base + 64 * (2 * c2 + 1)];
    q1w_smem[i] = pack16(lo, hi);
    q1w_smem[A * 512 + i] = pack16(-lo, -hi);
  }
  __syncthreads();
  const int t = threadIdx.x & 63;
  const uint64_t chunk = (uint64_t)blockIdx.y * 4 + (threadIdx.x >> 6);
  const uint64_t steps = 1ull << A;
  const uint64_t i0 = chunk * chunk_len;
  if (i0 >= steps) return;
  const uint64_t i1 = min(steps, i0 + chunk_len);
  const uint32_t* pos = q1w_smem + t;            // + row * 512 + c2 * 64
  const uint32_t* neg = q1w_smem + A * 512 + t;
  uint32_t E2[8];
  {
    const uint64_t p0 = gray64(i0);
#pragma unroll
    for (int c2 = 0; c2 < 8; ++c2) E2[c2] = pack16(BB[blk * 1024 + 128 * c2 + t], BB[blk * 1024 + 128 * c2 + 64 + t]);
    for (int k = 0; k < A; ++k)
      if ((p0 >> (A - 1 - k)) & 1) {
#pragma unroll
        for (int c2 = 0; c2 < 8; ++c2) E2[c2] = add16x2(E2[c2], pos[k * 512 + c2 * 64]);
      }
  }
  int best;
  uint64_t bi = i0;
  if ((chunk_len & 31) == 0) {
    best = 32768;  // above every int16
    uint32_t lp[2][2][8];  // rows of prefix bits 0 and 1 (variables A-1, A-2), on and off
#pragma unroll
    for (int kb = 0; kb < 2; ++kb)
#pragma unroll
      for (int c2 = 0; c2 < 8; ++c2) {
        lp[kb][0][c2] = pos[(A - 1 - kb) * 512 + c2 * 64];
        lp[kb][1][c2] = neg[(A - 1 - kb) * 512 + c2 * 64];
      }
    for (uint64_t ig = i0; ig < i1; ig += 32) {
      uint32_t aa[16];  // AA[ig .. ig + 31], two per word
      {
        const uint4* src = reinterpret_cast<const uint4*>(AA + ig);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint4 w = __ldg(src + q);
          aa[4 * q] = w.x;
          aa[4 * q + 1] = w.y;
          aa[4 * q + 2] = w.z;
          aa[4 * q + 3] = w.w;
        }
      }
      if (ig != i0) {  // the chunk's first step is its start state
        const int kb = __ffsll((long long)ig) - 1;  // >= 5
        const uint32_t* r = (((gray64(ig) >> kb) & 1) ? pos : neg) + (A - 1 - kb) * 512;
#pragma unroll
        for (int c2 = 0; c2 < 8; ++c2) E2[c2] = add16x2(E2[c2], r[c2 * 64]);
      }
      const uint32_t* r4 = (((ig >> 5) & 1) ? neg : pos) + (A - 5) * 512;  // prefix bit 4: off in odd groups
      uint32_t gm = 0u;
#pragma unroll
      for (int l = 0; l < 32; l += 2) {
        if (l) {
          const int kb = ctz5(l);  // >= 1
          const bool on = !((l >> (kb + 1)) & 1);
          const uint32_t* r = kb == 4 ? r4 : (on ? pos : neg) + (A - 1 - kb) * 512;
#pragma unroll
          for (int c2 = 0; c2 < 8; ++c2) E2[c2] = add16x2(E2[c2], kb == 1 ? lp[1][on ? 0 : 1][c2] : r[c2 * 64]);
        }
        const uint32_t m0 = min16x2_8(E2);
#pragma unroll
        for (int c2 = 0; c2 < 8; ++c2) E2[c2] = add16x2(E2[c2], lp[0][(l >> 1) & 1][c2]);
        const uint32_t m1 = min16x2_8(E2);
        const uint32_t tt = add16x2(min16x2(__byte_perm(m0, m1, 0x5410), __byte_perm(m0, m1, 0x7632)), aa[l >> 1]);
        gm = l ? min16x2(gm, tt) : tt;
      }
      const int g = min((int)(short)(gm & 0xffffu), (int)gm >> 16);
      if (g < best) {  // strict: the earliest group keeps a tie
        best = g;
        bi = ig;
      }
    }
  } else {
    auto step_min = [&]() -> int {
      const uint32_t m2 = min16x2_8(E2);
      return min((int)(short)(m2 & 0xffffu), (int)m2 >> 16);
    };
    best = wrap16((int)AA[i0] + step_min());
    for (uint64_t i = i0 + 1; i < i1; ++i) {
      const int kb = __ffsll((long long)i) - 1;
      const bool on = (gray64(i) >> kb) & 1;
      const uint32_t* r = (on ? pos : neg) + (A - 1 - kb) * 512;
#pragma unroll
      for (int c2 = 0; c2 < 8; ++c2) E2[c2] = add16x2(E2[c2], r[c2 * 64]);
      const int tt = wrap16((int)AA[i] + step_min());
      if (tt < best) {
        best = tt;
        bi = i;
      }
    }
  }
  const int tid = blk * 64 + t;
  atomicMin(key + tid, ((unsigned long long)(best + 32768) << 40) | (unsigned long long)bi);
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
                                                          const short* __restrict__ ABBA, const short* __restrict__ AA,
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
    for (int k = 0; k < A; ++k)
      if ((p >> (A - 1 - k)) & 1) v += ABBA[(size_t)k * (1 << kQbf1B) + col];
    v = wrap16(v);
  }
  val[warp][lane] = v;
  __syncthreads();
  if (warp == 0) {
    for (int c = 1; c < 16; ++c) v = min(v, val[c][lane]);
    const bool hit = in && wrap16((int)AA[in ? st : s0] + v) == best16;
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
