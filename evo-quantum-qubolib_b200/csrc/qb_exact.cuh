// qb_exact.cuh -- exact enumeration of state records (the "pass 2" kernel).
//
// One CTA per record, or per part of one.  A record is a set of 2^f states: a base state with f
// free bits (record_states in qb_common.cuh).  Energies are FP64, exact for integer Q with
// sum|Q| < 2^53.  The free bits split into up to 8 that select the thread, up to 5 that a
// thread holds as 32 energies in registers, and the rest, walked in Gray order by the whole CTA:
//   E(g, h) = c(h) + el_h[g]     g: register bits, h: walked bits
// c is the thread's energy with the register bits 0, el_h[g] what they add (their fields, which
// depend on the thread and on h, and their own couplings).  A walk step that flips variable o
// costs one add and one minimum per state: el[g] += +- sum of W_og over the set bits (a table in
// shared memory, the same for every thread), one c update, and the update of the walked
// variables' fields.  Only the minimum and its step are kept on the way; the threads within rounding of
// the CTA's minimum (usually one) then look for the state at that step (walking again where several
// steps attain the minimum), with the tie key, and the winner's energy is summed from scratch, so
// the reported value does not carry the walk's rounding.
//
// What bounds it: for one candidate record of 2^17 states in 16 parts (a 36-variable solve) the
// latency of one CTA's steps -- W from L2, the base state's fields and the start tables (all
// threads together), 32 energies, the CTA's minimum, one ordered sum: 15-18 us, against 29-54 us
// when every thread summed its start and its best state's energy alone (n = 20 .. 37).  Many states
// per CTA (2^19, qb_prefix_minima at n = 27): per state one FP64 add and one FP64 compare with two
// selects, two CTAs per SM (128 registers); 2^27 states 520 -> 69 us.  Where nearly all states tie,
// the second walk and the tie keys: 2^30 states of a zero matrix 2.0 ms, of a random one 0.46 ms.
// The 4096-problem batch's pass 2 1400 -> 507 us.
#pragma once
#include <cstring>

#include "qb_common.cuh"

namespace qb {

struct ExactOut {
  double e;
  uint64_t key;
  uint64_t x;
};

constexpr int kExactThreads = 256;
constexpr int kExactMaxFree = 40;
constexpr int kExactRegBits = 5;  // register bits: 32 FP64 energies per thread
constexpr int kExactLowWalk = 7;  // walked bits whose patterns' energies are a table

__device__ __forceinline__ double energy_from_scratch(const double* __restrict__ Ws, int n, uint64_t X) {
  double e = 0.0;
  uint64_t rem = X & mask64(n);
  while (rem) {
    int p = 63 - __clzll(rem);  // highest set bit = lowest variable index
    rem &= ~(1ull << p);
    int i = n - 1 - p;
    const double* row = Ws + i * n;
    e += row[i];
    uint64_t r2 = rem;  // variables after i
    while (r2) {
      int q = 63 - __clzll(r2);
      r2 &= ~(1ull << q);
      e += row[n - 1 - q];
    }
  }
  return e;
}

__device__ __forceinline__ bool lex_less(double e1, uint64_t k1, double e2, uint64_t k2) {
  return e1 < e2 || (e1 == e2 && k1 < k2);
}

// energy_from_scratch's sum, in its order, by one warp: the lanes lay the addends out in buf
// (k (k + 1) / 2 of them for k set bits; list: 64 ints), then every lane adds them up
__device__ __forceinline__ double energy_ordered(const double* __restrict__ Ws, int n, uint64_t X, double* buf,
                                                 int* list) {
  const int lane = threadIdx.x & 31;
  X &= mask64(n);
  const int k = __popcll(X);
  for (int v = lane; v < n; v += 32) {
    const int p = n - 1 - v;
    if ((X >> p) & 1) list[__popcll(X >> p) - 1] = v;
  }
  __syncwarp();
  for (int j = lane; j < k; j += 32) {
    const int v = list[j];
    int off = j;  // row i of the sum starts at i k - i (i - 1) / 2, its entry j >= i lies j - i further
#pragma unroll 4
    for (int i = 0; i <= j; ++i) {
      buf[off] = Ws[list[i] * n + v];
      off += k - i - 1;
    }
  }
  __syncwarp();
  double e = 0.0;
  const int cnt = k * (k + 1) / 2;
#pragma unroll 8
  for (int i = 0; i < cnt; ++i) e += buf[i];
  __syncwarp();
  return e;
}

__device__ __forceinline__ double min32d(const double (&el)[32]) {
  double m[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double a = el[4 * i] < el[4 * i + 1] ? el[4 * i] : el[4 * i + 1];
    const double b = el[4 * i + 2] < el[4 * i + 3] ? el[4 * i + 2] : el[4 * i + 3];
    m[i] = a < b ? a : b;
  }
#pragma unroll
  for (int w = 4; w >= 1; w >>= 1)
#pragma unroll
    for (int i = 0; i < w; ++i) m[i] = m[i] < m[i + w] ? m[i] : m[i + w];
  return m[0];
}

// order-preserving map of a double to an unsigned integer, and back
__host__ __device__ __forceinline__ uint64_t ord_f64(double e) {
#ifdef __CUDA_ARCH__
  uint64_t u = (uint64_t)__double_as_longlong(e);
#else
  uint64_t u;
  memcpy(&u, &e, 8);
#endif
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

__host__ __device__ __forceinline__ double unord_f64(uint64_t k) {
  uint64_t u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double e;
  memcpy(&e, &u, 8);
  return e;
#endif
}

// minimum of a double over the warp, by two 32-bit reductions of its ordered pattern (-0.0 sorts
// below +0.0, which changes no value)
__device__ __forceinline__ double warp_min_d(double v) {
  const uint64_t k = ord_f64(v);
  const uint32_t hi = __reduce_min_sync(0xffffffffu, (uint32_t)(k >> 32));
  const uint32_t lo = __reduce_min_sync(0xffffffffu, (uint32_t)(k >> 32) == hi ? (uint32_t)k : 0xffffffffu);
  return unord_f64(((uint64_t)hi << 32) | lo);
}

// One CTA (kExactThreads threads) evaluates record rid exactly -- or, with split_bits > 0,
// part `part` of it: the record's top split_bits free bits fixed to the bits of part (at
// most f - 8 of them) -- and returns the lexicographic (E, key) minimum in thread 0.
// smem_d: exact_smem_bytes(n, f) of dynamic shared memory.
__device__ __forceinline__ ExactOut exact_record_min(const ProblemDev& P, const TieRule& R, const RecGeom& G,
                                                     uint64_t rid, double* smem_d, int part, int split_bits) {
  const int n = P.n;
  constexpr int kWarps = kExactThreads / 32, kSlots = 4;
  __shared__ int var[kExactMaxFree];            // variables of the free bits, lowest bit first
  __shared__ double hs[64];                     // fields from the base state: sum of W_vq over its bits q != v
  __shared__ double q5[32];                     // energy of a register pattern alone
  __shared__ uint64_t xg[32];                   // its state bits
  __shared__ double qo[1 << kExactLowWalk];     // energy of a pattern of the low walked bits alone
  __shared__ double Wt[8][8];                   // couplings of the thread bits, W_vv + field on the diagonal
  __shared__ double ct[2][16];                  // energy of a pattern of thread bits 0-3, 4-7 from the base state
  __shared__ double ft[kExactMaxFree - 8][2][16];  // field of a register or walked bit from such a pattern
  __shared__ double red_e[kWarps];
  __shared__ uint64_t red_k[kWarps], red_x[kWarps];
  __shared__ double e_base;
  __shared__ int ncand;
  __shared__ ExactOut cand_out[kSlots];
  __shared__ int list[64];                      // energy_ordered's set variables
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;

  double* Ws = smem_d + ((n * n) & 1);  // n*n, then T at a 16-byte boundary
  double asum = 0.0;
  int whole = 1;
  for (int i = t; i < n * n; i += kExactThreads) {
    const double w = P.W[i];
    Ws[i] = w;
    asum += fabs(w);
    whole &= w == rint(w);
  }
  uint64_t base, fm;
  record_states(G, rid, &base, &fm);
  fm &= mask64(n);
  const int nfree = min(__popcll(fm), kExactMaxFree);
  const int sb = split_bits < nfree - 8 ? split_bits : (nfree > 8 ? nfree - 8 : 0);
  const int f = nfree - sb;  // the top sb free bits are fixed by part
  if (t < 64 && ((fm >> t) & 1)) {
    const int j = __popcll(fm & mask64(t));
    if (j < kExactMaxFree) var[j] = n - 1 - t;
  }
  for (int off = 16; off; off >>= 1) asum += __shfl_xor_sync(0xffffffffu, asum, off);
  if (lane == 0) red_e[warp] = asum;
  if (t == 0) ncand = 0;
  whole = __syncthreads_and(whole);
  for (int j = 0; j < sb; ++j)
    if ((part >> j) & 1) base |= 1ull << (n - 1 - var[f + j]);
  const int tb = f < 8 ? f : 8;                                                      // thread bits: var[L ..]
  const int L = f - tb, Lr = L < kExactRegBits ? L : kExactRegBits;  // register bits: var[0 .. Lr)
  const int Lo = L - Lr;                                             // walked bits: var[Lr .. L)
  double* T = Ws + n * n;                                            // [o][32]: walked variable o x register pattern
  double* at = T + Lo * 32;                                          // [o][thread]: fields of the walked variables
  double* buf = at + Lo * kExactThreads;                             // energy_ordered's addends
  asum = 0.0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) asum += red_e[w];
  {  // base fields, four threads per variable
    const int v = t >> 2;
    double h = 0.0;
    if (v < n) {
#pragma unroll 4
      for (int p = t & 3; p < n; p += 4) {
        const int u = n - 1 - p;
        const double w = Ws[u * n + v];
        h += ((base >> p) & 1) && u != v ? w : 0.0;
      }
    }
    h += __shfl_xor_sync(0xffffffffu, h, 1);
    h += __shfl_xor_sync(0xffffffffu, h, 2);
    if ((t & 3) == 0) hs[v] = h;
  }
  __syncthreads();
  // the tables of the thread's start, of the register patterns and of the walk steps
  if (warp == 0) {
    // the fields' sum counts every coupling twice: halved as a whole it stays a whole number for
    // integer W (single fields' halves would not, and FP64 holds halves only below 2^52)
    double e = 0.0, h = 0.0;
    for (int v = lane; v < n; v += 32)
      if ((base >> (n - 1 - v)) & 1) {
        e += Ws[v * n + v];
        h += hs[v];
      }
    for (int off = 16; off; off >>= 1) {
      e += __shfl_xor_sync(0xffffffffu, e, off);
      h += __shfl_xor_sync(0xffffffffu, h, off);
    }
    if (lane == 0) e_base = e + 0.5 * h;
  } else if (warp == 1) {
    double s = 0.0;  // register pattern g = lane
    uint64_t xs = 0;
#pragma unroll
    for (int u = 0; u < kExactRegBits; ++u) {
      if (u >= Lr) break;
      xs |= ((uint64_t)(lane >> u) & 1ull) << (n - 1 - var[u]);
      const double* row = Ws + var[u] * n;
      double r = row[var[u]];
#pragma unroll
      for (int w = 0; w < u; ++w) r += ((lane >> w) & 1) ? row[var[w]] : 0.0;
      s += ((lane >> u) & 1) ? r : 0.0;
    }
    q5[lane] = s;
    xg[lane] = xs;
  } else if (warp == 2) {
    const int half = lane >> 4, g = lane & 15;  // thread pattern g of bits 4 half ..
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (4 * half + u >= tb) break;
      const int v = var[L + 4 * half + u];
      const double* row = Ws + v * n;
      double r = row[v] + hs[v];
#pragma unroll
      for (int w = 0; w < u; ++w) r += ((g >> w) & 1) ? row[var[L + 4 * half + w]] : 0.0;
      s += ((g >> u) & 1) ? r : 0.0;
    }
    ct[half][g] = s;
  } else if (warp == 3) {
    for (int i = lane; i < 64; i += 32) {
      const int j = i >> 3, l = i & 7;
      Wt[j][l] = j < tb && l < tb ? Ws[var[L + j] * n + var[L + l]] : 0.0;
    }
  }
  for (int i = t; i < L * 32; i += kExactThreads) {
    const int o = i >> 5, half = (i >> 4) & 1, g = i & 15;
    const double* row = Ws + var[o] * n;
    double s = half ? 0.0 : hs[var[o]];
#pragma unroll
    for (int u = 0; u < 4; ++u) s += 4 * half + u < tb && ((g >> u) & 1) ? row[var[L + 4 * half + u]] : 0.0;
    ft[o][half][g] = s;
  }
  const int Ll = Lo < kExactLowWalk ? Lo : kExactLowWalk;  // low walked bits
  for (int i = t; i < (1 << Ll); i += kExactThreads) {
    double s = 0.0;
    for (int u = 0; u < Ll; ++u) {
      if (!((i >> u) & 1)) continue;
      const double* row = Ws + var[Lr + u] * n;
      s += row[var[Lr + u]];
#pragma unroll 4
      for (int w = 0; w < u; ++w) s += ((i >> w) & 1) ? row[var[Lr + w]] : 0.0;
    }
    qo[i] = s;
  }
  for (int i = t; i < Lo * 32; i += kExactThreads) {
    const double* row = Ws + var[Lr + (i >> 5)] * n;
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < kExactRegBits; ++u) s += ((i >> u) & 1) ? row[var[u]] : 0.0;
    T[i] = s;
  }
  __syncthreads();

  const bool active = t < (1 << tb);
  const int tl = t & 15, th = t >> 4;
  double c0 = 0.0;
#pragma unroll
  for (int j = 4; j < 8; ++j) {
    double s = 0.0;
#pragma unroll
    for (int l = 0; l < 4; ++l) s += ((tl >> l) & 1) ? Wt[j][l] : 0.0;
    c0 += ((th >> (j - 4)) & 1) ? s : 0.0;
  }
  c0 += ct[0][tl] + ct[1][th] + e_base;
  double a5[kExactRegBits];
#pragma unroll
  for (int u = 0; u < kExactRegBits; ++u) a5[u] = u < Lr ? ft[u][0][tl] + ft[u][1][th] : 0.0;

  // c = ch + A + qo: ch the thread's energy with the high walked bits' pattern, A the sum of the
  // set low walked bits' fields, qo their own energy
  double el[32], c = 0.0, ch = 0.0, A = 0.0;
  // el and c at the walk's start
  auto start = [&]() {
    c = ch = c0;
    A = 0.0;
    for (int o = 0; o < Lo; ++o) at[o * kExactThreads + t] = ft[Lr + o][0][tl] + ft[Lr + o][1][th];
    el[0] = 0.0;
#pragma unroll
    for (int u = 0; u < kExactRegBits; ++u)
#pragma unroll
      for (int g = 0; g < (1 << u); ++g) el[(1 << u) + g] = el[g] + a5[u];
#pragma unroll
    for (int g = 0; g < 32; ++g) el[g] = g < (1 << Lr) ? el[g] + q5[g] : inf;
  };
  // walk step st: flips walked variable ctz(st)
  auto step = [&](uint32_t st) {
    const int o = __ffs(st) - 1;
    const bool on = !((st >> (o + 1)) & 1u);
    const uint32_t gl = (st ^ (st >> 1)) & ((1u << Ll) - 1u);
    if (o < Ll) {
      const double a = at[o * kExactThreads + t];
      A = on ? A + a : A - a;
    } else {  // a high bit, every 2^Ll steps: of the low bits at most the top one is set
      const double* row = Ws + var[Lr + o] * n;
      const double d = row[var[Lr + o]] + at[o * kExactThreads + t];
      ch = on ? ch + d : ch - d;
      for (int o2 = 0; o2 < Lo; ++o2) {
        const double w = o2 == o ? 0.0 : row[var[Lr + o2]];
        at[o2 * kExactThreads + t] += on ? w : -w;
      }
      A = gl ? at[(Ll - 1) * kExactThreads + t] : 0.0;
    }
    c = ch + A + qo[gl];
    const double2* To = reinterpret_cast<const double2*>(T + o * 32);
    if (on) {
#pragma unroll
      for (int g = 0; g < 16; ++g) {
        const double2 w = To[g];
        el[2 * g] += w.x;
        el[2 * g + 1] += w.y;
      }
    } else {
#pragma unroll
      for (int g = 0; g < 16; ++g) {
        const double2 w = To[g];
        el[2 * g] -= w.x;
        el[2 * g + 1] -= w.y;
      }
    }
  };
  const uint32_t steps = 1u << Lo;
  // pass 0: the minimum, the walk step that first attains it and how many do.  Pass 1, the
  // threads that can hold the winner: the smallest key among the thread's states of minimal
  // energy, at that step (its el summed from the start) or, with several, by walking again.
  double best_e = inf, m = inf;
  uint64_t best_k = ~0ull, best_x = 0;
  uint32_t best_st = 0, best_cnt = 0;
  bool cand = active;
  // exact sums: the threads at the CTA's minimum; otherwise those within twice the walk's
  // rounding of it (per step and for the start's about 100 additions, 2^-53 sum |W| each)
  const bool exact = whole && asum < 9007199254740992.0;
  const double tol = exact ? 0.0 : ldexp(asum * (2.0 * (double)steps + 256.0), -52);
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    if (cand) {
      if (pass == 0 || steps > 1) start();  // without walked bits el still holds the start
      uint64_t Xh = 0;  // pass 1: the state's bits but for the register pattern's
      if (pass == 1) {
        Xh = base;
        for (int j = 0; j < tb; ++j)
          if ((t >> j) & 1) Xh |= 1ull << (n - 1 - var[L + j]);
      }
      uint32_t st = 0;
      double target = best_e;
      const bool seek = pass == 1 && best_cnt == 1;
      if (seek) {
        st = best_st;
        uint32_t h = st ^ (st >> 1), lower = 0;
#pragma unroll 1
        for (; h; h &= h - 1) {
          const int o = __ffs(h) - 1;
          const double* row = Ws + var[Lr + o] * n;
          double d = row[var[Lr + o]] + at[o * kExactThreads + t];
          for (uint32_t l = lower; l; l &= l - 1) d += row[var[Lr + __ffs(l) - 1]];
          c += d;
          lower |= 1u << o;
          Xh |= 1ull << (n - 1 - var[Lr + o]);
#pragma unroll
          for (int g = 0; g < 32; ++g) el[g] += T[o * 32 + g];
        }
        target = c + min32d(el);
      }
#pragma unroll 1
      for (;;) {
        const double e = c + min32d(el);
        if (pass == 0) {
          if (e < best_e) {
            best_e = e;
            best_st = st;
            best_cnt = 0;
          }
          best_cnt += e == best_e;
        } else if (e == target) {
          uint32_t hit = 0;
#pragma unroll
          for (int g = 0; g < 32; ++g) hit |= c + el[g] == target ? 1u << g : 0u;
#pragma unroll 1
          for (; hit; hit &= hit - 1) {
            const uint64_t X = Xh | xg[__ffs(hit) - 1];
            const uint64_t k = tie_key(R, X);
            if (k < best_k) {
              best_k = k;
              best_x = X;
            }
          }
        }
        if (seek || ++st == steps) break;
        step(st);
        Xh ^= 1ull << (n - 1 - var[Lr + __ffs(st) - 1]);
      }
    }
    if (pass == 0) {  // the CTA's minimum
      m = warp_min_d(best_e);
      __syncthreads();  // red_e was read as sum |W|
      if (lane == 0) red_e[warp] = m;
      __syncthreads();
#pragma unroll
      for (int w = 0; w < kWarps; ++w) m = red_e[w] < m ? red_e[w] : m;
      cand = active && best_e <= m + tol;
    }
  }
  if (cand) {
    const int slot = atomicAdd(&ncand, 1);
    if (slot < kSlots) cand_out[slot] = ExactOut{best_e, best_k, best_x};
  } else {
    best_e = inf;
  }
  __syncthreads();
  const int nc = ncand;
  if (nc <= kSlots) {  // usual: pick among the slots
    ExactOut b{inf, ~0ull, 0ull};
    if (warp == 0)
      for (int i = 0; i < nc; ++i) {
        ExactOut o = cand_out[i];
        if (!exact) o.e = energy_ordered(Ws, n, o.x, buf, list);
        if (lex_less(o.e, o.key, b.e, b.key)) b = o;
      }
    return b;
  }
  if (!exact && cand) best_e = energy_from_scratch(Ws, n, best_x);
  // CTA reduction of (e, key, x)
  for (int off = 16; off; off >>= 1) {
    double oe = __shfl_down_sync(0xffffffffu, best_e, off);
    uint64_t ok = __shfl_down_sync(0xffffffffu, best_k, off);
    uint64_t ox = __shfl_down_sync(0xffffffffu, best_x, off);
    if (lex_less(oe, ok, best_e, best_k)) {
      best_e = oe;
      best_k = ok;
      best_x = ox;
    }
  }
  if (lane == 0) {
    red_e[warp] = best_e;
    red_k[warp] = best_k;
    red_x[warp] = best_x;
  }
  __syncthreads();
  if (t == 0)
    for (int w = 1; w < kWarps; ++w)
      if (lex_less(red_e[w], red_k[w], best_e, best_k)) {
        best_e = red_e[w];
        best_k = red_k[w];
        best_x = red_x[w];
      }
  return ExactOut{best_e, best_k, best_x};
}

__device__ __forceinline__ void exact_record_body(const ProblemDev& P, const TieRule& R, const RecGeom& G,
                                                  uint64_t rid, ExactOut* __restrict__ out_slot, double* smem_d,
                                                  int part = 0, int split_bits = 0) {
  const ExactOut o = exact_record_min(P, R, G, rid, smem_d, part, split_bits);
  if (threadIdx.x == 0) *out_slot = o;
}

// rec_ids: candidate record indices (nullptr: record = rec_offset + block).
// count_ptr: number of valid entries (nullptr: count_static).
// split_bits: 2^split_bits CTAs per record (block = blockIdx.x >> split_bits); outputs are
// indexed (slot << split_bits) | part.
__global__ void __launch_bounds__(kExactThreads, 2)
exact_records_kernel(ProblemDev P, TieRule R, RecGeom G, const uint64_t* __restrict__ rec_ids,
                     const int* __restrict__ count_ptr, int64_t count_static, int64_t rec_offset,
                     ExactOut* __restrict__ out, int split_bits) {
  extern __shared__ __align__(16) double smem_d[];
  const int64_t blk = (int64_t)(blockIdx.x >> split_bits);
  const int part = (int)(blockIdx.x & ((1u << split_bits) - 1u));
  const int64_t slot = blk + (rec_ids ? rec_offset : 0);
  const int64_t count = count_ptr ? (int64_t)(*count_ptr) : count_static;
  if (slot >= count) return;
  const uint64_t rid = rec_ids ? rec_ids[slot] : (uint64_t)(rec_offset + blk);
  exact_record_body(P, R, G, rid, out + ((slot << split_bits) | part), smem_d, part, split_bits);
}

// qb_prefix_minima for prefixes of few states: out[p] = the minimum over the 2^B states of prefix p
// (natural order), every energy summed from scratch, a state per thread and W loaded once per CTA.
// In exact_records_kernel a prefix costs a CTA's whole set-up, which pays from 2^8 states on.  The
// whole call (f64, us) there and here: n = 20, B = 0 .. 7 25254 12658 6386 3196 1649 848 448 238 and
// 847 469 298 208 156 134 125 118; n = 22, B = 7 892 and 435; B = 8 there 470.
constexpr int kPrefixFewBits = 7;
__global__ void __launch_bounds__(kExactThreads)
prefix_few_states_kernel(ProblemDev P, int B, double* __restrict__ out) {
  extern __shared__ __align__(16) double smem_d[];
  __shared__ double red[kExactThreads / 32];
  const int n = P.n;
  for (int i = threadIdx.x; i < n * n; i += kExactThreads) smem_d[i] = P.W[i];
  __syncthreads();
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lb = min(B, 5), g = 1 << (B - lb);  // a prefix: 2^lb lanes of g neighbouring warps
  const uint64_t states = 1ull << n;
  for (uint64_t x0 = (uint64_t)blockIdx.x * kExactThreads; x0 < states; x0 += (uint64_t)gridDim.x * kExactThreads) {
    const uint64_t X = x0 + threadIdx.x;
    double m = X < states ? energy_from_scratch(smem_d, n, X) : inf;
    __syncwarp();
    for (int b = 0; b < lb; ++b) {
      const double o = __shfl_xor_sync(0xffffffffu, m, 1 << b);
      m = o < m ? o : m;
    }
    if (g > 1) {
      if (lane == 0) red[warp] = m;
      __syncthreads();
      for (int w = warp; w < warp + g && w < kExactThreads / 32; ++w) m = red[w] < m ? red[w] : m;
      __syncthreads();
    }
    if (X < states && (X & mask64(B)) == 0) out[X >> B] = m;
  }
}

// One solve's control words on the device, uploaded with W and copied back with the answer.
struct SolveCtl {
  uint32_t err;      // error word of the tensor-core kernels
  uint32_t min_key;  // smallest pass-1 record value (f2key)
  int count;         // candidate records
  uint32_t done[2];  // CTAs that have finished: exact_candidates_kernel, exact_row_kernel
  uint32_t pad;
  ExactOut best;     // exact_candidates_kernel's answer
  ExactOut row;      // exact_row_kernel's answer
};

// Every CTA's thread 0 holds b: the last CTA to arrive at *done writes the lexicographic minimum
// over all of them to *out.  part: gridDim.x entries.
__device__ __forceinline__ void last_cta_min(const ExactOut& b, ExactOut* __restrict__ part, uint32_t* done,
                                             ExactOut* __restrict__ out) {
  __shared__ int last;
  __shared__ ExactOut red[kExactThreads / 32];
  if (threadIdx.x == 0) {
    part[blockIdx.x] = b;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double be = __longlong_as_double(0x7ff0000000000000ll);
  uint64_t bk = ~0ull, bx = 0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += kExactThreads) {
    const double e = __ldcg(&part[i].e);
    const uint64_t k = __ldcg(reinterpret_cast<const unsigned long long*>(&part[i].key));
    if (lex_less(e, k, be, bk)) {
      be = e;
      bk = k;
      bx = __ldcg(reinterpret_cast<const unsigned long long*>(&part[i].x));
    }
  }
  for (int off = 16; off; off >>= 1) {
    const double oe = __shfl_down_sync(0xffffffffu, be, off);
    const uint64_t ok = __shfl_down_sync(0xffffffffu, bk, off);
    const uint64_t ox = __shfl_down_sync(0xffffffffu, bx, off);
    if (lex_less(oe, ok, be, bk)) {
      be = oe;
      bk = ok;
      bx = ox;
    }
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ExactOut{be, bk, bx};
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kExactThreads / 32; ++w)
      if (lex_less(red[w].e, red[w].key, be, bk)) {
        be = red[w].e;
        bk = red[w].key;
        bx = red[w].x;
      }
    *out = ExactOut{be, bk, bx};
  }
}

// The candidate records rec_ids[0 .. ctl->count) (rec_ids == nullptr: the records
// 0 .. count_static), each split into up to 2^split_bits parts, as a grid-stride loop over
// (record, part) items: the host launches it before it knows the count.  Parts repeat the set-up,
// so records are split only as far as all parts run at once (the whole call with 16 parts always
// and so: 2 candidates at n = 20 80 and 80 us, 64 at n = 24 166 and 116, 1024 at n = 33 1301 and
// 553, 8192 13.4 and 5.6 ms).  The lexicographic minimum over all of them goes to ctl->best.  With
// more candidates than cap nothing is done: the host starts over with a larger cap.
__global__ void __launch_bounds__(kExactThreads, 2)
exact_candidates_kernel(ProblemDev P, TieRule R, RecGeom G, const uint64_t* __restrict__ rec_ids, SolveCtl* ctl,
                        int64_t count_static, int cap, int split_bits, ExactOut* __restrict__ part_out) {
  extern __shared__ __align__(16) double smem_d[];
  const int64_t count = !rec_ids ? count_static : ctl->count <= cap ? (int64_t)ctl->count : 0;
  while (split_bits > 0 && (count << split_bits) > (int64_t)gridDim.x) --split_bits;
  const int64_t items = count << split_bits;
  ExactOut b{__longlong_as_double(0x7ff0000000000000ll), ~0ull, 0ull};
  for (int64_t w = blockIdx.x; w < items; w += gridDim.x) {
    __syncthreads();  // the previous item's shared-memory readers are done
    const int64_t slot = w >> split_bits;
    const int part = (int)(w & ((1 << split_bits) - 1));
    const ExactOut o = exact_record_min(P, R, G, rec_ids ? rec_ids[slot] : (uint64_t)slot, smem_d, part, split_bits);
    if (lex_less(o.e, o.key, b.e, b.key)) b = o;
  }
  last_cta_min(b, part_out, &ctl->done[0], &ctl->best);
}

// QB_F1's last step: the smallest 18-bit suffix among the states of ctl->best's prefix with its
// energy, as the natural-order minimum of that prefix's 2^18 states over gridDim.x = 2^kRowSplit
// CTAs, into ctl->row (left at +infinity where there is nothing to do).
constexpr int kRowSplit = 5;
__global__ void __launch_bounds__(kExactThreads, 2)
exact_row_kernel(ProblemDev P, SolveCtl* ctl, ExactOut* __restrict__ part_out) {
  extern __shared__ __align__(16) double smem_d[];
  ExactOut b{__longlong_as_double(0x7ff0000000000000ll), ~0ull, 0ull};
  const uint64_t x = ctl->best.x;
  if (x != 0ull) {
    RecGeom g{};
    g.kind = kGeomBlock;
    g.n = P.n;
    g.fbits = 18;
    const TieRule nat{kTieNatural, P.n, 0, 0, 0};
    b = exact_record_min(P, nat, g, x >> 18, smem_d, (int)blockIdx.x, kRowSplit);
  }
  last_cta_min(b, part_out, &ctl->done[1], &ctl->row);
}

inline size_t exact_smem_bytes(int n, int f) {
  const int lo = f > 8 + kExactRegBits ? f - 8 - kExactRegBits : 0;  // walked bits
  return ((size_t)n * n + 1 + (size_t)lo * (32 + kExactThreads) + (size_t)n * (n + 1) / 2) * sizeof(double);
}

}  // namespace qb
