// Sampling on the device from float32 logits [rows, vocab].
//
// greedy:      argmax, ties to the lowest token id.
// temperature / nucleus: p = softmax(logits / T); tokens are ranked by
// (-p, id); the head is the shortest prefix of that ranking whose mass reaches
// top_p; the draw u * mass(head) picks the first rank whose cumulative mass
// reaches it.  u is word 0 of Philox-4x32-10 with counter (pos_lo, pos_hi, 0, 0)
// and the request's 64-bit key, times 2^-32.  No sort is done: the rank that a
// target mass falls on is found on the bit pattern of p, up to 163,840 tokens digit by
// digit over histograms in shared memory (sample_cluster_kernel), beyond by bisection with a
// scratch of p in memory (sample_kernel: 32 block sums in a fixed order); then ties of that
// value are counted in id order.
// Every sum is taken in an order fixed by the vocabulary size alone, or is a sum of whole numbers.
#include <math_constants.h>

#include "common.cuh"

namespace {

constexpr int SAMPLE_THREADS = 1024;

__device__ __forceinline__ void philox_round(uint32_t& c0, uint32_t& c1, uint32_t& c2, uint32_t& c3,
                                             uint32_t k0, uint32_t k1) {
  const uint64_t p0 = (uint64_t)0xD2511F53u * c0;
  const uint64_t p1 = (uint64_t)0xCD9E8D57u * c2;
  const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
  const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
  const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
  c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
}

__device__ __forceinline__ uint32_t philox_word0(uint32_t pos_lo, uint32_t pos_hi, uint32_t k0,
                                                 uint32_t k1) {
  uint32_t c0 = pos_lo, c1 = pos_hi, c2 = 0u, c3 = 0u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    philox_round(c0, c1, c2, c3, k0, k1);
    if (r < 9) { k0 += 0x9E3779B9u; k1 += 0xBB67AE85u; }
  }
  return c0;
}

struct ArgMax {
  float v;
  int i;
};

__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

__device__ ArgMax block_argmax(const float* row, int vocab, float* sval, int* sidx) {
  ArgMax best{-CUDART_INF_F, 0x7fffffff};
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const float v = row[i];
    // NaN never wins; an all-NaN row gives token 0
    if (v > best.v || (v == best.v && i < best.i)) best = ArgMax{v, i};
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) { sval[warp] = best.v; sidx[warp] = best.i; }
  __syncthreads();
  ArgMax r{sval[0], sidx[0]};
  for (int w = 1; w < nwarps; ++w) r = better(r, ArgMax{sval[w], sidx[w]});
  if (r.i == 0x7fffffff) r.i = 0;
  return r;
}

__global__ void argmax_kernel(const float* __restrict__ logits, int* __restrict__ out, int vocab) {
  ls_dependency_sync();
  __shared__ float sval[32];
  __shared__ int sidx[32];
  const ArgMax r = block_argmax(logits + (int64_t)blockIdx.x * vocab, vocab, sval, sidx);
  if (threadIdx.x == 0) out[blockIdx.x] = r.i;
}

// mass of the tokens with p >= the value whose bits are `bits` (p >= 0, so the
// unsigned bit pattern orders like the value)
__device__ float mass_at_least(const float* p, int vocab, uint32_t bits, float* scratch) {
  float s = 0.f;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const float v = p[i];
    if (__float_as_uint(v) >= bits) s += v;
  }
  return ls_block_sum(s, scratch);
}

// The rank that `target` falls on: the token x with before(x) < target <=
// before(x) + p_x in the (-p, id) order.  Also returns the mass up to and
// including x.  If target exceeds the whole mass, the last rank is returned.
__device__ int select_rank(const float* p, int vocab, float target, float* mass_through,
                           float* scratch, int* iscratch) {
  // largest value v (as bits) with mass_at_least(v) >= target
  target = fmaxf(target, 1e-37f);  // a draw of exactly 0 falls on the first rank
  uint32_t lo = 0u, hi = 0x7f800000u;  // invariant: mass(lo) >= target or lo == 0
  for (int it = 0; it < 32 && lo < hi; ++it) {
    const uint32_t mid = lo + (hi - lo + 1u) / 2u;
    const float mass = mass_at_least(p, vocab, mid, scratch);
    if (mass >= target) lo = mid; else hi = mid - 1u;
  }
  // lo may lie between two values that occur: snap it to the smallest p >= lo
  float vmin = CUDART_INF_F;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const float v = p[i];
    if (__float_as_uint(v) >= lo) vmin = fminf(vmin, v);
  }
  vmin = -ls_warp_max(-vmin);
  {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) scratch[warp] = vmin;
    __syncthreads();
    vmin = scratch[0];
    for (int w = 1; w < nwarps; ++w) vmin = fminf(vmin, scratch[w]);
  }
  const uint32_t vbits = __float_as_uint(vmin);
  const float above = mass_at_least(p, vocab, vbits + 1u, scratch);  // mass of p > v
  // ties of value v in ascending id: the j-th (0-based) is the rank wanted
  int j = 0;
  if (vmin > 0.f) {
    const float need = target - above;
    j = (int)ceilf(need / vmin) - 1;
    if (j < 0) j = 0;
  }
  // count ties per thread over contiguous id ranges, then walk
  const int chunk = (vocab + blockDim.x - 1) / blockDim.x;
  const int begin = threadIdx.x * chunk;
  const int end = begin + chunk < vocab ? begin + chunk : vocab;
  int count = 0;
  for (int i = begin; i < end; ++i) count += (__float_as_uint(p[i]) == vbits);
  __syncthreads();
  iscratch[threadIdx.x] = count;
  __syncthreads();
  __shared__ int s_token, s_j;
  if (threadIdx.x == 0) {
    int total = 0;
    for (int t = 0; t < blockDim.x; ++t) total += iscratch[t];
    if (j >= total) j = total - 1;
    if (j < 0) j = 0;
    s_j = j;
    s_token = -1;
  }
  __syncthreads();
  j = s_j;
  // exclusive prefix of this thread
  int before = 0;
  for (int t = 0; t < (int)threadIdx.x; ++t) before += iscratch[t];
  if (j >= before && j < before + count) {
    int k = before;
    for (int i = begin; i < end; ++i) {
      if (__float_as_uint(p[i]) == vbits) {
        if (k == j) { s_token = i; break; }
        ++k;
      }
    }
  }
  __syncthreads();
  *mass_through = above + (float)(j + 1) * vmin;
  return s_token < 0 ? 0 : s_token;
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, float* __restrict__ probs,
              const float* __restrict__ temperature, const float* __restrict__ top_p,
              const uint32_t* __restrict__ keys, const uint32_t* __restrict__ positions,
              int* __restrict__ out, int vocab) {
  ls_dependency_sync();
  __shared__ float scratch[32];
  __shared__ int sidx[32];
  __shared__ int iscratch[SAMPLE_THREADS];
  const int r = blockIdx.x;
  const float* row = logits + (int64_t)r * vocab;
  float* p = probs + (int64_t)r * vocab;
  const float temp = temperature[r];
  const ArgMax top = block_argmax(row, vocab, scratch, sidx);
  if (!(temp > 0.f)) {
    if (threadIdx.x == 0) out[r] = top.i;
    return;
  }
  const float vmax = __fdiv_rn(top.v, temp);
  float s = 0.f;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const float e = expf(__fdiv_rn(row[i], temp) - vmax);
    p[i] = e;
    s += e;
  }
  const float z = ls_block_sum(s, scratch);
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) p[i] = __fdiv_rn(p[i], z);
  __syncthreads();

  const float u = (float)((double)philox_word0(positions[2 * r], positions[2 * r + 1], keys[2 * r],
                                               keys[2 * r + 1]) * 2.3283064365386963e-10);
  float head = 1.0f;
  const float tp = top_p[r];
  float through;
  if (tp < 1.0f) {
    select_rank(p, vocab, tp, &through, scratch, iscratch);
    head = through;
  } else {
    // the whole mass, summed in the order the bisection sums use
    head = mass_at_least(p, vocab, 0u, scratch);
  }
  const float draw = u * head;
  const int token = select_rank(p, vocab, draw, &through, scratch, iscratch);
  if (threadIdx.x == 0) out[r] = token;
}

// --------------------------------------------------------------------------
// The same sampling with a row spread over the 1, 2, 4 or 8 blocks of a cluster: a block keeps
// e = exp(l / T - max) of its contiguous part of the row in shared memory and finds the rank that
// a mass falls on digit by digit of e's bit pattern, highest first: 12 + 10 + 10 bits, a
// histogram of 1,024 bins a digit (e <= 1, so the first digit stays below 1,017).
//
// All masses are whole numbers.  The tokens of a bin share their exponent, so a bin's mass is the
// sum of their 24-bit mantissas, kept as two 32-bit sums (of the low and of the high 12 bits)
// that shared-memory atomics add in any order with the same result: no sum here depends on how
// the row is spread.  Over the first digit masses are counted in units of 2^-46 (163,840 tokens of
// e = 1 fit 64 bits; a bin's own sum is cut to a unit, 1e-14 of the largest token), below it in
// the mantissa units of the chosen bin, exactly.  Every block adds up the eight histograms by
// itself (one exchange a digit), so all take the same decisions.
//
// What bounds it: the exchanges (one for the maximum, one a digit: five digits with a nucleus,
// since the first digit's histogram serves both selections, else three), about 4 us each at eight
// blocks.  Bisecting on the bit pattern instead took 16 passes over registers and 17 exchanges a
// selection.  151,936 tokens with top-p, 1 / 8 / 64 rows: 37 / 39 / 89 us (bisecting: 106 / 107 /
// 526); 64 rows of 32,768: 32 us (510).
// --------------------------------------------------------------------------
constexpr int SAMPLE_CLUSTER = 8;                   // most blocks a row is spread over
// Largest vocabulary of this kernel.  Masses in units of 2^-46 fit 64 bits up to 262,143 tokens of e = 1, and eight blocks
// hold 393,216; above this line sample_kernel is what has been run.
constexpr int SAMPLE_MOST = 163840;
constexpr int SAMPLE_PART = 49152;                  // most tokens of a block: 192 KB of shared memory
static_assert(SAMPLE_MOST <= 4 * SAMPLE_PART, "clusters of four hold every row");
constexpr int SAMPLE_BINS = 1024;                   // a thread adds up one bin
constexpr int SAMPLE_UNIT = 46;                     // masses over the whole row: units of 2^-46
static_assert(SAMPLE_BINS == SAMPLE_THREADS, "a thread a bin");

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_addr(const void* mine, int rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(mine), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ uint2 ld_peer_u2(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}

struct SampleShare {
  uint2 hist[2][SAMPLE_BINS];       // sums of the low and high 12 bits of the mantissas; digits use the two in turn
  uint2 best;                       // this block's largest logit and its id
  float warp_v[32];
  int warp_i[32];
  unsigned long long warp_mass[32];
  unsigned long long total;         // of the row, in units of 2^-46
  unsigned long long above;         // mass in front of the chosen bin
  unsigned long long through;       // mass up to and including the chosen token (units of 2^-46)
  unsigned long long peer_sum[SAMPLE_CLUSTER];   // the chosen value's mass in each block
  int bin;
  int bad;                          // the row holds something that is no number
};

// The block's inclusive scan of `mass` in thread order (bins from the highest down: thread t has bin
// SAMPLE_BINS - 1 - t); `excl` is what lies in front of this thread.
__device__ unsigned long long sample_scan(SampleShare& sh, unsigned long long mass, unsigned long long& excl) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long incl = mass;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) sh.warp_mass[warp] = incl;
  __syncthreads();
  unsigned long long before = lane < warp ? sh.warp_mass[lane] : 0ull;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  incl += before;
  excl = incl - mass;
  return incl;
}

// One token's mantissa into its bin, for the lanes with `counts` (called by whole warps).  Where all of a
// warp's tokens share a bin, as in a flat row, the warp's sums go there at once: 64 atomics on one address
// would follow one another (a row of 151,936 equal logits 50 us, without this 126; a usual row pays 3 us).
__device__ __forceinline__ void sample_count(uint2* hist, bool counts, uint32_t bin, uint32_t bits) {
  const uint32_t lanes = __ballot_sync(0xffffffffu, counts);
  if (lanes == 0u) return;
  const uint32_t m = counts ? (bits & 0x7fffffu) | (bits >= 0x800000u ? 0x800000u : 0u) : 0u;
  const int first = __ffs(lanes) - 1;
  const uint32_t first_bin = __shfl_sync(0xffffffffu, bin, first);
  if (__all_sync(0xffffffffu, !counts || bin == first_bin)) {
    const uint32_t low = __reduce_add_sync(0xffffffffu, m & 0xfffu), high = __reduce_add_sync(0xffffffffu, m >> 12);
    if ((int)(threadIdx.x & 31) == first) {
      atomicAdd(&hist[bin].x, low);
      atomicAdd(&hist[bin].y, high);
    }
  } else if (counts) {
    atomicAdd(&hist[bin].x, m & 0xfffu);
    atomicAdd(&hist[bin].y, m >> 12);
  }
}

// The token that `target` (>= 1, at most the row's mass; units of 2^-46) falls on in the (-e, id)
// order, `l1_excl` and `l1_incl` being the scan of the first digit's bins.  Writes sh.through and,
// in the block that holds the token, *token_out where it is not null.  `turn`: the histogram free
// for the next digit (zeroed); every thread's own copy, the same in all.
template <int CL>
__device__ void sample_select(SampleShare& sh, const float* e, int live, int begin, int& turn, unsigned long long l1_excl,
                              unsigned long long l1_incl, unsigned long long target, int* token_out) {
  const int tid = threadIdx.x, b = SAMPLE_BINS - 1 - tid;
  if (l1_excl < target && target <= l1_incl) {
    sh.bin = b;
    sh.above = l1_excl;
  }
  __syncthreads();
  uint32_t prefix = (uint32_t)sh.bin;
  const unsigned long long l1_above = sh.above;
  // from here on in mantissa units of the bin: 2^(exponent - 150)
  const int exponent = (int)(prefix >> 3) > 0 ? (int)(prefix >> 3) : 1;
  const int shift = exponent - (150 - SAMPLE_UNIT);
  unsigned long long want = target - l1_above;
  want = shift >= 0 ? (want + ((1ull << shift) - 1)) >> shift : want << -shift;
  unsigned long long within = 0;                      // mantissa units in front, inside the first digit's bin
#pragma unroll 1
  for (int digit = 1; digit < 3; ++digit) {
    uint2* hist = sh.hist[turn];
    const int down = digit == 1 ? 10 : 0;
    for (int i0 = 0; i0 < live; i0 += SAMPLE_THREADS) {
      const uint32_t bits = i0 + tid < live ? __float_as_uint(e[i0 + tid]) : 0u;
      sample_count(hist, bits >> (down + 10) == prefix && bits != 0u, (bits >> down) & 1023u, bits);
    }
    cluster_sync_all();
    const int here = turn;
    turn ^= 1;
    sh.hist[turn][tid] = make_uint2(0u, 0u);          // nobody reads the digit before any more
    unsigned long long sum[CL], mass = 0;
#pragma unroll
    for (int r = 0; r < CL; ++r) {
      const uint2 v = ld_peer_u2(peer_addr(&sh.hist[here][b], r));
      sum[r] = v.x + ((unsigned long long)v.y << 12);
      mass += sum[r];
    }
    unsigned long long excl;
    const unsigned long long incl = sample_scan(sh, mass, excl);
    if (excl < want && want <= incl) {
      sh.bin = b;
      sh.above = excl;
      if (digit == 2) {
#pragma unroll
        for (int r = 0; r < CL; ++r) sh.peer_sum[r] = sum[r];
      }
    }
    __syncthreads();
    prefix = (prefix << 10) | (uint32_t)sh.bin;
    want -= sh.above;
    within += sh.above;
    __syncthreads();
  }
  // prefix is now the bit pattern of the chosen value; its tokens in ascending id, one mantissa each
  const unsigned long long m = (prefix & 0x7fffffu) | (prefix >= 0x800000u ? 0x800000u : 0u);
  const unsigned long long rank_j = (want + m - 1) / m - 1;         // want lies in 1 .. ties x m
  if (tid == 0) {
    const unsigned long long in = within + (rank_j + 1) * m;
    sh.through = l1_above + (shift >= 0 ? in << shift : in >> -shift);
  }
  if (token_out != nullptr) {
    unsigned long long before = 0;
    const int rank = (int)cluster_rank();
    for (int r = 0; r < rank; ++r) before += sh.peer_sum[r];
    const unsigned long long own = sh.peer_sum[rank] / m;
    before /= m;
    if (rank_j >= before && rank_j < before + own) {               // the same in all threads of a block
      const int per = (live + SAMPLE_THREADS - 1) / SAMPLE_THREADS;
      const int lo = min(tid * per, live), hi = min(lo + per, live);
      unsigned long long count = 0, excl;
      for (int i = lo; i < hi; ++i) count += __float_as_uint(e[i]) == prefix;
      sample_scan(sh, count, excl);
      unsigned long long k = before + excl;
      for (int i = lo; i < hi; ++i)
        if (__float_as_uint(e[i]) == prefix && k++ == rank_j) *token_out = begin + i;
    }
  }
  __syncthreads();
}

template <int CL>
__global__ void __launch_bounds__(SAMPLE_THREADS, 1)
sample_cluster_kernel(const float* __restrict__ logits, const float* __restrict__ temperature,
                      const float* __restrict__ top_p, const uint32_t* __restrict__ keys,
                      const uint32_t* __restrict__ positions, int* __restrict__ out, int vocab) {
  ls_dependency_sync();
  __shared__ SampleShare sh;
  extern __shared__ float sample_e[];                // this block's part of the row
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = blockIdx.x / CL;
  const int rank = (int)cluster_rank();
  const int part = (vocab + CL - 1) / CL;
  const int begin = rank * part;
  const int live = min(part, vocab - begin);         // may be negative: no tokens
  const float* row = logits + (int64_t)r * vocab + begin;
  // the row's argmax (ties to the lowest id; NaN never wins)
  ArgMax best{-CUDART_INF_F, 0x7fffffff};
#pragma unroll 8
  for (int i = tid; i < live; i += SAMPLE_THREADS) {
    const float v = row[i];
    sample_e[i] = v;
    if (v > best.v || (v == best.v && begin + i < best.i)) best = ArgMax{v, begin + i};
  }
  sh.hist[0][tid] = sh.hist[1][tid] = make_uint2(0u, 0u);
  if (tid == 0) sh.bad = 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  if (lane == 0) { sh.warp_v[warp] = best.v; sh.warp_i[warp] = best.i; }
  __syncthreads();
  best = ArgMax{sh.warp_v[lane], sh.warp_i[lane]};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  if (tid == 0) sh.best = make_uint2(__float_as_uint(best.v), (uint32_t)best.i);
  cluster_sync_all();
  {
    const uint2 peer = ld_peer_u2(peer_addr(&sh.best, lane & (CL - 1)));
    best = ArgMax{__uint_as_float(peer.x), (int)peer.y};
#pragma unroll
    for (int o = CL / 2; o > 0; o >>= 1) {
      ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
      best = better(best, other);
    }
  }
  if (best.i == 0x7fffffff) best.i = 0;
  const float temp = temperature[r];
  if (!(temp > 0.f)) {                       // the same branch in every block of the cluster
    if (rank == 0 && tid == 0) out[r] = best.i;
    cluster_sync_all();                      // no block leaves while a peer may still read its shared memory
    return;
  }
  const float vmax = __fdiv_rn(best.v, temp);
  // e, and the first digit's histogram; what is no number goes to the last bin
  for (int i0 = 0; i0 < live; i0 += SAMPLE_THREADS) {
    const int i = i0 + tid;
    uint32_t bits = 0u;
    if (i < live) {
      const float v = expf(__fdiv_rn(sample_e[i], temp) - vmax);
      sample_e[i] = v;
      bits = __float_as_uint(v);
      if (bits > 0x3f800000u) atomicAdd(&sh.hist[0][SAMPLE_BINS - 1].x, 1u);
    }
    sample_count(sh.hist[0], bits != 0u && bits <= 0x3f800000u, bits >> 20, bits);
  }
  cluster_sync_all();
  int turn = 1;
  unsigned long long l1_excl, l1_incl;
  {
    const int b = SAMPLE_BINS - 1 - tid;
    unsigned long long mass = 0;
#pragma unroll
    for (int q = 0; q < CL; ++q) {
      const uint2 v = ld_peer_u2(peer_addr(&sh.hist[0][b], q));
      mass += v.x + ((unsigned long long)v.y << 12);
    }
    if (b == SAMPLE_BINS - 1) {
      sh.bad = mass != 0;
      mass = 0;
    }
    const int shift = max(b >> 3, 1) - (150 - SAMPLE_UNIT);
    mass = shift >= 0 ? mass << shift : -shift < 64 ? mass >> -shift : 0ull;
    l1_incl = sample_scan(sh, mass, l1_excl);
    if (tid == SAMPLE_THREADS - 1) sh.total = l1_incl;
  }
  __syncthreads();
  if (sh.bad || sh.total == 0ull) {          // a row with something that is no number: token 0
    if (rank == 0 && tid == 0) out[r] = 0;
    cluster_sync_all();
    return;
  }
  const float u = (float)((double)philox_word0(positions[2 * r], positions[2 * r + 1], keys[2 * r],
                                               keys[2 * r + 1]) * 2.3283064365386963e-10);
  const float tp = top_p[r];
  unsigned long long head = sh.total;
  // a share of a mass, at least one unit (a draw of exactly 0 falls on the first rank) and at most the mass
  auto share_of = [](float share, unsigned long long mass) {
    const double d = ceil((double)share * (double)mass);
    return d < 1.0 ? 1ull : d >= (double)mass ? mass : (unsigned long long)d;
  };
  if (tp < 1.0f) {
    sample_select<CL>(sh, sample_e, live, begin, turn, l1_excl, l1_incl, share_of(tp, head), nullptr);
    head = sh.through;
  }
  sample_select<CL>(sh, sample_e, live, begin, turn, l1_excl, l1_incl, share_of(u, head), &out[r]);
  cluster_sync_all();                        // no block leaves while a peer may still read its shared memory
}

template <int CL>
cudaLaunchConfig_t sample_config(int rows, size_t smem, cudaStream_t stream, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(rows * CL));
  cfg.blockDim = dim3(SAMPLE_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ls_dependent_launch ? 2 : 1;
  return cfg;
}

// Rows that run at one time when each is spread over CL blocks (a block takes an SM's registers).
template <int CL>
int sample_rows_at_once() {
  static int rows = 0;
  if (rows == 0) {
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = sample_config<CL>(1, 0, nullptr, attr);
    if (cudaOccupancyMaxActiveClusters(&rows, sample_cluster_kernel<CL>, &cfg) != cudaSuccess || rows <= 0) {
      cudaGetLastError();
      rows = 96 / CL;
    }
  }
  return rows;
}

template <int CL>
int launch_sample_cluster(const float* logits, const float* temperature, const float* top_p, const uint32_t* keys,
                          const uint32_t* positions, int* out, int rows, int vocab, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(sample_cluster_kernel<CL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             SAMPLE_PART * (int)sizeof(float)) != cudaSuccess)
      return LS_E_SMEM;
    configured = true;
  }
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = sample_config<CL>(rows, (size_t)((vocab + CL - 1) / CL) * sizeof(float), stream, attr);
  LS_COUNT(LS_K_SAMPLE);
  cudaLaunchKernelEx(&cfg, sample_cluster_kernel<CL>, logits, temperature, top_p, keys, positions, out, vocab);
  return ls_launch_status();
}

// argmax in two stages, so that a few rows of a wide vocabulary fill the device:
// stage 1 reduces contiguous chunks of a row, stage 2 the chunks' winners.
constexpr int ARGMAX_CHUNKS = 64;

__global__ void argmax_chunk_kernel(const float* __restrict__ logits, float* __restrict__ cval,
                                    int* __restrict__ cidx, int vocab) {
  ls_dependency_sync();
  __shared__ float sval[32];
  __shared__ int sidx[32];
  const int r = blockIdx.x, c = blockIdx.y;
  const int per = (vocab + ARGMAX_CHUNKS - 1) / ARGMAX_CHUNKS;
  const int lo = c * per, hi = lo + per < vocab ? lo + per : vocab;
  ArgMax best{-CUDART_INF_F, 0x7fffffff};
  if (lo < hi) {
    const ArgMax local = block_argmax(logits + (int64_t)r * vocab + lo, hi - lo, sval, sidx);
    best.v = local.v;
    best.i = local.i + lo;
    // a chunk of NaN only: block_argmax reports index 0 with value -inf; keep it out of the way
    if (!(local.v > -CUDART_INF_F)) best.i = 0x7fffffff;
  }
  if (threadIdx.x == 0) {
    cval[r * ARGMAX_CHUNKS + c] = best.v;
    cidx[r * ARGMAX_CHUNKS + c] = best.i;
  }
}

__global__ void argmax_final_kernel(const float* __restrict__ cval, const int* __restrict__ cidx,
                                    int* __restrict__ out) {
  ls_dependency_sync();
  const int r = blockIdx.x;
  ArgMax best{cval[r * ARGMAX_CHUNKS + threadIdx.x], cidx[r * ARGMAX_CHUNKS + threadIdx.x]};
  // 64 candidates: two per lane of one warp
  if (threadIdx.x < 32) {
    ArgMax second{cval[r * ARGMAX_CHUNKS + 32 + threadIdx.x], cidx[r * ARGMAX_CHUNKS + 32 + threadIdx.x]};
    best = better(best, second);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgMax peer{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
      best = better(best, peer);
    }
    if (threadIdx.x == 0) out[r] = best.i == 0x7fffffff ? 0 : best.i;
  }
}

}  // namespace

// scratch: rows * 64 floats followed by rows * 64 ints (the caller's; rows * 512 bytes)
LS_API int ls_argmax(const float* logits, int* out, void* scratch, int rows, int vocab,
                     cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (scratch == nullptr || vocab < 4 * ARGMAX_CHUNKS) {
    LS_COUNT(LS_K_ARGMAX), ls_launch(argmax_kernel, rows, 512, 0, stream, logits, out, vocab);
    return ls_launch_status();
  }
  float* cval = (float*)scratch;
  int* cidx = (int*)(cval + (size_t)rows * ARGMAX_CHUNKS);
  LS_COUNT(LS_K_ARGMAX), ls_launch(argmax_chunk_kernel, dim3(rows, ARGMAX_CHUNKS), 256, 0, stream, logits, cval, cidx, vocab);
  ls_launch(argmax_final_kernel, rows, 32, 0, stream, cval, cidx, out);
  return ls_launch_status();
}

// How many floats of scratch ls_sample needs for its probabilities: none where a row fits the
// shared memory of a cluster (vocabularies up to 163,840), else rows x vocab.
LS_API long long ls_sample_scratch_floats(int rows, int vocab) {
  return vocab <= SAMPLE_MOST ? 0LL : (long long)rows * vocab;
}

// probs: scratch of ls_sample_scratch_floats(rows, vocab) floats (may be null when that is 0).
// keys, positions: [rows, 2] uint32 (low, high).
LS_API int ls_sample(const float* logits, float* probs, const float* temperature,
                     const float* top_p, const uint32_t* keys, const uint32_t* positions, int* out,
                     int rows, int vocab, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (vocab <= SAMPLE_MOST) {
    // as many blocks a row as still run all rows at once (a row's token does not depend on how it is
    // spread: 16 rows of 151,936 over 8 blocks each take two rounds, 66 us, over 4 one, 38); where no
    // spread does, the fewest blocks that hold a row
#define LS_SAMPLE_AS(CL) \
  return launch_sample_cluster<CL>(logits, temperature, top_p, keys, positions, out, rows, vocab, stream)
    if (rows <= sample_rows_at_once<8>()) LS_SAMPLE_AS(8);
    if (vocab > 2 * SAMPLE_PART || rows <= sample_rows_at_once<4>()) LS_SAMPLE_AS(4);
    if (vocab > SAMPLE_PART || rows <= sample_rows_at_once<2>()) LS_SAMPLE_AS(2);
    LS_SAMPLE_AS(1);
#undef LS_SAMPLE_AS
  }
  if (probs == nullptr) return LS_E_SIZE;
  LS_COUNT(LS_K_SAMPLE), ls_launch(sample_kernel, rows, SAMPLE_THREADS, 0, stream, logits, probs, temperature, top_p, keys,
                                                     positions, out, vocab);
  return ls_launch_status();
}

LS_API const char* ls_constants_sampling() {
  static char buf[256];
  static const LsConstant c[] = {{"argmax.chunks", ARGMAX_CHUNKS}, {"sample.threads", SAMPLE_THREADS},
                                 {"sample.cluster_blocks", SAMPLE_CLUSTER}, {"sample.cluster_vocab", SAMPLE_MOST}};
  return ls_format_constants(buf, sizeof buf, c, (int)(sizeof c / sizeof c[0]));
}
