// Causal attention of prompt portions over the paged cache on the CUDA cores, float32, head sizes
// 64 and 128: the sums of attention_tile_kernel (attention_simt.cu), element by element, for tiles
// of 32 or 64 tokens of one head.
//
// Why: the tile kernel's threads hold one row of queries each, so that every 16-byte piece of a
// key or a value read from shared memory feeds four FMAs.  Here a thread holds R rows (2 or 4):
// scores of R rows x 4 keys, outputs of R rows x D / 8 dimensions, so that a piece feeds 4 R FMAs;
// the next tile of keys and values is on its way (cp.async) while this one is used.  What bounds
// it: reads of shared memory (an SM delivers a 16-byte piece to 32 threads in 4 cycles, in which it
// does 16 of a warp's FMAs) and the FMAs.  16 heads of 128: prompts of 300, 600 and 900 tokens
// 339 us in tiles of 64 (559 us in tiles of 16), 1,024 tokens after 777 others 549 us (1,100), 173
// tokens in tiles of 32 36 us (55).
//
// The order of every sum is the tile kernel's: a score is one chain over the head's elements, an
// output one chain over the 32 keys of a tile (after its scaling), the weights of a tile are summed
// over groups of four neighbouring keys and then a tree, splits of LS_SPLIT keys at fixed positions
// are folded in ascending order.  A row's bits therefore depend on its own position only, and are
// those of a decoded token's splits and of the 16-token tiles.
//
// A key that a row does not see has the weight 0 and changes nothing, unless its value is an infinity
// or NaN: 0 times that is NaN, and larger tiles would carry it to rows whose 16-token tile never reads
// the key.  An item with a NaN among its results is therefore done again in groups of 16 tokens, each over
// the keys of its own 16-token tile (in an item without one this costs a vote of the block).
#include <math_constants.h>

#include "attention_fold.cuh"
#include "common.cuh"

namespace {

constexpr int KEYS = 32;          // keys of a tile: fixed by the order of the sums

__device__ __forceinline__ void copy16_or_zero(float* dst, const float* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int bytes = src != nullptr ? 16 : 0;             // 0: sixteen bytes of zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

template <int D, int R>
struct RowsShare {
  static constexpr int PITCH = D + 4;          // rows of Q and K: 16-byte pieces of eight rows fall into different banks
  static constexpr int PP = KEYS + 4;
  static constexpr int ROWS = 16 * R;
  float q[ROWS][PITCH];
  float k[2][KEYS][PITCH];
  float v[2][KEYS][D];
  float p[ROWS][PP];
};

struct RowsArgs {
  const float *__restrict__ q, *__restrict__ pages;
  float* __restrict__ out;
  const int *__restrict__ work, *__restrict__ block_table;
  int table_stride, nq, nkv, page_size, num_pages, window, keep_first;
  float scale, softcap;
  const float *__restrict__ slopes, *__restrict__ log_rates, *__restrict__ sinks;
  int* err;
};

// The rows of this block's item, or (ONE_GROUP) only those of a group of 16 tokens over the keys of its own 16-token
// tile.  Returns whether this thread has written a NaN.
template <int D, int R, bool ONE_GROUP>
__device__ __forceinline__ bool rows_pass(const RowsArgs& args, int group) {
  const float *__restrict__ q = args.q, *__restrict__ pages = args.pages;
  float* __restrict__ out = args.out;
  const float *__restrict__ slopes = args.slopes, *__restrict__ log_rates = args.log_rates, *__restrict__ sinks = args.sinks;
  const int nq = args.nq, nkv = args.nkv, page_size = args.page_size, num_pages = args.num_pages;
  const int window = args.window, keep_first = args.keep_first;
  const float scale = args.scale, softcap = args.softcap;
  int* err = args.err;
  typedef RowsShare<D, R> Share;
  extern __shared__ __align__(16) float rows_smem[];
  Share& sh = *reinterpret_cast<Share*>(rows_smem);
  const int* w = args.work + (int64_t)blockIdx.x * 8;
  const int req_row = w[0], tok0 = w[1], ntok = w[2], pos0 = w[3];
  const int h = (int)blockIdx.y, kvh = h / (nq / nkv);
  const int tid = threadIdx.x, mg = tid >> 3, sub = tid & 7;
  const int* table_row = args.block_table + (int64_t)req_row * args.table_stride;
  // (a group's bounds: what the plan of 16-token tiles has)
  const int first = ONE_GROUP ? pos0 + 16 * group : pos0;
  const int pos_last = ONE_GROUP ? min(first + 15, pos0 + ntok - 1) : pos0 + ntok - 1;
  const int key_lo_tile = ls_first_key(first, window);
  const int split_begin = ONE_GROUP ? key_lo_tile / LS_SPLIT : w[4];
  const int split_end = ONE_GROUP ? pos_last / LS_SPLIT + 1 : w[5];
  const int leading = ONE_GROUP ? min((keep_first + LS_SPLIT - 1) / LS_SPLIT, split_begin) : w[7];
  const float slope = slopes != nullptr ? slopes[h] : 0.f;
  const float log_rate = log_rates != nullptr ? log_rates[h] : 0.f;

  // the tiles of the item: splits split_begin .. split_end - 1 after the leading ones, tiles at fixed
  // offsets from a split's start; those wholly before the first row's window (and behind the kept
  // first keys) change nothing and are skipped
  struct Cursor { int turn, n0, s_hi; };
  auto enter = [&](Cursor& c) {
    const int split = c.turn < split_begin ? c.turn - (split_begin - leading) : c.turn;
    const int s_lo = split * LS_SPLIT;
    c.s_hi = min(s_lo + LS_SPLIT, pos_last + 1);
    c.n0 = key_lo_tile > s_lo && s_lo >= keep_first ? s_lo + ((key_lo_tile - s_lo) / KEYS) * KEYS : s_lo;
  };
  auto settle = [&](Cursor& c) {             // forward to a tile that counts; false at the end
    while (c.turn < split_end) {
      if (c.n0 < c.s_hi) {
        if (!(c.n0 >= keep_first && c.n0 + KEYS <= key_lo_tile)) return true;
        c.n0 += KEYS;
      } else if (++c.turn < split_end) {
        enter(c);
      }
    }
    return false;
  };
  auto fetch = [&](const Cursor& c, int buf) {   // four threads a key, its 16-byte pieces in turn
    const int n = tid >> 2, key = c.n0 + n;
    const float* kp = nullptr;
    if (key < c.s_hi && ls_sees(key, key_lo_tile, keep_first)) {
      const int page = table_row[key / page_size];
      if (page < 0 || page >= num_pages) ls_record_fault(err, LS_DEV_PAGE_RANGE, key);
      else kp = pages + ((((int64_t)page * 2) * nkv + kvh) * page_size + (key % page_size)) * D;
    }
    const int64_t to_v = (int64_t)nkv * page_size * D;
#pragma unroll
    for (int b = 0; b < D / 16; ++b) {
      const int c4 = 4 * ((tid & 3) + 4 * b);
      copy16_or_zero(&sh.k[buf][n][c4], kp != nullptr ? kp + c4 : nullptr);
      copy16_or_zero(&sh.v[buf][n][c4], kp != nullptr ? kp + to_v + c4 : nullptr);
    }
  };

  Cursor cur;
  cur.turn = split_begin - leading;
  enter(cur);
  bool more = settle(cur);
  if (more) fetch(cur, 0);
  for (int i = tid; i < Share::ROWS * (D / 4); i += 128) {
    const int r = i / (D / 4), c4 = 4 * (i - r * (D / 4));
    copy16_or_zero(&sh.q[r][c4], r < ntok ? q + ((int64_t)(tok0 + r) * nq + h) * D + c4 : nullptr);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");

  float acc_run[R][D / 8], m_run[R], l_run[R], m_s[R], l_s[R];
  float2 acc_s[R][D / 16];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    m_run[i] = m_s[i] = -CUDART_INF_F;
    l_run[i] = l_s[i] = 0.f;
#pragma unroll
    for (int j = 0; j < D / 8; ++j) acc_run[i][j] = 0.f;
#pragma unroll
    for (int j = 0; j < D / 16; ++j) acc_s[i][j] = make_float2(0.f, 0.f);
  }

  for (int buf = 0; more; buf ^= 1) {
    Cursor nxt = cur;
    nxt.n0 += KEYS;
    const bool next_more = settle(nxt);
    // (the buffer the next tile goes to was last read before the barrier that ended the tile before)
    if (next_more) fetch(nxt, buf ^ 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();

    // scores of rows mg + 16 i and keys sub + 8 j: each one chain over the head's elements
    float dot[R][4], alphas[R];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dot[i][j] = 0.f;
#pragma unroll 4
    for (int c = 0; c < D; c += 4) {
      float4 q4[R], k4[4];
#pragma unroll
      for (int i = 0; i < R; ++i) q4[i] = *reinterpret_cast<const float4*>(&sh.q[mg + 16 * i][c]);
#pragma unroll
      for (int j = 0; j < 4; ++j) k4[j] = *reinterpret_cast<const float4*>(&sh.k[buf][sub + 8 * j][c]);
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          dot[i][j] = fmaf(q4[i].x, k4[j].x, dot[i][j]);
          dot[i][j] = fmaf(q4[i].y, k4[j].y, dot[i][j]);
          dot[i][j] = fmaf(q4[i].z, k4[j].z, dot[i][j]);
          dot[i][j] = fmaf(q4[i].w, k4[j].w, dot[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int m = mg + 16 * i, qpos = pos0 + m;
      const int row_lo = ls_first_key(qpos, window);
      float s[4], tile_max = -CUDART_INF_F;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = cur.n0 + sub + 8 * j;
        const bool keep = m < ntok && key < cur.s_hi && key <= qpos && ls_sees(key, row_lo, keep_first);
        s[j] = !keep ? -CUDART_INF_F
               : log_rates != nullptr ? ls_capped(dot[i][j] * scale, softcap) - slope * log1pf(log_rate * (float)(qpos - key))
               : slopes != nullptr ? fmaf(slope, (float)(key - qpos), ls_capped(dot[i][j] * scale, softcap))
                                   : ls_capped(dot[i][j] * scale, softcap);
        tile_max = fmaxf(tile_max, s[j]);
      }
      tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 1));
      tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 2));
      tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 4));
      const float m_new = fmaxf(m_s[i], tile_max);
      float alpha = 1.f, p[4] = {0.f, 0.f, 0.f, 0.f};
      if (m_new != -CUDART_INF_F) {
        alpha = (m_s[i] == -CUDART_INF_F) ? 0.f : expf(m_s[i] - m_new);
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = (s[j] == -CUDART_INF_F) ? 0.f : expf(s[j] - m_new);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) sh.p[m][sub + 8 * j] = p[j];
      m_s[i] = m_new;
#pragma unroll
      for (int j = 0; j < D / 16; ++j) {
        acc_s[i][j].x = __fmul_rn(acc_s[i][j].x, alpha);
        acc_s[i][j].y = __fmul_rn(acc_s[i][j].y, alpha);
      }
      alphas[i] = alpha;
    }
    __syncwarp();                             // a row's weights are written and read by its eight lanes
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float4 g4 = *reinterpret_cast<const float4*>(&sh.p[mg + 16 * i][sub * 4]);
      float psum = 0.f;
      psum += g4.x;
      psum += g4.y;
      psum += g4.z;
      psum += g4.w;
      psum += __shfl_xor_sync(0xffffffffu, psum, 1);
      psum += __shfl_xor_sync(0xffffffffu, psum, 2);
      psum += __shfl_xor_sync(0xffffffffu, psum, 4);
      l_s[i] = __fmaf_rn(l_s[i], alphas[i], psum);
    }
    // outputs of rows mg + 16 i, dimensions sub * 4 + 32 jj + 0 .. 3: one chain over the tile's keys
#pragma unroll 2
    for (int n = 0; n < KEYS; n += 4) {
      float4 p4[R];
#pragma unroll
      for (int i = 0; i < R; ++i) p4[i] = *reinterpret_cast<const float4*>(&sh.p[mg + 16 * i][n]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
#pragma unroll
        for (int jj = 0; jj < D / 32; ++jj) {
          const float4 v4 = *reinterpret_cast<const float4*>(&sh.v[buf][n + e][sub * 4 + 32 * jj]);
#pragma unroll
          for (int i = 0; i < R; ++i) {
            const float pn = e == 0 ? p4[i].x : e == 1 ? p4[i].y : e == 2 ? p4[i].z : p4[i].w;
            ls_fma_pair(acc_s[i][2 * jj], pn, make_float2(v4.x, v4.y));
            ls_fma_pair(acc_s[i][2 * jj + 1], pn, make_float2(v4.z, v4.w));
          }
        }
      }
    }
    if (!next_more || nxt.turn != cur.turn) {   // the split ends: folded into the row
#pragma unroll
      for (int i = 0; i < R; ++i) {
        float alpha, beta, m_new;
        ls_fold_scales(m_run[i], m_s[i], alpha, beta, m_new);
        if (m_s[i] != -CUDART_INF_F) {
#pragma unroll
          for (int j = 0; j < D / 8; ++j)
            acc_run[i][j] = ls_fold_value(acc_run[i][j], alpha, j & 1 ? acc_s[i][j / 2].y : acc_s[i][j / 2].x, beta);
          l_run[i] = ls_fold_value(l_run[i], alpha, l_s[i], beta);
          m_run[i] = m_new;
        }
        m_s[i] = -CUDART_INF_F;
        l_s[i] = 0.f;
#pragma unroll
        for (int j = 0; j < D / 16; ++j) acc_s[i][j] = make_float2(0.f, 0.f);
      }
    }
    cur = nxt;
    more = next_more;
    __syncthreads();                          // everyone has read this tile: its buffer takes the one after the next
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");

  bool nan = false;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int m = mg + 16 * i;
    if (m >= ntok || (ONE_GROUP && i != group)) continue;
    if (sinks != nullptr) {
      // a sink: one more term exp(sinks[head]) in the softmax's denominator, with no value
      float alpha, beta, m_new;
      ls_fold_scales(m_run[i], sinks[h], alpha, beta, m_new);
#pragma unroll
      for (int j = 0; j < D / 8; ++j) acc_run[i][j] = __fmul_rn(acc_run[i][j], alpha);
      l_run[i] = ls_fold_value(l_run[i], alpha, 1.0f, beta);
    }
    float* o = out + ((int64_t)(tok0 + m) * nq + h) * D + sub * 4;
#pragma unroll
    for (int jj = 0; jj < D / 32; ++jj) {
      float4 y;
      y.x = l_run[i] > 0.f ? __fdiv_rn(acc_run[i][4 * jj], l_run[i]) : 0.f;
      y.y = l_run[i] > 0.f ? __fdiv_rn(acc_run[i][4 * jj + 1], l_run[i]) : 0.f;
      y.z = l_run[i] > 0.f ? __fdiv_rn(acc_run[i][4 * jj + 2], l_run[i]) : 0.f;
      y.w = l_run[i] > 0.f ? __fdiv_rn(acc_run[i][4 * jj + 3], l_run[i]) : 0.f;
      *reinterpret_cast<float4*>(o + 32 * jj) = y;
      nan |= !(y.x == y.x && y.y == y.y && y.z == y.z && y.w == y.w);
    }
  }
  return nan;
}

// (not inlined: the registers and the code of the usual pass stay its own)
template <int D, int R>
__device__ __noinline__ void rows_again(const RowsArgs& args, int ntok) {
  for (int group = 0; 16 * group < ntok; ++group) {
    __syncthreads();                          // everyone is done with the queries of the pass before
    rows_pass<D, R, true>(args, group);
  }
}

template <int D, int R>
__global__ void __launch_bounds__(128, 2) attention_rows_kernel(const __grid_constant__ RowsArgs args) {
  ls_dependency_sync();
  const int ntok = args.work[(int64_t)blockIdx.x * 8 + 2];
  if (ntok == 0) return;                     // padding item of a recorded launch
  if (__syncthreads_or(rows_pass<D, R, false>(args, 0))) rows_again<D, R>(args, ntok);
}

template <int D, int R>
int launch_rows(const RowsArgs& args, int n_work, cudaStream_t stream) {
  constexpr int smem = (int)sizeof(RowsShare<D, R>);
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(attention_rows_kernel<D, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return LS_E_SMEM;
    configured = true;
  }
  LS_COUNT(LS_K_ATTENTION_ROWS);
  ls_launch(attention_rows_kernel<D, R>, dim3(n_work, args.nq), 128, smem, stream, args);
  return ls_launch_status();
}

}  // namespace

// What the portions of a step (`tokens` in all, n16 / n32 / n64 tiles of 16 / 32 / 64 tokens) take in tiles of each
// size where there are many, in the same unit: a thread of the larger tiles holds all its rows whether they are
// filled or not, a row of the 16-token tile that is empty is half as dear as one that is not.  64 portions of 16 heads
// of 128 after 500 others, tiles of 16 / 32 / 64: of 2 tokens 219 / 442 / 518 us, of 8 279 / 442 / 517, of 14 414 / 483 / 584, of
// 17 674 / 490 / 571, of 40 1,109 / 867 / 593, of 65 1,759 / 1,370 / 1,210.
struct RowsCost {
  long long c16, c32, c64;
  RowsCost(int tokens, int n16, int n32, int n64) : c16(80LL * n16 + 5LL * tokens), c32(192LL * n32), c64(256LL * n64) {}
};

// The tile size that a step's portions are best cut into where there are many, whatever the heads.
LS_API int ls_attention_rows_tile_class(int tokens, int n16, int n32, int n64) {
  const RowsCost cost(tokens, n16, n32, n64);
  return cost.c64 < cost.c32 && cost.c64 < cost.c16 ? 64 : cost.c32 < cost.c16 ? 32 : 16;
}

// Tokens a work item should hold for portions of `tokens` tokens that make n16, n32 and n64 tiles: 16, which
// ls_attention_tile takes (as it does every other head size), 32 or 64.  More tiles than the two blocks an SM that run at
// one time: the cheapest, but 64 only where there are rows for most of the device's blocks (16 heads: 1,024 tokens
// after 777 others 549 us, with 32 705; 404 rows of 8 heads 39 us, with 32 25).  Fewer: a block's time counts and not their number, and
// 32 is faster down to a quarter of the SMs' rows (90 tokens of 16 heads 17.5 us, with 16 25.6; 16 portions of 8 tokens
// 10.1 and 13.2), or where tiles a quarter filled are on half of the SMs at most (4 portions of 8 tokens 7.6 and 10.3); fewer tokens take 16.
LS_API int ls_attention_rows_tile_tokens(int tokens, int n16, int n32, int n64, int nq, int d) {
  if ((d != 64 && d != 128) || tokens <= 0 || nq <= 0) return 16;
  const long long rows = (long long)tokens * nq, sms = ls_sm_count(), blocks = (long long)n32 * nq;
  if (blocks > 2 * sms) {
    const int best = ls_attention_rows_tile_class(tokens, n16, n32, n64);
    if (best != 64 || 2 * rows >= 64 * 3 * sms) return best;
    const RowsCost cost(tokens, n16, n32, n64);
    return cost.c32 < cost.c16 ? 32 : 16;
  }
  return 4 * rows >= 32 * sms || (2 * blocks <= sms && tokens >= 8LL * n32) ? 32 : 16;
}

// Work items as ls_attention_tile takes them in serial form, of up to `tile_tokens` (32 or 64) tokens.
LS_API int ls_attention_rows(const float* q, const float* pages, float* out, const int* work, int n_work, int tile_tokens,
                             const int* block_table, int table_stride, int nq, int nkv, int d, int page_size, int num_pages,
                             int window, int keep_first, float scale, float softcap, const float* slopes,
                             const float* log_rates, const float* sinks, int* err, cudaStream_t stream) {
  if (n_work <= 0) return 0;
  if (keep_first < 0 || (log_rates != nullptr && slopes == nullptr)) return LS_E_SIZE;
  if (nq <= 0 || nkv <= 0 || nq % nkv || nq > 65535 || page_size <= 0 || LS_SPLIT % page_size) return LS_E_SIZE;
  if (((uintptr_t)pages & 15) || ((uintptr_t)q & 15) || ((uintptr_t)out & 15)) return LS_E_ALIGN;
  const RowsArgs args = {q, pages, out, work, block_table, table_stride, nq, nkv, page_size, num_pages, window, keep_first,
                         scale, softcap, slopes, log_rates, sinks, err};
#define LS_ROWS(D, R) return launch_rows<D, R>(args, n_work, stream)
  if (d == 128 && tile_tokens == 64) LS_ROWS(128, 4);
  if (d == 128 && tile_tokens == 32) LS_ROWS(128, 2);
  if (d == 64 && tile_tokens == 64) LS_ROWS(64, 4);
  if (d == 64 && tile_tokens == 32) LS_ROWS(64, 2);
#undef LS_ROWS
  return LS_E_SIZE;
}

LS_API const char* ls_constants_attention_rows() {
  static char buf[128];
  static const LsConstant c[] = {{"attention_rows.keys", KEYS}, {"attention_rows.threads", 128}};
  return ls_format_constants(buf, sizeof buf, c, (int)(sizeof c / sizeof c[0]));
}
