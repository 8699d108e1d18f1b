// float32 attention of a decoded token: one token, one split of LS_SPLIT keys, one key head with its whole
// group of query heads; writes the partial that ls_attention_combine folds.  The sums of ls_attention_tile,
// element by element, so that a decoded row keeps the bits of the same row in a prompt: a score is one chain
// over the head's elements in ascending order, the weights of 32 keys are summed in groups of four neighbours and
// a tree, an output is one chain over the keys in ascending order with the rescaling of every 32 keys.
//
// What bounds it: the split's keys and values (2 x 256 x d floats, 256 KB at d = 128) and then two chains, d FMAs for the
// scores and 256 for the outputs.  attention_tile walks the split tile by tile, eight trips to memory one after the
// other with 2 of 16 rows in use.  Here the whole split is asked for at once (cp.async; all but the 32
// keys that hold the step's own token before the wait on the kernel before), a thread has one key's
// scores for all heads, a warp the 32 keys of a tile, and the maxima of the tiles are known together: three requests
// at contexts of 300 to 900, 16 query and 8 key heads of 128, 57 -> 6 us a layer.
#include <math_constants.h>

#include "common.cuh"

namespace {

constexpr int THREADS = LS_SPLIT;       // a thread a key
constexpr int TILE = 32;                // keys between two rescalings: attention_tile's
constexpr int TILES = LS_SPLIT / TILE;

__device__ __forceinline__ void copy16(float* dst, const float* src, bool live) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

struct Layout {
  int kp;          // pitch of a key row in floats
  int v_tiles;     // tiles of values beside the keys; the others take the keys' place after the scores
  size_t bytes;
};
// the keys, as many tiles of values as fit beside them (the rest where the keys were), the queries, the weights and
// the offsets of the keys
__host__ __device__ inline Layout layout(int d, int group) {
  Layout l;
  l.kp = d + 4;                         // 16-byte pieces stay aligned, eight rows read together fall into different banks
  const size_t fixed = sizeof(int64_t) * LS_SPLIT +
                       sizeof(float) * ((size_t)LS_SPLIT * l.kp + (size_t)group * (d + LS_SPLIT + 3 * TILES));
  const size_t tile = sizeof(float) * (size_t)TILE * d;
  const size_t room = (size_t)226 * 1024;
  l.v_tiles = fixed >= room ? 0 : (int)((room - fixed) / tile);
  if (l.v_tiles > TILES) l.v_tiles = TILES;
  l.bytes = fixed + l.v_tiles * tile;
  return l;
}

template <int G>
__global__ void __launch_bounds__(THREADS)
attention_split_kernel(const float* __restrict__ q, const float* __restrict__ pages, float* __restrict__ part_acc,
                       float* __restrict__ part_ml, const int* __restrict__ work, const int* __restrict__ block_table,
                       int table_stride, int nq, int nkv, int d, int page_size, int num_pages, int window, int keep_first,
                       float scale, int* err) {
  ls_dependency_trigger();
  extern __shared__ __align__(16) unsigned char smem[];
  const Layout l = layout(d, G);
  int64_t* offset = reinterpret_cast<int64_t*>(smem);                 // [256] of a key's row in `pages`, -1: not read
  float* Ks = reinterpret_cast<float*>(offset + LS_SPLIT);            // [256][kp]
  float* Vs = Ks + LS_SPLIT * l.kp;                                   // [32 v_tiles][d]
  float* Qs = Vs + (size_t)l.v_tiles * TILE * d;                      // [G][d]
  float* Ps = Qs + G * d;                                             // [G][256]
  float* tile_m = Ps + G * LS_SPLIT;                                  // [G][8] maxima, then
  float* tile_a = tile_m + G * TILES;                                 // [G][8] rescalings,
  float* tile_l = tile_a + G * TILES;                                 // [G][8] sums of weights

  const int* w = work + (int64_t)blockIdx.x * 8;
  if (w[2] == 0) return;                     // padding item of a recorded launch
  const int req_row = w[0], tok = w[1], pos = w[3], split = w[4], slot = w[6];
  const int kvh = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row_lo = ls_first_key(pos, window);
  const int s_lo = split * LS_SPLIT;
  int s_hi = s_lo + LS_SPLIT;
  if (s_hi > pos + 1) s_hi = pos + 1;
  const int tiles = (s_hi - s_lo + TILE - 1) / TILE;

  // (the work list, the block table and every key older than the step's own are there before the step's first kernel)
  const int key = s_lo + tid;
  const bool sees = key < s_hi && ls_sees(key, row_lo, keep_first);
  {
    int64_t at = -1;
    if (sees) {
      const int page = block_table[(int64_t)req_row * table_stride + key / page_size];
      if (page < 0 || page >= num_pages) ls_record_fault(err, LS_DEV_PAGE_RANGE, key);
      else at = ((((int64_t)page * 2) * nkv + kvh) * page_size + key % page_size) * d;
    }
    offset[tid] = at;
  }
  __syncthreads();
  const int pieces = d >> 2;
  const int64_t to_v = (int64_t)nkv * page_size * d;
  // tiles [from, to) of the keys or of the values, 16 bytes a copy; rows that are not read become zeros
  auto fetch = [&](bool values, int from, int to, float* dst, int pitch) {
    for (int i = tid + from * TILE * pieces; i < to * TILE * pieces; i += THREADS) {
      const int n = i / pieces, ch = i - n * pieces;
      const int64_t at = offset[n];
      copy16(dst + (size_t)(n - from * TILE) * pitch + ch * 4, at < 0 ? pages : pages + at + (values ? to_v : 0) + ch * 4, at >= 0);
    }
  };
  const int v_now = tiles < l.v_tiles ? tiles : l.v_tiles;            // tiles of values beside the keys
  const int old_tiles = pos < s_hi ? tiles - 1 : tiles;               // the split's last tile holds the step's own key
  const int old_v = old_tiles < v_now ? old_tiles : v_now;
  fetch(false, 0, old_tiles, Ks, l.kp);
  fetch(true, 0, old_v, Vs, d);
  ls_dependency_wait();
  fetch(false, old_tiles, tiles, Ks + (size_t)old_tiles * TILE * l.kp, l.kp);
  fetch(true, old_v, v_now, Vs + (size_t)old_v * TILE * d, d);
  for (int i = tid; i < G * d; i += THREADS) Qs[i] = q[((int64_t)tok * nq + kvh * G) * d + i];
  copies_done();
  __syncthreads();

  // scores of this thread's key for all heads of the group
  float s[G];
#pragma unroll
  for (int g = 0; g < G; ++g) s[g] = -CUDART_INF_F;
  if (sees) {
    float dot[G];
#pragma unroll
    for (int g = 0; g < G; ++g) dot[g] = 0.f;
    const float* kr = Ks + (size_t)tid * l.kp;
#pragma unroll 4
    for (int c = 0; c < d; c += 4) {
      const float4 k4 = *reinterpret_cast<const float4*>(kr + c);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float4 q4 = *reinterpret_cast<const float4*>(Qs + g * d + c);
        dot[g] = fmaf(q4.x, k4.x, dot[g]);
        dot[g] = fmaf(q4.y, k4.y, dot[g]);
        dot[g] = fmaf(q4.z, k4.z, dot[g]);
        dot[g] = fmaf(q4.w, k4.w, dot[g]);
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) s[g] = __fmul_rn(dot[g], scale);
  }
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const float m = ls_warp_max(s[g]);
    if (lane == 0) tile_m[g * TILES + warp] = m;
  }
  __syncthreads();                           // every thread has its scores: the keys' place is free
  if (v_now < tiles) fetch(true, v_now, tiles, Ks, d);

  // the running maximum after this warp's tile and before it: weights and the tile's rescaling
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float m_old = -CUDART_INF_F;
    for (int t = 0; t < warp; ++t) m_old = fmaxf(m_old, tile_m[g * TILES + t]);
    const float m_new = fmaxf(m_old, tile_m[g * TILES + warp]);
    float alpha = 1.f, p = 0.f;
    if (m_new != -CUDART_INF_F) {
      alpha = m_old == -CUDART_INF_F ? 0.f : expf(m_old - m_new);
      p = s[g] == -CUDART_INF_F ? 0.f : expf(s[g] - m_new);
    }
    Ps[g * LS_SPLIT + tid] = p;
    // four neighbouring keys in order, then a tree over the eight groups
    const int first = lane & ~3;
    float sum = 0.f;
    sum += __shfl_sync(0xffffffffu, p, first);
    sum += __shfl_sync(0xffffffffu, p, first + 1);
    sum += __shfl_sync(0xffffffffu, p, first + 2);
    sum += __shfl_sync(0xffffffffu, p, first + 3);
    sum += __shfl_xor_sync(0xffffffffu, sum, 4);
    sum += __shfl_xor_sync(0xffffffffu, sum, 8);
    sum += __shfl_xor_sync(0xffffffffu, sum, 16);
    if (lane == 0) {
      tile_a[g * TILES + warp] = alpha;
      tile_l[g * TILES + warp] = sum;
    }
  }
  __syncthreads();

  for (int u0 = 0; u0 < G * d; u0 += THREADS) {
    const int u = u0 + tid;
    const bool live = u < G * d;
    const int g = live ? u / d : 0, c = live ? u - g * d : 0;
    float a = 0.f;
    for (int t = 0; t < tiles; ++t) {
      if (u0 == 0 && t == v_now) {           // the values where the keys were
        copies_done();
        __syncthreads();
      }
      a = __fmul_rn(a, tile_a[g * TILES + t]);
      const float* vc = (t < v_now ? Vs + (size_t)t * TILE * d : Ks + (size_t)(t - v_now) * TILE * d) + c;
      const float* pr = Ps + g * LS_SPLIT + t * TILE;
#pragma unroll
      for (int n = 0; n < TILE; n += 4) {
        const float4 p4 = *reinterpret_cast<const float4*>(pr + n);
        a = fmaf(p4.x, vc[(n + 0) * d], a);
        a = fmaf(p4.y, vc[(n + 1) * d], a);
        a = fmaf(p4.z, vc[(n + 2) * d], a);
        a = fmaf(p4.w, vc[(n + 3) * d], a);
      }
    }
    if (live) part_acc[((int64_t)slot * nq + kvh * G + g) * d + c] = a;
  }
  if (tid < G) {
    float m = -CUDART_INF_F, sum = 0.f;
    for (int t = 0; t < tiles; ++t) {
      sum = __fmaf_rn(sum, tile_a[tid * TILES + t], tile_l[tid * TILES + t]);
      m = fmaxf(m, tile_m[tid * TILES + t]);
    }
    part_ml[((int64_t)slot * nq + kvh * G + tid) * 2 + 0] = m;
    part_ml[((int64_t)slot * nq + kvh * G + tid) * 2 + 1] = sum;
  }
}

template <int G>
int launch(const float* q, const float* pages, float* part_acc, float* part_ml, const int* work, int n_work,
           const int* block_table, int table_stride, int nq, int nkv, int d, int page_size, int num_pages, int window,
           int keep_first, float scale, int* err, cudaStream_t stream) {
  const Layout l = layout(d, G);
  static size_t configured = 0;
  if (l.bytes > configured) {
    if (cudaFuncSetAttribute(attention_split_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)l.bytes) !=
        cudaSuccess)
      return LS_E_SMEM;
    configured = l.bytes;
  }
  LS_COUNT(LS_K_ATTENTION_SPLIT), ls_launch(attention_split_kernel<G>, dim3(n_work, nkv), THREADS, l.bytes, stream, q, pages, part_acc,
            part_ml, work, block_table, table_stride, nq, nkv, d, page_size, num_pages, window, keep_first, scale, err);
  return ls_launch_status();
}

}  // namespace

// Work items of single tokens, a split each, as for ls_attention_tile with partials.  float32; groups of 1, 2, 4 and 8 heads
// (a thread keeps a score a head), head sizes to 128 that are multiples of 16 (half of the split's values fit
// beside its keys).  Returns LS_E_SIZE or LS_E_ALIGN for anything else, having launched nothing.
LS_API int ls_attention_split(const float* q, const float* pages, float* part_acc, float* part_ml, const int* work,
                              int n_work, const int* block_table, int table_stride, int nq, int nkv, int d, int page_size,
                              int num_pages, int window, int keep_first, float scale, int* err, cudaStream_t stream) {
  if (n_work <= 0) return 0;
  if (nq <= 0 || nkv <= 0 || nq % nkv || nkv > 65535 || keep_first < 0) return LS_E_SIZE;
  if (d < 16 || d > 128 || d % 16 || page_size <= 0 || LS_SPLIT % page_size) return LS_E_SIZE;
  if ((uintptr_t)pages & 15) return LS_E_ALIGN;
  const int group = nq / nkv;
  auto go = group == 1 ? launch<1> : group == 2 ? launch<2> : group == 4 ? launch<4> : group == 8 ? launch<8> : nullptr;
  if (go == nullptr) return LS_E_SIZE;
  return go(q, pages, part_acc, part_ml, work, n_work, block_table, table_stride, nq, nkv, d, page_size, num_pages, window,
            keep_first, scale, err, stream);
}
