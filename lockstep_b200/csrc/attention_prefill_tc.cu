// Attention of a portion of a prompt over the paged cache on the 5th-generation
// tensor cores: bfloat16, head sizes 64 and 128.  A block takes 128 query tokens of
// one request and one query head (a token is a row of the MMA tile, a lane of
// tensor memory, and a thread of a softmax team) and walks the keys in
// ascending tiles of 128, whose edges lie at multiples of 128 keys whatever the
// portion, so a row's arithmetic depends on its own position only.
//
//   S = Q K^T     tcgen05.mma, Q [128 x d] and the key tile [128 x d] K-major in
//                 shared memory (TMA, 128-byte swizzle), S in tensor memory
//   softmax       a thread reads its row's 128 scores from S with tcgen05.ld: maximum,
//                 p = exp2(s * scale * log2 e - m_ref), the sums of p over the tile's quarters; P
//                 rounded to bfloat16 goes back to tensor memory (tcgen05.st), two keys a column,
//                 over the scores it came from
//   PV            tcgen05.mma with P [128 x 128] as the A operand in tensor memory and the
//                 value tile [128 keys x d] as it lies in the cache (MN-major) in shared
//                 memory, adding to O in tensor memory over all tiles.  m_ref follows the
//                 row's maximum lazily (when it has grown by more than 8, a factor 256, the
//                 row of O is scaled and m_ref moved); O / l does not depend on m_ref.
//
// Twelve warps: warp 0 issues the MMAs, warp 1 fetches Q and the key tiles, warp 2 the value
// tiles (a lane per page of a tile: look-up and TMA box), warps 4..7 and 8..11 are two softmax
// teams that take the tiles in turn, a thread a row.  Tensor memory holds three S tiles and O, so
// S of the two tiles ahead is made while a tile's exponentials are taken.  Every wait is
// bounded; a wait that runs out records LS_DEV_WAIT_TIMEOUT and the block winds down and frees
// its tensor memory.
#include <cuda.h>
#include <math_constants.h>

#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int BLOCK_M = 128;              // query tokens per block
constexpr int BLOCK_N = 128;              // keys per tile
constexpr int STAGES = 2;                 // of Q, of keys and of values
constexpr int S_TILES = 3;                // S tiles in tensor memory
constexpr int UMMA_K = 16;
constexpr int HALF_BYTES = 128 * 128;     // 128 rows of 64 elements
constexpr uint32_t TMEM_COLS = 512;
constexpr int MMA_WARP = 0, K_WARP = 1, V_WARP = 2, TEAM_WARP = 4;
constexpr int THREADS = 12 * 32;
// Instances, so that none keeps registers for another's terms: plain scores; first keys that stay visible or sinks; a logarithmic bias; a
// linear bias, a cap or a scale that is not above 0 (times which -inf is not what a masked score is to be).  The last two take kept
// keys and sinks as well.
enum { PLAIN, KEPT_OR_SINK, LOG_BIAS, LINEAR_OR_CAP };
template <int V>
struct Kind {
  static constexpr int value = V;
};

// A key or value tile lies in groups of 8 keys, a group as its halves of 64 elements, a half as 8
// rows of 128 bytes (128-byte swizzle): what one TMA box of a page leaves (see encode_pages).
// MN-major operand (the value tile, d the major dimension): halves 1024 bytes apart (leading offset), groups of 8
// keys HALVES x 1024 (stride offset)
template <int HALVES>
__device__ __forceinline__ uint64_t desc_mn_major(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(1024 >> 4) << 16;
  d |= (uint64_t)((HALVES * 1024) >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// K-major operand whose groups of 8 rows are GROUP_BYTES apart
template <int GROUP_BYTES>
__device__ __forceinline__ uint64_t desc_k_major_groups(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(GROUP_BYTES >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int x0, int x1, int x2, int x3,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(smem_u32(bar)), "r"(x0), "r"(x1), "r"(x2), "r"(x3)
      : "memory");
}
// the same with the A operand in tensor memory (row = lane, two bfloat16 of neighbouring k a column)
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]),
        "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 2^x on the special-function unit, one instruction (inputs here are <= 0 or -inf)
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// tanh x = 1 - 2 / (1 + e^(2 x)), to float32 accuracy relative to one: what a capped score needs, which is this times the
// cap (the one-instruction tanh of the special-function unit keeps eleven bits)
__device__ __forceinline__ float tanh_of(float x) {
  return 1.0f - __fdividef(2.0f, 1.0f + ex2(x * 2.8853900817779268f));
}

// lg2 x on the special-function unit, one instruction (inputs here are >= 1)
__device__ __forceinline__ float lg2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two float32 lanes an instruction (sm_100: fma / add on pairs of registers) and the maximum of
// three: the softmax warps are short of issue slots, and each of these halves an instruction
// count without changing a result (every lane is rounded as the single instruction rounds it).
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// (x, y) = (a x + c, a y + c)
__device__ __forceinline__ void fma2(float& x, float& y, float a, float c) {
  uint64_t xy, aa, cc, r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(xy) : "f"(x), "f"(y));
  asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a));
  asm("mov.b64 %0, {%1, %1};" : "=l"(cc) : "f"(c));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(xy), "l"(aa), "l"(cc));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(r));
}
// (x, y) += (a, b)
__device__ __forceinline__ void add2(float& x, float& y, float a, float b) {
  uint64_t xy, ab, r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(xy) : "f"(x), "f"(y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(ab) : "f"(a), "f"(b));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(xy), "l"(ab));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(r));
}

// One work item of a block: up to 128 tokens of a request (rows of the MMA tile) and one query head.
struct Item {
  const int* table_row;
  int tok0, ntok, pos0, h, kvh;
  int pos_last, key_lo, tile_first, n_tiles;
  int lead;                  // tiles 0 .. lead - 1 come before tile_first (first keys that stay visible)
  // the place among all tiles of 128 keys of this item's tile `it`
  __device__ __forceinline__ int tile(int it) const { return it < lead ? it : tile_first + it - lead; }
};

// HALVES = d / 64.  Shared memory: two stages of Q [HALVES][128 rows][128 B], of K and of V [16 groups][HALVES][8 keys][128 B];
// barriers; what the teams hand each other.  Tensor memory: three S tiles (P over the S it came from), O.
//
// The kernel is persistent: a block per SM walks the items (work item x head, longest context
// first) in rounds, round r handing item r * blocks + b to block b, and every other round in the
// reverse order, so that a block with a long item gets a short one next.  Tiles count on over the items of
// a block (`g`): tile g is team g & 1's, lies in S tile g % 3 and in stage g & 1 of keys and values.  The
// MMA warp issues S two tiles ahead, into the next item too, whose Q has a stage of its own.
//
// What bounds it: MMAs (1,024 cycles a tile of 128 x 128 with d = 128), exponentials (1,024 on the special-function
// units), shared memory (160 KB a tile at 128 bytes a cycle) and L2 (64 KB a tile an SM) have to run side by side; a tile
// takes about 1,880 cycles, paced by S and PV one after the other and the issuing warp's waits between them (tensor pipe and
// special-function units half busy, L2 a quarter; a third stage of values changes nothing).  Measured, 16 query and 8 key heads of 128, pages of 16, with a
// head a block and four threads a row (two heads a block for the last two) / now: 2,048 tokens 30.5 / 25.9 us, 2,048 after
// 6,144 149.7 / 116.1 us, 8,192 277 / 248 us (1,110 TFLOP/s).
// Two teams on different tiles, with no chain between a tile's softmax and the next tile's S.  A row's sums need one
// order: m_ref of a row goes from team to team with the tiles (through shared memory and a named barrier of the two
// warps that share the row's quarter of tensor memory, before the exponentials are taken), and O is one accumulator.  The sum
// l of a row is four chains over the tiles, one of each quarter of a tile's keys (32), added in order at the end: a wholly
// masked tile changes none of them, so l does not depend on where the row's item begins.  The chains go from team to team with m_ref: at
// tile t a team gets them through tile t - 3, adds its own tile t - 2 and passes them on, so that none waits for exponentials; the team
// with the item's last tile adds the last two.  (With a sum of its own tiles a team, 2,048 tokens took 25.6 us and 8,192 245.8, now
// 25.9 and 247.7, but a row's bits depended on the parity of its tiles in the item.)
//
// KIND beyond PLAIN: the scores may get a bias that grows with the logarithm of the distance of key and query taken
// off (slopes[head] x ln(1 + log_rates[head] x distance): in the units of the exponentials,
// slopes[head] x lg2(1 + log_rates[head] x distance), one more special-function instruction a score),
// and the softmax's denominator one more term exp(sinks[head]) at the end of a row.  With slopes and no log_rates the
// bias is slopes[head] x distance, and with cap_log2 > 0 (a cap times lg2 e) the scaled score first becomes
// cap tanh(score / cap), again in the units of the exponentials.  keep_first > 0: the first
// keep_first keys of the sequence stay visible behind the window; their tiles come first.
template <int HALVES, int KIND>
__global__ void __launch_bounds__(THREADS, 1)
attention_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
                            __nv_bfloat16* __restrict__ out, const int* __restrict__ work, int n_work,
                            const int* __restrict__ block_table, int table_stride, int nq, int nkv, int page_size,
                            int num_pages, int window, int keep_first, float scale_log2, const float* __restrict__ slopes,
                            const float* __restrict__ log_rates, const float* __restrict__ sinks, float cap_log2, int* err) {
  ls_dependency_trigger();
  constexpr bool EXTRAS = KIND != PLAIN, BIASED = KIND == LOG_BIAS || KIND == LINEAR_OR_CAP;
  constexpr int D = HALVES * 64;
  constexpr int TILE_BYTES = HALVES * HALF_BYTES;        // K or V of one tile; also Q of one item
  constexpr int GROUP_BYTES = HALVES * 1024;             // 8 keys of a tile
  constexpr uint32_t O_COL = S_TILES * BLOCK_N;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t q_smem = base;                          // [STAGES]
  const uint32_t k_smem = q_smem + STAGES * TILE_BYTES;  // [STAGES]
  const uint32_t v_smem = k_smem + STAGES * TILE_BYTES;  // [STAGES]
  uint8_t* v_ptr = aligned + 2 * STAGES * TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(aligned + 3 * STAGES * TILE_BYTES);
  uint64_t* q_full = bars;             // [2] Q of an item landed
  uint64_t* q_free = bars + 2;         // [2] the item's last S product has read Q
  uint64_t* k_full = bars + 4;         // [2] keys of a tile landed
  uint64_t* v_full = bars + 6;         // [2] values landed
  uint64_t* k_free = bars + 8;         // [2] the S product has read the keys
  uint64_t* s_full = bars + 10;        // [3] S of a tile is in tensor memory
  uint64_t* p_full = bars + 13;        // [3] P of a tile is in tensor memory
  uint64_t* o_full = bars + 16;        // [2] PV of a tile has been added to O (and has read its values)
  uint64_t* o_free = bars + 18;        // the item's O has been read
  uint64_t* l_full = bars + 19;        // [4] the sums of the item's last tile but one lie in shared memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 23);
  volatile uint32_t* failed = tmem_slot + 1;
  float* hand_m = reinterpret_cast<float*>(bars + 32);   // [2 teams][128 rows] m_ref after a team's tile
  float4* hand_l = reinterpret_cast<float4*>(hand_m + 2 * 128);   // [2 teams][128 rows] the sums of weights through the tile two before
  float4* end_s = hand_l + 2 * 128;                      // [4][128 rows] the sums of an item's last tile but one
  float* end_f = reinterpret_cast<float*>(end_s + 4 * 128);       // [4][128 rows] and its rescaling

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total_items = n_work * nq;
  const int blocks = (int)gridDim.x;
  const int kept = EXTRAS ? keep_first : 0;

  // the item of this block in round `round`: 0 none is left, 1 an item, 2 a padding item (nothing to do)
  auto get_item = [&](int round, Item& I) -> int {
    const int idx = round * blocks + ((round & 1) ? blocks - 1 - (int)blockIdx.x : (int)blockIdx.x);
    if (idx >= total_items) return 0;
    const int wi = idx / nq;
    I.h = idx - wi * nq;
    const int* w = work + (int64_t)wi * 8;
    I.tok0 = w[1];
    I.ntok = w[2];
    I.pos0 = w[3];
    if (I.ntok == 0) return 2;
    I.table_row = block_table + (int64_t)w[0] * table_stride;
    I.kvh = I.h / (nq / nkv);
    I.pos_last = I.pos0 + I.ntok - 1;
    I.key_lo = ls_first_key(I.pos0, window);   // first key any row reads
    I.tile_first = I.key_lo / BLOCK_N;
    I.lead = kept > 0 ? min((kept + BLOCK_N - 1) / BLOCK_N, I.tile_first) : 0;
    I.n_tiles = I.pos_last / BLOCK_N + 1 - I.tile_first + I.lead;
    return 1;
  };

  const int rows_per_box = page_size < BLOCK_N ? page_size : BLOCK_N;
  const int boxes = BLOCK_N / rows_per_box;              // at most 16: lane b fetches box b of a tile
  // the page of this lane's box of tile `it` of an item, looked up one tile ahead (not yet checked)
  auto lookup = [&](const Item& I, int it) {
    int page = 0;
    if (it < I.n_tiles && lane < boxes) {
      int key = I.tile(it) * BLOCK_N + lane * rows_per_box;
      if (key > I.pos_last) key = I.pos_last;            // past the last key: any page that exists
      if (key >= kept && key < I.key_lo && key / page_size != I.key_lo / page_size)
        key = kept > 0 ? 0 : I.key_lo;                   // behind the window: pages may have been given back
      page = I.table_row[key / page_size];               // checked where it is used: the load stays in flight
    }
    return page;
  };
  // the work list and the block table are the step's inputs, older than the kernel before this
  // one: the first item's first look-up runs under the set-up below
  Item first_item;
  int first_page = 0;
  const bool producer = warp == K_WARP || warp == V_WARP;
  if (producer && get_item(0, first_item) == 1) first_page = lookup(first_item, 0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&q_free[s], 1);
      mbar_init(&k_full[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&k_free[s], 1);
      mbar_init(&o_full[s], 1);
    }
    for (int s = 0; s < S_TILES; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], 4);
    }
    for (int s = 0; s < 4; ++s) mbar_init(&l_full[s], 4);
    mbar_init(o_free, 4);
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_kv) : "memory");
  }
  if (warp == TEAM_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  ls_dependency_wait();                 // q and this step's keys and values come from the kernel before

  if (warp >= TEAM_WARP) {
    // ---- softmax: team 0 (warps 4..7) has the even tiles of the block, team 1 the odd ones; a
    // thread a row (a token, lane `row` of tensor memory), whose 128 scores lie in registers: the teams take
    // what the other warpgroup leaves of the block's 3 x 168 registers a thread ----
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    const int team = (warp - TEAM_WARP) >> 2;
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
    // O = sum of P V stays in tensor memory, the MMAs of every tile adding to it, in units of
    // 2^m_ref of its row.  m_ref follows the row's maximum lazily: only when the maximum has
    // grown by more than 8 (a factor 256, which bfloat16 P and float32 sums take easily) is the
    // row of O scaled down and m_ref moved, which after the first tiles hardly ever happens.
    // The quotient O / l does not depend on m_ref.
    constexpr float LAZY = 8.f;
    bool ok = true;
    int gt = 0, shared_items = 0;                 // tiles, and items of two or more tiles so far
    int s_tile = 0;                               // gt % 3
    uint32_t s_phase = 0;                         // (gt / 3) & 1

    // A wait that runs out clears `ok`; the loops still run to their ends, skipping the work, so
    // that every thread meets the named barriers of every tile of every item.
    for (int round = 0;; ++round) {
      Item I;
      const int kind = get_item(round, I);
      if (kind == 0) break;
      if (kind == 2) continue;
      const int pos0 = I.pos0, pos_last = I.pos_last, n_tiles = I.n_tiles;
      const int pos = pos0 + row;
      const int lo = ls_first_key(pos, window);
      const int lo_last = ls_first_key(pos_last, window);
      // m_ref: the row's, as this team knows it; quarter, factor: the sums of weights of this team's last tile, a sum a quarter
      // of its keys, and the tile's rescaling
      float m_ref = -CUDART_INF_F, factor = 1.f;
      float4 quarter = make_float4(0.f, 0.f, 0.f, 0.f);
      auto chained = [](float4 l, float f, float4 s) {
        return make_float4(fmaf(l.x, f, s.x), fmaf(l.y, f, s.y), fmaf(l.z, f, s.z), fmaf(l.w, f, s.w));
      };
      float bias_a = 0.f, bias_b = 0.f;
      if constexpr (KIND == LOG_BIAS) {
        bias_a = slopes[I.h];
        bias_b = log_rates[I.h];
      } else if constexpr (KIND == LINEAR_OR_CAP) {
        bias_a = slopes != nullptr ? slopes[I.h] * 1.4426950408889634f : 0.f;      // the slope in the exponentials' units
        bias_b = cap_log2 > 0.f ? scale_log2 / cap_log2 : 0.f;                     // score -> score x scale / cap
      }
      // with a bias the scores are put into the exponentials' units as they are read, and no scale is left
      const float scale_eff = BIASED ? 1.0f : scale_log2;
      for (int it = 0; it < n_tiles; ++it) {
        const int g = gt + it;
        const uint32_t s_addr = lane_base + (uint32_t)(s_tile * BLOCK_N);
        uint64_t* s_bar = &s_full[s_tile];
        uint64_t* p_bar = &p_full[s_tile];
        const uint32_t s_par = s_phase;
        if (++s_tile == S_TILES) {
          s_tile = 0;
          s_phase ^= 1u;
        }
        if ((g & 1) != team) continue;
        const int c0 = I.tile(it) * BLOCK_N;                         // first key of the tile
        if (ok && !mbar_wait(s_bar, s_par)) ok = false;
        fence_after_sync();
        // every key of the tile is seen by every row: no masks (uniform over the block); elsewhere a masked score
        // becomes -inf (selects and not branches), whose exponential is 0
        const bool full_tile = c0 + BLOCK_N - 1 <= pos0 && (c0 >= lo_last || c0 + BLOCK_N <= kept);
        if constexpr (BIASED) {
          // Bias and masks go over the scores in tensor memory, 32 at a time in a loop.  Unrolled over a row's 128 registers they are four
          // times the code, which a launch of a tile or two mostly fetches, and registers spilled (one instance for every bias).
          // 16 query and 8 key heads, us, that / this / four threads a row as it was before there were teams: logarithmic 2,048 tokens
          // 41.8 / 36.6 / 41.3, 2,048 after 6,144 in a window of 512 39.7 / 30.3 / 35.5; a cap 53.1 / 45.9 / 52.6; linear 46.0 / 38.2 / 39.4.
          // (A prompt of 25 tokens and two more in the 2,048 wide Malazen design: 1.31 / 1.26 / 1.27 ms.)
#pragma unroll 1
          for (int q0 = 0; q0 < BLOCK_N; q0 += 32) {
            uint32_t x[32];
            tmem_ld32(s_addr + q0, x);
            tmem_ld_wait();
            const int c = c0 + q0;
            const float d0 = (float)(pos - c);           // distance of the piece's first key (masked keys: clamped)
            if constexpr (KIND == LOG_BIAS) {
#pragma unroll
              for (int jj = 0; jj < 32; ++jj)
                x[jj] = __float_as_uint(fmaf(__uint_as_float(x[jj]), scale_log2, -bias_a * lg2(fmaf(bias_b, fmaxf(d0 - (float)jj, 0.f), 1.0f))));
            } else if (cap_log2 > 0.f) {
#pragma unroll
              for (int jj = 0; jj < 32; ++jj)
                x[jj] = __float_as_uint(fmaf(-bias_a, fmaxf(d0 - (float)jj, 0.f), cap_log2 * tanh_of(__uint_as_float(x[jj]) * bias_b)));
            } else {
#pragma unroll
              for (int jj = 0; jj < 32; ++jj)
                x[jj] = __float_as_uint(fmaf(-bias_a, fmaxf(d0 - (float)jj, 0.f), __uint_as_float(x[jj]) * scale_log2));
            }
            if (!full_tile) {
              const int after = pos - c;                             // the last place of the piece that the row sees
              const int from = kept > c ? kept - c : 0;              // between the kept keys and the window
              const uint32_t gap = lo - c > from ? (uint32_t)(lo - c - from) : 0u;
#pragma unroll
              for (int jj = 0; jj < 32; ++jj) x[jj] = (uint32_t)(jj - from) < gap ? __float_as_uint(-CUDART_INF_F) : x[jj];
#pragma unroll
              for (int jj = 0; jj < 32; ++jj) x[jj] = jj <= after ? x[jj] : __float_as_uint(-CUDART_INF_F);
            }
            tmem_st32(s_addr + q0, x);
          }
          tmem_st_wait();
        }
        uint32_t sc[BLOCK_N];
#pragma unroll
        for (int q0 = 0; q0 < BLOCK_N; q0 += 32) tmem_ld32(s_addr + q0, sc + q0);
        tmem_ld_wait();
        if (!BIASED && !full_tile) {
          const int after = pos - c0;                                // the last place of the tile that the row sees
          const int first = lo - c0;                                 // the first within its window
          if (c0 >= lo_last) {                                       // no window within the tile: the diagonal alone
#pragma unroll
            for (int jj = 0; jj < BLOCK_N; ++jj) sc[jj] = jj <= after ? sc[jj] : __float_as_uint(-CUDART_INF_F);
          } else if (EXTRAS && c0 < kept) {
            // between the kept keys and the window, then the diagonal (one condition for both took registers for 128 predicates)
            const int from = kept - c0;
            const uint32_t gap = first > from ? (uint32_t)(first - from) : 0u;
#pragma unroll
            for (int jj = 0; jj < BLOCK_N; ++jj) sc[jj] = (uint32_t)(jj - from) < gap ? __float_as_uint(-CUDART_INF_F) : sc[jj];
#pragma unroll
            for (int jj = 0; jj < BLOCK_N; ++jj) sc[jj] = jj <= after ? sc[jj] : __float_as_uint(-CUDART_INF_F);
          } else {
#pragma unroll
            for (int jj = 0; jj < BLOCK_N; ++jj) sc[jj] = jj >= first ? sc[jj] : __float_as_uint(-CUDART_INF_F);
#pragma unroll
            for (int jj = 0; jj < BLOCK_N; ++jj) sc[jj] = jj <= after ? sc[jj] : __float_as_uint(-CUDART_INF_F);
          }
        }
        float mx[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
        for (int jj = 0; jj < BLOCK_N; jj += 2)
          mx[(jj >> 1) & 3] = max3(mx[(jj >> 1) & 3], __uint_as_float(sc[jj]), __uint_as_float(sc[jj + 1]));
        const float tile_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        // m_ref after the tile before, from the other team (an item's first tile meets it too, for the
        // barrier's sake: a team may not announce two tiles before the other has taken the first)
        if (g > 0) asm volatile("bar.sync %0, 64;" ::"r"(1 + quad * 2 + ((g - 1) & 1)) : "memory");
        if (it > 0) m_ref = hand_m[((g - 1) & 1) * 128 + row];
        const float m_new = tile_max * scale_eff;
        const bool move = m_new > m_ref + LAZY;                      // true too for the first key a row sees
        // the chains through the other team's tile before the last come with m_ref, this team's last tile is added
        if (it > 1)
          hand_l[(g & 1) * 128 + row] =
              chained(it > 2 ? hand_l[((g - 1) & 1) * 128 + row] : make_float4(0.f, 0.f, 0.f, 0.f), factor, quarter);
        factor = move ? ((m_ref == -CUDART_INF_F) ? 0.f : ex2(m_ref - m_new)) : 1.f;
        if (move) m_ref = m_new;
        hand_m[(g & 1) * 128 + row] = m_ref;
        asm volatile("bar.arrive %0, 64;" ::"r"(1 + quad * 2 + (g & 1)) : "memory");
        // O is scaled only after the PV of the tile before has been added to it (and before this
        // tile's P is announced, so before the PV of this tile)
        if (it > 0 && __any_sync(0xffffffffu, move)) {
          if (ok && !mbar_wait(&o_full[(g - 1) & 1], (uint32_t)((g - 1) >> 1) & 1u)) ok = false;
          if (__all_sync(0xffffffffu, ok)) {
            fence_after_sync();
#pragma unroll
            for (int c = 0; c < D; c += 32) {
              uint32_t og[32];
              tmem_ld32(lane_base + O_COL + c, og);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 32; ++e) og[e] = __float_as_uint(__uint_as_float(og[e]) * factor);
              tmem_st32(lane_base + O_COL + c, og);
            }
          }
        }
        // p = exp2(s * scale - m_ref), rounded to bfloat16, two keys a column, written over scores this
        // thread has taken, from where the PV product takes it as its A operand; the sum of a quarter of the tile's keys
        // in four running sums, folded in a fixed order
        float sum[4];
        const bool dead = m_ref == -CUDART_INF_F;          // nothing seen yet by this row
        const float add = dead ? 0.f : -m_ref;
#pragma unroll
        for (int n0 = 0; n0 < BLOCK_N; n0 += 32) {
          uint32_t pk[16];
          float ps[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int jj = 0; jj < 32; jj += 4) {
            float p[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) p[e] = __uint_as_float(sc[n0 + jj + e]);
            fma2(p[0], p[1], scale_eff, add);
            fma2(p[2], p[3], scale_eff, add);
#pragma unroll
            for (int e = 0; e < 4; ++e) p[e] = ex2(p[e]);
            add2(ps[0], ps[1], p[0], p[1]);
            add2(ps[2], ps[3], p[2], p[3]);
            pk[jj >> 1] = pack_bf16(p[0], p[1]);
            pk[(jj >> 1) + 1] = pack_bf16(p[2], p[3]);
          }
          tmem_st16(s_addr + (n0 >> 1), pk);
          sum[n0 / 32] = (ps[0] + ps[1]) + (ps[2] + ps[3]);
        }
        if (__any_sync(0xffffffffu, dead && (sum[0] + sum[1]) + (sum[2] + sum[3]) != 0.f)) {
          // (a row that has seen scores that are no numbers and nothing else weighs nothing)
          tmem_st_wait();
#pragma unroll
          for (int c = 0; c < BLOCK_N / 2; c += 32) {
            uint32_t pk[32];
            tmem_ld32(s_addr + c, pk);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) pk[e] = dead ? 0u : pk[e];
            tmem_st32(s_addr + c, pk);
          }
          if (dead) sum[0] = sum[1] = sum[2] = sum[3] = 0.f;
        }
        // value rows of keys past the last position were never written: they must not be NaN,
        // since P is zero there and the MMA multiplies all the same
        if (c0 + BLOCK_N - 1 > pos_last) {
          if (ok && !mbar_wait(&v_full[g & 1], (uint32_t)(g >> 1) & 1u)) ok = false;
          if (ok && c0 + row > pos_last) {
            uint4* vrow = reinterpret_cast<uint4*>(v_ptr + (g & 1) * TILE_BYTES + (row >> 3) * GROUP_BYTES + (row & 7) * 128);
#pragma unroll
            for (int hh = 0; hh < HALVES; ++hh)
#pragma unroll
              for (int q8 = 0; q8 < 8; ++q8) vrow[hh * 64 + q8] = make_uint4(0u, 0u, 0u, 0u);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        tmem_st_wait();
        fence_before_sync();
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive(p_bar);
        quarter = make_float4(sum[0], sum[1], sum[2], sum[3]);
      }
      // ---- the item's end: the team that had the last tile takes what the other had of the tile before and writes
      // the rows out, while the other goes on to the next item ----
      const int g_last = gt + n_tiles - 1;
      const int lb = shared_items & 3;
      const uint32_t l_par = (uint32_t)(shared_items >> 2) & 1u;
      if ((g_last & 1) != team) {
        if (n_tiles > 1) {
          end_s[lb * 128 + row] = quarter;
          end_f[lb * 128 + row] = factor;
          __syncwarp();
          if (lane == 0) mbar_arrive(&l_full[lb]);
        }
      } else {
        float4 l = n_tiles > 2 ? hand_l[(g_last & 1) * 128 + row] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (n_tiles > 1) {
          if (ok && !mbar_wait(&l_full[lb], l_par)) ok = false;
          l = chained(l, end_f[lb * 128 + row], end_s[lb * 128 + row]);
        }
        l = chained(l, factor, quarter);
        float l_row = ((l.x + l.y) + l.z) + l.w;
        if constexpr (EXTRAS) {
          // the sink, in the units of this row's sums (2^m_ref)
          if (sinks != nullptr && m_ref != -CUDART_INF_F) l_row += ex2(fmaf(sinks[I.h], 1.4426950408889634f, -m_ref));
        }
        if (ok && !mbar_wait(&o_full[g_last & 1], (uint32_t)(g_last >> 1) & 1u)) ok = false;
        if (__all_sync(0xffffffffu, ok)) {
          fence_after_sync();
          uint32_t og[D];
#pragma unroll
          for (int c = 0; c < D; c += 32) tmem_ld32(lane_base + O_COL + c, og + c);
          tmem_ld_wait();
          fence_before_sync();                       // the next item's first PV overwrites O
          __syncwarp();
          if (lane == 0) mbar_arrive(o_free);
          if (row < I.ntok) {
            const float inv = l_row > 0.f ? 1.0f / l_row : 0.f;
            __nv_bfloat16* dst = out + ((int64_t)(I.tok0 + row) * nq + I.h) * D;
#pragma unroll
            for (int c = 0; c < D; c += 8) {
              uint4 v;
              v.x = pack_bf16(__uint_as_float(og[c]) * inv, __uint_as_float(og[c + 1]) * inv);
              v.y = pack_bf16(__uint_as_float(og[c + 2]) * inv, __uint_as_float(og[c + 3]) * inv);
              v.z = pack_bf16(__uint_as_float(og[c + 4]) * inv, __uint_as_float(og[c + 5]) * inv);
              v.w = pack_bf16(__uint_as_float(og[c + 6]) * inv, __uint_as_float(og[c + 7]) * inv);
              *reinterpret_cast<uint4*>(dst + c) = v;
            }
          }
        }
      }
      shared_items += n_tiles > 1 ? 1 : 0;
      gt += n_tiles;
    }
    // the announcement of the block's last tile is taken like any other
    if (gt > 0 && ((gt - 1) & 1) != team) asm volatile("bar.sync %0, 64;" ::"r"(1 + quad * 2 + ((gt - 1) & 1)) : "memory");
    if (!ok) {
      *failed = 1;
      if (lane == 0) ls_record_fault(err, LS_DEV_WAIT_TIMEOUT, 840 + quad);
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (producer) {
      // ---- producers: K_WARP fetches Q and the key tiles, V_WARP the value tiles: a key stage
      // is free earlier than the value stage of the same tile, and neither waits for the other's ----
      const bool keys = warp == K_WARP;
      uint64_t* free_bar = keys ? k_free : o_full;
      uint64_t* full_bar = keys ? k_full : v_full;
      const uint32_t dst_base = keys ? k_smem : v_smem;
      int g = 0, j = 0;                 // tiles and items of this block so far
      bool ok = true;
      for (int round = 0; ok; ++round) {
        Item I;
        const int kind = get_item(round, I);
        if (kind == 0) break;
        if (kind == 2) continue;
        int page = round == 0 ? first_page : lookup(I, 0);
        if (keys) {
          // a stage of Q is free once the last S product of the item before the one before has read it
          const int qs = j & 1;
          const uint32_t phase = (uint32_t)(j >> 1) & 1u;
          ok = __all_sync(0xffffffffu, *failed == 0 && mbar_wait(&q_free[qs], phase ^ 1u));
          if (!ok) {
            *failed = 1;
            if (lane == 0) ls_record_fault(err, LS_DEV_WAIT_TIMEOUT, 810);
            break;
          }
          if (lane == 0) {
            mbar_expect_tx(&q_full[qs], TILE_BYTES);
#pragma unroll
            for (int hh = 0; hh < HALVES; ++hh)
              tma_load_2d(q_smem + qs * TILE_BYTES + hh * HALF_BYTES, &map_q, I.h * D + hh * 64, I.tok0, &q_full[qs]);
          }
          __syncwarp();
        }
        ++j;
        for (int it = 0; it < I.n_tiles; ++it) {
          const int s = g & 1;
          const uint32_t phase = (uint32_t)(g >> 1) & 1u;
          const int c0 = I.tile(it) * BLOCK_N;
          ok = __all_sync(0xffffffffu, *failed == 0 && mbar_wait(&free_bar[s], phase ^ 1u));
          if (!ok) {
            *failed = 1;
            if (lane == 0) ls_record_fault(err, LS_DEV_WAIT_TIMEOUT, 800 + s);
            break;
          }
          if (lane == 0) mbar_expect_tx(&full_bar[s], TILE_BYTES);
          __syncwarp();
          if (lane < boxes) {
            if (page < 0 || page >= num_pages) {
              ls_record_fault(err, LS_DEV_PAGE_RANGE, c0 + lane * rows_per_box);
              page = 0;
            }
            const int in_page = ((c0 + lane * rows_per_box) % page_size) / rows_per_box * rows_per_box;
            const int y = ((page * 2 + (keys ? 0 : 1)) * nkv + I.kvh) * page_size + in_page;
            tma_load_4d(dst_base + (uint32_t)(s * TILE_BYTES + lane * (rows_per_box >> 3) * GROUP_BYTES), &map_kv, 0, 0, 0,
                        y >> 3, &full_bar[s]);
          }
          page = lookup(I, it + 1);     // after this tile's loads have gone out
          ++g;
        }
      }
      if (!ok && lane == 0) {
        // wait (bounded) for the copies still in flight before the block winds down
        for (int b = g > 2 ? g - 2 : 0; b < g; ++b) mbar_wait(&full_bar[b & 1], (uint32_t)(b >> 1) & 1u);
        if (keys)
          for (int b = j > 2 ? j - 2 : 0; b < j; ++b) mbar_wait(&q_full[b & 1], (uint32_t)(b >> 1) & 1u);
      }
    } else if (warp == MMA_WARP) {
      // ---- MMA issue: the whole warp walks the loop and one elected lane issues, so that the
      // instructions' operands are the same in every lane and stay in uniform registers (inside a
      // branch of one lane every MMA paid for moving them there) ----
      constexpr uint32_t idesc_s = instr_desc(BLOCK_M, BLOCK_N, false);
      constexpr uint32_t idesc_o = instr_desc(BLOCK_M, D, true);
      const bool issuer = elect_one();
      // two walks over the block's tiles: S runs two tiles ahead of PV
      struct Walk {
        int round, n, it, j, g;    // round to look at next; tiles of the item (0: none is left); tile, item and tiles so far
      };
      // What steers the loop comes out of a reduction over the warp, whose result lies in a uniform register: the
      // loop's state then stays there.  (Steered by values loaded from the work list, every MMA's descriptors and every
      // barrier's address were moved there one by one, 2,100 cycles of this warp a tile, and nothing else set the pace.)
      auto next_item = [&](Walk& w) {
        int n;
        do {
          Item I;
          const int kind = get_item(w.round, I);
          n = __reduce_max_sync(0xffffffffu, kind == 0 ? -1 : kind == 2 ? 0 : I.n_tiles);
          ++w.round;
        } while (n == 0);
        w.n = n > 0 ? n : 0;
        w.it = 0;
      };
      auto advance = [&](Walk& w) {
        ++w.g;
        if (++w.it == w.n) {
          ++w.j;
          next_item(w);
        }
      };
      const uint32_t tmem = __reduce_max_sync(0xffffffffu, tmem_base);
      const uint64_t q_desc = desc_k_major(q_smem), k_desc = desc_k_major_groups<GROUP_BYTES>(k_smem);
      const uint64_t v_desc = desc_mn_major<HALVES>(v_smem);
      Walk ws = {0, 0, 0, 0, 0};
      next_item(ws);
      Walk wp = ws;
      bool ok = true;
      int s_tile = 0;                   // ws.g % 3
      int p_tile = 0;                   // wp.g % 3 and the parity of wp.g / 3
      uint32_t p_phase = 0;
      // keys (and Q) of the tile at ws
      auto wait_s = [&]() {
        bool got = mbar_wait(&k_full[ws.g & 1], (uint32_t)(ws.g >> 1) & 1u);
        if (ws.it == 0) got = got && mbar_wait(&q_full[ws.j & 1], (uint32_t)(ws.j >> 1) & 1u);
        return got;
      };
      auto issue_s = [&]() {            // S of the tile at ws
        // (the S tile is free: the PV product of the tile that lay in it has been issued before)
        const int s = ws.g & 1, qs = ws.j & 1;
        if (issuer) {
#pragma unroll
          for (int k = 0; k < D / UMMA_K; ++k) {
            // (offsets in the descriptors' units of 16 bytes)
            const uint32_t qoff = (uint32_t)((k >> 2) * HALF_BYTES + (k & 3) * UMMA_K * 2) >> 4;
            const uint32_t koff = (uint32_t)((k >> 2) * 1024 + (k & 3) * UMMA_K * 2) >> 4;
            umma(tmem + s_tile * BLOCK_N, q_desc + (uint32_t)(qs * (TILE_BYTES >> 4)) + qoff,
                 k_desc + (uint32_t)(s * (TILE_BYTES >> 4)) + koff, idesc_s, k != 0 ? 1u : 0u);
          }
          umma_commit(&s_full[s_tile]);
          umma_commit(&k_free[s]);
          if (ws.it == ws.n - 1) umma_commit(&q_free[qs]);     // the item's last product with this Q
        }
        __syncwarp();
        if (++s_tile == S_TILES) s_tile = 0;
        advance(ws);
      };
      for (int ahead = 0; ahead < 2 && ok && ws.n != 0; ++ahead) {
        ok = __all_sync(0xffffffffu, wait_s());
        if (!ok) break;
        fence_after_sync();
        issue_s();
      }
      while (ok && wp.n != 0) {
        // what is there long before it is needed is waited for together, while the product before runs
        const int s = wp.g & 1;
        bool got = mbar_wait(&v_full[s], (uint32_t)(wp.g >> 1) & 1u);
        if (ws.n != 0) got = got && wait_s();
        ok = __all_sync(0xffffffffu, got);
        if (!ok) break;
        fence_after_sync();
        if (ws.n != 0) issue_s();
        got = mbar_wait(&p_full[p_tile], p_phase);
        // the first product of an item overwrites O
        if (wp.it == 0 && wp.j > 0) got = got && mbar_wait(o_free, (uint32_t)(wp.j - 1) & 1u);
        ok = __all_sync(0xffffffffu, got);
        if (!ok) break;
        fence_after_sync();
        if (issuer) {
#pragma unroll
          for (int k = 0; k < BLOCK_N / UMMA_K; ++k) {
            // P from tensor memory: 16 keys are 8 columns; V: 16 keys are two groups
            umma_ts(tmem + O_COL, tmem + p_tile * BLOCK_N + k * (UMMA_K / 2),
                    v_desc + (uint32_t)(s * (TILE_BYTES >> 4) + k * (2 * GROUP_BYTES >> 4)), idesc_o, (wp.it | k) != 0 ? 1u : 0u);
          }
          umma_commit(&o_full[s]);
        }
        __syncwarp();
        if (++p_tile == S_TILES) {
          p_tile = 0;
          p_phase ^= 1u;
        }
        advance(wp);
      }
      if (!ok) {
        *failed = 1;
        if (issuer) ls_record_fault(err, LS_DEV_WAIT_TIMEOUT, 820);
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == TEAM_WARP) {
    fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS)
                 : "memory");
  }
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
  static EncodeTiled fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
        qr == cudaDriverEntryPointSuccess)
      fn = (EncodeTiled)p;
  }
  return fn;
}

bool encode(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t rows, uint32_t box_rows) {
  EncodeTiled enc = encode_fn();
  if (enc == nullptr) return false;
  cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)inner * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  cuuint32_t elem[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The cache pages [rows = page, k or v, head, position][d] as {64 elements, 8 rows, halves, groups of 8 rows}: a box takes
// box_rows consecutive rows (a multiple of 8) and leaves them as groups of 8 rows, each as its halves, each 8 x 128 bytes.
// (One box a page instead of one a page and half: a warp gets a TMA load out about every 100 cycles.)
bool encode_pages(CUtensorMap* map, const void* ptr, uint64_t halves, uint64_t rows, uint32_t box_rows) {
  EncodeTiled enc = encode_fn();
  if (enc == nullptr) return false;
  const cuuint64_t pitch = (cuuint64_t)halves * 128;
  cuuint64_t dims[4] = {64, 8, (cuuint64_t)halves, (cuuint64_t)rows / 8};
  cuuint64_t strides[3] = {pitch, 128, 8 * pitch};
  cuuint32_t box[4] = {64, 8, (cuuint32_t)halves, box_rows / 8};
  cuuint32_t elem[4] = {1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, elem,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int sm_count() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  }
  return sms;
}

template <int HALVES, int KIND>
int launch(const CUtensorMap& map_q, const CUtensorMap& map_kv, void* out, const int* work, int n_work,
           const int* block_table, int table_stride, int nq, int nkv, int page_size, int num_pages, int window,
           int keep_first, float scale, const float* slopes, const float* log_rates, const float* sinks, float softcap,
           int* err, cudaStream_t stream) {
  constexpr size_t smem = (size_t)HALVES * HALF_BYTES * 3 * STAGES + 256 + (2 + 2 * 4 + 4 * 5) * 128 * 4 + 1024;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(attention_prefill_tc_kernel<HALVES, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
      return LS_E_SMEM;
    configured = true;
  }
  // a block per SM (its shared memory and its 512 columns of tensor memory fill one), or fewer items
  const long long items = (long long)n_work * nq;
  const int blocks = items < sm_count() ? (int)items : sm_count();
  LS_COUNT(LS_K_ATTENTION_PREFILL_TC), ls_launch(attention_prefill_tc_kernel<HALVES, KIND>, dim3(blocks), THREADS, smem, stream, map_q, map_kv,
            (__nv_bfloat16*)out, work, n_work, block_table, table_stride, nq, nkv, page_size, num_pages, window,
            keep_first, scale * 1.4426950408889634f, slopes, log_rates, sinks, softcap > 0.f ? softcap * 1.4426950408889634f : 0.f, err);
  return ls_launch_status();
}

}  // namespace

LS_API int ls_attention_prefill_tc_tile_tokens() { return BLOCK_M; }

// q, out: [tokens, nq * d] bfloat16; pages [num_pages, 2, nkv, page_size, d]; d 64 or 128; page
// sizes 8, 16, 32, 64, 128.  Work items as for ls_attention_tile with up to 128 tokens each
// (splits and slots are not used).  Returns LS_E_SIZE or LS_E_ALIGN for anything else, having
// launched nothing.
LS_API int ls_attention_prefill_tc(const void* q, const void* pages, void* out, int tokens, const int* work,
                                   int n_work, const int* block_table, int table_stride, int nq, int nkv, int d,
                                   int page_size, int num_pages, int window, int keep_first, float scale,
                                   const float* slopes, const float* log_rates, const float* sinks, float softcap,
                                   int* err, cudaStream_t stream) {
  if (n_work <= 0 || tokens <= 0) return 0;
  if (keep_first < 0) return LS_E_SIZE;
  if (log_rates != nullptr && (slopes == nullptr || softcap > 0.f)) return LS_E_SIZE;
  if (nq <= 0 || nkv <= 0 || nq % nkv || n_work > 65535) return LS_E_SIZE;
  if (d != 64 && d != 128) return LS_E_SIZE;
  if (page_size != 8 && page_size != 16 && page_size != 32 && page_size != 64 && page_size != 128) return LS_E_SIZE;
  const int64_t rows = (int64_t)num_pages * 2 * nkv * page_size;
  if (rows > 2147483647LL) return LS_E_SIZE;
  if (((uintptr_t)pages & 127) || ((uintptr_t)q & 15) || ((uintptr_t)out & 15)) return LS_E_ALIGN;
  CUtensorMap map_q, map_kv;
  if (!encode(&map_q, q, (uint64_t)nq * d, (uint64_t)tokens, BLOCK_M)) return LS_E_SIZE;
  if (!encode_pages(&map_kv, pages, (uint64_t)d / 64, (uint64_t)rows, page_size < BLOCK_N ? page_size : BLOCK_N)) return LS_E_SIZE;
  auto of = [&](auto kind) { return d == 64 ? launch<1, decltype(kind)::value> : launch<2, decltype(kind)::value>; };
  auto go = log_rates != nullptr ? of(Kind<LOG_BIAS>())
            : slopes != nullptr || softcap > 0.f || !(scale > 0.f) ? of(Kind<LINEAR_OR_CAP>())
            : sinks != nullptr || keep_first > 0 ? of(Kind<KEPT_OR_SINK>()) : of(Kind<PLAIN>());
  return go(map_q, map_kv, out, work, n_work, block_table, table_stride, nq, nkv, page_size, num_pages, window,
            keep_first, scale, slopes, log_rates, sinks, softcap, err, stream);
}

LS_API const char* ls_constants_attention_prefill_tc() {
  static char buf[256];
  static const LsConstant c[] = {{"attention_prefill_tc.queries", BLOCK_M}, {"attention_prefill_tc.keys", BLOCK_N},
                                 {"attention_prefill_tc.softmax_threads_per_row", 1}};
  return ls_format_constants(buf, sizeof buf, c, (int)(sizeof c / sizeof c[0]));
}
