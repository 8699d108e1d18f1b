// C[M, N] = A[M, K] * W[N, K]^T on the CUDA cores (FFMA, float32 accumulate).
//
// This is the true 32-bit matrix product of the engine and the fallback of the
// bfloat16 path for shapes the tensor-core kernel refuses.  An output element is
// one accumulator and one chain of FMAs over K in ascending order, so its value
// does not depend on M (the batch) or on where its row lies in the batch.  There
// is no split-K.  Three kernels make that same chain: the general one below (a
// block owns a 64x64 tile; any element type, any depth), one for up to 32
// float32 tokens and one for many float32 tokens.
//
// Epilogues:
//   0 store        C[m, n]  = acc                       (C of type TC)
//   1 residual     C[m, n] += acc                       (C float32, in place)
//   2 silu-mul     C[m, n]  = silu(acc_gate) * acc_up   (W holds gate rows [0, N)
//                                                        and up rows [N, 2N))
//   4 gelu         C[m, n]  = gelu_tanh(acc)
//   5 relu squared C[m, n]  = max(acc, 0)^2
#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, PAD = 4;

template <typename TA, typename TW, typename TC, int EPI>
__global__ void __launch_bounds__(256)
gemm_nt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TC* __restrict__ C, int M,
               int N, int K, int64_t lda, int64_t ldw, int64_t ldc) {
  ls_dependency_sync();
  __shared__ float As[BK][BM + PAD];
  __shared__ float Ws[BK][BN + PAD];
  __shared__ float Us[EPI == 2 ? BK : 1][BN + PAD];

  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

  float acc[4][4] = {};
  float acu[4][4] = {};

  // each thread stages 4 consecutive k of one row of A and of W
  const int lrow = tid >> 2;        // 0..63
  const int lk = (tid & 3) * 4;     // 0,4,8,12

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + lk + j;
      const int m = m0 + lrow, n = n0 + lrow;
      As[lk + j][lrow] = (m < M && k < K) ? ls_to_float<TA>(A[(int64_t)m * lda + k]) : 0.f;
      Ws[lk + j][lrow] = (n < N && k < K) ? ls_to_float<TW>(W[(int64_t)n * ldw + k]) : 0.f;
      if (EPI == 2)
        Us[lk + j][lrow] = (n < N && k < K) ? ls_to_float<TW>(W[(int64_t)(n + N) * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[4], w[4], u[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = Ws[k][tx * 4 + j];
      if (EPI == 2) {
#pragma unroll
        for (int j = 0; j < 4; ++j) u[j] = Us[k][tx * 4 + j];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
          if (EPI == 2) acu[i][j] = fmaf(a[i], u[j], acu[i][j]);
        }
    }
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      TC* c = C + (int64_t)m * ldc + n;
      if (EPI == 0) {
        *c = ls_from_float<TC>(acc[i][j]);
      } else if (EPI == 1) {
        *c = ls_from_float<TC>(ls_to_float<TC>(*c) + acc[i][j]);
      } else if (EPI == 4) {
        *c = ls_from_float<TC>(ls_gelu_tanh(acc[i][j]));
      } else if (EPI == 5) {
        *c = ls_from_float<TC>(ls_relu_squared(acc[i][j]));
      } else {
        const float g = acc[i][j];
        *c = ls_from_float<TC>(g / (1.0f + expf(-g)) * acu[i][j]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Few tokens (up to 32), float32: the decode step's products on the true 32-bit path.
// The tile kernel above would run a handful of blocks with most of their rows empty.  Here a
// warp's lanes are TL token lanes x 32 / TL feature lanes, a thread has FT features and MT tokens
// (silu-mul: the gate and the up row of every feature), each with the accumulator and the
// ascending chain of FMAs it has in the tile kernel (fmaf(a, w, acc) from k = 0 up), so the
// kernels give the same bits.  W and the token rows stream through a ring of shared-memory
// stages by 16-byte cp.async; the weights of the first stages are asked for before the wait on
// the kernel before.
//
// What bounds it: for a narrow weight the chain, 16 cycles for four steps of k, so its features
// are spread over the SMs; else what a thread reads from shared memory, (FT + MT) pieces of 16
// bytes (an SM delivers 32 of them in 4 cycles) for 4 FT MT FMAs, and for the widest (a head) the
// memory's rate.  3 tokens, weights 4,096 / 2 x 3,072 / 151,936 by 1,024: 7.5 / 13.0 / 135 us, 1,024 by
// 2,048 / 3,072: 9.5 / 14.6 us (a thread a feature and a token, 16 features a block: 13.5 / 24.8 / 280 and
// 17.5 / 25.1); floors of memory 2.6 / 3.9 / 96 and of the chain 4.2 / 6.3.
// ---------------------------------------------------------------------------
constexpr int SK_MAX_M = 32;

__device__ __forceinline__ void cp_async_16(float* dst, const float* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <bool GLU, int FT, int MT, int TL, int NW, int DEPTH>
struct Skinny {
  static constexpr int FL = 32 / TL;                     // feature lanes of a warp
  static constexpr int FEATURES = NW * FL * FT;          // of a block
  static constexpr int W_ROWS = GLU ? 2 * FEATURES : FEATURES;
  static constexpr int X_ROWS = TL * MT;
  static constexpr int PITCH = DEPTH + 4;                // rows: the pieces of eight of them fall into different banks
  static constexpr int STAGE = (W_ROWS + X_ROWS) * PITCH;          // floats
  static constexpr int FIT = 104 * 1024 / (STAGE * 4);
  static constexpr int STAGES = FIT > 8 ? 8 : FIT;
  static_assert(STAGES >= 2, "a stage too large");
};

// epilogue: 0, 1, 4 or 5 (silu-mul is the instance GLU)
template <bool GLU, int FT, int MT, int TL, int NW, int DEPTH>
__global__ void __launch_bounds__(32 * NW)
gemm_nt_skinny_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N,
                      int K, int64_t lda, int64_t ldw, int64_t ldc, int epilogue) {
  typedef Skinny<GLU, FT, MT, TL, NW, DEPTH> S;
  constexpr int FL = S::FL, PITCH = S::PITCH, STAGES = S::STAGES, THREADS = 32 * NW, CHUNKS = DEPTH / 4;
  ls_dependency_trigger();
  extern __shared__ __align__(16) float sk_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tl = lane % TL, fl = warp * FL * FT + lane / TL;       // feature j of this thread: fl + FL * j
  const int n0 = blockIdx.x * S::FEATURES;
  const int stages_total = (K + DEPTH - 1) / DEPTH;

  // pieces of 16 bytes this thread fetches per stage: W rows, then token rows.  Rows past N or
  // M and pieces past K are not fetched: what lies there is never stored (rows) or never
  // multiplied (the loops below stop at K)
  auto load_w = [&](int st) {
    float* ws = sk_smem + (st % STAGES) * S::STAGE;
    const int k0 = st * DEPTH;
#pragma unroll 4
    for (int i = tid; i < S::W_ROWS * CHUNKS; i += THREADS) {
      const int r = i / CHUNKS, ch = i - r * CHUNKS;
      const int f = r % S::FEATURES;
      if (n0 + f < N && k0 + ch * 4 < K)                           // up rows follow the gate rows at N
        cp_async_16(ws + r * PITCH + ch * 4, W + (int64_t)(n0 + f + (r >= S::FEATURES ? N : 0)) * ldw + k0 + ch * 4);
    }
  };
  auto load_x = [&](int st) {
    float* xs = sk_smem + (st % STAGES) * S::STAGE + S::W_ROWS * PITCH;
    const int k0 = st * DEPTH;
    for (int i = tid; i < S::X_ROWS * CHUNKS; i += THREADS) {
      const int r = i / CHUNKS, ch = i - r * CHUNKS;
      if (r < M && k0 + ch * 4 < K) cp_async_16(xs + r * PITCH + ch * 4, A + (int64_t)r * lda + k0 + ch * 4);
    }
  };

  const int ahead = stages_total < STAGES - 1 ? stages_total : STAGES - 1;
  for (int st = 0; st < ahead; ++st) load_w(st);          // weights do not depend on the kernel before
  ls_dependency_wait();
  for (int st = 0; st < STAGES - 1; ++st) {               // one group per stage, empty ones included
    if (st < ahead) load_x(st);
    cp_async_commit();
  }

  float acc[FT][MT], acu[GLU ? FT : 1][MT];
#pragma unroll
  for (int j = 0; j < FT; ++j)
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      acc[j][i] = 0.f;
      if (GLU) acu[GLU ? j : 0][i] = 0.f;
    }

  for (int st = 0; st < stages_total; ++st) {
    cp_async_wait<STAGES - 2>();                          // stage st has landed (for this thread)
    if (NW > 1) __syncthreads();                          // ... for every thread; and stage st - 1 is read
    else __syncwarp();
    if (st + STAGES - 1 < stages_total) {
      load_w(st + STAGES - 1);
      load_x(st + STAGES - 1);
    }
    cp_async_commit();
    const float* wr = sk_smem + (st % STAGES) * S::STAGE + fl * PITCH;
    const float* xr = sk_smem + (st % STAGES) * S::STAGE + (S::W_ROWS + tl) * PITCH;
    // four steps of k
    auto four = [&](int c) {
      float4 w[FT], u[GLU ? FT : 1], x[MT];
#pragma unroll
      for (int j = 0; j < FT; ++j) {
        w[j] = *reinterpret_cast<const float4*>(wr + FL * j * PITCH + 4 * c);
        if (GLU) u[GLU ? j : 0] = *reinterpret_cast<const float4*>(wr + (S::FEATURES + FL * j) * PITCH + 4 * c);
      }
#pragma unroll
      for (int i = 0; i < MT; ++i) x[i] = *reinterpret_cast<const float4*>(xr + TL * i * PITCH + 4 * c);
#pragma unroll
      for (int j = 0; j < FT; ++j)
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          acc[j][i] = fmaf(x[i].x, w[j].x, acc[j][i]);
          acc[j][i] = fmaf(x[i].y, w[j].y, acc[j][i]);
          acc[j][i] = fmaf(x[i].z, w[j].z, acc[j][i]);
          acc[j][i] = fmaf(x[i].w, w[j].w, acc[j][i]);
          if (GLU) {
            const float4 uj = u[GLU ? j : 0];
            float& a = acu[GLU ? j : 0][i];
            a = fmaf(x[i].x, uj.x, a);
            a = fmaf(x[i].y, uj.y, a);
            a = fmaf(x[i].z, uj.z, a);
            a = fmaf(x[i].w, uj.w, a);
          }
        }
    };
    const int left = (K - st * DEPTH) / 4;
    if (left >= CHUNKS) {
#pragma unroll 8
      for (int c = 0; c < CHUNKS; ++c) four(c);
    } else {
      for (int c = 0; c < left; ++c) four(c);
    }
  }
  cp_async_wait<0>();

#pragma unroll
  for (int j = 0; j < FT; ++j) {
    const int n = n0 + fl + FL * j;
    if (n >= N) continue;
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      const int m = tl + TL * i;
      if (m >= M) continue;
      float* c = C + (int64_t)m * ldc + n;
      const float g = acc[j][i];
      if (GLU) *c = g / (1.0f + expf(-g)) * acu[GLU ? j : 0][i];
      else if (epilogue == 1) *c = *c + g;
      else if (epilogue == 4) *c = ls_gelu_tanh(g);
      else if (epilogue == 5) *c = ls_relu_squared(g);
      else *c = g;
    }
  }
}

template <bool GLU, int FT, int MT, int TL, int NW, int DEPTH>
int launch_skinny_as(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw,
                     int64_t ldc, int epilogue, cudaStream_t stream) {
  typedef Skinny<GLU, FT, MT, TL, NW, DEPTH> S;
  constexpr size_t smem = (size_t)S::STAGES * S::STAGE * sizeof(float);
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_nt_skinny_kernel<GLU, FT, MT, TL, NW, DEPTH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
      return LS_E_SMEM;
    configured = true;
  }
  LS_COUNT(LS_K_GEMM_SIMT_FEW);
  ls_launch(gemm_nt_skinny_kernel<GLU, FT, MT, TL, NW, DEPTH>, dim3((N + S::FEATURES - 1) / S::FEATURES), 32 * NW, smem, stream,
            A, W, C, M, N, K, lda, ldw, ldc, epilogue);
  return ls_launch_status();
}

// Which thread makes an element changes no bit.  Narrow (a feature a thread, 8 features a block): a weight of
// 1,024 rows then lies on 128 SMs (16 a block: K = 3,072, 3 tokens, 22 us against 15).  Middle: two features a
// thread, to 8 tokens.  5 to 8 tokens in blocks of 16 features take 100 KB of stages each, two an SM, and above 32 features an
// SM would start another round over the device, so there blocks hold 32 (8 tokens of 4,736 / 4,800 / 6,144 / 9,472 features and K = 1,024:
// in blocks of 16 11.3 / 19.2 / 19.8 / 21.8 us, of 32 13.3 / 14.0 / 14.6 / 15.5).  17 to 32 tokens on four lanes, eight a thread, a feature each (32
// tokens of 2,560 / 6,144 / 8,192 features 26.1 / 51.1 / 51.3 us; with two features a thread 27.0 / 53.3 / 54.2).  Wide, more than eight blocks of 16 features an SM: two features a thread and the tokens on as
// few lanes as their number allows, since what is read from shared memory bounds it (8 tokens of a head: 185 us, a
// token a lane 265).
template <bool GLU>
int launch_skinny(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc,
                  int epilogue, cudaStream_t stream) {
#define LS_SKINNY(FT, MT, TL, NW, DEPTH) \
  return launch_skinny_as<GLU, FT, MT, TL, NW, DEPTH>(A, W, C, M, N, K, lda, ldw, ldc, epilogue, stream)
  if (N <= 2048) {
    if (M <= 4) LS_SKINNY(1, 1, 4, 1, 256);
    if (M <= 8) LS_SKINNY(1, 1, 8, 2, 256);
    if (M <= 16) LS_SKINNY(1, 2, 8, 2, 128);
    LS_SKINNY(1, 4, 8, 2, 64);
  }
  if (GLU || N <= 16 * 8 * ls_sm_count()) {
    if (M <= 4) LS_SKINNY(2, 1, 4, 1, 256);
    if (M <= 8 && !GLU && N > 32 * ls_sm_count()) LS_SKINNY(2, 2, 4, 2, 128);
    if (M <= 8) LS_SKINNY(2, 2, 4, 1, 256);
    if (M <= 16) LS_SKINNY(1, 2, 8, 4, 128);
    if (GLU) LS_SKINNY(1, 4, 8, 4, 128);
    LS_SKINNY(1, 8, 4, 2, 64);
  }
  if constexpr (!GLU) {
    if (M <= 4) LS_SKINNY(2, 4, 1, 2, 32);
    if (M <= 8) LS_SKINNY(2, 8, 1, 2, 32);
    if (M <= 16) LS_SKINNY(2, 8, 2, 2, 64);
    LS_SKINNY(2, 8, 4, 2, 64);
  }
  return LS_E_SIZE;
#undef LS_SKINNY
}

// float32 operands of up to 32 tokens whose rows can be fetched 16 bytes at a time
bool skinny_applies(const void* A, const void* W, int a_dtype, int c_dtype, int M, int K, int64_t lda, int64_t ldw) {
  return a_dtype == LS_F32 && c_dtype == LS_F32 && M <= SK_MAX_M && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
         ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
}

// ---------------------------------------------------------------------------
// Many tokens, float32: the prompt's products on the true 32-bit path.  A block owns TM tokens x WR
// rows of W (silu-mul: the gate rows and the up rows of WR / 2 features), a thread 8 x WR / 16 of
// them as 4 x 4 corners.  FMAs go out two lanes an instruction (PAIRS: two columns, one token) or one.  The next
// k-block is on its way from memory to registers while this one is multiplied.  Every element is
// still one accumulator and one ascending chain fmaf(a, w, acc), so the bits are those of the two
// kernels above.  What bounds it: FMAs and, beside them, what threads read from shared memory (an SM
// delivers a 16-byte piece to 32 threads in 4 cycles, in which it does 16 of a warp's FMAs), and with
// few tiles an SM the trip to memory of every k-block.  1,800 tokens, weights 4,096 and 2 x 3,072 by
// 1,024: 381 and 502 us (with single FMAs 435 and 571).
// ---------------------------------------------------------------------------
constexpr int LK = 16;

template <int EPI, int TM, int WR, bool PAIRS>
__global__ void __launch_bounds__(2 * TM, 256 / TM)
gemm_nt_large_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N,
                     int K, int64_t lda, int64_t ldw, int64_t ldc) {
  static_assert(WR == 128 || (WR == 64 && EPI != 2), "tile widths");
  constexpr int LR = TM / 2;                           // rows that are fetched side by side
  constexpr int FN = EPI == 2 ? WR / 2 : WR;           // features of the tile
  constexpr int HALVES = WR / 64;                      // 64-row halves of W a thread multiplies
  constexpr int WF = WR / LR;                          // pieces of W a thread fetches a k-block
  constexpr int WC = 4 * HALVES;                       // columns of a thread
  ls_dependency_sync();
  __shared__ __align__(16) float As[2][LK][TM + 4];
  __shared__ __align__(16) float Ws[2][LK][WR + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * FN;
  // staging: a thread fetches 4 consecutive k of rows lr + LR h of both operands
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  // row of W behind column c of the tile: silu-mul tiles hold gate rows, then the up rows
  auto w_row = [&](int c) -> int64_t {
    if (EPI == 2) return c < FN ? (n0 + c < N ? n0 + c : -1) : (n0 + c - FN < N ? (int64_t)N + n0 + c - FN : -1);
    return n0 + c < N ? n0 + c : -1;
  };
  float4 ra[2], rw[WF];
  auto fetch = [&](int k0) {
    const bool k_ok = k0 + lk < K;                      // K is a multiple of 4: a piece is whole or absent
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int m = m0 + lr + LR * half;
      ra[half] = (m < M && k_ok) ? *reinterpret_cast<const float4*>(A + (int64_t)m * lda + k0 + lk)
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int half = 0; half < WF; ++half) {
      const int64_t wr = w_row(lr + LR * half);
      rw[half] = (wr >= 0 && k_ok) ? *reinterpret_cast<const float4*>(W + wr * ldw + k0 + lk)
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int r = lr + LR * half;
      As[buf][lk + 0][r] = ra[half].x; As[buf][lk + 1][r] = ra[half].y;
      As[buf][lk + 2][r] = ra[half].z; As[buf][lk + 3][r] = ra[half].w;
    }
#pragma unroll
    for (int half = 0; half < WF; ++half) {
      const int r = lr + LR * half;
      Ws[buf][lk + 0][r] = rw[half].x; Ws[buf][lk + 1][r] = rw[half].y;
      Ws[buf][lk + 2][r] = rw[half].z; Ws[buf][lk + 3][r] = rw[half].w;
    }
  };

  float2 pair[8][WC / 2];                               // columns 2 j and 2 j + 1 of the thread's tile
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < WC / 2; ++j) pair[i][j] = make_float2(0.f, 0.f);

  fetch(0);
  stage(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += LK) {
    const bool more = k0 + LK < K;
    if (more) fetch(k0 + LK);
#pragma unroll
    for (int k = 0; k < LK; ++k) {
      const float4 a_lo = *reinterpret_cast<const float4*>(&As[buf][k][ty * 4]);
      const float4 a_hi = *reinterpret_cast<const float4*>(&As[buf][k][LR + ty * 4]);
      const float a[8] = {a_lo.x, a_lo.y, a_lo.z, a_lo.w, a_hi.x, a_hi.y, a_hi.z, a_hi.w};
      float2 w[WC / 2];
#pragma unroll
      for (int half = 0; half < HALVES; ++half) {
        const float4 w4 = *reinterpret_cast<const float4*>(&Ws[buf][k][64 * half + tx * 4]);
        w[2 * half + 0] = make_float2(w4.x, w4.y);
        w[2 * half + 1] = make_float2(w4.z, w4.w);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < WC / 2; ++j) {
          if constexpr (PAIRS) {
            ls_fma_pair(pair[i][j], a[i], w[j]);
          } else {
            pair[i][j].x = fmaf(a[i], w[j].x, pair[i][j].x);
            pair[i][j].y = fmaf(a[i], w[j].y, pair[i][j].y);
          }
        }
    }
    if (more) {
      stage(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }

  float acc[8][WC];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < WC; ++j) acc[i][j] = j & 1 ? pair[i][j / 2].y : pair[i][j / 2].x;
  // rows ty * 4 + i and LR + ty * 4 + i; columns tx * 4 + j and (128 rows of W) 64 + tx * 4 + j
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + (i < 4 ? ty * 4 + i : LR + ty * 4 + i - 4);
    if (m >= M) continue;
    float* crow = C + (int64_t)m * ldc;
    if (EPI == 2) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + tx * 4 + j;
        const float g = acc[i][j];
        if (n < N) crow[n] = g / (1.0f + expf(-g)) * acc[i][WC - 4 + j];
      }
    } else {
#pragma unroll
      for (int j = 0; j < WC; ++j) {
        const int n = n0 + (j < 4 ? tx * 4 + j : 64 + tx * 4 + j - 4);
        if (n < N) crow[n] = EPI == 1 ? crow[n] + acc[i][j] : EPI == 4 ? ls_gelu_tanh(acc[i][j])
                         : EPI == 5 ? ls_relu_squared(acc[i][j]) : acc[i][j];
      }
    }
  }
}

template <int EPI, int TM, int WR, bool PAIRS = true>
int launch_large_as(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw,
                    int64_t ldc, cudaStream_t stream) {
  constexpr int FN = EPI == 2 ? WR / 2 : WR;
  // (a grid has 65,535 rows of blocks at most: 4,194,240 tokens in tiles of 64; the tokens after them are a launch of their own)
  constexpr int MOST = 65535 * TM;
  for (; M > 0; M -= MOST, A += (int64_t)MOST * lda, C += (int64_t)MOST * ldc) {
    const int rows = M < MOST ? M : MOST;
    LS_COUNT(LS_K_GEMM_SIMT_MANY);
    ls_launch(gemm_nt_large_kernel<EPI, TM, WR, PAIRS>, dim3((N + FN - 1) / FN, (rows + TM - 1) / TM), 2 * TM, 0, stream, A, W, C, rows, N,
              K, lda, ldw, ldc);
  }
  return ls_launch_status();
}

template <int EPI>
int launch_large(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc,
                 cudaStream_t stream) {
  // The tile's size changes no sum.  Tiles of 64 x 128 (four blocks an SM) where there are three or more an SM:
  // 1,800 tokens of 4,096 features 334 us (64 x 64: 373, 128 x 64: 385).  With fewer tiles the trip to memory of
  // a k-block bounds a block, and more and smaller tiles are faster, 64 x 64 (600 tokens of 4,096 features 167 us,
  // 64 x 128: 195), up to two of them an SM; with more, tiles of 128 x 64 where they are at most two an SM (1,500 / 1,800
  // tokens of 1,024 features, K = 1,024: 114 / 114 us, 64 x 64: 118 / 122; 400 tokens of 2,560 features, 280 tiles of 64 x 64, K = 2,560:
  // 278 us, 64 x 64: 238).  These do their FMAs one by one from K = 4,096 on (800 tokens of 2,560 features, K = 9,728: 1,100
  // us, in pairs 1,195; 512 of 4,096, K = 4,096: 478 and 493) and in pairs below (2,048 of 1,024, K = 3,072: 349 and 335).
  const long long sms = ls_sm_count(), rows64 = (M + 63LL) / 64, rows128 = (M + 127LL) / 128;
  if (rows128 > 65535) return LS_E_SIZE;
  if constexpr (EPI != 2) {
    const long long columns = (N + 63) / 64;
    if (rows64 * ((N + 127) / 128) < 3 * sms) {
      if (rows64 * columns > 2 * sms && rows128 * columns <= 2 * sms) {
        if (K >= 4096) return launch_large_as<EPI, 128, 64, false>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        return launch_large_as<EPI, 128, 64>(A, W, C, M, N, K, lda, ldw, ldc, stream);
      }
      return launch_large_as<EPI, 64, 64>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    }
  }
  return launch_large_as<EPI, 64, 128>(A, W, C, M, N, K, lda, ldw, ldc, stream);
}

template <typename TA, typename TW, typename TC>
int launch(const void* A, const void* W, void* C, int M, int N, int K, int64_t lda, int64_t ldw,
           int64_t ldc, int epilogue, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return LS_E_SIZE;
  switch (epilogue) {
    case 0:
      LS_COUNT(LS_K_GEMM_SIMT), ls_launch(gemm_nt_kernel<TA, TW, TC, 0>, grid, 256, 0, stream, (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc);
      break;
    case 1:
      LS_COUNT(LS_K_GEMM_SIMT), ls_launch(gemm_nt_kernel<TA, TW, TC, 1>, grid, 256, 0, stream, (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc);
      break;
    case 2:
      LS_COUNT(LS_K_GEMM_SIMT), ls_launch(gemm_nt_kernel<TA, TW, TC, 2>, grid, 256, 0, stream, (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc);
      break;
    case 4:
      LS_COUNT(LS_K_GEMM_SIMT), ls_launch(gemm_nt_kernel<TA, TW, TC, 4>, grid, 256, 0, stream, (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc);
      break;
    case 5:
      LS_COUNT(LS_K_GEMM_SIMT), ls_launch(gemm_nt_kernel<TA, TW, TC, 5>, grid, 256, 0, stream, (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc);
      break;
    default:
      return LS_E_SIZE;
  }
  return ls_launch_status();
}

}  // namespace

// a_dtype is also the type of W; c_dtype is the type of C (float32 for the
// residual epilogue and for logits).
LS_API int ls_gemm_nt_simt(const void* A, const void* W, void* C, int a_dtype, int c_dtype, int M,
                           int N, int K, int64_t lda, int64_t ldw, int64_t ldc, int epilogue,
                           cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return LS_E_SIZE;
  if (epilogue == 1 && c_dtype != LS_F32) return LS_E_DTYPE;
  typedef __nv_bfloat16 bf16;
  if (skinny_applies(A, W, a_dtype, c_dtype, M, K, lda, ldw)) {
    const float* a = (const float*)A;
    const float* w = (const float*)W;
    if (epilogue == 2) return launch_skinny<true>(a, w, (float*)C, M, N, K, lda, ldw, ldc, epilogue, stream);
    if (epilogue == 0 || epilogue == 1 || epilogue == 4 || epilogue == 5)
      return launch_skinny<false>(a, w, (float*)C, M, N, K, lda, ldw, ldc, epilogue, stream);
    return LS_E_SIZE;
  }
  // float32 rows that can be fetched 16 bytes at a time, more than a few of them
  if (a_dtype == LS_F32 && c_dtype == LS_F32 && M > SK_MAX_M && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
      ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0) {
    const float* a = (const float*)A;
    const float* w = (const float*)W;
    if (epilogue == 0) return launch_large<0>(a, w, (float*)C, M, N, K, lda, ldw, ldc, stream);
    if (epilogue == 1) return launch_large<1>(a, w, (float*)C, M, N, K, lda, ldw, ldc, stream);
    if (epilogue == 2) return launch_large<2>(a, w, (float*)C, M, N, K, lda, ldw, ldc, stream);
    if (epilogue == 4) return launch_large<4>(a, w, (float*)C, M, N, K, lda, ldw, ldc, stream);
    if (epilogue == 5) return launch_large<5>(a, w, (float*)C, M, N, K, lda, ldw, ldc, stream);
    return LS_E_SIZE;
  }
  if (a_dtype == LS_F32 && c_dtype == LS_F32)
    return launch<float, float, float>(A, W, C, M, N, K, lda, ldw, ldc, epilogue, stream);
  if (a_dtype == LS_BF16 && c_dtype == LS_BF16)
    return launch<bf16, bf16, bf16>(A, W, C, M, N, K, lda, ldw, ldc, epilogue, stream);
  if (a_dtype == LS_BF16 && c_dtype == LS_F32)
    return launch<bf16, bf16, float>(A, W, C, M, N, K, lda, ldw, ldc, epilogue, stream);
  return LS_E_DTYPE;
}

LS_API const char* ls_constants_gemm_simt() {
  static char buf[256];
  static const LsConstant c[] = {{"gemm_simt.tile_m", BM}, {"gemm_simt.tile_n", BN}, {"gemm_simt.tile_k", BK},
                                 {"gemm_simt.few_tokens", SK_MAX_M},
                                 {"gemm_simt.many_tokens_depth", LK}};
  return ls_format_constants(buf, sizeof buf, c, (int)(sizeof c / sizeof c[0]));
}
