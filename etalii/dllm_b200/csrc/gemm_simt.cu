// The true 32-bit matrix product: float32 operands, one fused multiply-add chain per output over k ascending, on
// the CUDA cores. No tensor cores, no reduced-precision mode, no split of the reduction, so an output's bits depend
// only on its own row of A and row of W: not on M, on the tile it falls in, or on what else is in the batch.
#include "gemm_common.cuh"

namespace {
constexpr int BM = 64, BN = 64, BK = 16, THREADS = 256;

template <int EPI>
__global__ void __launch_bounds__(THREADS) gemm_f32_kernel(void* __restrict__ c, const float* __restrict__ a,
                                                           const float* __restrict__ w, int M, int N, int K) {
  __shared__ float as[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  int tid = threadIdx.x;
  int tx = tid & 15, ty = tid >> 4;
  int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  int lrow = tid >> 2, lk = (tid & 3) * 4;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    float4 va = make_float4(0.f, 0.f, 0.f, 0.f), vw = va;
    if (m0 + lrow < M && k0 + lk < K) va = *(const float4*)(a + (size_t)(m0 + lrow) * K + k0 + lk);
    if (n0 + lrow < N && k0 + lk < K) vw = *(const float4*)(w + (size_t)(n0 + lrow) * K + k0 + lk);
    as[lk + 0][lrow] = va.x; as[lk + 1][lrow] = va.y; as[lk + 2][lrow] = va.z; as[lk + 3][lrow] = va.w;
    ws[lk + 0][lrow] = vw.x; ws[lk + 1][lrow] = vw.y; ws[lk + 2][lrow] = vw.z; ws[lk + 3][lrow] = vw.w;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float4 ra = *(const float4*)&as[k][ty * 4];
      float4 rw = *(const float4*)&ws[k][tx * 4];
      float av[4] = {ra.x, ra.y, ra.z, ra.w}, wv[4] = {rw.x, rw.y, rw.z, rw.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int m = m0 + ty * 4 + i, n = n0 + tx * 4;
    epilogue_pair<EPI, float>(c, m, n, M, N, acc[i][0], acc[i][1]);
    epilogue_pair<EPI, float>(c, m, n + 2, M, N, acc[i][2], acc[i][3]);
  }
}

// ---- the same product for many rows: 128 x 128 tiles, 8 x 8 outputs a thread ---------------------------------------
// Two stages of shared memory; the next k tile travels from global memory into registers while this one is
// multiplied. A thread's 64 outputs are 2 x 2 groups of 4 x 4, so its shared-memory reads are four 16-byte loads per
// k. Every output is still one chain of fused multiply-adds over k ascending from zero: the same bits as above.
constexpr int LM = 128, LN = 128, LK = 16, LTHREADS = 256;

template <int EPI>
__global__ void __launch_bounds__(LTHREADS) gemm_f32_large_kernel(void* __restrict__ c, const float* __restrict__ a,
                                                                  const float* __restrict__ w, int M, int N, int K) {
  __shared__ __align__(16) float as[2][LK][LM + 4];
  __shared__ __align__(16) float ws[2][LK][LN + 4];
  int tid = threadIdx.x;
  int tx = tid & 15, ty = tid >> 4;             // 16 x 16 threads; outputs rows ty*4 + {0..3, 64..67}, cols likewise
  int m0 = blockIdx.y * LM, n0 = blockIdx.x * LN;
  int lrow = tid >> 2, lk = (tid & 3) * 4;      // a thread fetches rows lrow and lrow + 64, k lk .. lk + 3
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  float4 va[2], vw[2];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int r = lrow + 64 * h;
      va[h] = vw[h] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (m0 + r < M && k0 + lk < K) va[h] = *(const float4*)(a + (size_t)(m0 + r) * K + k0 + lk);
      if (n0 + r < N && k0 + lk < K) vw[h] = *(const float4*)(w + (size_t)(n0 + r) * K + k0 + lk);
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int r = lrow + 64 * h;
      as[buf][lk + 0][r] = va[h].x; as[buf][lk + 1][r] = va[h].y; as[buf][lk + 2][r] = va[h].z; as[buf][lk + 3][r] = va[h].w;
      ws[buf][lk + 0][r] = vw[h].x; ws[buf][lk + 1][r] = vw[h].y; ws[buf][lk + 2][r] = vw[h].z; ws[buf][lk + 3][r] = vw[h].w;
    }
  };
  fetch(0);
  stash(0);
  __syncthreads();
  int tiles = (K + LK - 1) / LK;
  for (int t = 0; t < tiles; ++t) {
    int buf = t & 1;
    if (t + 1 < tiles) fetch((t + 1) * LK);
#pragma unroll
    for (int k = 0; k < LK; ++k) {
      float4 a0 = *(const float4*)&as[buf][k][ty * 4], a1 = *(const float4*)&as[buf][k][64 + ty * 4];
      float4 w0 = *(const float4*)&ws[buf][k][tx * 4], w1 = *(const float4*)&ws[buf][k][64 + tx * 4];
      float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    if (t + 1 < tiles) {
      stash(buf ^ 1);  // (the other stage was last read before the barrier that ended the step before)
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int m = m0 + (i >> 2) * 64 + ty * 4 + (i & 3);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      int n = n0 + (j >> 2) * 64 + tx * 4 + (j & 3);
      epilogue_pair<EPI, float>(c, m, n, M, N, acc[i][j], acc[i][j + 1]);
    }
  }
}

// ---- and for a few rows (decode steps): the reduction streamed through a ring of stages -----------------------------
// One chain of fused multiply-adds per output over k ascending from zero, as above: a token's bits are the ones it gets
// in a long prompt. So a product cannot be faster than its K dependent multiply-adds (four cycles each: 3.1 us for
// K = 1536), and the split is made to come close to that: a block takes COLS columns, few enough that the columns
// spread over the whole device, a thread PER rows of one column, and W and A arrive by cp.async STAGES - 1 stages of
// DEPTH values ahead of the chain. W's first stages are asked for before the kernel in front has finished.
// Eight rows, 576 columns: K = 576 12.0 -> 3.3 us, K = 1536 27.5 -> 6.1 us (before: 32 columns a block, three stages of
// 32 values, which was 18 blocks for the device and a round trip to L2 every other stage); 49152 x 576 52 -> 28.5 us.
constexpr int SM_ROWS = 16;

__device__ __forceinline__ void cp_async_f4(float* smem, const float* gmem, bool ok) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int bytes = ok ? 16 : 0;  // (a copy of no bytes fills the 16 bytes with zeros)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}

template <int EPI, int COLS, int ROWS, int PER, int DEPTH, int STAGES>
__global__ void __launch_bounds__(COLS * ROWS / PER) gemm_f32_small_kernel(void* __restrict__ c, const float* __restrict__ a,
                                                                           const float* __restrict__ w, int M, int N,
                                                                           int K) {
  constexpr int T = COLS * ROWS / PER, LD = DEPTH + 4, PIECES = DEPTH / 4, STAGE = (COLS + ROWS) * LD;
  static_assert(T % 32 == 0 && (COLS * PIECES) % T == 0 && (ROWS * PIECES) % T == 0 && COLS % 2 == 0, "whole warps and copies");
  extern __shared__ __align__(16) float ring[];  // [STAGES][COLS of W, then ROWS of A][LD]
  int tid = threadIdx.x, col = tid % COLS, row0 = tid / COLS;  // rows row0 + i * (ROWS / PER)
  int n0 = blockIdx.x * COLS;
  int tiles = (K + DEPTH - 1) / DEPTH;
  pdl_launch_dependents();
  auto ask_w = [&](int t) {
    float* stage = ring + (t % STAGES) * STAGE;
#pragma unroll
    for (int i = 0; i < COLS * PIECES / T; ++i) {
      int at = tid + i * T, r = at / PIECES, k = (at % PIECES) * 4;
      bool ok = n0 + r < N && t * DEPTH + k < K;
      cp_async_f4(stage + r * LD + k, ok ? w + (size_t)(n0 + r) * K + t * DEPTH + k : w, ok);
    }
  };
  auto ask_a = [&](int t) {
    float* stage = ring + (t % STAGES) * STAGE + COLS * LD;
#pragma unroll
    for (int i = 0; i < ROWS * PIECES / T; ++i) {
      int at = tid + i * T, r = at / PIECES, k = (at % PIECES) * 4;
      bool ok = r < M && t * DEPTH + k < K;
      cp_async_f4(stage + r * LD + k, ok ? a + (size_t)r * K + t * DEPTH + k : a, ok);
    }
  };
  auto close = [] { asm volatile("cp.async.commit_group;\n" ::); };
  for (int t = 0; t < min(tiles, STAGES - 1); ++t) ask_w(t);
  pdl_wait();
  for (int t = 0; t < STAGES - 1; ++t) {
    if (t < tiles) ask_a(t);
    close();
  }
  float acc[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) acc[i] = 0.f;
  for (int t = 0; t < tiles; ++t) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // (this stage has arrived for everybody, and everybody is done with the one before it)
    if (t + STAGES - 1 < tiles) {
      ask_w(t + STAGES - 1);
      ask_a(t + STAGES - 1);
    }
    close();
    const float* stage = ring + (t % STAGES) * STAGE;
    const float* mine = stage + col * LD;
    const float* rows = stage + (COLS + row0) * LD;
    // (the values of the next GROUP pieces are on their way from shared memory while these are multiplied; the chains of
    // a thread go side by side, since a warp issues in order)
    constexpr int GROUP = PER == 1 ? 4 : 2;
    float4 wv[2][GROUP], av[2][GROUP][PER];
    auto load = [&](int slot, int k) {
#pragma unroll
      for (int g = 0; g < GROUP; ++g) {
        wv[slot][g] = *(const float4*)(mine + k + 4 * g);
#pragma unroll
        for (int i = 0; i < PER; ++i) av[slot][g][i] = *(const float4*)(rows + i * (ROWS / PER) * LD + k + 4 * g);
      }
    };
    load(0, 0);
#pragma unroll
    for (int k = 0; k < DEPTH; k += 4 * GROUP) {
      int slot = (k / (4 * GROUP)) & 1;
      if (k + 4 * GROUP < DEPTH) load(slot ^ 1, k + 4 * GROUP);
#pragma unroll
      for (int g = 0; g < GROUP; ++g) {
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = fmaf(av[slot][g][i].x, wv[slot][g].x, acc[i]);
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = fmaf(av[slot][g][i].y, wv[slot][g].y, acc[i]);
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = fmaf(av[slot][g][i].z, wv[slot][g].z, acc[i]);
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = fmaf(av[slot][g][i].w, wv[slot][g].w, acc[i]);
      }
    }
  }
  // pairs of columns are stored by the even lane (the SwiGLU epilogue needs gate and up together)
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    float other = __shfl_down_sync(0xffffffffu, acc[i], 1);
    if (!(col & 1)) epilogue_pair<EPI, float>(c, row0 + i * (ROWS / PER), n0 + col, M, N, acc[i], other);
  }
}

template <int EPI, int COLS, int ROWS, int PER, int DEPTH, int STAGES>
int launch_small(void* c, const float* a, const float* w, int M, int N, int K, cudaStream_t stream) {
  auto kernel = gemm_f32_small_kernel<EPI, COLS, ROWS, PER, DEPTH, STAGES>;
  constexpr int smem = STAGES * (COLS + ROWS) * (DEPTH + 4) * (int)sizeof(float);
  static std::atomic<unsigned long long> allowed{0};
  if (!dllm_allow_shared((const void*)kernel, smem, allowed)) return DLLM_LAUNCH_FAILED;
  return dllm_launch_pdl(kernel, dim3((N + COLS - 1) / COLS), dim3(COLS * ROWS / PER), smem, stream, c, a, w, M, N, K);
}

// How the columns are split, by what was fastest with eight rows (all of it bounded by latency, so by how the columns
// spread and how many chains a thread keeps going, not by the bytes):
//   up to 1,184 columns   8 a block: 148 blocks and more (576 x 1536: 6.1 us; four columns 6.5, sixteen 9.0 to 11.5);
//   up to 4,736           16 a block, two rows a thread, ten short stages (3072 x 576: 5.8 us; 8 columns 8.3, 32 6.7);
//   up to 18,944          16 a block, four rows a thread (8192 x 2048: 25 us; two rows 30 to 35, 32 columns 27 to 35);
//   more                  64 a block, eight rows a thread, which reads shared memory least (49152 x 576: 28.5 us, 4.0 TB/s;
//                         16 columns 40, 32 columns 32).
template <int EPI, int ROWS>
int launch_small_by_columns(void* c, const float* a, const float* w, int M, int N, int K, cudaStream_t stream) {
  if (N <= 8 * 148) return launch_small<EPI, 8, ROWS, ROWS / 8, 128, 6>(c, a, w, M, N, K, stream);
  if (N <= 32 * 148) return launch_small<EPI, 16, ROWS, 2, 64, 10>(c, a, w, M, N, K, stream);
  if (N <= 128 * 148) return launch_small<EPI, 16, ROWS, 4, 128, 4>(c, a, w, M, N, K, stream);
  return launch_small<EPI, 64, ROWS, 8, 64, 3>(c, a, w, M, N, K, stream);
}

template <int EPI>
int launch_small_by_rows(void* c, const float* a, const float* w, int M, int N, int K, cudaStream_t stream) {
  return M <= 8 ? launch_small_by_columns<EPI, 8>(c, a, w, M, N, K, stream)
                : launch_small_by_columns<EPI, 16>(c, a, w, M, N, K, stream);
}
}  // namespace

// C = A[M,K] * W[N,K]^T in float32; K a multiple of 4 (16-byte rows); N even for the SwiGLU epilogue (column pairs).
// Up to 16 rows take the kernel that streams the reduction, 17 to 64 the 64 x 64 tiles, more the 128 x 128 tiles;
// the three give an output the same bits.
DLLM_EXPORT int dllm_gemm_f32(void* c, const float* a, const float* w, int M, int N, int K, int epilogue,
                              cudaStream_t stream) {
  if (M <= 0 || N <= 0) return DLLM_OK;
  if (K <= 0 || (K & 3) || ((N & 1) && epilogue == EPI_SWIGLU)) return DLLM_UNSUPPORTED_SIZE;
  if (epilogue < 0 || epilogue > EPI_SWIGLU) return DLLM_BAD_ARGUMENT;
  if (epilogue == EPI_STORE_T) epilogue = EPI_STORE_F32;  // (the activation type is float32 here)
#define DLLM_BY_EPILOGUE(KERNEL, GRID, THREADS_)                                                      \
  switch (epilogue) {                                                                                 \
    case EPI_STORE_F32: KERNEL<EPI_STORE_F32><<<GRID, THREADS_, 0, stream>>>(c, a, w, M, N, K); break; \
    case EPI_RESIDUAL: KERNEL<EPI_RESIDUAL><<<GRID, THREADS_, 0, stream>>>(c, a, w, M, N, K); break;   \
    default: KERNEL<EPI_SWIGLU><<<GRID, THREADS_, 0, stream>>>(c, a, w, M, N, K); break;               \
  }
  if (M <= SM_ROWS) {
    switch (epilogue) {
      case EPI_STORE_F32: return launch_small_by_rows<EPI_STORE_F32>(c, a, w, M, N, K, stream);
      case EPI_RESIDUAL: return launch_small_by_rows<EPI_RESIDUAL>(c, a, w, M, N, K, stream);
      default: return launch_small_by_rows<EPI_SWIGLU>(c, a, w, M, N, K, stream);
    }
  } else if (M <= 64) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    DLLM_BY_EPILOGUE(gemm_f32_kernel, grid, THREADS)
  } else {
    dim3 grid((N + LN - 1) / LN, (M + LM - 1) / LM);
    if (grid.y > 65535) return DLLM_UNSUPPORTED_SIZE;
    DLLM_BY_EPILOGUE(gemm_f32_large_kernel, grid, LTHREADS)
  }
#undef DLLM_BY_EPILOGUE
  return dllm_launch_status();
}
