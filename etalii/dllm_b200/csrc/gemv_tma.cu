// Weight-streaming products for decode on large matrices (at most 16 rows of activations, bfloat16): C = X * W^T
// where reading W once from HBM is the whole cost, so what counts is how many bytes are on their way at any time.
// Here they travel into shared memory, not into registers: a producer warp issues bulk copies (cp.async.bulk, 2 KB
// of one row of W or X per copy, completion counted by an mbarrier) into a ring of stages that holds up to 216 KB
// per multiprocessor (less what resident rows of X take, below), and consumer warps multiply out of shared memory on the tensor cores (mma.sync m16n8k16
// with W as the 16-row operand, ldmatrix from rows padded by 16 bytes so that no two rows share a bank).
// Blocks are persistent: a block walks over its tiles of W and the ring runs on across tiles.
//   a tile is `height` rows (an even number from 16 to 32: the height that leaves the busiest multiprocessor the fewest
//   rows, e.g. 147 tiles of 28 for 4,096 rows, where 128 tiles of 32 left 20 multiprocessors idle). A stage of the ring
//   holds `height` rows, so that low tiles do not mean fewer bytes on their way;
//   ROWS = 32: tiles of 18 rows and more; ROWS = 16: of sixteen (few rows of W, and the q/k/v projection, whose tiles are
//   eight rotary pairs). With stages of 32 rows whatever the height, one row took 32.4 us for 1024 x 28672 instead of 22.1
//   and 20.2 for 2048 x 16384 instead of 14.3.
// Sixteen rows are the work of four consumer warps, which take 16-value steps in turn and add their sums in order: a
// step is a chain of ldmatrix and product, so one warp gets through one about every 35 cycles, and two warps for a tile
// could not keep up with memory. One row, W out of L2, before all of this (two consumers, tiles of 32 or 16) and now: 28672 x
// 4096 40.0 -> 34.1 us, 128256 x 4096 167 -> 144, 4096 x 14336 23.1 -> 19.6, 4096 x 4096 8.8 -> 7.9; eight rows of 28672 x
// 4096 50.1 -> 38.7, of 4096 x 14336 24.3 -> 23.0.
// RESIDENT: the rows of X lie in shared memory for the whole kernel, copied once, and the ring carries nothing but W. (As
// a part of every stage they cost a copy a row and stage: with eight rows a quarter of all copies.) Where they take more
// than 72 KB they stay a part of the stages. The ring is 144 to 213 KB beside them.
// Epilogues as the tile kernels: store (float32 / bfloat16), residual add in float32, SwiGLU on interleaved rows; rotation
// and cache write behind the q/k/v projection; the greedy choice behind the head. K must be a multiple of 64. Every wait on
// an mbarrier is bounded; a role that gives up records a status word.
#include "gemv_common.cuh"
#include "tcgen05.cuh"

namespace {
using namespace tc5;
typedef __nv_bfloat16 bf16;
constexpr int KC = 1024;                   // values of k per stage: 2 KB of every row (a bulk copy costs its
                                           // issuer about as much whatever its size, so copies are long)
constexpr int ROW_BYTES = KC * 2;
constexpr int PITCH = ROW_BYTES + 16;      // rows in shared memory: 16 bytes of padding (ldmatrix without conflicts)
constexpr int K_PARTS = 4;                 // consumer warps that share 16 rows of W
constexpr int RING_BYTES = 216 * 1024;

__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(unsigned* r, unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x2(unsigned* r, unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
using gemv::mma_bf16;

constexpr int RESIDENT_BYTES = 72 * 1024;  // the most that resident rows of X may take
// Stages a row of resident X may span (their arrivals are counted one by one): as many as the longest single row that fits.
constexpr int MAX_CHUNKS = (RESIDENT_BYTES / 2 + KC - 1) / KC;

template <int ROWS, int NT, bool RESIDENT> struct Shape {
  static constexpr int TOKENS = NT * 8;                          // token rows of a stage (those beyond M stay unused)
  static __host__ __device__ constexpr int stage_bytes(int height) { return (height + (RESIDENT ? 0 : TOKENS)) * PITCH; }
  static constexpr int MAX_STAGES = RING_BYTES / ((16 + (RESIDENT ? 0 : TOKENS)) * PITCH);  // (no tile is lower)
  static constexpr int CONSUMERS = ROWS / 16 * K_PARTS, THREADS = 32 * (1 + CONSUMERS);  // (warp 0 copies)
  static constexpr int SCRATCH_FLOATS = CONSUMERS * 16 * (TOKENS + 1);  // a 16 x TOKENS tile per consumer warp
  // (resident rows of X, then the ring in what is left)
  static int x_bytes(int M, int K) { return RESIDENT ? M * (2 * K + 16) : 0; }
  static int stages(int M, int K, int height) { return (RING_BYTES - x_bytes(M, K)) / stage_bytes(height); }
  static size_t smem(int M, int K, int height) {
    return (size_t)x_bytes(M, K) + (size_t)stages(M, K, height) * stage_bytes(height) + SCRATCH_FLOATS * sizeof(float) + 128;
  }
  static constexpr int MAX_SMEM = RING_BYTES + SCRATCH_FLOATS * (int)sizeof(float) + 128;
};

template <int ROWS, int NT, int EPI, bool RESIDENT>
__global__ void __launch_bounds__(Shape<ROWS, NT, RESIDENT>::THREADS, 1) gemv_tma_kernel(void* __restrict__ c, const bf16* __restrict__ x,
                                                              const bf16* __restrict__ w, int M, int N, int K,
                                                              int tiles, int height, int stages, int* __restrict__ status,
                                                              RopeArgs rope) {
  typedef Shape<ROWS, NT, RESIDENT> S;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* x_s = (unsigned char*)(((uintptr_t)smem_raw + 15) & ~(uintptr_t)15);
  const int x_pitch = 2 * K + 16;  // (K is a multiple of 64: the rows begin in different banks)
  unsigned char* ring = x_s + (RESIDENT ? (size_t)M * x_pitch : 0);
  const int stage_bytes = S::stage_bytes(ROWS == 16 ? 16 : height);
  float* scratch = reinterpret_cast<float*>(ring + (size_t)stages * stage_bytes);
  __shared__ uint64_t full_bar[S::MAX_STAGES], empty_bar[S::MAX_STAGES], x_bar[RESIDENT ? MAX_CHUNKS : 1];
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int chunks = K / KC + (K % KC ? 1 : 0);  // stages per tile; the last may be shorter (K is a multiple of 64)
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], S::CONSUMERS); }
    if (RESIDENT)
      for (int ch = 0; ch < chunks; ++ch) mbar_init(&x_bar[RESIDENT ? ch : 0], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (EPI == EPI_QKV_ROPE) gemv::prefetch_cache_pages(rope, M);

  if (warp == 0) {
    // ---- producer: lane r copies row r of the tile's W; lanes also copy the token rows of X. The weights are
    // nobody's output: the first trip round the ring asks for them before the wait on the kernel before, and adds
    // the rows of X (which that kernel may have written) after it.
    auto fill = [&](int s, int tile, int ch, bool weights, bool tokens) {
      int row0 = tile * height, rows_valid = min(height, N - row0), k0 = ch * KC;
      unsigned bytes = (unsigned)min(KC, K - k0) * 2u;
      unsigned char* stage = ring + (size_t)s * stage_bytes;
      if (weights) {
        if (lane == 0) mbar_expect_tx(&full_bar[s], bytes * (unsigned)(rows_valid + (RESIDENT ? 0 : M)));
        __syncwarp();
        for (int r = lane; r < rows_valid; r += 32) {
          int row = row0 + r;
          if (EPI == EPI_QKV_ROPE) {
            int head, dim0;
            bool paired;
            row = gemv::tile_row<EPI>(tile, r, N, rope, head, dim0, paired);
          }
          bulk_copy(stage + r * PITCH, w + (size_t)row * K + k0, bytes, &full_bar[s]);
        }
      }
      if (tokens && !RESIDENT)
        for (int m = lane; m < M; m += 32)
          bulk_copy(stage + (height + m) * PITCH, x + (size_t)m * K + k0, bytes, &full_bar[s]);
    };
    int filled = 0, tile = blockIdx.x, ch = 0;
    for (; filled < stages && tile < tiles; ++filled) {  // the first trip: weights only
      fill(filled, tile, ch, true, false);
      if (++ch == chunks) { ch = 0; tile += gridDim.x; }
    }
    pdl_wait();
    if (RESIDENT) {
      // (a lane a stage for what is expected, then a lane a copy: a row of 36 stages is two turns, not 36)
      auto stage_row = [&](int k) { return (unsigned)min(KC, K - k * KC) * 2u; };
      for (int k = lane; k < chunks; k += 32) mbar_expect_tx(&x_bar[RESIDENT ? k : 0], stage_row(k) * (unsigned)M);
      __syncwarp();
      for (int i = lane; i < chunks * M; i += 32) {
        int k = i / M, m = i % M;
        bulk_copy(x_s + (size_t)m * x_pitch + k * ROW_BYTES, x + (size_t)m * K + k * KC, stage_row(k), &x_bar[RESIDENT ? k : 0]);
      }
    } else {
      int tile2 = blockIdx.x, ch2 = 0;
      for (int s = 0; s < filled; ++s) {  // their rows of X
        fill(s, tile2, ch2, false, true);
        if (++ch2 == chunks) { ch2 = 0; tile2 += gridDim.x; }
      }
    }
    // (laps are counted along: divided by a number of stages that the compiler does not know, they cost 0.1 us a stage)
    int s = 0;
    unsigned lap = 0;
    while (tile < tiles) {
      if (!mbar_wait(&empty_bar[s], lap)) {
        if (lane == 0) *(volatile int*)status = 32;
        break;
      }
      fill(s, tile, ch, true, true);
      if (++ch == chunks) { ch = 0; tile += gridDim.x; }
      if (++s == stages) { s = 0; lap ^= 1; }
    }
  } else {
    // ---- consumers
    pdl_wait();  // C (for the residual) may come from the kernel before
    int cw = warp - 1, half = cw / K_PARTS, part = cw % K_PARTS;  // which 16 rows of the tile, which steps
    int g = lane >> 2, t = lane & 3;
    int row_base = half * 16;
    // ldmatrix addresses inside a stage: W rows (lane & 15), k offset 8 for the upper lanes; X rows (lane & 7),
    // k offset 8 for lanes 8..15 (and the second eight tokens for lanes 16..31 when NT == 2). Rows of W beyond the tile's
    // height are its last row again, rows of X beyond M whatever lies there, or the last row again where X is resident:
    // their results are not stored.
    unsigned a_off = (unsigned)(min(row_base + (lane & 15), height - 1) * PITCH + (lane >> 4) * 16);
    int token = (lane & 7) + (NT == 2 ? (lane >> 4) * 8 : 0);
    unsigned b_off = RESIDENT ? smem_u32(x_s) + (unsigned)(min(token, M - 1) * x_pitch + ((lane >> 3) & 1) * 16)
                              : (unsigned)((height + token) * PITCH + ((lane >> 3) & 1) * 16);
    constexpr int TILE_FLOATS = 16 * (S::TOKENS + 1);
    float* group = scratch + (size_t)half * K_PARTS * TILE_FLOATS;  // the tiles of the warps that share these rows
    float* mine = group + part * TILE_FLOATS;
    int member = part * 32 + lane;  // this thread among the group's
    int s = 0;  // the ring's next stage and lap
    unsigned lap = 0;
    auto meet = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + half), "n"(K_PARTS * 32) : "memory"); };
    bool ok = true;  // (a warp that gave up still meets the others of its group, tile by tile, and stores nothing)
    // (in the q/k/v projection a thread stores the same pair and token of every tile: the token's position and cache page
    // are asked for before the first product, the tile's angle before the tile's)
    static_assert(EPI != EPI_QKV_ROPE || (NT == 1 && ROWS == 16), "one pair and token a thread");
    int pos = 0, page = 0;
    if (EPI == EPI_QKV_ROPE && member < 64 && (member & 7) < M) {
      pos = rope.tok_pos[member & 7];
      if (rope.write_cache)
        page = rope.cache.page_table[(size_t)rope.slots[rope.tok_seq[member & 7]] * rope.cache.max_pages +
                                     pos / rope.cache.page_size];
    }
    // (EPI_ARGMAX: the largest value that this thread has seen over all tiles, and its feature; features ascend, so the
    // first of equal ones stays)
    static_assert(EPI != EPI_ARGMAX || NT == 1, "one pair and token a thread");
    float best_value = -INFINITY;
    int best_feature = 0x7fffffff;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      int head = 0, dim0 = 0;
      bool paired = false;
      float2 turn = make_float2(1.f, 0.f);
      if (EPI == EPI_QKV_ROPE) {
        gemv::tile_row<EPI>(tile, 0, N, rope, head, dim0, paired);
        if (paired && member < 64 && (member & 7) < M)
          turn = rope.table[(size_t)pos * (rope.rotary_dim / 2) + dim0 + (member >> 3)];
      }
      float acc[2][NT][4];  // two sets on alternate steps: a step does not wait for the one before
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[e][n][i] = 0.f;
      for (int ch = 0; ch < chunks && ok; ++ch) {
        if (!mbar_wait(&full_bar[s], lap) || (RESIDENT && !mbar_wait(&x_bar[RESIDENT ? ch : 0], 0))) {
          if (lane == 0) *(volatile int*)status = 33;
          ok = false;
          break;
        }
        unsigned stage = smem_u32(ring + (size_t)s * stage_bytes);
        unsigned x_at = RESIDENT ? b_off + (unsigned)(ch * ROW_BYTES) : stage + b_off;
        int steps = min(KC, K - ch * KC) / (16 * K_PARTS);  // (K is a multiple of 64: as many for every warp)
        auto step = [&](float (*into)[4], int j) {
          unsigned a[4], b[4];
          unsigned at = (unsigned)(j * K_PARTS + part) * 32u;
          ldmatrix_x4(a, stage + a_off + at);
          if (NT == 2) ldmatrix_x4(b, x_at + at);
          else ldmatrix_x2(b, x_at + at);
          mma_bf16(into[0], a, b[0], b[1]);
          if (NT == 2) mma_bf16(into[NT - 1], a, b[2], b[3]);
        };
        int j = 0;
#pragma unroll 4
        for (; j + 1 < steps; j += 2) {
          step(acc[0], j);
          step(acc[1], j + 1);
        }
        if (j < steps) step(acc[0], j);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[s]);  // this warp is done with the stage
        if (++s == stages) { s = 0; lap ^= 1; }
      }
      // the warp's 16 x TOKENS tile to shared memory, then one (pair of rows, token) per thread of the group and turn
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        mine[g * (S::TOKENS + 1) + n * 8 + 2 * t] = acc[0][n][0] + acc[1][n][0];
        mine[g * (S::TOKENS + 1) + n * 8 + 2 * t + 1] = acc[0][n][1] + acc[1][n][1];
        mine[(g + 8) * (S::TOKENS + 1) + n * 8 + 2 * t] = acc[0][n][2] + acc[1][n][2];
        mine[(g + 8) * (S::TOKENS + 1) + n * 8 + 2 * t + 1] = acc[0][n][3] + acc[1][n][3];
      }
      meet();
      int n0 = tile * height + row_base;
      for (int idx = member; idx < 8 * S::TOKENS && ok; idx += K_PARTS * 32) {
        int p = idx / S::TOKENS, m = idx % S::TOKENS;
        // (rows 2 p and 2 p + 1 of the sixteen, or p and p + 8 for rotary pairs)
        int r0 = EPI == EPI_QKV_ROPE ? p : 2 * p, r1 = EPI == EPI_QKV_ROPE ? p + 8 : 2 * p + 1;
        if (m >= M || (EPI != EPI_QKV_ROPE && row_base + r0 >= height)) continue;
        float v0 = 0.f, v1 = 0.f;
#pragma unroll
        for (int k = 0; k < K_PARTS; ++k) {
          v0 += group[k * TILE_FLOATS + r0 * (S::TOKENS + 1) + m];
          v1 += group[k * TILE_FLOATS + r1 * (S::TOKENS + 1) + m];
        }
        if (EPI == EPI_QKV_ROPE) {
          int hd = rope.cache.head_dim, nkv = rope.cache.kv_heads;
          int d0 = dim0 + p, d1 = d0 + (paired ? rope.rotary_dim / 2 : 8);
          if (paired) {
            float a = v0, b = v1;
            v0 = fmaf(a, turn.x, -(b * turn.y));
            v1 = fmaf(a, turn.y, b * turn.x);
          }
          bf16* dst;
          if (head < rope.heads) {
            dst = rope.q_out + ((size_t)m * rope.heads + head) * hd;
          } else {
            if (!rope.write_cache) continue;
            int which = head < rope.heads + nkv ? 0 : 1, kvh = head - rope.heads - which * nkv;
            dst = (bf16*)rope.cache.base + kv_offset(rope.cache, page, which, kvh, pos % rope.cache.page_size);
          }
          dst[d0] = __float2bfloat16_rn(v0);
          dst[d1] = __float2bfloat16_rn(v1);
        } else if (EPI == EPI_ARGMAX) {  // (a value that is not a number is never larger: it is never chosen)
          int n = n0 + 2 * p;
          if (n < N && v0 > best_value) { best_value = v0; best_feature = n; }
          if (n + 1 < N && v1 > best_value) { best_value = v1; best_feature = n + 1; }
        } else {
          epilogue_pair<EPI, bf16>(c, m, n0 + 2 * p, M, N, v0, v1);
        }
      }
      meet();  // the scratch is free for the next tile
    }
    if (EPI == EPI_ARGMAX) {
      // Pairs 0..3 of a token lie in the group's first warp, 4..7 in its second; every group leaves one candidate a token.
      auto better = [&](float value, int feature) {
        if (value > best_value || (value == best_value && feature < best_feature)) {
          best_value = value;
          best_feature = feature;
        }
      };
#pragma unroll
      for (int o = 8; o <= 16; o <<= 1) {
        float value = __shfl_xor_sync(0xffffffffu, best_value, o);
        int feature = __shfl_xor_sync(0xffffffffu, best_feature, o);
        better(value, feature);
      }
      if (part == 1 && lane < 8) {
        group[2 * lane] = best_value;
        group[2 * lane + 1] = __int_as_float(best_feature);
      }
      meet();
      if (part == 0 && lane < M) {
        better(group[2 * lane], __float_as_int(group[2 * lane + 1]));
        float* out = (float*)c + ((size_t)lane * 2 * gridDim.x + 2 * blockIdx.x + half) * 2;
        out[0] = best_value;
        out[1] = __int_as_float(best_feature);
      }
    }
  }
}

int multiprocessors() {
  static int sms = 0;
  if (sms == 0) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0) {
      sms = 0;
    }
  }
  return sms;
}

template <int ROWS, int NT, int EPI, bool RESIDENT>
int launch(void* c, const bf16* x, const bf16* w, int M, int N, int K, int height, int* status, const RopeArgs& rope,
           cudaStream_t stream) {
  typedef Shape<ROWS, NT, RESIDENT> S;
  static std::atomic<unsigned long long> allowed{0};
  int sms = multiprocessors();
  if (sms == 0 || !dllm_allow_shared((const void*)gemv_tma_kernel<ROWS, NT, EPI, RESIDENT>, S::MAX_SMEM, allowed))
    return DLLM_LAUNCH_FAILED;
  int tiles = (N + height - 1) / height;
  int blocks = tiles < sms ? tiles : sms;
  return dllm_launch_pdl(gemv_tma_kernel<ROWS, NT, EPI, RESIDENT>, dim3(blocks), dim3(S::THREADS), S::smem(M, K, height),
                         stream, c, x, w, M, N, K, tiles, height, S::stages(M, K, height), status, rope);
}

// (`resident_activations` of kernels/ops.py is the same rule: who asks it calls the entry points below that want it kept)
bool resident(int M, int K) { return M <= 8 && (long long)M * (2ll * K + 16) <= RESIDENT_BYTES; }

// The height that leaves the busiest multiprocessor the fewest rows, the larger one where several do.
int tile_height(int N, int sms) {
  int height = 32;
  long long fewest = 0;
  for (int h = 32; h >= 16; h -= 2) {
    long long rows = ((long long)((N + h - 1) / h) + sms - 1) / sms * h;
    if (h == 32 || rows < fewest) {
      fewest = rows;
      height = h;
    }
  }
  return height;
}

template <int NT, bool RESIDENT>
int dispatch(void* c, const bf16* x, const bf16* w, int M, int N, int K, int epilogue, int* status, cudaStream_t stream) {
  int sms = multiprocessors();
  if (sms == 0) return DLLM_LAUNCH_FAILED;
  int height = tile_height(N, sms);
  auto go = [&](auto low, auto high) {
    return (height == 16 ? low : high)(c, x, w, M, N, K, height, status, RopeArgs{}, stream);
  };
  switch (epilogue) {
    case EPI_STORE_F32: return go(launch<16, NT, EPI_STORE_F32, RESIDENT>, launch<32, NT, EPI_STORE_F32, RESIDENT>);
    case EPI_STORE_T: return go(launch<16, NT, EPI_STORE_T, RESIDENT>, launch<32, NT, EPI_STORE_T, RESIDENT>);
    case EPI_RESIDUAL: return go(launch<16, NT, EPI_RESIDUAL, RESIDENT>, launch<32, NT, EPI_RESIDUAL, RESIDENT>);
    case EPI_SWIGLU: return go(launch<16, NT, EPI_SWIGLU, RESIDENT>, launch<32, NT, EPI_SWIGLU, RESIDENT>);
    default: return DLLM_BAD_ARGUMENT;
  }
}
}  // namespace

// C = X[M,K] * W[N,K]^T for M <= 16, bfloat16 X and W, K a multiple of 64, N even for SwiGLU; X and W 16-byte
// aligned. `status` is a word the device can write; the kernel sets it non-zero if a bounded wait ran out
// (32: producer, 33: consumer).
DLLM_EXPORT int dllm_gemv_tma(void* c, const void* x, const void* w, int M, int N, int K, int epilogue, int* status,
                              cudaStream_t stream) {
  if (M <= 0 || N <= 0) return DLLM_OK;
  if (M > 16 || K <= 0 || (K & 63) || ((N & 1) && epilogue == EPI_SWIGLU) || ((uintptr_t)x & 15) ||
      ((uintptr_t)w & 15) || status == nullptr)
    return DLLM_UNSUPPORTED_SIZE;
  const bf16* xp = (const bf16*)x;
  const bf16* wp = (const bf16*)w;
  if (resident(M, K)) return dispatch<1, true>(c, xp, wp, M, N, K, epilogue, status, stream);
  if (M <= 8) return dispatch<1, false>(c, xp, wp, M, N, K, epilogue, status, stream);
  return dispatch<2, false>(c, xp, wp, M, N, K, epilogue, status, stream);
}

// The first stage of the greedy head product on the same ring (see EPI_ARGMAX), for up to eight tokens whose rows are
// resident: candidates [M][*count](value, feature), two a block and token, for dllm_argmax_candidates. *count is at most
// ceil(N / 16) for N of 4,736 and more; fewer rows of W are refused.
DLLM_EXPORT int dllm_gemv_tma_argmax(float* candidates, const void* x, const void* w, int M, int N, int K, int* count,
                                     int* status, cudaStream_t stream) {
  int sms = multiprocessors();
  if (sms == 0) return DLLM_LAUNCH_FAILED;
  if (M <= 0 || N < 32 * sms || K <= 0 || (K & 63) || !resident(M, K) || ((uintptr_t)x & 15) || ((uintptr_t)w & 15) ||
      status == nullptr || count == nullptr)
    return DLLM_UNSUPPORTED_SIZE;
  int height = tile_height(N, sms), tiles = (N + height - 1) / height;
  *count = 2 * (tiles < sms ? tiles : sms);
  return launch<32, 1, EPI_ARGMAX, true>(candidates, (const bf16*)x, (const bf16*)w, M, N, K, height, status, RopeArgs{},
                                         stream);
}

// The q/k/v projection of a decode step on the same ring, arguments as `dllm_gemv_qkv_rope` without a norm in front:
// for up to eight tokens whose rows are resident. head_dim and rotary_dim multiples of 16.
DLLM_EXPORT int dllm_gemv_tma_qkv_rope(const void* x, const void* w, int M, int K, void* q_out, void* cache_base,
                                       const int* page_table, int max_pages, int page_size, int heads, int kv_heads,
                                       int head_dim, const float* table, int rotary_dim, const int* tok_seq,
                                       const int* tok_pos, const int* slots, int write_cache, int prefetch_window,
                                       int* status, cudaStream_t stream) {
  if (M <= 0) return DLLM_OK;
  if (K <= 0 || (K & 63) || !resident(M, K) || heads <= 0 || kv_heads <= 0 || head_dim <= 0 || (head_dim & 15) ||
      rotary_dim < 0 || rotary_dim > head_dim || (rotary_dim & 15) || ((uintptr_t)x & 15) || ((uintptr_t)w & 15) ||
      status == nullptr)
    return DLLM_UNSUPPORTED_SIZE;
  RopeArgs rope{(bf16*)q_out, KvLayout{cache_base, page_table, max_pages, page_size, kv_heads, head_dim},
                (const float2*)table, table ? rotary_dim : 0, heads, tok_seq, tok_pos, slots, write_cache,
                prefetch_window};
  int N = (heads + 2 * kv_heads) * head_dim;
  return launch<16, 1, EPI_QKV_ROPE, true>(nullptr, (const bf16*)x, (const bf16*)w, M, N, K, 16, status, rope, stream);
}
