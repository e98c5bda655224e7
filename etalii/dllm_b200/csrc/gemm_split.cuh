// The tile product for hundreds of rows of activations and a long reduction (a short prompt): tiles of 128 x 128 whose
// reduction is shared by the 1, 2, 4 or 8 blocks of a thread-block cluster. Part of gemm_tcgen05.cu.
//
// What bounds such a product is W, read once from HBM, as long as every multiprocessor takes part and the activations are
// not read too often: tiles of 32 columns give enough blocks but move 16 KB of A for 4 KB of W, and a W of 4,096 rows has
// 32 tiles of 128 columns for 148 multiprocessors. So the columns are 128 and the cluster cuts the reduction. Block r of a
// cluster multiplies its stretch of the k tiles into tensor memory (the producer and issuer of gemm_tcgen05_kernel, one
// tile a block), puts the sums into its shared memory, and after a cluster barrier finishes its share of the tile's rows:
// a warp a row, four columns a lane, the blocks' sums added in the order of the stretches through distributed shared memory.
// Two blocks a multiprocessor.
#pragma once

namespace {
struct SplitShape {
  static constexpr int BN = 128, THREADS = 256, WARPS = THREADS / 32, STAGES = 3, BLOCKS_PER_SM = 2;
  static constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
  static constexpr int LD = BN + 4;  // floats per row of the sums
  static constexpr int RING = STAGES * (A_BYTES + B_BYTES), SUMS = BM * LD * 4;
  static constexpr size_t SMEM = (RING > SUMS ? RING : SUMS) + 1024;
};

template <int EPI, int HD>
__global__ void __launch_bounds__(SplitShape::THREADS, SplitShape::BLOCKS_PER_SM) gemm_split_kernel(
    const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, void* __restrict__ c, int M, int N,
    int K, int* __restrict__ status, RopeArgs rope, NormArgs norm) {
  typedef SplitShape S;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* tiles = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* sums = reinterpret_cast<float*>(tiles);  // (when every product has read its stage)
  __shared__ uint64_t full_bar[S::STAGES], empty_bar[S::STAGES], acc_full;
  __shared__ unsigned tmem_base_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = (int)gridDim.x, rank = (int)blockIdx.x, n_tile = (int)blockIdx.y;
  const int m0 = (int)blockIdx.z * BM, n0 = n_tile * S::BN;
  const int k_tiles = (K + BK - 1) / BK, kt_begin = rank * k_tiles / split, kt_end = (rank + 1) * k_tiles / split;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&acc_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(&tmem_base_s, S::BN);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const unsigned tmem_base = tmem_base_s;
  // (only now: a block of the next kernel that came first to this multiprocessor's tensor memory would hold it until this
  // grid has ended)
  pdl_launch_dependents();

  if (warp == 0) {
    if (lane == 0) {
      // W is nobody's output: its first tiles travel while the kernel in front ends
      int early = min(S::STAGES, kt_end - kt_begin);
      for (int i = 0; i < early; ++i) {
        mbar_expect_tx(&full_bar[i], S::A_BYTES + S::B_BYTES);
        tma_load_2d(tiles + i * (S::A_BYTES + S::B_BYTES) + S::A_BYTES, &map_w, &full_bar[i], (kt_begin + i) * BK, n0);
      }
      pdl_wait();
      for (int i = 0; i < early; ++i)
        tma_load_2d(tiles + i * (S::A_BYTES + S::B_BYTES), &map_a, &full_bar[i], (kt_begin + i) * BK, m0);
      for (int i = early, kt = kt_begin + early; kt < kt_end; ++kt, ++i) {
        int s = i % S::STAGES;
        if (!mbar_wait(&empty_bar[s], (i / S::STAGES - 1) & 1)) { *(volatile int*)status = 2; break; }
        mbar_expect_tx(&full_bar[s], S::A_BYTES + S::B_BYTES);
        unsigned char* at = tiles + s * (S::A_BYTES + S::B_BYTES);
        tma_load_2d(at, &map_a, &full_bar[s], kt * BK, m0);
        tma_load_2d(at + S::A_BYTES, &map_w, &full_bar[s], kt * BK, n0);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr unsigned idesc = instr_desc(BM, S::BN);
      for (int i = 0; i < kt_end - kt_begin; ++i) {
        int s = i % S::STAGES;
        if (!mbar_wait(&full_bar[s], (i / S::STAGES) & 1)) { *(volatile int*)status = 3; break; }
        fence_after_sync();
        unsigned a_addr = smem_u32(tiles + s * (S::A_BYTES + S::B_BYTES)), b_addr = a_addr + S::A_BYTES;
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma(tmem_base, smem_desc(a_addr + k * UMMA_K * 2), smem_desc(b_addr + k * UMMA_K * 2), idesc,
               (i > 0 || k > 0) ? 1u : 0u);
        tcgen05_commit(&empty_bar[s]);
      }
      tcgen05_commit(&acc_full);
    }
    __syncwarp();
  }
  pdl_wait();

  // This block's rows: a warp takes every WARPS-th of them. What the epilogue reads besides the sums is asked for first.
  constexpr bool SCALED = EPI != EPI_RESIDUAL;
  const int rows = min(BM, M - m0), height = (rows + split - 1) / split, row0 = rank * height;
  const int row_end = min(rows, row0 + height), per_warp = (height + S::WARPS - 1) / S::WARPS;  // (at most 16 rows a warp)
  float scale_mine = 1.f;  // lane i: the factor of the warp's i-th row
  int pos_mine = 0, page_mine = 0;
  {
    int row = row0 + warp + lane * S::WARPS, m = m0 + row;
    if (lane < per_warp && row < row_end) {
      if (SCALED) scale_mine = row_scale(norm, m, M);
      if (EPI == EPI_QKV_ROPE) {
        pos_mine = rope.tok_pos[m];
        if (rope.write_cache) {
          int slot = rope.slots[rope.tok_seq[m]];
          page_mine = rope.cache.page_table[(size_t)slot * rope.cache.max_pages + pos_mine / rope.cache.page_size];
        }
      }
    }
  }
  if (!mbar_wait(&acc_full, 0) && lane == 0) *(volatile int*)status = 4;
  __syncwarp();
  fence_after_sync();
  if ((warp & 3) * 32 < rows) {
    const int quarter = warp & 3, c0 = (warp >> 2) * (S::BN / 2);  // (a warp reads the tensor-memory lanes of its quarter)
    float* to = sums + (size_t)(quarter * 32 + lane) * S::LD + c0;
    unsigned acc = tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)c0;
#pragma unroll
    for (int cc = 0; cc < S::BN / 2; cc += 16) {
      unsigned v[16];
      tmem_load16(acc + (unsigned)cc, v);
#pragma unroll
      for (int i = 0; i < 16; i += 4)
        *reinterpret_cast<float4*>(to + cc + i) = make_float4(__uint_as_float(v[i]), __uint_as_float(v[i + 1]),
                                                              __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
    }
  }
  fence_before_sync();
  if (split > 1) asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
  else __syncthreads();

  const int n = n0 + lane * 4;  // the lane's columns (N is a multiple of 4)
  const bool inside = n < N;
  for (int at = 0; at < per_warp; ++at) {
    const int row = row0 + warp + at * S::WARPS, m = m0 + row;
    if (row >= row_end) break;  // (rows ascend)
    float4 old = make_float4(0.f, 0.f, 0.f, 0.f);
    if (EPI == EPI_RESIDUAL && inside) old = *reinterpret_cast<const float4*>((const float*)c + (size_t)m * N + n);
    const float* mine = sums + (size_t)row * S::LD + lane * 4;
    float4 v;
    if (split == 1) {
      v = *reinterpret_cast<const float4*>(mine);
    } else {
      unsigned local = smem_u32(mine);
      float4 part[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        if (r >= split) continue;
        unsigned far;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(far) : "r"(local), "r"(r));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(part[r].x), "=f"(part[r].y), "=f"(part[r].z), "=f"(part[r].w) : "r"(far));
      }
      v = part[0];
#pragma unroll
      for (int r = 1; r < 8; ++r) {
        if (r >= split) continue;
        v.x += part[r].x; v.y += part[r].y; v.z += part[r].z; v.w += part[r].w;
      }
    }
    const float scale = SCALED ? __shfl_sync(0xffffffffu, scale_mine, at) : 1.f;
    if (SCALED) { v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale; }
    auto pack = [](float4 f) {
      __nv_bfloat162 lo = __floats2bfloat162_rn(f.x, f.y), hi = __floats2bfloat162_rn(f.z, f.w);
      return make_uint2(*reinterpret_cast<unsigned*>(&lo), *reinterpret_cast<unsigned*>(&hi));
    };
    if (EPI == EPI_RESIDUAL) {
      float squares = 0.f;
      if (inside) {
        old.x += v.x; old.y += v.y; old.z += v.z; old.w += v.w;
        *reinterpret_cast<float4*>((float*)c + (size_t)m * N + n) = old;
        if (norm.copy_out != nullptr) {
          *reinterpret_cast<uint2*>(norm.copy_out + (size_t)m * N + n) = pack(old);
          squares = fmaf(old.x, old.x, fmaf(old.y, old.y, fmaf(old.z, old.z, old.w * old.w)));
        }
      }
      if (norm.ssq_out != nullptr) {
        squares = warp_sum(squares);
        if (lane == 0) norm.ssq_out[(size_t)n_tile * M + m] = squares;
      }
    } else if (EPI == EPI_QKV_ROPE) {
      // a tile is one head of 128 or two of 64; the rotary partner of a lane's columns lies half a head away
      constexpr int HEAD = HD > 0 ? HD : S::BN, HALF = HEAD / 2;
      float4 p;
      p.x = __shfl_xor_sync(0xffffffffu, v.x, HALF / 4);
      p.y = __shfl_xor_sync(0xffffffffu, v.y, HALF / 4);
      p.z = __shfl_xor_sync(0xffffffffu, v.z, HALF / 4);
      p.w = __shfl_xor_sync(0xffffffffu, v.w, HALF / 4);
      const int pos = __shfl_sync(0xffffffffu, pos_mine, at), page = __shfl_sync(0xffffffffu, page_mine, at);
      const int heads = rope.heads, nkv = rope.cache.kv_heads, head = n / HEAD, d = n % HEAD;
      if (inside && (head < heads || rope.write_cache)) {
        if (rope.table != nullptr && head < heads + nkv) {
          const bool low = d < HALF;
          const float2* cs = rope.table + (size_t)(low ? d : d - HALF) * rope.table_positions + pos;
          float2 t[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) t[i] = cs[(size_t)i * rope.table_positions];
          auto turn = [&](float own, float other, float2 a) {
            return low ? fmaf(own, a.x, -(other * a.y)) : fmaf(other, a.y, own * a.x);
          };
          v = make_float4(turn(v.x, p.x, t[0]), turn(v.y, p.y, t[1]), turn(v.z, p.z, t[2]), turn(v.w, p.w, t[3]));
        }
        bf16* dst;
        if (head < heads) {
          dst = rope.q_out + ((size_t)m * heads + head) * HEAD;
        } else {
          int which = head < heads + nkv ? 0 : 1;
          dst = (bf16*)rope.cache.base +
                kv_offset(rope.cache, page, which, head - heads - which * nkv, pos % rope.cache.page_size);
        }
        *reinterpret_cast<uint2*>(dst + d) = pack(v);
      }
    } else if (inside) {
      if (EPI == EPI_STORE_F32) {
        *reinterpret_cast<float4*>((float*)c + (size_t)m * N + n) = v;
      } else if (EPI == EPI_STORE_T) {
        *reinterpret_cast<uint2*>((bf16*)c + (size_t)m * N + n) = pack(v);
      } else {  // SwiGLU
        __nv_bfloat162 o = __floats2bfloat162_rn(silu_for<bf16>(v.x) * v.y, silu_for<bf16>(v.z) * v.w);
        *reinterpret_cast<__nv_bfloat162*>((bf16*)c + (size_t)m * (N / 2) + (n >> 1)) = o;
      }
    }
    __syncwarp();
  }
  // (nobody leaves while others still read its sums)
  if (split > 1) asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
  else __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, S::BN);
}

// How many blocks share a tile's reduction: as many as the device takes at once, each with two k tiles or more; 0 where the
// product does not belong here. Microseconds with tiles of 32 columns (up to 256 rows) or wider ones, and here, the residual
// sum unless noted:
//   4096 x 14336   65 rows 73.5 / 27.6   128 74.6 / 30.0   129 74.3 / 37.4   256 75.1 / 39.8   512 111.8 / 66.8
//   4096 x 4096            23.6 / 12.1       24.4 / 14.2       24.4 / 15.3       24.6 / 16.1        43.3 / 23.8
//   2048 x 8192            42.8 / 14.1       43.4 / 15.9       43.5 / 16.1       43.9 / 17.3        66.3 / 22.7
//   576 x 1536             10.2 / 5.7        10.8 / 6.5        10.9 / 7.2        11.3 / 7.9         10.7 / 8.9
//   28672 x 4096 SwiGLU    87.6 / 47.5       88.4 / 49.1      144.2 / 81.0      145.2 / 87.4       108.5 / 166.0
//   16384 x 2048 SwiGLU    24.3 / 16.9       24.5 / 18.4       43.7 / 21.4       44.1 / 22.2        31.6 / 41.5
// With 768, 1,145 and 1,536 rows: 2048 x 2048 27.1 / 15.7, 28.6 / 16.5, 31.3 / 23.0; 2048 x 8192 66.2 / 37.1, 67.8 / 39.6, 73.1 /
// 65.0; 576 x 1536 10.8 / 9.9, 10.9 / 10.1, 11.1 / 10.6, but with 2,048 12.2 / 14.2.
// Two and more tiles of rows come here while 256-wide tiles of gemm_tcgen05_kernel would leave multiprocessors without one
// (it takes those from 128 on: 28672 x 4096 with 129 and 256 rows 61.8 / 64.7, 16384 x 2048 18.8 / 19.3). A reduction of 576
// values has nothing to share: 576 x 576 5.7 / 5.7, 6.2 / 6.8, 6.5 / 7.0; 3072 x 576 5.2 / 5.9, 5.2 / 6.9, 5.5 / 7.5. The q/k/v
// product, whose epilogue is the longer part: 6144 x 4096 (heads of 128) 100 rows 33.0 / 19.3, 129 33.8 / 28.3, 300 34.3 / 31.5,
// 500 39.0 / 52.7; 6144 x 2048 (heads of 64) 13.9 / 12.9, 15.3 / 17.9, 15.2 / 19.6, 27.8 / 30.0.
template <int EPI> int split_stretches(int M, int N, int K) {
  const int k_tiles = (K + BK - 1) / BK, m_tiles = (M + BM - 1) / BM;
  if (M <= 64 || M > 1536 || (N & 3) || k_tiles < 16) return 0;
  if (EPI == EPI_QKV_ROPE && m_tiles > (K >= 4096 ? 3 : 1)) return 0;
  if (m_tiles > 1 && N % 256 == 0 && (long long)m_tiles * (N / 256) >= 128) return 0;
  const long long tiles = (long long)m_tiles * ((N + SplitShape::BN - 1) / SplitShape::BN);
  const long long places = (long long)SplitShape::BLOCKS_PER_SM * multiprocessors();
  if (m_tiles > 2 && tiles > places) return 0;
  int split = 1;
  while (split < 8 && tiles * split * 2 <= places && k_tiles >= 4 * split) split *= 2;
  return split;
}

template <int EPI, int HD = 0>
int launch_split(void* c, const void* a, const void* w, int M, int N, int K, int split, int* status, cudaStream_t stream,
                 const RopeArgs& rope, const NormArgs& norm) {
  alignas(64) CUtensorMap map_a, map_w;
  if (!make_map(&map_a, a, M, K, BM) || !make_map(&map_w, w, N, K, SplitShape::BN)) return DLLM_LAUNCH_FAILED;
  static std::atomic<unsigned long long> allowed{0};
  if (!dllm_allow_shared((const void*)gemm_split_kernel<EPI, HD>, (int)SplitShape::SMEM, allowed)) return DLLM_LAUNCH_FAILED;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(split, (N + SplitShape::BN - 1) / SplitShape::BN, (M + BM - 1) / BM);
  config.blockDim = dim3(SplitShape::THREADS);
  config.dynamicSmemBytes = SplitShape::SMEM;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = split;
  attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = dllm_pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&config, gemm_split_kernel<EPI, HD>, map_a, map_w, c, M, N, K, status, rope, norm) == cudaSuccess
             ? DLLM_OK
             : DLLM_LAUNCH_FAILED;
}
}  // namespace
