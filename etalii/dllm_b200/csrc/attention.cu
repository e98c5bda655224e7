// Attention over the paged cache, general form: any head size that is a multiple of 8 up to 256, any number of heads and
// groups, with or without a window, float32 and bfloat16, whole prompts and single tokens.
//
// Every kernel here computes the same thing in the same order, so that a (token, head) result has the same bits whichever
// kernel gives it, however the tokens were cut into steps or batched:
//   * keys are taken in chunks of 64 positions, aligned at multiples of 64 (the pages); a chunk's result depends on nothing
//     but the query and the visible keys in it: the largest score m, weights exp(s - m), their sum l, and o = sum of
//     weight * value per dimension, one chain of multiply-adds over ascending keys;
//   * a score is two chains of multiply-adds, over the even and the odd dimensions ascending, added and then scaled;
//   * the 64 weights are summed by a fixed tree: key + key 32 further, then the butterfly over 32;
//   * the chunks' results meet in ascending order (`merge`).
// Since chunks are independent, decoding gives each to a warp of its own (attention_chunks_kernel) and a prompt's tiles of
// queries take them one after another (attention_tile_kernel).
#include "common.cuh"

namespace {
constexpr int WARPS = 4;
constexpr int MAX_HEAD_DIM = 256;

template <typename T> struct Vec;  // 16-byte vectors of the element type
template <> struct Vec<float> { static constexpr int N = 4; };
template <> struct Vec<__nv_bfloat16> { static constexpr int N = 8; };

// Packed pairs of float32 (the even and the odd dimensions' chains of a score side by side).
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// The next dimensions of a score, sixteen bytes of a key: (even, odd) in `acc`.
__device__ __forceinline__ void score_piece(float2& acc, const float* q, float4 k) {
  acc.x = fmaf(q[0], k.x, acc.x);
  acc.y = fmaf(q[1], k.y, acc.y);
  acc.x = fmaf(q[2], k.z, acc.x);
  acc.y = fmaf(q[3], k.w, acc.y);
}
__device__ __forceinline__ void score_piece(float2& acc, const float* q, uint4 raw) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 k = __bfloat1622float2(p[i]);
    acc.x = fmaf(q[2 * i], k.x, acc.x);
    acc.y = fmaf(q[2 * i + 1], k.y, acc.y);
  }
}
// The score: a product of its own, never the front half of a fused multiply-add with what is subtracted from it later.
__device__ __forceinline__ float scaled(float2 dot, float scale) { return __fmul_rn(dot.x + dot.y, scale); }
__device__ __forceinline__ float4 load_vec(const float* k) { return *(const float4*)k; }
__device__ __forceinline__ uint4 load_vec(const __nv_bfloat16* k) { return *(const uint4*)k; }

// What is subtracted in an exponent: a chunk (or a run of chunks) whose scores are all -inf has weights of 0, not NaN.
__device__ __forceinline__ float finite_or_zero(float m) { return m == -INFINITY ? 0.f : m; }

// A chunk's result joins those before it: factors for the old and the new, the sum of weights and the maximum updated.
// The first chunk (m = -inf, l = 0, o = 0) joins like any other: 0 * its factor + the chunk's.
__device__ __forceinline__ void merge(float& m, float& l, float chunk_m, float chunk_l, float& keep, float& take) {
  float m_new = fmaxf(m, chunk_m), shift = finite_or_zero(m_new);
  keep = expf(m - shift);
  take = expf(chunk_m - shift);
  l = fmaf(l, keep, __fmul_rn(chunk_l, take));
  m = m_new;
}
__device__ __forceinline__ float merge_output(float o, float keep, float chunk_o, float take) {
  return fmaf(o, keep, __fmul_rn(chunk_o, take));
}

template <typename T>
__global__ void __launch_bounds__(WARPS * 32) attention_warp_kernel(
    T* __restrict__ out, const T* __restrict__ q, KvLayout cache, const int* __restrict__ tok_seq,
    const int* __restrict__ tok_pos, const int* __restrict__ slots, int tokens, int heads, float scale, int window) {
  __shared__ float q_s[WARPS][MAX_HEAD_DIM];
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long item = (long long)blockIdx.x * WARPS + warp;
  if (item >= (long long)tokens * heads) return;
  int t = (int)(item / heads), h = (int)(item % heads);
  int hd = cache.head_dim, ps = cache.page_size;
  int g = h / (heads / cache.kv_heads);
  int pos = tok_pos[t];
  const int* pages = cache.page_table + (size_t)slots[tok_seq[t]] * cache.max_pages;
  const T* qrow = q + ((size_t)t * heads + h) * hd;
  for (int d = lane; d < hd; d += 32) q_s[warp][d] = to_float(qrow[d]);
  __syncwarp();

  int end = pos + 1;
  int first = (window > 0 && end > window) ? end - window : 0;
  float m_run = -INFINITY, l_run = 0.f;
  float acc[MAX_HEAD_DIM / 32];
#pragma unroll
  for (int i = 0; i < MAX_HEAD_DIM / 32; ++i) acc[i] = 0.f;
  const T* base = (const T*)cache.base;

  for (int c0 = first / 64 * 64; c0 < end; c0 += 64) {
    float s[2], p[2];
    int page[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      int j = c0 + lane + 32 * u;
      bool valid = j >= first && j < end;
      page[u] = valid ? pages[j / ps] : 0;
      s[u] = -INFINITY;
      if (valid) {
        const T* krow = base + kv_offset(cache, page[u], 0, g, j % ps);
        float2 dot = make_float2(0.f, 0.f);
        for (int d = 0; d < hd; d += Vec<T>::N) score_piece(dot, &q_s[warp][d], load_vec(krow + d));
        s[u] = scaled(dot, scale);
      }
    }
    float m = warp_max(fmaxf(s[0], s[1])), shift = finite_or_zero(m);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      int j = c0 + lane + 32 * u;
      p[u] = j >= first && j < end ? expf(s[u] - shift) : 0.f;
    }
    float l = warp_sum(p[0] + p[1]), o[MAX_HEAD_DIM / 32];
#pragma unroll
    for (int i = 0; i < MAX_HEAD_DIM / 32; ++i) o[i] = 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      int from = max(0, first - c0 - 32 * u), to = min(32, end - c0 - 32 * u);
      for (int jj = from; jj < to; ++jj) {
        float pj = __shfl_sync(0xffffffffu, p[u], jj);
        int pg = __shfl_sync(0xffffffffu, page[u], jj);
        const T* vrow = base + kv_offset(cache, pg, 1, g, (c0 + 32 * u + jj) % ps);
#pragma unroll
        for (int i = 0; i < MAX_HEAD_DIM / 32; ++i) {
          int d = lane + 32 * i;
          if (d < hd) o[i] = fmaf(pj, to_float(vrow[d]), o[i]);
        }
      }
    }
    float keep, take;
    merge(m_run, l_run, m, l, keep, take);
#pragma unroll
    for (int i = 0; i < MAX_HEAD_DIM / 32; ++i) acc[i] = merge_output(acc[i], keep, o[i], take);
  }
  float inv = 1.0f / l_run;
  T* orow = out + ((size_t)t * heads + h) * hd;
#pragma unroll
  for (int i = 0; i < MAX_HEAD_DIM / 32; ++i) {
    int d = lane + 32 * i;
    if (d < hd) orow[d] = from_float<T>(acc[i] * inv);
  }
}

// ---- the same attention, blockwise ------------------------------------------------------------------------------
// A block serves one kv head and a run of consecutive tokens of the step; its warps are the (token, query head)
// pairs of that run, R tokens a warp. The block copies the keys and values of the kv head page by page (64
// positions, one chunk) into shared memory, with the next page on its way (cp.async) while the warps work on this one.
// Two keys a lane for the scores, one value dimension a lane for the weighted sum. Tokens of several sequences in one
// block are served sequence by sequence. This form takes what the float32 kernels below do not: bfloat16, prompts with
// other head sizes, single tokens whose chunks' results do not fit into a cluster's shared memory.
template <typename T> struct Pad { static constexpr int N = 16 / sizeof(T); };  // 16 bytes: rows in different banks

template <typename T>
__device__ __forceinline__ void stage_page(T* k_s, T* v_s, const KvLayout& cache, int page, int g, int hd, int ld,
                                           int tid, int threads) {
  const T* ksrc = (const T*)cache.base + kv_offset(cache, page, 0, g, 0);
  const T* vsrc = (const T*)cache.base + kv_offset(cache, page, 1, g, 0);
  constexpr int VN = Vec<T>::N;
  int pieces = hd / VN;  // 16-byte pieces of a row
  for (int i = tid; i < 64 * pieces; i += threads) {
    int r = i / pieces, c = (i % pieces) * VN;
    unsigned kd = (unsigned)__cvta_generic_to_shared(k_s + r * ld + c);
    unsigned vd = (unsigned)__cvta_generic_to_shared(v_s + r * ld + c);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(kd), "l"(ksrc + (size_t)r * hd + c));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(vd), "l"(vsrc + (size_t)r * hd + c));
  }
  asm volatile("cp.async.commit_group;\n" ::);
}

template <typename T, int R, int CHUNKS>  // CHUNKS: head_dim / 32 rounded up (value dimensions a lane owns)
__global__ void __launch_bounds__(512) attention_block_kernel(
    T* __restrict__ out, const T* __restrict__ q, KvLayout cache, const int* __restrict__ tok_seq,
    const int* __restrict__ tok_pos, const int* __restrict__ slots, int tokens, int heads, float scale, int window,
    int heads_per_pass, int stages) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // Values are multiplied without bounds over spans of keys that every token sees all of: the page, or for rows of 32 values
  // its halves (a page with an edge in it then keeps one: 8 heads of 32, prompt of 2,048 under a window of 100, 92 -> 50 us.
  // Longer rows have no registers for that beside short prompts' needs: 4 heads of 256, seven tokens each, 68.6 -> 76.4).
  constexpr int SPANS = R > 1 && CHUNKS == 1 ? 2 : 1, SPAN = 64 / SPANS;
  int hd = cache.head_dim, ld = hd + Pad<T>::N;
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  int token_slots = warps / heads_per_pass;       // warps = token_slots * heads_per_pass
  int block_tokens = token_slots * R;
  int slot_of_warp = warp / heads_per_pass, head_of_warp = warp % heads_per_pass;
  T* kv_s = reinterpret_cast<T*>(smem_raw);       // [stages][k|v][64][ld]
  float* q_all = reinterpret_cast<float*>(smem_raw + (size_t)stages * 2 * 64 * ld * sizeof(T));
  float* q_s = q_all + (size_t)warp * R * hd;                        // this warp's R queries
  float* p_s = q_all + (size_t)warps * R * hd + (size_t)warp * R * 64;  // and their weights for the page at hand
  int g = blockIdx.y, group = heads / cache.kv_heads;
  // (the last tokens of a prompt see the most keys: their blocks go first, the short ones fill the gaps behind)
  int t0 = (int)(gridDim.x - 1 - blockIdx.x) * block_tokens, t_stop = min(tokens, t0 + block_tokens);

  for (int pass = 0; pass < group; pass += heads_per_pass) {
    int h = g * group + pass + head_of_warp;
    bool head_ok = pass + head_of_warp < group;
    for (int run_begin = t0; run_begin < t_stop;) {
      // a run: the block's tokens of one sequence (positions ascend inside it)
      int seq = tok_seq[run_begin], run_end = run_begin + 1;
      while (run_end < t_stop && tok_seq[run_end] == seq) ++run_end;
      const int* pages = cache.page_table + (size_t)slots[seq] * cache.max_pages;
      int run_last = tok_pos[run_end - 1] + 1;   // keys [run_first, run_last) are read by somebody of the run
      int first_end = tok_pos[run_begin] + 1;
      int run_first = (window > 0 && first_end > window) ? first_end - window : 0;

      // this warp's tokens of the run
      int end[R], first[R];
      float m_run[R], l_run[R], acc[R][CHUNKS];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        int t = t0 + slot_of_warp * R + r;
        bool mine = head_ok && t >= run_begin && t < run_end;
        end[r] = mine ? tok_pos[t] + 1 : 0;
        first[r] = (window > 0 && end[r] > window) ? end[r] - window : 0;
        m_run[r] = -INFINITY;
        l_run[r] = 0.f;
#pragma unroll
        for (int i = 0; i < CHUNKS; ++i) acc[r][i] = 0.f;
        if (mine) {
          const T* qrow = q + ((size_t)t * heads + h) * hd;
          for (int d = lane; d < hd; d += 32) q_s[r * hd + d] = to_float(qrow[d]);
        }
      }
      __syncwarp();

      int page_first = run_first / 64, page_last = (run_last - 1) / 64;
      __syncthreads();  // (the stages may still be read by a warp that is behind in the run before)
      stage_page(kv_s, kv_s + 64 * ld, cache, pages[page_first], g, hd, ld, threadIdx.x, blockDim.x);
      for (int p = page_first; p <= page_last; ++p) {
        int stage = stages == 2 ? ((p - page_first) & 1) : 0;
        T* k_s = kv_s + (size_t)stage * 2 * 64 * ld;
        T* v_s = k_s + 64 * ld;
        if (stages == 2 && p < page_last) {
          T* next = kv_s + (size_t)(stage ^ 1) * 2 * 64 * ld;
          stage_page(next, next + 64 * ld, cache, pages[p + 1], g, hd, ld, threadIdx.x, blockDim.x);
          asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
          asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        // The warp's R tokens walk the page together: a key is loaded once for the R scores and a value once for the
        // R weighted sums (what a token computes, and in which order, is what it would compute alone).
        int j0 = p * 64;
        bool active[R], any = false, lower = false, upper = false, whole = hd == CHUNKS * 32;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          active[r] = j0 < end[r] && j0 + 64 > first[r];  // (warp-uniform) a visible key in this page
          any = any || active[r];
          lower = lower || (active[r] && first[r] < j0 + 32);
          upper = upper || (active[r] && j0 + 32 < end[r]);
          whole = whole && (!active[r] || (first[r] <= j0 && j0 + 64 <= end[r]));
        }
        if (any) {
          float weight[R][2], chunk_m[R], chunk_l[R];
          auto join = [&](int r, const float* o) {  // the page's result joins those before it
            float keep, take;
            merge(m_run[r], l_run[r], chunk_m[r], chunk_l[r], keep, take);
#pragma unroll
            for (int i = 0; i < CHUNKS; ++i) acc[r][i] = merge_output(acc[r][i], keep, o[i], take);
          };
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            if (!(u == 0 ? lower : upper)) {  // 32 keys that nobody sees: masked below, as any such key
#pragma unroll
              for (int r = 0; r < R; ++r) weight[r][u] = 0.f;
              continue;
            }
            const T* krow = k_s + (lane + 32 * u) * ld;
            float2 dot[R];
#pragma unroll
            for (int r = 0; r < R; ++r) dot[r] = make_float2(0.f, 0.f);
            if (hd == CHUNKS * 32) {
#pragma unroll 8
              for (int d = 0; d < CHUNKS * 32; d += Vec<T>::N) {
                auto key = load_vec(krow + d);
#pragma unroll
                for (int r = 0; r < R; ++r) score_piece(dot[r], &q_s[r * hd + d], key);
              }
            } else {
              for (int d = 0; d < hd; d += Vec<T>::N) {
                auto key = load_vec(krow + d);
#pragma unroll
                for (int r = 0; r < R; ++r) score_piece(dot[r], &q_s[r * hd + d], key);
              }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) weight[r][u] = scaled(dot[r], scale);
          }
          // (a single token a warp, as in decoding, hands its weights from lane to lane by shuffles; several go
          // through shared memory, four weights a load)
          if (R > 1) __syncwarp();  // (the weights of the page before have been read by every lane)
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (!active[r]) continue;
            bool valid[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              int j = j0 + lane + 32 * u;
              valid[u] = j >= first[r] && j < end[r];
              if (!valid[u]) weight[r][u] = -INFINITY;
            }
            chunk_m[r] = warp_max(fmaxf(weight[r][0], weight[r][1]));
            float shift = finite_or_zero(chunk_m[r]);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              weight[r][u] = valid[u] ? expf(weight[r][u] - shift) : 0.f;
              if (R > 1) p_s[r * 64 + 32 * u + lane] = weight[r][u];
            }
            chunk_l[r] = warp_sum(weight[r][0] + weight[r][1]);
          }
          if (R > 1) __syncwarp();
          const T* vtile = v_s + lane;
          auto weight_of = [&](int r, int jj) {
            return R > 1 ? p_s[r * 64 + jj] : __shfl_sync(0xffffffffu, jj < 32 ? weight[r][0] : weight[r][1], jj & 31);
          };
          if (hd == CHUNKS * 32 && (SPANS > 1 || whole)) {
            float o[R][CHUNKS];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int i = 0; i < CHUNKS; ++i) o[r][i] = 0.f;
#pragma unroll
            for (int span = 0; span < SPANS; ++span) {
              const int k0 = span * SPAN;
              bool sees[R], all = true;
#pragma unroll
              for (int r = 0; r < R; ++r) {
                sees[r] = SPANS > 1 ? active[r] && j0 + k0 < end[r] && j0 + k0 + SPAN > first[r] : active[r];
                if (SPANS > 1) all = all && (!sees[r] || (first[r] <= j0 + k0 && j0 + k0 + SPAN <= end[r]));
              }
              if (all) {  // every token that sees the span sees all of it: no bounds in the loop
#pragma unroll 4
                for (int jj = k0; jj < k0 + SPAN; jj += 4) {
                  float v[4][CHUNKS];
#pragma unroll
                  for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int i = 0; i < CHUNKS; ++i) v[u][i] = to_float(vtile[(jj + u) * ld + 32 * i]);
#pragma unroll
                  for (int r = 0; r < R; ++r) {
                    if (!sees[r]) continue;  // (a token that does not see the keys must not meet what lies there)
                    float4 pj;
                    if (R > 1) {
                      pj = *reinterpret_cast<const float4*>(&p_s[r * 64 + jj]);
                    } else {
                      float mine = jj < 32 ? weight[r][0] : weight[r][1];
                      pj.x = __shfl_sync(0xffffffffu, mine, jj & 31);
                      pj.y = __shfl_sync(0xffffffffu, mine, (jj & 31) + 1);
                      pj.z = __shfl_sync(0xffffffffu, mine, (jj & 31) + 2);
                      pj.w = __shfl_sync(0xffffffffu, mine, (jj & 31) + 3);
                    }
#pragma unroll
                    for (int i = 0; i < CHUNKS; ++i) {
                      o[r][i] = fmaf(pj.x, v[0][i], o[r][i]);
                      o[r][i] = fmaf(pj.y, v[1][i], o[r][i]);
                      o[r][i] = fmaf(pj.z, v[2][i], o[r][i]);
                      o[r][i] = fmaf(pj.w, v[3][i], o[r][i]);
                    }
                  }
                }
              } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  if (!sees[r]) continue;
                  int from = max(k0, first[r] - j0), to = min(k0 + SPAN, end[r] - j0);
                  for (int jj = from; jj < to; ++jj) {
                    float pj = weight_of(r, jj);
#pragma unroll
                    for (int i = 0; i < CHUNKS; ++i) o[r][i] = fmaf(pj, to_float(vtile[jj * ld + 32 * i]), o[r][i]);
                  }
                }
              }
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (active[r]) join(r, o[r]);
          } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
              if (!active[r]) continue;
              float o[CHUNKS];
#pragma unroll
              for (int i = 0; i < CHUNKS; ++i) o[i] = 0.f;
              int from = max(0, first[r] - j0), to = min(64, end[r] - j0);
              for (int jj = from; jj < to; ++jj) {
                float pj = weight_of(r, jj);
#pragma unroll
                for (int i = 0; i < CHUNKS; ++i)
                  if (lane + 32 * i < hd) o[i] = fmaf(pj, to_float(vtile[jj * ld + 32 * i]), o[i]);
              }
              join(r, o);
            }
          }
        }
        if (stages != 2) {
          __syncthreads();  // one stage: it is free only when every warp is done with it
          if (p < page_last) stage_page(kv_s, kv_s + 64 * ld, cache, pages[p + 1], g, hd, ld, threadIdx.x, blockDim.x);
        } else {
          __syncthreads();  // the stage read now is the one the copy after next writes
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        int t = t0 + slot_of_warp * R + r;
        if (head_ok && t >= run_begin && t < run_end) {
          float inv = 1.0f / l_run[r];
          T* orow = out + ((size_t)t * heads + h) * hd;
#pragma unroll
          for (int i = 0; i < CHUNKS; ++i) {
            int d = lane + 32 * i;
            if (d < hd) orow[d] = from_float<T>(acc[r][i] * inv);
          }
        }
      }
      run_begin = run_end;
    }
  }
}

template <typename T, int R, int CHUNKS>
int launch_blocks(void* out, const void* q, const KvLayout& cache, const int* tok_seq, const int* tok_pos,
                  const int* slots, int tokens, int heads, float scale, int window, cudaStream_t stream) {
  int group = heads / cache.kv_heads;
  int heads_per_pass = group < 16 ? group : 16;
  int token_slots = R == 1 ? 1 : (16 / heads_per_pass > 0 ? 16 / heads_per_pass : 1);
  int warps = token_slots * heads_per_pass;
  int ld = cache.head_dim + Pad<T>::N;
  size_t stage_bytes = (size_t)2 * 64 * ld * sizeof(T);
  size_t q_bytes = (size_t)warps * R * (cache.head_dim + 64) * sizeof(float);  // queries and a page's weights
  int stages = 2 * stage_bytes + q_bytes <= 200 * 1024 ? 2 : 1;
  size_t smem = stages * stage_bytes + q_bytes;
  static size_t configured = 0;
  if (smem > configured) {
    if (cudaFuncSetAttribute(attention_block_kernel<T, R, CHUNKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
      return DLLM_LAUNCH_FAILED;
    configured = smem;
  }
  int block_tokens = token_slots * R;
  dim3 grid((tokens + block_tokens - 1) / block_tokens, cache.kv_heads);
  attention_block_kernel<T, R, CHUNKS><<<grid, warps * 32, smem, stream>>>((T*)out, (const T*)q, cache, tok_seq, tok_pos,
                                                                  slots, tokens, heads, scale, window,
                                                                  heads_per_pass, stages);
  return dllm_launch_status();
}
// ---- float32 with heads of 64 and 128: tiles of 32 queries of one head -----------------------------------------------------
// Bound by multiply-adds and the shared-memory reads that feed them, so it is laid out like a product: a block takes 32
// consecutive new tokens of a sequence and one query head, a thread four tokens (ty + 8 i) by four keys (tx + 16 j) of the
// scores and by HD / 16 dimensions of the outputs; a key, value or weight read from shared memory serves four multiply-adds,
// the even and odd dimensions of a score and neighbouring output dimensions share a packed one. The next page's keys are on
// their way while values are multiplied, the next values while scores are. 32 queries rather than 64: a prompt of 2,048 with
// nine heads is 576 blocks, which level out over the device although the last ones see 32 times the keys of the first ones
// (those go first). Before, a warp walked the keys for four tokens, and read a value and a weight for every four
// multiply-adds: 492 us a layer at 2,048 tokens (9 query, 3 kv heads of 64), now 214 (23 TFLOP/s).
// A tile never spans two sequences, and one of up to eight tokens is one row a thread: a step in which many sequences bring a
// token or two beside a prompt is many small blocks side by side.
constexpr int TILE_Q = 32, TILE_THREADS = 128;

template <int HD>
struct TileShared {
  float q[TILE_Q][HD + 4], k[64][HD + 4], v[64][HD + 4], p[TILE_Q][64 + 4];
};

// One tile: `count` tokens, at most 8 * NI, from position pos0 of the sequence on; q and out at the first one's row.
template <int HD, int NI>
__device__ __forceinline__ void attend_tile(TileShared<HD>& sm, float* __restrict__ out, const float* __restrict__ q,
                                            const KvLayout& cache, const int* __restrict__ pages, int count, int pos0, int h,
                                            int g, int heads, float scale, int window) {
  constexpr int GROUPS = HD / 64;  // groups of four output dimensions a thread owns, 64 apart
  int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  auto copy_page = [&](float (*to)[HD + 4], int page, int which) {
    const float* from = (const float*)cache.base + kv_offset(cache, page, which, g, 0);
#pragma unroll 4
    for (int i = tid; i < 64 * (HD / 4); i += TILE_THREADS) {
      int r = i / (HD / 4), d = i % (HD / 4) * 4;
      unsigned at = (unsigned)__cvta_generic_to_shared(&to[r][d]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(at), "l"(from + (size_t)r * HD + d));
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  int run_first = (window > 0 && pos0 + 1 > window) ? pos0 + 1 - window : 0;  // keys from here on are seen by somebody
  int page_first = run_first / 64, page_last = (pos0 + count - 1) / 64;
  copy_page(sm.k, pages[page_first], 0);
  copy_page(sm.v, pages[page_first], 1);
  for (int i = tid; i < 8 * NI * (HD / 4); i += TILE_THREADS) {
    int r = i / (HD / 4), d = i % (HD / 4) * 4;
    float4 value = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < count) value = *(const float4*)(q + ((size_t)r * heads + h) * HD + d);
    *(float4*)&sm.q[r][d] = value;
  }
  int end[NI], first[NI];  // keys [first, end) are seen by row ty + 8 i
  float m_run[NI], l_run[NI];
  unsigned long long acc[NI][2 * GROUPS];
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    end[i] = ty + 8 * i < count ? pos0 + ty + 8 * i + 1 : 0;
    first[i] = (window > 0 && end[i] > window) ? end[i] - window : 0;
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
#pragma unroll
    for (int x = 0; x < 2 * GROUPS; ++x) acc[i][x] = 0;
  }
  for (int p = page_first; p <= page_last; ++p) {
    int j0 = p * 64;
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // the page's keys (its values may still be on their way)
    __syncthreads();
    float s[NI][4];
    {
      unsigned long long dot[NI][4];
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dot[i][j] = 0;
#pragma unroll 4
      for (int d = 0; d < HD; d += 4) {
        ulonglong2 key[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) key[j] = *(const ulonglong2*)&sm.k[tx + 16 * j][d];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          ulonglong2 query = *(const ulonglong2*)&sm.q[ty + 8 * i][d];
#pragma unroll
          for (int j = 0; j < 4; ++j) dot[i][j] = fma2(query.x, key[j].x, dot[i][j]);
#pragma unroll
          for (int j = 0; j < 4; ++j) dot[i][j] = fma2(query.y, key[j].y, dot[i][j]);
        }
      }
#pragma unroll
      for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = scaled(unpack2(dot[i][j]), scale);
        }
    }
    bool whole = true;  // every token of this thread that sees the page sees all of it
    float chunk_m[NI], chunk_l[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      bool sees = j0 < end[i] && j0 + 64 > first[i];  // (what a token that does not is given here is dropped below)
      whole = whole && (!sees || (first[i] <= j0 && j0 + 64 <= end[i]));
      bool valid[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        int key = j0 + tx + 16 * j;
        valid[j] = key >= first[i] && key < end[i];
        if (!valid[j]) s[i][j] = -INFINITY;
      }
      float m = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
      float shift = finite_or_zero(m);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = valid[j] ? expf(s[i][j] - shift) : 0.f;
        sm.p[ty + 8 * i][tx + 16 * j] = s[i][j];
      }
      float l = (s[i][0] + s[i][2]) + (s[i][1] + s[i][3]);
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
      chunk_m[i] = m;
      chunk_l[i] = l;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");  // the page's values
    __syncthreads();  // values and weights are there, everybody is done with the keys
    if (p < page_last) copy_page(sm.k, pages[p + 1], 0);
    unsigned long long o[NI][2 * GROUPS];
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
      for (int x = 0; x < 2 * GROUPS; ++x) o[i][x] = 0;
    if (__all_sync(0xffffffffu, whole)) {
#pragma unroll 2
      for (int jj = 0; jj < 64; jj += 4) {
        float4 weight[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) weight[i] = *(const float4*)&sm.p[ty + 8 * i][jj];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          unsigned long long value[2 * GROUPS];
#pragma unroll
          for (int x = 0; x < GROUPS; ++x) {
            ulonglong2 two = *(const ulonglong2*)&sm.v[jj + u][64 * x + 4 * tx];
            value[2 * x] = two.x;
            value[2 * x + 1] = two.y;
          }
#pragma unroll
          for (int i = 0; i < NI; ++i) {
            float one = u == 0 ? weight[i].x : u == 1 ? weight[i].y : u == 2 ? weight[i].z : weight[i].w;
            unsigned long long both = pack2(one, one);
#pragma unroll
            for (int x = 0; x < 2 * GROUPS; ++x) o[i][x] = fma2(both, value[x], o[i][x]);
          }
        }
      }
    } else {  // (a token must not meet what lies at positions that it does not see)
      int from = 64, to = 0;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        if (j0 < end[i] && j0 + 64 > first[i]) {
          from = min(from, max(0, first[i] - j0));
          to = max(to, min(64, end[i] - j0));
        }
      }
      for (int jj = from; jj < to; ++jj) {
        unsigned long long value[2 * GROUPS];
#pragma unroll
        for (int x = 0; x < GROUPS; ++x) {
          ulonglong2 two = *(const ulonglong2*)&sm.v[jj][64 * x + 4 * tx];
          value[2 * x] = two.x;
          value[2 * x + 1] = two.y;
        }
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          if (j0 + jj < first[i] || j0 + jj >= end[i]) continue;
          float one = sm.p[ty + 8 * i][jj];
          unsigned long long both = pack2(one, one);
#pragma unroll
          for (int x = 0; x < 2 * GROUPS; ++x) o[i][x] = fma2(both, value[x], o[i][x]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      if (j0 >= end[i] || j0 + 64 <= first[i]) continue;  // (no visible key in this page: it does not take part)
      float keep, take;
      merge(m_run[i], l_run[i], chunk_m[i], chunk_l[i], keep, take);
#pragma unroll
      for (int x = 0; x < 2 * GROUPS; ++x) {
        float2 before = unpack2(acc[i][x]), now = unpack2(o[i][x]);
        acc[i][x] = pack2(merge_output(before.x, keep, now.x, take), merge_output(before.y, keep, now.y, take));
      }
    }
    __syncthreads();  // everybody is done with the values and weights
    if (p < page_last) copy_page(sm.v, pages[p + 1], 1);
  }
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    if (end[i] == 0) continue;
    float inv = 1.0f / l_run[i];
    float* row = out + ((size_t)(ty + 8 * i) * heads + h) * HD;
#pragma unroll
    for (int x = 0; x < GROUPS; ++x) {
      float2 lo = unpack2(acc[i][2 * x]), hi = unpack2(acc[i][2 * x + 1]);
      *(float4*)(row + 64 * x + 4 * tx) = make_float4(lo.x * inv, lo.y * inv, hi.x * inv, hi.y * inv);
    }
  }
}

// `tile_seq` / `tile_first`: the sequence of each stretch of up to 64 new tokens and its first token among that sequence's, the
// longest contexts first. A stretch is two tiles, the later one first.
template <int HD>
__global__ void __launch_bounds__(TILE_THREADS, HD == 64 ? 4 : 2) attention_tile_kernel(
    float* __restrict__ out, const float* __restrict__ q, KvLayout cache, const int* __restrict__ tok_pos,
    const int* __restrict__ slots, const int* __restrict__ tile_seq, const int* __restrict__ tile_first,
    const int* __restrict__ cu_seqlens, int heads, float scale, int window) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TileShared<HD>& sm = *reinterpret_cast<TileShared<HD>*>(smem_raw);
  int h = blockIdx.x % heads, item = blockIdx.x / heads, seq = tile_seq[item >> 1];
  int t0 = cu_seqlens[seq] + tile_first[item >> 1] + (item & 1 ? 0 : TILE_Q);
  int count = min(TILE_Q, cu_seqlens[seq + 1] - t0);
  if (count <= 0) return;
  const int* pages = cache.page_table + (size_t)slots[seq] * cache.max_pages;
  const float* rows = q + (size_t)t0 * heads * HD;
  float* to = out + (size_t)t0 * heads * HD;
  int g = h / (heads / cache.kv_heads), pos0 = tok_pos[t0];  // (a sequence's new tokens have ascending positions)
  if (count <= 8) attend_tile<HD, 1>(sm, to, rows, cache, pages, count, pos0, h, g, heads, scale, window);
  else attend_tile<HD, 4>(sm, to, rows, cache, pages, count, pos0, h, g, heads, scale, window);
}

template <int HD>
int launch_tiles(float* out, const float* q, const KvLayout& cache, const int* tok_pos, const int* slots, const int* tile_seq,
                 const int* tile_first, const int* cu_seqlens, int tiles, int heads, float scale, int window,
                 cudaStream_t stream) {
  static std::atomic<unsigned long long> allowed{0};
  constexpr int smem = (int)sizeof(TileShared<HD>);
  if (!dllm_allow_shared((const void*)attention_tile_kernel<HD>, smem, allowed)) return DLLM_LAUNCH_FAILED;
  long long blocks = 2ll * tiles * heads;
  if (blocks > 0x7fffffffLL) return DLLM_UNSUPPORTED_SIZE;
  attention_tile_kernel<HD><<<(unsigned)blocks, TILE_THREADS, smem, stream>>>(
      out, q, cache, tok_pos, slots, tile_seq, tile_first, cu_seqlens, heads, scale, window);
  return dllm_launch_status();
}

// ---- float32 single tokens: chunks of keys side by side ------------------------------------------------------------------
// Bound by latency: one token's heads over a few thousand keys are little work, so the chunks of 64 keys are dealt out to
// the blocks of a cluster (chunk c to block c mod cluster size) and `per_round` of them at a time to the warps of a block,
// a warp per (chunk, head). Every chunk's (m, l, o) stays in the shared memory of the block that made it; after one cluster
// barrier each output dimension is merged over the chunks in ascending order by one thread of the cluster, reading them
// through distributed shared memory. A second barrier keeps the blocks' memory alive until everybody has read.
// Eight sequences of 50 to 700 tokens, 9 query and 3 kv heads of 64: 38.8 us a layer with a warp walking all keys of its
// head.
// Keys and values of earlier steps are nobody's output in this one, nor are positions, slots and page numbers: the first
// round's rows travel before the wait on the kernel in front, but for the newest, which that kernel writes. HD: the head
// size where it is known to the compiler (64 and 128: the copies' places are shifts then, and the loops over the dimensions
// are flat), 0 for all others. With that, page numbers read once a chunk instead of once a piece, the outputs dealt out to
// all blocks and sixteen chunks asked for at a time in the merge, us before and now: 9 query and 3 kv heads of 64, eight
// sequences of 50 to 700 13.4 -> 8.1, of 2,000 28.5 -> 19.0, sixteen of 260 13.0 -> 7.7; 32 and 8 heads of 128, four of 500
// 16.3 -> 10.8; 4 and 2 of 256, two of 500 27.4 -> 11.5.
constexpr int CHUNK_WARPS = 16;

template <int HD>
__global__ void __launch_bounds__(CHUNK_WARPS * 32) attention_chunks_kernel(
    float* __restrict__ out, const float* __restrict__ q, KvLayout cache, const int* __restrict__ tok_seq,
    const int* __restrict__ tok_pos, const int* __restrict__ slots, int heads, float scale, int window, int heads_per_block,
    int per_round, int room, int* __restrict__ status) {
  extern __shared__ __align__(16) float smem[];
  const int hd = HD ? HD : cache.head_dim, ld = hd + 4, pieces = hd / 4;
  int group = heads / cache.kv_heads;
  int size = (int)gridDim.x, rank = (int)blockIdx.x;  // (a cluster is a row of the grid)
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, threads = (int)blockDim.x;
  int parts = (group + heads_per_block - 1) / heads_per_block;
  int g = (int)blockIdx.y / parts, head0 = (int)blockIdx.y % parts * heads_per_block, t = (int)blockIdx.z;
  int here = min(heads_per_block, group - head0);    // heads of this block: g * group + head0 + [0, here)
  float* kv_s = smem;                                // [per_round][k|v][64][ld]
  float* q_s = kv_s + (size_t)per_round * 2 * 64 * ld;          // [heads_per_block][hd]
  float* result = q_s + (size_t)heads_per_block * hd;           // [room][heads_per_block][hd + 2]: o, m, l
  int end = tok_pos[t] + 1, first = (window > 0 && end > window) ? end - window : 0;
  const int* pages = cache.page_table + (size_t)slots[tok_seq[t]] * cache.max_pages;
  int chunk0 = first / 64, chunks = min((end + 63) / 64 - chunk0, room * size);
  // (`room` covers what the caller says; a token that sees more gets no number, and the host is told)
  bool told = chunks == (end + 63) / 64 - chunk0;
  int mine = warp / heads_per_block, head = warp % heads_per_block;
  auto copy_rows = [&](int n, int c, int from, int to) {  // rows [from, to) of chunk c's keys and values, to place n
    const float* base = (const float*)cache.base;
    size_t keys = kv_offset(cache, pages[chunk0 + c], 0, g, 0), values = kv_offset(cache, pages[chunk0 + c], 1, g, 0);
    int count = (to - from) * pieces;
    for (int i = threadIdx.x; i < 2 * count; i += threads) {
      int which = i >= count, j = i - which * count;
      int row = from + j / pieces, d = j % pieces * 4;
      unsigned at = (unsigned)__cvta_generic_to_shared(kv_s + ((size_t)(n * 2 + which) * 64 + row) * ld + d);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(at),
                   "l"(base + (which ? values : keys) + (size_t)row * hd + d));
    }
  };
  // Chunks c0, c0 + size, ... (per_round of them at most); nobody reads what lies behind the last key. `before`: the rows
  // that were there before this step; `newest`: the one that was not.
  auto ask = [&](int c0, bool before, bool newest) {
    for (int n = 0; n < per_round && c0 + n * size < chunks; ++n) {
      int c = c0 + n * size, last = min(64, end - (chunk0 + c) * 64);  // (rows of it that exist)
      bool has_newest = (chunk0 + c) * 64 + last == end;
      if (before) copy_rows(n, c, 0, has_newest ? last - 1 : last);
      if (newest && has_newest) copy_rows(n, c, last - 1, last);
    }
  };
  ask(rank, true, false);
  pdl_wait();
  if (!told && threadIdx.x == 0) *(volatile int*)status = 50;
  ask(rank, false, true);
  for (int i = threadIdx.x; i < here * hd; i += threads)
    q_s[i] = q[((size_t)t * heads + g * group + head0) * hd + i];
  for (int c0 = rank; c0 < chunks; c0 += size * per_round) {
    if (c0 != rank) {
      __syncthreads();  // (everybody is done with the round before)
      ask(c0, true, true);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    int c = c0 + mine * size;
    if (mine < per_round && head < here && c < chunks) {
      const float* k_s = kv_s + (size_t)mine * 128 * ld;
      const float* v_s = k_s + 64 * ld;
      const float* query = q_s + head * hd;
      int j0 = (chunk0 + c) * 64;
      float2 dot[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll (HD ? 8 : 4)
      for (int d = 0; d < hd; d += 4) {
        float4 piece = *(const float4*)(query + d);
        float values[4] = {piece.x, piece.y, piece.z, piece.w};
        score_piece(dot[0], values, load_vec(k_s + lane * ld + d));
        score_piece(dot[1], values, load_vec(k_s + (lane + 32) * ld + d));
      }
      float p[2];
      bool valid[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        int j = j0 + lane + 32 * u;
        valid[u] = j >= first && j < end;
        p[u] = valid[u] ? scaled(dot[u], scale) : -INFINITY;
      }
      float m = warp_max(fmaxf(p[0], p[1])), shift = finite_or_zero(m);
#pragma unroll
      for (int u = 0; u < 2; ++u) p[u] = valid[u] ? expf(p[u] - shift) : 0.f;
      float l = warp_sum(p[0] + p[1]);
      int from = max(0, first - j0), to = min(64, end - j0);
      float* slot = result + ((size_t)(c / size) * heads_per_block + head) * (hd + 2);
      for (int d0 = 0; d0 < hd; d0 += 64) {  // two dimensions a lane
        float o0 = 0.f, o1 = 0.f;
        const float* column = v_s + d0 + lane;
        bool has0 = d0 + lane < hd, has1 = d0 + lane + 32 < hd;
        auto step = [&](int at) {
          float w = __shfl_sync(0xffffffffu, at < 32 ? p[0] : p[1], at & 31);
          if (has0) o0 = fmaf(w, column[at * ld], o0);
          if (has1) o1 = fmaf(w, column[at * ld + 32], o1);
        };
        if (from == 0 && to == 64) {
#pragma unroll 16
          for (int at = 0; at < 64; ++at) step(at);
        } else {
          for (int at = from; at < to; ++at) step(at);
        }
        if (has0) slot[d0 + lane] = o0;
        if (has1) slot[d0 + lane + 32] = o1;
      }
      if (lane == 0) {
        slot[hd] = m;
        slot[hd + 1] = l;
      }
    }
  }
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
  pdl_launch_dependents();  // (behind the chunks: see the products of few rows in gemm_simt.cu)
  unsigned local = (unsigned)__cvta_generic_to_shared(result);
  // (the outputs are dealt out evenly: every block of the cluster has some)
  int total = here * hd, per = (total + size - 1) / size;
  for (int i = rank * per + (int)threadIdx.x; i < min(total, (rank + 1) * per); i += threads) {
    int head_at = i / hd, d = i % hd;
    float m_run = -INFINITY, l_run = 0.f, acc = 0.f;
    for (int base = 0; base < chunks; base += 16) {  // (sixteen chunks' values are asked for before the first is merged)
      float o[16], m[16], l[16];
#pragma unroll
      for (int x = 0; x < 16; ++x) {
        int c = base + x;
        if (c >= chunks) continue;
        int place = c / size;
        unsigned at = local + 4u * (unsigned)((place * heads_per_block + head_at) * (hd + 2)), far;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(far) : "r"(at), "r"(c - place * size));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(o[x]) : "r"(far + 4u * (unsigned)d));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(m[x]) : "r"(far + 4u * (unsigned)hd));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(l[x]) : "r"(far + 4u * (unsigned)hd + 4u));
      }
#pragma unroll
      for (int x = 0; x < 16; ++x) {
        if (base + x >= chunks) continue;
        float keep, take;
        merge(m_run, l_run, m[x], l[x], keep, take);
        acc = merge_output(acc, keep, o[x], take);
      }
    }
    out[((size_t)t * heads + g * group + head0) * hd + i] = told ? acc * (1.0f / l_run) : __int_as_float(0x7fffffff);
  }
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}

// Refuses (DLLM_UNSUPPORTED_SIZE) what does not fit and what the serial form (attention_block_kernel, the same bits) is faster
// at; the caller then takes that. `reach`: the most keys a token may see.
// A chunk costs more here than there, and there is a cluster barrier to pay, so it has to be worth it: enough chunks in a row
// that walking them one after another takes longer, and few enough (token, kv head) pairs that the device has room beside
// them. Microseconds here against there, 9 query and 3 kv heads of 64: one token of 30 keys 7.9 and 5.4, of 100 8.6 and 8.7,
// of 500 9.1 and 26.5, of 2,000 20.6 and 101; 2,000 keys and 32 tokens 58 and 103, 64 tokens 133 and 119, 128 tokens 243 and
// 138. Rows of 256 values, 4 query and 2 kv heads: 500 keys and 8 tokens 56 and 70, 16 tokens 84 and 70.
int launch_chunks(float* out, const float* q, const KvLayout& cache, const int* tok_seq, const int* tok_pos, const int* slots,
                  int tokens, int heads, float scale, int window, long long reach, int* status, cudaStream_t stream) {
  int group = heads / cache.kv_heads, hd = cache.head_dim, ld = hd + 4;
  // (a window of w keys may begin anywhere in its first chunk)
  long long chunks = (reach + 63) / 64;
  if (window > 0 && window < reach) chunks = ((long long)window + 126) / 64;
  if (tokens > 65535 || status == nullptr) return DLLM_UNSUPPORTED_SIZE;
  int heads_per_block = group < CHUNK_WARPS ? group : CHUNK_WARPS;
  int parts = (group + heads_per_block - 1) / heads_per_block;
  long long rows = (long long)cache.kv_heads * parts;
  if (rows > 65535) return DLLM_UNSUPPORTED_SIZE;
  // (two or three chunks: only where the serial form has many heads a block, or short rows and little else to do)
  long long values = rows * tokens * hd;
  bool few = chunks >= 2 && values <= 4096 && (group > 8 || hd <= 24);
  if (!(chunks >= 4 || few) || values > (hd <= 128 ? 8192 : 4096)) return DLLM_UNSUPPORTED_SIZE;
  // As many blocks a cluster as there are chunks, up to 8, while three a multiprocessor hold them all.
  int size = 1;
  while (size < 8 && size < chunks && rows * tokens * size * 2 <= 3 * 148) size *= 2;
  // As many chunks a round as give a block at least eight warps' work, within what shared memory holds beside the results.
  int room = (int)((chunks + size - 1) / size), per_round = 1;
  auto bytes = [&](int n) {
    return ((size_t)n * 128 * ld + (size_t)heads_per_block * hd + (size_t)room * heads_per_block * (hd + 2)) * sizeof(float);
  };
  if (bytes(1) > 200 * 1024 || room > 256) return DLLM_UNSUPPORTED_SIZE;
  while ((per_round + 1) * heads_per_block <= 8 && per_round < room && bytes(per_round + 1) <= 110 * 1024) ++per_round;
  // (more than one and a half rounds of blocks: 8 query heads of 128 to each of 8 kv heads, 8 tokens of 8,000: 597 and 500)
  long long resident = 148ll * (227 * 1024 / ((long long)bytes(per_round) + 2048));
  if (2 * rows * tokens * size > 3 * resident) return DLLM_UNSUPPORTED_SIZE;
  auto kernel = hd == 64 ? attention_chunks_kernel<64> : (hd == 128 ? attention_chunks_kernel<128> : attention_chunks_kernel<0>);
  static std::atomic<unsigned long long> allowed[3];
  if (!dllm_allow_shared((const void*)kernel, 200 * 1024, allowed[hd == 64 ? 0 : (hd == 128 ? 1 : 2)])) return DLLM_LAUNCH_FAILED;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(size, (unsigned)rows, tokens);
  config.blockDim = dim3(32 * heads_per_block * per_round);
  config.dynamicSmemBytes = bytes(per_round);
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = size;
  attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = dllm_pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&config, kernel, out, q, cache, tok_seq, tok_pos, slots, heads, scale, window,
                            heads_per_block, per_round, room, status) == cudaSuccess
             ? DLLM_OK
             : DLLM_LAUNCH_FAILED;
}
}  // namespace

DLLM_EXPORT int dllm_attention_general(void* out, const void* q, void* cache_base, const int* page_table,
                                       int max_pages, int page_size, int heads, int kv_heads, int head_dim,
                                       const int* tok_seq, const int* tok_pos, const int* slots, int tokens,
                                       float scale, int window, int dtype, cudaStream_t stream) {
  if (tokens <= 0) return DLLM_OK;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads) return DLLM_BAD_ARGUMENT;
  if (head_dim <= 0 || head_dim > MAX_HEAD_DIM || (head_dim & 7)) return DLLM_UNSUPPORTED_SIZE;
  KvLayout cache{cache_base, page_table, max_pages, page_size, kv_heads, head_dim};
  long long items = (long long)tokens * heads;
  unsigned blocks = (unsigned)((items + WARPS - 1) / WARPS);
  if (dtype == DLLM_F32)
    attention_warp_kernel<float><<<blocks, WARPS * 32, 0, stream>>>((float*)out, (const float*)q, cache, tok_seq,
                                                                    tok_pos, slots, tokens, heads, scale, window);
  else if (dtype == DLLM_BF16)
    attention_warp_kernel<__nv_bfloat16><<<blocks, WARPS * 32, 0, stream>>>(
        (__nv_bfloat16*)out, (const __nv_bfloat16*)q, cache, tok_seq, tok_pos, slots, tokens, heads, scale, window);
  else
    return DLLM_BAD_ARGUMENT;
  return dllm_launch_status();
}

// The same attention with the same arguments, blockwise; the same bits. `max_new`: the most new tokens a sequence brings
// in this step: with one each (decoding) a block serves one token's heads, else runs of tokens. `max_context`: the most
// keys any token of the step may see; one that sees more gets no number (NaN) and `status`, a word that the device can write,
// is set to 50. tile_seq / tile_first / cu_seqlens: for each of `tiles` stretches of up to 64 new tokens its sequence and its
// first token among that sequence's, and where the sequences' new tokens begin (may be absent, tiles = 0). Pages of 64
// positions, at most 65,535 kv heads.
// float32 takes the kernels made for it: single tokens their chunks side by side, prompts with heads of 64 and 128 in
// 16-byte aligned rows the tiles of queries.
DLLM_EXPORT int dllm_attention_blocks(void* out, const void* q, void* cache_base, const int* page_table,
                                      int max_pages, int page_size, int heads, int kv_heads, int head_dim,
                                      const int* tok_seq, const int* tok_pos, const int* slots, int tokens,
                                      int max_new, int max_context, const int* tile_seq, const int* tile_first,
                                      const int* cu_seqlens, int tiles, float scale, int window, int dtype, int* status,
                                      cudaStream_t stream) {
  if (tokens <= 0) return DLLM_OK;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads) return DLLM_BAD_ARGUMENT;
  if (head_dim <= 0 || head_dim > MAX_HEAD_DIM || (head_dim & 7) || page_size != 64 || kv_heads > 65535)
    return DLLM_UNSUPPORTED_SIZE;
  KvLayout cache{cache_base, page_table, max_pages, page_size, kv_heads, head_dim};
  bool runs = max_new > 1;
  int chunks = (head_dim + 31) / 32;
#define DLLM_GO(T, R, CHUNKS) \
  return launch_blocks<T, R, CHUNKS>(out, q, cache, tok_seq, tok_pos, slots, tokens, heads, scale, window, stream)
#define DLLM_BY_WIDTH(T, R)                   \
  if (chunks <= 1) DLLM_GO(T, R, 1);          \
  else if (chunks == 2) DLLM_GO(T, R, 2);     \
  else if (chunks <= 4) DLLM_GO(T, R, 4);     \
  else DLLM_GO(T, R, 8)
  if (dtype == DLLM_F32) {
    const float* rows = (const float*)q;
    float* to = (float*)out;
    bool tiled = (head_dim == 64 || head_dim == 128) && (((uintptr_t)q | (uintptr_t)out) & 15) == 0;
    if (!runs) {
      int done = launch_chunks(to, rows, cache, tok_seq, tok_pos, slots, tokens, heads, scale, window,
                               max_context > 0 ? max_context : (long long)max_pages * page_size, status, stream);
      if (done != DLLM_UNSUPPORTED_SIZE) return done;
    } else if (tiled && tiles > 0) {
      // A tile is one query head's, the serial form's block all heads' of a kv head: with many sequences of a token or two
      // and several heads a kv head, that is less work once tiles fill the device. 200 tokens of 300 keys and one prompt of
      // two, us here and there: 32 query and 8 kv heads of 128 702 and 570, 40 and 2 of 64 375 and 246, 9 and 3 of 64 96 and
      // 485; 32 tokens of 500 and a prompt of 100: 196 and 875, 108 and 386, 48 and 749.
      bool crowd = heads / kv_heads >= 4 && tokens < 4ll * tiles && (long long)tiles * heads * (head_dim / 64) >= 5000;
      if (!crowd)
        return (head_dim == 64 ? launch_tiles<64> : launch_tiles<128>)(to, rows, cache, tok_pos, slots, tile_seq,
                                                                       tile_first, cu_seqlens, tiles, heads, scale, window,
                                                                       stream);
    }
    if (runs) { DLLM_BY_WIDTH(float, 4); }
    DLLM_BY_WIDTH(float, 1);
  }
  if (dtype == DLLM_BF16) {
    if (runs) { DLLM_BY_WIDTH(__nv_bfloat16, 4); }
    DLLM_BY_WIDTH(__nv_bfloat16, 1);
  }
#undef DLLM_BY_WIDTH
#undef DLLM_GO
  return DLLM_BAD_ARGUMENT;
}
