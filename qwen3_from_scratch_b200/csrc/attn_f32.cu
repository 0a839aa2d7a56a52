// Paged causal attention in float32 for head sizes 64 and 128: the 32-bit path's attention (scores, probabilities and
// sums in float32, on CUDA cores), for whole prompts, portions and single tokens.
//
// A query's result depends only on its own keys, not on how the batch was cut or on the kernel that computes it.  The keys
// are taken in chunks of 64 by their absolute position, and for each chunk that holds a key the query sees:
//   s_n = scale * (q . k_n)        the dot product by runs of 32 values: eight chains of 4, added by halves, and the runs one
//                                  after the other (as close to 64 bits as the shuffle tree of attn_ref.cu; with chains of
//                                  16 the results for 2 to 65 keys were 2 to 11 % further off than that kernel's)
//   m_c = max s_n                  no lower than the lowest finite number
//   p_n = exp(s_n - m_c),  l_c = sum p_n  (keys t, t + 16, t + 32, t + 48 first, then over t by halves)
//   o_c = sum p_n v_n              ascending n
// and the chunks are folded together in ascending order: m' = max(m, m_c), l' = l exp(m - m') + l_c exp(m_c - m'), o likewise.
// Long contexts keep their accuracy (sums of 64, then one term per chunk), and the chunks of a single token can be
// computed side by side:
//   attn_f32_kernel        a block takes up to 32 (token, head) rows of one kv head and walks over the chunks
//   attn_f32_chunk_kernel  a block takes the heads of one token and one chunk and leaves (m_c, l_c, o_c)
//   attn_f32_fold_kernel   folds them
// Sizes of the 0.6B model (16 heads over 8 of 128), cold caches: 4 single tokens at contexts of 400 to 900 23.6 us, one at
// 4,096 36 us, prompts of 203 and 310 tokens 76 us; the walk over the keys one by one that served here before (attn_ref.cu,
// a warp per token and head) took 1,435, 6,600 and 453 us: some 1.6 us per key of the longest context, whatever the batch.
//
// Reference formulas: as in attn_ref.cu (models/attn.py:402-499, kernels/triton/paged_attn.py:89-181).
#include <float.h>

#include "common.cuh"

namespace q3 {

constexpr int AF_THREADS = 128, AF_CHUNK = 64;
constexpr float AF_MASKED = -1.0f;  // in place of a probability: the query does not see the key
// The maximum of a chunk is at least this if the query sees a key of it: where all the scores that it sees have fallen to
// minus infinity their weights are 0, not exp(-inf + inf), and the chunks beside it keep their values.
constexpr float AF_LOWEST = -FLT_MAX;

__device__ __forceinline__ void af_copy16(uint32_t dst, const float* src, bool in) {
  const int n = in ? 16 : 0;  // zero bytes read: the destination is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ float4 af_lds(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float af_dot4(float4 a, float4 b) {  // a chain; __fmul_rn: never joined with an addition of its result
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, __fmul_rn(a.x, b.x))));
}

// RPT: rows per thread; the block has 8 RPT (token, head) rows of one kv head, row r = token r / G, head r % G of the group.
template <int D, int RPT>
struct AfShape {
  static constexpr int ROWS = 8 * RPT;
  static constexpr size_t SMEM = ((size_t)(ROWS + 2 * AF_CHUNK) * D + (size_t)ROWS * AF_CHUNK) * sizeof(float);
};

// Grid (token tiles, kv heads, requests).
// Bound by shared-memory reads and the FMA pipe together (a 4 x 4 piece of the scores per thread: 8 reads of 16 bytes for
// 64 FMA); K of the next chunk is fetched under P V, V under the scores.
template <int D, int RPT>
__global__ void __launch_bounds__(AF_THREADS, D == 128 ? 2 : 3)  // (what an SM's shared memory holds)
attn_f32_kernel(const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
                float* __restrict__ out, const int* __restrict__ q_start, const int* __restrict__ kv_len,
                const int* __restrict__ block_table, int table_stride, int page_size, int num_pages, int Hq, int Hkv,
                float scale, int window, int* status) {
  constexpr int ROWS = 8 * RPT, D4 = D / 4, DV = D / 64;  // DV: pieces of four output columns per thread
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(128) float af_smem[];
  float* q_s = af_smem;                  // [ROWS][D], piece c of a row at place c ^ (row & 7)
  float* k_s = q_s + ROWS * D;           // [64][D], the same
  float* v_s = k_s + AF_CHUNK * D;       // [64][D], as it is
  float* p_s = v_s + AF_CHUNK * D;       // [ROWS][64], as Q
  __shared__ unsigned long long key_ok;  // bit n: key n of the chunk has a page

  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;  // rows ty + 8 i, keys tx + 16 j
  const int b = blockIdx.z, hk = blockIdx.y, G = Hq / Hkv;
  const int t0 = q_start[b], q_len = q_start[b + 1] - t0, len = kv_len[b];
  const int tokens = ROWS / G, tok0 = blockIdx.x * tokens;
  if (tok0 >= q_len) return;
  const int live_rows = min(tokens, q_len - tok0) * G;
  const int first_pos = len - q_len + tok0, last_pos = first_pos + min(tokens, q_len - tok0) - 1;
  const int first_key = (window > 0 && first_pos - window + 1 > 0) ? first_pos - window + 1 : 0;
  int chunk = first_key / AF_CHUNK;
  const int chunk_end = last_pos / AF_CHUNK + 1;
  if (first_pos < 0 && tid == 0) atomicOr(status, Q3_STATUS_BAD_POSITION);

  for (int e = tid; e < ROWS * D4; e += AF_THREADS) {
    const int r = e / D4, c = e % D4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < live_rows) v = af_lds(q + ((size_t)(t0 + tok0 + r / G) * Hq + hk * G + r % G) * D + c * 4);
    *reinterpret_cast<float4*>(q_s + r * D + ((c ^ (r & 7)) * 4)) = v;
  }
  int pos[RPT], lo[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int r = ty + 8 * i;
    pos[i] = r < live_rows ? first_pos + r / G : -1;
    lo[i] = (window > 0 && pos[i] - window + 1 > 0) ? pos[i] - window + 1 : 0;
  }
  const bool busy = (tid >> 5) * 2 < live_rows;  // the warp's first row is in use (its rows: 2 w, 2 w + 1, then by 8)

  const uint32_t k_addr = (uint32_t)__cvta_generic_to_shared(k_s), v_addr = (uint32_t)__cvta_generic_to_shared(v_s);
  const int* table = block_table + (size_t)b * table_stride;
  // two threads per key: its page, then its row piece by piece
  const int my_key = tid >> 1;
  auto fetch = [&](uint32_t dst, const float* pages, int c, bool swizzle, bool note) {
    const int n = c * AF_CHUNK + my_key;
    int page = -1;
    if (n >= first_key && n <= last_pos) {
      page = table_page(table, n / page_size, table_stride, status);
      if (page < 0 || page >= num_pages) {
        if (note) atomicOr(status, Q3_STATUS_BAD_PAGE);
        page = -1;
      }
    }
    const float* src = pages + (page < 0 ? 0 : (((size_t)page * Hkv + hk) * page_size + n % page_size) * D);
#pragma unroll
    for (int i = 0; i < D4 / 2; ++i) {
      const int piece = 2 * i + (tid & 1);
      af_copy16(dst + (my_key * D + (swizzle ? piece ^ (my_key & 7) : piece) * 4) * 4, src + piece * 4, page >= 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    return page >= 0;
  };

  float m[RPT], l[RPT], o[RPT][4 * DV];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int d = 0; d < 4 * DV; ++d) o[i][d] = 0.f;
  }
  bool have = false;
  if (chunk < chunk_end) have = fetch(k_addr, k_pages, chunk, true, true);
  for (; chunk < chunk_end; ++chunk) {
    if (tid == 0) key_ok = 0ull;
    __syncthreads();  // V and P of the chunk before have been read
    if (!(tid & 1) && have) atomicOr(&key_ok, 1ull << my_key);
    fetch(v_addr, v_pages, chunk, false, false);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // K and key_ok (and Q)
    const unsigned long long ok = key_ok;
    float oc[RPT][4 * DV], mc[RPT], lc[RPT];
    if (busy) {
      float s[RPT][4];
#pragma unroll
      for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 1
      for (int run = 0; run < D / 32; ++run) {
        float whole[RPT][4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float two[RPT][4], other[RPT][4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int piece = run * 8 + half * 4 + c;
            float4 kv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) kv[j] = af_lds(k_s + (tx + 16 * j) * D + ((piece ^ (tx & 7)) * 4));
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
              const float4 a = af_lds(q_s + (ty + 8 * i) * D + ((piece ^ ty) * 4));
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float p = af_dot4(a, kv[j]);
                if (c == 0) two[i][j] = p;
                else if (c == 1) two[i][j] += p;
                else if (c == 2) other[i][j] = p;
                else other[i][j] += p;
              }
            }
          }
#pragma unroll
          for (int i = 0; i < RPT; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float sum16 = two[i][j] + other[i][j];
              if (half == 0) whole[i][j] = sum16;
              else s[i][j] += whole[i][j] + sum16;
            }
        }
      }
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        bool sees[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = tx + 16 * j, n = chunk * AF_CHUNK + key;
          sees[j] = n >= lo[i] && n <= pos[i] && ((ok >> key) & 1ull);
        }
        mc[i] = sees[0] || sees[1] || sees[2] || sees[3] ? AF_LOWEST : -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = __fmul_rn(s[i][j], scale);  // (not contracted with the subtraction below)
          if (sees[j]) mc[i] = fmaxf(mc[i], s[i][j]);
        }
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) mc[i] = fmaxf(mc[i], __shfl_xor_sync(0xffffffffu, mc[i], x));
        lc[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float p = sees[j] ? expf(s[i][j] - mc[i]) : AF_MASKED;
          if (sees[j]) lc[i] += p;
          p_s[(ty + 8 * i) * AF_CHUNK + (((tx >> 2) + 4 * j) ^ ty) * 4 + (tx & 3)] = p;
        }
#pragma unroll
        for (int x = 8; x > 0; x >>= 1) lc[i] += __shfl_xor_sync(0xffffffffu, lc[i], x);
      }
    }
    __syncthreads();  // K has been read
    have = false;
    if (chunk + 1 < chunk_end) have = fetch(k_addr, k_pages, chunk + 1, true, true);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // V
    if (!busy) continue;
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
      for (int d = 0; d < 4 * DV; ++d) oc[i][d] = 0.f;
#pragma unroll 1
    for (int n4 = 0; n4 < AF_CHUNK; n4 += 4) {
      float4 p4[RPT];
#pragma unroll
      for (int i = 0; i < RPT; ++i) p4[i] = af_lds(p_s + (ty + 8 * i) * AF_CHUNK + ((n4 >> 2) ^ ty) * 4);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        float4 v[DV];
#pragma unroll
        for (int c = 0; c < DV; ++c) v[c] = af_lds(v_s + (n4 + n) * D + (tx + 16 * c) * 4);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const float p = n == 0 ? p4[i].x : n == 1 ? p4[i].y : n == 2 ? p4[i].z : p4[i].w;
          if (!(p < 0.f)) {  // a key that the query does not see takes no part, whatever its value holds
#pragma unroll
            for (int c = 0; c < DV; ++c) {
              oc[i][4 * c] = fmaf(p, v[c].x, oc[i][4 * c]);
              oc[i][4 * c + 1] = fmaf(p, v[c].y, oc[i][4 * c + 1]);
              oc[i][4 * c + 2] = fmaf(p, v[c].z, oc[i][4 * c + 2]);
              oc[i][4 * c + 3] = fmaf(p, v[c].w, oc[i][4 * c + 3]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      if (!(mc[i] == -INFINITY && lc[i] == 0.f)) {  // else: no key of the chunk is seen
        const float mn = fmaxf(m[i], mc[i]), f = expf(m[i] - mn), g = expf(mc[i] - mn);
        l[i] = fmaf(l[i], f, lc[i] * g);
#pragma unroll
        for (int d = 0; d < 4 * DV; ++d) o[i][d] = fmaf(o[i][d], f, oc[i][d] * g);
        m[i] = mn;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int r = ty + 8 * i;
    if (r >= live_rows) continue;
    const float inv = l[i] == 0.f && m[i] == -INFINITY ? 0.f : 1.0f / l[i];  // 0: no key seen
    float* dst = out + ((size_t)(t0 + tok0 + r / G) * Hq + hk * G + r % G) * D;
#pragma unroll
    for (int c = 0; c < DV; ++c)
      *reinterpret_cast<float4*>(dst + (tx + 16 * c) * 4) =
          make_float4(o[i][4 * c] * inv, o[i][4 * c + 1] * inv, o[i][4 * c + 2] * inv, o[i][4 * c + 3] * inv);
  }
}

// Single tokens: grid (chunks that a query can see, kv heads, requests), the G heads of one kv head against one chunk; leaves o_c, m_c and l_c of
// each head.  The same additions in the same order as above, shared out so that all four warps work whatever G is: a
// thread per key (and every second head) for the scores, a half-warp per head for the softmax, a thread per output
// column for P V (4 requests at contexts of 400 to 900, 16 heads over 8 of 128: 14.5 us with the kernel above cut by chunks,
// one of whose warps had rows, 13.0 us here; batch 1 at 4,096: 69 and 36 us with the fold).
template <int D, int G>
__global__ void __launch_bounds__(AF_THREADS, D == 128 ? 3 : 6)
attn_f32_chunk_kernel(const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
                      float* __restrict__ partial, const int* __restrict__ q_start, const int* __restrict__ kv_len,
                      const int* __restrict__ block_table, int table_stride, int page_size, int num_pages, int Hq, int Hkv,
                      float scale, int window, int max_chunks, int* status) {
  constexpr int D4 = D / 4;
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(128) float af_smem[];
  float* k_s = af_smem;                  // [64][D], piece c of a row at place c ^ (row & 7)
  float* v_s = k_s + AF_CHUNK * D;       // [64][D], as it is
  __shared__ __align__(16) float q_s[G][D];
  __shared__ __align__(16) float p_s[8][AF_CHUNK];
  __shared__ unsigned long long key_ok;  // bit n: key n of the chunk has a page
  const int tid = threadIdx.x, b = blockIdx.z, hk = blockIdx.y;
  const int t = q_start[b], pos = kv_len[b] - 1;
  if (q_start[b + 1] == t) return;
  if (pos < 0 && tid == 0 && blockIdx.x == 0) atomicOr(status, Q3_STATUS_BAD_POSITION);
  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  const int chunk = lo / AF_CHUNK + blockIdx.x;
  if (chunk * AF_CHUNK > pos || chunk >= max_chunks) return;  // (the fold reports a context beyond the scratch)
  if (tid == 0) key_ok = 0ull;

  const int my_key = tid >> 1, n_mine = chunk * AF_CHUNK + my_key;  // two threads per key bring its rows
  int page = -1;
  if (n_mine >= lo && n_mine <= pos) {
    page = table_page(block_table + (size_t)b * table_stride, n_mine / page_size, table_stride, status);
    if (page < 0 || page >= num_pages) {
      atomicOr(status, Q3_STATUS_BAD_PAGE);
      page = -1;
    }
  }
  const size_t row = page < 0 ? 0 : (((size_t)page * Hkv + hk) * page_size + n_mine % page_size) * D;
  const uint32_t k_addr = (uint32_t)__cvta_generic_to_shared(k_s), v_addr = (uint32_t)__cvta_generic_to_shared(v_s);
#pragma unroll
  for (int i = 0; i < D4 / 2; ++i) {
    const int piece = 2 * i + (tid & 1);
    af_copy16(k_addr + (my_key * D + (piece ^ (my_key & 7)) * 4) * 4, k_pages + row + piece * 4, page >= 0);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
  for (int i = 0; i < D4 / 2; ++i) {
    const int piece = 2 * i + (tid & 1);
    af_copy16(v_addr + (my_key * D + piece * 4) * 4, v_pages + row + piece * 4, page >= 0);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int e = tid; e < G * D4; e += AF_THREADS)
    *reinterpret_cast<float4*>(&q_s[e / D4][(e % D4) * 4]) =
        af_lds(q + ((size_t)t * Hq + hk * G + e / D4) * D + (e % D4) * 4);
  __syncthreads();
  if (!(tid & 1) && page >= 0) atomicOr(&key_ok, 1ull << my_key);
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();  // K, Q, key_ok
  const unsigned long long ok = key_ok;
  {
    constexpr int RH = (G + 1) / 2;  // heads of a thread: tid / 64, + 2, ..
    const int key = tid & 63;
    float s[RH];
#pragma unroll
    for (int i = 0; i < RH; ++i) s[i] = 0.f;
#pragma unroll 2
    for (int run = 0; run < D / 32; ++run) {
      float whole[RH];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float two[RH], other[RH];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int piece = run * 8 + half * 4 + c;
          const float4 kv = af_lds(k_s + key * D + ((piece ^ (key & 7)) * 4));
#pragma unroll
          for (int i = 0; i < RH; ++i) {
            const float p = af_dot4(af_lds(&q_s[min((tid >> 6) + 2 * i, G - 1)][piece * 4]), kv);
            if (c == 0) two[i] = p;
            else if (c == 1) two[i] += p;
            else if (c == 2) other[i] = p;
            else other[i] += p;
          }
        }
#pragma unroll
        for (int i = 0; i < RH; ++i) {
          const float sum16 = two[i] + other[i];
          if (half == 0) whole[i] = sum16;
          else s[i] += whole[i] + sum16;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < RH; ++i)
      if ((tid >> 6) + 2 * i < G) p_s[(tid >> 6) + 2 * i][key] = __fmul_rn(s[i], scale);
  }
  __syncthreads();
  const int tx = tid & 15, head = tid >> 4;
  float* dst = partial + ((size_t)(b * Hq + hk * G) * max_chunks + chunk) * (D + 4);
  const size_t dst_pitch = (size_t)max_chunks * (D + 4);
  if ((tid >> 5) * 2 < G) {  // whole warps, two heads each
    float s[4], mc = -INFINITY, lc = 0.f;
    bool sees[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int key = tx + 16 * j, n = chunk * AF_CHUNK + key;
      s[j] = head < G ? p_s[head][key] : 0.f;
      sees[j] = n >= lo && n <= pos && ((ok >> key) & 1ull);
      if (sees[j]) mc = fmaxf(mc, fmaxf(s[j], AF_LOWEST));
    }
#pragma unroll
    for (int x = 8; x > 0; x >>= 1) mc = fmaxf(mc, __shfl_xor_sync(0xffffffffu, mc, x));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float p = sees[j] ? expf(s[j] - mc) : AF_MASKED;
      if (sees[j]) lc += p;
      if (head < G) p_s[head][tx + 16 * j] = p;
    }
#pragma unroll
    for (int x = 8; x > 0; x >>= 1) lc += __shfl_xor_sync(0xffffffffu, lc, x);
    if (tx == 0 && head < G) *reinterpret_cast<float4*>(dst + head * dst_pitch + D) = make_float4(mc, lc, 0.f, 0.f);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();  // P and V
  if (tid < D) {
    float oc[G];
#pragma unroll
    for (int h = 0; h < G; ++h) oc[h] = 0.f;
#pragma unroll 4
    for (int n4 = 0; n4 < AF_CHUNK; n4 += 4) {
      float v[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) v[n] = v_s[(n4 + n) * D + tid];
#pragma unroll
      for (int h = 0; h < G; ++h) {
        const float4 p4 = af_lds(&p_s[h][n4]);
        const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
        for (int n = 0; n < 4; ++n)
          if (!(p[n] < 0.f)) oc[h] = fmaf(p[n], v[n], oc[h]);
      }
    }
#pragma unroll
    for (int h = 0; h < G; ++h) dst[h * dst_pitch + tid] = oc[h];
  }
}

// One block per (request, head), a thread per output value.
template <int D>
__global__ void __launch_bounds__(D)
attn_f32_fold_kernel(const float* __restrict__ partial, float* __restrict__ out, const int* __restrict__ q_start,
                     const int* __restrict__ kv_len, int Hq, int window, int max_chunks, int* status) {
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.y, head = blockIdx.x, d = threadIdx.x;
  const int t = q_start[b], pos = kv_len[b] - 1;
  if (q_start[b + 1] == t) return;
  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  const float* src = partial + (size_t)(b * Hq + head) * max_chunks * (D + 4);
  float m = -INFINITY, l = 0.f, o = 0.f;
  const int end = min(pos / AF_CHUNK + 1, max_chunks);
  if (pos >= 0 && pos / AF_CHUNK >= max_chunks && d == 0) atomicOr(status, Q3_STATUS_BAD_POSITION);
  constexpr int AT_ONCE = 8;  // chunks whose values are asked for together: the fold itself is a chain
  if (pos >= 0) {
    for (int c0 = lo / AF_CHUNK; c0 < end; c0 += AT_ONCE) {
      float oc[AT_ONCE];
      float2 ml[AT_ONCE];
#pragma unroll
      for (int u = 0; u < AT_ONCE; ++u) {
        const float* p = src + (size_t)min(c0 + u, end - 1) * (D + 4);
        oc[u] = p[d];
        ml[u] = c0 + u < end ? *reinterpret_cast<const float2*>(p + D) : make_float2(-INFINITY, 0.f);
      }
#pragma unroll
      for (int u = 0; u < AT_ONCE; ++u) {
        if (ml[u].x == -INFINITY && ml[u].y == 0.f) continue;
        const float mn = fmaxf(m, ml[u].x), f = expf(m - mn), g = expf(ml[u].x - mn);
        l = fmaf(l, f, ml[u].y * g);
        o = fmaf(o, f, oc[u] * g);
        m = mn;
      }
    }
  }
  out[((size_t)t * Hq + head) * D + d] = l == 0.f && m == -INFINITY ? 0.f : o * (1.0f / l);
}

template <int D, int G>
static int attn_f32_chunks(const float* q, const float* k_pages, const float* v_pages, float* out, float* partial,
                           const int* q_start, const int* kv_len, const int* block_table, int table_stride, int page_size,
                           int num_pages, int num_seqs, int Hq, int Hkv, float scale, int window, int max_chunks, int* status,
                           cudaStream_t stream) {
  constexpr size_t smem = (size_t)2 * AF_CHUNK * D * sizeof(float);
  auto kernel = attn_f32_chunk_kernel<D, G>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  // a window's keys lie in no more chunks than this (64 requests at contexts of 300, a window of 17 on 16 heads over 8: 19.5 us
  // with a block for every chunk of the context bucket of 1,024)
  const int seen = window > 0 && window <= (max_chunks - 1) * AF_CHUNK ? min(max_chunks, (window + AF_CHUNK - 2) / AF_CHUNK + 1)
                                                                       : max_chunks;
  q3::launch(kernel, dim3(seen, Hkv, num_seqs), dim3(AF_THREADS), smem, stream, q, k_pages, v_pages, partial, q_start,
             kv_len, block_table, table_stride, page_size, num_pages, Hq, Hkv, scale, window, max_chunks, status);
  q3::launch(attn_f32_fold_kernel<D>, dim3(Hq, num_seqs), dim3(D), 0, stream, partial, out, q_start, kv_len, Hq, window,
             max_chunks, status);
  return launch_status();
}

template <int D, int RPT>
static int attn_f32_walk(const float* q, const float* k_pages, const float* v_pages, float* out, const int* q_start,
                         const int* kv_len, const int* block_table, int table_stride, int page_size, int num_pages,
                         int num_seqs, int max_q_len, int Hq, int Hkv, float scale, int window, int* status,
                         cudaStream_t stream) {
  constexpr size_t smem = AfShape<D, RPT>::SMEM;
  auto kernel = attn_f32_kernel<D, RPT>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int tokens = 8 * RPT / (Hq / Hkv);
  q3::launch(kernel, dim3((max_q_len + tokens - 1) / tokens, Hkv, num_seqs), dim3(AF_THREADS), smem, stream, q, k_pages,
             v_pages, out, q_start, kv_len, block_table, table_stride, page_size, num_pages, Hq, Hkv, scale, window, status);
  return launch_status();
}

template <int D>
static int attn_f32_go(const float* q, const float* k_pages, const float* v_pages, float* out, float* partial,
                       const int* q_start, const int* kv_len, const int* block_table, int table_stride, int page_size,
                       int num_pages, int num_seqs, int max_q_len, int Hq, int Hkv, float scale, int window, int max_chunks,
                       int* status, cudaStream_t stream) {
  const int G = Hq / Hkv;
  if (max_chunks > 0) {
#define Q3_AF_CHUNKS(G_)                                                                                                    \
  return attn_f32_chunks<D, G_>(q, k_pages, v_pages, out, partial, q_start, kv_len, block_table, table_stride, page_size,    \
                                num_pages, num_seqs, Hq, Hkv, scale, window, max_chunks, status, stream)
    if (G == 1) Q3_AF_CHUNKS(1);
    if (G == 2) Q3_AF_CHUNKS(2);
    if (G == 4) Q3_AF_CHUNKS(4);
    Q3_AF_CHUNKS(8);
#undef Q3_AF_CHUNKS
  }
#define Q3_AF_WALK(RPT)                                                                                                     \
  return attn_f32_walk<D, RPT>(q, k_pages, v_pages, out, q_start, kv_len, block_table, table_stride, page_size, num_pages,   \
                               num_seqs, max_q_len, Hq, Hkv, scale, window, status, stream)
  if (max_q_len * G <= 8) Q3_AF_WALK(1);
  // 16 rows per block where blocks of 32 would leave SMs without one (37 tokens over 1,000 keys: 143 against 184 us), else
  // 32 (prompts of 203 and 310 tokens: 76 us against 90 with 16 rows, and 111 with 64, whose one warp per scheduler waits
  // for every shared-memory read)
  if ((long long)((max_q_len + 32 / G - 1) / (32 / G)) * Hkv * num_seqs < sm_count()) Q3_AF_WALK(2);
  Q3_AF_WALK(4);
#undef Q3_AF_WALK
}

}  // namespace q3

// float32; q, out: [T, Hq, D] with D 64 or 128; k_pages / v_pages: [num_pages, Hkv, page_size, D]; Hq / Hkv 1, 2, 4 or 8.
// q_start: int32 [num_seqs + 1]; kv_len: int32 [num_seqs] keys after this step's write; block_table: int32 [num_seqs,
// table_stride].  max_chunks > 0: every request brings one token, none has more than 64 max_chunks keys, and partial holds
// num_seqs * Hq * max_chunks * (D + 4) floats; 0: requests of up to max_q_len tokens, partial not used.  The results are
// the same bits either way.  window <= 0: all earlier keys.
extern "C" int q3_attn_f32(const float* q, const float* k_pages, const float* v_pages, float* out, float* partial,
                           const int* q_start, const int* kv_len, const int* block_table, int table_stride, int page_size,
                           int num_pages, int num_seqs, int max_q_len, int Hq, int Hkv, int D, float scale, int window,
                           int max_chunks, int* status, cudaStream_t stream) {
  if (num_seqs <= 0 || max_q_len <= 0) return 0;
  if (Hkv <= 0 || Hq % Hkv || page_size <= 0 || table_stride <= 0 || max_chunks < 0 || (max_chunks > 0 && !partial))
    return Q3_ERR_SIZE;
  const int G = Hq / Hkv;
  if ((G != 1 && G != 2 && G != 4 && G != 8) || Hkv > 65535 || num_seqs > 65535) return Q3_ERR_SIZE;
  if ((uintptr_t)q % 16 || (uintptr_t)k_pages % 16 || (uintptr_t)v_pages % 16 || (uintptr_t)out % 16 || (uintptr_t)partial % 16)
    return Q3_ERR_ALIGN;
#define Q3_AF_GO(D_)                                                                                                        \
  return q3::attn_f32_go<D_>(q, k_pages, v_pages, out, partial, q_start, kv_len, block_table, table_stride, page_size,      \
                             num_pages, num_seqs, max_q_len, Hq, Hkv, scale, window, max_chunks, status, stream)
  if (D == 64) Q3_AF_GO(64);
  if (D == 128) Q3_AF_GO(128);
#undef Q3_AF_GO
  return Q3_ERR_SIZE;
}
