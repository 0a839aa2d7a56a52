// Latent attention for prompt portions on the fifth-generation tensor cores (tcgen05), bfloat16, with the keys and values of
// every head formed from the latents first (see latent_attn.cu for the arithmetic).
//
// The cache holds one latent c and one rotated part r per token.  A query can be taken into the latent's space (the absorbed
// form of latent_attn_mma.cu: scores over rank + rot values, output rank values wide) or each head's key W_uk c and value
// W_uv c can be formed.  With 16 heads of 128 + 64 over a latent of 512 the absorbed form costs 1,088 multiply-adds per
// query, head and key, the formed one 320, and forming 131,072 per head and key, which a portion pays once for all its
// tokens.  At 2,048 tokens a layer's attention took 525 us absorbed (on mma.sync, with 25 us for the products around it); now
// 32 us of attention (670 TFLOP/s), 11 us for forming keys and values and 3 us for the gather.
//   latent_gather_kernel     brings a request's latents and rotated parts out of their pages into rows of their own
//   (a library product)      keys and values of all heads, [rows, H 128 | H 128]
//   latent_attn_tc_kernel    causal attention of one head's 128 query rows over the formed keys: scores over 128 + 64
//                            values (three swizzle atoms, the third from the shared rotated part), output 128 wide,
//                            multiplied by the head's gate in the epilogue
// The attention kernel is built like attn_tc.cu's: a loader thread each for K and V (TMA boxes of 128 rows x 64 values), an
// issuing thread, 512 softmax threads (four per query row), K, V and S double-buffered, P in tensor memory over its own S,
// a reference maximum that moves only when it must.  One block per SM (213 KB of shared memory, all 512 TMEM columns).  All
// mbarrier waits are bounded (tc_common.cuh).
#include "tc_common.cuh"
#include "tile_phase.h"

namespace q3 {

constexpr int LT_BM = 128, LT_BN = 128;        // query rows per block, keys per tile
constexpr int LT_D = 128, LT_ROT = 64;         // plain part of a key (and a value), rotated part
constexpr int LT_PARTS = 4, LT_PART = LT_BN / LT_PARTS;
constexpr int LT_SOFTMAX = LT_PARTS * LT_BM;
constexpr int LT_ISSUE_WARP = LT_SOFTMAX / 32, LT_LOAD_WARP = LT_ISSUE_WARP + 1;
constexpr int LT_THREADS = LT_SOFTMAX + 96;
constexpr int LT_ATOM = LT_BM * 128;           // bytes of a 128-row atom of 64 values
constexpr int LT_QK_ATOMS = (LT_D + LT_ROT) / 64;
constexpr int LT_Q_BYTES = LT_QK_ATOMS * LT_ATOM, LT_K_BYTES = LT_QK_ATOMS * LT_ATOM, LT_V_BYTES = (LT_D / 64) * LT_ATOM;
constexpr int LT_BAR_BYTES = 128, LT_XCHG_BYTES = 2 * LT_PARTS * LT_BM * 4;
constexpr size_t LT_SMEM = (size_t)LT_Q_BYTES + 2 * LT_K_BYTES + 2 * LT_V_BYTES + LT_BAR_BYTES + LT_XCHG_BYTES;
constexpr uint32_t LT_TMEM_COLS = 512;         // S: two buffers of 128 columns at 0 and 128, O: 128 columns at 256

// byte offset of value (row, col) in a [rows x 64] bfloat16 tile with the 128-byte swizzle
__device__ __forceinline__ uint32_t lt_offset(int row, int col) {
  return (uint32_t)row * 128u + ((((uint32_t)col >> 3) ^ ((uint32_t)row & 7u)) << 4) + (((uint32_t)col & 7u) << 1);
}

// Row b * pitch + n of the dense arrays: key n of request b (n < kv_len; later rows are left as they are, nobody reads what
// is made of them).  A thread per 16 bytes; a page that the table does not have leaves zeros and a bit in the status word.
__global__ void __launch_bounds__(256)
latent_gather_kernel(const __nv_bfloat16* __restrict__ c_pages, const __nv_bfloat16* __restrict__ r_pages,
                     const int* __restrict__ kv_len, const int* __restrict__ table, int stride, int page_size, int num_pages,
                     int rank, int rot, int pitch, __nv_bfloat16* __restrict__ c_rows, __nv_bfloat16* __restrict__ r_rows,
                     int* status) {
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.y, chunks = (rank + rot) / 8;
  const int idx = blockIdx.x * 256 + threadIdx.x, n = idx / chunks, c = (idx % chunks) * 8;
  if (n >= min(kv_len[b], pitch)) return;
  const int page = table_page(table + (size_t)b * stride, n / page_size, stride, status);
  uint4 v = make_uint4(0, 0, 0, 0);
  const size_t row = (size_t)b * pitch + n;
  if (page < 0 || page >= num_pages) {
    if (c == 0) atomicOr(status, Q3_STATUS_BAD_PAGE);
  } else {
    const size_t slot = (size_t)page * page_size + n % page_size;
    v = *reinterpret_cast<const uint4*>(c < rank ? c_pages + slot * rank + c : r_pages + slot * rot + (c - rank));
  }
  *reinterpret_cast<uint4*>(c < rank ? c_rows + row * rank + c : r_rows + row * rot + (c - rank)) = v;
}

// map_kv: [rows, 2 H 128], the heads' keys, then their values; map_r: [rows, 64]; both in boxes of 64 values x 128 rows.
// q_plain [T, H, 128], q_rot [T, H, 64], out [T, H, 128]; gate: float32 [T, H] or null; sink: float32 [H] or null.
__global__ void __launch_bounds__(LT_THREADS, 1)
latent_attn_tc_kernel(const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_r,
                      const __nv_bfloat16* __restrict__ q_plain, const __nv_bfloat16* __restrict__ q_rot,
                      __nv_bfloat16* __restrict__ out, const int* __restrict__ q_start, const int* __restrict__ kv_len,
                      int pitch, int H, float scale_log2, const float* __restrict__ gate, const float* __restrict__ sink,
                      int* status) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* q_s = smem_raw;
  unsigned char* k_s = q_s + LT_Q_BYTES;       // two stages
  unsigned char* v_s = k_s + 2 * LT_K_BYTES;   // two stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + 2 * LT_V_BYTES);
  uint64_t* k_full = bars + 0;   // [2]
  uint64_t* k_empty = bars + 2;  // [2]
  uint64_t* v_full = bars + 4;   // [2]
  uint64_t* v_empty = bars + 6;  // [2]
  uint64_t* s_ready = bars + 8;  // [2]
  uint64_t* p_ready = bars + 10;  // [2]
  uint64_t* pv_done = bars + 12;  // [2]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bars + 14);
  int* abort_word = reinterpret_cast<int*>(bars + 15);
  float* row_xchg = reinterpret_cast<float*>(v_s + 2 * LT_V_BYTES + LT_BAR_BYTES);  // [2][parts][128] row maxima, then sums
#define abort_flag (*abort_word)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x, b = blockIdx.z;
  const int qs = q_start[b];
  const int q_len = q_start[b + 1] - qs;
  const int len = kv_len[b];
  // the heads are x, so that the heaviest query tiles (late queries, many keys) of all heads start first
  const int qt = (int)gridDim.y - 1 - (int)blockIdx.y;
  const int row0 = qt * LT_BM;
  if (row0 >= q_len) return;  // before any barrier or allocation: the whole block leaves
  const int past = len - q_len;
  if (past < 0 || len > pitch) {  // more new tokens than the request holds, or more keys than there are rows
    if (threadIdx.x == 0) atomicOr(status, Q3_STATUS_BAD_POSITION);
    return;
  }
  const int pos_first = past + row0, pos_last = past + min(q_len, row0 + LT_BM) - 1;
  const int n_tiles = pos_last / LT_BN + 1;

  if (warp == LT_LOAD_WARP && lane == 0) {
    tma_prefetch_map(&map_kv);
    tma_prefetch_map(&map_r);
  }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    if (s_addr(smem_raw) & 1023u) {  // the swizzled tiles need this; never seen, but a wrong answer must not be silent
      abort_flag = 1;
      atomicOr(status, Q3_STATUS_TIMEOUT);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(k_full + i, 1);
      mbar_init(k_empty + i, 1);
      mbar_init(v_full + i, 1);
      mbar_init(v_empty + i, 1);
      mbar_init(s_ready + i, 1);
      mbar_init(p_ready + i, LT_SOFTMAX / 32);
      mbar_init(pv_done + i, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();  // queries, keys and values come from the kernels before this one
  pdl_launch_dependents();
  __syncthreads();  // the barriers exist; from here the loader warps go their own way until the end
  // Tensor memory is taken only after the wait: a block that holds TMEM while it waits for the
  // kernel before it could keep that kernel's own blocks from ever getting theirs.
  if (warp == LT_ISSUE_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_addr(tmem_holder)),
                 "r"(LT_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // the query tile, written in the swizzled K-major layout by the softmax threads
  if (warp < LT_ISSUE_WARP) {
    constexpr int CH = (LT_D + LT_ROT) / 8, PER_THREAD = LT_BM * CH / LT_SOFTMAX;  // 24 chunks of a row, 6 per thread
    uint4 v[PER_THREAD];
#pragma unroll
    for (int i = 0; i < PER_THREAD; ++i) {
      const int idx = threadIdx.x + i * LT_SOFTMAX, r = idx / CH, c = idx % CH;
      const size_t row = (size_t)(qs + row0 + r) * H + h;
      v[i] = row0 + r >= q_len ? make_uint4(0, 0, 0, 0)
                               : *reinterpret_cast<const uint4*>(c < LT_D / 8 ? q_plain + row * LT_D + c * 8
                                                                              : q_rot + row * LT_ROT + (c * 8 - LT_D));
    }
#pragma unroll
    for (int i = 0; i < PER_THREAD; ++i) {
      const int idx = threadIdx.x + i * LT_SOFTMAX, r = idx / CH, c = idx % CH;
      *reinterpret_cast<uint4*>(q_s + (c / 8) * LT_ATOM + lt_offset(r, (c % 8) * 8)) = v[i];
    }
    fence_async_proxy();
  }
  uint32_t tmem_s = 0, tmem_o = 0;
  if (warp < LT_LOAD_WARP) {
    // the query tile and the tensor memory address, among the softmax and issue warps only
    tcgen05_fence_before();
    asm volatile("bar.sync 2, %0;" ::"n"(LT_SOFTMAX + 32) : "memory");
    tcgen05_fence_after();
    tmem_s = *tmem_holder;           // S of tile j lives at column (j & 1) * 128
    tmem_o = tmem_s + 2 * LT_BN;
  }

  if (warp >= LT_LOAD_WARP) {
    // ------------------------------------------------------------------ loaders: one thread for K, one for V
    // Boxes past the request's keys bring rows of another request, rows never written or zeros: their scores are masked
    // and their values zeroed below.  The row is any number; a box's first value is a multiple of 64.
    if (lane == 0) {
      const bool is_v = warp != LT_LOAD_WARP;
      uint64_t* full = is_v ? v_full : k_full;
      uint64_t* empty = is_v ? v_empty : k_empty;
      bool ok = true;
      uint32_t issued = 0;  // tiles asked for
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int st = tile_slot(j), y = b * pitch + j * LT_BN;
        if (j > 1) ok = mbar_wait(empty + st, ((uint32_t)(j >> 1) - 1) & 1, &abort_flag);
        if (!ok) break;
        if (is_v) {
          mbar_expect_tx(full + st, LT_V_BYTES);
          for (int a = 0; a < LT_D / 64; ++a)
            tma_load_2d(v_s + st * LT_V_BYTES + a * LT_ATOM, &map_kv, full + st, (H + h) * LT_D + a * 64, y);
        } else if (j != tc_drop_copy) {  // left out only in the tests of the give-up path (see tc_common.cuh)
          mbar_expect_tx(full + st, LT_K_BYTES);
          for (int a = 0; a < LT_D / 64; ++a)
            tma_load_2d(k_s + st * LT_K_BYTES + a * LT_ATOM, &map_kv, full + st, h * LT_D + a * 64, y);
          tma_load_2d(k_s + st * LT_K_BYTES + (LT_D / 64) * LT_ATOM, &map_r, full + st, 0, y);
        }
        ++issued;
      }
      if (!ok) {
        abort_flag = 1;
        atomicOr(status, Q3_STATUS_TIMEOUT);
      }
      finish_copies(full, issued, 2, is_v ? -1 : tc_drop_copy, status);
    }
  } else if (warp == LT_ISSUE_WARP) {
    // ------------------------------------------------------------------ tensor-core issue
    if (lane == 0) {
      constexpr uint32_t idesc_s = umma_idesc(LT_BN, 0);  // 128 x 128, K and Q both K-major
      constexpr uint32_t idesc_o = umma_idesc(LT_D, 1);      // 128 x D, V MN-major
      // S of tile j + 1 is issued before the wait for tile j's probabilities, so it runs on the
      // tensor cores while the softmax threads work on tile j.
      // Descriptors are built once; inside the loops only constants are added to their address
      // field (in units of 16 bytes), so that the issuing thread is not held up by address arithmetic.
      const uint64_t q_desc = umma_desc_sw128(q_s);
      const uint64_t k_desc0 = umma_desc_sw128(k_s), k_desc1 = umma_desc_sw128(k_s + LT_K_BYTES);
      const uint64_t v_desc0 = umma_desc_sw128_mn(v_s, LT_ATOM), v_desc1 = umma_desc_sw128_mn(v_s + LT_V_BYTES, LT_ATOM);
      auto issue_s = [&](int j) -> bool {
        const int st = tile_slot(j);
        if (!mbar_wait(k_full + st, tile_parity(j), &abort_flag)) return false;
        tcgen05_fence_after();
        const uint64_t kd = st ? k_desc1 : k_desc0;
        const uint32_t acc = tmem_s + st * LT_BN;
#pragma unroll
        for (int t = 0; t < (LT_D + LT_ROT) / 16; ++t) {
          constexpr int ATOM16 = LT_ATOM >> 4;  // one 64-wide atom of 128 rows, in 16-byte units
          umma_f16(acc, q_desc + (uint64_t)((t / 4) * ATOM16 + 2 * (t % 4)), kd + (uint64_t)((t / 4) * ATOM16 + 2 * (t % 4)),
                   idesc_s, t != 0);
        }
        umma_commit(s_ready + st);
        umma_commit(k_empty + st);
        return true;
      };
      bool ok = issue_s(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int st = tile_slot(j);
        if (j + 1 < n_tiles && !issue_s(j + 1)) { ok = false; break; }
        if (!mbar_wait(p_ready + st, tile_parity(j), &abort_flag)) { ok = false; break; }
        if (!mbar_wait(v_full + st, tile_parity(j), &abort_flag)) { ok = false; break; }
        tcgen05_fence_after();
        const uint64_t vd = st ? v_desc1 : v_desc0;
        const uint32_t p_cols = tmem_s + st * LT_BN;
#pragma unroll
        for (int t = 0; t < LT_BN / 16; ++t)  // 16 keys: 8 packed columns of P, 16 rows (2048 bytes) of V
          umma_f16_ts(tmem_o, p_cols + 8 * t, vd + (uint64_t)(t * (2048 >> 4)), idesc_o, (j | t) != 0);
        umma_commit(v_empty + st);
        umma_commit(pv_done + st);  // last: the last tile's is waited for, so no arrival is still to come when the block ends
      }
      if (!ok) {
        abort_flag = 1;
        atomicOr(status, Q3_STATUS_TIMEOUT);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax, four threads per row
    // warps 4 p .. 4 p + 3 take keys 32 p .. 32 p + 31 of every tile; warp w sees TMEM lanes
    // (w % 4) * 32 .., i.e. row (w % 4) * 32 + lane.
    const int part = warp >> 2;
    const int rr = (warp & 3) * 32 + lane;
    const int R = row0 + rr;
    const bool valid_row = R < q_len;
    const int my_pos = valid_row ? past + R : pos_last;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const int soft_tid = threadIdx.x;  // 0 .. 511
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    // Every softmax thread runs every iteration and meets the others at the named barrier even
    // after a wait has run out (the barrier itself cannot time out); `ok` only switches the work off.
    for (int j = 0; j < n_tiles; ++j) {
      const int st = tile_slot(j);
      float* xchg = row_xchg + (j & 1) * (LT_PARTS * LT_BM);
      ok = ok && mbar_wait(s_ready + st, tile_parity(j), &abort_flag);
      tcgen05_fence_after();
      uint32_t sv[32];
      tmem_ld_32(tmem_s + st * LT_BN + part * LT_PART + lane_base, sv);
      tmem_wait_ld();
      const int tile_n = j * LT_BN;  // the tile's first key
      const int base_n = tile_n + part * LT_PART;
      float mx = -INFINITY;
      if (tile_n + LT_BN - 1 > pos_first) {  // the diagonal: keys beyond this row's position are hidden
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const bool seen = base_n + c <= my_pos;
          const float v = seen ? __uint_as_float(sv[c]) : -INFINITY;
          sv[c] = __float_as_uint(v);
          mx = fmaxf(mx, v);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 32; ++c) mx = fmaxf(mx, __uint_as_float(sv[c]));
      }
      // the threads of a row agree on its maximum
      xchg[part * LT_BM + rr] = mx;
      asm volatile("bar.sync 1, %0;" ::"n"(LT_SOFTMAX) : "memory");
#pragma unroll
      for (int o = 0; o < LT_PARTS; ++o) mx = fmaxf(mx, xchg[o * LT_BM + rr]);
      mx *= scale_log2;
      // the reference maximum moves only when it must: probabilities up to 2^8 are harmless
      float alpha = 1.f;
      if (mx > m_ref + 8.f) {
        alpha = m_ref == -INFINITY ? 0.f : exp2f(m_ref - mx);
        m_ref = mx;
      }
      const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        // O belongs to the tensor cores until the previous tile's P V has finished
        ok = ok && mbar_wait(pv_done + tile_slot(j - 1), tile_parity(j - 1), &abort_flag);
        tcgen05_fence_after();
        // the row's threads rescale 32 output columns each
        uint32_t ov[32];
        tmem_ld_32(tmem_o + lane_base + part * 32, ov);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) ov[c] = __float_as_uint(__uint_as_float(ov[c]) * alpha);
        tmem_st_32(tmem_o + lane_base + part * 32, ov);
        tmem_wait_st();
      }
      l *= alpha;
      float sum = 0.f;
      // P over the tile's own S: key k of the row goes to the half of column k / 2.  Every thread of
      // the row has its S in registers since the barrier above, so the columns may be overwritten.
      uint32_t pk[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float p0 = ex2_approx(fmaf(__uint_as_float(sv[2 * e]), scale_log2, -m_use));
        const float p1 = ex2_approx(fmaf(__uint_as_float(sv[2 * e + 1]), scale_log2, -m_use));
        sum += p0 + p1;
        pk[e] = pack2(__float_as_uint(p0), __float_as_uint(p1));
      }
      tmem_st_16(tmem_s + st * LT_BN + part * (LT_PART / 2) + lane_base, pk);
      tmem_wait_st();
      l += sum;
      // keys past the end of the sequence in the last tile: their V rows are not this request's; zero them
      if (tile_n + LT_BN > len) {
        ok = ok && mbar_wait(v_full + st, tile_parity(j), &abort_flag);
        const int first_bad = len - tile_n;
        for (int e = soft_tid; e < (LT_BN - first_bad) * (LT_D / 8); e += LT_SOFTMAX) {
          const int key = first_bad + e / (LT_D / 8), c = e % (LT_D / 8);
          *reinterpret_cast<uint4*>(v_s + st * LT_V_BYTES + (c / 8) * LT_ATOM + lt_offset(key, (c % 8) * 8)) =
              make_uint4(0, 0, 0, 0);
        }
      }
      // every thread has finished its own writes (the zeroed V rows go through the async proxy); one
      // arrival per warp then tells the issuing thread
      fence_async_proxy();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready + st);
    }
    if (!ok && lane == 0) {
      abort_flag = 1;
      atomicOr(status, Q3_STATUS_TIMEOUT);
    }
    // the last P V, then O / l with l summed over the row's threads; each writes 32 of the columns
    const bool done = ok && mbar_wait(pv_done + tile_slot(n_tiles - 1), tile_parity(n_tiles - 1), &abort_flag);
    float* xchg = row_xchg + (n_tiles & 1) * (LT_PARTS * LT_BM);
    xchg[part * LT_BM + rr] = l;
    asm volatile("bar.sync 1, %0;" ::"n"(LT_SOFTMAX) : "memory");
    constexpr int OUT_CH = LT_D / 8;
    if (done) {
      tcgen05_fence_after();
      float total = 0.f;
#pragma unroll
      for (int o = 0; o < LT_PARTS; ++o) total += xchg[o * LT_BM + rr];
      if (sink) total += exp2f(fmaf(sink[h], 1.4426950408889634f, -m_ref));
      float inv = total > 0.f ? 1.0f / total : 0.f;
      if (gate && valid_row) inv *= gate[(size_t)(qs + R) * H + h];
      // through shared memory (where the query tile was: every product that read it has finished), so that the tile leaves
      // in whole rows; chunk c of row r sits at place c ^ (r % 16), which spreads a warp's rows over the banks
      uint32_t ov[32];
      tmem_ld_32(tmem_o + lane_base + part * 32, ov);
      tmem_wait_ld();
#pragma unroll
      for (int v4 = 0; v4 < 4; ++v4) {
        uint32_t pk[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          pk[i] = pack2(__float_as_uint(__uint_as_float(ov[8 * v4 + 2 * i]) * inv),
                        __float_as_uint(__uint_as_float(ov[8 * v4 + 2 * i + 1]) * inv));
        const int c = part * 4 + v4;
        *reinterpret_cast<uint4*>(q_s + rr * (LT_D * 2) + ((c ^ (rr % OUT_CH)) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      }
    } else if (lane == 0) {
      abort_flag = 1;
      atomicOr(status, Q3_STATUS_TIMEOUT);
    }
    asm volatile("bar.sync 1, %0;" ::"n"(LT_SOFTMAX) : "memory");
    if (done) {
#pragma unroll
      for (int i = 0; i < LT_BM * OUT_CH / LT_SOFTMAX; ++i) {
        const int idx = threadIdx.x + i * LT_SOFTMAX, r = idx / OUT_CH, c = idx % OUT_CH;
        if (row0 + r < q_len)
          *reinterpret_cast<uint4*>(out + ((size_t)(qs + row0 + r) * H + h) * LT_D + c * 8) =
              *reinterpret_cast<const uint4*>(q_s + r * (LT_D * 2) + ((c ^ (r % OUT_CH)) << 4));
      }
    }
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (warp == LT_ISSUE_WARP) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_s), "r"(LT_TMEM_COLS) : "memory");
  }
#undef abort_flag
}

}  // namespace q3

// For the tests of the give-up path: see set_wait_test in tc_common.cuh.
extern "C" int q3_latent_attn_tc_wait_test(unsigned limit, int drop) { return q3::set_wait_test(limit, drop); }

// c_rows [B * pitch, rank], r_rows [B * pitch, rot] <- the latents and rotated parts of the first kv_len[b] keys of request
// b (never more than pitch), in rows b * pitch ...  bfloat16, rank and rot multiples of 8.
extern "C" int q3_latent_gather(const void* c_pages, const void* r_pages, const int* kv_len, const int* table, int stride,
                                int page_size, int num_pages, int B, int pitch, int rank, int rot, void* c_rows, void* r_rows,
                                int* status, cudaStream_t stream) {
  if (B <= 0 || pitch <= 0) return 0;
  if (rank <= 0 || rot < 0 || rank % 8 || rot % 8 || page_size <= 0 || stride <= 0 || B > 65535 ||
      (long long)pitch * ((rank + rot) / 8) > 0x7fffff00ll)
    return Q3_ERR_SIZE;
  if ((uintptr_t)c_pages % 16 || (uintptr_t)r_pages % 16 || (uintptr_t)c_rows % 16 || (uintptr_t)r_rows % 16)
    return Q3_ERR_ALIGN;
  using bf16 = __nv_bfloat16;
  const unsigned blocks = (unsigned)(((long long)pitch * ((rank + rot) / 8) + 255) / 256);
  q3::launch(q3::latent_gather_kernel, dim3(blocks, B), dim3(256), 0, stream, (const bf16*)c_pages, (const bf16*)r_pages,
             kv_len, table, stride, page_size, num_pages, rank, rot, pitch, (bf16*)c_rows, (bf16*)r_rows, status);
  return q3::launch_status();
}

// Causal attention of every request's tokens over its formed keys and values: kv [B * pitch, 2 H 128] (keys of all heads,
// then values), r_rows [B * pitch, 64], q_plain [T, H, 128], q_rot [T, H, 64], out [T, H, 128], all bfloat16; gate float32
// [T, H] or null; sink float32 [H] or null.  max_q_len: of the requests' new tokens.  A positive scale.
extern "C" int q3_latent_attn_tc(const void* q_plain, const void* q_rot, const void* kv, const void* r_rows, void* out,
                                 const int* q_start, const int* kv_len, int B, int pitch, int max_q_len, int H, float scale,
                                 const float* gate, const float* sink, int* status, cudaStream_t stream) {
  using namespace q3;
  if (B <= 0 || max_q_len <= 0) return 0;
  if (H <= 0 || H > 65535 || B > 65535 || pitch <= 0 || (long long)B * pitch > 0x7fffff00ll || !(scale > 0.f)) return Q3_ERR_SIZE;
  const long long tiles = ((long long)max_q_len + LT_BM - 1) / LT_BM;
  if (tiles > 65535) return Q3_ERR_SIZE;
  if ((uintptr_t)q_plain % 16 || (uintptr_t)q_rot % 16 || (uintptr_t)kv % 16 || (uintptr_t)r_rows % 16 || (uintptr_t)out % 16)
    return Q3_ERR_ALIGN;
  cudaError_t e = cudaFuncSetAttribute(latent_attn_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LT_SMEM);
  if (e != cudaSuccess) return (int)e;
  CUtensorMap map_kv, map_r;
  const uint64_t rows = (uint64_t)B * pitch;
  int code = cached_map(&map_kv, kv, rows, (uint64_t)2 * H * LT_D, LT_BN);
  if (code) return code;
  code = cached_map(&map_r, r_rows, rows, LT_ROT, LT_BN);
  if (code) return code;
  launch(latent_attn_tc_kernel, dim3(H, (unsigned)tiles, B), dim3(LT_THREADS), LT_SMEM, stream, map_kv, map_r,
         (const __nv_bfloat16*)q_plain, (const __nv_bfloat16*)q_rot, (__nv_bfloat16*)out, q_start, kv_len, pitch, H,
         scale * 1.4426950408889634f, gate, sink, status);
  return launch_status();
}
