// True float32 matrix product for the 32-bit path of the model:
//   C[M, N] = A[M, K] * W[N, K]^T      (the layout of a Linear weight: y = x W^T)
// FFMA on CUDA cores: no tensor cores, no TF32.
//
// The order of an output's additions depends on k alone, so a row's result does not depend on M, on the rest of the
// batch or on which of the two kernels below computes it.  With k = 1024 s + 256 j + 8 l + i (j < 4, l < 32, i < 8):
//   chain(s, l) = the FMA chain over j, then i, ascending, from zero            (32 terms)
//   T_g         = the chains of l = 8 g .. 8 g + 7, s by s, l ascending, added one after the other (g < 4)
//   C           = (T_0 + T_1) + (T_2 + T_3)
// It is made for both kernels: l is the lane that streams a weight row in pieces of 32 bytes where few rows of A make
// the product a stream over W, and g is one of four groups of threads that share the K of an output tile.  Short chains,
// summed by groups, are also closer to 64 bits than one sum over K in tiles of 16, which was the order before (of the result's
// norm, normal values: 1.24e-7 against 1.60e-7 at K = 1,024, 1.44e-7 against 2.56e-7 at K = 3,072).
#include "common.cuh"

namespace q3 {

constexpr int GF_SEG = 1024;  // values of k in a segment s
constexpr int GF_STEP = 256;  // from one j to the next
constexpr int GF_LANE = 8;    // values of k of a lane at a time

// ---------------------------------------------------------------- tiles
// 64 x 64 outputs per block, four groups of 64 threads; group g walks over its chains (s, l) with 8 x 8 outputs per thread
// and the four partial sums meet in shared memory (64 FMA per four 16-byte shared-memory reads).  The split over K inside
// the block gives a narrow product more blocks than wider tiles would (N = 1,024 and 500 rows: 128 tiles of 64 x 64, with
// eight warps each, against 32 of 128 x 128 for 148 SMs).  The FMA pipe is busy half of the time (513 x 4,096 x 1,024: 139.8 us,
// 31 of 74 TFLOP/s).  Of 5.4 us for a tile's 128 values of k the FMA loop alone takes 3.2 (49 TFLOP/s; such a loop over registers
// reaches 50 to 72, by how the compiler places them), and two warps per scheduler hide none of the rest: operand reads 1.2,
// copies 0.6, running sums 0.6.  Packed FMAs reach 61 to 73 in such a loop, and 0.8 to 1.0 of this kernel's speed in it where the
// tiles fill the SMs.
constexpr int GF_T = 64, GF_GROUPS = 4, GF_GROUP_THREADS = 64, GF_THREADS = GF_GROUPS * GF_GROUP_THREADS, GF_STAGES = 3;
constexpr int GF_STAGE_BYTES = 2 * GF_T * 128;                            // 64 rows of A, 64 of W, 32 values of k each
constexpr int GF_RED_PITCH = GF_T + 8;                                    // floats: a thread's rows fall on different banks
constexpr int GF_SMEM = GF_GROUPS * GF_STAGES * GF_STAGE_BYTES;           // 192 KB; the partial sums reuse it
static_assert(GF_GROUPS * GF_T * GF_RED_PITCH * 4 <= GF_SMEM, "the partial sums fit");

template <int BYTES>
__device__ __forceinline__ void gf_copy(uint32_t dst, const float* src, bool in) {
  const int n = in ? BYTES : 0;  // zero bytes read: the destination is filled with zeros
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ float4 gf_lds(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}

// VEC: K, lda, ldw are multiples of 4 and A, W are 16-byte aligned (copies of 16 bytes; otherwise of 4).
template <bool VEC>
__global__ void __launch_bounds__(GF_THREADS, 1)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                     int lda, int ldw, int ldc, int out_vec) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(1024) unsigned char gf_smem[];
  const int group = threadIdx.x / GF_GROUP_THREADS, t = threadIdx.x % GF_GROUP_THREADS;
  const int m_tiles = (M + GF_T - 1) / GF_T;  // tiles of the same W rows next to each other: a wave of blocks reads W once
  const int m0 = (blockIdx.x % m_tiles) * GF_T, n0 = (blockIdx.x / m_tiles) * GF_T;
  const uint32_t stages = (uint32_t)__cvta_generic_to_shared(gf_smem) + group * GF_STAGES * GF_STAGE_BYTES;

  // a stage: row r's 32 values of chain (s, l) as eight pieces of 16 bytes (piece c: j = c / 2, half c % 2), piece c at
  // place c ^ (r % 8), so that eight rows' equal pieces lie on different banks
  const int c = t & 7, r8 = t >> 3;
  const int k_piece = (c >> 1) * GF_STEP + (c & 1) * 4;
  const uint32_t dst0 = r8 * 128 + ((c ^ r8) << 4);
  // Only what holds a k below K is fetched and multiplied: of the last segment's chains those that begin there, and of a
  // chain's four pieces (j) those that do.  (K = 64: 8 of 32 chains and one piece of four in each.  What is left out would
  // add zeros to sums that are not negative zero: the bits are the same.)
  const int segs = (K + GF_SEG - 1) / GF_SEG, rem = K - (segs - 1) * GF_SEG - group * (8 * GF_LANE);
  const int items = (segs - 1) * 8 + max(0, min(8, (rem + GF_LANE - 1) / GF_LANE));  // chains of this group
  auto fetch = [&](int item) {
    const int k = (item >> 3) * GF_SEG + k_piece + (group * 8 + (item & 7)) * GF_LANE;
    if (k - (c & 1) * 4 >= K) return;  // the piece is not read
    const uint32_t dst = stages + (item % GF_STAGES) * GF_STAGE_BYTES + dst0;
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      const int r = r8 + 8 * (p & 7), row = (p < 8 ? m0 : n0) + r, rows = p < 8 ? M : N;
      const float* src = (p < 8 ? A + (size_t)min(row, M - 1) * lda : W + (size_t)min(row, N - 1) * ldw);
      if (VEC) {
        const bool in = row < rows && k < K;
        gf_copy<16>(dst + p * 1024, src + (in ? k : 0), in);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool in = row < rows && k + e < K;
          gf_copy<4>(dst + p * 1024 + 4 * e, src + (in ? k + e : 0), in);
        }
      }
    }
  };
#pragma unroll
  for (int i = 0; i < GF_STAGES - 1; ++i) {
    if (i < items) fetch(i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  const int tx = t & 7, ty = t >> 3;  // rows ty + 8 i of A, tx + 8 j of W
  float total[8][8], part[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) total[i][j] = 0.f;

  for (int item = 0; item < items; ++item) {
    asm volatile("cp.async.wait_group %0;" ::"n"(GF_STAGES - 2) : "memory");
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(GF_GROUP_THREADS) : "memory");  // the group's copies are there,
    if (item + GF_STAGES - 1 < items) fetch(item + GF_STAGES - 1);  // and the stage read in the last turn is free
    asm volatile("cp.async.commit_group;" ::: "memory");
    const uint32_t base = stages + (item % GF_STAGES) * GF_STAGE_BYTES;
    const uint32_t a_row = base + ty * 128, w_row = base + GF_T * 128 + tx * 128;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) part[i][j] = 0.f;
    auto multiply = [&](int q) {
      float4 a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = gf_lds(a_row + i * 1024 + ((q ^ ty) << 4));
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 w = gf_lds(w_row + j * 1024 + ((q ^ tx) << 4));
#pragma unroll
        for (int i = 0; i < 8; ++i) part[i][j] = fmaf(a[i].x, w.x, part[i][j]);
#pragma unroll
        for (int i = 0; i < 8; ++i) part[i][j] = fmaf(a[i].y, w.y, part[i][j]);
#pragma unroll
        for (int i = 0; i < 8; ++i) part[i][j] = fmaf(a[i].z, w.z, part[i][j]);
#pragma unroll
        for (int i = 0; i < 8; ++i) part[i][j] = fmaf(a[i].w, w.w, part[i][j]);
      }
    };
    const int left = min(GF_SEG, K - (item >> 3) * GF_SEG - (group * 8 + (item & 7)) * GF_LANE);
#pragma unroll 1
    for (int q = 0; q < 8 && q * (GF_STEP / 2) < left; q += 2) {
      multiply(q);
      multiply(q + 1);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) total[i][j] += part[i][j];
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* red = reinterpret_cast<float*>(gf_smem);
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) red[(group * GF_T + ty + 8 * i) * GF_RED_PITCH + tx + 8 * j] = total[i][j];
  __syncthreads();
  // four neighbouring outputs per thread and turn
  for (int e = threadIdx.x; e < GF_T * GF_T / 4; e += GF_THREADS) {
    const int r = e / (GF_T / 4), col = (e % (GF_T / 4)) * 4;
    if (m0 + r >= M || n0 + col >= N) continue;
    float4 T[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) T[g] = *reinterpret_cast<const float4*>(&red[(g * GF_T + r) * GF_RED_PITCH + col]);
    const float v[4] = {(T[0].x + T[1].x) + (T[2].x + T[3].x), (T[0].y + T[1].y) + (T[2].y + T[3].y),
                        (T[0].z + T[1].z) + (T[2].z + T[3].z), (T[0].w + T[1].w) + (T[2].w + T[3].w)};
    float* dst = C + (size_t)(m0 + r) * ldc + n0 + col;
    if (out_vec && n0 + col + 4 <= N) {
      *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (n0 + col + i < N) dst[i] = v[i];
    }
  }
}

// ---------------------------------------------------------------- short reductions
// K up to 128, where the tiles above would leave two or three of their four groups without a chain: 64 x 64 outputs per
// block, 4 x 4 per thread, all of K in shared memory at once, the chains one after the other (T_0, then T_1; the other two
// are zero).  34 KB for K = 64, so that several blocks share an SM and one's copies run under another's products.  Bound by
// shared-memory reads (eight of 16 bytes per 64 FMA) and, for the smallest K, by the stores: 2,048 x 4,096 outputs of K = 64
// 45 us (24 TFLOP/s; the tiles above 96), of K = 128 77 us (99); the kernel before these took 53 and 99 us.
constexpr int GFK_MAX = 128, GFK_THREADS = 256;

template <bool VEC>
__global__ void __launch_bounds__(GFK_THREADS)
gemm_f32_short_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                      int lda, int ldw, int ldc, int out_vec) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(16) float gfk_smem[];  // [64 rows of A, then 64 of W][pitch]
  const int chains = (K + GF_LANE - 1) / GF_LANE, pieces = 2 * chains, pitch = 8 * chains + 4;  // eight rows: other banks
  const int m_tiles = (M + GF_T - 1) / GF_T;
  const int m0 = (blockIdx.x % m_tiles) * GF_T, n0 = (blockIdx.x / m_tiles) * GF_T;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(gfk_smem);
  for (int e = threadIdx.x; e < 2 * GF_T * pieces; e += GFK_THREADS) {
    const int r = e / pieces, k = (e - r * pieces) * 4;
    const bool of_a = r < GF_T;
    const int row = of_a ? m0 + r : n0 + r - GF_T;
    const bool in_row = row < (of_a ? M : N);
    const float* src = of_a ? A + (size_t)min(row, M - 1) * lda : W + (size_t)min(row, N - 1) * ldw;
    const uint32_t dst = base + (r * pitch + k) * 4;
    if (VEC) {
      gf_copy<16>(dst, src + (k < K ? k : 0), in_row && k < K);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) gf_copy<4>(dst + 4 * i, src + (k + i < K ? k + i : 0), in_row && k + i < K);
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;  // rows ty + 16 i of A, tx + 16 j of W
  const uint32_t a_row = base + ty * pitch * 4, w_row = base + (GF_T + tx) * pitch * 4;
  float sum[4][4], T[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sum[i][j] = T[i][j] = 0.f;
#pragma unroll 2
  for (int l = 0; l < chains; ++l) {
    if (l == 8) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          sum[i][j] = T[i][j];
          T[i][j] = 0.f;
        }
    }
    float part[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) part[i][j] = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4 a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = gf_lds(a_row + (16 * i * pitch + 8 * l + 4 * h) * 4);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 w = gf_lds(w_row + (16 * j * pitch + 8 * l + 4 * h) * 4);
#pragma unroll
        for (int i = 0; i < 4; ++i) part[i][j] = fmaf(a[i].x, w.x, part[i][j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) part[i][j] = fmaf(a[i].y, w.y, part[i][j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) part[i][j] = fmaf(a[i].z, w.z, part[i][j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) part[i][j] = fmaf(a[i].w, w.w, part[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) T[i][j] += part[i][j];
  }
  // through shared memory, so that a row's values leave side by side
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) gfk_smem[(ty + 16 * i) * (GF_T + 4) + tx + 16 * j] = sum[i][j] + T[i][j];
  __syncthreads();
  for (int e = threadIdx.x; e < GF_T * GF_T / 4; e += GFK_THREADS) {
    const int r = e / (GF_T / 4), col = (e % (GF_T / 4)) * 4;
    if (m0 + r >= M || n0 + col >= N) continue;
    const float4 v = *reinterpret_cast<const float4*>(&gfk_smem[r * (GF_T + 4) + col]);
    float* dst = C + (size_t)(m0 + r) * ldc + n0 + col;
    if (out_vec && n0 + col + 4 <= N) {
      *reinterpret_cast<float4*>(dst) = v;
    } else {
      const float vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (n0 + col + i < N) dst[i] = vs[i];
    }
  }
}

// ---------------------------------------------------------------- a few rows of A
// Decoding: the product is one pass over W, so the weights go from memory straight into the registers that multiply them,
// 32 bytes per lane and load, and each warp takes R weight rows over one segment of 1,024 values of k (8 KB of loads in
// flight per warp with R = 4; the first of them before the wait on the kernel before, which never writes weights).  The
// rows of A come through L1, which the block's warps share.  The chains' sums meet in shared memory.
constexpr int GFS_WARPS = 8;
constexpr int GFS_MAX_ROWS = 16;
constexpr int GFS_MAX_SEGS = 16;  // K up to 16,384; times the groups of a block never more than this, whatever K

__device__ __forceinline__ void gf_load8(float (&v)[8], const float* p) {  // read once: not kept in L1
  asm volatile("ld.global.nc.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "l"(p));
}
__device__ __forceinline__ void gf_load8_shared(float (&v)[8], const float* p) {  // the block's warps all read it
  asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "l"(p));
}

// MT: rows of A (M <= MT; those past M repeat the last one and are not stored).  seg_warps: warps of the block that share
// a group of R weight rows, each with every seg_warps-th segment.  K, lda, ldw multiples of 8, A and W 32-byte aligned.
template <int MT, int R>
__global__ void __launch_bounds__(GFS_WARPS * 32, MT <= 8 ? 2 : 1)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                     int lda, int ldw, int ldc, int seg_warps) {
  extern __shared__ __align__(16) float gfs_sums[];  // [output of the block][segment][lane]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int segs = (K + GF_SEG - 1) / GF_SEG;
  const int groups = GFS_WARPS / seg_warps;  // of weight rows per block
  const int group = warp / seg_warps, first = warp % seg_warps;
  const int n0 = (blockIdx.x * groups + group) * R;
  const bool active = group < groups && n0 < N && first < segs;

  const float* w_row[R];
#pragma unroll
  for (int r = 0; r < R; ++r) w_row[r] = W + (size_t)min(n0 + r, N - 1) * ldw + lane * GF_LANE;
  float w[2][R][8];
  auto load_w = [&](float (&dst)[R][8], int s, int j) {
    const int k = s * GF_SEG + j * GF_STEP;
    const bool in = s < segs && k + lane * GF_LANE < K;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (in) {
        gf_load8(dst[r], w_row[r] + k);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) dst[r][i] = 0.f;
      }
    }
  };
  if (active) {
    load_w(w[0], first, 0);
    load_w(w[1], first, 1);
  }
  pdl_wait();
  pdl_launch_dependents();
  if (active) {
    for (int s = first; s < segs; s += seg_warps) {
      float acc[R][MT];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[r][m] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = s * GF_SEG + j * GF_STEP + lane * GF_LANE;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          float x[8];
          if (k < K) {
            gf_load8_shared(x, A + (size_t)min(m, M - 1) * lda + k);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = 0.f;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r][m] = fmaf(x[i], w[j & 1][r][i], acc[r][m]);
        }
        if (j < 2) load_w(w[j & 1], s, j + 2);
        else load_w(w[j & 1], s + seg_warps, j - 2);
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m)
          gfs_sums[((size_t)((group * R + r) * MT + m) * segs + s) * 32 + lane] = acc[r][m];
    }
  }
  __syncthreads();
  // four threads per output: T_g of the head of the file, then their sums
  const int outputs = groups * R * MT;
  for (int e0 = 0; e0 < outputs * 4; e0 += GFS_WARPS * 32) {  // whole warps: the shuffles below
    const int e = e0 + threadIdx.x, o = e >> 2, g = e & 3;
    const int m = o % MT, n = (blockIdx.x * groups) * R + o / MT;
    const bool live = o < outputs && m < M && n < N;
    float T = 0.f;
    if (live) {
      const float* p = gfs_sums + (size_t)o * segs * 32 + g * 8;
      for (int s = 0; s < segs; ++s) {
        const float4 a = *reinterpret_cast<const float4*>(p + s * 32), b = *reinterpret_cast<const float4*>(p + s * 32 + 4);
        T += a.x; T += a.y; T += a.z; T += a.w;
        T += b.x; T += b.y; T += b.z; T += b.w;
      }
    }
    T += __shfl_xor_sync(0xffffffffu, T, 1);
    T += __shfl_xor_sync(0xffffffffu, T, 2);
    if (live && g == 0) C[(size_t)m * ldc + n] = T;
  }
}

template <int MT, int R>
static int gemm_f32_rows_launch(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                                int segs, int seg_warps, cudaStream_t stream) {
  const int groups = GFS_WARPS / seg_warps;
  const size_t smem = (size_t)groups * R * MT * segs * 32 * sizeof(float);
  // The limit is the function's, for all threads: always set to the most that any K asks for, so that no call lowers it
  // under another's launch.
  constexpr size_t most = (size_t)R * MT * GFS_MAX_SEGS * 32 * sizeof(float);
  if (smem > most) return Q3_ERR_SIZE;
  auto kernel = gemm_f32_rows_kernel<MT, R>;
  if (most > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) return (int)e;
  }
  q3::launch(kernel, dim3((N + groups * R - 1) / (groups * R)), dim3(GFS_WARPS * 32), smem, stream, A, W, C, M, N, K, lda, ldw,
             ldc, seg_warps);
  return launch_status();
}

}  // namespace q3

// C[M, N] = A[M, K] * W[N, K]^T, all float32, row pitches lda / ldw / ldc in elements.
extern "C" int q3_gemm_f32_nt(const float* A, const float* W, float* C, int M, int N, int K, int lda,
                              int ldw, int ldc, cudaStream_t stream) {
  using namespace q3;
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return Q3_ERR_SIZE;
  const int segs = (K + GF_SEG - 1) / GF_SEG;
  // Up to 16 rows stream W once; the sums of up to 16 segments (K = 16,384) fit the block's shared memory.  A short reduction
  // gives a lane of that kernel little to do per row of A: there the kernels below are the faster ones (us for N = 4,096:
  // 8 rows, K = 32 5.5 against 3.5, K = 64 5.5 and 5.6; 16 rows, K = 64 7.7 and 4.8; 16 rows of N = 150,000, K = 192 222 and 175,
  // but 7.8 and 11.6 for N = 4,096, where the tiles are fewer than the SMs).
  const bool streams = K >= 256 || (K > GFK_MAX && (M <= 8 || (N + GF_T - 1) / GF_T * 2 <= sm_count())) ||
                       (K <= GFK_MAX && M <= 8 && K >= 8 * M);
  if (streams && M <= GFS_MAX_ROWS && segs <= GFS_MAX_SEGS && K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 &&
      (uintptr_t)A % 32 == 0 && (uintptr_t)W % 32 == 0) {
    const int seg_warps = segs < GFS_WARPS ? segs : GFS_WARPS;
    const int groups = GFS_WARPS / seg_warps;
    // four weight rows per warp share the reads of A; two where four would leave SMs without a block
    const bool four = (N + groups * 4 - 1) / (groups * 4) >= sm_count() * 3 / 4;
#define Q3_GFS_GO(MT)                                                                                              \
  return four ? gemm_f32_rows_launch<MT, 4>(A, W, C, M, N, K, lda, ldw, ldc, segs, seg_warps, stream)              \
              : gemm_f32_rows_launch<MT, 2>(A, W, C, M, N, K, lda, ldw, ldc, segs, seg_warps, stream)
    if (M == 1) Q3_GFS_GO(1);
    if (M == 2) Q3_GFS_GO(2);
    if (M <= 4) Q3_GFS_GO(4);
    if (M <= 8) Q3_GFS_GO(8);
    Q3_GFS_GO(16);
#undef Q3_GFS_GO
  }
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
  const int out_vec = ldc % 4 == 0 && (uintptr_t)C % 16 == 0;
  const long long m_tiles = (M + GF_T - 1) / GF_T, n_tiles = (N + GF_T - 1) / GF_T;
  if (m_tiles > 65535 || m_tiles * n_tiles > 0x7fffffffll) return Q3_ERR_SIZE;
  if (K <= GFK_MAX) {
    constexpr int most = 2 * GF_T * (GFK_MAX + 4) * (int)sizeof(float);
    const size_t smem = max((size_t)2 * GF_T * (8 * ((K + 7) / 8) + 4), (size_t)GF_T * (GF_T + 4)) * sizeof(float);
    auto kernel = vec ? gemm_f32_short_kernel<true> : gemm_f32_short_kernel<false>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return (int)e;
    q3::launch(kernel, dim3((unsigned)(m_tiles * n_tiles)), dim3(GFK_THREADS), smem, stream, A, W, C, M, N, K, lda, ldw, ldc, out_vec);
    return launch_status();
  }
  auto kernel = vec ? gemm_f32_tile_kernel<true> : gemm_f32_tile_kernel<false>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GF_SMEM);
  if (e != cudaSuccess) return (int)e;
  q3::launch(kernel, dim3((unsigned)(m_tiles * n_tiles)), dim3(GF_THREADS), GF_SMEM, stream, A, W, C, M, N, K, lda, ldw, ldc, out_vec);
  return launch_status();
}
