// Which of two mbarriers, and which phase of it, stands for tile j in the attention kernels that walk tiles of keys
// (attn_tc.cu, latent_attn_tc.cu).
//
// A wait on an mbarrier names only the parity of the phase that it waits for, so it is right only while the barrier's
// completed phases can be told apart by parity: when the wait is made, every phase before the wanted one must be known to
// be over and the one after it must not be over yet.  One barrier for all tiles does not give that.  After the scores of
// tile j are seen to be ready, the product P V of tile j - 2 is known to be over (the scores were issued behind it) but not
// that of tile j - 1, and a tile whose wait was slow to look can be overtaken by the next.  With a barrier for the even and
// one for the odd tiles, tile j follows tile j - 2 on its barrier, which is over, and tile j + 2 cannot be over before the
// waiting warp itself has handed on tile j + 1 (the issuing thread: tile j).  The tests walk every order of events of this.
#pragma once

#ifdef __CUDACC__
#define Q3_HOST_DEVICE __host__ __device__
#else
#define Q3_HOST_DEVICE
#endif

namespace q3 {

Q3_HOST_DEVICE constexpr int tile_slot(int j) { return j & 1; }
Q3_HOST_DEVICE constexpr unsigned tile_parity(int j) { return ((unsigned)j >> 1) & 1u; }

}  // namespace q3
