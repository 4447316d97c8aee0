// Which phases of their barriers the softmax warps of the prompt attention kernels wait for, written once for the kernels
// (attn_prefill_umma.cu, gqa_prefill_umma.cu) and for the host model of their hand-overs (tests/cabi/attn_phases_model.cpp).
//
// The product of tile `it` with its values arrives on a barrier of its own when it is done. A wait names a phase by its parity and
// cannot tell a phase from the one two before it, so a warp must have seen every phase of a barrier end before it waits for the
// next one. That the product is done follows from other barriers too (the tensor pipe works in order: the scores that are
// multiplied later arrive later), but not that its arrival is there: arrivals on different barriers keep no order. A wait for the phase behind one that
// was passed over would then be answered by the phase before it, and a row's sums rescaled while a product is still added to them.
//
// With BARRIERS barriers in turn a warp waits at the start of a tile for the product BARRIERS tiles before. With one, that is the tile before: for
// kernels whose scores are multiplied behind it. Where the scores of a tile are multiplied ahead of the product before, that product may or
// may not be done when they are there, and two barriers are needed: the phase that is waited for is then the last that can have
// ended on its barrier, since the next one needs this warp's weights of this tile.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define NFAI_PHD __host__ __device__ __forceinline__
#else
#define NFAI_PHD inline
#endif

namespace nfai {

template <uint32_t BARRIERS>
struct ValuePhases {
  static constexpr uint32_t kBarriers = BARRIERS;
  NFAI_PHD static uint32_t barrier(uint32_t it) { return it % BARRIERS; }
  NFAI_PHD static uint32_t parity(uint32_t it) { return it / BARRIERS & 1u; }
  // `wait(tile)` for what has to be seen at the start of a tile,
  template <typename W>
  NFAI_PHD static void at_tile(uint32_t it, W&& wait) {
    if (it >= BARRIERS) wait(it - BARRIERS);
  }
  // before the sums of a row are rescaled in it,
  template <typename W>
  NFAI_PHD static void at_rescaling(uint32_t it, W&& wait) {
    if (it) wait(it - 1);
  }
  // and behind the last of n tiles: the sums are complete, and no arrival is on its way when the CTA leaves.
  template <typename W>
  NFAI_PHD static void at_end(uint32_t n, W&& wait) {
    for (uint32_t it = n > BARRIERS ? n - BARRIERS : 0; it < n; ++it) wait(it);
  }
};

}  // namespace nfai
