// Prompt attention of Tutizen layers on the 5th-generation tensor cores: bfloat16 operands and caches, heads of 64 or 128.
//
// A CTA owns 128 tokens of one head, one accumulator lane each, and walks the key tiles (64 positions) from the causal edge back to
// the reach of the head's distance bias (gqa_common.cuh), newest first: with a bias the maximum is then found early.
//   warp 8     Q, then K and V tiles by TMA into a ring of 128-byte swizzled slots
//   warp 9     one lane issues S = Q K^T and O += P V (P in tensor memory, V as it lies in the cache: its rows run along N)
//   warps 0-7  softmax, two threads to a row (32 positions each): they add the bias to S, write the weights back and keep their
//              float32 sums; at the end they divide, gate and store half a row of O each
// The weights enter the second product as a bfloat16 head and remainder (relative error ~2^-17), as in the warp-level kernel; both
// fit where the scores lay. Two tiles' scores and O are 192 or 256 columns of tensor memory, so that the next tile's scores are
// there when this one's weights are done, and two CTAs share an SM. A row's sums are rescaled only when its maximum has grown by more
// than 8 (base 2): weights are then at most 2^8 and their relative rounding is what it was.
//
// What bounds it: issue slots of the softmax (bias, exponential, split: about 11 per pair of weights) are 53 % of a launch's, the rest is
// latency between a tile's steps and the last of 1.7 waves (41 us at 2011 tokens). Against the warp-level kernel of
// gqa_prefill.cu, prompts of 16 layers with 32 heads of 64 (ms): 2011 tokens 6.52 and 5.99 (about 75 and 41 us a layer), 1024: 4.00 and
// 3.91, 512: 3.04 and 2.99, 384: 2.88 and 2.83. Tiles of 128 positions, their weights over the scores of the only tile that fits beside
// O then: 6.18 at 2011 (spills, and the products wait for the weights and the weights for the products).
#include "attn_phases.h"
#include "gqa_common.cuh"
#include "umma.cuh"

namespace nfai {

namespace {

using namespace umma;
using namespace gqa_detail;
using attn_detail::kNegBig;

constexpr uint32_t kM = 128;        // tokens of a CTA
constexpr uint32_t kN = 64;         // positions per tile
constexpr int kThreads = 320;
constexpr float kGrowth = 8.0f;     // growth of a maximum (base 2) that the sums are carried through without rescaling
using Values = ValuePhases<2>;      // barriers of the products with the values: scores are multiplied one tile ahead of them

template <int D>
struct Smem {
  static constexpr uint32_t kQ = kM * D * 2;                 // D / 64 blocks of [128][64]
  static constexpr uint32_t kTile = kN * D * 2;              // a K or a V tile: D / 64 blocks of [64][64]
  static constexpr uint32_t kSlots = D == 64 ? 10 : 4;       // two CTAs on an SM
  static constexpr uint32_t kBarOff = kQ + kSlots * kTile;
  static constexpr uint32_t kSwapOff = kBarOff + 256;        // two floats per row: maxima of its halves, later their sums
  static constexpr uint32_t kTotal = kSwapOff + 2 * kM * 4 + 1024;
};

__device__ __forceinline__ uint32_t bf2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return reinterpret_cast<const uint32_t&>(h);
}

template <int D>
__global__ void __launch_bounds__(kThreads, 2) gqa_prefill_umma_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                                                                       const __grid_constant__ CUtensorMap mapV, const GqaParams p, const uint32_t T) {
  using SM = Smem<D>;
  constexpr uint32_t kLow = kN / 2, kO = 2 * kN;  // columns of tensor memory: weights, and their remainders, over the scores of either tile
  extern __shared__ unsigned char gu_raw[];
  unsigned char* const sm = reinterpret_cast<unsigned char*>(((uintptr_t)gu_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(sm + SM::kBarOff);
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * SM::kSlots + 5 + Values::kBarriers);
  const uint32_t full0 = s_u32(bars), empty0 = s_u32(bars + SM::kSlots), q_ready = s_u32(bars + 2 * SM::kSlots), s_ready = q_ready + 8,
                 p_ready = q_ready + 24, pv_done = q_ready + 40;  // (s_ready, p_ready, pv_done: one for each of two tiles)
  const GqaSpec& spec = p.spec;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;  // (warp: uniform)
  if (tid == 0) {
    for (uint32_t i = 0; i < SM::kSlots; ++i) {
      bar_init(full0 + 8 * i, 1);
      bar_init(empty0 + 8 * i, 1);
    }
    bar_init(q_ready, 1);
    for (uint32_t i = 0; i < 2; ++i) {
      bar_init(s_ready + 8 * i, 1);
      bar_init(p_ready + 8 * i, 8);
    }
    for (uint32_t i = 0; i < Values::kBarriers; ++i) bar_init(pv_done + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(256u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();  // queries and the newest cache rows come from the kernel launched just before

  // the last tokens of the heads that reach farthest start first
  const uint32_t h = spec.heads - 1 - blockIdx.x % spec.heads, row0 = (gridDim.x / spec.heads - 1 - blockIdx.x / spec.heads) * kM;
  const uint32_t g = h / (spec.heads / spec.kv_heads);
  const float sl = slope2(spec, h);
  const uint32_t far = reach(spec, sl), first_pos = p.pos0 + row0, last_pos = p.pos0 + min(T, row0 + kM) - 1;
  const uint32_t tile_lo = (first_pos > far ? first_pos - far : 0u) / kN, tile_hi = last_pos / kN, n = tile_hi - tile_lo + 1;
  bool ok = true;

  if (warp == 8) {
    if (elect_one()) {
      bar_expect_tx(q_ready, SM::kQ);
#pragma unroll
      for (uint32_t b = 0; b < D / 64; ++b) tma_load_2d(s_u32(sm) + b * (kM * 128), &mapQ, (int)(h * D + b * 64), (int)row0, q_ready);
    }
    __syncwarp();
    uint32_t j = 0;
    auto load = [&](const CUtensorMap* map, uint32_t tile) {
      const uint32_t s = j % SM::kSlots;
      if (j >= SM::kSlots && !warp_wait(empty0 + 8 * s, (j / SM::kSlots - 1) & 1)) return ok = false;
      if (elect_one()) {
        bar_expect_tx(full0 + 8 * s, SM::kTile);
#pragma unroll
        for (uint32_t b = 0; b < D / 64; ++b)
          tma_load_2d(s_u32(sm) + SM::kQ + s * SM::kTile + b * (kN * 128), map, (int)(g * D + b * 64), (int)(tile * kN), full0 + 8 * s);
      }
      __syncwarp();
      ++j;
      return true;
    };
    load(&mapK, tile_hi);
    for (uint32_t it = 0; it < n && ok; ++it) {
      if (it + 1 < n && !load(&mapK, tile_hi - it - 1)) break;
      if (!load(&mapV, tile_hi - it)) break;
    }
    if (ok) ok = drain_ring<SM::kSlots>(empty0, j);
  } else if (warp == 9) {
    // bfloat16 operands, float32 sums; A along K in both products; B along K (K tile) or along N (V tile)
    constexpr uint32_t types = (1u << 4) | (1u << 7) | (1u << 10);
    constexpr uint32_t idesc_s = types | ((kN >> 3) << 17) | ((kM >> 4) << 24);
    constexpr uint32_t idesc_o = types | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((kM >> 4) << 24);
    const uint32_t q_s = s_u32(sm);
    uint32_t j = 0;
    auto slot = [&](uint32_t& s) {  // wait for the next tile
      s = j % SM::kSlots;
      ok = warp_wait(full0 + 8 * s, (j / SM::kSlots) & 1);
      fence_after();
      ++j;
      return ok;
    };
    // (the weights of tile it - 2 lie where its scores go: products of one thread run in their order)
    auto scores = [&](uint32_t it) {
      uint32_t s;
      if (!slot(s)) return false;
      if (elect_one()) {
        const uint32_t k_s = q_s + SM::kQ + s * SM::kTile;
#pragma unroll
        for (uint32_t kk = 0; kk < D / 16; ++kk)
          umma_f16(tmem + (it & 1) * kN, smem_desc_sw128(q_s + (kk >> 2) * (kM * 128) + (kk & 3) * 32),
                   smem_desc_sw128(k_s + (kk >> 2) * (kN * 128) + (kk & 3) * 32), idesc_s, kk != 0);
        umma_commit(empty0 + 8 * s);
        umma_commit(s_ready + 8 * (it & 1));
      }
      __syncwarp();
      return true;
    };
    ok = warp_wait(q_ready, 0);
    fence_after();
    if (ok) scores(0);
    for (uint32_t it = 0; it < n && ok; ++it) {
      if (it + 1 < n && !scores(it + 1)) break;
      if (!(ok = warp_wait(p_ready + 8 * (it & 1), (it >> 1) & 1))) break;
      fence_after();
      uint32_t s;
      if (!slot(s)) break;
      if (elect_one()) {
        const uint32_t v_s = q_s + SM::kQ + s * SM::kTile, weights = tmem + (it & 1) * kN;
#pragma unroll
        for (uint32_t kk = 0; kk < kN / 16; ++kk) {
          const uint64_t v = smem_desc_mn_sw128(v_s + kk * 2048, kN * 128);
          umma_f16_ta(tmem + kO, weights + kk * 8, v, idesc_o, (it | kk) != 0);
          umma_f16_ta(tmem + kO, weights + kLow + kk * 8, v, idesc_o, 1);
        }
        umma_commit(empty0 + 8 * s);
        umma_commit(pv_done + 8 * Values::barrier(it));
      }
      __syncwarp();
    }
  } else {
    const uint32_t quarter = warp & 3, half = warp >> 2, col0 = half * (kN / 2), r_own = quarter * 32 + lane;
    const uint32_t row = row0 + r_own, limit = p.pos0 + min(row, T - 1);          // last position this row sees
    const uint32_t w_first = p.pos0 + min(row0 + quarter * 32, T - 1);            // ... and the warp's first row
    const uint32_t lanes = tmem + (quarter * 32u << 16);
    float* const swap = reinterpret_cast<float*>(sm + SM::kSwapOff);              // [2][kM]
    auto meet = [&]() { asm volatile("barrier.cta.sync %0, 64;" ::"r"(quarter + 1) : "memory"); };
    auto either = [&](bool mine) {  // a condition on a row of either warp
      uint32_t r;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %2, 0;\n\tbarrier.cta.red.or.pred q, %1, 64, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
          : "=r"(r)
          : "r"(quarter + 1), "r"((uint32_t)mine)
          : "memory");
      return r != 0;
    };
    auto value = [&](uint32_t j) {  // the product of tile j with its values is done
      ok = __all_sync(0xffffffffu, ok && bar_wait(pv_done + 8 * Values::barrier(j), Values::parity(j)));
    };
    float m = kNegBig, l = 0.f;
    for (uint32_t it = 0; it < n; ++it) {
      ok = __all_sync(0xffffffffu, ok && bar_wait(s_ready + 8 * (it & 1), (it >> 1) & 1));  // (a warp that gave up still meets the other one)
      Values::at_tile(it, value);
      const uint32_t n0 = (tile_hi - it) * kN + col0;
      const uint32_t tile = lanes + (it & 1) * kN;
      const float base = sl * (float)((int)n0 - (int)limit);  // bias of this half's first position
      // The weights are formed from the maximum as it stands; a row that turns out to have grown too far (the first tile always
      // has) makes its two warps raise their maxima and do the tile again.
      uint64_t sum[2];
      bool raise = it == 0;
      for (;;) {
        uint32_t s[kN / 2];
        fence_after();
        tmem_ld(tile + col0, s);
#pragma unroll
        for (uint32_t j = 0; j < kN / 2; ++j) s[j] = __float_as_uint(fmaf(sl, (float)j, __uint_as_float(s[j])));
        if (n0 + kN / 2 - 1 > w_first) {  // not every row of the warp sees the whole tile
#pragma unroll
          for (uint32_t j = 0; j < kN / 2; ++j)
            if (n0 + j > limit) s[j] = 0xff800000u;
        }
        float t[4] = {__uint_as_float(s[0]), __uint_as_float(s[1]), __uint_as_float(s[2]), __uint_as_float(s[3])};
#pragma unroll
        for (uint32_t j = 4; j < kN / 2; j += 8)
#pragma unroll
          for (uint32_t i = 0; i < 4; ++i)
            t[i] = j + 4 + i < kN / 2 ? fmaxf(fmaxf(t[i], __uint_as_float(s[j + i])), __uint_as_float(s[j + 4 + i])) : fmaxf(t[i], __uint_as_float(s[j + i]));
        float top = fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3])) + base;
        if (raise) {
          swap[half * kM + r_own] = top;
          meet();
          top = fmaxf(fmaxf(top, swap[(half ^ 1) * kM + r_own]), m);
          if (it) {
            Values::at_rescaling(it, value);
            fence_after();
            // a row that has seen no position yet: what zero weights left of values that are not finite goes, as if it had begun here
            const bool begins = m == kNegBig;
            const float f = gqa_ex2(m - top);
            l *= f;
#pragma unroll 1
            for (uint32_t c = half * (D / 2); c < (half + 1) * (D / 2); c += 16) {
              uint32_t o[16];
              tmem_ld(lanes + kO + c, o);
#pragma unroll
              for (int e = 0; e < 16; ++e) o[e] = begins ? 0u : __float_as_uint(__uint_as_float(o[e]) * f);
              tmem_st(lanes + kO + c, o);
            }
          }
          m = top;
        }
        sum[0] = sum[1] = 0;
        const uint64_t shift = pair(base - m, base - m);
        uint32_t hi[16], lo[16];
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j) {
          float a, b, ra, rb;
          unpair(add2(pair(__uint_as_float(s[2 * j]), __uint_as_float(s[2 * j + 1])), shift), a, b);
          a = gqa_ex2(a);
          b = gqa_ex2(b);
          const uint64_t w = pair(a, b);
          sum[j & 1] = add2(sum[j & 1], w);
          hi[j] = bf2(a, b);
          unpair(fma2(pair(__uint_as_float(hi[j] << 16), __uint_as_float(hi[j] & 0xffff0000u)), pair(-1.f, -1.f), w), ra, rb);
          lo[j] = bf2(ra, rb);
        }
        fence_before();  // (the other warp's scores may lie where this one's weights go: both have read theirs now)
        if (either(top > m + kGrowth) && !raise) {
          raise = true;
          continue;
        }
        fence_after();
        tmem_st(tile + col0 / 2, hi);
        tmem_st(tile + kLow + col0 / 2, lo);
        break;
      }
      float s0, s1;
      unpair(add2(sum[0], sum[1]), s0, s1);
      l += s0 + s1;
      tmem_st_wait();
      fence_before();
      __syncwarp();
      if (lane == 0) bar_arrive(p_ready + 8 * (it & 1));
    }
    swap[half * kM + r_own] = l;
    meet();
    l += swap[(half ^ 1) * kM + r_own];
    Values::at_end(n, value);
    if (ok) {
      fence_after();
      const float f = __fdiv_rn(1.0f, l) * (spec.head_gate && row < T ? head_sigmoid(p.in[(size_t)row * p.in_ld + spec.gate_row0() + h]) : 1.0f);
      __nv_bfloat16* const out = reinterpret_cast<__nv_bfloat16*>(p.ao) + (size_t)row * spec.out_cols() + (size_t)h * D;
#pragma unroll 1
      for (uint32_t c = half * (D / 2); c < (half + 1) * (D / 2); c += 32) {
        uint32_t o[32];
        tmem_ld(lanes + kO + c, o);
        if (row >= T) continue;
#pragma unroll
        for (int e = 0; e < 32; e += 8) {
          uint4 v;
          v.x = bf2(__uint_as_float(o[e]) * f, __uint_as_float(o[e + 1]) * f);
          v.y = bf2(__uint_as_float(o[e + 2]) * f, __uint_as_float(o[e + 3]) * f);
          v.z = bf2(__uint_as_float(o[e + 4]) * f, __uint_as_float(o[e + 5]) * f);
          v.w = bf2(__uint_as_float(o[e + 6]) * f, __uint_as_float(o[e + 7]) * f);
          *reinterpret_cast<uint4*>(out + c + e) = v;
        }
      }
    }
  }
  if (!ok) {
    if (lane == 0 && p.state) atomicOr(&p.state->err, 4u);
    // copies and products of this CTA may still be in flight: a bounded time for them to end before their memory is released
    for (volatile uint32_t spin = 0; spin < (1u << 20); ++spin) {
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
}

template <int D>
cudaError_t launch_umma(cudaStream_t s, const GqaParams& p, uint32_t T) {
  CUtensorMap mapQ, mapK, mapV;  // rows beyond the pass come as zeros: its own maps
  const uint64_t rows = (uint64_t)p.pos0 + T;
  if (!encode_tile_map16(&mapQ, p.q, T, p.spec.q_rows(), kM) || !encode_tile_map16(&mapK, p.k_cache, rows, p.spec.k_cols(), kN) ||
      !encode_tile_map16(&mapV, p.v_cache, rows, p.spec.v_cols(), kN))
    return cudaErrorInvalidValue;
  const cudaError_t e = cudaFuncSetAttribute(gqa_prefill_umma_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Smem<D>::kTotal);
  if (e != cudaSuccess) return e;
  const uint64_t grid = (uint64_t)((T + kM - 1) / kM) * p.spec.heads;
  if (grid > 0x7fffffffu) return cudaErrorInvalidValue;
  return launch_pdl(gqa_prefill_umma_kernel<D>, dim3((unsigned)grid), dim3(kThreads), Smem<D>::kTotal, s, prefill_pdl(), mapQ, mapK, mapV, p, T);
}

}  // namespace

// From 64 tokens on (ms, the warp-level kernel and this one: 64 tokens 2.134 and 2.105, 128: 2.260 and 2.254, 256: 2.445 and 2.454); half a
// tile of rows or less is work for the former.
bool gqa_prefill_umma_supported(const GqaParams& p, uint32_t T) {
  const GqaSpec& s = p.spec;
  if (p.dtype != 2 || s.dim != s.vdim || (s.dim != 64 && s.dim != 128)) return false;
  if ((((uintptr_t)p.q | (uintptr_t)p.k_cache | (uintptr_t)p.v_cache | (uintptr_t)p.ao) & 15) != 0) return false;
  return T >= 64;
}

cudaError_t launch_gqa_prefill_umma(cudaStream_t s, const GqaParams& p, uint32_t T) {
  return p.spec.dim == 64 ? launch_umma<64>(s, p, T) : launch_umma<128>(s, p, T);
}

}  // namespace nfai
