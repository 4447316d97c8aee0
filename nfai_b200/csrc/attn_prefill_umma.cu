// Causal attention over a chunk of prompt tokens on the 5th-generation tensor cores: float16 caches, heads of 64 or 128.
//
// The query heads of a KV group and the tokens are packed into one list of rows (row = token * G + head of the group); a CTA
// owns 128 of them, one accumulator lane each, and walks the cache in tiles of 128 positions:
//   warp 8   K and V tiles by TMA into a ring of 128-byte swizzled slots, in the order in which they are multiplied
//   warp 9   one lane issues S = Q K^T (both operands in shared memory) and O += P V (P in tensor memory, V as it lies in the
//            cache: its rows run along N); accumulators in tensor memory
//   warps 0-7  softmax, two threads to a row (64 positions each): they read S, write the weights back as the float16 operand of
//            the second product and keep their float32 sums; at the end they divide and store half a row of O each
// Exponentials and what goes with them, not the products (28 % of the time at d = 64), are what bounds it: two CTAs share an
// SM, 256 columns of tensor memory each, so that the exponentials of one run beside the products and waits of the other, four
// warps to a scheduler (one thread to a row, two warps to a scheduler, left 52 % of the issue slots idle: 763 us against 742 for
// 2048 tokens behind 28000, 32 heads of 64). With d = 64 there are columns left for the weights beside the scores: the next
// tile's scores are multiplied while this tile's exponentials run.
//
// A row's sums are rescaled only when its maximum has grown by more than 8 (base 2) since the last time: weights are then at
// most 2^8, far inside float16, and their relative rounding is what it was. The first tile sets the maximum.
// Precision as in attn_prefill_tc.cu: q (scaled) and weights rounded to float16 for the products, everything else float32.
//
// Against the warp-level kernel of attn_prefill_tc.cu (us): 2011 tokens, 32 heads of 64: 37 against 68; 24 heads of 128: 48
// against 98 (46 with elected issue); 2048 behind 28000, 32 heads of 64: 732 against 1783 (665 TFLOP/s); 9472 behind 18944: 2317
// against 5771 (793).
//
// Reference arithmetic replaced: AttentionScoreCalculationShader.cs:170-205, AttentionSoftmaxShader.cs:145-177,
// AttentionWeightedValueSumShader.cs:181-215, applied once per prompt token by LlamaModel.cs:103-126.
#include "attn_core.cuh"
#include "attn_phases.h"
#include "umma.cuh"

namespace nfai {

namespace {

using namespace umma;

constexpr uint32_t kUM = 128;        // rows (token, head of the group) per CTA
constexpr uint32_t kUN = 128;        // positions per tile
constexpr int kUThreads = 320;
constexpr float kGrowth = 8.0f;      // growth of a maximum (base 2) that the sums are carried through without rescaling
using Values = ValuePhases<1>;       // the barrier of the products with the values

// A row's sum, or a NaN where no weights add up to it: beyond any sum of them (2^kGrowth each) one of the scores was not a number;
// below `least` (the whole row's has the 1 of its maximum) all were -infinity, and only the polynomial's 2^-126 are in it.
__device__ __forceinline__ float known_sum(float l, float least) { return l >= least && l < 1e30f ? l : __uint_as_float(0x7fffffffu); }

// Pairs of every eight whose exponentials go to the multiply-add units instead of the special function unit. Measured at 2048
// tokens behind 28000 (d = 64, 32 heads): 0: 774 us, 1: 742, 2: 749, 3: 806, 4: 861; d = 128, 1024 behind 1024: 49.0, 48.8, 48.5,
// 50.0, 51.9 us: the issue slots that the polynomial takes soon cost more than the special function unit is relieved of.
constexpr int kPoly = 1;

template <int D>
struct USmem {
  static constexpr uint32_t kTile = kUN * D * 2;             // a K or a V tile: D / 64 blocks of [128][64]
  static constexpr uint32_t kSlots = D == 64 ? 5 : 2;        // two CTAs on an SM
  static constexpr uint32_t kQ = kUM * D * 2;
  static constexpr uint32_t kBarOff = kQ + kSlots * kTile;
  static constexpr uint32_t kSwapOff = kBarOff + 256;        // two floats per row: maxima of its halves, later their sums
  static constexpr uint32_t kTotal = kSwapOff + 2 * kUM * 4 + 1024;
};

__device__ __forceinline__ float u_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t u_half2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// 2^x of a pair on the fused multiply-add units, for x below 128: x = n + f with n whole and |f| <= 1/2 (adding 1.5 * 2^23 rounds),
// 2^f by its minimax polynomial of degree 5 (a linear program over the relative error; 2.1e-7 in float32, as much as the
// hardware's approximation is allowed), n added to the exponent. Anything below 2^-126 becomes that; a NaN becomes the largest
// finite number, which shows in the row's sum (known_sum; multiplying 2^n on would keep it one, but took 2392 us for 2378 at 9472 tokens
// behind 18944, 47.0 for 46.2 at 2011 tokens of 24 heads of 128, looking at each tile's sum as much; this takes nothing).
__device__ __forceinline__ void poly_ex2(uint64_t x2, float& a, float& b) {
  float x0, x1;
  unpair(x2, x0, x1);
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x0) : "f"(-126.f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x1) : "f"(-126.f));
  const float magic = 12582912.f;
  const uint64_t x = pair(x0, x1), t = add2(x, pair(magic, magic)), n = add2(t, pair(-magic, -magic)), f = fma2(n, pair(-1.f, -1.f), x);
  uint64_t q = pair(1.327646430581808e-3f, 1.327646430581808e-3f);
  q = fma2(q, f, pair(9.675540961325169e-3f, 9.675540961325169e-3f));
  q = fma2(q, f, pair(5.550713464617729e-2f, 5.550713464617729e-2f));
  q = fma2(q, f, pair(2.4022120237350464e-1f, 2.4022120237350464e-1f));
  q = fma2(q, f, pair(6.931469440460205e-1f, 6.931469440460205e-1f));
  q = fma2(q, f, pair(1.0000001192092896f, 1.0000001192092896f));
  float q0, q1, t0, t1;
  unpair(q, q0, q1);
  unpair(t, t0, t1);
  a = __uint_as_float((__float_as_uint(t0) << 23) + __float_as_uint(q0));
  b = __uint_as_float((__float_as_uint(t1) << 23) + __float_as_uint(q1));
}

template <int D>
__global__ void __launch_bounds__(kUThreads, 2) attn_prefill_umma_kernel(const __grid_constant__ CUtensorMap mapK,
                                                                         const __grid_constant__ CUtensorMap mapV, const AttnParams p,
                                                                         const uint32_t T, uint32_t* err) {
  using SM = USmem<D>;
  constexpr uint32_t kS = 0, kP = D == 64 ? 128 : 0, kO = D == 64 ? 192 : 128;  // columns of tensor memory
  constexpr bool kAhead = D == 64;  // scores of the next tile beside the weights of this one
  extern __shared__ unsigned char um_raw[];
  unsigned char* const sm = reinterpret_cast<unsigned char*>(((uintptr_t)um_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(sm + SM::kBarOff);
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * SM::kSlots + 5);
  const uint32_t full0 = s_u32(bars), empty0 = s_u32(bars + SM::kSlots), q_ready = s_u32(bars + 2 * SM::kSlots), s_ready = q_ready + 8,
                 s_free = q_ready + 16, p_ready = q_ready + 24, pv_done = q_ready + 32;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;  // (warp: uniform)
  if (tid == 0) {
    for (uint32_t i = 0; i < SM::kSlots; ++i) {
      bar_init(full0 + 8 * i, 1);
      bar_init(empty0 + 8 * i, 1);
    }
    bar_init(q_ready, 8);
    bar_init(s_ready, 1);
    bar_init(s_free, 8);
    bar_init(p_ready, 8);
    bar_init(pv_done, 1);
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
  pdl_wait();  // q and the chunk's cache rows come from the QKV GEMM launched just before

  // the longest walks start first
  const uint32_t G = p.qH / p.kvH, g = blockIdx.x % p.kvH, tile = gridDim.x / p.kvH - 1 - blockIdx.x / p.kvH;
  const uint32_t row0 = tile * kUM, p0 = p.seq_imm - 1;
  const uint32_t last_token = min(T, (row0 + kUM - 1) / G + 1) - 1;
  const uint32_t n = (p0 + last_token) / kUN + 1;  // tiles
  bool ok = true;

  if (warp == 8) {
    uint32_t j = 0;
    auto load = [&](const CUtensorMap* map, uint32_t it) {
      const uint32_t s = j % SM::kSlots;
      if (j >= SM::kSlots && !warp_wait(empty0 + 8 * s, (j / SM::kSlots - 1) & 1)) return ok = false;
      if (elect_one()) {
        bar_expect_tx(full0 + 8 * s, SM::kTile);
#pragma unroll
        for (uint32_t b = 0; b < D / 64; ++b)
          tma_load_2d(s_u32(sm) + SM::kQ + s * SM::kTile + b * (kUN * 128), map, (int)(g * D + b * 64), (int)(it * kUN), full0 + 8 * s);
      }
      ++j;
      return true;
    };
    if constexpr (kAhead) {
      load(&mapK, 0);
      for (uint32_t it = 0; it < n && ok; ++it) {
        if (it + 1 < n && !load(&mapK, it + 1)) break;
        if (!load(&mapV, it)) break;
      }
    } else {
      for (uint32_t it = 0; it < n && ok; ++it)
        if (!load(&mapK, it) || !load(&mapV, it)) break;
    }
    if (ok) ok = drain_ring<SM::kSlots>(empty0, j);
  } else if (warp == 9) {
    // float16 operands, float32 sums; A along K in both products; B along K (K tile) or along N (V tile)
    constexpr uint32_t idesc_s = (1u << 4) | ((kUN >> 3) << 17) | ((kUM >> 4) << 24);
    constexpr uint32_t idesc_o = (1u << 4) | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((kUM >> 4) << 24);
    const uint32_t q_s = s_u32(sm);
    uint32_t j = 0;
    auto slot = [&](uint32_t& s) {  // wait for the next tile
      s = j % SM::kSlots;
      ok = warp_wait(full0 + 8 * s, (j / SM::kSlots) & 1);
      fence_after();
      ++j;
      return ok;
    };
    auto scores = [&]() {
      uint32_t s;
      if (!slot(s)) return false;
      if (elect_one()) {
        const uint32_t k_s = q_s + SM::kQ + s * SM::kTile;
#pragma unroll
        for (uint32_t kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk >> 2) * (kUM * 128) + (kk & 3) * 32;
          umma_f16(tmem + kS, smem_desc_sw128(q_s + off), smem_desc_sw128(k_s + off), idesc_s, kk != 0);
        }
        umma_commit(empty0 + 8 * s);
        umma_commit(s_ready);
      }
      return true;
    };
    ok = warp_wait(q_ready, 0);
    fence_after();
    if (ok) scores();
    for (uint32_t it = 0; it < n && ok; ++it) {
      if (kAhead && it + 1 < n) {
        if (!(ok = warp_wait(s_free, it & 1))) break;
        fence_after();
        if (!scores()) break;
      }
      if (!(ok = warp_wait(p_ready, it & 1))) break;
      fence_after();
      uint32_t s;
      if (!slot(s)) break;
      if (elect_one()) {
        const uint32_t v_s = q_s + SM::kQ + s * SM::kTile;
#pragma unroll
        for (uint32_t kk = 0; kk < kUN / 16; ++kk)
          umma_f16_ta(tmem + kO, tmem + kP + kk * 8, smem_desc_mn_sw128(v_s + kk * 2048, kUN * 128), idesc_o, (it | kk) != 0);
        umma_commit(empty0 + 8 * s);
        umma_commit(pv_done);
      }
      // (the weights lie where the next scores go: products of one thread run in their order)
      if (!kAhead && it + 1 < n && !scores()) break;
    }
  } else {
    const uint32_t qDim = p.qH * D;
    {  // the rows of Q, scaled into the base-2 domain
      const float qscale = (1.0f / sqrtf((float)D)) * 1.4426950408889634f;
      constexpr uint32_t kLanes = D / 4, kRows = 32 / kLanes;
      const uint32_t c = (lane % kLanes) * 4;
#pragma unroll 8
      for (uint32_t i = 0; i < 16; i += kRows) {
        const uint32_t r = warp * 16 + i + lane / kLanes, token = (row0 + r) / G, h = g * G + (row0 + r) % G;
        const float4 v = token < T ? __ldcg(reinterpret_cast<const float4*>(p.q + (size_t)token * qDim + h * D + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<uint2*>(sm + (c >> 6) * (kUM * 128) + r * 128 + ((((c & 63) >> 3) ^ (r & 7)) << 4) + (c & 7) * 2) =
            make_uint2(u_half2(v.x * qscale, v.y * qscale), u_half2(v.z * qscale, v.w * qscale));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(q_ready);
    }
    const uint32_t quarter = warp & 3, half = warp >> 2, col0 = half * (kUN / 2), r_own = quarter * 32 + lane;
    const uint32_t row = row0 + r_own, token = row / G;
    const uint32_t limit = p0 + min(token, T - 1);                        // last position this row sees
    const uint32_t w_first = p0 + min((row0 + quarter * 32) / G, T - 1);  // ... and the warp's first row
    const uint32_t lanes = tmem + (quarter * 32u << 16);
    float* const swap = reinterpret_cast<float*>(sm + SM::kSwapOff);      // [2][kUM]
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
      ok = __all_sync(0xffffffffu, ok && bar_wait(pv_done, Values::parity(j)));
    };
    float m = 0.f, l = 0.f;
    for (uint32_t it = 0; it < n; ++it) {
      ok = __all_sync(0xffffffffu, ok && bar_wait(s_ready, it & 1));  // (a warp that gave up still meets the other one)
      if (!kAhead) Values::at_tile(it, value);
      const uint32_t n0 = it * kUN + col0;
      // The weights are formed from the maximum as it stands; a row that turns out to have grown too far (the first tile always
      // has) makes its two warps raise their maxima and do the tile again.
      uint64_t sum[2];
      bool raise = it == 0;
      for (;;) {
        uint32_t s[kUN / 2];
        fence_after();
        tmem_ld(lanes + kS + col0, s);
        if (n0 + kUN / 2 - 1 > w_first) {  // (causal: nothing of the earlier tiles is hidden from any row)
#pragma unroll
          for (uint32_t j = 0; j < kUN / 2; ++j)
            if (n0 + j > limit) s[j] = 0xff800000u;
        }
        float t[4] = {__uint_as_float(s[0]), __uint_as_float(s[1]), __uint_as_float(s[2]), __uint_as_float(s[3])};
#pragma unroll
        for (uint32_t j = 4; j < kUN / 2; j += 8)
#pragma unroll
          for (uint32_t i = 0; i < 4; ++i)
            t[i] = j + 4 + i < kUN / 2 ? fmaxf(fmaxf(t[i], __uint_as_float(s[j + i])), __uint_as_float(s[j + 4 + i])) : fmaxf(t[i], __uint_as_float(s[j + i]));
        float top = fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3]));
        if (raise) {
          swap[half * kUM + r_own] = top;
          meet();
          top = fmaxf(fmaxf(top, swap[(half ^ 1) * kUM + r_own]), it ? m : attn_detail::kNegBig);
          if (it) {
            Values::at_rescaling(it, value);
            fence_after();
            const float f = u_ex2(m - top);
            l = known_sum(l, 0.f) * f;
#pragma unroll 1
            for (uint32_t c = half * (D / 2); c < (half + 1) * (D / 2); c += 16) {
              uint32_t o[16];
              tmem_ld(lanes + kO + c, o);
#pragma unroll
              for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
              tmem_st(lanes + kO + c, o);
            }
          }
          m = top;
        }
        sum[0] = sum[1] = 0;
        const uint64_t minus_m = pair(-m, -m);
        uint32_t w[2][16];
        auto weights = [&](uint32_t c) {
#pragma unroll
          for (uint32_t j = 0; j < 16; ++j) {
            const uint64_t x = add2(pair(__uint_as_float(s[c * 32 + 2 * j]), __uint_as_float(s[c * 32 + 2 * j + 1])), minus_m);
            float a, b;
            if ((int)(j & 7) < kPoly) {
              poly_ex2(x, a, b);
            } else {
              unpair(x, a, b);
              a = u_ex2(a);
              b = u_ex2(b);
            }
            sum[j & 1] = add2(sum[j & 1], pair(a, b));
            w[c][j] = u_half2(a, b);
          }
        };
        weights(0);
        if (!kAhead) fence_before();  // (the other warp's scores may lie where this one's weights go: both have read theirs now)
        if (either(top > m + kGrowth) && !raise) {
          raise = true;
          continue;
        }
        if (!kAhead) fence_after();
        if (kAhead) {
          fence_before();
          __syncwarp();
          if (lane == 0) bar_arrive(s_free);
          Values::at_tile(it, value);  // the weights of the tile before have been used
          fence_after();
        }
        tmem_st(lanes + kP + col0 / 2, w[0]);
        weights(1);
        tmem_st(lanes + kP + col0 / 2 + 16, w[1]);
        break;
      }
      float s0, s1;
      unpair(add2(sum[0], sum[1]), s0, s1);
      l += s0 + s1;
      tmem_st_wait();
      fence_before();
      __syncwarp();
      if (lane == 0) bar_arrive(p_ready);
    }
    swap[half * kUM + r_own] = l;
    meet();
    l += swap[(half ^ 1) * kUM + r_own];
    Values::at_end(n, value);
    if (ok) {
      fence_after();
      const float inv = 1.0f / known_sum(l, 0.5f);
      __half* const out = p.out_half + (size_t)token * qDim + (size_t)(g * G + row % G) * D;
#pragma unroll 1
      for (uint32_t c = half * (D / 2); c < (half + 1) * (D / 2); c += 32) {
        uint32_t o[32];
        tmem_ld(lanes + kO + c, o);
        if (token >= T) continue;
#pragma unroll
        for (int e = 0; e < 32; e += 8) {
          uint4 v;
          v.x = u_half2(__uint_as_float(o[e]) * inv, __uint_as_float(o[e + 1]) * inv);
          v.y = u_half2(__uint_as_float(o[e + 2]) * inv, __uint_as_float(o[e + 3]) * inv);
          v.z = u_half2(__uint_as_float(o[e + 4]) * inv, __uint_as_float(o[e + 5]) * inv);
          v.w = u_half2(__uint_as_float(o[e + 6]) * inv, __uint_as_float(o[e + 7]) * inv);
          *reinterpret_cast<uint4*>(out + c + e) = v;
        }
      }
    }
  }
  if (!ok) {
    if (lane == 0 && err) atomicOr(err, 4u);
    // copies and products of this CTA may still be in flight: a bounded time for them to end before their memory is released
    for (volatile uint32_t spin = 0; spin < (1u << 20); ++spin) {
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
}

template <int D>
cudaError_t launch_umma(cudaStream_t s, const AttnParams& p, uint32_t T, uint32_t* err) {
  CUtensorMap mapK, mapV;
  // Rows beyond the chunk come as zeros, so a map is one pass's own: it is not kept (two per layer and pass would in time push
  // those of the weights out).
  const uint64_t rows = (uint64_t)p.seq_imm - 1 + T, width = (uint64_t)p.kvH * D;
  if (!encode_tile_map16(&mapK, p.kcache, rows, width, kUN) || !encode_tile_map16(&mapV, p.vcache, rows, width, kUN)) return cudaErrorInvalidValue;
  static thread_local int attr_device = -1;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (attr_device != dev) {
    e = cudaFuncSetAttribute(attn_prefill_umma_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)USmem<D>::kTotal);
    if (e != cudaSuccess) return e;
    attr_device = dev;
  }
  const uint64_t rows_q = (uint64_t)T * (p.qH / p.kvH), grid = (rows_q + kUM - 1) / kUM * p.kvH;
  if (grid > 0x7fffffffu) return cudaErrorInvalidValue;
  return launch_pdl(attn_prefill_umma_kernel<D>, dim3((unsigned)grid), dim3(kUThreads), USmem<D>::kTotal, s, prefill_pdl(), mapK, mapV, p, T, err);
}

}  // namespace

// The line to the warp-level kernel. A short walk is a few tiles, and the set-up of tensor memory and barriers counts as much:
// with few rows (tokens times heads) up to 320 positions belong to the warp-level kernel (us, there and here: 64 tokens, 32 heads of
// 64: 313 positions 8.9 and 9.4, 321: 9.4 and 8.9; 37 tokens, 24 heads of 128: 307: 11.5 and 13.1, 321: 13.0 and 13.2, 449: 16.7 and
// 14.9; 37 of 32 heads of 64 at 640: 14.1 and 11.2). From 6144 rows on, heads of 64 fill that kernel's SMs more than once: 192
// tokens of 32 heads at 257: 11.6 and 9.5 (160 tokens at 289: 9.4 and 10.1). Heads of 128 have one CTA of it on an SM and a tile of
// 128 positions here costs them most where there are many: 300 tokens of 24 heads at 321: 13.3 and 14.8, 384 at 448: 16.5 and 17.1,
// 449: 18.1 and 17.2.
bool attn_prefill_umma_supported(int kvdtype, const AttnParams& p, uint32_t T) {
  if (kvdtype != 1 || (p.d != 64 && p.d != 128)) return false;
  if ((((uintptr_t)p.kcache | (uintptr_t)p.vcache | (uintptr_t)p.q | (uintptr_t)p.out_half) & 15) != 0) return false;
  const uint64_t rows = (uint64_t)T * p.qH;
  const uint32_t short_walk = p.d == 64 ? (rows < 6144 ? 320 : 256) : (rows <= 4096 ? 320 : 448);
  return (uint64_t)p.seq_imm - 1 + T > short_walk;
}

cudaError_t launch_attn_prefill_umma(cudaStream_t s, const AttnParams& p, uint32_t T, uint32_t* err) {
  if (p.qH == 0 || p.kvH == 0 || p.qH % p.kvH != 0 || !p.out_half || !p.seq_imm || !T) return cudaErrorInvalidValue;
  return p.d == 64 ? launch_umma<64>(s, p, T, err) : p.d == 128 ? launch_umma<128>(s, p, T, err) : cudaErrorInvalidValue;
}

}  // namespace nfai
