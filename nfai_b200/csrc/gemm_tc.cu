// Prompt-ingestion GEMM on the 5th-generation tensor cores: C[M][N] = A[M][K] * W[N][K]^T, A and W float16 with K
// contiguous, float32 accumulation in tensor memory. M = prompt tokens of a chunk, N = output features.
//
// The reference has no batched prompt path (it pushes prompt tokens through the single-token shaders one by one:
// NFAI.Models.Llama3/LlamaModel.cs:103-126); results must equal that token-by-token evaluation within the FP16
// tolerance, so the fused epilogues below are the same ones the decode GEMVs use (RoPE + cache write, SiLU*up,
// residual add) applied row by row.
//
// Shape of one CTA (320 threads, one 128 x BN output tile):
//   warp 0      producer: the warp waits for a free stage, an elected lane issues the TMA tile loads (A 128x64, W BNx64
//               halves, 128-byte swizzle), completion counted on the stage's "full" mbarrier; at the end the warp waits
//               for the last stages to be free again;
//   warp 1      MMA: allocates BN tensor-memory columns; the warp waits for a full stage, an elected lane issues four
//               tcgen05.mma (K = 16 each) from shared-memory descriptors and commits to the stage's "empty" mbarrier so
//               that the producer may refill it, after the last stage also to "accumulator ready";
//   warps 2-9   epilogue: two for each quarter of the accumulator's rows (a warp may only read the lanes of its index modulo 4),
//               taking its column blocks in turn.
// K is split over several CTAs where the tiles alone leave SMs idle: they are a cluster and add up through each other's shared
// memory, or, where too few clusters run at once, through memory and a second kernel. Larger products go to pairs of CTAs, rows
// in groups to 128 x 256 tiles (both below). No tile copy is delivered to more than one CTA. Every mbarrier wait is bounded (one
// second): on a time-out the role records an error bit and leaves; the tensor memory is released on every path.
#include <cuda.h>

#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "gemm_tc.h"
#include "kernels.h"
#include "umma.cuh"

#include <stdlib.h>

#include <functional>
#include <type_traits>
#include <unordered_map>

namespace nfai {

namespace {

using namespace umma;

constexpr int kBM = 128;
constexpr int kBK = 64;  // halves per stage row = 128 bytes = one swizzle span
constexpr int kGemmThreads = 64 + 8 * 32;
constexpr uint32_t kEpiWarp = 32 * 32 * 4;  // an epilogue warp's shared memory

// ---- epilogue of an accumulator tile ------------------------------------------------------------------------------
// tcgen05.ld hands every lane one accumulator row; the output wants lanes along a row. A 32 x 32 block goes through 4 KB of
// shared memory in 16-byte quads (quad j of row r lies at place j ^ (r & 7): neither side conflicts) and comes back with 8 lanes
// on the 32 columns of a row, 4 rows per instruction, all of it in registers before the first store: 8 wide loads and stores per
// lane and block. Stores of single columns or pairs from the accumulator's layout touched 32 rows per instruction: 256 x 2048 at
// K = 64 took 8.0 us, now 3.6; 128 x 16384 x 2048 (67 MB of weights) 34, now 17.4 (19.5 with gates; 18.2 and 22.8 with four warps).

// Whether every quad of columns that lies below N can be read and written in one piece
template <int KIND>
__device__ __forceinline__ bool quads_fit(const GemmEpilogue& ep, uint32_t N) {
  auto aligned = [](const void* p, uint32_t bytes) { return ((uintptr_t)p & (bytes - 1)) == 0; };
  if (N & 3u) return false;
  const uint32_t act_bytes = ep.out_dtype == 0 ? 4 : 2;
  if constexpr (KIND == GEMM_EPI_STORE) return aligned(ep.out_f32, 16) && aligned(ep.resid, 16) && aligned(ep.bias, 16);
  if constexpr (KIND == GEMM_EPI_GATED) return aligned(ep.out_act, 2 * act_bytes) && aligned(ep.bias, 16);
  if constexpr (KIND == GEMM_EPI_GATED_CLAMPED) return (ep.gated_cols & 3u) == 0 && aligned(ep.out_act, 2 * act_bytes) && aligned(ep.out_f32, 16);
  if constexpr (KIND == GEMM_EPI_STORE_ACT) return aligned(ep.out_act, 4 * act_bytes) && aligned(ep.bias, 16);
  const uint32_t row = ep.kv_f16 ? 8 : 16;
  return ((ep.qDim | ep.kvDim | ep.d | ep.ropeDim) & 3u) == 0 && aligned(ep.out_f32, 16) && aligned(ep.kcache, row) && aligned(ep.vcache, row) &&
         aligned(ep.rope_cs, 16);
}
// two consecutive activations at element `at`, in their type
__device__ __forceinline__ void store_acts2(const GemmEpilogue& ep, size_t at, float a, float b) {
  if (ep.out_dtype == 1) *reinterpret_cast<__half2*>(reinterpret_cast<__half*>(ep.out_act) + at) = __floats2half2_rn(a, b);
  else if (ep.out_dtype == 2) *reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<__nv_bfloat16*>(ep.out_act) + at) = __floats2bfloat162_rn(a, b);
  else *reinterpret_cast<float2*>(reinterpret_cast<float*>(ep.out_act) + at) = make_float2(a, b);
}
__device__ __forceinline__ uint2 half_quad(const float4& v) {
  const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
__device__ __forceinline__ uint2 bf16_quad(const float4& v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

// One warp's share of a tile: columns from `acc` of tensor memory, rows [m0, M) of the output, the quarter lane_grp of the
// lanes, column blocks c_first, c_first + c_step, ... of `blocks`, 32 columns each, from n0; eb is its 4 KB of shared memory.
// What the epilogue reads besides the sums (residual, (cos, sin) pairs) is fetched a block ahead, first before the wait for the
// accumulator.
template <int KIND>
__device__ __forceinline__ bool tile_epilogue(const GemmEpilogue& ep, const uint32_t m0, const uint32_t M, const uint32_t n0, const uint32_t N,
                                              const int blocks, const uint32_t acc, const uint32_t lane_grp, const int c_first, const int c_step,
                                              const int lane, const uint32_t eb, const uint32_t tfull, const uint32_t parity) {
  constexpr bool kRope = KIND == GEMM_EPI_QKV_ROPE, kRows = KIND == GEMM_EPI_STORE || kRope;  // kRows: reads something per row
  const uint32_t quad = lane & 7, mrow = m0 + lane_grp * 32 + (lane >> 3);                     // rows mrow, mrow + 4, ... of the block
  const bool fit = quads_fit<KIND>(ep, N);
  float4 aux[8];
  // everything about a quad of Q/K/V that depends on the column only: which of Q, K, V; its place there; whether it is rotated
  struct Place {
    uint32_t seg, local, e;
    bool rot;
  };
  auto place = [&](uint32_t n) {
    Place c;
    c.seg = n < ep.qDim ? 0u : n < ep.qDim + ep.kvDim ? 1u : 2u;
    c.local = n - (c.seg == 0 ? 0u : c.seg == 1 ? ep.qDim : ep.qDim + ep.kvDim);
    c.e = c.local & (ep.d - 1);  // head dimensions are powers of two (32, 64, 128)
    c.rot = c.seg < 2 && c.e < ep.ropeDim;
    return c;
  };
  auto load_aux = [&](int b) {
    const uint32_t n = n0 + b * 32 + quad * 4;
    if constexpr (kRope) {
      const Place c = place(n);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        aux[i] = c.rot && n < N && mrow + 4 * i < M
                     ? __ldg(reinterpret_cast<const float4*>(ep.rope_cs + (size_t)(ep.pos0 + mrow + 4 * i) * (ep.ropeDim / 2) + (c.e >> 1)))
                     : make_float4(1.f, 0.f, 1.f, 0.f);
    } else {
      const float4 bias = ep.bias && n < N ? __ldg(reinterpret_cast<const float4*>(ep.bias + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ep.resid && n < N && mrow + 4 * i < M) r = __ldcg(reinterpret_cast<const float4*>(ep.resid + (size_t)(mrow + 4 * i) * N + n));
        aux[i] = make_float4(r.x + bias.x, r.y + bias.y, r.z + bias.z, r.w + bias.w);
      }
    }
  };
  if (kRows && fit && c_first < blocks) load_aux(c_first);
  bool good = bar_wait(tfull, parity);
  good = __all_sync(0xffffffffu, good);
  if (!good) return false;
  fence_after();
#pragma unroll 1
  for (int b = c_first; b < blocks; b += c_step) {
    const uint32_t nb = n0 + b * 32, n = nb + quad * 4;
    float4 x[8];
    {
      uint32_t v[32];
      tmem_ld(acc + ((lane_grp * 32u) << 16) + (uint32_t)b * 32u, v);
      if (m0 + lane_grp * 32 >= M || nb >= N) continue;  // (warp-uniform)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(eb + lane * 128 + ((j ^ (lane & 7)) << 4)), "r"(v[4 * j]), "r"(v[4 * j + 1]),
                     "r"(v[4 * j + 2]), "r"(v[4 * j + 3])
                     : "memory");
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t r = (lane >> 3) + 4 * i;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(x[i].x), "=f"(x[i].y), "=f"(x[i].z), "=f"(x[i].w)
                     : "r"(eb + r * 128 + ((quad ^ (r & 7)) << 4))
                     : "memory");
      }
      __syncwarp();
    }
    if (!fit) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t m = mrow + 4 * i;
        if (m >= M || n >= N) continue;
        epilogue_pair<KIND>(ep, m, n, N, x[i].x, x[i].y, epilogue_aux<KIND>(ep, m, n, N));
        if (n + 2 < N) epilogue_pair<KIND>(ep, m, n + 2, N, x[i].z, x[i].w, epilogue_aux<KIND>(ep, m, n + 2, N));
      }
      continue;
    }
    if constexpr (KIND == GEMM_EPI_STORE) {
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = make_float4(aux[i].x + x[i].x, aux[i].y + x[i].y, aux[i].z + x[i].z, aux[i].w + x[i].w);
    } else if constexpr (kRope) {
      if (n < N && place(n).rot) {  // value1 = cos*a - sin*b ; value2 = sin*a + cos*b, products rounded separately
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 cs = aux[i], v = x[i];
          x[i].x = __fsub_rn(__fmul_rn(cs.x, v.x), __fmul_rn(cs.y, v.y));
          x[i].y = __fadd_rn(__fmul_rn(cs.y, v.x), __fmul_rn(cs.x, v.y));
          x[i].z = __fsub_rn(__fmul_rn(cs.z, v.z), __fmul_rn(cs.w, v.w));
          x[i].w = __fadd_rn(__fmul_rn(cs.w, v.z), __fmul_rn(cs.z, v.w));
        }
      }
    }
    if constexpr (kRows) {
      if (b + c_step < blocks) load_aux(b + c_step);  // in flight during this block's stores
    }
    if (n >= N) continue;
    const int rows = mrow < M ? min(8u, (M - mrow + 3) / 4) : 0;  // of this lane's eight
    if constexpr (KIND == GEMM_EPI_STORE) {
      float* const out = ep.out_f32 + (size_t)mrow * N + n;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < rows) *reinterpret_cast<float4*>(out + (size_t)(4 * i) * N) = x[i];
    } else if constexpr (kRope) {
      const Place c = place(n);
      const size_t kv = (size_t)(ep.pos0 + mrow) * ep.kvDim + c.local;
      void* const cache = c.seg == 1 ? ep.kcache : ep.vcache;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i >= rows) continue;
        if (c.seg == 0) *reinterpret_cast<float4*>(ep.out_f32 + (size_t)(mrow + 4 * i) * ep.qDim + c.local) = x[i];
        else if (ep.kv_f16) *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(cache) + kv + (size_t)(4 * i) * ep.kvDim) = half_quad(x[i]);
        else *reinterpret_cast<float4*>(reinterpret_cast<float*>(cache) + kv + (size_t)(4 * i) * ep.kvDim) = x[i];
      }
    } else if constexpr (KIND == GEMM_EPI_GATED) {  // columns (2j, 2j+1) = (gate_j, up_j)
      const float4 bias = ep.bias ? __ldg(reinterpret_cast<const float4*>(ep.bias + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < rows)
          store_acts2(ep, (size_t)(mrow + 4 * i) * (N / 2) + (n >> 1), gated(ep.act, x[i].x + bias.x, x[i].y + bias.y),
                      gated(ep.act, x[i].z + bias.z, x[i].w + bias.w));
    } else if constexpr (KIND == GEMM_EPI_GATED_CLAMPED) {
      const uint32_t cols = ep.gated_cols ? ep.gated_cols : N;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i >= rows) continue;
        if (n < cols)
          store_acts2(ep, (size_t)(mrow + 4 * i) * (cols / 2) + (n >> 1), gated_clamped(x[i].x, x[i].y, ep.act_limit),
                      gated_clamped(x[i].z, x[i].w, ep.act_limit));
        else *reinterpret_cast<float4*>(ep.out_f32 + (size_t)(mrow + 4 * i) * (N - cols) + (n - cols)) = x[i];
      }
    } else {  // plain store in the operand type of the next product
      const float4 bias = ep.bias ? __ldg(reinterpret_cast<const float4*>(ep.bias + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i >= rows) continue;
        const float4 v = make_float4(x[i].x + bias.x, x[i].y + bias.y, x[i].z + bias.z, x[i].w + bias.w);
        const size_t at = (size_t)(mrow + 4 * i) * N + n;
        if (ep.out_dtype == 0) *reinterpret_cast<float4*>(reinterpret_cast<float*>(ep.out_act) + at) = v;
        else *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(ep.out_act) + at) = ep.out_dtype == 1 ? half_quad(v) : bf16_quad(v);
      }
    }
  }
  return true;
}

// Second kernel of a split GEMM: one thread per column pair adds the partials in split order and applies the epilogue.
__global__ void __launch_bounds__(256) gemm_finish_kernel(const float* __restrict__ part, uint32_t M, uint32_t N, uint32_t Z,
                                                          const GemmEpilogue ep) {
  pdl_launch_dependents();
  pdl_wait();  // the partial tiles come from the GEMM launched just before
  const uint32_t pairs = (N + 1) / 2;
  const size_t total = (size_t)M * pairs;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const uint32_t m = (uint32_t)(idx / pairs), n = (uint32_t)(idx % pairs) * 2;
    float a = 0.f, b = 0.f;
    for (uint32_t z = 0; z < Z; ++z) {
      const float* p = part + ((size_t)z * M + m) * N + n;
      a += p[0];
      if (n + 1 < N) b += p[1];
    }
    epilogue_pair(ep, m, n, N, a, b, epilogue_aux(ep, m, n, N));
  }
}

template <int BN, int STAGES>
struct GemmSmem {
  static constexpr uint32_t kABytes = kBM * kBK * 2;
  static constexpr uint32_t kBBytes = BN * kBK * 2;
  static constexpr uint32_t kStage = kABytes + kBBytes;
  static constexpr uint32_t kBarOff = STAGES * kStage;
  static constexpr uint32_t kEpiOff = kBarOff + 256;
  static constexpr uint32_t kTotal = kEpiOff + 8 * kEpiWarp + 1024;  // slack for the 1024-byte alignment
};

// KIND: the epilogue. A split of K over gridDim.z CTAs adds up in one of two ways. REDUCE: those CTAs are a cluster; each leaves
// its sums in its shared memory and, when all have, adds its share of the rows over the cluster (in split order) and applies the
// epilogue. Otherwise raw sums go into [split][M][N] and a finishing kernel adds them in the same order.
template <int BN, int STAGES, int KIND, bool REDUCE>
__global__ void __launch_bounds__(kGemmThreads) gemm_tc_kernel(const __grid_constant__ CUtensorMap mapA,
                                                               const __grid_constant__ CUtensorMap mapW, uint32_t M,
                                                               uint32_t N, uint32_t K, const GemmEpilogue ep,
                                                               uint32_t* err) {
  using SM = GemmSmem<BN, STAGES>;
  extern __shared__ unsigned char gsm_raw[];
  unsigned char* gsm = reinterpret_cast<unsigned char*>(((uintptr_t)gsm_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(gsm + SM::kBarOff);
  // bars[0..STAGES) full, [STAGES..2*STAGES) empty, [2*STAGES] accumulator ready; then the TMEM base address word
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);
  const uint32_t full0 = s_u32(bars), empty0 = s_u32(bars + STAGES), accbar = s_u32(bars + 2 * STAGES);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // (uniform)
  const uint32_t m0 = blockIdx.y * kBM, n0 = blockIdx.x * BN;
  // this CTA's share of the K tiles (split-K: blockIdx.z of gridDim.z; every share holds at least one tile)
  const uint32_t KT_all = (K + kBK - 1) / kBK;
  const uint32_t kt0 = (uint32_t)((uint64_t)KT_all * blockIdx.z / gridDim.z);
  const uint32_t KT = (uint32_t)((uint64_t)KT_all * (blockIdx.z + 1) / gridDim.z) - kt0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      bar_init(full0 + 8 * s, 1);
      bar_init(empty0 + 8 * s, 1);
    }
    bar_init(accbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // the MMA warp owns the tensor-memory allocation
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"((uint32_t)BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;
  // barriers and tensor memory are set up; the operands (and the residual) come from the previous kernel
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    for (uint32_t kt = 0; kt < KT; ++kt) {
      const uint32_t s = kt % STAGES;
      if (kt >= (uint32_t)STAGES) {
        if (!(ok = warp_wait(empty0 + 8 * s, ((kt / STAGES) - 1) & 1))) break;
      }
      if (elect_one()) {
        const uint32_t a_dst = s_u32(gsm + s * SM::kStage), b_dst = a_dst + SM::kABytes;
        bar_expect_tx(full0 + 8 * s, SM::kABytes + SM::kBBytes);
        tma_load_2d(a_dst, &mapA, (int)((kt0 + kt) * kBK), (int)m0, full0 + 8 * s);
        tma_load_2d(b_dst, &mapW, (int)((kt0 + kt) * kBK), (int)n0, full0 + 8 * s);
      }
    }
    if (ok) ok = drain_ring<STAGES>(empty0, KT);
  } else if (warp == 1) {
    // instruction descriptor: D float32, A and B of one 16-bit type (0 = float16, 1 = bfloat16), both K-major, N = BN, M = 128
    const uint32_t idesc = (1u << 4) | (ep.operands_bf16 << 7) | (ep.operands_bf16 << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
    for (uint32_t kt = 0; kt < KT; ++kt) {
      const uint32_t s = kt % STAGES;
      if (!(ok = warp_wait(full0 + 8 * s, (kt / STAGES) & 1))) break;
      fence_after();
      if (elect_one()) {
        const uint32_t a_s = s_u32(gsm + s * SM::kStage), b_s = a_s + SM::kABytes;
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) {
          umma_f16(tmem_base, smem_desc_sw128(a_s + k * 32), smem_desc_sw128(b_s + k * 32), idesc, (kt | (uint32_t)k) != 0);
        }
        umma_commit(empty0 + 8 * s);  // arrives when the MMAs above have finished reading the stage
        if (kt + 1 == KT) umma_commit(accbar);
      }
    }
  } else {
    // warp w may touch tensor-memory lanes 32*(w%4) .. +31
    const uint32_t lane_grp = (uint32_t)(warp & 3);
    const uint32_t eb = s_u32(gsm + SM::kEpiOff) + (warp - 2) * kEpiWarp;
    if constexpr (REDUCE) {  // quad q of row r at place q ^ r (of the row's BN / 4): neither the writes nor the reads conflict
      ok = __all_sync(0xffffffffu, bar_wait(accbar, 0));
      if (ok) {
        fence_after();
        const uint32_t r = lane_grp * 32 + lane;
#pragma unroll 1
        for (uint32_t b = (warp - 2) >> 2; b < BN / 32; b += 2) {
          uint32_t v[32];
          tmem_ld(tmem_base + ((lane_grp * 32u) << 16) + b * 32u, v);
#pragma unroll
          for (uint32_t q = 0; q < 8; ++q)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(s_u32(gsm) + r * (BN * 4) + (((b * 8 + q) ^ (r & (BN / 4 - 1))) << 4)),
                         "r"(v[4 * q]), "r"(v[4 * q + 1]), "r"(v[4 * q + 2]), "r"(v[4 * q + 3])
                         : "memory");
        }
      }
    } else if (gridDim.z > 1) {
      GemmEpilogue part;
      part.out_f32 = ep.scratch + (size_t)blockIdx.z * M * N;
      ok = tile_epilogue<GEMM_EPI_STORE>(part, m0, M, n0, N, BN / 32, tmem_base, lane_grp, (warp - 2) >> 2, 2, lane, eb, accbar, 0);
    } else {
      ok = tile_epilogue<KIND>(ep, m0, M, n0, N, BN / 32, tmem_base, lane_grp, (warp - 2) >> 2, 2, lane, eb, accbar, 0);
    }
  }
  if (!ok) {
    if (lane == 0 && err) atomicOr(err, 4u);
    // tile copies of this CTA may still be in flight: give them a bounded time to land before shared memory and
    // tensor memory are released
    for (volatile uint32_t spin = 0; spin < (1u << 20); ++spin) {
    }
  }
  if constexpr (REDUCE) {
    static_assert(BN == 128 && kBM * BN * 4 <= SM::kBarOff, "a lane for each quad, and the sums where the stages were");
    __syncwarp();
    cluster_sync();
    const uint32_t Z = gridDim.z, live = min((uint32_t)kBM, M - m0), per = (live + Z - 1) / Z;
    const uint32_t end = min(live, (blockIdx.z + 1) * per), n = n0 + lane * 4;
    for (uint32_t r = blockIdx.z * per + warp; r < end && n < N; r += kGemmThreads / 32) {
      const uint32_t m = m0 + r, at = s_u32(gsm) + r * (BN * 4) + ((lane ^ (r & 31)) << 4);
      const float2 aux0 = epilogue_aux<KIND>(ep, m, n, N), aux1 = n + 2 < N ? epilogue_aux<KIND>(ep, m, n + 2, N) : make_float2(0.f, 0.f);
      float4 part[8];
#pragma unroll
      for (uint32_t z = 0; z < 8; ++z) part[z] = z < Z ? ld_cluster(at, z) : make_float4(0.f, 0.f, 0.f, 0.f);
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (uint32_t z = 0; z < 8; ++z) x = make_float4(x.x + part[z].x, x.y + part[z].y, x.z + part[z].z, x.w + part[z].w);
      epilogue_pair<KIND>(ep, m, n, N, x.x, x.y, aux0);
      if (n + 2 < N) epilogue_pair<KIND>(ep, m, n + 2, N, x.z, x.w, aux1);
    }
    __syncwarp();
    cluster_sync();  // nobody reads the memory of a CTA that has left
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)BN) : "memory");
  }
}

// ---- rows in groups: 128 x 256 tiles, two accumulators in tensor memory -------------------------------------------
// One CTA per SM walks tiles blockIdx.x, + gridDim.x, ...; the accumulator alternates between two 256-column halves of tensor
// memory, so the epilogue of tile i (tcgen05.ld, fused epilogue, global stores) runs while the tensor pipe is on tile i + 1.
constexpr int kPBN = 256;
constexpr int kPStages = 4;
struct PSmem {
  static constexpr uint32_t kABytes = kBM * kBK * 2;
  static constexpr uint32_t kBBytes = kPBN * kBK * 2;
  static constexpr uint32_t kStage = kABytes + kBBytes;
  static constexpr uint32_t kBarOff = kPStages * kStage;
  static constexpr uint32_t kEpiOff = kBarOff + 256;
  static constexpr uint32_t kEpiBytes = 8 * kEpiWarp;
  static constexpr uint32_t kTotal = kEpiOff + kEpiBytes + 1024;
};

// Eight epilogue warps, two per quarter of the tensor-memory lanes (a warp may only read the lanes of its index modulo 4),
// each pair sharing the column blocks of its rows: with one warp per scheduler the SiLU epilogue (an exponential and
// an IEEE division per output) ran at the latency of its dependent instructions and took longer than the tile's MMAs.
constexpr int kPThreadsGemm = 64 + 8 * 32;
static_assert(PSmem::kTotal <= 227 * 1024, "shared memory of the grouped kernel");
// The tiles of rows come from a device list, each with the group whose matrix it is multiplied by; a tile may read rows of A or
// W beyond its group (they exist or are zero-filled), its epilogue stores the group's own.
template <int KIND>
__global__ void __launch_bounds__(kPThreadsGemm) gemm_tc_grouped_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapW,
                                                                       uint32_t N, uint32_t K, const GemmGroups grp, const GemmEpilogue ep,
                                                                       uint32_t* err) {
  using SM = PSmem;
  constexpr int STAGES = kPStages;
  extern __shared__ unsigned char gsm_raw[];
  unsigned char* gsm = reinterpret_cast<unsigned char*>(((uintptr_t)gsm_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(gsm + SM::kBarOff);
  // bars: [0, S) full, [S, 2S) empty, [2S, 2S+2) accumulator full, [2S+2, 2S+4) accumulator empty; then the TMEM base word
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  const uint32_t full0 = s_u32(bars), empty0 = s_u32(bars + STAGES), tfull0 = s_u32(bars + 2 * STAGES),
                 tempty0 = s_u32(bars + 2 * STAGES + 2);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // (uniform)
  const uint32_t KT = (K + kBK - 1) / kBK;
  const uint32_t ntiles = (N + kPBN - 1) / kPBN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      bar_init(full0 + 8 * s, 1);
      bar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      bar_init(tfull0 + 8 * a, 1);
      bar_init(tempty0 + 8 * a, 8);  // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;
  // barriers and tensor memory are set up; the operands (and the residual) come from the previous kernel
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t tiles = min(*grp.n_tiles, grp.max_tiles) * ntiles;
  struct Tile {
    uint32_t m0, m_end, n0, w0;  // rows [m0, m_end) of A and the output, columns from n0, rows of W from w0
  };
  auto tile_at = [&](uint32_t tile) {
    Tile t;
    // column tiles fastest: they share the rows of A, which few other tiles do
    const uint2 g = __ldcg(grp.tiles + tile / ntiles);
    t.m0 = g.y;
    t.m_end = __ldcg(grp.rows + g.x + 1);
    t.n0 = (tile % ntiles) * kPBN;
    t.w0 = g.x * N + t.n0;
    return t;
  };

  if (warp == 0) {
    uint32_t it = 0;
    for (uint32_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
      const Tile at = tile_at(tile);
      for (uint32_t kt = 0; kt < KT; ++kt, ++it) {
        const uint32_t s = it % STAGES;
        if (it >= (uint32_t)STAGES) {
          if (!(ok = warp_wait(empty0 + 8 * s, ((it / STAGES) - 1) & 1))) break;
        }
        if (elect_one()) {
          const uint32_t a_dst = s_u32(gsm + s * SM::kStage), b_dst = a_dst + SM::kABytes;
          bar_expect_tx(full0 + 8 * s, SM::kABytes + SM::kBBytes);
          tma_load_2d(a_dst, &mapA, (int)(kt * kBK), (int)at.m0, full0 + 8 * s);
          tma_load_2d(b_dst, &mapW, (int)(kt * kBK), (int)at.w0, full0 + 8 * s);
        }
      }
    }
    if (ok) ok = drain_ring<STAGES>(empty0, it);
  } else if (warp == 1) {
    const uint32_t idesc = (1u << 4) | (ep.operands_bf16 << 7) | (ep.operands_bf16 << 10) | ((uint32_t)(kPBN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
    uint32_t it = 0, i = 0;
    for (uint32_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++i) {
      const uint32_t acc = i & 1;
      if (i >= 2) {  // the epilogue must have drained this half of tensor memory (tile i - 2)
        if (!(ok = warp_wait(tempty0 + 8 * acc, ((i >> 1) - 1) & 1))) break;
        fence_after();
      }
      const uint32_t d = tmem_base + acc * (uint32_t)kPBN;
      for (uint32_t kt = 0; kt < KT; ++kt, ++it) {
        const uint32_t s = it % STAGES;
        if (!(ok = warp_wait(full0 + 8 * s, (it / STAGES) & 1))) break;
        fence_after();
        if (elect_one()) {
          const uint32_t a_s = s_u32(gsm + s * SM::kStage), b_s = a_s + SM::kABytes;
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) {
            umma_f16(d, smem_desc_sw128(a_s + k * 32), smem_desc_sw128(b_s + k * 32), idesc, (kt | (uint32_t)k) != 0);
          }
          umma_commit(empty0 + 8 * s);
          if (kt + 1 == KT) umma_commit(tfull0 + 8 * acc);
        }
      }
    }
  } else {
    const uint32_t lane_grp = (uint32_t)(warp & 3);
    uint32_t i = 0;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++i) {
      const uint32_t acc = i & 1;
      const Tile at = tile_at(tile);
      ok = tile_epilogue<KIND>(ep, at.m0, at.m_end, at.n0, N, kPBN / 32, tmem_base + acc * (uint32_t)kPBN, lane_grp, (warp - 2) >> 2, 2, lane,
                               s_u32(gsm + SM::kEpiOff) + (warp - 2) * kEpiWarp, tfull0 + 8 * acc, (i >> 1) & 1);
      if (!ok) break;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(tempty0 + 8 * acc);
    }
  }
  if (!ok) {
    if (lane == 0 && err) atomicOr(err, 4u);
    // tile copies of this CTA may still be in flight: give them a bounded time to land before shared memory and
    // tensor memory are released
    for (volatile uint32_t spin = 0; spin < (1u << 20); ++spin) {
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// ---- two SMs per tile: 256 x BN, each CTA of a pair holds 128 rows of A, half of the rows of W and 128 rows of the result ----
// A 128 x 256 tile per SM reads 48 KB of operands per 512 cycles of the tensor pipe; here it is 32 KB (BN = 256), so the copies
// keep up with the products, and narrower tiles (BN = 160: 83 bytes per cycle, below the 96 of the former) do so too: BN is
// chosen per shape so that the last wave of pairs is as full as possible (pair_columns). One CTA pair per two SMs walks tiles,
// token tiles fastest, so that pairs running together share one weight tile; two accumulators of 256 columns, so the epilogue of
// a tile runs beside the products of the next.
// Each CTA's warp 0 copies its own operands and counts them on the first CTA's barrier; the first CTA's warp 1 issues the
// products of both; epilogues by eight warps of each CTA, its rows. Measured against a 128 x 256 tile per SM (us, 1.9 GHz):
// 2011 x 16384 x 2048 105 against 120, 2011 x 3072 x 8192 78 and 103, 2011 x 5120 x 3072 50 and 65, 9472 x 16384 x 2048 470 and
// 528, 2011 x 2048 x 2048 18.4 and 21.8.
constexpr int kPairStages = 6;
struct PairSmem {
  static constexpr uint32_t kABytes = kBM * kBK * 2;
  static constexpr uint32_t kStage = kABytes + 128 * kBK * 2;
  static constexpr uint32_t kBarOff = kPairStages * kStage;
  static constexpr uint32_t kEpiOff = kBarOff + 256;
  static constexpr uint32_t kTotal = kEpiOff + PSmem::kEpiBytes + 1024;
};
static_assert(PairSmem::kTotal <= 227 * 1024, "shared memory of the pair kernel");

template <int KIND>
__global__ void __launch_bounds__(kPThreadsGemm) gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap mapA,
                                                                    const __grid_constant__ CUtensorMap mapW, const uint32_t M, const uint32_t N,
                                                                    const uint32_t K, const uint32_t BN, const GemmEpilogue ep, uint32_t* err) {
  using SM = PairSmem;
  constexpr int STAGES = kPairStages;
  extern __shared__ unsigned char gsm_raw[];
  unsigned char* gsm = reinterpret_cast<unsigned char*>(((uintptr_t)gsm_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(gsm + SM::kBarOff);
  // as in the grouped kernel; "full" and "accumulator empty" count in the first CTA, the others in both
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  const uint32_t full0 = s_u32(bars), empty0 = s_u32(bars + STAGES), tfull0 = s_u32(bars + 2 * STAGES), tempty0 = s_u32(bars + 2 * STAGES + 2);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // (uniform)
  const uint32_t rank = cluster_rank(), KT = (K + kBK - 1) / kBK;
  const uint32_t mtiles = (M + 2 * kBM - 1) / (2 * kBM), tiles = mtiles * ((N + BN - 1) / BN);
  const uint32_t first = blockIdx.x >> 1, step = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      bar_init(full0 + 8 * s, 1);
      bar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      bar_init(tfull0 + 8 * a, 1);
      bar_init(tempty0 + 8 * a, 16);  // the epilogue warps of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  cluster_sync();  // the other CTA's barriers are there
  fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    const uint32_t b_bytes = BN / 2 * kBK * 2;
    uint32_t it = 0;
    for (uint32_t tile = first; tile < tiles && ok; tile += step) {
      const uint32_t m0 = (tile % mtiles) * (2 * kBM) + rank * kBM, w0 = (tile / mtiles) * BN + rank * (BN / 2);
      for (uint32_t kt = 0; kt < KT; ++kt, ++it) {
        const uint32_t s = it % STAGES;
        if (it >= (uint32_t)STAGES) {
          if (!(ok = warp_wait(empty0 + 8 * s, ((it / STAGES) - 1) & 1))) break;
        }
        if (elect_one()) {
          const uint32_t a_dst = s_u32(gsm + s * SM::kStage), b_dst = a_dst + SM::kABytes, full = in_leader(full0 + 8 * s);
          if (rank == 0) bar_expect_tx(full0 + 8 * s, 2 * (SM::kABytes + b_bytes));
          tma_load_2d_pair(a_dst, &mapA, (int)(kt * kBK), (int)m0, full);
          tma_load_2d_pair(b_dst, &mapW, (int)(kt * kBK), (int)w0, full);
        }
      }
    }
    if (ok) ok = drain_ring<STAGES>(empty0, it);
  } else if (warp == 1) {
    if (rank == 0) {
      const uint32_t idesc = (1u << 4) | (ep.operands_bf16 << 7) | (ep.operands_bf16 << 10) | ((BN >> 3) << 17) | ((uint32_t)(2 * kBM >> 4) << 24);
      uint32_t it = 0, i = 0;
      for (uint32_t tile = first; tile < tiles && ok; tile += step, ++i) {
        const uint32_t acc = i & 1;
        if (i >= 2) {  // both epilogues must have drained this half of tensor memory
          if (!(ok = warp_wait_cluster(tempty0 + 8 * acc, ((i >> 1) - 1) & 1))) break;
          fence_after();
        }
        const uint32_t d = tmem_base + acc * 256u;
        for (uint32_t kt = 0; kt < KT; ++kt, ++it) {
          const uint32_t s = it % STAGES;
          if (!(ok = warp_wait_cluster(full0 + 8 * s, (it / STAGES) & 1))) break;
          fence_after();
          if (elect_one()) {
            const uint32_t a_s = s_u32(gsm + s * SM::kStage), b_s = a_s + SM::kABytes;
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              umma_f16_pair(d, smem_desc_sw128(a_s + k * 32), smem_desc_sw128(b_s + k * 32), idesc, (kt | (uint32_t)k) != 0);
            umma_commit_pair(empty0 + 8 * s);
            if (kt + 1 == KT) umma_commit_pair(tfull0 + 8 * acc);
          }
        }
      }
    }
  } else {
    const uint32_t lane_grp = (uint32_t)(warp & 3);
    uint32_t i = 0;
    for (uint32_t tile = first; tile < tiles; tile += step, ++i) {
      const uint32_t acc = i & 1, m0 = (tile % mtiles) * (2 * kBM) + rank * kBM, n0 = (tile / mtiles) * BN;
      ok = tile_epilogue<KIND>(ep, m0, M, n0, N, (int)(BN / 32), tmem_base + acc * 256u, lane_grp, (warp - 2) >> 2, 2, lane,
                               s_u32(gsm + SM::kEpiOff) + (warp - 2) * kEpiWarp, tfull0 + 8 * acc, (i >> 1) & 1);
      if (!ok) break;
      fence_before();
      __syncwarp();
      if (lane == 0) bar_arrive_cluster(in_leader(tempty0 + 8 * acc));
    }
  }
  if (!ok) {
    if (lane == 0 && err) atomicOr(err, 4u);
    // copies and products of the pair may still be in flight: a bounded time for them to end before their memory is released
    for (volatile uint32_t spin = 0; spin < (1u << 20); ++spin) {
    }
  }
  fence_before();
  __syncthreads();
  cluster_sync();  // nobody arrives on, or multiplies from, the memory of a CTA that has left
  fence_after();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
}

// ---- small producers of the float16 A operands ----------------------------------------------------------------
__global__ void __launch_bounds__(256) rmsnorm_to_half_kernel(const float* __restrict__ x, const float* __restrict__ gain,
                                                              float eps, uint32_t H, __half* __restrict__ out) {
  __shared__ float red[8];
  pdl_launch_dependents();
  pdl_wait();
  const float* xr = x + (size_t)blockIdx.x * H;
  float ss = 0.f;
  for (uint32_t i = threadIdx.x; i < H; i += 256) ss = fmaf(xr[i], xr[i], ss);
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) tot += red[w];
  const float rms = sqrtf(__fdiv_rn(tot, (float)H) + eps);
  __half* o = out + (size_t)blockIdx.x * H;
  for (uint32_t i = threadIdx.x; i < H; i += 256) o[i] = __float2half_rn(__fmul_rn(__fdiv_rn(xr[i], rms), gain[i]));
}

__global__ void embed_rows_kernel(const __half* __restrict__ E, const uint32_t* __restrict__ tokens, uint32_t H,
                                  float* __restrict__ x) {
  pdl_launch_dependents();
  pdl_wait();
  const __half* row = E + (size_t)tokens[blockIdx.x] * H;
  float* o = x + (size_t)blockIdx.x * H;
  for (uint32_t i = threadIdx.x; i < H; i += blockDim.x) o[i] = __half2float(row[i]);
}

__global__ void float_to_half_kernel(const float* __restrict__ in, __half* __restrict__ out, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = __float2half_rn(in[i]);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || !p) return nullptr;
  fn = (EncodeTiledFn)p;
  return fn;
}

// A descriptor depends only on (address, rows, K, box rows). Those of the weights, the same few hundred for every pass, are kept per
// host thread instead of being encoded again at each of ~110 launches, and with them those of the workspaces, a few per length of a
// pass.
struct MapKey {
  const void* base;
  uint64_t rows, K;
  uint32_t box_rows;
  bool operator==(const MapKey& o) const { return base == o.base && rows == o.rows && K == o.K && box_rows == o.box_rows; }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    return std::hash<uint64_t>()((uint64_t)(uintptr_t)k.base ^ (k.rows * 0x9E3779B97F4A7C15ull) ^ (k.K << 20) ^ k.box_rows);
  }
};

}  // namespace

bool encode_tile_map16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {K * 2};
  cuuint32_t box[2] = {(cuuint32_t)kBK, box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool encode_stack_map16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K, uint64_t layers, uint64_t stride, uint32_t box_rows,
                        uint32_t box_blocks) {
  EncodeTiledFn fn = encode_fn();
  if (!fn || K % kBK || stride % 16) return false;
  cuuint64_t dims[4] = {kBK, rows, K / kBK, layers};
  cuuint64_t strides[3] = {K * 2, kBK * 2, layers > 1 ? stride : rows * K * 2};
  cuuint32_t box[4] = {(cuuint32_t)kBK, box_rows, box_blocks, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool tile_map16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K, uint32_t box_rows) {
  static thread_local std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  const MapKey key{base, rows, K, box_rows};
  auto it = cache.find(key);
  if (it != cache.end()) {
    *map = it->second;
    return true;
  }
  if (!encode_tile_map16(map, base, rows, K, box_rows)) return false;
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, *map);
  return true;
}

namespace {

// Clusters of Z CTAs (along a split of K) that run at the same time: a cluster's CTAs share a group of 16 to 18 SMs.
template <int BN, int STAGES, int KIND>
uint32_t clusters_at_once(uint32_t Z) {
  static thread_local int device = -1, known[9] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (device != dev) {
    for (int& k : known) k = -1;
    device = dev;
  }
  if (known[Z] < 0) {
    auto kern = gemm_tc_kernel<BN, STAGES, KIND, true>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count() / Z, 1, Z);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = GemmSmem<BN, STAGES>::kTotal;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = Z;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    known[Z] = n;
  }
  return (uint32_t)known[Z];
}

template <int BN, int STAGES, int KIND, bool REDUCE = false>
cudaError_t launch_bn_kind(cudaStream_t s, const __half* A, const __half* W, uint32_t M, uint32_t N, uint32_t K,
                      const GemmEpilogue& ep, uint32_t* err, uint32_t Z) {
  CUtensorMap mapA, mapW;
  if (!tile_map16(&mapA, A, M, K, kBM) || !tile_map16(&mapW, W, N, K, BN)) return cudaErrorInvalidValue;
  auto kern = gemm_tc_kernel<BN, STAGES, KIND, REDUCE>;
  const size_t smem = GemmSmem<BN, STAGES>::kTotal;
  static thread_local int attr_device = -1;  // the attribute is per device: set it once per (thread, device)
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (attr_device != dev) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr_device = dev;
  }
  dim3 grid((N + BN - 1) / BN, (M + kBM - 1) / kBM, Z);
  if constexpr (REDUCE) return launch_pdl_cluster(kern, grid, dim3(kGemmThreads), dim3(1, 1, Z), smem, s, prefill_pdl(), mapA, mapW, M, N, K, ep, err);
  e = launch_pdl(kern, grid, dim3(kGemmThreads), smem, s, prefill_pdl(), mapA, mapW, M, N, K, ep, err);
  if (e != cudaSuccess || Z == 1) return e;
  const size_t pairs = (size_t)M * ((N + 1) / 2);
  const size_t want = (pairs + 255) / 256;
  return launch_pdl(gemm_finish_kernel, dim3((unsigned)(want < 1184 ? want : 1184)), dim3(256), 0, s, prefill_pdl(),
                    (const float*)ep.scratch, M, N, Z, ep);
}

// f(kind) with the epilogue kind as a constant
template <typename F>
cudaError_t with_kind(int kind, F f) {
  switch (kind) {
    case GEMM_EPI_STORE: return f(std::integral_constant<int, GEMM_EPI_STORE>{});
    case GEMM_EPI_GATED: return f(std::integral_constant<int, GEMM_EPI_GATED>{});
    case GEMM_EPI_GATED_CLAMPED: return f(std::integral_constant<int, GEMM_EPI_GATED_CLAMPED>{});
    case GEMM_EPI_STORE_ACT: return f(std::integral_constant<int, GEMM_EPI_STORE_ACT>{});
    default: return f(std::integral_constant<int, GEMM_EPI_QKV_ROPE>{});
  }
}

template <int BN, int STAGES>
cudaError_t launch_bn(cudaStream_t s, const __half* A, const __half* W, uint32_t M, uint32_t N, uint32_t K, const GemmEpilogue& ep, uint32_t* err,
                      uint32_t Z = 1) {
  return with_kind(ep.kind, [&](auto kind) { return launch_bn_kind<BN, STAGES, decltype(kind)::value>(s, A, W, M, N, K, ep, err, Z); });
}

// A split of K, at best Z ways: added up inside clusters when all of them run at once with at least two thirds as many ways, else
// through memory. (Of 8 CTAs 15 clusters run at once, of 6 22, of 4 33.) 128 x 2048 x 2048: 9.6 us nine ways through memory, 7.8 six
// ways in clusters; 128 x 3072 x 2048: 9.5 (six), 8.1 (five); 37 x 2048 x 8192: 13.6 (nine), 12.8 (six); 128 x 2048 x 8192: 15.0
// (nine), 14.4 (six), 16.7 (four).
cudaError_t launch_split(cudaStream_t s, const __half* A, const __half* W, uint32_t M, uint32_t N, uint32_t K, const GemmEpilogue& ep, uint32_t* err,
                         uint32_t Z) {
  return with_kind(ep.kind, [&](auto kind) {
    constexpr int KIND = decltype(kind)::value;
    const uint32_t tiles = ((M + kBM - 1) / kBM) * ((N + 127) / 128);
    for (uint32_t z = Z < 8 ? Z : 8; z > 1 && z * 3 >= Z * 2; --z)
      if (clusters_at_once<128, 4, KIND>(z) >= tiles) return launch_bn_kind<128, 4, KIND, true>(s, A, W, M, N, K, ep, err, z);
    return launch_bn_kind<128, 4, KIND>(s, A, W, M, N, K, ep, err, Z);
  });
}

template <int KIND>
cudaError_t launch_grouped(cudaStream_t s, const __half* A, const __half* W, uint32_t max_rows, uint32_t N, uint32_t K, const GemmGroups& grp,
                           const GemmEpilogue& ep, uint32_t* err) {
  CUtensorMap mapA, mapW;
  if (!tile_map16(&mapA, A, max_rows, K, kBM) || !tile_map16(&mapW, W, (uint64_t)grp.count * N, K, kPBN)) return cudaErrorInvalidValue;
  auto kern = gemm_tc_grouped_kernel<KIND>;
  static thread_local int attr_device = -1;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (attr_device != dev) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PSmem::kTotal);
    if (e != cudaSuccess) return e;
    attr_device = dev;
  }
  const uint32_t tiles = grp.max_tiles * ((N + kPBN - 1) / kPBN);
  return launch_pdl(kern, dim3(tiles < sm_count() ? tiles : sm_count()), dim3(kPThreadsGemm), PSmem::kTotal, s, prefill_pdl(), mapA, mapW, N, K,
                    grp, ep, err);
}

// Columns of a pair's tile: the width in steps of 32 that needs the least time in waves of pairs (a wave costs its width, and
// about 8 columns' worth of filling and draining), the wider one of two equal ones. Forced, with a residual and plain stores (us):
// 2011 x 3072 x 8192: 256: 90, 224: 87, 192 (the choice): 81, 160: 100, 128: 103; 2011 x 3072 x 2048: 33, 31, 28, 33, 30;
// 2011 x 16384 x 2048: 128 at 256 (the choice), 133 at 224, 137 at 192; 128 x 28672 x 4096: 63 at 256, 57 at 224 (the choice),
// 71 at 192.
uint32_t pair_columns(uint32_t M, uint32_t N) {
  const uint32_t pairs = sm_count() / 2, mt = (M + 2 * kBM - 1) / (2 * kBM);
  uint32_t best = 256, cost = ~0u;
  for (uint32_t bn = 256; bn >= 128; bn -= 32) {
    const uint32_t tiles = mt * ((N + bn - 1) / bn), c = (tiles + pairs - 1) / pairs * (bn + 8);
    if (c < cost) best = bn, cost = c;
  }
  return best;
}

template <int KIND>
cudaError_t launch_pair(cudaStream_t s, const __half* A, const __half* W, uint32_t M, uint32_t N, uint32_t K, const GemmEpilogue& ep, uint32_t* err) {
  const uint32_t BN = pair_columns(M, N);
  CUtensorMap mapA, mapW;
  if (!tile_map16(&mapA, A, M, K, kBM) || !tile_map16(&mapW, W, N, K, BN / 2)) return cudaErrorInvalidValue;
  auto kern = gemm_tc_pair_kernel<KIND>;
  static thread_local int attr_device = -1;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (attr_device != dev) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PairSmem::kTotal);
    if (e != cudaSuccess) return e;
    attr_device = dev;
  }
  const uint32_t tiles = (M + 2 * kBM - 1) / (2 * kBM) * ((N + BN - 1) / BN), pairs = sm_count() / 2;
  return launch_pdl_cluster(kern, dim3(2 * (tiles < pairs ? tiles : pairs)), dim3(kPThreadsGemm), dim3(2), PairSmem::kTotal, s, prefill_pdl(), mapA, mapW,
                            M, N, K, BN, ep, err);
}

}  // namespace

// A tile grid of fewer than 120 CTAs of 128 x 128 leaves SMs without work (a chunk of <= 128 prompt tokens times a
// 2048-column matrix is 16 tiles): divide K so that about one CTA per SM streams weights, at least two K tiles each.
uint32_t gemm_tc_splits(uint32_t M, uint32_t N, uint32_t K) {
  const uint32_t tiles = ((M + kBM - 1) / kBM) * ((N + 127) / 128);
  const uint32_t KT = (K + kBK - 1) / kBK;
  if (tiles >= 120) return 1;
  uint32_t z = sm_count() / tiles;
  if (z > KT / 2) z = KT / 2;
  if (z > 16) z = 16;
  return z < 1 ? 1 : z;
}

cudaError_t launch_gemm_tc(cudaStream_t s, const __half* A, const __half* W, uint32_t M, uint32_t N, uint32_t K,
                           const GemmEpilogue& ep, uint32_t* err) {
  if (!A || !W || !M || !N || !K || (K & 7u) || (((uintptr_t)A | (uintptr_t)W) & 15)) return cudaErrorInvalidValue;
  if ((ep.kind == GEMM_EPI_GATED || ep.kind == GEMM_EPI_GATED_CLAMPED || ep.kind == GEMM_EPI_QKV_ROPE) && (N & 1u)) return cudaErrorInvalidValue;
  if (ep.operands_bf16 > 1) return cudaErrorInvalidValue;
  // enough CTAs to pull weights with every SM when the chunk is a single row of tiles
  const uint32_t mtiles = (M + kBM - 1) / kBM;
  // enough tiles to occupy most pairs of SMs
  if (mtiles * ((N + 255) / 256) >= 96)
    return with_kind(ep.kind, [&](auto kind) { return launch_pair<decltype(kind)::value>(s, A, W, M, N, K, ep, err); });
  if (ep.scratch) {
    uint32_t Z = gemm_tc_splits(M, N, K);
    while (Z > 1 && (size_t)Z * M * N > ep.scratch_floats) --Z;
    if (Z > 1) return launch_split(s, A, W, M, N, K, ep, err, Z);
  }
  if (mtiles * ((N + 127) / 128) >= 120) return launch_bn<128, 4>(s, A, W, M, N, K, ep, err);
  if (mtiles * ((N + 63) / 64) >= 120) return launch_bn<64, 6>(s, A, W, M, N, K, ep, err);
  return launch_bn<32, 8>(s, A, W, M, N, K, ep, err);
}

cudaError_t launch_gemm_tc_grouped(cudaStream_t s, const __half* A, const __half* W, uint32_t max_rows, uint32_t N, uint32_t K,
                                   const GemmGroups& g, const GemmEpilogue& ep, uint32_t* err) {
  static_assert(kGroupTile == kBM, "the tile list is made for this kernel's tiles");
  if (!A || !W || !max_rows || !N || !K || (K & 7u) || (((uintptr_t)A | (uintptr_t)W) & 15) || !g.count || !g.max_tiles) return cudaErrorInvalidValue;
  if (ep.kind == GEMM_EPI_QKV_ROPE || ((ep.kind == GEMM_EPI_GATED || ep.kind == GEMM_EPI_GATED_CLAMPED) && (N & 1u)) || ep.bias || ep.resid || ep.operands_bf16 > 1) return cudaErrorInvalidValue;
  return with_kind(ep.kind, [&](auto kind) {
    if constexpr (decltype(kind)::value == GEMM_EPI_QKV_ROPE) return cudaErrorInvalidValue;
    else return launch_grouped<decltype(kind)::value>(s, A, W, max_rows, N, K, g, ep, err);
  });
}

bool prefill_pdl() {
  static const bool on = [] { const char* v = getenv("NFAI_PREFILL_PDL"); return !(v && atoi(v) == 0); }();
  return on;
}

cudaError_t launch_rmsnorm_to_half(cudaStream_t s, const float* x, const float* gain, float eps, uint32_t M, uint32_t H,
                                   __half* out, bool after_collective) {
  return launch_pdl(rmsnorm_to_half_kernel, dim3(M), dim3(256), 0, s, prefill_pdl() && !after_collective, x, gain, eps, H, out);
}

cudaError_t launch_embed_rows(cudaStream_t s, const __half* E, const uint32_t* tokens, uint32_t M, uint32_t H, float* x) {
  return launch_pdl(embed_rows_kernel, dim3(M), dim3(256), 0, s, prefill_pdl(), E, tokens, H, x);
}

cudaError_t launch_float_to_half(cudaStream_t s, const float* in, __half* out, size_t n) {
  size_t want = (n + 255) / 256;
  float_to_half_kernel<<<(unsigned)(want < 2368 ? want : 2368), 256, 0, s>>>(in, out, n);
  return cudaGetLastError();
}

}  // namespace nfai
