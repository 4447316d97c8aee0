// A decode step as ONE kernel that stays on the GPU from the embedding row to the arg-max: one CTA per SM, all resident
// (cooperative launch), the layers' products and attentions as phases of a loop. Models with float16 weights and a float16 cache on one
// GPU.
//
// What bounds a step is the stream of its weights out of HBM; what a step made of launches loses on top are its hand-overs: five a
// layer at about 2 us each (the wait for the last CTA, then x out of L2), during which only what a kernel requested before its
// wait is in flight. Here nothing in the weight stream waits for a result: a warp of its own copies this CTA's rows of every
// matrix, in the order they are used, through a ring of shared memory (tile copies, 176 KB per SM = 4 us of HBM time), and runs
// ahead of the products while those wait for x.
//
// For that to help, the ring must be emptied much faster than HBM fills it (23 bytes per clock and SM). With float32 arithmetic on
// the warps it was not: 25 bytes, half of the instructions conversions and sums across lanes, and little more with warp-level products (39
// bytes). So tcgen05 multiplies, exactly: float16 weights are the A operand as they lie in the
// ring, x is split into three float16 terms of 11 bits each, scaled to the largest element of its block, as the B operand. Every
// product is exact and sums are float32 in tensor memory (resident_plan says what they lose); one thread issues them, and no warp
// touches a weight.
//
// Hand-overs go through memory words of (value, tag), as between the ranks of a tensor-parallel group (xchg_protocol.h): a row's
// result is one 8-byte store, a reader polls the words it needs until each carries this step's tag. No flag, no fence, no
// barrier across the grid. Every phase of every layer has words of its own, so a word is written once per step, and the tag is the
// number of the step. All CTAs are on the GPU at the same time, so a poll ends; should it not within the context's budget
// (nfai_ctx_set_wait_ns), it gives up (error bit 4 of the step state, NFAI_ERR_TIMEOUT) and the kernel runs to its end without waiting
// for results again. It does wait, with a limit of its own, for what is on its way into a CTA's memory before that CTA leaves.
//
// Split of the work. Rows of every matrix are dealt evenly over the CTAs in contiguous blocks. A ring slot holds a tile of 16 rows
// and 512 columns, eight blocks of 64; warp b makes the terms of block b of every piece of x: it polls exactly those columns, and no
// x is read twice by a CTA. Sums meet across warps in shared memory, in a fixed order. Attention: one CTA per query head and
// range of positions; the rows of earlier positions are requested before the new row's words are polled; ranges are merged by the
// CTAs that made them, a slice each.
//
// Measured (B200, us a step, sequence of launches -> this kernel): 1B architecture (121 MB a layer) at position 128 619 -> 535, 391 629
// -> 550, 700 675 -> 558, 2 000 691 -> 629, 4 000 734 -> 725; 3B at 128 1 477 -> 1 332, 1 000 1 672 -> 1 485; 8B at 128 2 886 -> 2 747,
// 1 000 3 036 -> 2 948. What single choices are worth, below, is at position 128 of the 1B architecture with a head of 32 768 rows (478 to
// 481 from one board to the next).
#include <math.h>

#include <algorithm>

#include "attn_core.cuh"
#include "common.cuh"
#include "kernels.h"
#include "step_resident.h"
#include "umma.cuh"

namespace nfai {

namespace {

constexpr uint32_t kThreads = 256;                // that make x, finish rows and attend
constexpr uint32_t kWarps = kThreads / 32;
constexpr uint32_t kAllThreads = kThreads + 64;   // a warp that copies, a warp that issues the products
constexpr uint32_t kSlots = 11;                   // of the ring
constexpr uint32_t kTileRows = 16, kPiece = 512;  // a slot: rows, columns
constexpr uint32_t kBlocks = kPiece / 64;         // blocks of 64 columns: the operand's rows are (block, row) pairs
constexpr uint32_t kSlotBytes = kTileRows * kPiece * 2;
static_assert(kBlocks == kWarps, "a warp makes the terms of one block of every piece");
constexpr uint32_t kAhead = 5;                    // copies in flight (feed)
constexpr uint32_t kXSlots = 8, kXBytes = 4096;   // ring of pieces of x: [32 rows: block, term][64 columns]
constexpr uint32_t kNarrow = 8;                   // most pieces that a phase keeps for all its rows
constexpr uint32_t kChunk = 4;                    // pieces at a time where x is longer
static_assert(kNarrow == 2 * kChunk && kXSlots == 2 * kChunk, "two chunks are polled, and kept, at a time");
constexpr uint32_t kAcc = 8, kAccColumns = 32;    // accumulators in tensor memory
constexpr uint32_t kBlockRows = 128;              // rows whose sums meet in shared memory at a time
constexpr uint32_t kPartFloats = 2 * kBlockRows * 4;  // two buffers of four warps' sums
constexpr uint32_t kMaxNarrow = kNarrow * kPiece, kMaxWide = 16384;
constexpr unsigned long long kLeaveNs = 1000000000ull;     // a CTA that leaves: for its copies and products to end
constexpr unsigned long long kArrivalsNs = 100000ull;      // ... and, where waits have given up, for arrivals that nobody counts

// ---- barriers, copies, words ---------------------------------------------------------------------------------------------
using umma::bar_arrive;
using umma::bar_expect_tx;
using umma::bar_init;
using umma::bar_try;
__device__ __forceinline__ uint32_t s_addr(const void* p) { return umma::s_u32(p); }
__device__ __forceinline__ void copy_box(unsigned long long policy, uint32_t dst, const void* map, int row, int block, int layer, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4, %5}], [%6], %7;" ::"r"(dst),
      "l"(map), "r"(0), "r"(row), "r"(block), "r"(layer), "r"(bar), "l"(policy)
      : "memory");
}
// The thread's number, asked for where it is used: the compiler would otherwise derive things from it once and keep them over all phases
// of all layers (168 registers a thread, 144 so; beyond 200 they would go to local memory, which here means L2: next to the ring
// there is no L1 to speak of).
__device__ __forceinline__ uint32_t thread_id() {
  uint32_t t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}
// the threads that multiply
__device__ __forceinline__ void sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

__device__ __forceinline__ uint4 ld_words(const uint4* p) {  // two (value, tag) words
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_word(uint2* p, float v, uint32_t tag) {
  asm volatile("st.volatile.global.v2.u32 [%0], {%1,%2};" ::"l"(p), "r"(__float_as_uint(v)), "r"(tag) : "memory");
}
__device__ __forceinline__ void st_words(uint2* p, float a, float b, uint32_t tag) {
  asm volatile("st.volatile.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(__float_as_uint(a)), "r"(tag), "r"(__float_as_uint(b)), "r"(tag) : "memory");
}

__device__ __forceinline__ void sts4(uint32_t at, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory"); }

// ---- shared memory ---------------------------------------------------------------------------------------------------------
enum Phase { PH_QKV, PH_O, PH_GATEUP, PH_DOWN, PH_HEAD, kPhases };

// This CTA's part of a matrix.
struct Share {
  uint32_t row0, rows, K;
  uint32_t pieces;               // slots of a tile
};

struct Shared {
  // The launch's parameters. From where they are, a constant bank, a phase's first look at one is a miss up to HBM when the weights
  // have passed through L2 since the last: 1.3 us for the epsilon of a norm.
  ResidentArgs p;
  unsigned long long full[kSlots], empty[kSlots];      // ring of weights: copies to products and back
  unsigned long long x_full[kXSlots], x_empty[kXSlots];      // ring of pieces of x: warps to products and back
  unsigned long long acc_full[kAcc], acc_empty[kAcc];        // accumulators: products to warps and back
  unsigned long long drained;                                // the last product is done
  Share share[kPhases];
  uint32_t dead;                 // 1: a poll gave up, no further one is begun; 2: a wait on a barrier did, nothing is issued any more
  uint32_t tmem;
  alignas(16) float squares[kThreads];  // each thread's part of the sum of squares of x
  float scale[kMaxWide / kPiece / kChunk][kBlocks];  // what undoes the scaling of a chunk's blocks
  alignas(16) float resid[kBlockRows];  // the residual at this CTA's rows of O and down
  float best_v[kBlockRows / 2];  // of the head's rows that a thread has finished
  uint32_t best_i[kBlockRows / 2];
  float2 rope[64];               // this step's row of the table
  uint32_t tag, pos, tok;        // this step's
  bool keep;                     // the position is inside the cache
};

// The kernel's shared memory. The ring lies first: what the products read behind a tile of fewer than 16 rows is a slot or x.
constexpr uint32_t aligned(uint32_t bytes) { return (bytes + 1023) / 1024 * 1024; }
constexpr uint32_t kXOffset = kSlots * kSlotBytes, kSharedOffset = kXOffset + kXSlots * kXBytes, kPartOffset = kSharedOffset + aligned(sizeof(Shared)),
                   kWorkOffset = kPartOffset + kPartFloats * 4, kSmem = kWorkOffset + (kWarps * (128 + 4) + 3 * 128) * 4;
static_assert(kSmem <= 227 * 1024, "shared memory of a CTA");

__device__ __forceinline__ uint32_t dead(const Shared& sh) { return *reinterpret_cast<const volatile uint32_t*>(&sh.dead); }
__device__ __forceinline__ void give_up(Shared& sh, StepState* state, uint32_t how) {
  atomicMax(&sh.dead, how);
  atomicOr(&state->err, 4u);
}
// (inlined: 481.1 us a step, 484.7 as a function of its own)
__device__ __forceinline__ void wait_slowly(Shared& sh, StepState* state, uint32_t bar, uint32_t parity, unsigned long long limit) {
  const unsigned long long t0 = global_timer_ns();
  for (uint32_t polls = 1; !bar_try(bar, parity) && dead(sh) < 2; ++polls)
    if ((polls & 63u) == 0 && global_timer_ns() - t0 > limit) return give_up(sh, state, 2);
}
// Pairs of words at(0) .. at(N - 1) until each carries the tag; those that carry it from the start are not read.
template <int N, typename At>
__device__ __forceinline__ void poll_words(Shared& sh, StepState* state, uint32_t tag, At at, uint4 (&w)[N]) {
  unsigned long long t0 = 0;
#pragma unroll 1
  for (uint32_t polls = 1;; ++polls) {
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (w[j].y != tag || w[j].w != tag) w[j] = ld_words(at(j));
    bool all = true;
#pragma unroll
    for (int j = 0; j < N; ++j) all = all && w[j].y == tag && w[j].w == tag;
    if (all) return;
    if ((polls & 3u) == 1) {
      if (dead(sh)) return;
      if (t0 == 0) t0 = global_timer_ns();
      else if (global_timer_ns() - t0 > sh.p.wait_ns) return give_up(sh, state, 1);
    }
  }
}

// Where a role is in a ring of barriers.
struct Cursor {
  uint32_t slot = 0, turn = 0;   // turn: the parity of the phase that ends next
  __device__ __forceinline__ void next(uint32_t slots) {
    if (++slot == slots) {
      slot = 0;
      turn ^= 1u;
    }
  }
};

struct Step {
  Shared& sh;
  uint32_t ring, xs;             // addresses: weights, pieces of x
  float* const work;             // the warps' attention states
  float* const part;             // row sums

  // (four times the budget: what arrives here may have polled for words before)
  __device__ __forceinline__ void wait(unsigned long long& bar, uint32_t parity) const {
    if (!bar_try(s_addr(&bar), parity)) wait_slowly(sh, sh.p.state, s_addr(&bar), parity, 4 * sh.p.wait_ns);
  }
  // For a CTA that leaves: whether or not waits have given up.
  __device__ __forceinline__ void wait_out(unsigned long long& bar, uint32_t parity) const {
    const unsigned long long t0 = global_timer_ns();
    while (!bar_try(s_addr(&bar), parity) && global_timer_ns() - t0 < kLeaveNs) {}
  }
  // For roles of a whole warp, whose lanes stay together: one answer. False: a wait on a barrier has given up, nothing is issued any more.
  __device__ __forceinline__ bool warp_wait(unsigned long long& bar, uint32_t parity) const {
    if (__all_sync(0xffffffffu, bar_try(s_addr(&bar), parity))) return true;
    wait_slowly(sh, sh.p.state, s_addr(&bar), parity, 4 * sh.p.wait_ns);
    return !__any_sync(0xffffffffu, dead(sh) >= 2);
  }
  // N pairs of words, kPiece elements apart from `first` on; those from `left` elements on read as zero
  template <int N>
  __device__ __forceinline__ void poll(const uint2* first, uint32_t left, float2 (&v)[N]) const {
    const uint32_t tag = sh.tag;
    uint4 w[N];
#pragma unroll
    for (int j = 0; j < N; ++j) w[j] = make_uint4(0, j * kPiece < left ? ~tag : tag, 0, tag);
    poll_words<N>(sh, sh.p.state, tag, [&](int j) { return reinterpret_cast<const uint4*>(first + j * kPiece); }, w);
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = make_float2(__uint_as_float(w[j].x), __uint_as_float(w[j].z));
  }
};

__device__ __forceinline__ Share share_of(uint32_t N, uint32_t unit, uint32_t K) {
  const uint32_t n = N / unit, c = blockIdx.x, G = gridDim.x;
  Share s;
  s.row0 = (uint32_t)((uint64_t)n * c / G) * unit;
  s.rows = (uint32_t)((uint64_t)n * (c + 1) / G) * unit - s.row0;
  s.K = K;
  s.pieces = (K + kPiece - 1) / kPiece;
  return s;
}

// ---- x ------------------------------------------------------------------------------------------------------------------------
// Three terms of 11 bits, each 2^11 times as large as it counts (exact; nothing is left of what is not finite).
__device__ __forceinline__ void split2(float2 x, float up, uint32_t (&term)[3]) {
  float2 r = make_float2(x.x * up, x.y * up);
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const __half2 h = __floats2half2_rn(r.x, r.y);
    const float2 f = __half22float2(h);
    r.x = fabsf(f.x) < INFINITY ? (r.x - f.x) * 2048.f : 0.f;
    r.y = fabsf(f.y) < INFINITY ? (r.y - f.y) * 2048.f : 0.f;
    term[t] = reinterpret_cast<const uint32_t&>(h);
  }
}

// Row `block` * 4 + term of a piece of x holds a term of its block's 64 columns: 128 bytes under the 128-byte swizzle, 8 rows a
// group, the fourth row of a block zero. The address of columns 2 lane, 2 lane + 1 in the first term's row.
__device__ __forceinline__ uint32_t x_row(uint32_t piece, uint32_t block, uint32_t term, uint32_t lane) {
  const uint32_t row = (block & 1) * 4 + term;
  return piece + (block >> 1) * 1024 + row * 128 + (((lane >> 2) ^ row) << 4) + (lane & 3) * 4;
}

// ---- products ---------------------------------------------------------------------------------------------------------------
// A slot is the A operand of four instructions as it lies: [8 blocks of 64 columns][16 rows][128 bytes] are 128 lines (block, row) of
// 64 columns. The last rows of a share come in boxes of 8, 4 and 2 rows (feed), one behind the other: lines all the same. The B
// operand's 32 columns are (block, term); of the 128 x 32 sums those whose blocks agree are wanted, the others cost nothing: four such
// instructions take 389 cycles, 42 bytes of weights a clock and SM where HBM brings 23, and with fewer columns as long.
// Sub-products of a phase: chunks of K (one, where x is short enough to be kept), in a chunk tiles of 16 rows, in a tile pieces.
__device__ __forceinline__ uint32_t chunk_of(const Share& s) { return s.pieces <= kNarrow ? s.pieces : kChunk; }

__device__ __forceinline__ void issue_products(const Step& st) {
  const ResidentArgs& p = st.sh.p;
  Shared& sh = st.sh;
  constexpr uint32_t idesc = (1u << 4) | (kAccColumns >> 3) << 17 | (128u >> 4) << 24;
  const uint64_t a0 = umma::smem_desc_sw128(st.ring), b0 = umma::smem_desc_sw128(st.xs);  // (addresses in units of 16 bytes, below 2^14)
  const uint32_t tmem = sh.tmem, empty = s_addr(&sh.empty[0]);
  Cursor w, x0, acc;             // weights, the chunk's first piece of x, accumulators
  const uint32_t end = p.L * 4 + (p.with_head ? 1 : 0);
#pragma unroll 1
  for (uint32_t k = 0; k < end; ++k) {
    const Share& s = sh.share[k < p.L * 4 ? k & 3u : (uint32_t)PH_HEAD];
    const uint32_t rows = s.rows, pieces = s.pieces, chunk = chunk_of(s);
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < pieces; c0 += chunk) {
      const uint32_t n = min(chunk, pieces - c0);
#pragma unroll 1
      for (uint32_t r = 0; r < rows; r += kTileRows, acc.next(kAcc)) {
        const uint32_t d = tmem + acc.slot * kAccColumns;
        const bool last = r + kTileRows >= rows;
        Cursor x = x0;
        st.wait(sh.acc_empty[acc.slot], acc.turn ^ 1u);
#pragma unroll 1
        for (uint32_t i = 0; i < n; ++i, w.next(kSlots), x.next(kXSlots)) {
          // (one decision a piece: with votes behind the other two waits as well 486.6 us a step, 481.5 so)
          if (r == 0) st.wait(sh.x_full[x.slot], x.turn);
          if (!st.warp_wait(sh.full[w.slot], w.turn)) return;
          umma::fence_after();
          if (umma::elect_one()) {
            const uint64_t a = a0 + w.slot * (kSlotBytes / 16), b = b0 + x.slot * (kXBytes / 16);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) umma::umma_f16(d, a + 2 * j, b + 2 * j, idesc, (i | j) != 0);
            umma::umma_commit(empty + 8 * w.slot);
            if (last) umma::umma_commit(s_addr(&sh.x_empty[x.slot]));
            if (i + 1 == n) umma::umma_commit(s_addr(&sh.acc_full[acc.slot]));
          }
          __syncwarp();
        }
      }
      for (uint32_t i = 0; i < n; ++i) x0.next(kXSlots);
    }
  }
}

// The words of layer l - 1: queries, keys and values, then in this order. The embedding row is what the layer before the first leaves.
__device__ __forceinline__ uint2* layer_words(const ResidentArgs& p, uint32_t l) { return reinterpret_cast<uint2*>(p.words) + (size_t)l * p.words_per_layer; }
__device__ __forceinline__ uint32_t words_att(const ResidentArgs& p) { return (p.qH + 2 * p.kvH) * p.d; }
__device__ __forceinline__ uint32_t words_mid(const ResidentArgs& p) { return words_att(p) + p.qH * p.d; }
__device__ __forceinline__ uint32_t words_hid(const ResidentArgs& p) { return words_mid(p) + p.H; }
__device__ __forceinline__ uint32_t words_out(const ResidentArgs& p) { return words_hid(p) + p.F; }
__device__ __forceinline__ uint32_t words_part(const ResidentArgs& p) { return words_out(p) + p.H; }
template <int D>
__device__ __forceinline__ __half* layer_cache(const ResidentArgs& p, void* cache, uint32_t l) {
  return reinterpret_cast<__half*>(cache) + (size_t)l * p.ctx * (p.kvH * D);
}

// The lowest index among the maxima.
__device__ __forceinline__ void take_best(float& v, uint32_t& i, float ov, uint32_t oi) {
  if (oi != 0xffffffffu && (i == 0xffffffffu || ov > v || (ov == v && oi < i))) {
    v = ov;
    i = oi;
  }
}

// The pair of rows `row`, `row` + 1 (`local` within the share) of phase `ph` of layer l; both: the second one is a row of this CTA
// too.
template <int D>
__device__ __forceinline__ void finish_pair(const Step& st, uint32_t l, uint32_t ph, uint32_t row, uint32_t local, float a, float b, bool both) {
  const ResidentArgs& p = st.sh.p;
  Shared& sh = st.sh;
  uint2* const words = layer_words(p, l + 1);
  if (ph == PH_QKV) {
    const uint32_t qDim = p.qH * D, kvDim = p.kvH * D;
    if (row < qDim + kvDim && row % D < p.ropeDim) {  // products rounded separately, as the other kernels do
      const float2 cs = sh.rope[row % D >> 1];
      const float v1 = __fsub_rn(__fmul_rn(cs.x, a), __fmul_rn(cs.y, b));
      const float v2 = __fadd_rn(__fmul_rn(cs.y, a), __fmul_rn(cs.x, b));
      a = v1;
      b = v2;
    }
    if (row >= qDim && sh.keep) {
      const bool key = row < qDim + kvDim;
      __half* k = layer_cache<D>(p, key ? p.kc : p.vc, l) + (size_t)sh.pos * kvDim + (row - qDim - (key ? 0 : kvDim));
      store_as(k, a);
      store_as(k + 1, b);
    }
    st_words(words + row, a, b, sh.tag);
  } else if (ph == PH_GATEUP) {
    st_word(words + words_hid(p) + (row >> 1), gated(ACT_SILU, a, b), sh.tag);
  } else if (ph == PH_HEAD) {
    float v = sh.best_v[local & (kBlockRows / 2 - 1)];
    uint32_t i = sh.best_i[local & (kBlockRows / 2 - 1)];
    p.logits[row] = a;
    take_best(v, i, a, row);
    if (both) {
      p.logits[row + 1] = b;
      take_best(v, i, b, row + 1);
    }
    sh.best_v[local & (kBlockRows / 2 - 1)] = v;
    sh.best_i[local & (kBlockRows / 2 - 1)] = i;
  } else {
    a = sh.resid[2 * local] + a;
    b = sh.resid[2 * local + 1] + b;
    st_words(words + (ph == PH_O ? words_mid(p) : words_out(p)) + row, a, b, sh.tag);
    *reinterpret_cast<float2*>(p.xbuf + (size_t)(2 * l + (ph == PH_O ? 1 : 2)) * p.H + row) = make_float2(a, b);
  }
}

// This warp's block of the kNarrow pieces from c0 on of x, from the words of the phase before. The norm's gain is multiplied in here,
// its root mean square divides the product's sums (product): nothing waits for a sum over the CTA that way. This CTA's rows of
// x as they came are kept for the epilogue that adds them to its sums.
__device__ __forceinline__ void fetch_x(const Step& st, uint32_t l, uint32_t ph, uint32_t t, uint32_t c0, float2 (&v)[kNarrow]) {
  const ResidentArgs& p = st.sh.p;
  Shared& sh = st.sh;
  const uint32_t column0 = c0 * kPiece + (t >> 5) * 64 + 2 * (t & 31), K = sh.share[ph].K, left = K > column0 ? K - column0 : 0;
  const bool norm = ph != PH_O && ph != PH_DOWN;
  float2 g[kNarrow];
  if (norm) {
    const float* gain = (ph == PH_HEAD ? p.out_norm : reinterpret_cast<const float*>(reinterpret_cast<const char*>(ph == PH_QKV ? p.attn_norm : p.ffn_norm) + l * p.layer_stride)) + column0;
#pragma unroll
    for (int j = 0; j < (int)kNarrow; ++j) g[j] = j * kPiece < left ? __ldg(reinterpret_cast<const float2*>(gain + j * kPiece)) : make_float2(0.f, 0.f);
  }
  const uint32_t at = ph == PH_O ? words_att(p) : ph == PH_GATEUP ? words_mid(p) : ph == PH_DOWN ? words_hid(p) : words_out(p);
  st.poll<kNarrow>(layer_words(p, ph == PH_QKV || ph == PH_HEAD ? l : l + 1) + at + column0, left, v);
  if (norm) {
    const uint32_t mine = column0 - sh.share[PH_O].row0, keep = sh.share[PH_O].rows;  // (down has the same rows)
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < (int)kNarrow; ++j) {
      ss = fmaf(v[j].x, v[j].x, ss);
      ss = fmaf(v[j].y, v[j].y, ss);
      if (mine + j * kPiece < keep) *reinterpret_cast<float2*>(&sh.resid[mine + j * kPiece]) = v[j];
      v[j] = make_float2(v[j].x * g[j].x, v[j].y * g[j].y);
    }
    sh.squares[t] = ss;
  }
}
// The first n of them, a chunk, go as terms to the ring of x; the others move up.
__device__ __forceinline__ void put_x(const Step& st, Cursor& xc, uint32_t t, uint32_t n, uint32_t scale_slot, float2 (&v)[kNarrow]) {
  Shared& sh = st.sh;
  const uint32_t block = t >> 5, lane = t & 31;
  // the chunk's largest element of the block to [2^14, 2^15): the next terms are below 2^15 too. Exponents at the ends keep the factors
  // finite.
  float top = 0.f;
#pragma unroll
  for (int j = 0; j < (int)kNarrow; ++j)
    if (j < (int)n) top = fmaxf(top, fmaxf(fabsf(v[j].x), fabsf(v[j].y)));
  const uint32_t e = __reduce_max_sync(0xffffffffu, __float_as_uint(top)) >> 23;
  const int shift = min(max((int)e, 15), 254) - 127 - 14;
  const float up = __uint_as_float((uint32_t)(127 - shift) << 23);
  if (lane == 0) sh.scale[scale_slot][block] = __uint_as_float((uint32_t)(127 + shift) << 23);
#pragma unroll 1
  for (uint32_t j = 0; j < n; ++j) {
    uint32_t term[3];
    split2(v[0], up, term);
    st.wait(sh.x_empty[xc.slot], xc.turn ^ 1u);
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i) sts4(x_row(st.xs + xc.slot * kXBytes, block, i, lane), term[i]);
    // (a fence a piece: the products begin with the first while the others are made; one for all of a chunk 502.0 us a step, 477.8 so)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) bar_arrive(s_addr(&sh.x_full[xc.slot]));
    xc.next(kXSlots);
#pragma unroll
    for (int i = 1; i < (int)kNarrow; ++i) v[i - 1] = v[i];
  }
}

// The sums of a tile of `rows` rows out of its accumulator, to part[quarter of the lines][row]; four warps, a quarter of the lines each.
// All lines of a quarter are of one box.
__device__ __forceinline__ void take_tile(const Step& st, const Cursor& acc, uint32_t t, uint32_t rows, uint32_t scale_slot, bool add, float* part) {
  Shared& sh = st.sh;
  const uint32_t lane = t & 31, quarter = (t >> 5) & 3;
  uint32_t first = 0, row = 0, size = 0;  // the quarter's box: its first line and row, the logarithm of its rows
#pragma unroll
  for (uint32_t i = 4; i >= 1; --i) {
    if (rows >> i & 1u) {
      if (size == 0) size = quarter * 32 - first < (kBlocks << i) ? i : 0;
      if (size == 0) {
        first += kBlocks << i;
        row += 1u << i;
      }
    }
  }
  const uint32_t block = (quarter * 32 + lane - first) >> size;
  st.wait(sh.acc_full[acc.slot], acc.turn);
  umma::fence_after();
  uint32_t c[kAccColumns];
  umma::tmem_ld(sh.tmem + acc.slot * kAccColumns + (quarter << 21), c);
  umma::fence_before();
  __syncwarp();
  if (lane == 0) bar_arrive(s_addr(&sh.acc_empty[acc.slot]));
  float a = 0.f, b = 0.f, d = 0.f;  // the terms' sums of the lane's own block
#pragma unroll
  for (uint32_t i = 0; i < kBlocks; ++i) {
    if (block == i) {
      a = __uint_as_float(c[4 * i]);
      b = __uint_as_float(c[4 * i + 1]);
      d = __uint_as_float(c[4 * i + 2]);
    }
  }
  float v = 0.f;
  // (what an infinite weight makes of the later terms, infinity times zero, does not count)
  if (size && block < kBlocks) v = sh.scale[scale_slot][block] * (fabsf(a) < INFINITY ? fmaf(d, 0x1p-22f, fmaf(b, 0x1p-11f, a)) : a);
#pragma unroll 1
  for (uint32_t o = 1u << size; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  // rows that are another quarter's: nothing from this one
  part += quarter * kBlockRows;
  const bool here = size && lane >= row && lane < row + (1u << size);
  const float got = __shfl_sync(0xffffffffu, v, here ? lane - row : 0);
  if (lane < rows) part[lane] = (add ? part[lane] : 0.f) + (here ? got : 0.f);
}

// The product of this CTA's share in phase ph of layer l with x, and its epilogue.
template <int D>
__device__ __forceinline__ void product(const Step& st, Cursor& xc, Cursor& acc, uint32_t l, uint32_t ph) {
  const ResidentArgs& p = st.sh.p;
  const Share& s = st.sh.share[ph];
  const uint32_t t = thread_id(), chunk = chunk_of(s), pieces = s.pieces;
  const uint32_t chunks = (pieces + chunk - 1) / chunk;
  float2 v[kNarrow];
  uint32_t turn = 0;
#pragma unroll 1
  for (uint32_t r0 = 0; r0 < s.rows; r0 += kBlockRows, turn ^= 1u) {  // blocks take turns in two buffers; a phase of several chunks has one
    const uint32_t n = min(kBlockRows, s.rows - r0);
    float* const part = st.part + turn * (kBlockRows * 4);
    // x goes two chunks ahead of the sums and is polled before the sums that its place in the ring waits for
#pragma unroll 1
    for (uint32_t i = r0 ? 2 : 0; i < chunks + 2; ++i) {
      if (i < chunks && (i * chunk) % kNarrow == 0) fetch_x(st, l, ph, t, i * chunk, v);
      if (i >= 2) {
#pragma unroll 1
        for (uint32_t r = 0; r < n; r += kTileRows, acc.next(kAcc))
          if (((r / kTileRows) & 1u) == (t >> 7)) take_tile(st, acc, t, min(kTileRows, (n - r + 1) & ~1u), i - 2, i != 2, part + r);
      }
      if (i < chunks) put_x(st, xc, t, min(chunk, pieces - i * chunk), i, v);
    }
    sync();
    if ((t & ~31u) < (n + 1) / 2) {
      float rms = 1.f;
      if (ph != PH_O && ph != PH_DOWN) {
        float4 ss = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (uint32_t i = 0; i < kThreads / 128; ++i) {
          const float4 o = *reinterpret_cast<const float4*>(&st.sh.squares[i * 128 + (t & 31) * 4]);
          ss = make_float4(ss.x + o.x, ss.y + o.y, ss.z + o.z, ss.w + o.w);
        }
        rms = sqrtf(__fdiv_rn(warp_sum((ss.x + ss.y) + (ss.z + ss.w)), (float)s.K) + p.eps);
      }
      float2 v = make_float2(0.f, 0.f);
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
        const float2 o = *reinterpret_cast<const float2*>(part + i * kBlockRows + 2 * min(t, kBlockRows / 2 - 1));
        v.x += o.x;
        v.y += o.y;
      }
      if (t < (n + 1) / 2)
        finish_pair<D>(st, l, ph, s.row0 + r0 + 2 * t, ph == PH_HEAD ? t : r0 / 2 + t, __fdiv_rn(v.x, rms), __fdiv_rn(v.y, rms), 2 * t + 1 < n);
    }
  }
}

// ---- attention -------------------------------------------------------------------------------------------------------------
using attn_detail::kNegBig;
using KV8 = attn_detail::KV8<__half>;
// as the cache will hold it
__device__ __forceinline__ float as_cached(float v) { return __half2float(__float2half_rn(v)); }

// Positions a CTA takes before the range is split: two batches of what its lanes request at once. Splitting costs a hand-over
// (the merge), a batch more about as much.
constexpr uint32_t kRequests = 4;  // of a lane, each for keys and values
constexpr uint32_t attn_batch(uint32_t d) { return kWarps * (32 / (d / 8)) * kRequests; }

template <int D>
__device__ __forceinline__ void attention(const Step& st, uint32_t l) {
  constexpr uint32_t LPP = D / 8, PPW = 32 / LPP, UNR = kRequests, NW = kWarps, SSTR = D + 4;  // lanes of a position, positions of a warp
  const ResidentArgs& p = st.sh.p;
  const uint32_t seq = st.sh.pos + 1;
  uint32_t chunk = (seq + p.splits - 1) / p.splits;
  chunk = max(chunk, attn_batch(D));
  if (seq <= 2 * attn_batch(D)) chunk = seq;
  const uint32_t S = (seq + chunk - 1) / chunk, items = p.qH * S, kvDim = p.kvH * D;
  float* const wpart = st.work;              // [NW][SSTR]
  float* const qs = st.work + NW * SSTR;     // query, newest key, newest value
#pragma unroll 1
  for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
    const uint32_t s = item / p.qH, h = item - s * p.qH, g = h / (p.qH / p.kvH);
    const uint32_t t1 = min(seq, (s + 1) * chunk), newest = seq - 1;
    const uint32_t tid = thread_id(), lane = tid & 31, warp = tid >> 5, grp = lane / LPP, sub = lane % LPP;
    uint32_t base = s * chunk + warp * PPW;
    const __half* kc = layer_cache<D>(p, p.kc, l) + g * D + sub * 8;
    const __half* vc = layer_cache<D>(p, p.vc, l) + g * D + sub * 8;
    KV8::Raw kr[UNR], vr[UNR];
    auto request = [&]() {
#pragma unroll
      for (uint32_t u = 0; u < UNR; ++u) {
        const uint32_t t = base + u * (NW * PPW) + grp;
        const bool there = t < t1 && t != newest;
        kr[u] = there ? KV8::ld<true>(kc + (size_t)t * kvDim) : KV8::zero();
        vr[u] = there ? KV8::ld<true>(vc + (size_t)t * kvDim) : KV8::zero();
      }
    };
    const float scale = 1.0f / sqrtf((float)D);
    float q[8], acc[8], m = kNegBig, ls = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = q[e] = 0.f;
    auto take = [&](const float (&kf)[8], const float (&vf)[8], bool live) {
      float dot = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) dot = fmaf(q[e], kf[e], dot);
#pragma unroll
      for (uint32_t o = 1; o < LPP; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      if (live) {
        const float sc = dot * scale;
        const float m_new = fmaxf(m, sc);
        const float alpha = __expf(m - m_new), pr = __expf(sc - m_new);
        ls = fmaf(ls, alpha, pr);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = fmaf(acc[e], alpha, pr * vf[e]);
        m = m_new;
      }
    };
#pragma unroll 1
    for (bool first = true;; first = false) {
      request();
      if (first) {
        sync();  // (what the work area held before is no longer read)
        if (tid < 3 * D / 2) {  // the query, and the KV head's newest rows
          const uint32_t i = 2 * tid, part = i / D, e = i % D;
          float2 v[1];
          st.poll<1>(layer_words(p, l + 1) + (part == 0 ? h * D : p.qH * D + (part - 1) * kvDim + g * D) + e, 1, v);
          *reinterpret_cast<float2*>(qs + i) = part == 0 ? v[0] : make_float2(as_cached(v[0].x), as_cached(v[0].y));
        }
        sync();
#pragma unroll
        for (int e = 0; e < 8; ++e) q[e] = qs[sub * 8 + e];
      }
#pragma unroll
      for (uint32_t u = 0; u < UNR; ++u) {
        const uint32_t t = base + u * (NW * PPW) + grp;
        if (base + u * (NW * PPW) >= t1) break;  // the whole warp
        float kf[8], vf[8];
        KV8::unpack(kr[u], kf);
        KV8::unpack(vr[u], vf);
        take(kf, vf, t < t1 && t != newest);
      }
      base += NW * PPW * UNR;
      if (base >= t1) break;
    }
    if (t1 == seq && warp == NW - 1) {
      float kf[8], vf[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        kf[e] = qs[D + sub * 8 + e];
        vf[e] = qs[2 * D + sub * 8 + e];
      }
      take(kf, vf, grp == 0);
    }
    // lane groups of the warp, then warps
#pragma unroll 1
    for (uint32_t o = LPP; o < 32; o <<= 1) {
      const float m_o = __shfl_xor_sync(0xffffffffu, m, o), l_o = __shfl_xor_sync(0xffffffffu, ls, o);
      const float m_new = fmaxf(m, m_o), a = __expf(m - m_new), b = __expf(m_o - m_new);
      ls = ls * a + l_o * b;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = acc[e] * a + __shfl_xor_sync(0xffffffffu, acc[e], o) * b;
      m = m_new;
    }
    if (grp == 0) {
      float* wp = wpart + warp * SSTR + sub * 8;
      *reinterpret_cast<float4*>(wp) = make_float4(acc[0], acc[1], acc[2], acc[3]);
      *reinterpret_cast<float4*>(wp + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
      if (sub == 0) *reinterpret_cast<float2*>(wpart + warp * SSTR + D) = make_float2(m, ls);
    }
    sync();
    if (tid < D) {
      float M = kNegBig, o = 0.f, Ls = 0.f;
#pragma unroll
      for (uint32_t x = 0; x < NW; ++x) M = fmaxf(M, wpart[x * SSTR + D]);
#pragma unroll
      for (uint32_t x = 0; x < NW; ++x) {
        const float* wp = wpart + x * SSTR;
        const float sc = __expf(wp[D] - M);
        Ls = fmaf(wp[D + 1], sc, Ls);
        o = fmaf(wp[tid], sc, o);
      }
      if (S == 1) {
        st_word(layer_words(p, l + 1) + words_att(p) + h * D + tid, o * (1.0f / Ls), st.sh.tag);
      } else {
        uint2* pw = layer_words(p, l + 1) + words_part(p) + ((size_t)h * p.splits + s) * (D + 2);
        st_word(pw + tid, o, st.sh.tag);
        if (tid == 0) st_words(pw + D, M, Ls, st.sh.tag);
      }
    }
    sync();
  }
  if (S == 1) return;
  // every CTA merges its share of its head's elements
#pragma unroll 1
  for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) {
    const uint32_t s = item / p.qH, h = item - s * p.qH;
    const uint32_t i = D * s / S + thread_id();
    if (i >= D * (s + 1) / S) continue;
    const uint2* pw = layer_words(p, l + 1) + words_part(p) + (size_t)h * p.splits * (D + 2);
    float M = kNegBig, Ls = 0.f, o = 0.f;
#pragma unroll 1
    for (uint32_t k0 = 0; k0 < S; k0 += 4) {  // online over groups of four ranges, their words polled together
      uint4 w[8];  // the sum of element i beside its neighbour's; m and l
#pragma unroll
      for (int k = 0; k < 4; ++k) w[2 * k] = w[2 * k + 1] = make_uint4(0, k0 + k < S ? ~st.sh.tag : st.sh.tag, 0, st.sh.tag);
      poll_words<8>(st.sh, p.state, st.sh.tag, [&](int x) { return reinterpret_cast<const uint4*>(pw + (k0 + x / 2) * (D + 2) + (x & 1 ? D : i & ~1u)); }, w);
      float mx = M;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k0 + k < S) mx = fmaxf(mx, __uint_as_float(w[2 * k + 1].x));
      const float kept = __expf(M - mx);
      Ls *= kept;
      o *= kept;
      M = mx;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k0 + k < S) {
          const float e = __expf(__uint_as_float(w[2 * k + 1].x) - M);
          Ls = fmaf(__uint_as_float(w[2 * k + 1].z), e, Ls);
          o = fmaf(__uint_as_float(i & 1u ? w[2 * k].z : w[2 * k].x), e, o);
        }
      }
    }
    st_word(layer_words(p, l + 1) + words_att(p) + h * D + i, o * (1.0f / Ls), st.sh.tag);
  }
}

// ---- the weights' way into the ring -----------------------------------------------------------------------------------------
// A warp copies this CTA's shares in the order they are used: tile by tile, 512 columns at a time. A slot's copies are begun when it
// is free and the ones kAhead before them have landed: what is in flight keeps HBM busy and no more, because everything else that
// misses L2 (words that were written, gains, K and V) queues behind it. (The whole ring in flight is 4 us of HBM time; it made no
// difference at short positions, 480.0 us a step and 481.1.) The last rows of a share come in boxes of 8, 4 and 2, so that no row is read
// that is another CTA's. (One copy per row instead, 1 KB each, took a step of two layers half as long again: they are issued one by
// one.) The warp's waits are votes: its lanes on their own ahead of one vote took 484.8 us a step, 478.7 so.
__device__ __forceinline__ void feed(const Step& st, const ResidentStep& launch) {
  const ResidentArgs& p = st.sh.p;
  Shared& sh = st.sh;
  unsigned long long once;       // weights are read once a step: they give way to everything else in L2 (502.3 us a step without, 481.1 with)
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
  Cursor c, landed;
  uint32_t begun = 0, seen = 0;  // copies, and those that were waited for
  const uint32_t end = p.L * 4 + (p.with_head ? 1 : 0);
#pragma unroll 1
  for (uint32_t k = 0; k < end; ++k) {
    const uint32_t l = k >> 2, ph = l < p.L ? k & 3u : (uint32_t)PH_HEAD;
    const Share s = sh.share[ph];
    const uint32_t chunk = chunk_of(s);
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < s.pieces; c0 += chunk) {
#pragma unroll 1
      for (uint32_t r = 0; r < s.rows; r += kTileRows) {
        const uint32_t rows = (min(kTileRows, s.rows - r) + 1) & ~1u;
#pragma unroll 1
        for (uint32_t piece = c0; piece < min(s.pieces, c0 + chunk); ++piece, ++begun, c.next(kSlots)) {
          const uint32_t full = s_addr(&sh.full[c.slot]);
          if (begun >= kAhead) {
            if (!st.warp_wait(sh.full[landed.slot], landed.turn)) goto drain;
            landed.next(kSlots);
            ++seen;
          }
          if (begun >= kSlots && !st.warp_wait(sh.empty[c.slot], c.turn ^ 1u)) goto drain;
          if (__any_sync(0xffffffffu, dead(sh) >= 2)) goto drain;  // nothing more goes into a slot that may still be read or written
          if (umma::elect_one()) {
            bar_expect_tx(full, rows * (kPiece * 2));
            uint32_t dst = st.ring + c.slot * kSlotBytes, at = s.row0 + r;
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
              const uint32_t R = kTileRows >> i;
              if (rows & R) {
                copy_box(once, dst, launch.maps[ph][i], (int)at, (int)(piece * kBlocks), ph == PH_HEAD ? 0 : (int)l, full);
                dst += R * (kPiece * 2);
                at += R;
              }
            }
          }
          __syncwarp();
        }
      }
    }
  }
drain:  // nothing is on its way into this CTA's memory when it leaves, neither copies nor the products' arrivals on the slots' barriers
  for (; seen < begun; ++seen, landed.next(kSlots)) st.wait_out(sh.full[landed.slot], landed.turn);
  if (dead(sh) < 2) {  // (else the products of the last copies may never have been issued: kArrivalsNs)
    for (uint32_t i = 0; i < min(begun, kSlots); ++i) st.wait_out(sh.empty[i], (begun - 1 - i) / kSlots & 1u);
  }
}

// ---- the step ----------------------------------------------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(kAllThreads, 1) step_resident_kernel(const __grid_constant__ ResidentStep launch) {
  extern __shared__ __align__(1024) char smem[];
  Shared& sh = *reinterpret_cast<Shared*>(smem + kSharedOffset);
  const Step st{sh, s_addr(smem), s_addr(smem + kXOffset), reinterpret_cast<float*>(smem + kWorkOffset), reinterpret_cast<float*>(smem + kPartOffset)};
  const ResidentArgs& p = sh.p;
  const uint32_t tid = threadIdx.x;
  if (tid == 0) {
    sh.p = launch;
    const uint32_t qDim = p.qH * D, kvDim = p.kvH * D;
    sh.share[PH_QKV] = share_of(qDim + 2 * kvDim, 2, p.H);
    sh.share[PH_O] = share_of(p.H, 2, qDim);
    sh.share[PH_GATEUP] = share_of(2 * p.F, 2, p.H);
    sh.share[PH_DOWN] = share_of(p.H, 2, p.F);
    sh.share[PH_HEAD] = share_of(p.V, 1, p.H);
    sh.dead = 0;
    for (uint32_t i = 0; i < kSlots; ++i) {
      bar_init(s_addr(&sh.full[i]), 1);
      bar_init(s_addr(&sh.empty[i]), 1);
    }
    for (uint32_t i = 0; i < kXSlots; ++i) {
      bar_init(s_addr(&sh.x_full[i]), kWarps);
      bar_init(s_addr(&sh.x_empty[i]), 1);
    }
    for (uint32_t i = 0; i < kAcc; ++i) {
      bar_init(s_addr(&sh.acc_full[i]), 1);
      bar_init(s_addr(&sh.acc_empty[i]), 4);
    }
    bar_init(s_addr(&sh.drained), 1);
    const uint32_t pos = __ldcg(&p.state->pos), tok = p.prompt ? __ldcg(p.prompt + __ldcg(&p.state->prompt_idx)) : __ldcg(&p.state->cur_token);
    sh.tag = __ldcg(p.epoch) + 1;
    sh.keep = pos < p.ctx;
    sh.pos = sh.keep ? pos : p.ctx - 1;
    sh.tok = tok < p.V ? tok : 0;
    if (blockIdx.x == 0 && !sh.keep) atomicOr(&p.state->err, 2u);
    if (blockIdx.x == 0 && tok >= p.V) atomicOr(&p.state->err, 1u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (tid < launch.ropeDim / 2) sh.rope[tid] = __ldg(launch.rope_cs + (size_t)min(__ldcg(&launch.state->pos), launch.ctx - 1) * (launch.ropeDim / 2) + tid);
  if (tid < kBlockRows / 2) {
    sh.best_v[tid] = -INFINITY;
    sh.best_i[tid] = 0xffffffffu;
  }
  for (uint32_t i = tid; i < kXSlots * kXBytes / 16; i += kAllThreads) *reinterpret_cast<uint4*>(smem + kXOffset + 16 * i) = make_uint4(0, 0, 0, 0);
  const uint32_t warp = tid >> 5;
  if (warp == kWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_addr(&sh.tmem)), "r"(kAcc * kAccColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  umma::fence_before();
  __syncthreads();
  umma::fence_after();
  if (warp == kWarps) {
    feed(st, launch);
  } else if (warp == kWarps + 1) {
    issue_products(st);
    // the last products, and their arrivals on the barriers of x, before the memory goes
    if (umma::elect_one()) umma::umma_commit(s_addr(&sh.drained));
    __syncwarp();
    st.wait_out(sh.drained, 0);
    if (dead(sh) >= 2) {  // arrivals of products that are done, on barriers that are not waited for any more
      const unsigned long long t0 = global_timer_ns();
      while (global_timer_ns() - t0 < kArrivalsNs) {}
    }
  } else {
    {  // this CTA's columns of the embedding row
      const uint32_t i = 2 * tid, at = sh.share[PH_O].row0 + i;
      if (i < sh.share[PH_O].rows) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(reinterpret_cast<const __half*>(p.embd) + (size_t)sh.tok * p.H + at));
        st_words(layer_words(p, 0) + words_out(p) + at, v.x, v.y, sh.tag);
        *reinterpret_cast<float2*>(p.xbuf + at) = v;
      }
    }
    Cursor xc, acc;
    const uint32_t end = p.L * 4 + (p.with_head ? 1 : 0);
#pragma unroll 1
    for (uint32_t k = 0; k < end; ++k) {
      const uint32_t l = k >> 2, ph = l < p.L ? k & 3u : (uint32_t)PH_HEAD;
      if (ph == PH_O) {
        attention<D>(st, l);
        sync();
      }
      product<D>(st, xc, acc, l, ph);
      sync();
    }
    if (warp == 0 && dead(sh) < 2)  // (the products' arrivals on the last pieces of x)
      for (uint32_t i = 0; i < kXSlots; ++i, xc.next(kXSlots)) st.wait_out(sh.x_empty[xc.slot], xc.turn ^ 1u);
  }

  umma::fence_before();
  __syncthreads();
  if (warp == kWarps + 1) {
    umma::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem), "r"(kAcc * kAccColumns));
  }
  // ---- arg-max and the state of the next step, by the CTA that comes last
  if (tid >= 32) return;
  float bv = -INFINITY;
  uint32_t bi = 0xffffffffu;
  auto reduce = [&]() {
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
      take_best(bv, bi, ov, oi);
    }
  };
  if (p.with_head) {
    for (uint32_t i = tid; i < kBlockRows / 2; i += 32) take_best(bv, bi, sh.best_v[i], sh.best_i[i]);
    reduce();
  }
  uint32_t last = 0;
  if (tid == 0) {
    if (p.with_head) {
      p.part_val[blockIdx.x] = bv;
      p.part_idx[blockIdx.x] = bi;
    }
    __threadfence();
    last = atomicAdd(p.ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
    __threadfence();
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return;
  if (p.with_head) {
    bv = -INFINITY;
    bi = 0xffffffffu;
    for (uint32_t i = tid; i < gridDim.x; i += 32) take_best(bv, bi, __ldcg(p.part_val + i), __ldcg(p.part_idx + i));
    reduce();
  }
  if (tid == 0) {
    StepState* state = p.state;
    if (p.with_head) {
      const uint32_t token = bi == 0xffffffffu ? 0u : bi;
      if (state->steps < p.history_cap) p.history[state->steps] = token;
      state->last_argmax = token;
      state->cur_token = token;  // greedy feedback: the next step embeds this token unless the host overwrites it
      state->steps += 1;
    } else {
      state->prompt_idx += 1;
    }
    state->pos += 1;
    *p.ticket = 0;
    *p.epoch += 1;
  }
}

using Kernel = void (*)(const ResidentStep);
Kernel pick(uint32_t d) { return d == 32 ? step_resident_kernel<32> : d == 64 ? step_resident_kernel<64> : step_resident_kernel<128>; }

}  // namespace

// Positions up to which this kernel's attention keeps the step ahead of the sequence of launches. What grows with them is a CTA's
// share of a head, position / splits rows of d keys and values, read while no product has its x: the line is at 65 536 elements of each.
// us a step, launches and this kernel: 1B (32 heads of 64, 4 ranges: 4 096) at 4 070 666 and 651; 3B (24 of 128, 6 ranges: 3 072) at
// 3 060 1 691 and 1 675, 3 400 1 713 and 1 706, 4 000 1 736 and 1 774; 8B (32 of 128, 4 ranges: 2 048) at 1 600 3 052 and 3 039,
// 1 900 3 055 and 3 079, 3 060 3 150 and 3 217; 7B with as many KV heads at 2 300 2 883 and 2 873, 2 500 2 896 and 2 903; 8 layers
// with 64 heads of 64 (2 ranges: 2 048), 8 KV heads: 2 800 728 and 719, 3 100 736 and 739, 64 KV heads: 1 300 786 and 776, 1 600 794 and 805.
uint32_t resident_positions(const ResidentArgs& p) { return std::min(65536u * p.splits / p.d, 4096u); }

uint32_t resident_splits(uint32_t qH) {
  const uint32_t s = sm_count() / qH;
  return s < 1 ? 1 : s > 16 ? 16 : s;
}

size_t resident_words_per_layer(uint32_t H, uint32_t qH, uint32_t kvH, uint32_t d, uint32_t F) {
  return (size_t)2 * qH * d + 2 * kvH * d + 2 * H + F + (size_t)qH * resident_splits(qH) * (d + 2);
}

bool resident_plan(int wdtype, int kvdtype, ResidentStep* p) {
  const uint32_t qDim = p->qH * p->d, G = sm_count();
  // Sums inside the tensor core lose more than sums in registers, the more the longer they are. A float16 cache rounds by a thousand times
  // as much, and logits are off by the same either way; with a float32 cache they were off by more (1B architecture, two layers, position
  // 0: 7.1e-7 for 4.8e-7 as launches, one layer's rows 8.5e-7 for 3.4e-7). Shorter sums, a 512-column piece each, are as exact as
  // the launches and take what the one kernel gains (480 -> 546 us a step).
  if (wdtype != 1 || kvdtype != 1) return false;
  if (p->d != 32 && p->d != 64 && p->d != 128) return false;
  if (p->H % 64 || qDim % 64 || p->F % 64) return false;  // rows of whole blocks of 64 columns
  if (p->H > kMaxNarrow || qDim > kMaxNarrow || p->F > kMaxWide) return false;
  // Weights of a layer that are worth it even if it is the only one and stays in L2: layers of 18 MB, position 128, launches and this
  // kernel: one layer 24.8 and 28.9 us a step, two 43.2 and 45.3, four 82.2 and 73.9; of 39 MB: 32.9 and 33.0, 56.4 and 51.4; of 56
  // MB: 35.1 and 35.9, 61.2 and 56.1; of 116 MB: 45.1 and 43.9, 78.1 and 71.8.
  if (((uint64_t)p->H * (2 * qDim + 2 * p->kvH * p->d) + (uint64_t)3 * p->H * p->F) * 2 < (32u << 20)) return false;
  if (p->H / 2 / G + 1 > 32) return false;                // the kept residual; rows of down are one block
  if (p->H / 2 < G || (p->qH + 2 * p->kvH) * p->d / 2 < G || p->F < G || p->V < G) return false;  // no CTA without a row
  int dev = 0, limit = 0, coop = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return false;
  if (kSmem > (uint32_t)limit) return false;
  p->splits = resident_splits(p->qH);
  p->words_per_layer = (uint32_t)resident_words_per_layer(p->H, p->qH, p->kvH, p->d, p->F);
  const uint64_t rows[kPhases] = {qDim + 2 * p->kvH * p->d, p->H, 2 * p->F, p->H, p->V}, cols[kPhases] = {p->H, qDim, p->H, p->F, p->H};
  for (int i = 0; i < kPhases; ++i)
    for (int b = 0; b < 4; ++b)
      if (!encode_stack_map16(reinterpret_cast<CUtensorMap*>(p->maps[i][b]), p->w[i], rows[i], cols[i], i == PH_HEAD ? 1 : p->L, p->layer_stride, kTileRows >> b, kPiece / 64))
        return false;
  const Kernel k = pick(p->d);
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, (int)kAllThreads, kSmem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return false;
  }
  return true;
}

cudaError_t launch_step_resident(cudaStream_t s, const ResidentStep& p) {
  const Kernel k = pick(p.d);
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sm_count());
  cfg.blockDim = dim3(kAllThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, p);
}

}  // namespace nfai
