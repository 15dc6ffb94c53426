// One generation step of a GPT-2 model (one new token for each of up to 8 sequences) as ONE
// persistent kernel: embedding, every transformer block over the K/V caches, final LayerNorm and
// the vocabulary head.
//
// The arithmetic is that of the reference's modules (src/py/model_inference.py:39-190: pre-LN
// blocks, LayerNorm :96-107, tanh GELU :109-117), evaluated for a single position per sequence
// with the keys and values of earlier positions cached.
//
// What bounds it: every weight is read once per step (GPT-2 XL: 3.1 GB, 0.48 ms at the measured
// copy bandwidth), and a layer is five dependent operations across all SMs, each at least one trip
// through L2 (about 1000 clocks one way and the wait for it).  As one launch per operation the step
// is 250 kernels, each of which starts with an idle memory system.
//
//   stream       Four warps per CTA run through the CTA's share of ALL weights and of the cached keys
//                and values in order and copy it into a ring of shared-memory stages; they wait only
//                for ring slots, never for the other CTAs, and fill the ring while those wait.  (One
//                warp, or a lane per row, does not issue the copies fast enough: 1000 clocks a stage.)
//   exchange     No barrier between the operations.  Every value that one CTA hands to others is a
//                32-bit word, bf16 in the upper half and the generation of its buffer in the lower:
//                a reader loads the words it needs and loads again until the generation is right.
//                One trip instead of the four of data, fence, counter and poll.  A buffer is
//                written again only by CTAs that hold something which depends on everybody's having
//                read it (its reader's own output, a few operations on).
//   work split   Output columns of a layer (rows of W) are cut evenly over the CTAs, so a CTA's
//                share is one contiguous piece of W.  It is taken in tiles of at most 12 rows, K in
//                pieces of d_model columns or half of that where they are more than 800: a ring stage.
//   ahead        Before an operation's weights go into the ring, the next one's are sent for as far as
//                L2: the ring is too short (154 KB of the 415 KB a CTA reads per XL layer) to keep the
//                memory busy while the operations wait for one another.  One operation ahead: XL 785
//                us per step against 832 without and 790 with two (before the ring and the split were
//                as they are now: 985, 1085, 1014, and 1152 and 1255 with three and four); with the
//                cached rows sent for in the same way it was slower, 2030 against 1860 at 8 sequences.
//   tensor path  mma.sync m16n8k16 with W as the 16-row operand and the (up to 8) tokens as the
//                8-column operand: at 8 tokens a scalar product per weight costs more issue slots
//                than the stream leaves.  tcgen05 needs 64 or 128 rows of one operand per CTA and
//                gives nothing here, the memory pipe is the limit.  The 8 warps split K: a warp has the
//                same part of every row, which lies in one ring stage, so it waits for one barrier
//                per tile, holds its input in registers over all tiles, and the partial tiles meet in
//                shared memory.  Per step of GPT-2 small / XL, 1 sequence, 100 rows, us: 242 / 1138
//                with 16 warps that all go over all stages, 228 / 1083 with 8, 178 / 1078 with a
//                warp to a whole stage (shared memory is the limit for XL: the input is read again
//                for every tile), 153 / 770 like this.
//   attention    a (sequence, head) pair per CTA, up to two where there are more pairs than CTAs,
//                split over several CTAs from 768 rows on.  q.K on the tensor
//                path with the cached rows as the 16-row operand, P.V on packed fp32.  The cached
//                rows come through the ring, ahead of the query; the new row comes through the
//                exchange, so nobody waits for the caches.
//   precision    bf16 weights, activations rounded to bf16 where the layer-by-layer path rounds
//                them, fp32 accumulation; the residual stream accumulates in fp32 in the shared
//                memory of the CTA that owns the column.
//   what counts  Between two exchanges a warp runs a few hundred instructions at 4 to 8 clocks each
//                (dependent, few warps): their number, the trips to L2 and the CTA barriers are the
//                time.  Nothing but an operation's own input is fetched after that input, and
//                nothing may spill: shared memory leaves so little L1 that a spilled register costs
//                a trip to L2 (a build with 300 bytes of spills per thread took 2.5 ms per GPT-2 XL
//                step).  step_tid keeps one operation's addresses out of the other's registers.
//
// The grid is launched cooperatively (CTAs wait on one another).  Every wait is bounded: one that
// runs out leaves its code in the status words and the kernel drains.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "add_layernorm_sm100.cuh"   // ln_unpack8
#include "fa_fwd_sm100.cuh"          // Watch and the watchdog codes
#include "linear_small_sm100.cuh"    // gelu_tanh

namespace fa {

constexpr int kStepWarps = 8;                         // computing warps
constexpr int kStepLgWarps = 3;
static_assert(kStepWarps == 1 << kStepLgWarps, "warps are divided by shifts");
constexpr int kStepCompute = kStepWarps * 32;
constexpr int kStepStreamWarps = 4;
constexpr int kStepThreads = kStepCompute + 32 * kStepStreamWarps;
// Registers: the computing warpgroups take what the streaming one gives up.  (setmaxnreg.inc waits
// without a limit for registers of this CTA's launch allocation, hence the check; the host refuses a
// build whose launch allocation is another.)
constexpr int kStepLaunchRegs = 168, kStepComputeRegs = 216, kStepStreamRegs = 40;
static_assert(kStepCompute * kStepComputeRegs + 32 * kStepStreamWarps * kStepStreamRegs <= kStepThreads * kStepLaunchRegs,
              "setmaxnreg budget exceeds the launch allocation: the kernel would hang");
constexpr int kStepMaxRows = 8;                       // sequences (the 8-column side of the MMA)
constexpr int kStepMaxLayers = 64;
constexpr int kStepMaxPairs = 256;                    // (sequence, head) pairs
constexpr int kStepMaxVocab = 1 << 24;                // step_cut multiplies row counts by block indices in 32 bits
constexpr int kStepTile = 12;                         // rows of W per stage (of the MMA's 16)
constexpr int kStepMmaRows = 16;
constexpr int kStepGroup = 4;                         // tiles whose partial sums are added up together
constexpr int kStepRedPitch = 20;                     // partial tiles: [token][row], conflict-free for the MMA's layout
constexpr int kStepRed = kStepRedPitch * kStepMaxRows;
constexpr int kStepOutputs = kStepMmaRows * kStepMaxRows;
constexpr int kStepUnit = 32;                         // columns of W per warp step: 64 bytes
constexpr int kStepChunkUnits = 25;                   // columns per stage: at most 800
constexpr int kStepStageBytes = kStepTile * kStepChunkUnits * 64;
constexpr int kStepStages = 8;                        // one per warp: a group of tiles has at most as many
static_assert(kStepStages >= kStepWarps, "a wait by parity is for the slot's next stage only while the one before is not given back");
constexpr uint32_t kStepAheadBytes = 192 * 1024, kStepAheadPiece = 2048;
constexpr int kStepMaxWidth = 1600;                   // d_model: the fragments of 8 rows fill sm.x
constexpr int kStepMaxUnits = kStepMaxWidth / kStepUnit;
constexpr int kStepQuads = (kStepMaxWidth / 4 + 31) / 32;     // 13: columns / 4 of a row per lane of a warp
constexpr int kStepTake = 8;                          // words of a batch: 32 lanes x kStepTake x 4
constexpr int kStepSegs = 2;                          // attention units of one CTA
constexpr int kStepBlocks = 4;                        // blocks of 16 cached rows (K, then V) per stage
static_assert(kStepBlocks == kStepWarps / 2 && kStepStages % 2 == 0, "half the warps to a stage, by the slot's parity");
static_assert(kStepBlocks * 16 * 256 <= kStepStageBytes, "cached rows fit a stage");
// Rows of a unit where pairs are split over CTAs, from twice as many on.  Merging costs a fence and an
// atomic per part: 1 x 900 rows, small / XL, us per step: unsplit 204 / 997, parts of 384 191 / 927, of
// 192 191 / 956.
constexpr int kStepSplitRows = 384;
// Bounds of the waits: of barriers by the clock (a poll of one may suspend the thread), of exchange words by
// their number (a trip to L2 each, 0.3 to 1 us).  A wait behind one that has run out runs out as well.
#ifdef FA_WAIT_TEST
// Test build: short waits, and block 0 keeps back its words of the embedding, for which every block waits.
constexpr uint32_t kStepWaitNs = 2u * 1000 * 1000, kStepWordPolls = 1u << 12;
constexpr bool kStepKeepsBack = true;
#else
constexpr uint32_t kStepWaitNs = 500u * 1000 * 1000, kStepWordPolls = 1u << 21;
constexpr bool kStepKeepsBack = false;
#endif

// Rows of a stage lie 64 bytes (mod 128) apart: the 8 lanes of a 128-bit load phase read two rows of
// 64 bytes each, which then cover all banks (an even `units` is at most 24).
constexpr int step_pitch(int units) { return units * 64 + ((units & 1) ? 0 : 64); }

struct StepLayer {       // one transformer block's parameters (device memory, built once per model)
  const __nv_bfloat16 *ln1_g, *ln1_b, *qkv_w, *qkv_b, *proj_w, *proj_b;
  const __nv_bfloat16 *ln2_g, *ln2_b, *fc_w, *fc_b, *out_w, *out_b;
};

struct StepParams {
  const StepLayer* layers;
  const __nv_bfloat16 *tok_emb, *pos_emb, *lnf_g, *lnf_b, *head_w;
  const long long* ids;            // [M], ids_stride apart
  long long ids_stride;
  long long* pos_ptr;              // device position (cache row of the new token), or null: `pos`
  int* len_ptr;                    // with pos_ptr and advance: set to the new length + 1
  int pos, advance;
  int n_layers, C, H, V, M;
  int stage_units, lg_chunks;      // units of 32 columns per ring stage, stages per d_model columns: 1 or 2
  int stage_pitch;                 // bytes between a stage's rows, see step_pitch
  int batch_units;                 // units whose exchange words a warp takes at once
  float inv_c;                     // 1 / C
  int cache_rows, n_positions;
  float eps, scale_log2;
  long long c_sb;                  // cache strides in elements: sequence, row, head
  int c_sn, c_sh;
  // workspace: the exchange buffers (words: bf16 << 16 | generation) ...
  uint32_t *x_att, *x_mlp;         // [M][C] residual stream after attention and after the MLP (or embedding)
  uint32_t* qkv;                   // [M][3C]
  uint32_t* ctx;                   // [C / 32][M][32]: fragment order
  uint32_t* h;                     // [4C / 32][M][32]
  uint32_t* generation;            // of the last launch's last layer
  // ... and what is behind fences
  float* part_o;                   // [pairs * splits, 64]
  float2* part_ml;                 // [pairs * splits]
  unsigned int* arrived;           // per pair: CTAs whose partial is in; zero between launches
  unsigned long long* best;        // [8] packed argmax keys
  unsigned int* done;              // CTAs that have delivered their argmax
  long long* next_ids;             // argmax of the logits, M ids next_stride apart, or null
  long long next_stride;
  __nv_bfloat16* logits;           // [M, V]
  unsigned int* status;
  __nv_bfloat16* k_cache[kStepMaxLayers];
  __nv_bfloat16* v_cache[kStepMaxLayers];
};

// How a [N, K] weight is cut: rows of this CTA, tiles of `tile` rows, taken in groups of 1 << lg_group.
struct __align__(16) StepCut {
  int row0, rows;
  short tiles, tile;
  int lg_group;
};
__device__ __forceinline__ StepCut step_cut(int N, bool head) {          // N < kStepMaxVocab, grid <= 160
  StepCut c;
  c.row0 = static_cast<int>(blockIdx.x * static_cast<uint32_t>(N) / gridDim.x);
  c.rows = static_cast<int>((blockIdx.x + 1) * static_cast<uint32_t>(N) / gridDim.x) - c.row0;
  const int tiles = (c.rows + kStepTile - 1) / kStepTile;
  c.tiles = static_cast<short>(tiles);
  c.tile = static_cast<short>(tiles > 0 ? (c.rows + tiles - 1) / tiles : 0);
  c.lg_group = 0;
  while ((1 << c.lg_group) < (head ? kStepGroup : min(tiles, kStepGroup))) ++c.lg_group;
  return c;
}
// Which columns of a row are a warp's: `units` units from unit `first`, in ring stage `stage` of the
// 1 << lg_stages that hold a tile, from unit `at` of that stage.
struct StepPart {
  int stage, lg_stages, first, units, at;
  __device__ __forceinline__ StepPart(int warp, int lg, int stage_units) {
    lg_stages = lg;
    stage = warp >> (kStepLgWarps - lg);
    const int parts = kStepWarps >> lg, per = (stage_units + parts - 1) / parts;
    at = (warp & (parts - 1)) * per;
    units = max(min(per, stage_units - at), 0);
    first = stage * stage_units + at;
  }
};

enum StepOp : int { kStepQkv = 0, kStepProj = 1, kStepFc = 2, kStepOut = 3, kStepHead = 4 };

// How the attention over the `rows` earlier positions is cut: `splits` units per (sequence, head)
// pair, the units evenly over the first CTAs; a CTA has at most kStepSegs.
struct StepAttnCut {
  int rows, splits;
  int first, count;                      // units of this CTA
  __device__ __forceinline__ StepAttnCut(int pairs, int earlier) {
    rows = earlier;
    splits = min(static_cast<int>(gridDim.x) / pairs, (rows + kStepSplitRows - 1) / kStepSplitRows);
    if (splits < 1 || rows < 2 * kStepSplitRows) splits = 1;
    const int units = pairs * splits, ctas = min(static_cast<int>(gridDim.x), units);
    first = count = 0;
    if (static_cast<int>(blockIdx.x) < ctas) {
      first = blockIdx.x * units / ctas;
      count = (blockIdx.x + 1) * units / ctas - first;
    }
  }
};
// A unit's rows and addresses: the same in every layer, worked out once.
struct StepUnit {
  long long head;                        // offset of the head in a cache, elements
  int pair, slot;                        // which of the pair's units
  int row0, rows;
  int query;                             // offset of the pair's q in p.qkv
  int out;                               // offset of its output in p.ctx
};

struct __align__(128) StepSmem {
  uint8_t ring[kStepStages][kStepStageBytes];
  uint4 x[kStepMaxUnits * 32];                              // LayerNorm's output as MMA fragments
  float red[kStepGroup][kStepWarps][kStepRed];              // partial tiles of the warps
  float red_one[kStepWarps][kStepRed];                      // ... where the input comes through the exchange
  float seg[kStepSegs][kStepWarps + 1][68];                 // attention partials: m, l, -, -, o[64]
  uint2 norm[2][kStepMaxWidth / 4];                         // scale and shift of the coming LayerNorm
  alignas(16) float2 stat[kStepWarps];                      // LayerNorm: sums of a warp's part
  float own[kStepOutputs];                                  // this CTA's columns of the residual stream
  unsigned long long keys[kStepMaxRows][2];                 // best logits: a token's of two warps
  StepUnit unit[kStepSegs];                                 // this CTA's attention units
  int units, splits;
  StepCut cut[5];                                           // by StepOp
  StepLayer layers[kStepMaxLayers];
  uint64_t full[kStepStages];
  uint64_t empty[kStepStages];
  uint32_t seg_last;                                        // the CTA completes its pair
  uint32_t abort, abort_who;
};
constexpr int kStepSmemBytes = sizeof(StepSmem) + 128;
static_assert(kStepSmemBytes <= 227 * 1024, "one CTA per SM");

enum StepWaitId : uint32_t { kWaitStepFull = 17, kWaitStepEmpty = 18, kWaitStepWords = 19 };

// The thread index, read anew: what is computed from it stays in the operation that computes it
// instead of being hoisted out of the loop over the operations.
__device__ __forceinline__ int step_tid() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}
__device__ __forceinline__ void step_bar() {           // the computing warps only
  asm volatile("bar.sync 1, %0;" ::"n"(kStepCompute) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t a) {
  uint4 r;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(a) : "memory");
  return r;
}
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(reinterpret_cast<uint64_t>(src)) : "memory");
}
// Untiled bulk copy global -> shared (both 16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               :: "r"(dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar) : "memory");
}
// (16-byte aligned, a multiple of 16 bytes)
__device__ __forceinline__ void bulk_prefetch_l2(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<uint64_t>(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<uint64_t>(p)));
}

struct StepRing {
  uint32_t stage = 0, parity = 0;
  __device__ __forceinline__ void next() {
    if (++stage == kStepStages) { stage = 0; parity ^= 1; }
  }
  __device__ __forceinline__ void skip(uint32_t n) {      // n <= kStepWarps
    stage += n;
    if (stage >= kStepStages) { stage -= kStepStages; parity ^= 1; }
  }
  __device__ __forceinline__ void skip_any(uint32_t n) {
    stage += n;
    parity ^= (stage / kStepStages) & 1;
    stage %= kStepStages;
  }
};

struct StepCta {            // what a computing warp carries from operation to operation
  StepSmem* sm;
  StepRing ring;
  bool ok;                  // false: a wait has run out somewhere in the CTA, wait for nothing more
};

__device__ __forceinline__ void step_give_up(StepSmem& sm, uint32_t id) {
  volatile uint32_t* abort = &sm.abort;
  if (*abort == 0) {
    sm.abort_who = threadIdx.x;
    *abort = kWatchdogBase | id;
  }
}
// A bounded wait of a converged warp, small because it is inlined in the loops.  (A step of GPT-2 small, 1
// sequence / XL, 8 sequences at 900 rows, us: 148.4 / 1451 with the clock read at every poll but the first,
// 148.8 / 1455 at every 256th, 152.5 / 1466 at every 64th in one loop; by a count of polls 147.9 / 1460.)
__device__ __forceinline__ bool step_wait(uint32_t bar, uint32_t parity, StepSmem& sm, uint32_t id) {
  bool ok = mbar_try_wait(bar, parity);
  if (!ok) {
    const uint32_t since = globaltimer_lo_ns();
#pragma unroll 1
    do ok = mbar_try_wait(bar, parity);
    while (!ok && globaltimer_lo_ns() - since < kStepWaitNs);
  }
  ok = __all_sync(0xffffffffu, ok);
  if (!ok) step_give_up(sm, id);
  return ok;
}

// ------------------------------------------------------------------------------ exchange words
__device__ __forceinline__ uint32_t step_word(float v, uint32_t gen) {
  return (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v))) << 16) | gen;
}
__device__ __forceinline__ void step_put(uint32_t* dst, float v, uint32_t gen) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(dst), "r"(step_word(v, gen)) : "memory");
}
__device__ __forceinline__ uint4 step_peek(const uint32_t* src) {       // four words, past L1
  uint4 r;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(src) : "memory");
  return r;
}
__device__ __forceinline__ uint32_t step_stale(const uint4& w, uint32_t gen) {    // 0: all of this generation
  return ((w.x ^ gen) | (w.y ^ gen) | (w.z ^ gen) | (w.w ^ gen)) & 0xffffu;
}
__device__ __forceinline__ uint32_t step_pair(uint32_t lo, uint32_t hi) {         // two words' values as bf16x2
  return __byte_perm(lo, hi, 0x7632);
}
// Asynchronous copies of this thread so far: the barrier's phase cannot complete before they have.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
// (Only by warps whose waits have been met: others would arrive out of turn, more often than a phase has
// arrivals left.  Where one has run out the stream's waits run out too.)
__device__ __forceinline__ void mbar_arrive_many(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void st_shared_v2(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
// Loads kN times four words, the i-th from at(i), until all have this generation.
template <int kN, class At>
__device__ __forceinline__ void step_take(StepCta& c, uint32_t gen, uint4 (&w)[kN], At at) {
#pragma unroll 1
  for (uint32_t polls = 0;; ++polls) {
    uint32_t bad = 0;
#pragma unroll
    for (int i = 0; i < kN; ++i) w[i] = step_peek(at(i));
#pragma unroll
    for (int i = 0; i < kN; ++i) bad |= step_stale(w[i], gen);
    if (!c.ok || !__any_sync(0xffffffffu, bad != 0)) break;
    if (polls >= kStepWordPolls || *const_cast<volatile uint32_t*>(&c.sm->abort)) {
      step_give_up(*c.sm, kWaitStepWords);
      c.ok = false;
    }
  }
}

__device__ __forceinline__ unsigned long long step_key(float v, int n) {
  // orders by value (NaN above all, as torch.argmax has it), then by the lower index
  uint32_t b = __float_as_uint(v);
  b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  if (v != v) b = 0xffffffffu;
  return (static_cast<unsigned long long>(b) << 32) | (0xffffffffu - static_cast<uint32_t>(n));
}

// ---------------------------------------------------------------------------------- operations
// y[n, token] for this CTA's rows of W.  Every warp takes its columns (StepPart) of every tile, so it waits
// for one barrier per tile; the partial tiles meet in shared memory, a group of tiles at a time.
// Fragments: the 16 bytes of lane 4 token + q hold columns 32 unit + 8 q .. + 7 of the token.  (Which k
// meets which does not matter to a sum: both operands use the order in which a 16-byte vector comes out
// of memory.)

// Adds kN (<= 4) units: `w` and `x(i)` are this lane's 16 bytes of row g and of token g.  Past unit `last`
// that unit again: x is zero there, and what lies behind it in shared memory may not be a number.
template <int kN, class X>
__device__ __forceinline__ void step_mma(float (&a)[4][4], uint32_t w, int last, uint32_t pitch, X x) {
  uint4 r[kN], s[kN];
#pragma unroll
  for (int i = 0; i < kN; ++i) {
    const uint32_t at = w + min(i, last) * 64;
    r[i] = ld_shared_v4(at);
    s[i] = ld_shared_v4(at + 8 * pitch);         // (rows past the tile's: their products are used by nobody)
  }
#pragma unroll
  for (int i = 0; i < kN; ++i) mma_16816(a[i], r[i].x, s[i].x, r[i].y, s[i].y, x(i).x, x(i).y);
#pragma unroll
  for (int i = 0; i < kN; ++i) mma_16816(a[i], r[i].z, s[i].z, r[i].w, s[i].w, x(i).z, x(i).w);
}
__device__ __forceinline__ void step_red_store(float* red, const float (&a)[4][4], int g, int q) {
  float* at = red + 2 * q * kStepRedPitch + g;
  at[0] = (a[0][0] + a[1][0]) + (a[2][0] + a[3][0]);
  at[kStepRedPitch] = (a[0][1] + a[1][1]) + (a[2][1] + a[3][1]);
  at[8] = (a[0][2] + a[1][2]) + (a[2][2] + a[3][2]);
  at[kStepRedPitch + 8] = (a[0][3] + a[1][3]) + (a[2][3] + a[3][3]);
}
// Output o of a group: token o >> (4 + lg), row (o & 15) of tile (o >> 4) of the group: neighbouring
// lanes have neighbouring rows, which lie next to each other wherever outputs go.
struct StepOutput {
  int row, n, tok, tile;
  bool mine;
  __device__ __forceinline__ StepOutput(const StepCut& cut, int t0, int o, int M) {
    const int in_tile = o & (kStepMmaRows - 1);
    tile = (o >> 4) & ((1 << cut.lg_group) - 1);
    tok = o >> (4 + cut.lg_group);
    row = (t0 + tile) * cut.tile + in_tile;
    n = cut.row0 + row;
    mine = in_tile < cut.tile && row < cut.rows && tok < M;
  }
};
__device__ __forceinline__ uint32_t step_bias(const __nv_bfloat16* bias, int n) {
  return __ldg(reinterpret_cast<const unsigned short*>(bias) + n);
}
__device__ __forceinline__ float step_red_sum(const float* red) {
  float v[kStepWarps];
#pragma unroll
  for (int w = 0; w < kStepWarps; ++w) v[w] = red[w * kStepRed];
  return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
}

constexpr int kStepPart = (kStepChunkUnits + kStepWarps / 2 - 1) / (kStepWarps / 2);     // 7 units of a warp
static_assert(kStepChunkUnits <= kStepPart * kStepWarps && kStepMaxUnits <= kStepPart * kStepWarps, "columns fit the warps");

// ... of the LayerNorm's output in sm.x: QKV projection, first MLP layer, head.
__device__ __forceinline__ StepCta step_linear(StepCta c, const StepParams& p, const StepPart& part, int op, int layer,
                                               int pos, uint32_t gen, const __nv_bfloat16* bias) {
  const int tid = step_tid(), warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3, M = p.M;
  unsigned long long key[2] = {0ull, 0ull};      // best of this thread's logits, of its two tokens
  const StepCut cut = c.sm->cut[op];
  uint32_t raw_bias = 0;                         // of the first output: comes while the tiles are multiplied
  {
    const StepOutput out(cut, 0, tid, M);
    if (bias != nullptr && out.mine) raw_bias = step_bias(bias, out.n);
  }
  uint4 xv[kStepPart];
#pragma unroll
  for (int i = 0; i < kStepPart; ++i) {
    xv[i] = make_uint4(0u, 0u, 0u, 0u);
    if (i < part.units && g < M) xv[i] = c.sm->x[(part.first + i) * 4 * M + lane];
  }
  const uint32_t pitch = p.stage_pitch, base = smem_u32(c.sm->ring[0]) + part.at * 64 + g * pitch + q * 16;
#pragma unroll 1
  for (int t0 = 0; t0 < cut.tiles; t0 += kStepGroup) {
    const int tiles = min(kStepGroup, cut.tiles - t0);
#pragma unroll 1
    for (int t = 0; t < tiles; ++t) {
      StepRing at = c.ring;
      at.skip(part.stage);
      c.ring.skip(1 << part.lg_stages);
      if (c.ok) c.ok = step_wait(smem_u32(&c.sm->full[at.stage]), at.parity, *c.sm, kWaitStepFull);
      const uint32_t w = base + at.stage * kStepStageBytes;
      float a[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) a[i][j] = 0.f;
      if (part.units > 0) step_mma<4>(a, w, part.units - 1, pitch, [&](int i) -> const uint4& { return xv[i]; });
      if (part.units > 4) step_mma<kStepPart - 4>(a, w + 256, part.units - 5, pitch, [&](int i) -> const uint4& { return xv[4 + i]; });
      __syncwarp();
      if (lane == 0 && c.ok) mbar_arrive_many(smem_u32(&c.sm->empty[at.stage]), 1u << part.lg_stages);
      step_red_store(c.sm->red[t][warp], a, g, q);
    }
    step_bar();
#pragma unroll
    for (int k = 0; k < 2; ++k) {                // at most 512 outputs
      const int o = tid + k * kStepCompute;
      const StepOutput out(cut, t0, o, M);
      if (out.mine) {
        if (bias != nullptr && (k > 0 || t0 > 0)) raw_bias = step_bias(bias, out.n);
        const float val = __uint_as_float(raw_bias << 16) + step_red_sum(&c.sm->red[out.tile][0][out.tok * kStepRedPitch + (o & (kStepMmaRows - 1))]);
        const int n = out.n, tok = out.tok;
        if (op == kStepQkv) {
          step_put(p.qkv + tok * 3 * p.C + n, val, gen);
          if (n >= p.C) {                          // the caches get the row too, for the steps to come
            const bool is_k = n < 2 * p.C;
            const int nn = n - (is_k ? p.C : 2 * p.C);
            (is_k ? p.k_cache[layer] : p.v_cache[layer])[tok * p.c_sb + static_cast<long long>(pos) * p.c_sn + static_cast<long long>(nn >> 6) * p.c_sh + (nn & 63)] =
                __float2bfloat16_rn(val);
          }
        } else if (op == kStepFc) {
          step_put(p.h + ((n >> 5) * M + tok) * 32 + (n & 31), gelu_tanh(val), gen);
        } else {
          const __nv_bfloat16 b = __float2bfloat16_rn(val);
          p.logits[static_cast<long long>(tok) * p.V + n] = b;
          const unsigned long long kk = step_key(__bfloat162float(b), n);
          key[k] = kk > key[k] ? kk : key[k];
        }
      }
    }
    if (t0 + kStepGroup < cut.tiles) step_bar();     // before the partial tiles are overwritten
  }
  if (op == kStepHead) {                         // groups of 4 tiles: 64 rows, so two warps per token
#pragma unroll
    for (int k = 0; k < 2; ++k) {
#pragma unroll
      for (int o = 1; o <= 16; o <<= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, key[k], o);
        key[k] = other > key[k] ? other : key[k];
      }
      if (lane == 0) c.sm->keys[(warp >> 1) + 4 * k][warp & 1] = key[k];
    }
  }
  return c;
}
static_assert(kStepGroup == 4 && kStepWarps == 8 && kStepMaxRows == 8, "512 outputs of a group, two per thread; a token's are two warps'");

// ... of an exchange buffer, for the few rows (one tile) of the attention's projection and the second MLP
// layer: a warp takes the words of its own columns, 32 unit rows at a time, and packs them into its piece
// of sm.x.
__device__ __forceinline__ StepCta step_linear_words(StepCta c, const StepParams& p, const StepPart& part, const uint32_t* src,
                                                     uint32_t* dst, int op, uint32_t gen, const __nv_bfloat16* bias) {
  const int tid = step_tid(), warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3, M = p.M;
  const uint32_t* words = src + (part.first * M * 8 + lane) * 4;
  uint4 raw[kStepTake];
  auto peek = [&](int b0, int nb) {                            // the words of units b0 .. + nb
#pragma unroll
    for (int i = 0; i < kStepTake; ++i) {
      raw[i] = make_uint4(gen, gen, gen, gen);
      if (i * 32 + lane < nb * M * 8) raw[i] = step_peek(words + b0 * M * 32 + i * 128);
    }
  };
  const int batch = p.batch_units, units = part.units;
  peek(0, min(batch, units));
  const StepCut cut = c.sm->cut[op];
  const StepOutput out(cut, 0, tid, M);
  uint32_t raw_bias = 0;
  if (bias != nullptr && out.mine) raw_bias = step_bias(bias, out.n);
  if (cut.tiles > 0) {
    StepRing at = c.ring;
    at.skip(part.stage);
    c.ring.skip(1 << part.lg_stages);
    if (c.ok) c.ok = step_wait(smem_u32(&c.sm->full[at.stage]), at.parity, *c.sm, kWaitStepFull);
    const uint32_t pitch = p.stage_pitch;
    uint32_t w = smem_u32(c.sm->ring[0]) + at.stage * kStepStageBytes + part.at * 64 + g * pitch + q * 16;
    const uint32_t pack = smem_u32(c.sm->x) + warp * (kStepTake * 256), x0 = pack + lane * 16, x_step = M * 64;
    float a[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) a[i][j] = 0.f;
#pragma unroll 1
    for (int b0 = 0; b0 < units; b0 += batch) {
      const int nb = min(batch, units - b0);
#pragma unroll 1
      for (uint32_t polls = 0;; ++polls) {
        uint32_t bad = 0;
#pragma unroll
        for (int i = 0; i < kStepTake; ++i) bad |= step_stale(raw[i], gen);
        if (!c.ok || !__any_sync(0xffffffffu, bad != 0)) break;
        if (polls >= kStepWordPolls || *const_cast<volatile uint32_t*>(&c.sm->abort)) {
          step_give_up(*c.sm, kWaitStepWords);
          c.ok = false;
        }
        peek(b0, nb);
      }
#pragma unroll
      for (int i = 0; i < kStepTake; ++i)
        if (i * 32 < nb * M * 8)                 // (what lies past the end of the units is not read)
          st_shared_v2(pack + (i * 32 + lane) * 8, step_pair(raw[i].x, raw[i].y), step_pair(raw[i].z, raw[i].w));
      __syncwarp();
      if (b0 + batch < units) peek(b0 + batch, min(batch, units - b0 - batch));
      uint32_t x = x0;
#pragma unroll 1
      for (int u = 0; u < nb; u += 4) {          // four units at a time: their loads overlap
        uint4 xv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          xv[i] = make_uint4(0u, 0u, 0u, 0u);
          if (u + i < nb && g < M) xv[i] = ld_shared_v4(x + i * x_step);
        }
        step_mma<4>(a, w + u * 64, nb - 1 - u, pitch, [&](int i) -> const uint4& { return xv[i]; });
        x += 4 * x_step;
      }
      w += nb * 64;
      __syncwarp();                              // before the words are overwritten, the stage given back
    }
    if (lane == 0 && c.ok) mbar_arrive_many(smem_u32(&c.sm->empty[at.stage]), 1u << part.lg_stages);
    step_red_store(c.sm->red_one[warp], a, g, q);
  }
  step_bar();
  if (out.mine) {
    const float val = __uint_as_float(raw_bias << 16) + step_red_sum(&c.sm->red_one[0][out.tok * kStepRedPitch + out.row]) + c.sm->own[tid];
    c.sm->own[tid] = val;
    step_put(dst + out.tok * p.C + out.n, val, gen);
  }
  return c;
}

// How the warps share the token rows: warp w serves token w / wpt; its lane the groups of four
// columns (w % wpt) * 32 + lane, + 32 wpt, ...
struct StepRows {
  int tok, first, stride, lg;
  __device__ __forceinline__ StepRows(int M, int warp, int lane) {
    lg = M <= 1 ? 3 : (M <= 2 ? 2 : (M <= 4 ? 1 : 0));      // log2 of warps per token
    tok = warp >> lg;
    first = (warp & ((1 << lg) - 1)) * 32 + lane;
    stride = 32 << lg;
  }
};

// LayerNorm of the residual stream (exchange words at `x`) into the fragments sm.x.  One pass: sums
// of x - s and (x - s)^2 with s the mean of the row's first four columns.  However far a row lies from 0, s
// is a value of that row, and no value is more than sqrt(C) standard deviations from the mean: the difference
// of squares loses at most a factor C (1600 * 2^-24 = 1e-4, a twentieth of the rounding of the result to
// bf16), and a few units in the last place on rows without such an outlier in front.  (With the mean of the
// LayerNorm before, and 0 in the first, the loss had no bound: rows of 448 + {0, 2} were off by 1 %.)
// kN: rounds of the warps over a row's groups of four columns, at least as many as there are.  (One kN for
// the widest row of a warp, with the rounds that are not there branched around, took 2300 clocks where
// there was one round.)
template <int kN>
__device__ __forceinline__ StepCta step_layernorm(StepCta c, const StepParams& p, const uint32_t* x, uint32_t gen,
                                                  const StepRows& rw) {
  const int lane = step_tid() & 31, warp = step_tid() >> 5;
  const int quads = p.C >> 2;
  uint4 w[kN], front;                            // front: columns 0 .. 3
  {                                              // (past the end the last quad again, unused)
    const uint32_t* src = x + min(rw.tok, p.M - 1) * p.C;
#pragma unroll 1
    for (uint32_t polls = 0;; ++polls) {
      front = step_peek(src);
#pragma unroll
      for (int i = 0; i < kN; ++i) w[i] = step_peek(src + 4 * min(rw.first + i * rw.stride, quads - 1));
      uint32_t bad = step_stale(front, gen);
#pragma unroll
      for (int i = 0; i < kN; ++i) bad |= step_stale(w[i], gen);
      if (!c.ok || !__any_sync(0xffffffffu, bad != 0)) break;
      if (polls >= kStepWordPolls || *const_cast<volatile uint32_t*>(&c.sm->abort)) {
        step_give_up(*c.sm, kWaitStepWords);
        c.ok = false;
      }
    }
  }
  auto value = [](uint32_t word) { return __uint_as_float(word & 0xffff0000u); };
  const float shift = 0.25f * ((value(front.x) + value(front.y)) + (value(front.z) + value(front.w)));
  float sum = 0.f, sq = 0.f;
#pragma unroll
  for (int i = 0; i < kN; ++i) {
    w[i].x &= 0xffff0000u; w[i].y &= 0xffff0000u; w[i].z &= 0xffff0000u; w[i].w &= 0xffff0000u;   // now fp32
    const float f = rw.first + i * rw.stride < quads ? 1.f : 0.f;
    const float d0 = __uint_as_float(w[i].x) - shift, d1 = __uint_as_float(w[i].y) - shift;
    const float d2 = __uint_as_float(w[i].z) - shift, d3 = __uint_as_float(w[i].w) - shift;
    sum = fmaf(f, (d0 + d1) + (d2 + d3), sum);
    sq = fmaf(f, fmaf(d0, d0, d1 * d1) + fmaf(d2, d2, d3 * d3), sq);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    sq += __shfl_xor_sync(0xffffffffu, sq, o);
  }
  if (lane == 0) c.sm->stat[warp] = make_float2(sum, sq);
  asm volatile("cp.async.wait_all;" ::: "memory");
  step_bar();                                    // sm.stat and sm.norm are complete
  if (rw.lg > 0) {                               // 1, 2 or 4 pairs of warps
    const float4* st = reinterpret_cast<const float4*>(c.sm->stat + ((rw.tok << rw.lg) & (kStepWarps - 1)));
    float4 two[kStepWarps / 2];
#pragma unroll
    for (int i = 0; i < kStepWarps / 2; ++i) two[i] = i < 1 << (rw.lg - 1) ? st[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    sum = ((two[0].x + two[0].z) + (two[1].x + two[1].z)) + ((two[2].x + two[2].z) + (two[3].x + two[3].z));
    sq = ((two[0].y + two[0].w) + (two[1].y + two[1].w)) + ((two[2].y + two[2].w) + (two[3].y + two[3].w));
  }
  const float off = sum * p.inv_c;
  const float rstd = rsqrtf(fmaxf(sq * p.inv_c - off * off, 0.f) + p.eps);
  const float mean = shift + off;
  uint2* out = reinterpret_cast<uint2*>(c.sm->x) + rw.tok * 8;
#pragma unroll
  for (int i = 0; i < kN; ++i) {
    const int v = rw.first + i * rw.stride;      // columns 4 v .. 4 v + 3
    if (rw.tok < p.M && v < quads) {
      const uint2 gm = c.sm->norm[0][v], bt = c.sm->norm[1][v];
      const float y0 = fmaf((__uint_as_float(w[i].x) - mean) * rstd, __uint_as_float(gm.x << 16), __uint_as_float(bt.x << 16));
      const float y1 = fmaf((__uint_as_float(w[i].y) - mean) * rstd, __uint_as_float(gm.x & 0xffff0000u), __uint_as_float(bt.x & 0xffff0000u));
      const float y2 = fmaf((__uint_as_float(w[i].z) - mean) * rstd, __uint_as_float(gm.y << 16), __uint_as_float(bt.y << 16));
      const float y3 = fmaf((__uint_as_float(w[i].w) - mean) * rstd, __uint_as_float(gm.y & 0xffff0000u), __uint_as_float(bt.y & 0xffff0000u));
      out[(v >> 3) * 8 * p.M + (v & 7)] = make_uint2(pack_bf16(y0, y1), pack_bf16(y2, y3));
    }
  }
  step_bar();
  return c;
}
// Scale and shift of the coming LayerNorm on their way to sm.norm; the LayerNorm waits for them.
__device__ __forceinline__ void step_fetch_norm(StepSmem& sm, const __nv_bfloat16* gamma, const __nv_bfloat16* beta,
                                                int nvec) {
  const int tid = step_tid();
  const bool second = tid >= kStepCompute / 2;
  const uint32_t dst = smem_u32(sm.norm[second ? 1 : 0]);
  const uint4* src = reinterpret_cast<const uint4*>(second ? beta : gamma);
#pragma unroll 1
  for (int v = second ? tid - kStepCompute / 2 : tid; v < nvec; v += kStepCompute / 2) cp_async_16(dst + v * 16, src + v);
}

// Adds a block of 16 cached rows, K at `ks` in shared memory and V behind the stage's K, of which left > 0 count, to a
// lane group's running maximum, sum and outputs.  release() once the rows are in registers.
template <class Release>
__device__ __forceinline__ void step_attend(uint32_t ks, int left, const uint4& q0, const uint4& q1, float scale_log2, int lane,
                                            float& m, float& l, uint64_t (&acc)[4], Release release) {
  const int g = lane >> 2, q = lane & 3, grp = lane >> 3, col = lane & 7;
  const int swap = (g & 1) << 2, vswap = (grp & 1) << 2;
  const uint4 k0 = ld_shared_v4(ks + g * 128 + (q ^ swap) * 16), k1 = ld_shared_v4(ks + g * 128 + ((q + 4) ^ swap) * 16);
  const uint4 k2 = ld_shared_v4(ks + (g + 8) * 128 + (q ^ swap) * 16), k3 = ld_shared_v4(ks + (g + 8) * 128 + ((q + 4) ^ swap) * 16);
  uint4 vr[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) vr[j] = ld_shared_v4(ks + (kStepBlocks * 16 + grp + 4 * j) * 128 + (col ^ vswap) * 16);
  release();
  // scores of rows g ([0], equal in the lanes of a quad and in [1]) and g + 8 ([2], [3]): every
  // column of the 8-column operand is the query
  float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
  mma_16816(s0, k0.x, k2.x, k0.y, k2.y, q0.x, q0.y);
  mma_16816(s1, k0.z, k2.z, k0.w, k2.w, q0.z, q0.w);
  mma_16816(s0, k1.x, k3.x, k1.y, k3.y, q1.x, q1.y);
  mma_16816(s1, k1.z, k3.z, k1.w, k3.w, q1.z, q1.w);
  const float sa = g < left ? (s0[0] + s1[0]) * scale_log2 : -INFINITY;
  const float sb = g + 8 < left ? (s0[2] + s1[2]) * scale_log2 : -INFINITY;
  float sc[4];                             // rows grp + 4 j: lane 4 (row % 8) has them
#pragma unroll
  for (int j = 0; j < 4; ++j) sc[j] = __shfl_sync(0xffffffffu, j < 2 ? sa : sb, ((grp + 4 * j) & 7) * 4);
  const float m_new = fmaxf(fmaxf(m, fmaxf(sc[0], sc[1])), fmaxf(sc[2], sc[3]));
  const float f = ex2_approx(m - m_new);
  const uint64_t f2 = pack_f32x2(f, f);
  m = m_new;
  l *= f;
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] = mul_f32x2(acc[e], f2);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float pr = ex2_approx(sc[j] - m);
    l += pr;
    const uint64_t p2 = pack_f32x2(pr, pr);
    acc[0] = fma_f32x2(p2, bf16x2_to_f32x2(vr[j].x), acc[0]);
    acc[1] = fma_f32x2(p2, bf16x2_to_f32x2(vr[j].y), acc[1]);
    acc[2] = fma_f32x2(p2, bf16x2_to_f32x2(vr[j].z), acc[2]);
    acc[3] = fma_f32x2(p2, bf16x2_to_f32x2(vr[j].w), acc[3]);
  }
}

__device__ __forceinline__ StepCta step_attention(StepCta c, const StepParams& p, int layer, uint32_t gen) {
  const int tid = step_tid(), warp = tid >> 5, lane = tid & 31, count = c.sm->units, splits = c.sm->splits;
  const int q = lane & 3, grp = lane >> 3, col = lane & 7;
#pragma unroll 1
  for (int i = 0; i < count; ++i) {
    const StepUnit un = c.sm->unit[i];
    uint4 q0, q1;
    {
      uint4 w[4];                                // columns 8 q .. + 7 and 32 + 8 q .. + 7
      const uint32_t* src = p.qkv + un.query + q * 8;
      step_take<4>(c, gen, w, [&](int k) { return src + (k >> 1) * 32 + (k & 1) * 4; });
      q0 = make_uint4(step_pair(w[0].x, w[0].y), step_pair(w[0].z, w[0].w), step_pair(w[1].x, w[1].y), step_pair(w[1].z, w[1].w));
      q1 = make_uint4(step_pair(w[2].x, w[2].y), step_pair(w[2].z, w[2].w), step_pair(w[3].x, w[3].y), step_pair(w[3].z, w[3].w));
    }
    float m = kNoScore, l = 0.f;
    uint64_t acc[4] = {0ull, 0ull, 0ull, 0ull};
    // Stages of kStepBlocks blocks of 16 rows, one warp to a block: warps 0 to 3 take the even ring slots, 4
    // to 7 the odd ones (so a warp that waits for a slot has also waited for the slot's stage before).  A
    // row's odd-numbered neighbour has its 64-byte halves swapped (see step_stream_rows): no bank conflicts.
    // Lane group grp (of 8 lanes) sums rows grp, grp + 4, + 8, + 12 of the blocks with a maximum of its own.
    // A GPT-2 XL unit of 900 rows, clocks: 8900 with one maximum per warp and waits for all stages, 7500 so.
    // A stage goes back as soon as its rows are in registers: the stream of rows, not the arithmetic, is what the
    // longer caches wait for.  us per step, given back behind the arithmetic / so: GPT-2 small 8 x 900 rows 228 / 223,
    // medium 8 x 600 446 / 439, XL 8 x 900 1467 / 1457, 4 x 500 944 / 940; two blocks at a time on top: 231, 449, 1499.
    {
      const int stages = (un.rows + kStepBlocks * 16 - 1) / (kStepBlocks * 16);
      const uint32_t own = (c.ring.stage & 1) == warp / kStepBlocks ? 0 : 1;
      const uint32_t first = smem_u32(c.sm->ring) + (warp & (kStepBlocks - 1)) * 16 * 128;
      StepRing at = c.ring;
      at.skip(own);
      c.ring.skip_any(stages);
      int left = un.rows - (static_cast<int>(own) * kStepBlocks + (warp & (kStepBlocks - 1))) * 16;   // rows of the block and after
#pragma unroll 1
      for (int st = own; st < stages; st += 2, left -= 2 * kStepBlocks * 16) {
        if (c.ok) c.ok = step_wait(smem_u32(&c.sm->full[at.stage]), at.parity, *c.sm, kWaitStepFull);
        const uint32_t ks = first + at.stage * kStepStageBytes;
        auto release = [&]() {               // the rows are in registers: the stage may be filled again
          __syncwarp();
          if (lane == 0 && c.ok) mbar_arrive_many(smem_u32(&c.sm->empty[at.stage]), kStepWarps / kStepBlocks);
        };
        if (left > 0) step_attend(ks, left, q0, q1, p.scale_log2, lane, m, l, acc, release);
        else release();
        at.skip(2);
      }
    }
    {                                            // the four groups' maxima, and their sums
      float m_all = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
      m_all = fmaxf(m_all, __shfl_xor_sync(0xffffffffu, m_all, 16));
      const float f = ex2_approx(m - m_all);
      const uint64_t f2 = pack_f32x2(f, f);
      m = m_all;
      l *= f;
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = mul_f32x2(acc[e], f2);
      l += __shfl_xor_sync(0xffffffffu, l, 8);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
    }
    float* dst = c.sm->seg[i][warp];
    if (lane == 0) { dst[0] = m; dst[1] = l; }
#pragma unroll
    for (int e = 0; e < 4; ++e) {                // the four row groups
      float o0, o1;
      unpack_f32x2(acc[e], o0, o1);
      o0 += __shfl_xor_sync(0xffffffffu, o0, 8);
      o1 += __shfl_xor_sync(0xffffffffu, o1, 8);
      o0 += __shfl_xor_sync(0xffffffffu, o0, 16);
      o1 += __shfl_xor_sync(0xffffffffu, o1, 16);
      if (grp == 0) *reinterpret_cast<float2*>(dst + 4 + 8 * col + 2 * e) = make_float2(o0, o1);
    }
    if (warp == kStepWarps - 1) {              // the new row, a partial of its own (of one unit)
      // lanes 0-15: four columns each; the other half of the warp repeats them
      const uint32_t* src = p.qkv + un.query + (lane & 15) * 4;
      uint4 w[3];
      step_take<3>(c, gen, w, [&](int k) { return src + k * p.C; });
      auto val = [](uint32_t x) { return __uint_as_float(x & 0xffff0000u); };
      float s = val(w[0].x) * val(w[1].x) + val(w[0].y) * val(w[1].y) + val(w[0].z) * val(w[1].z) + val(w[0].w) * val(w[1].w);
#pragma unroll
      for (int o = 1; o <= 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      float* fresh = c.sm->seg[i][kStepWarps];
      const bool counts = un.slot == 0;
      if (lane == 0) { fresh[0] = counts ? s * p.scale_log2 : kNoScore; fresh[1] = counts ? 1.f : 0.f; }
      if (lane < 16)
        *reinterpret_cast<float4*>(fresh + 4 + 4 * lane) = make_float4(val(w[2].x), val(w[2].y), val(w[2].z), val(w[2].w));
    }
  }
  step_bar();
  const int i = tid >> 6, e = tid & 63;
  if (i < count) {
    const StepUnit un = c.sm->unit[i];
    const float(&seg)[kStepWarps + 1][68] = c.sm->seg[i];
    float mm = kNoScore, ll = 0.f, oo = 0.f;
#pragma unroll
    for (int w = 0; w <= kStepWarps; ++w) mm = fmaxf(mm, seg[w][0]);
#pragma unroll
    for (int w = 0; w <= kStepWarps; ++w) {      // (a warp without rows: m = kNoScore, l = o = 0)
      const float f = ex2_approx(seg[w][0] - mm);
      ll = fmaf(seg[w][1], f, ll);
      oo = fmaf(seg[w][4 + e], f, oo);
    }
    bool write = true;
    if (splits > 1) {                        // (then the CTA has one unit)
      float* po = p.part_o + un.pair * splits * 64 + e;
      float2* pm = p.part_ml + un.pair * splits;
      __stcg(po + un.slot * 64, oo);
      if (e == 0) __stcg(pm + un.slot, make_float2(mm, ll));
      __threadfence();
      asm volatile("bar.sync 2, 64;" ::: "memory");
      if (e == 0) c.sm->seg_last = atomicAdd(p.arrived + un.pair, 1u) + 1 == splits;
      asm volatile("bar.sync 2, 64;" ::: "memory");
      write = c.sm->seg_last;
      if (write) {                               // all partials are in: merge them
        __threadfence();
        if (e == 0) p.arrived[un.pair] = 0;
        mm = kNoScore; ll = 0.f; oo = 0.f;
#pragma unroll 1
        for (int k = 0; k < splits; ++k) {
          const float2 ml = __ldcg(pm + k);
          const float v = __ldcg(po + k * 64);
          const float m_new = fmaxf(mm, ml.x), f = ex2_approx(mm - m_new), fi = ex2_approx(ml.x - m_new);
          ll = ll * f + ml.y * fi;
          oo = oo * f + v * fi;
          mm = m_new;
        }
      }
    }
    if (write) step_put(p.ctx + un.out + (e >> 5) * p.M * 32 + (e & 31), __fdividef(oo, ll), gen);
  }
  return c;
}

// Pulls a layer's vectors into L2, spread over the grid: nobody should be the first to touch them
// between two exchanges.
__device__ __forceinline__ void step_prefetch(const StepSmem& sm, const StepParams& p, int layer) {
  const int tid = step_tid();
  const StepLayer& L = sm.layers[layer];
  const int at = (blockIdx.x + tid * gridDim.x) * 64;        // 64 elements per 128-byte line
  if (at < 4 * p.C) {
    prefetch_l2(L.fc_b + at);
    if (at < 3 * p.C && L.qkv_b) prefetch_l2(L.qkv_b + at);
    if (at < p.C) {
      prefetch_l2(L.ln1_g + at); prefetch_l2(L.ln1_b + at); prefetch_l2(L.ln2_g + at); prefetch_l2(L.ln2_b + at);
      prefetch_l2(L.proj_b + at); prefetch_l2(L.out_b + at);
    }
  }
}

// The streaming warps' ops in order: 4 per layer, then the head.
__device__ __forceinline__ const __nv_bfloat16* step_weight(const StepSmem& sm, const StepParams& p, int i, int& op) {
  if (i >= 4 * p.n_layers) { op = kStepHead; return p.head_w; }
  op = i & 3;
  const StepLayer& L = sm.layers[i >> 2];
  return op == kStepQkv ? L.qkv_w : (op == kStepProj ? L.proj_w : (op == kStepFc ? L.fc_w : L.out_w));
}
__device__ __forceinline__ void step_ahead(const StepSmem& sm, const StepParams& p, int i, int sw, int lane) {
  if (i > 4 * p.n_layers) return;
  int op;
  const __nv_bfloat16* w = step_weight(sm, p, i, op);
  const StepCut& cut = sm.cut[op];
  const uint32_t row = (op == kStepOut ? 4 * p.C : p.C) * 2u, bytes = min(cut.rows * row, kStepAheadBytes);
  const char* at = reinterpret_cast<const char*>(w) + static_cast<long long>(cut.row0) * row;
#pragma unroll 1
  for (uint32_t b = (sw * 32 + lane) * kStepAheadPiece; b < bytes; b += 32 * kStepStreamWarps * kStepAheadPiece)
    bulk_prefetch_l2(at + b, min(kStepAheadPiece, bytes - b));
}
// Streaming warp `sw`: its quarter of this CTA's rows of one matrix into the ring.
__device__ __forceinline__ bool step_stream(StepSmem& sm, const StepParams& p, StepRing& ring, uint32_t& issued,
                                            const __nv_bfloat16* w, int op, int sw) {
  const StepCut cut = sm.cut[op];
  const long long ldw = op == kStepOut ? 4 * p.C : p.C;
  const int stages = 1 << (p.lg_chunks + (op == kStepOut ? 2 : 0));
  const uint32_t bytes = static_cast<uint32_t>(p.stage_units) * 64;
  w += (cut.row0 + sw) * ldw;
#pragma unroll 1
  for (int t = 0; t < cut.tiles; ++t) {
    // rows sw, sw + 4, ... of the tile
    const int rows = (min(cut.tile, cut.rows - t * cut.tile) - sw + kStepStreamWarps - 1) / kStepStreamWarps;
    const __nv_bfloat16* src = w + t * cut.tile * ldw;
#pragma unroll 1
    for (int st = 0; st < stages; ++st) {
      if (issued >= kStepStages &&
          !step_wait(smem_u32(&sm.empty[ring.stage]), ring.parity ^ 1, sm, kWaitStepEmpty))
        return false;
      if (elect_one()) {
        fence_proxy_async_smem();                // (the stage may have held cached rows, written by plain copies)
        const uint32_t bar = smem_u32(&sm.full[ring.stage]);
        uint32_t dst = smem_u32(sm.ring[ring.stage]) + sw * p.stage_pitch;
        mbar_arrive_expect_tx(bar, bytes * rows);
#pragma unroll
        for (int r = 0; r < kStepTile / kStepStreamWarps; ++r)
          if (r < rows) bulk_load(dst + r * kStepStreamWarps * p.stage_pitch, src + r * kStepStreamWarps * ldw, bytes, bar);
      }
      __syncwarp();
      ring.next();
      ++issued;
      src += p.stage_units * kStepUnit;
    }
  }
  return true;
}

// The cached rows of this CTA's attention units in a layer, kStepBlocks * 16 rows of K and then of V
// per stage, every fourth group of four rows by streaming warp `sw`.  Odd rows have their 64-byte
// halves swapped.  Rows past the end are the last row again.
__device__ __forceinline__ bool step_stream_rows(StepSmem& sm, const StepParams& p, StepRing& ring, uint32_t& issued,
                                                 int layer, int sw, int lane) {
  const int chunk = lane & 7, first = sw * 4 + (lane >> 3);    // four rows of eight 16-byte chunks per copy
  const uint32_t off = first * 128 + ((chunk ^ ((first & 1) << 2)) * 16);
#pragma unroll 1
  for (int i = 0; i < sm.units; ++i) {
    const StepUnit& un = sm.unit[i];
    const long long at = un.head + static_cast<long long>(un.row0) * p.c_sn + chunk * 8;
    const __nv_bfloat16 *kb = p.k_cache[layer] + at, *vb = p.v_cache[layer] + at;
    const long long step = 4ll * kStepStreamWarps * p.c_sn, ahead = static_cast<long long>(first) * p.c_sn;
    const __nv_bfloat16 *kr = kb + ahead, *vr = vb + ahead;      // this lane's first row of the stage
#pragma unroll 1
    for (int r = 0; r < un.rows; r += kStepBlocks * 16) {
      if (issued >= kStepStages &&
          !step_wait(smem_u32(&sm.empty[ring.stage]), ring.parity ^ 1, sm, kWaitStepEmpty))
        return false;
      const uint32_t dst = smem_u32(sm.ring[ring.stage]) + off, bar = smem_u32(&sm.full[ring.stage]);
      if (un.rows - r >= kStepBlocks * 16) {
#pragma unroll
        for (int j = 0; j < kStepBlocks * 16; j += 4 * kStepStreamWarps) {
          cp_async_16(dst + j * 128, kr);
          cp_async_16(dst + (kStepBlocks * 16 + j) * 128, vr);
          kr += step;
          vr += step;
        }
      } else {
        const int rows = (un.rows - r + 15) & ~15;
#pragma unroll 1
        for (int j = 0; j < rows; j += 4 * kStepStreamWarps) {
          const long long row = static_cast<long long>(min(r + j + first, un.rows - 1)) * p.c_sn;
          cp_async_16(dst + j * 128, kb + row);
          cp_async_16(dst + (kStepBlocks * 16 + j) * 128, vb + row);
        }
      }
      cp_async_arrive(bar);
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
      ring.next();
      ++issued;
    }
  }
  return true;
}

__global__ void __launch_bounds__(kStepThreads, 1) fa_gpt_step_kernel(const __grid_constant__ StepParams p) {
  extern __shared__ uint8_t step_raw[];
  StepSmem& sm = *reinterpret_cast<StepSmem*>(step_raw + ((128u - (smem_u32(step_raw) & 127u)) & 127u));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int C = p.C, M = p.M;
  const long long pos64 = p.pos_ptr ? *p.pos_ptr : static_cast<long long>(p.pos);
  // (reduced here: past 2^32 the remainders would repeat one, and a word of the layer before pass for new)
  const uint32_t generation = *p.generation % 65535u;
  const int last = min(p.cache_rows, p.n_positions) - 1;
  const int pos = pos64 < 0 ? 0 : (pos64 > last ? last : static_cast<int>(pos64));
  const StepAttnCut cut(M * p.H, pos);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStepStages; ++i) {
      mbar_init(smem_u32(&sm.full[i]), kStepStreamWarps);
      mbar_init(smem_u32(&sm.empty[i]), kStepWarps);
    }
    sm.abort = 0;
    sm.abort_who = 0;
    fence_mbar_init();
    if (blockIdx.x == 0) {                       // used at the very end, by CTAs that depend on this one's output
      *p.done = 0;
      for (int t = 0; t < kStepMaxRows; ++t) p.best[t] = 0ull;
      __threadfence();
    }
  }
  {
    constexpr int kPtrs = sizeof(StepLayer) / sizeof(void*);
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(p.layers);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(sm.layers);
    for (int i = threadIdx.x; i < p.n_layers * kPtrs; i += kStepThreads) dst[i] = src[i];
  }
  if (threadIdx.x == 0) {
    sm.units = cut.count;
    sm.splits = cut.splits;
  }
  if (static_cast<int>(threadIdx.x) < cut.count) {
    const int u = cut.first + threadIdx.x, pair = u / cut.splits, part = u - pair * cut.splits;
    const int b = pair / p.H, h = pair - b * p.H;
    StepUnit un;
    un.pair = pair;
    un.slot = part;
    un.row0 = static_cast<int>(static_cast<long long>(part) * cut.rows / cut.splits);
    un.rows = static_cast<int>(static_cast<long long>(part + 1) * cut.rows / cut.splits) - un.row0;
    un.head = b * p.c_sb + static_cast<long long>(h) * p.c_sh;
    un.query = b * 3 * C + h * 64;
    un.out = (2 * h * M + b) * 32;
    sm.unit[threadIdx.x] = un;
  }
  if (threadIdx.x < 5) {
    const int op = threadIdx.x;
    sm.cut[op] = step_cut(op == kStepQkv ? 3 * C : (op == kStepFc ? 4 * C : (op == kStepHead ? p.V : C)),
                          op == kStepHead);
  }
  __syncthreads();

  if (warp >= kStepWarps) {
    reg_dealloc<kStepStreamRegs>();              // all four warps of the warpgroup
    // ------------------------------------------------------------------ stream
    const int sw = warp - kStepWarps;
    StepRing ring;
    uint32_t issued = 0;
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i <= 4 * p.n_layers && ok; ++i) {
      int op;
      const __nv_bfloat16* w = step_weight(sm, p, i, op);
      step_ahead(sm, p, i + 1, sw, lane);
      ok = step_stream(sm, p, ring, issued, w, op, sw);
      if (ok && op == kStepQkv) ok = step_stream_rows(sm, p, ring, issued, i >> 2, sw, lane);
    }
    // leave no copy in flight, whatever the computing warps did: the last use of every stage
#pragma unroll 1
    for (uint32_t i = 0; i < kStepStages && i < issued; ++i)
      step_wait(smem_u32(&sm.full[(issued - 1 - i) % kStepStages]), ((issued - 1 - i) / kStepStages) & 1, sm, kWaitDrain);
  } else {
    reg_alloc<kStepComputeRegs>();
    // ------------------------------------------------------------------ computing warps
    StepCta c;
    c.sm = &sm;
    c.ok = true;
    {  // this CTA's columns of the residual stream: the embeddings' sum
      const StepOutput out(sm.cut[kStepProj], 0, threadIdx.x, M);
      const int tok = out.tok, n = out.n;
      if (out.mine) {
        long long id = p.ids[tok * p.ids_stride];
        id = id < 0 ? 0 : (id >= p.V ? p.V - 1 : id);
        const float v = __bfloat162float(__float2bfloat16_rn(
            __bfloat162float(p.tok_emb[id * C + n]) + __bfloat162float(p.pos_emb[static_cast<long long>(pos) * C + n])));
        sm.own[threadIdx.x] = v;
        if (!kStepKeepsBack || blockIdx.x > 0) step_put(p.x_mlp + tok * C + n, v, generation % 65535u + 1u);
      }
    }
    step_prefetch(sm, p, 0);
    const StepPart narrow(warp, p.lg_chunks, p.stage_units), wide(warp, p.lg_chunks + 2, p.stage_units);
#pragma unroll 1
    for (int i = 0; i <= 4 * p.n_layers; ++i) {
      const int l = min(i >> 2, p.n_layers - 1);
      const int op = i == 4 * p.n_layers ? static_cast<int>(kStepHead) : (i & 3);
      const StepLayer& L = sm.layers[l];
      const uint32_t before = (generation + l) % 65535u + 1u, gen = (generation + l + 1) % 65535u + 1u;
      const __nv_bfloat16* bias = op == kStepQkv ? L.qkv_b : (op == kStepProj ? L.proj_b : (op == kStepFc ? L.fc_b : (op == kStepOut ? L.out_b : nullptr)));
      if (op & 1) {
        const bool proj = op == kStepProj;
        c = step_linear_words(c, p, proj ? narrow : wide, proj ? p.ctx : p.h, proj ? p.x_att : p.x_mlp, op, gen, bias);
      } else {
        step_fetch_norm(sm, op == kStepQkv ? L.ln1_g : (op == kStepFc ? L.ln2_g : p.lnf_g),
                        op == kStepQkv ? L.ln1_b : (op == kStepFc ? L.ln2_b : p.lnf_b), C >> 3);
        const uint32_t* x = op == kStepFc ? p.x_att : p.x_mlp;
        const uint32_t want = op == kStepQkv ? before : gen;
        const StepRows rw(M, step_tid() >> 5, step_tid() & 31);
        if (C <= 8 * rw.stride) c = step_layernorm<2>(c, p, x, want, rw);
        else if (C <= 16 * rw.stride) c = step_layernorm<4>(c, p, x, want, rw);
        else if (C <= 28 * rw.stride) c = step_layernorm<7>(c, p, x, want, rw);
        else c = step_layernorm<kStepQuads>(c, p, x, want, rw);
        c = step_linear(c, p, narrow, op, l, pos, gen, bias);
      }
      if (op == kStepQkv && sm.units > 0) {
        c = step_attention(c, p, l, gen);
      }
      if (op == kStepOut && l + 1 < p.n_layers) step_prefetch(sm, p, l + 1);
    }
    if (p.next_ids) {
      step_bar();
      if (warp == 0) {
        if (lane < M) {
          unsigned long long key = 0ull;
#pragma unroll
          for (int w = 0; w < 2; ++w) key = sm.keys[lane][w] > key ? sm.keys[lane][w] : key;
          atomicMax(p.best + lane, key);
        }
        __threadfence();
        __syncwarp();
        if (lane == 0 && atomicAdd(p.done, 1u) + 1 == gridDim.x) {   // the last CTA: all keys are in
          __threadfence();
          for (int t = 0; t < M; ++t)
            p.next_ids[t * p.next_stride] = static_cast<long long>(0xffffffffu - static_cast<uint32_t>(__ldcg(p.best + t)));
        }
      }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // everyone has read these: their output is in ours
      *p.generation = generation + p.n_layers + 1;
      if (p.pos_ptr && p.advance) {
        *p.pos_ptr = pos64 + 1;
        if (p.len_ptr) *p.len_ptr = static_cast<int>(pos64) + 2;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && sm.abort != 0) {
    if (atomicCAS(p.status, 0u, sm.abort) == 0u) {
      p.status[1] = blockIdx.x;
      p.status[2] = sm.abort_who & 0xffffu;
      p.status[3] = sm.abort_who >> 16;
    }
  }
}

}  // namespace fa
