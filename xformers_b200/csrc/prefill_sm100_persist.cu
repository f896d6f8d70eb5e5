// Attention forward (prefill) on tcgen05: one persistent CTA per SM.
//
// A work item is a block of 256 query rows of one (sequence, query head): two
// 128-row query tiles that share every K/V tile TMA brings in.  (One tile, where
// the tiles of the whole launch are no more than the SMs.)  Where the heads of a
// GQA group read the same keys, the rows of a tile are (token, head of the group)
// pairs, which the box of the Q copies lays out that way.  Items are
// handed out by one atomic counter, heaviest first (the last row block of every
// head, then the one before, ...) inside groups of heads whose keys and values
// fit the L2 together, so the SMs stay evenly loaded whatever the sequence
// lengths are, a K/V tile comes from DRAM once and from the L2 for the other row
// blocks of its head, and everything a CTA sets up -- tensor memory, barriers,
// tensor-map prefetch -- is paid once per SM instead of once per block of rows.
// The roles of the 16 warps:
//
//   warps 0-3    softmax of query tile 0   (thread <-> row <-> TMEM lane)
//   warps 4-7    softmax of query tile 1
//   warps 8-11   output: O_t / l -> global memory, log-sum-exp.  They work on
//                item i while every other warp is already on item i + 1, so
//                the tensor pipe does not wait for the write-back.
//   warp 12/13   MMA issuer of P_t V of tile 0 / 1 (one lane issues)
//   warp 14      scheduler + TMA producer: pulls the next item one item ahead of
//                time, works out its geometry once and announces it to the other
//                warps through a small ring of descriptors in shared memory,
//                loads Q (per tile) and the K/V tiles into 2-deep rings that run
//                on across item boundaries.  Items in which no query sees any
//                key (possible when the key axis is sharded) never enter the
//                ring: this warp writes their zeros and -inf itself.
//   warp 15      MMA issuer of Q_t K^T, both tiles in turn
//
// Tensor memory: S | P0 | P1 | O0 | O1.  There is one buffer of scores: as soon
// as the softmax of a tile has its 128 scores in registers, the buffer goes to
// Q K^T of the other tile, which is through long before that tile's softmax asks
// for it.  So nothing a tile's softmax waits for hangs on its own last step except
// P V (P_t is free and O_t may be rescaled once that is through), and the two
// tiles stay half a step apart: one is in its exponentials while the other reads
// scores and looks for the maximum.  Across items the first PV of a tile waits until the
// output warps have read the previous O_t out of tensor memory.
//
// What bounds a step of 2 x 128 rows x 128 keys: 2048 clocks of MMAs and 2048 clocks of exponentials
// (4 per clock and scheduler).  Its period is 2760 clocks (D = 128, no mask), given by the buffer
// of scores: per tile 220 to read it, 570-650 for the MMAs, the rest barriers and latency of the
// pipe.  Before, P_t overwrote S_t, so that the scores of the next step had to wait for softmax
// and P V of this one: 3500 clocks.
//
// Instruction fetch is what such a kernel trips over: softmax and issuers run different
// code side by side, two tiles half a step apart, and the cache of an SM holds little.  With the
// issuers unrolled per tile, a lane chosen by `lane == 0` (every MMA operand is then brought to uniform registers one by one),
// and long wait loops, the kernel had 110 KB of code, 21 % of the instruction requests missed (the former design: 10 %) and the
// schedule above took 3900 clocks.  Hence: one copy of the code for both tiles, short loops,
// elect.sync, a warp index known to be uniform, a wait loop of a few instructions, one place
// per role that reports an error: 60 KB, 1.5 % misses.
//
// Softmax: thread = row.  If the maximum of a step exceeds the row's reference maximum by
// more than 2^8 the row is re-based at once; otherwise the reference stays and nothing is rescaled -- one vote and
// one rarely taken branch per step.  Then the probabilities are formed and stored as P chunk by chunk.  On diagonal and ragged tiles a
// small loop first writes -inf over the hidden scores in tensor memory; the step
// itself is one piece of code for every tile.
// An additive bias is added behind the load (kernel variants of their own).  When the first half of P (keys 0-63) is stored the softmax
// arrives on a barrier of its own and the PV warp issues that half while the other half is still being computed.
//
// Masks are index arithmetic on (row, key) positions; K/V heads of a GQA group
// are indexed, never expanded; V rows past a sequence's end are zeroed in
// shared memory and K garbage is masked by select, so NaN in padding cannot
// leak.  Every wait is bounded: a wait that runs out records a code in the
// device status word, all warps leave their loops, tensor memory is freed and
// the CTA returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "internal.h"
#include "prefill_sm100.h"
#include "ptx.cuh"

namespace xfb {
namespace pst {

constexpr int kBM = 128;    // rows per query tile
constexpr int kTiles = 2;   // query tiles per item
constexpr int kBN = 128;    // keys per step
constexpr int kMaxStages = 2;  // depth of the K and of the V ring
constexpr int kSched = 4;   // depth of the ring that announces work items
constexpr int kThreads = 512;
constexpr int kOutWarp0 = 8, kPvWarp0 = 12, kTmaWarp = 14, kQkWarp = 15;
constexpr int kItemReaders = 15;  // warps that read every announced item (all but the scheduler)
// registers per thread after setmaxnreg; the sum over the 16 warps must fit what the CTA was launched with
#ifndef XFB_PST_REGS_SOFTMAX
#define XFB_PST_REGS_SOFTMAX 184
#endif
#ifndef XFB_PST_REGS_OUT
#define XFB_PST_REGS_OUT 64
#endif
#ifndef XFB_PST_REGS_AUX
#define XFB_PST_REGS_AUX 80
#endif
constexpr int kRegsLaunch = 128, kRegsSoftmax = XFB_PST_REGS_SOFTMAX, kRegsOut = XFB_PST_REGS_OUT, kRegsAux = XFB_PST_REGS_AUX;
static_assert(8 * kRegsSoftmax + 4 * kRegsOut + 4 * kRegsAux <= 16 * kRegsLaunch, "setmaxnreg would ask for more registers than the CTA owns");
constexpr float kRescaleThreshold = 8.0f;  // a row is re-based when its maximum grew by more than 2^8: probabilities stay below 2^8
constexpr uint32_t kHalfBytes = 128 * 128;  // one 64-column block of a 128-row tile

// Geometry of a work item, worked out once by the scheduler warp and read by the others from shared memory.
struct Item {
  int idx;  // item number, -1 = no more work
  int b, head, kv_head, tb;
  int g, h;
  int q_row0, k_row0, qlen, klen;
  int m0, shift, n_base;
  int shift2;  // two key ranges in one tensor: what `shift` is for the keys from row kv_split on
  int jlo[kTiles], jhi[kTiles];  // key-step range of each query tile, in steps of kBN keys from n_base
  int j_begin, j_end;            // steps any tile takes part in
};

struct __align__(8) Barriers {
  uint64_t sched_full[kSched], sched_empty[kSched];
  uint64_t q_full[kTiles], q_empty[kTiles];
  uint64_t k_full[kMaxStages], v_full[kMaxStages], k_empty[kMaxStages], v_empty[kMaxStages];
  uint64_t s_full[kTiles], s_empty;          // s_empty: the scores are in registers (the two tiles share one buffer)
  uint64_t p_half[kTiles], p_full[kTiles];   // p_half: the probabilities of keys 0-63 are stored
  uint64_t pv_done[kTiles];                  // P_t has been read, O_t is quiescent
  uint64_t o_full[kTiles], o_empty[kTiles];
  uint64_t stats_full[kTiles], stats_empty[kTiles];
  Item sched_item[kSched];
  uint32_t tmem_base;
  uint32_t abort_flag;
};

template <int D>
struct Smem {
  // above 128 columns an item is one tile (two outputs do not fit the tensor memory), and the rings hold one step
  static constexpr int kQTiles = D > 128 ? 1 : kTiles, kStages = D > 128 ? 1 : kMaxStages;
  static constexpr int kQTile = kBM * D * 2;
  static constexpr int kKV = kBN * D * 2;
  static constexpr int kQ = 0;
  static constexpr int kK = kQ + kQTiles * kQTile;
  static constexpr int kV = kK + kStages * kKV;
  static constexpr int kStats = kV + kStages * kKV;          // float2 [kTiles][kBM]: running maximum (log2 units), row sum
  static constexpr int kBar = kStats + kTiles * kBM * 8;
  static constexpr int kBias = kBar + 1024;  // with a bias only: one unit of 32 rows x 64 bytes for each softmax warp
  static constexpr int kBiasUnit = 32 * 64;
  static constexpr int kTotal = kBar + 1024 + 1024;
  static constexpr int kTotalBiased = kTotal + 8 * kBiasUnit;
};
static_assert(sizeof(Barriers) <= 1024, "barrier block");

// Columns of the tensor memory: scores (fp32, one buffer in which the two tiles take turns), probabilities (16-bit pairs), output
// (fp32).  At D = 128 these are all 512 columns, as at D = 256, where there is one tile; at D = 64 a buffer of scores per tile would fit, but then nothing keeps the
// tiles half a step apart (4 x 4096 rows, 32 heads, no mask: 778 us with two buffers, 664 with one).
template <int D>
struct Tmem {
  static constexpr uint32_t kS = 0;
  __device__ static constexpr uint32_t p(int t) { return kBN + t * (kBN / 2); }
  __device__ static constexpr uint32_t o(int t) { return 2 * kBN + t * D; }
};

// Packed fp32 pairs live in 64-bit registers; building and splitting them with
// mov.b64 keeps everything in registers (no address-taken locals).
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t fadd2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fmul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
template <bool kBf16>
__device__ __forceinline__ void unpack_pair(uint32_t x, float& lo, float& hi) {
  if constexpr (kBf16) {
    lo = __uint_as_float(x << 16);
    hi = __uint_as_float(x & 0xffff0000u);
  } else {
    const float2 f = __half22float2(*reinterpret_cast<__half2*>(&x));
    lo = f.x, hi = f.y;
  }
}
template <bool kBf16>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
  if constexpr (kBf16) {
    __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
  } else {
    __half2 t = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
  }
}

#ifdef XFB_PST_PROFILE
// Timing build only: per-CTA cycle counters of the softmax warps (16 slots each, 0-127) and of the two MMA issuers
// (128-143 / 144-159), read back with xfb200_debug_read_prefill_profile.
__device__ long long g_prof[160][160];
#define XFB_PROF_DECL(n) long long prof_acc[n] = {0}; long long prof_t = clock64();
#define XFB_PROF_LAP(k) { const long long _n = clock64(); prof_acc[k] += _n - prof_t; prof_t = _n; }
#define XFB_PROF_COUNT(k) { prof_acc[k] += 1; }
#define XFB_PROF_STORE(base, n) { if (lane == 0 && blockIdx.x < 160) for (int _i = 0; _i < (n); ++_i) g_prof[blockIdx.x][(base) + _i] += prof_acc[_i]; }
#else
#define XFB_PROF_DECL(n)
#define XFB_PROF_LAP(k)
#define XFB_PROF_COUNT(k)
#define XFB_PROF_STORE(base, n) {}
#endif

// Records the first code a launch gives up with (kept until the host reads it) and marks the
// launch, so that CTAs that have not started yet leave at once.
__device__ __forceinline__ void give_up(const Sm100Args& a, int code) {
  atomicCAS(a.status, 0, code);
  reinterpret_cast<volatile int32_t*>(a.status)[1] = int32_t(a.epoch);
}

// Order in which the sequences of a packed batch are taken: longest first (lane r holds the sequence of rank r).  Contexts of a
// chunked prefill differ by an order of magnitude, and items are only ordered inside a sequence: the long ones must not come
// last (8 sequences of 835 to 6822 keys, 150 to 480 new tokens each: 206 -> 191 us with the rotary pass; simulated item by item the
// launch goes from 162 to 128, 120 being the mean over the SMs).  A warp ranks up to 32 sequences, one per lane; a longer batch keeps
// the order it came in (not measured there: one long context behind many short ones still ends the launch alone).
__device__ __forceinline__ int sequence_order(const Sm100Args& a, int lane) {
  if (a.seqstart_q == nullptr || a.batch > 32) return lane;
  int keys = -1;
  if (lane < a.batch && a.seqstart_q[lane + 1] > a.seqstart_q[lane])
    keys = a.seqlen_k != nullptr ? a.seqlen_k[lane] : a.seqstart_k[lane + 1] - a.seqstart_k[lane];
  int rank = lane < a.batch ? 0 : lane;
  for (int s = 0; s < a.batch; ++s) {
    const int other = __shfl_sync(0xffffffffu, keys, s);
    if (lane < a.batch && (other > keys || (other == keys && s < lane))) ++rank;
  }
  int order = lane;
  for (int s = 0; s < a.batch; ++s)
    if (__shfl_sync(0xffffffffu, rank, s) == lane) order = s;
  return order;
}

// Returns false when the item has no query row at all (a row block past the end of its sequence).  Called by a whole warp.
__device__ __forceinline__ bool decode_item(const Sm100Args& a, int order, int idx, Item& it) {
  it.idx = idx;
  const int n_heads = (a.groups * a.heads_per_group) >> a.pack_shift;  // (or groups of packed heads)
  const int n_bh = n_heads * a.batch;
  const int tile_rows = kBM >> a.pack_shift;  // query rows (tokens) of a tile
  // Heaviest (latest) row blocks first, but not over all heads at once: the CTAs of a launch run side by side, and
  // the keys and values they read should fit the L2 (a K/V tile is read once per row block of its head: from DRAM
  // the first time only, if it is still there).  Heads are taken in groups of heads_per_wave; inside a group the
  // row blocks go from the last to the first, so the launch still ends with light items.
  const int kHeadsPerWave = a.heads_per_wave;
  const int grp = idx / (kHeadsPerWave * a.q_tiles);
  const int first_bh = grp * kHeadsPerWave;
  const int in_grp = min(kHeadsPerWave, n_bh - first_bh);
  const int rr = idx - grp * kHeadsPerWave * a.q_tiles;
  const int qt = a.q_tiles - 1 - rr / in_grp;
  const int bh = first_bh + rr % in_grp;
  it.b = bh / n_heads;
  if (a.seqstart_q != nullptr && a.batch <= 32) it.b = __shfl_sync(0xffffffffu, order, it.b);
  it.head = (bh % n_heads) << a.pack_shift;
  it.g = it.head / a.heads_per_group, it.h = it.head % a.heads_per_group;
  it.kv_head = it.g * (a.kv_h_is_broadcast ? 1 : a.heads_per_group) + (a.kv_h_is_broadcast ? 0 : it.h);
  it.q_row0 = 0, it.k_row0 = 0, it.qlen = a.mq, it.klen = a.mkv, it.tb = it.b;
  if (a.seqstart_q != nullptr) {
    it.q_row0 = a.seqstart_q[it.b];
    it.qlen = a.seqstart_q[it.b + 1] - it.q_row0;
    it.k_row0 = a.seqstart_k[it.b];
    it.klen = a.seqlen_k != nullptr ? a.seqlen_k[it.b] : a.seqstart_k[it.b + 1] - it.k_row0;
    it.tb = 0;
  }
  const int item_rows = a.item_rows >> a.pack_shift;
  it.m0 = qt * item_rows;
  if (it.m0 >= it.qlen) return false;
  it.shift = (a.bottom_right ? it.klen - it.qlen : 0) - a.kv_offset;
  it.qlen = min(it.qlen, it.m0 + item_rows);  // (an item of one tile has no row of the other)
  it.shift2 = -a.kv_offset2;
  it.n_base = 0;
  if (a.window_left >= 0) it.n_base = max(0, it.m0 + it.shift - a.window_left) / kBN * kBN;
  it.j_begin = 0x7fffffff, it.j_end = 0;
#pragma unroll
  for (int t = 0; t < kTiles; ++t) {
    const int mt0 = it.m0 + t * tile_rows;
    int hi = it.klen, lo = it.n_base;
    if (a.window_right >= 0) hi = min(hi, mt0 + tile_rows + it.shift + a.window_right);
    if (a.kv_split > 0) {
      // Two key ranges back to back (causal, the second one later in the sequence): rows that see any key of the
      // second range see all of the first, so the visible keys are still one run of rows of the tensor.
      const int hi1 = min(it.klen - a.kv_split, mt0 + tile_rows + it.shift2);
      hi = hi1 > 0 ? a.kv_split + hi1 : min(a.kv_split, mt0 + tile_rows + it.shift);
    }
    if (a.window_left >= 0) lo = max(it.n_base, max(0, mt0 + it.shift - a.window_left) / kBN * kBN);
    if (mt0 >= it.qlen) hi = lo;  // no valid row in this tile
    it.jlo[t] = (lo - it.n_base) / kBN;
    it.jhi[t] = hi > lo ? (hi - it.n_base + kBN - 1) / kBN : it.jlo[t];
    if (it.jhi[t] > it.jlo[t]) {
      it.j_begin = min(it.j_begin, it.jlo[t]);
      it.j_end = max(it.j_end, it.jhi[t]);
    }
  }
  if (it.j_end == 0) it.j_begin = 0;
  return true;
}

// D: columns of the tiles (64, 128 or 256).  kVariant:
//   kExact   the head dim is D
//   kPadded  the head dim a.head_dim is smaller than D; the copies fill the columns behind it with zeros, the products
//            leave out what lies wholly behind it, the output is written up to it
//   kBiasedSame, kBiasedOther, kBiasedF32  an additive bias of the type of q, of the other 16-bit type, of 32 bits, which the step
//            knows at compile time; the head dim may be D or smaller
constexpr int kExact = 0, kPadded = 1, kBiasedSame = 2, kBiasedOther = 3, kBiasedF32 = 4;
template <int D, bool kBf16, int kVariant>
__global__ void __launch_bounds__(kThreads, 1) prefill_sm100_persist_kernel(const __grid_constant__ Sm100Args a) {
  using L = Smem<D>;
  using T = Tmem<D>;
  constexpr bool kPad = kVariant != kExact, kBias = kVariant >= kBiasedSame, kBiasF32 = kVariant == kBiasedF32;
  constexpr int kHalves = D / 64;
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);  // an offset, so that the compiler keeps seeing shared memory
  Barriers* bar = reinterpret_cast<Barriers*>(smem + L::kBar);
  float2* stats = reinterpret_cast<float2*>(smem + L::kStats);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int n_items = a.n_items;
  const int pack_shift = kBias ? 0 : a.pack_shift;
  const int tile_rows = kBM >> pack_shift;  // query rows (tokens) of a tile
  const uint32_t budget = a.wait_budget;
  const int head_dim = kPad ? a.head_dim : D;

  // a CTA of this launch already gave up: take no work (the counters are still settled below)
  const bool drained = reinterpret_cast<volatile int32_t*>(a.status)[1] == int32_t(a.epoch);

  if (!drained) {
    if (threadIdx.x == 0) {
      for (int i = 0; i < kSched; ++i) {
        mbar_init(&bar->sched_full[i], 1);
        mbar_init(&bar->sched_empty[i], kItemReaders);
      }
      for (int i = 0; i < kMaxStages; ++i) {
        mbar_init(&bar->k_full[i], 1);
        mbar_init(&bar->k_empty[i], 1);
        mbar_init(&bar->v_full[i], 1);
        mbar_init(&bar->v_empty[i], kTiles);  // released by both PV warps
      }
      for (int t = 0; t < kTiles; ++t) {
        mbar_init(&bar->q_full[t], 1);
        mbar_init(&bar->q_empty[t], 1);
        mbar_init(&bar->s_full[t], 1);
        mbar_init(&bar->p_half[t], 4);  // one arrival per softmax warp of the tile
        mbar_init(&bar->p_full[t], 4);
        mbar_init(&bar->pv_done[t], 1);
        mbar_init(&bar->o_full[t], 1);
        mbar_init(&bar->o_empty[t], 128);
        mbar_init(&bar->stats_full[t], 128);
        mbar_init(&bar->stats_empty[t], 128);
      }
      mbar_init(&bar->s_empty, 4);
      bar->abort_flag = 0;
      mbar_fence_init();
    }
    if (warp == kQkWarp) {
      tmem_alloc(&bar->tmem_base, 512);
      tmem_relinquish();
    }
    if (warp == kTmaWarp && elect_one()) {
      prefetch_tensormap(&a.tm_q);
      prefetch_tensormap(&a.tm_k);
      prefetch_tensormap(&a.tm_v);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bar->tmem_base;
    volatile uint32_t* abort_flag = &bar->abort_flag;
    // (barriers, tensor memory and its allocation do not wait for the kernel ahead in the stream; everything below does)
    grid_dep_wait();
    // (not with a bias: 128 items of one launch and the next one's on the SMs beside them, 82.5 -> 83.6 us for 2 x 2048 x 2048)
    // (nor where SMs are to stay free for another stream's kernels: the CTAs of the next launch would take these and wait there)
    if constexpr (!kBias)
      if (a.sm_margin == 0) grid_dep_launch();

    // Next announced item (every announced item has key steps): its number, -1 after the last one, -2 when the
    // wait ran out.  `take` copies what the caller needs out of the descriptor before the slot is handed back.
    auto pop_item = [&](int& seq, auto&& take) -> int {
      const int slot = seq % kSched;
      if (!mbar_wait(&bar->sched_full[slot], (seq / kSched) & 1, abort_flag, budget)) return -2;
      const Item* d = &bar->sched_item[slot];
      const int idx = d->idx;
      if (idx >= 0) take(*d);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->sched_empty[slot]);
      ++seq;
      return idx;
    };

    if (warp >= kPvWarp0) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsAux));
      if (warp == kTmaWarp) {
        // ============================================ scheduler + TMA producer
        // All lanes run the loop, because pulling an item (a broadcast) and writing the rows of an item without
        // visible keys are done by the whole warp; one lane issues the copies.
        const int order = sequence_order(a, lane);
        int seq = 0;           // items announced
        int ks = 0, kph = 1;   // K stage / parity its release is waited for with
        int vs = 0, vph = 1;
        uint32_t qph = 3;      // parities of the two Q buffers
        int code = 0;
        // Pulls item numbers until one has key steps.  Row blocks past the end of their sequence are
        // skipped; blocks whose rows see no key at all get their result here: zeros and -inf.
        // Where there are no more items than CTAs, and all alike, each has its own: the counter's answer takes 0.4 us, which nothing
        // hides yet (2 x 100 rows, 16 heads: 8.5 -> 8.1 us).  Otherwise the first CTAs to run have to get the first, heaviest items
        // (8 sequences of chunked prefill, first items by CTA number: 142 -> 146 us; causal, 333 rows, 8 heads: 8.7 -> 8.9).
        int own = n_items <= int(gridDim.x) && (a.window_right < 0 || a.mkv <= kBN) ? int(blockIdx.x) : -1;
        auto next_item = [&](Item& it) {
          for (;;) {
            int idx = own;
            if (own < 0) {
              if (lane == 0) idx = atomicAdd(a.counters, 1);
              idx = __shfl_sync(0xffffffffu, idx, 0);
            } else {
              own = n_items;
            }
            if (idx >= n_items) {
              it.idx = -1;
              return;
            }
            if (!decode_item(a, order, idx, it)) continue;
            if (it.j_end > it.j_begin) return;
            const int nrows = (it.qlen - it.m0) << pack_shift, head_mask = (1 << pack_shift) - 1;
            const int osz = a.out_dtype == XFB200_F32 ? 4 : 2;
            const int chunks = head_dim * osz / 16;
            uint8_t* ob = reinterpret_cast<uint8_t*>(a.out);
            const int64_t base = int64_t(it.tb) * a.os.b + int64_t(it.q_row0 + it.m0) * a.os.m + int64_t(it.g) * a.os.g + int64_t(it.h) * a.os.h;
#pragma unroll 1
            for (int i = lane; i < nrows * chunks; i += 32) {
              const int r = i / chunks, c = i % chunks;
              *reinterpret_cast<uint4*>(ob + (base + int64_t(r >> pack_shift) * a.os.m + int64_t(r & head_mask) * a.os.h) * osz + c * 16) = make_uint4(0, 0, 0, 0);
            }
            if (a.lse != nullptr) {
              const int64_t lo = a.seqstart_q != nullptr ? int64_t(it.g) * a.lse_g + int64_t(it.h) * a.lse_h + it.q_row0 + it.m0
                                                         : int64_t(it.b) * a.lse_b + int64_t(it.g) * a.lse_g + int64_t(it.h) * a.lse_h + it.m0;
#pragma unroll 1
              for (int r = lane; r < nrows; r += 32) a.lse[lo + (r >> pack_shift) + int64_t(r & head_mask) * a.lse_h] = -INFINITY;
            }
          }
        };
        // one tile of 128 rows (Q, K or V), as blocks of 64 columns
        const int blocks = D > 128 && kPad ? (head_dim + 63) / 64 : kHalves;
        auto load_tile = [&](int at, const CUtensorMap* tm, uint64_t* full, int head, int row, int tb) {
          if (elect_one()) {
            mbar_expect_tx(full, blocks * kHalfBytes);
#pragma unroll
            for (int hf = 0; hf < kHalves; ++hf)
              if (hf < blocks) tma_load_4d(smem + at + hf * kHalfBytes, tm, full, hf * 64, head, row, tb);
          }
        };
        // The V tile of a step is loaded behind the K tile of the step after it: its stage comes free a softmax later
        // than the K stage, which must not wait for that.
        int pend_row = -1, pend_head = 0, pend_tb = 0;
        auto load_pending_v = [&]() -> bool {
          if (pend_row < 0) return true;
          if (!mbar_wait(&bar->v_empty[vs], vph, abort_flag, budget)) {
            code = 12;
            return false;
          }
          load_tile(L::kV + vs * L::kKV, &a.tm_v, &bar->v_full[vs], pend_head, pend_row, pend_tb);
          if (++vs == L::kStages) vs = 0, vph ^= 1;
          pend_row = -1;
          return true;
        };
        Item cur;
        next_item(cur);
        while (true) {
          const int slot = seq % kSched;
          if (!mbar_wait(&bar->sched_empty[slot], ((seq / kSched) & 1) ^ 1, abort_flag, budget)) {
            code = 10;
            break;
          }
          if (lane == 0) {
            bar->sched_item[slot] = cur;
            mbar_arrive(&bar->sched_full[slot]);  // (release: the descriptor is visible to whoever sees the phase)
          }
          ++seq;
          if (cur.idx < 0) {
            load_pending_v();
            break;
          }
          Item nxt;
          bool have_next = false;
#pragma unroll 1
          for (int j = cur.j_begin; j < cur.j_end; ++j) {
            const int row = cur.k_row0 + cur.n_base + j * kBN;
            if (!mbar_wait(&bar->k_empty[ks], kph, abort_flag, budget)) {
              code = 11;
              break;
            }
            // (testing aid: the CTA that got the first item leaves out its last key tile, so that the wait for it runs out)
            if (!((a.debug_flags & 1) && cur.idx == 0 && j == cur.j_end - 1))
              load_tile(L::kK + ks * L::kKV, &a.tm_k, &bar->k_full[ks], cur.kv_head, row, cur.tb);
            if (++ks == L::kStages) ks = 0, kph ^= 1;
            if (!load_pending_v()) break;
            if (j == cur.j_begin) {
              // Q behind what does not wait for it: its buffers come free with the very last QK^T of the previous item
#pragma unroll 1
              for (int t = 0; t < kTiles; ++t) {
                if (t == 0 ? cur.jhi[0] <= cur.jlo[0] : cur.jhi[1] <= cur.jlo[1]) continue;
                if (!mbar_wait(&bar->q_empty[t], (qph >> t) & 1, abort_flag, budget)) {
                  code = 13;
                  break;
                }
                qph ^= 1u << t;
                load_tile(L::kQ + t * L::kQTile, &a.tm_q, &bar->q_full[t], cur.head, cur.q_row0 + cur.m0 + t * tile_rows, cur.tb);
              }
              if (code != 0) break;
            }
            pend_row = row, pend_head = cur.kv_head, pend_tb = cur.tb;
            // The first two steps fit the rings at once; from here on every load waits for a stage to
            // come free, so this is the moment to pull the next item: its latency costs nothing.
            if (!have_next && (j == cur.j_begin + 1 || j == cur.j_end - 1)) {
              next_item(nxt);
              have_next = true;
            }
          }
          if (code != 0) break;
          cur = nxt;
        }
        if (code != 0) {
          if (lane == 0) give_up(a, code);
          *abort_flag = 1;
        }
      } else {
        // ====================================================== MMA issuers
        // Warp 15 issues every QK^T, warps 12 and 13 the PV of tile 0 and 1.  A thread that issues tcgen05.mma stands still
        // while two or so are ahead of it in the tensor pipe, and for some 140 clocks at every commit; what one of the
        // three warps loses in that way, or in a wait, the others fill.  Their code is kept small (one copy for both
        // tiles, short loops): it shares the instruction cache with the softmax.
        XFB_PROF_DECL(16)
        // Shared-memory descriptors: the upper word is constant (stride between
        // 8-row groups = 1024 B, version 1, 128B swizzle); the lower word holds
        // (address >> 4) and the leading-dimension offset, so stepping through a
        // tile is one 32-bit add per operand.
        constexpr uint32_t kDescHi = 64u | (1u << 14) | (2u << 29);
        auto desc = [](uint32_t lo) -> uint64_t {
          uint64_t d;
          asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(kDescHi));
          return d;
        };
        int seq = 0, code = 0;
        int st = 0, ph = 0;  // K (or V) stage / phase of the step
        if (warp == kQkWarp) {
          constexpr uint32_t idesc_qk = umma_idesc(kBM, kBN, kBf16, false, false);
          // (a padded head dim: steps of 16 columns as far as it goes)
          const int qk_steps = kPad ? (head_dim + 15) / 16 : D / 16;
          const uint32_t q_lo = (smem_u32(smem + L::kQ) >> 4) | (1u << 16);
          const uint32_t k_lo = (smem_u32(smem + L::kK) >> 4) | (1u << 16);
          uint32_t sph = 1, qph = 0;  // parities: buffer of the scores (released), Q tiles (loaded)
          while (code == 0) {
            int j, j_end, jlo0, jhi0, jlo1, jhi1;
            const int idx = pop_item(seq, [&](const Item& d) {
              j = d.j_begin, j_end = d.j_end;
              jlo0 = d.jlo[0], jhi0 = d.jhi[0], jlo1 = d.jlo[1], jhi1 = d.jhi[1];
            });
            if (idx < 0) {
              if (idx == -2) code = 20;
              break;
            }
#pragma unroll 1
            for (; j < j_end; ++j) {
              if (!mbar_wait(&bar->k_full[st], ph, abort_flag, budget)) {
                code = 21;
                break;
              }
              XFB_PROF_LAP(1)  // wait for K
#pragma unroll 1
              for (int t = 0; t < kTiles; ++t) {
                const int jlo = t == 0 ? jlo0 : jlo1, jhi = t == 0 ? jhi0 : jhi1;
                if (j < jlo || j >= jhi) continue;
                bool ok = true;
                if (j == jlo) {
                  ok = mbar_wait(&bar->q_full[t], (qph >> t) & 1, abort_flag, budget);
                  qph ^= 1u << t;
                }
                // the scores that were here before have to be in registers
                if (!ok || !mbar_wait(&bar->s_empty, sph, abort_flag, budget)) {
                  code = 23 + t;
                  break;
                }
                sph ^= 1;
                tc_fence_after();
                XFB_PROF_LAP(2)  // wait for Q, for the buffer of the scores
                if (elect_one()) {
                  uint32_t ql = q_lo + t * (L::kQTile >> 4), kl = k_lo + st * (L::kKV >> 4);
#pragma unroll 1
                  for (int hf = 0; hf < kHalves; ++hf) {
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                      if (!kPad || hf * 4 + kk < qk_steps) umma_ss(tmem + T::kS, desc(ql + kk * 2), desc(kl + kk * 2), idesc_qk, kk > 0 ? 1u : uint32_t(hf));
                    ql += kHalfBytes >> 4, kl += kHalfBytes >> 4;
                  }
                  tc_commit(&bar->s_full[t]);
                  if (j == jhi - 1) tc_commit(&bar->q_empty[t]);
                }
                __syncwarp();
                XFB_PROF_LAP(3)  // QK^T issued
                XFB_PROF_COUNT(7)
              }
              if (code != 0) break;
              if (elect_one()) tc_commit(&bar->k_empty[st]);
              if (++st == L::kStages) st = 0, ph ^= 1;
            }
          }
        } else {
          const int t = warp - kPvWarp0;
          // (a padded head dim: a width that is a multiple of 16)
          const uint32_t idesc_pv = umma_idesc(kBM, kPad ? (head_dim + 15) / 16 * 16 : D, kBf16, false, true);
          const uint32_t v_lo = (smem_u32(smem + L::kV) >> 4) | ((kHalfBytes >> 4) << 16);
          const uint32_t tp = tmem + T::p(t), to = tmem + T::o(t);
          int cnt = 0, items = 0;  // products, items of this tile so far
          while (code == 0) {
            int j, j_end, jlo, jhi, n_base, klen;
            const int idx = pop_item(seq, [&](const Item& d) {
              j = d.j_begin, j_end = d.j_end, n_base = d.n_base, klen = d.klen;
              jlo = d.jlo[t], jhi = d.jhi[t];
            });
            if (idx < 0) {
              if (idx == -2) code = 20;
              break;
            }
#pragma unroll 1
            for (; j < j_end; ++j) {
              if (!mbar_wait(&bar->v_full[st], ph, abort_flag, budget)) {
                code = 22;
                break;
              }
              XFB_PROF_LAP(1)  // wait for V
              if (j >= jlo && j < jhi) {
                const int n0 = n_base + j * kBN;
                if (a.seqstart_k != nullptr && n0 + kBN > klen) {
                  // V rows past the end of the sequence may hold anything; P is 0 there.  (Behind the end of the tensor, where
                  // every sequence of a dense batch ends, the copy fills in zeros.)
                  // Both PV warps write the same zeros: no ordering between them is needed.
                  const int first = max(klen - n0, 0);
                  uint8_t* vt = smem + L::kV + st * L::kKV;
#pragma unroll 1
                  for (int hf = 0; hf < kHalves; ++hf)
#pragma unroll 1
                    for (int i = first * 8 + lane; i < kBN * 8; i += 32) *reinterpret_cast<uint4*>(vt + hf * kHalfBytes + i * 16) = make_uint4(0, 0, 0, 0);
                  fence_proxy_async_smem();
                  __syncwarp();
                }
                // the first product of an item overwrites O_t: the output warps must have read the previous one
                if (j == jlo && !mbar_wait(&bar->o_empty[t], (items++ & 1) ^ 1, abort_flag, budget)) {
                  code = 25 + t;
                  break;
                }
                // The first half of the product runs while the softmax is still busy with the second half of P.
                uint32_t vl = v_lo + st * (L::kKV >> 4), pt = tp;
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                  if (!mbar_wait(half == 0 ? &bar->p_half[t] : &bar->p_full[t], cnt & 1, abort_flag, budget)) {
                    code = 27 + t;
                    break;
                  }
                  tc_fence_after();
                  XFB_PROF_LAP(2 + 2 * half)  // wait for a half of P
                  if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < kBN / 32; ++kk)  // A = P_t: packed 16-bit pairs, 8 columns of tensor memory per 16 keys
                      umma_ts(to, pt + kk * 8, desc(vl + ((kk * 16 * 128) >> 4)), idesc_pv, kk > 0 ? 1u : uint32_t(j > jlo || half > 0));
                    if (half > 0) {
                      tc_commit(&bar->pv_done[t]);
                      if (j == jhi - 1) tc_commit(&bar->o_full[t]);
                    }
                  }
                  __syncwarp();
                  XFB_PROF_LAP(3 + 2 * half)  // half of PV issued
                  vl += (64 * 128) >> 4, pt += 32;
                }
                if (code != 0) break;
                ++cnt;
                XFB_PROF_COUNT(7)
              }
              if (elect_one()) tc_commit(&bar->v_empty[st]);
              if (++st == L::kStages) st = 0, ph ^= 1;
            }
          }
        }
        if (warp != kPvWarp0 + 1) XFB_PROF_STORE(128 + (warp == kQkWarp ? 0 : 16), 16)
        if (code != 0) {
          if (lane == 0) give_up(a, code);
          *abort_flag = 1;
        }
      }
    } else if (warp >= kOutWarp0) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOut));
      // ================================================================ output
      const int row = (warp & 3) * 32 + lane;  // TMEM lane == row inside the tile
      const uint32_t lane_sel = uint32_t((warp & 3) * 32) << 16;
      int seq = 0, code = 0;
      uint32_t oph = 0;  // parities of the two tiles
      while (code == 0) {
        struct {
          int b, tb, g, h, q_row0, m0, qlen, jlo0, jhi0, jlo1, jhi1;
        } it;
        const int idx = pop_item(seq, [&](const Item& d) {
          it.b = d.b, it.tb = d.tb, it.g = d.g, it.h = d.h, it.q_row0 = d.q_row0, it.m0 = d.m0, it.qlen = d.qlen;
          it.jlo0 = d.jlo[0], it.jhi0 = d.jhi[0], it.jlo1 = d.jlo[1], it.jhi1 = d.jhi[1];
        });
        if (idx < 0) {
          if (idx == -2) code = 40;
          break;
        }
#pragma unroll 1
        for (int t = 0; t < kTiles; ++t) {
          const int i_loc = it.m0 + t * tile_rows + (row >> pack_shift), h_loc = row & ((1 << pack_shift) - 1);
          const bool valid_row = i_loc < it.qlen;
          const bool active = t == 0 ? it.jhi0 > it.jlo0 : it.jhi1 > it.jlo1;
          if (!active && it.m0 + t * tile_rows >= it.qlen) continue;  // no row of this tile exists
          float m_run = -INFINITY, l_run = 0.f;
          const uint32_t tmem_o = tmem + T::o(t) + lane_sel;
          if (active) {
            bool ok = mbar_wait(&bar->stats_full[t], (oph >> t) & 1, abort_flag, budget);
            if (ok) {
              const float2 st = stats[t * kBM + row];
              m_run = st.x, l_run = st.y;
              mbar_arrive(&bar->stats_empty[t]);
              ok = mbar_wait(&bar->o_full[t], (oph >> t) & 1, abort_flag, budget);
            }
            if (!ok) {
              code = 41 + t;
              break;
            }
            oph ^= 1u << t;
            tc_fence_after();
          }
          const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
          const int64_t o_off = int64_t(it.tb) * a.os.b + int64_t(it.q_row0 + i_loc) * a.os.m + int64_t(it.g) * a.os.g + int64_t(it.h + h_loc) * a.os.h;
#pragma unroll 1
          for (int col = 0; col < D; col += 16) {
            uint32_t orr[16];
            if (active) {
              XFB_TMEM_LD_16(tmem_o + col, orr);
              XFB_TMEM_WAIT_LD_16(orr);
              if (col == D - 16) {
                // O_t is in registers: the next item's first PV may overwrite it
                tc_fence_before();
                mbar_arrive(&bar->o_empty[t]);
              }
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) orr[i] = 0;
            }
            if (valid_row) {
              if (a.out_dtype == XFB200_F32) {
                float* dst = reinterpret_cast<float*>(a.out) + o_off + col;
#pragma unroll
                for (int i = 0; i < 16; i += 4)
                  if (!kPad || col + i < head_dim)
                    *reinterpret_cast<float4*>(dst + i) = make_float4(__uint_as_float(orr[i]) * inv, __uint_as_float(orr[i + 1]) * inv,
                                                                      __uint_as_float(orr[i + 2]) * inv, __uint_as_float(orr[i + 3]) * inv);
              } else {
                uint16_t* dst = reinterpret_cast<uint16_t*>(a.out) + o_off + col;
#pragma unroll
                for (int i = 0; i < 16; i += 8) {
                  uint32_t w[4];
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    const float x0 = __uint_as_float(orr[i + 2 * e]) * inv, x1 = __uint_as_float(orr[i + 2 * e + 1]) * inv;
                    w[e] = a.out_dtype == XFB200_BF16 ? pack_pair<true>(x0, x1) : pack_pair<false>(x0, x1);
                  }
                  if (!kPad || col + i < head_dim) *reinterpret_cast<uint4*>(dst + i) = make_uint4(w[0], w[1], w[2], w[3]);
                }
              }
            }
          }
          if (valid_row && a.lse != nullptr) {
            const float lse = l_run > 0.f ? (m_run + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
            const int64_t lo = a.seqstart_q != nullptr ? int64_t(it.g) * a.lse_g + int64_t(it.h + h_loc) * a.lse_h + it.q_row0 + i_loc
                                                       : int64_t(it.b) * a.lse_b + int64_t(it.g) * a.lse_g + int64_t(it.h + h_loc) * a.lse_h + i_loc;
            a.lse[lo] = lse;
          }
        }
      }
      if (code != 0) {
        give_up(a, code);
        *abort_flag = 1;
      }
      tc_fence_before();
    } else {
      asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
      // ================================================================ softmax
      const int t = warp >> 2;                  // query tile of this warpgroup
      const int row = (warp & 3) * 32 + lane;   // TMEM lane == row inside the tile
      const uint32_t lane_sel = uint32_t((warp & 3) * 32) << 16;
      const uint32_t tmem_s = tmem + T::kS + lane_sel, tmem_p = tmem + T::p(t) + lane_sel, tmem_o = tmem + T::o(t) + lane_sel;
      // what brings the scores to log2 units; with an additive bias they are brought there before it is added, since the bias itself
      // times 1 / scale would overflow where the bias does not, and a large score would lose against its own maximum what the
      // product rounds
      const float sl2 = kBias ? 1.f : a.scale_log2;
      const uint64_t sc2 = f2_pack(sl2, sl2);
      int seq = 0;
      int cnt = 0;  // steps of this tile so far, over all items
      int ka = 0;   // items in which this tile took part so far
      int code = 0;
      XFB_PROF_DECL(16)

      // visibility of the 32 columns starting at key `col0` for this thread's row: hidden scores become -inf
      int col_lo = 0, col_hi = 0;
      auto mask_chunk = [&](float* sc, int col0) {
        // one bit per column, then a test and a select per score
        const int hr = col_hi - col0, lr = col_lo - col0;
        const uint32_t below_hi = hr >= 32 ? 0xffffffffu : (hr <= 0 ? 0u : (1u << hr) - 1u);
        const uint32_t from_lo = lr <= 0 ? 0xffffffffu : (lr >= 32 ? 0u : ~((1u << lr) - 1u));
        const uint32_t vis = below_hi & from_lo;
#pragma unroll
        for (int c = 0; c < 32; ++c) sc[c] = (vis & (1u << c)) != 0u ? sc[c] : -INFINITY;
      };
      auto chunk_max = [](const float* sc) -> float {
        float m0 = fmax3(sc[0], sc[1], sc[2]), m1 = fmax3(sc[3], sc[4], sc[5]), m2 = fmax3(sc[6], sc[7], sc[8]), m3 = fmax3(sc[9], sc[10], sc[11]);
        m0 = fmax3(m0, sc[12], sc[13]), m1 = fmax3(m1, sc[14], sc[15]), m2 = fmax3(m2, sc[16], sc[17]), m3 = fmax3(m3, sc[18], sc[19]);
        m0 = fmax3(m0, sc[20], sc[21]), m1 = fmax3(m1, sc[22], sc[23]), m2 = fmax3(m2, sc[24], sc[25]), m3 = fmax3(m3, sc[26], sc[27]);
        m0 = fmax3(m0, sc[28], sc[29]), m1 = fmax3(m1, sc[30], sc[31]);
        return fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
      };
      // 32 score columns -> 16 packed probability pairs against the maximum -m (nm2 = (-m, -m)), summed into
      // sum2 and stored to the 16 columns of P_t that start at `col`
      auto exp_store = [&](const uint32_t* sr, int col, uint64_t nm2, uint64_t (&sum2)[4]) {
        uint32_t pr[16];
        // (blocks of 16 independent elements: all FMAs, then all exp2, then the sums and packs -- a lone warp per
        // scheduler hides no latency by switching warps, the instruction stream has to)
#pragma unroll
        for (int h = 0; h < 32; h += 16) {
          float e[16];
#pragma unroll
          for (int i = 0; i < 16; i += 2)
            if constexpr (kBias)
              f2_unpack(fadd2(f2_pack(__uint_as_float(sr[h + i]), __uint_as_float(sr[h + i + 1])), nm2), e[i], e[i + 1]);
            else
              f2_unpack(ffma2(f2_pack(__uint_as_float(sr[h + i]), __uint_as_float(sr[h + i + 1])), sc2, nm2), e[i], e[i + 1]);
#pragma unroll
          for (int i = 0; i < 16; ++i) e[i] = fast_exp2(e[i]);
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            sum2[(i / 2) & 3] = fadd2(sum2[(i / 2) & 3], f2_pack(e[i], e[i + 1]));
            pr[(h + i) / 2] = pack_pair<kBf16>(e[i], e[i + 1]);
          }
        }
        XFB_TMEM_ST_16(tmem_p + col, pr);
      };
      // O_t *= alpha (per row), through registers
      auto rescale_o = [&](float alpha) {
        const uint64_t al2 = f2_pack(alpha, alpha);
#pragma unroll
        for (int cblk = 0; cblk < D / 16; ++cblk) {
          uint32_t orr[16];
          XFB_TMEM_LD_16(tmem_o + cblk * 16, orr);
          XFB_TMEM_WAIT_LD_16(orr);
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            float x0, x1;
            f2_unpack(fmul2(f2_pack(__uint_as_float(orr[i]), __uint_as_float(orr[i + 1])), al2), x0, x1);
            orr[i] = __float_as_uint(x0);
            orr[i + 1] = __float_as_uint(x1);
          }
          XFB_TMEM_ST_16(tmem_o + cblk * 16, orr);
        }
        tc_wait_st();
      };

      // ---- additive bias.  Bound by how its bytes reach the registers: a row per thread is the layout of the
      // scores, and reading memory that way costs one sector request per element (2048 x 2048 x 16 heads, bf16: 600 us).
      // A warp therefore reads its 32 rows in units of 64 bytes per row, four lanes to a row and 16 bytes to a lane, holds
      // the units of a step in registers from before the wait for the scores on, and turns one after the other into
      // rows through 2 KB of shared memory (16-byte chunks XOR-ed with row / 2, no bank conflict either way): 69 us for the
      // same call (34 GFLOP, 134 MB of bias).  A unit is
      // 32 columns of a 16-bit bias (four units: a step) or 16 of an f32 one (eight).
      //   An f32 bias takes 128 registers a step, as do the scores.  So its scores come 32 at a time, get their bias and go back to tensor
      // memory, from where the step reads them as it does without a bias; six units are asked for before the wait, the last two when
      // the first two are through.  With row and half a step of bias in registers together, the second half asked for when the first was
      // used up, the step spilled, and the type asked for at run time made it worse: 3 x 3000 x 3000, 12 heads of 64, bf16, f32 bias 457
      // -> 369 us (413 before the row was kept in registers), 8 heads x 700, causal, 39.8 -> 35.6; f16 with a bf16 bias 329 -> 271 and 31.7 -> 27.6.
      constexpr float kLog2e = 1.4426950408889634f;
      const uint64_t scale2 = f2_pack(a.scale_log2, a.scale_log2), log2e2 = f2_pack(kLog2e, kLog2e);
      uint8_t* const bias_smem = smem + L::kBias + warp * L::kBiasUnit;
      // Row r reads its visible keys only, [r + rel_lo, min(r + rel_hi, n_keys)), and has 0 for the others: their scores are -inf
      // already, and what the bias holds there, a NaN perhaps, must not meet that.  (Masking behind the addition instead costs the
      // step registers: 75.5 -> 86.7 us for 2 x 2048 x 2048, 8 heads, no mask at all.)  `whole`: a step of which every row and key
      // counts, and rows on 16-byte boundaries; its loads need no test (the tests cost that call 3.4 us).
      auto bias_load = [&](uint4* w, auto n_units, int64_t off, int mt0, int qlen, int col_first, int n_keys, int rel_lo, int rel_hi, bool whole) {
        constexpr int kUnits = decltype(n_units)::value, esz = kBiasF32 ? 4 : 2, per16 = 16 / esz;
        if (whole) {
          const int r = mt0 + (warp & 3) * 32 + (lane >> 2);
          const uint8_t* src = reinterpret_cast<const uint8_t*>(a.bias) + (off + int64_t(r) * a.bias_m + col_first + (lane & 3) * per16) * esz;
          const int64_t step = 8 * a.bias_m * esz;
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int u = 0; u < kUnits; ++u) w[u * 4 + i] = __ldg(reinterpret_cast<const uint4*>(src + i * step + u * 64));
          return;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = mt0 + (warp & 3) * 32 + i * 8 + (lane >> 2);
          const int lo = r + rel_lo, hi = min(r + rel_hi, n_keys);
          const uint8_t* src = reinterpret_cast<const uint8_t*>(a.bias) + (off + int64_t(r) * a.bias_m) * esz;
#pragma unroll
          for (int u = 0; u < kUnits; ++u) {
            const int col = col_first + (u * 4 + (lane & 3)) * per16;
            uint4 x = make_uint4(0, 0, 0, 0);
            if (r < qlen && col < hi) {
              auto seen = [&](int k) { return col + k < hi && col + k >= lo; };
              if (a.bias_vec && col + per16 <= hi && col >= lo) {
                x = __ldg(reinterpret_cast<const uint4*>(src + col * esz));
              } else if (esz == 4) {
                const uint32_t* e = reinterpret_cast<const uint32_t*>(src) + col;
                if (seen(0)) x.x = e[0];
                if (seen(1)) x.y = e[1];
                if (seen(2)) x.z = e[2];
                if (seen(3)) x.w = e[3];
              } else {
                const uint16_t* e = reinterpret_cast<const uint16_t*>(src) + col;
                auto el = [&](int k) -> uint32_t { return seen(k) ? e[k] : 0; };
                x = make_uint4(el(0) | el(1) << 16, el(2) | el(3) << 16, el(4) | el(5) << 16, el(6) | el(7) << 16);
              }
            }
            w[u * 4 + i] = x;
          }
        }
      };
      auto bias_prefetch = [&](int64_t off, int mt0, int qlen, int col_first, int n_keys) {
        constexpr int esz = kBiasF32 ? 4 : 2;
        const int r = mt0 + row;
        const uint8_t* src = reinterpret_cast<const uint8_t*>(a.bias) + (off + int64_t(r) * a.bias_m) * esz;
        for (int col = col_first; col < col_first + kBN; col += 128 / esz)
          if (r < qlen && col < n_keys) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + int64_t(col) * esz));
      };
      // 32 scores of this thread's row become (score * scale + bias) * log2 e; w: the unit (two, f32) of their columns
      auto bias_add = [&](uint32_t* sc, const uint4* w) {
        auto to_rows = [&](int u, uint4 (&mine)[4]) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(bias_smem + (i * 8 + (lane >> 2)) * 64 + (((lane & 3) ^ ((lane >> 3) & 3)) << 4)) = w[u * 4 + i];
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) mine[k] = *reinterpret_cast<const uint4*>(bias_smem + lane * 64 + ((k ^ ((lane >> 1) & 3)) << 4));
          __syncwarp();
        };
        auto add = [&](int c, float x) { sc[c] = __float_as_uint(fmaf(__uint_as_float(sc[c]), a.scale_log2, x * kLog2e)); };
        if constexpr (kBiasF32) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint4 mine[4];
            to_rows(h, mine);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              add(h * 16 + k * 4, __uint_as_float(mine[k].x)), add(h * 16 + k * 4 + 1, __uint_as_float(mine[k].y));
              add(h * 16 + k * 4 + 2, __uint_as_float(mine[k].z)), add(h * 16 + k * 4 + 3, __uint_as_float(mine[k].w));
            }
          }
          return;
        }
        uint4 mine[4];
        to_rows(0, mine);
        auto add2 = [&](int c, uint32_t x) {
          float lo, hi;
          unpack_pair<kBf16 == (kVariant == kBiasedSame)>(x, lo, hi);
          f2_unpack(ffma2(f2_pack(__uint_as_float(sc[c]), __uint_as_float(sc[c + 1])), scale2, fmul2(f2_pack(lo, hi), log2e2)), lo, hi);
          sc[c] = __float_as_uint(lo), sc[c + 1] = __float_as_uint(hi);
        };
#pragma unroll
        for (int k = 0; k < 4; ++k)
          add2(k * 8, mine[k].x), add2(k * 8 + 2, mine[k].y), add2(k * 8 + 4, mine[k].z), add2(k * 8 + 6, mine[k].w);
      };

      while (code == 0) {
        struct {
          int jlo, jhi, m0, shift, shift2, n_base, klen, qlen;
          int64_t bias_off;  // of the item's (batch, head) in the additive bias, in elements
        } it;
        const int idx = pop_item(seq, [&](const Item& d) {
          it.jlo = d.jlo[t], it.jhi = d.jhi[t];
          it.m0 = d.m0, it.shift = d.shift, it.shift2 = d.shift2, it.n_base = d.n_base, it.klen = d.klen, it.qlen = d.qlen;
          it.bias_off = kBias ? int64_t(d.b) * a.bias_b + int64_t(d.g) * a.bias_g + int64_t(d.h) * a.bias_h : 0;
        });
        if (idx < 0) {
          if (idx == -2) code = 30;
          break;
        }
        const int jlo = it.jlo, jhi = it.jhi;
        if (jhi <= jlo) continue;  // this tile sees no key in this item
        const int mt0 = it.m0 + t * tile_rows;
        const int i_loc = mt0 + (row >> pack_shift);
        const bool causal = a.window_right >= 0;
        col_hi = causal ? min(it.klen, i_loc + it.shift + a.window_right + 1) : it.klen;
        col_lo = a.window_left >= 0 ? i_loc + it.shift - a.window_left : 0;
        // m_run: the reference maximum the probabilities and O_t are taken against (log2 units; at most 2^8 below
        // the true running maximum); l_run: the row sum against m_run
        float m_run = -INFINITY, l_run = 0.f;

        XFB_PROF_LAP(0)  // between items: statistics hand-over, next descriptor
        for (int j = jlo; j < jhi; ++j, ++cnt) {
          int n0 = it.n_base + j * kBN;
          int klen = it.klen, shift = it.shift;
          if (a.kv_split > 0) {
            // which of the two key ranges this step lies in: positions and limits are relative to that range
            const bool second = n0 >= a.kv_split;
            klen = second ? it.klen - a.kv_split : a.kv_split;
            shift = second ? it.shift2 : it.shift;
            n0 -= second ? a.kv_split : 0;
            col_hi = min(klen, i_loc + shift + 1);
          }
          const bool need_mask = (n0 + kBN > klen) || (causal && n0 + kBN - 1 > mt0 + shift + a.window_right) ||
                                 (a.window_left >= 0 && n0 < mt0 + tile_rows - 1 + shift - a.window_left);
          uint4 bw[kBiasF32 ? 24 : kBias ? 16 : 1];
          bool whole = false;
          int rel_lo = 0, rel_hi = 0;  // visible keys of row r: from r + rel_lo, below r + rel_hi
          if constexpr (kBias) {
            // asked for before the wait for the scores, which hides most of their latency; the next step's are asked
            // into the L2 at the same time
            rel_lo = a.window_left >= 0 ? shift - a.window_left : -0x3fffffff;
            rel_hi = causal ? shift + a.window_right + 1 : 0x3fffffff;
            whole = a.bias_vec && !need_mask && mt0 + kBM <= it.qlen;
            bias_load(bw, std::integral_constant<int, kBiasF32 ? 6 : 4>{}, it.bias_off, mt0, it.qlen, n0, klen, rel_lo, rel_hi, whole);
            bias_prefetch(it.bias_off, mt0, it.qlen, n0 + kBN, j + 1 < jhi ? klen : 0);
          }
          if (!mbar_wait(&bar->s_full[t], cnt & 1, abort_flag, budget)) {
            code = 31 + t;
            break;
          }
          XFB_PROF_LAP(1)  // wait for the scores
          tc_fence_after();
          if (need_mask) {
            // Diagonal and ragged tiles: hidden scores are turned into -inf where they lie, in tensor memory, by this
            // small loop; the step itself then is the same code for every tile (one copy of it in the instruction
            // cache).  The rows of a warp are consecutive and both limits grow with the row, so the limits of the
            // first and the last row tell which chunks are fully visible to the warp (left alone) or fully hidden
            // (overwritten without being read).
            const int hi_first = __shfl_sync(0xffffffffu, col_hi, 0), hi_last = __shfl_sync(0xffffffffu, col_hi, 31);
            const int lo_first = __shfl_sync(0xffffffffu, col_lo, 0), lo_last = __shfl_sync(0xffffffffu, col_lo, 31);
            uint32_t sm[32], ninf[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) ninf[i] = 0xff800000u;
#pragma unroll 1
            for (int c = 0; c < kBN / 32; ++c) {
              const int col0 = n0 + c * 32;
              if (col0 >= lo_last && col0 + 32 <= hi_first) continue;  // every row of the warp sees the whole chunk
              if (col0 >= hi_last || col0 + 32 <= lo_first) {
                // no row of the warp sees any of it (the same eight registers serve every store: nothing to wait for)
#pragma unroll
                for (int i = 0; i < 4; ++i) XFB_TMEM_ST_8(tmem_s + c * 32 + i * 8, ninf);
              } else {
                tc_wait_st();  // (an earlier round's store may still be reading the registers)
                XFB_TMEM_LD_32(tmem_s + c * 32, sm);
                XFB_TMEM_WAIT_LD_32(sm);
                mask_chunk(reinterpret_cast<float*>(sm), col0);
                XFB_TMEM_ST_32(tmem_s + c * 32, sm);
              }
            }
            tc_wait_st();
            XFB_PROF_LAP(3)  // the visibility test
          }
          {
            // ---- the row's 128 scores come into registers, and the buffer is free for the next QK^T
            if constexpr (kBiasF32) {
              uint32_t sc[32];
#pragma unroll
              for (int c = 0; c < kBN / 32; ++c) {
                if (c > 0) tc_wait_st();  // (the store may still be reading the registers)
                XFB_TMEM_LD_32(tmem_s + c * 32, sc);
                XFB_TMEM_WAIT_LD_32(sc);
                bias_add(sc, bw + c % 3 * 8);
                XFB_TMEM_ST_32(tmem_s + c * 32, sc);
                if (c == 0) bias_load(bw, std::integral_constant<int, 2>{}, it.bias_off, mt0, it.qlen, n0 + 96, klen, rel_lo, rel_hi, whole);
              }
              tc_wait_st();
            }
            uint32_t s0[32], s1[32], s2[32], s3[32];
            XFB_TMEM_LD_32(tmem_s, s0);
            XFB_TMEM_LD_32(tmem_s + 32, s1);
            if constexpr (kBias && !kBiasF32) {
              XFB_TMEM_WAIT_LD_32(s0);
              XFB_TMEM_WAIT_LD_32(s1);
              bias_add(s0, bw);
              bias_add(s1, bw + 4);
            }
            XFB_TMEM_LD_32(tmem_s + 64, s2);
            XFB_TMEM_LD_32(tmem_s + 96, s3);
            XFB_TMEM_WAIT_LD_32(s0);
            XFB_TMEM_WAIT_LD_32(s1);
            XFB_TMEM_WAIT_LD_32(s2);
            XFB_TMEM_WAIT_LD_32(s3);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar->s_empty);
            if constexpr (kBias && !kBiasF32) {
              bias_add(s2, bw + 8);
              bias_add(s3, bw + 12);
            }
            XFB_PROF_LAP(5)  // scores read
            float mx = fmaxf(chunk_max(reinterpret_cast<float*>(s0)), chunk_max(reinterpret_cast<float*>(s1)));
            mx = fmaxf(mx, fmaxf(chunk_max(reinterpret_cast<float*>(s2)), chunk_max(reinterpret_cast<float*>(s3))));
            const float ms = mx * sl2;  // scale > 0 (host guarantees)
            XFB_PROF_LAP(8)  // their maximum
            // ---- the previous product of the tile has to be through: P_t is free again, O_t quiescent
            if (!mbar_wait(&bar->pv_done[t], (cnt & 1) ^ 1, abort_flag, budget)) {
              code = 35 + t;
              break;
            }
            tc_fence_after();
            XFB_PROF_LAP(7)  // wait for the previous product
            // ---- the reference follows the maximum only when it has to (a fresh row: from -inf)
            if (__any_sync(0xffffffffu, ms > m_run + kRescaleThreshold)) {
              const float m_new = ms > m_run + kRescaleThreshold ? ms : m_run;
              const float alpha = m_new == m_run ? 1.f : (m_run == -INFINITY ? 0.f : fast_exp2(m_run - m_new));
              if (j > jlo) rescale_o(alpha);
              l_run *= alpha;
              m_run = m_new;
            }
            // ---- probabilities
            const float m_use = m_run == -INFINITY ? 0.f : m_run;
            const uint64_t nm2 = f2_pack(-m_use, -m_use);
            uint64_t sum2[4] = {f2_pack(0.f, 0.f), f2_pack(0.f, 0.f), f2_pack(0.f, 0.f), f2_pack(0.f, 0.f)};
            exp_store(s0, 0, nm2, sum2);
            exp_store(s1, 16, nm2, sum2);
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar->p_half[t]);
            XFB_PROF_LAP(2)  // first half of the probabilities
            exp_store(s2, 32, nm2, sum2);
            exp_store(s3, 48, nm2, sum2);
            {
              float x0, x1, y0, y1;
              f2_unpack(fadd2(sum2[0], sum2[1]), x0, x1);
              f2_unpack(fadd2(sum2[2], sum2[3]), y0, y1);
              l_run += (x0 + x1) + (y0 + y1);
            }
          }
          XFB_PROF_COUNT(6)
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar->p_full[t]);
          XFB_PROF_LAP(4)  // second half
        }
        if (code != 0) break;
        // hand the row's statistics to the output warps
        if (!mbar_wait(&bar->stats_empty[t], (ka++ & 1) ^ 1, abort_flag, budget)) {
          code = 33 + t;
          break;
        }
        stats[t * kBM + row] = make_float2(m_run, l_run);
        mbar_arrive(&bar->stats_full[t]);
      }
      if (code != 0) {
        give_up(a, code);
        *abort_flag = 1;
      }
      tc_fence_before();
      XFB_PROF_STORE(warp * 16, 16)
    }

    __syncthreads();
    if (warp == kQkWarp) {
      tc_fence_after();
      tmem_dealloc(tmem, 512);
    }
  }

  // The last CTA to finish puts the work counters back to zero for the next launch.
  if (threadIdx.x == 0) {
    __threadfence();
    const int done = atomicAdd(a.counters + 1, 1);
    if (done == int(gridDim.x) - 1) {
      atomicExch(a.counters, 0);
      atomicExch(a.counters + 1, 0);
    }
  }
}

template <int D, bool kBf16, int kVariant>
static int launch_t(Sm100Args a, cudaStream_t stream) {
  auto kern = prefill_sm100_persist_kernel<D, kBf16, kVariant>;
  constexpr int smem = kVariant >= kBiasedSame ? Smem<D>::kTotalBiased : Smem<D>::kTotal;
  static_assert(smem <= 227 * 1024, "shared memory of one CTA");
  static bool configured[kMaxDevices] = {false};  // the attribute belongs to the device's context
  if (first_use_on_device(configured)) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return cuda_fail("prefill(sm100, persistent): cudaFuncSetAttribute", e);
  }
  const int64_t items = ((int64_t(a.groups) * a.heads_per_group) >> a.pack_shift) * a.batch * a.q_tiles;
  if (items > 0x3fffffff) return set_error(XFB200_E_UNSUPPORTED, "prefill: too many blocks of query rows");
  a.n_items = int32_t(items);
  int sms = sm_count() - a.sm_margin;
  if (sms < 1) sms = 1;
  const unsigned grid = unsigned(items < sms ? items : sms);
  if (a.sm_margin > 0) {  // the free SMs are for others from its first CTA to its last
    kern<<<grid, kThreads, smem, stream>>>(a);
    return check_launch("prefill_sm100_persist_kernel");
  }
  const cudaError_t e = launch_early(kern, grid, kThreads, smem, stream, a);
  return e != cudaSuccess ? cuda_fail("prefill_sm100_persist_kernel launch", e) : XFB200_OK;
}

}  // namespace pst

#ifdef XFB_PST_PROFILE
extern "C" __attribute__((visibility("default"))) int xfb200_debug_read_prefill_profile(long long* out, int clear) {
  cudaDeviceSynchronize();
  cudaError_t e = cudaMemcpyFromSymbol(out, pst::g_prof, sizeof(long long) * 160 * 160);
  if (e == cudaSuccess && clear) {
    static long long zeros[160 * 160] = {0};
    e = cudaMemcpyToSymbol(pst::g_prof, zeros, sizeof(zeros));
  }
  return e == cudaSuccess ? 0 : -3;
}
#endif

template <int D, int kVariant>
static int persist_launch_d(const Sm100Args& a, bool bf16, cudaStream_t stream) {
  return bf16 ? pst::launch_t<D, true, kVariant>(a, stream) : pst::launch_t<D, false, kVariant>(a, stream);
}

int prefill_sm100_persist_launch(Sm100Args a, int head_dim, bool bf16, cudaStream_t stream) {
  if (a.bias != nullptr && a.bias_dtype == XFB200_F32)
    return head_dim > 64 ? persist_launch_d<128, pst::kBiasedF32>(a, bf16, stream) : persist_launch_d<64, pst::kBiasedF32>(a, bf16, stream);
  if (a.bias != nullptr && a.bias_dtype == (bf16 ? XFB200_F16 : XFB200_BF16))
    return head_dim > 64 ? persist_launch_d<128, pst::kBiasedOther>(a, bf16, stream) : persist_launch_d<64, pst::kBiasedOther>(a, bf16, stream);
  if (a.bias != nullptr) return head_dim > 64 ? persist_launch_d<128, pst::kBiasedSame>(a, bf16, stream) : persist_launch_d<64, pst::kBiasedSame>(a, bf16, stream);
  if (head_dim > 128) return head_dim == 256 ? persist_launch_d<256, pst::kExact>(a, bf16, stream) : persist_launch_d<256, pst::kPadded>(a, bf16, stream);
  if (head_dim == 128) return persist_launch_d<128, pst::kExact>(a, bf16, stream);
  if (head_dim == 64) return persist_launch_d<64, pst::kExact>(a, bf16, stream);
  return head_dim > 64 ? persist_launch_d<128, pst::kPadded>(a, bf16, stream) : persist_launch_d<64, pst::kPadded>(a, bf16, stream);
}

}  // namespace xfb
