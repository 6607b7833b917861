// Persistent, warp-specialised, mbarrier-pipelined LoRA shrink / expand kernels (the fast path).
//
// Two CTAs per SM (a grid of 2 x SM count) walk their share of the work items (item i belongs to CTA i mod gridDim.x).
// Two producer warps feed a ring of shared-memory stages with bulk asynchronous copies (cp.async.bulk + mbarrier
// complete_tx): the lanes of the first resolve 32 upcoming items in parallel (tile record -> table entries -> pool rows
// and token ids), then both run the same deterministic allocation, the first copying adapter rows and the second
// activations (after a CTA's first stages also some of the rows).  Eight consumer warps wait on a stage's "full" barrier,
// do the arithmetic (mma.sync, lora_warp_mma.cuh) and release the stage through its "empty" barrier.  Consumer warps
// never wait for each other (shrink: each warp owns a K-slice and the last warp to finish an item, elected by an atomic
// counter, adds the partial sums; expand: each warp owns a 2048-element span of the B chunk).  Every wait is an mbarrier
// wait with a time limit, but for the meetings of the two producers, each of which only has such waits in between.
//
// What bounds a launch (measured on B200, clock64 around the phases of every warp): a stage's round trip - a consumer's
// release, the producers' reaction, the copies' issue, memory, the consumers - with two or three stages of 34 to 49 KB
// per CTA in flight.  What it is made of, and what was done about it:
// * A bulk copy's operands are uniform registers: a warp issues its lanes' copies one after the other, 52 cycles each with
//   the SM to itself and 75 to 140 beside working consumers.  So copies are few and large (one per pool row that a B
//   chunk touches, not one per power-of-two piece: 18 -> 6 copies a stage at row stride 5120) and two warps issue.
// * Divisions: a 64-bit one costs hundreds of cycles, and a stage had five.  The producers use FastDiv and shifts: the
//   expand's producer time per stage 3300 -> 1900 cycles (q,k,v expand of the 13B-shaped batch 83.8 -> 69.2 us).
// * Consumers on the tensor pipe: a stage of eight tokens at rank 64 took 3150 cycles of FMA and shuffles, now 1750
//   (q,k,v expand of the 70B-shaped batch 77.6 -> 55.1 us); the shrink's accumulators became one C fragment whatever the
//   item's size, so that an item can have sixteen rows and its tokens are staged a quarter as often (208 -> 106 us).
// * Copies per worker warp with cp.async instead (every consumer its own ring of 4 KB stages, no producers) were correct
//   and slower, 343 against 216 us per layer of the 13B-shaped batch: the addresses of 16-byte copies and the ring's
//   bookkeeping are then paid per 4 KB.
//
// Programmatic dependent launch: the first producer copies the adapter rows of the first stages (rows that no kernel on
// the stream writes) before griddepcontrol.wait; the second waits for the grid right before its first activation copy.
// Two CTAs fit on an SM: in steady state both belong to the running kernel, and as CTAs of the running kernel retire the
// next kernel's CTAs take their place and run their prologue under this kernel's tail.
//
// Shrink stage  = one item (tile, projection, block of 4, 8 or 16 rows), or a K-chunk of it when the item exceeds
//                 kMaxStageBytes: [adapter-row chunks][token-row chunks]; sums stay in registers across the chunks.
// Expand stage  = one item (tile, projection, 16384-element chunk of B): [B chunk][n y segments][n delta rows].
//                 y is read through the stage and written back with plain vector stores.
#pragma once

#include "lora_common.cuh"
#include "lora_warp_mma.cuh"

namespace slora {

constexpr int kSlots = 8;  // stage descriptors (barrier pairs) in flight
#ifndef SLORA_RING_KB
#define SLORA_RING_KB 96
#endif
#ifndef SLORA_STAGE_KB
#define SLORA_STAGE_KB 49
#endif
#ifndef SLORA_SHRINK_RING_KB
#define SLORA_SHRINK_RING_KB 98
#endif
// ring + control block (+ the shrink's reduction buffers) stay below half an SM's shared memory
constexpr int kRingBytes = SLORA_RING_KB * 1024;
constexpr int kShrinkRingBytes = SLORA_SHRINK_RING_KB * 1024;
#ifndef SLORA_EXPAND_RING_KB
#define SLORA_EXPAND_RING_KB 104
#endif
// The expand's control block is 8 KB smaller (no reduction buffers): with 104 KB three of its ~34 KB stages (a B chunk
// and one token's y segment and delta row) are in flight instead of two.  Used by the EXACT instantiation (q,k,v expand
// of the 13B-shaped batch 74.3 us with 96 KB, 72.6 with 104).  The padded one was given 96 KB when its consumers were
// FMA loops and short launches 2 % slower with 104; with the present ones 104 would be the better size there too (rank-8
// decode batch 9.3 -> 9.1 us, 77 tokens of mixed ranks 11.9 -> 11.3, 70B-shaped batch 55.4 -> 53.5).
constexpr int kExpandRingBytes = SLORA_EXPAND_RING_KB * 1024;
constexpr int kPipeCtasPerSm = 2;      // persistent CTAs per SM
// Producer warps: the first resolves items and copies adapter rows, the second copies activations.
constexpr int kProducerWarps = 2;
constexpr int kRowsAhead = 3;  // a CTA's first stages: all their adapter rows are the first producer's
constexpr int kConsumerWarps = 8;
constexpr int kPipeThreads = 32 * (kProducerWarps + kConsumerWarps);
constexpr int kMaxStageBytes = SLORA_STAGE_KB * 1024;  // a shrink item is cut into K-chunks no larger than this
constexpr int kPipeChunk = 16384;          // flat B elements per expand item (32 KB)
constexpr int kSpanRows = 6;    // pool rows a B chunk may touch: one copy each (lanes 0..5); y copies use lanes
                                // 16..23, delta rows 24..31
constexpr int kItemRows = 16;   // widest shrink item: adapter rows (ShrinkArgs::rows_per_cta picks 4, 8 or 16)
constexpr int kActLane = 16;    // lanes kActLane.. carry a stage's activation copies
constexpr int kCompactTiles = 640;  // tiles whose item counts fit the control block (two CTAs per SM leave little room)

constexpr int FLAG_FIRST = 1, FLAG_LAST = 2, FLAG_END = 4;
constexpr uint32_t FULL_MASK = 0xffffffffu;
constexpr long long kWaitCycles = 400000000ll;  // about 0.2 s of SM clock: far beyond any legitimate wait here

// Wait for a barrier phase for a bounded time (SM cycle counter); false on timeout.
__device__ __forceinline__ bool mbar_wait_timed(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 1024; ++i) {
      if (mbar_try_wait(bar, parity)) return true;
    }
    if (clock64() - t0 > kWaitCycles) return false;
  }
}

// Shared-memory control block of one pipeline.
struct PipeCtl {
  uint64_t full[kSlots];
  uint64_t empty[kSlots];
  int meta[kSlots][16];
  // the 32 items a batch resolves, one per lane of the first producer warp, parked here for the lanes that carry the
  // copies: pool rows and the item's description
  int32_t d_l[32][kItemRows];
  int d_i[32][16];
  uint32_t valid_mask;
  // planned batches of mixed ranks: items up to and including each tile (see build_item_map)
  uint16_t item_end[kCompactTiles];
  int tp_gave_up;  // in-band signalling: a wait for another rank's values ran out; nobody in this CTA waits again
};

// Shrink only: per-item partial sums of the consumer warps and the arrival counter that elects the last warp.  (Kept
// out of PipeCtl so that the expand, which has no use for it, can give those 8 KB to its ring.)
// Rows of a C fragment: half h holds rows 8h + lane / 4, tokens 2 (lane % 4) and the next; four, eight or sixteen rows
// are a half fragment (the lanes below 16), one or two.  8 KB hold the shrink_buffers() of a launch.
struct ShrinkRed {
  float2 sum[4 * kConsumerWarps * 32];
  int cnt[kSlots];
};

// Producer-side ring state (identical in all 32 lanes, but for `off`).
struct Ring {
  int role = 0;       // which producer warp this is
  uint32_t g = 0;     // next stage index
  uint32_t tail = 0;  // oldest stage not yet known to be released
  uint32_t head = 0;  // next free byte
  uint32_t off = 0;   // lane s: byte offset of the stage in slot s
  bool pre = true;    // still before the grid-dependency wait
  bool dead = false;  // a bounded wait ran out
  uint32_t cap = kRingBytes;  // bytes of the ring
  uint32_t slots = kSlots;    // stages in flight at most
  const TpLink* tp = nullptr;  // expand under tensor parallelism: flags to wait for before activations are read
  int32_t* status = nullptr;
  bool trigger_after_wait = false;  // shrink whose expand starts early: dependents may launch once this has waited
};

constexpr long long kTpLinkWaitCycles = 4000000000ll;  // about 2 s: ranks drift by host-side jitter, not more

// Expand side of the tensor-parallel link: lanes 0..n_parts-1 wait until every rank's columns of this exchange have
// landed in this rank's delta buffer.  Bounded; false when the wait ran out.
__device__ __forceinline__ bool tp_link_wait(const TpLink& tp, int lane) {
  bool seen = true;
  if (lane < tp.n_parts) {
    const int seq = tp.seq_state[tp.half] + 1;
    const int32_t* flag = tp.flags[tp.my_part] + tp.half * tp.n_parts + lane;
    const long long t0 = clock64();
    seen = false;
    while (!seen) {
      int v;
      asm volatile("ld.acquire.sys.global.b32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
      seen = v >= seq;
      if (!seen && clock64() - t0 > kTpLinkWaitCycles) break;
    }
  }
  return __all_sync(0xffffffffu, seen);
}

// End of a linked launch (whole-launch flags): the last CTA to get here either raises this rank's flag on every rank
// (shrink: all its columns have been written and fenced) or counts the exchange as done (expand: every CTA has read
// its number).  One system-scope fence per CTA, by the thread that then bumps the arrival counter: the CTA barrier
// before it orders every thread's stores before that fence, and a fence is cumulative.  (A fence by each of the CTA's
// threads, as this was first written, serialises in the memory system: measured, it cost more than the exchange
// itself.)  The expand's bookkeeping stays on this GPU and needs no system-scope fence at all.
__device__ __forceinline__ void tp_link_finish(const TpLink& tp, bool is_shrink) {
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    if (is_shrink) {
      __threadfence_system();
    } else {
      __threadfence();
    }
    s_last = atomicAdd(tp.counter, 1) == static_cast<int>(gridDim.x) - 1;
  }
  __syncthreads();
  if (!s_last) return;
  const int seq = tp.seq_state[tp.half] + 1;
  if (threadIdx.x == 0) {
    *tp.counter = 0;
    __threadfence();  // the other CTAs' arrivals (device-scope atomics) before what follows
  }
  __syncthreads();
  if (is_shrink) {
    if (static_cast<int>(threadIdx.x) < tp.n_parts) {
      asm volatile("st.release.sys.global.b32 [%0], %1;" ::"l"(tp.flags[threadIdx.x] + tp.half * tp.n_parts + tp.my_part),
                   "r"(seq)
                   : "memory");
    }
  } else if (threadIdx.x == 0) {
    tp.seq_state[tp.half] = seq;
  }
}

// ---- in-band signalling (TpLink::inband) ------------------------------------------------------------------------
// No flag and no fence at all: the delta buffers start out filled with a bit pattern no result can have (kTpEmpty: a
// NaN that the float-to-16-bit conversion never produces), the shrink stores its results into every rank's buffer
// with plain stores, and the expand checks the delta values themselves: a consumer lane that finds the pattern among
// the eight values it is about to use re-reads them from global memory until they have arrived (bounded).  Each
// 16-bit element is written by one store, so checking every element that is used is enough - no ordering between
// elements is needed.  The last CTA of the expand refills the half it consumed; no rank can write that half again
// before this rank has finished its next exchange on the other half, which starts after this kernel.
constexpr uint32_t kTpEmpty2 = 0xffffffffu;  // two elements of the pattern 0xffff
__device__ __forceinline__ bool tp_has_empty(const uint4& v) {
  // (bitwise ors: no short-circuit branches)
  auto e = [](uint32_t w) { return ((w & 0xffffu) == 0xffffu) | ((w >> 16) == 0xffffu); };
  return (e(v.x) | e(v.y) | e(v.z) | e(v.w)) != 0;
}
// Eight delta values from global memory, polled until none is the empty pattern; false when the wait ran out.
__device__ __forceinline__ bool tp_poll_delta(const void* src, uint4& v, volatile int* gave_up) {
  const long long t0 = clock64();
  for (;;) {
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(src)
                 : "memory");
    if (!tp_has_empty(v)) return true;
    if (*gave_up != 0) return false;
    if (clock64() - t0 > kTpLinkWaitCycles) {
      *gave_up = 1;
      return false;
    }
  }
}
// End of an expand with in-band signalling: the last CTA refills the consumed half with the empty pattern.  No fence
// before the arrival: what has to precede the refill is the other CTAs' LOADS of the values, and a load has
// returned its value before the code that follows it (the arrival) runs.
__device__ __forceinline__ void tp_inband_finish(const TpLink& tp, void* half_base, int64_t bytes) {
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(tp.counter, 1) == static_cast<int>(gridDim.x) - 1;
  __syncthreads();
  if (!s_last) return;
  uint4* p = reinterpret_cast<uint4*>(half_base);
  const uint4 e = make_uint4(kTpEmpty2, kTpEmpty2, kTpEmpty2, kTpEmpty2);
  const int64_t n16 = bytes / 16, nthr = blockDim.x;
  int64_t i = threadIdx.x;
  for (; i + 3 * nthr < n16; i += 4 * nthr) {  // four independent stores per thread and round
    p[i] = e;
    p[i + nthr] = e;
    p[i + 2 * nthr] = e;
    p[i + 3 * nthr] = e;
  }
  for (; i < n16; i += nthr) p[i] = e;
  if (threadIdx.x == 0) *tp.counter = 0;
}

// The grid-dependency wait of a producer warp.  The one that copies activations does it before its first copy (and, under
// tensor parallelism with flags, waits for the other ranks' there); the one that copies adapter rows, which no kernel
// on the stream writes, only before it first waits for ring space.
__device__ __forceinline__ void ring_enter(Ring& r, int lane) {
  if (!r.pre) return;
  r.pre = false;
  pdl_wait();
  if (r.trigger_after_wait) pdl_launch_dependents();
  if (r.role != 0 && r.tp != nullptr && !r.tp->inband && !tp_link_wait(*r.tp, lane)) {
    // the copies still go out (the consumers' barriers expect them); the result is flagged as not to be trusted
    if (lane == 0) set_status(r.status, SLORA_STATUS_TIMEOUT);
  }
}

// Where `sz` bytes go in a ring of `cap` bytes whose next free byte is `head` and whose oldest stage in use starts at
// `oldest` (`empty`: none is in use).
__host__ __device__ __forceinline__ bool ring_fits(uint32_t head, bool empty, uint32_t oldest, uint32_t cap, uint32_t sz,
                                                   uint32_t& at) {
  at = 0;
  if (empty) return true;
  if (head <= oldest) {  // wrapped
    at = head;
    return head + sz <= oldest && head != oldest;
  }
  if (head + sz > cap) return sz <= oldest;
  at = head;
  return true;
}

// Reserve `sz` bytes (a multiple of 128) and a descriptor for stage r.g, once all stages before `released` have been
// released; returns the byte offset, or 0xffffffff when a wait ran out.  The lanes poll the barriers one by one, so every
// turn of the loop brings them together again: each issues copies of its own, and a lane that saw another stage's offset
// would send its copy into a stage in use.  What they share of earlier stages therefore goes through shuffles and votes,
// not through shared memory.
__device__ __forceinline__ uint32_t ring_alloc(Ring& r, PipeCtl& c, uint32_t sz, int lane, uint32_t released = 0) {
  for (;;) {
    uint32_t cand;
    const uint32_t oldest = __shfl_sync(FULL_MASK, r.off, r.tail % kSlots);
    const bool ok = ring_fits(r.head, r.tail == r.g, oldest, r.cap, sz, cand);
    if (ok && r.g - r.tail < r.slots && static_cast<int32_t>(r.tail - released) >= 0) {
      r.head = cand + sz;
      if (lane == static_cast<int>(r.g % kSlots)) r.off = cand;
      return cand;
    }
    ring_enter(r, lane);
    if (!__all_sync(FULL_MASK, mbar_wait_timed(&c.empty[r.tail % kSlots], (r.tail / kSlots) & 1))) {
      r.dead = true;
      return 0xffffffffu;
    }
    ++r.tail;
  }
}

// The copies of a stage: lane `lane` carries (dst, src, bytes) or bytes == 0.  A bulk copy's operands are uniform
// registers, so a warp issues its lanes' copies one after the other (measured on B200: 52 cycles a copy with the SM to
// itself, 75 to 140 beside working consumers), while two warps issue side by side: each producer warp works out the same
// stages and calls this for its share of the lanes.  The stage's byte count is announced by one arrival (the first
// warp's); copies of the other warp may complete before it.
__device__ __forceinline__ void ring_issue(Ring& r, PipeCtl& c, uint32_t slot, uint32_t dst, const void* src,
                                           uint32_t bytes) {
  if (bytes != 0) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(&c.full[slot]))
                 : "memory");
  }
  ++r.g;
}

// The producer warps meet: before a batch of items is resolved (all of them are done with the previous one) and after.
__device__ __forceinline__ void producers_sync() {
  __syncwarp();  // (a barrier of whole warps)
  asm volatile("bar.sync 1, %0;" ::"n"(kProducerWarps * 32) : "memory");
}

// Finish: flush a prologue that never ended, then post the end marker.
__device__ __forceinline__ void ring_finish(Ring& r, PipeCtl& c, int32_t* status, int lane) {
  ring_enter(r, lane);
  if (!r.dead) ring_alloc(r, c, 0, lane);
  if (r.dead) {
    if (lane == 0) set_status(status, SLORA_STATUS_TIMEOUT);
    return;
  }
  const uint32_t slot = r.g % kSlots;
  if (lane == 0 && r.role == 0) {
    c.meta[slot][0] = FLAG_END;
    mbar_arrive(&c.full[slot]);
  }
}

__device__ __forceinline__ void pipe_init(PipeCtl& c, int tid) {
  if (tid == 0) {
    c.tp_gave_up = 0;
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(&c.full[s], 1);
      mbar_init(&c.empty[s], kConsumerWarps);
    }
    fence_barrier_init();
    fence_proxy_async();
  }
  __syncthreads();
}

template <typename P>
__device__ __forceinline__ P pick3(P const (&arr)[3], int p) {
  return p == 0 ? arr[0] : (p == 1 ? arr[1] : arr[2]);
}

__host__ __device__ __forceinline__ uint32_t round128(uint32_t v) { return (v + 127u) & ~127u; }

// ------------------------------------------------------------------------------------------------------------
// Which items does a launch have?  A tile yields a number of items that depends on its adapter's rank (row blocks
// of the shrink, B chunks of the expand).  Enumerating a fixed number of slots per tile, sized for the widest rank,
// and skipping the empty ones leaves the CTAs (item i belongs to CTA i mod gridDim.x) with unequal shares as soon
// as ranks differ - the empty slots recur with the period of the slot grid.  With a plan the items are therefore
// counted exactly: in closed form when every tile has the same rank (the plan's header says so), else through a
// per-tile running count that the CTA builds in shared memory from the tile records (all threads fetch the
// records, the first producer warp scans the counts; before the grid-dependency wait: the plan is complete by then).
// Without a plan, or with more tiles or items than the control block holds, the padded enumeration stays.  The exact
// count costs the start of a launch a few hundred nanoseconds (its arithmetic sits between the header and the first
// tile record), which a launch of ten microseconds over same-rank adapters does not earn back: the kernels are
// therefore built both ways (EXACT) and the caller, who can ask the plan what it holds (slora_plan_info), picks with
// SLORA_FLAG_EXACT_ITEMS.
// ------------------------------------------------------------------------------------------------------------
struct ItemMap {
  int mode = 0;      // 0 padded slots, 1 same count for every tile, 2 running count in PipeCtl::item_end
  int per_tile = 0;  // modes 0 and 1
  int uniform = 0;   // mode 1: the slot rows of every tile
  int n_tiles = 0;
  int64_t n_items = 0;
};

// Does this launch count its items per tile (ranks differ, or big groups go elsewhere), and over how many tiles?
__device__ __forceinline__ bool needs_item_counts(const TileSrc& src, int& n_tiles, int& uniform) {
  // the three header words in one go: their loads are on the launch's critical path
  const int32_t* hdr = src.plan;
  const int nt = hdr[PH_NTILES], uni = hdr[PH_UNIFORM], nbig = hdr[PH_NBIG];
  n_tiles = min(nt, src.slots);
  uniform = uni;
  const bool some_elsewhere = src.seg_split > 0 && nbig > 0;  // big groups the tensor-core launch serves
  return !(uni > 0 && !some_elsewhere);
}

// All threads of the CTA: items of every tile into PipeCtl::item_end (one tile record per thread and round, so the
// loads overlap); the caller follows with __syncthreads().
template <typename F>
__device__ __forceinline__ void fill_item_counts(const TileSrc& src, const Tables& tb, PipeCtl& c, int tid,
                                                 F items_of_rank) {
  if (src.mode != MODE_PLAN) return;
  int n_tiles, uniform;
  if (!needs_item_counts(src, n_tiles, uniform) || n_tiles > kCompactTiles) return;
  for (int tile = tid; tile < n_tiles; tile += kPipeThreads) {
    const int4* rec = reinterpret_cast<const int4*>(src.plan + PH_WORDS + kTileWords * tile);
    const int4 r0 = rec[0];
    const int n = r0.z, r = r0.w;
    bool elsewhere = false;
    if (src.seg_split > 0) elsewhere = rec[1].y != 0 && r > 0 && tb.pool_stride % r == 0 && r <= src.mma_max_rows;
    const int cnt = (n > 0 && r > 0 && !elsewhere) ? items_of_rank(r, n) : 0;
    c.item_end[tile] = static_cast<uint16_t>(min(cnt, 0xffff));
  }
}

// Producer warp, after fill_item_counts and the barrier: the launch's item map; with mixed ranks the counts in
// item_end become running counts (each lane sums a contiguous run, the warp scans the lane sums).
template <typename F>
__device__ __forceinline__ ItemMap build_item_map(const TileSrc& src, int padded_per_tile, PipeCtl& c, int lane,
                                                  int role, F items_of_rank) {
  ItemMap m;
  m.per_tile = padded_per_tile;
  if (src.mode != MODE_PLAN) {
    m.n_tiles = src.slots;
    m.n_items = static_cast<int64_t>(m.n_tiles) * padded_per_tile;
    return m;
  }
  int uniform;
  const bool counted = needs_item_counts(src, m.n_tiles, uniform);
  m.n_items = static_cast<int64_t>(m.n_tiles) * padded_per_tile;
  if (!counted) {
    m.mode = 1;
    m.uniform = uniform;
    m.per_tile = items_of_rank(uniform, kTileTokens);
    m.n_items = static_cast<int64_t>(m.n_tiles) * m.per_tile;
    return m;
  }
  if (m.n_tiles > kCompactTiles) return m;
  const int per = (m.n_tiles + 31) / 32;
  const int lo = min(lane * per, m.n_tiles), hi = min(lo + per, m.n_tiles);
  int sum = 0;
  for (int i = lo; i < hi; ++i) sum += c.item_end[i];
  int incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(FULL_MASK, incl, d);
    if (lane >= d) incl += v;
  }
  const int total = __shfl_sync(FULL_MASK, incl, 31);
  if (total > 0xffff) return m;  // too many items for 16-bit counts (same decision in every lane)
  producers_sync();  // every producer warp has read the counts; one of them turns them into running counts
  if (role == 0) {
    int run = incl - sum;
    for (int i = lo; i < hi; ++i) {
      run += c.item_end[i];
      c.item_end[i] = static_cast<uint16_t>(run);
    }
  }
  __syncwarp();  // (only the first producer warp looks items up)
  m.mode = 2;
  m.n_items = total;
  return m;
}

// The padded enumeration alone.  Nothing is read from the plan here: the first batch of items is bounded by the tile
// slots the workspace has (tile_lookup tells which of them hold tiles), so that its loads do not queue behind a
// load of the tile count; later batches use the count (padded_item_count), which has arrived by then.
__device__ __forceinline__ ItemMap padded_item_map(const TileSrc& src, int padded_per_tile) {
  ItemMap m;
  m.per_tile = padded_per_tile;
  m.n_tiles = src.slots;
  m.n_items = static_cast<int64_t>(m.n_tiles) * padded_per_tile;
  return m;
}
__device__ __forceinline__ int64_t padded_item_count(const TileSrc& src, int padded_per_tile) {
  return static_cast<int64_t>(tile_count(src)) * padded_per_tile;
}

// Item q -> its tile and its index among that tile's items.
__device__ __forceinline__ void item_to_tile(const ItemMap& m, const FastDiv& padded, const PipeCtl& c, int64_t q,
                                             int& tile, int& local) {
  if (m.mode != 2) {
    if (q < 0x7fffffff) {
      const uint32_t q32 = static_cast<uint32_t>(q);
      tile = m.mode == 0 ? padded.div(static_cast<int>(q32)) : static_cast<int>(q32 / static_cast<uint32_t>(m.per_tile));
    } else {
      tile = static_cast<int>(q / m.per_tile);
    }
    local = static_cast<int>(q - static_cast<int64_t>(tile) * m.per_tile);
    return;
  }
  int lo = 0, hi = m.n_tiles - 1;  // first tile whose running count exceeds q
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (static_cast<int64_t>(c.item_end[mid]) > q) {
      hi = mid;
    } else {
      lo = mid + 1;
    }
  }
  tile = lo;
  local = static_cast<int>(q) - (lo > 0 ? c.item_end[lo - 1] : 0);
}

// ------------------------------------------------------------------------------------------------------------
// shrink
// stage meta: [0] flags [1] nrows [2] n [3] j0 [4] projection [5] klen [6] ring offset, [8..15] token ids
// stage bytes: nrows chunks of klen elements (adapter rows), then n chunks of klen elements (token rows)
// ------------------------------------------------------------------------------------------------------------
// Row blocks a tile of rr slot rows has per projection (rows beyond the delta buffers' width are not enumerated).
__device__ __forceinline__ int shrink_rows_of(const ShrinkArgs& a, int rr) {
  return min(rr * a.rank_mult, a.max_rb * a.rows_per_cta);
}
__device__ __forceinline__ int shrink_blocks_of(const ShrinkArgs& a, int rr) {
  return (shrink_rows_of(a, rr) + a.rows_per_cta - 1) >> (31 - __clz(a.rows_per_cta));  // 4, 8 or 16
}
__device__ __forceinline__ int shrink_items_of(const ShrinkArgs& a, int rr) { return a.nproj * shrink_blocks_of(a, rr); }

// Item `rem` of a tile's nb items per projection: which projection (the last one takes what is beyond: its row block
// is then past the adapter's rows).
__device__ __forceinline__ int proj_of(int rem, int nb, int nproj) {
  return min((rem >= nb ? 1 : 0) + (rem >= 2 * nb ? 1 : 0), nproj - 1);
}

// Chunk j of a stage starts (j + 1) / 2 * kChunkPad bytes after j chunks' values: two rows that lie next to each other
// start in different halves of the banks, so that the eight lanes that read 64 bytes of each do not collide.
constexpr int kChunkPad = 64;
__host__ __device__ __forceinline__ int chunk_at(int j, int bytes) { return j * bytes + ((j + 1) >> 1) * kChunkPad; }
// K elements of a shrink stage of `chunks` rows and tokens, in pairs of units of kKUnit: what fits kMaxStageBytes, at
// least one pair.
constexpr int kKUnit = 512;
constexpr int stage_pairs(int c) {
  const int p = (kMaxStageBytes - 64 - (c + 1) / 2 * kChunkPad) / (c * kKUnit * 4);
  return p < 1 ? 1 : (p > 255 ? 255 : p);
}
struct StagePairs {
  uint64_t w[3];  // a byte per number of chunks (1..24)
};
constexpr StagePairs stage_pairs_table() {
  StagePairs s = {{0, 0, 0}};
  for (int c = 1; c <= 24; ++c) s.w[(c - 1) / 8] |= static_cast<uint64_t>(stage_pairs(c)) << (8 * ((c - 1) % 8));
  return s;
}
constexpr uint64_t kPairs0 = stage_pairs_table().w[0], kPairs1 = stage_pairs_table().w[1],
                   kPairs2 = stage_pairs_table().w[2];
__host__ __device__ __forceinline__ int stage_k(int chunks) {
  const int i = chunks - 1;
  const uint64_t w = i < 8 ? kPairs0 : (i < 16 ? kPairs1 : kPairs2);
  return static_cast<int>((w >> (8 * (i & 7))) & 255u) * (2 * kKUnit);
}
// Reduction buffers of a launch: items whose last stage may be in flight at once.  Item i sums in buffer i mod
// buffers, so its last stage goes out only when item i - buffers has been released.  Up to eight rows there are as many
// buffers as stages may be in flight, which is all it takes.  Items of sixteen rows have two (4 KB each): how many stages
// an item has depends on its rows and tokens (eight rows and a token are one up to 2048 elements, two rows up to 8192),
// so the producers count items and not stages, and the ring's bytes bound the stages.  (At hidden 256 to 1024 the ring
// would hold more than the four stages of items of eight rows; q,k,v launches of such items and of taller ones take 0.31
// to 0.85 of the time of FMA consumers with eight stages of four rows there.)
__host__ __device__ __forceinline__ uint32_t shrink_buffers(int rows_per_item) {
  return rows_per_item > 8 ? 2 : (rows_per_item > 4 ? 4 : 8);
}
__host__ __device__ __forceinline__ uint32_t shrink_slots(int rows_per_item) {
  return rows_per_item > 8 ? kSlots : shrink_buffers(rows_per_item);
}
// The ends of the two items before the current one, as the number of stages up to there.
struct ItemEnds {
  uint32_t previous = 0, before = 0;
  // The stages that have to be released before the next one goes out.
  __host__ __device__ __forceinline__ uint32_t released(bool item_ends, int rows_per_item) const {
    return item_ends && rows_per_item > 8 ? before : 0;
  }
  __host__ __device__ __forceinline__ void end_item(uint32_t stages) {
    before = previous;
    previous = stages;
  }
};

template <typename T, bool EXACT>
__device__ __forceinline__ void shrink_producer(const ShrinkArgs& a, unsigned char* ring_mem, PipeCtl& c, int lane,
                                                int role) {
  const int h_in = a.h_in;
  const int64_t S = a.tb.pool_stride;
  const T* w = reinterpret_cast<const T*>(a.w);
  const T* x = reinterpret_cast<const T*>(a.x);
  const int64_t G = gridDim.x;
  const uint32_t ring_base = smem_u32(ring_mem);
  const int RB = a.rows_per_cta;
  Ring r;
  r.role = role;
  r.cap = kShrinkRingBytes;
  r.slots = shrink_slots(RB);
  ItemEnds ends;
  r.trigger_after_wait = a.tp.enabled && a.tp.inband >= 2;
  const ItemMap map = EXACT ? build_item_map(a.src, a.nproj * a.max_rb, c, lane, role,
                                             [&](int rr, int) { return shrink_items_of(a, rr); })
                            : padded_item_map(a.src, a.nproj * a.max_rb);
  const int mode = EXACT ? map.mode : 0;
  int64_t n_items = map.n_items;
  const int rpp = static_cast<int>(a.rows_per_row.d);  // A rows per pool row (a whole number here)

  // (a producer warp whose wait ran out goes on meeting the other one)
  for (int64_t batch0 = blockIdx.x; batch0 < n_items; batch0 += 32 * G) {
    producers_sync();
    // ---- 32 items resolved in parallel, one per lane of the first producer warp:
    //      d_i[lane] = {-, n, nrows, j0, p, slot rows, -, -, tok[8]}, d_l[lane] = pool row of each A row ----
    if (role == 0) {
      const int64_t item = batch0 + lane * G;
      int valid = 0;
      if (item < n_items) {
        int tile, rem;
        item_to_tile(map, a.per_tile, c, item, tile, rem);
        // projection and row block: known before the tile record arrives unless ranks are mixed
        int nb = mode == 0 ? a.max_rb : shrink_blocks_of(a, map.uniform);
        // resolved tiles: where projection and row block follow from the item index alone, the pool rows of the
        // item are fetched now, together with the header and the record that will say whether they count
        int4 rows4[kItemRows / 4];
        const bool entry = a.src.mode == MODE_PLAN && a.src.xoff > 0 && rpp == 1;
        auto fetch_rows = [&](int qk, int j0) {
          const int32_t* xt = a.src.plan + a.src.xoff + static_cast<int64_t>(tile) * (kXtHead + 4 * a.src.xrcap) + kXtHead +
                              qk * a.src.xrcap;
#pragma unroll
          for (int v = 0; v < kItemRows / 4; ++v) {
            rows4[v] = make_int4(-1, -1, -1, -1);
            if (4 * v < RB && j0 + 4 * v < a.src.xrcap) rows4[v] = *reinterpret_cast<const int4*>(xt + j0 + 4 * v);
          }
        };
        if (entry && mode != 2) {
          const int p_s = proj_of(rem, nb, a.nproj);
          fetch_rows(pick3(a.qkvo, p_s), (rem - p_s * nb) * RB);
        }
        TileInfo t;
        if (lookup_tile(a.src, a.tb, tile, t, a.status)) {
          if (mode == 2) nb = shrink_blocks_of(a, t.r);
          const int p = proj_of(rem, nb, a.nproj), j0 = (rem - p * nb) * RB;
          const int rows_total = shrink_rows_of(a, t.r);  // A rows of the projection (rows may be shorter than a pool row)
          if (j0 < rows_total) {
            const int nrows = min(RB, rows_total - j0);
            const int qk = pick3(a.qkvo, p);
            bool ok = true;
            if (entry && t.xok) {
              if (j0 + nrows > t.r) ok = false;
              if (mode == 2) fetch_rows(qk, j0);
#pragma unroll
              for (int v = 0; v < kItemRows / 4; ++v) {
                if (4 * v < nrows) {
                  const int4 e = rows4[v];
                  auto bad = [&](int row, int j) { return j < nrows && (row < 0 || row >= a.tb.pool_rows); };
                  if (bad(e.x, 4 * v) || bad(e.y, 4 * v + 1) || bad(e.z, 4 * v + 2) || bad(e.w, 4 * v + 3)) ok = false;
                  *reinterpret_cast<int4*>(&c.d_l[lane][4 * v]) = e;
                }
              }
            } else {
              for (int v = 0; v < nrows; v += 4) {
                int64_t e[4];  // four loads in flight
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const int pr = a.rows_per_row.div(min(j0 + v + j, rows_total - 1));
                  e[j] = pr < t.r ? tile_loc(t, a.tb, qk, pr) : -1;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  if (e[j] < 0 || e[j] >= a.tb.pool_rows) ok = false;
                  c.d_l[lane][v + j] = static_cast<int32_t>(e[j]);  // (pool_rows < 2^31 here)
                }
              }
            }
            if (ok) {
              int tok[kTileTokens];
#pragma unroll
              for (int i = 0; i < kTileTokens; ++i) tok[i] = i < t.n ? tile_token(t, i) : 0;
              int4* di = reinterpret_cast<int4*>(c.d_i[lane]);
              di[0] = make_int4(0, t.n, nrows, j0);
              di[1] = make_int4(p, t.r, 0, 0);
              di[2] = make_int4(tok[0], tok[1], tok[2], tok[3]);
              di[3] = make_int4(tok[4], tok[5], tok[6], tok[7]);
              valid = 1;
            } else {
              set_status(a.status, SLORA_STATUS_BAD_TABLE);
            }
          }
        }
      }
      const uint32_t mask = __ballot_sync(FULL_MASK, valid != 0);
      if (lane == 0) c.valid_mask = mask;
    }
    producers_sync();
    const uint32_t valid_mask = c.valid_mask;

    // ---- feed the ring, item by item (lane j < 16 carries adapter row j, lane 16 + i carries token i) ----
    for (uint32_t left = valid_mask; left != 0 && !r.dead; left &= left - 1) {
      const int k = __ffs(left) - 1;
      const int* di = c.d_i[k];
      const int4 d0 = *reinterpret_cast<const int4*>(di);
      const int n = d0.y, nrows = d0.z, m_j0 = d0.w, m_p = di[4], m_rows = di[5];
      const bool is_w = lane < nrows;
      const bool is_x = lane >= kActLane && lane < kActLane + n;
      const int mytok = lane >= kActLane ? di[8 + (lane & 7)] : 0;
      const T* src0;
      if (lane < kActLane) {
        const int row = m_j0 + lane;
        const int pr = a.rows_per_row.div(row);
        src0 = w + c.d_l[k][lane] * S + static_cast<int64_t>(row - pr * rpp) * h_in;
      } else {
        src0 = x + static_cast<int64_t>(mytok) * a.x_stride;
      }
      const int myslot = is_w ? lane : nrows + (lane - kActLane);  // position of this lane's chunk in the stage
      // the item goes through the ring in K-chunks of whole units of kKUnit elements (so the element -> consumer lane
      // mapping, and with it the summation order, does not depend on how many rows or tokens share the stage)
      const int kc_elems = stage_k(nrows + n);
      for (int k0 = 0; k0 < h_in; k0 += kc_elems) {
        const int klen = min(kc_elems, h_in - k0);
        const uint32_t bytes = static_cast<uint32_t>(klen) * sizeof(T);
        const uint32_t sz = round128(chunk_at(nrows + n, bytes));
        const bool last = k0 + klen >= h_in;
        const uint32_t off = ring_alloc(r, c, sz, lane, ends.released(last, RB));
        if (r.dead) break;
        const uint32_t slot = r.g % kSlots;
        if (role == 0) {
          if (lane == 0) {  // the stage record in two 16-byte stores; [7] = slot rows of the adapter
            int4* mrec = reinterpret_cast<int4*>(c.meta[slot]);
            mrec[0] = make_int4((k0 == 0 ? FLAG_FIRST : 0) | (last ? FLAG_LAST : 0), nrows, n, m_j0);
            mrec[1] = make_int4(m_p, klen, static_cast<int>(off), m_rows);
          } else if (lane >= kActLane && lane < kActLane + kTileTokens) {
            c.meta[slot][8 + lane - kActLane] = mytok;
          }
          __syncwarp();  // the arrive below publishes every lane's part of the stage record
          if (lane == 0) mbar_expect_tx(&c.full[slot], static_cast<uint32_t>(nrows + n) * bytes);
        }
        // after a CTA's first stages the second producer takes some of the rows as well: half of all copies each
        if (role != 0) ring_enter(r, lane);
        const bool mine = role == 0 ? is_w && (r.g < kRowsAhead || lane < (nrows + n + 1) / 2)
                                    : is_x || (is_w && r.g >= kRowsAhead && lane >= (nrows + n + 1) / 2);
        ring_issue(r, c, slot, ring_base + off + chunk_at(myslot, bytes), src0 + k0,
                   mine ? bytes : 0u);
        if (last) ends.end_item(r.g);
      }
    }
    __syncwarp();
    if (!EXACT && a.src.mode == MODE_PLAN) n_items = padded_item_count(a.src, a.nproj * a.max_rb);
  }
  ring_finish(r, c, a.status, lane);
}

// Sums of one warp over its slices of an item.  K goes by units of kKUnit elements; warp cw owns [cw * 64, +64) of each, two
// fragments of 32.  A fragment of a unit is a chain of two mma from zero, added to the fragment's sum in unit order: an mma
// truncates what it adds to its accumulator, and with accumulators kept over the whole row (sixteen steps at 8192) 1.6 of a
// thousand intermediates were not the nearest 16-bit value, 0.9 with FMA sums.  The two fragments may share one
// instruction: where rows and tokens leave half of it empty (SPLIT), the second fragment's rows and tokens take those places.
struct ShrinkAcc {
  float d[2][4];  // [fragment; 0 alone when they share][C fragment]
};
enum ShrinkForm {
  FORM_FULL,   // rows 0..7 and 8..15, tokens 0..7
  FORM_WIDE,   // rows 0..7, tokens 0..7
  FORM_ROWS8,  // rows 0..7, tokens 0..3: the second fragment in rows 8..15 and columns 4..7
  FORM_ROWS4   // rows 0..3, tokens 0..3: the second fragment in rows 4..7 and columns 4..7
};
__device__ __forceinline__ int shrink_form(int rows_per_item, int nrows, int n) {
  if (rows_per_item > 8) return FORM_FULL;
  if (n > 4) return FORM_WIDE;
  return nrows > 4 ? FORM_ROWS8 : FORM_ROWS4;
}

// Lane (g, t) reads 16-byte vector t of the 64 bytes of a row or token; lanes beyond the real rows and tokens repeat the last
// one (what they compute is in rows and columns that nobody reads), and in the last round of a row (END) what lies beyond
// its end is zero: rows end anywhere on a multiple of eight elements.  A stage starts at a whole unit.  The loads of a
// round are issued before its first mma: the warp has nothing else to hide their latency with.  (A round of two units:
// with four or eight an item of four rows and one token took 1 to 4 % longer.  Checks of row, token and end at every load
// instead: 1160 cycles an item of 4096 elements against 1050 and, in batches of single tokens, where two stages a CTA are
// all that is in flight, 4 to 6 % of the launch.)
constexpr int kRoundUnits = 2;
template <int FORM>
struct ShrinkShape {
  static constexpr bool SPLIT = FORM == FORM_ROWS8 || FORM == FORM_ROWS4;
  static constexpr int NA = FORM == FORM_ROWS4 ? 1 : 2, NB = FORM == FORM_FULL ? 2 : 0, NX = SPLIT ? 1 : 2;
};
template <typename T, int FORM, bool END>
__device__ __forceinline__ void shrink_round(ShrinkAcc& acc, const unsigned char* pa, const unsigned char* pb,
                                             const unsigned char* px, int left_a, int left_x) {
  using S = ShrinkShape<FORM>;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4 va[kRoundUnits][S::NA], vb[kRoundUnits][S::NB ? S::NB : 1], vx[kRoundUnits][S::NX];
#pragma unroll
  for (int u = 0; u < kRoundUnits; ++u) {
    const int k = u * kKUnit;
    auto load = [&](const unsigned char* from, int h, int left) {
      return !END || k + 32 * h < left ? *reinterpret_cast<const uint4*>(from + 2 * (k + 32 * h)) : zero;
    };
#pragma unroll
    for (int h = 0; h < S::NA; ++h) va[u][h] = load(pa, h, left_a);
#pragma unroll
    for (int h = 0; h < S::NB; ++h) vb[u][h] = load(pb, h, left_a);
#pragma unroll
    for (int h = 0; h < S::NX; ++h) vx[u][h] = load(px, h, left_x);
  }
#pragma unroll
  for (int u = 0; u < kRoundUnits; ++u) {
    // (rows 8..15 of the two forms without them are not summed)
    constexpr int NSUM = FORM == FORM_FULL || FORM == FORM_ROWS8 ? 4 : 2;
    float first[4], second[4];
    if (FORM == FORM_ROWS4) {
      mma_k32<T>(first, va[u][0], zero, vx[u][0]);
    } else if (FORM == FORM_ROWS8) {
      mma_k32<T>(first, va[u][0], va[u][S::NA - 1], vx[u][0]);
    } else {
      mma_k32<T>(first, va[u][0], S::NB ? vb[u][0] : zero, vx[u][0]);
      mma_k32<T>(second, va[u][S::NA - 1], S::NB ? vb[u][S::NB ? S::NB - 1 : 0] : zero, vx[u][S::NX - 1]);
    }
#pragma unroll
    for (int i = 0; i < NSUM; ++i) {
      acc.d[0][i] += first[i];
      if (!S::SPLIT) acc.d[1][i] += second[i];
    }
  }
}
template <typename T, int FORM>
__device__ __forceinline__ void shrink_accumulate(ShrinkAcc& acc, const unsigned char* st, int nrows, int n, int klen,
                                                  int cw, int lane) {
  using S = ShrinkShape<FORM>;
  constexpr int ROUND = kRoundUnits * kKUnit;
  const int g = lane >> 2, t = lane & 3;
  const int bytes = klen * static_cast<int>(sizeof(T));
  const int row = FORM == FORM_ROWS4 ? (g & 3) : g, tok = S::SPLIT ? (g & 3) : g;
  const int ka = cw * (kKUnit / kConsumerWarps) + 8 * t + (FORM == FORM_ROWS4 ? 32 * (g >> 2) : 0);
  const int kx = cw * (kKUnit / kConsumerWarps) + 8 * t + (S::SPLIT ? 32 * (g >> 2) : 0);
  const unsigned char* pa = st + chunk_at(min(row, nrows - 1), bytes) + ka * 2;
  const unsigned char* pb = st + chunk_at(min(g + 8, nrows - 1), bytes) + ka * 2;
  const unsigned char* px = st + chunk_at(nrows + min(tok, n - 1), bytes) + kx * 2;
  int k0 = 0;
#pragma unroll 1
  for (; k0 + ROUND <= klen; k0 += ROUND) {
    shrink_round<T, FORM, false>(acc, pa, pb, px, 0, 0);
    pa += 2 * ROUND, pb += 2 * ROUND, px += 2 * ROUND;
  }
  if (k0 < klen) shrink_round<T, FORM, true>(acc, pa, pb, px, klen - k0 - ka, klen - k0 - kx);
}
// The warp's partial sums in C-fragment order: [0], [1] row g columns 2t, 2t + 1; [2], [3] row g + 8.
template <int FORM>
__device__ __forceinline__ void shrink_partials(const ShrinkAcc& acc, float (&out)[4]) {
  float first[4], second[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    first[i] = acc.d[0][i];
    second[i] = acc.d[1][i];
  }
  if (FORM == FORM_ROWS4) {  // the second fragment's sums sit four rows and four columns on: eighteen lanes
#pragma unroll
    for (int i = 0; i < 2; ++i) second[i] = __shfl_down_sync(FULL_MASK, first[i], 18);
  } else if (FORM == FORM_ROWS8) {
#pragma unroll
    for (int i = 0; i < 2; ++i) second[i] = __shfl_down_sync(FULL_MASK, first[2 + i], 2);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) out[i] = first[i] + second[i];
}

// At the item's last chunk the warps' partial sums meet in shared memory; the warp that arrives last (an atomic counter,
// no waiting) adds them in a fixed order and writes delta.  A reduction buffer is reused only after the last warp released
// the stage it was summing in (shrink_buffers).
template <typename T, bool EXACT>
__device__ __forceinline__ void shrink_consumer(const ShrinkArgs& a, const unsigned char* ring_mem, PipeCtl& c,
                                                ShrinkRed& red, int lane, int cw) {
  pdl_wait();
  int tp_slot = a.tp.half;  // which part of every rank's delta buffer this exchange writes
  if (a.tp.enabled && a.tp.inband == 3) {
    // rotating thirds (see TpLink::inband): the exchange's number picks the third; this CTA's share of the third
    // the PREVIOUS exchange used - whose expand on this GPU is complete: it is what the wait above waited for - goes
    // back to the empty pattern; one thread tells this exchange's expand its number
    const int e = *reinterpret_cast<volatile const int32_t*>(a.tp.seq_state);
    tp_slot = e % 3;
    const int64_t third = 3 * a.tp.full_tokens * static_cast<int64_t>(a.tp.n_parts) * a.delta_width;  // elements
    uint4* prev = reinterpret_cast<uint4*>(reinterpret_cast<T*>(a.tp.full[a.tp.my_part]) + ((e + 2) % 3) * third);
    const int64_t n16 = third * static_cast<int64_t>(sizeof(T)) / 16;
    const uint4 ev = make_uint4(kTpEmpty2, kTpEmpty2, kTpEmpty2, kTpEmpty2);
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * (kConsumerWarps * 32) + cw * 32 + lane; i < n16;
         i += static_cast<int64_t>(gridDim.x) * (kConsumerWarps * 32))
      prev[i] = ev;
    if (blockIdx.x == 0 && cw == 0 && lane == 0) {
      a.tp.seq_state[1] = e;
      __threadfence();  // before this thread lets dependents launch
    }
    __syncwarp();
  }
  if (a.tp.enabled && a.tp.inband >= 2) pdl_launch_dependents();
  const bool tall = a.rows_per_cta > 8;
  const uint32_t buffers = shrink_buffers(a.rows_per_cta);
  const int lanes = a.rows_per_cta > 4 ? 32 : 16;  // that hold rows of the item
  ShrinkAcc acc = {};
  uint32_t item_seq = 0;
  for (uint32_t g = 0;; ++g) {
    const uint32_t slot = g % kSlots;
    if (!mbar_wait_timed(&c.full[slot], (g / kSlots) & 1)) {
      if (lane == 0) set_status(a.status, SLORA_STATUS_TIMEOUT);
      return;
    }
    const int* m = c.meta[slot];
    const int4 m0 = *reinterpret_cast<const int4*>(m), m1 = *reinterpret_cast<const int4*>(m + 4);
    const int flags = m0.x;
    if (flags & FLAG_END) return;
    const int nrows = m0.y, n = m0.z, klen = m1.y;
    if (flags & FLAG_FIRST) acc = ShrinkAcc{};
    const unsigned char* st = ring_mem + m1.z;
    const int form = shrink_form(a.rows_per_cta, nrows, n);
    switch (form) {
      case FORM_FULL: shrink_accumulate<T, FORM_FULL>(acc, st, nrows, n, klen, cw, lane); break;
      case FORM_WIDE: shrink_accumulate<T, FORM_WIDE>(acc, st, nrows, n, klen, cw, lane); break;
      case FORM_ROWS8: shrink_accumulate<T, FORM_ROWS8>(acc, st, nrows, n, klen, cw, lane); break;
      default: shrink_accumulate<T, FORM_ROWS4>(acc, st, nrows, n, klen, cw, lane); break;
    }
    if (flags & FLAG_LAST) {
      const uint32_t buf = item_seq % buffers;
      ++item_seq;
      // buffer of this item: eight warps' fragments, one half (rows 0..7) or two
      const int halves = tall ? 2 : 1;
      float2* mine = red.sum + (buf * kConsumerWarps + cw) * halves * lanes;
      float part[4];
      switch (form) {
        case FORM_ROWS4: shrink_partials<FORM_ROWS4>(acc, part); break;
        case FORM_ROWS8: shrink_partials<FORM_ROWS8>(acc, part); break;
        default: shrink_partials<FORM_FULL>(acc, part); break;
      }
      if (lane < lanes) mine[lane] = make_float2(part[0], part[1]);
      if (tall) mine[32 + lane] = make_float2(part[2], part[3]);
      __syncwarp();
      int old = 0;
      if (lane == 0) {
        __threadfence_block();
        old = atomicAdd(&red.cnt[buf], 1);
      }
      old = __shfl_sync(FULL_MASK, old, 0);
      if (old == kConsumerWarps - 1) {
        __threadfence_block();
        for (int h = 0; h < halves; ++h) {
          float2 sum = make_float2(0.f, 0.f);
#pragma unroll
          for (int w = 0; w < kConsumerWarps; ++w) {
            const float2 v = red.sum[((buf * kConsumerWarps + w) * halves + h) * lanes + (lane & (lanes - 1))];
            sum.x += v.x;
            sum.y += v.y;
          }
          const int j = 8 * h + (lane >> 2);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int i = 2 * (lane & 3) + q;
            if (j < nrows && i < n && m0.w + j < a.delta_width) {
              const T v = from_f32<T>(q == 0 ? sum.x : sum.y);
              if (a.tp.enabled) {
                // tensor parallelism: this rank's rows go straight into every rank's delta buffer (NVLink stores)
                const int64_t R = static_cast<int64_t>(a.tp.n_parts) * a.delta_width;
                const int64_t at = ((static_cast<int64_t>(tp_slot) * 3 + m1.x) * a.tp.full_tokens + m[8 + i]) * R +
                                   static_cast<int64_t>(a.tp.my_part) * m1.w + m0.w + j;
                for (int p = 0; p < a.tp.n_parts; ++p) reinterpret_cast<T*>(a.tp.full[p])[at] = v;
              } else {
                T* d = reinterpret_cast<T*>(pick3(a.delta, m1.x));
                d[static_cast<int64_t>(m[8 + i]) * a.delta_stride + m0.w + j] = v;
              }
            }
          }
        }
        if (lane == 0) red.cnt[buf] = 0;
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&c.empty[slot]);
  }
}

// A segment call sends its long segments to the tensor-core kernels and launches these kernels beside them for the
// short ones.  When there are none (a pure prefill batch) the launch has nothing to do: every CTA finds that out from
// the segment table with one round of loads per table (a thread per segment) and leaves before it sets up its ring,
// instead of resolving every tile slot of every segment first.  A segment whose table entries look wrong counts as
// this launch's, whose normal path reports it.
__device__ __forceinline__ bool segments_all_elsewhere(const TileSrc& s, const Tables& tb) {
  if (s.mode != MODE_SEGMENT || s.seg_split <= 0) return false;
  bool mine = false;
  for (int i = threadIdx.x; i < s.n_seg; i += blockDim.x) {
    const int64_t len = s.seg_len[i];
    if (len <= 0) continue;
    const int64_t ad = s.ids[i];
    if (len < s.seg_split || ad < 0 || ad >= tb.n_adapters) {
      mine = true;
      continue;
    }
    const int64_t r4 = tb.ranks4[ad], st = tb.start[ad], r = r4 >> 2;
    if (r4 < 0 || st < 0 || st + r4 > tb.loc_len ||
        !(r >= 8 && r <= 128 && r % 8 == 0 && tb.pool_stride % r == 0 && r <= s.mma_max_rows))
      mine = true;
  }
  return __syncthreads_or(mine) == 0;
}

template <typename T, bool EXACT>
__global__ void __launch_bounds__(kPipeThreads, kPipeCtasPerSm) lora_shrink_pipe_kernel(const ShrinkArgs a) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ __align__(16) PipeCtl ctl;
  __shared__ __align__(16) ShrinkRed red;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (segments_all_elsewhere(a.src, a.tb)) return;
  if (tid < kSlots) red.cnt[tid] = 0;
  pipe_init(ctl, tid);
  // (a shrink whose expand starts early lets its dependents launch only after its own grid-dependency wait, thread
  // by thread: see TpLink::inband)
  if (!(a.tp.enabled && a.tp.inband >= 2)) pdl_launch_dependents();
  if (EXACT) {
    fill_item_counts(a.src, a.tb, ctl, tid, [&](int rr, int) { return shrink_items_of(a, rr); });
    __syncthreads();
  }
  if (warp < kProducerWarps) {
    shrink_producer<T, EXACT>(a, ring_mem, ctl, lane, warp);
  } else {
    shrink_consumer<T, EXACT>(a, ring_mem, ctl, red, lane, warp - kProducerWarps);
  }
  if (a.tp.enabled && !a.tp.inband) tp_link_finish(a.tp, true);
}

// ------------------------------------------------------------------------------------------------------------
// expand
// stage meta: [0] flags [1] n [2] r [3] projection [4] clen [5] first output [6] scale bits [7] ring offset,
//             [8..15] token ids
// stage bytes: B chunk (clen elements), then n y segments of clen / r elements, then n delta rows of r elements
// ------------------------------------------------------------------------------------------------------------
// The expand takes ranks 8..128 in powers of two that the delta buffers hold; B chunks of projection p for rank rk;
// items of a tile of rr slot rows.
__device__ __forceinline__ bool expand_rank_ok(const ExpandArgs& a, int rk) {
  return (rk == 8 || rk == 16 || rk == 32 || rk == 64 || rk == 128) && rk <= a.max_rank;
}
__device__ __forceinline__ int expand_chunks_of(const ExpandArgs& a, int p, int rk) {
  const int64_t flat = static_cast<int64_t>(pick3(a.h_out, p)) * rk;
  return static_cast<int>(min(static_cast<int64_t>(a.chunk_begin[p + 1] - a.chunk_begin[p]),
                              (flat + kPipeChunk - 1) / kPipeChunk));
}
__device__ __forceinline__ int expand_items_of(const ExpandArgs& a, int rr) {
  const int rk = rr * a.rank_mult;
  if (!expand_rank_ok(a, rk)) return 1;  // one item, which reports the rank
  int n = 0;
  for (int p = 0; p < a.nproj; ++p) n += expand_chunks_of(a, p, rk);
  return n;
}

template <typename T, bool EXACT>
__device__ __forceinline__ void expand_producer(const ExpandArgs& a, unsigned char* ring_mem, PipeCtl& c, int lane,
                                                int role) {
  const int total_chunks = a.chunk_begin[a.nproj];
  const int64_t S = a.tb.pool_stride;
  const T* w = reinterpret_cast<const T*>(a.w);
  const int64_t G = gridDim.x;
  const uint32_t ring_base = smem_u32(ring_mem);
  Ring r;
  r.role = role;
  r.cap = EXACT ? kExpandRingBytes : kRingBytes;  // see kExpandRingBytes
  r.tp = a.tp.enabled ? &a.tp : nullptr;
  r.status = a.status;
  if (a.tp.enabled && a.tp.inband >= 2) r.pre = false;  // early start: nothing to wait for (see TpLink::inband)
  int64_t delta_off = 0;  // rotating thirds: elements from the first third to this exchange's
  if (a.tp.enabled && a.tp.inband == 3) {
    const int e = *reinterpret_cast<volatile const int32_t*>(a.tp.seq_state + 1);  // left by this exchange's shrink
    delta_off = (e % 3) * 3 * a.tp.full_tokens * a.delta_stride;
    if (blockIdx.x == 0 && lane == 0 && role == 0) a.tp.seq_state[0] = e + 1;  // the next shrink reads it after its own wait
  }
  auto rank_ok = [&](int rk) { return expand_rank_ok(a, rk); };
  auto chunks_of = [&](int p, int rk) { return expand_chunks_of(a, p, rk); };
  const ItemMap map = EXACT ? build_item_map(a.src, total_chunks, c, lane, role, [&](int rr, int) { return expand_items_of(a, rr); })
                            : padded_item_map(a.src, total_chunks);
  const int mode = EXACT ? map.mode : 0;
  int64_t n_items = map.n_items;

  // (a producer warp whose wait ran out goes on meeting the other one)
  for (int64_t batch0 = blockIdx.x; batch0 < n_items; batch0 += 32 * G) {
    producers_sync();
    // d_i[lane] = {log2 r, n, r, p, clen, first output, scale bits, chunk start inside its first pool row, tok[8]},
    // d_l[lane][j] = pool row of the chunk's j-th slot row
    if (role == 0) {
      const int64_t item = batch0 + lane * G;
      int valid = 0;
      if (item < n_items) {
        int tile, ch;
        item_to_tile(map, a.per_tile, c, item, tile, ch);
        // projection and chunk: known before the tile record arrives unless ranks are mixed
        int p = 0;
        auto split = [&](int rk) {
          while (p + 1 < a.nproj && ch >= chunks_of(p, rk)) {
            ch -= chunks_of(p, rk);
            ++p;
          }
        };
        if (mode == 0) {
          while (p + 1 < a.nproj && ch >= a.chunk_begin[p + 1]) ++p;
          ch -= a.chunk_begin[p];
        } else if (mode == 1 && rank_ok(map.uniform * a.rank_mult)) {
          split(map.uniform * a.rank_mult);
        }
        // resolved tiles: where projection and chunk follow from the item index alone, the chunk's pool rows are
        // fetched now, together with the header and the record that will say whether they count
        const bool entry = a.src.mode == MODE_PLAN && a.src.xoff > 0;
        int64_t row[kSpanRows];
        auto fetch_rows = [&](int qk, int pr) {
          const int32_t* xt = a.src.plan + a.src.xoff + static_cast<int64_t>(tile) * (kXtHead + 4 * a.src.xrcap) + kXtHead +
                              qk * a.src.xrcap;
#pragma unroll
          for (int j = 0; j < kSpanRows; ++j) row[j] = xt[min(pr + j, a.src.xrcap - 1)];
        };
        if (entry && mode != 2) fetch_rows(pick3(a.qkvo, p), a.stride.div(min(ch, 0x7fffffff / kPipeChunk) * kPipeChunk));
        TileInfo t;
        if (lookup_tile(a.src, a.tb, tile, t, a.status)) {
          const int rk = t.r * a.rank_mult;
          if (mode == 2 && rank_ok(rk)) split(rk);
          const int h_out = pick3(a.h_out, p);
          const int64_t flat_total = static_cast<int64_t>(h_out) * rk;
          const int64_t c0 = static_cast<int64_t>(ch) * kPipeChunk;
          if (c0 < flat_total) {
            if (!rank_ok(rk)) {
              set_status(a.status, SLORA_STATUS_BAD_RANK);
            } else {
              const int clen = static_cast<int>(min(static_cast<int64_t>(kPipeChunk), flat_total - c0));
              const int qk = pick3(a.qkvo, p);
              const int pr0 = a.stride.div(static_cast<int>(c0)), pr1 = a.stride.div(static_cast<int>(c0) + clen - 1);
              bool ok = pr1 - pr0 < kSpanRows && pr1 < t.r;
              if (ok) {
                if (!t.xok) {
#pragma unroll
                  for (int j = 0; j < kSpanRows; ++j) row[j] = tile_loc(t, a.tb, qk, min(pr0 + j, pr1));
                } else if (mode == 2) {
                  fetch_rows(qk, pr0);
                }
#pragma unroll
                for (int j = 0; j < kSpanRows; ++j) {
                  if (pr0 + j <= pr1) {
                    if (row[j] < 0 || row[j] >= a.tb.pool_rows) ok = false;
                    c.d_l[lane][j] = static_cast<int32_t>(row[j]);  // (pool_rows < 2^31 here)
                  }
                }
              }
              if (ok) {
                int tok[kTileTokens];
#pragma unroll
                for (int i = 0; i < kTileTokens; ++i) tok[i] = i < t.n ? tile_token(t, i) : 0;
                const int lg = 31 - __clz(rk);  // rk is a power of two (rank_ok)
                // the scale's 16 bits: from the resolved tile when it counts and carries one, else from the table
                T sc;
                if (t.xok && (t.xscale & 0x10000)) {
                  const unsigned short bits = static_cast<unsigned short>(t.xscale & 0xffff);
                  sc = *reinterpret_cast<const T*>(&bits);
                } else {
                  sc = reinterpret_cast<const T*>(a.scales)[t.adapter];
                }
                int4* di = reinterpret_cast<int4*>(c.d_i[lane]);
                di[0] = make_int4(lg, t.n, rk, p);
                di[1] = make_int4(clen, static_cast<int>(c0) >> lg, __float_as_int(to_f32<T>(sc)),
                                  static_cast<int>(c0 - static_cast<int64_t>(pr0) * S));
                di[2] = make_int4(tok[0], tok[1], tok[2], tok[3]);
                di[3] = make_int4(tok[4], tok[5], tok[6], tok[7]);
                valid = 1;
              } else {
                set_status(a.status, SLORA_STATUS_BAD_TABLE);
              }
            }
          }
        }
      }
      const uint32_t mask = __ballot_sync(FULL_MASK, valid != 0);
      if (lane == 0) c.valid_mask = mask;
    }
    producers_sync();
    const uint32_t valid_mask = c.valid_mask;

    // one copy per lane: 0..5 the B chunk's pool rows, 16..23 y segments, 24..31 delta rows.  Everything that does
    // not depend on where the stage lands in the ring is worked out BEFORE the wait for ring space: what follows the
    // wait is on the path from a consumer's release of a stage to the next copy's issue.
    for (uint32_t left = valid_mask; left != 0 && !r.dead; left &= left - 1) {
      const int k = __ffs(left) - 1;
      const int* di = c.d_i[k];
      const int4 d0 = *reinterpret_cast<const int4*>(di), d1 = *reinterpret_cast<const int4*>(di + 4);
      const int n = d0.y, rk = d0.z, p = d0.w, clen = d1.x, obase = d1.y, m_scale = d1.z, col0 = d1.w;
      const int nout = clen >> d0.x;
      const uint32_t b_bytes = static_cast<uint32_t>(clen) * sizeof(T);
      const uint32_t y_bytes = static_cast<uint32_t>(nout) * sizeof(T);
      const uint32_t d_bytes = static_cast<uint32_t>(rk) * sizeof(T);
      const uint32_t total = b_bytes + static_cast<uint32_t>(n) * (y_bytes + d_bytes);
      const uint32_t sz = round128(total);
      const int mytok = lane >= 16 ? di[8 + (lane & 7)] : 0;
      uint32_t rel = 0, bytes = 0;  // this lane's copy: offset inside the stage, size
      const T* src = w;
      bool is_act = false;
      if (lane < kSpanRows) {
        // the chunk's part of pool row pr0 + lane: one copy per pool row, whole rows except at the chunk's ends
        const int64_t start = lane * S - col0;  // (before the chunk for row 0)
        if (start < clen) {
          const int poff = max(static_cast<int>(start), 0), col = lane == 0 ? col0 : 0;
          src = w + c.d_l[k][lane] * S + col;
          rel = static_cast<uint32_t>(poff) * sizeof(T);
          bytes = static_cast<uint32_t>(min(static_cast<int>(S) - col, clen - poff)) * sizeof(T);
        }
      } else if (lane >= 16 && lane < 16 + n) {
        src = reinterpret_cast<const T*>(pick3(a.y, p)) + static_cast<int64_t>(mytok) * pick3(a.y_stride, p) + obase;
        rel = b_bytes + static_cast<uint32_t>(lane - 16) * y_bytes;
        bytes = y_bytes;
        is_act = true;
      } else if (lane >= 24 && lane < 24 + n) {
        src = reinterpret_cast<const T*>(pick3(a.delta, p)) + delta_off + static_cast<int64_t>(mytok) * a.delta_stride;
        rel = b_bytes + static_cast<uint32_t>(n) * y_bytes + static_cast<uint32_t>(lane - 24) * d_bytes;
        bytes = d_bytes;
        is_act = true;
      }
      const uint32_t off = ring_alloc(r, c, sz, lane);
      if (r.dead) break;
      const uint32_t slot = r.g % kSlots;
      if (role == 0) {
        if (lane == 0) {  // the stage record in two 16-byte stores
          int4* mrec = reinterpret_cast<int4*>(c.meta[slot]);
          mrec[0] = make_int4(0, n, rk, p);
          mrec[1] = make_int4(clen, obase, m_scale, static_cast<int>(off));
        } else if (lane >= kActLane && lane < kActLane + kTileTokens) {
          c.meta[slot][8 + lane - kActLane] = mytok;
        }
        __syncwarp();  // the arrive below publishes every lane's part of the stage record
        if (lane == 0) mbar_expect_tx(&c.full[slot], total);
      }
      if (role != 0) ring_enter(r, lane);
      ring_issue(r, c, slot, ring_base + off + rel, src, is_act == (role != 0) ? bytes : 0u);
    }
    __syncwarp();
    if (!EXACT && a.src.mode == MODE_PLAN) n_items = padded_item_count(a.src, total_chunks);
  }
  ring_finish(r, c, a.status, lane);
}

// Tensor parallelism with in-band signalling: before a warp uses a stage, it looks at the delta values the stage's
// copy brought.  The common case - everything had landed - costs each lane one look at the vectors it is going to
// use (the 16 bytes at its own k offset of each of the n rows) and the warp one vote.  Otherwise the warp settles the
// whole delta block: lane l takes the vectors l, l + 32, ...; one that still holds the empty pattern is fetched again
// from global memory until it has arrived (bounded) and put into the stage.  Every warp does this by itself (the
// warps do not wait for one another; they write the same values), so the arithmetic that follows is the same
// straight loop as without tensor parallelism.
template <typename T>
__device__ __noinline__ void expand_settle_slow(T* ds, const int* m, int r, const T* dglobal, int64_t dglobal_stride,
                                                int32_t* status, volatile int* gave_up, int lane);

template <typename T>
__device__ __forceinline__ void expand_settle_delta(T* ds, const int* m, int r, const T* dglobal, int64_t dglobal_stride,
                                                    int32_t* status, volatile int* gave_up, int lane) {
  const int n = m[1];
  const int kp = (lane & (r / 8 - 1)) * 8;  // r is a power of two (expand_rank_ok)
  bool missing = false;
  for (int tt = 0; tt < n; ++tt) missing |= tp_has_empty(*reinterpret_cast<const uint4*>(ds + tt * r + kp));
  if (__any_sync(FULL_MASK, missing)) expand_settle_slow<T>(ds, m, r, dglobal, dglobal_stride, status, gave_up, lane);
}

// (kept out of line: it runs once in a long while and its polling loop would only bloat the consumers' hot loop)
template <typename T>
__device__ __noinline__ void expand_settle_slow(T* ds, const int* m, int r, const T* dglobal, int64_t dglobal_stride,
                                                int32_t* status, volatile int* gave_up, int lane) {
  const int n = m[1];
  const int vec_per_row = r / 8;
  for (int v = lane; v < n * vec_per_row; v += 32) {
    const int tt = v / vec_per_row, k0 = (v - tt * vec_per_row) * 8;
    uint4 dv = *reinterpret_cast<const uint4*>(ds + tt * r + k0);
    if (tp_has_empty(dv)) {
      if (!tp_poll_delta(dglobal + static_cast<int64_t>(m[8 + tt]) * dglobal_stride + k0, dv, gave_up)) {
        set_status(status, SLORA_STATUS_TIMEOUT);
        dv = make_uint4(0u, 0u, 0u, 0u);
      }
      *reinterpret_cast<uint4*>(ds + tt * r + k0) = dv;
      fence_proxy_async();  // this store before the bulk copy that will reuse the stage's bytes
    }
  }
  __syncwarp();
}

// One consumer warp's part of an expand stage of rank R and at most NT tokens: flat elements [cw * 2048, +2048) of the
// chunk on the tensor pipe (expand_group), then y = y + scale * v with y read from the stage as vectors and written
// back as vectors.
template <typename T, int R, int NT, bool INBAND>
__device__ __forceinline__ void expand_stage(const T* bs, const int* m, T* y, int64_t y_stride, int lane, int cw,
                                             const T* dglobal, int64_t dglobal_stride, int32_t* status,
                                             volatile int* gave_up) {
  using S = ExpandShape<R>;
  using K = TokenSplit<NT>;
  const int n = m[1], clen = m[4], obase = m[5];
  if (cw * (kPipeChunk / kConsumerWarps) >= clen) return;
  const int nout = clen / R;
  const float scale = __int_as_float(m[6]);
  const T* ys = bs + clen;
  const T* ds = ys + n * nout;
  // in-band signalling: have this stage's delta values all arrived?
  if (INBAND) expand_settle_delta<T>(const_cast<T*>(ds), m, R, dglobal, dglobal_stride, status, gave_up, lane);
  const int g = lane >> 2, t = lane & 3;
  const DeltaFrag<R> f = load_delta_frag<T, R>(ds, K::column(g, n), t);
  const int tok0 = K::tok0(t);
  const int x = expand_x<R>(g);
  constexpr int ROUNDS = (S::NG + K::DUP - 1) / K::DUP;
#pragma unroll 1
  for (int r = 0; r < ROUNDS; ++r) {
    float acc[S::VPL][2];
    expand_round<T, R, NT>(acc, bs, f, cw, r, nout, lane);
    const int gr = r * K::DUP + K::di(t);
    const int o = expand_out<R>(cw, gr, g);
    const bool live = gr < S::NG && o < nout;
#pragma unroll
    for (int c = 0; c < K::TPL; ++c) {
      float v[S::VPL], yv[S::VPL];
#pragma unroll
      for (int i = 0; i < S::VPL; ++i) v[i] = acc[i][c];
      xor_index(v, x);
      const int tok = tok0 + c;
      if (live && tok < n) {
        load_vec<T>(yv, ys + tok * nout + o);
#pragma unroll
        for (int i = 0; i < S::VPL; ++i) yv[i] = fmaf(scale, v[i], yv[i]);
        store_vec<T>(y + static_cast<int64_t>(m[8 + tok]) * y_stride + obase + o, yv);
      }
    }
  }
}

template <typename T, int R, bool INBAND>
__device__ __forceinline__ void expand_stage_tokens(const T* bs, const int* m, T* y, int64_t y_stride, int lane, int cw,
                                                    const T* dg, int64_t dgs, int32_t* status, volatile int* gave_up) {
  const int n = m[1];
  if (n <= 1) {
    expand_stage<T, R, 1, INBAND>(bs, m, y, y_stride, lane, cw, dg, dgs, status, gave_up);
  } else if (n <= 2) {
    expand_stage<T, R, 2, INBAND>(bs, m, y, y_stride, lane, cw, dg, dgs, status, gave_up);
  } else if (n <= 4) {
    expand_stage<T, R, 4, INBAND>(bs, m, y, y_stride, lane, cw, dg, dgs, status, gave_up);
  } else {
    expand_stage<T, R, 8, INBAND>(bs, m, y, y_stride, lane, cw, dg, dgs, status, gave_up);
  }
}

template <typename T, bool INBAND>
__device__ __forceinline__ void expand_consumer(const ExpandArgs& a, const unsigned char* ring_mem, PipeCtl& c,
                                                int lane, int cw) {
  if (!(a.tp.enabled && a.tp.inband >= 2)) pdl_wait();
  int64_t delta_off = 0;
  if (INBAND && a.tp.inband == 3)
    delta_off = (*reinterpret_cast<volatile const int32_t*>(a.tp.seq_state + 1) % 3) * 3 * a.tp.full_tokens *
                a.delta_stride;
  for (uint32_t g = 0;; ++g) {
    const uint32_t slot = g % kSlots;
    if (!mbar_wait_timed(&c.full[slot], (g / kSlots) & 1)) {
      if (lane == 0) set_status(a.status, SLORA_STATUS_TIMEOUT);
      return;
    }
    const int* m = c.meta[slot];
    if (m[0] & FLAG_END) return;
    const T* bs = reinterpret_cast<const T*>(ring_mem + m[7]);
    const int p = m[3];
    T* y = reinterpret_cast<T*>(pick3(a.y, p));
    const int64_t ystr = pick3(a.y_stride, p);
    const T* dg = INBAND ? reinterpret_cast<const T*>(pick3(a.delta, p)) + delta_off : nullptr;
    const int64_t dgs = a.delta_stride;
    switch (m[2]) {
      case 8: expand_stage_tokens<T, 8, INBAND>(bs, m, y, ystr, lane, cw, dg, dgs, a.status, &c.tp_gave_up); break;
      case 16: expand_stage_tokens<T, 16, INBAND>(bs, m, y, ystr, lane, cw, dg, dgs, a.status, &c.tp_gave_up); break;
      case 32: expand_stage_tokens<T, 32, INBAND>(bs, m, y, ystr, lane, cw, dg, dgs, a.status, &c.tp_gave_up); break;
      case 64: expand_stage_tokens<T, 64, INBAND>(bs, m, y, ystr, lane, cw, dg, dgs, a.status, &c.tp_gave_up); break;
      default: expand_stage_tokens<T, 128, INBAND>(bs, m, y, ystr, lane, cw, dg, dgs, a.status, &c.tp_gave_up); break;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&c.empty[slot]);
  }
}

// INBAND: the instantiation for tensor parallelism with in-band signalling (TpLink::inband); the plain one carries
// none of its checks.
template <typename T, bool EXACT, bool INBAND = false>
__global__ void __launch_bounds__(kPipeThreads, kPipeCtasPerSm) lora_expand_pipe_kernel(const ExpandArgs a) {
  extern __shared__ __align__(128) unsigned char ring_mem[];
  __shared__ __align__(16) PipeCtl ctl;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (segments_all_elsewhere(a.src, a.tb)) return;
  pipe_init(ctl, tid);
  pdl_launch_dependents();
  if (EXACT) {
    fill_item_counts(a.src, a.tb, ctl, tid, [&](int rr, int) { return expand_items_of(a, rr); });
    __syncthreads();
  }
  if (warp < kProducerWarps) {
    expand_producer<T, EXACT>(a, ring_mem, ctl, lane, warp);
  } else {
    expand_consumer<T, INBAND>(a, ring_mem, ctl, lane, warp - kProducerWarps);
  }
  if (a.tp.enabled && a.tp.inband != 3) {  // (rotating thirds: nothing to do at the end of an expand)
    if (INBAND) {
      // what this exchange used of its half of the delta buffer: [nproj][full_tokens][delta_stride] elements from
      // delta[0] on
      tp_inband_finish(a.tp, const_cast<void*>(a.delta[0]),
                       a.nproj * a.tp.full_tokens * a.delta_stride * static_cast<int64_t>(sizeof(T)));
    } else {
      tp_link_finish(a.tp, false);
    }
  }
}

}  // namespace slora
