// Scheduling and DAG bookkeeping of the persistent fabric: how a worker finds its
// next tiles, and what happens when a stage's last tile completes.
//
// What is fixed by the wire protocol (the reference's, csrc/fabric/runtime.cuh:155-509,
// because its Python program builder, its state readers and its tests see it):
//   * a ring entry is tag << 20 | stage; tags are 12 bits, 0 = never activated;
//   * a ring has a reservation counter, a published tail and a consumer head;
//     entries become visible in reservation order;
//   * StageRuntime::tag_next = tag << 32 | next tile; a claim is ONE fetch-and-add on
//     it, valid only if the word still carried the entry's tag and tiles were left;
//   * a stage is armed (tag_next := tag << 32) before its entry is published;
//   * link stages are taken only under one of the lane's `cap` slots;
//   * the host mirror's write order (end time before count; running before gen).
// Everything else here is this library's own: the scheduler is a whole warp that
// probes up to 32 ring entries at once, drops a run of exhausted head entries with a
// single compare-and-swap, walks a visiting order computed once per epoch, and sizes
// claims for a 148-SM machine; completion releases a stage's successors 32 at a time.
//
// A stage that does next to nothing is a chain of round trips to the L2 (0.7 us each): from the count that completes it
// to its successor's published word, and from there through a worker's reading of the rings, its claim, the tile and its
// operands.  The polling of an idle worker is one load of all words it depends on, and what a step of the chain does not need from
// the one before it goes out beside it.  From publish to the end of the pass, a step of 39 stages (Teganex, 32 sequences) 1014 -> 862
// us, of 57 stages (a mixture-of-experts decoder, 32 sequences) 2478 -> 2217.  Polls without a back-off beside another lane cost it nothing
// that shows: 128 sequences decoded beside prompts of 4 x 2048 tokens, four layers, all experts in HBM, with a back-off of 4 us and with
// none: 8.2 and 8.2 ms a step, 14.3 and 13.1 ms a prompt pass; half of the experts in host memory 60.5 and 62.5, 242 and 209.
#pragma once
#include <cstddef>

#include "fabric_types.h"
#include "ptx.cuh"

namespace mf {
namespace fab {

constexpr uint32_t kStageBits = 20;
constexpr uint32_t kStageMask = (1u << kStageBits) - 1;
constexpr uint32_t kTagMask = 0xfffu;
constexpr int kWorklistCap = 448;   // bounded by the worker's shared memory; an overflow is reported, not fatal
// A claim takes about 1/256 of what is left of a stage, at least one tile and at most
// eight: with one worker per SM the first round over a large stage hands out eights,
// and the tail is shared out tile by tile so that the workers finish together.
constexpr uint32_t kClaimMax = 8;
constexpr uint32_t kClaimShareLog2 = 8;
constexpr unsigned long long kRingWaitBudgetNs = 2000000000ull;
constexpr unsigned kWarp = 0xffffffffu;

enum : uint32_t { kCmdRun = 0, kCmdIdle = 1, kCmdExit = 2 };

template <class T>
__device__ __forceinline__ T ld_volatile(const T* p) { return *reinterpret_cast<const volatile T*>(p); }
__device__ __forceinline__ unsigned int ld_acq(const unsigned int* p) { return ld_acquire_gpu(p); }
__device__ __forceinline__ unsigned long long ld_acq(const unsigned long long* p) { return ld_acquire_gpu64(p); }
// The count before one is taken off; what the threads that took the others off had written, or knew of, is known here behind it.
__device__ __forceinline__ unsigned int take_one_acq(unsigned int* p) {
  unsigned int before;
  asm volatile("atom.acquire.gpu.global.add.u32 %0, [%1], %2;" : "=r"(before) : "l"(p), "r"(0xffffffffu) : "memory");
  return before;
}
__device__ __forceinline__ void st_rel(unsigned int* p, unsigned int v) { st_release_gpu(p, v); }
__device__ __forceinline__ void st_rel(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void raise_error(DeviceState& S, unsigned long long bit) {
  const unsigned long long now = atomicOr(&S.error, bit) | bit;
  if (S.mirror) st_release_sys64(&S.mirror->error, now);   // pinned host memory
}

__device__ __forceinline__ void trace_stage(DeviceState& S, uint32_t lane, uint32_t s, uint32_t event, uint32_t tag) {
  const uint32_t cap = ld_volatile(&S.trace_cap);
  if (cap == 0) return;
  const uint32_t i = atomicAdd(&S.trace_n, 1u);
  if (i >= cap) return;
  unsigned long long* r = reinterpret_cast<unsigned long long*>(ld_volatile(&S.trace_ptr)) + 2ull * i;
  r[0] = static_cast<unsigned long long>(s) | (static_cast<unsigned long long>(lane) << 32) |
         (static_cast<unsigned long long>(event) << 40) | (static_cast<unsigned long long>(tag & kTagMask) << 48);
  r[1] = globaltimer_ns();
}

enum MirrorField { kMirrorIterations, kMirrorGen, kMirrorRunning, kMirrorMark };
__device__ __forceinline__ void mirror_lane(DeviceState& S, uint32_t lane, MirrorField what, unsigned long long v) {
  if (!S.mirror) return;
  LaneMirror& m = S.mirror->lane[lane];
  if (what == kMirrorIterations) st_release_sys64(&m.iterations, v);
  else if (what == kMirrorGen) st_release_sys64(&m.gen, v);
  else if (what == kMirrorRunning) st_release_sys64(&m.running, v);
  else {
    st_release_sys64(&m.mark_ns, globaltimer_ns());   // the time is there before the mark that announces it
    st_release_sys64(&m.mark, v);
  }
}

// ------------------------------------------------------------------ wire words
struct StageWord {   // decoded StageRuntime::tag_next
  uint32_t tag, next;
  __device__ explicit StageWord(unsigned long long w) : tag(static_cast<uint32_t>(w >> 32) & kTagMask), next(static_cast<uint32_t>(w)) {}
};
__device__ __forceinline__ uint32_t ring_word(uint32_t stage, uint32_t tag) {
  return ((tag & kTagMask) << kStageBits) | (stage & kStageMask);
}
__device__ __forceinline__ unsigned long long armed_word(uint32_t tag) {
  return static_cast<unsigned long long>(tag & kTagMask) << 32;
}

// Completed stages a releasing warp still has to process (shared memory; lane 0 owns it).
template <int kCap>
struct WorklistOf {
  uint32_t v[kCap];
  int n;
  bool overflow;
  __device__ void clear() { n = 0; overflow = false; }
  __device__ void push(uint32_t s) {
    if (n < kCap) v[n++] = s; else overflow = true;
  }
  __device__ uint32_t pop() { return v[--n]; }
};
using Worklist = WorklistOf<kWorklistCap>;
using SmallWorklist = WorklistOf<16>;   // the scheduler's: it only ever releases the empty stages at a program's start

// ---------------------------------------------------------------------- rings
// Producer side, any one thread: move the published tail over the m places at `at`, which are filled, once every
// earlier reservation has been published (next: that is known already).  The wait for earlier producers is
// bounded; if it runs out the entries stay unpublished and the host sees kFabErrRingWait.
__device__ __forceinline__ void ring_announce(DeviceState& S, Ring& R, unsigned long long at, int m, bool next) {
  if (!next) {
    const unsigned long long give_up = globaltimer_ns() + kRingWaitBudgetNs;
    for (unsigned int pause = 32; ld_acq(&R.tail) != at; pause = pause < 512 ? pause * 2 : pause) {
      __nanosleep(pause);
      if (globaltimer_ns() > give_up) {
        raise_error(S, kFabErrRingWait);
        return;
      }
    }
  }
  st_rel(&R.tail, at + m);
}
// One word.
__device__ __forceinline__ void ring_publish(DeviceState& S, Ring& R, uint32_t word) {
  const unsigned long long at = atomicAdd(&R.reserve, 1ull);
  R.ids[at & (kRingCap - 1)] = word;
  ring_announce(S, R, at, 1, false);
}

// ---------------------------------------------------------------------- claims
// The tables of a program as a worker keeps them: the descriptor itself does not change while a lane runs it.
struct ProgView {
  const ProgramDesc* prog;
  StageStatic* stages;
  StageRuntime* runtime;
  const TileDesc* tiles;
  const uint32_t* succ;
  uint32_t n_stages, gen;
};
// The WHOLE warp.  gen: of the lane, which is new for every program it is given (an address may come back).
__device__ __forceinline__ void view_program(ProgView& v, const ProgramDesc* P, uint32_t gen) {
  if (v.prog == P && v.gen == gen) return;
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    v.stages = ld_volatile(&P->stages);
    v.runtime = ld_volatile(&P->runtime);
    v.tiles = ld_volatile(&P->tiles);
    v.succ = ld_volatile(&P->succ);
    v.n_stages = ld_volatile(&P->n_stages);
    v.prog = P;
    v.gen = gen;
  }
  __syncwarp();
}

// What a work record keeps of it.
struct ProgTables {
  const ProgramDesc* prog;
  StageStatic* stages;
  StageRuntime* runtime;
  const uint32_t* succ;
};

struct Claim {
  uint32_t stage, first_tile, n;
};
// What a probe of a ring entry found; left = 0: its stage has moved on to another activation or has been handed out.
struct Probe {
  uint32_t left, first, count;
};

__device__ __forceinline__ uint2 stage_tiles(const StageStatic* st) {   // (first, count) by one load
  const unsigned long long v = ld_volatile(reinterpret_cast<const unsigned long long*>(st));
  return make_uint2(static_cast<uint32_t>(v), static_cast<uint32_t>(v >> 32));
}

// A read-only probe; the claim itself re-checks.  The two loads may be answered in either order: a stage's tiles change only
// while it is closed (tag 0), which the claim sees.
__device__ __forceinline__ Probe probe_entry(const ProgView& V, uint32_t word) {
  Probe p{0, 0, 0};
  const uint32_t s = word & kStageMask;
  if (s >= V.n_stages) return p;
  const unsigned long long tn = ld_volatile(&V.runtime[s].tag_next);
  const uint2 t = stage_tiles(V.stages + s);
  const StageWord w(tn);
  p.first = t.x;
  p.count = t.y;
  if (w.tag == (word >> kStageBits) && w.next < p.count) p.left = p.count - w.next;
  return p;
}

// The fetch-and-add.  `left` is the probe's answer and only sizes the claim.
__device__ __forceinline__ bool claim_tiles(const ProgView& V, uint32_t word, Probe p, Claim& c) {
  const uint32_t s = word & kStageMask;
  uint32_t want = p.left >> kClaimShareLog2;
  want = want < 1 ? 1 : (want > kClaimMax ? kClaimMax : want);
  const StageWord before(atomicAdd(&V.runtime[s].tag_next, static_cast<unsigned long long>(want)));
  // The add may land on a later activation of the stage (or on a stage that was closed, tag 0).
  // On a later activation it hands out that activation's tiles, which is as good; on a closed
  // stage, or past the end, it hands out nothing and the overshoot is harmless: `next` is only
  // ever compared with the count.
  if (before.tag == 0) return false;
  if (before.tag != (word >> kStageBits)) {   // a later activation: its stage record may be newer than the probe saw
    __threadfence();
    const uint2 t = stage_tiles(V.stages + s);
    p.first = t.x;
    p.count = t.y;
  }
  if (before.next >= p.count) return false;
  c.stage = s;
  c.first_tile = p.first + before.next;
  c.n = min(want, p.count - before.next);
  return true;
}

// Consumer side, the WHOLE warp: lane i probes entry head + i; a run of exhausted entries at the
// head is dropped with one compare-and-swap; the first entry that still has tiles is claimed.
// head and tail come from one reading of both: a pair out of step only looks empty, or begins at
// entries that are exhausted and fail the compare-and-swap.  V comes from the same reading, whose words are not ordered among
// themselves: against the tables of a program that the lane ran before, entries of the one it runs now would pass for exhausted.
// Entries are dropped only where the lane's program, read behind the tail, is still V's.
__device__ __forceinline__ bool ring_take(const LaneState& L, Ring& R, unsigned long long head, unsigned long long tail, const ProgView& V, Claim& c) {
  const int lane = threadIdx.x & 31;
  if (tail <= head) return false;
  const int n = static_cast<int>(min(tail - head, 32ull));
  uint32_t word = 0;
  Probe p{0, 0, 0};
  unsigned long long prog = 0;
  uint32_t gen = 0;
  if (lane == 0) {   // beside the entries
    prog = ld_volatile(&L.prog);
    gen = ld_volatile(&L.gen);
  }
  if (lane < n) {
    word = ld_volatile(&R.ids[(head + lane) & (kRingCap - 1)]);
    p = probe_entry(V, word);
  }
  unsigned live = __ballot_sync(kWarp, p.left != 0);
  const int spent = live ? __ffs(live) - 1 : n;   // exhausted entries in front of the first live one
  if (spent > 0 && lane == 0 && prog == reinterpret_cast<unsigned long long>(V.prog) && gen == V.gen) atomicCAS(&R.head, head, head + spent);   // losing the race is fine: someone else dropped them
  while (live) {
    const int src = __ffs(live) - 1;
    live &= live - 1;
    int ok = 0;
    if (lane == src) ok = claim_tiles(V, word, p, c);
    ok = __shfl_sync(kWarp, ok, src);
    if (ok) {
      c.stage = __shfl_sync(kWarp, c.stage, src);
      c.first_tile = __shfl_sync(kWarp, c.first_tile, src);
      c.n = __shfl_sync(kWarp, c.n, src);
      return true;
    }
  }
  return false;
}

// -------------------------------------------------------- iterations of a lane
// The program a lane should be running according to the latest published plan.
__device__ __forceinline__ void planned_program(DeviceState& S, uint32_t lane, ProgramDesc*& prog, uint32_t& gen) {
  for (unsigned long long e = ld_acq(&S.published);;) {
    const Snapshot& sn = S.snap[e & 1];
    prog = ld_volatile(&sn.prog[lane]);
    gen = ld_volatile(&sn.prog_gen[lane]);
    const unsigned long long again = ld_acq(&S.published);   // the snapshot is double-buffered: re-read if a publish intervened
    if (again == e) return;
    e = again;
  }
}

// Arm stage s for activation `tag`.  Returns true if it has tiles (the caller publishes its ring
// word), false if it is empty and therefore complete at once (pushed on the worklist).
template <class WL>
__device__ __forceinline__ bool arm_stage(DeviceState& S, uint32_t lane, const ProgramDesc* P, uint32_t s, uint32_t tag,
                                          WL& wl) {
  trace_stage(S, lane, s, 0, tag);
  if (ld_volatile(&P->stages[s].count) == 0) {
    wl.push(s);
    return false;
  }
  atomicExch(&P->runtime[s].tag_next, armed_word(tag));
  return true;
}

// One thread.  Opens the next activation wave of a lane's program: a new tag (never 0) and the
// program's first stage.  `switched`: P is not the program the lane ran before.
template <class WL>
__device__ __forceinline__ void open_wave(DeviceState& S, uint32_t lane, const ProgramDesc* P, uint32_t gen, bool switched,
                                          WL& wl) {
  LaneState& L = S.lane[lane];
  if (switched) {
    for (Ring& R : L.ring) atomicExch(&R.head, ld_acq(&R.tail));   // what is left in the rings belongs to the old program
    L.iter_in_prog = 0;
    st_rel(&L.prog, reinterpret_cast<unsigned long long>(P));
    st_rel(&L.gen, gen);
    mirror_lane(S, lane, kMirrorGen, gen);
  }
  uint32_t tag = (ld_volatile(&L.tag) + 1) & kTagMask;
  if (tag == 0) tag = 1;
  st_rel(&L.tag, tag);
  const uint32_t s = P->first_stage;
  if (arm_stage(S, lane, P, s, tag, wl)) {
    ring_publish(S, L.ring[(ld_volatile(&P->stages[s].flags) & kStageLink) ? 1 : 0], ring_word(s, tag));
  }
}

// One thread.  The reset stage completed: count the iteration, then switch to a newer program,
// stop after the program's last iteration, or go round again.  Returns the program now current.
template <class WL>
__device__ __forceinline__ const ProgramDesc* close_iteration(DeviceState& S, uint32_t lane, const ProgramDesc* P, WL& wl) {
  LaneState& L = S.lane[lane];
  StageRuntime& reset = P->runtime[P->reset_stage];   // the reset tiles re-armed every stage but their own
  reset.done = 0;
  reset.deps = ld_volatile(&P->stages[P->reset_stage].deps_init);
  const uint32_t done_iterations = ++L.iter_in_prog;
  if (S.mirror) {
    st_release_sys64(&S.mirror->lane[lane].iter_ns, globaltimer_ns());
    mirror_lane(S, lane, kMirrorIterations, ld_volatile(&S.mirror->lane[lane].iterations) + 1);
  }
  ProgramDesc* wanted;
  uint32_t wanted_gen;
  planned_program(S, lane, wanted, wanted_gen);
  if (wanted != nullptr && wanted_gen != ld_volatile(&L.gen)) {
    open_wave(S, lane, wanted, wanted_gen, true, wl);
    return wanted;
  }
  if (P->iterations != 0 && done_iterations >= P->iterations) {
    st_rel(&L.running, 0u);
    mirror_lane(S, lane, kMirrorRunning, 0);
    return P;
  }
  open_wave(S, lane, P, ld_volatile(&L.gen), false, wl);
  return P;
}

// The WHOLE warp.  Counts down and arms the successors succ[first ..) of a completed stage, the 32 lanes side by side, and
// publishes their ring words in two publications (ungated, link), so a stage with 128 successors releases them in a few
// microseconds.  Each step is a round trip to the L2 that every stage of a program waits for, so what does not depend
// on one another goes out together: the record of a successor beside its count, unless a tile of the program writes that record
// (kSuccLate) and may do so ahead of another predecessor than this one (kSuccJoin); then it is read behind the count.
template <class WL>
__device__ __forceinline__ void release_stage(DeviceState& S, uint32_t lane_id, StageStatic* stages, StageRuntime* runtime,
                                              const uint32_t* succs, uint32_t first, uint32_t count, uint32_t tag, bool tracing, WL& wl) {
  const int lane = threadIdx.x & 31;
  LaneState& L = S.lane[lane_id];
  for (uint32_t base = 0; base < count; base += 32) {
    enum { kNone, kUngated, kLink, kEmpty };
    int fate = kNone;
    uint32_t word = 0, succ = 0;
    if (base + lane < count) {
      const uint32_t entry = ld_volatile(succs + first + base + lane);
      succ = entry & kStageMask;
      // a skipped stage keeps its count: one taken off late would be missed by the next iteration, whose end does not wait for it
      uint32_t skip = 0;
      if (entry & kSuccLate) skip = ld_volatile(&stages[succ].flags) & kStageSkip;
      uint32_t flags = ld_volatile(&stages[succ].flags), tiles = ld_volatile(&stages[succ].count);
      const unsigned int before = skip ? 0u : take_one_acq(&runtime[succ].deps);
      if (before == 1u && (entry & kSuccLate) && (entry & kSuccJoin)) {
        flags = ld_volatile(&stages[succ].flags);
        tiles = ld_volatile(&stages[succ].count);
      }
      if (before == 1u && !(flags & kStageSkip)) {
        if (tracing) trace_stage(S, lane_id, succ, 0, tag);
        if (tiles == 0) {
          fate = kEmpty;
        } else {
          atomicExch(&runtime[succ].tag_next, armed_word(tag));
          word = ring_word(succ, tag);
          fate = (flags & kStageLink) ? kLink : kUngated;
        }
      }
    }
#pragma unroll
    for (int want = kUngated; want <= kLink; ++want) {
      const unsigned mask = __ballot_sync(kWarp, fate == want);
      if (mask == 0) continue;
      Ring& R = L.ring[want == kLink ? 1 : 0];
      unsigned long long got = 0;
      if (lane == 0) got = atomicAdd(&R.reserve, static_cast<unsigned long long>(__popc(mask)));
      else if (lane == 1) got = ld_acq(&R.tail);   // the earlier publishers' entries go on with the release behind it
      const unsigned long long at = __shfl_sync(kWarp, got, 0), tail = __shfl_sync(kWarp, got, 1);
      if (fate == want) R.ids[(at + __popc(mask & ((1u << lane) - 1))) & (kRingCap - 1)] = word;
      __syncwarp();   // the stages' tags and words, by all lanes, are in front of lane 0's release
      if (lane == 0) ring_announce(S, R, at, __popc(mask), tail == at);
    }
    const unsigned empty = __ballot_sync(kWarp, fate == kEmpty);
    if (empty) __threadfence();   // what was acquired above goes on with the counts that these stages' completion takes from
    for (unsigned mask = empty; mask; mask &= mask - 1) {
      const uint32_t v = __shfl_sync(kWarp, succ, __ffs(mask) - 1);
      if (lane == 0) wl.push(v);
    }
  }
}

// The WHOLE warp.  Processes the worklist: for every completed stage, lane 0 reports marks and
// handles the iteration boundary; then its successors are released.
template <class WL>
__device__ __forceinline__ void release_successors(DeviceState& S, uint32_t lane_id, const ProgramDesc* P, WL& wl) {
  const int lane = threadIdx.x & 31;
  LaneState& L = S.lane[lane_id];
  for (;;) {
    uint32_t first = 0, count = 0, tag = 0;
    int have = 0;
    if (lane == 0) {
      while (wl.n > 0 && !have) {
        const uint32_t s = wl.pop();
        trace_stage(S, lane_id, s, 1, ld_volatile(&L.tag));
        const StageStatic& st = P->stages[s];
        const uint32_t flags = ld_volatile(&st.flags);
        if (flags & kStageMark) mirror_lane(S, lane_id, kMirrorMark, ld_volatile(&st.mark));
        if (flags & kStageReset) {
          P = close_iteration(S, lane_id, P, wl);
        } else {
          tag = ld_volatile(&L.tag) & kTagMask;
          first = ld_volatile(&st.succ_first);
          count = ld_volatile(&st.succ_count);
          have = 1;
        }
      }
    }
    if (!__shfl_sync(kWarp, have, 0)) break;
    first = __shfl_sync(kWarp, first, 0);
    count = __shfl_sync(kWarp, count, 0);
    tag = __shfl_sync(kWarp, tag, 0);
    const ProgramDesc* Pw = reinterpret_cast<const ProgramDesc*>(__shfl_sync(kWarp, reinterpret_cast<unsigned long long>(P), 0));
    release_stage(S, lane_id, Pw->stages, Pw->runtime, Pw->succ, first, count, tag, true, wl);
  }
  if (lane == 0 && wl.overflow) raise_error(S, kFabErrWorklist);
}

// The WHOLE warp.  n tiles of stage s are done; the warp whose tiles complete the stage releases
// its successors.  What that takes of the stage's record is loaded beside the count.
__device__ __forceinline__ void tiles_completed(DeviceState& S, uint32_t lane_id, const ProgTables& V, uint32_t s, uint32_t n, Worklist& wl) {
  int last = 0;
  uint32_t count = 0, first = 0, n_succ = 0, flags = 0, tag = 0, tracing = 0;
  if ((threadIdx.x & 31) == 0) {
    const unsigned int done = atomicAdd(&V.runtime[s].done, n) + n;
    const StageStatic* st = V.stages + s;
    count = ld_volatile(&st->count);
    first = ld_volatile(&st->succ_first);
    n_succ = ld_volatile(&st->succ_count);
    flags = ld_volatile(&st->flags);
    tag = ld_volatile(&S.lane[lane_id].tag);
    tracing = ld_volatile(&S.trace_cap);
    last = done == count;
  }
  if (!__shfl_sync(kWarp, last, 0)) return;
  __threadfence();   // the other workers' tiles of the stage are visible before its successors start
  const bool plain = !(__shfl_sync(kWarp, flags, 0) & (kStageMark | kStageReset));
  if ((threadIdx.x & 31) == 0) {
    wl.clear();
    if (!plain) wl.push(s);
    else if (tracing) trace_stage(S, lane_id, s, 1, tag);
  }
  __syncwarp();
  if (plain)
    release_stage(S, lane_id, V.stages, V.runtime, V.succ, __shfl_sync(kWarp, first, 0), __shfl_sync(kWarp, n_succ, 0),
                  __shfl_sync(kWarp, tag, 0) & kTagMask, __shfl_sync(kWarp, tracing, 0) != 0, wl);
  __syncwarp();
  release_successors(S, lane_id, V.prog, wl);
}

// ------------------------------------------------------------------ the worker
// Scheduling state of one worker (shared memory).  Written by lane 0 of the scheduler warp
// between warp barriers; the link accounting is also read by the completing exec thread.
struct WorkerState {
  unsigned long long epoch;
  uint32_t worker, lane, n_lanes, idle_ns;
  uint32_t cap[kMaxLanes], prog_gen[kMaxLanes];
  ProgramDesc* prog_snap[kMaxLanes];
  uint32_t visit[kMaxLanes];   // lanes in the order this worker looks for work: its own, then the borrowing order
  uint32_t n_visit;
  ProgView view;               // of the program looked at last
  uint32_t idle, polls;        // the last round found nothing; rounds that found nothing, ever
  // the current claim
  ProgTables prog;
  const TileDesc* tiles;
  uint32_t stage, tile_lane, link, next_index, left;
  uint32_t row_block;   // a kind-45 tile runs as one record per row block: the block of its next record
  // The link slot this worker holds (kNoLane = none).  The worker runs its records through a pipeline
  // behind the scheduler, so the slot goes back only when the exec warps have finished the last link
  // record issued under it.
  uint32_t slot_lane;
  uint32_t link_last;                  // records issued up to and including the last link record
  const volatile unsigned int* done;   // records the exec warps have finished
};

// Lane 0 of the scheduler warp.
__device__ __forceinline__ void give_slot_back(DeviceState& S, WorkerState& ws) {
  if (ws.slot_lane == kNoLane) return;
  if (ws.done) {   // bounded: after a second the slot goes back regardless (the fabric is stuck or stopping)
    const unsigned long long give_up = globaltimer_ns() + 1000000000ull;
    while (static_cast<int>(*ws.done - ws.link_last) < 0 && globaltimer_ns() < give_up) __nanosleep(64);
  }
  atomicSub(&S.lane[ws.slot_lane].slots, 1u);
  ws.slot_lane = kNoLane;
}

__device__ __forceinline__ bool take_slot(LaneState& L, uint32_t cap) {
  for (unsigned int held = ld_volatile(&L.slots); held < cap;) {
    const unsigned int seen = atomicCAS(&L.slots, held, held + 1);
    if (seen == held) return true;
    held = seen;
  }
  return false;
}

// The WHOLE scheduler warp.  Adopt a newer published plan: lane l < 4 reads lane l's share of the
// snapshot, lane 0 the rest; the read is repeated if a publish intervened.
__device__ __forceinline__ void adopt_epoch(DeviceState& S, WorkerState& ws) {
  const int lane = threadIdx.x & 31;
  unsigned long long e = 0;
  if (lane == 0) e = ld_acq(&S.published);
  e = __shfl_sync(kWarp, e, 0);
  if (e == ws.epoch) return;
  __shared__ uint32_t s_order[kMaxLanes];
  for (;;) {
    const Snapshot& sn = S.snap[e & 1];
    if (lane < kMaxLanes) {
      ws.cap[lane] = ld_volatile(&sn.cap[lane]);
      s_order[lane] = ld_volatile(&sn.order[lane]);
      ws.prog_gen[lane] = ld_volatile(&sn.prog_gen[lane]);
      ws.prog_snap[lane] = ld_volatile(&sn.prog[lane]);
    }
    if (lane == 0) {
      ws.n_lanes = min(ld_volatile(&sn.n_lanes), static_cast<uint32_t>(kMaxLanes));
      ws.lane = ld_volatile(&sn.map[ws.worker]);
    }
    unsigned long long again = 0;
    if (lane == 0) again = ld_acq(&S.published);
    again = __shfl_sync(kWarp, again, 0);
    if (again == e) break;
    e = again;
  }
  __syncwarp();
  if (lane == 0) {
    ws.n_visit = 0;
    if (ws.lane < ws.n_lanes) ws.visit[ws.n_visit++] = ws.lane;
    for (uint32_t i = 0; i < ws.n_lanes; ++i)
      if (s_order[i] != ws.lane && s_order[i] < kMaxLanes) ws.visit[ws.n_visit++] = s_order[i];
    ws.epoch = e;
    if (S.mirror) {
      st_release_sys64(&S.mirror->worker_epoch_ns[ws.worker], globaltimer_ns());
      st_release_sys64(&S.mirror->worker_epoch[ws.worker], e);
    }
  }
  __syncwarp();
}

// The WHOLE scheduler warp.  A lane whose planned program is not the one it runs, and that is not
// running, is started by whichever worker gets there first.
__device__ __forceinline__ void start_waiting_lanes(DeviceState& S, WorkerState& ws, SmallWorklist& wl) {
  const int lane = threadIdx.x & 31;
  for (uint32_t l = 0; l < ws.n_lanes; ++l) {
    int mine = 0;
    ProgramDesc* P = ws.prog_snap[l];
    if (lane == 0 && P != nullptr) {
      LaneState& L = S.lane[l];
      if (ws.prog_gen[l] != ld_acq(&L.gen) && ld_acq(&L.running) == 0 && atomicCAS(&L.running, 0u, 1u) == 0u) {
        mirror_lane(S, l, kMirrorRunning, 1);
        wl.clear();
        open_wave(S, l, P, ws.prog_gen[l], true, wl);
        mine = 1;
      }
    }
    if (__shfl_sync(kWarp, mine, 0)) release_successors(S, l, P, wl);   // an empty first stage completes at once
  }
}

// The words a round of scheduling depends on, one for each lane of the scheduler warp: lanes 7 l .. 7 l + 6 read lane l's
// published tails (ungated, link), held link slots, running flag, generation, ungated head and program; lane 30 the
// published epoch, lane 31 the shutdown flag (low half) and the idle cap.  One load instead of a chain of them: an idle
// worker sees a new stage a round trip after it is published, and has its ring's ends and program in hand.
constexpr int kWordsPerLane = 7, kEpochLane = 30, kStopLane = 31;
static_assert(kWordsPerLane * kMaxLanes <= kEpochLane, "one word for each lane of a warp");
static_assert(offsetof(LaneState, slots) % 8 == 0 && offsetof(LaneState, inflight_max) % 8 == 0 && offsetof(LaneState, gen) % 8 == 0 &&
              offsetof(LaneState, running) == offsetof(LaneState, inflight_max) + 4 && offsetof(DeviceState, shutdown) % 8 == 0 &&
              offsetof(DeviceState, idle_cap) == offsetof(DeviceState, shutdown) + 4, "pairs read as one word");
enum { kWTail, kWLinkTail, kWSlots, kWRunning, kWGen, kWHead, kWProg };
__device__ __forceinline__ const unsigned long long* polled_word(DeviceState& S, int lane) {
  if (lane == kEpochLane) return &S.published;
  if (lane == kStopLane) return reinterpret_cast<const unsigned long long*>(&S.shutdown);
  if (lane >= kWordsPerLane * kMaxLanes) return nullptr;
  LaneState& L = S.lane[lane / kWordsPerLane];
  switch (lane % kWordsPerLane) {
    case kWTail: return &L.ring[0].tail;
    case kWLinkTail: return &L.ring[1].tail;
    case kWSlots: return reinterpret_cast<const unsigned long long*>(&L.slots);
    case kWRunning: return reinterpret_cast<const unsigned long long*>(&L.inflight_max);
    case kWGen: return reinterpret_cast<const unsigned long long*>(&L.gen);
    case kWHead: return &L.ring[0].head;
    default: return &L.prog;
  }
}

// The WHOLE scheduler warp.  Look for tiles in lane l: link stages first, under a slot; then the
// ungated ring.  On success the claim is in ws (written by lane 0).
__device__ __forceinline__ bool look_in_lane(DeviceState& S, WorkerState& ws, uint32_t l, unsigned long long words) {
  const int lane = threadIdx.x & 31;
  LaneState& L = S.lane[l];
  auto word = [&](int which) { return __shfl_sync(kWarp, words, l * kWordsPerLane + which); };
  const unsigned long long running = word(kWRunning), tail = word(kWTail), link_tail = word(kWLinkTail), gen = word(kWGen),
                           head = word(kWHead), prog = word(kWProg);
  if (!running || !prog) return false;
  unsigned long long link_head = 0;
  if (link_tail) {
    if (lane == 0) link_head = ld_volatile(&L.ring[1].head);
    link_head = __shfl_sync(kWarp, link_head, 0);
  }
  if (tail <= head && link_tail <= link_head) return false;
  ProgView& V = ws.view;
  view_program(V, reinterpret_cast<const ProgramDesc*>(prog), static_cast<uint32_t>(gen));
  auto took = [&](const Claim& c, uint32_t link) {
    if (lane == 0) {
      ws.prog = ProgTables{V.prog, V.stages, V.runtime, V.succ}; ws.tiles = V.tiles; ws.stage = c.stage; ws.tile_lane = l; ws.link = link; ws.next_index = c.first_tile; ws.left = c.n;
    }
  };
  Claim c;
  if (link_tail > link_head) {
    int held = 0;
    if (lane == 0) {
      held = ws.slot_lane == l;
      if (held && ld_volatile(&L.slots) > ws.cap[l]) {   // the grant shrank under this worker
        give_slot_back(S, ws);
        held = 0;
      }
      if (!held) {
        give_slot_back(S, ws);   // a slot of another lane
        if (take_slot(L, ws.cap[l])) {
          ws.slot_lane = l;
          held = 1;
        }
      }
    }
    if (__shfl_sync(kWarp, held, 0)) {
      if (ring_take(L, L.ring[1], link_head, link_tail, V, c)) {
        took(c, 1);
        return true;
      }
      if (lane == 0) give_slot_back(S, ws);
    }
  }
  if (!ring_take(L, L.ring[0], head, tail, V, c)) return false;
  if (lane == 0) give_slot_back(S, ws);
  took(c, 0);
  return true;
}

// The WHOLE scheduler warp.  One scheduling round: kCmdRun with a claim in ws, kCmdExit when the
// host asked the fabric to stop, or kCmdIdle.  `at` is this lane's polled word, `seen` what it was in the last round: a round in
// which no word has changed since one that found nothing is only the reading of the words.  The back-off grows to the idle cap, and
// while a lane runs, to 1/128 of it, which by default is none to speak of (a stage is over in microseconds).
constexpr uint32_t kBusyCapLog2 = 7;
__device__ __forceinline__ uint32_t schedule(DeviceState& S, WorkerState& ws, SmallWorklist& wl, const unsigned long long* at,
                                             unsigned long long& seen) {
  const int lane = threadIdx.x & 31, which = lane % kWordsPerLane;
  const bool of_lane = lane < kWordsPerLane * kMaxLanes;
  const uint32_t n_lanes = ws.n_lanes;
  unsigned long long words = 0;
  if (lane >= kEpochLane || (of_lane && lane / kWordsPerLane < n_lanes)) words = ld_acq(at);
  __syncwarp();
  if (of_lane && (which == kWSlots || which == kWGen)) words &= 0xffffffffull;
  if (of_lane && which == kWRunning) words >>= 32;
  const bool changed = __any_sync(kWarp, words != seen && !(of_lane && which == kWHead));
  auto idle = [&](bool found_nothing, bool more = false) {
    const bool busy = __any_sync(kWarp, of_lane && which == kWRunning && words != 0);
    const uint32_t cap = max(64u, static_cast<uint32_t>(__shfl_sync(kWarp, words, kStopLane) >> 32)), most = busy ? max(32u, cap >> kBusyCapLog2) : cap;
    if (lane == 0) {
      ws.idle = found_nothing && !more;
      ++ws.polls;
      if (found_nothing) {
        __nanosleep(min(ws.idle_ns, most));
        ws.idle_ns = min(ws.idle_ns * 2, most);
      }
    }
    __syncwarp();
    return kCmdIdle;
  };
  if (ws.idle && !changed) return idle(true);
  seen = words;
  if (static_cast<uint32_t>(__shfl_sync(kWarp, words, kStopLane)) != 0) {
    if (lane == 0) give_slot_back(S, ws);
    return kCmdExit;
  }
  if (__shfl_sync(kWarp, words, kEpochLane) != ws.epoch) {
    adopt_epoch(S, ws);
    return idle(false);   // the words of the plan's lanes are read next
  }
  const unsigned long long running = __shfl_up_sync(kWarp, words, kWGen - kWRunning);
  const uint32_t l = lane / kWordsPerLane;
  const bool starts = of_lane && which == kWGen && l < n_lanes && running == 0 && ws.prog_snap[l] != nullptr &&
                      ws.prog_gen[l] != static_cast<uint32_t>(words);
  if (__any_sync(kWarp, starts)) {
    start_waiting_lanes(S, ws, wl);
    __syncwarp();
    return idle(false);
  }
  const uint32_t n_visit = ws.n_visit;
  for (uint32_t i = 0; i < n_visit; ++i) {
    if (ws.visit[i] >= n_lanes) continue;
    if (look_in_lane(S, ws, ws.visit[i], words)) {
      if (lane == 0) {
        ws.idle_ns = 64;
        ws.idle = 0;
      }
      __syncwarp();
      return kCmdRun;
    }
  }
  if (lane == 0) give_slot_back(S, ws);
  // Entries past the 32 that were probed, and link stages (whose ring's head and slots are read apart), are looked at again.
  const unsigned long long head = __shfl_down_sync(kWarp, words, kWHead - kWTail);
  const bool more = of_lane && ((which == kWTail && words > head + 32) || (which == kWLinkTail && words != 0));
  return idle(true, __any_sync(kWarp, more));
}

}  // namespace fab
}  // namespace mf
