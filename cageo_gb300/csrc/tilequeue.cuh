// tilequeue.cuh -- the asynchronous tile work queue of the persistent
// relaxation kernels (the pit fill's floods and the flat-surface BFS).
//
// Tiles are processed as soon as they are queued, by whichever warp is free:
// no grid-wide pass barriers.  Both users run monotone relaxations (values
// only fall), so the order of the updates does not change their limit; what
// must not happen is two warps processing one tile at once (a slower warp's
// write-back could undo a faster one's lower values).  Each tile therefore
// has a state: idle, queued, processing, processing and queued again
// meanwhile (re-queued when its processing ends).  The ring (cap slots, -1 =
// empty) holds each queued tile once, so cap = 2 * tiles + the tickets warps
// may hold ahead of the pushes (kRingSlack > warps in flight) never overflows.
//
// The queue is drained when as many tiles have been finished as were ever
// pushed: a tile is pushed by a warp that has not finished its own yet, so
// reading `done` first and `tail` after it and finding them equal means that
// no tile was queued or in process at the first read (a fence lies between a
// warp's pushes and its addition to `done`: a warp that saw the latter without
// the former would leave with a ticket that a later push fills).  Warps add their
// finished tiles to `done` only when they find no tile waiting, and a warp
// pushes all the neighbours of a visit with one addition to `tail`: two
// same-address atomics a visit, against five with a counter of pending tiles
// (the fill's flood 1.09 -> 1.07 ms at 8192^2).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace cageo {

enum : int { kIdle = 0, kQueued = 1, kBusy = 2, kBusyQueued = 3 };
constexpr int kEmptySlot = -1;
constexpr int kRingSlack = 8192;

struct TileQueue {
  int* state;              // per tile
  int* ring;               // cap slots
  unsigned int cap;
  unsigned int* head;      // tickets handed out (own 128-byte line)
  unsigned int* tail;      // entries pushed (own line)
  unsigned int* done;      // tiles finished (own line)
  int* err;                // set to 3 when a state change keeps failing
};

// A plain store: the taker swaps the slot for "empty" and retries while it
// reads empty.
__device__ __forceinline__ void tq_store(const TileQueue& q, unsigned int pos, int t) {
  ((volatile int*)q.ring)[pos % q.cap] = t;
}

// The whole warp: each lane with `want` queues its tile t, unless it is queued
// already: idle -> queued, processing -> processing and queued again
// (its owner pushes it then).  A single compare-and-swap when the state is the
// one expected.
__device__ __forceinline__ void tq_enqueue(const TileQueue& q, bool want, int t) {
  bool push = false;
  if (want) {
    int expect = kIdle;
    bool settled = false;
    for (int it = 0; it < 256 && !settled; it++) {
      const int old = atomicCAS(&q.state[t], expect, expect == kIdle ? kQueued : kBusyQueued);
      settled = old == expect || (old != kIdle && old != kBusy);
      push = old == expect && expect == kIdle;
      expect = old;
    }
    if (!settled) atomicCAS(q.err, 0, 3);
  }
  __syncwarp();
  const unsigned int ball = __ballot_sync(0xffffffffu, push);
  if (!ball) return;
  const int lane = (int)(threadIdx.x & 31), leader = __ffs(ball) - 1;
  unsigned int pos = 0;
  if (lane == leader) pos = atomicAdd(q.tail, (unsigned int)__popc(ball));
  pos = __shfl_sync(0xffffffffu, pos, leader);
  if (push) tq_store(q, pos + __popc(ball & ((1u << lane) - 1u)), t);
}

// Lane 0 (the other lanes follow after a __syncwarp, which hands them the order
// that lane 0's fence makes): take the next queued tile.  A warp takes a ticket (the next ring
// position) as soon as it is free and keeps it until the slot is filled --
// possibly by a later push -- so no claim ever fails (looking whether the
// ring holds an entry first would be one more L2 access a visit).  Returns
// the tile, or -1 while waiting; *ticket carries the ticket between calls
// (-1: none).
__device__ __forceinline__ int tq_try_dequeue(const TileQueue& q, long long* ticket) {
  if (*ticket < 0) *ticket = atomicAdd(q.head, 1u);
  const int t = atomicExch(&q.ring[(unsigned int)*ticket % q.cap], kEmptySlot);
  if (t == kEmptySlot) return -1;
  *ticket = -1;
  // Queued -> processing: only the taker changes a queued tile's state.
  // The fence puts the change before the staging loads, so a neighbour
  // that writes the halo later sees "processing" and queues the tile again.
  ((volatile int*)q.state)[t] = kBusy;
  __threadfence();
  return t;
}

// Lane 0, after the tile's write-back (and a fence): idle again, or pushed
// again if a neighbour queued it while it was processed.  The caller counts the
// finished tile.
__device__ __forceinline__ void tq_finish(const TileQueue& q, int t) {
  if (atomicCAS(&q.state[t], kBusy, kIdle) != kBusy) {
    // Processing and queued again: only the owner changes that state.  The
    // fence keeps this store ahead of the entry, whose taker changes the state
    // next: landing after that, it would leave the tile "queued" with no entry.
    ((volatile int*)q.state)[t] = kQueued;
    const unsigned int pos = atomicAdd(q.tail, 1u);
    __threadfence();
    tq_store(q, pos, t);
  }
}

// Lane 0, when no tile is waiting: adds the tiles this warp has finished since
// the last call; whether the queue is drained.
__device__ __forceinline__ bool tq_drained(const TileQueue& q, unsigned int* finished) {
  unsigned int d;
  if (*finished) {
    __threadfence();  // the pushes of these tiles' visits before their end is counted
    d = atomicAdd(q.done, *finished) + *finished;
    *finished = 0;
  } else {
    d = *(volatile unsigned int*)q.done;
  }
  __threadfence();
  return d == *(volatile unsigned int*)q.tail;
}

}  // namespace cageo
