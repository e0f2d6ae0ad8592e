// Hand-over of claimed tasks inside a pair of CTAs: a ring of kPairQueue slots, of which each CTA has its own copy.
//
//   scheduler (leader)  writes a task into the slot of both CTAs; each copy completes the slot's `full` barrier there
//   readers             every role of either CTA waits for `full`, reads its CTA's copy and arrives on its CTA's `empty`
//   forwarder (peer)    a warp that stores nothing: tells the leader's `empty` that all readers of the peer have arrived on theirs
//
// The scheduler overwrites the PEER's shared memory, so a reader's access there has to happen before a write from another CTA.  Barriers order
// that only in the scope they are used with: the readers' arrivals are CTA-wide, and the forwarder's one arrival and the waits for what comes
// from the other CTA are cluster-wide.  Were the readers to arrive at the leader's barrier themselves, each would need a release of
// cluster scope, and an epilogue warp's waits for its outstanding stores to global memory first.
//
// `Port` is what the ring is made of: barriers and shared memory in the kernels, a checker of scopes in the CPU test.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define MMOE_QUEUE_FN __host__ __device__ __forceinline__
#else
#define MMOE_QUEUE_FN inline
#endif

namespace mmoe {

constexpr uint32_t kPairQueue = 4;   // tasks that the scheduler may be ahead of the slowest role
enum PairBarrier { kPairFull = 0, kPairEmpty = 1 };

// arrivals that complete the barriers of a slot: `readers` of the leader or of the peer
MMOE_QUEUE_FN constexpr uint32_t pair_full_count() { return 1; }
MMOE_QUEUE_FN constexpr uint32_t pair_empty_count(bool leader, uint32_t readers) { return readers + (leader ? 1u : 0u); }

MMOE_QUEUE_FN uint32_t pair_slot(uint32_t n) { return n % kPairQueue; }
MMOE_QUEUE_FN uint32_t pair_lap(uint32_t n) { return (n / kPairQueue) & 1u; }

// Each returns false when the call is being abandoned.
// scheduler: the n-th task, to both CTAs
template <class Port>
MMOE_QUEUE_FN bool pair_put(Port& port, uint32_t n, int task) {
  if (!port.wait_pair(kPairEmpty, pair_slot(n), pair_lap(n) ^ 1u)) return false;       // passes in the first lap
  port.send(pair_slot(n), task);
  return true;
}
// a role of either CTA: reads the n-th task
template <class Port>
MMOE_QUEUE_FN bool pair_take(Port& port, uint32_t n, int* task) {
  if (!port.wait_pair(kPairFull, pair_slot(n), pair_lap(n))) return false;
  *task = port.read(pair_slot(n));
  port.arrive_own(kPairEmpty, pair_slot(n));
  return true;
}
// forwarder: whether there is anything behind the n-th task it has to look up itself, between these two
template <class Port>
MMOE_QUEUE_FN bool pair_peek(Port& port, uint32_t n, int* task) {
  if (!port.wait_pair(kPairFull, pair_slot(n), pair_lap(n))) return false;
  *task = port.read(pair_slot(n));
  return true;
}
template <class Port>
MMOE_QUEUE_FN bool pair_forward(Port& port, uint32_t n) {
  if (!port.wait_own(kPairEmpty, pair_slot(n), pair_lap(n))) return false;
  port.arrive_leader(kPairEmpty, pair_slot(n));
  return true;
}

}  // namespace mmoe
