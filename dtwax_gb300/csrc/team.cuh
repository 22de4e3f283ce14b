// Teams of warps that sweep the strips of a work item as a pipeline (sdtw.cu,
// refdel.cu).
#pragma once

#include "warp_ops.cuh"

namespace dtwx {

// A strip's row needs only rows of the left neighbour that it has already
// computed, so strip s + 1 runs a window of rows behind strip s on another warp,
// fed by the seam column that strip s leaves in global scratch: every cell sees
// the operations, in the order, of one warp that sweeps strip after strip.
//
// Strips are handed out in sequence (all of an item's, then the next item's),
// so a strip's left neighbour was always handed out before it, and no warp
// waits for work that has not begun.  Strip `seq` of a team writes its seam
// column into buffer seq % buffers (two per warp, or as few as one more than
// the warps); prog[] of that buffer holds the sequence number and how much of
// it is complete (32-row windows in sdtw.cu, rows in refdel.cu).
struct TeamState {
  uint32_t lock;
  uint32_t abort;  // a wait of this CTA gave up: every warp leaves
  int32_t item;    // item being handed out
  int32_t next;    // its next strip
  int32_t total;   // its strips
  uint32_t seq;    // strips handed out so far
  int32_t dealt;   // items begun (p.deal); in an ordered deal the CTA's next item
  int32_t end;     // ordered deal: the item after the CTA's last
};
static_assert(sizeof(TeamState) == kTeamStateBytes, "shared-memory layout of the team");

constexpr uint32_t kStripDone = 0xffffffffu;  // prog[]: every row of the strip is complete

__device__ __forceinline__ uint32_t ld_shared_volatile(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ void st_shared_volatile(uint32_t addr, uint32_t v) {
  asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Bounded wait until prog word `addr` reaches `target`; false when the limit
// is reached or another warp of the CTA gave up.  The limit grows with the
// rows of a strip (the longest wait that can be in order is a strip's sweep);
// for a 2,000-row read it ends after a fraction of a second.
__device__ __forceinline__ bool team_wait(uint32_t addr, uint64_t target, uint32_t abort_addr, int rows) {
  const uint32_t limit = (1u << 22) + 256u * (uint32_t)min(rows, 1 << 23);
  for (uint32_t it = 0; it < limit; ++it) {
    uint64_t v;
    asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
    if (__all_sync(FULL_MASK, v >= target)) {
      __threadfence_block();
      return true;
    }
    if (__any_sync(FULL_MASK, ld_shared_volatile(abort_addr) != 0)) return false;
    __nanosleep(40);
  }
  return false;
}

// One look at a prog word, without waiting.
__device__ __forceinline__ bool team_ready(uint32_t addr, uint64_t target) {
  uint64_t v;
  asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  const bool ready = __all_sync(FULL_MASK, v >= target);
  __threadfence_block();
  return ready;
}

// `done` windows or rows of the strip are complete (kStripDone: all of it): the
// seam values and offsets every lane stored before are visible to the CTA's
// other warps first.
__device__ __forceinline__ void team_publish(uint32_t addr, uint32_t seq, uint32_t done) {
  __threadfence_block();
  __syncwarp();
  const uint64_t v = ((uint64_t)(seq + 1) << 32) | done;
  asm volatile("st.volatile.shared.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

// Take the team's lock (lane 0's atomic, every lane's wait).  False when the
// limit is reached or another warp of the team gave up; the lock is then free
// or never was held.
__device__ __forceinline__ bool team_lock(uint32_t lock_addr, uint32_t abort_addr, uint32_t is0) {
  for (uint32_t it = 0; it < (1u << 22); ++it) {
    if (__shfl_sync(FULL_MASK, lock_if(lock_addr, is0), 0) == 0) {
      __threadfence_block();
      if (!__any_sync(FULL_MASK, ld_shared_volatile(abort_addr) != 0)) return true;
      st_shared_volatile(lock_addr, 0);
      return false;
    }
    __nanosleep(20);
  }
  return false;
}

__device__ __forceinline__ void team_unlock(uint32_t lock_addr) {
  __threadfence_block();
  __syncwarp();
  st_shared_volatile(lock_addr, 0);
}

}  // namespace dtwx
