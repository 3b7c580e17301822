// The end of a wait that a whole warp keeps.
#pragma once

namespace bogus_gpu {

// Every lane of a converged warp: late, its own wait ran out; stopped, it saw that another's did. True when the warp gives
// up, with the reason in *status.
__device__ __forceinline__ bool warp_gives_up(bool late, bool stopped, int lane, int* status, int timeout) {
  const bool ran_out = __any_sync(0xffffffffu, late);  // the lanes' clocks need not agree: any of them decides
  if (ran_out && lane == 0) atomicCAS(status, 0, timeout);
  return __any_sync(0xffffffffu, ran_out || stopped);
}

}  // namespace bogus_gpu
