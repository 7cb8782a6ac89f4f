// Which phase of a pair of mbarriers a warp waits for next, and which copies are in
// flight: the bookkeeping of a double buffer that bulk copies fill. Plain C++, so it
// is checked on the CPU.
//
// A barrier completes one phase per copy, and a wait for parity p returns at once
// where the phase of the other parity is the one in progress. So a buffer's parity
// moves on only with a wait that saw its copy arrive: after one that gave up, parity()
// is still that of the copy in flight, and the wait before the block leaves its shared
// memory is for that copy.
#pragma once

#ifdef __CUDACC__
#define LRD_HD __host__ __device__ __forceinline__
#else
#define LRD_HD inline
#endif

namespace lrd {

struct CopyPhases {
  unsigned phase = 0;    // bit b: the parity of buffer b's next copy to arrive
  unsigned pending = 0;  // bit b: a copy into buffer b that this warp issued is in flight
  bool ok = true;        // no wait has given up

  LRD_HD unsigned parity(int b) const { return (phase >> b) & 1u; }
  LRD_HD bool in_flight(int b) const { return (pending >> b) & 1u; }
  LRD_HD void issued(int b) { pending |= 1u << b; }
  LRD_HD void waited(int b, bool arrived) {
    ok = arrived;
    if (!arrived) return;
    phase ^= 1u << b;
    pending &= ~(1u << b);
  }
};

}  // namespace lrd
