// rift_bar.cuh -- arithmetic of the grid barrier's word, also for the host (a
// test plays arrivals in every order against it).
//
// One 64-bit word counts both: arrivals in the high half (monotonic; it wraps
// off the top), events raised in the low half.  An arrival that raises an event
// adds to both halves at once, and the high half alone decides when the barrier
// is passed, so no event lets a CTA leave early and every CTA reads the same
// number of events.  (The low half would carry after 2^32 events of one launch:
// every CTA of the largest grid raising one at two million barriers.)
#pragma once

#ifdef __CUDACC__
#define RIFT_BAR_FN __host__ __device__ __forceinline__
#else
#define RIFT_BAR_FN inline
#endif

namespace rift {

typedef unsigned long long BarWord;

// what an arrival adds
RIFT_BAR_FN BarWord barArrival(bool raise) { return (1ull << 32) + (raise ? 1ull : 0ull); }
// `target` arrivals are in (within 2^31 of it)
RIFT_BAR_FN bool barPassed(BarWord v, unsigned target) { return (int)((unsigned)(v >> 32) - target) >= 0; }
// events raised so far, modulo 2^32
RIFT_BAR_FN unsigned barEvents(BarWord v) { return (unsigned)v; }

}  // namespace rift
