// rift_bar.cuh -- arithmetic of the grid barrier's word, also for the host (a
// test plays arrivals in every order against it).
//
// One 32-bit word counts both: an arrival adds 1, an arrival that raises an event
// 1 + 2^16.  `target` is the word at which the barrier is passed, with the events
// counted so far.  The low half of word - target is the difference in arrivals
// whatever was raised since: its sign alone passes the barrier (fewer than 2^15
// CTAs, at most one barrier apart), so no event lets a CTA leave early.  Once
// passed, the high half is the number of events since: every CTA reads the same.
// (Compared as one number, the arrival that raised the first event was past the
// target for whoever polled next.  A 64-bit word, or the count kept apart from the
// target, cost 0.3 to 0.5 us of 15.8 a step on 456 CTAs.)
#pragma once

#ifdef __CUDACC__
#define RIFT_BAR_FN __host__ __device__ __forceinline__
#else
#define RIFT_BAR_FN inline
#endif

namespace rift {

// what an arrival adds
RIFT_BAR_FN unsigned barArrival(bool raise) { return raise ? 0x10001u : 1u; }
RIFT_BAR_FN bool barPassed(unsigned v, unsigned target) { return (int)((v - target) << 16) >= 0; }
// events raised since those in `target` (the barrier passed)
RIFT_BAR_FN unsigned barEvents(unsigned v, unsigned target) { return (v - target) >> 16; }
// the target with k more events counted
RIFT_BAR_FN unsigned barSeen(unsigned target, unsigned k) { return target + (k << 16); }

}  // namespace rift
