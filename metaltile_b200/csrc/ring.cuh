// Who waits for what in the shared-memory rings of the tcgen05 kernels: rules that the kernels follow and a host program can walk through (no CUDA in
// this file; tests/test_ring.py plays them against a model of the barriers).
#pragma once

#ifdef __CUDACC__
#define MTC_HD __host__ __device__
#else
#define MTC_HD
#endif

namespace mtc {
namespace ring {

// The two copy warps of the dense product (warp 0 and 1 here).  What TMA copies is issued by warp 0 alone, everything else by both.  A warp waits only for
// buffers that it helps to fill.  A wait by parity is sound while the waiter is at most one phase behind: a buffer that a warp waits for and nobody waits for
// that warp's arrival at can be filled, read and released again before it looks, and its phase then reads as not complete, for good where the buffer is
// not used again.
constexpr int kCopyWarps = 2;
MTC_HD constexpr bool fills(bool by_tma, int warp) { return !by_tma || warp == 0; }
// arrivals that fill a buffer: one thread's, or those of all threads of both warps
MTC_HD constexpr int fill_arrivals(bool by_tma) { return by_tma ? 1 : kCopyWarps * 32; }

// Giving up.  A CTA whose waits ran out leaves only when what it set in motion has come to rest: use u of a ring takes slot u % slots, so of `issued` uses
// the last one of a slot completes the phase of this parity (-1: none took it).  Where a phase also takes arrivals of warps that convert (use u is that
// of team u % teams), those that have left owe theirs for the uses from `done` on that were issued: `owed`.
MTC_HD constexpr int last_parity(unsigned issued, int slots, int slot) {
    return issued <= static_cast<unsigned>(slot) ? -1 : static_cast<int>((issued - 1 - slot) / slots & 1);
}
MTC_HD constexpr bool owed(unsigned use, int teams, int team) { return static_cast<int>(use % teams) == team; }

}  // namespace ring
}  // namespace mtc
