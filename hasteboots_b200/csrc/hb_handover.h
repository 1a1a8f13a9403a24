// hb_handover.h -- the named barriers of bootstrap_tc_kernel's handovers (hb_boot_tc.cuh).
//
// A step has units + 2 handovers, units even: handover 0 hands the first pair's digits to the auxiliary
// warps, handover u + 1 ends stage u. Compute threads arrive and go on; the MMA and the key warp wait. A
// barrier counts arrivals, so a thread that arrives at the same barrier twice before the auxiliary warps came
// once completes it in their place: from then on the counts are off by a warp and the CTA waits for good.
//
// Between two handovers of a step the compute threads wait for the MMAs issued after the first of them, which
// both auxiliary warps have then passed. The last handover of a step issues no MMA, and the next one (the
// following step's first, or the one that stops the auxiliary warps) waits for nothing of theirs. So the
// handovers take two barriers in turn: an arrival then only meets the handover two before it, which such a wait
// has covered. The number of handovers in a step is even, so the turn follows from the handover's place in
// its step.
#pragma once

#if defined(__CUDACC__)
#define HB_HANDOVER_HD __host__ __device__
#else
#define HB_HANDOVER_HD
#endif

namespace hb {

constexpr int kTcHandoverEven = 5, kTcHandoverOdd = 7;  // 1 to 4: the gates' groups, 6: barrier_stop

// The barrier of a step's handover k.
HB_HANDOVER_HD constexpr int tc_handover_barrier(unsigned k) { return k % 2 == 0 ? kTcHandoverEven : kTcHandoverOdd; }

}  // namespace hb
