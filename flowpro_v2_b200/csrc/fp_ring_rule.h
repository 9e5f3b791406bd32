// Slots of the ring sweep (fp_ilu_ring.cu) and the rule that keeps their barriers unambiguous; plain
// C++, so that the rule can be tested on the host.
//
// Position k of a thread block uses slot k % kRingSlots, lap k / kRingSlots.  A slot's two barriers count
// laps by one parity bit, which says "the lap before mine is over" only as long as a waiting thread is at
// most one lap ahead.  A group that waits for the blocks of position k has finished position k -
// inflight, and other groups may still be anywhere behind it: bulk copies land in any order, and the
// positions of finished cases need none.  So position k - kRingSlots, the slot's previous user, has to
// be released before any group can reach k.  That holds if position k - inflight was requested
// only when every position up to k - kRingSlots had been released.
#pragma once

namespace fp {

constexpr int kRingSlots = 64;

// whether position k may be requested when the positions below tail have been released and inflight
// groups of warps take the positions in turn
constexpr bool ring_may_request(int k, int tail, int inflight) { return k - tail < kRingSlots - inflight; }

// parity that the barriers of position k's slot are waited on with
constexpr unsigned ring_lap_parity(int k) { return (unsigned)(k / kRingSlots) & 1u; }

}  // namespace fp
