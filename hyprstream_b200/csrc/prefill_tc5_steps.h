// Which mbarrier of a query tile, and which phase of it, says that P.V of step u is complete (prefill_tc5.cu).
//
// A wait by parity tells a barrier's current phase from the one before it, no more: the phase before the one waited for has to be
// known to be over, and the one after it must not be able to complete before the waiter has looked.  One barrier per step parity
// gives both.  Behind step u on its barrier comes step u + 2, whose P the waiter itself has yet to write; in front of it lies step
// u - 2, and the scores of step u, which the waiter has seen, are issued behind P.V_{u-2}.  (One barrier for all steps gives only
// the first half: the scores of step u say nothing of P.V_{u-1}, and a warp that first waits for that phase, late, after its last P
// is handed over, may find P.V_u complete as well - then the parity it waits for never comes.)
#pragma once

namespace hs {

constexpr int kT5OBars = 2;
constexpr int t5_odone_bar(int u) { return u & 1; }
constexpr unsigned t5_odone_parity(int u) { return static_cast<unsigned>(u >> 1) & 1u; }

}  // namespace hs
