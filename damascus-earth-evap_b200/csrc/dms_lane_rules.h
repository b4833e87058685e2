// Rules of the lane loop that need nothing of the device, so that they can be tested on the CPU.
#pragma once

#include "dms_philox.h"

namespace dms
{
namespace lane
{

// The sets of counts in which a block in lockstep votes.  A pass has one barrier: each warp adds to the pass's set
// before it and reads that set after it.  One warp clears the next pass's set before the barrier too: no warp
// adds to that set until it is past the barrier, and each has read it (two passes earlier) before
// the barrier of the pass before this one.  With two sets the clear would have to come after the barrier, where a
// warp with an almost empty pass may already be adding.
constexpr int VOTE_SETS = 3;
DMS_HD int next_vote_set(int set) { return set + 1 == VOTE_SETS ? 0 : set + 1; }

}	// namespace lane
}	// namespace dms
