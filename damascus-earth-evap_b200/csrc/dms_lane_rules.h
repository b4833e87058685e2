// Rules of the lane loop that need nothing of the device, so that they can be tested on the CPU.
#pragma once

#include <cmath>

#include "dms_constants.h"
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

// When lanes that wait for a rare phase (scatterings, terminations) get it, asked once per pass: when `waiting` of them
// reach `batch` in `per` lanes of a full group, when the first of them has waited `wait` passes, or when no lane is
// stepping.  `passes` counts since the first of them arrived (0 before it).  `lanes` is the size of the group;
// with fewer lanes at work, `full`, batch and wait shrink.
DMS_HD bool rare_phase_due(int& passes, int waiting, int stepping, int batch, int per, int wait, int lanes, int full)
{
	if(waiting == 0)
		return false;
	passes++;
	const bool go = per * waiting >= batch * full || stepping == 0 || passes * lanes >= wait * full;
	if(go)
		passes = 0;
	return go;
}

// Whether the time to the surface (src/Simulation_Trajectory.cpp:886-899) of a particle outside it cannot be
// below `step`, by a margin far above its rounding.  along = x . v.
DMS_HD bool surface_is_far(double r, double along, double step)
{
	return (along >= 0.0) | ((r - DMS_RSUN_KM) * r * (1.0 - 1.0e-9) > -along * step);
}

// The same from the propagator's radial speed, for a state whose event has not been formed.  The event's
// x . v is off r v_radial by some 1e-15 r speed, since its components and axes are rounded: far below
// the margin only above 1e-4 of the speed.  False below that, where the event decides.
DMS_HD bool surface_is_far_by_speed(double r, double v_radial, double speed, double step)
{
	return (fabs(v_radial) > 1.0e-4 * speed) & surface_is_far(r, r * v_radial, step);
}

}	// namespace lane
}	// namespace dms
