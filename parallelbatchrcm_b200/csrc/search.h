// search.h -- the end of a breadth-first pass of a team.
#pragma once

#include "hd.h"

namespace pbrcm {

// look() reads what the pass left in the queue: every CTA finds the next start
// and the kind of the next pass by itself, from the same records.  The barrier
// behind it keeps the next pass, whose first levels CTA 0 may run alone, from
// writing the queue while another CTA still looks, so that all of them decide
// the same; and it keeps CTA 0 from opening the gate again while another CTA
// still reads the state of this one.  Returns false if the team must stop.
template <class TeamT, class Look>
PBRCM_DEV bool end_pass(TeamT& team, Look look)
{
    look();
    return team.size == 1 || team.sync(8);
}

}  // namespace pbrcm
