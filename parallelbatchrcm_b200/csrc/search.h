// search.h -- decisions of the start search: the end of a team's pass, and
// which matrices search in discovery order from the first pass on.
#pragma once

#include <cstdint>

#include "hd.h"

namespace pbrcm {

// Stencils wider than 5 and 7 points: more than 8 entries a row, most rows of
// about the largest valence (random geometric graphs: half of it).  Their
// breadth-first levels end in a face or an edge, not in a corner, so that a
// start-search pass always needs discovery order.
PBRCM_HD inline bool wide_stencil(uint32_t n, uint32_t nnz, uint32_t maxdeg)
{
    return nnz / 8u > n && 4ull * nnz >= 3ull * maxdeg * n;
}

// Longest row that an unordered pass of one thread group puts together with
// others: a warp takes a longer one alone (solo.cuh), eight lanes take one in
// 5 and more rounds (resident.cu).
constexpr uint32_t kLevelRow = 31;

// Whether one group's unordered passes are no faster than ordered ones.  Solo
// engine, 200 matrices at once, 20,000 nodes each: geometric graphs of 35
// entries a row 21.4 ms unordered, 13.4 in order; random graphs of 41 a row 13.6
// / 9.9, of 15 (rows of 31 to 35) 4.59 / 4.69.  Shared-memory engine, 96 hub
// paths of 4,000 nodes with rows of 403 entries: 0.63 / 0.49; of 103 0.47 /
// 0.33; of 43 0.62 / 0.48.  (A team's chunks take rows of any length up to
// theirs together: 100,000-node geometric graphs of 29 entries a row 1.15 /
// 0.97, of 21 0.59-1.27 / 0.87-1.15, a mesh with stars of 101 6.3 / 9.5.)
PBRCM_HD inline bool long_rows(uint32_t maxdeg) { return maxdeg > kLevelRow; }

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
