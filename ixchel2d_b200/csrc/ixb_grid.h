// ixb_grid.h -- what the CTAs of a resident kernel wait on (ixb_grid.cuh).
#pragma once

namespace ixb {

// how a launch ended early
enum { GRID_GAVE_UP = 1,  // a wait between phases ran out: the fields are part-swept
       GRID_NOT_MET = 2   // not all CTAs started in time: nothing has been written
};
// for tests (ixb_expire_grid_wait): the wait that expects one CTA more than there are
enum { GRID_EXPIRE_NONE = 0, GRID_EXPIRE_MEET = 1, GRID_EXPIRE_SYNC = 2 };

struct GridWords {
  unsigned bar, met;  // arrivals at the barriers, CTAs started: zero at the start of a launch
  int gave_up;        // GRID_*, kept over the launches of a call
  int passes;         // passes done (energy passes)
};
struct GridWaits {
  GridWords* words;
  int expire;
};

}  // namespace ixb
