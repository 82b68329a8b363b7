// mcd_lanes.h - launch of the small-run transport kernel (mcd_lanes.cu).
#ifndef MCD_LANES_H
#define MCD_LANES_H

#include "mcd_tally.cuh"

namespace mcd {

// One simulation with `group` (8, 16 or 32) lanes per electron.
template <class T>
int launch_lanes(const SimConst<T>& c, int group, mcd_tally* tally, const ElOut& eo, const mcd_event_ring& ring,
                 bool rec, uint32_t* status, cudaStream_t st);

}  // namespace mcd

#endif  // MCD_LANES_H
