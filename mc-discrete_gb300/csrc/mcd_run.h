// mcd_run.h - launch of the resident kernel of one large simulation (mcd_run.cu).
#ifndef MCD_RUN_H
#define MCD_RUN_H

#include "mcd_tally.cuh"

namespace mcd {

int launch_run(const SimConst<float>& c, int sms, mcd_tally* tally, const mcd_electron_out& rows,
               const mcd_event_ring& ring, bool rec, uint32_t* status, cudaStream_t st);

}  // namespace mcd

#endif  // MCD_RUN_H
