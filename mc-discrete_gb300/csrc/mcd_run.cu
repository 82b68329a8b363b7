// mcd_run.cu - one FP32 simulation of more electrons than the small-run kernel
// takes, one resident block per SM.
//
// Block b runs every gridDim.x-th electron: its lanes take the next of its
// share as they fall idle, and when the share is handed out the block runs down
// with compaction (mcd_drain.cuh).  No queue in global memory is needed, since
// the shares of the SMs are statistically alike.
#include <cuda_runtime.h>
#include <stdint.h>

#include "mcd_drain.cuh"
#include "mcd_run.h"

namespace mcd {

// Threads of a block: 512 where they hold its share of the electrons, else as
// many as leave 72 registers each, enough for the constants (HotConst) but in
// the discrete model with a ring, which spills 232 bytes (and is still twice as
// fast as independent threads: 152000 Au 10 keV electrons 3.6 ms against 7.2).
// Against 1024 threads at 64 registers, with the constants in shared memory:
// 1e6 electrons Si 5.65 / 6.04 ms, Au 12.9 / 13.5, Cu without a table 12.6 /
// 12.5, continuous Cu 70 deg 2.50 / 2.65; 1e5: Si 0.94 / 1.06, Au 3.28 / 3.54,
// Cu 2.39 / 2.54; 768 threads lose 2 to 8% of the large runs.
constexpr int kThreadsMost = 896;

template <int MODE, bool REC, int THREADS>
__global__ void __launch_bounds__(THREADS) k_run(const SimConst<float> cp, const __grid_constant__ RoundKeys keys,
                                                 mcd_tally* tally, const mcd_electron_out eo,
                                                 const mcd_event_ring ring, uint32_t* status) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ BlockTally bt[THREADS / 32];   // a copy per warp
    __shared__ SimConst<float> c;
    __shared__ mcd_electron_out rows;
    if (threadIdx.x == 0) {
        c = cp;
        rows = eo;
    }
    bt_zero(bt, THREADS / 32);
    __syncthreads();
    const HotConst<float> hot(c, MODE == MCD_MODE_CONT ? &keys : nullptr);
    const OneSim<MODE, HotConst<float>> run{c, hot, bt[threadIdx.x >> 5], tally, rows};
    const unsigned count = (unsigned)(((unsigned long long)c.num_el - blockIdx.x + gridDim.x - 1) / gridDim.x);
    auto take = [&](unsigned k, Lane<float>& L, ElecRng& rng, int& sim) {
        rng = elec_rng(c, c.first + blockIdx.x + (uint64_t)k * gridDim.x);
        lane_init(L, c);
        sim = 0;
    };
    const bool chan = (c.bits & kBitChan) != 0;
    const uint32_t st = MODE == MCD_MODE_DS && chan ? drain_run<REC, true>(run, count, take, smem, ring, false)
                                                    : drain_run<REC, false>(run, count, take, smem, ring, false);
    or_status(status, st);
    __syncthreads();
    bt_fold(bt, 1, THREADS / 32);
    __syncthreads();
    if (threadIdx.x == 0) bt_flush(bt[0], tally, chan);
}

template <int MODE, bool REC>
static int launch_threads(const SimConst<float>& c, int sms, mcd_tally* tally, const mcd_electron_out& rows,
                          const mcd_event_ring& ring, uint32_t* status, cudaStream_t st) {
    const unsigned grid = (unsigned)(c.num_el < sms ? c.num_el : sms);
    if (grid == 0) return MCD_OK;
    const RoundKeys keys = round_keys(c);
    if (c.num_el <= (int64_t)512 * sms)
        k_run<MODE, REC, 512><<<grid, 512, drain_smem(512), st>>>(c, keys, tally, rows, ring, status);
    else
        k_run<MODE, REC, kThreadsMost><<<grid, kThreadsMost, drain_smem(kThreadsMost), st>>>(c, keys, tally, rows, ring, status);
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}

int launch_run(const SimConst<float>& c, int sms, mcd_tally* tally, const mcd_electron_out& rows,
               const mcd_event_ring& ring, bool rec, uint32_t* status, cudaStream_t st) {
    if (c.mode == MCD_MODE_DS)
        return rec ? launch_threads<MCD_MODE_DS, true>(c, sms, tally, rows, ring, status, st)
                   : launch_threads<MCD_MODE_DS, false>(c, sms, tally, rows, ring, status, st);
    return rec ? launch_threads<MCD_MODE_CONT, true>(c, sms, tally, rows, ring, status, st)
               : launch_threads<MCD_MODE_CONT, false>(c, sms, tally, rows, ring, status, st);
}

}  // namespace mcd
