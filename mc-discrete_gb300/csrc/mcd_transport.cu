// mcd_transport.cu - trajectory kernels and their C-ABI entry points.
//
//  k_plain    one thread per electron, one launch per simulation
//             (replaces multiTraj_DS/_cont, MC/tools/multiScatter.py:66-229)
//             (small runs: several lanes per electron, mcd_lanes.cu; large FP32
//             ones: a resident block per SM, mcd_run.cu)
//  k_batched  persistent grid over many simulations; a global queue hands
//             out electrons and a warp takes new ones as soon as `refill` of
//             its lanes are idle, so uneven trajectory lengths do not idle
//             the warp (replaces MapScatterer's pool, MC/doScatter.py:22-95)
//
// Tallies are gathered per block in shared memory and flushed once per block
// with global atomics; exit-energy/angle histograms go straight to global
// memory (one atomic per backscattered electron).
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "mcd_drain.cuh"
#include "mcd_lanes.h"
#include "mcd_run.h"

namespace mcd {

// ---------------------------------------------------------------------------
// plain kernel: one thread per electron
// ---------------------------------------------------------------------------
// The constant block arrives as a by-value kernel parameter and is copied to
// shared memory before use.  Reading it through a reference to the parameter
// itself made nvcc 13.0 (sm_103a, -O3) drop the loop-carried energy update of
// the lane state initialised from it; the shared-memory copy is also what the
// batched kernel reads.
// The continuous model keeps the constants in registers and reads the round keys
// from the constant bank (RoundKeys): its events are short, and a run of a warp or
// two per scheduler waits for each load and addition on the way to the random
// words.  6080 electrons of Au 30 keV 0.675 -> 0.579 ms, of Al 0.266 -> 0.231, 36480 of
// Cu 0.446 -> 0.398, 1e6 of Al 5 keV 0.917 -> 0.891.
template <class T, int MODE, bool REC>
__global__ void __launch_bounds__(256) k_plain(const SimConst<T> cp, const __grid_constant__ RoundKeys keys,
                                               mcd_tally* tally, const ElOut eo, const mcd_event_ring ring,
                                               uint32_t* status) {
    __shared__ BlockTally bt;
    __shared__ SimConst<T> c;
    if (threadIdx.x == 0) c = cp;
    bt_zero(&bt, 1);
    __syncthreads();
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t st = 0;
    if (i < (uint64_t)c.num_el) {
        Lane<T> L;
        lane_init(L, c);
        const ElecRng rng = elec_rng(c, c.first + i);
        const bool chan = (c.tally_flags & MCD_TALLY_CHANNELS) != 0;
        const HotConst<T> hot(c, MODE == MCD_MODE_CONT ? &keys : nullptr);   // (continuous)
        while (L.outcome == MCD_OUT_NONE) {
            EventOut<T> ev;
            RingTicket tk{};
            if (REC) {
                const bool rec = L.step < c.max_scatt, takes = ring_takes(ring, (uint32_t)i);
                tk = ring_reserve(ring, rec && takes);
                if (rec && !takes) st |= MCD_FLAG_RING_INDEX;
            }
            const int ch = (MODE == MCD_MODE_DS) ? ds_event<T, REC>(L, c, rng, &ev, c.sig != nullptr)
                                                 : cont_event<T, REC>(L, hot, rng, &ev);
            if (REC) ring_write(ring, ring_slot(ring, tk), (uint32_t)i, L.step, ev);
            if (chan && ch > MCD_CH_RUTH) atomicAdd(&bt.channel[ch], 1ull);
        }
        st |= finish_electron(c, L, i, bt, tally, eo);
    }
    or_status(status, st);
    __syncthreads();
    if (threadIdx.x == 0) bt_flush(bt, tally, (c.bits & kBitChan) != 0);
}

// ---------------------------------------------------------------------------
// batched persistent kernel
// ---------------------------------------------------------------------------
struct BatchHeader {
    unsigned long long queue;   // next electron to hand out
    unsigned long long live;    // electrons listed for the run-down kernel
    unsigned long long total;   // electrons over all simulations
    int32_t nsims;
    int32_t chan;               // some simulation counts channels
    uint32_t* list;             // the list's seats, or nullptr
    int32_t list_cap;           // ... how many
    int32_t pad_[5];
};
static_assert(sizeof(BatchHeader) == 64, "the workspace's layout");

constexpr int kBatchMaxSims = 256;

// Workspace layout: header | prefix[nsims+1] (u64, by queue position) |
// perm[nsims] (i32: queue position -> simulation) | pad | SimConst[nsims].
__host__ __device__ constexpr size_t batch_prefix_off() { return sizeof(BatchHeader); }
__host__ __device__ constexpr size_t batch_perm_off(int nsims) {
    return sizeof(BatchHeader) + sizeof(unsigned long long) * (size_t)(nsims + 1);
}
__host__ __device__ constexpr size_t batch_consts_off(int nsims) {
    return (batch_perm_off(nsims) + sizeof(int32_t) * (size_t)nsims + 255) & ~(size_t)255;
}
// ... | per-electron row pointers[nsims] | FP64 constants (table build only)
// | cross-section tables.  The no-alloc path copies only the core (through
// the row pointers) and has no table slots.
__host__ __device__ constexpr size_t batch_elout_off(int nsims) {
    return batch_consts_off(nsims) + sizeof(SimConst<float>) * (size_t)nsims;
}
__host__ __device__ constexpr size_t batch_core_bytes(int nsims) {
    return batch_elout_off(nsims) + sizeof(mcd_electron_out) * (size_t)nsims;
}
static_assert(sizeof(SimConst<float>) % 8 == 0, "row pointers follow the constant blocks");

// The row pointers of each simulation (zero: none), as the kernel reads them.
inline void pack_rows(const mcd_sim* sims, int nsims, uint8_t* host) {
    mcd_electron_out* eo = reinterpret_cast<mcd_electron_out*>(host + batch_elout_off(nsims));
    for (int k = 0; k < nsims; ++k) {
        if (sims[k].electrons) eo[k] = *sims[k].electrons;
        else memset(&eo[k], 0, sizeof(mcd_electron_out));
    }
}
__host__ __device__ constexpr size_t batch_dconsts_off(int nsims) {
    return (batch_core_bytes(nsims) + 255) & ~(size_t)255;
}
__host__ __device__ constexpr size_t batch_sig_off(int nsims) {
    return (batch_dconsts_off(nsims) + sizeof(SimConst<double>) * (size_t)nsims + 255) & ~(size_t)255;
}
__host__ __device__ constexpr size_t batch_sig_bytes() {   // one table slot per simulation
    return sizeof(float) * (size_t)kSigRowsMax * kSigStride;
}
__host__ __device__ constexpr size_t batch_bytes(int nsims) {
    return batch_sig_off(nsims) + batch_sig_bytes() * (size_t)nsims;
}
// The electrons still on their way when the queue ran empty are listed (seats
// as in mcd_drain.cuh) in a buffer of its own, scratch of one launch that
// batches may share: at most one electron per lane of the launch, and no more
// than the batch has.
constexpr int kLiveSeats = 1 << 18;

__host__ __device__ constexpr size_t batch_smem(int nsims) {
    return sizeof(SimConst<float>) * nsims + sizeof(unsigned long long) * (nsims + 1) +
           sizeof(int32_t) * ((nsims + 1) & ~1) + sizeof(BlockTally) * nsims;
}
// Copies of the tallies in the run-down kernel (bt_fold): one for each of its 16
// warps while they take no more than 17 KB.
__host__ __device__ constexpr int drain_copies(int nsims) {
    int c = kDrainThreads / 32;
    while (c > 1 && c * nsims > 80) c /= 2;
    return c;
}
// Its shared memory: that of the batch, the other copies, the drain's seats.
__host__ __device__ constexpr size_t batch_drain_off(int nsims) {
    return (batch_smem(nsims) + sizeof(BlockTally) * nsims * (drain_copies(nsims) - 1) + 15) & ~(size_t)15;
}

// Queue order: simulations with the longest expected trajectories first, so
// that the last electrons handed out are short ones and the grid drains
// evenly.  The key is the energy to lose, less for tilted beams (which
// backscatter more).  Results do not depend on the order: every electron
// keeps its own (sim, electron, event) Philox counters.
static void batch_order(const mcd_sim* sims, int nsims, int32_t* perm) {
    for (int k = 0; k < nsims; ++k) perm[k] = k;
    auto key = [&](int k) {
        const double t = sims[k].s_tilt * kPi / 180.0;
        return (sims[k].E0 - sims[k].Emin) * cos(0.5 * t);
    };
    for (int a = 1; a < nsims; ++a) {      // stable insertion sort, descending key
        const int v = perm[a];
        const double kv = key(v);
        int b = a - 1;
        while (b >= 0 && key(perm[b]) < kv) {
            perm[b + 1] = perm[b];
            --b;
        }
        perm[b + 1] = v;
    }
}

template <bool REC, bool CHAN>
__device__ __forceinline__ void batched_body(uint8_t* ws, mcd_tally* tallies, int refill, uint32_t* status,
                                             const mcd_event_ring& ring, int flags);

// Two register budgets of the same kernel: up to 1024 threads per block at
// 64 registers (32 warps per SM: one block of 1024), or two blocks of up to
// 576 per SM at 56 registers (36 warps, two copies of the constant blocks in
// shared memory); neither spills.  On the 64-simulation workload the second, in
// blocks of 576, takes 72.4 ms against 74.2; five blocks of 256 at 48 registers
// were 26% slower.
// REC: append every event to the ring.  The event loop exists twice, CHAN
// for batches in which some simulation counts channels, so that the others
// test nothing per event (one test there cost 1% of the 64 simulations); the
// counts of members that do not ask are dropped at the flush.
template <bool REC = false>
__global__ void __launch_bounds__(1024) k_batched(uint8_t* ws, mcd_tally* tallies, int refill,
                                                  uint32_t* status, const mcd_event_ring ring = mcd_event_ring{},
                                                  int flags = 0) {
    if (reinterpret_cast<const BatchHeader*>(ws)->chan) batched_body<REC, true>(ws, tallies, refill, status, ring, flags);
    else batched_body<REC, false>(ws, tallies, refill, status, ring, flags);
}

template <bool REC = false>
__global__ void __launch_bounds__(576, 2) k_batched_lr(uint8_t* ws, mcd_tally* tallies, int refill,
                                                       uint32_t* status, const mcd_event_ring ring = mcd_event_ring{},
                                                       int flags = 0) {
    if (reinterpret_cast<const BatchHeader*>(ws)->chan) batched_body<REC, true>(ws, tallies, refill, status, ring, flags);
    else batched_body<REC, false>(ws, tallies, refill, status, ring, flags);
}

// What a batched block keeps in shared memory: the simulations' constants,
// queue prefix sums, order and tallies.
struct BatchShared {
    SimConst<float>* c;
    unsigned long long* pre;
    int32_t* perm;
    BlockTally* t;
    __device__ __forceinline__ BatchShared(uint8_t* smem, int nsims)
        : c(reinterpret_cast<SimConst<float>*>(smem)),
          pre(reinterpret_cast<unsigned long long*>(smem + sizeof(SimConst<float>) * nsims)),
          perm(reinterpret_cast<int32_t*>(pre + (nsims + 1))),
          t(reinterpret_cast<BlockTally*>(perm + ((nsims + 1) & ~1))) {}
    __device__ __forceinline__ void load(const uint8_t* ws, int nsims, int copies = 1) const {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(ws + batch_consts_off(nsims));
        uint32_t* dst = reinterpret_cast<uint32_t*>(c);
        const int words = (int)(sizeof(SimConst<float>) / 4) * nsims;
        for (int k = threadIdx.x; k < words; k += blockDim.x) dst[k] = src[k];
        const unsigned long long* p = reinterpret_cast<const unsigned long long*>(ws + batch_prefix_off());
        for (int k = threadIdx.x; k <= nsims; k += blockDim.x) pre[k] = p[k];
        const int32_t* q = reinterpret_cast<const int32_t*>(ws + batch_perm_off(nsims));
        for (int k = threadIdx.x; k < nsims; k += blockDim.x) perm[k] = q[k];
        bt_zero(t, nsims * copies);
    }
    __device__ __forceinline__ void flush(mcd_tally* tallies, int nsims) const {
        for (int k = threadIdx.x; k < nsims; k += blockDim.x)
            bt_flush(t[k], tallies + k, (c[k].bits & kBitChan) != 0);
    }
};

constexpr int kRunInline = 1;   // evaluate cross sections instead of reading the tables
constexpr int kRunList = 2;     // list the electrons left when the queue is empty, if the list holds them

template <bool REC, bool CHAN>
__device__ __forceinline__ void batched_body(uint8_t* ws, mcd_tally* tallies, int refill, uint32_t* status,
                                             const mcd_event_ring& ring, int flags) {
    extern __shared__ __align__(16) uint8_t smem[];
    BatchHeader* hdr = reinterpret_cast<BatchHeader*>(ws);
    const int nsims = hdr->nsims;
    const unsigned long long total = hdr->total;
    const int inline_sigma = flags & kRunInline;
    if ((unsigned long long)hdr->list_cap < min(total, (unsigned long long)gridDim.x * blockDim.x)) flags &= ~kRunList;
    const BatchShared sh(smem, nsims);
    SimConst<float>* s_c = sh.c;
    unsigned long long* s_pre = sh.pre;
    int32_t* s_perm = sh.perm;
    BlockTally* s_t = sh.t;
    sh.load(ws, nsims);
    __syncthreads();

    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    Lane<float> L;
    int sim = 0;
    ElecRng rng{0u, 0u, 0u};
    bool have = false;
    bool exhausted = false;
    uint32_t st = 0;
    const mcd_electron_out* rows = reinterpret_cast<const mcd_electron_out*>(ws + batch_elout_off(nsims));
    while (true) {
        // the lanes without an electron; voted again only after a refill,
        // so a step with every lane busy costs one vote
        unsigned idle = __ballot_sync(0xffffffffu, !have);
        if (!exhausted && idle && (__popc(idle) >= refill || idle == 0xffffffffu)) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(&hdr->queue, (unsigned long long)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (!have) {
                const unsigned long long g = base + __popc(idle & lt);
                if (g < total) {
                    int lo = 0, hi = nsims;  // s_pre[lo] <= g < s_pre[hi] (queue positions)
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if (s_pre[mid] <= g) lo = mid; else hi = mid;
                    }
                    sim = s_perm[lo];
                    rng = elec_rng(s_c[sim], s_c[sim].first + (g - s_pre[lo]));
                    lane_init(L, s_c[sim]);
                    have = true;
                }
            }
            // (a batch no larger than the launch is handed out in one claim per warp)
            if (base + __popc(idle) >= total || total <= (unsigned long long)gridDim.x * blockDim.x) exhausted = true;
            idle = __ballot_sync(0xffffffffu, !have);
            if (exhausted && (flags & kRunList)) {
                // the run-down kernel takes the warp's electrons over
                const unsigned busy = ~idle;
                unsigned long long at = 0;
                if (lane == 0 && busy) at = atomicAdd(&hdr->live, (unsigned long long)__popc(busy));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (have)
                    seat_put(Seats{hdr->list, hdr->list_cap}, (int)at + __popc(busy & lt), L, rng, sim);
                break;
            }
        }
        if (idle == 0xffffffffu) {
            if (exhausted) break;
            continue;
        }
        if (have) {
            const SimConst<float>& c = s_c[sim];
            EventOut<float> ev;
            RingTicket tk{};
            uint32_t el = 0;
            if (REC) {
                el = (uint32_t)(elec_index(c, rng) - c.first);
                const bool rec = L.step < c.max_scatt;
                tk = ring_reserve(ring, rec && ring_takes(ring, el));
                if (rec && !ring_takes(ring, el)) st |= MCD_FLAG_RING_INDEX;
            }
            int ch;
            if (!(c.bits & kBitCont))
                ch = ds_event<float, REC>(L, c, rng, &ev, !inline_sigma && c.sig != nullptr);
            else
                ch = cont_event<float, REC>(L, c, rng, &ev);
            if (REC) ring_write(ring, ring_slot(ring, tk), el, L.step, ev);
            if (CHAN && ch > MCD_CH_RUTH) atomicAdd(&s_t[sim].channel[ch], 1ull);
            if (L.outcome != MCD_OUT_NONE) {
                const mcd_electron_out& r = rows[sim];
                const ElOut eo{r.outcome, r.flags, r.final_E, r.dir, r.last_pos, r.max_z, r.n_events};
                st |= finish_electron(c, L, elec_index(c, rng) - c.first, s_t[sim], tallies + sim, eo);
                have = false;
            }
        }
    }
    or_status(status, st);
    __syncthreads();
    sh.flush(tallies, nsims);
}

// The electrons that a batched launch listed, to their end: block b of the
// grid takes every gridDim.x-th of them, so that each SM gets its part of
// every simulation's.  ONE: the batch has one simulation, whose constants, in
// DS mode, stay in registers (40000 Au 30 keV electrons 4.63 -> 4.05 ms, with
// every event to the ring 6.14 -> 5.94 ms).
template <bool REC, bool ONE>
__global__ void __launch_bounds__(kDrainThreads) k_rundown(uint8_t* ws, mcd_tally* tallies, uint32_t* status,
                                                           const mcd_event_ring ring, int flags) {
    extern __shared__ __align__(16) uint8_t smem[];
    const BatchHeader* hdr = reinterpret_cast<const BatchHeader*>(ws);
    const int nsims = hdr->nsims;
    const unsigned live = (unsigned)hdr->live;
    if (blockIdx.x >= live) return;
    const BatchShared sh(smem, nsims);
    const int copies = drain_copies(nsims);
    sh.load(ws, nsims, copies);
    __syncthreads();
    BlockTally* mine = sh.t + (int)(threadIdx.x >> 5) % copies * nsims;
    const ManySims run{sh.c, mine, tallies, reinterpret_cast<const mcd_electron_out*>(ws + batch_elout_off(nsims))};
    const Seats list{hdr->list, hdr->list_cap};
    const unsigned count = (live - blockIdx.x + gridDim.x - 1) / gridDim.x;
    auto take = [&](unsigned k, Lane<float>& L, ElecRng& rng, int& sim) {
        seat_get(list, (int)(blockIdx.x + k * gridDim.x), L, rng, sim);
    };
    uint8_t* seats = smem + batch_drain_off(nsims);
    const bool inl = (flags & kRunInline) != 0;
    uint32_t st;
    if (ONE && !(sh.c[0].bits & kBitCont)) {
        const HotConst<float> hot(sh.c[0]);
        const OneSim<MCD_MODE_DS, HotConst<float>> one{sh.c[0], hot, mine[0], tallies, run.rows(0)};
        st = hdr->chan ? drain_run<REC, true>(one, count, take, seats, ring, inl)
                       : drain_run<REC, false>(one, count, take, seats, ring, inl);
    } else {
        st = hdr->chan ? drain_run<REC, true>(run, count, take, seats, ring, inl)
                       : drain_run<REC, false>(run, count, take, seats, ring, inl);
    }
    or_status(status, st);
    __syncthreads();
    bt_fold(sh.t, nsims, copies);
    __syncthreads();
    sh.flush(tallies, nsims);
}

// Cross-section tables of a prepared batch: one thread per (table slot, grid
// point); a slot is built when its simulation leads a group sharing it.  The
// exact FP64 expressions of the inline path, stored as FP32 E * running sums
// in pick order.
// Row i of a table on the grid (l0, inv): [E total, E running sums Ruth,
// +Moller, +Gryz[k] ... (the sum through Quinn is the total)], padding
// FLT_MAX: never below a target.
__device__ __forceinline__ void sig_row(const SimConst<double>& c, float l0, float inv, int S, int i,
                                        float* row) {
    const double E = exp2((double)l0 + (double)i / (double)inv);
    const double invE = 1.0 / E;
    double cum = sig_ruth<double>(c, E);
    int col = 1;
    row[col++] = (float)(E * cum);
    cum += sig_moller<double>(c, E, invE);
    row[col++] = (float)(E * cum);
    for (int k = 0; k < c.nsh; ++k) {
        cum += sig_gryz<double>(c, E, invE, k);
        row[col++] = (float)(E * cum);
    }
    cum += sig_quinn<double>(c, E, invE);
    row[0] = (float)(E * cum);
    for (; col < S; ++col) row[col] = 3.402823466e38f;
}

__global__ void __launch_bounds__(256) k_sigtab(uint8_t* ws, int nsims) {
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (long long)nsims * kSigRowsMax) return;
    const int s = (int)(gid / kSigRowsMax), i = (int)(gid % kSigRowsMax);
    const SimConst<float>& cf = reinterpret_cast<const SimConst<float>*>(ws + batch_consts_off(nsims))[s];
    const float* slot = reinterpret_cast<const float*>(ws + batch_sig_off(nsims) + batch_sig_bytes() * s);
    if (cf.sig != slot || i >= cf.sig_rows) return;
    const SimConst<double>& c = reinterpret_cast<const SimConst<double>*>(ws + batch_dconsts_off(nsims))[s];
    float* row = reinterpret_cast<float*>(ws + batch_sig_off(nsims) + batch_sig_bytes() * s) + (size_t)i * cf.sig_S;
    sig_row(c, cf.sig_l0, cf.sig_inv, cf.sig_S, i, row);
}

// The table of one simulation (mcd_build_sigma_table): one thread per row.
__global__ void __launch_bounds__(256) k_sigtab_one(const SimConst<double> c, float l0, float inv, int rows,
                                                     int S, float* table) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows) return;
    sig_row(c, l0, inv, S, i, table + (size_t)i * S);
}

// The FP64 table of one simulation (mcd_build_sigma_table for FP64
// transport; layout at kSig64Cells): one thread per (octave, cell).  It
// evaluates the mean free path and the running-sum fractions at the cell's
// four nodes E_n = 2^e (1 + (i - 1 + n) / cells), n = 0..3, and stores the
// coefficients of the cubic through them in the offset f = (E - E_1) / h:
// with v_n the node values, c0 = v_1, c1 = -v_0/3 - v_1/2 + v_2 - v_3/6,
// c2 = v_0/2 - v_1 + v_2/2, c3 = (v_3 - v_0)/6 + (v_1 - v_2)/2 (the
// Lagrange cubic written in powers of f).
__global__ void __launch_bounds__(128) k_sigtab64(const SimConst<double> c, int e_lo, int blocks,
                                                   double* table) {
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= blocks * kSig64Cells) return;
    const int blk = gid / kSig64Cells, i = gid % kSig64Cells;
    const int K = c.nsh + 3;
    const double base = ldexp(1.0, e_lo + blk), h = base / kSig64Cells;
    double v[4][3 + MCD_MAX_SHELLS];
    for (int n = 0; n < 4; ++n) {
        const double E = base + (double)(i - 1 + n) * h;
        const double invE = 1.0 / E;
        double run[3 + MCD_MAX_SHELLS];
        double cum = sig_ruth<double>(c, E);
        run[1] = cum;
        cum += sig_moller<double>(c, E, invE);
        run[2] = cum;
        for (int k = 0; k < c.nsh; ++k) {
            cum += sig_gryz<double>(c, E, invE, k);
            run[3 + k] = cum;
        }
        cum += sig_quinn<double>(c, E, invE);
        const double inv = 1.0 / cum;
        v[n][0] = inv;
        for (int k = 1; k < K; ++k) v[n][k] = run[k] * inv;
    }
    double* rec = table + (size_t)gid * sig64_stride(K);
    const double E1 = base + (double)(i - 1) * h, E4 = E1 + 3.0 * h;
    auto in = [&](double x) { return x >= E1 && x <= E4; };
    // below 2 Wc the Moller cross section is negative and falls to -inf at
    // Wc (MC/tools/crossSections.py:183-208), which no cubic follows
    bool kink = in(c.Wc) || in(c.Epl) || E1 < 2.0 * c.Wc;
    for (int k = 0; k < c.nsh; ++k) kink |= in(c.gEs[k]);
    rec[0] = kink ? 1.0 : 0.0;
    rec[1] = 0.0;
    for (int k = 0; k < K; ++k) {
        const double a = v[0][k], b = v[1][k], d = v[2][k], e = v[3][k];
        double* q = rec + 2 + 4 * k;
        q[0] = b;
        q[1] = -a / 3.0 - b / 2.0 + d - e / 6.0;
        q[2] = a / 2.0 - b + d / 2.0;
        q[3] = (e - a) / 6.0 + (b - d) / 2.0;
    }
}

// Do two simulations have the same channel cross sections at every energy?
// (material, Wc and density enter; beam, range and Bethe settings do not)
inline bool same_sigma(const SimConst<double>& a, const SimConst<double>& b) {
    if (a.nsh != b.nsh) return false;
    if (a.cRs != b.cRs || a.aS != b.aS || a.ruth_r2 != b.ruth_r2 || a.pM != b.pM || a.Wc != b.Wc) return false;
    if (a.qK != b.qK || a.qC1 != b.qC1 || a.qInvEf != b.qInvEf || a.qB != b.qB || a.Epl != b.Epl) return false;
    for (int k = 0; k < a.nsh; ++k)
        if (a.gEs[k] != b.gEs[k] || a.gP[k] != b.gP[k] || a.gInvEs[k] != b.gInvEs[k]) return false;
    return true;
}

// Group the DS simulations of a batch by same_sigma; each group shares the
// table in its first member's slot, on a log2 grid over the union of the
// members' [Emin, E0] ranges.
inline void share_sigma_tables(const mcd_sim* sims, int nsims, const SimConst<double>* cd, SimConst<float>* cs,
                               const uint8_t* ws_dev) {
    for (int k = 0; k < nsims; ++k) {
        if (sims[k].mode != MCD_MODE_DS) continue;
        int lead = k;
        for (int j = 0; j < k; ++j)
            if (sims[j].mode == MCD_MODE_DS && cs[j].sig == reinterpret_cast<const float*>(
                                                                ws_dev + batch_sig_off(nsims) + batch_sig_bytes() * j) &&
                same_sigma(cd[j], cd[k])) {
                lead = j;
                break;
            }
        cs[k].sig = reinterpret_cast<const float*>(ws_dev + batch_sig_off(nsims) + batch_sig_bytes() * lead);
    }
    for (int k = 0; k < nsims; ++k) {
        if (sims[k].mode != MCD_MODE_DS) continue;
        const float* slot = reinterpret_cast<const float*>(ws_dev + batch_sig_off(nsims) + batch_sig_bytes() * k);
        if (cs[k].sig != slot) continue;
        double lo = sims[k].Emin, hi = sims[k].E0;
        for (int j = k + 1; j < nsims; ++j)
            if (cs[j].sig == slot) {
                lo = fmin(lo, sims[j].Emin);
                hi = fmax(hi, sims[j].E0);
            }
        float l0, inv, tmax;
        int32_t rows;
        sigma_grid(lo, hi, &l0, &inv, &tmax, &rows);
        for (int j = k; j < nsims; ++j)
            if (cs[j].sig == slot) {
                cs[j].sig_l0 = l0;
                cs[j].sig_inv = inv;
                cs[j].sig_tmax = tmax;
                cs[j].sig_rows = rows;
                cs[j].sig_off = -l0 * inv;
            }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
template <class T, int MODE, bool REC>
static int launch_plain(const SimConst<T>& c, int block, mcd_tally* tally, const ElOut& eo,
                        const mcd_event_ring& ring, uint32_t* status, cudaStream_t st) {
    const unsigned long long grid = ((unsigned long long)c.num_el + block - 1) / block;
    if (grid == 0) return MCD_OK;
    if (grid > 0x7fffffffull) return MCD_ETOOBIG;
    k_plain<T, MODE, REC><<<(unsigned)grid, block, 0, st>>>(c, round_keys(c), tally, eo, ring, status);
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}

template <class T>
static int dispatch_plain(const SimConst<T>& c, int block, mcd_tally* tally, const ElOut& eo,
                          const mcd_event_ring& ring, bool rec, uint32_t* status, cudaStream_t st) {
    if (c.mode == MCD_MODE_DS)
        return rec ? launch_plain<T, MCD_MODE_DS, true>(c, block, tally, eo, ring, status, st)
                   : launch_plain<T, MCD_MODE_DS, false>(c, block, tally, eo, ring, status, st);
    return rec ? launch_plain<T, MCD_MODE_CONT, true>(c, block, tally, eo, ring, status, st)
               : launch_plain<T, MCD_MODE_CONT, false>(c, block, tally, eo, ring, status, st);
}

// Lanes per electron of an automatic run (mcd_lanes.cu): 0 for a thread per
// electron.  More lanes make an electron's chain shorter, but a warp issues
// for fewer electrons, so the width falls as the run fills the GPU; the lines
// (in electrons per SM) lie where the two sides measured equal on 152 SMs,
// kernel times in ms, 0 = a thread per electron (in FP32 DS as mcd_run.cu runs
// it):
//   FP32 DS (Si, table)  2500: 0.35 / 0.39 with 32 / 16;  3500: 0.49 / 0.43;
//                        4500: 0.48 / 0.49 with 16 / 8;  7500: 0.55 / 0.56
//                        with 8 / 0;  10000: 0.67 / 0.59
//   (Au: 3500 1.07 / 1.26 with 32 / 16, 4500 1.35 / 1.34 with 16 / 8, 7500
//   1.53 / 1.63 with 8 / 0, 10000 1.83 / 1.72; Cu without a table: 3500 0.88 /
//   0.85, 4500 0.95 / 1.08, 7500 1.21 / 1.23, 10000 1.36 / 1.32)
//   FP32 continuous (44 parameter sets of all materials, 32 / 8 lanes over 0, the
//                        mean and the worst): 10 per SM 0.91, 0.95 / 0.97, 0.99; 14:
//                        1.02, 1.13 / 0.97, 0.98;  18: 1.15, 1.33 / 1.01, 1.06; 33:
//                        1.54, 2.08 / 1.08, 1.19
//   FP64 DS (with their host calls; Si, table)  1200: 2.15 / 2.31 with 32 / 16,
//                        1400: 2.63 / 2.37;  2100: 2.60 / 2.82 with 16 / 8, 2500:
//                        3.76 / 3.10 (up to two warps per scheduler, both);
//                        6500: 4.9 / 5.35 with 8 / 0, 7500: 5.6 / 5.34
//   (Au: 1200 6.00 / 6.20 with 32 / 16, 1400 6.01 / 6.25, 2100 6.64 / 7.80 with
//   16 / 8, 2500 6.99 / 8.14, 9000 21.2 / 26.3 with 8 / 0)
//   without a table      Si 7000: 15.7 / 16.5 with 8 / 0, 9000 19.9 / 16.7; Cu
//                        9000: 25.4 / 29.8, 11000 35.3 / 29.0; Au 14000: 63 / 116
//                        (the plain kernel evaluates a cross section per
//                        shell in every event)
//   FP64 continuous (Cu) 450: 3.72 / 3.82 with 32 / 8, 700: 4.21 / 3.85;  2500:
//                        4.53 / 4.83 with 8 / 0, 4000: 5.93 / 5.08
static int lanes_per_electron(const mcd_sim& s, const mcd_material& m, int sms) {
    const int64_t e = s.num_el / sms;   // electrons per SM
    if (s.precision == MCD_FP32) {
        if (s.mode != MCD_MODE_DS) return e < 12 ? 32 : e < 16 ? 8 : 0;
        return e < 20 ? 32 : e < 33 ? 16 : e < 58 ? 8 : 0;
    }
    if (s.mode != MCD_MODE_DS) return e < 3 ? 32 : e < 18 ? 8 : 0;
    const int most = s.sigma_table ? 47 : 16 * (m.n_shells > 3 ? m.n_shells : 3);
    return e < 8 ? 32 : e < 16 ? 16 : e < most ? 8 : 0;
}

// Does an automatic run of a thread per electron take one resident block per
// SM that refills its lanes and compacts its warps (mcd_run.cu), or blocks of
// independent threads?  The first keeps warps full where trajectory lengths
// differ; its barriers and its own loop cost a few percent where they do not.
// Kernel times in ms, this against independent threads:
//   FP32 DS    always (10000 electrons: Cu 1.32 / 1.96, Au 1.72 / 2.74, Si 0.59
//              / 0.75; 80000: Cu 2.23 / 2.66, Au 3.16 / 4.01, Si 0.88 / 0.98;
//              1e6: Cu 12.6 / 21.5, Au 12.9 / 33.4, Si 5.7 / 8.0)
//              but for the thinnest films, of an event or two, while the independent
//              threads are all resident at once (30 A at 5 keV, 300 to 1000 electrons
//              per SM: 1.0 to 1.14 of their time; 100 A at 15 keV 0.9 to 1.16; 100 A at
//              5 keV 0.5 to 1.1, at 30 keV 0.96 to 1.14)
//   FP32 continuous, whose lengths differ by backscattering alone: only where
//              they differ much (tilted beams, heavy elements) and the run is
//              large; up to 1024 electrons per SM the independent threads are all
//              resident at once.  The line moves up as trajectories get shorter,
//              as the ends weigh more.  Time over that of independent threads:
//                electrons per SM      300   400   600   800  1000  1300  2500  5000
//                Al  5 keV 60 deg     1.20  1.16  1.09  1.01  1.01  1.03  0.96  0.91
//                Al  5 keV 75 deg     1.24  1.16  1.08  1.02  0.97  0.86  0.85  0.78
//                Al 10 keV 60 deg     1.17  1.07  1.02  0.94  0.99  1.02  0.92  0.87
//                Al 30 keV 60 deg     1.09  1.00  0.93  0.84  0.92  0.96  0.87  0.82
//                Al 30 keV  0 deg     1.17  1.01  1.01  0.92  1.26  1.19  1.07  0.99
//                Cu  5 keV 60 deg     1.16  1.07  1.00  0.89  0.93  0.82  0.82  0.74
//                Cu 30 keV 60 deg     1.06  0.92  0.84  0.73  0.76  0.74  0.69  0.67
//                Cu 30 keV  0 deg     1.08  0.98  0.92  0.81  1.10  0.95  0.94  0.86
//                Au  5 keV  0 deg     1.11  0.96  0.89  0.77  0.78  0.74  0.76  0.68
//                Au 30 keV  0 deg     1.04  0.88  0.81  0.69  0.73  0.73  0.68  0.66
//                Au 30 keV 75 deg     0.93  0.77  0.71  0.56  0.56  0.48  0.40  0.37
//              (500: within 0.1 above 400; films of 1000 A, in which light elements
//              and fast beams make short trajectories: Al 10 keV 60 deg 500: 1.18,
//              1000: 1.06, 2500: 0.80; Cu 30 keV 75 deg 1.13, 1.15, 0.81; Cu 10 keV
//              80 deg 0.98, 0.70, 0.47)
static bool one_block_per_sm(const mcd_sim& s, const mcd_material& m, int sms) {
    const int64_t e = s.num_el / sms;   // electrons per SM
    if (s.precision != MCD_FP32 || e > INT32_MAX / 2) return false;
    const bool film = s.thickness > 0 && s.thickness < 1e30;
    if (s.mode == MCD_MODE_DS) return !(film && s.thickness < 0.007 * s.E0 && e <= 1024);
    if (s.E0 < 10.0 * s.Emin) return false;   // short trajectories: the start and the end weigh more
    if (film && (m.Z < 25 || s.E0 > 15e3) && e <= 1024) return false;
    if (m.Z >= 40) return e >= (s.E0 >= 10e3 || s.s_tilt >= 60.0 ? 400 : 600);
    if (s.s_tilt >= 60.0 && m.Z >= 25) return e >= (s.E0 >= 20e3 ? 400 : 600);
    if (s.s_tilt >= 60.0) return e >= (s.E0 >= 8e3 ? 800 : 1300);
    return m.Z >= 25 && e >= 4000;
}

}  // namespace mcd

using namespace mcd;

extern "C" int mcd_run(const mcd_sim* sim, const mcd_material* mat, const mcd_table* moller,
                       const mcd_table* gryz, mcd_tally* tally, const mcd_electron_out* electrons,
                       const mcd_event_ring* ring, uint32_t* status, int32_t block_size, void* stream) {
    if (!sim || !mat || !tally || !status) return MCD_EINVAL;
    const int rc = check_sim(*sim, *mat, moller, gryz);
    if (rc != MCD_OK) return rc;
    // automatic: a small run takes several lanes per electron (mcd_lanes.cu),
    // a larger one a thread per electron
    int group = 0, sms = 0;
    bool resident = false;
    if (block_size <= 0) {
        block_size = 128;
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return MCD_ECUDA;
        group = lanes_per_electron(*sim, *mat, sms);
        resident = group == 0 && one_block_per_sm(*sim, *mat, sms);
        // a thread per electron: 128 threads, halved (down to 8) while the
        // grid would leave SMs idle, so that a small job spreads over the GPU;
        // FP64 further, down to 2 while the grid stays within one warp per
        // scheduler (4 per SM): fewer lanes per warp diverge less
        while (block_size > 8 && (sim->num_el + block_size - 1) / block_size < sms) block_size /= 2;
        if (sim->precision == MCD_FP64)
            while (block_size > 2 && 2 * ((sim->num_el + block_size - 1) / block_size) <= 4ll * sms) block_size /= 2;
    }
    if (!(block_size < 32 ? (block_size & (block_size - 1)) == 0 : block_size % 32 == 0) || block_size > 256)
        return MCD_EINVAL;
    ElOut eo{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    if (electrons) {
        eo.outcome = electrons->outcome;
        eo.flags = electrons->flags;
        eo.final_E = electrons->final_E;
        eo.dir = electrons->dir;
        eo.last_pos = electrons->last_pos;
        eo.max_z = electrons->max_z;
        eo.n_events = electrons->n_events;
    }
    mcd_event_ring rg{nullptr, 0, nullptr};
    bool rec = false;
    if (ring && ring->rec && ring->cursor && ring->capacity > 0) {
        if (ring->fields & ~(MCD_EV_ALL | MCD_EV_PACKED_HEAD)) return MCD_EINVAL;
        if ((ring->fields & MCD_EV_PACKED_HEAD) && sim->num_el > (1ll << 28)) return MCD_EINVAL;
        rg = *ring;
        rec = true;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const mcd_table* tm = sim->mode == MCD_MODE_DS ? moller : nullptr;
    const mcd_table* tg = sim->mode == MCD_MODE_DS ? gryz : nullptr;
    if (sim->precision == MCD_FP64) {
        const SimConst<double> c = make_consts<double>(*sim, *mat, tm, tg);
        if (group) return launch_lanes<double>(c, group, tally, eo, rg, rec, status, st);
        return dispatch_plain<double>(c, block_size, tally, eo, rg, rec, status, st);
    }
    const SimConst<float> c = make_consts<float>(*sim, *mat, tm, tg);
    if (group) return launch_lanes<float>(c, group, tally, eo, rg, rec, status, st);
    if (resident) return launch_run(c, sms, tally, electrons ? *electrons : mcd_electron_out{}, rg, rec, status, st);
    return dispatch_plain<float>(c, block_size, tally, eo, rg, rec, status, st);
}

extern "C" size_t mcd_sigma_table_bytes(void) { return kSigTableBytes; }

extern "C" int mcd_build_sigma_table(const mcd_sim* sim, const mcd_material* mat, void* table, void* stream) {
    if (!sim || !mat || !table) return MCD_EINVAL;
    if (sim->mode != MCD_MODE_DS) return MCD_EINVAL;
    if (sim->precision != MCD_FP32 && sim->precision != MCD_FP64) return MCD_EINVAL;
    if (sim->elastic < MCD_ELASTIC_RUTH || sim->elastic > MCD_ELASTIC_NIGRAM_WDEFL) return MCD_EINVAL;
    if (!(sim->E0 > sim->Emin) || !(sim->Emin > 0) || !(sim->Wc > 0)) return MCD_EINVAL;
    if (mat->n_shells < 0 || mat->n_shells > MCD_MAX_SHELLS || mat->atnd <= 0) return MCD_EINVAL;
    if ((reinterpret_cast<uintptr_t>(table) & 15) != 0) return MCD_EINVAL;   // rows are read as float4
    if (sim->precision == MCD_FP64 && sigma_bytes64(sim->Emin, sim->E0, mat->n_shells + 3) > kSigTableBytes)
        return MCD_ETOOBIG;
    mcd_sim s = *sim;
    s.sigma_table = table;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (sim->precision == MCD_FP64) {
        const SimConst<double> c = make_consts<double>(s, *mat, nullptr, nullptr);
        const int n = c.sig_rows * kSig64Cells;
        k_sigtab64<<<(n + 127) / 128, 128, 0, st>>>(c, (int)c.sig_l0, c.sig_rows, static_cast<double*>(table));
        return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
    }
    s.precision = MCD_FP32;
    SimConst<double> c = make_consts<double>(s, *mat, nullptr, nullptr);
    k_sigtab_one<<<(c.sig_rows + 255) / 256, 256, 0, st>>>(c, c.sig_l0, c.sig_inv, c.sig_rows, c.sig_S,
                                                            static_cast<float*>(table));
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}

extern "C" size_t mcd_batch_workspace_bytes(int32_t nsims) {
    if (nsims <= 0 || nsims > kBatchMaxSims) return 0;
    return batch_bytes(nsims);
}

extern "C" size_t mcd_batch_list_bytes(int64_t electrons) {
    if (electrons <= 0) return 0;
    return sizeof(uint32_t) * kSeatWords * (size_t)(electrons < kLiveSeats ? electrons : kLiveSeats);
}

extern "C" size_t mcd_batch_upload_bytes(int32_t nsims) {
    if (nsims <= 0 || nsims > kBatchMaxSims) return 0;
    return batch_sig_off(nsims);
}

extern "C" int mcd_batch_prepare(const mcd_sim* sims, int32_t nsims, const mcd_material* mats,
                                 const int32_t* sim_material, const mcd_table* tables, const int32_t* sim_moller,
                                 const int32_t* sim_gryz, void* workspace, size_t workspace_bytes, void* stream) {
    return mcd_batch_prepare_list(sims, nsims, mats, sim_material, tables, sim_moller, sim_gryz, workspace,
                                  workspace_bytes, nullptr, 0, stream);
}

extern "C" int mcd_batch_prepare_list(const mcd_sim* sims, int32_t nsims, const mcd_material* mats,
                                      const int32_t* sim_material, const mcd_table* tables,
                                      const int32_t* sim_moller, const int32_t* sim_gryz, void* workspace,
                                      size_t workspace_bytes, void* list, size_t list_bytes, void* stream) {
    if (!sims || !mats || !sim_material || !workspace) return MCD_EINVAL;
    if (nsims <= 0) return MCD_EINVAL;
    if (nsims > kBatchMaxSims) return MCD_ETOOBIG;
    if (workspace_bytes < batch_bytes(nsims)) return MCD_EINVAL;
    if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0) return MCD_EINVAL;
    if ((reinterpret_cast<uintptr_t>(list) & 3) != 0) return MCD_EINVAL;
    const size_t bytes = batch_sig_off(nsims);   // everything but the tables, which the GPU fills
    uint8_t* host = static_cast<uint8_t*>(calloc(1, bytes));
    if (!host) return MCD_EINVAL;
    SimConst<double>* cd = reinterpret_cast<SimConst<double>*>(host + batch_dconsts_off(nsims));
    BatchHeader* h = reinterpret_cast<BatchHeader*>(host);
    unsigned long long* pre = reinterpret_cast<unsigned long long*>(host + batch_prefix_off());
    int32_t* perm = reinterpret_cast<int32_t*>(host + batch_perm_off(nsims));
    SimConst<float>* cs = reinterpret_cast<SimConst<float>*>(host + batch_consts_off(nsims));
    int rc = MCD_OK;
    for (int k = 0; k < nsims && rc == MCD_OK; ++k) {
        const mcd_sim& s = sims[k];
        const mcd_material& m = mats[sim_material[k]];
        const mcd_table* tm = nullptr;
        const mcd_table* tg = nullptr;
        if (s.mode == MCD_MODE_DS) {
            if (!tables || !sim_moller || !sim_gryz) { rc = MCD_EINVAL; break; }
            tm = &tables[sim_moller[k]];
            tg = &tables[sim_gryz[k]];
        }
        rc = check_sim(s, m, tm, tg);
        if (rc != MCD_OK) break;
        if (s.precision != MCD_FP32) { rc = MCD_EINVAL; break; }
        cs[k] = make_consts<float>(s, m, tm, tg);
        cd[k] = make_consts<double>(s, m, tm, tg);
    }
    if (rc == MCD_OK) share_sigma_tables(sims, nsims, cd, cs, static_cast<const uint8_t*>(workspace));
    if (rc == MCD_OK) pack_rows(sims, nsims, host);
    batch_order(sims, nsims, perm);
    unsigned long long acc = 0;
    for (int q = 0; q < nsims; ++q) {
        pre[q] = acc;
        acc += (unsigned long long)sims[perm[q]].num_el;
    }
    pre[nsims] = acc;
    h->queue = 0;
    h->total = acc;
    h->nsims = nsims;
    for (int k = 0; k < nsims; ++k) h->chan |= (sims[k].tally_flags & MCD_TALLY_CHANNELS) ? 1 : 0;
    const size_t seats = list ? list_bytes / (sizeof(uint32_t) * kSeatWords) : 0;
    h->list = static_cast<uint32_t*>(list);
    h->list_cap = (int32_t)(seats < (size_t)kLiveSeats ? seats : (size_t)kLiveSeats);
    if (rc == MCD_OK) {
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        const unsigned grid = (unsigned)(((long long)nsims * kSigRowsMax + 255) / 256);
        if (cudaMemcpyAsync(workspace, host, bytes, cudaMemcpyHostToDevice, st) != cudaSuccess) rc = MCD_ECUDA;
        else {
            k_sigtab<<<grid, 256, 0, st>>>(static_cast<uint8_t*>(workspace), nsims);
            if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) rc = MCD_ECUDA;
        }
    }
    free(host);
    return rc;
}

// The launch tuning of a batched run; MCD_OK or why it is refused.
static int read_tune(const mcd_tune* tune, int* block, int* per_sm, int* refill) {
    *block = 256;
    *per_sm = 0;
    *refill = 1;
    if (tune) {
        if (tune->block_size > 0) *block = tune->block_size;
        if (tune->blocks_per_sm > 0) *per_sm = tune->blocks_per_sm;
        if (tune->refill > 0) *refill = tune->refill;
    }
    if (*block % 32 != 0 || *block > 1024 || *refill < 1 || *refill > 32 || (tune && tune->reserved != 0))
        return MCD_EINVAL;
    return MCD_OK;
}

// The persistent launch and, where the list can hold an electron per lane and
// the run-down kernel's block fits, that kernel after it.
template <bool REC>
static int launch_batched(void* workspace, int nsims, mcd_tally* tallies, const mcd_tune* tune,
                          const mcd_event_ring& ring, uint32_t* status, bool lowreg, cudaStream_t st) {
    int block, per_sm, refill;
    if (read_tune(tune, &block, &per_sm, &refill) != MCD_OK) return MCD_EINVAL;
    int flags = (tune && (tune->variant & 2)) ? kRunInline : 0;
    if (lowreg && block > 576) return MCD_EINVAL;
    int dev = 0, sms = 0, most = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return MCD_ECUDA;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return MCD_ECUDA;
    if (cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return MCD_ECUDA;
    const size_t smem = batch_smem(nsims), smem2 = batch_drain_off(nsims) + drain_smem(kDrainThreads);
    auto kern = k_batched<REC>;
    if constexpr (!REC) kern = lowreg ? k_batched_lr<false> : k_batched<false>;
    if (allow_smem((const void*)kern, smem) != MCD_OK) return MCD_ECUDA;
    int fit = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, block, smem) != cudaSuccess) return MCD_ECUDA;
    if (fit < 1) return MCD_ETOOBIG;
    if (per_sm <= 0 || per_sm > fit) per_sm = fit;
    if ((long long)sms * per_sm * block <= kLiveSeats && smem2 + 1024 <= (size_t)most) flags |= kRunList;
    auto down = nsims == 1 ? k_rundown<REC, true> : k_rundown<REC, false>;
    if ((flags & kRunList) && allow_smem((const void*)down, smem2) != MCD_OK) return MCD_ECUDA;
    // reset the queue and the list (the first two words of the workspace)
    if (cudaMemsetAsync(workspace, 0, 2 * sizeof(unsigned long long), st) != cudaSuccess) return MCD_ECUDA;
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    kern<<<sms * per_sm, block, smem, st>>>(ws, tallies, refill, status, ring, flags);
    if (cudaGetLastError() != cudaSuccess) return MCD_ECUDA;
    if (flags & kRunList) down<<<sms, kDrainThreads, smem2, st>>>(ws, tallies, status, ring, flags);
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}

extern "C" int mcd_run_batched(void* workspace, int32_t nsims, mcd_tally* tallies, const mcd_tune* tune,
                               uint32_t* status, void* stream) {
    if (!workspace || !tallies || !status) return MCD_EINVAL;
    if (nsims <= 0) return MCD_EINVAL;
    if (nsims > kBatchMaxSims) return MCD_ETOOBIG;
    return launch_batched<false>(workspace, nsims, tallies, tune, mcd_event_ring{}, status,
                                 tune && (tune->variant & 1), static_cast<cudaStream_t>(stream));
}

// Batched run that also appends every event to a device ring (the streaming
// path): the caller drains the ring between launches (mcd.stream).
extern "C" int mcd_run_batched_ring(void* workspace, int32_t nsims, mcd_tally* tallies, const mcd_tune* tune,
                                    const mcd_event_ring* ring, uint32_t* status, void* stream) {
    if (!workspace || !tallies || !status || !ring || !ring->rec || !ring->cursor || ring->capacity == 0)
        return MCD_EINVAL;
    if (ring->fields & ~(MCD_EV_ALL | MCD_EV_PACKED_HEAD)) return MCD_EINVAL;
    if (nsims <= 0) return MCD_EINVAL;
    if (nsims > kBatchMaxSims) return MCD_ETOOBIG;
    return launch_batched<true>(workspace, nsims, tallies, tune, *ring, status, false,
                                static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------
// Batched run that allocates nothing.
//
// Some callers cannot call cudaMalloc: an application that embeds this
// library and owns all device memory through its own arena, or a caller on a
// latency budget for which an allocation (which can synchronise the device)
// is not acceptable.  This variant keeps the batched kernel's scratch (queue
// counter, electron prefix sums and packed simulation constants) in a
// file-scope device array instead of a caller workspace.  The array holds at
// most kStaticMaxSims simulations and stays resident on every GPU that loads
// the library until the process exits.  Every call shares it and rewrites it
// in full (the queue counter starts at zero each call), so calls that overlap
// on the GPU - two streams, or two host threads - race on it and must not be
// issued concurrently.
//
// The host packs the scratch and hands it to a staging kernel as one
// by-value argument (kernel arguments may take up to 32764 bytes), which
// writes it into the array ahead of the transport launch on the same
// stream: no host buffer has to outlive the call, and nothing is copied
// from pageable memory.
// ---------------------------------------------------------------------------
#include <mutex>

namespace mcd {

constexpr int kStaticMaxSims = MCD_STATIC_MAX_SIMS;
constexpr size_t kStaticHeadBytes = batch_consts_off(kStaticMaxSims);
constexpr size_t kStaticScratchBytes = batch_core_bytes(kStaticMaxSims);
static_assert(kStaticScratchBytes % 16 == 0, "the scratch is staged as 16-byte words");

struct StaticBlock {
    uint4 w[kStaticScratchBytes / 16];
};
static_assert(sizeof(StaticBlock) + 16 <= 32764, "the packed scratch must fit the kernel argument space");

static __device__ __align__(256) uint8_t g_static_scratch[kStaticScratchBytes];

// Writes the first `words` 16-byte words of the packed block to dst.
__global__ void __launch_bounds__(256) k_static_stage(uint4* dst, const StaticBlock blk, uint32_t words) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x)
        dst[i] = blk.w[i];
}

constexpr int kStaticMaxDevices = 64;
static std::mutex g_static_mu;
static void* g_static_ptr[kStaticMaxDevices];

// The device address of g_static_scratch on the current device, looked up
// once per device (host code may not use the symbol itself as an address).
// The address belongs to the device's primary context: a cudaDeviceReset
// makes it stale, so the library must not be used across one.
static int static_scratch(void** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return MCD_ECUDA;
    if (dev < 0 || dev >= kStaticMaxDevices) return MCD_EINVAL;
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || !p) return MCD_ECUDA;
        g_static_ptr[dev] = p;
    }
    *out = g_static_ptr[dev];
    return MCD_OK;
}

}  // namespace mcd

extern "C" int mcd_run_batched_noalloc(const mcd_sim* sims, int32_t nsims, const mcd_material* mats,
                                       const int32_t* sim_material, const mcd_table* tables,
                                       const int32_t* sim_moller, const int32_t* sim_gryz, mcd_tally* tallies,
                                       const mcd_tune* tune, uint32_t* status, void* stream) {
    if (!sims || !mats || !sim_material || !tallies || !status) return MCD_EINVAL;
    if (nsims <= 0) return MCD_EINVAL;
    if (nsims > kStaticMaxSims) return MCD_ETOOBIG;
    int block = 256, per_sm = 0, refill = 1;
    if (tune) {
        if (tune->block_size > 0) block = tune->block_size;
        if (tune->blocks_per_sm > 0) per_sm = tune->blocks_per_sm;
        if (tune->refill > 0) refill = tune->refill;
    }
    if (block % 32 != 0 || block > 1024 || refill < 1 || refill > 32 || (tune && tune->reserved != 0))
        return MCD_EINVAL;
    // the variant bits of mcd_run_batched: bit 0 the 56-register kernel,
    // bit 1 inline cross sections (a caller-built sigma_table is then not read)
    const bool lowreg = tune && (tune->variant & 1);
    const int inline_sigma = (tune && (tune->variant & 2)) ? 1 : 0;
    if (lowreg && block > 576) return MCD_EINVAL;

    // pack on the host: header (queue = 0), prefix sums, constants, row pointers
    StaticBlock blk;
    uint8_t* host = reinterpret_cast<uint8_t*>(&blk);
    memset(host, 0, kStaticHeadBytes);
    BatchHeader* h = reinterpret_cast<BatchHeader*>(host);
    unsigned long long* pre = reinterpret_cast<unsigned long long*>(host + batch_prefix_off());
    int32_t* perm = reinterpret_cast<int32_t*>(host + batch_perm_off(nsims));
    SimConst<float>* cs = reinterpret_cast<SimConst<float>*>(host + batch_consts_off(nsims));
    for (int k = 0; k < nsims; ++k) {
        const mcd_sim& s = sims[k];
        const mcd_material& m = mats[sim_material[k]];
        const mcd_table* tm = nullptr;
        const mcd_table* tg = nullptr;
        if (s.mode == MCD_MODE_DS) {
            if (!tables || !sim_moller || !sim_gryz) return MCD_EINVAL;
            tm = &tables[sim_moller[k]];
            tg = &tables[sim_gryz[k]];
        }
        const int rc = check_sim(s, m, tm, tg);
        if (rc != MCD_OK) return rc;
        if (s.precision != MCD_FP32) return MCD_EINVAL;
        cs[k] = make_consts<float>(s, m, tm, tg);
    }
    batch_order(sims, nsims, perm);
    unsigned long long acc = 0;
    for (int q = 0; q < nsims; ++q) {
        pre[q] = acc;
        acc += (unsigned long long)sims[perm[q]].num_el;
    }
    pre[nsims] = acc;
    h->queue = 0;
    h->total = acc;
    h->nsims = nsims;
    for (int k = 0; k < nsims; ++k) h->chan |= (sims[k].tally_flags & MCD_TALLY_CHANNELS) ? 1 : 0;
    pack_rows(sims, nsims, host);
    // the core only: cross sections come from the callers' tables or are
    // evaluated inline
    const uint32_t words = (uint32_t)((batch_core_bytes(nsims) + 15) / 16);

    void* scratch = nullptr;
    int rc = static_scratch(&scratch);
    if (rc != MCD_OK) return rc;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return MCD_ECUDA;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return MCD_ECUDA;
    const size_t smem = batch_smem(nsims);
    auto kern = lowreg ? k_batched_lr<false> : k_batched<false>;
    if (allow_smem((const void*)kern, smem) != MCD_OK) return MCD_ECUDA;
    int fit = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, block, smem) != cudaSuccess) return MCD_ECUDA;
    if (fit < 1) return MCD_ETOOBIG;
    if (per_sm <= 0 || per_sm > fit) per_sm = fit;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    k_static_stage<<<(words + 255) / 256, 256, 0, st>>>(static_cast<uint4*>(scratch), blk, words);
    if (cudaGetLastError() != cudaSuccess) return MCD_ECUDA;
    kern<<<sms * per_sm, block, smem, st>>>(static_cast<uint8_t*>(scratch), tallies, refill, status,
                                            mcd_event_ring{}, inline_sigma ? kRunInline : 0);
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}
