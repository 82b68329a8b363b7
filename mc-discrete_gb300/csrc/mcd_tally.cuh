// mcd_tally.cuh - per-block tallies and per-electron rows, shared by the
// transport kernels.
#ifndef MCD_TALLY_CUH
#define MCD_TALLY_CUH

#include "mcd_device.cuh"

namespace mcd {

// Per-block sums; the per-event counters (events, channels) are 64-bit, as
// one persistent block can see more than 2^32 events of a channel.
// Channel counts (MCD_TALLY_CHANNELS): every event of an electron has one
// channel, so only the others are counted event by event and Rutherford's
// count is the rest of `events` at the flush.  Counting it per event too put
// up to 32 lanes of every warp on one 64-bit shared counter, a serialised
// compare-and-swap loop: six uneven simulations (5.5e7 events) took 17.5 ms
// for it, 9.4 ms without.
struct BlockTally {
    unsigned int outcome[8];
    unsigned int double_rows, nan_events, clamped, long_path, table_range, pad_;
    unsigned long long events;
    double sum_E, sum_E2, sum_steps2;
    unsigned long long channel[MCD_MAX_CHANNELS];
};
static_assert(sizeof(BlockTally) == 14 * 4 + (1 + 3 + MCD_MAX_CHANNELS) * 8, "bt_fold's fields");

__device__ __forceinline__ void bt_zero(BlockTally* t, int n) {
    unsigned int* p = reinterpret_cast<unsigned int*>(t);
    const int words = n * (int)(sizeof(BlockTally) / 4);
    for (int i = threadIdx.x; i < words; i += blockDim.x) p[i] = 0u;
}

// A block of many warps keeps several copies of its n tallies, so that fewer warps
// meet at one: FP64 and 64-bit additions in shared memory are compare-and-swap
// loops.  Adds copies 1 .. (n tallies apart) to the first; called by the whole
// block after a barrier.
// Measured, one copy for the 28 warps of the resident kernel and one for each: a
// 30 A film, 1e6 Si electrons 1.52 -> 0.13 ms; 152000 Si 5 keV electrons with channel
// counts 2.19 -> 0.87, 1e6 13.5 -> 3.65; 150000 film electrons as a batch 0.16 -> 0.07.
__device__ __forceinline__ void bt_fold(BlockTally* t, int n, int copies) {
    constexpr int kWords = 14, kFields = kWords + 1 + 3 + MCD_MAX_CHANNELS;   // 32-bit; events; sums; channels
    auto fold = [&](auto* p) {
        auto s = *p;
        for (int c = 1; c < copies; ++c) {
            p = reinterpret_cast<decltype(p)>(reinterpret_cast<uint8_t*>(p) + sizeof(BlockTally) * n);
            s += *p;
        }
        return s;
    };
    for (int k = threadIdx.x; k < n * kFields; k += blockDim.x) {
        BlockTally& a = t[k / kFields];
        const int f = k % kFields;
        if (f < kWords) reinterpret_cast<unsigned int*>(&a)[f] = fold(reinterpret_cast<unsigned int*>(&a) + f);
        else if (f == kWords) a.events = fold(&a.events);
        else if (f < kWords + 4) (&a.sum_E)[f - kWords - 1] = fold(&a.sum_E + (f - kWords - 1));
        else a.channel[f - kWords - 4] = fold(&a.channel[f - kWords - 4]);
    }
}

__device__ __forceinline__ void add_u64(unsigned long long* p, unsigned long long v) {
    if (v) atomicAdd(p, v);
}

__device__ __forceinline__ void bt_flush(const BlockTally& t, mcd_tally* g, bool chan) {
    // called by one thread per simulation
    unsigned long long others = 0;
    for (int k = 1; chan && k < MCD_MAX_CHANNELS; ++k) others += t.channel[k];
    bool any = t.events != 0 || others != 0;
    for (int k = 0; k < 8; ++k) any |= t.outcome[k] != 0;
    if (!any) return;
    for (int k = 0; k < 8; ++k) add_u64(&g->outcome[k], t.outcome[k]);
    add_u64(&g->events, t.events);
    add_u64(&g->double_rows, t.double_rows);
    add_u64(&g->nan_events, t.nan_events);
    add_u64(&g->clamped, t.clamped);
    add_u64(&g->long_path, t.long_path);
    add_u64(&g->table_range, t.table_range);
    if (chan) {
        for (int k = 1; k < MCD_MAX_CHANNELS; ++k) add_u64(&g->channel[k], t.channel[k]);
        // an electron's events are counted where it ends, which may be
        // another block than ran some of them: the differences add up modulo
        // 2^64
        add_u64(&g->channel[MCD_CH_RUTH], t.events - others);
    }
    if (t.sum_E != 0.0) atomicAdd(&g->sum_E_bks, t.sum_E);
    if (t.sum_E2 != 0.0) atomicAdd(&g->sum_E2_bks, t.sum_E2);
    if (t.sum_steps2 != 0.0) atomicAdd(&g->sum_steps2, t.sum_steps2);
}

struct ElOut {
    uint8_t* outcome;
    uint8_t* flags;
    void* final_E;
    void* dir;
    void* last_pos;
    void* max_z;
    int32_t* n_events;
};

template <class T, class C>
__device__ __forceinline__ uint32_t finish_electron(const C& c, const Lane<T>& L, uint64_t i, BlockTally& bt,
                                                    mcd_tally* gt, const ElOut& eo) {
    atomicAdd(&bt.outcome[L.outcome & 7], 1u);
    atomicAdd(&bt.events, (unsigned long long)L.step);
    atomicAdd(&bt.sum_steps2, (double)L.step * (double)L.step);
    if (L.flags & F_DOUBLE_ROW) atomicAdd(&bt.double_rows, 1u);
    if (L.odd_n) atomicAdd((c.bits & kBitCont) ? &bt.long_path : &bt.nan_events, L.odd_n);
    if (L.flags & F_CLAMPED) atomicAdd(&bt.clamped, 1u);
    if (L.flags & F_TABLE_RANGE) atomicAdd(&bt.table_range, 1u);
    if (L.outcome == MCD_OUT_BKS) {
        const double e = (double)L.E_row;
        atomicAdd(&bt.sum_E, e);
        atomicAdd(&bt.sum_E2, e * e);
        if (c.hE > 0) {
            const T f = L.E_row * c.invWE;
            if (f >= (T)0 && f < (T)c.hE) atomicAdd(&gt->hist_E[(int)f], 1ull);
        }
        if (c.hT > 0) {
            const T th = Ops<T>::acos_deg(-L.dz) * c.invWT;
            if (th >= (T)0 && th < (T)c.hT) atomicAdd(&gt->hist_T[(int)th], 1ull);
        }
    }
    if (eo.outcome) eo.outcome[i] = (uint8_t)L.outcome;
    if (eo.flags) eo.flags[i] = (uint8_t)(L.flags & (F_DOUBLE_ROW | F_NAN));
    const size_t n = (size_t)c.num_el;
    if (eo.final_E) static_cast<T*>(eo.final_E)[i] = L.E_row;
    if (eo.dir) {
        T* d = static_cast<T*>(eo.dir);
        d[i] = L.dx;
        d[n + i] = L.dy;
        d[2 * n + i] = L.dz;
    }
    if (eo.last_pos) {
        T* p = static_cast<T*>(eo.last_pos);
        p[i] = L.x;
        p[n + i] = L.y;
        p[2 * n + i] = L.z;
    }
    if (eo.max_z) static_cast<T*>(eo.max_z)[i] = L.max_z;
    if (eo.n_events) eo.n_events[i] = (int32_t)L.step;
    uint32_t st = 0;
    if (L.flags & F_NAN) st |= MCD_FLAG_NAN;
    if (L.flags & F_TABLE_RANGE) st |= MCD_FLAG_TABLE_RANGE;
    if (L.flags & F_CLAMPED) st |= MCD_FLAG_CLAMPED;
    if (L.flags & F_LONG_PATH) st |= MCD_FLAG_LONG_PATH;
    if (L.outcome == MCD_OUT_LONG) st |= MCD_FLAG_LONG;
    return st;
}

// Called by every thread of the block; a block smaller than a warp (plain
// launches of 1 to 16 threads) leaves lanes that never exist, so the
// reduction names the lanes present (and meets them: they leave the event
// loop one by one).
__device__ __forceinline__ void or_status(uint32_t* status, uint32_t st) {
    const unsigned present = blockDim.x < 32 ? (1u << blockDim.x) - 1u : 0xffffffffu;
    const uint32_t w = __reduce_or_sync(present, st);
    if ((threadIdx.x & 31) == 0 && w) atomicOr(status, w);
}

}  // namespace mcd

#endif  // MCD_TALLY_CUH
