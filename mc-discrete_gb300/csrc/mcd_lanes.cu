// mcd_lanes.cu - transport of small runs, several lanes of a warp per electron.
//
// A small run lasts as long as its longest trajectory, one dependent chain of
// instructions (about five cycles an instruction where a scheduler has one
// warp), and most lanes of a GPU are idle.  Here the G lanes of a group run
// their electron's events in lockstep (every lane holds the same state) and
// share the work that need not be on the chain:
//  - each lane computes, for one of the G events that follow, what does not
//    depend on the trajectory: the event's Philox block, ln U of its step, the
//    azimuth's cos and sin, the uniforms of the channel pick and of the polar
//    angle.  The values pass through shared memory, two blocks of G events
//    deep, so that an event's are loaded while the one before it runs;
//  - the cross sections depend on the energy alone, which most events leave as
//    it is (62% in Si, 90% in Au), so they are evaluated where it changes, one
//    column of the table (or one shell's expression) per lane, and an event's
//    channel is one comparison per lane and a vote;
//  - a W table's interval is found by comparing the guide's range of entries
//    with the draw, one entry per lane;
//  - in FP64, whose pipe the warps of an SM share, the polar angles of the events
//    ahead are computed one per lane, again where the energy changes, and the
//    direction update's components one per lane (mcd_group.cuh).
// The trajectories are the plain kernel's, bit for bit.
#include <cuda_runtime.h>
#include <stdint.h>

#include "mcd_group.cuh"
#include "mcd_lanes.h"

namespace mcd {

// Blocks per SM that the registers must leave room for: what the automatic
// rule gives an SM at most (in FP64 the narrow groups' alone; spilling more
// there costs as much as it gains).
template <class T>
constexpr int lanes_blocks(int group) {
    return sizeof(T) == 4 ? (group == 8 ? 20 : 16) : (group == 8 ? 16 : 1);
}

// where the continuous FP64 event leaves its sin^2(theta/2)
__device__ __forceinline__ double* turn_s2(GroupTurn* t, double) { return &t->t.s2; }
__device__ __forceinline__ float* turn_s2(GroupTurn*, float) { return nullptr; }

template <class T, int MODE, bool REC, int G>
__global__ void __launch_bounds__(32, lanes_blocks<T>(G)) k_lanes(const SimConst<T> cp, mcd_tally* tally, const ElOut eo,
                                              const mcd_event_ring ring, uint32_t* status) {
    __shared__ BlockTally bt;
    __shared__ SimConst<T> full;
    __shared__ EventPre<T> pre[2][32];
    __shared__ GroupAngle angles[32];   // (FP64 DS) of the block of events under way
    if (threadIdx.x == 0) full = cp;
    bt_zero(&bt, 1);
    __syncwarp();
    const HotConst<T> c(full);
    const int lane = threadIdx.x;
    const GroupLanes<G> g(lane);
    const uint64_t i = (uint64_t)blockIdx.x * (32 / G) + (uint64_t)(lane / G);
    bool active = i < (uint64_t)full.num_el;
    const ElecRng rng = elec_rng(full, full.first + i);
    const uint4 w = event_words(c);   // sim id and Philox key words, event limit
    const bool chan = (full.tally_flags & MCD_TALLY_CHANNELS) != 0;
    const T zmax = group_zmax<T>(c);
    const uint32_t plain = group_plain(full);
    const bool use_tab = c.sig != nullptr;
    const T ang = MODE == MCD_MODE_DS ? c.a0 : (T)1;
    Lane<T> L;
    lane_init(L, full);
    GroupSig<T, G> sig;
    if (MODE == MCD_MODE_DS) group_sig<T, G>(c, L.E, use_tab, g.t, g.h0, g.gmask, sig);
    // every electron of the warp that still runs is at the same event
    uint32_t step = 0, st = 0;
    pre[0][lane] = event_pre<T>(c, philox_event(rng, (uint32_t)g.t, w), ang);
    __syncwarp();
    EventPre<T> cur = pre[0][g.h0];
    constexpr bool kAngles = sizeof(T) == 8 && MODE == MCD_MODE_DS;
    GroupTurn turn{};
    turn.changed = true;   // angles[] are of another block or energy
    while (G == 32 ? active : __any_sync(0xffffffffu, active)) {
        if ((step & (G - 1)) == 0) {   // the block of events after this one
            __syncwarp();   // it takes the place of one whose values other lanes may still be reading
            pre[(step / G + 1) & 1][lane] = event_pre<T>(c, philox_event(rng, step + G + (uint32_t)g.t, w), ang);
            __syncwarp();
            turn.changed = true;
        }
        GroupAngle angle_next{};
        if constexpr (kAngles) {
            if (G == 32 ? turn.changed : __any_sync(0xffffffffu, turn.changed)) {
                __syncwarp();
                angles[lane] = group_angle(c, L.E, pre[(step / G) & 1][lane]);
                __syncwarp();
                turn.t = angles[g.h0 + (int)(step & (G - 1))];
                turn.changed = false;
            }
            angle_next = angles[g.h0 + (int)((step + 1) & (G - 1))];
        }
        const EventPre<T> next = pre[((step + 1) / G) & 1][g.h0 + (int)((step + 1) & (G - 1))];
        EventOut<T> ev;
        RingTicket tk{};
        if (REC) {
            const bool rec = g.t == 0 && active && step < w.w, takes = ring_takes(ring, (uint32_t)i);
            tk = ring_reserve(ring, rec && takes);
            if (rec && !takes) st |= MCD_FLAG_RING_INDEX;
        }
        int ch = kGroupNone;
        turn.due = false;
        if (MODE == MCD_MODE_DS) {
            ch = group_event<T, REC, G>(L, sig, c, cur, active, w.w, plain, g, zmax, use_tab, &ev, &turn);
        } else if (active) {
            if (step >= w.w) {
                lane_long(L);
            } else {
                L.step = step + 1;
                ch = cont_event_r<T, REC>(L, c, make_uint4(0u, 0u, cur.rz, cur.rw), &ev, &cur,
                                          turn_s2(&turn, (T)0));
                if (sizeof(T) == 8) turn.t = group_deflect(turn.t.s2, (double)cur.cph, (double)cur.sph);
                turn.due = L.outcome == MCD_OUT_NONE;
            }
        }
        if constexpr (sizeof(T) == 8) {
            if (G < 32) __syncwarp();
            group_turn<G>(L, turn, cur.cph, cur.sph, g);
        }
        if (REC) ring_write(ring, ring_slot(ring, tk), (uint32_t)i, L.step, ev);
        if (ch != kGroupPlain && active) {
            if (g.t == 0 && chan && ch > MCD_CH_RUTH) atomicAdd(&bt.channel[ch], 1ull);
            if (L.outcome != MCD_OUT_NONE) {
                if (g.t == 0) st |= finish_electron(full, L, i, bt, tally, eo);
                active = false;
            }
        }
        cur = next;
        if (kAngles) turn.t = angle_next;
        ++step;
    }
    or_status(status, st);
    __syncwarp();
    if (lane == 0) bt_flush(bt, tally, chan);
}

template <class T, int MODE, bool REC, int G>
static int launch_g(const SimConst<T>& c, mcd_tally* tally, const ElOut& eo, const mcd_event_ring& ring,
                    uint32_t* status, cudaStream_t st) {
    const unsigned long long grid = ((unsigned long long)c.num_el + 32 / G - 1) / (32 / G);
    if (grid == 0) return MCD_OK;
    if (grid > 0x7fffffffull) return MCD_ETOOBIG;
    k_lanes<T, MODE, REC, G><<<(unsigned)grid, 32, 0, st>>>(c, tally, eo, ring, status);
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}

template <class T, int G>
static int launch_mode(const SimConst<T>& c, mcd_tally* tally, const ElOut& eo, const mcd_event_ring& ring, bool rec,
                       uint32_t* status, cudaStream_t st) {
    if (c.mode == MCD_MODE_DS)
        return rec ? launch_g<T, MCD_MODE_DS, true, G>(c, tally, eo, ring, status, st)
                   : launch_g<T, MCD_MODE_DS, false, G>(c, tally, eo, ring, status, st);
    return rec ? launch_g<T, MCD_MODE_CONT, true, G>(c, tally, eo, ring, status, st)
               : launch_g<T, MCD_MODE_CONT, false, G>(c, tally, eo, ring, status, st);
}

template <class T>
int launch_lanes(const SimConst<T>& c, int group, mcd_tally* tally, const ElOut& eo, const mcd_event_ring& ring,
                 bool rec, uint32_t* status, cudaStream_t st) {
    switch (group) {
        case 32: return launch_mode<T, 32>(c, tally, eo, ring, rec, status, st);
        case 16: return launch_mode<T, 16>(c, tally, eo, ring, rec, status, st);
        default: return launch_mode<T, 8>(c, tally, eo, ring, rec, status, st);
    }
}

template int launch_lanes<float>(const SimConst<float>&, int, mcd_tally*, const ElOut&, const mcd_event_ring&, bool,
                                 uint32_t*, cudaStream_t);
template int launch_lanes<double>(const SimConst<double>&, int, mcd_tally*, const ElOut&, const mcd_event_ring&, bool,
                                  uint32_t*, cudaStream_t);

}  // namespace mcd
