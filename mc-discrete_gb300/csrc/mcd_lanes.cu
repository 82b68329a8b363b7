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
//    with the draw, one entry per lane.
// The trajectories are the plain kernel's, bit for bit.
#include <cuda_runtime.h>
#include <stdint.h>

#include "mcd_lanes.h"

namespace mcd {

// What an electron's energy says about its next event.  Column k = 1, 2, ..
// is the running sum of the cross sections through channel k in pick order
// (Ruth, Moller, Gryz[0] ..), in the units of the draw's level U all; lane t
// of the group holds columns t, t + G, ..
template <class T, int G>
struct GroupSig {
    static constexpr int N = (kSigStride + G - 1) / G;
    T all, tot, mfp;   // level of U = 1; of the channels before diffraction; 1/sum(sigma)
    T col[N];
    bool tab;          // from a table, not the expressions
};

// The group's lanes evaluate the cross sections at E.
template <class T, int G, class C>
__device__ __forceinline__ void group_sig(const C& c, T E, bool use_tab, int t, int h0, unsigned gmask,
                                          GroupSig<T, G>& k) {
    constexpr int N = GroupSig<T, G>::N;
    constexpr T kBig = sizeof(T) == 4 ? (T)3.402823466e38 : (T)1.7976931348623157e308;
    const bool diff = (c.bits & kBitDiff) != 0;
    k.tab = use_tab;
    if (use_tab) {
        if constexpr (sizeof(T) == 4) {
            const SigRow row = sig_row_at(c, E);
            const int S = bits_S(c);
#pragma unroll
            for (int q = 0; q < N; ++q) {
                const int col = t + q * G;
                k.col[q] = kBig;
                if (col < S) {
                    const float x = __ldg(row.r0 + col), y = __ldg(row.r0 + S + col);
                    k.col[q] = fmaf(row.f, y - x, x);
                }
            }
            k.tot = __shfl_sync(gmask, k.col[0], h0);
            k.all = diff ? fmaf(E, c.dS, k.tot) : k.tot;
            k.mfp = Ops<T>::div(E, k.all);
            return;
        } else {
            const Sig64Cell cell = sig64_cell(c, E);
            if (cell.smooth()) {
                const int K = bits_K(c);
#pragma unroll
                for (int q = 0; q < N; ++q) {
                    const int col = t + q * G;
                    k.col[q] = col < K ? cell.at(col) : kBig;
                }
                k.mfp = __shfl_sync(gmask, k.col[0], h0);
                k.tot = 1.0;
                k.all = 1.0;
                if (diff) {
                    k.all = fma((double)c.dS, k.mfp, 1.0);
                    k.mfp = k.mfp / k.all;
                }
                return;
            }
            k.tab = false;
        }
    }
    // the expressions: one shell per lane, the sums in channel order
    const T invE = Ops<T>::div((T)1, E);
    const T sR = sig_ruth<T>(c, E);
    const T sM = sig_moller<T>(c, E, invE);
    const T sQ = sig_quinn<T>(c, E, invE);
    const T sG = t < c.nsh ? sig_gryz<T>(c, E, invE, t & (MCD_MAX_SHELLS - 1)) : (T)0;
    T cum = sR + sM;
    const T after_moller = cum;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        const int col = t + q * G;
        k.col[q] = col == 1 ? sR : col == 2 ? after_moller : kBig;
    }
    for (int s = 0; s < c.nsh; ++s) {
        cum += __shfl_sync(gmask, sG, h0 + s);
#pragma unroll
        for (int q = 0; q < N; ++q)
            if (t + q * G == 3 + s) k.col[q] = cum;
    }
    cum += sQ;
    k.tot = cum;
    k.all = diff ? cum + c.dS : cum;
    k.mfp = Ops<T>::div((T)1, k.all);
}

// The W table's draw (table_pick): the row, then the entries of the guide's
// range compared one per lane.
template <class T, int G>
__device__ __forceinline__ T group_table_pick(const TableDev& tb, T E, T U, int t, int h0, unsigned gmask,
                                              bool* oor) {
    const TableSpan sp = table_span<T>(tb, E, U, oor);
    const float* row = tb.cdf + (size_t)sp.row * (tb.nW - 1);
    int lo = sp.lo, hi = sp.hi;
    while (hi - lo > G) {   // masked entries (0) act as +inf
        const int mid = (lo + hi) >> 1;
        const float v = __ldg(row + mid);
        if (v != 0.0f && (T)v < U) lo = mid + 1; else hi = mid;
    }
    if (lo < hi) {   // the entries below U are a prefix of the range
        const float v = lo + t < hi ? __ldg(row + lo + t) : 0.0f;
        lo += __popc(__ballot_sync(gmask, v != 0.0f && (T)v < U));
    }
    return (T)__ldg(tb.Ws + lo);
}

template <class T>
__device__ __forceinline__ void event_out(EventOut<T>& ev, const Lane<T>& L, T E, T W, T path, T s2, uint32_t rw,
                                          int ch) {
    ev.E = E;
    ev.W = W;
    ev.pathl = path;
    ev.c2 = (T)1 - s2;
    ev.half_phi = (T)3.141592653589793 * Ops<T>::unit(rw);
    ev.x = L.x;
    ev.y = L.y;
    ev.z = L.z;
    ev.ch = ch;
}

template <class T, int MODE, bool REC, int G>
__global__ void __launch_bounds__(32) k_lanes(const SimConst<T> cp, mcd_tally* tally, const ElOut eo,
                                              const mcd_event_ring ring, uint32_t* status) {
    __shared__ BlockTally bt;
    __shared__ SimConst<T> c;
    __shared__ EventPre<T> pre[2][32];
    if (threadIdx.x == 0) c = cp;
    bt_zero(&bt, 1);
    __syncwarp();
    const int lane = threadIdx.x, t = lane & (G - 1), h0 = lane & ~(G - 1);
    const unsigned gones = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u, gmask = gones << h0;
    const uint64_t i = (uint64_t)blockIdx.x * (32 / G) + (uint64_t)(lane / G);
    bool active = i < (uint64_t)c.num_el;
    const ElecRng rng = elec_rng(c, c.first + i);
    const uint4 w = event_words(c);   // sim id and Philox key words, event limit
    const bool chan = (c.tally_flags & MCD_TALLY_CHANNELS) != 0;
    const T zmax = (c.bits & kBitFilm) ? c.thickness : (T)INFINITY;   // the bottom face
    const bool use_tab = c.sig != nullptr, diff = (c.bits & kBitDiff) != 0;
    Lane<T> L;
    lane_init(L, c);
    GroupSig<T, G> sig;
    if (MODE == MCD_MODE_DS) group_sig<T, G>(c, L.E, use_tab, t, h0, gmask, sig);
    // every electron of the warp that still runs is at the same event
    uint32_t step = 0, st = 0;
    pre[0][lane] = event_pre<T, MODE>(c, philox_event(rng, (uint32_t)t, w));
    __syncwarp();
    EventPre<T> cur = pre[0][h0];
    while (G == 32 ? active : __any_sync(0xffffffffu, active)) {
        if ((step & (G - 1)) == 0) {   // the block of events after this one
            pre[(step / G + 1) & 1][lane] = event_pre<T, MODE>(c, philox_event(rng, step + G + (uint32_t)t, w));
            __syncwarp();
        }
        const EventPre<T> next = pre[((step + 1) / G) & 1][h0 + (int)((step + 1) & (G - 1))];
        int j = 0;         // columns passed: 0 Rutherford, 1 Moller, 2.. Gryz, K-1 Quinn
        bool dif = false;
        if (MODE == MCD_MODE_DS) {
            const T level = cur.ux * sig.all;
            unsigned below = 0;
#pragma unroll
            for (int q = 0; q < GroupSig<T, G>::N; ++q) {
                const unsigned b = __ballot_sync(0xffffffffu, sig.col[q] < level);
                below |= ((b >> h0) & gones) << (q * (G & 31));
            }
            below >>= 1;   // column 0 is no channel's
            // (an FP32 table counts them, the others stop at the first)
            j = sizeof(T) == 4 && sig.tab ? __popc(below) : __ffs(~below) - 1;
            dif = diff && level > sig.tot;
        }
        // what a Rutherford event does; the others replace it
        const T E = L.E;
        T W = (T)0, s2 = (T)0, path = (T)0;
        int ch = MCD_CH_RUTH;
        bool plain = false;
        if (MODE == MCD_MODE_DS) {
            s2 = ruth_s2<T>(c, E, cur.a0u, cur.uzc);
            path = -cur.ln_y * sig.mfp;
            if (sizeof(T) == 4) {
                // a Rutherford event that stays in the sample changes nothing
                // but the position and the directions: FP32 takes it on a
                // path of its own with one branch (37 Au electrons 1.12 ->
                // 0.74 ms); in FP64, where the groups of a warp would each
                // issue their own rotation, it lost (1000 Si electrons 2.42
                // -> 2.96 ms)
                const T nz = L.z + path * L.dz;
                plain = j == 0 && !dif && !(nz <= (T)0) && !(nz >= zmax) && step < w.w;
            }
        }
        if (active && plain) {
            EventOut<T> ev;
            if (REC) event_out<T>(ev, L, E, W, path, s2, cur.rw, ch);
            L.step = step + 1;
            lane_move(L, c, path);
            lane_rotate_cs(L, s2, cur.cph, cur.sph);
            if (REC && t == 0) st |= ring_append(ring, (uint32_t)i, L.step, ev);
        } else if (active) {
            if (step >= w.w) {   // the 'long' check that opens every event (MC/tools/singleScatter.py:19-23)
                lane_long(L);
            } else {
                L.step = step + 1;
                EventOut<T> ev;
                if (MODE == MCD_MODE_DS) {
                    bool loss = false;
                    if (j != 0 || dif) {
                        const int K = bits_K(c);
                        // a table's diffraction is tested first, the
                        // expressions' after every other channel
                        if (dif && (sig.tab || j >= K - 1)) ch = MCD_CH_DIFF;
                        else if (j == 0) ch = MCD_CH_RUTH;
                        else if (j == 1) ch = MCD_CH_MOLLER;
                        else if (j >= K - 1) ch = MCD_CH_QUINN;
                        else ch = MCD_CH_GRYZ0 + (j - 2);
                        loss = ch != MCD_CH_RUTH && ch != MCD_CH_DIFF;
                        if (ch == MCD_CH_DIFF) {
                            path = -cur.ln_y * c.xip;
                            s2 = (T)0;
                        } else if (ch == MCD_CH_QUINN) {
                            W = c.Epl;
                            s2 = (T)0;
                        } else if (loss) {
                            bool oor = false;
                            W = group_table_pick<T, G>(c.tab[ch != MCD_CH_MOLLER], E, Ops<T>::unit(cur.rz), t, h0,
                                                       gmask, &oor);
                            if (oor) L.flags |= F_TABLE_RANGE;
                            s2 = collide(L, c, E, W);
                        }
                        const T after = E - W;
                        if (loss && after > c.Emin) group_sig<T, G>(c, after, use_tab, t, h0, gmask, sig);
                    }
                    if (REC) event_out<T>(ev, L, E, W, path, s2, cur.rw, ch);
                    lane_move(L, c, path, ch == MCD_CH_DIFF);
                    if (loss && (L.outcome == MCD_OUT_NONE || (c.bits & MCD_Q_CROSSING_STEP))) lane_lose(L, c, W);
                    if (L.outcome == MCD_OUT_NONE) lane_rotate_cs(L, s2, cur.cph, cur.sph);
                } else {
                    cont_event_r<T, REC>(L, c, make_uint4(0u, 0u, cur.rz, cur.rw), &ev, &cur);
                }
                if (t == 0) {
                    if (REC) st |= ring_append(ring, (uint32_t)i, L.step, ev);
                    if (chan && ch > MCD_CH_RUTH) atomicAdd(&bt.channel[ch], 1ull);
                }
            }
            if (L.outcome != MCD_OUT_NONE) {
                if (t == 0) st |= finish_electron(c, L, i, bt, tally, eo);
                active = false;
            }
        }
        cur = next;
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
