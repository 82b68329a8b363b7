// mcd_group.cuh - a DS event run by the G lanes of a group in lockstep, every
// lane holding the electron's state (mcd_lanes.cu says why).
#ifndef MCD_GROUP_CUH
#define MCD_GROUP_CUH

#include "mcd_tally.cuh"

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
    constexpr int NS = (MCD_MAX_SHELLS + G - 1) / G;
    T sG[NS];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        const int s = t + q * G;
        sG[q] = s < c.nsh ? sig_gryz<T>(c, E, invE, s & (MCD_MAX_SHELLS - 1)) : (T)0;
    }
    T cum = sR + sM;
    const T after_moller = cum;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        const int col = t + q * G;
        k.col[q] = col == 1 ? sR : col == 2 ? after_moller : kBig;
    }
#pragma unroll
    for (int p = 0; p < NS; ++p) {
        for (int s = p * G; s < c.nsh && s < (p + 1) * G; ++s) {
            cum += __shfl_sync(gmask, sG[p], h0 + s - p * G);
#pragma unroll
            for (int q = 0; q < N; ++q)
                if (t + q * G == 3 + s) k.col[q] = cum;
        }
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

// The lanes of one group
template <int G>
struct GroupLanes {
    int t, h0;               // lane within the group; its first lane
    unsigned gmask;
    static constexpr unsigned ones = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
    __device__ __forceinline__ explicit GroupLanes(int lane)
        : t(lane & (G - 1)), h0(lane & ~(G - 1)), gmask(ones << (lane & ~(G - 1))) {}
};

// (FP64) A Rutherford event's sin^2(theta/2) and what the direction update takes
// of it: cos(theta) and sin(theta) cos(phi), sin(theta) sin(phi).  They depend on
// the energy and on the event's random values alone, so each lane computes them
// for its event of those ahead, and again when the energy has changed: 23 of the
// event's 48 FP64 instructions, which most events then need not issue.  1000 Si 10
// keV electrons 2.30 -> 2.03 ms, 1000 Au 20 keV 7.75 -> 5.50 (with their host
// calls).  In FP32, where the instructions are cheap and the shared memory's
// latency is not, the same lost 3 to 6%.
struct GroupAngle {
    double s2, cth, a, b;
};
__device__ __forceinline__ GroupAngle group_deflect(double s2, double cph, double sph) {
    const double sth = 2.0 * Ops<double>::sqrt_(s2 * (1.0 - s2));   // the operations of lane_rotate_cs
    return GroupAngle{s2, 1.0 - 2.0 * s2, sth * cph, sth * sph};
}
template <class C>
__device__ __forceinline__ GroupAngle group_angle(const C& c, double E, const EventPre<double>& p) {
    return group_deflect(ruth_s2<double>(c, E, p.a0u, p.uzc), p.cph, p.sph);
}

// What an FP64 event takes of the angles computed ahead and leaves to group_turn
struct GroupTurn {
    GroupAngle t;    // of the event as a Rutherford one; then the event's
    bool due;        // the direction is to be updated
    bool changed;    // the energy has changed, and goes on
};

// lane_rotate_cs by the lanes of a group, called by the whole warp: lane q of
// the first six computes component q mod 3 of the new direction (q < 3) or of
// the new y axis with the operations of lane_rotate_cs in their order, and
// every lane of the group receives all six.  The FP64 pipe takes 16 cycles for
// a warp instruction and a small run's warps share it, so 25 of the event's 77
// FP64 instructions (35 of the update become 10) are time, and the shuffles
// that come instead are not: 1000 Si 10 keV electrons 2.72 -> 2.37 ms, 700 Au 20
// keV 9.76 -> 7.98, 3000 Si 3.74 -> 3.22, 1000 Cu in the continuous model 4.08 ->
// 3.82 (with their host calls).
template <int G>
__device__ __forceinline__ void group_turn(Lane<double>& L, const GroupTurn& turn, double cph, double sph,
                                           const GroupLanes<G>& g) {
    const double cth = turn.t.cth, a = turn.t.a, b = turn.t.b;
    const int q = g.t % 6, i = q % 3;
    const bool axis = q >= 3;
    auto pick = [](int k, double x, double y, double z) { return k == 0 ? x : k == 1 ? y : z; };
    const double d0 = pick(i, L.dx, L.dy, L.dz), d1 = pick(i, L.dy, L.dz, L.dx), d2 = pick(i, L.dz, L.dx, L.dy);
    const double y0 = pick(i, L.yx, L.yy, L.yz), y1 = pick(i, L.yy, L.yz, L.yx), y2 = pick(i, L.yz, L.yx, L.yy);
    const double x = fma(y1, d2, -(y2 * d1));
    const double v = fma(y0, axis ? 0.0 : b, fma(axis ? y0 : d0, axis ? cph : cth, x * (axis ? -sph : a)));
    const int src = g.h0 + (axis ? 3 : 0);
    const double u0 = __shfl_sync(0xffffffffu, v, src), u1 = __shfl_sync(0xffffffffu, v, src + 1),
                 u2 = __shfl_sync(0xffffffffu, v, src + 2);
    const double w = v * Ops<double>::renorm(fma(u2, u2, fma(u0, u0, u1 * u1)));
    double n[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) n[k] = __shfl_sync(0xffffffffu, w, g.h0 + k);
    if (!turn.due) return;
    L.dx = n[0];
    L.dy = n[1];
    L.dz = n[2];
    L.yx = n[3];
    L.yy = n[4];
    L.yz = n[5];
}

constexpr int kGroupNone = -1;    // the group took no event (no electron, or at the event limit)
constexpr int kGroupPlain = -2;   // a Rutherford event that stays in the sample

// One DS event of every group of a warp, but in FP64 for its direction update,
// which is left in *turn (called by all its lanes; active: the group has an
// electron; cur: its event's values computed ahead).  Returns the channel code,
// kGroupNone or kGroupPlain; the step counter has advanced unless it is
// kGroupNone.  plain: the events below which an event that loses no energy may
// go on without the test E > Emin: the limit, or 0 for a beam that is not above
// Emin (group_plain), whose electrons end with their first event.
template <class T, bool REC, int G, class C>
__device__ __forceinline__ int group_event(Lane<T>& L, GroupSig<T, G>& sig, const C& c, const EventPre<T>& cur,
                                           bool active, uint32_t limit, uint32_t plain, const GroupLanes<G>& g, T zmax,
                                           bool use_tab, EventOut<T>* ev, GroupTurn* turn = nullptr) {
    // the columns passed: 0 Rutherford, 1 Moller, 2.. Gryz, K-1 Quinn
    const T level = cur.ux * sig.all;
    unsigned below = 0;
#pragma unroll
    for (int q = 0; q < GroupSig<T, G>::N; ++q) {
        const unsigned b = __ballot_sync(0xffffffffu, sig.col[q] < level);
        below |= ((b >> g.h0) & GroupLanes<G>::ones) << (q * (G & 31));
    }
    below >>= 1;   // column 0 is no channel's
    // (an FP32 table counts them, the others stop at the first)
    const int j = sizeof(T) == 4 && sig.tab ? __popc(below) : __ffs(~below) - 1;
    const bool dif = (c.bits & kBitDiff) && level > sig.tot;
    if (!active) return kGroupNone;
    // what a Rutherford event does; the others replace it
    const T E = L.E;
    T W = (T)0, s2, path = -cur.ln_y * sig.mfp;
    if constexpr (sizeof(T) == 8) s2 = turn->t.s2;
    else s2 = ruth_s2<T>(c, E, cur.a0u, cur.uzc);
    int ch = MCD_CH_RUTH;
    if (sizeof(T) == 4) {
        // a Rutherford event that stays in the sample changes nothing but the
        // position and the directions: FP32 takes it on a path of its own
        // with one branch (37 Au electrons 1.12 -> 0.74 ms); in FP64, where
        // the groups of a warp would each issue their own rotation, it lost
        // (1000 Si electrons 2.42 -> 2.96 ms)
        const T nz = L.z + path * L.dz;
        if (j == 0 && !dif && !(nz <= (T)0) && !(nz >= zmax) && L.step < plain) {
            if (REC) event_out<T>(*ev, L, E, W, path, s2, cur.rw, ch);
            L.step += 1;
            lane_move(L, c, path);
            lane_rotate_cs(L, s2, cur.cph, cur.sph);
            return kGroupPlain;
        }
    }
    if (L.step >= limit) {   // the 'long' check that opens every event (MC/tools/singleScatter.py:19-23)
        lane_long(L);
        return kGroupNone;
    }
    L.step += 1;
    bool loss = false;
    if (j != 0 || dif) {
        const int K = bits_K(c);
        // a table's diffraction is tested first, the expressions' after
        // every other channel
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
            W = group_table_pick<T, G>(c.tab[ch != MCD_CH_MOLLER], E, Ops<T>::unit(cur.rz), g.t, g.h0, g.gmask, &oor);
            if (oor) L.flags |= F_TABLE_RANGE;
            s2 = collide(L, c, E, W);
        }
        const T after = E - W;
        if (loss && after > c.Emin) {
            group_sig<T, G>(c, after, use_tab, g.t, g.h0, g.gmask, sig);
            if constexpr (sizeof(T) == 8) turn->changed = true;
        }
    }
    if (REC) event_out<T>(*ev, L, E, W, path, s2, cur.rw, ch);
    lane_move(L, c, path, ch == MCD_CH_DIFF);
    if ((loss || plain == 0) && (L.outcome == MCD_OUT_NONE || (c.bits & MCD_Q_CROSSING_STEP))) lane_lose(L, c, W);
    if constexpr (sizeof(T) == 8) {
        if (ch != MCD_CH_RUTH) turn->t = group_deflect(s2, cur.cph, cur.sph);
        turn->due = L.outcome == MCD_OUT_NONE;
    } else if (L.outcome == MCD_OUT_NONE) {
        lane_rotate_cs(L, s2, cur.cph, cur.sph);
    }
    return ch;
}

// group_event's `plain`: FP32 can round E0 to Emin (E0 > Emin is checked in FP64)
template <class T>
__device__ __forceinline__ uint32_t group_plain(const SimConst<T>& c) {
    return sizeof(T) == 8 || c.E0 > c.Emin ? c.max_scatt : 0u;
}

// the bottom face as group_event tests it
template <class T, class C>
__device__ __forceinline__ T group_zmax(const C& c) {
    return (c.bits & kBitFilm) ? c.thickness : (T)INFINITY;
}

}  // namespace mcd

#endif  // MCD_GROUP_CUH
