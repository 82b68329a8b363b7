// mcd_drain.cuh - running down the electrons of FP32 simulations that no new
// ones follow.
//
// Trajectory lengths differ by an order of magnitude, so once no electrons are
// left to refill lanes with (or where there never were more than lanes) warps
// run on with a few lanes each, and a warp with one busy lane issues as many
// instructions as a full one.  Here a block, one per SM, takes its share of the
// electrons (the ones a persistent kernel listed when its queue ran empty, or
// the whole of a run of middling size), refills its lanes from the share, and
// then advances in windows of kWindow events with a barrier after each.  There
// the electrons of its emptiest warps move, through shared memory, into the
// idle lanes of the others, so that as few warps as possible carry them; once
// the block has no more electrons than an eighth of its threads, they go on as
// the small-run kernel runs them (mcd_lanes.cu): eight lanes per electron in
// windows, then, when there are no more than one in 32, a warp per electron to
// the end.  No electron's draws or arithmetic depend on where it runs.
#ifndef MCD_DRAIN_CUH
#define MCD_DRAIN_CUH

#include "mcd_group.cuh"

namespace mcd {

constexpr int kDrainThreads = 512;   // one block per SM at up to 128 registers
// Events between meetings, one lane and eight lanes per electron.  Windows of 32,
// 64, 128 and 256 events were within 3% of each other (1e5 Au, 20011 Cu electrons).
constexpr int kWindow = 128;
constexpr int kGroupWindow = 64;
// Warps that keep electrons while there are enough: two per scheduler; below,
// fuller warps only diverge more, above, a warp issues for fewer lanes.  14, 20 and
// 28 take 0.99, 1.04 and 1.10 of the time for 1e5 Au electrons, 1.06 for 20011 Cu,
// 1.05 to 1.19 for a stream's chunk of 40000 Au.  (The continuous model, whose
// events are short, keeps one per scheduler: drain_run.)
constexpr int kKeepWarps = 8;

// An electron in shared memory: kSeatWords words at stride `stride`.
constexpr int kSeatWords = 17;
struct Seats {
    uint32_t* w;
    int stride;
};

__device__ __forceinline__ void seat_put(const Seats& p, int s, const Lane<float>& L, const ElecRng& g, int sim) {
    const float f[11] = {L.E, L.x, L.y, L.z, L.dx, L.dy, L.dz, L.yx, L.yy, L.yz, L.max_z};
    const uint32_t u[6] = {L.step, L.flags | ((uint32_t)sim << 8), L.odd_n, g.b, g.d, g.e};
#pragma unroll
    for (int k = 0; k < 11; ++k) p.w[k * p.stride + s] = __float_as_uint(f[k]);
#pragma unroll
    for (int k = 0; k < 6; ++k) p.w[(11 + k) * p.stride + s] = u[k];
}

__device__ __forceinline__ void seat_get(const Seats& p, int s, Lane<float>& L, ElecRng& g, int& sim) {
    const auto f = [&](int k) { return __uint_as_float(p.w[k * p.stride + s]); };
    L.E = f(0);
    L.x = f(1);
    L.y = f(2);
    L.z = f(3);
    L.dx = f(4);
    L.dy = f(5);
    L.dz = f(6);
    L.yx = f(7);
    L.yy = f(8);
    L.yz = f(9);
    L.max_z = f(10);
    L.step = p.w[11 * p.stride + s];
    const uint32_t u = p.w[12 * p.stride + s];
    L.flags = u & 0xffu;
    sim = (int)(u >> 8);
    L.odd_n = p.w[13 * p.stride + s];
    g.b = p.w[14 * p.stride + s];
    g.d = p.w[15 * p.stride + s];
    g.e = p.w[16 * p.stride + s];
    L.outcome = MCD_OUT_NONE;
    L.E_row = L.E;
}

// Seats of a block of b threads: for the moves between warps, and for the
// electrons that run several lanes wide, with one buffer of values computed
// ahead per warp that runs them.
__host__ __device__ constexpr int drain_move_seats(int b) { return b / 4; }
__host__ __device__ constexpr int drain_group_seats(int b) { return b / 8; }
__host__ __device__ constexpr int drain_solo_seats(int b) { return b / 32; }
__host__ __device__ constexpr size_t drain_group_bytes(int b) {
    return ((size_t)kSeatWords * 4 * drain_group_seats(b) + 15) & ~(size_t)15;
}
__host__ __device__ constexpr size_t drain_smem(int b) {
    const size_t a = (size_t)kSeatWords * 4 * drain_move_seats(b);
    const size_t g = drain_group_bytes(b) + sizeof(EventPre<float>) * (size_t)b;
    return a > g ? a : g;
}

// The block's count of electrons: every thread learns all warps' counts.
struct BlockCount {
    int mine;     // lane l: the count of warp l
    int total;
    int warps;    // warps with an electron
};
__device__ __forceinline__ BlockCount block_count(int count, int (*s_cnt)[32], int& parity) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) s_cnt[parity][warp] = count;
    __syncthreads();
    BlockCount b;
    b.mine = lane < (int)(blockDim.x >> 5) ? s_cnt[parity][lane] : 0;
    parity ^= 1;   // the other buffer next time: this one may still be read
    b.total = __reduce_add_sync(0xffffffffu, b.mine);
    b.warps = __popc(__ballot_sync(0xffffffffu, b.mine > 0));
    return b;
}

__device__ __forceinline__ int warp_exclusive(int v, int warp) {   // sum of lanes 0 .. warp - 1
    int incl = v;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    return __shfl_sync(0xffffffffu, incl - v, warp);
}

// Moves the electrons of the block's emptiest (last) warps into the idle lanes
// of the first ones when that frees a warp.  Called by the whole block.
__device__ __forceinline__ void drain_compact(const BlockCount& b, const Seats& seats, Lane<float>& L, ElecRng& rng,
                                              int& sim, bool& have, int least) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int keep = max((b.total + 31) / 32, least);
    if (b.warps <= keep) return;
    // high half: electrons that move; low half: idle lanes that stay
    const int v = lane < (int)(blockDim.x >> 5) ? (lane < keep ? 32 - b.mine : b.mine << 16) : 0;
    const int before = warp_exclusive(v, warp);
    const int moving = __reduce_add_sync(0xffffffffu, v) >> 16;
    if (moving > drain_move_seats((int)blockDim.x)) return;
    const unsigned m = __ballot_sync(0xffffffffu, have);
    if (warp >= keep && have) {
        seat_put(seats, (before >> 16) + __popc(m & lt), L, rng, sim);
        have = false;
    }
    __syncthreads();
    if (warp < keep && !have) {
        const int s = (before & 0xffff) + __popc(~m & lt);
        if (s < moving) {
            seat_get(seats, s, L, rng, sim);
            have = true;
        }
    }
}

// What a block's electrons need besides their state: the constants, block
// tallies, tallies and rows of their simulations.  MODE: the one mode they
// run, or kMixed.
constexpr int kMixed = 2;
struct ManySims {
    static constexpr int MODE = kMixed;
    const SimConst<float>* c_;
    BlockTally* t_;
    mcd_tally* tallies_;
    const mcd_electron_out* rows_;
    __device__ __forceinline__ const SimConst<float>& c(int sim) const { return c_[sim]; }
    __device__ __forceinline__ const SimConst<float>& full(int sim) const { return c_[sim]; }
    __device__ __forceinline__ BlockTally& t(int sim) const { return t_[sim]; }
    __device__ __forceinline__ mcd_tally* tally(int sim) const { return tallies_ + sim; }
    __device__ __forceinline__ const mcd_electron_out& rows(int sim) const { return rows_[sim]; }
};
template <int M, class C>
struct OneSim {
    static constexpr int MODE = M;
    const SimConst<float>& full_;
    const C& c_;   // what its events read: the same, or a HotConst
    BlockTally& t_;
    mcd_tally* tally_;
    const mcd_electron_out& rows_;
    __device__ __forceinline__ const C& c(int) const { return c_; }
    __device__ __forceinline__ const SimConst<float>& full(int) const { return full_; }
    __device__ __forceinline__ BlockTally& t(int) const { return t_; }
    __device__ __forceinline__ mcd_tally* tally(int) const { return tally_; }
    __device__ __forceinline__ const mcd_electron_out& rows(int) const { return rows_; }
};

template <class Sims>
__device__ __forceinline__ uint32_t run_finish(const Sims& s, int sim, const Lane<float>& L, const ElecRng& rng) {
    const SimConst<float>& c = s.full(sim);
    const mcd_electron_out& r = s.rows(sim);
    const ElOut eo{r.outcome, r.flags, r.final_E, r.dir, r.last_pos, r.max_z, r.n_events};
    return finish_electron(c, L, elec_index(c, rng) - c.first, s.t(sim), s.tally(sim), eo);
}

template <class Sims, class C>
__device__ __forceinline__ bool run_cont(const C& c) {
    return Sims::MODE == MCD_MODE_CONT || (Sims::MODE == kMixed && (c.bits & kBitCont));
}

// Runs the electrons of a warp's groups, which have had an event (so that their
// energy is above Emin), for up to `events` events each.
template <bool REC, bool CHAN, int G, class Sims>
__device__ __forceinline__ uint32_t group_run(const Sims& s, int sim, Lane<float>& L, const ElecRng& rng, bool& have,
                                              int events, EventPre<float>* buf, const mcd_event_ring& ring,
                                              bool inline_sigma) {
    const int lane = threadIdx.x & 31;
    const GroupLanes<G> g(lane);
    const auto& c = s.c(sim);
    const uint4 w = event_words(c);
    const bool cont = run_cont<Sims>(c);
    const bool use_tab = !inline_sigma && c.sig != nullptr;
    const float zmax = group_zmax<float>(c), ang = cont ? 1.0f : c.a0;
    GroupSig<float, G> sig{};
    if (have && !cont) group_sig<float, G>(c, L.E, use_tab, g.t, g.h0, g.gmask, sig);
    uint32_t st = 0;
    EventPre<float> cur{}, next{};
    for (int k = 0; k < events; ++k) {
        if (!__any_sync(0xffffffffu, have)) break;
        if ((k & (G - 1)) == 0) {   // the next G events' values, one event per lane
            __syncwarp();
            buf[lane] = event_pre<float>(c, philox_event(rng, L.step + (uint32_t)g.t, w), ang);
            __syncwarp();
            cur = buf[g.h0];
        } else {
            cur = next;
        }
        next = buf[g.h0 + ((k + 1) & (G - 1))];
        EventOut<float> ev;
        RingTicket tk{};
        uint32_t el = 0;
        if (REC) {
            el = (uint32_t)(elec_index(s.full(sim), rng) - s.full(sim).first);
            const bool rec = g.t == 0 && have && L.step < w.w;
            tk = ring_reserve(ring, rec && ring_takes(ring, el));
            if (rec && !ring_takes(ring, el)) st |= MCD_FLAG_RING_INDEX;
        }
        int ch = kGroupNone;
        if (Sims::MODE != MCD_MODE_CONT)
            ch = group_event<float, REC, G>(L, sig, c, cur, have && !cont, w.w, w.w, g, zmax, use_tab, &ev);
        if (have && cont) {
            if (L.step >= w.w) {
                lane_long(L);
            } else {
                L.step += 1;
                ch = cont_event_r<float, REC>(L, c, make_uint4(0u, 0u, cur.rz, cur.rw), &ev, &cur);
            }
        }
        if (REC) ring_write(ring, ring_slot(ring, tk), el, L.step, ev);
        if (ch != kGroupPlain && have) {
            if (CHAN && g.t == 0 && ch > MCD_CH_RUTH) atomicAdd(&s.t(sim).channel[ch], 1ull);
            if (L.outcome != MCD_OUT_NONE) {
                if (g.t == 0) st |= run_finish(s, sim, L, rng);
                have = false;
            }
        }
    }
    __syncwarp();
    return st;
}

// The block's last electrons (at most drain_group_seats), several lanes wide,
// to their end.  Called by the whole block.
template <bool REC, bool CHAN, class Sims>
__device__ __forceinline__ uint32_t drain_groups(const Sims& s, BlockCount b, uint8_t* smem, int (*s_cnt)[32], int parity,
                                              Lane<float> L, ElecRng rng, int sim, bool have,
                                              const mcd_event_ring& ring, bool inline_sigma) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int threads = (int)blockDim.x;
    const Seats seats{reinterpret_cast<uint32_t*>(smem), drain_group_seats(threads)};
    EventPre<float>* bufs = reinterpret_cast<EventPre<float>*>(smem + drain_group_bytes(threads));
    uint32_t st = 0;
    bool wide = false;   // `have` is per group of eight lanes
    for (;;) {
        // the electrons take seats in order
        const unsigned m = __ballot_sync(0xffffffffu, have && (!wide || (lane & 7) == 0));
        const int at = warp_exclusive(b.mine, warp) + __popc(m & lt);
        if ((m >> lane) & 1u) seat_put(seats, at, L, rng, sim);
        __syncthreads();
        const bool solo = b.total <= drain_solo_seats(threads);
        const int slot = solo ? warp : warp * 4 + (lane >> 3);
        have = slot < b.total;
        if (have) seat_get(seats, slot, L, rng, sim);
        if (__any_sync(0xffffffffu, have)) {
            if (!have) sim = 0;
            EventPre<float>* buf = bufs + warp * 32;
            if (solo) return st | group_run<REC, CHAN, 32>(s, sim, L, rng, have, 0x7fffffff, buf, ring, inline_sigma);
            st |= group_run<REC, CHAN, 8>(s, sim, L, rng, have, kGroupWindow, buf, ring, inline_sigma);
        } else if (solo) {
            return st;
        }
        wide = true;
        b = block_count(__popc(__ballot_sync(0xffffffffu, have && (lane & 7) == 0)), s_cnt, parity);
        if (b.total == 0) return st;
    }
}

// Runs a block's share of electrons: `count` of them, the k-th (claimed by one
// lane) put into a lane by take(k, L, rng, sim).  Called by the whole block
// with the tallies zeroed and the constants in place.
template <bool REC, bool CHAN, class Sims, class Take>
__device__ __forceinline__ uint32_t drain_run(const Sims& run, unsigned count, Take take, uint8_t* smem,
                                              const mcd_event_ring& ring, bool inline_sigma) {
    __shared__ int s_cnt[2][32];
    __shared__ unsigned s_next;
    if (threadIdx.x == 0) s_next = blockDim.x;   // with more electrons than threads every thread has one
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int threads = (int)blockDim.x;
    Lane<float> L;
    ElecRng rng{0u, 0u, 0u};
    int sim = 0;
    uint32_t st = 0;
    // the first electrons go evenly to as few warps as hold them, but to
    // kKeepWarps at least; the others to lanes as they fall idle
    const int least = Sims::MODE == MCD_MODE_CONT ? 4 : kKeepWarps;
    const unsigned wide = min(max((count + 31u) / 32u, (unsigned)least), blockDim.x >> 5);
    const unsigned first = (unsigned)lane * wide + (threadIdx.x >> 5);
    bool have = (threadIdx.x >> 5) < wide && first < count;
    if (have) take(first, L, rng, sim);
    auto event = [&]() {
        const auto& c = run.c(sim);
        EventOut<float> ev;
        RingTicket tk{};
        uint32_t el = 0;
        if (REC) {
            el = (uint32_t)(elec_index(run.full(sim), rng) - run.full(sim).first);
            const bool rec = L.step < event_words(c).w;
            tk = ring_reserve(ring, rec && ring_takes(ring, el));
            if (rec && !ring_takes(ring, el)) st |= MCD_FLAG_RING_INDEX;
        }
        int ch;
        if (run_cont<Sims>(c)) ch = cont_event<float, REC>(L, c, rng, &ev);
        else ch = ds_event<float, REC>(L, c, rng, &ev, !inline_sigma && c.sig != nullptr);
        if (REC) ring_write(ring, ring_slot(ring, tk), el, L.step, ev);
        if (CHAN && ch > MCD_CH_RUTH) atomicAdd(&run.t(sim).channel[ch], 1ull);
        if (L.outcome != MCD_OUT_NONE) {
            st |= run_finish(run, sim, L, rng);
            have = false;
        }
    };
    for (bool more = count > blockDim.x; more;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !have);
        if (idle) {   // the idle lanes take the share's next electrons
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(&s_next, (unsigned)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, 0);
            const unsigned k = base + (unsigned)__popc(idle & lt);
            if (!have && k < count) {
                take(k, L, rng, sim);
                have = true;
            }
            more = base + (unsigned)__popc(idle) < count;
        }
        if (have) event();
    }
    for (int parity = 0;;) {
        for (int k = 0; have && k < kWindow; ++k) event();
        __syncwarp();
        const BlockCount b = block_count(__popc(__ballot_sync(0xffffffffu, have)), s_cnt, parity);
        if (b.total == 0) break;
        if (b.total <= (Sims::MODE == MCD_MODE_CONT ? drain_solo_seats(threads) : drain_group_seats(threads))) {
            st |= drain_groups<REC, CHAN>(run, b, smem, s_cnt, parity, L, rng, sim, have, ring, inline_sigma);
            break;
        }
        drain_compact(b, Seats{reinterpret_cast<uint32_t*>(smem), drain_move_seats(threads)}, L, rng, sim, have, least);
    }
    return st;
}

}  // namespace mcd

#endif  // MCD_DRAIN_CUH
