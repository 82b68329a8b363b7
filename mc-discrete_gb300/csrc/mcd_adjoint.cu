// mcd_adjoint.cu - pathwise gradients of continuous-mode exit-energy tallies.
//
// Continuous mode (MC/tools/singleScatter.py:205-239) changes the energy
// only through E_{k+1} = E_k - s_k S(E_k), with s_k = -ln(U_k) / sigma'(E_k)
// the Rutherford step (MC/tools/scattering.py:802-826) and S the Bethe law
// (MC/tools/stoppingPowers.py:112-215).  With the random numbers and the
// event sequence frozen (the event k* in which an electron leaves through
// the surface is fixed), the exit energy E_{k*} is a smooth function of the
// Bethe mean ionisation energy J and of the density n.  Its derivative follows
// the same recursion: with e_k = dE_k/dJ,
//
//   e_{k+1} = e_k (1 + s_k (dlnsig/dE S - dS/dE)) - s_k dS/dJ
//   dL/dJ   = sum over electrons of dL/dE_exit e_{k*};   dL/dn = 0  (s ~ 1/n, S ~ n)
//
// For one parameter that is as cheap as the adjoint recursion and needs no
// event twice: the forward pass carries e along, and the backward pass is one
// multiplication per electron.  The deepest z instead takes a reverse sweep: its
// derivative through the rotations grows by orders of magnitude along deep
// trajectories, so that another order of evaluation in FP32 gives other
// gradients there.  Its forward pass stores the state every 64 events; the
// backward pass recomputes each 64-event segment from its checkpoint and the
// Philox counters, then sweeps it in reverse.  Tallies are Gaussian-soft bins of
// the exit energy (or deepest z) of backscattered electrons,
// h_b = (1/N) sum exp(-(q - c_b)^2 / (2 sigma^2)),
// and their sum.
#include <cuda_runtime.h>
#include <stdint.h>

#include "mcd_device.cuh"

namespace mcd {

constexpr int kSeg = 64;  // events per checkpoint segment

struct AdjBuf {
    void* ckpt;        // T, [num_el] dE/dJ_scale, or (depth) max_ckpt x 8 x num_el (checkpoint-major)
    int32_t* kstar;    // exit event of 'bks' electrons, -1 otherwise
    void* E_exit;      // T
    int32_t max_ckpt;
    unsigned long long* queue;   // the forward pass's work queue, or nullptr
};

struct SoftHist {
    int32_t nbins;
    int32_t quantity;   // MCD_ADJ_EXIT_E or MCD_ADJ_MAX_DEPTH
    double lo, width, inv2s2, inv_s2;
    double inv_width, reach;   // 1 / width; 8 sigma
    // the same in FP32, for FP32 runs: their soft bins are evaluated in FP32
    // (and summed in FP64), so that an FP32 run issues no FP64 arithmetic
    // per electron -- the backward takes its electrons a few lanes at a time,
    // and the FP64 unit charges each of those instructions in full
    float f_lo, f_inv_width, f_width, f_inv2s2, f_inv_s2, f_reach;
};

constexpr int kDepthState = 8;   // E, z, d (3), y (3) per depth checkpoint

// Gaussian soft bins within 8 sigma of the quantity q, in the transport
// precision T: calls f(bin, weight, d = q - c_b)
template <class T>
__device__ __forceinline__ void soft_consts(const SoftHist& sh, T& lo, T& w, T& iw, T& i2, T& reach) {
    if constexpr (sizeof(T) == 8) {
        lo = sh.lo, w = sh.width, iw = sh.inv_width, i2 = sh.inv2s2, reach = sh.reach;
    } else {
        lo = sh.f_lo, w = sh.f_width, iw = sh.f_inv_width, i2 = sh.f_inv2s2, reach = sh.f_reach;
    }
}
template <class T>
__device__ __forceinline__ void soft_range(const SoftHist& sh, T q, T lo, T iw, T reach, int& b0, int& b1) {
    b0 = (int)floor((q - reach - lo) * iw - (T)0.5);
    b1 = (int)ceil((q + reach - lo) * iw - (T)0.5);
    b0 = b0 < 0 ? 0 : b0;
    b1 = b1 > sh.nbins - 1 ? sh.nbins - 1 : b1;
}
template <class T, class F>
__device__ __forceinline__ void soft_bins(const SoftHist& sh, T q, F f) {
    T lo, w, iw, i2, reach;
    soft_consts<T>(sh, lo, w, iw, i2, reach);
    int b0, b1;
    soft_range(sh, q, lo, iw, reach, b0, b1);
    for (int b = b0; b <= b1; ++b) {
        const T d = q - (lo + ((T)b + (T)0.5) * w);
        f(b, exp(-d * d * i2), d);
    }
}

template <class T, class C>
__device__ __forceinline__ T step_len(const C& c, T E, const ElecRng& g, int64_t k) {
    const uint4 r = philox_event(g, (uint32_t)k, event_words(c));
    return -Ops<T>::ln_step_word(r.y) * Ops<T>::div((T)1, sig_ruth<T>(c, E));
}

// dS/dE and dS/dJ_scale of the Bethe law at E (S itself returned in *S)
template <class T, class C>
__device__ __forceinline__ void stopping_derivs(const C& c, T E, T* S, T* SE, T* Sj) {
    const T s = stopping<T>(c, E);
    *S = s;
    if (c.bethe == MCD_BETHE_CLASSICAL) {
        *SE = Ops<T>::div(c.bP, E * E) - Ops<T>::div(s, E);
        *Sj = -Ops<T>::div(c.bP, E);                       // J dS/dJ, J = J0 * J_scale
    } else if (c.bethe == MCD_BETHE_JL) {
        *SE = Ops<T>::div(c.bP, E * (E + c.bkJ)) - Ops<T>::div(s, E);
        *Sj = Ops<T>::div(c.bP, E) * (Ops<T>::div(c.bkJ, E + c.bkJ) - (T)1);
    } else {
        *SE = Ops<T>::div(c.bX * c.bW, E * E) - Ops<T>::div(s, E);
        *Sj = (T)0;
    }
}

// d ln(sigma'_R)/dE
template <class T, class C>
__device__ __forceinline__ T dlnsig(const C& c, T E) {
    const T rel = (c.bits & kBitR2) ? (T)2 * (Ops<T>::div((T)1, E + (T)511000) - Ops<T>::div((T)1, E + (T)1024000))
                            : (T)0;
    return rel - Ops<T>::div((T)1, E + c.aS);
}

// dE/dJ_scale after an event of step s and loss dE = s S at the energy E, from
// its value e before it; ij = 1 / J_scale.  In terms of dE and s bP / E, which
// the event has computed, the derivatives of s and S take a dozen instructions.
// In FP64 the quotients share one reciprocal, of the product of their
// denominators: the FP64 pipe bounds the pass, and the four or five divisions
// were some 45 of the derivative's 57 FP64 instructions (the forward pass of 30000
// electrons, ms, without the derivative / with the divisions / with the
// reciprocal: Al 15 keV 4.70 / 5.73 / 5.20, Au 20 keV 17.8 / 21.3 / 19.9; the
// backward pass that it replaces, 5.07 and 12.7).  The explicit law has no J: its
// e stays the 0 it starts from.
template <class C>
__device__ __forceinline__ double tangent(const C& c, double E, double s, double dE, double e, double ij) {
    if (c.bethe != MCD_BETHE_CLASSICAL && c.bethe != MCD_BETHE_JL) return e;
    const double A = E + c.aS, D = c.bethe == MCD_BETHE_JL ? E + c.bkJ : 1.0;
    const double EA = E * A, N = c.bethe == MCD_BETHE_JL ? EA * D : EA;
    double r, iEA;   // 1 / N, 1 / EA
    double up;       // d ln(sigma'_R)/dE + 1/E = aS / (E A) + 2 (1/B - 1/C)
    if (c.bits & kBitR2) {
        const double BC = (E + 511000.0) * (E + 1024000.0), q = rcp_pos(N * BC);
        r = BC * q;
        iEA = c.bethe == MCD_BETHE_JL ? D * r : r;
        up = fma(c.aS, iEA, 2.0 * (1024000.0 - 511000.0) * (N * q));
    } else {
        r = rcp_pos(N);
        iEA = c.bethe == MCD_BETHE_JL ? D * r : r;
        up = c.aS * iEA;
    }
    const double iE = A * iEA;
    if (c.bethe == MCD_BETHE_CLASSICAL) {
        const double sb = s * (c.bP * iE);
        return fma(e, fma(dE, up, -(sb * iE)), fma(ij, sb, e));
    }
    const double sb = s * (c.bP * iE), q = EA * r, sq = sb * q;
    return fma(e, fma(dE, up, -sq), fma(ij, fma(-c.bkJ, sq, sb), e));
}
template <class C>
__device__ __forceinline__ float tangent(const C& c, float E, float s, float dE, float e, float ij) {
    using T = float;
    const T iE = Ops<T>::div((T)1, E), up = dE * (dlnsig<T>(c, E) + iE);   // s (dlnsig S + S / E)
    if (c.bethe == MCD_BETHE_CLASSICAL) {
        const T sb = s * Ops<T>::div(c.bP, E);
        return e + e * (up - sb * iE) + ij * sb;
    }
    if (c.bethe == MCD_BETHE_JL) {
        const T sb = s * Ops<T>::div(c.bP, E), q = Ops<T>::div((T)1, E + c.bkJ);
        return e + e * (up - sb * q) + ij * (sb - sb * (c.bkJ * q));
    }
    return e + e * (up - s * Ops<T>::div(c.bX, E) * c.bW * iE);
}

// The forward pass: every electron's full transport, with (exit energy) the
// derivative of its energy carried along or (depth) its checkpoints every kSeg
// events.  With a queue word (buf.queue) the grid is resident and
// a lane that finishes its electron takes the next from the queue, so that
// lanes do not idle while the longest trajectory of their warp runs (one
// thread per electron kept about 18 of 32 lanes busy); without one, each
// warp takes `range` = 32 consecutive electrons, one per lane.  An electron
// that ends leaves its event and its quantity; the soft bins are a pass of
// their own (k_adj_bins), for which all lanes of a warp work on one electron:
// here a lane or two at a time would evaluate some five bins each and add them
// to shared FP64 sums by compare-and-swap.  With the constants in registers
// and one vote per event, forward and backward with their host calls: exit
// energy of 1e6 Al electrons 2.97 -> 2.65 ms, depth of 3e5 1.76 -> 1.61 ms.  The
// derivative carried along costs the exit-energy pass 4% (1.69 -> 1.76 ms)
// and leaves 0.09 of the backward's 0.51 ms: together 2.62 -> 2.22 ms.  Its
// FP32 error against FP64 along the same events, over 40 parameter sets, is
// 3.6e-7 rms, the reverse sweep's was 4.0e-7.
template <class T, bool DEPTH>
__global__ void __launch_bounds__(256) k_adj_fwd(const SimConst<T> cp, const AdjBuf buf, uint32_t range,
                                                 double inv_j, mcd_tally* tally, uint32_t* status) {
    __shared__ SimConst<T> full;
    __shared__ unsigned long long s_cnt[9];
    if (threadIdx.x == 0) full = cp;
    if (threadIdx.x < 9) s_cnt[threadIdx.x] = 0ull;
    __syncthreads();
    const HotConst<T> c(full);
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const uint64_t n = (uint64_t)full.num_el;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint64_t pos = warp * range;
    const uint64_t end = buf.queue ? n : (pos + range < n ? pos + range : n);
    bool exhausted = false;
    T* ck = static_cast<T*>(buf.ckpt);
    uint32_t st = 0;
    Lane<T> L;
    uint64_t i = 0;
    ElecRng rng{0u, 0u, 0u};
    bool have = false;
    int mstar = 0;   // (depth) events up to the deepest point
    T zbest = (T)0;
    const T ij = (T)inv_j;
    T tan = (T)0;    // (exit energy) dE/dJ_scale
    while (true) {
        // the lanes without an electron; voted again only after a refill
        unsigned idle = __ballot_sync(0xffffffffu, !have);
        if (idle && !exhausted) {   // the idle lanes take the next electrons
            const unsigned cnt = (unsigned)__popc(idle);
            unsigned long long base = pos;
            if (buf.queue) {
                if (lane == 0) base = atomicAdd(buf.queue, (unsigned long long)cnt);
                base = __shfl_sync(0xffffffffu, base, 0);
            } else {
                pos += cnt;
            }
            const uint64_t j = base + (uint64_t)__popc(idle & lt);
            if (!have && j < end) {
                i = j;
                lane_init(L, full);
                rng = elec_rng(full, full.first + i);
                if (DEPTH) {
                    mstar = 0;
                    zbest = (T)0;
                } else {
                    tan = (T)0;
                }
                have = true;
            }
            if (base + cnt >= end) exhausted = true;
            idle = __ballot_sync(0xffffffffu, !have);
        }
        if (idle == 0xffffffffu) {
            if (exhausted) break;
            continue;
        }
        if (!have) continue;
        if (DEPTH && (L.step % kSeg) == 0) {
            const int64_t m = L.step / kSeg;
            if (m < buf.max_ckpt) {
                T* q = ck + (size_t)m * kDepthState * n + i;
                q[0] = L.E;
                q[n] = L.z;
                q[2 * n] = L.dx;
                q[3 * n] = L.dy;
                q[4 * n] = L.dz;
                q[5 * n] = L.yx;
                q[6 * n] = L.yy;
                q[7 * n] = L.yz;
            }
        }
        EventOut<T> ev;   // (exit energy) the event's E and step; the rest is not stored
        cont_event<T, !DEPTH>(L, c, rng, &ev);
        if (DEPTH && L.max_z > zbest) {
            zbest = L.max_z;
            mstar = (int)L.step;
        }
        if (L.outcome == MCD_OUT_NONE) {
            if constexpr (!DEPTH) tan = tangent(c, ev.E, ev.pathl, ev.W, tan, ij);
            continue;
        }
        // the electron is done; a 'bks' one left in its last event
        const bool bks = L.outcome == MCD_OUT_BKS;
        const int key = DEPTH ? mstar : (int)(L.step - 1);
        if (bks && key > 0 && (key - 1) / kSeg >= buf.max_ckpt) st |= MCD_FLAG_CKPT;
        buf.kstar[i] = bks ? key : -1;
        static_cast<T*>(buf.E_exit)[i] = DEPTH ? L.max_z : L.E_row;
        if (!DEPTH) ck[i] = tan;
        if (tally) {
            atomicAdd(&s_cnt[L.outcome & 7], 1ull);
            atomicAdd(&s_cnt[8], (unsigned long long)L.step);
        }
        if (L.flags & F_CLAMPED) st |= MCD_FLAG_CLAMPED;
        if (L.flags & F_LONG_PATH) st |= MCD_FLAG_LONG_PATH;
        if (L.outcome == MCD_OUT_LONG) st |= MCD_FLAG_LONG;
        have = false;
    }
    const uint32_t w = __reduce_or_sync(0xffffffffu, st);
    if (lane == 0 && w) atomicOr(status, w);
    if (!tally) return;
    __syncthreads();
    if (threadIdx.x < 9 && s_cnt[threadIdx.x]) {
        if (threadIdx.x < 8) atomicAdd(&tally->outcome[threadIdx.x], s_cnt[threadIdx.x]);
        else atomicAdd(&tally->events, s_cnt[8]);
    }
}

// A positive normal weight as a double (the build flushes subnormals, also in
// the comparison with zero before the sum).  In FP32 by its bits, as the
// conversion would hold the FP64 pipe, which bounds the pass, for as long as
// the addition does: the pass over 1M Cu electrons and 100 bins 80 us with the
// conversion, 45 us without.
__device__ __forceinline__ double widen(double x) { return x; }
__device__ __forceinline__ double widen(float x) {
    const uint32_t b = __float_as_uint(x);
    return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

// The soft bins, the sum and the number of the backscattered electrons of a
// forward pass.  A warp reads 32 electrons at a time and takes the
// backscattered ones in turn, lane l evaluating bins l, l + 32, .. in T and
// summing them in FP64 registers; NB = ceil(nbins / 32).  It reads 8 or 12
// bytes per electron; what it issues is one exponential per lane and bin group
// in reach.
template <class T, int NB>
__global__ void __launch_bounds__(256) k_adj_bins(const SoftHist sh, const AdjBuf buf, int64_t n, double* hout) {
    __shared__ double s_h[MCD_HIST_E_MAX + 2];
    for (int b = threadIdx.x; b < sh.nbins + 2; b += blockDim.x) s_h[b] = 0.0;
    __syncthreads();
    T lo, w, iw, i2, reach;
    soft_consts<T>(sh, lo, w, iw, i2, reach);
    const int lane = threadIdx.x & 31;
    double acc[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) acc[j] = 0.0;
    double sum = 0.0;
    unsigned count = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t i = first; i - lane < n; i += stride) {   // whole warps
        const bool bks = i < n && buf.kstar[i] >= 0;
        T q = (T)0;
        if (bks) {
            q = static_cast<const T*>(buf.E_exit)[i];
            sum += (double)q;
            ++count;
        }
        for (unsigned m = __ballot_sync(0xffffffffu, bks); m; m &= m - 1u) {
            const T v = __shfl_sync(0xffffffffu, q, __ffs(m) - 1);
            int b0, b1;
            soft_range(sh, v, lo, iw, reach, b0, b1);
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                const int b = lane + 32 * j;
                if (b >= b0 && b <= b1) {
                    const T d = v - (lo + ((T)b + (T)0.5) * w);
                    const T x = exp(-d * d * i2);
                    if (x > (T)0) acc[j] += widen(x);
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < NB; ++j)
        if (acc[j] != 0.0) atomicAdd(&s_h[lane + 32 * j], acc[j]);
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    count = __reduce_add_sync(0xffffffffu, count);
    if (lane == 0 && count) {
        atomicAdd(&s_h[sh.nbins], sum);
        atomicAdd(&s_h[sh.nbins + 1], (double)count);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < sh.nbins + 2; b += blockDim.x)
        if (s_h[b] != 0.0) atomicAdd(&hout[b], s_h[b]);
}

template <class T>
static void launch_bins(const SoftHist& sh, const AdjBuf& ab, int64_t n, int sms, double* hout, cudaStream_t st) {
    const int64_t blocks = (n + 255) / 256, cap = 4ll * sms;
    const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
    if (sh.nbins <= 32) k_adj_bins<T, 1><<<grid, 256, 0, st>>>(sh, ab, n, hout);
    else if (sh.nbins <= 64) k_adj_bins<T, 2><<<grid, 256, 0, st>>>(sh, ab, n, hout);
    else k_adj_bins<T, MCD_HIST_E_MAX / 32><<<grid, 256, 0, st>>>(sh, ab, n, hout);
}

// Reverse sweep of the deepest depth Z = z_{m*} = sum_{k < m*} s_k d_z,k
// along the frozen sequence.  Per event k, with the step s(E), the energy
// update E' = E - s S(E), the Rutherford sin^2(theta/2) = s2(E) and the
// rotation of the frame (d, y, x = y cross d)
//     d' = d cos(theta) + x sin(theta) cos(phi) + y sin(theta) sin(phi)
//     y' = y cos(phi) - x sin(phi)
// the adjoints of (E, d, y) run backwards from zero at m* (Z does not
// depend on the state after m*), g = dL/dZ feeds the z term of every event:
//     lE  = lE' (1 + s dlnsig S - s dS/dE) - g d_z s dlnsig
//           + lD' . (-2 ds2/dE d + dsin(theta)/dE (x cos(phi) + y sin(phi)))
//     lD  = cos(theta) lD' + w cross y + g s e_z
//     lY  = sin(theta) sin(phi) lD' + cos(phi) lY' + d cross w,
//           w = sin(theta) cos(phi) lD' - sin(phi) lY'
//     dL/dJ += lE' (-s dS/dJ);  dL/dn += g d_z (-s / n)  (E' does not depend on n)
// (the renormalisation of d and y after each rotation is left out: it moves
// a unit vector by rounding only).  Each segment is recomputed from its
// checkpoint with the forward's own event code.
// The adjoints a depth sweep carries from one segment to the one before it,
// and the electron's parameter sums.
template <class T>
struct DepthAdj {
    T lE, ldx, ldy, ldz, lyx, lyy, lyz, sj, sn;
};

// Segment m of electron i's depth sweep (the segments run last to first).
template <class T, class C>
__device__ __forceinline__ void depth_segment(const C& c, const AdjBuf& buf, uint64_t i, const ElecRng& rng, int mstar,
                                              int m, T g, T ij, T ins, DepthAdj<T>& A) {
    const T* ck = static_cast<const T*>(buf.ckpt);
    const size_t n = (size_t)c.num_el;
    T lE = A.lE, ldx = A.ldx, ldy = A.ldy, ldz = A.ldz, lyx = A.lyx, lyy = A.lyy, lyz = A.lyz;
    T sj = A.sj, sn = A.sn;
    // the segment's recorded states (E, d and y before each event); the
    // event's step, polar angle and uniforms are recomputed from its Philox
    // block in the sweep (the recorded arrays pass through local memory,
    // and four more of them cost more traffic than the recomputation)
    T aE[kSeg], aD[3][kSeg], aY[3][kSeg];
    {
        const int k0 = m * kSeg;
        const int len = min(kSeg, mstar - k0);
        const T* q = ck + (size_t)m * kDepthState * n + i;
        Lane<T> L;
        lane_init(L, c);
        L.E = q[0];
        L.z = q[n];
        L.dx = q[2 * n];
        L.dy = q[3 * n];
        L.dz = q[4 * n];
        L.yx = q[5 * n];
        L.yy = q[6 * n];
        L.yz = q[7 * n];
        L.step = k0;
        for (int j = 0; j < len; ++j) {   // the forward's events, recorded
            aE[j] = L.E;
            aD[0][j] = L.dx;
            aD[1][j] = L.dy;
            aD[2][j] = L.dz;
            aY[0][j] = L.yx;
            aY[1][j] = L.yy;
            aY[2][j] = L.yz;
            EventOut<T> ev;
            cont_event<T, false>(L, c, rng, &ev);
        }
        for (int j = len - 1; j >= 0; --j) {   // reverse sweep
            const T E = aE[j];
            // the event's step and angles as cont_event_r computed them
            const uint4 r = philox_event(rng, (uint32_t)(k0 + j), event_words(c));
            const T s = -Ops<T>::ln_step_word(r.y) * Ops<T>::div((T)1, sig_ruth<T>(c, E));
            const T a_r = Ops<T>::div(c.a0, E);
            const T s2 = Ops<T>::div(a_r * Ops<T>::unit(r.z), a_r + Ops<T>::unit_c(r.z));
            const T dx = aD[0][j], dy = aD[1][j], dz = aD[2][j];
            const T yx = aY[0][j], yy = aY[1][j], yz = aY[2][j];
            T S, SE, Sj;
            stopping_derivs<T>(c, E, &S, &SE, &Sj);
            const T dl = dlnsig<T>(c, E);
            // angles of the event
            T sp, cp;
            Ops<T>::sincos_pi(Ops<T>::unit(r.w), &sp, &cp);
            if (c.quirks & MCD_Q_HALF_PHI_FOLD) cp = fabs(cp);
            const T cph = (T)1 - (T)2 * sp * sp, sph = (T)2 * sp * cp;
            const T cth = (T)1 - (T)2 * s2;
            const T sth = (T)2 * Ops<T>::sqrt_(s2) * Ops<T>::sqrt_((T)1 - s2);
            // d s2 / dE with s2 = a U / (a + 1 - U), a = a0 / E
            const T a = a_r, U = Ops<T>::unit(r.z), Uc = (T)1 - U;
            const T den = a + Uc;
            const T ds2 = -Ops<T>::div(a, E) * Ops<T>::div(U * Uc, den * den);
            const T dsth = sth > (T)0 ? Ops<T>::div((T)2 * cth * ds2, sth) : (T)0;
            const T xx = yy * dz - yz * dy, xy = yz * dx - yx * dz, xz = yx * dy - yy * dx;
            const T sa = sth * cph, sb = sth * sph;
            // parameter gradients use the adjoint of the event's outputs
            sj += lE * (-s * Sj * ij);
            sn += g * dz * (-s * ins);
            const T rot = ldx * (-(T)2 * ds2 * dx + dsth * (cph * xx + sph * yx)) +
                          ldy * (-(T)2 * ds2 * dy + dsth * (cph * xy + sph * yy)) +
                          ldz * (-(T)2 * ds2 * dz + dsth * (cph * xz + sph * yz));
            const T nE = lE * ((T)1 + s * dl * S - s * SE) - g * dz * s * dl + rot;
            const T wx = sa * ldx - sph * lyx, wy = sa * ldy - sph * lyy, wz = sa * ldz - sph * lyz;
            const T ndx = cth * ldx + (wy * yz - wz * yy);
            const T ndy = cth * ldy + (wz * yx - wx * yz);
            const T ndz = cth * ldz + (wx * yy - wy * yx) + g * s;
            const T nyx = sb * ldx + cph * lyx + (dy * wz - dz * wy);
            const T nyy = sb * ldy + cph * lyy + (dz * wx - dx * wz);
            const T nyz = sb * ldz + cph * lyz + (dx * wy - dy * wx);
            lE = nE;
            ldx = ndx;
            ldy = ndy;
            ldz = ndz;
            lyx = nyx;
            lyy = nyy;
            lyz = nyz;
        }
    }
    A = DepthAdj<T>{lE, ldx, ldy, ldz, lyx, lyy, lyz, sj, sn};
}

// d(loss)/d(exit quantity) of electron i: the soft-bin weights' derivative
// plus the sum term, in T, with gh[b] = dL/dh_b / N and gh[nbins] = dL/dsum
template <class T>
__device__ __forceinline__ T exit_adjoint(const SoftHist& sh, const AdjBuf& buf, const T* gh, uint64_t i) {
    const T q = static_cast<const T*>(buf.E_exit)[i];
    const T is2 = sizeof(T) == 8 ? (T)sh.inv_s2 : (T)sh.f_inv_s2;
    T g = gh[sh.nbins];
    soft_bins<T>(sh, q, [&](int b, T w, T d) { g += gh[b] * (-d * is2) * w; });
    return g;
}

// Adds the threads' sums to grad; called by the whole block, red[2] zeroed
__device__ __forceinline__ void add_grad(double* red, double dj, double dn, double* grad) {
    for (int o = 16; o > 0; o >>= 1) {
        dj += __shfl_down_sync(0xffffffffu, dj, o);
        dn += __shfl_down_sync(0xffffffffu, dn, o);
    }
    if ((threadIdx.x & 31u) == 0) {
        atomicAdd(&red[0], dj);
        atomicAdd(&red[1], dn);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(&grad[0], red[0]);
        atomicAdd(&grad[1], red[1]);
    }
}

// The depth's backward pass runs only for backscattered electrons, a fraction
// of the launch, and a warp's lanes run as long as the longest of their
// sequences: a block sorts the backscattered electrons of its range by the
// length of their sequences (into bins, the longest first) and its warps take
// them 32 at a time.  Handing electrons in index order to lanes that had become
// idle, a segment per trip, kept 12 of 32 lanes busy: the backward of Al 15 keV
// 300000 electrons 0.48 ms, sorted 0.26; Au 25 keV 1.07 and 0.70; 30000 Al
// electrons 0.41 and 0.24.
// The range is the shortest of 1024, 2048 and 4096 electrons that leaves at most
// one block per SM: up to there a block lasts as long as its longest sequences
// and its other warps' work hides behind them, beyond it a longer range sorts
// better.  Ranges of 1024 / 2048 / 4096, ms: 150000 Al 0.23 / 0.26 / 0.33, Au
// 0.62 / 0.69 / 0.86; 300000 Al 0.29 / 0.26 / 0.34, Au 0.77 / 0.71 / 0.88;
// 500000 Al 0.41 / 0.33 / 0.35, Au 1.03 / 0.92 / 0.90; 1500000 Al 0.81 / 0.70 /
// 0.63, Au 2.28 / 1.91 / 1.73.
constexpr int kBwdThreads = 256, kBwdRange = 4096;
constexpr int kBwdBins = 64;
__device__ __forceinline__ int length_bin(int k) {   // of k > 0 events; 0 is the longest
    const int b = k <= 128 ? (k - 1) / 4 : 32 + min((k - 129) / 32, 31);
    return kBwdBins - 1 - b;
}

template <class T>
__global__ void __launch_bounds__(kBwdThreads, 4) k_adj_depth(const SimConst<T> cp, const SoftHist sh, const AdjBuf buf, int range,
                                                      const double* grad_h, double inv_n, double inv_j,
                                                      double inv_ns, double* grad) {
    __shared__ SimConst<T> c;
    __shared__ double red[2];
    __shared__ T gh[MCD_HIST_E_MAX + 1];
    __shared__ unsigned s_bin[kBwdBins], s_next;
    __shared__ uint16_t s_el[kBwdRange];
    if (threadIdx.x == 0) {
        c = cp;
        red[0] = red[1] = 0.0;
        s_next = 0u;
    }
    if (threadIdx.x < kBwdBins) s_bin[threadIdx.x] = 0u;
    for (int b = threadIdx.x; b <= sh.nbins; b += blockDim.x) gh[b] = (T)(b < sh.nbins ? grad_h[b] * inv_n : grad_h[b]);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t lo = (uint64_t)blockIdx.x * range, left = (uint64_t)c.num_el - lo;
    const int len = left < (uint64_t)range ? (int)left : range;
    auto events = [&](int j) {   // of a backscattered electron with a checkpointed sweep, else 0
        const int k = buf.kstar[lo + j];
        return k > 0 && (k - 1) / kSeg < buf.max_ckpt ? k : 0;
    };
    for (int j = threadIdx.x; j < len; j += blockDim.x) {
        const int k = events(j);
        if (k) atomicAdd(&s_bin[length_bin(k)], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 32) {   // bins to their first places
        const unsigned a = s_bin[2 * lane], b = s_bin[2 * lane + 1];
        unsigned incl = a + b;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        s_bin[2 * lane] = incl - a - b;
        s_bin[2 * lane + 1] = incl - b;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < len; j += blockDim.x) {
        const int k = events(j);
        if (k) s_el[atomicAdd(&s_bin[length_bin(k)], 1u)] = (uint16_t)j;
    }
    __syncthreads();
    const unsigned count = s_bin[kBwdBins - 1];   // (now the bins' ends)
    double gj = 0.0, gn = 0.0;
    const T ij = (T)inv_j, ins = (T)inv_ns;
    while (true) {
        unsigned first = 0;
        if (lane == 0) first = atomicAdd(&s_next, 32u);
        first = __shfl_sync(0xffffffffu, first, 0);
        if (first >= count) break;
        const bool have = first + lane < count;
        const uint64_t i = lo + (have ? s_el[first + lane] : 0);
        const int ks = have ? events((int)(i - lo)) : 0;
        int m = have ? (ks - 1) / kSeg : -1;
        const ElecRng rng = elec_rng(c, c.first + i);
        const T g = have ? exit_adjoint<T>(sh, buf, gh, i) : (T)0;
        DepthAdj<T> dA{};
        while (__any_sync(0xffffffffu, m >= 0)) {   // the segments, last to first
            if (m >= 0) depth_segment<T>(c, buf, i, rng, ks, m, g, ij, ins, dA);
            --m;
        }
        gj += (double)dA.sj;
        gn += (double)dA.sn;
    }
    add_grad(red, gj, gn, grad);
}

// The exit energy's gradient: every backscattered electron's dL/dE_exit times
// the derivative that the forward pass left.  It reads 8 to 12 bytes per
// electron and evaluates the few bins in reach.  Sums in FP64; the density does
// not enter the exit energy (s ~ 1/n, S ~ n), and its sum shows only a gradient
// that is not finite.
template <class T>
__global__ void __launch_bounds__(256) k_adj_exit(const SoftHist sh, const AdjBuf buf, int64_t n, const double* grad_h,
                                                  double inv_n, double* grad) {
    __shared__ double red[2];
    __shared__ T gh[MCD_HIST_E_MAX + 1];
    if (threadIdx.x < 2) red[threadIdx.x] = 0.0;
    for (int b = threadIdx.x; b <= sh.nbins; b += blockDim.x) gh[b] = (T)(b < sh.nbins ? grad_h[b] * inv_n : grad_h[b]);
    __syncthreads();
    const T* ck = static_cast<const T*>(buf.ckpt);
    double gj = 0.0, gn = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int k = buf.kstar[i];
        if (k <= 0 || (k - 1) / kSeg >= buf.max_ckpt) continue;
        const T g = exit_adjoint<T>(sh, buf, gh, (uint64_t)i);
        gj += (double)(g * ck[i]);
        gn += (double)(g * (T)0);
    }
    __syncwarp();
    add_grad(red, gj, gn, grad);
}

template <class T>
static void launch_exit(const SoftHist& sh, const AdjBuf& ab, int64_t n, int sms, const double* grad_h, double inv_n,
                        double* grad, cudaStream_t st) {
    const int64_t blocks = (n + 255) / 256, cap = 8ll * sms;
    k_adj_exit<T><<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, st>>>(sh, ab, n, grad_h, inv_n, grad);
}

// E_{k*}(J, n) along the frozen event sequence only (no geometry): the
// function the adjoint differentiates, for finite-difference checks.
template <class T>
__global__ void __launch_bounds__(256) k_adj_chain(const SimConst<T> cp, const SoftHist sh, const AdjBuf buf,
                                                   double* hout) {
    __shared__ SimConst<T> c;
    __shared__ double sh_h[MCD_HIST_E_MAX + 2];
    if (threadIdx.x == 0) c = cp;
    for (int b = threadIdx.x; b < sh.nbins + 2; b += blockDim.x) sh_h[b] = 0.0;
    __syncthreads();
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (uint64_t)c.num_el) {
        const int kstar = buf.kstar[i];
        if (kstar >= 0) {
            const ElecRng rng = elec_rng(c, c.first + i);
            T Ed;
            if (sh.quantity == MCD_ADJ_MAX_DEPTH) {
                // the forward's own events up to the deepest point
                Lane<T> L;
                lane_init(L, c);
                for (int k = 0; k < kstar; ++k) {
                    EventOut<T> ev;
                    cont_event<T, false>(L, c, rng, &ev);
                }
                Ed = L.z;
            } else {
                T E = c.E0;
                for (int k = 0; k < kstar; ++k) {
                    const T s = step_len<T>(c, E, rng, k);
                    E = E - Ops<T>::mul_rn(s, stopping<T>(c, E));
                }
                Ed = E;
            }
            soft_bins<T>(sh, Ed, [&](int b, T w, T) { if (w > (T)0) atomicAdd(&sh_h[b], (double)w); });
            atomicAdd(&sh_h[sh.nbins], (double)Ed);
            atomicAdd(&sh_h[sh.nbins + 1], 1.0);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < sh.nbins + 2; b += blockDim.x)
        if (sh_h[b] != 0.0) atomicAdd(&hout[b], sh_h[b]);
}

// multiprocessors of the current device, 0 on an error
static int sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return sms;
}

static int adj_args(const mcd_sim* sim, const mcd_material* mat, const mcd_softhist* hist,
                    const mcd_adjoint_buf* buf, SoftHist* sh, AdjBuf* ab) {
    if (!sim || !mat || !hist || !buf) return MCD_EINVAL;
    const int rc = check_sim(*sim, *mat, nullptr, nullptr);
    if (rc != MCD_OK) return rc;
    if (sim->mode != MCD_MODE_CONT) return MCD_EINVAL;
    if (hist->nbins < 1 || hist->nbins > MCD_HIST_E_MAX) return MCD_ETOOBIG;
    if (!(hist->sigma > 0) || !(hist->hi > hist->lo)) return MCD_EINVAL;
    if (!buf->ckpt || !buf->kstar || !buf->E_exit || buf->max_ckpt < 1) return MCD_EINVAL;
    if (hist->quantity != MCD_ADJ_EXIT_E && hist->quantity != MCD_ADJ_MAX_DEPTH) return MCD_EINVAL;
    if (!(sim->J_scale >= 0) || !(sim->n_scale >= 0)) return MCD_EINVAL;
    sh->nbins = hist->nbins;
    sh->quantity = hist->quantity;
    sh->lo = hist->lo;
    sh->width = (hist->hi - hist->lo) / hist->nbins;
    sh->inv2s2 = 1.0 / (2.0 * hist->sigma * hist->sigma);
    sh->inv_s2 = 1.0 / (hist->sigma * hist->sigma);
    sh->inv_width = 1.0 / sh->width;
    sh->reach = 8.0 * hist->sigma;
    sh->f_lo = (float)sh->lo;
    sh->f_width = (float)sh->width;
    sh->f_inv_width = (float)sh->inv_width;
    sh->f_inv2s2 = (float)sh->inv2s2;
    sh->f_inv_s2 = (float)sh->inv_s2;
    sh->f_reach = (float)sh->reach;
    ab->ckpt = buf->ckpt;
    ab->kstar = buf->kstar;
    ab->E_exit = buf->E_exit;
    ab->max_ckpt = buf->max_ckpt;
    ab->queue = buf->queue;
    return MCD_OK;
}

}  // namespace mcd

using namespace mcd;

extern "C" int mcd_adjoint_forward(const mcd_sim* sim, const mcd_material* mat, const mcd_softhist* hist,
                                   const mcd_adjoint_buf* buf, double* hist_out, mcd_tally* tally,
                                   uint32_t* status, void* stream) {
    SoftHist sh;
    AdjBuf ab;
    int rc = adj_args(sim, mat, hist, buf, &sh, &ab);
    if (rc != MCD_OK) return rc;
    if (!hist_out || !status) return MCD_EINVAL;
    if (sim->num_el == 0) return MCD_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t range = 32;
    unsigned long long grid = ((unsigned long long)sim->num_el + 255) / 256;   // one thread per electron
    const int sms = sm_count();
    if (sms <= 0) return MCD_ECUDA;
    const double inv_j = 1.0 / (sim->J_scale > 0 ? sim->J_scale : 1.0);
    const bool depth = sh.quantity == MCD_ADJ_MAX_DEPTH, fp64 = sim->precision == MCD_FP64;
    const void* kern = fp64 ? (depth ? (const void*)k_adj_fwd<double, true> : (const void*)k_adj_fwd<double, false>)
                            : (depth ? (const void*)k_adj_fwd<float, true> : (const void*)k_adj_fwd<float, false>);
    if (ab.queue) {
        // a resident grid: as many blocks as fit on the GPU at once, and no
        // more than there are electrons for
        int blocks = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, 256, 0) != cudaSuccess) return MCD_ECUDA;
        const unsigned long long resident = (unsigned long long)sms * (blocks > 0 ? blocks : 1);
        grid = grid < resident ? grid : resident;
        if (cudaMemsetAsync(ab.queue, 0, sizeof(unsigned long long), st) != cudaSuccess) return MCD_ECUDA;
    }
    if (grid > 0x7fffffffull) return MCD_ETOOBIG;
    const unsigned g = (unsigned)grid;
    if (fp64) {
        const SimConst<double> c = make_consts<double>(*sim, *mat, nullptr, nullptr);
        if (depth) k_adj_fwd<double, true><<<g, 256, 0, st>>>(c, ab, range, inv_j, tally, status);
        else k_adj_fwd<double, false><<<g, 256, 0, st>>>(c, ab, range, inv_j, tally, status);
        if (cudaGetLastError() != cudaSuccess) return MCD_ECUDA;
        launch_bins<double>(sh, ab, sim->num_el, sms, hist_out, st);
    } else {
        const SimConst<float> c = make_consts<float>(*sim, *mat, nullptr, nullptr);
        if (depth) k_adj_fwd<float, true><<<g, 256, 0, st>>>(c, ab, range, inv_j, tally, status);
        else k_adj_fwd<float, false><<<g, 256, 0, st>>>(c, ab, range, inv_j, tally, status);
        if (cudaGetLastError() != cudaSuccess) return MCD_ECUDA;
        launch_bins<float>(sh, ab, sim->num_el, sms, hist_out, st);
    }
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}

extern "C" int mcd_adjoint(const mcd_sim* sim, const mcd_material* mat, const mcd_softhist* hist,
                           const mcd_adjoint_buf* buf, const double* grad_hist, double* grad, void* stream) {
    SoftHist sh;
    AdjBuf ab;
    int rc = adj_args(sim, mat, hist, buf, &sh, &ab);
    if (rc != MCD_OK) return rc;
    if (!grad_hist || !grad) return MCD_EINVAL;
    if (sim->num_el == 0) return MCD_OK;
    const double inv_n = 1.0 / (double)sim->num_el;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int sms = sm_count();
    if (sms <= 0) return MCD_ECUDA;
    if (sh.quantity != MCD_ADJ_MAX_DEPTH) {
        if (sim->precision == MCD_FP64) launch_exit<double>(sh, ab, sim->num_el, sms, grad_hist, inv_n, grad, st);
        else launch_exit<float>(sh, ab, sim->num_el, sms, grad_hist, inv_n, grad, st);
        return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
    }
    int range = kBwdRange / 4;
    while (range < kBwdRange && sim->num_el > (int64_t)range * sms) range *= 2;
    const unsigned long long grid = ((unsigned long long)sim->num_el + range - 1) / range;
    if (grid > 0x7fffffffull) return MCD_ETOOBIG;
    const double js = 1.0 / (sim->J_scale > 0 ? sim->J_scale : 1.0);
    const double ns = 1.0 / (sim->n_scale > 0 ? sim->n_scale : 1.0);
    const unsigned g = (unsigned)grid;
    if (sim->precision == MCD_FP64)
        k_adj_depth<double><<<g, kBwdThreads, 0, st>>>(make_consts<double>(*sim, *mat, nullptr, nullptr), sh, ab,
                                                       range, grad_hist, inv_n, js, ns, grad);
    else
        k_adj_depth<float><<<g, kBwdThreads, 0, st>>>(make_consts<float>(*sim, *mat, nullptr, nullptr), sh, ab,
                                                      range, grad_hist, inv_n, js, ns, grad);
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}

extern "C" int mcd_adjoint_chain(const mcd_sim* sim, const mcd_material* mat, const mcd_softhist* hist,
                                 const mcd_adjoint_buf* buf, double* hist_out, void* stream) {
    SoftHist sh;
    AdjBuf ab;
    int rc = adj_args(sim, mat, hist, buf, &sh, &ab);
    if (rc != MCD_OK) return rc;
    if (!hist_out) return MCD_EINVAL;
    const unsigned long long grid = ((unsigned long long)sim->num_el + 255) / 256;
    if (grid == 0) return MCD_OK;
    if (grid > 0x7fffffffull) return MCD_ETOOBIG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (sim->precision == MCD_FP64)
        k_adj_chain<double><<<(unsigned)grid, 256, 0, st>>>(make_consts<double>(*sim, *mat, nullptr, nullptr), sh, ab,
                                                             hist_out);
    else
        k_adj_chain<float><<<(unsigned)grid, 256, 0, st>>>(make_consts<float>(*sim, *mat, nullptr, nullptr), sh, ab,
                                                            hist_out);
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}
