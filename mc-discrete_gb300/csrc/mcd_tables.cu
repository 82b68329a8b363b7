// mcd_tables.cu - FP64 fill of the sampled energy-loss CDF tables.
//
// Restates probTable.computeBlock (MC/tools/probTables.py:415-462): for each
// E row, the trapezoid of dsigma/dW between consecutive float32 grid points
// W_k, W_k+1 (their float32 difference times the mean of the two values),
// a cumulative sum along W and a division by the row total.  An interval
// whose upper edge exceeds Wmax(E) = (E - Ef)/2, evaluated in float32 as the
// reference's float32 meshes are, is masked and stored as 0
// (MC/tools/probTables.py:428-439, 507).
//
// One warp per E row: the unmasked intervals are a prefix of the row, whose
// values are dealt out to the lanes in contiguous runs of equal length; a lane
// leaves its running sums in shared memory, the warp scans the 32 partial sums,
// and a coalesced pass writes the sums divided by the row total.  dsigma/dW
// (MC/tools/extFunctions.py:159-219) is evaluated in FP64, once per grid
// point, up to a factor that is constant along the row: it divides out.
//
// What bounds it: the FP64 pipe, two lanes per SM on this part (a warp
// instruction occupies it for 16 cycles, whatever its active lanes), at 86%
// of its peak in the first version, which evaluated every dsigma/dW twice
// with pow, log, sqrt and five divisions: about 280 FP64 instructions per
// Gryzinski value.  With eps = W/E and epsB = Eb/E,
//   eps (1 - eps)^(epsB/(epsB+eps)) ((1-epsB) + 4 epsB L / (3 eps)) / W^3
//     = (1/E) (1 - eps)^(Eb/(Eb+W)) ((1-epsB) W^-2 + (4/3) Eb W^-3 L),
//   L = ln(2.7 + sqrt((1 - eps)/epsB)),
// so the exponent and the powers of W belong to the column: a block computes
// them once into shared memory and its warps run many rows.  A value is then
// two table-driven logarithms, one table-driven exponential and one square root
// from the hardware's approximation, 34 FP64 instructions with the trapezoid;
// exponents, table indices, halvings and the rounding to float32 are integer
// operations.  The Moller value is a^2 + b^2 - a b with a = 1/W (column) and
// b = 1/(E - W), over E.
// Measured: the Au 30 keV tol 1e-4 pair (20000 x 499 and 100000 x 599 values)
// 67.7 ms in the first version; 7.24 ms with tables of 256 and 64 breakpoints
// and their longer series, conversions on the FP64 pipe and the masked
// intervals' lanes idle (58 instructions per value); 4.95 ms without the
// former, 4.19 ms with the lanes sharing the unmasked prefix (FP64 pipe 85%
// busy).  The float32 tables are bit for bit the same in all of them.
#include <cuda_runtime.h>
#include <stdint.h>

#include "mcd_device.cuh"

namespace mcd {

struct FillParams {
    const float* Es;
    const float* Ws;
    float* cdf32;
    double* cdf64;
    int32_t* nvalid;
    uint16_t* guide;
    int32_t nE, nW;
    int32_t kind;
    double Eb;     // Gryzinski binding energy
    float Ef32;
};

// The tables of the fill's logarithms and exponential: 1024 breakpoints, so
// that the remainder's series is one FP64 instruction per term shorter per
// factor of four (256 or 64 breakpoints took 20 FP64 instructions more per
// value).  r_j is 1/(1 + (j + 1/2)/1024) rounded to 24 bits, so that
// t = m r_j - 1 is one fused operation, |t| < 2^-10.99; the entries are
// evaluated at compile time in double-double arithmetic and are the doubles
// nearest to their values.
constexpr int kFillSteps = 1024;
struct FillTabs {
    double r[kFillSteps];
    double ln1[kFillSteps];       // -ln r_j
    double ln0[kFillSteps];       // -ln r_j - ln 2
    double e[kFillSteps + 1];     // exp(-j/1024)
    double eln2[64];              // j ln 2
};
constexpr CxDD cx_exp_neg(double num, double den) {   // exp(-num/den), num/den <= 1
    const CxDD x = cx_div(CxDD{-num, 0.0}, den);
    CxDD term{1.0, 0.0}, sum{0.0, 0.0};
    for (int k = 0; k < 24; ++k) {
        sum = cx_add(sum, term);
        term = cx_div(cx_mul(term, x), k + 1.0);
    }
    return sum;
}
constexpr FillTabs cx_fill_tabs() {
    FillTabs t{};
    CxDD coarse[257] = {}, fine[33] = {}, block[33] = {};
    for (int j = 0; j <= 256; ++j) coarse[j] = cx_ln_ratio(j);   // ln(1 + j/256)
    const CxDD ln2 = coarse[256];
    for (int j = 0; j <= 32; ++j) {
        fine[j] = cx_exp_neg(j, 1024.0);
        block[j] = cx_exp_neg(j, 32.0);
    }
    for (int j = 0; j < kFillSteps; ++j) {
        const double r = (double)(float)(1.0 / (1.0 + (j + 0.5) / kFillSteps));
        // r (1 + i/256) = 1 - d, exact, |d| <= 1/256:
        // -ln r = ln(1 + i/256) - ln(1 - d), -ln(1 - d) = 2 atanh(d / (2 - d))
        const int i = (j + 2) / 4;
        const double d = 1.0 - r * (1.0 + i / 256.0);
        const CxDD l = cx_add(coarse[i], cx_atanh2(d, 2.0 - d, 8));
        const CxDD l0 = cx_add(l, CxDD{-ln2.hi, -ln2.lo});
        t.r[j] = r;
        t.ln1[j] = l.hi + l.lo;
        t.ln0[j] = l0.hi + l0.lo;
    }
    for (int j = 0; j <= kFillSteps; ++j) {
        const CxDD e = cx_mul(block[j / 32], fine[j % 32]);
        t.e[j] = e.hi + e.lo;
    }
    for (int j = 0; j < 64; ++j) {
        const CxDD l = cx_mul(ln2, CxDD{(double)j, 0.0});
        t.eln2[j] = l.hi + l.lo;
    }
    return t;
}
static __device__ const FillTabs kFillTabs = cx_fill_tabs();

// ln of a double's mantissa m in [1, 2) from its high word's breakpoint, onto
// the entry `base` of the breakpoint: base + ln(m r_j), to t^4 (the next term is
// below 6e-18)
__device__ __forceinline__ double ln_mantissa(double x, const double* base) {
    const int hi = __double2hiint(x), j = (hi >> 10) & (kFillSteps - 1);
    const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(x));
    const double t = fma(m, __ldg(&kFillTabs.r[j]), -1.0);
    return fma(t, fma(t, fma(t, fma(t, -0.25, 1.0 / 3.0), -0.5), 1.0), __ldg(&base[j]));
}

// ln x of a positive normal x, absolute error about 2e-16 max(1, |ln x|): the
// scheme of ln_word (256 breakpoints, series of the remainder) on a double
__device__ __forceinline__ double ln_pos(double x) {
    const long long b = __double_as_longlong(x);
    const int j = (int)(b >> 44) & 255;
    const double m = __longlong_as_double((b & 0x000fffffffffffffll) | 0x3ff0000000000000ll);
    const double mj = __longlong_as_double((b & 0x000ff00000000000ll) | 0x3ff0000000000000ll);
    const double t = (m - mj) * __ldg(&kF64Tabs.invm[j]);
    const double q = t * fma(t, fma(t, fma(t, fma(t, fma(t, -1.0 / 6.0, 0.2), -0.25), 1.0 / 3.0), -0.5), 1.0);
    return fma((double)((int)(b >> 52) - 1023), 0.6931471805599453, __ldg(&kF64Tabs.lnm[j]) + q);
}

// ln x for x in [1/2, 1), elsewhere ln_pos (not on the reference's grids:
// W <= (E - Ef)/2); absolute error about 2e-16
__device__ __forceinline__ double ln_half(double x) {
    if ((__double2hiint(x) >> 20) != 0x3fe) return ln_pos(x);
    return ln_mantissa(x, kFillTabs.ln0);
}
// ln x for x in [1, 2^64), elsewhere ln_pos
__device__ __forceinline__ double ln_above(double x) {
    const unsigned e = ((unsigned)__double2hiint(x) >> 20) - 1023u;
    if (e >= 64u) return ln_pos(x);
    return ln_mantissa(x, kFillTabs.ln1) + __ldg(&kFillTabs.eln2[e]);
}

// exp(y) for y in (-0.99, 0], elsewhere exp: exp(-j/1024) of the nearest j times
// the series of the remainder |r| <= 2^-11 to r^4 (the next term is below
// 3e-19); j is read from the low bits of 1.5 2^52 - 1024 y
__device__ __forceinline__ double exp_unit(double y) {
    const unsigned h = (unsigned)__double2hiint(y);
    if (!(h - 0x80000000u < 0x3fefae14u || h == 0u)) return exp(y);
    const double v = fma(y, -1024.0, 6755399441055744.0);
    const double e = __ldg(&kFillTabs.e[__double2loint(v)]);
    const double r = fma(v - 6755399441055744.0, 1.0 / 1024.0, y);
    const double p = fma(r, fma(r, fma(r, 1.0 / 24.0, 1.0 / 6.0), 0.5), 1.0);
    return fma(e * r, p, e);
}

// sqrt(x) of a positive normal x (within one ulp): the hardware reciprocal
// square root r (some 20 bits), whose error one Newton step on s = x r squares
// and one on the residual x - s^2 removes; r/2 by its exponent
__device__ __forceinline__ double sqrt_pos(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double h = __hiloint2double(__double2hiint(r) - 0x00100000, __double2loint(r));
    double s = x * r;
    s = fma(s, fma(-s, h, 0.5), s);
    return fma(fma(-s, s, x), h, s);
}

// A double in [0, 1] rounded to the nearest float (ties to even), by its bits:
// the conversion would hold the FP64 pipe.  Outside the normal floats of that
// range the conversion itself.
__device__ __forceinline__ float round_unit(double v) {
    if ((unsigned)__double2hiint(v) - 0x38100000u > 0x3ff00000u - 0x38100000u) return __double2float_rn(v);
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return __uint_as_float((uint32_t)((b + 0x0fffffffull + ((b >> 29) & 1ull)) >> 29) - 0xc0000000u);
}

// What a grid point W contributes to every row: W itself, Gryzinski the
// exponent Eb/(Eb + W), W^-2 and (4/3) Eb W^-3, Moller 1/W and W^-2; and half
// the interval up to it from the point before (in float32, as the reference's
// grids are).
struct FillCol {
    double W, a, b, c, half;
};
__device__ __forceinline__ FillCol fill_col(const FillParams& p, int k) {
    const float w = p.Ws[k];
    const double W = (double)w, w1 = 1.0 / W, w2 = w1 * w1;
    const double half = k ? (double)__fmul_rn(__fsub_rn(w, p.Ws[k - 1]), 0.5f) : 0.0;
    if (p.kind == MCD_TABLE_MOLLER) return FillCol{W, w1, w2, 0.0, half};
    return FillCol{W, p.Eb / (p.Eb + W), w2, (4.0 / 3.0) * p.Eb * w2 * w1, half};
}

// dsigma/dW at (E, W) up to a factor of the row
__device__ __forceinline__ double fill_value(const FillParams& p, double E, double invE, double c1, double invEb,
                                             const FillCol& q) {
    if (p.kind == MCD_TABLE_MOLLER) {
        const double b = rcp_pos(E - q.W);
        return fma(b, b - q.a, q.b);
    }
    const double x = fma(-q.W, invE, 1.0);
    const double pw = exp_unit(q.a * ln_half(x));
    const double L = ln_above(2.7 + sqrt_pos(x * invEb));
    return pw * fma(q.c, L, c1 * q.b);
}

constexpr int kFillCols = 1024;   // intervals a row may have to pass through shared memory

// Shared memory of a block of w warps: the columns of nW grid points, and per
// warp the row's running sums (then, each in its slot, the float values) and
// the lanes' offsets.
constexpr size_t fill_smem(int w, int nW) {
    return sizeof(FillCol) * nW + (size_t)w * sizeof(double) * (nW + 32);
}

// SMEM: the row's sums pass through shared memory; rows wider than kFillCols
// evaluate their values a second time instead.
template <bool SMEM>
__global__ void __launch_bounds__(256) k_fill(const FillParams p) {
    extern __shared__ __align__(16) uint8_t fill_sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int nint = p.nW - 1;
    FillCol* cols = reinterpret_cast<FillCol*>(fill_sm);
    double* sums = reinterpret_cast<double*>(cols + p.nW) + (size_t)warp * (p.nW + 32);
    double* offs = sums + p.nW;
    if (SMEM) {
        for (int k = threadIdx.x; k < p.nW; k += blockDim.x) cols[k] = fill_col(p, k);
        __syncthreads();
    }
    for (int row = blockIdx.x * nwarps + warp; row < p.nE; row += gridDim.x * nwarps) {
        const float e32 = p.Es[row];
        const double E = (double)e32;
        const float wmax = __fmul_rn(__fsub_rn(e32, p.Ef32), 0.5f);
        const double invE = 1.0 / E, epsB = p.Eb * invE, c1 = 1.0 - epsB, invEb = E / p.Eb;
        const bool open = p.kind == MCD_TABLE_MOLLER || epsB < 1.0;   // below the binding energy: 0
        // W ascends, so the unmasked intervals are a prefix; the values at
        // their ends are dealt out to the lanes in contiguous runs
        int nval = 0;
        for (int hi = nint; nval < hi;) {
            const int mid = (nval + hi) >> 1;
            if (p.Ws[mid + 1] <= wmax) nval = mid + 1;
            else hi = mid;
        }
        const int nvals = nval ? nval + 1 : 0;
        const int per = (nval + 32) / 32;   // of nval + 1
        const int v0 = min(lane * per, nvals), v1 = min(v0 + per, nvals);
        // the lane's running sums of its intervals k - 1 (those that end at its
        // values k), but for the part of its first value's predecessor;
        // f(interval, running sum) sees each.  `last` is the lane's last value.
        double last = 0.0;
        auto sweep = [&](double run, auto f) {
            last = 0.0;
            for (int k = v0; k < v1; ++k) {
                const FillCol q = SMEM ? cols[k] : fill_col(p, k);
                const double v = open && p.Ws[k] < e32 ? fill_value(p, E, invE, c1, invEb, q) : 0.0;
                run = fma(q.half, last + v, run);
                if (k) f(k - 1, run);
                last = v;
            }
            return run;
        };
        double part = sweep(0.0, [&](int k, double run) {
            if (SMEM) sums[k] = run;
        });
        double first = __shfl_up_sync(0xffffffffu, last, 1);   // the predecessor's part, in all of the lane's sums
        first = lane && v0 < v1 ? first * (SMEM ? cols[v0].half : fill_col(p, v0).half) : 0.0;
        part += first;
        // warp scan of the partial sums (exclusive)
        double incl = part;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const double total = __shfl_sync(0xffffffffu, incl, 31);
        const double before = (incl - part) + first;
        const size_t base = (size_t)row * nint;
        // the reference's last valid entry is cum/cum = 1 exactly
        auto store = [&](int k, double run) {
            const double v = (k == nval - 1) ? 1.0 : fmin(run / total, 1.0);
            const float v32 = __double2float_rn(v);
            p.cdf32[base + k] = v32;
            if (p.cdf64) p.cdf64[base + k] = v;
            return v32;
        };
        if (SMEM) {
            const double inv = 1.0 / total;
            offs[lane] = before * inv;
            __syncwarp();
            for (int k = lane; k < nint; k += 32) {
                double v = 0.0;
                if (k < nval - 1) {
                    v = fma(sums[k], inv, offs[(k + 1) / per]);
                    if ((unsigned)__double2hiint(v) >= 0x3ff00000u) v = fmin(v, 1.0);   // 1 and above, NaN, negative
                } else if (k == nval - 1) {
                    v = 1.0;
                }
                const float v32 = round_unit(v);
                p.cdf32[base + k] = v32;
                if (p.cdf64) p.cdf64[base + k] = v;
                reinterpret_cast<float*>(sums + k)[0] = v32;
            }
        } else {
            sweep(before, [&](int k, double run) { store(k, run); });
            for (int k = nval + lane; k < nint; k += 32) {
                p.cdf32[base + k] = 0.0f;
                if (p.cdf64) p.cdf64[base + k] = 0.0;
            }
        }
        __syncwarp();
        if (lane == 0 && p.nvalid) p.nvalid[row] = nval;
        if (p.guide) {
            // guide[k] = first entry >= k/G among the unmasked prefix (as the
            // sampler's bisection sees the row); the row was written by this warp
            const float* r = SMEM ? reinterpret_cast<const float*>(sums) : p.cdf32 + base;
            constexpr int step = SMEM ? 2 : 1;
            for (int k = lane; k <= MCD_GUIDE; k += 32) {
                const float q = (float)k / (float)MCD_GUIDE;
                int lo = 0, hi = nval;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    const float v = r[mid * step];
                    if (v != 0.0f && v < q) lo = mid + 1; else hi = mid;
                }
                p.guide[(size_t)row * (MCD_GUIDE + 1) + k] = (uint16_t)lo;
            }
        }
        __syncwarp();   // the next row reuses the warp's shared memory
    }
}

}  // namespace mcd

using namespace mcd;

extern "C" int mcd_build_table(int kind, const mcd_material* mat, int shell, int32_t nE, int32_t nW,
                               const float* Es, const float* Ws, float* cdf32, double* cdf64, int32_t* nvalid,
                               uint16_t* guide, void* stream) {
    if (!mat || !Es || !Ws || !cdf32) return MCD_EINVAL;
    if (nE < 1 || nW < 2) return MCD_EINVAL;
    if (guide && nW - 1 > 65535) return MCD_EINVAL;   // column indices must fit 16 bits
    if (kind != MCD_TABLE_MOLLER && kind != MCD_TABLE_GRYZ) return MCD_EINVAL;
    FillParams p;
    p.Es = Es;
    p.Ws = Ws;
    p.cdf32 = cdf32;
    p.cdf64 = cdf64;
    p.nvalid = nvalid;
    p.guide = guide;
    p.nE = nE;
    p.nW = nW;
    p.kind = kind;
    p.Ef32 = (float)mat->fermi_e;
    if (kind == MCD_TABLE_MOLLER) {
        p.Eb = 0.0;
    } else {
        if (shell < 0 || shell >= mat->n_shells) return MCD_EINVAL;
        p.Eb = mat->shell_E[shell];
    }
    int dev = 0, sms = 0, fit = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return MCD_ECUDA;
    // eight rows per block, fewer while that would leave SMs (and so their
    // FP64 pipes) idle; a resident grid whose warps stride over the rows, so
    // that the columns are computed once per block
    int w = 8;
    while (w > 1 && (nE + w - 1) / w < sms) w /= 2;
    const bool smem = nW - 1 <= kFillCols;
    const size_t bytes = smem ? fill_smem(w, nW) : 0;
    auto kern = smem ? k_fill<true> : k_fill<false>;
    if (allow_smem((const void*)kern, bytes) != MCD_OK) return MCD_ECUDA;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, 32 * w, bytes) != cudaSuccess) return MCD_ECUDA;
    if (fit < 1) return MCD_ETOOBIG;
    const long long rows = ((long long)nE + w - 1) / w, cap = (long long)sms * fit;
    kern<<<(unsigned)(rows < cap ? rows : cap), 32 * w, bytes, static_cast<cudaStream_t>(stream)>>>(p);
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}
