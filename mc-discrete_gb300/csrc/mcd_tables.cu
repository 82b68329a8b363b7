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
// One warp per E row: each lane owns a contiguous run of intervals and leaves
// its running sums in shared memory, the warp scans the 32 partial sums, and
// a coalesced pass writes the sums divided by the row total.  dsigma/dW
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
// two table-driven logarithms, one table-driven exponential and one
// Newton-refined square root, about 50 FP64 instructions.  The Moller value
// is a^2 + b^2 - a b with a = 1/W (column) and b = 1/(E - W), over E.
// Measured: the Au 30 keV tol 1e-4 pair (20000 x 499 and 100000 x 599 values)
// 67.7 -> 7.3 ms, float32 tables bit for bit the same.
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

// exp(-j/64), j = 0..63, each correctly rounded (its Taylor series in the
// double-double arithmetic of the other tables)
struct ExpTab {
    double e[64];
};
constexpr ExpTab cx_exp_tab() {
    ExpTab t{};
    for (int j = 0; j < 64; ++j) {
        const CxDD x = cx_div(CxDD{-(double)j, 0.0}, 64.0);
        CxDD term{1.0, 0.0}, sum{0.0, 0.0};
        for (int k = 0; k < 24; ++k) {
            sum = cx_add(sum, term);
            term = cx_div(cx_mul(term, x), k + 1.0);
        }
        t.e[j] = sum.hi + sum.lo;
    }
    return t;
}
static __device__ const ExpTab kExpTab = cx_exp_tab();

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

// exp(y) for y in (-1, 0]: exp(-j/64) times the series of the remainder
// r in (-1/64, 0] to r^6 (the next term is below 5e-17)
__device__ __forceinline__ double exp_unit(double y) {
    if (!(y > -0.99)) return exp(y);   // outside the table (not on the reference's grids)
    const int j = (int)(y * -64.0);
    const double r = fma((double)j, 1.0 / 64.0, y);
    const double p = fma(r, fma(r, fma(r, fma(r, fma(r, 1.0 / 720.0, 1.0 / 120.0), 1.0 / 24.0), 1.0 / 6.0), 0.5), 1.0);
    const double e = __ldg(&kExpTab.e[j]);
    return fma(e * r, p, e);
}

// sqrt(x) of a positive normal x: the hardware reciprocal square root, one
// Newton step on it, and one on the root itself (within one ulp)
__device__ __forceinline__ double sqrt_pos(double x) {
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double h = 0.5 * r;
    r = fma(h, fma(-x * r, r, 1.0), r);
    const double s = x * r;
    return fma(0.5 * r, fma(-s, s, x), s);
}

// What a grid point W contributes to every row: Gryzinski the exponent
// Eb/(Eb + W), W^-2 and (4/3) Eb W^-3; Moller 1/W.
struct FillCol {
    double a, b, c;
};
__device__ __forceinline__ FillCol fill_col(const FillParams& p, double W) {
    const double w1 = 1.0 / W;
    if (p.kind == MCD_TABLE_MOLLER) return FillCol{w1, 0.0, 0.0};
    const double w2 = w1 * w1;
    return FillCol{p.Eb / (p.Eb + W), w2, (4.0 / 3.0) * p.Eb * w2 * w1};
}

// dsigma/dW at (E, W) up to a factor of the row
__device__ __forceinline__ double fill_value(const FillParams& p, double E, double invE, double c1, double invEb,
                                             double W, const FillCol& q) {
    if (p.kind == MCD_TABLE_MOLLER) {
        const double b = rcp_pos(E - W);
        return fma(b, b - q.a, q.a * q.a);
    }
    const double x = fma(-W, invE, 1.0);
    const double pw = exp_unit(q.a * ln_pos(x));
    const double L = ln_pos(2.7 + sqrt_pos(x * invEb));
    return pw * fma(q.c, L, c1 * q.b);
}

constexpr int kFillCols = 1024;   // intervals a row may have to pass through shared memory

// Shared memory of a block of w warps: the columns of nW grid points, and per
// warp the row's running sums, its float values and the lanes' offsets.
constexpr size_t fill_smem(int w, int nW) {
    return sizeof(FillCol) * nW + (size_t)w * (sizeof(double) * (nW + 32) + sizeof(float) * nW);
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
    float* vals = reinterpret_cast<float*>(reinterpret_cast<double*>(cols + p.nW) + (size_t)nwarps * (p.nW + 32)) +
                  (size_t)warp * p.nW;
    if (SMEM) {
        for (int k = threadIdx.x; k < p.nW; k += blockDim.x) cols[k] = fill_col(p, (double)p.Ws[k]);
        __syncthreads();
    }
    const int per = (nint + 31) / 32;
    const int k0 = lane * per;
    const int k1 = min(k0 + per, nint);
    for (int row = blockIdx.x * nwarps + warp; row < p.nE; row += gridDim.x * nwarps) {
        const float e32 = p.Es[row];
        const double E = (double)e32;
        const float wmax = __fmul_rn(__fsub_rn(e32, p.Ef32), 0.5f);
        const double invE = 1.0 / E, epsB = p.Eb * invE, c1 = 1.0 - epsB, invEb = E / p.Eb;
        const bool open = p.kind == MCD_TABLE_MOLLER || epsB < 1.0;   // below the binding energy: 0
        // the lane's intervals (W ascends, so the unmasked ones are a prefix);
        // f(k, running sum) sees each
        auto sweep = [&](double run, auto f) {
            int k = k0;
            if (k < k1 && p.Ws[k + 1] <= wmax) {
                float wa = p.Ws[k];
                auto value = [&](int j, float w) {
                    if (!open || !((double)w < E)) return 0.0;
                    return fill_value(p, E, invE, c1, invEb, (double)w, SMEM ? cols[j] : fill_col(p, (double)w));
                };
                double fa = value(k, wa);
                for (; k < k1; ++k) {
                    const float wb = p.Ws[k + 1];
                    if (!(wb <= wmax)) break;
                    const double fb = value(k + 1, wb);
                    run = fma((double)__fmul_rn(__fsub_rn(wb, wa), 0.5f), fa + fb, run);
                    f(k, run);
                    wa = wb;
                    fa = fb;
                }
            }
            return run;
        };
        int valid = 0;
        const double part = sweep(0.0, [&](int k, double run) {
            if (SMEM) sums[k] = run;
            ++valid;
        });
        // warp scan of the partial sums (exclusive)
        double incl = part;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const double total = __shfl_sync(0xffffffffu, incl, 31);
        const int nval = __reduce_add_sync(0xffffffffu, valid);
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
            offs[lane] = incl - part;
            __syncwarp();
            const double inv = 1.0 / total;
            for (int k = lane; k < nint; k += 32) {
                double v = 0.0;
                if (k < nval) v = (k == nval - 1) ? 1.0 : fmin((sums[k] + offs[k / per]) * inv, 1.0);
                const float v32 = __double2float_rn(v);
                p.cdf32[base + k] = v32;
                if (p.cdf64) p.cdf64[base + k] = v;
                vals[k] = v32;
            }
        } else {
            sweep(incl - part, [&](int k, double run) { store(k, run); });
            for (int k = max(k0, nval); k < k1; ++k) {
                p.cdf32[base + k] = 0.0f;
                if (p.cdf64) p.cdf64[base + k] = 0.0;
            }
        }
        __syncwarp();
        if (lane == 0 && p.nvalid) p.nvalid[row] = nval;
        if (p.guide) {
            // guide[k] = first entry >= k/G among the unmasked prefix (as the
            // sampler's bisection sees the row); the row was written by this warp
            const float* r = SMEM ? vals : p.cdf32 + base;
            for (int k = lane; k <= MCD_GUIDE; k += 32) {
                const float q = (float)k / (float)MCD_GUIDE;
                int lo = 0, hi = nval;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    const float v = r[mid];
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
    if (bytes > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
        return MCD_ECUDA;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, 32 * w, bytes) != cudaSuccess) return MCD_ECUDA;
    if (fit < 1) return MCD_ETOOBIG;
    const long long rows = ((long long)nE + w - 1) / w, cap = (long long)sms * fit;
    kern<<<(unsigned)(rows < cap ? rows : cap), 32 * w, bytes, static_cast<cudaStream_t>(stream)>>>(p);
    return cudaGetLastError() == cudaSuccess ? MCD_OK : MCD_ECUDA;
}
