// Cell moments: the far wings of 2^cshift consecutive lines as one short
// series (CellHead in xs_internal.cuh has the formulas).
#include <cuda_runtime.h>

#include "xs_internal.cuh"

namespace xs {
namespace {

constexpr int kCellWarps = 4;

// Sums over the warp: on return lane L holds in v[0] the sum of v[L] over all
// lanes.  31 exchanges of doubles instead of 5 for each of the 32 values.
__device__ __forceinline__ void transpose_sum(double (&v)[32], int lane) {
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
        const bool up = (lane & w) != 0;
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const double give = up ? v[i] : v[i + w];
            const double got = __shfl_xor_sync(0xffffffffu, give, w);
            v[i] = (up ? v[i + w] : v[i]) + got;
        }
    }
}

// FP64: one warp per (cell, group of conditions), lanes over the cell's lines;
// y and pref of each (line, condition) from step one's RecV64 or, GROUPED,
// CondRec64.  30 terms x 6 FP64 operations per (line, condition), the pipe busy 41 %
// of the time at 14 warps per SM (116 registers; 1e6 lines); 1e7 lines 0.22 ms.
template <bool GROUPED, int C>
__global__ void __launch_bounds__(kCellWarps * 32) k_cells(CellArgs a) {
    constexpr int PM = kCellTerms64;
    const int lane = threadIdx.x & 31;
    const int cell = int(blockIdx.x) * kCellWarps + int(threadIdx.x >> 5);
    if (cell >= a.ncell) return;
    const int g = int(blockIdx.y);
    const long i0 = long(cell) << a.cshift;
    const long i1 = i0 + (1L << a.cshift) < a.n ? i0 + (1L << a.cshift) : a.n;
    const double c0 = 0.5 * (a.nu[i0] + a.nu[i1 - 1]);

    auto load = [&](long i, int k, double& y, double& pref) {
        const size_t c = size_t(g) * C + k;
        if constexpr (GROUPED) {
            const CondRec64& r = static_cast<const CondRec64*>(a.rec)[(size_t(g) * size_t(a.n) + size_t(i)) * C + k];
            y = r.y;
            pref = r.pref;
        } else {
            const RecV64& r = static_cast<const RecV64*>(a.rec)[c * size_t(a.n) + size_t(i)];
            y = r.y;
            pref = r.pref;
        }
    };
    const double s2 = 0.70710678118654752440;

    // The scale q (every |zeta|), the reach of W4's regions II-IV, and
    // whether every line is an ordinary one (else the cell is never far).
    float q = 0.0f, reach = 0.0f;
    bool good = true;
    for (long i = i0 + lane; i < i1; i += 32) {
        const double nu = a.nu[i];
        const double d = fabs(nu - c0);
        good = good && nu > 0.0;
#pragma unroll 1
        for (int k = 0; k < C; ++k) {
            double y, pref;
            load(i, k, y, pref);
            const double w = nu * a.dpw[g * C + k];
            const double re = fma(s2, w, d), gam = y * w;
            const float z = __double2float_ru(sqrt(fma(re, re, gam * gam)));
            const float h = __double2float_ru(d + (y < 15.0 ? (15.0 - y) * w : 0.0));
            // (a NaN fails the comparisons)
            good = good && w > 0.0 && z < 1.0e30f && h < 1.0e30f && fabs(pref) < 1.0e280;
            q = fmaxf(q, z);
            reach = fmaxf(reach, h);
        }
    }
    // non-negative floats order as their bit patterns
    q = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(q)));
    reach = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(reach)));
    good = __all_sync(0xffffffffu, good) && q > 0.0f;
    const size_t at = size_t(g) * size_t(a.ncell) + size_t(cell);
    if (lane == 0) {
        CellHead h;
        h.c0 = c0;
        // two grid steps beyond the regions: their intervals are placed on the
        // analytic grid, the tiles by the grid's own values
        h.dmin = good ? fmaxf(kCellKappa * q * 1.000001f, reach * 1.000001f + __double2float_ru(2.0 * a.df))
                      : __int_as_float(0x7f800000);
        h.q = q;
        a.head[at] = h;
    }
    if (!good) return;
    const double rq = 1.0 / double(q);
    double* M = a.mom + at * size_t(PM * C);
#pragma unroll 1
    for (int k = 0; k < C; ++k) {
        double m[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) m[j] = 0.0;
        const double dpw = a.dpw[g * C + k];
#pragma unroll 1
        for (long i = i0 + lane; i < i1; i += 32) {
            double y, pref;
            load(i, k, y, pref);
            const double nu = a.nu[i];
            const double w = nu * dpw;
            const double A = pref * w * (0.5 * kW4C * rq);
            const double d = (nu - c0) * rq, s = s2 * w * rq, gam = y * w * rq;
            // I_k = A Im(zeta^k) of both poles by
            // I_{k+1} = 2 Re(zeta) I_k - |zeta|^2 I_{k-1}
            const double p = d + s, n = d - s, g2 = gam * gam;
            const double p2 = 2.0 * p, n2 = 2.0 * n;
            const double pp = -fma(p, p, g2), nn = -fma(n, n, g2);
            double u0 = 0.0, u1 = A * gam, v0 = 0.0, v1 = u1;
#pragma unroll
            for (int j = 0; j < PM; ++j) {
                m[j] += u1 + v1;
                const double u = fma(p2, u1, pp * u0);
                u0 = u1;
                u1 = u;
                const double v = fma(n2, v1, nn * v0);
                v0 = v1;
                v1 = v;
            }
        }
        transpose_sum(m, lane);
        if (lane < PM) M[size_t(lane) * C + k] = m[0];
    }
}

// Mixed precision, from the (y, c pref) pairs of the group layouts: the same in
// FP32, the two poles as one packed FP32x2 operand, the sums over the lanes in
// FP64.  The amplitudes c pref w are formed from c pref times a power of two that
// brings the cell's largest to [1, 2), so that they are normal numbers however
// weak the lines are (S below 1e-38 leaves c pref w, and its reciprocal, outside
// the FP32 range); a moment is off by about 1e-7 of itself, as one FP32 evaluation
// of the line is.
// 16 terms x 3 packed operations per (line, condition).  Issue slots 66 %, XU (the
// conversions from FP64) 47 %, FMA pipe 36 % at 1e6 lines; 40 conditions x 1e7 lines
// 4.77 ms in FP64, 2.45 in FP32.
template <int C>
__global__ void __launch_bounds__(kCellWarps * 32) k_cells_f32(CellArgs a) {
    constexpr int PM = kCellTermsMixed;
    static_assert(PM == 16, "the transposed sum below is for 16 values");
    const int lane = threadIdx.x & 31;
    const int cell = int(blockIdx.x) * kCellWarps + int(threadIdx.x >> 5);
    if (cell >= a.ncell) return;
    const int g = int(blockIdx.y);
    const long i0 = long(cell) << a.cshift;
    const long i1 = i0 + (1L << a.cshift) < a.n ? i0 + (1L << a.cshift) : a.n;
    const double c0 = 0.5 * (a.nu[i0] + a.nu[i1 - 1]);
    const float2* yp = a.cyp + size_t(g) * C * size_t(a.n);
    const float s2 = 0.70710678f;

    // scale and reach (widened by 1e-6, far more than their FP32 rounding) and
    // the largest |c pref|
    float z2 = 0.0f, reach = 0.0f, big[C];
    bool good = true;
#pragma unroll
    for (int k = 0; k < C; ++k) big[k] = 0.0f;
    for (long i = i0 + lane; i < i1; i += 32) {
        const double nu = a.nu[i];
        const float d = fabsf(float(nu - c0)), nuf = float(nu);
        good = good && nu > 0.0;
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const float2 v = yp[size_t(k) * size_t(a.n) + size_t(i)];
            const float w = nuf * float(a.dpw[g * C + k]);
            const float re = fmaf(s2, w, d), gam = v.x * w;
            const float z = fmaf(re, re, gam * gam);
            const float h = d + (v.x < 15.0f ? (15.0f - v.x) * w : 0.0f);
            const float A = fabsf(v.y) * w;
            // (a NaN fails the comparisons)
            good = good && w > 0.0f && z < 1.0e30f && h < 1.0e30f && A < 1.0e37f;
            z2 = fmaxf(z2, z);
            reach = fmaxf(reach, h);
            big[k] = fmaxf(big[k], fabsf(v.y));
        }
    }
    // non-negative floats order as their bit patterns
    auto warp_max = [](float v) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v))); };
    z2 = warp_max(z2);
    reach = warp_max(reach);
    const float q = sqrtf(z2) * 1.000001f;
    good = __all_sync(0xffffffffu, good) && q > 0.0f;
    const size_t at = size_t(g) * size_t(a.ncell) + size_t(cell);
    if (lane == 0) {
        CellHead h;
        h.c0 = c0;
        // two grid steps beyond the regions: their intervals are placed on the
        // analytic grid, the tiles by the grid's own values
        h.dmin = good ? fmaxf(kCellKappa * q * 1.000001f, reach * 1.000002f + __double2float_ru(2.0 * a.df))
                      : __int_as_float(0x7f800000);
        h.q = q;
        a.head[at] = h;
    }
    if (!good) return;
    const double rq = 1.0 / double(q);
    double* M = a.mom + at * size_t(PM * C);
#pragma unroll 1
    for (int k = 0; k < C; ++k) {
        float bk = 0.0f;
#pragma unroll
        for (int j = 0; j < C; ++j) bk = j == k ? big[j] : bk;
        bk = warp_max(bk);
        // 2^(127 - e), e the biased exponent of bk (0: zero or subnormal)
        const int e = int(__float_as_uint(bk) >> 23);
        const float sv = __uint_as_float(unsigned(max(254 - e, 1)) << 23);
        const double wq = a.dpw[g * C + k] * rq;
        float2 m[PM];
#pragma unroll
        for (int j = 0; j < PM; ++j) m[j] = make_float2(0.0f, 0.0f);
#pragma unroll 1
        for (long i = i0 + lane; i < i1; i += 32) {
            const float2 v = yp[size_t(k) * size_t(a.n) + size_t(i)];
            const double nu = a.nu[i];
            const float w = float(nu * wq), d = float((nu - c0) * rq);  // in units of q
            // c pref sv w, |c pref| sv < 2, through nu dpw as above
            const float A = (v.y * sv) * (float(nu) * float(a.dpw[g * C + k]));
            const float s = s2 * w, gam = v.x * w, g2 = gam * gam;
            // I_k = A Im(zeta^k) of both poles by
            // I_{k+1} = 2 Re(zeta) I_k - |zeta|^2 I_{k-1}
            const float p = d + s, n = d - s;
            const float2 r2 = make_float2(2.0f * p, 2.0f * n);
            const float2 nn = make_float2(-fmaf(p, p, g2), -fmaf(n, n, g2));
            float2 u0 = make_float2(0.0f, 0.0f), u1 = make_float2(A * gam, A * gam);
#pragma unroll
            for (int j = 0; j < PM; ++j) {
                m[j] = __fadd2_rn(m[j], u1);
                const float2 u = __ffma2_rn(r2, u1, __fmul2_rn(nn, u0));
                u0 = u1;
                u1 = u;
            }
        }
        // sums over the lanes in FP64: lane L ends with moment L & 15
        double t[PM];
#pragma unroll
        for (int j = 0; j < PM; ++j) t[j] = double(m[j].x) + double(m[j].y);
#pragma unroll
        for (int w = PM / 2; w >= 1; w >>= 1) {
            const bool up = (lane & w) != 0;
#pragma unroll
            for (int i = 0; i < w; ++i) {
                const double got = __shfl_xor_sync(0xffffffffu, up ? t[i] : t[i + w], w);
                t[i] = (up ? t[i + w] : t[i]) + got;
            }
        }
        t[0] += __shfl_xor_sync(0xffffffffu, t[0], 16);
        // A stands for c pref w sv; the series wants c pref w / (2 q)
        if (lane < PM) M[size_t(lane) * C + k] = t[0] * (0.5 / double(sv) * rq);
    }
}

}  // namespace

cudaError_t launch_cells(bool mixed, const CellArgs& a, cudaStream_t stream) {
    if (a.ncell <= 0 || a.ncond <= 0) return cudaSuccess;
    const dim3 grid(unsigned((a.ncell + kCellWarps - 1) / kCellWarps),
                    unsigned(a.group > 1 ? a.ncond / a.group : a.ncond));
    auto go = [&](auto kernel) {
        kernel<<<grid, kCellWarps * 32, 0, stream>>>(a);
        return cudaGetLastError();
    };
    switch (a.group) {
        case 0: return mixed ? cudaErrorInvalidValue : go(k_cells<false, 1>);
        case 1: return mixed ? go(k_cells_f32<1>) : cudaErrorInvalidValue;
        case 2: return mixed ? go(k_cells_f32<2>) : go(k_cells<true, 2>);
        case 4: return mixed ? go(k_cells_f32<4>) : go(k_cells<true, 4>);
        case 8: return mixed ? go(k_cells_f32<8>) : go(k_cells<true, 8>);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace xs
