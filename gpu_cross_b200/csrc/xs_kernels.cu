// sm_100a kernels of the cross-section engine.
//
//  k_grid_check   validates the grid (ascending, uniform step) once per run.
//  k_prep         "step one" per (line, condition): intensity S(T), Lorentz
//                 width, Doppler width, the exact window of grid indices each
//                 line reaches, and a packed record for step two.
//  k_cells        (xs_cells.cu) per cell of consecutive lines, the moments that
//                 stand for the lines' far wings.
//  k_steptwo_*    "step two": a persistent grid of warps takes work items
//                 (condition or group of conditions, tile of grid points) from
//                 an atomic counter.  A warp finds the lines whose windows meet
//                 its tile with a 32-way ballot search over the window arrays,
//                 streams the records of those that are too near the tile for
//                 their cells through a per-warp shared memory stage
//                 (cp.async), accumulates the tile in registers -- a lane per
//                 point or a lane per line -- and adds the far cells' series: a
//                 fixed summation order, no atomics on the result.
//
// The reference computes the same sums with one CTA per grid point that scans
// the whole chunk (cross_kernal.cu:924-997, :654-723).
#include <cuda_runtime.h>

#include <cfloat>
#include <climits>
#include <cmath>
#include <type_traits>

#include "xs_internal.cuh"

namespace xs {
namespace {

// Depth of the per-warp cp.async staging pipeline (groups of 32 records).
constexpr int kStages = 3;

// Offsets (in Doppler widths) from which a line's every pair takes the
// per-pair path, x from its FP64 centre ("whole" lines): FP32 offsets and
// the region-I sums are exact enough below it.
constexpr double kWholeXMax = 1.0e8;
// Lines whose x^2 + y^2 stays below kPairUMax over their tiles and whose
// |Pc| stays below kPairPcMax, for every condition of the group ("narrow"
// lines, the usual case), share reciprocals between two lines or points: their
// denominators lie in [1, 6.3e18], so dA dB lies in [1, 4e37] and its
// reciprocal is a normal FP32 number, and the numerators |Pc (u + 1)| stay
// below 2.5e17, so the cross products nA dB of two lines stay below 1.6e36
// (and, d being >= 1, never fall below |n|).  Other lines are marked
// kLineWide.
constexpr double kPairUMax = 2.5e9;
constexpr double kPairPcMax = 1.0e8;
// Wide lines below these take a reciprocal per pair with no test: u^2 stays below
// 1e36 and Pc (u + 1) below 1e36.
constexpr double kSoloUMax = 1.0e18, kSoloPcMax = 1.0e18;


// ---------------------------------------------------------------------------
// Small complex arithmetic for the W4 regions II-IV.
// ---------------------------------------------------------------------------
struct cplx {
    double re, im;
};
__device__ __forceinline__ cplx operator+(double a, cplx b) { return {a + b.re, b.im}; }
__device__ __forceinline__ cplx operator-(double a, cplx b) { return {a - b.re, -b.im}; }
__device__ __forceinline__ cplx operator*(cplx a, cplx b) {
    return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__device__ __forceinline__ cplx operator*(cplx a, double b) { return {a.re * b, a.im * b}; }
// Real part of a / b.
__device__ __forceinline__ double div_re(cplx a, cplx b) {
    return (a.re * b.re + a.im * b.im) / (b.re * b.re + b.im * b.im);
}

// Re w(x + iy) by Humlicek's W4 (JQSRT 27 (1982) 437): four regions chosen
// on s = |x| + y and y vs 0.195|x| - 0.176 (the region tests and the
// coefficient table are Humlicek's, as used by cross_kernal.cu:149-181 and
// profiles.cpp:9-42).  Region I is evaluated as a real rational, the others
// with complex Horner schemes.
__device__ double w4_re(double x, double y) {
    const double s = fabs(x) + y;
    if (s >= 15.0) {
        const double x2 = x * x, y2 = y * y;
        const double dr = 0.5 + y2 - x2;
        return kW4C * y * (0.5 + x2 + y2) / (dr * dr + 4.0 * x2 * y2);
    }
    const cplx t = {y, -x};
    if (s >= 5.5) {
        const cplx u = t * t;
        const cplx num = t * (1.410474 + u * .5641896);
        const cplx den = .75 + u * (3. + u);
        return div_re(num, den);
    }
    if (y >= 0.195 * fabs(x) - 0.176) {
        const cplx num = 16.4955 + t * (20.20933 + t * (11.96482 + t * (3.778987 + t * .5642236)));
        const cplx den =
            16.4955 + t * (38.82363 + t * (39.27121 + t * (21.69274 + t * (6.699398 + t))));
        return div_re(num, den);
    }
    const cplx u = t * t;
    double sn, cs;
    sincos(u.im, &sn, &cs);
    const double eu = exp(u.re);
    const cplx num =
        36183.31 - u * (3321.9905 - u * (1540.787 - u * (219.0313 - u * (35.76683 - u * (1.320522 - u * .56419)))));
    const cplx den =
        32066.6 - u * (24322.84 - u * (9022.228 - u * (2186.181 - u * (364.2191 - u * (61.57037 - u * (1.841439 - u))))));
    return eu * cs - div_re(t * num, den);
}

// First j in [s, e) with pred(j) true (pred monotone false..true), or e.
// Starts from a guess and walks; falls back to bisection after 8 steps.
template <class Pred>
__device__ int find_first(int s, int e, double guess, Pred pred) {
    long j;
    if (!(guess > double(s))) j = s;  // also catches NaN
    else if (guess > double(e)) j = e;
    else j = long(guess);
    for (int it = 0; it < 8; ++it) {
        if (j > s && pred(int(j - 1))) { --j; continue; }
        if (j < e && !pred(int(j))) { ++j; continue; }
        return int(j);
    }
    int lo = s, hi = e;
    while (lo < hi) {
        int mid = lo + (hi - lo) / 2;
        if (pred(mid)) hi = mid; else lo = mid + 1;
    }
    return lo;
}

__device__ __forceinline__ int clamp_index(double v, int lo, int hi) {
    if (!(v > double(lo))) return lo;  // NaN -> lo
    if (v > double(hi)) return hi;
    return int(v);
}

// ---------------------------------------------------------------------------
// Grid check.
// ---------------------------------------------------------------------------
// Also clears the words step one and step two start from (kc, counter; NULL:
// left alone), which saves two memsets per call.
__global__ void k_grid_check(GridDev g, unsigned* err, int* kc, unsigned* counter) {
    if (blockIdx.x == 0 && kc) {
        for (int t = threadIdx.x; t < kKcWords; t += blockDim.x) kc[t] = 0;
        if (threadIdx.x == 0) *counter = 0;
    }
    const int j = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (j >= g.npoints_total) return;
    const double f0 = g.freq[0];
    const double fj = g.freq[j];
    bool bad = !(fj > g.freq[j - 1]);
    bad |= !(fabs(fj - (f0 + double(j) * g.df)) <= 0.01 * g.df);
    if (bad) atomicOr(err, kErrGrid);
}

// ---------------------------------------------------------------------------
// Step one.
// ---------------------------------------------------------------------------
// Mixed multi-condition layout: outside x^2 + y^2 < kNearR2 the region-I
// rational stays below 2 Pc (u >= 1), so step two adds it there on every
// line; inside, only the lines within the core-candidate reach can have
// pairs, and step two tests u on them.
constexpr double kNearR2 = 1.5;
// Grid indices [jlo, jhi] of the window [lo, hi) where |x| + y < lim, with
// x = (nu - f_j) g in FP64 on the analytic grid f_j = f0 + j df: the region
// choice of the FP64 path (up to the grid's last-bit rounding), so that no
// pair changes region with the FP32 rounding of x.  Empty: jlo > jhi.
// md = (nu - f0) / df, q = 1 / (g df) and tb = |md| + (|nu| + |f0|) / df
// (the line's part of the rounding tolerance below) come precomputed; md and
// q place the interval's ends, and the region test itself decides where an
// end is close to a grid point.
__device__ __forceinline__ double region_tol_base(double nu, double f0, double df, double md) {
    return fabs(md) + (fabs(nu) + fabs(f0)) / df;
}
__device__ __forceinline__ void region_interval_q(double nu, double g, double y, double lim, int lo, int hi, double f0,
                                  double df, double md, double q, double tb, int& jlo, int& jhi) {
    jlo = 1;
    jhi = 0;
    if (!(y < lim) || lo >= hi) return;
    const double hq = (lim - y) * q;
    // x_j = (md - j) / q, so the points inside are the integers of
    // (md - hq, md + hq).  The region test's roundings (f_j, nu - f_j, the
    // product with g, md and hq themselves) move both ends by a few 1e-16 of
    // |md|, (|nu| + |f0|) / df and hq grid steps; where each end lies further
    // than `tol` (a thousand times that, and at least 1e-6) from an integer,
    // the exact region test of every point agrees with [ceil(md - hq),
    // ceil(md + hq) - 1], clamped to the window, and is not evaluated.
    // Otherwise the walks below decide.
    {
        const double bl = md - hq, bh = md + hq;
        const double tol = 1.0e-6 + 1.0e-13 * (tb + hq);
        if (fabs(bl) < 1.0e9 && fabs(bh) < 1.0e9 && fabs(bl - rint(bl)) > tol && fabs(bh - rint(bh)) > tol) {
            // ceil to int in one conversion, clamped in integers (lo < hi)
            const int jl = min(max(__double2int_ru(bl), lo), hi), jh = min(max(__double2int_ru(bh), lo), hi);
            if (jl < jh) {
                jlo = jl;
                jhi = jh - 1;
            }
            return;
        }
    }
    auto fa = [&](int j) { return fma(double(j), df, f0); };
    auto inside = [&](int j) { return !(fabs((nu - fa(j)) * g) + y >= lim); };
    const int jl = find_first(lo, hi, ceil(md - hq), [&](int j) { return fa(j) > nu || inside(j); });
    const int jh = find_first(lo, hi, floor(md + hq) + 1.0, [&](int j) { return fa(j) > nu && !inside(j); });
    if (jl < jh) {
        jlo = jl;
        jhi = jh - 1;
    }
}

// The intervals of region II-IV (|x| + y < 15) and of regions III-IV
// (|x| + y < 5.5), with md, q and tb computed once for both.
__device__ void region_intervals(double nu, double g, double y, int lo, int hi, double f0, double df, int& j15,
                                 int& k15, int& j55, int& k55) {
    const double md = (nu - f0) / df, q = 1.0 / (g * df);
    const double tb = region_tol_base(nu, f0, df, md);
    region_interval_q(nu, g, y, 15.0, lo, hi, f0, df, md, q, tb, j15, k15);
    region_interval_q(nu, g, y, 5.5, lo, hi, f0, df, md, q, tb, j55, k55);
}

// Step one of one (line, condition).  Returns the line's core half-width in
// grid points (Voigt; 0 otherwise).  `reach` (mixed Voigt): the largest
// distance, in grid points, from the line's nearest grid index to its region
// interval (the core pass's reach).  The mixed-precision multi-condition
// layout has its own step one (k_prep_lines_x); the FP64 one is written here.
template <int KIND, int CONV, bool MIXED>
__device__ __forceinline__ int prep_line(const PrepArgs& a, long i, int c, int* reach = nullptr) {
    const CondDev& C = a.cond[c];
    const double* F = a.G.freq;
    const double f0 = F[0];
    const double df = a.G.df;
    const int s = a.G.start, e = a.G.start + a.G.points;
    const double nu = a.L.nu[i];
    if (c == 0 && i > 0 && nu < a.L.nu[i - 1]) atomicOr(a.err, kErrUnsorted);
    const bool streamed = KIND == kVoigt && CONV == kConvGpu && a.L.s32 != nullptr;
    // per-temperature cache: read S(T) and (T_ref/T)^n, or compute and store
    const bool tc_read = a.L.tc_mode == 1, tc_write = a.L.tc_mode == 2;
    const bool from_lines = !streamed && !tc_read;
    const double ei = from_lines ? a.L.energies[i] : 0.0;
    const double aif = from_lines ? a.L.aif[i] : 0.0;
    const double gns = from_lines ? double(a.L.gns[i]) : 0.0;
    const double cut = C.cut;
    const size_t ci = size_t(c) * size_t(a.L.n) + size_t(i);
    int kcl = 0;

    // Intensity, centre used for offsets, and the reference window.
    double S, nu_p;
    int lo, hi;
    if (CONV == kConvGpu) {
        if (KIND == kVoigt) {
            // device_compute_cross_section_voigt_stepone, cross_kernal.cu:775-779
            double nu_if = nu;
            if (nu_if == 0) nu_if = 1e-6;
            if (streamed) {
                S = double(a.L.s32[i]);
            } else if (tc_read) {
                S = a.L.tc_s[i];
            } else {
                S = C.cmcoef * aif * gns * kISQRTPI * exp(-C.beta * ei) * (1.0 - exp(-C.beta * nu_if)) /
                    (nu_if * nu_if * C.partition);
                if (gns == -1) S = aif;
            }
        } else if (tc_read) {
            S = a.L.tc_s[i];
        } else {
            // doppler_stepone / stepone, cross_kernal.cu:645-648, :487-490
            S = C.cmcoef * aif * gns * exp(-C.beta * ei) * (1.0 - exp(-C.beta * nu)) /
                (nu * nu * C.partition);
            if (nu == 0) S = 0.0;
        }
        nu_p = nu;  // step two reads the uploaded centre (cross_kernal.cu:951)
        if (KIND == kGauss) {
            // |f - nu| <= cut with dnu = f - nu (cross_kernal.cu:599-602)
            lo = find_first(s, e, ceil((nu - cut - f0) / df),
                            [&](int j) { return !(F[j] - nu < -cut); });
            hi = find_first(s, e, ceil((nu + cut - f0) / df),
                            [&](int j) { return F[j] - nu > cut; });
        } else {
            // -cut <= nu - f <= cut (cross_kernal.cu:952-957, :684-687)
            lo = find_first(s, e, ceil((nu - cut - f0) / df),
                            [&](int j) { return !(nu - F[j] > cut); });
            hi = find_first(s, e, ceil((nu + cut - f0) / df),
                            [&](int j) { return nu - F[j] < -cut; });
        }
    } else {
        // OpenMPManager::ComputeVoigt / ComputeDoppler, OpenMPManager.cpp:196-208, :151-163
        double nu_if = nu;
        if (nu_if == 0) nu_if = 1e-6;
        if (tc_read)
            S = a.L.tc_s[i];
        else if (KIND == kVoigt)
            S = C.cmcoef * aif * gns * kISQRTPI * exp(-C.beta * ei) * (1.0 - exp(-C.beta * nu_if)) /
                (nu_if * nu_if * C.partition);
        else
            S = C.cmcoef * aif * gns * exp(-C.beta * ei) * (1.0 - exp(-C.beta * nu_if)) /
                (nu_if * nu_if * C.partition);
        nu_p = nu_if;
        const double rb = round((nu_if - cut - f0) / df);
        const double re = round((nu_if + cut - f0) / df);
        // ib = max(rb, start), ie = min(re, start + points); both clamped into
        // [s, e] so the arrays stay monotone (an empty range stays empty).
        lo = clamp_index(rb > double(s) ? rb : double(s), s, e);
        hi = clamp_index(re < double(e) ? re : double(e), s, e);
        // Lines with S == 0 are skipped (OpenMPManager.cpp:163, :208); they
        // keep their window (monotone arrays) and add exactly 0 below.
    }

    if (tc_write) a.L.tc_s[i] = S;
    if (KIND == kVoigt) {
        // an empty window has length 0 (a negative cut, from a negative pressure,
        // puts hi below lo; step two takes hi - lo as unsigned)
        if (hi < lo) hi = lo;
        double pw = 0.0;
        if (!streamed) {
            pw = tc_read ? a.L.tc_pw[i] : pow(C.tratio, a.L.nexp[i]);
            if (tc_write) a.L.tc_pw[i] = pw;
        }
        const double gl = streamed ? double(a.L.gl32[i]) : a.L.gamma[i] * C.gamma_scale * pw;
        const double g = 1.0 / (nu_p * C.dpw);  // gammaG, cross_kernal.cu:958
        const double y = gl * g;
        const double pref = (CONV == kConvCpu && S == 0.0) ? 0.0 : S * g;
        const double y2 = y * y;
        const double Pc = pref * kW4C * y;
        const double Cy = y2 - 0.5;
        const double D2 = 2.0 * y2;
        const double m = rint((nu_p - f0) / df);
        // Grid indices where |x| + y < 15 is possible (region I not
        // guaranteed), with a margin of two points either side.
        double clo_d = 3.0e7, chi_d = -3.0e7;
        if (y < 15.0) {
            double h = (15.0 - y) / g;
            h = h * (1.0 + 1e-9) + 1e-12 * fabs(nu_p);
            clo_d = floor((nu_p - h - f0) / df) - 2.0;
            chi_d = ceil((nu_p + h - f0) / df) + 2.0;
            if (!(clo_d > -3.0e7)) clo_d = -3.0e7;
            if (!(chi_d < 3.0e7)) chi_d = 3.0e7;
        }
        // FP32 offsets need |m| < 2^24 and x below ~1e8 over the window;
        // otherwise every pair of the line takes the per-pair path.
        bool whole = false;
        if (MIXED) {
            const double xw = (cut + double(a.mixed_tile_span + 4) * df) * g;
            whole = !(fabs(m) < 16000000.0) || !(xw < kWholeXMax);
        }
        if (whole) {
            clo_d = -3.0e7;
            chi_d = 3.0e7;
            kcl = 30000000;
        } else if (chi_d >= clo_d) {
            const double w = fmax(m - clo_d, chi_d - m) + 1.0;
            kcl = w < 3.0e7 ? int(w) : 30000000;
        }
        if (c == 0) a.mi[i] = int(fmin(fmax(m, -1073741824.0), 1073741824.0));
        if (!MIXED && a.group > 0) {
            // FP64 multi-condition layout (conditions of a group share the
            // window).
            const int C = a.group;
            const int cg = c / C, cl = c - cg * C;
            const size_t gi = size_t(cg) * size_t(a.L.n) + size_t(i);
            int core = -1;
            if (whole) {
                core = 0x7fff | (0x7fff << 16);
            } else if (chi_d >= clo_d) {
                const int aa = int(fmin(m - clo_d, 32767.0));
                const int bb = int(fmin(chi_d - m, 32767.0));
                core = aa | (bb << 16);
            }
            {
                CondRec64 cr;
                cr.g = g;
                cr.Cy = Cy;
                cr.D2 = D2;
                cr.Pc = Pc;
                cr.y = y;
                cr.pref = pref;
                cr.core = core;
                cr.pad0 = cr.pad1 = cr.pad2 = 0;
                reinterpret_cast<CondRec64*>(a.rec)[gi * C + cl] = cr;
                if (cl == 0) {
                    LineSh64 ls;
                    ls.nu = nu_p;
                    ls.lo = lo;
                    ls.hi = hi;
                    reinterpret_cast<LineSh64*>(a.lsh)[gi] = ls;
                }
            }
            if (cl == 0) {
                a.wlo[gi] = lo;
                a.whi[gi] = hi;
            }
            return kcl;
        }
        if (MIXED && a.group == 1) {
            // one condition per group of the line-parallel step two: offsets
            // scaled by g, x = (m - j) dfn + rn
            LineShX ls;
            const double xw = (cut + double(a.mixed_tile_span + 4) * df) * g;
            ls.m = float(fabs(m) < 16000000.0 ? m : 0.0);
            ls.dfn = float(df * g);
            ls.rn = float(((nu_p - f0) - m * df) * g);
            ls.flags = (whole || !(xw * xw + y2 < kSoloUMax) || !(fabs(Pc) < kSoloPcMax) ? kLineWhole : 0) |
                       (!(xw * xw + y2 < kPairUMax) || !(fabs(Pc) < kPairPcMax) ? kLineWide : 0);
            ls.lo = lo;
            ls.hi = hi;
            ls.nu = nu_p;
            reinterpret_cast<LineShX*>(a.lsh)[ci] = ls;
            CoreIv iv;
            region_intervals(nu_p, g, y, lo, hi, f0, df, iv.lo15, iv.hi15, iv.lo55, iv.hi55);
            int rch = 0;
            if (iv.lo15 <= iv.hi15) {
                const double w = fmax(m - double(iv.lo15), double(iv.hi15) - m);
                rch = w < 3.0e7 ? int(w) : 30000000;
                if (!(w < 3.0e7)) atomicOr(a.err, kErrReach);
            }
            if (reach) *reach = rch;
            kcl = 0;
            a.civ[ci] = iv;
            a.cyp[ci] = make_float2(float(y), float(pref * kW4C));
        } else if (MIXED) {
            RecV32 rr;
            rr.m = float(fabs(m) < 16000000.0 ? m : 0.0);
            rr.ra = float(((nu_p - f0) - m * df) * g);
            rr.dfa = float(whole ? -df * g : df * g);  // negative: x from the FP64 centre
            rr.Cy = float(Cy);
            rr.D2 = float(D2);
            rr.Pc = float(Pc);
            rr.pref = float(pref);
            rr.y = float(y);
            rr.lo = float(lo);
            rr.hi = float(hi);
            // exact intervals: step two leaves [clo, chi] to the core pass
            int j15, k15, j55, k55;
            region_intervals(nu_p, g, y, lo, hi, f0, df, j15, k15, j55, k55);
            int rch = 0;
            if (j15 <= k15) {
                const double w = fmax(m - double(j15), double(k15) - m);
                rch = w < 3.0e7 ? int(w) : 30000000;
                if (!(w < 3.0e7)) atomicOr(a.err, kErrReach);  // the core pass would not find it
            }
            if (reach) *reach = rch;
            kcl = whole ? 30000000 : rch;  // a whole line is a core candidate of every tile
            rr.clo = float(j15);
            rr.chi = float(k15);
            rr.lo55 = float(j55);
            rr.hi55 = float(k55);
            rr.nu = nu_p;
            reinterpret_cast<RecV32*>(a.rec)[ci] = rr;
        } else {
            RecV64 rr;
            rr.nu = nu_p;
            rr.g = g;
            rr.Cy = Cy;
            rr.D2 = D2;
            rr.Pc = Pc;
            rr.y = y;
            rr.pref = pref;
            rr.pad = 0.0;
            rr.lo = lo;
            rr.hi = hi;
            rr.clo = int(clo_d);
            rr.chi = int(chi_d);
            reinterpret_cast<RecV64*>(a.rec)[ci] = rr;
        }
    } else {
        // Doppler / Gaussian: pairs whose two erf arguments are both beyond
        // kErfSat on the same side add exactly 0; narrow the window to the
        // rest (with margins), keeping it monotone in nu.
        double g = 0.0, lo_f, hi_f;
        if (KIND == kDoppler) {
            g = 1.0 / (nu_p * C.dpw);
            const double w = kErfSat * C.dpw * (1.0 + 1e-6);
            const double abs_m = a.x0 * (1.0 + 1e-6) + 2.0 * df;
            lo_f = nu_p * (1.0 - w) - abs_m;
            hi_f = nu_p * (1.0 + w) + abs_m;
        } else {
            const double wg = (kErfSat + a.x0g) / a.xg * (1.0 + 1e-6) + 2.0 * df;
            lo_f = nu_p - wg;
            hi_f = nu_p + wg;
        }
        const int alo = clamp_index(floor((lo_f - f0) / df), s, e);
        const int ahi = clamp_index(ceil((hi_f - f0) / df) + 1.0, s, e);
        if (alo > lo) lo = alo;
        if (ahi < hi) hi = ahi;
        RecE64 rr;
        rr.nu = nu_p;
        rr.s = (CONV == kConvCpu && S == 0.0) ? 0.0 : S;
        rr.g = g;
        rr.pad = 0.0;
        rr.lo = lo;
        rr.hi = hi;
        rr.pad0 = rr.pad1 = 0;
        reinterpret_cast<RecE64*>(a.rec)[ci] = rr;
    }
    a.wlo[ci] = lo;
    a.whi[ci] = hi;
    return kcl;
}

template <int KIND, int CONV, bool MIXED>
__global__ void __launch_bounds__(256) k_prep(PrepArgs a) {
    const long i = a.line0 + long(blockIdx.x) * blockDim.x + threadIdx.x;
    const int c = blockIdx.y;
    int kcl = 0, rch = 0;
    if (i < (a.line1 > 0 ? a.line1 : a.L.n)) kcl = prep_line<KIND, CONV, MIXED>(a, i, c, &rch);
    if (KIND == kVoigt) {
        // Block maxima of the core widths (kc) and, mixed, of the core pass's
        // reach (kc + kMaxCond), one atomic each per block.
        __shared__ int smax[2][8];
        kcl = __reduce_max_sync(0xffffffffu, kcl);
        rch = __reduce_max_sync(0xffffffffu, rch);
        if ((threadIdx.x & 31) == 0) {
            smax[0][threadIdx.x >> 5] = kcl;
            smax[1][threadIdx.x >> 5] = rch;
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            int m = 0;
            for (int w = 0; w < int(blockDim.x >> 5); ++w) m = smax[threadIdx.x][w] > m ? smax[threadIdx.x][w] : m;
            if (m > 0) atomicMax(a.kc + threadIdx.x * kMaxCond + c, m);
        }
    }
}

// Step one of the mixed-precision multi-condition layout, one thread per line
// over every group of C conditions.  The line's data is read once; the
// intensity, the Lorentz temperature power and 1/Doppler width of each
// temperature class (conditions with the same beta, Q, T_ref/T and Doppler
// width; the 40-condition sweep has 10) are computed once per line and kept
// in shared memory (up to kMaxClassCache classes; beyond, each condition
// computes its own); what groups with the same cut share -- the window, the
// condition-free offsets (LineShX) -- is written once per run of such
// groups; the conditions follow in order, their loop not unrolled, which
// keeps the code small.  Each value takes the FP64 path's operations in the
// same order (the W4 region intervals are the FP64 region choice).  Every
// store but the window data's is coalesced (conditions outermost); step two
// forms the region-I constants from (y, pref) itself, which took 12 bytes per
// line and condition and the L1's store bandwidth here (4-byte stores 96 bytes
// apart).  The core-candidate reach (kc) covers the
// pairs where x^2 + y^2 < kNearR2, at least one grid point beyond: there the
// region-I rational may exceed W4 by far, and step two tests u on the lines
// of that reach.
template <int CONV, int C>
__global__ void __launch_bounds__(256, 3) k_prep_lines_x(PrepArgs a) {
    static_assert(C % 2 == 0, "conditions come in pairs");
    extern __shared__ __align__(16) double cls[];  // [3][ncache][256]: S, (T_ref/T)^n, g
    __shared__ int smax[2][kMaxCond][8];
    const int ngroups = a.ncond / C;
    const long i = a.line0 + long(blockIdx.x) * 256 + threadIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool live = i < (a.line1 > 0 ? a.line1 : a.L.n);
    const double* F = a.G.freq;
    const double f0 = F[0];
    const double df = a.G.df;
    const int s = a.G.start, e = a.G.start + a.G.points;

    double nu = 0.0, ei = 0.0, aif = 0.0, gns = 0.0, gam = 0.0, nex = 0.0;
    if (live) {
        nu = a.L.nu[i];
        if (i > 0 && nu < a.L.nu[i - 1]) atomicOr(a.err, kErrUnsorted);
        ei = a.L.energies[i];
        aif = a.L.aif[i];
        gns = double(a.L.gns[i]);
        gam = a.L.gamma[i];
        nex = a.L.nexp[i];
    }
    double nu_if = nu;
    if (nu_if == 0) nu_if = 1e-6;
    // step two reads the uploaded centre in the GPU convention
    // (cross_kernal.cu:951), the nu = 0 guarded one in the CPU convention
    const double nu_p = CONV == kConvGpu ? nu : nu_if;
    const double md = (nu_p - f0) / df;
    const double m = rint(md);
    const double nu_df = nu_p / df;  // q = 1 / (g df) = nu_df * dpw
    const double tb = region_tol_base(nu_p, f0, df, md);
    const bool far_m = !(fabs(m) < 16000000.0);
    const int im = int(fmin(fmax(m, -1073741824.0), 1073741824.0));
    if (live) a.mi[i] = im;

    // device_compute_cross_section_voigt_stepone, cross_kernal.cu:775-779
    // (GPU); OpenMPManager.cpp:196-200 (CPU)
    auto class_values = [&](const CondDev& Cd, double& S, double& pw, double& g) {
        S = Cd.cmcoef * aif * gns * kISQRTPI * exp(-Cd.beta * ei) * (1.0 - exp(-Cd.beta * nu_if)) /
            (nu_if * nu_if * Cd.partition);
        if (CONV == kConvGpu && gns == -1) S = aif;
        pw = pow(Cd.tratio, nex);
        g = 1.0 / (nu_p * Cd.dpw);  // gammaG, cross_kernal.cu:958
    };
    const int ncache = a.nclass <= kMaxClassCache ? a.nclass : 0;
    double* cS = cls;
    double* cP = cls + ncache * 256;
    double* cG = cls + 2 * ncache * 256;
    if (live) {
        for (int t = 0; t < ncache; ++t)
            class_values(a.cond[a.class_rep[t]], cS[t * 256 + tid], cP[t * 256 + tid], cG[t * 256 + tid]);
    }

    // Window data (LineShX, lo, hi) once per run of groups with the same cut
    // (a.wslot), written when the run ends: its wide flag covers every
    // condition of the run.
    double cut_prev = -1.0;
    int lo = s, hi = s;
    int slot = -1;
    bool wide = false, far = false;
    auto flush_window = [&]() {
        if (!live || slot < 0) return;
        const size_t wi = size_t(slot) * size_t(a.L.n) + size_t(i);
        LineShX ls;
        ls.m = float(far_m ? 0.0 : m);
        ls.dfn = float(df / nu_p);
        ls.rn = float(((nu_p - f0) - m * df) / nu_p);
        ls.flags = (far_m ? kLineWhole : 0) | (wide ? kLineWide : 0) | (far ? kLineFar : 0);
        ls.lo = lo;
        ls.hi = hi;
        ls.nu = nu_p;
        reinterpret_cast<LineShX*>(a.lsh)[wi] = ls;
        a.wlo[wi] = lo;
        a.whi[wi] = hi;
    };
    for (int cg = 0; cg < ngroups; ++cg) {
        if (a.wslot[cg] != slot) {
            flush_window();
            slot = a.wslot[cg];
            wide = far = false;
            const double cut = a.cond[cg * C].cut;  // a run of groups shares its cut
            cut_prev = cut;
            if (live) {
                if (CONV == kConvGpu) {
                    // -cut <= nu - f <= cut (cross_kernal.cu:952-957)
                    lo = find_first(s, e, ceil((nu - cut - f0) / df), [&](int j) { return !(nu - F[j] > cut); });
                    hi = find_first(s, e, ceil((nu + cut - f0) / df), [&](int j) { return nu - F[j] < -cut; });
                } else {
                    // OpenMPManager.cpp:196-208
                    const double rb = round((nu_if - cut - f0) / df);
                    const double re = round((nu_if + cut - f0) / df);
                    lo = clamp_index(rb > double(s) ? rb : double(s), s, e);
                    hi = clamp_index(re < double(e) ? re : double(e), s, e);
                }
            }
        }
#pragma unroll 1
        for (int k = 0; k < C; ++k) {
            const int c = cg * C + k;
            const CondDev& Cd = a.cond[c];
            int kcl = 0, rch = 0;
            if (live) {
                double S, pw, g;
                if (ncache) {
                    const int t = a.tclass[c];
                    S = cS[t * 256 + tid];
                    pw = cP[t * 256 + tid];
                    g = cG[t * 256 + tid];
                } else {
                    class_values(Cd, S, pw, g);
                }
                const double gl = gam * Cd.gamma_scale * pw;
                const double y = gl * g;
                const double pref = (CONV == kConvCpu && S == 0.0) ? 0.0 : S * g;
                const double y2 = y * y;
                const double Pc = pref * kW4C * y;
                const double xw = (cut_prev + double(a.mixed_tile_span + 4) * df) * g;
                const bool whole = far_m || !(xw < kWholeXMax);
                // the shared reciprocals need the products in range
                wide = wide || !(xw * xw + y2 < kPairUMax) || !(fabs(Pc) < kPairPcMax);
                far = far || whole || !(xw * xw + y2 < kSoloUMax) || !(fabs(Pc) < kSoloPcMax);
                CoreIv iv;
                const double q = nu_df * Cd.dpw;
                region_interval_q(nu_p, g, y, 15.0, lo, hi, f0, df, md, q, tb, iv.lo15, iv.hi15);
                region_interval_q(nu_p, g, y, 5.5, lo, hi, f0, df, md, q, tb, iv.lo55, iv.hi55);
                if (iv.lo15 <= iv.hi15) {
                    // in integers where m is one (|m| < 1.6e7, grid indices
                    // below 1.5e7: no overflow)
                    bool over;
                    if (far_m) {
                        const double w = fmax(m - double(iv.lo15), double(iv.hi15) - m);
                        over = !(w < 3.0e7);
                        rch = over ? 30000000 : int(w);
                    } else {
                        rch = max(im - iv.lo15, iv.hi15 - im);
                        over = rch >= 30000000;
                        if (over) rch = 30000000;
                    }
                    if (over) atomicOr(a.err, kErrReach);  // the core pass would not find it
                    // |md - j| < sqrt(kNearR2 - y^2) q, |md - m| <= 1/2, one
                    // point of margin, plus one (0: none)
                    // (in FP32, widened by 1e-6 for its rounding)
                    if (y2 < kNearR2)
                        kcl = int(fminf(ceilf(sqrtf(float(kNearR2 - y2)) * float(q) * 1.000001f + 0.5f), 3.0e7f)) + 2;
                }
                if (whole) kcl = 30000000;  // a core candidate of every tile
                const size_t ci = size_t(c) * size_t(a.L.n) + size_t(i);
                a.civ[ci] = iv;
                a.cyp[ci] = make_float2(float(y), float(pref * kW4C));
            }
            kcl = __reduce_max_sync(0xffffffffu, kcl);
            rch = __reduce_max_sync(0xffffffffu, rch);
            if (lane == 0) {
                smax[0][c][warp] = kcl;
                smax[1][c][warp] = rch;
            }
        }
    }
    flush_window();
    // block maxima of the core-candidate widths (kc) and of the core pass's
    // reach (kc + kMaxCond), one atomic each per block and condition
    __syncthreads();
    for (int idx = tid; idx < 2 * a.ncond; idx += 256) {
        const int which = idx / a.ncond, c = idx - which * a.ncond;
        int mx = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) mx = smax[which][c][w] > mx ? smax[which][c][w] : mx;
        if (mx > 0) atomicMax(a.kc + (which ? kMaxCond : 0) + c, mx);
    }
}

// ---------------------------------------------------------------------------
// Step two helpers.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// First i in [lo, hi) with pred(i) true (pred monotone), or hi; 32-way
// ballot search by one warp.  Lanes 0..30 probe the ends of 31 segments of
// `step` indices; lane 31 stands for the rest of the range and is taken as
// true, so the ballot is never empty inside the loop.
template <class Pred>
__device__ long warp_lower_bound(long lo, long hi, int lane, Pred pred) {
    while (hi - lo > 32) {
        const long step = (hi - lo + 31) / 32;
        const long q = lo + long(lane + 1) * step - 1;
        const bool v = (lane < 31 && q < hi) ? pred(q) : true;
        const unsigned b = __ballot_sync(0xffffffffu, v);
        const int f = __ffs(b) - 1;
        const long nlo = lo + long(f) * step;
        if (f < 31) {
            const long qf = lo + long(f + 1) * step - 1;
            hi = qf < hi ? qf : hi;
        }
        lo = nlo;
    }
    const long q = lo + lane;
    const bool v = (q < hi) ? pred(q) : true;
    const unsigned b = __ballot_sync(0xffffffffu, v);
    if (b == 0u) return hi;
    const long r = lo + (__ffs(b) - 1);
    return r < hi ? r : hi;
}

// First i in [lo, hi) with v[i] >= key (v ascending), or hi.  One copy of the
// search for the kernels whose code has to stay small.
__device__ __noinline__ int warp_search(const int* v, int lo, int hi, int key, int lane) {
    return int(warp_lower_bound(lo, hi, lane, [&](long i) { return v[i] >= key; }));
}

// Copy `cnt` records of REC (sizeof a multiple of 16) into shared memory,
// 16 bytes per lane per step.
template <class REC>
__device__ __forceinline__ void stage(REC* dst, const REC* src, int cnt, int lane) {
    constexpr int kChunks = sizeof(REC) / 16;
    const int total = cnt * kChunks;
    const char* s = reinterpret_cast<const char*>(src);
    char* d = reinterpret_cast<char*>(dst);
    for (int q = lane; q < total; q += 32) cp_async16(d + 16 * q, s + 16 * q);
}

// The same for the first BYTES of records STRIDE bytes apart.
template <int BYTES, int STRIDE>
__device__ __forceinline__ void stage_rec(void* dst, const void* src, int cnt, int lane) {
    constexpr int kChunks = BYTES / 16;
    const char* s = static_cast<const char*>(src);
    char* d = static_cast<char*>(dst);
    for (int q = lane; q < cnt * kChunks; q += 32)
        cp_async16(d + 16 * q, s + (BYTES == STRIDE ? 16 * q : (q / kChunks) * STRIDE + (q % kChunks) * 16));
}

struct WorkItem {
    int c, t0, t1, s;
};

// Items are (condition, tile, split), splits innermost: the parts of one
// tile run side by side and share its records in L2.
__device__ __forceinline__ bool next_item(const StepArgs& a, int P, int lane, WorkItem& w) {
    int item = 0;
    if (lane == 0) item = int(atomicAdd(a.counter, 1u));
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= a.n_items) return false;
    const int per_cond = a.tiles_per_cond * a.splits;
    w.c = item / per_cond;
    const int rem = item - w.c * per_cond;
    const int tile = rem / a.splits;
    w.s = rem - tile * a.splits;
    w.t0 = a.G.start + tile * 32 * P;
    const int end = a.G.start + a.G.points;
    w.t1 = w.t0 + 32 * P < end ? w.t0 + 32 * P : end;
    return true;
}

// Split s of `splits` takes the 32-line groups s, s + splits, s + 2 splits,
// ... of the tile's lines [La, Lb): interleaved, so that the costly lines
// near the tile (cores) are shared evenly between the splits.
__device__ __forceinline__ int split_groups(long nl, int splits, int s) {
    const int all = int((nl + 31) / 32);
    return all > s ? (all - s + splits - 1) / splits : 0;
}

// Where item (c, s) puts the sum of grid point j: added to out, or stored to
// its part when the tile is split.
__device__ __forceinline__ void put_result(const StepArgs& a, int c, int s, int j, double v) {
    if (a.splits <= 1)
        a.out[size_t(a.row[c]) * a.out_stride + size_t(j)] += v;
    else
        a.part[(size_t(c) * a.splits + s) * a.part_stride + size_t(j - a.G.start)] = v;
}

// ---------------------------------------------------------------------------
// Cells: which of a tile's lines are taken through their cells' moments.
// ---------------------------------------------------------------------------
// A tile's lines [La, Lb) as three runs taken line by line -- [La, r1),
// [b2, e2), [b3, Lb) -- and two runs of cells [fa, fb), [fc, fd) taken by their
// moments.  Without usable cells the first run is all of [La, Lb).
struct LineRuns {
    long La, r1, b2, e2, b3, Lb;
    int fa, fb, fc, fd;
    int g1, g2, total;  // 32-line groups of the first and the second run, of all three

    // First line of the idx-th 32-line group, and the end of its run.
    __device__ __forceinline__ long start(int idx, long& end) const {
        if (idx < g1) {
            end = r1;
            return La + 32L * idx;
        }
        if (idx < g1 + g2) {
            end = e2;
            return b2 + 32L * (idx - g1);
        }
        end = Lb;
        return b3 + 32L * (idx - g1 - g2);
    }
    // Groups of split s of S: s, s + S, s + 2 S, ...
    __device__ __forceinline__ int groups_of(int S, int s) const { return total > s ? (total - s + S - 1) / S : 0; }
};

// [fs, fe): the lines whose windows cover the tile, whose grid points lie in
// [ftlo, fthi] cm-1.  The cells inside it are taken by their moments from each
// end up to the first one that is too near the tile; the cells in between are
// taken line by line.
__device__ __forceinline__ LineRuns line_runs(const CellHead* H, int ncell, int shift, long n, long La, long Lb,
                                              long fs, long fe, double ftlo, double fthi, int lane) {
    LineRuns r;
    r.La = La;
    r.Lb = Lb;
    r.r1 = r.b2 = r.e2 = r.b3 = Lb;
    r.fa = r.fb = r.fc = r.fd = 0;
    if (ncell > 0) {
        const int ca = int((fs + (1L << shift) - 1) >> shift);
        const int cb = fe >= n ? ncell : int(fe >> shift);
        if (ca < cb) {
            auto near = [&](int ci) {
                const CellHead h = H[ci];
                return !(fmax(ftlo - h.c0, h.c0 - fthi) >= double(h.dmin));
            };
            int nl = cb, nr;
            for (int b = ca; b < cb; b += 32) {
                const unsigned m = __ballot_sync(0xffffffffu, b + lane < cb && near(b + lane));
                if (m) {
                    nl = b + __ffs(m) - 1;
                    break;
                }
            }
            nr = nl;
            for (int e = cb; e > nl; e -= 32) {
                const unsigned m = __ballot_sync(0xffffffffu, e - 1 - lane >= nl && near(e - 1 - lane));
                if (m) {
                    nr = e - (__ffs(m) - 1);
                    break;
                }
            }
            auto line_of = [&](int c) { return c >= ncell ? n : long(c) << shift; };
            r.fa = ca;
            r.fb = nl;
            r.fc = nr;
            r.fd = cb;
            r.r1 = line_of(ca);
            r.b2 = line_of(nl);
            r.e2 = line_of(nr);
            r.b3 = line_of(cb);
        }
    }
    r.g1 = int((r.r1 - r.La + 31) / 32);
    r.g2 = int((r.e2 - r.b2 + 31) / 32);
    r.total = r.g1 + r.g2 + int((r.Lb - r.b3 + 31) / 32);
    return r;
}

// Terms evaluated of a cell at the tile's least distance from it: enough for
// (p + 1) r^p to lie below 2^-bits.  Even, so that moments load in pairs.
template <int PM>
__device__ __forceinline__ int cell_terms(float bits, double dist, float q) {
    const int p = int(__fdividef(bits, __log2f(float(dist) / q))) + 3;
    return p >= PM ? PM : (p & ~1);
}

// 1/x to FP64 rounding: the hardware approximation and two Newton-Raphson
// steps (r <- r + r (1 - x r)).
__device__ __forceinline__ double rcp_newton2_f64(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = fma(r, fma(-x, r, 1.0), r);
    return fma(r, fma(-x, r, 1.0), r);
}

// Adds the far cells of split s of S to the sum v of this lane's point f (one
// condition).  The heads of 32 cells are read at once, a cell per lane, and handed
// round; two cells are summed side by side, so that the latency of their moments'
// loads and of the chain is shared (one head and one chain at a time: 7.1 ms of
// step two for the FP64 single point, 5.1 so).  The SUB neighbouring lanes of a
// point take every SUB-th cell each (sub = this lane's); their sums are left apart.
template <int PM, int SUB>
__device__ __forceinline__ void add_far_cells(const CellHead* H, const double* M, const LineRuns& r, int S, int s,
                                              float bits, double ftlo, double fthi, double f, double& v, int lane,
                                              int sub) {
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const int c1 = h ? r.fd : r.fb;
#pragma unroll 1
        for (int b = (h ? r.fc : r.fa) + s; b < c1; b += 32 * S) {
            const int cnt = min(32, (c1 - b + S - 1) / S);
            const CellHead hd = H[min(b + lane * S, c1 - 1)];
            const int terms = cell_terms<PM>(bits, fmax(ftlo - hd.c0, hd.c0 - fthi), hd.q);
#pragma unroll 1
            for (int k = 0; k < cnt; k += 2 * SUB) {
                double t[2], a[2] = {0.0, 0.0};
                const double2* m[2];
                int np = 0;
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const int kk = k + w * SUB + sub;
                    const bool ok = kk < cnt;
                    const int at = ok ? kk : cnt - 1;
                    const double cc = __shfl_sync(0xffffffffu, hd.c0, at);
                    const float q = __shfl_sync(0xffffffffu, hd.q, at);
                    np = max(np, __shfl_sync(0xffffffffu, terms, at));
                    m[w] = reinterpret_cast<const double2*>(M + size_t(b + at * S) * PM);
                    t[w] = ok ? double(q) * rcp_newton2_f64(f - cc) : 0.0;  // (past the end: adds 0)
                }
                if constexpr (SUB > 1) np = __reduce_max_sync(0xffffffffu, np);
#pragma unroll 2
                for (int i = np / 2 - 1; i >= 0; --i) {
                    const double2 m0 = __ldg(m[0] + i), m1 = __ldg(m[1] + i);
                    a[0] = fma(fma(a[0], t[0], m0.y), t[0], m0.x);
                    a[1] = fma(fma(a[1], t[1], m1.y), t[1], m1.x);
                }
                v = fma(a[0] * t[0], t[0], v);
                v = fma(a[1] * t[1], t[1], v);
            }
        }
    }
}

// The same for one point and N of the C conditions of a group (M: at the first of
// them).
template <int C, int N, int PM, int LS = 1>
__device__ __forceinline__ void add_far_cells_mc(const CellHead* H, const double* M, const LineRuns& r, int S, int s,
                                                 float bits, double ftlo, double fthi, double f, double (&v)[N],
                                                 int lane, int sub = 0) {
    constexpr int W = N <= 4 ? 2 : 1;  // cells side by side
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const int c1 = h ? r.fd : r.fb;
#pragma unroll 1
        for (int b = (h ? r.fc : r.fa) + s; b < c1; b += 32 * S) {
            const int cnt = min(32, (c1 - b + S - 1) / S);
            const CellHead hd = H[min(b + lane * S, c1 - 1)];
            const int terms = cell_terms<PM>(bits, fmax(ftlo - hd.c0, hd.c0 - fthi), hd.q);
#pragma unroll 1
            for (int k = 0; k < cnt; k += W * LS) {
                double t[W], a[W][N];
                const double* m[W];
                int np = 0;
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    const int kk = k + w * LS + sub;
                    const bool ok = kk < cnt;
                    const int at = ok ? kk : cnt - 1;
                    const double cc = __shfl_sync(0xffffffffu, hd.c0, at);
                    const float q = __shfl_sync(0xffffffffu, hd.q, at);
                    np = max(np, __shfl_sync(0xffffffffu, terms, at));
                    m[w] = M + size_t(b + at * S) * (PM * C);
                    t[w] = ok ? double(q) * rcp_newton2_f64(f - cc) : 0.0;  // (past the end: adds 0)
#pragma unroll
                    for (int q2 = 0; q2 < N; ++q2) a[w][q2] = 0.0;
                }
                if constexpr (LS > 1) np = __reduce_max_sync(0xffffffffu, np);
#pragma unroll 2
                for (int i = np - 1; i >= 0; --i) {
#pragma unroll
                    for (int w = 0; w < W; ++w) {
                        if constexpr (N % 2 == 0) {
#pragma unroll
                            for (int q = 0; q < N; q += 2) {
                                const double2 mk = __ldg(reinterpret_cast<const double2*>(m[w] + i * C + q));
                                a[w][q] = fma(a[w][q], t[w], mk.x);
                                a[w][q + 1] = fma(a[w][q + 1], t[w], mk.y);
                            }
                        } else {
                            a[w][0] = fma(a[w][0], t[w], __ldg(m[w] + i * C));
                        }
                    }
                }
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    const double t2 = t[w] * t[w];
#pragma unroll
                    for (int q = 0; q < N; ++q) v[q] = fma(a[w][q], t2, v[q]);
                }
            }
        }
    }
}

// Sum of v over the warp's LS lane subsets, to every lane.
template <int LS>
__device__ __forceinline__ double sum_subsets(double v) {
#pragma unroll
    for (int o = 32 / LS; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------
// Step two, Voigt.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float rcp_approx_f32(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// 1/x: the hardware approximation refined by one Newton-Raphson step
// (r <- r + r (1 - x r)), which squares its relative error.
__device__ __forceinline__ double rcp_refined_f64(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, e, r);
}

struct fcplx {
    float re, im;
};

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 f2s(float a) { return make_float2(a, a); }
__device__ __forceinline__ fcplx operator+(float a, fcplx b) { return {a + b.re, b.im}; }
__device__ __forceinline__ fcplx operator*(fcplx a, fcplx b) {
    return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}

// a / b for the FP32 W4 forms of regions II and III (no cancellation
// follows there): the hardware reciprocal and one product, within 2 ulp; the
// denominators lie between about 0.5 and 1e6, far from the range where the
// approximation fails.  Region IV, which subtracts, keeps the IEEE division.
__device__ __forceinline__ float region_div(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double region_div(double a, double b) { return a * rcp_newton2_f64(b); }

// W4 region II (5.5 <= |x| + y < 15): T (a + b U) / (c + U (3 + U)), T = y - ix,
// U = T^2, a = 1.410474, b = .5641896, c = .75.  Its denominator has the roots
// U = -(3 -+ sqrt 6) / 2 = -B1, -B2, so it is T [A1 / (U + B1) + A2 / (U + B2)]
// with A1 + A2 = b, A1 B2 + A2 B1 = a, and as Re[T / (U + B)] =
// y (v + B) / ((v - B)^2 + 4 B y^2), v = x^2 + y^2 (region I is the same with
// B = 1/2), its real part is a sum of positive terms: no cancellation, and half
// the operations of the complex form's real part.
constexpr double kW4Root6 = 2.44948974278317809820;
constexpr double kW4B1 = 0.5 * (3.0 - kW4Root6), kW4B2 = 0.5 * (3.0 + kW4Root6);
constexpr double kW4A1 = (1.410474 - .5641896 * kW4B1) / kW4Root6;
constexpr double kW4A2 = (.5641896 * kW4B2 - 1.410474) / kW4Root6;
// Per unit c = kW4C, from u = x^2 + y^2 - 1/2 = v - 1/2: in FP32 this order and
// these constants leave an rms error of 0.9e-7 and a mean of 4e-9 over the
// region (the complex form's real part: 1.8e-7 and 3e-8).
template <class R>
__device__ __forceinline__ R w4_region2_c(R x, R y) {
    const R y2 = y * y, u = x * x + (y2 - R(0.5));
    const R e1 = u + R(0.5 - kW4B1), e2 = u + R(0.5 - kW4B2);
    const R d1 = e1 * e1 + R(2) * y2 * R(2.0 * kW4B1), d2 = e2 * e2 + R(2) * y2 * R(2.0 * kW4B2);
    const R p1 = y * R(kW4A1 / kW4C), p2 = y * R(kW4A2 / kW4C);
    const R n1 = u * p1 + p1 * R(0.5 + kW4B1), n2 = u * p2 + p2 * R(0.5 + kW4B2);
    return region_div(n1 * d2 + n2 * d1, d1 * d2);
}
template <class R>
__device__ __forceinline__ R w4_region2_re(R x, R y) {
    return R(kW4C) * w4_region2_c(x, y);
}
// The same for one line at several points: what depends on y alone, times f.
struct Region2F64 {
    double d1, d2, p1, p2, q1, q2;
    __device__ __forceinline__ Region2F64(double y, double f) {
        const double y2 = y * y;
        d1 = y2 * (4.0 * kW4B1);
        d2 = y2 * (4.0 * kW4B2);
        p1 = y * (f * kW4A1);
        p2 = y * (f * kW4A2);
        q1 = p1 * (0.5 + kW4B1);
        q2 = p2 * (0.5 + kW4B2);
    }
    // u = x^2 + y^2 - 1/2
    __device__ __forceinline__ double operator()(double u) const {
        const double e1 = u + (0.5 - kW4B1), e2 = u + (0.5 - kW4B2);
        const double g1 = fma(e1, e1, d1), g2 = fma(e2, e2, d2);
        return fma(fma(u, p1, q1), g2, fma(u, p2, q2) * g1) * rcp_newton2_f64(g1 * g2);
    }
};

// The region-I rational of W4 in FP32 per unit c pref, as step two evaluates
// it: y (u + 1) / (u^2 + 2 y^2), u = x^2 + y^2 - 0.5.  The core pass
// takes it back off the pairs where step two added it.
__device__ __forceinline__ float w4_region1_c(float x, float y) {
    const float y2 = y * y;
    const float u = fmaf(x, x, y2 - 0.5f);
    return region_div(y * (u + 1.0f), fmaf(u, u, 2.0f * y2));
}

// W4 region III in FP32 (there y >= 0.195|x| - 0.176, so Re w is not small
// next to |w| and the complex form keeps its accuracy).
__device__ __forceinline__ float w4_region3_re_f32(float x, float y) {
    const fcplx t = {y, -x};
    const fcplx num = 16.4955f + t * (20.20933f + t * (11.96482f + t * (3.778987f + t * fcplx{.5642236f, 0.f})));
    const fcplx den = 16.4955f + t * (38.82363f + t * (39.27121f + t * (21.69274f + t * (6.699398f + t))));
    return region_div(num.re * den.re + num.im * den.im, den.re * den.re + den.im * den.im);
}

// a - u p for the region IV Horner schemes.
__device__ __forceinline__ fcplx fms(float a, fcplx u, fcplx p) {
    return {a - (u.re * p.re - u.im * p.im), -(u.re * p.im + u.im * p.re)};
}

// W4 region IV in FP32: Re[exp(U) - T P(U) / Q(U)], U = T^2, with
// exp(U) = exp(y^2 - x^2) (cos 2xy + i ...).  Over the region (|x| + y < 5.5,
// y < 0.195|x| - 0.176) this stays within 7e-6 of the FP64 evaluation at the
// same FP32 x, y (sampled densely with y down to 1e-9).
__device__ float w4_region4_re_f32(float x, float y) {
    const float e = expf(fmaf(y, y, -x * x)) * cosf(2.0f * x * y);
    const fcplx t = {y, -x};
    const fcplx u = t * t;
    fcplx num = fms(1.320522f, u, fcplx{.56419f, 0.f});
    num = fms(35.76683f, u, num);
    num = fms(219.0313f, u, num);
    num = fms(1540.787f, u, num);
    num = fms(3321.9905f, u, num);
    num = fms(36183.31f, u, num);
    fcplx den = fms(1.841439f, u, fcplx{1.f, 0.f});
    den = fms(61.57037f, u, den);
    den = fms(364.2191f, u, den);
    den = fms(2186.181f, u, den);
    den = fms(9022.228f, u, den);
    den = fms(24322.84f, u, den);
    den = fms(32066.6f, u, den);
    const fcplx r = t * num;
    return e - (r.re * den.re + r.im * den.im) / (den.re * den.re + den.im * den.im);
}

// Persistent step two.  For a tile [t0, t1) the lines [La, Lb) meet it;
// since the window bounds lo[] and hi[] are ascending in line order, the
// lines covering the whole tile form one contiguous run [fs, fe), and among
// those the ones whose core may reach the tile ([E, F), from the ascending
// nearest-grid-index array mi[] and the condition's widest core kc) form
// another.  So every staged group splits into at most five contiguous runs:
//   partial [La, fs) | fast [fs, E) | core [E, F) | fast [F, fe) | partial [fe, Lb)
// Fast lines evaluate W4 region I on every pair with no test at all.  Core
// and partial lines classify whole rows (outside the window: skipped; inside
// and clear of the core band: as fast; otherwise lane by lane).  Pairs of W4
// regions II-IV are left out there: the FP64 kernels take them in a pass of
// their own after the tile's lines (core_row_f64, lane = line), the mixed ones
// in separate kernels.

// W4 regions III and IV in FP64, real parts; complex Horner schemes (T = y - ix).
__device__ __forceinline__ double w4_region3_re_f64(double x, double y) {
    const cplx t = {y, -x};
    const cplx num = 16.4955 + t * (20.20933 + t * (11.96482 + t * (3.778987 + t * .5642236)));
    const cplx den = 16.4955 + t * (38.82363 + t * (39.27121 + t * (21.69274 + t * (6.699398 + t))));
    return (num.re * den.re + num.im * den.im) * rcp_newton2_f64(den.re * den.re + den.im * den.im);
}
__device__ __forceinline__ double w4_region4_re_f64(double x, double y) {
    const cplx t = {y, -x};
    const cplx u = t * t;
    const cplx num = t * (36183.31 - u * (3321.9905 - u * (1540.787 - u * (219.0313 -
                          u * (35.76683 - u * (1.320522 - u * .56419))))));
    const cplx den = 32066.6 - u * (24322.84 - u * (9022.228 - u * (2186.181 -
                          u * (364.2191 - u * (61.57037 - u * (1.841439 - u))))));
    return exp(u.re) * cos(u.im) -
           (num.re * den.re + num.im * den.im) * rcp_newton2_f64(den.re * den.re + den.im * den.im);
}

// Per-warp table of the FP64 core pass: [point of the row][lane].
constexpr int kCoreRow64 = 33;
constexpr size_t kCoreTable64 = sizeof(double) * 32 * kCoreRow64;

// W4 regions II-IV of the FP64 path on one row of 32 grid points [r0, r0 + 32):
// the lines [E, Fc) are taken 32 at a time (batches s, s + S, ...), lane = line,
// each lane going over its line's points jlo..jhi (core band and window, from
// `get`) and adding to its own column of the table T; the columns are added up
// in lane order at the end, so the order of every sum is fixed.  Region II and
// regions III-IV run in loops of their own: neighbouring lines have nearly the
// same intervals, so a warp step runs one region's code on most of its lanes.
// x, y and the region choice are the reference's.  Returns this lane's point's
// sum.
//
// Rows with at most kFewCore candidates (sparse lists) go lane = point.
// Before, the pairs went through a shared-memory queue, 32 at a time over all
// regions, between step two's lines.
constexpr long kFewCore = 3;
template <class Get>
__device__ __forceinline__ double core_row_f64(double (*T)[kCoreRow64], const double* F, long E, long Fc, int r0,
                                               int S, int s, int lane, Get get) {
    // Few candidate lines (sparse lists, small calls): 2 or 4 lanes to a line,
    // on every second or fourth point, so that one batch's chain is shorter.
    if (Fc - E <= kFewCore) {
        // one to a few lines: lane = point, without the table
        double v = 0.0;
        for (long i = E; i < Fc && s == 0; ++i) {
            double nu = 0.0, g = 0.0, y = 0.0, pref = 0.0;
            int jlo = 1, jhi = 0;
            get(i, nu, g, y, pref, jlo, jhi);
            const int j = r0 + lane;
            if (jlo > jhi || j < jlo || j > jhi) continue;
            const double ax = fabs((nu - F[j]) * g), sx = ax + y;
            if (sx >= 15.0) continue;
            v += pref * (sx >= 5.5 ? w4_region2_re<double>(ax, y)
                         : y >= 0.195 * ax - 0.176 ? w4_region3_re_f64(ax, y) : w4_region4_re_f64(ax, y));
        }
        __syncwarp();
        return v;
    }
    const int sh = Fc - E <= 8L * S ? 2 : (Fc - E <= 16L * S ? 1 : 0);
    const int nb = 32 >> sh, sub = lane & ((1 << sh) - 1), step = 1 << sh;
    if (E + long(nb) * s >= Fc) return 0.0;
#pragma unroll 4
    for (int q = 0; q < 32; ++q) T[q][lane] = 0.0;
    bool any = false;
    for (long b = E + long(nb) * s; b < Fc; b += long(nb) * S) {
        const long i = b + (lane >> sh);
        double nu = 0.0, g = 0.0, y = 0.0, pref = 0.0;
        int jlo = 1, jhi = 0;
        if (i < Fc) get(i, nu, g, y, pref, jlo, jhi);
        int b0 = INT_MAX, b1 = -1;
        for (int j = jlo + sub; j <= jhi; j += step) {
            const double ax = fabs((nu - F[j]) * g);
            const double sx = ax + y;
            if (sx >= 15.0) continue;
            any = true;
            if (sx >= 5.5) {
                T[j - r0][lane] += pref * w4_region2_re<double>(ax, y);
            } else {
                b0 = min(b0, j);
                b1 = j;
            }
        }
        for (int j = b0; j <= b1; j += step) {
            const double ax = fabs((nu - F[j]) * g);
            const double w = y >= 0.195 * ax - 0.176 ? w4_region3_re_f64(ax, y) : w4_region4_re_f64(ax, y);
            T[j - r0][lane] += pref * w;
        }
    }
    any = __any_sync(0xffffffffu, any);
    __syncwarp();
    if (!any) return 0.0;
    double sum = 0.0;
#pragma unroll 8
    for (int q = 0; q < 32; ++q) sum += T[lane][q];
    __syncwarp();
    return sum;
}

// Resident blocks per SM the step-two Voigt kernel asks the compiler to fit
// (register budget), FP32 path at 4 warps per block: 28 warps per SM at 4
// points per thread (72 registers), 32 at 1 or 2 (64 registers; 8 blocks of
// 24.6 KB of staging fit in shared memory); 24 for its other shapes up to 4
// points per thread.
template <int P, int WARPS, bool MIXED>
constexpr int voigt_min_blocks() {
    return (MIXED && P == 4 && WARPS == 4) ? 7 : (MIXED && P <= 2 && WARPS == 4) ? 8 : (MIXED && P <= 4) ? 24 / WARPS : 1;
}

// Shared memory of one warp of it.
constexpr size_t voigt_warp_smem(bool mixed) {
    const size_t staged = size_t(32) * kStages * (mixed ? sizeof(RecV32) : size_t(kRecV64Staged));
    return mixed || staged > kCoreTable64 ? staged : kCoreTable64;
}

template <int P, int WARPS, bool MIXED>
__global__ void __launch_bounds__(WARPS * 32, (voigt_min_blocks<P, WARPS, MIXED>()))
    k_steptwo_voigt(StepArgs a) {
    using REC = typename std::conditional<MIXED, RecV32, RecV64>::type;
    using T = typename std::conditional<MIXED, float, double>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    // staged records, kStages groups of 32; the FP64 core pass's table takes
    // the same space after the tile's lines
    constexpr int kRec = MIXED ? int(sizeof(REC)) : kRecV64Staged;
    unsigned char* const mine = smem_raw + size_t(warp) * voigt_warp_smem(MIXED);
    const REC* recs_all = reinterpret_cast<const REC*>(a.rec);
    const double* F = a.G.freq;

    WorkItem w;
    while (next_item(a, P, lane, w)) {
        const size_t cbase = size_t(w.c) * size_t(a.n);
        const int* whi = a.whi + cbase;
        const int* wlo = a.wlo + cbase;
        const int* mi = a.mi;
        const int kc = a.kc[w.c];
        const int t0 = w.t0, t1 = w.t1, tl = t1 - 1;
        const long La = warp_lower_bound(0, a.n, lane, [&](long i) { return whi[i] > t0; });
        const long Lb = warp_lower_bound(La, a.n, lane, [&](long i) { return wlo[i] >= t1; });
        const long fs = warp_lower_bound(La, Lb, lane, [&](long i) { return whi[i] >= t1; });
        const long Cb = warp_lower_bound(La, Lb, lane, [&](long i) { return wlo[i] > t0; });
        const long fe = Cb > fs ? Cb : fs;
        const long E = warp_lower_bound(fs, fe, lane, [&](long i) { return mi[i] >= t0 - kc; });
        const long Fc = warp_lower_bound(E, fe, lane, [&](long i) { return mi[i] > tl + kc; });
        const REC* recs = recs_all + cbase;
        int jj[P];
        float jf[P];
        double fj[P];
        float accf[P], sumf[P], cmpf[P];
        double accd[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            jj[p] = t0 + lane + 32 * p;
            jf[p] = float(jj[p]);
            fj[p] = MIXED ? 0.0 : F[jj[p] < t1 ? jj[p] : tl];
            accf[p] = sumf[p] = cmpf[p] = 0.0f;
            accd[p] = 0.0;
        }

        // Region I on every row: u = x^2 + Cy, acc += Pc (u + 1) / (u^2 + D2);
        // in FP32 two rows at a time as packed FP32x2 operations.
        auto fast_line = [&](const unsigned char* r) {
            if (MIXED) {
                const float4* q = reinterpret_cast<const float4*>(r);
                const float4 v0 = q[0], v1 = q[1];
                if constexpr (P % 2 == 0) {
#pragma unroll
                    for (int p = 0; p < P; p += 2) {
                        const float2 d = __fadd2_rn(f2s(v0.x), f2(-jf[p], -jf[p + 1]));
                        const float2 xs = __ffma2_rn(d, f2s(v0.z), f2s(v0.y));
                        const float2 u = __ffma2_rn(xs, xs, f2s(v0.w));
                        const float2 den = __ffma2_rn(u, u, f2s(v1.x));
                        const float2 num = __ffma2_rn(u, f2s(v1.y), f2s(v1.y));
                        const float2 acc = __ffma2_rn(num, f2(rcp_approx_f32(den.x), rcp_approx_f32(den.y)),
                                                      f2(accf[p], accf[p + 1]));
                        accf[p] = acc.x;
                        accf[p + 1] = acc.y;
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < P; ++p) {
                        const float xs = fmaf(v0.x - jf[p], v0.z, v0.y);
                        const float u = fmaf(xs, xs, v0.w);
                        accf[p] = fmaf(fmaf(u, v1.y, v1.y), rcp_approx_f32(fmaf(u, u, v1.x)), accf[p]);
                    }
                }
            } else {
                const double2* q = reinterpret_cast<const double2*>(r);
                const double2 v0 = q[0], v1 = q[1], v2 = q[2];
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const double xs = (v0.x - fj[p]) * v0.y;
                    const double u = fma(xs, xs, v1.x);
                    accd[p] = fma(fma(u, v2.x, v2.x), rcp_refined_f64(fma(u, u, v1.y)), accd[p]);
                }
            }
        };
        // Whole lines: Pc / u to FP32 rounding from u = 1e12 on; u^2 overflows from
        // 1.8e19 and Pc u may, and infinity times 0 is NaN.
        auto whole_far = [](bool whole, float u, float Pc, float& num, float& den) {
            if (whole && u > 1.0e12f) num = Pc, den = u;
        };
        // `full`: the line's window covers the whole tile.
        auto slow_line = [&](const unsigned char* r, bool full) {
            if (MIXED) {
                // region I except the pairs of the region interval [clo, chi]
                // (the core pass takes those)
                const float4* q = reinterpret_cast<const float4*>(r);
                const float4 v0 = q[0], v1 = q[1], v2 = q[2];
                const float m = v0.x, ra = v0.y, dfa = v0.z, Cy = v0.w;
                const float D2 = v1.x, Pc = v1.y;
                const float lo = v2.x, hi = v2.y, clo = v2.z, chi = v2.w;
                const bool whole = dfa < 0.0f;
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const float r0 = float(t0 + 32 * p), r1 = r0 + 31.0f;
                    if (!full && (r0 >= hi || r1 < lo)) continue;
                    const bool row_in = full || (r0 >= lo && r1 < hi);
                    const bool row_core = whole || !(r1 < clo || r0 > chi);
                    const float xs = whole ? float((reinterpret_cast<const RecV32*>(r)->nu - F[jj[p] < t1 ? jj[p] : tl]) / reinterpret_cast<const RecV32*>(r)->nu) * a.kx[w.c]
                                           : fmaf(m - jf[p], dfa, ra);
                    const float u = fmaf(xs, xs, Cy);
                    float num = fmaf(u, Pc, Pc), den = fmaf(u, u, D2);
                    whole_far(whole, u, Pc, num, den);
                    const float rr = rcp_approx_f32(den);
                    if (row_in && !row_core) {
                        accf[p] = fmaf(num, rr, accf[p]);
                        continue;
                    }
                    const bool in = row_in || (jf[p] >= lo && jf[p] < hi);
                    const bool core = jf[p] >= clo && jf[p] <= chi;
                    // beyond x ~ 1e18 (whole lines only) region I is taken as 0
                    const bool keep = in && !core && fabsf(xs) < 1.0e18f;
                    accf[p] += keep ? num * rr : 0.0f;
                }
            } else {
                const double2* q = reinterpret_cast<const double2*>(r);
                const double2 v0 = q[0], v1 = q[1], v2 = q[2];
                const int4 vi = reinterpret_cast<const int4*>(r)[3];
                const double nu = v0.x, g = v0.y, Cy = v1.x, D2 = v1.y, Pc = v2.x, y = v2.y;
                const int lo = vi.x, hi = vi.y, clo = vi.z, chi = vi.w;
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const int r0 = t0 + 32 * p, r1 = r0 + 31;
                    if (!full && (r0 >= hi || r1 < lo)) continue;
                    const bool row_in = full || (r0 >= lo && r1 < hi);
                    const bool row_core = !(r1 < clo || r0 > chi);
                    const double xs = (nu - fj[p]) * g;
                    if (row_in && !row_core) {
                        const double u = fma(xs, xs, Cy);
                        accd[p] = fma(fma(u, Pc, Pc), rcp_refined_f64(fma(u, u, D2)), accd[p]);
                        continue;
                    }
                    const bool in = row_in || (jj[p] >= lo && jj[p] < hi);
                    // x and y are bit-identical to the reference's, so the
                    // region choice below is the reference's.
                    const double ax = fabs(xs);
                    const bool exact = row_core && jj[p] >= clo && jj[p] <= chi && !(ax + y >= 15.0);
                    if (in && !exact) {
                        const double u = fma(xs, xs, Cy);
                        accd[p] = fma(fma(u, Pc, Pc), rcp_refined_f64(fma(u, u, D2)), accd[p]);
                    }
                }
            }
        };

        // A line whose window covers only part of the tile and whose core
        // band misses it: rows outside the window are skipped, the boundary
        // row is masked lane by lane.
        auto partial_line = [&](const unsigned char* r) {
            if (MIXED) {
                const float4* q = reinterpret_cast<const float4*>(r);
                const float4 v0 = q[0], v1 = q[1], v2 = q[2];
                const float lo = v2.x, hi = v2.y;
                // region interval reaching the tile, or a whole line
                if (v0.z < 0.0f || !(v2.w < float(t0) || v2.z > float(tl))) {
                    slow_line(r, false);
                    return;
                }
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const float r0 = float(t0 + 32 * p), r1 = r0 + 31.0f;
                    if (r0 >= hi || r1 < lo) continue;
                    const float xs = fmaf(v0.x - jf[p], v0.z, v0.y);
                    const float u = fmaf(xs, xs, v0.w);
                    float rr = rcp_approx_f32(fmaf(u, u, v1.x));
                    if (!(r0 >= lo && r1 < hi)) rr = (jf[p] >= lo && jf[p] < hi) ? rr : 0.0f;
                    accf[p] = fmaf(fmaf(u, v1.y, v1.y), rr, accf[p]);
                }
            } else {
                const double2* q = reinterpret_cast<const double2*>(r);
                const double2 v0 = q[0], v1 = q[1], v2 = q[2];
                const int4 vi = reinterpret_cast<const int4*>(r)[3];
                const int lo = vi.x, hi = vi.y;
                if (!(vi.w < t0 || vi.z > tl)) {
                    slow_line(r, false);
                    return;
                }
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const int r0 = t0 + 32 * p, r1 = r0 + 31;
                    if (r0 >= hi || r1 < lo) continue;
                    const double xs = (v0.x - fj[p]) * v0.y;
                    const double u = fma(xs, xs, v1.x);
                    double rr = rcp_refined_f64(fma(u, u, v1.y));
                    if (!(r0 >= lo && r1 < hi)) rr = (jj[p] >= lo && jj[p] < hi) ? rr : 0.0;
                    accd[p] = fma(fma(u, v2.x, v2.x), rr, accd[p]);
                }
            }
        };
        // A line whose window covers the tile and whose core band may reach
        // it: region I on every row except the band's pairs outside region I.
        auto core_line = [&](const unsigned char* r) {
            if (MIXED) {
                const float4* q = reinterpret_cast<const float4*>(r);
                const float4 v0 = q[0], v1 = q[1], v2 = q[2];
                const float clo = v2.z, chi = v2.w;
                const bool whole = v0.z < 0.0f;
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const float r0 = float(t0 + 32 * p), r1 = r0 + 31.0f;
                    const float xs = whole ? float((reinterpret_cast<const RecV32*>(r)->nu - F[jj[p] < t1 ? jj[p] : tl]) / reinterpret_cast<const RecV32*>(r)->nu) * a.kx[w.c]
                                           : fmaf(v0.x - jf[p], v0.z, v0.y);
                    const float u = fmaf(xs, xs, v0.w);
                    float num = fmaf(u, v1.y, v1.y), den = fmaf(u, u, v1.x);
                    whole_far(whole, u, v1.y, num, den);
                    const float rr = rcp_approx_f32(den);
                    if (!whole && (r1 < clo || r0 > chi)) {
                        accf[p] = fmaf(num, rr, accf[p]);
                        continue;
                    }
                    // region I except the pairs of the region interval
                    const bool core = jf[p] >= clo && jf[p] <= chi;
                    const bool keep = !core && fabsf(xs) < 1.0e18f;
                    accf[p] += keep ? num * rr : 0.0f;
                }
            } else {
                const double2* q = reinterpret_cast<const double2*>(r);
                const double2 v0 = q[0], v1 = q[1], v2 = q[2];
                const int4 vi = reinterpret_cast<const int4*>(r)[3];
                const int clo = vi.z, chi = vi.w;
                const double y = v2.y;
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const int r0 = t0 + 32 * p, r1 = r0 + 31;
                    const double xs = (v0.x - fj[p]) * v0.y;
                    if (r1 < clo || r0 > chi) {
                        const double u = fma(xs, xs, v1.x);
                        accd[p] = fma(fma(u, v2.x, v2.x), rcp_refined_f64(fma(u, u, v1.y)), accd[p]);
                        continue;
                    }
                    const double ax = fabs(xs);
                    const bool exact = jj[p] >= clo && jj[p] <= chi && !(ax + y >= 15.0);
                    if (!exact) {
                        const double u = fma(xs, xs, v1.x);
                        accd[p] = fma(fma(u, v2.x, v2.x), rcp_refined_f64(fma(u, u, v1.y)), accd[p]);
                    }
                }
            }
        };

        // this item's groups of 32 lines: gi-th starts at La + 32 (s + gi S)
        const int ngroups = split_groups(Lb - La, a.splits, w.s);
        auto gstart = [&](int gi) { return La + 32L * (w.s + long(gi) * a.splits); };
        // kStages-deep cp.async pipeline: groups gi+1 .. gi+kStages-1 are in
        // flight while group gi is evaluated (one commit per step, empty
        // commits past the end keep the group count uniform).
        auto issue = [&](int g) {
            if (g < ngroups) {
                const long b = gstart(g);
                const long rem = Lb - b;
                stage_rec<kRec, int(sizeof(REC))>(mine + (g % kStages) * 32 * kRec, recs + b, int(rem < 32 ? rem : 32),
                                                  lane);
            }
            cp_async_commit();
        };
#pragma unroll
        for (int g = 0; g < kStages - 1; ++g) issue(g);
        for (int gi = 0; gi < ngroups; ++gi) {
            issue(gi + kStages - 1);
            cp_async_wait<kStages - 1>();
            __syncwarp();
            const unsigned char* R0 = mine + (gi % kStages) * 32 * kRec;
            auto R = [&](int t) { return R0 + t * kRec; };
            const long gb = gstart(gi);
            const long ge = Lb - gb < 32 ? Lb : gb + 32;
            auto lo_of = [&](long v) { return int((v < gb ? gb : (v > ge ? ge : v)) - gb); };
            const int a0 = lo_of(La), a1 = lo_of(fs);
            const int b1 = lo_of(E), c1 = lo_of(Fc), d1 = lo_of(fe), e1 = lo_of(Lb);
            // slow lines of the three slow runs, one loop: t in [a0, a1) and
            // [d1, e1) are partial, [b1, c1) cover the tile
            for (int t = a0; t < e1; ++t) {
                if (t == a1) t = b1;  // skip the first fast run
                if (t == c1) t = d1;  // skip the second fast run
                if (t >= e1) break;
                if (t >= b1 && t < c1) core_line(R(t));
                else partial_line(R(t));
            }
            {
                int t = a1;
                for (; t + 1 < b1; t += 2) {
                    fast_line(R(t));
                    fast_line(R(t + 1));
                }
                if (t < b1) fast_line(R(t));
                t = c1;
                for (; t + 1 < d1; t += 2) {
                    fast_line(R(t));
                    fast_line(R(t + 1));
                }
                if (t < d1) fast_line(R(t));
            }
            if (MIXED) {
                // compensated (Kahan) fold of this group's FP32 partials
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    const float part = accf[p];
                    const float yk = part - cmpf[p];
                    const float tk = sumf[p] + yk;
                    cmpf[p] = (tk - sumf[p]) - yk;
                    sumf[p] = tk;
                    accf[p] = 0.0f;
                }
            }
            __syncwarp();
        }
        cp_async_wait<0>();
        __syncwarp();
        double v[P];
#pragma unroll
        for (int p = 0; p < P; ++p) v[p] = MIXED ? double(sumf[p]) - double(cmpf[p]) : accd[p];
        if constexpr (!MIXED) {
            // W4 regions II-IV (one search for the tile, so that a tile without
            // candidates, the usual one of a sparse list, makes none per row)
            double (*T)[kCoreRow64] = reinterpret_cast<double (*)[kCoreRow64]>(mine);
            const long Ta = warp_lower_bound(La, Lb, lane, [&](long i) { return mi[i] >= t0 - kc; });
            const long Tb = warp_lower_bound(Ta, Lb, lane, [&](long i) { return mi[i] > tl + kc; });
            const int mt = Ta + lane < Tb ? mi[Ta + lane] : INT_MAX;
#pragma unroll 1
            for (int p = 0; p < P && Ta < Tb; ++p) {
                const int r0 = t0 + 32 * p, r1 = min(r0 + 32, t1) - 1;
                if (r0 > r1) break;
                long E0 = Ta, E1 = Tb;
                if (P > 1 && Tb - Ta <= 32) {
                    E0 = Ta + __popc(__ballot_sync(0xffffffffu, mt < r0 - kc));
                    E1 = Ta + __popc(__ballot_sync(0xffffffffu, mt <= r1 + kc));
                } else if (P > 1) {
                    E0 = warp_lower_bound(Ta, Tb, lane, [&](long i) { return mi[i] >= r0 - kc; });
                    E1 = warp_lower_bound(E0, Tb, lane, [&](long i) { return mi[i] > r1 + kc; });
                }
                const double add =
                    core_row_f64(T, F, E0, E1, r0, a.splits, w.s, lane,
                                 [&](long i, double& nu, double& g, double& y, double& pref, int& jlo, int& jhi) {
                                     const RecV64& r = recs[i];
                                     const int4 iv = *reinterpret_cast<const int4*>(&r.lo);
                                     nu = r.nu;
                                     g = r.g;
                                     y = r.y;
                                     pref = r.pref;
                                     jlo = max(max(iv.x, iv.z), r0);
                                     jhi = min(min(iv.y - 1, iv.w), r1);
                                 });
#pragma unroll
                for (int q = 0; q < P; ++q)
                    if (q == p) v[q] += add;
            }
        }
#pragma unroll
        for (int p = 0; p < P; ++p)
            if (jj[p] < t1) put_result(a, w.c, w.s, jj[p], v[p]);
    }
}

// Multi-condition step two, FP64: a work item is (group of C conditions that
// share one window, row of 32 / LS grid points); each lane owns one grid point,
// every LS-th line of the row's and C accumulators (LS = 4: 8-point rows for
// coarse grids over dense lists, where a 32-point row is much wider than the
// zone that has to be taken line by line).  The line runs are found as in k_steptwo_voigt (windows and
// grid indices are shared by the group; the core run uses the group's widest
// core), and every line loads its shared record once and one small record
// per condition.
template <int C, int WARPS, int LS>
__global__ void __launch_bounds__(WARPS * 32) k_steptwo_voigt_mc(StepArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    // two stages of 32 lines; the core pass's table takes the same space
    static_assert(64 * (sizeof(LineSh64) + 2 * sizeof(CondRec64)) >= kCoreTable64, "the table fits the stages");
    unsigned char* const mine = smem_raw + size_t(warp) * 64 * (sizeof(LineSh64) + C * sizeof(CondRec64));
    LineSh64* lsb = reinterpret_cast<LineSh64*>(mine);
    CondRec64* crb = reinterpret_cast<CondRec64*>(mine + 64 * sizeof(LineSh64));
    const double* F = a.G.freq;
    constexpr int PT = 32 / LS;  // points of a row
    const int sub = lane / PT;

    for (;;) {
        int item = 0;
        if (lane == 0) item = int(atomicAdd(a.counter, 1u));
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.n_items) break;
        const int per_cond = a.tiles_per_cond * a.splits;
        const int cg = item / per_cond;
        const int tile = (item - cg * per_cond) / a.splits;
        const int split = item - cg * per_cond - tile * a.splits;
        const int t0 = a.G.start + tile * PT;
        const int end = a.G.start + a.G.points;
        const int t1 = t0 + PT < end ? t0 + PT : end;
        const int tl = t1 - 1;
        const size_t gbase = size_t(cg) * size_t(a.n);
        const int* whi = a.whi + gbase;
        const int* wlo = a.wlo + gbase;
        const int* mi = a.mi;
        int kc = 0;
#pragma unroll
        for (int c = 0; c < C; ++c) kc = max(kc, a.kc[cg * C + c]);
        const long La = warp_lower_bound(0, a.n, lane, [&](long i) { return whi[i] > t0; });
        const long Lb = warp_lower_bound(La, a.n, lane, [&](long i) { return wlo[i] >= t1; });
        const long fs = warp_lower_bound(La, Lb, lane, [&](long i) { return whi[i] >= t1; });
        const long Cb = warp_lower_bound(La, Lb, lane, [&](long i) { return wlo[i] > t0; });
        const long fe = Cb > fs ? Cb : fs;
        // core candidates among all the tile's lines (partial ones included):
        // only lines in [E, Fc) can have a core band that reaches the row
        const long E = warp_lower_bound(La, Lb, lane, [&](long i) { return mi[i] >= t0 - kc; });
        const long Fc = warp_lower_bound(E, Lb, lane, [&](long i) { return mi[i] > tl + kc; });
        const LineSh64* lsh = reinterpret_cast<const LineSh64*>(a.lsh) + gbase;
        const CondRec64* crec = reinterpret_cast<const CondRec64*>(a.rec) + gbase * C;

        const size_t cell0 = size_t(cg) * size_t(a.ncell);
        const LineRuns runs =
            line_runs(a.chead + cell0, a.ncell, a.cshift, a.n, La, Lb, fs, fe, F[t0], F[tl], lane);

        const int jj = t0 + lane % PT;
        const double fj = F[jj < t1 ? jj : tl];
        double accd[C];
#pragma unroll
        for (int c = 0; c < C; ++c) accd[c] = 0.0;

        // x (in Doppler widths) of this lane's point for condition record r.
        auto offset = [&](const LineSh64& s, const CondRec64& r) { return (s.nu - fj) * r.g; };
        auto region1 = [&](double xs, const CondRec64& r, double mask, int c) {
            const double u = fma(xs, xs, r.Cy);
            accd[c] = fma(fma(u, r.Pc, r.Pc), rcp_refined_f64(fma(u, u, r.D2)) * mask, accd[c]);
        };
        // One condition of a partial line, or of a line whose core band may
        // reach this row; `in`: this lane's point lies in the line's window.
        auto core_cond = [&](const LineSh64& s, const CondRec64& r, int mline, bool in, int c) {
            const double xs = offset(s, r);
            const double ax = xs < 0.0 ? -xs : xs;
            const double sx = ax + r.y;
            bool band = false;
            if (r.core != -1) {
                const int aa = r.core & 0xffff, bb = (r.core >> 16) & 0xffff;
                const int rel = jj - mline;
                band = (aa == 0x7fff || rel >= -aa) && (bb == 0x7fff || rel <= bb);
            }
            // x and y are bit-identical to the reference's, so |x| + y < 15
            // is the reference's region choice.
            const bool special = in && band && sx < 15.0;
            region1(xs, r, (in && !special) ? 1.0 : 0.0, c);
        };

        // this item's groups of 32 lines
        const int ngroups = runs.groups_of(a.splits, split);
        auto gstart = [&](int gi, long& end) { return runs.start(split + gi * a.splits, end); };
        auto stage_group = [&](int bufi, long b, int cnt) {
            stage(lsb + bufi * 32, lsh + b, cnt, lane);
            stage(crb + bufi * 32 * C, crec + b * C, cnt * C, lane);
        };
        if (ngroups > 0) {
            long end;
            const long b = gstart(0, end);
            stage_group(0, b, int(end - b < 32 ? end - b : 32));
            cp_async_commit();
        }
        for (int gi = 0; gi < ngroups; ++gi) {
            if (gi + 1 < ngroups) {
                long end;
                const long b = gstart(gi + 1, end);
                const long rem = end - b;
                stage_group((gi + 1) & 1, b, int(rem < 32 ? rem : 32));
                cp_async_commit();
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncwarp();
            const LineSh64* SL = lsb + (gi & 1) * 32;
            const CondRec64* SC = crb + (gi & 1) * 32 * C;
            long end;
            const long gb = gstart(gi, end);
            const long ge = end - gb < 32 ? end : gb + 32;
            auto lo_of = [&](long v) { return int((v < gb ? gb : (v > ge ? ge : v)) - gb); };
            const int b1 = lo_of(E), c1 = lo_of(Fc);  // the core candidates
            // Lines [x, y) that are not core candidates: region I, the window
            // as a lane mask (one loop for the lines before and after the
            // candidates, full and partial ones alike); with LS > 1 a lane
            // past its last line takes the run's last one with weight 0.
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int x = h ? c1 : 0, y = h ? int(ge - gb) : b1;
                for (int b = x; b < y; b += LS) {
                    const int t = min(b + sub, y - 1);
                    const LineSh64 s = SL[t];
                    const double mask = (b + sub < y && jj >= s.lo && jj < s.hi) ? 1.0 : 0.0;
#pragma unroll
                    for (int c = 0; c < C; ++c) region1(offset(s, SC[t * C + c]), SC[t * C + c], mask, c);
                }
            }
            // Core candidates.  Per condition: when its core band misses the
            // row, region I with the window as a lane mask; otherwise the
            // lane-by-lane core path.
            auto cand_run = [&](int x, int y) {
                for (int b = x; b < y; b += LS) {
                    const int t = min(b + sub, y - 1);
                    const LineSh64 s = SL[t];
                    const bool in = b + sub < y && jj >= s.lo && jj < s.hi;
                    const double mask = in ? 1.0 : 0.0;
                    const int mline = mi[gb + t];
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        const CondRec64& r = SC[t * C + c];
                        bool hit = false;
                        if (r.core != -1) {
                            const int aa = r.core & 0xffff, bb = (r.core >> 16) & 0xffff;
                            hit = (aa == 0x7fff || mline - aa <= tl) && (bb == 0x7fff || mline + bb >= t0);
                        }
                        if (!hit) {
                            region1(offset(s, r), r, mask, c);
                        } else {
                            core_cond(s, r, mline, in, c);
                        }
                    }
                }
            };
            cand_run(b1, c1);
            __syncwarp();
        }
        if (runs.fa < runs.fb || runs.fc < runs.fd)
            add_far_cells_mc<C, C, kCellTerms64, LS>(a.chead + cell0, a.cmom + cell0 * (kCellTerms64 * C), runs,
                                                     a.splits, split, kCellBits64, F[t0], F[tl], fj, accd, lane, sub);
#pragma unroll
        for (int c = 0; c < C; ++c) accd[c] = sum_subsets<LS>(accd[c]);
        // W4 regions II-IV (point p of the row in lane p)
        double (*T)[kCoreRow64] = reinterpret_cast<double (*)[kCoreRow64]>(mine);
#pragma unroll 1
        for (int c = 0; c < C; ++c) {
            const double add = core_row_f64(
                T, F, E, Fc, t0, a.splits, split, lane,
                [&](long i, double& nu, double& g, double& y, double& pref, int& jlo, int& jhi) {
                    const CondRec64& r = crec[i * C + c];
                    if (r.core == -1) return;
                    const LineSh64 ls = lsh[i];
                    const int aa = r.core & 0xffff, bb = (r.core >> 16) & 0xffff, m = mi[i];
                    nu = ls.nu;
                    g = r.g;
                    y = r.y;
                    pref = r.pref;
                    jlo = max(aa == 0x7fff ? t0 : max(m - aa, t0), ls.lo);
                    jhi = min(bb == 0x7fff ? tl : min(m + bb, tl), ls.hi - 1);
                });
#pragma unroll
            for (int q = 0; q < C; ++q)
                if (q == c) accd[q] += add;
        }
        if (sub == 0 && jj < t1) {
#pragma unroll
            for (int c = 0; c < C; ++c) put_result(a, cg * C + c, split, jj, accd[c]);
        }
    }
}

// ---------------------------------------------------------------------------
// Mixed-precision multi-condition step two (Voigt), packed FP32x2.
//
// Work items and line runs are those of k_steptwo_voigt_mc.  Per (line, point)
// one condition-free offset X = (m - j) dfn + rn and X^2 are formed; conditions
// are then taken in pairs, each pair one packed FP32x2 operation per step of
// the region-I rational (u = X^2 k^2 + Cy, u^2 + D2, Pc (u + 1)), two lines
// sharing one reciprocal.  The rational is added at every pair of the window
// except, on core candidates, where u < 1; k_core_mcx adds W4 less the rational
// (where it was added) inside the W4 region intervals (|x| + y < 15, from step
// one).
//
// A row is 64 / LS points; each lane owns two of them and every LS-th line
// (LS = 2: rows of 32; LS = 8: rows of 8, for coarse grids over dense lists --
// 40 conditions, 1e7 lines, 0.1 cm-1 grid: a 32-point row has 6.4 cm-1 of lines
// whose windows end in it and 3.2 of its own width beside the 2 near it, an
// 8-point one 1.6 and 0.8).  What bounds it is shared memory: a lane needs 24 +
// 8 C bytes of every line it takes, 128 bytes a wavefront for the warp, so two
// points per lane halve it, and 2 y^2 comes from Cy = y^2 - 1/2 instead of a
// third array.  After each group of 32 lines the FP32 sums (32 / LS lines deep)
// are added up over the lane subsets by halving exchanges, each lane keeping
// 2 C / LS of them in FP64.  (Every LS groups only, 0.6 of 24.8 ms less for the
// 40-condition sweep, the error at 10 atm is 0.23e-7 instead of 0.18e-7, and
// 0.57e-7 instead of 0.43e-7 for a tenth of the lines.)
// ---------------------------------------------------------------------------
// Resident blocks per SM the mixed multi-condition kernel asks the compiler
// to fit (register budget): 20 warps per SM at 8 conditions and 4 warps per
// block, 16 at 8 and 8, 24 otherwise -- the occupancy points the autotuner
// chooses between through the block size.
template <int C, int WARPS>
constexpr int voigt_mcx_min_blocks() {
    return (C == 8 && WARPS == 8) ? 2 : (C == 8 && WARPS == 4) ? 5 : 24 / WARPS;
}

// Region-I constants of a line for the C conditions of its group, in condition
// order: conditions 2k and 2k+1 are one packed FP32x2 operand, conditions
// 4k..4k+3 one 16-byte load.  Formed in shared memory from the (y, c pref) pairs
// of step one when a group of lines has arrived.
template <int C>
struct __align__(C == 2 ? 8 : 16) LineR1 {
    float Cy[C], Pc[C];
};
// (the core pass repeats step two's choice on u = X^2 k^2 + Cy: one definition)
__device__ __forceinline__ float region1_cy(float y) { return fmaf(y, y, -0.5f); }
// D2 = 2 y^2 of a packed pair of conditions: within 6e-8 of max(1, 2 y^2), and it
// is added to u^2 with u >= 1.
__device__ __forceinline__ float2 region1_d2(float2 cy) { return __ffma2_rn(cy, f2s(2.0f), f2s(1.0f)); }

// Shared memory of one warp: two stages of 32 lines' offsets and flags (16 B),
// windows (8 B) and (y, c pref) (8 B per condition), and 32 lines' constants.
template <int C>
constexpr size_t mcx_warp_smem() {
    return 64 * (sizeof(float4) + sizeof(int2) + C * sizeof(float2)) + 32 * sizeof(LineR1<C>);
}

// Sums w[0..V) over the lane bits 16 .. LP by halving exchanges: a lane ends
// with kept() values from base() on (fewer values than lanes: every
// lane of the remaining bits holds the same one).
template <int V, int LP, class R = float>
struct Halving {
    static constexpr int kept() { return V * LP / 32 > 1 ? V * LP / 32 : 1; }
    __device__ static __forceinline__ void sum(R (&w)[V], int lane) {
        int n = V;
#pragma unroll
        for (int o = 16; o >= LP; o >>= 1) {
            if (n > 1) {
                n /= 2;
                const bool up = (lane & o) != 0;
#pragma unroll
                for (int i = 0; i < V / 2; ++i)
                    if (i < n) {
                        const R got = __shfl_xor_sync(0xffffffffu, up ? w[i] : w[i + n], o);
                        w[i] = (up ? w[i + n] : w[i]) + got;
                    }
            } else {
                w[0] += __shfl_xor_sync(0xffffffffu, w[0], o);
            }
        }
    }
    // First of the lane's values, and whether another lane holds the same ones.
    __device__ static __forceinline__ int base(int lane, bool& copy) {
        int n = V, at = 0;
        copy = false;
#pragma unroll
        for (int o = 16; o >= LP; o >>= 1) {
            if (n > 1) {
                n /= 2;
                if (lane & o) at += n;
            } else if (lane & o) {
                copy = true;
            }
        }
        return at;
    }
};

template <int C, int WARPS, int LS>
__global__ void __launch_bounds__(WARPS * 32, (voigt_mcx_min_blocks<C, WARPS>()))
    k_steptwo_voigt_mcx(StepArgs a) {
    static_assert(C % 2 == 0, "conditions come in pairs");
    constexpr int NP = C / 2;
    constexpr int LP = 32 / LS, PT = 2 * LP;  // lane points, points of a row
    using Sum = Halving<2 * C, LP>;
    constexpr int VF = Sum::kept();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    using R1 = LineR1<C>;
    // staged per line: the offsets and flags of LineShX, its window and the
    // conditions' (y, c pref), [condition][line]; a whole line's FP64 centre is
    // read from memory when needed
    unsigned char* const mine = smem_raw + size_t(warp) * mcx_warp_smem<C>();
    float4* lsb = reinterpret_cast<float4*>(mine);
    R1* SR = reinterpret_cast<R1*>(mine + 64 * sizeof(float4));
    float2* ypb = reinterpret_cast<float2*>(mine + 64 * sizeof(float4) + 32 * sizeof(R1));
    int2* lhb = reinterpret_cast<int2*>(ypb + 64 * C);
    const int sub = lane / LP;
    const double* F = a.G.freq;

    for (;;) {
        int item = 0;
        if (lane == 0) item = int(atomicAdd(a.counter, 1u));
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.n_items) break;
        const int per_cond = a.tiles_per_cond * a.splits;
        const int cg = item / per_cond;
        const int tile = (item - cg * per_cond) / a.splits;
        const int split = item - cg * per_cond - tile * a.splits;
        const int t0 = a.G.start + tile * PT;
        const int gend = a.G.start + a.G.points;
        const int t1 = t0 + PT < gend ? t0 + PT : gend;
        const int tl = t1 - 1;
        const size_t wbase = size_t(a.wslot[cg]) * size_t(a.n);  // the group's window data
        const int* whi = a.whi + wbase;
        const int* wlo = a.wlo + wbase;
        const int* mi = a.mi;
        int kc = 0;
#pragma unroll
        for (int c = 0; c < C; ++c) kc = max(kc, a.kc[cg * C + c]);
        // line indices fit 32 bits (at most 2^31 - 1 lines per call)
        const int La = warp_search(whi, 0, int(a.n), t0 + 1, lane);
        const int Lb = warp_search(wlo, La, int(a.n), t1, lane);
        const int fs = warp_search(whi, La, Lb, t1, lane);
        const int Cb = warp_search(wlo, La, Lb, t0 + 1, lane);
        const int fe = Cb > fs ? Cb : fs;
        // core candidates [E, Fc): the lines whose near-centre pairs may
        // fall in the tile (kc: the group's widest reach plus one; 0: no
        // line of the group has such pairs)
        int E = La, Fc = La;
        if (kc > 0) {
            E = warp_search(mi, La, Lb, t0 - (kc - 1), lane);
            Fc = warp_search(mi, E, Lb, tl + kc, lane);
        }
        const LineShX* lsh = reinterpret_cast<const LineShX*>(a.lsh) + wbase;
        const float2* yp = a.cyp + size_t(cg) * C * size_t(a.n);
        const size_t cell0 = size_t(cg) * size_t(a.ncell);
        const LineRuns runs =
            line_runs(a.chead + cell0, a.ncell, a.cshift, a.n, La, Lb, fs, fe, F[t0], F[tl], lane);

        const int j0 = t0 + lane % LP, j1 = j0 + LP;  // this lane's points
        const float jf0 = float(j0), jf1 = float(j1);
        float2 k2[NP];
        float2 acc[2][NP];
        double sum[VF];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            k2[p] = f2(a.kx2[cg * C + 2 * p], a.kx2[cg * C + 2 * p + 1]);
            acc[0][p] = acc[1][p] = f2(0.0f, 0.0f);
        }
#pragma unroll
        for (int v = 0; v < VF; ++v) sum[v] = 0.0;

        // Two narrow lines A, B that are not core candidates, at once: per
        // condition one reciprocal for both lines, to += (nA dB + nB dA)
        // / (dA dB) (u >= 1 on such lines, so dA, dB >= 1; narrow lines
        // keep dA dB and the products with Pc in range, kPairUMax).  inA,
        // inB: the point takes the line (a line left out adds exactly 0).
        auto pair_step = [&](float XA2, float XB2, float2 cyA, float2 d2A, float2 pcA, float2 cyB, float2 d2B,
                             float2 pcB, int p, bool inA, bool inB, float2& to) {
            const float2 uA = __ffma2_rn(f2s(XA2), k2[p], cyA);
            const float2 uB = __ffma2_rn(f2s(XB2), k2[p], cyB);
            const float2 dA = __ffma2_rn(uA, uA, d2A);
            const float2 dB = __ffma2_rn(uB, uB, d2B);
            float2 nA = __ffma2_rn(uA, pcA, pcA);
            float2 nB = __ffma2_rn(uB, pcB, pcB);
            if (!inA) nA = f2(0.0f, 0.0f);
            if (!inB) nB = f2(0.0f, 0.0f);
            const float2 q = __fmul2_rn(dA, dB);
            const float2 sn = __ffma2_rn(nB, dA, __fmul2_rn(nA, dB));
            to = __ffma2_rn(sn, f2(rcp_approx_f32(q.x), rcp_approx_f32(q.y)), to);
        };
        // One line (wide, or in a wide one's company) at one point, not a core
        // candidate: a reciprocal per pair.
        auto solo_step = [&](float X2, float2 cy, float2 pc, int p, bool in, float2& to) {
            const float2 u = __ffma2_rn(f2s(X2), k2[p], cy);
            const float2 den = __ffma2_rn(u, u, region1_d2(cy));
            float2 num = __ffma2_rn(u, pc, pc);
            if (!in) num = f2(0.0f, 0.0f);
            to = __ffma2_rn(num, f2(rcp_approx_f32(den.x), rcp_approx_f32(den.y)), to);
        };
        // One line (far, whole or a core candidate, or any in their company)
        // at one point: a reciprocal per pair.  NEAR: a pair is kept only where
        // u >= 1 (core candidates: the core pass takes u < 1).  Pc / u to FP32
        // rounding from u = 1e12 on (u^2 overflows from 1.8e19); beyond x = 1e18
        // region I is taken as 0.  A pair that is left out adds exactly 0: the
        // product itself is selected, so an infinite reciprocal never counts.
        auto line_step = [&](bool near, float X, const R1& r, int p, bool in, float2& to) {
            const float2 cy = *reinterpret_cast<const float2*>(&r.Cy[2 * p]);
            const float2 pc = *reinterpret_cast<const float2*>(&r.Pc[2 * p]);
            const float2 u = __ffma2_rn(f2s(X * X), k2[p], cy);
            float2 den = __ffma2_rn(u, u, region1_d2(cy));
            float2 num = __ffma2_rn(u, pc, pc);
            if (u.x > 1.0e12f) den.x = u.x, num.x = pc.x;
            if (u.y > 1.0e12f) den.y = u.y, num.y = pc.y;
            const float aX = fabsf(X);
            const bool k0 = in && !(near && u.x < 1.0f) && aX * a.kx[cg * C + 2 * p] < 1.0e18f;
            const bool k1 = in && !(near && u.y < 1.0f) && aX * a.kx[cg * C + 2 * p + 1] < 1.0e18f;
            to.x += k0 ? num.x * rcp_approx_f32(den.x) : 0.0f;
            to.y += k1 ? num.y * rcp_approx_f32(den.y) : 0.0f;
        };
        // A narrow core candidate at one point, two pairs of conditions with one
        // reciprocal per two evaluations: a condition's pair is kept where the
        // point takes the line (`in`) and u >= 1; a pair that is not kept enters
        // the shared product as 1 and adds exactly zero.
        auto near_step = [&](float X2, const float4& cy, const float4& pc, int p, bool in, float2& toA, float2& toB) {
            const float2 cA = f2(cy.x, cy.y), cB = f2(cy.z, cy.w);
            const float2 uA = __ffma2_rn(f2s(X2), k2[p], cA);
            const float2 uB = __ffma2_rn(f2s(X2), k2[p + 1], cB);
            const bool q0 = in && !(uA.x < 1.0f), q1 = in && !(uA.y < 1.0f);
            const bool q2 = in && !(uB.x < 1.0f), q3 = in && !(uB.y < 1.0f);
            const float2 dA0 = __ffma2_rn(uA, uA, region1_d2(cA));
            const float2 dB0 = __ffma2_rn(uB, uB, region1_d2(cB));
            const float2 nA = __ffma2_rn(uA, f2(pc.x, pc.y), f2(pc.x, pc.y));
            const float2 nB = __ffma2_rn(uB, f2(pc.z, pc.w), f2(pc.z, pc.w));
            const float2 dA = f2(q0 ? dA0.x : 1.0f, q1 ? dA0.y : 1.0f);
            const float2 dB = f2(q2 ? dB0.x : 1.0f, q3 ? dB0.y : 1.0f);
            const float2 q = __fmul2_rn(dA, dB);
            const float2 rq = f2(rcp_approx_f32(q.x), rcp_approx_f32(q.y));
            const float2 iA = __fmul2_rn(dB, rq);
            const float2 iB = __fmul2_rn(dA, rq);
            toA = __ffma2_rn(nA, f2(q0 ? iA.x : 0.0f, q1 ? iA.y : 0.0f), toA);
            toB = __ffma2_rn(nB, f2(q2 ? iB.x : 0.0f, q3 ? iB.y : 0.0f), toB);
        };

        const int ngroups = runs.groups_of(a.splits, split);
        auto gstart = [&](int gi, int& end) {
            long e;
            const int b = int(runs.start(split + gi * a.splits, e));
            end = int(e);
            return b;
        };
        auto stage_group = [&](int gi) {
            int end;
            const int b = gstart(gi, end), bufi = gi & 1;
            if (b + lane < end) {
                cp_async16(lsb + bufi * 32 + lane, lsh + b + lane);
                cp_async8(lhb + bufi * 32 + lane, &lsh[b + lane].lo);
#pragma unroll
                for (int c = 0; c < C; ++c) cp_async8(ypb + (bufi * C + c) * 32 + lane, yp + size_t(c) * size_t(a.n) + b + lane);
            }
            cp_async_commit();
        };
        if (ngroups > 0) stage_group(0);
        for (int gi = 0; gi < ngroups; ++gi) {
            if (gi + 1 < ngroups) {
                stage_group(gi + 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncwarp();
            const float4* SL = lsb + (gi & 1) * 32;  // m, df/nu, r/nu, flags
            const int2* SW = lhb + (gi & 1) * 32;    // window [lo, hi)
            {
                // this lane's line's constants (lanes past the group's end
                // convert what an earlier group left: never used)
                R1& r = SR[lane];
#pragma unroll
                for (int c = 0; c < C; c += 2) {
                    const float2 v0 = ypb[((gi & 1) * C + c) * 32 + lane], v1 = ypb[((gi & 1) * C + c + 1) * 32 + lane];
                    *reinterpret_cast<float2*>(&r.Cy[c]) = f2(region1_cy(v0.x), region1_cy(v1.x));
                    *reinterpret_cast<float2*>(&r.Pc[c]) = f2(v0.y * v0.x, v1.y * v1.x);
                }
            }
            __syncwarp();
            int end;
            const int gb = gstart(gi, end);
            const int ge = end - gb < 32 ? end : gb + 32;
            auto lo_of = [&](int v) { return (v < gb ? gb : (v > ge ? ge : v)) - gb; };
            const int b1 = lo_of(E), c1 = lo_of(Fc);  // the core candidates
            // Lines [x, y) that are not core candidates, two at a time, the
            // window as a lane mask.  Lane subset `sub` takes lines x + sub,
            // x + sub + LS, ...; a lane past the run's end takes its last line
            // with `in` false.  One loop for the lines before and after the
            // candidates (and for full and partial ones alike): the body is
            // large, and six copies of it ran out of the instruction cache.
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int x = h ? c1 : 0, y = h ? ge - gb : b1;
#pragma unroll 1
                for (int b = x; b < y; b += 2 * LS) {
                    const int tA = min(b + sub, y - 1), tB = min(b + sub + LS, y - 1);
                    const float4 sA = SL[tA];
                    const float4 sB = SL[tB];
                    const int2 wA = SW[tA], wB = SW[tB];
                    const float XA0 = fmaf(sA.x - jf0, sA.y, sA.z), XA1 = fmaf(sA.x - jf1, sA.y, sA.z);
                    const float XB0 = fmaf(sB.x - jf0, sB.y, sB.z), XB1 = fmaf(sB.x - jf1, sB.y, sB.z);
                    const int flags = __float_as_int(sA.w) | __float_as_int(sB.w);
                    const bool wide = (flags & kLineWide) != 0;
                    const bool okA = b + sub < y, okB = b + sub + LS < y;
                    const bool inA0 = okA && j0 >= wA.x && j0 < wA.y, inA1 = okA && j1 >= wA.x && j1 < wA.y;
                    const bool inB0 = okB && j0 >= wB.x && j0 < wB.y, inB1 = okB && j1 >= wB.x && j1 < wB.y;
                    const R1 &rA = SR[tA], &rB = SR[tB];
                    if (!__any_sync(0xffffffffu, wide)) {
                        auto both = [&](float2 cyA, float2 pcA, float2 cyB, float2 pcB, int p) {
                            const float2 d2A = region1_d2(cyA), d2B = region1_d2(cyB);
                            pair_step(XA0 * XA0, XB0 * XB0, cyA, d2A, pcA, cyB, d2B, pcB, p, inA0, inB0, acc[0][p]);
                            pair_step(XA1 * XA1, XB1 * XB1, cyA, d2A, pcA, cyB, d2B, pcB, p, inA1, inB1, acc[1][p]);
                        };
                        if constexpr (NP % 2 == 0) {
                            // conditions 4q..4q+3: one 16-byte load per array and line
#pragma unroll
                            for (int p = 0; p < NP; p += 2) {
                                const float4 cyA = *reinterpret_cast<const float4*>(&rA.Cy[2 * p]);
                                const float4 pcA = *reinterpret_cast<const float4*>(&rA.Pc[2 * p]);
                                const float4 cyB = *reinterpret_cast<const float4*>(&rB.Cy[2 * p]);
                                const float4 pcB = *reinterpret_cast<const float4*>(&rB.Pc[2 * p]);
                                both(f2(cyA.x, cyA.y), f2(pcA.x, pcA.y), f2(cyB.x, cyB.y), f2(pcB.x, pcB.y), p);
                                both(f2(cyA.z, cyA.w), f2(pcA.z, pcA.w), f2(cyB.z, cyB.w), f2(pcB.z, pcB.w), p + 1);
                            }
                        } else {
                            both(*reinterpret_cast<const float2*>(&rA.Cy[0]), *reinterpret_cast<const float2*>(&rA.Pc[0]),
                                 *reinterpret_cast<const float2*>(&rB.Cy[0]), *reinterpret_cast<const float2*>(&rB.Pc[0]), 0);
                        }
                    } else if (!__any_sync(0xffffffffu, (flags & (kLineFar | kLineWhole)) != 0)) {
#pragma unroll
                        for (int p = 0; p < NP; ++p) {
                            const float2 cyA = *reinterpret_cast<const float2*>(&rA.Cy[2 * p]);
                            const float2 pcA = *reinterpret_cast<const float2*>(&rA.Pc[2 * p]);
                            const float2 cyB = *reinterpret_cast<const float2*>(&rB.Cy[2 * p]);
                            const float2 pcB = *reinterpret_cast<const float2*>(&rB.Pc[2 * p]);
                            solo_step(XA0 * XA0, cyA, pcA, p, inA0, acc[0][p]);
                            solo_step(XA1 * XA1, cyA, pcA, p, inA1, acc[1][p]);
                            solo_step(XB0 * XB0, cyB, pcB, p, inB0, acc[0][p]);
                            solo_step(XB1 * XB1, cyB, pcB, p, inB1, acc[1][p]);
                        }
                    } else {
#pragma unroll
                        for (int p = 0; p < NP; ++p)
#pragma unroll 1
                            for (int q = 0; q < 2; ++q) {
                                line_step(false, q ? XB0 : XA0, q ? rB : rA, p, q ? inB0 : inA0, acc[0][p]);
                                line_step(false, q ? XB1 : XA1, q ? rB : rA, p, q ? inB1 : inA1, acc[1][p]);
                            }
                    }
                }
            }
            // Core candidates: region I where u >= 1, per condition (the
            // core pass takes the pairs with u < 1, deciding on the same FP32
            // u).
#pragma unroll 1
            for (int b = b1; b < c1; b += LS) {
                const int t = min(b + sub, c1 - 1);
                const float4 s = SL[t];
                const int flags = __float_as_int(s.w);
                const int2 win = SW[t];
                const bool ok = b + sub < c1;
                const bool in0 = ok && j0 >= win.x && j0 < win.y, in1 = ok && j1 >= win.x && j1 < win.y;
                const R1& r = SR[t];
                if (NP % 2 == 0 && !__any_sync(0xffffffffu, (flags & (kLineWhole | kLineWide)) != 0)) {
                    const float X0 = fmaf(s.x - jf0, s.y, s.z), X1 = fmaf(s.x - jf1, s.y, s.z);
#pragma unroll
                    for (int p = 0; p + 1 < NP; p += 2) {
                        const float4 cy = *reinterpret_cast<const float4*>(&r.Cy[2 * p]);
                        const float4 pc = *reinterpret_cast<const float4*>(&r.Pc[2 * p]);
                        near_step(X0 * X0, cy, pc, p, in0, acc[0][p], acc[0][p + 1]);
                        near_step(X1 * X1, cy, pc, p, in1, acc[1][p], acc[1][p + 1]);
                    }
                    continue;
                }
                // whole lines: X from the FP64 centre (rare; the grid value is
                // read here rather than held for every line)
                double nu = 0.0;
                if (flags & kLineWhole) nu = lsh[gb + t].nu;
                const float X0 = (flags & kLineWhole) ? float((nu - F[min(j0, tl)]) / nu) : fmaf(s.x - jf0, s.y, s.z);
                const float X1 = (flags & kLineWhole) ? float((nu - F[min(j1, tl)]) / nu) : fmaf(s.x - jf1, s.y, s.z);
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    line_step(true, X0, r, p, in0, acc[0][p]);
                    line_step(true, X1, r, p, in1, acc[1][p]);
                }
            }
            {
                float w[2 * C];
#pragma unroll
                for (int v = 0; v < C; ++v) {
                    const float2 x = acc[v / NP][v % NP];  // values 2 v, 2 v + 1
                    w[2 * v] = x.x;
                    w[2 * v + 1] = x.y;
                    acc[v / NP][v % NP] = f2(0.0f, 0.0f);
                }
                Sum::sum(w, lane);
#pragma unroll
                for (int v = 0; v < VF; ++v) sum[v] += double(w[v]);
            }
            __syncwarp();
        }
        // value (point, condition) = point * C + condition
        bool copy;
        const int base = Sum::base(lane, copy);
        const int c0 = base % C, jj = base / C ? j1 : j0;
        if (runs.fa < runs.fb || runs.fc < runs.fd)
            add_far_cells_mc<C, VF, kCellTermsMixed>(a.chead + cell0, a.cmom + cell0 * (kCellTermsMixed * C) + c0, runs,
                                                     a.splits, split, kCellBitsMixed, F[t0], F[tl],
                                                     F[jj < t1 ? jj : tl], sum, lane);
        if (!copy && jj < t1) {
#pragma unroll
            for (int v = 0; v < VF; ++v) put_result(a, cg * C + c0 + v, split, jj, sum[v]);
        }
    }
}

// The core passes' per-warp table: row = point of the 32-point row, column =
// lane (stride kCoreRow floats keeps rows 16-byte aligned and a quarter-warp's
// 128-bit row reads on distinct banks).  It starts all zero; each lane adds its
// lines' entries to its own column, and every kCoreBatches batches of 32 lines
// every lane sums its point's row into FP64 and clears it: FP32 sums at most
// kCoreBatches + 9 deep in a fixed order.  (One sum and one clearing per batch
// took a quarter of the pass: few entries per batch and line.)
constexpr int kCoreRow = 36;
constexpr int kCoreBatches = 8;
__device__ __forceinline__ void core_table_clear(float (*T)[kCoreRow], int lane) {
#pragma unroll
    for (int q = 0; q < 32; q += 4) *reinterpret_cast<float4*>(&T[lane][q]) = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
}
// Sum of this lane's row, which is cleared.  Warp-uniform.
__device__ __forceinline__ double core_table_take(float (*T)[kCoreRow], int lane) {
    __syncwarp();
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int q = 0; q < 32; q += 4) {
        float4* row = reinterpret_cast<float4*>(&T[lane][q]);
        const float4 v = *row;
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
        *row = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncwarp();
    return double(s.x) + double(s.y) + double(s.z) + double(s.w);
}

// Core pass of the mixed multi-condition layout.  A warp takes a (condition,
// row of 32 grid points); the lines whose region interval may reach the row
// form one run (the nearest grid index mi[] is ascending; the condition's
// widest interval bounds the reach), taken 32 at a time: each lane evaluates
// W4 regions II-IV (region III-IV interval from step one, region III or IV
// by Humlicek's test on the FP32 x, y) at the row's points inside its line's
// interval, less the region-I rational where step two added it, and adds
// them to its column of a per-warp table; every few batches each lane sums its
// point's row into FP64, in a fixed order.  With line splits (blockIdx.z = split) a
// row's batches are shared out as in step two and the sums go to the parts.
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_core_mcx(CoreArgs a) {
    __shared__ __align__(16) float tab[WARPS][32][kCoreRow];  // [point][line of the batch]
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    // blockIdx.x = condition, so that the blocks of one set of rows run
    // together and the lines' shared data (LineShX, mi) comes from DRAM once
    // for all conditions; blockIdx.y steps over the sets of WARPS rows.
    const int c = int(blockIdx.x);
    const int end = a.G.start + a.G.points;
    const int row_sets = (a.G.points + 32 * WARPS - 1) / (32 * WARPS);
    float (*T)[kCoreRow] = tab[warp];
    core_table_clear(T, lane);
    const int K = a.kc[kMaxCond + c];  // the condition's core-pass reach
    const int g = c / a.group;
    const CoreIv* civ = a.civ + size_t(c) * size_t(a.n);
    const float2* cyp = a.cyp + size_t(c) * size_t(a.n);
    const LineShX* lsh = a.lsh + size_t(a.wslot[g]) * size_t(a.n);
    // step two's core candidates of a row: the group's reach (kc - 1)
    int kcg = 0;
    for (int q = 0; q < a.group; ++q) kcg = max(kcg, a.kc[g * a.group + q]);
    const float k = a.kx[c], k2 = a.kx2[c];
    const int split = int(blockIdx.z), S = a.splits;
    for (int rs = int(blockIdx.y); rs < row_sets; rs += int(gridDim.y)) {
        const int t0 = a.G.start + (rs * WARPS + warp) * 32;
        if (t0 >= end) break;  // warp-uniform; later sets start further on
        const int t1 = t0 + 32 < end ? t0 + 32 : end;
        const int tl = t1 - 1;
        const long E = warp_lower_bound(0, a.n, lane, [&](long i) { return a.mi[i] >= t0 - K; });
        const long F = warp_lower_bound(E, a.n, lane, [&](long i) { return a.mi[i] > tl + K; });
        double acc = 0.0;
        int held = 0;  // batches in the table
        for (long b = E + 32L * split; b < F; b += 32L * S) {
            const long i = b + lane;
            int jlo = 1, jhi = 0;
            if (i < F) {
                const CoreIv iv = civ[i];
                jlo = max(iv.lo15, t0);
                jhi = min(iv.hi15, tl);
                if (jlo <= jhi) {
                    const LineShX s = lsh[i];
                    const float2 yp = cyp[i];
                    const int mline = a.mi[i];
                    const bool cand = kcg > 0 && mline >= t0 - (kcg - 1) && mline <= tl + (kcg - 1);
                    const float cy = region1_cy(yp.x);  // step two's u
                    for (int j = jlo; j <= jhi; ++j) {
                        const float X = (s.flags & kLineWhole) ? float((s.nu - a.freq[j]) / s.nu)
                                                               : fmaf(s.m - float(j), s.dfn, s.rn);
                        const float ax = fabsf(X) * k, y = yp.x;
                        float w;
                        if (j >= iv.lo55 && j <= iv.hi55)
                            w = float(1.0 / kW4C) * ((y >= fmaf(0.195f, ax, -0.176f)) ? w4_region3_re_f32(ax, y)
                                                                                       : w4_region4_re_f32(ax, y));
                        else
                            w = w4_region2_c(ax, y);
                        // step two added the region-I rational here unless the
                        // line was its core candidate and u < 1 (the same FP32 u)
                        if (!(cand && fmaf(X * X, k2, cy) < 1.0f)) w -= w4_region1_c(ax, y);
                        T[j - t0][lane] += yp.y * w;
                    }
                }
            }
            held += __any_sync(0xffffffffu, jlo <= jhi) ? 1 : 0;
            if (held == kCoreBatches) {
                acc += core_table_take(T, lane);
                held = 0;
            }
        }
        if (held > 0) acc += core_table_take(T, lane);
        const int jj = t0 + lane;
        if (jj < t1) {
            if (S <= 1)
                a.out[size_t(a.row[c]) * a.out_stride + size_t(jj)] += acc;
            else
                a.part[(size_t(c) * S + split) * a.part_stride + size_t(jj - a.G.start)] += acc;
        }
    }
}

// Core pass of the single-condition mixed layout (RecV32): as k_core_mcx,
// with the region intervals [clo, chi] and [lo55, hi55] of the records; a
// line marked whole (dfa < 0) takes x from its FP64 centre.
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_core_v32(StepArgs a) {
    __shared__ __align__(16) float tab[WARPS][32][kCoreRow];  // [point][line of the batch]
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int c = int(blockIdx.y);
    const int t0 = a.G.start + (int(blockIdx.x) * WARPS + warp) * 32;
    const int end = a.G.start + a.G.points;
    if (t0 >= end) return;
    float (*T)[kCoreRow] = tab[warp];
    core_table_clear(T, lane);
    const int t1 = t0 + 32 < end ? t0 + 32 : end;
    const int tl = t1 - 1;
    const int K = a.kc[kMaxCond + c];  // the condition's core-pass reach
    const long E = warp_lower_bound(0, a.n, lane, [&](long i) { return a.mi[i] >= t0 - K; });
    const long F = warp_lower_bound(E, a.n, lane, [&](long i) { return a.mi[i] > tl + K; });
    const RecV32* recs = reinterpret_cast<const RecV32*>(a.rec) + size_t(c) * size_t(a.n);
    const float k = a.kx[c];
    const int split = int(blockIdx.z), S = a.splits;
    double acc = 0.0;
    int held = 0;  // batches in the table
    for (long b = E + 32L * split; b < F; b += 32L * S) {
        const long i = b + lane;
        int jlo = 1, jhi = 0;
        if (i < F) {
            const RecV32 r = recs[i];
            const bool whole = r.dfa < 0.0f;
            jlo = max(int(r.clo), t0);
            jhi = min(int(r.chi), tl);
            for (int j = jlo; j <= jhi; ++j) {
                const float xs = whole ? float((r.nu - a.G.freq[j]) / r.nu) * k : fmaf(r.m - float(j), r.dfa, r.ra);
                const float ax = fabsf(xs), y = r.y;
                float w;
                if (float(j) >= r.lo55 && float(j) <= r.hi55)
                    w = (y >= fmaf(0.195f, ax, -0.176f)) ? w4_region3_re_f32(ax, y) : w4_region4_re_f32(ax, y);
                else
                    w = w4_region2_re<float>(ax, y);
                T[j - t0][lane] += r.pref * w;
            }
        }
        held += __any_sync(0xffffffffu, jlo <= jhi) ? 1 : 0;
        if (held == kCoreBatches) {
            acc += core_table_take(T, lane);
            held = 0;
        }
    }
    if (held > 0) acc += core_table_take(T, lane);
    const int jj = t0 + lane;
    if (jj < t1) {
        if (S <= 1)
            a.out[size_t(a.row[c]) * a.out_stride + size_t(jj)] += acc;
        else
            a.part[(size_t(c) * S + split) * a.part_stride + size_t(jj - a.G.start)] += acc;
    }
}

// ---------------------------------------------------------------------------
// Mixed-precision single-condition step two with cells, lane = line.
//
// With the far wings taken by cells, what is left of a tile is a few thousand
// lines on few points, so the lanes go over the lines: a warp takes a tile of PT
// points and 32 lines at a time, each lane evaluating its own line at every
// point of the tile into PT accumulators.  The line's constants are read once
// per lane (a broadcast to every lane costs a shared-memory wavefront per 4
// bytes), and the lines of a group, being neighbours, are in the same W4 region
// at the same point.  Every 4 groups of lines the accumulators are summed over
// the lanes by halving exchanges and added in FP64 (sums 4 + 5 deep; 3e5 lines on
// 5e4 points at 10 atm: 1.66e-8 of the result in the 2-norm, 1.93e-8 and 2 % less
// time with 8 groups; a lane per point 2.25e-8).  Tiles of 16 points (32: 2.72 against
// 2.50 ms at the sizes below), of 8 on coarse grids over dense lists, where 16
// points are wider than the near zone.
//
// Two evaluations share one reciprocal, 1/dA = dB / (dA dB) (narrow lines,
// kPairUMax); groups with wide lines take one each (3000 lines, 50000 points, cut
// 100: 189 us with all their pairs in the loop below, 102 so).  Groups with lines
// of the core reach choose region I or II per pair by the exact region intervals;
// the pairs of regions III and IV, and all pairs of groups with whole lines, are
// evaluated in a loop by their own line's lane into a per-warp table with a column
// per lane.  (Few unrolled
// bodies: with every region unrolled a third of the time went to instruction
// fetches.)
//
// B200, 1e7 lines, 7.5e5 points: 2.6 ms against 3.5 + 1.2 ms for the
// point-parallel kernel with cells and its core pass.  The same kernel over
// 32 / C points and C = 8 conditions was slower than k_steptwo_voigt_mcx on the
// coarse sweep (20.7 against 12.6 ms).
// ---------------------------------------------------------------------------
constexpr int kNearRow = 33;
// Two stages of offsets and flags, windows and (y, pref), and the table.
template <int PT>
constexpr size_t near_warp_smem() {
    return 64 * (sizeof(float4) + sizeof(int2) + sizeof(float2)) + sizeof(float) * PT * kNearRow;
}
// Sum over the lanes of one tile point's sub-lanes (neighbours), to each of them.
template <int SUB>
__device__ __forceinline__ double sum_neighbours(double v) {
#pragma unroll
    for (int o = 1; o < SUB; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int PT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 20 / WARPS) k_steptwo_near(StepArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    constexpr int SUB = 32 / PT;  // lanes to a point where lanes stand for points
    using Sum = Halving<PT, 1>;   // lane ends with point lane / SUB
    unsigned char* const mine = smem_raw + size_t(threadIdx.x >> 5) * near_warp_smem<PT>();
    float4* lsb = reinterpret_cast<float4*>(mine);
    float2* ypb = reinterpret_cast<float2*>(mine + 64 * sizeof(float4));
    int2* lhb = reinterpret_cast<int2*>(ypb + 64);
    float (*T)[kNearRow] = reinterpret_cast<float (*)[kNearRow]>(lhb + 64);
    const double* F = a.G.freq;
    const int* mi = a.mi;
#pragma unroll 4
    for (int q = 0; q < PT; ++q) T[q][lane] = 0.0f;
    __syncwarp();

    for (;;) {
        int item = 0;
        if (lane == 0) item = int(atomicAdd(a.counter, 1u));
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.n_items) break;
        const int per_cond = a.tiles_per_cond * a.splits;
        const int cond = item / per_cond;
        const int tile = (item - cond * per_cond) / a.splits;
        const int split = item - cond * per_cond - tile * a.splits;
        const int t0 = a.G.start + tile * PT;
        const int gend = a.G.start + a.G.points;
        const int t1 = t0 + PT < gend ? t0 + PT : gend;
        const int tl = t1 - 1;
        const size_t cbase = size_t(cond) * size_t(a.n);
        const int* whi = a.whi + cbase;
        const int* wlo = a.wlo + cbase;
        const int K = a.kc[kMaxCond + cond];  // the condition's core reach
        const int La = warp_search(whi, 0, int(a.n), t0 + 1, lane);
        const int Lb = warp_search(wlo, La, int(a.n), t1, lane);
        const int fs = warp_search(whi, La, Lb, t1, lane);
        const int Cb = warp_search(wlo, La, Lb, t0 + 1, lane);
        const int fe = Cb > fs ? Cb : fs;
        const int E = warp_search(mi, La, Lb, t0 - K, lane);
        const int Fc = warp_search(mi, E, Lb, tl + K + 1, lane);
        const LineShX* lsh = reinterpret_cast<const LineShX*>(a.lsh) + cbase;
        const float2* yp = a.cyp + cbase;
        const CoreIv* civ = a.civ + cbase;
        const size_t cell0 = size_t(cond) * size_t(a.ncell);
        const LineRuns runs =
            line_runs(a.chead + cell0, a.ncell, a.cshift, a.n, La, Lb, fs, fe, F[t0], F[tl], lane);

        const float t0f = float(t0);
        float2 acc[PT / 2];  // points 2 q, 2 q + 1
#pragma unroll
        for (int v = 0; v < PT / 2; ++v) acc[v] = f2(0.0f, 0.0f);
        double sum = 0.0;
        bool cored = false;  // the table holds something

        // Region-I constants of the line.
        struct R1 {
            float2 cy, d2, pc;
        };
        auto constants = [&](float2 v) {
            R1 r;
            r.cy = f2s(region1_cy(v.x));
            r.d2 = f2s(2.0f * v.x * v.x);
            r.pc = f2s(v.y * v.x);
            return r;
        };
        auto offsets = [&](float mj, const float4& s, int q) {
            const float2 d = __fadd2_rn(f2s(mj), f2(-float(2 * q), -float(2 * q + 1)));
            return __ffma2_rn(d, f2s(s.y), f2s(s.z));
        };
        // to += num / den for both halves, one reciprocal.
        auto add_pair = [&](float2 num, float2 den, float2& to) {
            const float rq = rcp_approx_f32(den.x * den.y);
            to = __ffma2_rn(num, __fmul2_rn(f2(den.y, den.x), f2s(rq)), to);
        };
        // One group of lines, region I only; MASK: some windows cover the tile
        // partly (or there are fewer than 32 lines).
        auto plain_group = [&](auto mask, float4 s, int2 win, float2 v) {
            const float mj = s.x - t0f;
            const unsigned wlen = unsigned(win.y - win.x);
            const int w0 = t0 - win.x;
            const R1 r = constants(v);
#pragma unroll
            for (int q = 0; q < PT / 2; ++q) {
                const float2 x = offsets(mj, s, q);
                const float2 u = __ffma2_rn(x, x, r.cy);
                float2 num = __ffma2_rn(u, r.pc, r.pc);
                if constexpr (decltype(mask)::value)
                    num = f2(unsigned(w0 + 2 * q) < wlen ? num.x : 0.0f, unsigned(w0 + 2 * q + 1) < wlen ? num.y : 0.0f);
                add_pair(num, __ffma2_rn(u, u, r.d2), acc[q]);
            }
        };
        // A group with wide lines: region I with a reciprocal per pair.
        auto solo_group = [&](float4 s, int2 win, float2 v, const CoreIv& iv) {
            const float mj = s.x - t0f;
            const unsigned wlen = unsigned(win.y - win.x);
            const int w0 = t0 - win.x, d15 = t0 - iv.lo15;
            const unsigned n15 = iv.lo15 <= iv.hi15 ? unsigned(iv.hi15 - iv.lo15) + 1u : 0u;
            const R1 r = constants(v);
#pragma unroll
            for (int q = 0; q < PT / 2; ++q) {
                const float2 x = offsets(mj, s, q);
                const float2 u = __ffma2_rn(x, x, r.cy);
                const float2 den = __ffma2_rn(u, u, r.d2);
                float2 num = __ffma2_rn(u, r.pc, r.pc);
                const int pa = 2 * q, pb = 2 * q + 1;
                if (!(unsigned(w0 + pa) < wlen) || unsigned(d15 + pa) < n15) num.x = 0.0f;
                if (!(unsigned(w0 + pb) < wlen) || unsigned(d15 + pb) < n15) num.y = 0.0f;
                acc[q] = __ffma2_rn(num, f2(rcp_approx_f32(den.x), rcp_approx_f32(den.y)), acc[q]);
            }
        };
        // A group of narrow lines with core candidates: region I or II chosen
        // per pair by the region intervals; the pairs of regions III and IV are
        // left to inner_pairs.
        auto core_group = [&](float4 s, int2 win, float2 v, const CoreIv& iv) {
            const float mj = s.x - t0f;
            const unsigned wlen = unsigned(win.y - win.x);
            const int w0 = t0 - win.x;
            // an interval's start relative to t0 and its length (empty: far off)
            const int d15 = iv.lo15 <= iv.hi15 ? t0 - iv.lo15 : -0x40000000;
            const int d55 = iv.lo55 <= iv.hi55 ? t0 - iv.lo55 : -0x40000000;
            const unsigned l15 = unsigned(iv.hi15 - iv.lo15), l55 = unsigned(iv.hi55 - iv.lo55);
            const unsigned n15 = iv.lo15 <= iv.hi15 ? l15 : 0u, n55 = iv.lo55 <= iv.hi55 ? l55 : 0u;
            const R1 r = constants(v);
            const float2 p1 = __fmul2_rn(r.pc, f2s(float(kW4A1 / kW4C)));
            const float2 p2 = __fmul2_rn(r.pc, f2s(float(kW4A2 / kW4C)));
#pragma unroll
            for (int q = 0; q < PT / 2; ++q) {
                const float2 x = offsets(mj, s, q);
                const float2 u = __ffma2_rn(x, x, r.cy);
                float2 den = __ffma2_rn(u, u, r.d2);
                float2 num = __ffma2_rn(u, r.pc, r.pc);
                // region II, v = u + 1/2 (r.d2 = 2 y^2)
                const float2 e1 = __fadd2_rn(u, f2s(float(0.5 - kW4B1)));
                const float2 e2 = __fadd2_rn(u, f2s(float(0.5 - kW4B2)));
                const float2 d1 = __ffma2_rn(e1, e1, __fmul2_rn(r.d2, f2s(float(2.0 * kW4B1))));
                const float2 d2 = __ffma2_rn(e2, e2, __fmul2_rn(r.d2, f2s(float(2.0 * kW4B2))));
                const float2 n1 = __ffma2_rn(u, p1, __fmul2_rn(p1, f2s(float(0.5 + kW4B1))));
                const float2 n2 = __ffma2_rn(u, p2, __fmul2_rn(p2, f2s(float(0.5 + kW4B2))));
                const float2 n = __ffma2_rn(n1, d2, __fmul2_rn(n2, d1));
                const float2 dd = __fmul2_rn(d1, d2);
                const int pa = 2 * q, pb = 2 * q + 1;
                const bool ca = unsigned(d15 + pa) <= n15, cb = unsigned(d15 + pb) <= n15;
                const bool ka = unsigned(w0 + pa) < wlen && !(unsigned(d55 + pa) <= n55);
                const bool kb = unsigned(w0 + pb) < wlen && !(unsigned(d55 + pb) <= n55);
                // (a pair left out enters the product as 1)
                num = f2(ka ? (ca ? n.x : num.x) : 0.0f, kb ? (cb ? n.y : num.y) : 0.0f);
                den = f2(ka ? (ca ? dd.x : den.x) : 1.0f, kb ? (cb ? dd.y : den.y) : 1.0f);
                add_pair(num, den, acc[q]);
            }
        };
        // The pairs jlo .. jhi of the line in the tile, a lane going over its own:
        // regions III and IV, or (`mixed`) regions by the intervals; whole lines: X
        // from the FP64 centre (beyond x = 1e18 region I is taken as 0).
        auto inner_pairs = [&](float4 s, float2 v, const CoreIv& iv, int i, int jlo, int jhi, bool mixed) {
            const bool whole = (__float_as_int(s.w) & kLineWhole) != 0;
            jlo = max(jlo, t0);
            jhi = min(jhi, tl);
            if (!__any_sync(0xffffffffu, jlo <= jhi)) return;
            cored = true;
            const double nu = whole ? lsh[i].nu : 0.0;
            const float y = v.x;
#pragma unroll 1
            for (int j = jlo; j <= jhi; ++j) {
                const float ax =
                    fabsf(whole ? float((nu - F[j]) / nu) * a.kx[cond] : fmaf(s.x - float(j), s.y, s.z));
                // (a line at nu = 0 in the GPU convention has infinite or NaN x, y
                // and pref: the pair is left out, not multiplied by 0)
                if (!(ax < 1.0e18f)) continue;
                float wf;
                if (!mixed || (j >= iv.lo55 && j <= iv.hi55)) {
                    wf = float(1.0 / kW4C) *
                         ((y >= fmaf(0.195f, ax, -0.176f)) ? w4_region3_re_f32(ax, y) : w4_region4_re_f32(ax, y));
                } else if (j >= iv.lo15 && j <= iv.hi15) {
                    wf = w4_region2_c(ax, y);
                } else {
                    // (u + 1) / (u^2 + 2 y^2) is 1 / u to FP32 rounding from u = 1e12
                    // on (2 y^2 < u there), and u^2 overflows from 1.8e19
                    const float u = fmaf(ax, ax, region1_cy(y));
                    const float rat = u > 1.0e12f ? rcp_approx_f32(u)
                                                  : (u + 1.0f) * rcp_approx_f32(fmaf(u, u, 2.0f * y * y));
                    wf = y * rat;
                }
                T[j - t0][lane] += v.y * wf;
            }
            __syncwarp();
        };
        // The lanes' partial sums, into point lane / SUB.
        auto fold = [&]() {
            float s[PT];
#pragma unroll
            for (int v = 0; v < PT / 2; ++v) {
                s[2 * v] = acc[v].x;
                s[2 * v + 1] = acc[v].y;
                acc[v] = f2(0.0f, 0.0f);
            }
            Sum::sum(s, lane);
            sum += double(s[0]);
            if (cored) {
                cored = false;
                __syncwarp();
                double t = 0.0;
#pragma unroll 4
                for (int q = 0; q < 32; q += SUB) t += double(T[lane / SUB][q + lane % SUB]);
                sum += sum_neighbours<SUB>(t);
                __syncwarp();
#pragma unroll 4
                for (int q = 0; q < PT; ++q) T[q][lane] = 0.0f;
            }
        };

        const int ngroups = runs.groups_of(a.splits, split);
        auto gstart = [&](int gi, int& end) {
            long e;
            const int b = int(runs.start(split + gi * a.splits, e));
            end = int(e);
            return b;
        };
        auto issue = [&](int gi) {
            if (gi < ngroups) {
                int end;
                const int b = gstart(gi, end), at = (gi & 1) * 32 + lane;
                if (b + lane < end) {
                    cp_async16(lsb + at, lsh + b + lane);
                    cp_async8(lhb + at, &lsh[b + lane].lo);
                    cp_async8(ypb + at, yp + b + lane);
                }
            }
            cp_async_commit();
        };
        issue(0);
        for (int gi = 0; gi < ngroups; ++gi) {
            issue(gi + 1);
            cp_async_wait<1>();
            // (each lane reads only what it copied)
            int end;
            const int gb = gstart(gi, end);
            const int ge = end - gb < 32 ? end : gb + 32;
            float4 s = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(0));  // a line that adds nothing
            int2 win = make_int2(0, 0);
            float2 v = f2(1.0f, 0.0f);
            const bool live = gb + lane < ge;
            if (live) {
                const int at = (gi & 1) * 32 + lane;
                s = lsb[at];
                win = lhb[at];
                v = ypb[at];
            }
            const bool odd = __any_sync(0xffffffffu, (__float_as_int(s.w) & (kLineWhole | kLineWide)) != 0);
            // (the reach is the widest of the whole list: the group's own
            // intervals decide)
            CoreIv iv = {1, 0, 1, 0};
            bool core = odd;
            if (odd || (ge > E && gb < Fc)) {
                if (live) iv = civ[gb + lane];
                core = __any_sync(0xffffffffu, odd || (iv.lo15 <= tl && iv.hi15 >= t0 && iv.lo15 <= iv.hi15));
            }
            if (core) {
                if (!odd) {
                    core_group(s, win, v, iv);
                    inner_pairs(s, v, iv, gb + lane, iv.lo55, iv.hi55, false);
                } else if (__any_sync(0xffffffffu, (__float_as_int(s.w) & kLineWhole) != 0)) {
                    inner_pairs(s, v, iv, gb + lane, win.x, win.y - 1, true);
                } else {
                    solo_group(s, win, v, iv);
                    inner_pairs(s, v, iv, gb + lane, iv.lo15, iv.hi15, true);
                }
            } else if (gb >= fs && ge <= fe && ge - gb == 32) {
                plain_group(std::false_type(), s, win, v);
            } else {
                plain_group(std::true_type(), s, win, v);
            }
            if ((gi & 3) == 3) fold();
        }
        cp_async_wait<0>();
        fold();

        const int jj = t0 + lane / SUB;
        if (runs.fa < runs.fb || runs.fc < runs.fd) {
            double far = 0.0;
            add_far_cells<kCellTermsMixed, SUB>(a.chead + cell0, a.cmom + cell0 * kCellTermsMixed, runs, a.splits, split,
                                                kCellBitsMixed, F[t0], F[tl], F[min(jj, tl)], far, lane, lane % SUB);
            sum += sum_neighbours<SUB>(far);
        }
        if (lane % SUB == 0 && jj < t1) put_result(a, cond, split, jj, sum);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// FP64 single-condition step two on narrow tiles, lane = line.
//
// As k_steptwo_near: a warp takes a tile of PT points and 32 lines at a time,
// each lane evaluating its own line (80-byte record, staged; a lane's reads of
// its record are conflict-free at that stride) at the tile's points, whose grid
// values are read from shared memory.  Groups without core candidates add
// region I into PT accumulators; groups with core candidates go over the points
// in a loop, choosing the region per pair with the reference's own test on x
// and y, into a per-warp table with a column per lane.  At the end the lanes'
// sums are added up by halving exchanges.  PT = 8: coarse
// grids over dense lists, where a 32-point tile is wider than the near zone.
//
// Bound by issue slots and the FP64 pipe (50 and 34 % at 1e6 lines): 8 FP64
// operations and about 4 others per region-I pair.  B200, 1e7 lines, 7.5e5 points with cells: 4.0
// ms, with 32-point tiles 5.1 (64 more registers); the point-parallel kernel needed
// 7.0, 26 % of the FP64 pipe and three other instructions for each FP64 one.  16
// warps per SM (128 registers): 20 spill and take 4.15 ms.
// ---------------------------------------------------------------------------
template <int PT>
constexpr size_t near64_warp_smem() {
    return 64 * sizeof(RecV64) + sizeof(double) * PT * kCoreRow64 + sizeof(double) * PT;
}

template <int PT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS) k_steptwo_near64(StepArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    constexpr int SUB = 32 / PT;        // lanes to a point where lanes stand for points
    using Sum = Halving<PT, 1, double>;  // lane ends with point lane / SUB
    unsigned char* const mine = smem_raw + size_t(threadIdx.x >> 5) * near64_warp_smem<PT>();
    RecV64* buf = reinterpret_cast<RecV64*>(mine);
    double (*T)[kCoreRow64] = reinterpret_cast<double (*)[kCoreRow64]>(mine + 64 * sizeof(RecV64));
    double* fj = &T[PT][0];  // the tile's grid values
    const double* F = a.G.freq;
    const int* mi = a.mi;
#pragma unroll 4
    for (int q = 0; q < PT; ++q) T[q][lane] = 0.0;

    for (;;) {
        int item = 0;
        if (lane == 0) item = int(atomicAdd(a.counter, 1u));
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.n_items) break;
        const int per_cond = a.tiles_per_cond * a.splits;
        const int c = item / per_cond;
        const int tile = (item - c * per_cond) / a.splits;
        const int split = item - c * per_cond - tile * a.splits;
        const int t0 = a.G.start + tile * PT;
        const int gend = a.G.start + a.G.points;
        const int t1 = t0 + PT < gend ? t0 + PT : gend;
        const int tl = t1 - 1;
        const size_t cbase = size_t(c) * size_t(a.n);
        const int* whi = a.whi + cbase;
        const int* wlo = a.wlo + cbase;
        const int kc = a.kc[c];
        const int La = warp_search(whi, 0, int(a.n), t0 + 1, lane);
        const int Lb = warp_search(wlo, La, int(a.n), t1, lane);
        const int fs = warp_search(whi, La, Lb, t1, lane);
        const int Cb = warp_search(wlo, La, Lb, t0 + 1, lane);
        const int fe = Cb > fs ? Cb : fs;
        const int E = warp_search(mi, La, Lb, t0 - kc, lane);
        const int Fc = warp_search(mi, E, Lb, tl + kc + 1, lane);
        const RecV64* recs = reinterpret_cast<const RecV64*>(a.rec) + cbase;
        const size_t cell0 = size_t(c) * size_t(a.ncell);
        const LineRuns runs =
            line_runs(a.chead + cell0, a.ncell, a.cshift, a.n, La, Lb, fs, fe, F[t0], F[tl], lane);

        if (lane < PT) fj[lane] = F[min(t0 + lane, tl)];
        double acc[PT];
#pragma unroll
        for (int p = 0; p < PT; ++p) acc[p] = 0.0;
        bool cored = false;  // the table holds something
        __syncwarp();

        // One group of lines, region I only; MASK: some windows cover the tile
        // partly (or there are fewer than 32 lines).
        auto plain_group = [&](auto mask, const RecV64& r, int w0, unsigned wlen) {
            const double nu = r.nu, g = r.g, Cy = r.Cy, D2 = r.D2, Pc = r.Pc;
#pragma unroll
            for (int p = 0; p < PT; ++p) {
                const double xs = (nu - fj[p]) * g;
                const double u = fma(xs, xs, Cy);
                double rr = rcp_refined_f64(fma(u, u, D2));
                if constexpr (decltype(mask)::value) rr = unsigned(w0 + p) < wlen ? rr : 0.0;
                acc[p] = fma(fma(u, Pc, Pc), rr, acc[p]);
            }
        };
        // A group whose core bands reach the tile, two points at a time.  x, y
        // and the region choice are the reference's.
        auto core_group = [&](const RecV64& r, int w0, unsigned wlen) {
            const double nu = r.nu, g = r.g, Cy = r.Cy, D2 = r.D2, Pc = r.Pc, y = r.y, pref = r.pref;
            const Region2F64 region2(y, pref);
            cored = true;
#pragma unroll 1
            for (int p0 = 0; p0 < PT; p0 += 2) {
                double ax[2], sx[2], u[2], v[2];
                bool in[2], core[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double xs = (nu - fj[p0 + h]) * g;
                    ax[h] = fabs(xs);
                    sx[h] = ax[h] + y;
                    u[h] = fma(xs, xs, Cy);
                    in[h] = unsigned(w0 + p0 + h) < wlen;
                    core[h] = in[h] && sx[h] < 15.0;
                    v[h] = 0.0;
                }
                if (__any_sync(0xffffffffu, (in[0] && !core[0]) || (in[1] && !core[1]))) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const double rr = rcp_refined_f64(fma(u[h], u[h], D2));
                        v[h] = in[h] && !core[h] ? fma(u[h], Pc, Pc) * rr : 0.0;
                    }
                }
                if (__any_sync(0xffffffffu, core[0] || core[1])) {
                    const bool c0 = core[0] && sx[0] < 5.5, c1 = core[1] && sx[1] < 5.5;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const double w = region2(u[h]);
                        if (core[h] && sx[h] >= 5.5) v[h] = w;
                    }
                    if (__any_sync(0xffffffffu, c0 || c1)) {
#pragma unroll 1
                        for (int h = 0; h < 2; ++h) {
                            if (!(h ? c1 : c0)) continue;
                            const double x = h ? ax[1] : ax[0];
                            const double w = pref * (y >= 0.195 * x - 0.176 ? w4_region3_re_f64(x, y) : w4_region4_re_f64(x, y));
                            if (h) v[1] = w;
                            else v[0] = w;
                        }
                    }
                }
                T[p0][lane] += v[0];
                T[p0 + 1][lane] += v[1];
            }
        };

        const int ngroups = runs.groups_of(a.splits, split);
        auto gstart = [&](int gi, int& end) {
            long e;
            const int b = int(runs.start(split + gi * a.splits, e));
            end = int(e);
            return b;
        };
        auto issue = [&](int gi) {
            if (gi < ngroups) {
                int end;
                const int b = gstart(gi, end);
                stage(buf + (gi & 1) * 32, recs + b, min(end - b, 32), lane);
            }
            cp_async_commit();
        };
        issue(0);
        for (int gi = 0; gi < ngroups; ++gi) {
            issue(gi + 1);
            cp_async_wait<1>();
            __syncwarp();
            int end;
            const int gb = gstart(gi, end);
            const int cnt = min(end - gb, 32);
            // (a lane past the group's end takes its last line, outside every
            // window)
            const RecV64& r = buf[(gi & 1) * 32 + min(lane, cnt - 1)];
            const int w0 = t0 - r.lo;
            const unsigned wlen = lane < cnt ? unsigned(r.hi - r.lo) : 0u;
            // (kc is the widest band of the whole list: the group's own decide)
            const bool core = gb + cnt > E && gb < Fc && __any_sync(0xffffffffu, r.clo <= tl && r.chi >= t0);
            if (core) core_group(r, w0, wlen);
            else if (gb >= fs && gb + cnt <= fe && cnt == 32) plain_group(std::false_type(), r, w0, wlen);
            else plain_group(std::true_type(), r, w0, wlen);
            __syncwarp();
        }
        cp_async_wait<0>();
        // point lane / SUB, the lanes' sums by halving exchanges
        Sum::sum(acc, lane);
        double sum = acc[0];
        if (cored) {
            __syncwarp();
            double t = 0.0;
#pragma unroll 8
            for (int q = 0; q < 32; q += SUB) t += T[lane / SUB][q + lane % SUB];
            sum += sum_neighbours<SUB>(t);
            __syncwarp();
#pragma unroll 4
            for (int q = 0; q < PT; ++q) T[q][lane] = 0.0;
        }
        const int jj = t0 + lane / SUB;
        if (runs.fa < runs.fb || runs.fc < runs.fd) {
            double far = 0.0;
            add_far_cells<kCellTerms64, SUB>(a.chead + cell0, a.cmom + cell0 * kCellTerms64, runs, a.splits, split,
                                             kCellBits64, F[t0], F[tl], F[min(jj, tl)], far, lane, lane % SUB);
            sum += sum_neighbours<SUB>(far);
        }
        if (lane % SUB == 0 && jj < t1) put_result(a, c, split, jj, sum);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Step two, Doppler and Gaussian (bin-integrated erf differences, FP64).
//
// A line reaches a dozen points or so (the rest of its window adds exactly 0),
// so a lane per point idles most lanes.  The (line, point) pairs of 32 lines and
// the tile are numbered through instead (a prefix sum of the lines' points in the
// tile) and taken 32 at a time, a pair per lane, each lane finding its line by a
// search over the prefix sums.  Lanes l and l + 16 add to column l of a per-warp
// table, one after the other; at the end each lane adds up its points' rows: a
// fixed order.  Bound by erf (two per pair, about 40 FP64 operations each; issue
// slots 69 %, FP64 pipe 43 %).
// B200, 1e6 lines on 1e6 points (12 pairs per line): 200 us, 421 with a lane per
// point.
// ---------------------------------------------------------------------------
constexpr int kErfCols = 16;
template <int P>
constexpr size_t erf_warp_smem() {
    return 64 * sizeof(RecE64) + sizeof(double) * 32 * P * (kErfCols + 1);
}

template <int KIND, int CONV, int P, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_steptwo_erf(StepArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    unsigned char* const mine = smem_raw + size_t(threadIdx.x >> 5) * erf_warp_smem<P>();
    RecE64* buf = reinterpret_cast<RecE64*>(mine);
    double (*T)[kErfCols + 1] = reinterpret_cast<double (*)[kErfCols + 1]>(mine + 64 * sizeof(RecE64));
    const RecE64* recs_all = reinterpret_cast<const RecE64*>(a.rec);
    const double* F = a.G.freq;
    auto clear = [&]() {
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
            for (int q = 0; q < kErfCols; ++q) T[lane + 32 * p][q] = 0.0;
        __syncwarp();
    };
    clear();

    WorkItem w;
    while (next_item(a, P, lane, w)) {
        const size_t cbase = size_t(w.c) * size_t(a.n);
        const int* whi = a.whi + cbase;
        const int* wlo = a.wlo + cbase;
        const int t0 = w.t0, t1 = w.t1;
        const long La = warp_lower_bound(0, a.n, lane, [&](long i) { return whi[i] > t0; });
        const long Lb = warp_lower_bound(La, a.n, lane, [&](long i) { return wlo[i] >= t1; });
        const RecE64* recs = recs_all + cbase;
        // this item's groups of 32 lines: gi-th starts at La + 32 (s + gi S)
        const int ngroups = split_groups(Lb - La, a.splits, w.s);
        auto gstart = [&](int gi) { return La + 32L * (w.s + long(gi) * a.splits); };
        if (ngroups > 0) {
            const long b = gstart(0);
            stage(buf, recs + b, int(Lb - b < 32 ? Lb - b : 32), lane);
            cp_async_commit();
        }
        for (int gi = 0; gi < ngroups; ++gi) {
            if (gi + 1 < ngroups) {
                const long b = gstart(gi + 1);
                const long rem = Lb - b;
                stage(buf + ((gi + 1) & 1) * 32, recs + b, int(rem < 32 ? rem : 32), lane);
                cp_async_commit();
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncwarp();
            const RecE64* R = buf + (gi & 1) * 32;
            const long gbase = gstart(gi);
            const int cnt = int(Lb - gbase < 32 ? Lb - gbase : 32);
            // this lane's line's points in the tile, and their prefix sum
            int pts = 0;
            if (lane < cnt) pts = max(0, min(R[lane].hi, t1) - max(R[lane].lo, t0));
            int incl = pts;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            for (int base = 0; base < total; base += 32) {
                const int q = base + lane;
                // the line of pair q: the number of lines whose pairs end at or
                // before it
                int line = 0;
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1)
                    if (__shfl_sync(0xffffffffu, incl, line + o - 1) <= q) line += o;
                line = min(line, 31);
                const int first = __shfl_sync(0xffffffffu, incl - pts, line);
                double v = 0.0;
                int row = 0;
                const bool live = q < total;
                if (live) {
                    const double2* rq = reinterpret_cast<const double2*>(&R[line]);
                    const double2 v0 = rq[0], v1 = rq[1];
                    const double nu = v0.x, S = v0.y, g = v1.x;
                    const int j = max(R[line].lo, t0) + (q - first);
                    row = j - t0;
                    const double fj = F[j];
                    double xp, xm;
                    if (KIND == kDoppler) {
                        // cross_kernal.cu:684-698 (GPU), OpenMPManager.cpp:165-170 (CPU)
                        const double d = (CONV == kConvGpu) ? nu - fj : fabs(nu - fj);
                        xp = g * ((d) + a.x0);
                        xm = g * ((d) - a.x0);
                    } else {
                        // Gaussian erf bin with dnu = f - nu (cross_kernal.cu:599-609)
                        const double d = fj - nu;
                        xp = a.xg * (d) + a.x0g;
                        xm = a.xg * (d) - a.x0g;
                    }
                    v = S * (erf(xp) - erf(xm));
                }
                if (live && lane < kErfCols) T[row][lane] += v;
                __syncwarp();
                if (live && lane >= kErfCols) T[row][lane - kErfCols] += v;
                __syncwarp();
            }
        }
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const int jj = t0 + lane + 32 * p;
            double sum = 0.0;
#pragma unroll
            for (int q = 0; q < kErfCols; ++q) sum += T[lane + 32 * p][q];
            if (jj < t1) put_result(a, w.c, w.s, jj, sum);
        }
        clear();
    }
}

// ---------------------------------------------------------------------------
// Sampled FP64 re-evaluation (mixed-precision error statement).
// ---------------------------------------------------------------------------
__global__ void k_check_snapshot(CheckArgs a) {
    const int c = blockIdx.y, k = blockIdx.x, lane = threadIdx.x;
    const int j = a.rows[k] + lane;
    const bool in = j < a.G.start + a.G.points;
    a.before[(size_t(c) * a.nrows + k) * 32 + lane] =
        in ? a.out[size_t(a.row[c]) * a.out_stride + size_t(j)] : 0.0;
}

// One warp per (sampled row, condition).  The lines whose window may meet the
// row are taken 32 at a time, lane = line: each lane computes its line's
// intensity, widths and window in FP64 as step one does for the FP64 path
// (cross_kernal.cu:758-790 / OpenMPManager.cpp:183-208); then, line by line
// in order, every lane adds the line's W4 value at its own point (the
// reference's region choice, w4_re) when the point lies in the line's window.
template <int CONV>
__global__ void __launch_bounds__(32) k_check_rows(CheckArgs a) {
    const int k = blockIdx.x, c = blockIdx.y, lane = threadIdx.x;
    const CondDev& C = a.cond[c];
    const double* F = a.G.freq;
    const double f0 = F[0], df = a.G.df;
    const int s = a.G.start, e = a.G.start + a.G.points;
    const int t0 = a.rows[k];
    const int t1 = t0 + 32 < e ? t0 + 32 : e;
    const int j = t0 + lane;
    const bool mine = j < t1;
    const double fj = F[mine ? j : t1 - 1];
    const double cut = C.cut;
    // lines with nu in [F[t0] - cut - 2 df, F[t1 - 1] + cut + 2 df]
    const double lo_nu = F[t0] - cut - 2.0 * df, hi_nu = F[t1 - 1] + cut + 2.0 * df;
    const long La = warp_lower_bound(0, a.L.n, lane, [&](long i) { return a.L.nu[i] >= lo_nu; });
    const long Lb = warp_lower_bound(La, a.L.n, lane, [&](long i) { return a.L.nu[i] > hi_nu; });
    double acc = 0.0;
    for (long b = La; b < Lb; b += 32) {
        const long i = b + lane;
        double nu_p = 0.0, g = 0.0, y = 0.0, pref = 0.0;
        int ib = 0, ie = 0;
        if (i < Lb) {
            const double nu = a.L.nu[i];
            const double ei = a.L.energies[i], aif = a.L.aif[i], gns = double(a.L.gns[i]);
            double nu_if = nu;
            if (nu_if == 0) nu_if = 1e-6;
            double S = C.cmcoef * aif * gns * kISQRTPI * exp(-C.beta * ei) *
                       (1.0 - exp(-C.beta * nu_if)) / (nu_if * nu_if * C.partition);
            if (CONV == kConvGpu && gns == -1) S = aif;
            nu_p = CONV == kConvGpu ? nu : nu_if;
            const double gl = a.L.gamma[i] * C.gamma_scale * pow(C.tratio, a.L.nexp[i]);
            g = 1.0 / (nu_p * C.dpw);
            y = gl * g;
            pref = (CONV == kConvCpu && S == 0.0) ? 0.0 : S * g;
            if (CONV == kConvCpu) {
                const double rb = round((nu_if - cut - f0) / df);
                const double re = round((nu_if + cut - f0) / df);
                ib = clamp_index(rb > double(s) ? rb : double(s), s, e);
                ie = clamp_index(re < double(e) ? re : double(e), s, e);
            }
        }
        const int cnt = Lb - b < 32 ? int(Lb - b) : 32;
        for (int t = 0; t < cnt; ++t) {
            const double lnu = __shfl_sync(0xffffffffu, nu_p, t);
            const double lg = __shfl_sync(0xffffffffu, g, t);
            const double ly = __shfl_sync(0xffffffffu, y, t);
            const double lp = __shfl_sync(0xffffffffu, pref, t);
            const int lib = __shfl_sync(0xffffffffu, ib, t);
            const int lie = __shfl_sync(0xffffffffu, ie, t);
            const double d = lnu - fj;
            const bool in = CONV == kConvGpu ? (!(d > cut) && !(d < -cut)) : (j >= lib && j < lie);
            if (mine && in) acc += lp * w4_re(d * lg, ly);
        }
    }
    a.ref[(size_t(c) * a.nrows + k) * 32 + lane] = mine ? acc : 0.0;
}

// Per condition: the comparison of what the call added at the sampled
// points (out after minus out before) with the FP64 sums.
__global__ void __launch_bounds__(32) k_check_stats(CheckArgs a) {
    const int c = blockIdx.x, lane = threadIdx.x;
    const int e = a.G.start + a.G.points;
    double peak = 0.0;
    for (int k = 0; k < a.nrows; ++k) {
        const double r = a.ref[(size_t(c) * a.nrows + k) * 32 + lane];
        peak = fmax(peak, fabs(r));
    }
    for (int o = 16; o > 0; o >>= 1) peak = fmax(peak, __shfl_xor_sync(0xffffffffu, peak, o));
    double mx = 0.0, sr = 0.0, sd = 0.0;
    for (int k = 0; k < a.nrows; ++k) {
        const int j = a.rows[k] + lane;
        if (j >= e) continue;
        const size_t q = (size_t(c) * a.nrows + k) * 32 + lane;
        const double r = a.ref[q];
        const double got = a.out[size_t(a.row[c]) * a.out_stride + size_t(j)] - a.before[q];
        if (fabs(r) > 1e-6 * peak) mx = fmax(mx, fabs(got - r) / fabs(r));
        sr += r;
        sd += got - r;
    }
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        sd += __shfl_xor_sync(0xffffffffu, sd, o);
    }
    if (lane == 0) {
        a.stats[4 * c + 0] = mx;
        a.stats[4 * c + 1] = sr;
        a.stats[4 * c + 2] = sd;
        a.stats[4 * c + 3] = peak;
    }
}

// Sums the parts of split tiles in part order and adds them to out.
__global__ void k_reduce_splits(StepArgs a, int ncond_out) {
    const long i = long(blockIdx.x) * blockDim.x + threadIdx.x;
    const long pts = a.G.points;
    if (i >= pts * ncond_out) return;
    const int c = int(i / pts);
    const long j = i - long(c) * pts;
    const double* p = a.part + size_t(c) * a.splits * a.part_stride + size_t(j);
    double v = 0.0;
    for (int s = 0; s < a.splits; ++s) v += p[size_t(s) * a.part_stride];
    a.out[size_t(a.row[c]) * a.out_stride + size_t(a.G.start + j)] += v;
}

template <class K>
int blocks_per_sm(K kernel, int threads, size_t smem) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess)
        return 1;
    return n > 0 ? n : 1;
}

template <class K>
cudaError_t run_group_kernel(K kernel, int threads, size_t smem, int blocks, const StepArgs& a, cudaStream_t st,
                             int* occ) {
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess)
        return cudaGetLastError();
    if (occ) {
        *occ = blocks_per_sm(kernel, threads, smem);
        return cudaSuccess;
    }
    kernel<<<blocks, threads, smem, st>>>(a);
    return cudaGetLastError();
}

template <int P, int WARPS, bool MIXED>
cudaError_t run_voigt(int blocks, const StepArgs& a, cudaStream_t st, int* occ) {
    const size_t smem = size_t(WARPS) * voigt_warp_smem(MIXED);
    if (smem > 48 * 1024) {
        if (cudaFuncSetAttribute(k_steptwo_voigt<P, WARPS, MIXED>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess)
            return cudaGetLastError();
    }
    if (occ) {
        *occ = blocks_per_sm(k_steptwo_voigt<P, WARPS, MIXED>, WARPS * 32, smem);
        return cudaSuccess;
    }
    k_steptwo_voigt<P, WARPS, MIXED><<<blocks, WARPS * 32, smem, st>>>(a);
    return cudaGetLastError();
}

template <int C, int WARPS, int LS, bool MIXED>
cudaError_t run_group(int blocks, const StepArgs& a, cudaStream_t st, int* occ) {
    if constexpr (MIXED)
        return run_group_kernel(k_steptwo_voigt_mcx<C, WARPS, LS>, WARPS * 32, size_t(WARPS) * mcx_warp_smem<C>(),
                                blocks, a, st, occ);
    else
        return run_group_kernel(k_steptwo_voigt_mc<C, WARPS, LS>, WARPS * 32,
                                size_t(WARPS) * 64 * (sizeof(LineSh64) + C * sizeof(CondRec64)), blocks, a, st, occ);
}

// Rows of 32 or 8 points (FP64: one point per lane, mixed: two).
template <int C, int WARPS, bool MIXED>
cudaError_t dispatch_mc_ls(int row, int blocks, const StepArgs& a, cudaStream_t st, int* occ) {
    if (row == 32) return run_group<C, WARPS, MIXED ? 2 : 1, MIXED>(blocks, a, st, occ);
    if (row == 8) return run_group<C, WARPS, MIXED ? 8 : 4, MIXED>(blocks, a, st, occ);
    return cudaErrorInvalidValue;
}

template <int WARPS, bool MIXED>
cudaError_t dispatch_mc_c(int C, int row, int blocks, const StepArgs& a, cudaStream_t st, int* occ) {
    switch (C) {
        case 2: return dispatch_mc_ls<2, WARPS, MIXED>(row, blocks, a, st, occ);
        case 4: return dispatch_mc_ls<4, WARPS, MIXED>(row, blocks, a, st, occ);
        case 8: return dispatch_mc_ls<8, WARPS, MIXED>(row, blocks, a, st, occ);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t dispatch_mc(bool mixed, int C, int warps, int row, int blocks, const StepArgs& a,
                        cudaStream_t st, int* occ) {
    if (warps == 4) return mixed ? dispatch_mc_c<4, true>(C, row, blocks, a, st, occ)
                                 : dispatch_mc_c<4, false>(C, row, blocks, a, st, occ);
    if (warps == 8) return mixed ? dispatch_mc_c<8, true>(C, row, blocks, a, st, occ)
                                 : dispatch_mc_c<8, false>(C, row, blocks, a, st, occ);
    return cudaErrorInvalidValue;
}

template <int KIND, int CONV, int P, int WARPS>
cudaError_t run_erf(int blocks, const StepArgs& a, cudaStream_t st, int* occ) {
    return run_group_kernel(k_steptwo_erf<KIND, CONV, P, WARPS>, WARPS * 32, size_t(WARPS) * erf_warp_smem<P>(), blocks,
                            a, st, occ);
}

template <int WARPS, bool MIXED>
cudaError_t dispatch_voigt_p(int P, int blocks, const StepArgs& a, cudaStream_t st, int* occ) {
    switch (P) {
        case 1: return run_voigt<1, WARPS, MIXED>(blocks, a, st, occ);
        case 2: return run_voigt<2, WARPS, MIXED>(blocks, a, st, occ);
        case 4: return run_voigt<4, WARPS, MIXED>(blocks, a, st, occ);
        case 8: return run_voigt<8, WARPS, MIXED>(blocks, a, st, occ);
        default: return cudaErrorInvalidValue;
    }
}

template <int KIND, int CONV, int WARPS>
cudaError_t dispatch_erf_p(int P, int blocks, const StepArgs& a, cudaStream_t st, int* occ) {
    switch (P) {
        case 1: return run_erf<KIND, CONV, 1, WARPS>(blocks, a, st, occ);
        case 2: return run_erf<KIND, CONV, 2, WARPS>(blocks, a, st, occ);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t dispatch_steptwo(int kind, int conv, bool mixed, int P, int warps, int blocks,
                             const StepArgs& a, cudaStream_t st, int* occ) {
    if (kind == kVoigt) {
        if (warps == 4) return mixed ? dispatch_voigt_p<4, true>(P, blocks, a, st, occ)
                                     : dispatch_voigt_p<4, false>(P, blocks, a, st, occ);
        if (warps == 8) return mixed ? dispatch_voigt_p<8, true>(P, blocks, a, st, occ)
                                     : dispatch_voigt_p<8, false>(P, blocks, a, st, occ);
        return cudaErrorInvalidValue;
    }
    if (warps != 4 && warps != 8) return cudaErrorInvalidValue;
    if (kind == kDoppler) {
        if (conv == kConvGpu)
            return warps == 4 ? dispatch_erf_p<kDoppler, kConvGpu, 4>(P, blocks, a, st, occ)
                              : dispatch_erf_p<kDoppler, kConvGpu, 8>(P, blocks, a, st, occ);
        return warps == 4 ? dispatch_erf_p<kDoppler, kConvCpu, 4>(P, blocks, a, st, occ)
                          : dispatch_erf_p<kDoppler, kConvCpu, 8>(P, blocks, a, st, occ);
    }
    if (kind == kGauss)
        return warps == 4 ? dispatch_erf_p<kGauss, kConvGpu, 4>(P, blocks, a, st, occ)
                          : dispatch_erf_p<kGauss, kConvGpu, 8>(P, blocks, a, st, occ);
    return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_grid_check(const GridDev& g, unsigned* err, int* kc, unsigned* counter, cudaStream_t stream) {
    if (g.npoints_total < 2 && !kc) return cudaSuccess;
    const int n = g.npoints_total > 2 ? g.npoints_total - 1 : 1;
    k_grid_check<<<(n + 255) / 256, 256, 0, stream>>>(g, err, kc, counter);
    return cudaGetLastError();
}

cudaError_t launch_check_snapshot(const CheckArgs& a, cudaStream_t stream) {
    if (a.nrows <= 0 || a.ncond <= 0) return cudaSuccess;
    k_check_snapshot<<<dim3(unsigned(a.nrows), unsigned(a.ncond)), 32, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_check_rows(const CheckArgs& a, cudaStream_t stream) {
    if (a.nrows <= 0 || a.ncond <= 0) return cudaSuccess;
    const dim3 grid(unsigned(a.nrows), unsigned(a.ncond));
    if (a.conv == kConvGpu) k_check_rows<kConvGpu><<<grid, 32, 0, stream>>>(a);
    else k_check_rows<kConvCpu><<<grid, 32, 0, stream>>>(a);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    k_check_stats<<<unsigned(a.ncond), 32, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_reduce_splits(const StepArgs& a, int ncond_out, cudaStream_t stream) {
    if (a.splits <= 1 || a.G.points <= 0 || ncond_out <= 0) return cudaSuccess;
    const long n = long(a.G.points) * ncond_out;
    k_reduce_splits<<<unsigned((n + 255) / 256), 256, 0, stream>>>(a, ncond_out);
    return cudaGetLastError();
}

cudaError_t launch_prep(int kind, int conv, bool mixed, const PrepArgs& a, cudaStream_t stream) {
    const long count = (a.line1 > 0 ? a.line1 : a.L.n) - a.line0;
    if (count <= 0 || a.ncond <= 0) return cudaSuccess;
    const dim3 grid(unsigned((count + 255) / 256), unsigned(a.ncond));
    if (kind == kVoigt && mixed && a.group > 1) {
        // (precomputed-intensity lists run one condition at a time)
        if (a.L.s32 != nullptr || a.ncond % a.group != 0) return cudaErrorInvalidValue;
        const unsigned nblk = unsigned((count + 255) / 256);
        const int ncache = a.nclass <= kMaxClassCache ? a.nclass : 0;
        const size_t smem = sizeof(double) * 3 * size_t(ncache) * 256;
        auto go = [&](auto kernel) {
            // (the kernel's static arrays count against the 48 KB that need no
            // attribute: 8 classes are exactly 48 KB without them)
            if (smem + sizeof(int) * 2 * kMaxCond * 8 > 48 * 1024 &&
                cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess)
                return cudaGetLastError();
            kernel<<<nblk, 256, smem, stream>>>(a);
            return cudaGetLastError();
        };
        switch (a.group) {
            case 2: return conv == kConvGpu ? go(k_prep_lines_x<kConvGpu, 2>) : go(k_prep_lines_x<kConvCpu, 2>);
            case 4: return conv == kConvGpu ? go(k_prep_lines_x<kConvGpu, 4>) : go(k_prep_lines_x<kConvCpu, 4>);
            case 8: return conv == kConvGpu ? go(k_prep_lines_x<kConvGpu, 8>) : go(k_prep_lines_x<kConvCpu, 8>);
            default: return cudaErrorInvalidValue;
        }
    } else if (kind == kVoigt) {
        if (conv == kConvGpu) {
            if (mixed) k_prep<kVoigt, kConvGpu, true><<<grid, 256, 0, stream>>>(a);
            else k_prep<kVoigt, kConvGpu, false><<<grid, 256, 0, stream>>>(a);
        } else {
            if (mixed) k_prep<kVoigt, kConvCpu, true><<<grid, 256, 0, stream>>>(a);
            else k_prep<kVoigt, kConvCpu, false><<<grid, 256, 0, stream>>>(a);
        }
    } else if (kind == kDoppler) {
        if (conv == kConvGpu) k_prep<kDoppler, kConvGpu, false><<<grid, 256, 0, stream>>>(a);
        else k_prep<kDoppler, kConvCpu, false><<<grid, 256, 0, stream>>>(a);
    } else if (kind == kGauss) {
        k_prep<kGauss, kConvGpu, false><<<grid, 256, 0, stream>>>(a);
    } else {
        return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_steptwo(int kind, int conv, bool mixed, int P, int warps, int blocks,
                           const StepArgs& a, cudaStream_t stream) {
    if (blocks <= 0 || a.n_items <= 0) return cudaSuccess;
    return dispatch_steptwo(kind, conv, mixed, P, warps, blocks, a, stream, nullptr);
}

int steptwo_blocks_per_sm(int kind, int conv, bool mixed, int P, int warps) {
    StepArgs dummy{};
    int occ = 0;
    if (dispatch_steptwo(kind, conv, mixed, P, warps, 0, dummy, nullptr, &occ) != cudaSuccess)
        return 0;
    return occ;
}

cudaError_t launch_core_v32(const StepArgs& a, int ncond, cudaStream_t stream) {
    if (a.n <= 0 || a.G.points <= 0 || ncond <= 0) return cudaSuccess;
    constexpr int W = 4;
    const int rows = (a.G.points + 31) / 32;
    const unsigned S = unsigned(a.splits > 1 ? a.splits : 1);
    k_core_v32<W><<<dim3(unsigned((rows + W - 1) / W), unsigned(ncond), S), W * 32, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_core_mcx(const CoreArgs& a, int ncond, cudaStream_t stream) {
    if (a.n <= 0 || a.G.points <= 0 || ncond <= 0) return cudaSuccess;
    constexpr int W = 4;
    const int rows = (a.G.points + 31) / 32;
    const unsigned S = unsigned(a.splits > 1 ? a.splits : 1);
    const int sets = (rows + W - 1) / W;
    k_core_mcx<W><<<dim3(unsigned(ncond), unsigned(sets < 65535 ? sets : 65535), S), W * 32, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_steptwo_mc(bool mixed, int C, int warps, int row, int blocks, const StepArgs& a,
                              cudaStream_t stream) {
    if (blocks <= 0 || a.n_items <= 0) return cudaSuccess;
    return dispatch_mc(mixed, C, warps, row, blocks, a, stream, nullptr);
}

template <int WARPS>
static cudaError_t dispatch_near_w(bool mixed, int row, int blocks, const StepArgs& a, cudaStream_t st, int* occ) {
    auto go = [&](auto kernel, size_t smem) {
        return run_group_kernel(kernel, WARPS * 32, WARPS * smem, blocks, a, st, occ);
    };
    if (row == 16)
        return mixed ? go(k_steptwo_near<16, WARPS>, near_warp_smem<16>())
                     : go(k_steptwo_near64<16, WARPS>, near64_warp_smem<16>());
    if (row == 8)
        return mixed ? go(k_steptwo_near<8, WARPS>, near_warp_smem<8>())
                     : go(k_steptwo_near64<8, WARPS>, near64_warp_smem<8>());
    return cudaErrorInvalidValue;
}

static cudaError_t dispatch_near(bool mixed, int row, int warps, int blocks, const StepArgs& a, cudaStream_t st,
                                 int* occ) {
    if (warps == 4) return dispatch_near_w<4>(mixed, row, blocks, a, st, occ);
    if (warps == 8) return dispatch_near_w<8>(mixed, row, blocks, a, st, occ);
    return cudaErrorInvalidValue;
}

cudaError_t launch_steptwo_near(bool mixed, int row, int warps, int blocks, const StepArgs& a, cudaStream_t stream) {
    if (blocks <= 0 || a.n_items <= 0) return cudaSuccess;
    return dispatch_near(mixed, row, warps, blocks, a, stream, nullptr);
}

int steptwo_near_blocks_per_sm(bool mixed, int row, int warps) {
    StepArgs dummy{};
    int occ = 0;
    return dispatch_near(mixed, row, warps, 0, dummy, nullptr, &occ) == cudaSuccess ? occ : 0;
}

int steptwo_mc_blocks_per_sm(bool mixed, int C, int warps, int row) {
    StepArgs dummy{};
    int occ = 0;
    if (dispatch_mc(mixed, C, warps, row, 0, dummy, nullptr, &occ) != cudaSuccess) return 0;
    return occ;
}

size_t record_bytes(int kind, bool mixed) {
    if (kind == kVoigt) return mixed ? sizeof(RecV32) : sizeof(RecV64);
    return sizeof(RecE64);
}

ScratchPlan plan_scratch(int kind, bool mixed, size_t n, int ncond, size_t base_off, int group) {
    auto al = [](size_t v) { return (v + 255) / 256 * 256; };
    ScratchPlan p;
    const size_t nwin = group > 0 ? size_t((ncond + group - 1) / group) : size_t(ncond);
    // records: per (line, condition); the mixed multi-condition layout has
    // (y, pref) and the region intervals below instead
    const size_t rec_bytes = group > 0 ? (mixed ? 0 : sizeof(CondRec64) * n * size_t(ncond))
                                       : record_bytes(kind, mixed) * n * size_t(ncond);
    p.off_rec = al(base_off);
    p.off_wlo = al(p.off_rec + rec_bytes);
    p.off_whi = al(p.off_wlo + sizeof(int) * n * nwin);
    p.off_mi = al(p.off_whi + sizeof(int) * n * nwin);
    p.off_kc = al(p.off_mi + sizeof(int) * n);
    p.off_lsh = al(p.off_kc + sizeof(int) * size_t(kKcWords));
    const size_t lsh = mixed ? sizeof(LineShX) : sizeof(LineSh64);
    p.off_civ = al(p.off_lsh + (group > 0 ? lsh * n * nwin : 0));
    const bool core = mixed && group > 0;
    p.off_cyp = al(p.off_civ + (core ? sizeof(CoreIv) * n * size_t(ncond) : 0));
    p.need = al(p.off_cyp + (core ? sizeof(float2) * n * size_t(ncond) : 0));
    return p;
}

}  // namespace xs
