// physics64.cuh -- FP64 point physics of the TSUNER scheme, evaluated in the
// reference's exact operation order so that the fused kernels reproduce the
// reference CUDA build bit for bit (both are compiled with -fmad=false, and
// double division and sqrt are IEEE round-to-nearest on the device).
//
// What differs from the reference is WHERE things are computed, not how:
// per-run constants (settling velocity, pow() terms, sqrt(FR), sqrt(OC)) are
// evaluated once per run with the reference expressions (TsuConsts), cell
// velocities are evaluated once per cell instead of five times, and face
// states / edge fluxes never leave shared memory.
#pragma once
#include <math_constants.h>

#include <cfloat>
#include <cstdint>

#include "ieee64.h"
#include "tsuner_b200.h"

namespace tsu {

constexpr double kG = 9.81;              // Sim_parameters.hxx:34
constexpr double kEpsilon = DBL_EPSILON; // Sim_parameters.hxx:28
constexpr double kEps = 1e-6;            // Sim_parameters.hxx:35
constexpr double kVmax = 10.0;           // Sim_parameters.hxx:36

// Scalar parameters the stage kernels need, packed once per run.
struct Phys64 {
    double FR, eps_h, Opar, OC, Q, HQB, porosity, CFL, dx, dy, inv_dx, inv_dy;
    TsuConsts k;
    int npx, npy;
    int order, wbc, bedload, suspension, read_files, bedload_law;
    double grass_ag;
    int rk, manning;
    // Row slab of a decomposed grid: npy is the number of rows this solver
    // owns, starting at global row j0 of a grid of ny_glob rows; gs / gn
    // ghost rows (0 or 2) below / above the owned rows are stored in the
    // state and mask planes and filled by the halo exchange.  A whole grid
    // has ny_glob = npy, j0 = 0, gs = gn = 0.
    int ny_glob, j0, gs, gn;
    // 1: an edge whose two faces are both dry returns zero fluctuations
    // without evaluating the Riemann solver (see edge_flux)
    int dry_skip;
    double inv_vs;  // RN(1 / k.vs)
    // 1: the source terms always take the ordinary operators (Manning friction,
    // or a divisor that the branch-free form could not take: see sources())
    int plain_sources;
    // High word of a speed s such that two components below it leave the bed
    // at rest for certain: Opar (s^2 + s^2) < 0.99 OC (0: no such speed).
    unsigned still_hi;
    __device__ __forceinline__ bool still(double u) const { return (hi32(u) & 0x7fffffffu) < still_hi; }
};

// IEEE quotient and square root with the zero cases answered directly:
// (+-0)/b for finite non-zero b is a zero with the XOR of the signs, and
// sqrt(+-0) = +-0.  Value-identical to `/` and sqrt(); still water and dry
// land make such operands the common case of this scheme.
__device__ __forceinline__ double ddiv(double a, double b) {
    if (a == 0.0 && b != 0.0 && isfinite(b)) return (signbit(a) != signbit(b)) ? -0.0 : 0.0;
    return a / b;
}
__device__ __forceinline__ double dsqrt(double x) { return (x == 0.0) ? x : sqrt(x); }
// As ddiv, also answering a non-zero, non-NaN numerator over a zero divisor
// (an infinity with the XOR of the signs).
__device__ __forceinline__ double ddiv_inf(double a, double b) {
    if (b == 0.0 && a != 0.0 && !isnan(a)) return (signbit(a) != signbit(b)) ? -CUDART_INF : CUDART_INF;
    return ddiv(a, b);
}

// x is neither NaN nor an infinity (exponent field not all ones), with
// integer instructions only (the FP64 pipe is the stage kernels' bottleneck)
__device__ __forceinline__ bool finite64(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

// SGN (Sim_parameters.hxx:29)
__device__ __forceinline__ int sgn(double x) { return (fabs(x) < kEpsilon) ? 0 : ((x) > 0) ? 1 : -1; }

// u_calculator_double (GPU/SedFlux.cuh:39-49).  `modb` receives the modulus
// of the returned velocity exactly as bedload() recomputes it
// (GPU/SedFlux.cuh:157): when no clamping happened it is the same expression
// on the same operands, so it is reused instead of a second sqrt.
// A dry state (h < EPS) gives u = (q / (h + EPSILON)) * 0, i.e. a zero with
// the sign of q; that is produced directly when the operands are finite and
// h + EPSILON > 0, which is value-identical and skips two divisions.
__device__ __forceinline__ void velocity(double h, double qx, double qy, double &ux, double &uy, double &modb) {
    double d = h + kEpsilon;
    if (!(h >= kEps) && d > 0.0 && !isnan(qx) && !isnan(qy)) {
        ux = copysign(0.0, qx);
        uy = copysign(0.0, qy);
        modb = 0.0;
        return;
    }
    double u = ddiv(qx, d) * (double)(h >= kEps);
    double v = ddiv(qy, d) * (double)(h >= kEps);
    double modu = dsqrt(u * u + v * v);
    if (modu > kVmax) {
        u = u / modu * kVmax;
        v = v / modu * kVmax;
        modb = dsqrt(u * u + v * v);
    } else {
        modb = modu;
    }
    ux = u;
    uy = v;
}
__device__ __forceinline__ void velocity(double h, double qx, double qy, double &ux, double &uy) {
    double m;
    velocity(h, qx, qy, ux, uy, m);
}

// avg, the van-Leer-type limiter (GPU/Reconstructor.cu:19-31).  When the
// numerator is a (signed) zero -- slopes of opposite sign or a zero slope --
// the quotient equals the numerator, so the division is skipped.
__device__ __forceinline__ double limiter(double a, double b) {
    double aa = fabs(a), bb = fabs(b);
    double den = aa + bb;
    if (!(den > kEpsilon)) return 0.0;
    double num = a * bb + b * aa;
    if (num == 0.0) return num;
    return num / den;
}

// state_filter_double (GPU/SedFlux.cuh:118-132)
__device__ __forceinline__ void positivity_filter(double &h, double &qx, double &qy, double &hc) {
    h = h * (double)(h > 0.0);
    double c = ddiv(hc, h + kEpsilon);
    c = c * (double)(c > 0.0);
    double ux, uy;
    velocity(h, qx, qy, ux, uy);
    qx = h * ux;
    qy = h * uy;
    hc = h * c;
}

struct State5 {
    double h, qx, qy, H, hc;
};

// What an edge needs of the face on one side: depth, bed, the velocity and
// the concentration that RiemannSolver_Vols computes from the filtered face
// (GPU/VolumeSolver.cu:28-36).  They are formed where the face is, because
// the filter already divides by the same h + EPSILON; the discharge and load
// themselves are not used by the edge.
struct Face5 {
    double h, u, v, H, c;
};

// Every formula below that divides or takes roots exists in two forms with
// the same operations in the same order.  FAST: the branch-free quotients and
// roots of ieee64.h, with `ok` cleared when an operand lies outside the range
// they are exact in (the results are then not used).  Otherwise: the ordinary
// operators, any operand.  The range tests read the high words only (integer
// instructions: the FP64 pipe is the scarcer one).
template <bool FAST>
struct Divisor {
    double d, y;
    // FAST: 2^-800 <= |d| < 2^800 and a quotient between 2^-1000 and 2^1000 are
    // the caller's to know (each use below says from what)
    __device__ __forceinline__ Divisor(double d_, bool &ok) : d(d_), y(0.0) {
        if (FAST) {
            y = recip(d);
            ok &= recip_ok(d);
        }
    }
    // numerator / d; FAST tests 2^-800 <= |a| < 2^800 or a zero
    __device__ __forceinline__ double of(double a, bool &ok) const {
        if (!FAST) return ddiv(a, d);
        ok &= mid_or_zero(a);
        return quot(a, d, y);
    }
    // FAST: the same without the test
    __device__ __forceinline__ double of(double a) const { return FAST ? quot(a, d, y) : ddiv(a, d); }
    // the same for a numerator near q0 * d
    __device__ __forceinline__ double near(double a, double q0) const {
        return FAST ? quot_from(a, d, y, q0) : ddiv(a, d);
    }
};
template <bool FAST>
__device__ __forceinline__ double root_of(double x) {
    return FAST ? root(x) : dsqrt(x);
}

// h + EPSILON of a wet state: 2^-19 <= d < 2^100 (d >= 2^-19 implies h > EPS)
__device__ __forceinline__ bool wet_divisor(double d) { return hi32(d) - 0x3ec00000u < 0x07700000u; }
// u = q / d of such a state is exact and cannot be clamped together with its
// other component: q is a zero or 2^-700 <= |u| < 7 (7^2 + 7^2 < VMAX^2)
__device__ __forceinline__ bool calm(double q, double u) {
    return ((hi32(u) & 0x7fffffffu) - 0x14300000u < 0x401c0000u - 0x14300000u) |
           (((hi32(q) & 0x7fffffffu) | lo32(q)) == 0u);
}
static_assert(kVmax == 10.0 && kEps < 0x1p-19, "calm, wet_divisor");

// What the tests above send away -- films below the velocity cutoff, speeds up
// to and beyond the clamp, every coast has some -- goes through a second
// branch-free form (`near_front`, in functions of their own: inlined, its code
// slowed the common path by 4 %), and only what that cannot take through the
// ordinary operators.  On a grid of one tile per SM a single such face set the
// time of the stage: 6400 cycles by the ordinary operators, of 10000 in all.
// h above the velocity cutoff EPS = 1e-6 for certain (and below 2^100), or
// zero or positive and below it for certain; the few depths whose high word is
// EPS's own are neither
constexpr uint32_t kEpsHi = 0x3eb0c6f7u;
static_assert(kEps == 1e-6, "kEpsHi");
__device__ __forceinline__ bool wet(double h) { return hi32(h) - (kEpsHi + 1u) < 0x46300000u - (kEpsHi + 1u); }
__device__ __forceinline__ bool film(double h) { return hi32(h) < kEpsHi; }
// u = q / d of a wet state is exact: q is a zero or 2^-700 <= |u| < 2^256
__device__ __forceinline__ bool sane(double q, double u) {
    return ((hi32(u) & 0x7fffffffu) - 0x14300000u < 0x4ff00000u - 0x14300000u) |
           (((hi32(q) & 0x7fffffffu) | lo32(q)) == 0u);
}
// The largest double whose square root rounds to at most VMAX = 10: with
// ulp(10) = 2^-49, sqrt(100 + 2^-46) = 10 + 0.8 * 2^-50 rounds to 10 and
// sqrt(100 + 2^-45) = 10 + 1.6 * 2^-50 to the next double.
constexpr double kVmax2 = 100.0 + 0x1p-46;
// the velocity clamp of u_calculator_double; sane components
__device__ __forceinline__ void clamp_speed(double &u, double &v, bool &ok) {
    const double m2 = u * u + v * v;
    if (m2 > kVmax2) {
        const Divisor<true> m(root(m2), ok);
        u = m.of(u) * kVmax;
        v = m.of(v) * kVmax;
    }
}

// u_calculator_double with d = h + EPSILON.  A film stands still: a zero
// reciprocal (left in dv) makes its quotients zeros.
__device__ __forceinline__ void velocity_near_front(double h, double qx, double qy, Divisor<true> &dv, double &u,
                                                    double &v, bool &ok) {
    const bool still = film(h);
    dv.y = still ? 0.0 : dv.y;
    u = dv.of(qx);
    v = dv.of(qy);
    const bool zero = ((hi32(u) | hi32(v)) << 1 | lo32(u) | lo32(v)) == 0u;  // q was finite
    ok &= still ? zero : wet(h) & sane(qx, u) & sane(qy, v);
    clamp_speed(u, v, ok);
}

// |x| < 2^100: what a face's differences are made of must be (see limit)
__device__ __forceinline__ bool limited(double x) { return (hi32(x) & 0x7fffffffu) < 0x46300000u; }

// dry land: a state of zeros
__device__ __forceinline__ bool empty(double h, double qx, double qy, double hc) {
    return ((hi32(h) | hi32(qx) | hi32(qy) | hi32(hc)) << 1 | lo32(h) | lo32(qx) | lo32(qy) | lo32(hc)) == 0u;
}

// Velocity and concentration of an unfiltered state (a cell, a ghost).  FAST
// takes only states whose depth, velocity and concentration are limited().
template <bool FAST>
__device__ __forceinline__ Face5 face_of(double h, double qx, double qy, double H, double hc, bool &ok) {
    Face5 f;
    f.h = h;
    f.H = H;
    if (FAST) {  // wet and unclamped, or empty (zero over EPSILON throughout)
        const Divisor<true> d(h + kEpsilon, ok);
        f.u = d.of(qx);
        f.v = d.of(qy);
        ok &= small_or_zero(hc);
        f.c = d.of(hc);
        ok &= (wet_divisor(d.d) & calm(qx, f.u) & calm(qy, f.v)) | empty(h, qx, qy, hc);
    } else {
        velocity(h, qx, qy, f.u, f.v);
        f.c = ddiv(hc, h + kEpsilon);
    }
    return f;
}

// A state through the positivity filter (state_filter_double,
// GPU/SedFlux.cuh:118-132), and the velocity and concentration of the result;
// h, qx, qy, hc become the filtered ones.  FAST: a wet, unclamped state (six
// quotients by the same h + EPSILON) or one without water, which comes out as
// zeros.
template <bool FAST>
__device__ __forceinline__ Face5 filter_face(double &h, double &qx, double &qy, double H, double &hc, bool &ok) {
    if (!FAST) {
        positivity_filter(h, qx, qy, hc);
        return face_of<false>(h, qx, qy, H, hc, ok);
    }
    bool in = true;
    Divisor<true> d(h + kEpsilon, in);
    // without water: a zero reciprocal makes every quotient below a zero
    const bool dry = (h == 0.0) & (fabs(qx) + fabs(qy) + fabs(hc) < 1e30);
    d.y = dry ? 0.0 : d.y;
    double c = d.of(hc, in);
    const double u = d.of(qx), v = d.of(qy);
    in &= wet_divisor(d.d) & calm(qx, u) & calm(qy, v);
    ok &= in | dry;
    c = (c > 0.0) ? c : 0.0;
    qx = h * u;
    qy = h * v;
    hc = h * c;
    Face5 f;
    f.h = h;
    f.H = H;
    f.u = d.near(qx, u);
    f.v = d.near(qy, v);
    f.c = d.near(hc, c);
    return f;
}

// filter_face for films and any speed; h >= 0
__device__ __forceinline__ Face5 filter_near_front(double h, double &qx, double &qy, double H, double &hc, bool &ok) {
    const Divisor<true> d(h + kEpsilon, ok);
    Divisor<true> dv = d;
    double u, v;
    velocity_near_front(h, qx, qy, dv, u, v, ok);
    double c = d.of(hc, ok);
    c = (c > 0.0) ? c : 0.0;
    qx = h * u;
    qy = h * v;
    hc = h * c;
    Face5 f;
    f.h = h;
    f.H = H;
    f.u = dv.near(qx, u);
    f.v = dv.near(qy, v);
    clamp_speed(f.u, f.v, ok);
    f.c = d.of(hc, ok);
    return f;
}

// avg, the van-Leer-type limiter (GPU/Reconstructor.cu:19-31): with a and b
// of the same sign (a |b| + b |a|) / (|a| + |b|) is 2 a b / (a + b), every
// operation rounding alike; of opposite sign its numerator is an exact zero.
// Both only while nothing overflows: FAST needs a and b below 2^101 (larger
// ones and infinities give a NaN by the general form, not a zero), which also
// bounds s, and 2 p / s from below, by 2^-900.
template <bool FAST>
__device__ __forceinline__ double limit(double a, double b, bool &ok) {
    if (!FAST) return limiter(a, b);
    const double p = a * b, s = a + b;
    const bool live = (p > 0.0) & (fabs(s) > kEpsilon);
    bool in = mid(p);
    const Divisor<true> d(s, in);
    const double q = d.of(p + p);
    ok &= in | !live;  // else q is not used
    return live ? q : 0.0;
}

// bedload (GPU/SedFlux.cuh:150-168), or the Grass law when selected; modu
// is |u| as bedload() computes it.  The Ashida-Michiue product
// K1*Q*max(O-OC,0)*max(sqrt(O)-sqrt(OC),0)*(h>HQB)*(h>5DS) has the sign of
// u (K1 = 17u/(|u|+eps), every other factor >= +0), so whenever one factor
// vanishes it is a zero with the sign of u and the return value -qb is
// -copysign(0, u): that case skips the division and the sqrt.
__device__ __forceinline__ double bedload_flux(const Phys64 &P, double h, double ux, double modu) {
    if (P.bedload_law == 1) return -ddiv(P.grass_ag * ux * modu * modu, 1.0 - P.porosity);
    double O = P.Opar * modu * modu;
    if (!isnan(O) && (O <= P.OC || h <= P.HQB || h <= P.k.DS5)) return -copysign(0.0, ux);
    double K1 = ddiv(17.0 * ux, modu + kEpsilon);
    double qb = K1 * P.Q * fmax(O - P.OC, 0.0) * fmax(dsqrt(O) - P.k.sqrt_OC, 0.0) *
                (double)(h > P.HQB) * (double)(h > P.k.DS5);
    return -qb;
}

// The bed component of Cflux (GPU/SedFlux.cuh:171-179) of a face with depth h
// and velocity (u, v).  With the bedload switched off or a fixed bed it is
// bedload * 0, a zero (NaN for a NaN velocity).
__device__ __forceinline__ double bed_flux(const Phys64 &P, double h, double u, double v, bool moves) {
    const double m2 = u * u + v * v;
    if (isnan(m2)) return m2;
    if (!moves) return 0.0;
    return bedload_flux(P, h, u, dsqrt(m2)) * (double)P.bedload;
}
// bedload_flux without branches for the Ashida-Michiue law
__device__ __forceinline__ double bed_flux_fast(const Phys64 &P, double h, double u, double v, bool &ok) {
    const double m2 = u * u + v * v;
    ok &= mid_or_zero(m2);
    const double m = root(m2), O = P.Opar * m * m;
    ok &= mid_or_zero(O);
    const double K1 = Divisor<true>(m + kEpsilon, ok).of(17.0 * u, ok);  // 2^-52 <= m + EPSILON < 2^5
    const double e = O - P.OC, f = root(O) - P.k.sqrt_OC;
    const bool live = (e > 0.0) & (f > 0.0) & (h > P.HQB) & (h > P.k.DS5);
    const double qb = K1 * P.Q * e * f;
    return live ? -qb * (double)P.bedload : 0.0;
}

// One edge: RiemannSolver_Vols (GPU/VolumeSolver.cu:19-126) in the frame of
// its normal: a is the face the normal leaves, b the one it enters, u / v
// their velocities along n and along n turned left.  Dm is the fluctuation
// into side a, Dp into side b, components (h, qn, qt, H, hc).
template <bool FAST>
__device__ __forceinline__ bool edge_flux(const Phys64 &P, const Face5 &a, const Face5 &b, int fixed, double Dm[5],
                                          double Dp[5]) {
    bool ok = true;
    // hydrostatic reconstruction (:37-40)
    const double zmH = fmin(a.H, b.H);
    double h0 = a.h - a.H + zmH, h1 = b.h - b.H + zmH;
    h0 = (h0 > 0.0) ? h0 : 0.0;  // fmax(h0, 0)
    h1 = (h1 > 0.0) ? h1 : 0.0;
    const double deta = h1 - h0;
    if (FAST && h0 == 0.0 && h1 == 0.0 && (P.bedload_law == 0 || (a.u == 0.0 && b.u == 0.0))) {
        // no water stands against either side (both faces dry, or water below
        // the other side's bed): F and DU are zeros, and so is everything the
        // finite wave speeds multiply (the Grass law's bed flux has no depth in
        // it: there the water has to stand still too).  Dry land makes this a
        // common edge.
        const double z = 0.0 * (a.u + a.v + a.c + b.u + b.v + b.c);
#pragma unroll
        for (int i = 0; i < 5; i++) Dm[i] = Dp[i] = z;
        return true;
    }
    double F0[5], F1[5];  // [3], the bed, comes last
    const double hc0 = h0 * a.c, hc1 = h1 * b.c;
    F0[0] = h0 * a.u;
    F0[1] = F0[0] * a.u;
    F0[2] = F0[0] * a.v;
    F0[4] = hc0 * a.u;
    F1[0] = h1 * b.u;
    F1[1] = F1[0] * b.u;
    F1[2] = F1[0] * b.v;
    F1[4] = hc1 * b.u;

    // Roe average + wave-speed bounds (GPU/SedFlux.cuh:181-199)
    const double hm = 0.5 * (h0 + h1);
    // depths below 2^80 and velocities up to 10 m/s bound every divisor below:
    // 2^-400 <= s0q + s1q < 2^41, 2^-52 < dS < 2^45
    if (FAST) ok &= small_or_zero(h0) & small_or_zero(h1);
    const double s0q = root_of<FAST>(h0), s1q = root_of<FAST>(h1);
    const double ghm = kG * hm;
    double SL = a.u - root_of<FAST>(kG * h0), SR = b.u + root_of<FAST>(kG * h1);
    const double cm = root_of<FAST>(ghm);
    // two zero depths: 0/0, as in the reference, and the bounds below ignore it
    const double umx = Divisor<FAST>(s0q + s1q, ok).of(s0q * a.u + s1q * b.u, ok);
    const double sl = umx - cm, sr = umx + cm;
    SL = (sl < SL) ? sl : SL;  // fmin / fmax of a possibly NaN second operand
    SR = (sr > SR) ? sr : SR;

    double a0, a1;
    const double dS = SR - SL;
    if (FAST) {
        const Divisor<true> d(dS, ok);
        ok &= dS > kEpsilon;
        a0 = d.of(SR * fabs(SL) - SL * fabs(SR), ok);
        a1 = d.of(fabs(SR) - fabs(SL), ok);
    } else if (dS > kEpsilon) {
        a0 = ddiv(SR * fabs(SL) - SL * fabs(SR), dS);
        a1 = ddiv(fabs(SR) - fabs(SL), dS);
    } else {
        a0 = fmax(fabs(SL), fabs(SR));
        a1 = 0.0;
    }

    double df[5], DU[5];
    df[0] = F1[0] - F0[0];
    df[1] = (F1[1] - F0[1]) + ghm * deta;
    df[2] = F1[2] - F0[2];
    df[4] = F1[4] - F0[4];
    DU[0] = deta;
    DU[1] = df[0];  // q = u h, the mass flux
    DU[2] = b.v * h1 - a.v * h0;
    DU[4] = hc1 - hc0;
#pragma unroll
    for (int i = 0; i < 5; i++) {
        if (i == 3) continue;
        const double vis = a0 * DU[i] + a1 * df[i];
        Dm[i] = 0.5 * (df[i] - vis) + F0[i];
        Dp[i] = 0.5 * (df[i] + vis) - F1[i];
    }
    // the bed component (upwinded by its own sign, :100-120): zeros where the
    // bed is fixed or at rest on both sides
    const bool moves = (fixed != 0) & (P.bedload != 0);
    Dm[3] = Dp[3] = 0.0;
    if (!FAST || (moves & ((P.bedload_law != 0) | !(P.still(a.u) & P.still(a.v) & P.still(b.u) & P.still(b.v))))) {
        double f0, f1;
        if (!FAST || P.bedload_law != 0) {
            f0 = bed_flux(P, h0, a.u, a.v, moves);
            f1 = bed_flux(P, h1, b.u, b.v, moves);
        } else {
            f0 = bed_flux_fast(P, h0, a.u, a.v, ok);
            f1 = bed_flux_fast(P, h1, b.u, b.v, ok);
        }
        const double d = f1 - f0;
        const int s0 = sgn(b.H - a.H), s2 = sgn(a1);
        const int s1 = sgn(d) * s0;  // s1 / s0 for s0 = +-1, 0 for s0 = 0
        const double vis = (s2 == s1) ? a1 * d : -a1 * d;
        Dm[3] = 0.5 * (d - vis) + f0;
        Dp[3] = 0.5 * (d + vis) - f1;
    }
    return ok;
}

// MUSCL-Hancock half-step predictor (RK == 0, GPU/Reconstructor.cu:280-342)
// on a cell's four faces before the state filter: L/R along x, D/U along y.
// hi is the cell's depth, detx/dety its hydrostatic slopes (the pressure
// terms Tpx/Tpy of :199-201,276-278).  The face velocities are taken once,
// before any face is updated, and each update reads the faces as the
// previous ones left them -- the order of the reference.  Its bedload terms
// use bedload() directly (no mask, no BEDLOAD switch), as the reference does.
__device__ __forceinline__ void hancock_predictor(const Phys64 &P, double dt, double hi, double detx, double dety,
                                                  State5 &L, State5 &R, State5 &D, State5 &U) {
    const double Tpx = kG * hi * detx;
    const double Tpy = kG * hi * dety;
    double uRx, uRy, mR, uLx, uLy, mL, uUx, uUy, mU, uDx, uDy, mD;
    velocity(R.h, R.qx, R.qy, uRx, uRy, mR);
    velocity(L.h, L.qx, L.qy, uLx, uLy, mL);
    velocity(U.h, U.qx, U.qy, uUx, uUy, mU);
    velocity(D.h, D.qx, D.qy, uDx, uDy, mD);
    const double hdt = 0.5 * dt;
    double qhx = (R.qx - L.qx) * P.inv_dx;
    double qhy = (U.qy - D.qy) * P.inv_dy;
    double up = hdt * (qhx + qhy);
    L.h -= up;
    R.h -= up;
    D.h -= up;
    U.h -= up;
    qhx = (R.qx * uRx - L.qx * uLx) * P.inv_dx;
    qhy = (U.qx * uUy - D.qx * uDy) * P.inv_dy;
    up = hdt * (qhx + qhy);
    L.qx -= up;
    R.qx -= up;
    D.qx -= up;
    U.qx -= up;
    qhx = (R.qx * uRy - L.qx * uLy) * P.inv_dx;
    qhy = (U.qy * uUy - D.qy * uDy) * P.inv_dy;
    up = hdt * (qhx + qhy);
    L.qy -= up;
    R.qy -= up;
    D.qy -= up;
    U.qy -= up;
    qhx = (bedload_flux(P, R.h, uRx, mR) - bedload_flux(P, L.h, uLx, mL)) * P.inv_dx;
    qhy = (bedload_flux(P, U.h, uUx, mU) - bedload_flux(P, D.h, uDx, mD)) * P.inv_dy;
    up = hdt * (qhx + qhy);
    L.H -= up;
    R.H -= up;
    D.H -= up;
    U.H -= up;
    qhx = (R.hc * uRx - L.hc * uLx) * P.inv_dx;
    qhy = (U.hc * uUy - D.hc * uDy) * P.inv_dy;
    up = hdt * (qhx + qhy);
    L.hc -= up;
    R.hc -= up;
    D.hc -= up;
    U.hc -= up;
    up = hdt * P.inv_dx * Tpx;
    L.qx -= up;
    U.qx -= up;
    D.qx -= up;
    R.qx -= up;
    up = hdt * P.inv_dy * Tpy;
    L.qy -= up;
    U.qy -= up;
    D.qy -= up;
    R.qy -= up;
}

// interpolate_time (GPU/VolumeSolver.cu:172-203): boundary state from the
// CC series at segment `seg`; replaces h, H, qx, qy and zeroes hc.
__device__ __forceinline__ void series_state(const double *__restrict__ CC, const double *__restrict__ tCC,
                                             double t, int npx, int npy, int seg, State5 &g) {
    double dt = tCC[1] - tCC[0];
    int it = int((t - tCC[0]) / dt);
    it *= (it > 0);
    int tp = it + 1;
    long long nseg4 = (long long)(2 * npx + 2 * npy) * 4;
    long long posCC = it * nseg4 + (long long)seg * 4;
    long long posCCp = tp * nseg4 + (long long)seg * 4;
    double m = (CC[posCCp] - CC[posCC]) / dt;
    double b = CC[posCC] - m * tCC[it];
    double h1 = m * t + b;
    m = (CC[posCCp + 3] - CC[posCC + 3]) / dt;
    b = CC[posCC + 3] - m * tCC[it];
    double zb1 = m * t + b;
    h1 += zb1;
    m = (CC[posCCp + 1] - CC[posCC + 1]) / dt;
    b = CC[posCC + 1] - m * tCC[it];
    double qx = m * t + b;
    qx *= h1;
    m = (CC[posCCp + 2] - CC[posCC + 2]) / dt;
    b = CC[posCC + 2] - m * tCC[it];
    double qy = m * t + b;
    qy *= h1;
    g.h = h1;
    g.H = zb1;
    g.qx = qx;
    g.qy = qy;
    g.hc = 0.0;
}

// GetDeltaT per cell (GPU/Volume_kernel.cu:28-41)
__device__ __forceinline__ double cfl_dt(const Phys64 &P, double h, double qx, double qy) {
    double ux, uy;
    velocity(h, qx, qy, ux, uy);
    double cg = dsqrt(kG * h);
    double lx = fabs(ux) + cg;
    double ly = fabs(uy) + cg;
    return P.CFL * 0.5 * fmin(ddiv_inf(P.dx, lx), ddiv_inf(P.dy, ly));
}

// The same from the velocity of the cell's filtered state.  On square
// cells the smaller of dx / lx and dy / ly is dx over the larger speed (the
// rounded quotient does not increase with the divisor).
__device__ __forceinline__ bool cfl_dt_fast(const Phys64 &P, const Face5 &f, double &dt) {
    bool ok = mid(f.h);  // f.h of a wet filtered state: 2^-20 < h < 2^100, and so is lx, ly from below
    if (f.h == 0.0) {  // no speed: an infinite step
        dt = CUDART_INF;
        return true;
    }
    const double cg = root(kG * f.h);
    const double lx = fabs(f.u) + cg, ly = fabs(f.v) + cg;
    double q;
    if (P.dx == P.dy) {
        q = Divisor<true>((lx > ly) ? lx : ly, ok).of(P.dx, ok);
    } else {
        const double qx = Divisor<true>(lx, ok).of(P.dx, ok), qy = Divisor<true>(ly, ok).of(P.dy, ok);
        q = (qx < qy) ? qx : qy;
    }
    dt = P.CFL * 0.5 * q;
    return ok;
}

}  // namespace tsu
