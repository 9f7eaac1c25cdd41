// pn_fix.cuh -- the star-pair terms of the FP64 sweeps in 64-bit fixed point.
//
// A GB300 scheduler issues an FP64 warp instruction every 64 cycles, a 32 x 32 + 64 bit integer
// multiply-add every 4 (both measured); a product of two 62-bit numbers is three of the latter and carries
// 9 more bits than a double.  The pair terms are therefore formed as fixed-point numbers of 58 to 62
// fraction bits.  Host and device compile the same functions (a CPU run checks the device's arithmetic).
//
// Units.  Lengths in units of 2^eL, the power of two with 1 <= eps / 2^eL < 2; masses in units of
// the power of two of the BH's mass; velocities in units of 2^ev, the power of two above the fastest
// |u| (below) of the two tiles at hand.  "S = k" at a variable says that it holds its value times 2^k.
//
// One pair (i, j), d = x_j - x_i:
//   X   BH-relative positions, 96 bits, S = 62: d is exact to 2^-62 eps.
//   y   FP32 estimate of Q = (|d|^2 + eps^2)^(-1/2) (MUFU), raised above Q: y = f 2^-ey, 1 <= f < 2.
//   D   = d 2^-ey, S = 62: |D| <= 1 whatever the distance (the only per-pair normalisation)
//   RHO = |D|^2 + eps^2 2^(-2 ey), S = 60, in (1/4, 1]
//   r   = 1 - RHO f^2, |r| < 2^-18.8;  Q 2^ey = f (1 + r/2 + 3 r^2/8): the binomial series of
//         (1 - r)^(-1/2), whose next term is below 2^-58 (2^-60 on average).
//   n   = d Q, S = 60, the softened unit vector
// and the terms of pn_device.cuh's sums, with w_j = sqrt(3) v_j, u_i = (4 / sqrt(3)) v_i:
//   G   += (m Q^2) n         S0 += (m Q^2) Q
//   W   += (H + C) n + ct w,   H = m Q^2 F,  F = u.w + (w.n)^2 / 2,  ct = m Q^2 (u.n - w.n),
//          C = (g1 - g3 qe_i) Q^2 + k,  g1 = m (c1 - 2 |v|^2), g3 = m c3, k = g3 + k35
//          (C, which spans the range of R_j^3, is formed in FP64; c3 rho Q^2 = c3 is in k)
//   Phi += m Q,  U += mu3 Q  (FP64; in the energy sweep Phi in integers)
//   Psi += m Q (7 u.w + (u.n)(w.n))  (four times the energy's)
// The small (cross) parts of the dot products u.w, u.n, w.n are FP32: their rounding, 2^-54 of the
// velocity unit, is random from pair to pair.  The sums over one j-tile are accumulated as integers
// relative to the tile's own sums of magnitudes (a first FP32 pass over the tile finds their exponents),
// so the smallest kept bit is 2^-62 of that sum; the tile sums are added in FP64.  The pair of a star
// with itself (d = 0: no G, no W) would raise that scale to m / eps^2; it is left out of the integer
// sums and its S0, and in the energy sweep Phi and Psi, added in FP64.
// Two of these errors do not shrink with their term, as FP64's do: n's, 2^-61 also where d is far below eps (the
// sweep forms such rows again in FP64), and the velocity terms' in the unit of a tile's fastest star (velocity_limit).
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define PNF __host__ __device__ __forceinline__
#else
#define PNF inline
#endif

namespace pn {
namespace fix {

typedef long long i64;
typedef unsigned long long u64;

// limits of the fixed-point range (host constants of the units, checked per star by k_prep)
constexpr int POS_BITS = 24;   // |s| / 2^eL < 2^24 (the FP32 seed then stays within 2^-20)
constexpr int EV_MAX = 200;    // speeds below 2^200 (slower ones than 2^-200 count as at rest)
constexpr int E0_MAX = 300;    // the BH's mass within 2^-300 .. 2^300
constexpr double W_SCALE = 1.7320508075688772935;  // w / v
constexpr u64 W_MANT = 0xDDB3D742C265539DULL;      // sqrt(3) 2^63
constexpr u64 U_MANT = 0x93CD3A2C8198E269ULL;      // 4 / sqrt(3) 2^62

// rounding constants of right shifts
constexpr i64 half(int s) { return 1LL << (s - 1); }

PNF float fmaf_(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    return ::fmaf(a, b, c);
#else
    return __builtin_fmaf(a, b, c);
#endif
}
PNF float as_float(unsigned b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float f;
    std::memcpy(&f, &b, 4);
    return f;
#endif
}
PNF int to_int(float x) {  // rounded
#ifdef __CUDA_ARCH__
    return __float2int_rn(x);
#else
    return (int)__builtin_rintf(x);
#endif
}
PNF double fma_(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return ::fma(a, b, c);
#else
    return __builtin_fma(a, b, c);
#endif
}

// value = h 2^32 + l with both limbs signed 32-bit, so that limb products need no sign repair
struct B2 {
    int h, l;
};
PNF B2 bal(i64 v) {
    B2 b;
    b.l = (int)v;
    b.h = (int)(v >> 32) + (int)((unsigned)b.l >> 31);
    return b;
}
PNF i64 limbs(int h, int l) { return (i64)(((u64)(unsigned)h << 32) + (u64)(i64)l); }
PNF i64 mw(int a, int b, i64 c) { return (i64)a * b + c; }                           // IMAD.WIDE
PNF u64 muw(unsigned a, unsigned b, u64 c) { return (u64)a * b + c; }                // IMAD.WIDE.U32
PNF i64 cross(B2 a, B2 b, i64 c) { return mw(a.h, b.l, mw(a.l, b.h, c)); }
// A factor: value = h 2^32 + l, the high part an integer (and as a float, for the cross products), the
// low part a float; |h| < 2^31, so the value keeps 55 bits below its scale's top.  A product is
// h h' 2^64 + (h l' + l h') 2^32: one integer multiply-add for the first part, which may be summed
// over terms, and two FP32 FMAs for the second, which likewise.
struct V {
    int h;
    float hf, l;
};
PNF V vec(B2 b) {
    V r;
    r.h = b.h;
    r.hf = (float)b.h;
    r.l = (float)b.l;
    return r;
}
PNF float crossf(const V &a, const V &b, float c) { return fmaf_(a.hf, b.l, fmaf_(a.l, b.hf, c)); }

PNF u64 mulhi(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}
// a >> s for 0 <= s (0 from 64 on, and for s < 0)
PNF u64 shr(u64 a, int s) {
#ifdef __CUDA_ARCH__
    u64 r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(s));
    return r;
#else
    return (unsigned)s > 63u ? 0 : a >> s;
#endif
}

// Sums of a product and a 32-bit part as carry additions of their halves: as the addend of a multiply-add the
// part would have to be moved and extended into a register pair, by moves on the pipe that bounds the
// sweep (N = 65,536: 77.3 -> 71.7 ms).
// a + (c >> 32)
PNF i64 plus_hi(i64 a, i64 c) {
#ifdef __CUDA_ARCH__
    const int ch = (int)(c >> 32);
    unsigned lo, hi;
    asm("add.cc.u32 %0, %2, %4;\n\taddc.u32 %1, %3, %5;"
        : "=r"(lo), "=r"(hi) : "r"((unsigned)a), "r"((unsigned)((u64)a >> 32)), "r"(ch), "r"(ch >> 31));
    return (i64)(((u64)hi << 32) | lo);
#else
    return a + (c >> 32);
#endif
}
// hi 2^32 + a + (c >> 32), unsigned
PNF u64 plus_hi(u64 a, u64 c, unsigned h) {
#ifdef __CUDA_ARCH__
    unsigned lo, hi;
    asm("add.cc.u32 %0, %2, %4;\n\taddc.u32 %1, %3, %5;"
        : "=r"(lo), "=r"(hi) : "r"((unsigned)a), "r"((unsigned)(a >> 32)), "r"((unsigned)(c >> 32)), "r"(h));
    return ((u64)hi << 32) | lo;
#else
    return a + (((u64)h << 32) | (c >> 32));
#endif
}

// a + t
PNF i64 plus_small(i64 a, unsigned t) {
#ifdef __CUDA_ARCH__
    unsigned lo, hi;
    asm("add.cc.u32 %0, %2, %4;\n\taddc.u32 %1, %3, 0;"
        : "=r"(lo), "=r"(hi) : "r"((unsigned)a), "r"((unsigned)((u64)a >> 32)), "r"(t));
    return (i64)(((u64)hi << 32) | lo);
#else
    return a + t;
#endif
}
// a + t 2^B
template <int B> PNF i64 plus_low(i64 a, int t) {
#ifdef __CUDA_ARCH__
    unsigned lo, hi;
    asm("add.cc.u32 %0, %2, %4;\n\taddc.u32 %1, %3, %5;"
        : "=r"(lo), "=r"(hi)
        : "r"((unsigned)a), "r"((unsigned)((u64)a >> 32)), "r"((unsigned)t << B), "r"(t >> (32 - B)));
    return (i64)(((u64)hi << 32) | lo);
#else
    return a + (i64)((u64)(i64)t << B);
#endif
}

// hi + x f, x a sum of cross products and f its unit; |x f| < 2^(31 + B), rounded to 2^B
template <int B> PNF i64 merge(i64 hi, float x, float f) {
    return plus_low<B>(hi, to_int(x * (f * (1.f / (1 << B)))));
}
struct X96 {
    unsigned w0, w1, w2;
};
// (b - a) >> e, 0 <= e < 32, of two 96-bit integers whose difference fits 62 bits after the shift
PNF i64 diff_shift(const X96 &b, const X96 &a, int e) {
#ifdef __CUDA_ARCH__
    unsigned d0, d1, d2;
    asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
        : "=r"(d0), "=r"(d1), "=r"(d2)
        : "r"(b.w0), "r"(b.w1), "r"(b.w2), "r"(a.w0), "r"(a.w1), "r"(a.w2));
    const unsigned lo = __funnelshift_r(d0, d1, e), hi = __funnelshift_r(d1, d2, e);
    return (i64)(((u64)hi << 32) | lo);
#else
    const u64 bl = ((u64)b.w1 << 32) | b.w0, al = ((u64)a.w1 << 32) | a.w0;
    const u64 lo = bl - al;
    const unsigned hi = b.w2 - a.w2 - (bl < al ? 1u : 0u);
    const unsigned __int128 d = ((unsigned __int128)(u64)(i64)(int)hi << 64) | lo;
    return (i64)(u64)((__int128)d >> e);
#endif
}

// ------------------------------------------------------------------ conversions (O(N))
PNF u64 bits_of(double x) {
#ifdef __CUDA_ARCH__
    return (u64)__double_as_longlong(x);
#else
    u64 b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
// exponent e of a finite normal x = +-1.f 2^e
PNF int expo(double x) { return (int)((bits_of(x) >> 52) & 0x7ff) - 1023; }
// x 2^(62 - eL) truncated to a 96-bit integer (|x| 2^-eL < 2^33)
PNF X96 to_x96(double x, int eL) {
    const u64 b = bits_of(x);
    const int be = (int)((b >> 52) & 0x7ff);
    const u64 m = be ? ((b & 0xfffffffffffffULL) | 0x10000000000000ULL) : 0;
    const int s = be - 1075 + 62 - eL;
    u64 lo, hi = 0;
    if (s >= 0) {
        lo = m << s;
        if (s > 11) hi = m >> (64 - s);
    } else {
        lo = s > -64 ? m >> -s : 0;
    }
    if (b >> 63) {
        lo = 0 - lo;
        hi = ~hi + (lo == 0 ? 1 : 0);
    }
    X96 r;
    r.w0 = (unsigned)lo;
    r.w1 = (unsigned)(lo >> 32);
    r.w2 = (unsigned)hi;
    return r;
}
// x (mant / 2^k) 2^(S - ev) truncated to a 64-bit integer, for |result| < 2^62; mant = k-bit scale
PNF i64 to_scaled(double x, u64 mant, int k, int S, int ev) {
    const u64 b = bits_of(x);
    const int be = (int)((b >> 52) & 0x7ff);
    const u64 m = be ? ((b & 0xfffffffffffffULL) | 0x10000000000000ULL) << 11 : 0;  // S = 63 of 1.f
    const u64 p = mulhi(m, mant);                                                     // S = 63 + k - 64
    const int s = (k - 1) - (S - ev + (be - 1023));                                   // right shift to S
    const u64 v = s <= 0 ? p << (s < -63 ? 63 : -s) : shr(p, s);
    return (b >> 63) ? -(i64)v : (i64)v;
}
// positive x = M 2^-64 2^e with 2^63 <= M < 2^64 (x = 0: M = 0)
PNF u64 mantissa(double x, int &e) {
    const u64 b = bits_of(x);
    const int be = (int)((b >> 52) & 0x7ff);
    e = be - 1022;
    return be ? ((b & 0xfffffffffffffULL) | 0x10000000000000ULL) << 11 : 0;
}

// the smallest ev with |u| = (4 / sqrt(3)) |v| < 2^ev, from |v|^2 (0: the smallest of all)
PNF int speed_exp(double v2) {
    const int be = (int)((bits_of(v2) >> 52) & 0x7ff);
    const int e = ((be - 1022) >> 1) + 2;
    return be == 0 || e < -EV_MAX ? -EV_MAX : e;
}

// The largest velocity unit 2^ev of a system whose 1PN terms have the weight inv_c2: inv_c2 4^ev <= 64, which every
// speed up to that of light is within (and up to 2.8 times it at inv_c2 = 1).  The velocity terms' rounding, 2^-58 of
// the unit's square and 2^-55 of the unit times the star's own speed for each m Q^2, does not shrink with
// the slow stars of a tile that holds a fast one.
// Median errors of W over sum m Q^2 |n| of 128 stars of speeds about 0.3 and one light fast one, in units of 2^-53
// (inv_c2 = 1; here and in FP64): speed 1: 0.50, 0.70; 2.8: 1.3, 0.80; 11: 6.8, 1.0; 45: 124, 0.4; 300: 6,100, 0.4.
inline int velocity_limit(double inv_c2) {
    if (!(inv_c2 > 0.0)) return EV_MAX;  // (no velocity terms)
    const double lim = 64.0 / inv_c2;
    const int e = lim > 0.0 ? __builtin_ilogb(lim) >> 1 : -EV_MAX - 1;
    return e < EV_MAX ? e : EV_MAX;
}

// Whether the sweep covers a star of mass m at s with |v|^2 = v2 beside a BH of mass m0 (a star outside sends the
// whole system to the FP64 sweep): |s| < 2^POS_BITS in units, speeds below 2^EV_MAX and (for the FP32 sums of C's
// magnitudes) |v|^2 below 2^60 m0 / 2^eL, the star's mass 0 or 2^-32 .. 2^59 of the BH's, the speed within
// velocity_limit, the BH's mass positive and within 2^-E0_MAX .. 2^E0_MAX; infinities and NaN are outside.
// The units of a tile's integer sums are then powers of two that a double holds (the sweep's pow2): with the BH's mass
// about 2^e0, |e0| <= 300, |eL| <= 60, a tile's FP32 sum of m Q^2 below 2^67 (2^-126 stands for none), -200 <= ev
// and ev < 200, their exponents lie within
//   G, S0      e0 - 2 eL - 188 .. e0 - 3 eL + 7          -608 .. 487
//   C + H      2 e0 - 3 eL - 187 .. 2 e0 - 3 eL + 67     -967 .. 847
//   ct, ct w   e0 - 2 eL - 200 + 2 ev .. e0 - 2 eL + 5 + 2 ev    -1020 .. 825
PNF bool in_range(const double *s, double v2, double m, double m0, int eL, int ev_max) {
    auto e = [](double x) { return (int)((bits_of(x) >> 52) & 0x7ff); };
    const int e0 = expo(m0);
    bool in = !(bits_of(m0) >> 63) && e0 >= -E0_MAX && e0 <= E0_MAX && e(v2) < 1023 + 2 * EV_MAX - 10 &&
              e(v2) < 1023 + 60 + e0 - eL;
    for (int k = 0; k < 3; ++k) in = in && e(s[k]) < 1023 + POS_BITS + eL;
    return in && speed_exp(v2) <= ev_max && !(bits_of(m) >> 63) && (m == 0.0 || (e(m) >= 1023 + e0 - 32 && e(m) < 1023 + e0 + 59));
}

// ------------------------------------------------------------------ one pair
enum : int { F_NEWTON = 0, F_FORCE = 1, F_ENERGY = 2, F_FORCE_ENERGY = 3 };  // as PairMode

struct StarI {  // the accumulating star
    X96 x, y, z;
    V ux, uy, uz;  // u_i in units of its own power of two 2^(ev - d), S = 62
    int d;         // (per tile)
    float fd;      // 2^-d
    double qe;     // |s_i|^2 + eps^2
};
struct StarJ {
    X96 x, y, z;
    unsigned mh;        // mantissa of m, S = 64: its high 32 bits as an integer,
    float mhf, ml;      // and both halves as floats times 2^-34
    int em;             // its exponent (in the units above)
    B2 wx, wy, wz;      // w_j, S = 60
    double m, mu3;      // m and mu3 = m R^3, in the system's units
    double g1, g3, k;   // the coefficients of C, in the system's units
};
struct Scale {
    int g;     // the tile's sums: m Q^2 < 2^g (or m Q, energy)
    int c;     // ... |C + H| < 2^c (the system's units): c one above the larger of C's and H's exponents
    int rh;    // right shift of H from its own exponent to 2^c
    int q;     // exponent of the system's Q over the units' Q: -eL
    // left shifts of the velocity terms' factors, from S = 60 relative to 2^g to S = 62 relative to the
    // tile's own sums: |m Q^2 F| < 2^(g + 2 - lh + 2 ev), |ct| < 2^(g + 2 - lt + ev); 2^(lh - 32), 2^(lt - 32)
    int lh, lt;
};
struct Acc {  // h 2^64 + x 2^32
    i64 h;
    float x;
};
struct Acci {  // ... all integers
    i64 h, x;
};
struct Sums {
    Acci g[3];  // G, S = 122 relative to 2^g
    Acci c[3];  // W's part along n, S = 122 relative to 2^c
    Acci t[3];  // W's part along w, S = 122 relative to 2^(g + 2 - lt + 2 ev)
    i64 s0;     // S0, S = 60 relative to 2^g
    i64 ct;     // sum of ct, S = 62 relative to 2^(g + 2 - lt + ev)
    i64 phi;    // energy: Phi, S = 62 relative to 2^g
    Acc psi;    // energy: Psi, S = 121 relative to 2^(g + 2 ev)
    double dphi, du;  // force: Phi, U (FP64)
    double dpsi;      // force and energy: Psi (FP64, times 2^59, relative to 2^(2 ev))
};

template <int MODE> PNF void clear(Sums &a) {
    for (int k = 0; k < 3; ++k) {
        a.g[k].h = a.g[k].x = a.c[k].h = a.c[k].x = a.t[k].h = a.t[k].x = 0;
    }
    a.s0 = a.ct = a.phi = a.psi.h = 0;
    a.psi.x = 0.f;
    a.dphi = a.du = a.dpsi = 0.0;
}
// Moves the cross sums into the high sums, at least every 8 pairs (see the bounds at pair()).
PNF void fold(Acc &a) {  // (what is below 2^35 stays in the FP32 sum: 12582912 = 1.5 2^23 rounds to an integer)
    const float t = fmaf_(a.x, 0x1p-36f, 12582912.f) - 12582912.f;
    a.h = mw(to_int(t), 16, a.h);
    a.x = fmaf_(t, -0x1p36f, a.x);
}
PNF void fold(Acci &a) {
    a.h += a.x >> 32;
    a.x &= 0xffffffffLL;
}
template <int MODE> PNF void fold(Sums &a) {
    if (MODE == F_ENERGY) {
        fold(a.psi);
        return;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        fold(a.g[k]);
        if (MODE != F_NEWTON) {
            fold(a.c[k]);
            fold(a.t[k]);
        }
    }
}

// The sums after the last fold, S lowered by 60 (the integer ones) or 61
PNF i64 top(const Acci &a) { return (i64)((u64)a.h << 4) + (a.x >> 28); }
PNF i64 top(const Acc &a) { return (i64)((u64)a.h << 3) + to_int(a.x * 0x1p-29f); }
// The shifts of Scale from the exponents of the tile's sums of m Q^2, m Q^2 |F| and |ct|
// (at most by `most`: beyond that the terms are small beside |v_i|^2 times the tile's sum)
PNF int lift(int g, int e, int most) { return 2 + (g - e < 0 ? 0 : g - e > most ? most : g - e); }
constexpr int LIFT_H = 16, LIFT_T = 12;
// Scale::c and rh from C's exponent and H's own (in the system's units)
PNF void join(Scale &E, int ec, int eh) {
    E.c = (ec > eh ? ec : eh) + 1;
    E.rh = E.c - eh < 63 ? E.c - eh : 63;
}

PNF double scale_down(double x, int e) {  // x 2^-e, x > 0 and normal, result normal
#ifdef __CUDA_ARCH__
    return __hiloint2double(__double2hiint(x) - (e << 20), __double2loint(x));
#else
    u64 b = bits_of(x) - ((u64)(i64)e << 52);
    double r;
    std::memcpy(&r, &b, 8);
    return r;
#endif
}
PNF double u2d(u64 v) {
#ifdef __CUDA_ARCH__
    return __ull2double_rn(v);
#else
    return (double)v;
#endif
}

PNF void add(Acci &s, B2 a, B2 b) {
    s.h = mw(a.h, b.h, s.h);
    s.x = cross(a, b, s.x);
}
PNF void add(Acc &s, const V &a, const V &b) {
    s.h = mw(a.h, b.h, s.h);
    s.x = crossf(a, b, s.x);
}
PNF Acc dot(const V &ax, const V &ay, const V &az, const V &bx, const V &by, const V &bz) {
    Acc s;
    s.h = mw(ax.h, bx.h, 0);
    s.x = fmaf_(ax.hf, bx.l, ax.l * bx.hf);
    add(s, ay, by);
    add(s, az, bz);
    return s;
}

// One pair.  ybits: the bits of the FP32 seed y (0 < y <= 1 + 2^-20).  eps60: eps^2 in the units
// above, S = 60 (1 <= eps^2 < 4).
// Bounds: |D| <= 1 (+ 2^-18), |n| <= 1, |u| < 1 and |w| < 3/4 (the unit 2^ev), the tile's sums of P, H, t
// and C below 2^62, so the high sums stay below 2^62.  Integer cross sums of 8 pairs: ah bl with the sum of
// |ah| <= 2^30, |bl| <= 2^31, and al bh <= 8 2^31 2^28 (t w: 8 2^31 0.75 2^28): below 2^62.6.
template <int MODE>
PNF void pair(Sums &a, const StarI &I, const StarJ &J, const Scale &E, unsigned ybits, u64 eps60) {
    ybits += 8;  // a seed above Q (by 2^-21 .. 2^-20 less its error): Q 2^ey < 2, so Q^2 fits
    const int ey = 127 - (int)(ybits >> 23);
    const unsigned F = (ybits & 0x7fffffu) | 0x800000u;
    const B2 bx = bal(diff_shift(J.x, I.x, ey)), by = bal(diff_shift(J.y, I.y, ey)), bz = bal(diff_shift(J.z, I.z, ey));
    // RHO, S = 60 (its cross products in integers: its rounding error would enter every term)
    const i64 dt = mw(bz.h, bz.l, mw(by.h, by.l, mw(bx.h, bx.l, half(31))));
    const u64 rho = (u64)(mw(bz.h, bz.h, mw(by.h, by.h, mw(bx.h, bx.h, dt >> 31)))) + shr(eps60, 2 * ey);
    // r = 1 - RHO f^2, S = 58
    const unsigned F8 = F << 8;
    const u64 U = plus_hi(muw((unsigned)(rho >> 32), F8, 0), muw((unsigned)rho, F8, half(32)), 0u);  // RHO f, S = 59
    const i64 r = (i64)((1ULL << 58) - plus_hi(muw((unsigned)(U >> 32), F8, 0), muw((unsigned)U, F8, half(32)), 0u));
    const int rs = (int)(r >> 12);                          // S = 46 (below 2^28)
    const int rsq = (int)(mw(rs, rs, 0) >> 32);             // r^2, S = 60
    const i64 c = plus_small(r << 5, 6u * (unsigned)rsq);  // r/2 + 3 r^2/8, S = 64
    const int F7 = (int)(F << 7);
    const u64 Q = plus_hi((u64)mw(F7, (int)(c >> 32), 0), muw((unsigned)F7, (unsigned)c, 0), (unsigned)F7);  // S = 62
    const B2 bq = bal((i64)Q);
    // n = d Q, S = 60
    const B2 mx = bal(plus_hi(mw(bx.h, bq.h, 0), cross(bx, bq, half(32)))), my = bal(plus_hi(mw(by.h, bq.h, 0), cross(by, bq, half(32)))),
             mz = bal(plus_hi(mw(bz.h, bq.h, 0), cross(bz, bq, half(32))));
    if (MODE == F_ENERGY) {
        const V q = vec(bq);
        const u64 mQ = muw(J.mh, (unsigned)q.h, 0) + ((u64)(i64)to_int(fmaf_(J.mhf, q.l, J.ml * q.hf)) << 2);  // S = 62
        const u64 P = shr(mQ, E.g - J.em + ey);  // m Q relative to 2^g
        a.phi += (i64)P;
        const V p = vec(bal((i64)P));
        const V nx = vec(mx), ny = vec(my), nz = vec(mz), wx = vec(J.wx), wy = vec(J.wy), wz = vec(J.wz);
        const Acc uw = dot(I.ux, I.uy, I.uz, wx, wy, wz), un = dot(I.ux, I.uy, I.uz, nx, ny, nz), wn = dot(wx, wy, wz, nx, ny, nz);
        const V b = vec(bal(merge<4>((un.h << 4) >> I.d, un.x, I.fd * 0x1p-28f))), w = vec(bal(merge<5>(wn.h << 6, wn.x, 0x1p-26f)));
        // 7 u.w + (u.n)(w.n), S = 59 (below 6.1)
        const V z = vec(bal(merge<5>(((14 * uw.h) >> I.d) + (mw(b.h, w.h, 0) >> 1), fmaf_(14.f * I.fd, uw.x, 0.5f * crossf(b, w, 0.f)), 0x1p-32f)));
        add(a.psi, p, z);
        return;
    }
    const unsigned qh = (unsigned)(Q >> 32);
    const u64 Q2 = muw(qh, qh, muw(qh, (unsigned)Q, 0) >> 31) << 2;  // S = 62
    const float q2h = (float)(unsigned)(Q2 >> 32), q2l = (float)(unsigned)Q2;
    const u64 mQ2 = muw(J.mh, (unsigned)(Q2 >> 32), 0) + ((u64)(i64)to_int(fmaf_(J.mhf, q2l, J.ml * q2h)) << 2);  // S = 62
    const B2 p = bal((i64)shr(mQ2, E.g - J.em + 2 * ey));  // m Q^2, S = 62 relative to 2^g
    add(a.g[0], p, mx);
    add(a.g[1], p, my);
    add(a.g[2], p, mz);
    if (MODE == F_NEWTON) return;
    a.s0 += plus_hi(mw(p.h, bq.h, 0), cross(p, bq, 0)) >> ey;  // m Q^3 = (m Q^2) Q
    // velocity terms: the dot products' small parts in FP32, the sums in integers
    const V nx = vec(mx), ny = vec(my), nz = vec(mz), wx = vec(J.wx), wy = vec(J.wy), wz = vec(J.wz);
    const Acc uw = dot(I.ux, I.uy, I.uz, wx, wy, wz), un = dot(I.ux, I.uy, I.uz, nx, ny, nz), wn = dot(wx, wy, wz, nx, ny, nz);
    const i64 b = merge<4>((un.h << 4) >> I.d, un.x, I.fd * 0x1p-28f), w = merge<5>(wn.h << 6, wn.x, 0x1p-26f);  // S = 62
    const V wv = vec(bal(w));
    // F = u.w + (w.n)^2 / 2, S = 62
    const B2 f = bal(merge<4>(mw(wv.h, 2 * wv.h, (uw.h << 4) >> I.d), fmaf_(4.f * wv.hf, wv.l, (16.f * I.fd) * uw.x), 0x1p-32f));
    const i64 H = ((i64)((u64)mw(p.h, f.h, 0) << E.lh) + (cross(p, f, 0) >> (32 - E.lh))) >> E.rh;
    const B2 k = bal(b - w);
    const i64 ct = (i64)((u64)mw(p.h, k.h, 0) << E.lt) + (cross(p, k, 0) >> (32 - E.lt));
    a.ct += ct;
    const B2 t = bal(ct);
    add(a.t[0], t, J.wx);
    add(a.t[1], t, J.wy);
    add(a.t[2], t, J.wz);
    // FP64: Phi, U and C, which then joins the integers
    const double qd = scale_down(u2d(Q), 62 + ey - E.q);
    a.dphi = fma_(J.m, qd, a.dphi);
    a.du = fma_(J.mu3, qd, a.du);
    const u64 co = bits_of(fma_(fma_(-I.qe, J.g3, J.g1), qd * qd, J.k));
    const u64 cm = ((co & 0xfffffffffffffULL) | 0x10000000000000ULL) << 9;  // S = 61 of 1.f
    const i64 sg = (i64)co >> 63;
    const B2 C = bal((i64)(((u64)shr(cm, E.c + 1022 - (int)((co >> 52) & 0x7ff)) ^ (u64)sg) - (u64)sg) + H);  // S = 62
    add(a.c[0], C, mx);
    add(a.c[1], C, my);
    add(a.c[2], C, mz);
    if (MODE == F_FORCE_ENERGY) {
        const V bv = vec(bal(b));
        const i64 z = merge<5>(((14 * uw.h) >> I.d) + (mw(bv.h, wv.h, 0) >> 1), fmaf_(14.f * I.fd, uw.x, 0.5f * crossf(bv, wv, 0.f)), 0x1p-32f);  // S = 59
        a.dpsi = fma_(J.m * qd, (double)z, a.dpsi);
    }
}

}  // namespace fix
}  // namespace pn
