// pn_fix.cuh -- the star-pair terms of the FP64 sweeps in 64-bit fixed point.
//
// A GB300 SM issues one FP64 warp instruction every 16 cycles (64 per scheduler; measured) but a
// 32 x 32 + 64 bit integer multiply-add every second cycle per scheduler, so a product of two
// 62-bit numbers on the integer pipe costs about a tenth of an FP64 multiply and carries 9 more bits.  The
// pair terms are therefore formed as fixed-point numbers of 58 to 62 fraction bits; no
// intermediate has fewer bits than a double.  Host and device compile the same functions (the
// arithmetic is integer, so a CPU run gives the device's bits for the same seed).
//
// Units.  Lengths in units of 2^eL, the power of two with 1 <= eps / 2^eL < 2; masses in units of
// the power of two of the BH's mass; velocities in units of 2^ev, the power of two above the fastest
// |u| (below) of the two tiles at hand.
// "S = k" at a variable says that it holds its value times 2^k.
//
// One pair (i, j), d = x_j - x_i:
//   X   BH-relative positions, 96 bits, S = 62: d is exact to 2^-62 eps.
//   y   FP32 estimate of Q = (|d|^2 + eps^2)^(-1/2) (MUFU), raised above Q: y = f 2^-ey, 1 <= f < 2.
//   D   = d 2^-ey, S = 62: |D| <= 1 whatever the distance (the only per-pair normalisation)
//   RHO = |D|^2 + eps^2 2^(-2 ey), S = 60, in (1/4, 1]
//   r   = 1 - RHO f^2, |r| < 2^-18.8;  Q 2^ey = f (1 + r/2 + 3 r^2/8): the binomial series of
//         (1 - r)^(-1/2), whose next term is below 2^-58 (2^-60 on average).
//   n   = d Q, S = 59, the softened unit vector
// and the terms of pn_device.cuh's sums, with w_j = sqrt(3) v_j, u_i = (4 / sqrt(3)) v_i:
//   G   += (m Q^2) n         Phi += m Q      S0 += m Q^3      U += mu3 Q
//   W   += [m Q^2 (u.w + (w.n)^2 / 2)] n + ct w,   ct = m Q^2 (u.n - w.n)
//   W64 += [(g1 - g3 qe_i) Q^2 + k] n,  g1 = m (c1 - 2 |v|^2), g3 = m c3, k = g3 + k35
//          (FP64: its coefficients span the range of R_j^3; c3 rho Q^2 = c3 is in k)
//   Psi += m Q (7 u.w + (u.n)(w.n))  (four times the energy's)
// The sums of one j-tile are accumulated as integers relative to the tile's own sum of
// magnitudes (a first FP32 pass over the tile finds its exponent), so the smallest kept bit is
// 2^-62 of that sum; the tile sums are added in FP64.  The pair of a star with itself (d = 0: no G,
// no W) would raise that scale to m / eps^2; it is left out and its Phi, S0, U, Psi added in FP64.
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
constexpr int EV_MAX = 300;    // speeds below 2^300 (slower ones than 2^-300 count as at rest)
constexpr double W_SCALE = 1.7320508075688772935;  // w / v
constexpr u64 W_MANT = 0xDDB3D742C265539DULL;      // sqrt(3) 2^63
constexpr u64 U_MANT = 0x93CD3A2C8198E269ULL;      // 4 / sqrt(3) 2^62

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
PNF u64 mulhi(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}
// a >> s for 0 <= s (0 from 64 on)
PNF u64 shr(u64 a, int s) {
#ifdef __CUDA_ARCH__
    u64 r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(s));
    return r;
#else
    return s > 63 ? 0 : a >> s;
#endif
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

// ------------------------------------------------------------------ one pair
enum : int { F_NEWTON = 0, F_FORCE = 1, F_ENERGY = 2, F_FORCE_ENERGY = 3 };  // as PairMode

struct StarI {  // the accumulating star
    X96 x, y, z;
    B2 ux, uy, uz;  // u_i, S = 62
    double qe;      // |s_i|^2 + eps^2
};
struct StarJ {
    X96 x, y, z;
    u64 m, m3;      // mantissas of m and mu3 = m R^3
    int em, em3;    // their exponents (in the units above)
    B2 wx, wy, wz;  // w_j, S = 60
    double g1, g3, k;  // FP64 coefficients (g1, g3 times 2^(-62 - 2 eL))
};
struct Scale {  // the tile's exponents: sum of m Q^2, m Q, m Q^3, mu3 Q is below 2^e
    int g, p, s, u;
};
struct Sums {
    i64 gh[3], gx[3];  // G: h 2^64 + x 2^32, S = 121 relative to 2^g
    i64 wh[3], wx[3];  // W: likewise, S = 121
    i64 phi, s0, u;    // S = 62, 61, 62 relative to 2^p, 2^s, 2^u
    i64 ct;            // S = 61 relative to 2^g
    i64 ph, px;        // Psi: h 2^64 + x 2^32, S = 120 relative to 2^p
    double w[3];       // W64 (times 2^59)
};

template <int MODE> PNF void clear(Sums &a) {
    for (int k = 0; k < 3; ++k) a.gh[k] = a.gx[k] = a.wh[k] = a.wx[k] = 0;
    a.phi = a.s0 = a.u = a.ct = a.ph = a.px = 0;
}

// Moves the cross sums' upper halves into the high sums; at least every 4 pairs (the cross sums
// of 4 pairs stay below 2^63: see the bounds at pair()).
template <int MODE> PNF void carry(Sums &a) {
    if (MODE != F_ENERGY) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a.gh[k] += a.gx[k] >> 32;
            a.gx[k] &= 0xffffffffLL;
            if (MODE != F_NEWTON) {
                a.wh[k] += a.wx[k] >> 32;
                a.wx[k] &= 0xffffffffLL;
            }
        }
    }
    if (MODE == F_ENERGY || MODE == F_FORCE_ENERGY) {
        a.ph += a.px >> 32;
        a.px &= 0xffffffffLL;
    }
}

PNF double scale_down(double x, int e) {  // x 2^-e, x > 0 and normal, result normal
#ifdef __CUDA_ARCH__
    return __hiloint2double(__double2hiint(x) - (e << 20), __double2loint(x));
#else
    u64 b = bits_of(x) - ((u64)e << 52);
    double r;
    std::memcpy(&r, &b, 8);
    return r;
#endif
}

// rounding constants of right shifts
constexpr i64 half(int s) { return 1LL << (s - 1); }

// u.w (S = 58 as h + x / 2^32), and u.n, w.n with S = 61
struct Dots {
    i64 vh, vx, un, wn;
};
PNF Dots dots(const StarI &I, const StarJ &J, B2 nx, B2 ny, B2 nz) {
    Dots d;
    d.vx = cross(I.uz, J.wz, cross(I.uy, J.wy, cross(I.ux, J.wx, 0)));
    d.vh = mw(I.uz.h, J.wz.h, mw(I.uy.h, J.wy.h, mw(I.ux.h, J.wx.h, 0)));
    const i64 ux = cross(I.uz, nz, cross(I.uy, ny, cross(I.ux, nx, half(28))));
    const i64 uh = mw(I.uz.h, nz.h, mw(I.uy.h, ny.h, mw(I.ux.h, nx.h, 0)));
    const i64 wx = cross(J.wz, nz, cross(J.wy, ny, cross(J.wx, nx, half(26))));
    const i64 wh = mw(J.wz.h, nz.h, mw(J.wy.h, ny.h, mw(J.wx.h, nx.h, 0)));
    d.un = (uh << 4) + (ux >> 28);
    d.wn = (wh << 6) + (wx >> 26);
    return d;
}
// Psi's term: m Q (7 u.w + (u.n)(w.n)); p = m Q (S = 62), the bracket S = 58 (below 6.1)
PNF void psi_term(Sums &a, const Dots &d, B2 p) {
    const B2 un = bal(d.un), wn = bal(d.wn);
    const B2 z = bal(7 * d.vh + mw(un.h, wn.h, (7 * (d.vx >> 3) + (cross(un, wn, half(32)) >> 3)) >> 29));
    a.ph = mw(p.h, z.h, a.ph);
    a.px = cross(p, z, a.px);
}

// One pair.  ybits: the bits of the FP32 seed y (0 < y <= 1 + 2^-20).  eps60: eps^2 in the units
// above, S = 60 (1 <= eps^2 < 4).
// Bounds: |D| <= 1 (+ 2^-20), |n| <= 1, |u| < 1 and |w| < 3/4 (the unit 2^ev), the tile's sum of P <= 2^62.
//   cross sums of G, 4 pairs: sum Ph nl <= 2^30 2^31, Pl nh <= 4 2^31 2^27: 1.5 2^61
//   cross sums of W, 4 pairs: |H| <= 1.03 2^62 in all, |ct| <= 1.75 2^61 in all, hence
//     Hh nl <= 1.03 2^61, Hl nh <= 2^60, cth wl <= 0.88 2^61, ctl wh <= 0.75 2^61: 3.2 2^61 < 2^63
//   cross sums of Psi, 4 pairs: Ph zl <= 2^61, Pl zh <= 4 2^31 6.1 2^26: 1.8 2^61
template <int MODE>
PNF void pair(Sums &a, const StarI &I, const StarJ &J, const Scale &E, unsigned ybits, u64 eps60) {
    ybits += 8;  // a seed above Q (by 2^-21 .. 2^-20 less its error): Q 2^ey < 2, so Q^2 and Q^3 fit
    const int ey = 127 - (int)(ybits >> 23);
    const unsigned F = (ybits & 0x7fffffu) | 0x800000u;
    const B2 dx = bal(diff_shift(J.x, I.x, ey)), dy = bal(diff_shift(J.y, I.y, ey)),
             dz = bal(diff_shift(J.z, I.z, ey));
    // RHO, S = 60
    const i64 dt = mw(dz.h, dz.l, mw(dy.h, dy.l, mw(dx.h, dx.l, half(31))));
    const u64 rho = (u64)(mw(dz.h, dz.h, mw(dy.h, dy.h, mw(dx.h, dx.h, dt >> 31)))) + shr(eps60, 2 * ey);
    // r = 1 - RHO f^2, S = 58
    const unsigned F8 = F << 8;
    const u64 U = muw((unsigned)(rho >> 32), F8, muw((unsigned)rho, F8, half(32)) >> 32);  // RHO f, S = 59
    const i64 r = (i64)((1ULL << 58) - muw((unsigned)(U >> 32), F8, muw((unsigned)U, F8, half(32)) >> 32));
    const int rs = (int)(r >> 12);                          // S = 46 (below 2^28)
    const int rsq = (int)(mw(rs, rs, 0) >> 32);             // r^2, S = 60
    const i64 c = mw(6, rsq, r << 5);                       // r/2 + 3 r^2/8, S = 64
    const int F7 = (int)(F << 7);
    const u64 Q = (u64)mw(F7, (int)(c >> 32), (i64)(((u64)F7 << 32) | (muw((unsigned)F7, (unsigned)c, 0) >> 32)));  // S = 62
    const B2 q = bal((i64)(Q >> 1));  // S = 61
    const i64 n0 = mw(dx.h, q.h, cross(dx, q, half(32)) >> 32), n1 = mw(dy.h, q.h, cross(dy, q, half(32)) >> 32),
              n2 = mw(dz.h, q.h, cross(dz, q, half(32)) >> 32);
    const B2 nx = bal(n0), ny = bal(n1), nz = bal(n2);  // S = 59
    if (MODE == F_ENERGY) {
        const i64 pq = (i64)shr(mulhi(J.m, Q), E.p - J.em + ey);  // m Q, S = 62
        a.phi += pq;
        psi_term(a, dots(I, J, nx, ny, nz), bal(pq));
        return;
    }
    const u64 Q2 = mulhi(Q, Q) << 2;  // S = 62
    const B2 p = bal((i64)shr(mulhi(J.m, Q2), E.g - J.em + 2 * ey));  // m Q^2, S = 62 relative to 2^g
    a.gh[0] = mw(p.h, nx.h, a.gh[0]);
    a.gh[1] = mw(p.h, ny.h, a.gh[1]);
    a.gh[2] = mw(p.h, nz.h, a.gh[2]);
    a.gx[0] = cross(p, nx, a.gx[0]);
    a.gx[1] = cross(p, ny, a.gx[1]);
    a.gx[2] = cross(p, nz, a.gx[2]);
    if (MODE == F_NEWTON) return;
    const u64 Q3 = mulhi(Q2, Q) << 1;  // S = 61
    const i64 pq = (i64)shr(mulhi(J.m, Q), E.p - J.em + ey);
    a.phi += pq;
    a.s0 += (i64)shr(mulhi(J.m, Q3), E.s - J.em + 3 * ey);
    a.u += (i64)shr(mulhi(J.m3, Q), E.u - J.em3 + ey);
    // velocity terms
    const Dots v = dots(I, J, nx, ny, nz);
    const B2 wb = bal(v.wn), kb = bal(v.un - v.wn);
    // F = u.w + (w.n)^2 / 2, S = 60
    const B2 f = bal((v.vh << 2) + (mw(wb.h, wb.h, 0) << 1) + ((v.vx + mw(wb.h, wb.l, half(30))) >> 30));
    const B2 H = bal((mw(p.h, f.h, 0) << 4) + (cross(p, f, half(28)) >> 28));   // S = 62
    const i64 ct = (mw(p.h, kb.h, 0) << 2) + (cross(p, kb, half(30)) >> 30);    // S = 61
    a.ct += ct;
    const B2 cb = bal(ct);
    a.wh[0] = mw(H.h, nx.h, mw(cb.h, J.wx.h, a.wh[0]));
    a.wh[1] = mw(H.h, ny.h, mw(cb.h, J.wy.h, a.wh[1]));
    a.wh[2] = mw(H.h, nz.h, mw(cb.h, J.wz.h, a.wh[2]));
    // (with the products of the low limbs: slow stars leave H and ct few high bits)
    a.wx[0] = cross(H, nx, cross(cb, J.wx, a.wx[0] + (mw(H.l, nx.l, mw(cb.l, J.wx.l, 0)) >> 32)));
    a.wx[1] = cross(H, ny, cross(cb, J.wy, a.wx[1] + (mw(H.l, ny.l, mw(cb.l, J.wy.l, 0)) >> 32)));
    a.wx[2] = cross(H, nz, cross(cb, J.wz, a.wx[2] + (mw(H.l, nz.l, mw(cb.l, J.wz.l, 0)) >> 32)));
    if (MODE == F_FORCE_ENERGY) psi_term(a, v, bal(pq));
    // FP64 part (g1, g3 carry 2^-62 for Q2's S)
#ifdef __CUDA_ARCH__
    const double q2 = scale_down(__ull2double_rn(Q2), 2 * ey);
    const double co = ::fma(::fma(-I.qe, J.g3, J.g1), q2, J.k);
    a.w[0] = ::fma(co, __ll2double_rn(n0), a.w[0]);
    a.w[1] = ::fma(co, __ll2double_rn(n1), a.w[1]);
    a.w[2] = ::fma(co, __ll2double_rn(n2), a.w[2]);
#else
    const double q2 = scale_down((double)Q2, 2 * ey);
    const double co = __builtin_fma(__builtin_fma(-I.qe, J.g3, J.g1), q2, J.k);
    a.w[0] = __builtin_fma(co, (double)n0, a.w[0]);
    a.w[1] = __builtin_fma(co, (double)n1, a.w[1]);
    a.w[2] = __builtin_fma(co, (double)n2, a.w[2]);
#endif
}

// h 2^64 + x 2^32 (x carried: 0 <= x < 2^32) divided by 2^(64 - B)
template <int B> PNF i64 top(i64 h, i64 x) { return (i64)((u64)h << B) + (x >> (32 - B)); }
// bits kept, and the S of the result
constexpr int TOP_G = 5, S_G = 62, TOP_W = 4, S_W = 61, TOP_P = 4, S_P = 60;

}  // namespace fix
}  // namespace pn
