// The fixed-point pair terms (pn_fix.cuh) on the CPU, over one star's row: stdin has
//   mode n i eps m0 seed_error, then n lines "sx sy sz vx vy vz m" (BH-relative positions)
// and stdout one line per sum (Gx Gy Gz Phi S0 U Wx Wy Wz Psi): fixed point, FP64 as the plain
// sweep sums it, the errors of the two against long double, and the sum of the terms' magnitudes (for G
// and W without the pair of the star with itself, whose term is zero).
#include <cmath>
#include <cstdio>
#include <vector>

#include "../pn_gb300/csrc/pn_fix.cuh"

using namespace pn::fix;
typedef long double L;

struct Star {
    double s[3], v[3], m;
};

static double two(int e) { return std::ldexp(1.0, e); }
static int mag_exp(float x) { x *= 1.001f; unsigned b; std::memcpy(&b, &x, 4); return (int)(b >> 23) - 126; }

template <typename T> struct Terms { T t[10], mag[10]; };

template <typename T>
static void plain(const std::vector<Star> &st, int i, T eps, T m0, Terms<T> &o) {
    for (int q = 0; q < 10; ++q) o.t[q] = o.mag[q] = 0;
    const Star &a = st[i];
    const T e2 = eps * eps;
    T qe = e2, vi2 = 0;
    for (int k = 0; k < 3; ++k) { qe += (T)a.s[k] * a.s[k]; vi2 += (T)a.v[k] * a.v[k]; }
    for (const Star &b : st) {
        T d[3], dv[3], rho = e2, R = e2, vdj = 0, vdi = 0, dv2 = 0, vv = 0;
        for (int k = 0; k < 3; ++k) {
            d[k] = (T)b.s[k] - a.s[k];
            dv[k] = (T)b.v[k] - a.v[k];
            rho += d[k] * d[k];
            R += (T)b.s[k] * b.s[k];
            vdj += b.v[k] * d[k];
            vdi += a.v[k] * d[k];
            dv2 += dv[k] * dv[k];
            vv += (T)a.v[k] * b.v[k];
        }
        const T Q = 1 / std::sqrt(rho);
        R = 1 / std::sqrt(R);
        const T m = b.m, mu3 = m * R * R * R, c1 = (T)1.25 * m0 * R, c3 = (T)0.25 * m0 * R * R * R, k35 = (T)3.5 * m0 * mu3;
        const T mq3 = m * Q * Q * Q;
        const T br = c1 + c3 * (rho - qe) + vi2 - 2 * dv2 + (T)1.5 * vdj * vdj * Q * Q;
        const T cd = mq3 * br + k35 * Q, cv = mq3 * (4 * vdi - 3 * vdj);
        T x[10];
        for (int k = 0; k < 3; ++k) { x[k] = mq3 * d[k]; x[6 + k] = cd * d[k] + cv * dv[k]; }
        x[3] = m * Q; x[4] = mq3; x[5] = mu3 * Q;
        x[9] = m * Q * (7 * vv + vdi * vdj * Q * Q);
        const T dn = std::sqrt(rho), dvn = std::sqrt(dv2);
        for (int q = 0; q < 10; ++q) o.t[q] += x[q];
        if (&b == &a) {
            for (int q = 3; q < 6; ++q) o.mag[q] += x[q];
            o.mag[9] += x[9];
            continue;
        }
        for (int k = 0; k < 3; ++k) {
            o.mag[k] += mq3 * dn;
            o.mag[6 + k] += (mq3 * (std::fabs(c1) + c3 * std::fabs(rho - qe) + vi2 + 2 * dv2 + (T)1.5 * vdj * vdj * Q * Q) + k35 * Q) * dn
                            + mq3 * (4 * std::fabs(vdi) + 3 * std::fabs(vdj)) * dvn;
        }
        for (int q = 3; q < 6; ++q) o.mag[q] += x[q];
        o.mag[9] += m * Q * (7 * std::fabs(vv) + std::fabs(vdi * vdj) * Q * Q);
    }
}

int main() {
    int mode, n, i;
    double eps, m0, err;
    if (scanf("%d %d %d %lf %lf %lf", &mode, &n, &i, &eps, &m0, &err) != 6) return 2;
    std::vector<Star> st(n);
    for (Star &b : st)
        if (scanf("%lf %lf %lf %lf %lf %lf %lf", &b.s[0], &b.s[1], &b.s[2], &b.v[0], &b.v[1], &b.v[2], &b.m) != 7) return 2;
    const int eL = std::ilogb(eps);
    int ev = -EV_MAX;
    for (const Star &b : st) {
        const int e = speed_exp(b.v[0] * b.v[0] + b.v[1] * b.v[1] + b.v[2] * b.v[2]);
        if (e > ev) ev = e;
    }
    const double eq = std::ldexp(eps, -eL);
    const u64 eps60 = (u64)std::ldexp(eq * eq, 60);
    const int e0 = expo(m0);
    const double eps2 = eps * eps;
    std::vector<StarJ> J(n);
    std::vector<float> mf(n), g1f(n), g3f(n), kf(n), wn(n);
    float un = 0;
    StarI I;
    double vi2 = 0;
    for (int j = 0; j < n; ++j) {
        const Star &b = st[j];
        const double q = b.s[0] * b.s[0] + b.s[1] * b.s[1] + b.s[2] * b.s[2], R = 1.0 / std::sqrt(q + eps2), R3 = R * R * R;
        const double mu3 = b.m * R3, c1 = 1.25 * m0 * R, c3 = 0.25 * m0 * R3, k35 = 3.5 * m0 * mu3;
        const double v2 = b.v[0] * b.v[0] + b.v[1] * b.v[1] + b.v[2] * b.v[2];
        StarJ &p = J[j];
        p.x = to_x96(b.s[0], eL); p.y = to_x96(b.s[1], eL); p.z = to_x96(b.s[2], eL);
        p.wx = bal(to_scaled(b.v[0], W_MANT, 63, 60, ev));
        p.wy = bal(to_scaled(b.v[1], W_MANT, 63, 60, ev));
        p.wz = bal(to_scaled(b.v[2], W_MANT, 63, 60, ev));
        const u64 mm = mantissa(b.m, p.em);
        p.em = mm ? p.em - e0 : -8192;
        p.mh = (unsigned)(mm >> 32);
        p.mhf = (float)p.mh * 0x1p-34f;
        p.ml = (float)(unsigned)mm * 0x1p-34f;
        p.m = b.m;
        p.mu3 = mu3;
        p.g1 = b.m * (c1 - 2.0 * v2);
        p.g3 = b.m * c3;
        p.k = std::fma(b.m, c3, k35);
        mf[j] = (float)(b.m * two(-e0));
        g1f[j] = (float)std::fabs(p.g1 * two(eL - 2 * e0));
        g3f[j] = (float)(p.g3 * two(3 * eL - 2 * e0));
        kf[j] = (float)(p.k * two(3 * eL - 2 * e0));
        wn[j] = std::sqrt((float)(3.0 * v2 * two(-2 * ev))) * 1.00001f;
        if (j == i) {
            un = (float)two(-(ev - speed_exp(v2) < 63 ? ev - speed_exp(v2) : 63));
            I.x = p.x; I.y = p.y; I.z = p.z;
            const int eu = speed_exp(v2);
            I.ux = vec(bal(to_scaled(b.v[0], U_MANT, 62, 62, eu)));
            I.uy = vec(bal(to_scaled(b.v[1], U_MANT, 62, 62, eu)));
            I.uz = vec(bal(to_scaled(b.v[2], U_MANT, 62, 62, eu)));
            I.d = ev - eu < 63 ? ev - eu : 63;
            I.fd = (float)two(-I.d);
            I.qe = q + eps2;
            vi2 = v2;
        }
    }
    const float qef = (float)(I.qe * two(-2 * eL));
    const bool energy = mode == F_ENERGY;
    double tot[12] = {0};
    Sums A;
    double phi = 0, us = 0;
    unsigned rnd = 12345;
    for (int t = 0; t < n; t += 128) {
        const int e = t + 128 < n ? t + 128 : n;
        std::vector<unsigned> yb(128);
        float mg = 0, mc = 0, mh = 0, mt = 0;
        for (int j = t; j < e; ++j) {
            double rho = eq * eq;
            for (int k = 0; k < 3; ++k) { const double d = (st[j].s[k] - st[i].s[k]) * two(-eL); rho += d * d; }
            rnd = rnd * 1664525u + 1013904223u;  // a seed off by at most err
            const float y = (float)((1.0 / std::sqrt(rho)) * (1.0 + err * (2.0 * (rnd / 4294967296.0) - 1.0)));
            std::memcpy(&yb[j - t], &y, 4);
            if (j != i) {
                const float my2 = mf[j] * y * y;
                mh += my2 * wn[j] * (un + 0.5f * wn[j]);
                mt += my2 * (un + wn[j]);
            }
            if (j != i) mg += energy ? mf[j] * y : mf[j] * y * y;
            if (j != i) mc += (g3f[j] * qef + g1f[j]) * (y * y) + kf[j];
        }
        const int lh = lift(mag_exp(mg), mag_exp(mh), LIFT_H), lt = lift(mag_exp(mg), mag_exp(mt), LIFT_T);
        Scale E{mag_exp(mg), 0, 0, -eL, lh, lt};
        join(E, mag_exp(mc) + 2 * e0 - 3 * eL, E.g + e0 - 2 * eL + 2 - lh + 2 * ev);
        clear<F_FORCE_ENERGY>(A);
        for (int j = t; j < e; ++j) {
            const int em = J[j].em;
            if (j == i) J[j].em = -8192;
            if (mode == 0) pair<F_NEWTON>(A, I, J[j], E, yb[j - t], eps60);
            else if (mode == 1) pair<F_FORCE>(A, I, J[j], E, yb[j - t], eps60);
            else if (mode == 2) pair<F_ENERGY>(A, I, J[j], E, yb[j - t], eps60);
            else pair<F_FORCE_ENERGY>(A, I, J[j], E, yb[j - t], eps60);
            J[j].em = em;
            if ((j & 7) == 7 || j + 1 == e) {
                if (energy) fold<F_ENERGY>(A);
                else fold<F_FORCE>(A);
            }
        }
        const int gn = E.g + e0 - (energy ? 1 : 2) * eL;
        for (int k = 0; k < 3; ++k) {
            tot[k] += (double)top(A.g[k]) * two(gn - 62);
            tot[4 + k] += (double)top(A.t[k]) * two(gn + 2 - lt - 62 + 2 * ev);
            tot[7 + k] += (double)top(A.c[k]) * two(E.c - 62);
        }
        tot[3] += (double)A.s0 * two(gn - eL - 60);
        tot[10] += (double)A.ct * two(gn + 2 - lt - 62 + ev);
        if (energy) {
            tot[0] += (double)A.phi * two(gn - 62);
            tot[1] += (double)top(A.psi) * two(gn - 62 + 2 * ev);
        }
        tot[11] += A.dpsi * two(2 * ev - 61);
        phi += A.dphi;
        us += A.du;
    }
    const double Qs = 1.0 / eps, mi = st[i].m;
    double f[10] = {0};
    if (energy) {
        f[3] = std::fma(mi, Qs, tot[0]);
        f[9] = std::fma(7.0 * vi2, mi * Qs, tot[1]);
    } else {
        for (int k = 0; k < 3; ++k) {
            f[k] = tot[k];
            f[6 + k] = std::fma(-W_SCALE * tot[10], st[i].v[k], tot[4 + k]) + std::fma(-vi2, f[k], tot[7 + k]);
        }
        f[3] = phi;
        f[4] = std::fma(mi, (double)(1.0L / ((L)eps * eps * eps)), tot[3]);
        f[5] = us;
        f[9] = tot[11];
    }
    Terms<double> d;
    Terms<L> x;
    plain<double>(st, i, eps, m0, d);
    plain<L>(st, i, (L)eps, (L)m0, x);
    for (int q = 0; q < 10; ++q)
        printf("%.17g %.17g %.17g %.17g %.17g\n", f[q], d.t[q], (double)((L)f[q] - x.t[q]), (double)((L)d.t[q] - x.t[q]),
               (double)x.mag[q]);
    return 0;
}
