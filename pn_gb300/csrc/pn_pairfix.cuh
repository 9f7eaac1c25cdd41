// pn_pairfix.cuh -- the FP64 pair sweep on the integer pipes (the pair terms: pn_fix.cuh).
//
// The same sums, to FP64 accuracy, as k_pair<double, MODE> (pn_pair.cuh), which is bound by the
// FP64 pipe.  A CTA of 128 threads owns 128 / JS stars i; JS consecutive lanes share one i and
// split each j-tile; blockIdx.y selects one of gsplit ranges of j-tiles.  Tiles of 128 stars are
// copied to shared memory by the TMA engine, double buffered, with bounded waits.  Each tile is
// passed twice: in FP32 for the magnitude of the tile's sums (the integer sums' exponents), then
// for the sums themselves, which are added to FP64 totals in shared memory at the tile's end.
//
// Why: FP64 issues one warp instruction per 64 cycles and scheduler here, so k_pair<double>'s 51 per
// pair take that pipe 3,264 cycles per warp of pairs (3,610 measured); this form takes 672, of which the
// multiply-add pipe is busy 71 % and the FP64 pipe 59 % (6 operations per pair). One force evaluation at
// N = 65,536: 385 -> 71.5 ms, N = 10,000: 9.3 -> 1.85 ms.  Its error against long double sums is below
// the FP64 sweep's (medians at N = 2,049: 1.46e-16 against 2.22e-16 at c = 1000, 5.2e-16 against
// 7.4e-16 at c = 1).  Measured on the way there, at N = 65,536: every product in integers and C's sum
// in FP64 (4 conversions and 5 FMA per pair) 104 ms; the dot products' small parts in FP32, Phi and U in
// FP64 and C's sum in integers 88.2 ms; one sum along n for C and H 77.3 ms, carry additions 71.7 ms; the sums' small
// parts in FP32 too (before that) 76 against 88 ms, but with twice the FP64 sweep's error at c = 1.
//
// n = d Q has an absolute error of 2^-61, whatever d: G's is up to 2^-61 sum m Q^2, where FP64's is about 2^-53 of
// the terms, sum m Q^2 |n|.  So a row whose stars (of its j-range, weighted by m Q^2) lie so far inside the softening
// that the mean of |n|^2 may be below 1 / 128 is formed once more in FP64, by the whole CTA, before it leaves: two
// stars 1e-8 eps apart and alone kept 5e-11 of their force without that.  For one such pair to dominate a
// row its stars have to be within 0.13 eps; of N = 65,536 stars at eps = 0.04 / N^(1/3), one in a hundred systems has one.
//
// The integer range covers the systems that k_prep has checked star by star (fix::in_range: positions within
// 2^24 eps, masses zero or 2^-32 .. 2^59 of the BH's, which is positive and not extreme, speeds up to that of light
// and somewhat beyond, all finite); for any other the same launch runs k_pair<double>'s block instead.
#pragma once

#include "pn_fix.cuh"
#include "pn_pair.cuh"

namespace pn {

constexpr int FIX_TJ = 128;
constexpr int FIX_GENERAL_JS = 16;  // lanes per star in k_pair<double>'s block
// Rows with sum m Q^2 |n|^2 < sum m Q^2 / NEAR go to FP64 (fix_row_fp64).
constexpr float NEAR = 128.f;

template <int MODE> struct FixInfo {
    static constexpr int NG = MODE == MODE_NEWTON ? 5 : MODE == MODE_ENERGY ? 8 : 11;  // streamed 16-byte groups
    // sums over the tiles in shared memory: G; or G, S0, W along n, ct, W along w, Phi, U (and Psi); or Phi, Psi
    static constexpr int NT = MODE == MODE_NEWTON ? 3 : MODE == MODE_ENERGY ? 2 : MODE == MODE_FORCE ? 13 : 14;
};

template <int MODE>
__host__ __device__ constexpr size_t fix_tot_bytes() {
    return (size_t)PAIR_NT * (FixInfo<MODE>::NT * sizeof(double) + sizeof(float));
}
template <int MODE>
inline size_t fix_smem_bytes() {
    const size_t fast = 128 + fix_tot_bytes<MODE>() + 2 * (size_t)FixInfo<MODE>::NG * FIX_TJ * 16;
    const size_t gen = pair_smem_bytes(ModeInfo<MODE>::NG64, FIX_TJ, sizeof(double2));
    return fast > gen ? fast : gen;
}

// a velocity component (h, l) of the pack, 2^-s times it
__device__ __forceinline__ fix::B2 slower(unsigned h, unsigned l, int s) {
    return fix::bal(fix::limbs((int)h, (int)l) >> s);
}
// exponent e with x < 2^e, x >= 0 (x within FP32 range)
__device__ __forceinline__ int mag_exp(float x) {
    return (int)(__float_as_uint(x * 1.001f) >> 23) - 126;
}
__device__ __forceinline__ double pow2(int e) {  // 2^e, -1022 <= e <= 1023
    return __hiloint2double((e + 1023) << 20, 0);
}

// Row i's sums with the stars j0 .. j1 - 1 in FP64, by the whole CTA, to out[slot * npad].  red: 4 NACC doubles of
// shared memory.
template <int MODE>
__device__ __forceinline__ void fix_row_fp64(const double2 *pk, int npad, int i, int j0, int j1, double eps2, double *red,
                                          double *out) {
    constexpr int NACC = ModeInfo<MODE>::NACC;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto grp = [&](int g, int j) { return pk[(size_t)g * npad + j]; };
    IState<double> I{};
    I.ex = grp(0, i).x;
    I.ey = grp(0, i).y;
    I.ez = grp(1, i).x;
    I.vx = grp(2, i).x;
    I.vy = grp(2, i).y;
    I.vz = grp(3, i).x;
    I.qe = grp(5, i).y;
    I.vi2 = pn_fma(I.vz, I.vz, pn_fma(I.vy, I.vy, I.vx * I.vx));
    double acc[NACC];
#pragma unroll
    for (int q = 0; q < NACC; ++q) acc[q] = 0.0;
#pragma unroll 1
    for (int j = j0 + tid; j < j1; j += PAIR_NT) {
        const double2 g0 = grp(0, j), g1 = grp(1, j), g2 = grp(2, j), g3 = grp(3, j), g4 = grp(4, j), g5 = grp(5, j);
        pair_accumulate<MODE, double>(acc, I, g0.x, g0.y, g1.x, 0.0, 0.0, 0.0, g1.y, g2.x, g2.y, g3.x, g3.y, g4.x, g4.y,
                                      g5.x, eps2);
    }
#pragma unroll
    for (int q = 0; q < NACC; ++q) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], off);
        if (lane == 0) red[warp * NACC + q] = acc[q];
    }
    __syncthreads();
    if (tid < NACC) out[(size_t)tid * npad] = (red[tid] + red[NACC + tid]) + (red[2 * NACC + tid] + red[3 * NACC + tid]);
    __syncthreads();  // red is free again
}

template <int MODE, int JS>
__device__ __forceinline__ bool fix_block(const PairArgs &a, int ibase, int split, uint64_t *bars, double *tot,
                                          uint4 *buf, uint32_t &seq) {
    using namespace fix;
    constexpr int NT = PAIR_NT, NI = NT / JS, NG = FixInfo<MODE>::NG, TJ = FIX_TJ;
    constexpr int NACC = ModeInfo<MODE>::NACC;
    constexpr bool FORCE = mode_has_force(MODE);
    constexpr bool PSI = MODE == MODE_ENERGY || MODE == MODE_FORCE_ENERGY;
    const int tid = threadIdx.x, sub = tid % JS, grp = tid / JS;
    const int t0 = (int)(((long long)a.ntiles * split) / a.gsplit);
    const int t1 = (int)(((long long)a.ntiles * (split + 1)) / a.gsplit);
    const int i = ibase + grp;
    const bool valid = i < a.nstar;
    const int il = valid ? i : 0;
    const uint4 *pk = a.fpack;
    const float epsf = (float)((double)a.fu.eps60 * (1.0 / 1152921504606846976.0));

    StarI I;
    {
        const uint4 g2 = pk[(size_t)2 * a.npad + il], g3 = pk[(size_t)3 * a.npad + il];
        I.x = {g2.x, g2.y, g2.z};
        I.y = {g2.w, g3.x, g3.y};
        I.z = {g3.z, g3.w, pk[(size_t)4 * a.npad + il].x};
        const uint4 u1 = pk[(size_t)12 * a.npad + il];
        I.qe = __hiloint2double((int)u1.w, (int)u1.z);
    }
    // u_i is stored in its own velocity unit 2^eu, w_j in that of its tile; a pair of tiles uses the larger
    // of theirs
    const int ei = __float_as_int(a.torg[ibase / TJ].pad0);
    int ev = -100000, eu = 0;
    if constexpr (MODE != MODE_NEWTON) {
        const uint4 k = pk[(size_t)10 * a.npad + il], u0 = pk[(size_t)11 * a.npad + il], u1 = pk[(size_t)12 * a.npad + il];
        I.ux = vec(slower(u0.x, u0.y, 0));
        I.uy = vec(slower(u0.z, u0.w, 0));
        I.uz = vec(slower(u1.x, u1.y, 0));
        eu = (int)k.w;
    }
    const int e0 = fix::expo(a.m[0]), eL = a.fu.eL;
    const int eg = e0 - (MODE == MODE_ENERGY ? 1 : 2) * eL;  // exponents of the units of m Q^2 (m Q)
    const int ec = 2 * e0 - 3 * eL;                          // ... and of C
    const float qef = FORCE ? (float)(I.qe * pow2(-2 * eL)) : 0.f;
    // the i position in units of 2^eL as an FP32 pair (for the seeds' differences)
    float sh[3], sl[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double s = a.spos[(size_t)k * a.npad + il] * a.fu.inv_len;
        sh[k] = (float)s;
        sl[k] = (float)(s - (double)sh[k]);
    }
    Sums A;
    // sum of m Q^2 (units; without S0, of m Q^2 (1 - NEAR |n|^2)) over this lane's stars
    float &near = reinterpret_cast<float *>(tot + FixInfo<MODE>::NT * NT)[tid];
    near = 0.f;
    if (sub == 0)
#pragma unroll
        for (int q = 0; q < FixInfo<MODE>::NT; ++q) tot[q * NT + grp] = 0.0;

    constexpr uint32_t gbytes = TJ * 16u;
    auto issue = [&](int t, int stage) {
        mbar_arrive_expect_tx(&bars[stage], NG * gbytes);
#pragma unroll
        for (int g = 0; g < NG; ++g)
            bulk_g2s(buf + (size_t)(stage * NG + g) * TJ, pk + (size_t)g * a.npad + (size_t)t * TJ, gbytes, &bars[stage]);
    };
    if (tid == 0 && t0 < t1) issue(t0, (int)(seq & 1u));

    for (int t = t0; t < t1; ++t) {
        const uint32_t it = seq + (uint32_t)(t - t0);
        const int stage = (int)(it & 1u);
        const uint32_t phase = (it >> 1) & 1u;
        const bool next = t + 1 < t1;
        if (tid == 0 && next) issue(t + 1, stage ^ 1);
        const bool ok = mbar_wait_bounded(&bars[stage], phase);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicOr(a.err, DEVERR_TIMEOUT);
                mbar_wait_bounded(&bars[stage], phase);
                if (next) mbar_wait_bounded(&bars[stage ^ 1], ((it + 1) >> 1) & 1u);
            }
            return false;
        }
        const uint4 *b = buf + (size_t)stage * NG * TJ;
        const int jself = i - t * TJ;  // the star itself, where this tile holds it
        if constexpr (MODE != MODE_NEWTON) {
            const int et = __float_as_int(a.torg[t].pad0), e = max(ei, et);
            if (e != ev) {
                ev = e;
                I.d = min(e - eu, 63);
                I.fd = __int_as_float((127 - I.d) << 23);
            }
            if (e > et) {  // (the whole CTA) bring the tile's velocities to the larger unit, in place
                uint4 *q = buf + (size_t)(stage * NG + 5) * TJ + tid;
                const uint4 g5 = q[0], g6 = q[TJ];
                const int sft = min(e - et, 63);
                const B2 wx = slower(g5.x, g5.y, sft), wy = slower(g5.z, g5.w, sft), wz = slower(g6.x, g6.y, sft);
                q[0] = make_uint4((unsigned)wx.h, (unsigned)wx.l, (unsigned)wy.h, (unsigned)wy.l);
                q[TJ] = make_uint4((unsigned)wz.h, (unsigned)wz.l, g6.z, g6.w);
                fence_before_bulk();  // (the stage is refilled by a bulk copy)
                __syncthreads();
            }
        }
        float ex, ey, ez, lx, ly, lz;  // s_i relative to the tile's origin, hi and lo
        {
            const TileOrigin &o = a.torg[t];
            float e;
            ex = two_diff(sh[0], o.hx, e);
            lx = e + (sl[0] - o.lx);
            ey = two_diff(sh[1], o.hy, e);
            ly = e + (sl[1] - o.ly);
            ez = two_diff(sh[2], o.hz, e);
            lz = e + (sl[2] - o.lz);
        }
        auto seed = [&](const float4 &h, const float4 &l) {
            const float dx = (h.x - ex) + (l.x - lx), dy = (h.y - ey) + (l.y - ly), dz = (h.z - ez) + (l.z - lz);
            float y;
            asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, epsf)))));
            return y;
        };
        // ---- the tile's sums in FP32: their exponents
        Scale E;
        {
            float mg = 0.f, mb = 0.f, mc = 0.f, mh = 0.f, mt = 0.f;
            const float down = FORCE ? exp2f((float)(__float_as_int(a.torg[t].pad0) - ev)) : 0.f;  // w to units of 2^ev
#pragma unroll 4
            for (int j = sub; j < TJ; j += JS) {
                const float4 h = reinterpret_cast<const float4 *>(b)[j], l = reinterpret_cast<const float4 *>(b)[TJ + j];
                const float y = seed(h, l);
                const float my = j == jself ? 0.f : h.w * y;
                const float my2 = my * y;
                mg += MODE == MODE_ENERGY ? my : my2;
                if constexpr (MODE == MODE_NEWTON) mb = fmaf(my2, y * y, mb);
                if constexpr (FORCE) {
                    const float4 g7 = reinterpret_cast<const float4 *>(b)[7 * TJ + j];
                    mc += j == jself ? 0.f : fmaf(fmaf(g7.z, qef, g7.y), y * y, g7.w);
                    const float wn = __uint_as_float(b[10 * TJ + j].z) * down;  // |F| <= |u| |w| + |w|^2 / 2, |ct| <= |u| + |w|, |u| <= 2^-d
                    mh = fmaf(my2 * wn, fmaf(0.5f, wn, I.fd), mh);
                    mt = fmaf(my2, I.fd + wn, mt);
                }
            }
            if constexpr (MODE == MODE_NEWTON) near = fmaf(NEAR * epsf, mb, fmaf(1.f - NEAR, mg, near));
#pragma unroll
            for (int off = JS / 2; off > 0; off >>= 1) {
                mg += __shfl_xor_sync(0xffffffffu, mg, off);
                if constexpr (FORCE) {
                    mc += __shfl_xor_sync(0xffffffffu, mc, off);
                    mh += __shfl_xor_sync(0xffffffffu, mh, off);
                    mt += __shfl_xor_sync(0xffffffffu, mt, off);
                }
            }
            if constexpr (FORCE) near += mg;
            E.g = mag_exp(mg);
            E.q = -eL;
            E.lh = lift(E.g, mag_exp(mh), LIFT_H);
            E.lt = lift(E.g, mag_exp(mt), LIFT_T);
            join(E, mag_exp(mc) + ec, E.g + eg + 2 - E.lh + 2 * ev);
        }
        // ---- the sums
        clear<MODE>(A);
        constexpr int FOLD = TJ / JS < 8 ? TJ / JS : 8;
        for (int j0 = sub; j0 < TJ; j0 += FOLD * JS) {
#pragma unroll 4  // (2: 1 % slower; 8: 28 %, the loop leaves the instruction cache)
            for (int j = j0; j < j0 + FOLD * JS; j += JS) {
                const float4 h = reinterpret_cast<const float4 *>(b)[j], l = reinterpret_cast<const float4 *>(b)[TJ + j];
                const uint4 g2 = b[2 * TJ + j], g3 = b[3 * TJ + j], g4 = b[4 * TJ + j];
                auto uf = [](unsigned u) { return __uint_as_float(u); };
                StarJ J;
                J.x = {g2.x, g2.y, g2.z};
                J.y = {g2.w, g3.x, g3.y};
                J.z = {g3.z, g3.w, g4.x};
                J.mh = g4.y;
                J.mhf = uf(g4.z);
                J.ml = uf(g4.w);
                J.em = j == jself ? -8192 : __float_as_int(l.w);
                if constexpr (MODE != MODE_NEWTON) {
                    const uint4 g5 = b[5 * TJ + j], g6 = b[6 * TJ + j];
                    J.wx = {(int)g5.x, (int)g5.y};
                    J.wy = {(int)g5.z, (int)g5.w};
                    J.wz = {(int)g6.x, (int)g6.y};
                }
                if constexpr (FORCE) {
                    const double2 g8 = reinterpret_cast<const double2 *>(b)[8 * TJ + j], g9 = reinterpret_cast<const double2 *>(b)[9 * TJ + j];
                    J.m = g8.x;
                    J.mu3 = g8.y;
                    J.g1 = g9.x;
                    J.g3 = g9.y;
                    J.k = reinterpret_cast<const double2 *>(b)[10 * TJ + j].x;
                }
                fix::pair<MODE>(A, I, J, E, __float_as_uint(seed(h, l)), a.fu.eps60);
            }
            fold<MODE>(A);
        }
        // ---- the JS lanes' integer sums share their exponents: added exactly; then the FP64 totals
        i64 v[FixInfo<MODE>::NT];
        int ve[FixInfo<MODE>::NT];  // exponent of the value's unit
        const int gn = E.g + eg;
        if constexpr (MODE == MODE_ENERGY) {
            v[0] = A.phi;
            ve[0] = gn - 62;
            v[1] = top(A.psi);
            ve[1] = gn - 60 + 2 * ev - 2;
        } else {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                v[k] = top(A.g[k]);
                ve[k] = gn - 62;
            }
        }
        if constexpr (FORCE) {
            v[3] = A.s0;
            ve[3] = gn - eL - 60;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                v[4 + k] = top(A.c[k]);
                ve[4 + k] = E.c - 62;
                v[8 + k] = top(A.t[k]);
                ve[8 + k] = gn + 2 - E.lt - 62 + 2 * ev;
            }
            v[7] = A.ct;
            ve[7] = gn + 2 - E.lt - 62 + ev;
        }
        constexpr int NI64 = FORCE ? 11 : FixInfo<MODE>::NT;
#pragma unroll
        for (int q = 0; q < NI64; ++q) {
            i64 x = v[q];
#pragma unroll
            for (int off = JS / 2; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
            if (sub == 0) tot[q * NT + grp] = ::fma(__ll2double_rn(x), pow2(ve[q]), tot[q * NT + grp]);
        }
        if constexpr (FORCE) {
            const double d[3] = {A.dphi, A.du, A.dpsi};
#pragma unroll
            for (int q = 0; q < FixInfo<MODE>::NT - NI64; ++q) {
                double x = d[q];
#pragma unroll
                for (int off = JS / 2; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
                double &t = tot[(NI64 + q) * NT + grp];
                if (sub == 0) t = q < 2 ? t + x : ::fma(x, pow2(2 * ev - 61), t);
            }
        }
        __syncthreads();  // every thread is done with this stage before it is refilled
    }

    if (sub == 0 && valid) {
        auto T = [&](int q) { return tot[q * NT + grp]; };
        auto out = [&](int slot, double x) { a.out[((size_t)split * NACC + slot) * a.npad + i] = x; };
        // the pair of the star with itself: in the FP64 sums where they are formed (self at Q = 1 / eps),
        // left out of the integer sums and added here by the range that holds its tile
        const double mi = i / TJ >= t0 && i / TJ < t1 ? a.m[i + 1] : 0.0;
        double v[3] = {0.0, 0.0, 0.0}, vi2 = 0.0;
        if constexpr (MODE != MODE_NEWTON) {
#pragma unroll
            for (int k = 0; k < 3; ++k) v[k] = a.v[(size_t)(i + 1) * a.vsp + k * a.vsk];
            vi2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
        }
        if constexpr (MODE == MODE_NEWTON) {
            for (int k = 0; k < 3; ++k) out(A_GX + k, T(k));
        } else if constexpr (MODE == MODE_ENERGY) {
            out(E_PHI, ::fma(mi, a.fu.inv_eps, T(0)));
            out(E_PSI, ::fma(7.0 * vi2, mi * a.fu.inv_eps, T(1)));
        } else {
            out(A_PHI, T(11));
            out(A_S0, ::fma(mi, a.fu.inv_eps3, T(3)));
            out(A_U, T(12));
            // the velocity factors of the star itself: -|v_i|^2 G and -3/4 u_i sum ct = -sqrt(3) v_i sum ct
            const double cs = -fix::W_SCALE * T(7);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double g = T(k);
                out(A_GX + k, g);
                out(A_WX + k, ::fma(cs, v[k], T(8 + k)) + ::fma(-vi2, g, T(4 + k)));
            }
            if constexpr (MODE == MODE_FORCE_ENERGY) out(A_PSI, T(13));
        }
    }
    if constexpr (MODE != MODE_ENERGY) {
        // rows whose stars lie far inside the softening: in FP64 (above), by |n|^2 = 1 - eps^2 Q^2 or, at no cost per
        // pair, by |n|^2 >= 1 - eps Q and S0 = sum m Q^2 Q (without the star itself)
        bool lost = sub == 0 && valid;
        if constexpr (FORCE) {
            lost = lost && tot[3 * NT + grp] > (double)(near * (1.f - 1.f / NEAR)) * pow2(eg) * a.fu.inv_eps;
        } else {
            float w = near;
#pragma unroll
            for (int off = JS / 2; off > 0; off >>= 1) w += __shfl_xor_sync(0xffffffffu, w, off);
            lost = lost && w > 0.f;
        }
        if (__syncthreads_or(lost)) {
            int *flag = reinterpret_cast<int *>(buf);  // (every copy to the stages has been consumed)
            double *red = reinterpret_cast<double *>(buf + PAIR_NT);
            if (sub == 0) flag[grp] = lost;
            __syncthreads();
#pragma unroll 1
            for (int r = 0; r < NI; ++r)
                if (flag[r])
                    fix_row_fp64<MODE>(static_cast<const double2 *>(a.pack), a.npad, ibase + r, t0 * TJ, min(t1 * TJ, a.nstar),
                                       a.eps2, red, a.out + (size_t)split * NACC * a.npad + ibase + r);
        }
    }
    seq += (uint32_t)(t1 - t0 > 0 ? t1 - t0 : 0);
    return true;
}

template <int MODE, int JS>
__global__ void __launch_bounds__(PAIR_NT, 3) k_pair_fix(const PairArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    uint32_t seq = 0;
    const int ibase = blockIdx.x * (PAIR_NT / JS);
    if (__builtin_expect(*a.fix_bad != 0, 0)) {
        // The launch's shape fits the sweep below, whose CTAs are few and unequally many per SM; in FP64 the fullest SM
        // then sets the time, so the CTAs take smaller items in turn (N = 3,000 1,026 -> 892 us, 9,000 7.96 -> 7.53 ms,
        // 30,000 82.8 -> 80.6 ms; 8 lanes per star: 872 us, 7.58 and 80.5 ms, but 64 stars 42 -> 55 us).
        constexpr int BI = PAIR_NT / FIX_GENERAL_JS;
        int &cur = *reinterpret_cast<int *>(smem + 64);  // (behind the barriers)
        const int items = (a.nstar + BI - 1) / BI * a.gsplit;
        for (;;) {
            if (threadIdx.x == 0) cur = atomicAdd(a.fix_bad + 1, 1);
            __syncthreads();
            const int w = cur;
            __syncthreads();  // everyone has read cur before thread 0 fetches the next item
            if (w >= items) break;
            if (!pair_block<double, MODE, 1, FIX_GENERAL_JS>(a, w / a.gsplit * BI, w % a.gsplit, bars,
                                                             reinterpret_cast<double2 *>(smem + 128), seq)) break;
        }
        return;
    }
    double *tot = reinterpret_cast<double *>(smem + 128);
    uint4 *buf = reinterpret_cast<uint4 *>(smem + 128 + fix_tot_bytes<MODE>());
    fix_block<MODE, JS>(a, ibase, blockIdx.y, bars, tot, buf, seq);
}

}  // namespace pn
