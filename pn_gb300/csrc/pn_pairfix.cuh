// pn_pairfix.cuh -- the FP64 pair sweep on the integer pipes (the pair terms: pn_fix.cuh).
//
// The same sums, to FP64 accuracy, as k_pair<double, MODE> (pn_pair.cuh), which is bound by the
// FP64 pipe.  A CTA of 128 threads owns 128 / JS stars i; JS consecutive lanes share one i and
// split each j-tile; blockIdx.y selects one of gsplit ranges of j-tiles.  Tiles of 128 stars are
// copied to shared memory by the TMA engine, double buffered, with bounded waits.  Each tile is
// passed twice: in FP32 for the magnitude of the tile's sums (the integer sums' exponents), then
// for the sums themselves, which are added to FP64 totals in shared memory at the tile's end.
//
// Why: FP64 issues one warp instruction per 64 cycles and scheduler here and k_pair<double>'s 51 per
// pair keep that pipe busy for 3580 cycles per warp of pairs; this form takes 970, of which the
// integer multiply pipe is busy 79 % and the FP64 pipe (5 FMA, 4 conversions) 62 %.  One force
// evaluation at N = 65,536: 385 -> 104 ms, at N = 16,384: 24.0 -> 6.55 ms; its error against long
// sums is a third of the FP64 sweep's (5.6e-16 against 1.6e-15 there, c = 1).
//
// The integer range covers the systems that k_prep has checked star by star (positions within
// 2^24 eps, masses zero or 2^-32 .. 2^59 of the BH's, all finite); for any other
// the same launch runs k_pair<double>'s block instead.
#pragma once

#include "pn_fix.cuh"
#include "pn_pair.cuh"

namespace pn {

constexpr int FIX_TJ = 128;

template <int MODE> struct FixInfo {
    static constexpr int NG = MODE == MODE_NEWTON ? 5 : MODE == MODE_ENERGY ? 7 : 9;  // streamed 16-byte groups
    // tile totals: G, Phi, S0, U, W, ct, Psi as the mode has them
    static constexpr int NT = MODE == MODE_NEWTON ? 3 : MODE == MODE_ENERGY ? 2 : MODE == MODE_FORCE ? 10 : 11;
};

template <int MODE>
__host__ __device__ constexpr size_t fix_tot_bytes() {
    return (size_t)FixInfo<MODE>::NT * PAIR_NT * sizeof(double);
}
template <int MODE>
inline size_t fix_smem_bytes() {
    const size_t fast = 128 + fix_tot_bytes<MODE>() + 2 * (size_t)FixInfo<MODE>::NG * FIX_TJ * 16;
    const size_t gen = pair_smem_bytes(ModeInfo<MODE>::NG64, FIX_TJ, sizeof(double2));
    return fast > gen ? fast : gen;
}

// exponent e with x < 2^e, x >= 0 (x within FP32 range)
__device__ __forceinline__ int mag_exp(float x) {
    return (int)(__float_as_uint(x * 1.001f) >> 23) - 126;
}
__device__ __forceinline__ double pow2(int e) {  // 2^e, -1022 <= e <= 1023
    return __hiloint2double((e + 1023) << 20, 0);
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
        const uint4 u1 = pk[(size_t)10 * a.npad + il];
        I.qe = __hiloint2double((int)u1.w, (int)u1.z);
    }
    // u_i is stored in its own tile's velocity unit 2^ei, w_j in tile t's; a pair of tiles uses the larger
    const int ei = __float_as_int(a.torg[ibase / TJ].pad0);
    int ev = -100000;
    // the i position in units of 2^eL as an FP32 pair (for the seeds' differences)
    float sh[3], sl[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double s = a.spos[(size_t)k * a.npad + il] * a.fu.inv_len;
        sh[k] = (float)s;
        sl[k] = (float)(s - (double)sh[k]);
    }
    Sums A;
    A.w[0] = A.w[1] = A.w[2] = 0.0;
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
                const uint4 u0 = pk[(size_t)9 * a.npad + il], u1 = pk[(size_t)10 * a.npad + il];
                I.ux = bal(limbs((int)u0.y, (int)u0.x) >> min(e - ei, 63));
                I.uy = bal(limbs((int)u0.w, (int)u0.z) >> min(e - ei, 63));
                I.uz = bal(limbs((int)u1.y, (int)u1.x) >> min(e - ei, 63));
            }
            if (e > et) {  // (the whole CTA) bring the tile's velocities to the larger unit, in place
                uint4 *q = buf + (size_t)(stage * NG + 5) * TJ + tid;
                const uint4 g5 = q[0], g6 = q[TJ];
                const int s = min(e - et, 63);
                const B2 wx = bal(limbs((int)g5.y, (int)g5.x) >> s), wy = bal(limbs((int)g5.w, (int)g5.z) >> s),
                         wz = bal(limbs((int)g6.y, (int)g6.x) >> s);
                q[0] = make_uint4((unsigned)wx.l, (unsigned)wx.h, (unsigned)wy.l, (unsigned)wy.h);
                q[TJ] = make_uint4((unsigned)wz.l, (unsigned)wz.h, g6.z, g6.w);
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
            float mg = 0.f, mp = 0.f, ms = 0.f, mu = 0.f;
#pragma unroll 4
            for (int j = sub; j < TJ; j += JS) {
                const float4 h = reinterpret_cast<const float4 *>(b)[j], l = reinterpret_cast<const float4 *>(b)[TJ + j];
                const float y = seed(h, l);
                const float my = j == jself ? 0.f : h.w * y, my2 = my * y;
                if constexpr (MODE != MODE_ENERGY) mg += my2;
                if constexpr (MODE != MODE_NEWTON) mp += my;
                if constexpr (FORCE) {
                    ms = fmaf(my2, y, ms);
                    mu = fmaf(j == jself ? 0.f : __uint_as_float(b[4 * TJ + j].w), y, mu);
                }
            }
#pragma unroll
            for (int off = JS / 2; off > 0; off >>= 1) {
                if constexpr (MODE != MODE_ENERGY) mg += __shfl_xor_sync(0xffffffffu, mg, off);
                if constexpr (MODE != MODE_NEWTON) mp += __shfl_xor_sync(0xffffffffu, mp, off);
                if constexpr (FORCE) {
                    ms += __shfl_xor_sync(0xffffffffu, ms, off);
                    mu += __shfl_xor_sync(0xffffffffu, mu, off);
                }
            }
            E.g = mag_exp(mg);
            E.p = mag_exp(mp);
            E.s = mag_exp(ms);
            E.u = mag_exp(mu);
        }
        // ---- the sums
        clear<MODE>(A);
        constexpr int CARRY = TJ / JS < 4 ? TJ / JS : 4;
        for (int j0 = sub; j0 < TJ; j0 += CARRY * JS) {
#pragma unroll
            for (int c = 0; c < CARRY; ++c) {
                const int j = j0 + c * JS;
                const float4 h = reinterpret_cast<const float4 *>(b)[j], l = reinterpret_cast<const float4 *>(b)[TJ + j];
                const uint4 g2 = b[2 * TJ + j], g3 = b[3 * TJ + j], g4 = b[4 * TJ + j];
                StarJ J;
                J.x = {g2.x, g2.y, g2.z};
                J.y = {g2.w, g3.x, g3.y};
                J.z = {g3.z, g3.w, g4.x};
                J.m = ((u64)g4.z << 32) | g4.y;
                J.em = j == jself ? -8192 : __float_as_int(l.w);
                if constexpr (MODE != MODE_NEWTON) {
                    const uint4 g5 = b[5 * TJ + j], g6 = b[6 * TJ + j];
                    J.wx = {(int)g5.y, (int)g5.x};
                    J.wy = {(int)g5.w, (int)g5.z};
                    J.wz = {(int)g6.y, (int)g6.x};
                    J.m3 = ((u64)g6.w << 32) | g6.z;
                }
                if constexpr (FORCE) {
                    const uint4 g7 = b[7 * TJ + j], g8 = b[8 * TJ + j];
                    J.em3 = j == jself ? -8192 : (int)g7.x;
                    J.g1 = __hiloint2double((int)g7.w, (int)g7.z);
                    J.g3 = __hiloint2double((int)g8.y, (int)g8.x);
                    J.k = __hiloint2double((int)g8.w, (int)g8.z);
                }
                fix::pair<MODE>(A, I, J, E, __float_as_uint(seed(h, l)), a.fu.eps60);
            }
            carry<MODE>(A);
        }
        // ---- the JS lanes' integer sums share their exponents: added exactly; then the FP64 totals
        i64 v[FixInfo<MODE>::NT];
        int ve[FixInfo<MODE>::NT];  // exponent of the value's unit
        int nv = 0;
        auto put = [&](i64 x, int e) {
            v[nv] = x;
            ve[nv++] = e;
        };
        if constexpr (MODE != MODE_ENERGY)
#pragma unroll
            for (int k = 0; k < 3; ++k) put(top<TOP_G>(A.gh[k], A.gx[k]), E.g - S_G);
        if constexpr (MODE != MODE_NEWTON) put(A.phi, E.p - 62);
        if constexpr (FORCE) {
            put(A.s0, E.s - 61);
            put(A.u, E.u - 62);
#pragma unroll
            for (int k = 0; k < 3; ++k) put(top<TOP_W>(A.wh[k], A.wx[k]), E.g - S_W + 2 * ev);
            put(A.ct, E.g - 61 + ev);
        }
        if constexpr (PSI) put(top<TOP_P>(A.ph, A.px), E.p - S_P + 2 * ev - 2);
#pragma unroll
        for (int q = 0; q < FixInfo<MODE>::NT; ++q) {
            i64 x = v[q];
#pragma unroll
            for (int off = JS / 2; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
            if (sub == 0) tot[q * NT + grp] = ::fma(__ll2double_rn(x), pow2(ve[q]), tot[q * NT + grp]);
        }
        __syncthreads();  // every thread is done with this stage before it is refilled
    }

    if constexpr (FORCE)
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int off = JS / 2; off > 0; off >>= 1) A.w[k] += __shfl_xor_sync(0xffffffffu, A.w[k], off);
    if (sub == 0 && valid) {
        // back to the system's units
        const int e0 = fix::expo(a.m[0]), eL = a.fu.eL;
        const double fp = pow2(e0 - eL), fg = pow2(e0 - 2 * eL);
        // the pair of the star with itself belongs to the range that holds its tile
        const bool has_self = i / TJ >= t0 && i / TJ < t1;
        const double mi = has_self ? a.m[i + 1] : 0.0, Qs = a.fu.inv_eps;
        auto T = [&](int q) { return tot[q * NT + grp]; };
        auto out = [&](int slot, double x) { a.out[((size_t)split * NACC + slot) * a.npad + i] = x; };
        double v[3] = {0.0, 0.0, 0.0}, vi2 = 0.0;
        if constexpr (MODE != MODE_NEWTON) {
#pragma unroll
            for (int k = 0; k < 3; ++k) v[k] = a.v[(size_t)(i + 1) * a.vsp + k * a.vsk];
            vi2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
        }
        if constexpr (MODE == MODE_NEWTON) {
            for (int k = 0; k < 3; ++k) out(A_GX + k, fg * T(k));
        } else if constexpr (MODE == MODE_ENERGY) {
            out(E_PHI, ::fma(mi, Qs, fp * T(0)));
            out(E_PSI, ::fma(7.0 * vi2, mi * Qs, fp * T(1)));
        } else {
            const uint4 g6 = pk[(size_t)6 * a.npad + i], g7 = pk[(size_t)7 * a.npad + i];
            const u64 m3 = has_self ? ((u64)g6.w << 32) | g6.z : 0;
            const double mu3 = m3 ? scale_down(__ull2double_rn(m3), 64 - ((int)g7.x + e0 - 3 * eL)) : 0.0;
            out(A_PHI, ::fma(mi, Qs, fp * T(3)));
            out(A_S0, ::fma(mi, a.fu.inv_eps3, pow2(e0 - 3 * eL) * T(4)));
            out(A_U, ::fma(mu3, Qs, pow2(e0 - 4 * eL) * T(5)));
            // the velocity factors of the star itself: -|v_i|^2 G and -3/4 u_i sum ct = -sqrt(3) v_i sum ct
            const double cs = -fix::W_SCALE * fg * T(9);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double g = fg * T(k);
                out(A_GX + k, g);
                out(A_WX + k, ::fma(cs, v[k], fg * T(6 + k)) + ::fma(-vi2, g, A.w[k] * (1.0 / 576460752303423488.0)));
            }
            if constexpr (MODE == MODE_FORCE_ENERGY)
                out(A_PSI, ::fma(7.0 * vi2, mi * Qs, fp * T(10)));
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
    if (*a.fix_bad == 0) {
        double *tot = reinterpret_cast<double *>(smem + 128);
        uint4 *buf = reinterpret_cast<uint4 *>(smem + 128 + fix_tot_bytes<MODE>());
        fix_block<MODE, JS>(a, ibase, blockIdx.y, bars, tot, buf, seq);
    } else {
        pair_block<double, MODE, 1, JS>(a, ibase, blockIdx.y, bars, reinterpret_cast<double2 *>(smem + 128), seq);
    }
}

}  // namespace pn
