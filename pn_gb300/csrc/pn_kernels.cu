// pn_kernels.cu -- the O(N) kernels of libpn's force path (FP64 throughout).
//
//   k_prep          per-star quantities, the j-particle pack, the global sums
//   k_finish        per-star accelerations (Limit-sticky9.c:36-51 BH column, :213-274,
//                   the closed-form parts of :276-422), the BH's acceleration (:36-51 BH row,
//                   :54-211), and optionally one stage of the integration step (:853-891)
//   k_energy_finish the energies (:445-556) from the energy pair sweep
//
// Reductions over particles are two-level and deterministic: each CTA writes its partial,
// and the last CTA to finish (atomic ticket) sums all partials in block order and resets
// the ticket, so results do not depend on scheduling.
#include <cstdio>

#include "pn_fix.cuh"
#include "pn_kernels.h"

namespace pn {

// ------------------------------------------------------------------ small helpers
__device__ __forceinline__ double ld_x(const double *p, long long sp, long long sk, int i, int k) {
    return p[(long long)i * sp + (long long)k * sk];
}

// Double-double accumulation (TwoSum, Knuth TAOCP vol. 2 4.2.2) for the compensated sums.
struct DD {
    double hi, lo;
};
__device__ __forceinline__ DD dd_add(DD a, DD b) {
    double s = a.hi + b.hi;
    double bb = s - a.hi;
    double e = (a.hi - (s - bb)) + (b.hi - bb);
    e += a.lo + b.lo;
    double t = s + e;
    return DD{t, e - (t - s)};
}

// Sums over the block, NQ (8 or 4) values per thread, in a fixed order.  Within a warp the lanes
// first trade halves of the values (each keeps and adds one half), so that NQ values take NQ - 1
// additions down to one value per lane and log2(32 / NQ) more across the remaining lanes: 9 FP64
// additions for 8 values instead of 40, which matters at one FP64 warp instruction per 64 cycles.
// Then thread q < NQ adds the warps' sums in order; the result is thread q's.  Every thread calls;
// scratch holds (blockDim.x / 32) * NQ values and is free again on return.
template <int NQ, typename T, typename Add, typename Shfl>
__device__ __forceinline__ T block_sum(T (&v)[NQ], T *scratch, Add add, Shfl shfl) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int off = 16;
#pragma unroll
    for (int h = NQ / 2; h >= 1; h >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int q = 0; q < h; ++q) {
            const T give = up ? v[q] : v[q + h], keep = up ? v[q + h] : v[q];
            v[q] = add(keep, shfl(give, off));
        }
    }
    constexpr int PER = 32 / NQ;  // lanes that hold partial sums of the same value
#pragma unroll
    for (int o = PER / 2; o >= 1; o >>= 1) v[0] = add(v[0], shfl(v[0], o));
    if (lane % PER == 0) scratch[warp * NQ + lane / PER] = v[0];
    __syncthreads();
    T r = scratch[threadIdx.x % NQ];
    if (threadIdx.x < NQ)
        for (int w = 1; w < nw; ++w) r = add(r, scratch[w * NQ + threadIdx.x]);
    __syncthreads();
    return r;
}
template <int NQ>
__device__ __forceinline__ double block_sum(double (&v)[NQ], double *scratch) {
    return block_sum<NQ, double>(
        v, scratch, [](double a, double b) { return a + b; },
        [](double a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); });
}
template <int NQ>
__device__ __forceinline__ DD block_sum(DD (&v)[NQ], DD *scratch) {
    return block_sum<NQ, DD>(v, scratch, dd_add, [](DD a, int o) {
        return DD{__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)};
    });
}
// The same over nblk block partials part[b * NQ + q] (thread t adds the blocks t / NQ, t / NQ +
// blockDim.x / NQ, ... of value t % NQ, then the threads of a value are added in order): the
// result is thread q's, q < NQ.  scratch holds blockDim.x values.
template <int NQ, typename T, typename Add, typename Load>
__device__ __forceinline__ T partials_sum(int nblk, T zero, T *scratch, Add add, Load load) {
    const int q = threadIdx.x % NQ, first = threadIdx.x / NQ, step = blockDim.x / NQ;
    T t = zero;
    for (int b = first; b < nblk; b += step) t = add(t, load(b, q));
    scratch[threadIdx.x] = t;
    __syncthreads();
    const int have = min(step, nblk);
    if (threadIdx.x < NQ)
        for (int k = 1; k < have; ++k) t = add(t, scratch[k * NQ + threadIdx.x]);
    return t;
}

// Last-CTA election after each CTA published its partial.
__device__ __forceinline__ bool last_block(unsigned *ticket, int nblk) {
    __shared__ bool am_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = atomicAdd(ticket, 1u);
        am_last = (t == (unsigned)nblk - 1u);
    }
    __syncthreads();
    return am_last;
}

// ------------------------------------------------------------------ prep
// The fixed-point sweep's pack of star j (pn_pairfix.cuh): s, its tile's origin o and velocity unit
// 2^ev, v, m, mu3 and the FP64 coefficients of the W sum.  A padding star has no mass and sits at its tile's origin.
__device__ __forceinline__ void prep_fix(const PrepArgs &a, int j, bool real, const double *s, const double *o,
                                         const double *v, double v2, int ev, double m, double mu3, double c1,
                                         double c3, double k35, double qe, double m0) {
    using namespace fix;
    const FixUnits &u = a.fu;
    const int e0 = expo(m0);
    const bool in = in_range(s, v2, m, m0, u.eL, u.ev_max);
    if (real && !in) atomicOr(a.fix_bad, 1);
    if (!in) return;
    float hi[3], lo[3];
    X96 x[3];
    B2 w[3], q[3];
    const float down = __int_as_float((127 - u.eL) << 23);
    const int eu = speed_exp(v2);  // the star's own velocity unit
    for (int k = 0; k < 3; ++k) {
        to_f32_pair(real ? s[k] - o[k] : 0.0, hi[k], lo[k]);
        hi[k] *= down;
        lo[k] *= down;
        x[k] = to_x96(real ? s[k] : o[k], u.eL);
        w[k] = bal(to_scaled(v[k], W_MANT, 63, 60, ev));
        q[k] = bal(to_scaled(v[k], U_MANT, 62, 62, eu));
    }
    int em;
    const u64 mm = mantissa(m, em);
    em = mm ? em - e0 : -8192;
    const double g1 = m * fma(-2.0, v2, c1), g3 = m * c3, kk = fma(m, c3, k35);
    // FP32 magnitudes in the sweep's units, for the exponents of a tile's sums
    const float mf = to_f32(scale2(m, -e0)), g1f = fabsf(to_f32(scale2(g1, u.eL - 2 * e0))),
                g3f = to_f32(scale2(g3, 3 * u.eL - 2 * e0)), kf = to_f32(scale2(kk, 3 * u.eL - 2 * e0));
    uint4 *p = a.fpack + j;
    const size_t n = a.npad;
    auto fu = [](float f) { return __float_as_uint(f); };
    auto lw = [](double d) { return (unsigned)__double2loint(d); };
    auto hw = [](double d) { return (unsigned)__double2hiint(d); };
    const float down34 = 5.8207660913467407e-11f;  // 2^-34
    p[0] = make_uint4(fu(hi[0]), fu(hi[1]), fu(hi[2]), fu(mf));
    p[n] = make_uint4(fu(lo[0]), fu(lo[1]), fu(lo[2]), (unsigned)em);
    p[2 * n] = make_uint4(x[0].w0, x[0].w1, x[0].w2, x[1].w0);
    p[3 * n] = make_uint4(x[1].w1, x[1].w2, x[2].w0, x[2].w1);
    p[4 * n] = make_uint4(x[2].w2, (unsigned)(mm >> 32), fu((float)(unsigned)(mm >> 32) * down34), fu((float)(unsigned)mm * down34));
    auto un = [](int i) { return (unsigned)i; };
    p[5 * n] = make_uint4(un(w[0].h), un(w[0].l), un(w[1].h), un(w[1].l));
    p[6 * n] = make_uint4(un(w[2].h), un(w[2].l), 0u, 0u);
    p[7 * n] = make_uint4(0u, fu(g1f), fu(g3f), fu(kf));
    p[8 * n] = make_uint4(lw(m), hw(m), lw(mu3), hw(mu3));
    p[9 * n] = make_uint4(lw(g1), hw(g1), lw(g3), hw(g3));
    // (|w| in the tile's unit, rounded up)
    p[10 * n] = make_uint4(lw(kk), hw(kk), fu(sqrtf(to_f32(scale2(3.0 * v2, -2 * ev))) * 1.00001f), (unsigned)eu);
    p[11 * n] = make_uint4(un(q[0].h), un(q[0].l), un(q[1].h), un(q[1].l));
    p[12 * n] = make_uint4(un(q[2].h), un(q[2].l), lw(qe), hw(qe));
}

// Per star j (particle p = j + 1): s = x_p - x_0, q = |s|^2, R = (q + eps^2)^(-1/2) (the
// reference's rsqrt, Limit-sticky9.c:15-19), and the pack entries; global sums
// A1 = sum m R, B3 = sum m R^3 s, C = sum m R^3 q, P = sum m v.
//
// Bound by the latency of its FP64 instructions (64 cycles each per warp and scheduler, so a block
// is four warps, one per scheduler): conversions and scalings by powers of two are integer
// operations, the square root and its inverse one rsqrt, the block's sums 9 additions per warp.
__device__ __forceinline__ void prep_body(const PrepArgs &a, int blk, int nblk) {
    __shared__ double red[ON_NT];
    const int j = blk * ON_NT + threadIdx.x;
    const double x0 = ld_x(a.x, a.sp, a.sk, 0, 0), y0 = ld_x(a.x, a.sp, a.sk, 0, 1),
                 z0 = ld_x(a.x, a.sp, a.sk, 0, 2);
    const double m0 = a.m[0];
    const bool real = j < a.nstar;
    double s[3] = {0, 0, 0}, vv[3] = {0, 0, 0}, o[3] = {0, 0, 0}, mj = 0, R = 0, q = 0, qe = 0;
    if (real) {
        const int p = j + 1;
        s[0] = ld_x(a.x, a.sp, a.sk, p, 0) - x0;
        s[1] = ld_x(a.x, a.sp, a.sk, p, 1) - y0;
        s[2] = ld_x(a.x, a.sp, a.sk, p, 2) - z0;
        vv[0] = ld_x(a.v, a.sp, a.sk, p, 0);
        vv[1] = ld_x(a.v, a.sp, a.sk, p, 1);
        vv[2] = ld_x(a.v, a.sp, a.sk, p, 2);
        mj = a.m[p];
        q = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
        qe = q + a.eps2;
        R = rsqrt(qe);
    }
    const double R3 = R * R * R;
    const double mu3 = mj * R3;
    const double c1 = (1.25 * m0) * R, c3 = (0.25 * m0) * R3, k35 = (3.5 * m0) * mu3;
    const double v2 = vv[0] * vv[0] + vv[1] * vv[1] + vv[2] * vv[2];
    // the tile origin (the tile's first star)
    const int jt = (j / a.tj) * a.tj;
    if ((a.f32 || a.fpack) && jt < a.nstar) {
        o[0] = ld_x(a.x, a.sp, a.sk, jt + 1, 0) - x0;
        o[1] = ld_x(a.x, a.sp, a.sk, jt + 1, 1) - y0;
        o[2] = ld_x(a.x, a.sp, a.sk, jt + 1, 2) - z0;
    }
    a.spos[j] = s[0];
    a.spos[a.npad + j] = s[1];
    a.spos[2 * a.npad + j] = s[2];
    if (a.f32) {
        // position relative to the tile origin as an FP32 hi/lo pair
        float hi[3], lo[3], v[3];
        for (int k = 0; k < 3; ++k) {
            to_f32_pair(real ? s[k] - o[k] : 0.0, hi[k], lo[k]);
            v[k] = to_f32(vv[k]);
        }
        const float qf = to_f32(qe), c3f = to_f32(c3);
        if (a.pack) {  // the scalar sweep's pack (not needed when only the packed sweep runs)
            float4 *pk = static_cast<float4 *>(a.pack);
            pk[j] = make_float4(hi[0], hi[1], hi[2], to_f32(mj));
            pk[a.npad + j] = make_float4(lo[0], lo[1], lo[2], to_f32(mu3));
            pk[2 * a.npad + j] = make_float4(v[0], v[1], v[2], qf);
            pk[3 * a.npad + j] = make_float4(to_f32(c1), c3f, to_f32(k35), 0.f);
        }
        if (a.spack) {  // scaled as the paired pack
            constexpr double K = X2_K, IK = 1.0 / K, IK3 = 1.0 / (K * K * K);
            float4 *p = a.spack + j;
            const size_t n = a.npad;
            p[0] = make_float4(hi[0], hi[1], hi[2], to_f32(mj * IK3));
            p[n] = make_float4(lo[0], lo[1], lo[2], to_f32(mu3 * IK));
            p[2 * n] = make_float4(to_f32(X2_SQRT3 * vv[0]), to_f32(X2_SQRT3 * vv[1]), to_f32(X2_SQRT3 * vv[2]),
                                   to_f32(fma(-2.0, v2, c1)));
            p[3 * n] = make_float4(c3f, to_f32(k35 * IK), qf, 0.f);
        }
        if (a.pack2) {  // paired layout: star j is lane (j & 1) of pair j / 2; scaled
            const int lane = j & 1;
            const size_t prow = (size_t)a.npad / 2;
            float *p2 = reinterpret_cast<float *>(a.pack2 + j / 2);
            constexpr double K = X2_K, IK = 1.0 / K, IK3 = 1.0 / (K * K * K);
            const float vals[7][2] = {{hi[0], hi[1]},
                                      {hi[2], to_f32(mj * IK3)},
                                      {lo[0], lo[1]},
                                      {lo[2], to_f32(mu3 * IK)},
                                      {to_f32(X2_SQRT3 * vv[0]), to_f32(X2_SQRT3 * vv[1])},
                                      {to_f32(X2_SQRT3 * vv[2]), to_f32(fma(-2.0, v2, c1))},
                                      {c3f, to_f32(k35 * IK)}};
            for (int g = 0; g < 7; ++g) {
                p2[g * prow * 4 + lane] = vals[g][0];
                p2[g * prow * 4 + 2 + lane] = vals[g][1];
            }
            a.ipack[j] = make_float4(v[0], v[1], v[2], qf);
        }
        if (j % a.tj == 0 && real) {
            TileOrigin t{s[0], s[1], s[2], 0.0};
            to_f32_pair(s[0], t.hx, t.lx);
            to_f32_pair(s[1], t.hy, t.ly);
            to_f32_pair(s[2], t.hz, t.lz);
            t.pad0 = t.pad1 = 0.f;
            a.torg[j / a.tj] = t;
        }
    } else {
        double2 *pk = static_cast<double2 *>(a.pack);
        pk[j] = make_double2(s[0], s[1]);
        pk[a.npad + j] = make_double2(s[2], mj);
        pk[2 * a.npad + j] = make_double2(vv[0], vv[1]);
        pk[3 * a.npad + j] = make_double2(vv[2], mu3);
        pk[4 * a.npad + j] = make_double2(c1, c3);
        pk[5 * a.npad + j] = make_double2(k35, qe);
        if (a.fpack) {
            if (j == 0) a.fix_bad[1] = 0;
            // the tile's velocity unit (a block is one tile of 128)
            static_assert(ON_NT == 128, "one tile per block");
            __shared__ int wev[4];
            const int we = __reduce_max_sync(0xffffffffu, fix::speed_exp(v2));
            if ((threadIdx.x & 31) == 0) wev[threadIdx.x >> 5] = we;
            __syncthreads();
            const int ev = max(max(wev[0], wev[1]), max(wev[2], wev[3]));
            prep_fix(a, j, real, s, o, vv, v2, ev, mj, mu3, c1, c3, k35, qe, m0);
            if (j % a.tj == 0 && real) {  // in units of 2^eL
                TileOrigin t{};
                const float down = __int_as_float((127 - a.fu.eL) << 23);
                to_f32_pair(s[0], t.hx, t.lx);
                to_f32_pair(s[1], t.hy, t.ly);
                to_f32_pair(s[2], t.hz, t.lz);
                t.hx *= down; t.hy *= down; t.hz *= down;
                t.lx *= down; t.ly *= down; t.lz *= down;
                t.pad0 = __int_as_float(ev);
                a.torg[j / a.tj] = t;
            }
        }
    }
    // (mj = mu3 = 0 and finite s, q, v for a slot without a star)
    double g[8] = {mj * R, mu3 * s[0], mu3 * s[1], mu3 * s[2], mu3 * q, mj * vv[0], mj * vv[1], mj * vv[2]};
    static_assert(NGLOB == 8 && G_A1 == 0 && G_B3X == 1 && G_C == 4 && G_PX == 5, "order of g");
    const double r = block_sum<8>(g, red);
    if (threadIdx.x < 8) a.part[(size_t)blk * 8 + threadIdx.x] = r;
    if (last_block(a.ticket, nblk)) {
        const double t = partials_sum<8>(nblk, 0.0, red, [](double u, double w) { return u + w; },
                                         [&](int b, int k) { return __ldcg(&a.part[(size_t)b * 8 + k]); });
        if (threadIdx.x < 8) a.glob[threadIdx.x] = t;
        if (threadIdx.x == 0) *a.ticket = 0u;
    }
}

// ------------------------------------------------------------------ finish
// Stage updates of the integration step (Limit-sticky9.c:853-891) without FMA contraction,
// so the state arithmetic is rounded exactly as the reference's.
// a / 6, correctly rounded, in three operations: with c = RN(1/6), q = RN(a c) and the exact
// remainder r = a - 6 q, RN(q + r c) is the rounded quotient (Markstein, IBM J. Res. Dev. 34, 1990);
// outside the range where that holds, the division itself.
__device__ __forceinline__ double sixth(double a) {
    const int be = (__double2hiint(a) >> 20) & 0x7ff;
    if (be < 128 || be > 2040) return __ddiv_rn(a, 6.0);
    constexpr double c = 1.0 / 6.0;
    const double q = __dmul_rn(a, c);
    return __fma_rn(__fma_rn(-6.0, q, a), c, q);
}

// What a stage reads of particle p's component k, loaded ahead of the arithmetic (the stores of one
// component would hold back the loads of the next).
struct StageIn {
    double x, v, vs, hx, hv;
};
__device__ __forceinline__ StageIn stage_load(const FinishArgs &a, int p, int k) {
    const size_t o = (size_t)k * a.ld + p;
    StageIn r{a.st.x[o], a.st.v[o], 0.0, 0.0, 0.0};
    if (a.stage != 1 && a.stage != STAGE_RK4_1) {
        r.vs = a.st.vs[o];
        r.hx = a.st.hx[o];
        r.hv = a.st.hv[o];
    }
    return r;
}
__device__ __forceinline__ void stage_update_k(const FinishArgs &a, int p, int k, double acc, const StageIn &in) {
    const double dt = a.dt;
    const size_t o = (size_t)k * a.ld + p;
    const double x = in.x, v = in.v, vprev = in.vs;
    if (a.stage >= STAGE_RK4_1) {
        // classic fourth-order Runge-Kutta (optional integrator; hx, hv accumulate
        // k1 + 2 k2 + 2 k3 of the position and velocity slopes)
        if (a.stage == STAGE_RK4_1) {
            a.st.xs[o] = x + 0.5 * dt * v;
            a.st.vs[o] = v + 0.5 * dt * acc;
            a.st.hx[o] = v;
            a.st.hv[o] = acc;
        } else if (a.stage == STAGE_RK4_4) {
            a.st.x[o] = x + (dt / 6.0) * (in.hx + vprev);
            a.st.v[o] = v + (dt / 6.0) * (in.hv + acc);
        } else {
            const double f = a.stage == STAGE_RK4_2 ? 0.5 * dt : dt;
            a.st.xs[o] = x + f * vprev;
            a.st.vs[o] = v + f * acc;
            a.st.hx[o] = in.hx + 2.0 * vprev;
            a.st.hv[o] = in.hv + 2.0 * acc;
        }
    } else if (a.stage == 1) {  // :853-860
        const double x1 = __dadd_rn(x, __dmul_rn(__dmul_rn(0.5, v), dt));
        const double v1 = __dadd_rn(v, __dmul_rn(__dmul_rn(0.5, acc), dt));
        a.st.xs[o] = x1;
        a.st.vs[o] = v1;
        a.st.hx[o] = x1;
        a.st.hv[o] = v1;
    } else if (a.stage == 2) {  // :864-871
        const double x1 = __dadd_rn(x, __dmul_rn(__dmul_rn(0.5, vprev), dt));
        const double v1 = __dadd_rn(v, __dmul_rn(__dmul_rn(0.5, acc), dt));
        a.st.xs[o] = x1;
        a.st.vs[o] = v1;
        a.st.hx[o] = __dadd_rn(in.hx, x1);
        a.st.hv[o] = __dadd_rn(in.hv, v1);
    } else {  // :875-891
        const double x3 = __dadd_rn(x, __dmul_rn(vprev, dt));
        const double v3 = __dadd_rn(v, __dmul_rn(acc, dt));
        a.st.x[o] = sixth(__dadd_rn(__dadd_rn(x, x3), __dmul_rn(2.0, in.hx)));
        a.st.v[o] = sixth(__dadd_rn(__dadd_rn(v, v3), __dmul_rn(2.0, in.hv)));
    }
}

// Star i's first NK pair sums over the j-range splits, in order, the loads of several splits in flight
// at once (one split after the other, they were half of the kernel's time with 8 splits: N = 1,000 mixed
// 25.6 -> 19.8 us with a cold cache).
template <int NK>
__device__ __forceinline__ void split_sums(const FinishArgs &a, int i, double (&S)[NACC_MAX]) {
#pragma unroll
    for (int k = NK; k < NACC_MAX; ++k) S[k] = 0.0;
    if (a.accf) {  // FP32 pairs, added in FP32 without loss of their low parts
        constexpr int U = 4;
        const float2 *p = reinterpret_cast<const float2 *>(a.acc) + i;
        float h[NK], l[NK];
#pragma unroll
        for (int k = 0; k < NK; ++k) h[k] = l[k] = 0.f;
        for (int g = 0; g < a.gsplit; g += U) {
            float2 t[U][NK];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int k = 0; k < NK; ++k)
                    t[u][k] = g + u < a.gsplit ? p[((size_t)(g + u) * a.nacc + k) * a.npad] : make_float2(0.f, 0.f);
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int k = 0; k < NK; ++k) pair_add(h[k], l[k], t[u][k]);
        }
#pragma unroll
        for (int k = 0; k < NK; ++k) S[k] = to_f64(h[k]) + to_f64(l[k]);
        S[A_PHI] *= X2_K * X2_K;  // the packed sweep's scale
    } else {
        constexpr int U = 3;
        const double *p = a.acc + i;
#pragma unroll
        for (int k = 0; k < NK; ++k) S[k] = p[(size_t)k * a.npad];
        for (int g = 1; g < a.gsplit; g += U) {
            double t[U][NK];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int k = 0; k < NK; ++k) t[u][k] = g + u < a.gsplit ? p[((size_t)(g + u) * a.nacc + k) * a.npad] : 0.0;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (g + u < a.gsplit)
#pragma unroll
                    for (int k = 0; k < NK; ++k) S[k] += t[u][k];
        }
    }
}

// Bound by its FP64 instructions (about 150 per star, 64 cycles each per warp and scheduler): one
// warp per scheduler and block, no division per star but the reference's own q, common factors
// R^3 and m R^3 taken out of the sums.  Whatever it reads is loaded first: the latency of a load is
// that of ten of them.
__device__ __forceinline__ void finish_body(const FinishArgs &a, int blk, int nblk) {
    __shared__ double red[ON_NT];
    const int i = blk * ON_NT + threadIdx.x;
    const double m0 = a.m[0];
    const double eps2 = a.eps2, ic2 = a.inv_c2;
    const double *G = a.glob;
    double bh[4] = {0.0, 0.0, 0.0, 0.0};
    bool bad = false;

    if (i < a.nstar) {
        const int p = i + 1;
        const double s[3] = {a.spos[i], a.spos[a.npad + i], a.spos[2 * a.npad + i]};
        const double mi = a.m[p];
        double v[3] = {0.0, 0.0, 0.0}, glob[NGLOB] = {0.0};
        StageIn in[3] = {};
        if (a.pn1) {
#pragma unroll
            for (int k = 0; k < 3; ++k) v[k] = ld_x(a.v, a.vsp, a.vsk, p, k);
#pragma unroll
            for (int k = 0; k < NGLOB; ++k) glob[k] = G[k];
        }
        if (a.stage)
#pragma unroll
            for (int k = 0; k < 3; ++k) in[k] = stage_load(a, p, k);
        const double q = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
        const double R = rsqrt(q + eps2);
        const double R3 = R * R * R;
        // the force slots only (a fused-energy sweep has one more, read by the energy kernel)
        const int nk = a.nacc < NACC_MAX ? a.nacc : NACC_MAX;
        double S[NACC_MAX];
        if (nk == NACC_MAX) split_sums<NACC_MAX>(a, i, S);
        else split_sums<3>(a, i, S);
        if (a.sums_out)
#pragma unroll
            for (int k = 0; k < NACC_MAX; ++k)
                if (k < nk) a.sums_out[(size_t)k * a.npad + i] = S[k];
        const double Gv[3] = {S[A_GX], S[A_GY], S[A_GZ]};
        double acc3[3];
        const double mb = m0 * R3;
        for (int k = 0; k < 3; ++k) acc3[k] = fma(-mb, s[k], Gv[k]);  // Newton incl. BH column
        if (a.pn1) {
            const double P[3] = {glob[G_PX], glob[G_PY], glob[G_PZ]};
            const double B3[3] = {glob[G_B3X], glob[G_B3Y], glob[G_B3Z]};
            const double A1 = glob[G_A1], C = glob[G_C];
            const double Phi = S[A_PHI], S0 = S[A_S0], U = S[A_U];
            const double W[3] = {S[A_WX], S[A_WY], S[A_WZ]};
            const double vi2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
            const double vis = v[0] * s[0] + v[1] * s[1] + v[2] * s[2];
            const double viP = v[0] * P[0] + v[1] * P[1] + v[2] * P[2];
            const double Ps = P[0] * s[0] + P[1] * s[1] + P[2] * s[2];
            const double sB3 = s[0] * B3[0] + s[1] * B3[1] + s[2] * B3[2];
            const double sG = s[0] * Gv[0] + s[1] * Gv[1] + s[2] * Gv[2];
            const double m0R = m0 * R;
            // star i: :215-238 (a_BH), :249-274 (ac direct), :276-382 summed over j (t1..t4, W),
            // minus the self-pair removal :392-422.  The s part, over R^3 but for the U term:
            //   m0 [ -(4 m0 R - v^2) - (4 Phi + 1.25 A1 - 0.25 C + 0.5 s.B3)
            //        + m_i (9.75 R + 0.5 / eps + 0.25 q R^3) ] - 8 m_i v^2 + 4 v.P
            const double aa = 4.0 * Phi + 1.25 * A1 + fma(0.5, sB3, -0.25 * C);
            const double bm = fma(9.75, R, fma(0.25 * q, R3, 0.5 * a.inv_eps));
            const double br = fma(mi, bm, vi2 - fma(4.0, m0R, aa));
            const double cs = fma(R3, fma(m0, br, fma(-8.0 * mi, vi2, 4.0 * viP)), (3.5 * m0) * U);
            const double cv = R3 * fma(vis, fma(14.0, mi, -4.0 * m0), -3.0 * Ps);
            const double cg = 4.0 * m0R, cb = -3.5 * m0R, cp = -4.0 * R3 * vis;
            for (int k = 0; k < 3; ++k) {
                const double pn = fma(cs, s[k], fma(cv, v[k], fma(cg, Gv[k], fma(cb, B3[k], fma(cp, P[k], W[k])))));
                acc3[k] = fma(ic2, pn, acc3[k]);
            }
            // this star's share of the BH's 1PN acceleration: :58-95 (a1), :101-115 (single),
            // :118-174 summed over j, minus :179-207 (removal, with its 1.25*eps)
            const double im0 = 1.0 / m0;
            const double T = fma(eps2, S0, -Phi) - 2.0 * sG;
            const double mR3 = mi * R3;
            const double bs = fma(5.0, m0R, fma(-2.0, vi2, 1.5 * (vis * vis / q)))          // a1
                              + fma(4.0, A1, fma(1.25, Phi, 0.25 * T))                      // pair
                              + mi * fma(8.0, R, 1.25 * a.eps)                              // single, -removal
                              - (4.0 * im0) * fma(mi, vi2, viP);
            const double bv = fma(vis, fma(7.0 * mi, im0, 3.0), (4.0 * im0) * Ps);
            const double bg = -3.5 * R * mi, bp = 3.0 * im0 * vis;
            for (int k = 0; k < 3; ++k) bh[k] = fma(mR3, fma(bs, s[k], fma(bv, v[k], bp * P[k])), bg * Gv[k]);
        }
        for (int k = 0; k < 3; ++k) {
            if (!isfinite(acc3[k])) bad = true;
            if (a.a) a.a[(long long)p * a.asp + (long long)k * a.ask] = acc3[k];
        }
        if (a.stage)
#pragma unroll
            for (int k = 0; k < 3; ++k) stage_update_k(a, p, k, acc3[k], in[k]);
    }
    if (bad) atomicOr(a.err, DEVERR_NONFINITE);
    const double r = block_sum<4>(bh, red);
    if (threadIdx.x < 4) a.part[(size_t)blk * 4 + threadIdx.x] = r;
    if (last_block(a.ticket, nblk)) {
        const int k = threadIdx.x;
        StageIn in{};
        if (a.stage && k < 3) in = stage_load(a, 0, k);
        const double t = partials_sum<4>(nblk, 0.0, red, [](double u, double w) { return u + w; },
                                         [&](int b, int k) { return __ldcg(&a.part[(size_t)b * 4 + k]); });
        // BH: Newtonian pull of the stars (:36-51, row 0) plus the 1PN sum; thread k < 3 holds component k
        if (k < 3) {
            const double acc = a.pn1 ? fma(ic2, t, G[G_B3X + k]) : G[G_B3X + k];
            if (!isfinite(acc)) atomicOr(a.err, DEVERR_NONFINITE);
            if (a.a) a.a[(long long)k * a.ask] = acc;
            if (a.stage) stage_update_k(a, 0, k, acc, in);
        }
        if (k == 0) {
            if (a.fix_bad) *a.fix_bad = 0;
            *a.ticket = 0u;
        }
    }
}

// ------------------------------------------------------------------ energy
// Per star (Limit-sticky9.c:452-556): kinetic, Newtonian potential row, O(N) 1PN term and the
// pairwise 1PN energy with its self-pair removal; compensated (double-double) sums.
__device__ __forceinline__ void energy_body(const EnergyArgs &a, int blk, int nblk) {
    __shared__ DD red[ON_NT];
    const int i = blk * ON_NT + threadIdx.x;
    const double m0 = a.m[0], eps2 = a.eps2, ie = a.inv_eps;
    const double v0[3] = {ld_x(a.v, a.sp, a.sk, 0, 0), ld_x(a.v, a.sp, a.sk, 0, 1),
                          ld_x(a.v, a.sp, a.sk, 0, 2)};
    const double A1 = a.glob[G_A1];
    DD e[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};  // kin, pot, pot_pn, pn2
    if (i < a.nstar) {
        const int p = i + 1;
        const double s[3] = {a.spos[i], a.spos[a.npad + i], a.spos[2 * a.npad + i]};
        const double v[3] = {ld_x(a.v, a.sp, a.sk, p, 0), ld_x(a.v, a.sp, a.sk, p, 1),
                             ld_x(a.v, a.sp, a.sk, p, 2)};
        const double mi = a.m[p];
        double Phi = 0.0, Psi = 0.0;
        if (a.accf) {
            const float2 *p = reinterpret_cast<const float2 *>(a.acc) + i;
            float h[2] = {0.f, 0.f}, l[2] = {0.f, 0.f};
            for (int g = 0; g < a.gsplit; ++g) {
                pair_add(h[0], l[0], p[((size_t)g * a.nacc + a.sphi) * a.npad]);
                pair_add(h[1], l[1], p[((size_t)g * a.nacc + a.spsi) * a.npad]);
            }
            Phi = (to_f64(h[0]) + to_f64(l[0])) * (X2_K * X2_K);
            Psi = to_f64(h[1]) + to_f64(l[1]);
        } else {
            for (int g = 0; g < a.gsplit; ++g) {
                Phi += a.acc[((size_t)g * a.nacc + a.sphi) * a.npad + i];
                Psi += a.acc[((size_t)g * a.nacc + a.spsi) * a.npad + i];
            }
        }
        const double q = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
        const double R = rsqrt(q + eps2);
        const double vi2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
        const double v0vi = v0[0] * v[0] + v0[1] * v[1] + v0[2] * v[2];
        const double sv0 = s[0] * v0[0] + s[1] * v0[1] + s[2] * v0[2];
        const double svi = s[0] * v[0] + s[1] * v[1] + s[2] * v[2];
        const double mR = m0 * R;
        e[0].hi = mi * vi2;
        e[1].hi = (-(mR + Phi) + mi * ie) * mi;
        e[2].hi = 0.375 * mi * vi2 * vi2 + 1.5 * mR * mi * vi2 + 0.5 * mR * mR * mi
                  + 0.5 * mR * mi * (3.0 * vi2 - 7.0 * v0vi - sv0 * svi * R * R);
        e[3].hi = 0.25 * mi * (6.0 * vi2 * Phi - Psi) + m0 * mi * R * Phi + 0.5 * m0 * mi * R * A1
                  - mi * mi * (-0.25 * ie * vi2 + m0 * R * (ie + 0.5 * R));
    }
    const DD r = block_sum<4>(e, red);
    if (threadIdx.x < 4) {
        a.part[((size_t)blk * 4 + threadIdx.x) * 2] = r.hi;
        a.part[((size_t)blk * 4 + threadIdx.x) * 2 + 1] = r.lo;
    }
    if (last_block(a.ticket, nblk)) {
        DD t = partials_sum<4>(nblk, DD{0.0, 0.0}, red, dd_add, [&](int b, int q) {
            return DD{__ldcg(&a.part[((size_t)b * 4 + q) * 2]), __ldcg(&a.part[((size_t)b * 4 + q) * 2 + 1])};
        });
        __shared__ double tot[4];
        if (threadIdx.x < 4) tot[threadIdx.x] = t.hi + t.lo;
        __syncthreads();
        if (threadIdx.x == 0) {
            const double kin0 = m0 * (v0[0] * v0[0] + v0[1] * v0[1] + v0[2] * v0[2]);
            const double kin = 0.5 * (tot[0] + kin0);
            const double pot = 0.5 * (tot[1] - m0 * A1);
            const double potpn = a.inv_c2 * tot[2];
            const double pn2 = a.inv_c2 * tot[3];
            a.out[0] = pot;
            a.out[1] = kin;
            a.out[2] = potpn;
            a.out[3] = kin + pot + potpn + pn2;
            if (a.fix_bad) *a.fix_bad = 0;
            *a.ticket = 0u;
        }
    }
}

// ------------------------------------------------------------------ kernels
// One system: the block index is the block within the system.
__global__ void __launch_bounds__(ON_NT) k_prep(const PrepArgs a) { prep_body(a, blockIdx.x, gridDim.x); }
__global__ void __launch_bounds__(ON_NT) k_finish(const FinishArgs a) { finish_body(a, blockIdx.x, gridDim.x); }
__global__ void __launch_bounds__(ON_NT) k_energy_finish(const EnergyArgs a) {
    energy_body(a, blockIdx.x, gridDim.x);
}

// An ensemble in one launch: blockmap[b] = (cluster, block within the cluster, blocks of the
// cluster); each cluster's arguments come from a device table.
__global__ void __launch_bounds__(ON_NT) k_prep_ens(const PrepArgs *tab, const int4 *blockmap) {
    const int4 bm = blockmap[blockIdx.x];
    const PrepArgs a = tab[bm.x];
    prep_body(a, bm.y, bm.z);
}
__global__ void __launch_bounds__(ON_NT) k_finish_ens(const FinishArgs *tab, const int4 *blockmap) {
    const int4 bm = blockmap[blockIdx.x];
    const FinishArgs a = tab[bm.x];
    finish_body(a, bm.y, bm.z);
}
__global__ void __launch_bounds__(ON_NT) k_energy_ens(const EnergyArgs *tab, const int4 *blockmap) {
    const int4 bm = blockmap[blockIdx.x];
    const EnergyArgs a = tab[bm.x];
    energy_body(a, bm.y, bm.z);
}

// ------------------------------------------------------------------ launchers
cudaError_t launch_prep_ens(const PrepArgs *tab, const int4 *blockmap, int nblocks, cudaStream_t s) {
    k_prep_ens<<<nblocks, ON_NT, 0, s>>>(tab, blockmap);
    return cudaGetLastError();
}
cudaError_t launch_finish_ens(const FinishArgs *tab, const int4 *blockmap, int nblocks, cudaStream_t s) {
    k_finish_ens<<<nblocks, ON_NT, 0, s>>>(tab, blockmap);
    return cudaGetLastError();
}
cudaError_t launch_energy_ens(const EnergyArgs *tab, const int4 *blockmap, int nblocks, cudaStream_t s) {
    k_energy_ens<<<nblocks, ON_NT, 0, s>>>(tab, blockmap);
    return cudaGetLastError();
}

cudaError_t launch_prep(const PrepArgs &a, cudaStream_t s) {
    const int nb = a.nfill / ON_NT;
    k_prep<<<nb, ON_NT, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_finish(const FinishArgs &a, cudaStream_t s) {
    const int nb = a.nstar > 0 ? (a.nstar + ON_NT - 1) / ON_NT : 1;
    k_finish<<<nb, ON_NT, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_energy_finish(const EnergyArgs &a, cudaStream_t s) {
    const int nb = a.nstar > 0 ? (a.nstar + ON_NT - 1) / ON_NT : 1;
    k_energy_finish<<<nb, ON_NT, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace pn
