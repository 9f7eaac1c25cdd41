// pn_pairsym.cuh -- the mixed-precision force sweep over unordered pairs.
//
// As k_pair2<MODE_FORCE> (pn_pair2.cuh), but each pair of stars is formed once and serves both: their
// difference, inverse distance and dot products are shared, so an ordered pair costs 37.5 packed FP32
// operations instead of 50 (27 for the pair, 24 per star).
//
// A CTA of 128 threads holds 512 rows i in registers, four per thread, two to an f32x2 operand, and
// runs over a range of 128-star tiles j, from the tiles of its own rows on.  In each 32-star part of a
// tile lane l meets star (l + s) mod 32 at step s, so the lanes' stars differ and star j's sums travel with
// it from lane to lane, one shuffle per sum and step; after 32 steps they are back at its lane.  The four
// warps' sums of a tile are added in order and written to slot b (the CTA's row block) of star j.  A
// tile of the CTA's own rows is swept in both orders and gives row sums only.  Row sums are folded per
// tile with compensation, as in k_pair2, and written per range of tiles; k_sym_reduce adds a star's slots
// in order.  No atomics: the sums do not depend on scheduling.  The slots take 36 bytes per star and row
// block, so the stars j are swept in panels, as wide as a fixed workspace allows.
//
// The operands are k_pair2's scaled ones, but both sides hold w = sqrt(3) v: with a = w_i.w_j, P = w_i.d,
// S = w_j.d (d = x_j - x_i) star i's bracket has 4 a / 3 + S^2 Q'^2 and its ct the factor 4 P / 3 - S;
// star j's 4 a / 3 + P^2 Q'^2 and, with d reversed, P - 4 S / 3.  The terms -|v|^2 of the brackets and
// -w sum ct are applied once per tile.
//
// Row sums run over SPAN terms before they are folded, star j's over 64 in each half of an operand.
// SPAN is what k_pair2's tiles give: 128 for one system of 8,000 stars or more (256-star tiles),
// 64 for an ensemble, whose clusters may be small (128-star tiles; folding twice per tile costs 1 % there, and 4 %
// at N = 262,144).  Against FP64 the median error of the accelerations is 0.93 to 0.99 of k_pair2's for
// one system (N = 8,100 to 32,767, inv_c2 = 1e-6; 0.75 to 0.85 at 1); for ensembles of 128 to 4,000 stars
// the error of the whole vector is 0.95 of k_pair2's in the mean (with 128 terms it was 1.15 of it).
//
// Bound by the FP32 FMA pipe (75 % active at N = 16,384) and, with two warps per scheduler, by the latency
// between its instructions.  Per step of a warp that pipe takes 300 cycles, the shared-memory pipe of
// the SM 144 (16 wavefronts of loads and 20 shuffles for each of four warps): with half the rows it
// would be the limit.  Measured at N = 65,536: stars as pairs of equal values in shared memory (twice the
// loads) 6.09 ms, single values 5.71, two steps unrolled 5.47, four 5.50; three CTAs per SM (168 registers,
// spills) 5.74; k_pair2 6.31.  N = 262,144: 101.0 -> 84.5 ms; 16,384: 426 -> 365 us.
#pragma once

#include "pn_pair2.cuh"

namespace pn {

inline size_t sym2_smem_bytes() {
    return 128 + (size_t)2 * SYM2_NS * 4 * PAIR_NT * 4 + (size_t)4 * 10 * SYM2_TJ * 4 + (size_t)2 * SYM2_NG * SYM2_TJ * 16;
}

struct Row2 {  // two rows
    f2 ex, ey, ez, lx, ly, lz, wx, wy, wz, m, mu3, c1, c3, k35, qe;
};
struct Star2 {  // one star in both lanes
    f2 x, y, z, lx, ly, lz, wx, wy, wz, m, mu3, c1, c3, k35, qe;
};

// Sums: G, Phi, S0, U, W, ct (star j's with G and W negated)
template <bool BOTH>
__device__ __forceinline__ void sym2_pair(f2 *y, f2 *z, const Row2 &I, const Star2 &J, f2 eps2) {
    const f2 dx = add2(sub2(J.x, I.ex), sub2(J.lx, I.lx));
    const f2 dy = add2(sub2(J.y, I.ey), sub2(J.ly, I.ly));
    const f2 dz = add2(sub2(J.z, I.ez), sub2(J.lz, I.lz));
    const f2 rhoe = fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, eps2)));
    const f2 Q = rsqrt2k(rhoe), Q2 = mul2(Q, Q), Q3 = mul2(Q2, Q);
    const f2 P = fma2(I.wz, dz, fma2(I.wy, dy, mul2(I.wx, dx)));
    const f2 S = fma2(J.wz, dz, fma2(J.wy, dy, mul2(J.wx, dx)));
    const f2 a = fma2(I.wz, J.wz, fma2(I.wy, J.wy, mul2(I.wx, J.wx)));
    const f2 c43 = f2_bcast((float)(4.0 / 3.0));
    const f2 third = f2_bcast((float)(1.0 / 3.0));
    {
        const f2 mQ3 = mul2(J.m, Q3);
        y[0] = fma2(mQ3, dx, y[0]);
        y[1] = fma2(mQ3, dy, y[1]);
        y[2] = fma2(mQ3, dz, y[2]);
        y[3] = fma2(J.m, Q, y[3]);
        y[4] = add2(y[4], mQ3);
        y[5] = fma2(J.mu3, Q, y[5]);
        const f2 br = fma2(mul2(S, S), Q2, fma2(c43, a, fma2(sub2(rhoe, I.qe), J.c3, J.c1)));
        const f2 cd = fma2(mQ3, br, mul2(J.k35, Q));
        const f2 ct = mul2(mQ3, fma2(third, P, sub2(P, S)));
        y[6] = fma2(cd, dx, fma2(ct, J.wx, y[6]));
        y[7] = fma2(cd, dy, fma2(ct, J.wy, y[7]));
        y[8] = fma2(cd, dz, fma2(ct, J.wz, y[8]));
        y[9] = add2(y[9], ct);
    }
    if constexpr (BOTH) {
        const f2 mQ3 = mul2(I.m, Q3);
        z[0] = fma2(mQ3, dx, z[0]);
        z[1] = fma2(mQ3, dy, z[1]);
        z[2] = fma2(mQ3, dz, z[2]);
        z[3] = fma2(I.m, Q, z[3]);
        z[4] = add2(z[4], mQ3);
        z[5] = fma2(I.mu3, Q, z[5]);
        const f2 br = fma2(mul2(P, P), Q2, fma2(c43, a, fma2(sub2(rhoe, J.qe), I.c3, I.c1)));
        const f2 cd = fma2(mQ3, br, mul2(I.k35, Q));
        const f2 ct = mul2(mQ3, fma2(third, S, sub2(S, P)));
        z[6] = fma2(cd, dx, fma2(ct, I.wx, z[6]));
        z[7] = fma2(cd, dy, fma2(ct, I.wy, z[7]));
        z[8] = fma2(cd, dz, fma2(ct, I.wz, z[8]));
        z[9] = add2(z[9], ct);
    }
}

// Star q of a tile in shared memory.
__device__ __forceinline__ void sym2_load(Star2 &J, const float4 *b, int q) {
    const float4 g0 = b[q], g1 = b[SYM2_TJ + q], g2 = b[2 * SYM2_TJ + q], g3 = b[3 * SYM2_TJ + q];
    J.x = f2_bcast(g0.x); J.y = f2_bcast(g0.y); J.z = f2_bcast(g0.z); J.m = f2_bcast(g0.w);
    J.lx = f2_bcast(g1.x); J.ly = f2_bcast(g1.y); J.lz = f2_bcast(g1.z); J.mu3 = f2_bcast(g1.w);
    J.wx = f2_bcast(g2.x); J.wy = f2_bcast(g2.y); J.wz = f2_bcast(g2.z); J.c1 = f2_bcast(g2.w);
    J.c3 = f2_bcast(g3.x); J.k35 = f2_bcast(g3.y); J.qe = f2_bcast(g3.z);
}

template <bool BOTH, int SPAN>
__device__ __forceinline__ void sym2_span(f2 (&y)[2][10], float *zs, const Row2 (&I)[2], const float4 *b, f2 eps2, int k0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int from = (lane + 1) & 31;
    for (int k = k0; k < k0 + SPAN; k += 32) {
        f2 z[10];
#pragma unroll
        for (int c = 0; c < 10; ++c) z[c] = 0ull;
#pragma unroll 2
        for (int s = 0; s < 32; ++s) {
            Star2 J;
            sym2_load(J, b, k + ((lane + s) & 31));
            sym2_pair<BOTH>(y[0], z, I[0], J, eps2);
            sym2_pair<BOTH>(y[1], z, I[1], J, eps2);
            if constexpr (BOTH)
#pragma unroll
                for (int c = 0; c < 10; ++c) z[c] = __shfl_sync(0xffffffffu, z[c], from);
        }
        if constexpr (BOTH)
#pragma unroll
            for (int c = 0; c < 10; ++c) zs[(warp * 10 + c) * SYM2_TJ + k + lane] = f2_sum(z[c]);
    }
}

// One work item: row block blk against range y of the panel's tiles.  seq: the tiles that this CTA has
// consumed before (pair_block).  Returns false when a bounded wait gave up.
template <int SPAN>
__device__ __forceinline__ bool sym2_block(const Pair2SymArgs &a, int blk, int y, unsigned char *smem, uint32_t &seq) {
    constexpr int NT = PAIR_NT, TJ = SYM2_TJ, NS = SYM2_NS;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    float *kahan = reinterpret_cast<float *>(smem + 128);          // [2][9][4][128]
    float *zs = kahan + 2 * NS * 4 * NT;                           // [4][10][128]
    float4 *buf = reinterpret_cast<float4 *>(zs + 4 * 10 * TJ);    // [2][8][128]
    const int tid = threadIdx.x;
    const int tc = a.p0 + y * a.chunk, t0 = max(4 * blk, tc), t1 = min(a.p1, tc + a.chunk);
    if (t0 >= t1) return true;
    const f2 eps2 = f2_bcast((float)a.eps2);
    float sh[3][4], sl[3][4];
    Row2 I[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        float v[9][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = 2 * p + h, i = blk * SYM2_ROWS + tid + r * NT;
            const bool valid = i < a.nstar;
#pragma unroll
            for (int k = 0; k < 3; ++k) to_f32_pair(valid ? a.spos[(size_t)k * a.npad + i] : 0.0, sh[k][r], sl[k][r]);
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 g0 = valid ? a.pack[i] : zero, g1 = valid ? a.pack[(size_t)a.npad + i] : zero,
                         g2 = valid ? a.pack[(size_t)2 * a.npad + i] : zero, g3 = valid ? a.pack[(size_t)3 * a.npad + i] : zero;
            v[0][h] = g2.x; v[1][h] = g2.y; v[2][h] = g2.z; v[3][h] = g0.w; v[4][h] = g1.w;
            v[5][h] = g2.w; v[6][h] = g3.x; v[7][h] = g3.y; v[8][h] = g3.z;
        }
        I[p].wx = f2_pack(v[0][0], v[0][1]); I[p].wy = f2_pack(v[1][0], v[1][1]); I[p].wz = f2_pack(v[2][0], v[2][1]);
        I[p].m = f2_pack(v[3][0], v[3][1]); I[p].mu3 = f2_pack(v[4][0], v[4][1]); I[p].c1 = f2_pack(v[5][0], v[5][1]);
        I[p].c3 = f2_pack(v[6][0], v[6][1]); I[p].k35 = f2_pack(v[7][0], v[7][1]); I[p].qe = f2_pack(v[8][0], v[8][1]);
    }
    auto ksum = [&](int q, int r) -> float & { return kahan[(q * 4 + r) * NT + tid]; };
    auto kcmp = [&](int q, int r) -> float & { return kahan[((NS + q) * 4 + r) * NT + tid]; };
#pragma unroll
    for (int q = 0; q < NS; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) ksum(q, r) = kcmp(q, r) = 0.f;

    constexpr uint32_t gbytes = TJ * 16u;
    auto issue = [&](int t, int stage) {
        mbar_arrive_expect_tx(&bars[stage], SYM2_NG * gbytes);
#pragma unroll
        for (int g = 0; g < SYM2_NG; ++g)
            bulk_g2s(buf + (size_t)(stage * SYM2_NG + g) * TJ, a.pack + (size_t)g * a.npad + (size_t)t * TJ, gbytes, &bars[stage]);
    };
    if (tid == 0) issue(t0, (int)(seq & 1u));
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
        {
            const TileOrigin &o = a.torg[t];
            const float oh[3] = {o.hx, o.hy, o.hz}, ol[3] = {o.lx, o.ly, o.lz};
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                float h[3][2], l[3][2];
#pragma unroll
                for (int k = 0; k < 3; ++k)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float err;
                        h[k][e] = two_diff(sh[k][2 * p + e], oh[k], err);
                        l[k][e] = err + (sl[k][2 * p + e] - ol[k]);
                    }
                I[p].ex = f2_pack(h[0][0], h[0][1]); I[p].ey = f2_pack(h[1][0], h[1][1]); I[p].ez = f2_pack(h[2][0], h[2][1]);
                I[p].lx = f2_pack(l[0][0], l[0][1]); I[p].ly = f2_pack(l[1][0], l[1][1]); I[p].lz = f2_pack(l[2][0], l[2][1]);
            }
        }
        const float4 *b = buf + (size_t)stage * SYM2_NG * TJ;
        const bool both = t >= 4 * blk + 4;  // (the whole CTA)
#pragma unroll 1
        for (int k = 0; k < TJ; k += SPAN) {
            f2 y[2][10];
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int c = 0; c < 10; ++c) y[p][c] = 0ull;
            if (both)
                sym2_span<true, SPAN>(y, zs, I, b, eps2, k);
            else
                sym2_span<false, SPAN>(y, zs, I, b, eps2, k);
            // rows: -w sum ct and -|v|^2 G into W, then the running sums
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const f2 third = f2_bcast((float)(-1.0 / 3.0));
                const f2 nv2 = mul2(third, fma2(I[p].wz, I[p].wz, fma2(I[p].wy, I[p].wy, mul2(I[p].wx, I[p].wx))));
                const f2 nct = sub2(0ull, y[p][9]);
                y[p][6] = fma2(nct, I[p].wx, fma2(nv2, y[p][0], y[p][6]));
                y[p][7] = fma2(nct, I[p].wy, fma2(nv2, y[p][1], y[p][7]));
                y[p][8] = fma2(nct, I[p].wz, fma2(nv2, y[p][2], y[p][8]));
#pragma unroll
                for (int q = 0; q < NS; ++q) {
                    float ts[2];
                    f2_unpack(y[p][q], ts[0], ts[1]);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float sum = ksum(q, 2 * p + e), comp = kcmp(q, 2 * p + e);
                        kahan_add(sum, comp, ts[e]);
                        ksum(q, 2 * p + e) = sum;
                        kcmp(q, 2 * p + e) = comp;
                    }
                }
            }
        }
        __syncthreads();
        if (both) {  // star j = tid of the tile: the warps' sums in order, its own velocity terms
            float s[10];
#pragma unroll
            for (int c = 0; c < 10; ++c)
                s[c] = (zs[c * TJ + tid] + zs[(10 + c) * TJ + tid]) + (zs[(20 + c) * TJ + tid] + zs[(30 + c) * TJ + tid]);
            const float wx = b[2 * TJ + tid].x, wy = b[2 * TJ + tid].y, wz = b[2 * TJ + tid].z;
            const float v2 = (1.f / 3.f) * fmaf(wz, wz, fmaf(wy, wy, wx * wx));
            s[6] = fmaf(s[9], wx, fmaf(v2, s[0], -s[6]));
            s[7] = fmaf(s[9], wy, fmaf(v2, s[1], -s[7]));
            s[8] = fmaf(s[9], wz, fmaf(v2, s[2], -s[8]));
            float *out = a.cols + (size_t)blk * NS * a.cstride + (size_t)(t - a.p0) * TJ + tid;
#pragma unroll
            for (int q = 0; q < NS; ++q) out[(size_t)q * a.cstride] = q < 3 ? -s[q] : s[q];
            __syncthreads();  // every thread is done with this stage and zs
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = blk * SYM2_ROWS + tid + r * NT;
        if (i < a.nstar)
#pragma unroll
            for (int q = 0; q < NS; ++q)
                a.rows[((size_t)y * NS + q) * a.rstride + i] = make_float2(ksum(q, r), -kcmp(q, r));
    }
    seq += (uint32_t)(t1 - t0);
    return true;
}

__device__ __forceinline__ void sym2_init(unsigned char *smem) {
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
}

__global__ void __launch_bounds__(PAIR_NT, 2) k_pair2_sym(const Pair2SymArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    sym2_init(smem);
    uint32_t seq = 0;
    sym2_block<128>(a, blockIdx.x, blockIdx.y, smem, seq);
}

// Ensemble form, as k_pair2_ens: items (cluster, row block, range, 0), one panel per cluster.
__global__ void __launch_bounds__(PAIR_NT, 2)
    k_pair2_sym_ens(const Pair2SymArgs *tab, const int4 *items, int nitems, unsigned *counter) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int cur;
    sym2_init(smem);
    uint32_t seq = 0;
    for (;;) {
        if (threadIdx.x == 0) cur = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int w = cur;
        __syncthreads();  // everyone has read cur before thread 0 fetches the next item
        if (w >= nitems) break;
        const int4 it = items[w];
        const Pair2SymArgs a = tab[it.x];
        if (!sym2_block<64>(a, it.y, it.z, smem, seq)) break;
    }
}

// Adds a star's slots of a panel in order: the row sums of its block's ranges, then the column sums from
// the row blocks before its own (a star of an earlier panel only has row sums there, on top of its
// sums so far).  One thread per (star, sum).
__device__ __forceinline__ void sym_reduce_star(const Pair2SymArgs &a, int i, int q) {
    if (i >= min(a.nstar, a.p1 * SYM2_TJ)) return;
    const int blk = i / SYM2_ROWS, nchunk = (a.p1 - a.p0 + a.chunk - 1) / a.chunk, j = i - a.p0 * SYM2_TJ;
    float2 *out = a.out + (size_t)q * a.npad + i;
    float h = 0.f, l = 0.f;
    if (j < 0) {
        const float2 o = *out;
        h = o.x;
        l = o.y;
    }
    const int c0 = max(0, 4 * blk - a.p0) / a.chunk;
    const float2 *rows = a.rows + (size_t)q * a.rstride + i;
    const size_t rs = (size_t)SYM2_NS * a.rstride, cs = (size_t)SYM2_NS * a.cstride;
    for (int c = c0; c < nchunk; c += 16) {  // (16 loads in flight; adding zeros changes nothing)
        float2 t[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) t[u] = c + u < nchunk ? rows[(c + u) * rs] : make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 16; ++u) pair_add(h, l, t[u]);
    }
    if (j >= 0) {
        const float *cols = a.cols + (size_t)q * a.cstride + j;
        for (int b = 0; b < blk; b += 16) {
            float t[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) t[u] = b + u < blk ? cols[(b + u) * cs] : 0.f;
#pragma unroll
            for (int u = 0; u < 16; ++u) pair_add(h, l, make_float2(t[u], 0.f));
        }
    }
    *out = make_float2(h, l);
}
__global__ void __launch_bounds__(256) k_sym_reduce(const Pair2SymArgs a) {
    sym_reduce_star(a, blockIdx.x * 256 + threadIdx.x, blockIdx.y);
}
__global__ void __launch_bounds__(128) k_sym_reduce_ens(const Pair2SymArgs *tab, const int4 *blockmap) {
    const int4 bm = blockmap[blockIdx.x];
    const Pair2SymArgs a = tab[bm.x];
    sym_reduce_star(a, bm.y * 128 + threadIdx.x, blockIdx.y);
}

}  // namespace pn
