// pn_pair_sym.cu -- launcher of the mixed force sweep over unordered pairs (pn_pairsym.cuh).
#include <algorithm>

#include "pn_internal.h"
#include "pn_pairsym.cuh"

namespace pn {

// A panel is the widest range of tiles whose sums fit SYM_PANEL_BYTES: from tile p0 to the result.
static size_t panel_bytes(int p0, int p1, int chunk) {
    const size_t w = p1 - p0, blocks = (p1 + 3) / 4;
    return SYM2_NS * SYM2_TJ * (blocks * w * sizeof(float) + (w + chunk - 1) / chunk * (size_t)p1 * sizeof(float2));
}
static int panel_end(int p0, int ntiles, int chunk) {
    int lo = p0 + 4, hi = (ntiles - p0 + 3) / 4 * 4 + p0;  // (multiples of 4 beyond p0)
    while (lo < hi) {
        const int mid = lo + (hi - lo + 4) / 8 * 4;
        if (panel_bytes(p0, mid, chunk) <= SYM_PANEL_BYTES) lo = mid;
        else hi = mid - 4;
    }
    return std::min(lo, ntiles);
}

size_t sym_bytes(int nstar, int chunk) {
    const int ntiles = (nstar + SYM2_TJ - 1) / SYM2_TJ;
    size_t most = 0;
    for (int p0 = 0, p1; p0 < ntiles; p0 = p1) {
        p1 = panel_end(p0, ntiles, chunk);
        most = std::max(most, panel_bytes(p0, p1, chunk));
    }
    return most;
}

int sym_panels(int nstar, int chunk) {
    const int ntiles = (nstar + SYM2_TJ - 1) / SYM2_TJ;
    int n = 0;
    for (int p0 = 0; p0 < ntiles; p0 = panel_end(p0, ntiles, chunk)) ++n;
    return n;
}

size_t sym_ens_bytes(int nstar, int chunk) { return panel_bytes(0, (nstar + SYM2_TJ - 1) / SYM2_TJ, chunk); }

void sym_ens_args(Pair2SymArgs *a, int nstar, int chunk, void *work) {
    a->nstar = nstar;
    a->chunk = chunk;
    a->p0 = 0;
    a->p1 = (nstar + SYM2_TJ - 1) / SYM2_TJ;
    a->rstride = a->cstride = a->p1 * SYM2_TJ;
    a->rows = static_cast<float2 *>(work);
    a->cols = reinterpret_cast<float *>(a->rows + (size_t)((a->p1 + chunk - 1) / chunk) * SYM2_NS * a->rstride);
}

cudaError_t launch_pair_sym_ens(const Pair2SymArgs *tab, const int4 *items, int nitems, const int4 *blockmap,
                                int nblocks, int sms, unsigned *counter, cudaStream_t s) {
    if (nitems <= 0) return cudaSuccess;
    const size_t smem = sym2_smem_bytes();
    cudaError_t e = cudaFuncSetAttribute(k_pair2_sym_ens, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_pair2_sym_ens<<<2 * sms, PAIR_NT, smem, s>>>(tab, items, nitems, counter);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_sym_reduce_ens<<<dim3(nblocks, SYM2_NS), 128, 0, s>>>(tab, blockmap);
    return cudaGetLastError();
}

cudaError_t launch_pair_sym(const PairCfg &c, const PairArgs &q, void *work, cudaStream_t s) {
    if (q.nstar <= 0) return cudaSuccess;
    if (c.tj != SYM2_TJ || c.gsplit < 1 || !work) return cudaErrorInvalidValue;
    const size_t smem = sym2_smem_bytes();
    cudaError_t e = cudaFuncSetAttribute(k_pair2_sym, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    Pair2SymArgs a{};
    a.pack = static_cast<const float4 *>(q.pack);
    a.torg = q.torg; a.spos = q.spos; a.out = reinterpret_cast<float2 *>(q.out); a.err = q.err;
    a.nstar = q.nstar; a.npad = q.npad; a.chunk = c.gsplit; a.eps2 = q.eps2;
    const int ntiles = (q.nstar + SYM2_TJ - 1) / SYM2_TJ;
    for (; a.p0 < ntiles; a.p0 = a.p1) {
        a.p1 = panel_end(a.p0, ntiles, a.chunk);
        const int w = a.p1 - a.p0, nchunk = (w + a.chunk - 1) / a.chunk, blocks = (a.p1 + 3) / 4;
        a.rstride = a.p1 * SYM2_TJ;
        a.cstride = w * SYM2_TJ;
        a.rows = static_cast<float2 *>(work);
        a.cols = reinterpret_cast<float *>(a.rows + (size_t)nchunk * SYM2_NS * a.rstride);
        k_pair2_sym<<<dim3(blocks, nchunk), PAIR_NT, smem, s>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        k_sym_reduce<<<dim3((std::min(a.p1 * SYM2_TJ, a.nstar) + 255) / 256, SYM2_NS), 256, 0, s>>>(a);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace pn
