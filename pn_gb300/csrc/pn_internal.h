// pn_internal.h -- host-side declarations shared by libpn's translation units.
#pragma once

#include <cuda_runtime.h>

#include "pn_pair.cuh"

namespace pn {

struct PairCfg {
    int ipt = 2;     // i-particles per thread
    int js = 1;      // lanes sharing one i-set
    int tj = 128;    // stars per j-tile
    int gsplit = 1;  // j-range splits across CTAs
    int x2 = 0;      // FP32: the packed f32x2 sweep (pn_pair2.cuh; js = 1, ipt 1 or 2);
                     // 2 / 3 = the same sized for 3 / 4 CTAs per SM (ipt 2, force sweeps)
                     // 4 = the sweep over unordered pairs (pn_pairsym.cuh; MODE_FORCE, tj 128,
                     // gsplit = tiles per CTA)
                     // FP64: 1 = the fixed-point sweep (pn_pairfix.cuh; ipt 1, tj 128)
};

// j-range splits that the sweep's partial sums have
inline int acc_splits(const PairCfg &c) { return c.x2 == 4 ? 1 : c.gsplit; }

// Launches k_pair for the given precision/mode/shape (returns cudaErrorInvalidValue for an
// unsupported (ipt, js) combination).  Implemented in pn_pair_f32.cu / pn_pair_f64.cu.
cudaError_t launch_pair_f32(int mode, const PairCfg &c, const PairArgs &a, cudaStream_t s);
cudaError_t launch_pair_f64(int mode, const PairCfg &c, const PairArgs &a, cudaStream_t s);
// The FP64 sweep on the integer pipes (PairCfg::x2 = 1 in FP64; pn_pair_fix.cu): ipt 1, js 1..16,
// tiles of 128.
cudaError_t launch_pair_fix(int mode, const PairCfg &c, const PairArgs &a, cudaStream_t s);
constexpr int FIX_GROUPS = 13;  // 16-byte groups per star of its pack
// Its units for a softening and a weight of the 1PN terms; false where its range does not cover the softening.
bool fix_units(double eps, double inv_c2, FixUnits *u);
bool pair_shape_supported(int ipt, int js);
// The mixed force sweep over unordered pairs (PairCfg::x2 = 4; pn_pair_sym.cu), whose partial sums take
// sym_bytes of work, at most SYM_PANEL_BYTES (or one panel of 4 tiles).
constexpr size_t SYM_PANEL_BYTES = (size_t)512 << 20;
size_t sym_bytes(int nstar, int chunk);
int sym_panels(int nstar, int chunk);
// (its argument block: pn_pairsym.cuh)
constexpr int SYM2_ROWS = 512, SYM2_TJ = 128, SYM2_NG = 4, SYM2_NS = 9;

struct Pair2SymArgs {
    const float4 *pack;      // [SYM2_NG][npad]: (x y z m) (lx ly lz mu3) (wx wy wz c1) (c3 k35 qe 0), scaled (k_prep)
    const TileOrigin *torg;  // per tile of 128
    const double *spos;
    float2 *rows;            // [chunks][9][rstride] row sums (sum, -compensation) of each range of tiles
    float *cols;             // [blocks][9][cstride] sums of the panel's star j from row block b
    float2 *out;             // [9][npad]
    int *err;
    int nstar, npad, chunk;  // tiles per range
    int p0, p1;              // tiles of this panel (multiples of 4, or the last tile)
    int rstride, cstride;
    double eps2;
};
// Its ensemble form: one panel per cluster (tab[c]), items (cluster, row block, range of chunk tiles, 0);
// blockmap, nblocks: the O(N) kernels' blocks of 128 stars.  sym_ens_bytes: a cluster's partial sums.
size_t sym_ens_bytes(int nstar, int chunk);
void sym_ens_args(Pair2SymArgs *a, int nstar, int chunk, void *work);
cudaError_t launch_pair_sym_ens(const Pair2SymArgs *tab, const int4 *items, int nitems, const int4 *blockmap,
                                int nblocks, int sms, unsigned *counter, cudaStream_t s);
cudaError_t launch_pair_sym(const PairCfg &c, const PairArgs &a, void *work, cudaStream_t s);

// Persistent ensemble sweep (k_pair_ens): (ipt, js) in {(1,1), (2,1), (1,4)}; tjmax = the
// largest tile size among the clusters; grid <= 0 = one wave of resident CTAs.
cudaError_t launch_pair_ens_f32(int mode, int ipt, int js, int tjmax, int grid, const PairArgs *tab,
                                const int4 *items, int nitems, unsigned *counter, cudaStream_t s);
cudaError_t launch_pair_ens_f64(int mode, int ipt, int js, int tjmax, int grid, const PairArgs *tab,
                                const int4 *items, int nitems, unsigned *counter, cudaStream_t s);
// the packed FP32x2 form of the ensemble sweep (tab[c].pack2 / ipack set; js = 1, ipt 1 or 2)
cudaError_t launch_pair2_ens_f32(int mode, int ipt, int tjmax, int grid, const PairArgs *tab,
                                 const int4 *items, int nitems, unsigned *counter, cudaStream_t s);
inline bool ens_shape_supported(int ipt, int js) {
    return (js == 1 && (ipt == 1 || ipt == 2)) || (ipt == 1 && js == 4);
}

inline int pair_ng(bool f32, int mode) {
    if (f32) return mode == MODE_NEWTON ? ModeInfo<MODE_NEWTON>::NG32
                  : mode_has_force(mode) ? ModeInfo<MODE_FORCE>::NG32
                                         : ModeInfo<MODE_ENERGY>::NG32;
    return mode == MODE_NEWTON ? ModeInfo<MODE_NEWTON>::NG64
         : mode_has_force(mode) ? ModeInfo<MODE_FORCE>::NG64
                                : ModeInfo<MODE_ENERGY>::NG64;
}

inline int pair_nacc(int mode) {
    return mode == MODE_NEWTON ? ModeInfo<MODE_NEWTON>::NACC
         : mode == MODE_FORCE  ? ModeInfo<MODE_FORCE>::NACC
         : mode == MODE_FORCE_ENERGY ? ModeInfo<MODE_FORCE_ENERGY>::NACC
                               : ModeInfo<MODE_ENERGY>::NACC;
}

inline int pair_block_i(const PairCfg &c) { return PAIR_NT * c.ipt / c.js; }

}  // namespace pn
