// pn_pair_fix.cu -- instantiations and launcher of the fixed-point FP64 sweep (pn_pairfix.cuh).
#include "pn_internal.h"
#include "pn_pairfix.cuh"

namespace pn {

template <int MODE, int JS>
static cudaError_t launch_one(const PairCfg &c, const PairArgs &a, cudaStream_t s) {
    const size_t smem = fix_smem_bytes<MODE>();
    auto fn = k_pair_fix<MODE, JS>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int bi = PAIR_NT / JS;
    dim3 grid((unsigned)((a.nstar + bi - 1) / bi), (unsigned)c.gsplit);
    fn<<<grid, PAIR_NT, smem, s>>>(a);
    return cudaGetLastError();
}

template <int MODE>
static cudaError_t launch_mode(const PairCfg &c, const PairArgs &a, cudaStream_t s) {
    switch (c.js) {
        case 1: return launch_one<MODE, 1>(c, a, s);
        case 2: return launch_one<MODE, 2>(c, a, s);
        case 4: return launch_one<MODE, 4>(c, a, s);
        case 8: return launch_one<MODE, 8>(c, a, s);
        case 16: return launch_one<MODE, 16>(c, a, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_pair_fix(int mode, const PairCfg &c, const PairArgs &a, cudaStream_t s) {
    if (a.nstar <= 0) return cudaSuccess;
    if (c.ipt != 1 || c.tj != FIX_TJ || !a.fpack) return cudaErrorInvalidValue;
    switch (mode) {
        case MODE_NEWTON: return launch_mode<MODE_NEWTON>(c, a, s);
        case MODE_FORCE: return launch_mode<MODE_FORCE>(c, a, s);
        case MODE_ENERGY: return launch_mode<MODE_ENERGY>(c, a, s);
        case MODE_FORCE_ENERGY: return launch_mode<MODE_FORCE_ENERGY>(c, a, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace pn
