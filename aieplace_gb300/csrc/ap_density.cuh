// Density of a pair of bins from the fixed-point maps, shared by the density
// kernel (k_density.cu) and the field solve's first pass (k_field_fft.cu).
#pragma once

#include "ap_kernels.h"

namespace ap {

// The two bins' maps as loaded (fl: filler cells, zero without them).
struct BinPair {
    longlong2 mv, fs, fx, fl;
};

__device__ __forceinline__ BinPair load_pair(const RhoArgs &a, int p) {
    BinPair b;
    b.mv = __ldcg(reinterpret_cast<const longlong2 *>(a.mov_q) + p);
    b.fs = __ldg(reinterpret_cast<const longlong2 *>(a.fixs_q) + p);
    b.fx = __ldg(reinterpret_cast<const longlong2 *>(a.fix_q) + p);
    b.fl = a.fill_q ? __ldcg(reinterpret_cast<const longlong2 *>(a.fill_q) + p) : make_longlong2(0, 0);
    return b;
}

// Clears pair p of the moving maps for the next evaluation, adds to the
// overflow sums and returns the solver's input.
__device__ __forceinline__ float2 take_pair(const RhoArgs &a, int p, const BinPair &b, long long &over,
                                            long long &over_abs) {
    reinterpret_cast<longlong2 *>(a.mov_q)[p] = make_longlong2(0, 0);
    if (a.fill_q) reinterpret_cast<longlong2 *>(a.fill_q)[p] = make_longlong2(0, 0);
    const long long m[2] = {b.mv.x, b.mv.y}, sq[2] = {b.fs.x, b.fs.y}, f[2] = {b.fx.x, b.fx.y};
    const long long fil[2] = {b.fl.x, b.fl.y};
    float d[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const long long tot = m[k] + sq[k];
        const long long t = tot - a.cap_q;
        over += t > 0 ? t : 0;
        const long long ab = m[k] + f[k] - a.ab_q;
        over_abs += ab > 0 ? ab : 0;
        d[k] = fmaf(ll2f_rn_bits(tot + fil[k]), a.inv_ab_f, -a.d_shift);
    }
    return make_float2(d[0], d[1]);
}

}  // namespace ap
