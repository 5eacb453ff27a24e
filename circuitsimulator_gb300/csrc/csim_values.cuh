// csim_values.cuh — a state's exact sum as the estimators' doubles, by one warp.
// Shared by k_tree_values (csim_tree.cu) and k_seg_values (csim_batch_kernels.cu).
#pragma once

#include <cstdint>

#include "csim_warp.cuh"

namespace csim {

// z to double, to nearest even as the host's conversion: the top 64 bits with the
// rest folded into the lowest one convert with a single rounding
__device__ __forceinline__ double int128_to_double(__int128 z) {
    const bool neg = z < 0;
    const unsigned __int128 a = neg ? -(unsigned __int128)z : (unsigned __int128)z;
    const uint64_t hi = (uint64_t)(a >> 64), lo = (uint64_t)a;
    double d;
    if (hi == 0ull) {
        d = __ull2double_rn(lo);
    } else {
        const int s = 64 - __clzll((long long)hi);  // 1..64
        const uint64_t top = s == 64 ? hi : ((hi << (64 - s)) | (lo >> s));
        const uint64_t rest = s == 64 ? lo : lo << (64 - s);
        d = __dmul_rn(__ull2double_rn(top | (rest != 0ull ? 1ull : 0ull)), __hiloint2double((1023 + s) << 20, 0));
    }
    return neg ? -d : d;
}

__device__ __forceinline__ __int128 shfl_xor_i128(__int128 v, int m) {
    const uint64_t lo = shfl_xor64((uint64_t)v, m), hi = shfl_xor64((uint64_t)((unsigned __int128)v >> 64), m);
    return (__int128)(((unsigned __int128)hi << 64) | lo);
}

// Lane q < 4 holds coordinate q of a sum z in Z[w], scaled by 2^t, and for
// exactProjector's rows (`row`) coordinate q of the diagonal term d.  Returns
// factor times z (or d + 2 Re z, innerprod.c:187-195) as a + i b, with the host's own
// roundings (csim_host::zomega_to_complex: no fused multiply-adds).
__device__ __forceinline__ void warp_value(__int128 z, bool row, __int128 d, int t, double factor, double& a, double& b) {
    const int q = lane_id() & 3;
    // coordinates 0..3 give z0, z1 - z3, z2, z1 + z3
    const __int128 other = shfl_xor_i128(z, 2);
    __int128 v = q == 1 ? z - other : (q == 3 ? other + z : z);
    if (row) {  // warp-uniform; 2 Re(o) = 2 o0 + (o1 - o3) (w - w^3)
        const __int128 dother = shfl_xor_i128(d, 2);
        v = q == 0 ? d + 2 * z : (q == 1 ? d - dother + 2 * v : (q == 2 ? d : dother + d));
    }
    const double x = int128_to_double(v);
    const double s = 0.70710678118654752440;
    const double x0 = __shfl_sync(kFull, x, 0), x1 = __shfl_sync(kFull, x, 1), x2 = __shfl_sync(kFull, x, 2),
                 x3 = __shfl_sync(kFull, x, 3);
    const double unit = __hiloint2double((1023 - t) << 20, 0);  // 2^-t
    a = __dmul_rn(__dmul_rn(__dadd_rn(x0, __dmul_rn(x1, s)), unit), factor);
    b = __dmul_rn(__dmul_rn(__dadd_rn(x2, __dmul_rn(x3, s)), unit), factor);
}
// singleProjectorSample's value 2^t |a + i b|^2 (innerprod.c:142)
__device__ __forceinline__ double sample_value(double a, double b, int t) {
    return __dmul_rn(__hiloint2double((1023 + t) << 20, 0), __dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)));
}

}  // namespace csim
