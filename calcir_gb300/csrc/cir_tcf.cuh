// The sums of the correlation terms, for the contraction (k_tcf.cu) and the propagation's small
// products, whose epilogue contracts the tile it holds (k_gemm.cu).
#ifndef CIR_TCF_CUH_
#define CIR_TCF_CUH_

#include <float.h>

namespace {

// A sum held as an unevaluated pair of floats (Knuth's two-sum), on the FP32 pipe: in double the eight
// sums of a warp (40 adds, 16 clocks each for the warp) were most of the kernel.  48 bits for sums of FP32
// products: IR, VV and VH of random F, against 64 bits and relative to the vectors' norms, 3.1e-9,
// 7.5e-10 and 4.2e-10 at order 100, 1.8e-9, 4.0e-10 and 1.8e-10 at 2048 (with sums in double, in
// the order of the rows, 4.1e-9, 1.2e-9 and 5.4e-10; 2.0e-9, 4.6e-10 and 1.8e-10): the products' rounding.
// hi is the plain FP32 sum; where it is not finite, lo is NaN and hi is the sum (pair_value).
struct Pair {
    float hi, lo;
};
__device__ __forceinline__ Pair pair_add(Pair a, float x) {
    const float s = __fadd_rn(a.hi, x), v = __fsub_rn(s, a.hi);
    return {s, __fadd_rn(a.lo, __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, v)), __fsub_rn(x, v)))};
}
__device__ __forceinline__ Pair pair_add(Pair a, Pair b) {
    Pair r = pair_add(a, b.hi);
    r.lo = __fadd_rn(r.lo, b.lo);
    return r;
}
__device__ __forceinline__ double pair_value(Pair a) {
    return (double)a.hi + (fabsf(a.hi) <= FLT_MAX ? (double)a.lo : 0.0);
}
__device__ __forceinline__ Pair pair_xor(Pair a, int o) {
    return {__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)};
}

// the four sums (re, im) of one row's (partial) psi with m(t): IR, iiFii, ijFij, iiFjj
__device__ __forceinline__ void tcf_sums(const float (&pr)[9], const float (&pi)[9], const float (&c)[9], Pair (&acc)[8]) {
    acc[0] = pair_add(acc[0], c[0] * pr[0] + c[1] * pr[1] + c[2] * pr[2]);
    acc[1] = pair_add(acc[1], c[0] * pi[0] + c[1] * pi[1] + c[2] * pi[2]);
    acc[2] = pair_add(acc[2], c[3] * pr[3] + c[4] * pr[4] + c[5] * pr[5]);
    acc[3] = pair_add(acc[3], c[3] * pi[3] + c[4] * pi[4] + c[5] * pi[5]);
    acc[4] = pair_add(acc[4], c[6] * pr[6] + c[7] * pr[7] + c[8] * pr[8]);
    acc[5] = pair_add(acc[5], c[6] * pi[6] + c[7] * pi[7] + c[8] * pi[8]);
    // xx->yy, xx->zz, yy->xx, yy->zz, zz->xx, zz->yy (psi index 3, 4, 5 = xx, yy, zz)
    acc[6] = pair_add(acc[6], (c[4] + c[5]) * pr[3] + (c[3] + c[5]) * pr[4] + (c[3] + c[4]) * pr[5]);
    acc[7] = pair_add(acc[7], (c[4] + c[5]) * pi[3] + (c[3] + c[5]) * pi[4] + (c[3] + c[4]) * pi[5]);
}

// A warp's eight sums meet by halves: the lanes whose bit is set keep the upper half of what is
// left, so nine exchanges do for all eight.  Lane l gets sum l >> 2.
__device__ __forceinline__ double tcf_reduce(Pair (&acc)[8]) {
    const int lane = threadIdx.x & 31;
    #pragma unroll
    for (int w = 4; w > 0; w >>= 1) {
        const bool up = lane & (4 * w);
        #pragma unroll
        for (int q = 0; q < w; q++) {
            const Pair send = up ? acc[q] : acc[q + w], keep = up ? acc[q + w] : acc[q];
            acc[q] = pair_add(keep, pair_xor(send, 4 * w));
        }
    }
    acc[0] = pair_add(acc[0], pair_xor(acc[0], 2));
    acc[0] = pair_add(acc[0], pair_xor(acc[0], 1));
    return pair_value(acc[0]);
}

// a warp whose lane l < 8 holds sum l adds IR, VV, VH (re, im) to out
__device__ __forceinline__ void tcf_add(double s, double *out) {
    const int lane = threadIdx.x & 31, im = lane & 1;
    const double ii = __shfl_sync(0xffffffffu, s, 2 + im), ij = __shfl_sync(0xffffffffu, s, 4 + im),
                 jj = __shfl_sync(0xffffffffu, s, 6 + im);
    if (lane < 6)
        atomicAdd(out + lane, lane < 2 ? s : lane < 4 ? (3.0 * ii + jj + 4.0 * ij) / 15.0 : (2.0 * ii - jj + 6.0 * ij) / 30.0);
}

}  // namespace

#endif
