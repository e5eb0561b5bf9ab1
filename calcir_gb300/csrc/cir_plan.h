// Host-side planning of the batched runners (no CUDA): included by cir_api.cu and compiled
// on its own by the CPU tests.
#pragma once

#include <algorithm>
#include <cmath>

// Chunk length for K steps of St origins, at most kn_max steps a chunk.  The
// tridiagonalisation runs `wave` matrices at a time, and a chunk whose last wave is nearly
// empty pays for about a third of a wave while its few blocks run alone (measured with 456
// blocks resident: 3232 matrices of order 1024, 7.09 waves, 525 ms; 3168, 6.95 waves, 501 ms).
// Of the chunkings into as few chunks as kn_max allows, equal in length but the last, the
// one with the least estimated time is taken: whole waves, a part-filled last wave counted
// as at least 0.3 of one; ties go to the longer chunks.
inline int cir_plan_chunk(int K, int St, int kn_max, int wave) {
    kn_max = std::max(1, std::min(kn_max, K));
    wave = std::max(1, wave);
    const int nc = (K + kn_max - 1) / kn_max, kn_min = (K + nc - 1) / nc;
    double best = 1e300;
    int pick = kn_max;
    for (int kn = kn_max; kn >= kn_min; kn--) {
        double cost = 0.0;
        for (int k0 = 0; k0 < K && cost < best; k0 += kn) {
            const double w = (double)St * std::min(kn, K - k0) / wave, f = w - std::floor(w);
            cost += std::floor(w) + (f > 0.0 ? std::max(f, 0.3) : 0.0);
        }
        if (cost < best - 1e-9) {
            best = cost;
            pick = kn;
        }
    }
    return pick;
}

// The first part of a chunk's eigensolver batch split over two streams: whole waves of the
// tridiagonalisation, all but the last one (0: no split, fewer than two waves).
inline int cir_split_first_part(int nmat, int wave) {
    wave = std::max(1, wave);
    return nmat >= 2 * wave ? (nmat / wave - 1) * wave : 0;
}

// The tridiagonalisation's kernel, by order and number of matrices alone: what the autotuner measured
// on other batches of that order changes neither a batch's kernel nor its bits.  Orders up to 192, and
// up to 256 in a single wave, stay in shared memory, the more warps per matrix the fewer matrices there
// are (n = 128: 0.25 ms a matrix in 8 warps; n = 256, 320 matrices: 2.1 ms resident, one per SM, 2.0
// ms streaming, two per SM).  Above, two blocks of 8 warps per SM fill each other's barriers (512: 5.5
// ms per 304 matrices, one block of 16 warps 6.3), a single wave is better off with 16 warps (3.1
// against 3.6 ms); orders above 512 take a block of 16 warps or a cluster of them.
enum CirTridiagForm { CIR_TRI_RES4, CIR_TRI_RES8, CIR_TRI_STREAM8, CIR_TRI_WIDE };
inline CirTridiagForm cir_tridiag_form(int n, int nmat, int sms) {
    if (n <= 128 && nmat > 2 * sms) return CIR_TRI_RES4;
    if (n <= 192 || (n <= 256 && nmat <= sms)) return CIR_TRI_RES8;
    return n <= 512 && nmat > sms ? CIR_TRI_STREAM8 : CIR_TRI_WIDE;
}

// The autotuner's blocks per SM, measured on more than two waves of one block per SM, where a batch
// is as large; else 0, the kernel's own number.
inline int cir_tridiag_limit(int tuned, int nmat, int sms) { return nmat > 2 * sms ? tuned : 0; }

// Whether the field's sums take a warp per chromophore (wide) or a thread.  In us: the wide form by
// the chromophores on the whole device (each block stages all molecules, so that large boxes leave few
// blocks an SM), the other as long as one thread's run over its molecules until it fills the device.
// Fits to 1..1000 molecules and 1..3000 frames; measured, wide against narrow: 5 x 1000 14.5 / 10.4,
// 40 x 100 21 / 29, 100 x 30 34 / 56, 100 x 100 82 / 63, 343 x 10 65 / 109, 343 x 30 168 / 119, 1000 x 2
// 160 / 234, 1000 x 4 280 / 236, 1000 x 30 1958 / 500.
inline bool cir_build_wide(int n, int nmol, int nframes, int sms) {
    const double m = nmol, wide = 5.0 + 1e-3 * n * nframes * (1.0 + 0.02 * m + 1.2e-5 * m * m) * 152.0 / sms;
    return wide < 8.0 + std::min(0.42 * m, 42.0 + 0.18 * m);
}

// The FP32 product's kernel (k_gemm.cu): the least of four fits in us to 1800 measurements on 152 SMs
// (M, N, K 8..2048, batches 1..600, operands' and outputs' rows aligned to 16 bytes and not, with and without C = D - A B; within
// 6% of the fastest in 95% of them).  Tiles of 32 with four groups along K while there are few, of 64 for
// many products of order 24 to about 110 and for short K, of 128 for some of order 65 to 112 in large
// batches, and the tensor cores.  Measured (small, 64, 128, tensor cores): 128 x 256 x 128 6.6, 10, 25,
// 15; 65 x 130 x 65 in 150, rows not aligned, 30, 28, 22, 29; 50 x 100 x 50 in 300 31, 15, 19, 21; 686 x 686 x
// 128 in 64, C = D - A B, not aligned, 514, 297, 324, 739; aligned 474, 244, 282, 175; 512 x 1024 x 512 29, 27,
// 76, 29; 1024 x 2048 x 1024 154, 138, 146, 50.
enum CirGemmForm { CIR_GEMM_SMALL, CIR_GEMM_TILE64, CIR_GEMM_TILE128, CIR_GEMM_TC };
inline CirGemmForm cir_gemm_form(int M, int N, int K, int batch, int epilogue, bool in16, bool out16, int sms) {
    auto tiles = [&](int t) { return (double)((M + t - 1) / t) * ((N + t - 1) / t) * batch; };
    auto slices = [&](int k) { return (double)((K + k - 1) / k); };
    const double b32 = tiles(32) / sms, b64 = tiles(64) / sms, t128 = tiles(128), sub = epilogue == 2 ? 1.0 : 0.0;
    const double t[4] = {
        4.4 + slices(128) * std::max(1.92, 1.14 * b32) + 0.46 * b32,
        4.9 + slices(16) * std::max(0.63, 0.556 * b64) * (in16 ? 1.0 : 1.09) + 0.24 * sub * b64,
        2.7 + std::ceil(t128 / (2 * sms)) * (1.054 * slices(8) * (t128 > sms ? 1.57 : 1.0) * (in16 ? 1.0 : 1.035) + 2.76),
        3.5 + std::ceil(t128 / sms) * (out16 ? (in16 ? 1.44 : 1.75) * slices(32) + 4.8 + 2.0 * sub : 2.3 * slices(32) + 8.5 + 38.0 * sub)};
    return static_cast<CirGemmForm>(std::min_element(t, t + 4) - t);
}
