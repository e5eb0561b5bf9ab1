// Lineshape transform: the unnormalised inverse real DFT of the zero-padded TCF with
// cuFFT's C2R convention (calcIR.cu:790-825): only X_0..X_{n/2} are read, Im X_0 (and
// Im X_{n/2} for even n) is ignored, and y_k = sum_j Z_j exp(+2 pi i j k / n) over the
// Hermitian extension Z; n = ntcfpoints + nzeros (25750 = 2 * 5^3 * 103 by default).  The
// printed rows (calcIR.cu:890-919) are written in FP32, the arithmetic is FP64.
//
// k_lineshape sums the ntcfpoints terms that are not padding directly:
//     y_j, y_{n-j} = a_0 + sum_k a_k cos(k t_j) -+ b_k sin(k t_j),  t_j = 2 pi j / n,
// a_k = 2 Re X_k, b_k = 2 Im X_k, so a thread gives two outputs of up to three spectra for one
// cosine and one sine per k, each by the three-term recurrence (one FMA), restarted from
// sincospi every LS_SEG terms (rounding grows with the square of the terms since a restart, at
// most 64^2 eps = 5e-13 of the terms' sum; 4e-15 to 7e-15 for n 2650 to 40040, so that the FP32 rows round
// as the FFT's).  Bound by the FP64 pipe (two FMAs per SM and clock).  A whole lineshape
// call at 150 points and n = 25750: 528 -> 84 us, of which the seven launches of the FFT were
// 437 us; the twelve transforms of a job with n = 25624 = 8 * 3203 took the FFT 33 ms.
//
// Above 40 terms per unit of the sum of n's prime factors the self-sorting mixed-radix
// Stockham FFT is the shorter way, one pass per prime factor; each output of a radix-p pass is
//     out[k' + L' j'] = sum_q exp(+2 pi i q k'/L') in[(k' mod L) + L (j' + r' q)],
// L' = L p, r' = n / L'.  A term of a pass takes a sincospi (measured 1.4e-10 s per output and
// term at n = 25750, against 3.3e-12 s per output and k of the direct sum: a ratio of 42).
#include "cir_device.cuh"
#include <vector>

namespace {

constexpr int LS_SEG = 64;             // terms between restarts of the recurrence
constexpr int LS_TILE = 4 * LS_SEG;    // terms staged in shared memory
constexpr int LS_J = 64;               // output pairs of a block

// Row of the printed lineshape for output i, both parts of the selection (an output near n/2
// can appear in both).
__device__ __forceinline__ void ls_store(float *out, const LsRows &r, int i, double y) {
    const float v = (float)y / r.norm;
    if (i >= r.i0 && i < r.i0 + r.cnt1) out[i - r.i0] = v;
    if (i < r.cnt2) out[r.cnt1 + i] = v;
}

// Spectra Q*blockIdx.y .. of X [nq][K]; threadIdx.y shares the terms of an output pair.
template <int Q>
__global__ void __launch_bounds__(LS_J * 4) k_lineshape(const double2 *X, int nq, int K, LsRows r, float *out) {
    __shared__ double2 xs[Q][LS_TILE];
    __shared__ double part[3][2 * Q][LS_J];
    const int n = r.n, NC = blockDim.y, c = threadIdx.y, tid = c * LS_J + threadIdx.x;
    const int j = blockIdx.x * LS_J + threadIdx.x, q0 = Q * blockIdx.y;
    const int kmax = min(K - 1, n / 2);    // terms 1 .. kmax
    double C[Q], S[Q];
    #pragma unroll
    for (int q = 0; q < Q; q++) C[q] = S[q] = 0.0;
    double s1, c1;
    sincospi(2.0 * (double)j / (double)n, &s1, &c1);
    const double cc = 2.0 * c1;
    for (int t0 = 1; t0 <= kmax; t0 += LS_TILE) {
        __syncthreads();
        for (int i = tid; i < Q * LS_TILE; i += LS_J * NC) {
            const int q = i / LS_TILE, k = t0 + i % LS_TILE;
            double2 v = make_double2(0.0, 0.0);
            if (k <= kmax && q0 + q < nq) {
                v = X[(size_t)(q0 + q) * K + k];
                if (2 * k == n) v.y = 0.0;
                else v = make_double2(2.0 * v.x, 2.0 * v.y);
            }
            xs[q][i % LS_TILE] = v;
        }
        __syncthreads();
        for (int g = c; g * LS_SEG < min(LS_TILE, kmax - t0 + 1); g += NC) {
            const int k0 = t0 + g * LS_SEG, cnt = min(LS_SEG, kmax - k0 + 1);
            double s, co;
            sincospi(2.0 * (double)((long long)j * k0 % n) / (double)n, &s, &co);
            double cp = co * c1 + s * s1, sp = s * c1 - co * s1;   // of k0 - 1
            for (int i = 0; i < cnt; i++) {
                #pragma unroll
                for (int q = 0; q < Q; q++) {
                    const double2 v = xs[q][g * LS_SEG + i];
                    C[q] = fma(v.x, co, C[q]);
                    S[q] = fma(v.y, s, S[q]);
                }
                const double cn = fma(cc, co, -cp), sn = fma(cc, s, -sp);
                cp = co; co = cn;
                sp = s; s = sn;
            }
        }
    }
    if (NC > 1) {
        if (c > 0)
            #pragma unroll
            for (int q = 0; q < Q; q++) { part[c - 1][2 * q][threadIdx.x] = C[q]; part[c - 1][2 * q + 1][threadIdx.x] = S[q]; }
        __syncthreads();
        if (c > 0) return;
        for (int w = 0; w < NC - 1; w++)
            #pragma unroll
            for (int q = 0; q < Q; q++) { C[q] += part[w][2 * q][threadIdx.x]; S[q] += part[w][2 * q + 1][threadIdx.x]; }
    }
    if (j > n / 2) return;
    #pragma unroll
    for (int q = 0; q < Q; q++) {
        if (q0 + q >= nq) break;
        const double a0 = X[(size_t)(q0 + q) * K].x;
        float *o = out + (size_t)(q0 + q) * (r.cnt1 + r.cnt2);
        ls_store(o, r, j, a0 + (C[q] - S[q]));
        if (j > 0 && 2 * j != n) ls_store(o, r, n - j, a0 + (C[q] + S[q]));
    }
}

__global__ void k_hermitian(const double2 *X, int nx, int n, double2 *Z) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int src = j <= n / 2 ? j : n - j;
    double2 v = src < nx ? X[src] : make_double2(0.0, 0.0);
    if (src == 0 || (2 * src == n)) v.y = 0;
    if (j > n / 2) v.y = -v.y;
    Z[j] = v;
}

__global__ void k_stockham(const double2 *in, double2 *out, int n, int L, int p) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n) return;
    const int Lp = L * p, rp = n / Lp;
    const int kp = idx % Lp, jp = idx / Lp, k = kp % L;
    double re = 0, im = 0;
    for (int q = 0; q < p; q++) {
        const long long ph = ((long long)q * kp) % Lp;
        double s, c;
        sincospi(2.0 * (double)ph / (double)Lp, &s, &c);
        const double2 v = in[k + (size_t)L * (jp + (size_t)rp * q)];
        re += c * v.x - s * v.y;
        im += c * v.y + s * v.x;
    }
    out[idx] = make_double2(re, im);
}

__global__ void k_rows(const double2 *z, LsRows r, float *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < r.n) ls_store(out, r, i, z[i].x);
}

// dL/dy of L = sum (row - target)^2 for two spectra, and L; one block, sums in a fixed order.
__global__ void __launch_bounds__(1024) k_ls_residual(const float *rows, const float *target, int nls, float norm,
                                                      double *dy, double *loss) {
    __shared__ double red[32];
    double l = 0.0;
    for (int i = threadIdx.x; i < 2 * nls; i += 1024) {
        const double d = (double)rows[i] - (double)target[i];
        l += d * d;
        dy[i] = 2.0 * d / (double)norm;
    }
    l = warp_sum_d(l);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x < 32) {
        l = warp_sum_d(red[threadIdx.x]);
        if (threadIdx.x == 0) *loss = l;
    }
}

// dL/dX_k of two spectra, y_i = Re X_0 + 2 sum_k Re(X_k e^{2 pi i ik/n}): block k sums
// dy_i e^{2 pi i ik/n} over the rows, each thread a stride of rows by one rotation a step.
constexpr int LA_NT = 256;
__global__ void __launch_bounds__(LA_NT) k_ls_adjoint(const double *dy, LsRows r, int K, double *g) {
    __shared__ double red[4][LA_NT / 32];
    const int k = blockIdx.x, n = r.n, nls = r.cnt1 + r.cnt2, tid = threadIdx.x;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    double ss, sc;
    sincospi(2.0 * (double)((long long)k * LA_NT % n) / (double)n, &ss, &sc);
    for (int half = 0; half < 2; half++) {
        const int r0 = half ? r.cnt1 : 0, r1 = half ? nls : r.cnt1, base = half ? 0 : r.i0;
        double s, c;
        sincospi(2.0 * (double)((long long)k * (base + tid) % n) / (double)n, &s, &c);
        for (int i = r0 + tid; i < r1; i += LA_NT) {
            const double d0 = dy[i], d1 = dy[nls + i];
            acc[0] = fma(d0, c, acc[0]);
            acc[1] = fma(d0, s, acc[1]);
            acc[2] = fma(d1, c, acc[2]);
            acc[3] = fma(d1, s, acc[3]);
            const double cn = c * sc - s * ss;
            s = s * sc + c * ss;
            c = cn;
        }
    }
    #pragma unroll
    for (int q = 0; q < 4; q++) {
        acc[q] = warp_sum_d(acc[q]);
        if ((tid & 31) == 0) red[q][tid >> 5] = acc[q];
    }
    __syncthreads();
    if (tid < 4) {
        double t = 0.0;
        for (int w = 0; w < LA_NT / 32; w++) t += red[tid][w];
        // re and im of spectrum tid / 2; X_0 counts once and its imaginary part not at all
        const double f = tid & 1 ? (k ? -2.0 : 0.0) : (k ? 2.0 : 1.0);
        g[((size_t)(tid >> 1) * K + k) * 2 + (tid & 1)] = f * t;
    }
}

std::vector<int> prime_factors(int n) {
    std::vector<int> fac;
    for (int p = 2; (long long)p * p <= n; p++)
        while (n % p == 0) { fac.push_back(p); n /= p; }
    if (n > 1) fac.push_back(n);
    return fac;
}

}  // namespace

size_t cir_lineshape_work_bytes(int K, int n) {
    int sum = 0;
    for (int p : prime_factors(n)) sum += p;
    const int kmax = K - 1 < n / 2 ? K - 1 : n / 2;
    return (long long)kmax <= 40LL * sum ? 0 : (size_t)2 * n * sizeof(double2);
}

cudaError_t cir_launch_lineshape(const double *X, int nq, int K, const LsRows &r, void *work, float *out,
                                 cudaStream_t s, int *launches) {
    const int n = r.n;
    const double2 *x = reinterpret_cast<const double2 *>(X);
    if (r.cnt1 + r.cnt2 < 1) return cudaSuccess;
    if (!work) {
        const int jb = (n / 2 + LS_J) / LS_J;
        // three spectra a thread share the cosines (a job's IR, VV and VH); an output's terms are
        // shared by four threads while that fills the SMs (one group of spectra: 202 blocks)
        const int Q = nq % 3 == 0 ? 3 : 1;
        const dim3 grid(jb, nq / Q), blk(LS_J, nq <= 3 && K > LS_SEG ? 4 : 1);
        if (Q == 3) k_lineshape<3><<<grid, blk, 0, s>>>(x, nq, K, r, out);
        else k_lineshape<1><<<grid, blk, 0, s>>>(x, nq, K, r, out);
        if (launches) *launches += 1;
        return cudaGetLastError();
    }
    const std::vector<int> fac = prime_factors(n);
    const int T = 256, G = (n + T - 1) / T;
    for (int q = 0; q < nq; q++) {
        double2 *a = static_cast<double2 *>(work), *b = a + n;
        k_hermitian<<<G, T, 0, s>>>(x + (size_t)q * K, K, n, a);
        int L = 1;
        for (int p : fac) {
            k_stockham<<<G, T, 0, s>>>(a, b, n, L, p);
            double2 *t = a; a = b; b = t;
            L *= p;
        }
        k_rows<<<G, T, 0, s>>>(a, r, out + (size_t)q * (r.cnt1 + r.cnt2));
        if (launches) *launches += (int)fac.size() + 2;
    }
    return cudaGetLastError();
}

cudaError_t cir_launch_ls_adjoint(const float *rows, const float *target, int K, const LsRows &r, double *dy,
                                  double *loss, double *g, cudaStream_t s, int *launches) {
    k_ls_residual<<<1, 1024, 0, s>>>(rows, target, r.cnt1 + r.cnt2, r.norm, dy, loss);
    k_ls_adjoint<<<K, LA_NT, 0, s>>>(dy, r, K, g);
    if (launches) *launches += 2;
    return cudaGetLastError();
}
