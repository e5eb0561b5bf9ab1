// Correlation-function contraction and spectral density.
//
// k_tcf: psi_a = F m_a(0) for the 9 dipole/polarisability vectors, then the 15 unconjugated dot
// products with m_b(t) the reference evaluates as separate magma_cgemv + magma_cdotu pairs
// (calcIR.cu:628-745), combined directly into
//     IR = sum_a mu_a(t).F.mu_a(0)
//     VV = (3 iiFii + iiFjj + 4 ijFij) / 15,   VH = (2 iiFii - iiFjj + 6 ijFij) / 30.
// A warp takes R rows of F at a time, a column per lane.  The terms are linear in psi, so a
// lane contracts its own partial psi with m(t) and the sums over columns and rows meet as pairs of
// floats, in double per block.  Few rows are bound by the chain of loads and sums, many by the loads
// in flight (four rows a warp, two columns of each: more spill).  One matrix of order 128: 44 us
// with the 18 partial psi of every row reduced over the warp, 13.6 with one partial psi a lane and
// its sums in double, 5.4 so; ten of order 1024 120, 82 and 37.
// Nothing leaves the device.
//
// k_spec_mu2 / k_spec_sum: M = V^T mu (calcIR.cu:462-467) and the Lorentzian sum
// S(w_i) += sum_j |M_j|^2 g / ((w_i - l_j - avef)^2 + g^2) / pi, g = hbar/(2 T1)
// (get_spectral_density, calcIR.cu:1414-1444).
#include "cir_device.cuh"
#include "cir_tcf.cuh"

namespace {

constexpr int TCF_WARPS = 8;

// the block's sums into out
__device__ __forceinline__ void tcf_finish(Pair (&acc)[8], double *out) {
    __shared__ double part[TCF_WARPS][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double v = tcf_reduce(acc);
    if ((lane & 3) == 0) part[warp][lane >> 2] = v;
    __syncthreads();
    if (warp == 0) {
        double s = 0.0;
        if (lane < 8)
            #pragma unroll
            for (int w = 0; w < TCF_WARPS; w++) s += part[w][lane];
        tcf_add(s, out);
    }
}

// rows: the block's rows (a multiple of TCF_WARPS * R).  One row a warp reads m(0) as it needs it
// (the loads of all its columns are in flight at once), four share it in shared memory.
template <int R>
__global__ void __launch_bounds__(TCF_WARPS * 32, 2) k_tcf(TcfArgs t, int rows) {
    extern __shared__ float m0s[];   // [9][n]
    const int b = blockIdx.y;
    const float *F = t.F + (size_t)b * t.sF;
    const float *m0 = t.m0 + (size_t)b * t.sm0;
    const float *mt = t.mt + (size_t)b * t.smt;
    const int n = t.n;
    if (R > 1) {
        for (int i = threadIdx.x; i < n; i += TCF_WARPS * 32)
            #pragma unroll
            for (int a = 0; a < 9; a++) m0s[a * n + i] = m0[(size_t)a * t.ldv + i];
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Pair acc[8] = {};
    const int rend = min(n, ((int)blockIdx.x + 1) * rows);
    for (int r0 = blockIdx.x * rows + warp * R; r0 < rend; r0 += TCF_WARPS * R) {
        float pr[R][9], pi[R][9];
        const float2 *row[R];
        #pragma unroll
        for (int i = 0; i < R; i++) {
            row[i] = reinterpret_cast<const float2 *>(F + (size_t)min(r0 + i, n - 1) * t.ldf);
            #pragma unroll
            for (int a = 0; a < 9; a++) pr[i][a] = pi[i][a] = 0.f;
        }
        #pragma unroll R > 1 ? 2 : 4
        for (int q = lane; q < n; q += 32) {
            float2 f[R];
            #pragma unroll
            for (int i = 0; i < R; i++) f[i] = row[i][q];
            #pragma unroll
            for (int a = 0; a < 9; a++) {
                const float m = R > 1 ? m0s[a * n + q] : __ldg(m0 + (size_t)a * t.ldv + q);
                #pragma unroll
                for (int i = 0; i < R; i++) {
                    pr[i][a] = fmaf(f[i].x, m, pr[i][a]);
                    pi[i][a] = fmaf(f[i].y, m, pi[i][a]);
                }
            }
        }
        #pragma unroll
        for (int i = 0; i < R; i++) {
            if (r0 + i >= rend) break;
            float c[9];
            #pragma unroll
            for (int a = 0; a < 9; a++) c[a] = mt[(size_t)a * t.ldv + r0 + i];
            tcf_sums(pr[i], pi[i], c, acc);
        }
    }
    tcf_finish(acc, t.out + (size_t)b * t.sout);
}

// The same contraction with F stored transposed as a split BF16 pair (the mixed form's
// pre-split propagation): F[r][q] = Ft[(2q)*ldft + r] + i Ft[(2q+1)*ldft + r], hi + lo.
// The correlation terms are linear in psi, so each block takes 64 rows and a quarter of the
// q range and contracts its partial psi with m(t) directly.  Thread (rr, ql) = (t & 63,
// t >> 6) handles row r = 64 blockIdx.x + rr and every fourth q of the block's range.
constexpr int TT_ROWS = 64, TT_QSPLIT = 4;

__global__ void __launch_bounds__(256) k_tcf_t(TcfArgs t) {
    extern __shared__ float mq[];    // [9][qchunk]
    const int b = blockIdx.z, n = t.n;
    const int qchunk = (n + TT_QSPLIT - 1) / TT_QSPLIT;
    const int qb = blockIdx.y * qchunk, qe = min(n, qb + qchunk);
    const float *m0 = t.m0 + (size_t)b * t.sm0;
    const float *mt = t.mt + (size_t)b * t.smt;
    for (int i = threadIdx.x; i < 9 * qchunk; i += blockDim.x) {
        const int a = i / qchunk, q = qb + i % qchunk;
        mq[i] = q < n ? m0[(size_t)a * t.ldv + q] : 0.f;
    }
    __syncthreads();
    const int rr = threadIdx.x & 63, ql = threadIdx.x >> 6;
    const int r = blockIdx.x * TT_ROWS + rr;
    Pair acc[8] = {};
    if (r < n) {
        const __nv_bfloat16 *fh = t.Ft.hi + (size_t)b * t.sFt + r, *fl = t.Ft.lo + (size_t)b * t.sFt + r;
        float pr[9], pi[9], c[9];
        #pragma unroll
        for (int a = 0; a < 9; a++) pr[a] = pi[a] = 0.f;
        for (int q = qb + ql; q < qe; q += TT_QSPLIT) {
            const size_t o = (size_t)(2 * q) * t.ldft;
            const float re = __bfloat162float(fh[o]) + __bfloat162float(fl[o]);
            const float im = __bfloat162float(fh[o + t.ldft]) + __bfloat162float(fl[o + t.ldft]);
            #pragma unroll
            for (int a = 0; a < 9; a++) {
                const float m = mq[a * qchunk + (q - qb)];
                pr[a] = fmaf(re, m, pr[a]);
                pi[a] = fmaf(im, m, pi[a]);
            }
        }
        #pragma unroll
        for (int a = 0; a < 9; a++) c[a] = mt[(size_t)a * t.ldv + r];
        tcf_sums(pr, pi, c, acc);
    }
    tcf_finish(acc, t.out + (size_t)b * t.sout);
}

// |M_j|^2 of frame blockIdx.y, a warp per eigenvector
__global__ void k_spec_mu2(const float *V, int ld, long long sV, const float *dip, int ldv, long long sdip, int n,
                           float *mu2) {
    const int lane = threadIdx.x & 31;
    const int j = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (j >= n) return;
    const float *col = V + (size_t)blockIdx.y * sV + (size_t)j * ld, *d = dip + (size_t)blockIdx.y * sdip;
    float mx = 0, my = 0, mz = 0;
    for (int i = lane; i < n; i += 32) {
        const float v = col[i];
        mx = fmaf(v, d[i], mx);
        my = fmaf(v, d[ldv + i], my);
        mz = fmaf(v, d[2 * ldv + i], mz);
    }
    mx = warp_sum(mx); my = warp_sum(my); mz = warp_sum(mz);
    if (lane == 0) mu2[(size_t)blockIdx.y * n + j] = mx * mx + my * my + mz * mz;
}

// Lorentzian sums of the frames of set blockIdx.y (S consecutive frames): SP_W frequencies a
// block, the eigenvalues shared by SP_J threads each, the frames one after another, their sums
// added in double in the frames' order.  Bound by the two divisions of a term; one thread per
// frequency on 24 blocks, a launch per frame, was 102 us a frame at n = 1024.
constexpr int SP_W = 32, SP_J = 16;
__global__ void __launch_bounds__(SP_W * SP_J) k_spec_sum(const float *mu2, const float *w, long long sw, int n, int S,
                                                          double *Sw, float *Swf, int nomega, float omegaStart,
                                                          int omegaStep, float gamma, float avef) {
    __shared__ float part[SP_J][SP_W + 1];
    const int il = threadIdx.x, g = threadIdx.y, i = blockIdx.x * SP_W + il;
    const float wi = (float)(omegaStart + omegaStep * i);
    double tot = 0.0;
    for (int f = blockIdx.y * S; f < ((int)blockIdx.y + 1) * S; f++) {
        const float *m = mu2 + (size_t)f * n, *l = w + (size_t)f * sw;
        float s = 0.f;
        for (int j = g; j < n; j += SP_J) {
            const float dw = wi - (l[j] + avef);
            s += m[j] * gamma / (dw * dw + gamma * gamma) / (float)CIR_PI;
        }
        part[g][il] = s;
        __syncthreads();
        if (g == 0)
            for (int q = 0; q < SP_J; q++) tot += (double)part[q][il];
        __syncthreads();
    }
    if (g || i >= nomega) return;
    if (Swf) Swf[i] += (float)tot;
    else Sw[(size_t)blockIdx.y * nomega + i] += tot;
}

}  // namespace

cudaError_t cir_launch_tcf(const TcfArgs &t, int batch, cudaStream_t s, int *launches) {
    if (t.Ft.hi) {
        const size_t sm = sizeof(float) * 9 * (size_t)((t.n + TT_QSPLIT - 1) / TT_QSPLIT);
        cudaError_t e = cir_allow_smem(k_tcf_t, sm);
        if (e != cudaSuccess) return e;
        k_tcf_t<<<dim3((t.n + TT_ROWS - 1) / TT_ROWS, TT_QSPLIT, batch), 256, sm, s>>>(t);
        if (launches) *launches += 1;
        return cudaGetLastError();
    }
    // four rows a warp at a time share the reads of m(0) where that leaves two blocks per SM,
    // and a block takes up to 64 rows so that staging m(0) stays small beside them
    const long long all = (long long)t.n * batch, two = 2LL * cir_sms();
    const int R = all >= two * TCF_WARPS * 4 ? 4 : 1, rows = TCF_WARPS * (R == 4 && all >= two * 64 ? 8 : R);
    const size_t smem = R == 4 ? sizeof(float) * 9 * (size_t)t.n : 0;
    auto kern = R == 4 ? k_tcf<4> : k_tcf<1>;
    cudaError_t e = cir_allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    kern<<<dim3((t.n + rows - 1) / rows, batch), TCF_WARPS * 32, smem, s>>>(t, rows);
    if (launches) *launches += 1;
    return cudaGetLastError();
}

cudaError_t cir_launch_spectral(const float *V, int ld, long long sV, const float *w, long long sw, const float *dip, int ldv,
                                long long sdip, int n, int S, int sets, float *mu2, double *Sw, float *Swf, int nomega,
                                float omegaStart, int omegaStep, float t1, float avef, cudaStream_t s, int *launches) {
    k_spec_mu2<<<dim3((n + 7) / 8, S * sets), 256, 0, s>>>(V, ld, sV, dip, ldv, sdip, n, mu2);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const float gamma = (float)(CIR_HBAR / (t1 * 2.0));
    k_spec_sum<<<dim3((nomega + SP_W - 1) / SP_W, sets), dim3(SP_W, SP_J), 0, s>>>(mu2, w, sw, n, S, Sw, Swf, nomega,
                                                                                 omegaStart, omegaStep, gamma, avef);
    if (launches) *launches += 2;
    return cudaGetLastError();
}
