// Kernels of the differentiation form: the gradient of a spectrum-mismatch loss with respect
// to the 13 map and coupling coefficients (calcIR.cu:1207-1242) by the adjoint of the
// propagation and of the eigendecomposition.
//
// Only F m_c(0) enters the correlation functions (calcIR.cu:628-745), so the forward state
// is psi_c(k) = F(k) m_c(0) for the nine vectors c (dipole x, y, z; polarisability xx .. zx),
// stored per origin as an n x 18 row-major array of (re, im) pairs and propagated with the
// two products of F's step (U_k = V_k exp(i L_k dt/hbar) V_k^T).  The adjoint lambda_c obeys
// lambda_c(k) = w_c(k) + U_{k+1} lambda_c(k+1) (U is complex symmetric), w_c(k) being the
// coefficient vector of psi_c(k) in dL.  The gradient with respect to H_k is
// G_k = V_k R_k V_k^T, R_k = Re(Phi o sum_c (V_k^T lambda_c(k)) (V_k^T psi_c(k-1))^T), where
// Phi_mn = i tau exp(i tau (l_m + l_n)/2) sinc(tau (l_m - l_n)/2) is the divided difference of
// exp(i tau l) (Daleckii-Krein), exact and finite for equal eigenvalues.  V_k^T psi(k-1) and
// V_k^T lambda(k) are the half-way points of the two recursions and are kept from them; all steps'
// R, G and contractions are then independent and share their launches.  k_dtheta contracts
// G_k and dL/dm(k) with the derivatives of the maps.
#include "cir_device.cuh"

#include <algorithm>

namespace {

constexpr int PSI_LD = CIR_PSI_LD;   // 9 complex columns

__device__ __forceinline__ double dblock_sum(double v, double *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double r = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) r += red[w];
    return r;
}

// psi(0) = m(0): grid (ceil(n/256), S)
__global__ void k_psi_init(const float *M, long long sM, int ld, int n, float *psi) {
    const int s = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *m = M + (size_t)s * sM;
    float *p = psi + ((size_t)s * n + i) * PSI_LD;
    #pragma unroll
    for (int c = 0; c < 9; c++) {
        p[2 * c] = m[(size_t)c * ld + i];
        p[2 * c + 1] = 0.f;
    }
}

// IR, VV, VH of every origin (blockIdx.x) and step (blockIdx.y) from psi(k) and m(k) (the terms
// of calcIR.cu:628-745 with psi_a = F m_a(0)): out[s*sout + 6 k + 0..5] = (re, im) of each.
__global__ void __launch_bounds__(256) k_tcf_psi(const float *psi, const float *M, long long sM, int ld, int n,
                                                 double *out, long long sout) {
    __shared__ double red[8];
    const int s = blockIdx.x, k = blockIdx.y;
    const float *m = M + (size_t)s * sM + (size_t)k * 9 * ld;
    const float *p = psi + ((size_t)k * gridDim.x + s) * n * PSI_LD;
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};   // ir, ii, jj, ij (re, im)
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        float mv[9], pr[9], pi[9];
        #pragma unroll
        for (int c = 0; c < 9; c++) {
            mv[c] = m[(size_t)c * ld + i];
            pr[c] = p[(size_t)i * PSI_LD + 2 * c];
            pi[c] = p[(size_t)i * PSI_LD + 2 * c + 1];
        }
        // term(a, b) = m_b . psi_a
        acc[0] += (double)(mv[0] * pr[0] + mv[1] * pr[1] + mv[2] * pr[2]);
        acc[1] += (double)(mv[0] * pi[0] + mv[1] * pi[1] + mv[2] * pi[2]);
        acc[2] += (double)(mv[3] * pr[3] + mv[4] * pr[4] + mv[5] * pr[5]);
        acc[3] += (double)(mv[3] * pi[3] + mv[4] * pi[4] + mv[5] * pi[5]);
        acc[4] += (double)(mv[4] * pr[3] + mv[5] * pr[3] + mv[3] * pr[4] + mv[5] * pr[4] + mv[3] * pr[5] + mv[4] * pr[5]);
        acc[5] += (double)(mv[4] * pi[3] + mv[5] * pi[3] + mv[3] * pi[4] + mv[5] * pi[4] + mv[3] * pi[5] + mv[4] * pi[5]);
        acc[6] += (double)(mv[6] * pr[6] + mv[7] * pr[7] + mv[8] * pr[8]);
        acc[7] += (double)(mv[6] * pi[6] + mv[7] * pi[7] + mv[8] * pi[8]);
    }
    double v[8];
    for (int q = 0; q < 8; q++) v[q] = dblock_sum(acc[q], red);
    if (threadIdx.x == 0) {
        double *o = out + (size_t)s * sout + 6 * k;
        o[0] = v[0];
        o[1] = v[1];
        o[2] = (3 * v[2] + v[4] + 4 * v[6]) / 15.0;
        o[3] = (3 * v[3] + v[5] + 4 * v[7]) / 15.0;
        o[4] = (2 * v[2] - v[4] + 6 * v[6]) / 30.0;
        o[5] = (2 * v[3] - v[5] + 6 * v[7]) / 30.0;
    }
}

// component c of w(k) at one chromophore: conj(g_ir) m_c (c < 3), conj(g_vv) (2 m_c + m3 + m4 +
// m5)/15 (c = 3..5), conj(g_vv) 4 m_c/15 (c = 6..8); m at this chromophore, stride ld
__device__ __forceinline__ float2 lambda_src(const PsiSource &q, const float *m, int ld, int c) {
    const float mc = m[(size_t)c * ld];
    const float v = c < 3 ? mc : c < 6 ? (2.f * mc + (m[3LL * ld] + m[4LL * ld] + m[5LL * ld])) / 15.f : 4.f * mc / 15.f;
    return c < 3 ? make_float2(q.gir_r * v, -q.gir_i * v) : make_float2(q.gvv_r * v, -q.gvv_i * v);
}

// lambda = w(k)
__global__ void k_lambda_init(float *lam, PsiSource q, int ld, int n) {
    const int s = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2 *l = reinterpret_cast<float2 *>(lam + ((size_t)s * n + i) * PSI_LD);
    for (int c = 0; c < 9; c++) l[c] = lambda_src(q, q.M + (size_t)s * q.sM + i, ld, c);
}

// The symmetric part of R, which is all that G = V R V^T needs (H is symmetric):
//   R[m][n'] = Re(Phi_mn' sum_c (a[m][c] b[n'][c] + a[n'][c] b[m][c]) / 2),
// a = V^T lambda, b = V^T psi(k-1) (n x 18 each; matrix z at z * sab), Phi from the eigenvalues
// l of the step's frame (W + z * sW).  A block computes one 32 x 32 tile at or above the diagonal
// and writes it twice; the sines bound it, so each pair is evaluated once.
__global__ void __launch_bounds__(256) k_build_R(const float *a, const float *b, long long sab, const float *W, long long sW,
                                                 int n, float tau, float *R, int ldr, long long sR) {
    if (blockIdx.x < blockIdx.y) return;
    __shared__ float am[32][PSI_LD + 1], bm[32][PSI_LD + 1], an[32][PSI_LD + 1], bn[32][PSI_LD + 1];
    __shared__ float tr[32][33], la[32], lb[32];
    const int z = blockIdx.z;
    const int m0 = blockIdx.y * 32, n0 = blockIdx.x * 32;
    const float *A = a + (size_t)z * sab, *B = b + (size_t)z * sab, *w = W + (size_t)z * sW;
    for (int q = threadIdx.x; q < 32 * PSI_LD; q += blockDim.x) {
        const int r = q / PSI_LD, c = q % PSI_LD;
        am[r][c] = m0 + r < n ? A[(size_t)(m0 + r) * PSI_LD + c] : 0.f;
        bm[r][c] = m0 + r < n ? B[(size_t)(m0 + r) * PSI_LD + c] : 0.f;
        an[r][c] = n0 + r < n ? A[(size_t)(n0 + r) * PSI_LD + c] : 0.f;
        bn[r][c] = n0 + r < n ? B[(size_t)(n0 + r) * PSI_LD + c] : 0.f;
    }
    if (threadIdx.x < 32) {
        la[threadIdx.x] = m0 + (int)threadIdx.x < n ? w[m0 + threadIdx.x] : 0.f;
        lb[threadIdx.x] = n0 + (int)threadIdx.x < n ? w[n0 + threadIdx.x] : 0.f;
    }
    __syncthreads();
    float *Rz = R + (size_t)z * sR;
    const int c = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < 32; r += 8) {
        float sr = 0.f, si = 0.f;
        #pragma unroll
        for (int k = 0; k < 9; k++) {
            const float ar = am[r][2 * k], ai = am[r][2 * k + 1], br = bn[c][2 * k], bi = bn[c][2 * k + 1];
            const float cr = an[c][2 * k], ci = an[c][2 * k + 1], dr = bm[r][2 * k], di = bm[r][2 * k + 1];
            sr += (ar * br - ai * bi) + (cr * dr - ci * di);
            si += (ar * bi + ai * br) + (cr * di + ci * dr);
        }
        const float x = 0.5f * tau * (la[r] - lb[c]);
        const float sinc = fabsf(x) < 1e-3f ? 1.f - x * x * (1.f / 6.f) : sinf(x) / x;
        float sp, cp;
        sincosf(0.5f * tau * (la[r] + lb[c]), &sp, &cp);
        // Phi = i tau (cp + i sp) sinc = tau sinc (-sp + i cp); Re(Phi S) = tau sinc (-sp sr - cp si)
        const float v = 0.5f * tau * sinc * (-sp * sr - cp * si);
        tr[r][c] = v;
        if (m0 + r < n && n0 + c < n) Rz[(size_t)(m0 + r) * ldr + n0 + c] = v;
    }
    if (m0 == n0) return;
    __syncthreads();
    for (int r = threadIdx.x >> 5; r < 32; r += 8)
        if (n0 + r < n && m0 + c < n) Rz[(size_t)(n0 + r) * ldr + m0 + c] = tr[c][r];
}

// The geometric factor of the transition dipole coupling between chromophore i (position t,
// direction u) and chromophore o (position and direction) of a frame (calcIR.cu:1352-1399 without
// the x and mu' factors); rb = 1 / b.  QUICK takes the nearest image from products with rb and
// clears ok where cir_mi3 would ask cir_mi.
template <bool QUICK>
__device__ __forceinline__ float tdc_kappa(const float3 &t, const float3 &u, const float (&o)[6], const float3 &b, const float3 &rb, bool &ok) {
    float dx = t.x - o[0], dy = t.y - o[1], dz = t.z - o[2];
    if (QUICK) ok &= cir_mi3_quick(dx, dy, dz, b.x, b.y, b.z, rb.x, rb.y, rb.z);
    else cir_mi3(dx, dy, dz, b.x, b.y, b.z, rb.x, rb.y, rb.z);
    const float ir = cir_rsqrt(dx * dx + dy * dy + dz * dz);
    const float uu = u.x * o[3] + u.y * o[4] + u.z * o[5];
    const float un = (u.x * dx + u.y * dy + u.z * dz) * ir;
    const float vn = (o[3] * dx + o[4] * dy + o[5] * dz) * ir;
    return (uu - 3.0f * un * vn) * (ir * ir * ir) * CIR_TDC;
}

// Contraction of the gradients of every origin and step with the map derivatives: blockIdx.y is
// the matrix b = s*K + k (frame table, box and G of step k of origin s; psi(k) of it).
// A warp takes 32 rows i of one matrix, DT_R at a time, its lanes the columns j: G (symmetric) is
// read once, along its rows, and the table's values of j serve DT_R pairs; lane l keeps the sums
// of row l, so that the arithmetic in double is done once for 32 rows.  For each i
//   cw = G_ii (on d omega), a_i = sum_j inter 2 G_ij kappa_ij q_j (q = mu' x),
//   the intramolecular sums, and dL/dm_b,i (the correlation terms at this step, plus
//   Re lambda_c(0) at step 0, where psi(0) = m(0) and there is no G),
// folded into coefficients on d omega, d x, d p and d mu'; the 13 products with the derivatives
// of those four maps (plus the direct intramolecular ones) are added to out[13].
// The pair arithmetic bounds it.  Four matrices of order 512 a step, 100 steps: 49.4 ms with a
// thread a row and a launch a step, 0.37 so (1.6 with the branches of the image and of the
// intramolecular pairs in the loop).
constexpr int DT_R = 4, DT_W = 4;             // rows at a time, warps
__global__ void __launch_bounds__(32 * DT_W) k_dtheta(DthetaArgs d) {
    __shared__ double tot[DT_W][13];
    const int s = blockIdx.y / d.K, k = blockIdx.y - s * d.K, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = d.n, ld = d.ld, nc = d.nchrom_mol, w0 = (blockIdx.x * DT_W + warp) * 32;
    const float *ct = d.ct + (size_t)blockIdx.y * CT_NROW * ld;
    const float *b = d.box + 3 * (size_t)blockIdx.y;
    const float3 box = make_float3(b[0], b[1], b[2]), rbox = make_float3(1.f / b[0], 1.f / b[1], 1.f / b[2]);
    const CirMaps &mp = d.maps;
    const bool pairs = k > 0 && d.ispecies != 1 && d.ispecies != 2;
    const float *G = d.G + (size_t)blockIdx.y * d.sG;
    float sa = 0.f;                                          // row w0 + lane's
    for (int i0 = w0; pairs && i0 < min(n, w0 + 32); i0 += DT_R) {
        float a[DT_R] = {};
        float3 t[DT_R], u[DT_R];
        const float *Gr[DT_R];
        int mol[DT_R];
        #pragma unroll
        for (int r = 0; r < DT_R; r++) {
            const int i = min(i0 + r, n - 1);
            t[r] = make_float3(ct[CT_TX * ld + i], ct[CT_TY * ld + i], ct[CT_TZ * ld + i]);
            u[r] = make_float3(ct[CT_UX * ld + i], ct[CT_UY * ld + i], ct[CT_UZ * ld + i]);
            Gr[r] = G + (size_t)i * d.ldg;
            mol[r] = i / nc * nc;                            // the molecule's first chromophore
        }
        for (int j = lane; j < n; j += 32) {
            const float qj = 2.f * ct[CT_MUP * ld + j] * ct[CT_X * ld + j];
            const float o[6] = {ct[CT_TX * ld + j], ct[CT_TY * ld + j], ct[CT_TZ * ld + j],
                                ct[CT_UX * ld + j], ct[CT_UY * ld + j], ct[CT_UZ * ld + j]};
            float g[DT_R], kap[DT_R];
            bool ok = true;
            #pragma unroll
            for (int r = 0; r < DT_R; r++) g[r] = Gr[r][j] * qj;
            #pragma unroll
            for (int r = 0; r < DT_R; r++) kap[r] = tdc_kappa<true>(t[r], u[r], o, box, rbox, ok);
            if (!ok)
                for (int r = 0; r < DT_R; r++) kap[r] = tdc_kappa<false>(t[r], u[r], o, box, rbox, ok);
            #pragma unroll
            for (int r = 0; r < DT_R; r++)
                a[r] += (unsigned)(j - mol[r]) >= (unsigned)nc ? g[r] * kap[r] : 0.f;
        }
        #pragma unroll
        for (int r = 0; r < DT_R; r++) {
            const float v = warp_sum(a[r]);
            if (lane == i0 - w0 + r) sa = v;
        }
    }
    double th[13] = {};
    const int i = w0 + lane;
    if (i < n) {
        const float Ei = ct[CT_E * ld + i], w = ct[CT_W * ld + i], xi = ct[CT_X * ld + i], mup = ct[CT_MUP * ld + i];
        const float ux = ct[CT_UX * ld + i], uy = ct[CT_UY * ld + i], uz = ct[CT_UZ * ld + i];
        const float cw = k > 0 ? G[(size_t)i * d.ldg + i] : 0.f;
        float sax = 0.f, sbp = 0.f, s10 = 0.f, s11 = 0.f, s12 = 0.f;   // intramolecular map (calcIR.cu:1339)
        for (int j = i / nc * nc; pairs && j < min(n, i / nc * nc + nc); j++) {
            if (j == i) continue;
            const float g = G[(size_t)i * d.ldg + j], xj = ct[CT_X * ld + j], pj = ct[CT_P * ld + j], ee = Ei + ct[CT_E * ld + j];
            sax += 2.f * g * (mp.wi[0] + mp.wi[1] * ee) * xj;
            sbp += 2.f * g * mp.wi[2] * pj;
            s10 += g * xi * xj;
            s11 += g * ee * xi * xj;
            s12 += g * ct[CT_P * ld + i] * pj;
        }
        // dL/dm_b,i: the correlation terms of this step, plus Re lambda(0) at step 0
        const int S = gridDim.y / d.K;
        const float *ps = d.psi + (((size_t)k * S + s) * n + i) * PSI_LD;
        const float gir_r = (float)d.g[4 * k], gir_i = (float)d.g[4 * k + 1];
        const float gvv_r = (float)d.g[4 * k + 2], gvv_i = (float)d.g[4 * k + 3];
        float gm[9];
        {
            float pr[9], pi[9];
            #pragma unroll
            for (int c = 0; c < 9; c++) { pr[c] = ps[2 * c]; pi[c] = ps[2 * c + 1]; }
            // Re(conj(g) v) = gr vr + gi vi
            #pragma unroll
            for (int c = 0; c < 3; c++) gm[c] = gir_r * pr[c] + gir_i * pi[c];
            const float sr = pr[3] + pr[4] + pr[5], si = pi[3] + pi[4] + pi[5];
            #pragma unroll
            for (int c = 3; c < 6; c++) gm[c] = (gvv_r * (2.f * pr[c] + sr) + gvv_i * (2.f * pi[c] + si)) / 15.f;
            #pragma unroll
            for (int c = 6; c < 9; c++) gm[c] = 4.f * (gvv_r * pr[c] + gvv_i * pi[c]) / 15.f;
            if (k == 0) {
                const float *l0 = d.lam0 + ((size_t)s * n + i) * PSI_LD;
                #pragma unroll
                for (int c = 0; c < 9; c++) gm[c] += l0[2 * c];
            }
        }
        const float sq = gm[0] * ux + gm[1] * uy + gm[2] * uz;
        const float sx = gm[3] * (4.6f * ux * ux + 1.f) + gm[4] * (4.6f * uy * uy + 1.f) + gm[5] * (4.6f * uz * uz + 1.f) +
                         gm[6] * 4.6f * ux * uy + gm[7] * 4.6f * uy * uz + gm[8] * 4.6f * uz * ux;
        // coefficients on d omega, d x, d p, d mu' (q = mu' x: dq = dmu' x + mu' dx)
        const double cx = (double)sax + sx + (double)mup * (sa + sq);
        const double cp = sbp, cm = (double)xi * (sa + sq);
        const double e1 = Ei, e2 = (double)Ei * Ei;
        const double base = cw + cx * mp.x[1] + cp * mp.p[1];   // d omega feeds omega, x and p
        th[0] = base; th[1] = base * e1; th[2] = base * e2;
        th[3] = cx; th[4] = cx * w;
        th[5] = cp; th[6] = cp * w;
        th[7] = cm; th[8] = cm * e1; th[9] = cm * e2;
        th[10] = s10; th[11] = s11; th[12] = s12;
    }
    #pragma unroll
    for (int q = 0; q < 13; q++) {
        const double v = warp_sum_d(th[q]);
        if (lane == 0) tot[warp][q] = v;
    }
    __syncthreads();
    if (threadIdx.x < 13) {
        double v = 0.0;
        for (int wv = 0; wv < DT_W; wv++) v += tot[wv][threadIdx.x];
        atomicAdd(d.out + threadIdx.x, v);
    }
}

// One propagation step of every origin's nine vectors, psi <- V e^{i L dt/hbar} V^T psi (the
// F propagation of calcIR.cu:596-617 applied to psi = F m(0)), as two passes over the step's
// eigenvectors (row j of V = eigenvector j, stride ld, a multiple of 4):
//   k_psi_rows: raw[j][.] = sum_k V[j][k] psi[k][.], X[j][.] = e^{i w_j dt/hbar} raw[j][.]
//   k_psi_cols: psi'[i][.] = sum_j V[j][i] X[j][.] (+ w_i(k), the adjoint's source)
// psi and X are n x 18 floats per origin (nine complex vectors, (re, im) pairs).
// The steps follow one another, so a step's latency counts: blocks of 16 rows (columns) and 16
// slices of the sum, one thread each, fill the SMs from few origins, and every load of V is in
// flight before the vectors are staged.  Shared-memory reads bound the sums (5 of 16 bytes for
// 18 FMAs); where a wave of blocks is full, a thread takes two rows (columns) for each of them.
// Four origins of order 512, a step: 39 us with blocks of 64 rows and 32 columns, 18 so;
// twenty of order 1024 184, 120 so.
constexpr int PSI_B = 16, PSI_G = 16;        // rows or columns (of a thread's RP), slices of the sum
constexpr int PSI_KC = 512;                  // depth staged at a time
constexpr int PSI_TWO = 4;                   // blocks an SM above which two rows a thread (four origins of order
                                             // 512, 128 blocks on 152 SMs: 18.5 / 24.6 us; twenty, 640: 45.2 / 44.4)
constexpr int PSI_SX = 20;                   // shared stride of a row of vectors: 16-byte reads
__host__ __device__ inline int psi_kc(int n) { return n < PSI_KC ? (n + 63) & ~63 : PSI_KC; }

// rows k0 .. of an n x 18 array into shared memory, zero past n
__device__ __forceinline__ void psi_stage(const float *P, int n, int k0, int kc, float *xs) {
    for (int t = threadIdx.x; t < kc * (PSI_LD / 2); t += PSI_B * PSI_G) {
        const int k = t / (PSI_LD / 2), u = t - k * (PSI_LD / 2);
        const float2 v = k0 + k < n ? *reinterpret_cast<const float2 *>(P + (size_t)(k0 + k) * PSI_LD + 2 * u)
                                    : make_float2(0.f, 0.f);
        *reinterpret_cast<float2 *>(xs + k * PSI_SX + 2 * u) = v;
    }
}
template <int RP>
__device__ __forceinline__ void psi_fma(const float (&z)[RP], const float *x, float (&acc)[RP][PSI_LD]) {
    float v[PSI_LD];
    #pragma unroll
    for (int q = 0; q < 16; q += 4) *reinterpret_cast<float4 *>(v + q) = *reinterpret_cast<const float4 *>(x + q);
    *reinterpret_cast<float2 *>(v + 16) = *reinterpret_cast<const float2 *>(x + 16);
    #pragma unroll
    for (int r = 0; r < RP; r++)
        #pragma unroll
        for (int q = 0; q < PSI_LD; q++) acc[r][q] = fmaf(z[r], v[q], acc[r][q]);
}
// the slices' sums of RP * PSI_B rows, through shared memory (a row of slices: 19 floats apart)
template <int RP>
__device__ __forceinline__ void psi_park(const float (&acc)[RP][PSI_LD], float *part) {
    const int r = threadIdx.x & (PSI_B - 1), g = threadIdx.x / PSI_B;
    #pragma unroll
    for (int u = 0; u < RP; u++)
        #pragma unroll
        for (int q = 0; q < PSI_LD; q++) part[(g * RP * PSI_B + u * PSI_B + r) * (PSI_LD + 1) + q] = acc[u][q];
}
template <int RP>
__device__ __forceinline__ float psi_total(const float *part, int r, int q) {
    float v = 0.f;
    #pragma unroll
    for (int g = 0; g < PSI_G; g++) v += part[(g * RP * PSI_B + r) * (PSI_LD + 1) + q];
    return v;
}

template <int RP>
__global__ void __launch_bounds__(PSI_B * PSI_G) k_psi_rows(const float *V, int ld, long long sV, int n, const float *w,
                                                            long long sw, float dtoh, const float *psi, float *X,
                                                            float *raw) {
    extern __shared__ __align__(16) float sm[];
    constexpr int NR = RP * PSI_B;
    const int b = blockIdx.y, j0 = blockIdx.x * NR, kcm = psi_kc(n), vld = kcm + 4;
    float *vs = sm, *xs = sm + NR * vld;
    const float *Vb = V + (size_t)b * sV, *P = psi + (size_t)b * n * PSI_LD;
    const int r = threadIdx.x & (PSI_B - 1), g = threadIdx.x / PSI_B;
    float acc[RP][PSI_LD] = {};
    for (int k0 = 0; k0 < n; k0 += kcm) {
        const int q4 = kcm / 4;
        __syncthreads();
        #pragma unroll 8
        for (int t = threadIdx.x; t < NR * q4; t += PSI_B * PSI_G) {
            const int row = t / q4, k = 4 * (t - row * q4);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j0 + row < n && k0 + k < n) {
                v = *reinterpret_cast<const float4 *>(Vb + (size_t)(j0 + row) * ld + k0 + k);
                // the row's padding past n is not part of V (0 * a non-finite pad is NaN)
                if (k0 + k + 1 >= n) v.y = 0.f;
                if (k0 + k + 2 >= n) v.z = 0.f;
                if (k0 + k + 3 >= n) v.w = 0.f;
            }
            *reinterpret_cast<float4 *>(vs + row * vld + k) = v;
        }
        psi_stage(P, n, k0, kcm, xs);
        __syncthreads();
        for (int k = 4 * g; k < kcm; k += 4 * PSI_G) {
            float4 z[RP];
            #pragma unroll
            for (int u = 0; u < RP; u++) z[u] = *reinterpret_cast<const float4 *>(vs + (u * PSI_B + r) * vld + k);
            #pragma unroll
            for (int q = 0; q < 4; q++) {
                float zq[RP];
                #pragma unroll
                for (int u = 0; u < RP; u++) zq[u] = q == 0 ? z[u].x : q == 1 ? z[u].y : q == 2 ? z[u].z : z[u].w;
                psi_fma<RP>(zq, xs + (k + q) * PSI_SX, acc);
            }
        }
    }
    __syncthreads();
    psi_park<RP>(acc, sm);
    __syncthreads();
    for (int t = threadIdx.x; t < NR * (PSI_LD / 2); t += PSI_B * PSI_G) {
        const int row = t / (PSI_LD / 2), q = 2 * (t - row * (PSI_LD / 2)), j = j0 + row;
        if (j >= n) continue;
        float re = psi_total<RP>(sm, row, q), im = psi_total<RP>(sm, row, q + 1);
        const size_t o = ((size_t)b * n + j) * PSI_LD + q;
        if (raw) *reinterpret_cast<float2 *>(raw + o) = make_float2(re, im);
        cir_rotate(cir_phase(w[(size_t)b * sw + j] * dtoh), re, im);
        *reinterpret_cast<float2 *>(X + o) = make_float2(re, im);
    }
}

template <int RP>
__global__ void __launch_bounds__(PSI_B * PSI_G) k_psi_cols(const float *V, int ld, long long sV, int n, const float *X,
                                                            float *psi, PsiSource src) {
    extern __shared__ __align__(16) float sm[];
    constexpr int NC = RP * PSI_B, U = 16 / RP;
    const int b = blockIdx.y, i0 = blockIdx.x * NC, kcm = psi_kc(n);
    const int c = threadIdx.x & (PSI_B - 1), g = threadIdx.x / PSI_B;
    const float *Vb = V + (size_t)b * sV, *Xb = X + (size_t)b * n * PSI_LD;
    float acc[RP][PSI_LD] = {};
    for (int k0 = 0; k0 < n; k0 += kcm) {
        for (int h = 0; h < kcm; h += U * PSI_G) {
            float z[U][RP];
            #pragma unroll
            for (int t = 0; t < U; t++)
                #pragma unroll
                for (int u = 0; u < RP; u++) {
                    const int j = k0 + h + t * PSI_G + g, i = i0 + u * PSI_B + c;
                    z[t][u] = h + t * PSI_G < kcm && j < n && i < n ? Vb[(size_t)j * ld + i] : 0.f;
                }
            if (h == 0) {
                __syncthreads();
                psi_stage(Xb, n, k0, kcm, sm);
                __syncthreads();
            }
            #pragma unroll
            for (int t = 0; t < U; t++)
                if (h + t * PSI_G < kcm) psi_fma<RP>(z[t], sm + (h + t * PSI_G + g) * PSI_SX, acc);
        }
    }
    __syncthreads();
    psi_park<RP>(acc, sm);
    __syncthreads();
    for (int t = threadIdx.x; t < NC * (PSI_LD / 2); t += PSI_B * PSI_G) {
        const int row = t / (PSI_LD / 2), q = t - row * (PSI_LD / 2), i = i0 + row;
        if (i >= n) continue;
        float2 v = make_float2(psi_total<RP>(sm, row, 2 * q), psi_total<RP>(sm, row, 2 * q + 1));
        if (src.M) {
            const float2 l = lambda_src(src, src.M + (size_t)b * src.sM + i, ld, q);
            v.x += l.x;
            v.y += l.y;
        }
        *reinterpret_cast<float2 *>(psi + ((size_t)b * n + i) * PSI_LD + 2 * q) = v;
    }
}

template <int RP>
cudaError_t psi_launch(const float *V, int ld, long long sV, int n, const float *w, long long sw, float dtoh,
                       const float *in, float *out, float *X, float *raw, const PsiSource &src, int S, cudaStream_t s) {
    constexpr int NR = RP * PSI_B;
    const int kcm = psi_kc(n), grid = (n + NR - 1) / NR;
    const size_t part = (size_t)PSI_G * NR * (PSI_LD + 1);
    const size_t smem_r = 4 * std::max((size_t)NR * (kcm + 4) + (size_t)kcm * PSI_SX, part);
    const size_t smem_c = 4 * std::max((size_t)kcm * PSI_SX, part);
    cudaError_t e = cir_allow_smem(k_psi_rows<RP>, smem_r);
    if (e == cudaSuccess) e = cir_allow_smem(k_psi_cols<RP>, smem_c);
    if (e != cudaSuccess) return e;
    k_psi_rows<RP><<<dim3(grid, S), PSI_B * PSI_G, smem_r, s>>>(V, ld, sV, n, w, sw, dtoh, in, X, raw);
    k_psi_cols<RP><<<dim3(grid, S), PSI_B * PSI_G, smem_c, s>>>(V, ld, sV, n, X, out, src);
    return cudaGetLastError();
}

}  // namespace

cudaError_t cir_psi_step(const float *V, int ld, long long sV, int n, const float *w, long long sw, float dt_over_hbar,
                         const float *in, float *out, float *tmp, float *raw, const PsiSource *src, int S,
                         cudaStream_t s) {
    if (n < 1 || S < 1 || S > 65535 || ld < n || (ld & 3) || (sV & 3) || (reinterpret_cast<uintptr_t>(V) & 15))
        return cudaErrorInvalidValue;
    const PsiSource q = src ? *src : PsiSource{};
    const bool two = (long long)S * ((n + PSI_B - 1) / PSI_B) > (long long)PSI_TWO * cir_sms();
    return two ? psi_launch<2>(V, ld, sV, n, w, sw, dt_over_hbar, in, out, tmp, raw, q, S, s)
               : psi_launch<1>(V, ld, sV, n, w, sw, dt_over_hbar, in, out, tmp, raw, q, S, s);
}

cudaError_t cir_adj_psi_init(const float *M, long long sM, int ld, int n, int S, float *psi, cudaStream_t s) {
    k_psi_init<<<dim3((n + 255) / 256, S), 256, 0, s>>>(M, sM, ld, n, psi);
    return cudaGetLastError();
}

cudaError_t cir_adj_tcf(const float *psi, const float *M, long long sM, int ld, int n, int S, int K, double *out,
                        long long sout, cudaStream_t s) {
    k_tcf_psi<<<dim3(S, K), 256, 0, s>>>(psi, M, sM, ld, n, out, sout);
    return cudaGetLastError();
}

cudaError_t cir_adj_lambda_init(float *lam, const PsiSource &src, int ld, int n, int S, cudaStream_t s) {
    k_lambda_init<<<dim3((n + 255) / 256, S), 256, 0, s>>>(lam, src, ld, n);
    return cudaGetLastError();
}

cudaError_t cir_adj_build_R(const float *a, const float *b, long long sab, const float *W, long long sW, int n, int batch,
                            float tau, float *R, int ldr, long long sR, cudaStream_t s) {
    const int t = (n + 31) / 32;
    k_build_R<<<dim3(t, t, batch), 256, 0, s>>>(a, b, sab, W, sW, n, tau, R, ldr, sR);
    return cudaGetLastError();
}

cudaError_t cir_adj_dtheta(const DthetaArgs &d, int S, cudaStream_t s) {
    const int rows = 32 * DT_W;
    k_dtheta<<<dim3((d.n + rows - 1) / rows, (unsigned)(S * d.K)), 32 * DT_W, 0, s>>>(d);
    return cudaGetLastError();
}
