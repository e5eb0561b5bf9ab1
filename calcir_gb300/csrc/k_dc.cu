// Divide-and-conquer eigensolver for the symmetric tridiagonal T = Q^T H Q left by the
// tridiagonalisation (the method magma_ssyevd uses, calcIR.cu:420-448: LAPACK stedc /
// laed0-laed4 in FP32), batched over matrices and run level by level:
//
//   * The index range [0, n) is halved recursively to a uniform depth D (block b of level
//     l is [b n >> l, (b+1) n >> l)), leaves of at most DC_LEAF rows.  At every internal
//     boundary m the coupling beta = e[m-1] is torn out (Cuppen): d[m-1] and d[m] lose |beta|
//     and the merge that joins the two sides adds back rho u u^T, rho = |beta|,
//     u = e_{m-1} + sign(beta) e_m.
//   * k_dc_leaf: one warp per leaf solves its block by implicit QR (Wilkinson shift), every
//     lane applying the rotations to its row of the leaf's eigenvector block, and writes the
//     eigenvalues ascending with their vectors.
//   * k_dc_merge (a block or a cluster per merge): z = (last row of Q1, sign(beta) first row of Q2)/sqrt2,
//     rho = 2|beta|; the two sorted eigenvalue lists are merged; small components of z and
//     close pairs are deflated (close pairs by a Givens rotation, LAPACK laed2 rules with
//     tol = 8 eps max(|D|, |z|)); the secular equation 1/rho + sum z_j^2/(D_j - lambda) = 0
//     is solved for each root by a safeguarded rational (Gragg "middle way") iteration on
//     tau = lambda - D_origin, origin the nearer pole, so D_j - lambda is formed as
//     (D_j - D_origin) - tau without cancellation; z is recomputed from the roots
//     (Gu-Eisenstat), which keeps the vectors orthogonal; the block's K x K rotation
//     U = P G W (merge permutation, deflation rotations, secular vectors) is written
//     row-major, and the eigenvalues ascending.
//   * k_dc_gemm: Q_new = diag(Q1, Q2) U for every merge, as two products of the diagonal
//     blocks with the matching rows of U (64 x 64 tiles, FP32).
// The eigenvectors of H are then V = Q_H Q_T, the reflectors of the tridiagonalisation
// applied to Q_T in compact WY blocks (k_backtransform.cu): FP32 GEMMs in the plain form,
// the tensor-core GEMM (a.precision) in the mixed forms.
#include "cir_device.cuh"
#include "cir_tcgen05.cuh"

#include <cstdlib>
#include <float.h>

namespace {

constexpr int DC_LEAF = 32;
constexpr float DC_EPS = 5.9604645e-8f;   // 2^-24

__host__ __device__ inline int dc_off(int level, int b, int n) { return (int)(((long long)b * n) >> level); }

// ---------------------------------------------------------------------------------------
// Leaves: warp w of the block handles leaf blockIdx.x * 4 + w of matrix blockIdx.y.  The chain
// of a sweep's rotations bounds it: d and e stay in registers, an entry a lane, those a
// rotation meets are fetched one rotation ahead, its (c, s) come from one refined reciprocal
// square root, and the sweep's range from a ballot.  One matrix of order 128: 256 us with a square root,
// two divisions and a round trip through shared memory a rotation and the range searched entry by
// entry, 88 so; 200 of order 1024: 763, 387.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_dc_leaf(EighArgs a, int depth, float *Qout) {
    __shared__ float Zs[4][32][DC_LEAF + 1];
    __shared__ float dS[4][32];
    __shared__ int rk[4][32];
    const int n = a.n, ld = a.ld;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int leaf = blockIdx.x * 4 + warp;
    if (leaf >= (1 << depth)) return;
    const int m = blockIdx.y;
    float *dw = a.DE + (size_t)m * 3 * ld;          // d in, eigenvalues out
    const float *ev = dw + ld;                      // e
    float *Q = Qout + (size_t)m * a.mstride;
    const int a0 = dc_off(depth, leaf, n), a1 = dc_off(depth, leaf + 1, n);
    const int s = a1 - a0;
    float *d = dS[warp];
    float(*Z)[DC_LEAF + 1] = Zs[warp];
    float dl = 0.f, el = 0.f;                       // lane i: d[i], e[i]
    if (lane < s) {
        dl = dw[a0 + lane];
        if (lane == 0 && a0 > 0) dl -= fabsf(ev[a0 - 1]);
        if (lane == s - 1 && a1 < n) dl -= fabsf(ev[a1 - 1]);
        el = lane < s - 1 ? ev[a0 + lane] : 0.f;
    }
    for (int c = 0; c < s; c++) Z[lane][c] = lane == c ? 1.f : 0.f;
    auto at = [](float v, int i) { return __shfl_sync(0xffffffffu, v, i); };
    // implicit QR with the Wilkinson shift; every lane runs the same scalar recurrence
    float tn = fabsf(dl) + 2.f * fabsf(el);
    for (int o = 16; o > 0; o >>= 1) tn = fmaxf(tn, __shfl_xor_sync(0xffffffffu, tn, o));
    const float tiny = 1e-12f * tn + FLT_MIN;
    int cm = s - 1, nsweep = 0;
    const int cap = a.test_sweep_cap > 0 ? a.test_sweep_cap : 30 * s + 30;
    while (cm > 0 && nsweep < cap) {
        // the couplings that are negligible, and the unreduced range l .. cm that ends last
        const float du = __shfl_down_sync(0xffffffffu, dl, 1);
        const bool neg = lane < s - 1 && (fabsf(el) <= DC_EPS * (fabsf(dl) + fabsf(du)) || fabsf(el) <= tiny);
        const unsigned cut = __ballot_sync(0xffffffffu, neg);
        while (cm > 0 && (cut >> (cm - 1) & 1)) cm--;
        if (cm == 0) break;
        const int l = 32 - __clz(cut & ((1u << (cm - 1)) - 1));
        const float bb = at(el, cm - 1), dm = at(dl, cm);
        const float t = 0.5f * (at(dl, cm - 1) - dm);
        const float den = t + copysignf(sqrtf(t * t + bb * bb), t);
        const float mu = dm - (den != 0.f ? bb * bb / den : 0.f);
        float dk = at(dl, l), ek = at(el, l), dn = at(dl, l + 1), en = at(el, l + 1);
        float x = dk - mu, z = ek, z0 = Z[lane][l];
        for (int k = l; k < cm; k++) {
            const float dk1 = dn, ek1 = k + 1 < cm ? en : 0.f, z1 = Z[lane][k + 1];
            dn = at(dl, k + 2);
            en = at(el, k + 2);
            const float r2 = x * x + z * z;
            float rs = rsqrtf(r2);
            rs = fmaf(rs, fmaf(-0.5f * r2 * rs, rs, 0.5f), rs);
            const bool turn = r2 > 0.f;
            const float c = turn ? x * rs : 1.f, sn = turn ? z * rs : 0.f;
            const float dd = dk - dk1;
            const float g = sn * dd - 2.f * c * ek;
            x = (c * c - sn * sn) * ek - c * sn * dd;
            if (lane == k - 1 && k > l) el = turn ? r2 * rs : 0.f;
            if (lane == k) dl = dk - sn * g;
            Z[lane][k] = c * z0 + sn * z1;
            z0 = c * z1 - sn * z0;
            dk = dk1 + sn * g;
            ek = c * ek1;
            z = sn * ek1;
        }
        if (lane == cm) dl = dk;
        if (lane == cm - 1) el = x;
        Z[lane][cm] = z0;
        nsweep++;
    }
    __syncwarp();
    if (lane < s) d[lane] = dl;
    __syncwarp();
    if (lane == 0 && nsweep >= cap && a.status) a.status[m] = 1;
    // ascending order (ties by index)
    if (lane < s) {
        int r = 0;
        for (int i = 0; i < s; i++) r += cir_before(d[i], i, d[lane], lane);
        rk[warp][lane] = r;
    }
    __syncwarp();
    if (lane < s) dw[a0 + rk[warp][lane]] = d[lane];
    for (int c = 0; c < s; c++)
        if (lane < s) Q[(size_t)(a0 + rk[warp][c]) * ld + a0 + lane] = Z[lane][c];
}

// ---------------------------------------------------------------------------------------
// Merges of one level.
// ---------------------------------------------------------------------------------------
struct DcSmem {      // offsets (floats) of the merge block's arrays for a merge of size <= KM
    int D, Ds, zs, z2, Dn, tau, zh, inv, vals, perm, kind, nidx, defl, org, src, rot, red, total;
    __host__ __device__ DcSmem(int KM) {
        int o = 0;
        D = o; o += KM;
        Ds = o; o += KM;
        zs = o; o += KM;
        z2 = o; o += KM;
        Dn = o; o += KM;
        tau = o; o += KM;
        zh = o; o += KM;
        inv = o; o += KM;
        vals = o; o += KM;
        perm = o; o += KM;     // int
        kind = o; o += KM;     // int: index among the non-deflated, or -1
        nidx = o; o += KM;     // int: sorted index of non-deflated i
        defl = o; o += KM;     // int: sorted index of deflated q
        org = o; o += KM;      // int
        src = o; o += KM;      // int: final column -> value index
        rot = o; o += 4 * KM;  // rotations (p, j as int; c, s)
        red = o; o += 64;
        total = o;
    }
};

template <int NT>
__device__ float dc_block_max(float v, float *red) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float r = 0.f;
    for (int w = 0; w < NT / 32; w++) r = fmaxf(r, red[w]);
    return r;
}

template <int NT>
__device__ float dc_block_sum(float v, float *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[32 + (threadIdx.x >> 5)] = v;
    __syncthreads();
    float r = 0.f;
    for (int w = 0; w < NT / 32; w++) r += red[32 + w];
    return r;
}

// sum over the G lanes of a root (every lane gets the same bits)
__device__ __forceinline__ float dc_lanes(float v, int G, unsigned mask) {
    for (int o = G >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
    return v;
}

// root i of 1/rho + sum_j z2_j / (Dn_j - lambda); returns the origin index, *tau = lambda - Dn[origin].
// G lanes of a warp (mask) share it, this one with the terms j = gl modulo G; ONE: G is 1 (the
// compiler unrolls the loops and reads the terms by fours).
template <bool ONE>
__device__ int dc_root(int i, int Kp, const float *Dn, const float *z2, float rho, float z2sum, int gl, int lanes,
                       unsigned mask, float *tau_out, int *iters) {
    const int G = ONE ? 1 : lanes;
    if (ONE) gl = 0;
    const float rinv = 1.f / rho;
    int o;
    float lo, hi, t;
    // the interval and a first value: the root of the two poles about it (the last two, for the
    // last root) with the other terms as they are in the middle (LAPACK laed4).  Starting in the
    // middle took 4 evaluations a root and 24 for the slowest of a merge, the last root halving its
    // way to a small z; so it takes 3, and 9.
    if (i < Kp - 1) {
        const float gap = Dn[i + 1] - Dn[i];
        const float mid = 0.5f * gap;
        const float base = Dn[i];
        float g = 0.f;
        for (int j = gl; j < Kp; j += G) g += z2[j] / ((Dn[j] - base) - mid);
        g = rinv + dc_lanes(g, G, mask);
        const float za = z2[i], zb = z2[i + 1], c = g - (zb - za) / mid;
        if (g >= 0.f) {
            o = i; lo = 0.f; hi = mid;
            const float p = fmaf(c, gap, za + zb), q = za * gap, disc = sqrtf(fabsf(p * p - 4.f * q * c));
            t = p > 0.f ? 2.f * q / (p + disc) : (p - disc) / (2.f * c);
        } else {
            o = i + 1; lo = mid - gap; hi = 0.f;
            const float p = fmaf(c, gap, -za - zb), q = zb * gap, disc = sqrtf(fabsf(p * p + 4.f * q * c));
            t = p < 0.f ? 2.f * q / (p - disc) : -(p + disc) / (2.f * c);
        }
    } else {
        o = i; lo = 0.f; hi = rho * z2sum;
        t = 0.f;
        if (Kp > 1) {
            const float base = Dn[i], mid = 0.5f * hi, gap = base - Dn[i - 1], za = z2[i - 1], zb = z2[i];
            float c = 0.f;
            for (int j = gl; j < Kp - 2; j += G) c += z2[j] / ((Dn[j] - base) - mid);
            c = rinv + dc_lanes(c, G, mask);
            const float p = fmaf(c, gap, -za - zb), q = zb * gap, disc = sqrtf(fabsf(p * p + 4.f * q * c));
            t = p > 0.f ? 2.f * q / (p + disc) : (disc - p) / (2.f * c);
        }
    }
    if (!(t > lo && t < hi)) t = 0.5f * (lo + hi);
    const float dorg = Dn[o];
    const int ip = i < Kp - 1 ? i : Kp - 2;   // poles ip, ip+1 of the local model
    int it = 0;
    for (; it < 64; it++) {
        // the poles up to ip (psi) and beyond (phi); one reciprocal per term, approximate (1 ulp),
        // well inside the 8 eps sum(|terms|) convergence bound below
        float psi = 0.f, phi = 0.f, dpsi = 0.f, dphi = 0.f;
        if (ONE) {
            for (int j = 0; j <= ip; j++) {
                const float rl = __fdividef(1.f, (Dn[j] - dorg) - t);
                const float q = z2[j] * rl;
                psi += q;
                dpsi = fmaf(q, rl, dpsi);
            }
            for (int j = ip + 1; j < Kp; j++) {
                const float rl = __fdividef(1.f, (Dn[j] - dorg) - t);
                const float q = z2[j] * rl;
                phi += q;
                dphi = fmaf(q, rl, dphi);
            }
        } else {   // one loop: the lanes' boundaries differ
            #pragma unroll 4
            for (int j = gl; j < Kp; j += G) {
                const float rl = __fdividef(1.f, (Dn[j] - dorg) - t);
                const float q = z2[j] * rl;
                if (j <= ip) { psi += q; dpsi = fmaf(q, rl, dpsi); }
                else { phi += q; dphi = fmaf(q, rl, dphi); }
            }
        }
        psi = dc_lanes(psi, G, mask);
        phi = dc_lanes(phi, G, mask);
        dpsi = dc_lanes(dpsi, G, mask);
        dphi = dc_lanes(dphi, G, mask);
        const float di = ip >= 0 ? (Dn[ip] - dorg) - t : 0.f;
        const float dj = ip + 1 < Kp ? (Dn[ip + 1] - dorg) - t : 0.f;
        const float g = rinv + psi + phi;
        const float errb = 8.f * (fabsf(psi) + fabsf(phi)) + 2.f * rinv;
        if (fabsf(g) <= DC_EPS * errb) break;
        if (g < 0.f) lo = t;
        else hi = t;
        float eta;
        if (Kp == 1) {
            eta = -g / (dpsi + dphi);
        } else {
            const float C = g - di * dpsi - dj * dphi;
            const float A = (di + dj) * g - di * dj * (dpsi + dphi);
            const float B = di * dj * g;
            const float disc = sqrtf(fabsf(A * A - 4.f * B * C));
            if (C == 0.f) eta = A != 0.f ? B / A : -g / (dpsi + dphi);
            else if (A <= 0.f) eta = (A - disc) / (2.f * C);
            else eta = 2.f * B / (A + disc);
            if (g * eta >= 0.f) eta = -g / (dpsi + dphi);
        }
        float tn = t + eta;
        if (!(tn > lo && tn < hi)) tn = 0.5f * (lo + hi);
        const bool done = tn == t || hi - lo <= DC_EPS * fmaxf(fabsf(lo), fabsf(hi));
        t = tn;
        if (done) break;
    }
    *tau_out = t;
    *iters = it + 1;
    return o;
}

// positions of the i < K with pred(i), in order: emit(i, position, pred); returns their number
template <int NT, class P, class E>
__device__ __forceinline__ int dc_compact(int K, int *wsum, P pred, E emit) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int base = 0;
    for (int i0 = 0; i0 < K; i0 += NT) {
        const int i = i0 + threadIdx.x;
        const bool p = i < K && pred(i);
        const unsigned m = __ballot_sync(0xffffffffu, p);
        if (lane == 0) wsum[warp] = __popc(m);
        __syncthreads();
        int off = base;
        for (int w = 0; w < NT / 32; w++) {
            if (w < warp) off += wsum[w];
            base += wsum[w];
        }
        if (i < K) emit(i, off + __popc(m & ((1u << lane) - 1)), p);
        __syncthreads();
    }
    return base;
}

// One merge per block, or per cluster of C blocks (CL): every block forms the sorted lists and
// deflates them for itself; the roots, the recomputed z, the norms, the ranks and the columns of U
// are dealt to all threads of the cluster, G lanes to a root where there are more threads than
// roots, and pushed to every block.  The roots' terms bound the large merges of many matrices
// (and 200 blocks on 152 SMs leave a second wave of 48), the serial chain (the deflation's scan, a
// root's terms on one lane) those of few.  The scan is parallel but for the pairs that deflate.
// Measured with a lane a root from the middle of its interval, one block a merge and a serial scan,
// and so (us): the top three levels of one matrix of order 1024 2075, 336; one merge of 128 73, 31;
// 200 merges of 1024 1723, 1298; 1600 of 128 308, 219.
template <int NT, bool CL, bool ONE>
__global__ void __launch_bounds__(NT) k_dc_merge(EighArgs a, int level, int KM, const float *Qin, float *Uout) {
    extern __shared__ __align__(16) float sm[];
    const DcSmem L(KM);
    float *D = sm + L.D, *Ds = sm + L.Ds, *zs = sm + L.zs, *z2 = sm + L.z2, *Dn = sm + L.Dn, *tau = sm + L.tau;
    float *zh = sm + L.zh, *inv = sm + L.inv, *vals = sm + L.vals, *red = sm + L.red;
    int *perm = reinterpret_cast<int *>(sm + L.perm), *kind = reinterpret_cast<int *>(sm + L.kind);
    int *nidx = reinterpret_cast<int *>(sm + L.nidx), *defl = reinterpret_cast<int *>(sm + L.defl);
    int *org = reinterpret_cast<int *>(sm + L.org), *src = reinterpret_cast<int *>(sm + L.src);
    int *wsum = reinterpret_cast<int *>(red + 48);
    float *rot = sm + L.rot;
    __shared__ int s_m;
    const int C = CL ? (int)cl_size() : 1, rank = CL ? (int)cl_rank() : 0;
    // optional per-phase timers of the merges (EighArgs.phase_ns slots 7-11, summed over merges)
    unsigned long long *pt = a.phase_ns && rank == 0 ? a.phase_ns + (size_t)blockIdx.y * CIR_EIG_PROF_SLOTS : nullptr;
    unsigned long long tl = 0;
    auto mark = [&](int slot) {
        if (!pt) return;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (slot >= 0) atomicAdd(pt + slot, t - tl);
            tl = t;
        }
    };
    mark(-1);
    const int n = a.n, ld = a.ld, tid = threadIdx.x;
    const int mat = blockIdx.y, b = blockIdx.x / C;
    const int NTT = NT * C, gid = rank * NT + tid;       // all threads of the merge
    auto all_sync = [&] {
        if (CL) cl_sync();
        else __syncthreads();
    };
    // a word of this block's shared memory, in every block of the cluster
    auto put = [&](float *p, float v) {
        if (!CL) { *p = v; return; }
        for (int c = 0; c < C; c++) cl_store(cl_map(p, c), v);
    };
    auto puti = [&](int *p, int v) { put(reinterpret_cast<float *>(p), __int_as_float(v)); };
    const int a0 = dc_off(level, b, n), a1 = dc_off(level, b + 1, n), mid = dc_off(level + 1, 2 * b + 1, n);
    const int K = a1 - a0, k1 = mid - a0;
    float *dw = a.DE + (size_t)mat * 3 * ld;
    const float beta = dw[ld + mid - 1];
    const float *Q = Qin + (size_t)mat * a.mstride;
    float *U = Uout + (size_t)mat * a.mstride;
    const float rho = 2.f * fabsf(beta);
    const float sgn = beta >= 0.f ? 1.f : -1.f;
    // z and the two sorted lists
    for (int i = tid; i < K; i += NT) {
        D[i] = dw[a0 + i];
        zs[i] = (i < k1 ? Q[(size_t)(a0 + i) * ld + mid - 1] : sgn * Q[(size_t)(a0 + i) * ld + mid]) * 0.70710678118654752f;
    }
    __syncthreads();
    for (int i = tid; i < K; i += NT) {
        int rnk;
        const float v = D[i];
        // (both halves ascend in the order of cir_before, NaN last, so the ranks are a permutation)
        if (i < k1) {   // number of D2 < v
            int lo = k1, hi = K;
            while (lo < hi) { const int md = (lo + hi) >> 1; if (cir_lt(D[md], v)) lo = md + 1; else hi = md; }
            rnk = i + (lo - k1);
        } else {        // number of D1 <= v
            int lo = 0, hi = k1;
            while (lo < hi) { const int md = (lo + hi) >> 1; if (cir_le(D[md], v)) lo = md + 1; else hi = md; }
            rnk = (i - k1) + lo;
        }
        perm[rnk] = i;
    }
    __syncthreads();
    float mx = 0.f;
    for (int r = tid; r < K; r += NT) {
        const int i = perm[r];
        Ds[r] = D[i];
        z2[r] = zs[i];       // z in sorted order (z2 reused below for z^2)
        mx = fmaxf(mx, fmaxf(fabsf(D[i]), fabsf(zs[i])));
    }
    const float tol = 8.f * DC_EPS * dc_block_max<NT>(mx, red);
    __syncthreads();
    for (int r = tid; r < K; r += NT) zs[r] = z2[r];
    __syncthreads();
    // Deflation (LAPACK laed2).  Small components leave first; the rest (lst, M of them) are scanned
    // for close pairs |t c s| <= tol, c = z_j / tt, s = -z_pj / tt, tt^2 = z_j^2 + z_pj^2 (multiplied
    // through by tt^2: no division unless the pair deflates).  A pair's test depends on the one
    // before it only where that one deflated, so all pairs are tested as they stand, and one thread
    // follows the chains that start at those that pass.
    int *lst = org, *hot = src;          // (both free until the roots are known)
    const int M = dc_compact<NT>(K, wsum, [&](int j) { return !(rho * fabsf(zs[j]) <= tol); }, [&](int j, int pos, bool p) {
        kind[j] = p ? 0 : -1;
        if (p) lst[pos] = j;
    });
    auto close = [&](int i) {
        const int j = lst[i], p = lst[i - 1];
        const float zj = zs[j], zp = zs[p], t = Ds[j] - Ds[p];
        return fabsf(t * zj * zp) <= tol * fmaf(zj, zj, zp * zp);
    };
    const int nhot = dc_compact<NT>(M, wsum, [&](int i) { return i > 0 && close(i); }, [&](int i, int pos, bool p) {
        if (p) hot[pos] = i;
    });
    if (tid == 0) {
        int m = 0, next = 1;             // pairs before next are done
        for (int q = 0; q < nhot; q++) {
            if (hot[q] < next) continue;
            int i = hot[q];
            for (; i < M && close(i); i++) {
                const int j = lst[i], p = lst[i - 1];
                const float tt = hypotf(zs[j], zs[p]);
                const float c = zs[j] / tt, s = -zs[p] / tt;
                zs[j] = tt;
                zs[p] = 0.f;
                reinterpret_cast<int *>(rot)[4 * m] = p;
                reinterpret_cast<int *>(rot)[4 * m + 1] = j;
                rot[4 * m + 2] = c;
                rot[4 * m + 3] = s;
                m++;
                const float t2 = Ds[p] * c * c + Ds[j] * s * s;
                Ds[j] = Ds[p] * s * s + Ds[j] * c * c;
                Ds[p] = t2;
                kind[p] = -1;
            }
            next = i + 1;
        }
        s_m = m;
    }
    __syncthreads();
    const int nrot = s_m;
    const int Kp = dc_compact<NT>(K, wsum, [&](int j) { return kind[j] == 0; }, [&](int j, int pos, bool p) {
        if (p) nidx[pos] = j;
        else defl[j - pos] = j;
        kind[j] = p ? pos : -1;
    });
    float zpart = 0.f;
    for (int i = tid; i < Kp; i += NT) {
        const int r = nidx[i];
        Dn[i] = Ds[r];
        const float zz = zs[r];
        z2[i] = zz * zz;
        zh[i] = zz;          // sign carrier until the recomputation below
        zpart += zz * zz;
    }
    const float z2sum = dc_block_sum<NT>(zpart, red);
    __syncthreads();
    mark(7);
    // secular roots, G lanes each
    int lanes = 1;
    while (!ONE && lanes < 32 && 2 * lanes * Kp <= NTT) lanes *= 2;
    const int G = ONE ? 1 : lanes, gl = ONE ? 0 : gid & (G - 1);
    const int gi = gid / G, ng = NTT / G;
    const unsigned gmask = (G == 32 ? 0xffffffffu : (1u << G) - 1) << (tid & 31 & ~(G - 1));
    if (CL) cl_sync();                   // every block has its lists: their words may be written
    int nit = 0, nroot = 0;
    for (int i = gi; i < Kp; i += ng) {
        float t;
        int itc;
        const int o = dc_root<ONE>(i, Kp, Dn, z2, rho, z2sum, gl, G, gmask, &t, &itc);
        if (gl == 0) {
            puti(org + i, o);
            put(tau + i, t);
        }
        nit += itc;
        nroot++;
    }
    if (a.phase_ns && gl == 0 && nit) {
        unsigned long long *ps = a.phase_ns + (size_t)blockIdx.y * CIR_EIG_PROF_SLOTS;
        atomicAdd(ps + 18, (unsigned long long)nit);
        atomicAdd(ps + 19, (unsigned long long)nroot);
    }
    all_sync();
    mark(8);
    // Gu-Eisenstat: zh_j^2 = -prod_i (Dn_j - lambda_i) / prod_{i != j} (Dn_j - Dn_i)
    for (int j = gi; j < Kp; j += ng) {
        const float dj = Dn[j];
        float p = gl == 0 ? (dj - Dn[org[j]]) - tau[j] : 1.f;
        for (int i = gl; i < Kp; i += G)
            if (i != j) p *= ((dj - Dn[org[i]]) - tau[i]) / (dj - Dn[i]);
        for (int o = G >> 1; o > 0; o >>= 1) p *= __shfl_xor_sync(gmask, p, o);
        if (gl == 0) put(zh + j, copysignf(sqrtf(fmaxf(-p, 0.f)), zh[j]));
    }
    all_sync();
    for (int i = gi; i < Kp; i += ng) {
        const float base = Dn[org[i]], ti = tau[i];
        float sq = 0.f;
        for (int j = gl; j < Kp; j += G) {
            const float u = __fdividef(zh[j], (Dn[j] - base) - ti);
            sq = fmaf(u, u, sq);
        }
        sq = dc_lanes(sq, G, gmask);
        if (gl == 0) put(inv + i, 1.f / sqrtf(sq));
    }
    // eigenvalues: roots then deflated values; ascending rank (ties by index)
    for (int q = tid; q < K; q += NT) vals[q] = q < Kp ? Dn[org[q]] + tau[q] : Ds[defl[q - Kp]];
    int *touched = reinterpret_cast<int *>(D);   // D is free once the two lists are merged
    const int *rotp = reinterpret_cast<const int *>(rot);
    for (int r = tid; r < K; r += NT) touched[r] = 0;
    __syncthreads();
    for (int t = tid; t < nrot; t += NT) {
        touched[rotp[4 * t]] = 1;
        touched[rotp[4 * t + 1]] = 1;
    }
    mark(9);
    for (int q = gi; q < K; q += ng) {
        const float v = vals[q];
        int r = 0;
        for (int i = gl; i < K; i += G) r += cir_before(vals[i], i, v, q);
        for (int o = G >> 1; o > 0; o >>= 1) r += __shfl_xor_sync(gmask, r, o);
        if (gl == 0) {
            puti(src + r, q);
            dw[a0 + r] = v;
        }
    }
    all_sync();
    mark(10);
    // U = P G W without an intermediate: G = G_0 G_1 ... G_{nrot-1} are the deflation
    // rotations (G_t mixes the sorted rows p_t, j_t: p' = c p - s j, j' = s p + c j), W the
    // secular vectors in the sorted basis; rows that no rotation touches take W directly.
    // The deflation scan leaves the rotations in chains: rotation t+1 continues the chain of
    // rotation t when p_{t+1} = j_t, and no other rotation touches p_t or j_t.  Applied from
    // the last to the first, rotation t therefore reads row p_t from W and row j_t from the
    // previous step's p row (or from W at the end of a chain); row j_t is then final, and
    // row p_t is carried to rotation t-1 or, at the start of a chain, written.  The values
    // and the order of the operations are those of applying every rotation to a full copy.
    // A warp takes 32 columns and every nr-th row of them.
    const int nc = (K + 31) / 32, nw = NTT / 32, nr = ONE ? 1 : max(1, nw / nc);
    for (int u = gid >> 5; u < nc * nr; u += nw) {
        const int c = 32 * (u % nc) + (tid & 31), rg = u / nc;
        if (c >= K) continue;
        const int q = src[c];
        const bool root = q < Kp;
        const float base = root ? Dn[org[q]] : 0.f, ti = root ? tau[q] : 0.f, sc = root ? inv[q] : 0.f;
        const int pd = root ? -1 : defl[q - Kp];
        auto w = [&](int r) -> float {   // W[r][c]: secular vector entry, or the deflated unit vector
            if (!root) return r == pd ? 1.f : 0.f;
            const int jn = kind[r];
            return jn >= 0 ? zh[jn] / ((Dn[jn] - base) - ti) * sc : 0.f;
        };
        float *Uc = U + (size_t)a0 * ld + a0 + c;
        for (int r = rg; r < K; r += nr)
            if (!touched[r]) Uc[(size_t)perm[r] * ld] = w(r);
        if (rg) continue;
        float carry = 0.f;
        for (int t = nrot - 1; t >= 0; t--) {
            const int p = rotp[4 * t], j = rotp[4 * t + 1];
            const float cc = rot[4 * t + 2], ss = rot[4 * t + 3];
            const float rp = w(p), rj = (t + 1 < nrot && rotp[4 * (t + 1)] == j) ? carry : w(j);
            carry = cc * rp - ss * rj;
            Uc[(size_t)perm[j] * ld] = ss * rp + cc * rj;
            if (t == 0 || rotp[4 * (t - 1) + 1] != p) Uc[(size_t)perm[p] * ld] = carry;
        }
    }
    mark(11);
}

// Q_new = diag(Q1, Q2) U for every merge of a level: blockIdx.y = matrix, blockIdx.x =
// (merge, half, tile over (rows of the half) x (K columns)).  Q column-major (ld), U row-major
// (ld), 64 x 64 tiles, 16-deep k steps, 4 x 4 outputs per thread.
__global__ void __launch_bounds__(256) k_dc_gemm(EighArgs a, int level, int tiles, const float *Qin, const float *Uin,
                                                 float *Qout) {
    __shared__ float As[16][64 + 4];
    __shared__ float Bs[16][64 + 4];
    const int n = a.n, ld = a.ld;
    const int z = blockIdx.x / tiles, half = z & 1, b = z >> 1;
    const int mat = blockIdx.y;
    const int a0 = dc_off(level, b, n), a1 = dc_off(level, b + 1, n), mid = dc_off(level + 1, 2 * b + 1, n);
    const int K = a1 - a0;
    const int h0 = half ? mid : a0, hK = half ? a1 - mid : mid - a0;   // rows/k range of this half
    const int tr = (hK + 63) / 64, tc = (K + 63) / 64;
    const int tile = blockIdx.x - z * tiles;
    if (tile >= tr * tc) return;
    const int r0 = (tile % tr) * 64, c0 = (tile / tr) * 64;
    const float *Q = Qin + (size_t)mat * a.mstride;
    const float *U = Uin + (size_t)mat * a.mstride;
    float *C = Qout + (size_t)mat * a.mstride;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < hK; k0 += 16) {
        for (int q = threadIdx.x; q < 16 * 64; q += 256) {
            const int kk = q >> 6, i = q & 63;
            const int k = k0 + kk;
            As[kk][i] = (k < hK && r0 + i < hK) ? Q[(size_t)(h0 + k) * ld + h0 + r0 + i] : 0.f;
            Bs[kk][i] = (k < hK && c0 + i < K) ? U[(size_t)(h0 + k) * ld + a0 + c0 + i] : 0.f;
        }
        __syncthreads();
        #pragma unroll
        for (int kk = 0; kk < 16; kk++) {
            float av[4], bv[4];
            #pragma unroll
            for (int i = 0; i < 4; i++) av[i] = As[kk][ty + 16 * i];
            #pragma unroll
            for (int j = 0; j < 4; j++) bv[j] = Bs[kk][tx + 16 * j];
            #pragma unroll
            for (int i = 0; i < 4; i++)
                #pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
    #pragma unroll
    for (int j = 0; j < 4; j++) {
        const int c = c0 + tx + 16 * j;
        if (c >= K) continue;
        #pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = r0 + ty + 16 * i;
            if (r < hK) C[(size_t)(a0 + c) * ld + h0 + r] = acc[i][j];
        }
    }
}

// W (ascending eigenvalues) and the IPR histograms (calcIR.cu:493-538) of V's columns.  UNIT:
// the columns are first scaled to length one.  The reflectors' and merges' rounding leaves their
// lengths off by 5e-7, and by 1e-7..5e-7 on average, which every propagation step multiplies
// into F: 40 steps at n = 200 gave correlation functions 1.5e-6..4.3e-6 off, 0.4e-6..0.8e-6 with
// unit columns.  A warp takes a column at a time; reading V bounds it, so a matrix is spread over
// FIN_ROWS columns a block (200 matrices of order 1024, with the histograms: 1.05 ms with a
// block a matrix and no scaling, 0.26 so).
constexpr int FIN_WARPS = 8, FIN_ROWS = 32;

template <bool UNIT>
__global__ void __launch_bounds__(32 * FIN_WARPS) k_dc_finish(EighArgs a) {
    const int n = a.n, ld = a.ld, mat = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float *dw = a.DE + (size_t)mat * 3 * ld;
    float *V = a.A + (size_t)mat * a.mstride;
    const int j1 = min(n, ((int)blockIdx.x + 1) * FIN_ROWS);
    for (int j = blockIdx.x * FIN_ROWS + warp; j < j1; j += FIN_WARPS) {
        if (lane == 0) a.W[(size_t)mat * a.wstride + j] = dw[j];
        if (!UNIT && !a.hist_count) continue;
        float *col = V + (size_t)j * ld;
        float c = 0.f;                                   // column *= 1 - c
        if (UNIT) {
            float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
            for (int i = 4 * lane; i < n; i += 128) {
                const float4 v = *reinterpret_cast<const float4 *>(col + i);
                s0 = fmaf(v.x, v.x, s0);
                if (i + 1 < n) s1 = fmaf(v.y, v.y, s1);
                if (i + 2 < n) s2 = fmaf(v.z, v.z, s2);
                if (i + 3 < n) s3 = fmaf(v.w, v.w, s3);
            }
            const float d = (float)(warp_sum_d((double)s0 + s1 + s2 + s3) - 1.0);
            if (fabsf(d) < 1e-3f) c = d * (0.5f - 0.375f * d);   // 1 - 1/sqrt(1 + d)
        }
        float s4 = 0.f, m4 = 0.f;
        for (int i = 4 * lane; i < n; i += 128) {
            float4 v = *reinterpret_cast<const float4 *>(col + i);
            if (UNIT) {
                v = make_float4(fmaf(v.x, -c, v.x), fmaf(v.y, -c, v.y), fmaf(v.z, -c, v.z), fmaf(v.w, -c, v.w));
                *reinterpret_cast<float4 *>(col + i) = v;
            }
            const float x = v.x * v.x, y = i + 1 < n ? v.y * v.y : 0.f;
            const float z = i + 2 < n ? v.z * v.z : 0.f, w = i + 3 < n ? v.w * v.w : 0.f;
            s4 += (x * x + y * y) + (z * z + w * w);
            if (a.nchrom_mol == 2) m4 += (x + y) * (x + y) + (z + w) * (z + w);
        }
        if (!a.hist_count) continue;
        s4 = warp_sum(s4);
        m4 = a.nchrom_mol == 2 ? warp_sum(m4) : s4;
        if (lane == 0) {
            const float wi = dw[j] + a.avef;
            const int bin = (int)roundf((wi - a.omegaStart) / (float)a.omegaStep);
            const size_t grp = a.hist_group > 0 ? (size_t)(mat / a.hist_group) : 0;
            const int wgt = a.hist_weight ? a.hist_weight[mat] : 1;   // a frame shared by origins counts for each
            if (bin >= 0 && bin < a.nomega) {
                atomicAdd(a.hist_count + grp * a.nomega + bin, (unsigned long long)wgt);
                atomicAdd(a.hist_ipr + grp * a.nomega + bin, (double)wgt * (double)(1.f / s4));
                atomicAdd(a.hist_mipr + grp * a.nomega + bin, (double)wgt * (double)(1.f / m4));
            } else {
                atomicAdd(a.out_of_range + grp, (unsigned long long)wgt);
            }
        }
    }
}

// CIR_Q_PAIR=0: the top merge writes Q_T in FP32 and the back-transform splits it (for comparison)
bool pair_q_enabled() {
    static const bool on = [] {
        const char *v = getenv("CIR_Q_PAIR");
        return !(v && v[0] == '0');
    }();
    return on;
}

// Threads nt and blocks C of a merge of up to KM rows: the block that suits many merges (a thread
// a root, small blocks so that many share an SM), widened while the merges leave threads of the
// SMs idle, up to DC_LANES lanes a root and a block of the cluster per 128 rows.
constexpr int DC_LANES = 16;
void dc_shape(long long merges, int KM, int sms, int &nt, int &C) {
    while (nt < 512 && nt < DC_LANES * KM && merges * 2 * nt <= 2048LL * sms) nt *= 2;
    while (nt == 512 && C < 8 && 256 * C <= KM && merges * 2 * nt * C <= 2048LL * sms) C *= 2;
}

int dc_depth(int n) {
    int D = 0;
    while (((n + (1 << D) - 1) >> D) > DC_LEAF) D++;
    return D;
}

}  // namespace

size_t cir_dc_bytes(int n, int ld) { return sizeof(float) * 3 * (size_t)n * ld; }

// Stage 2 of the divide-and-conquer eigensolver: everything after the tridiagonalisation
// (DE holds d, e, tau; A the reflectors).  a.DC: 3 buffers of a.mstride floats per matrix
// (Q_T ping, pong, U), laid out [buffer][matrix]; a.Z is scratch of the back-transform.
cudaError_t cir_launch_dc(const EighArgs &a, int nmat, cudaStream_t s, int *launches) {
    const int n = a.n, ld = a.ld;
    const int D = dc_depth(n);
    float *buf[3] = {a.DC, a.DC + (size_t)nmat * a.mstride, a.DC + 2 * (size_t)nmat * a.mstride};
    const int nleaf = 1 << D;
    int dev = 0, sms = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    k_dc_leaf<<<dim3((nleaf + 3) / 4, nmat), 128, 0, s>>>(a, D, buf[0]);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    int nl = 1;
    int cur = 0;
    // the split-BF16 back-transform takes Q_T as a BF16 pair: the top merge's tensor-core
    // product writes it so directly, and the back-transform skips its own split of Q_T
    const bool q_pair = a.precision == CIR_PREC_BF16X3 && (ld & 7) == 0 && n > 2 && pair_q_enabled();
    bool q_split = false;
    for (int level = D - 1; level >= 0; level--) {
        const int KM = ((n + (1 << level) - 1) >> level);
        const DcSmem L(KM);
        const size_t smem = sizeof(float) * L.total;
        const int other = cur ^ 1;
        const int base = KM <= 64 ? 64 : KM <= 128 ? 128 : KM <= 512 ? 256 : 512;
        int nt = base, C = 1;
        dc_shape((1 << level) * (long long)nmat, KM, sms, nt, C);
        auto merge = [&](auto kern) -> cudaError_t {
            cudaError_t r = cir_allow_smem(kern, smem);
            if (r != cudaSuccess) return r;
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at[1];
            cfg.gridDim = dim3((unsigned)C << level, nmat);
            cfg.blockDim = dim3(nt);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = s;
            if (C > 1) {
                at[0].id = cudaLaunchAttributeClusterDimension;
                at[0].val.clusterDim.x = C;
                at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
                cfg.attrs = at;
                cfg.numAttrs = 1;
            }
            return cudaLaunchKernelEx(&cfg, kern, a, level, KM, (const float *)buf[cur], buf[2]);
        };
        const bool one = nt * C < 2 * KM;      // a lane a root
        e = C > 1 ? (one ? merge(k_dc_merge<512, true, true>) : merge(k_dc_merge<512, true, false>))
          : nt == 64 ? merge(k_dc_merge<64, false, true>)
          : nt == 128 ? (one ? merge(k_dc_merge<128, false, true>) : merge(k_dc_merge<128, false, false>))
          : nt == 256 ? (one ? merge(k_dc_merge<256, false, true>) : merge(k_dc_merge<256, false, false>))
                      : (one ? merge(k_dc_merge<512, false, true>) : merge(k_dc_merge<512, false, false>));
        if (e != cudaSuccess) return e;
        // One batched product per merge half on the tensor cores: the mixed forms' top three levels
        // where every offset keeps 16-byte alignment, and in FP32 (three BF16 terms) every merge of
        // 256 rows or more besides that gives a launch 32 tiles (200 matrices of order 1024, top three
        // levels: 10.4 -> 2.6 ms; 320 each of 256, 432, 686, whose halves are odd, and 1024 in the
        // mixed form 7.0 -> 3.8; below, k_dc_gemm's one launch a level is faster: four merges of 512
        // rows 35 us, eight products of 8 tiles 84).
        bool tc = level <= 2 && a.precision != CIR_PREC_FP32;
        for (int b = 0; tc && b < (1 << level); b++)
            tc = (dc_off(level, b, n) & 3) == 0 && (dc_off(level + 1, 2 * b + 1, n) & 3) == 0;
        const long long tiles = (long long)((KM + 127) / 128) * ((KM + 255) / 256) * nmat;
        if (tc || (KM >= 256 && tiles >= 32)) {
            for (int b = 0; b < (1 << level); b++) {
                const int a0 = dc_off(level, b, n), a1 = dc_off(level, b + 1, n), mid = dc_off(level + 1, 2 * b + 1, n);
                for (int half = 0; half < 2; half++) {
                    const int h0 = half ? mid : a0, hK = half ? a1 - mid : mid - a0;
                    // column-major Q_new block = Q_half U_half; in the row-major view the
                    // transpose: C^T = U_half^T Q_half^T
                    GemmArgs g{};
                    g.A = buf[2] + (size_t)h0 * ld + a0;        // U rows h0.., columns a0.. (row-major)
                    g.B = buf[cur] + (size_t)h0 * ld + h0;      // Q block (column-major)
                    g.C = buf[other] + (size_t)a0 * ld + h0;
                    g.M = a1 - a0;
                    g.N = hK;
                    g.K = hK;
                    g.lda = g.ldb = g.ldc = ld;
                    g.sA = g.sB = g.sC = a.mstride;
                    g.a_colmajor = true;
                    g.epilogue = 0;
                    g.err = a.err;
                    if (tc && level == 0 && q_pair) {
                        __nv_bfloat16 *pb = reinterpret_cast<__nv_bfloat16 *>(buf[other]) + (size_t)a0 * ld + h0;
                        g.Chi = pb;
                        g.Clo = pb + a.mstride;
                    }
                    e = tc ? cir_launch_tc_gemm(g, nmat, a.precision, s, nullptr) : cir_launch_gemm(g, nmat, s, nullptr);
                    if (e != cudaSuccess) return e;
                    nl++;
                }
            }
            nl++;
            if (tc && level == 0 && q_pair) q_split = true;
        } else {
            const int tiles = ((KM / 2 + 1 + 63) / 64) * ((KM + 63) / 64);
            k_dc_gemm<<<dim3(tiles * (1 << level) * 2, nmat), 256, 0, s>>>(a, level, tiles, buf[cur], buf[2], buf[other]);
            nl += 2;
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        cur = other;
    }
    // V = Q_H Q_T into a.A: the reflectors applied to Q_T (buf[cur]) in compact WY blocks,
    // with the free ping-pong buffer as scratch
    e = cir_launch_backtransform(a, buf[cur], buf[cur ^ 1], buf[2], nmat, s, &nl, q_split);
    if (e != cudaSuccess) return e;
    // optional FP64 refinement of the eigenpairs (eigenvalues in DE row 0) before W and the
    // distributions are written
    if (a.Href) {
        e = cir_launch_refine(a.Href, a.A, a.mstride, ld, n, a.DE, 3LL * ld, nmat, a.refine_iters, a.RW,
                              a.refine_chunk, s, &nl);
        if (e != cudaSuccess) return e;
    }
    const dim3 grid((n + FIN_ROWS - 1) / FIN_ROWS, nmat);
    if (a.precision == CIR_PREC_FP32 && !a.Href) k_dc_finish<true><<<grid, 32 * FIN_WARPS, 0, s>>>(a);
    else k_dc_finish<false><<<grid, 32 * FIN_WARPS, 0, s>>>(a);
    nl += 1;
    if (launches) *launches += nl;
    return cudaGetLastError();
}
