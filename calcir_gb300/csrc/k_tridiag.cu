// Householder tridiagonalisation Q^T H Q = T of a batch of symmetric matrices (the sytrd step
// of magma_ssyevd_gpu, calcIR.cu:420-448): LAPACK's lower storage and slarfg conventions, the
// reflectors left below the subdiagonal of A, d, e and tau in a.DE.
//
// One thread block, or one cluster of C blocks, per matrix.  Per column k, whose updated
// entries c (rows k+1..) every block holds in shared memory:
//   (1) y' = A c over the lower triangle as it stood at the start of the panel, in 32 x 32
//       tiles, each owned by one warp for good: warp (a, b) has the tile rows I = a and the
//       tile columns J = b modulo the warp grid, so the row sums of the B warp columns and
//       the column sums of the A warp rows go to A + B partial products in all, no word of
//       which two warps write; with it W^T c and V^T c of the panel's earlier columns;
//   (2) the reflector: v = scale (c - beta e), e the unit vector of row k+1, so A v = scale (y' -
//       beta A[:, k+1]): the pass over the matrix does not wait for the norm of c;
//       w = tau (A v - V t1 - W t2) - (tau/2)(w.v) v, t1 = W^T v, t2 = V^T v, where w.v =
//       tau (v.Av - 2 t1.t2) and v.Av follows from c.y' (summed tile by tile in (1)), so it
//       needs no pass and no barrier of its own; and column k + 1,
//       c = A[:, k+1] - V W[k+1,:]^T - W V[k+1,:]^T including the new pair, and its norm.
// Two block barriers a column.  The panel's V and W (NB columns) stay in shared memory.  After
// a panel the rank-2NB update A -= V W^T + W V^T is applied by the pass of the next column's
// (1): a tile is read, updated, written and multiplied.
//
// Alternate columns walk the tile columns in opposite orders, each starting on the tiles last read.
//
// Clusters (few matrices in flight, or orders above 1024): rows are dealt to the blocks in
// chunks of 32; a block sums its own tiles' y' and pushes each row to its owner and the dot
// products' partial sums to every block through distributed shared memory (one cluster
// barrier); the owner forms w and column k + 1 for its rows and pushes that column to every
// block (a second barrier).  Orders up to 256 keep the whole triangle in shared memory.
// Bound: with many matrices by the triangle's stream (152 matrices of order 1024 in flight
// hold 320 MB, so about two thirds of it come from HBM), with few by the barriers of a column.
// Measured against one block of 256 threads per matrix with per-warp partial products, the
// panel in L2 and the update as a pass of its own (ms): 608 matrices of order 1024 122 -> 76,
// 320 of order 432 8.7 -> 6.3, 320 of order 256 3.9 -> 2.0, one of order 1024 36 -> 7.1, of 2048
// 214 -> 22, of 128 0.58 -> 0.25.  Measured and not taken: tiles by TMA into a ring per warp
// (91 ms per 608: the copies of 128-byte rows run at 24 bytes a clock), tile rows unrolled with
// their sums in registers and packed FMAs (80 ms: the code no longer fits the registers).
#include "cir_device.cuh"
#include "cir_plan.h"
#include "cir_tcgen05.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

namespace {

constexpr int TQ_NB = 8;        // panel width (a multiple of 8, a lane's columns of a tile; 16 measured
                                // level: 76.3 against 75.9 ms per 608 matrices of order 1024)

__device__ __forceinline__ unsigned long long tq_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__host__ __device__ inline int tq_cluster_rows(int C) { return C >= 16 ? 4 : C >= 4 ? 2 : 1; }

struct TqSmem {      // offsets in floats
    int VS, WS, YR, X, X2, YIN, TIN, NIN, YWIN, VW, WW, T, TQ, red, tile, total;
    __host__ __device__ TqSmem(int n, int nt, bool res, int C) {
        const int n32 = (n + 31) & ~31, tn = n32 / 32, nw = nt / 32, B = 4, A = nw / B;
        const int R = 32 * ((tn + C - 1) / C);
        int o = 0;
        VS = o; o += TQ_NB * R;
        WS = o; o += TQ_NB * R;
        YR = o; o += (A + B) * n32;
        X = o; o += n32;
        X2 = YIN = TIN = NIN = YWIN = VW = WW = o;
        if (C > 1) {
            X2 = o; o += n32;
            YIN = o; o += C * R;
            TIN = o; o += C * (2 * TQ_NB + 1);
            NIN = o; o += C;
            YWIN = o; o += C * TQ_NB;
            VW = o; o += TQ_NB * TQ_NB;
            WW = o; o += TQ_NB * TQ_NB;
        }
        T = o; o += 2 * TQ_NB;
        red = o; o += 64;
        o = (o + 3) & ~3;
        TQ = o; o += 4 * TQ_NB * nw;
        o = (o + 31) & ~31;
        tile = o;
        if (res) o += 1024 * (tn * (tn + 1) / 2);
        total = o;
    }
};

// walk over the tiles (I, J), I >= J >= j0, I = wa mod At, J = wb mod Bt (powers of two),
// columns outermost, in rising or falling order
struct TqWalk {
    int I, J;
    __device__ __forceinline__ bool first(int j0, int tn, int wa, int wb, int At, int Bt, bool rev) {
        J = rev ? tn - 1 - ((tn - 1 - wb) & (Bt - 1)) : j0 + ((wb - j0) & (Bt - 1));
        return settle(j0, tn, wa, At, Bt, rev);
    }
    __device__ __forceinline__ bool settle(int j0, int tn, int wa, int At, int Bt, bool rev) {
        for (; J >= j0 && J < tn; J += rev ? -Bt : Bt) {
            I = rev ? tn - 1 - ((tn - 1 - wa) & (At - 1)) : J + ((wa - J) & (At - 1));
            if (I >= J && I < tn) return true;
        }
        return false;
    }
    __device__ __forceinline__ bool next(int j0, int tn, int wa, int At, int Bt, bool rev) {
        I += rev ? -At : At;
        if (I >= J && I < tn) return true;
        J += rev ? -Bt : Bt;
        return settle(j0, tn, wa, At, Bt, rev);
    }
};

// W32: the addresses of a tile as 32-bit offsets, half the registers and adds (152 matrices of order
// 1024 20.0 -> 19.3 ms); where the arguments come from a table it spills instead (62.2 against 60.2
// ms for four sizes of 256 to 1024, 320 each).
template <int NT, bool RES, bool CL, int D, bool W32>
__device__ __forceinline__ void tridiag(const EighArgs &a, int mat) {
    constexpr int NW = NT / 32, GB = 4, GA = NW / GB, NB = TQ_NB;
    static_assert(GA * GB == NW, "a warp per place of the warp grid");
    constexpr int RW = (CL ? 2048 : RES ? 256 : NT == 256 ? 512 : 1024) / NT;   // rows of n per thread
    constexpr int RS = CL ? 1024 / NT : RW;                                      // own rows per thread
    extern __shared__ __align__(128) float smem[];
    const int n = a.n, ld = a.ld, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n32 = (n + 31) & ~31, tn = n32 >> 5;
    const int C = CL ? (int)cl_size() : 1, rank = CL ? (int)cl_rank() : 0;
    const int R = 32 * ((tn + C - 1) / C);
    const TqSmem L(n, NT, RES, C);
    float *VS = smem + L.VS, *WS = smem + L.WS, *YR = smem + L.YR, *T = smem + L.T, *red = smem + L.red,
          *tiles = smem + L.tile;
    float4 *Tq = reinterpret_cast<float4 *>(smem + L.TQ) + NB * warp;   // this warp's (t1, t2, W[k+1], V[k+1])
    float *X = smem + L.X;
    float *A = a.A + (size_t)mat * a.mstride;
    float *Wg = a.Z + (size_t)mat * a.mstride;                              // the panel's W (clusters)
    float *dd = a.DE + (size_t)mat * 3 * ld, *ee = dd + ld, *tau = dd + 2 * ld;
    // this warp's tiles
    const int Ca = CL ? tq_cluster_rows(C) : 1, Cb = C / Ca;
    const int At = GA * Ca, Bt = GB * Cb;
    const int wa = (rank / Cb) * GA + warp / GB, wb = (rank % Cb) * GB + warp % GB;
    float *yrow = YR + (size_t)(warp % GB) * n32, *ycol = YR + (size_t)(GB + warp / GB) * n32;
    const int g = lane & 7, h = lane >> 3;

    if (a.status && tid == 0 && rank == 0) a.status[mat] = 0;
    unsigned long long *pt = a.phase_ns && rank == 0 ? a.phase_ns + (size_t)mat * CIR_EIG_PROF_SLOTS : nullptr;
    unsigned long long tlast = 0;
    if (pt && tid == 0) pt[0] = tlast = tq_ns();
    // optional phase timers (slots 12-17), read after a block-wide barrier
    auto mark = [&](int slot) {
        if (!pt) return;
        __syncthreads();
        if (tid == 0) {
            const unsigned long long t = tq_ns();
            pt[slot] += t - tlast;
            tlast = t;
        }
    };
    if (n < 3) {
        if (tid == 0 && rank == 0) {
            for (int i = 0; i < n; i++) { dd[i] = A[(size_t)i * ld + i]; tau[i] = 0.f; ee[i] = 0.f; }
            if (n == 2) ee[0] = A[1];
            if (pt) pt[1] = tq_ns();
        }
        return;
    }
    // own row l of this block's slice -> row of the matrix
    auto own_row = [&](int l) { return CL ? (((l >> 5) * C + rank) << 5) + (l & 31) : l; };

    for (int i = tid; i < L.T; i += NT) smem[i] = 0.f;   // V, W, partial products, vectors: rows >= n stay zero
    // and the panel's W in the scratch, read in whole tiles from the first update on but written only below
    // each column's reflector: what a call before left there (a NaN times the zeros of c is a NaN)
    if (CL)
        for (int i = rank * NT + tid; i < NB * ld; i += C * NT) Wg[i] = 0.f;
    if (RES) {
        for (int J = 0, q = 0; J < tn; J++)
            for (int I = J; I < tn; I++, q++) {
                if (q % NW != warp) continue;
                float *t = tiles + 1024 * q;
                for (int c = 0; c < 32; c++) {
                    const int r = 32 * I + lane, cc = 32 * J + c;
                    t[32 * c + lane] = (r < n && cc < n) ? A[(size_t)cc * ld + r] : 0.f;
                }
            }
    }
    else if (ld > n) {   // the rows of the padding may hold anything
        for (int i = tid; i < n * (ld - n); i += NT) A[(size_t)(i / (ld - n)) * ld + n + i % (ld - n)] = 0.f;
    }
    auto tile_ptr = [&](int I, int J) { return tiles + 1024 * (J * tn - J * (J - 1) / 2 + I - J); };
    __syncthreads();

    const int klast = n - 3;
    // column 0
    float part = 0.f;
    for (int r = tid; r < n; r += NT) {
        const float v = __ldcg(A + r);
        if (r == 0) { if (rank == 0) dd[0] = v; }
        else { X[r] = v; part += r == 1 ? 0.f : v * v; }
    }
    part = warp_sum(part);
    if (lane == 0) red[warp] = part;
    __syncthreads();
    if (CL) {   // every block has read the whole column: its norm as if pushed by block 0
        if (tid < C) {
            float s = 0.f;
            for (int w = 0; w < NW; w++) s += red[w];
            smem[L.NIN + tid] = tid == 0 ? s : 0.f;
        }
        cl_sync();
    }

    for (int k = 0; k <= klast; k++) {
        const int kk = k % NB, p0 = k - kk, j0 = (k + 1) >> 5;
        const bool upd = kk == 0 && k > 0;
        // the reflector (slarfg: v[0] = 1, beta = -sign(alpha) norm), by every thread
        float xn2 = 0.f;
        if (CL) xn2 = lane < C ? smem[L.NIN + lane] : 0.f;
        else xn2 = lane < NW ? red[lane] : 0.f;
        xn2 = warp_sum(xn2);
        const float alpha = X[k + 1];
        float tk = 0.f, beta = alpha, scale = 0.f;
        if (xn2 > 0.f) {
            beta = -copysignf(sqrtf(alpha * alpha + xn2), alpha);
            tk = (beta - alpha) / beta;
            scale = 1.f / (alpha - beta);
        }
        if (tid == 0 && rank == 0) { ee[k] = beta; tau[k] = tk; }
        // column k + 1 at the start of the panel: own rows, its diagonal, the panel window's rows
        float creg[RS], a11 = 0.f, awin = 0.f;
        #pragma unroll
        for (int i = 0; i < RS; i++) creg[i] = 0.f;
        auto fetch = [&] {
            const float *col = A + (size_t)(k + 1) * ld;
            #pragma unroll
            for (int i = 0; i < RS; i++) {
                const int l = tid + i * NT, r = own_row(l);
                if (l < R && r > k && r < n) creg[i] = __ldcg(col + r);
            }
            a11 = __ldcg(col + k + 1);
            if (CL && tid < NB && p0 + 1 + tid > k && p0 + 1 + tid < n) awin = __ldcg(col + p0 + 1 + tid);
        };
        if (!RES && !upd) fetch();
        mark(13);
        // (1) y' = A c (after a panel: with its update), scale c.y' (c.y' itself, a product of three factors
        // of the matrix's size, leaves FP32's range from 1e12 on), and the panel's dot products
        {
            const bool rev = (k & 1) != 0;
            float cac = 0.f, yc[8];
            #pragma unroll
            for (int t = 0; t < 8; t++) yc[t] = 0.f;
            // lane (g, h): rows 32I + 4g .. + 3 of columns 32J + 8h .. + 7
            // (rows and columns past the end are read at the last ones: the zeros of c beyond row n - 1
            // discard them, so whatever a tile can meet there has to be finite where the matrix is)
            auto load = [&](float4 (&v)[8], int I, int J) {
                if (RES) {
                    const float *t = tile_ptr(I, J) + 4 * g + 32 * 8 * h;
                    #pragma unroll
                    for (int q = 0; q < 8; q++) v[q] = *reinterpret_cast<const float4 *>(t + 32 * q);
                    return;
                }
                const int c0 = 32 * J + 8 * h;
                if (W32) {
                    const char *base = reinterpret_cast<const char *>(A);
                    const unsigned r0 = 4u * min(32 * I + 4 * g, ld - 4), row = 4u * ld;
                    if (J + 1 < tn) {
                        const unsigned o = r0 + c0 * row;
                        #pragma unroll
                        for (int q = 0; q < 8; q++) v[q] = __ldcg(reinterpret_cast<const float4 *>(base + (o + q * row)));
                    } else {
                        #pragma unroll
                        for (int q = 0; q < 8; q++) v[q] = __ldcg(reinterpret_cast<const float4 *>(base + (r0 + min(c0 + q, n - 1) * row)));
                    }
                    return;
                }
                const float *p = A + min(32 * I + 4 * g, ld - 4);
                if (J + 1 < tn) {
                    p += (size_t)c0 * ld;
                    #pragma unroll
                    for (int q = 0; q < 8; q++) v[q] = __ldcg(reinterpret_cast<const float4 *>(p + (size_t)q * ld));
                } else {
                    #pragma unroll
                    for (int q = 0; q < 8; q++) v[q] = __ldcg(reinterpret_cast<const float4 *>(p + (size_t)min(c0 + q, n - 1) * ld));
                }
            };
            auto update = [&](float4 (&v)[8], int I, int J) {
                const int r0 = 32 * I + 4 * g, c0 = 32 * J + 8 * h, o0 = p0 - NB;
                #pragma unroll 4
                for (int j = 0; j < NB; j++) {
                    float4 vr, wr, vc0, vc1, wc0, wc1;
                    if (CL) {
                        const float *vg = A + (size_t)(o0 + j) * ld, *wg = Wg + (size_t)j * ld;
                        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                        // (finished rows and columns, where V holds what the matrix does above the
                        // reflectors, stay as they are: what is multiplied by zeros must not overflow)
                        const bool ri = r0 >= p0 && r0 < n, c0i = c0 >= p0 && c0 < n, c4i = c0 >= p0 && c0 + 4 < n;
                        vr = ri ? __ldcg(reinterpret_cast<const float4 *>(vg + r0)) : z;
                        wr = ri ? __ldcg(reinterpret_cast<const float4 *>(wg + r0)) : z;
                        vc0 = c0i ? __ldcg(reinterpret_cast<const float4 *>(vg + c0)) : z;
                        vc1 = c4i ? __ldcg(reinterpret_cast<const float4 *>(vg + c0 + 4)) : z;
                        wc0 = c0i ? __ldcg(reinterpret_cast<const float4 *>(wg + c0)) : z;
                        wc1 = c4i ? __ldcg(reinterpret_cast<const float4 *>(wg + c0 + 4)) : z;
                    } else {
                        const float *vs = VS + (size_t)j * R, *ws = WS + (size_t)j * R;
                        vr = *reinterpret_cast<const float4 *>(vs + r0);
                        wr = *reinterpret_cast<const float4 *>(ws + r0);
                        vc0 = *reinterpret_cast<const float4 *>(vs + c0);
                        vc1 = *reinterpret_cast<const float4 *>(vs + c0 + 4);
                        wc0 = *reinterpret_cast<const float4 *>(ws + c0);
                        wc1 = *reinterpret_cast<const float4 *>(ws + c0 + 4);
                    }
                    const float vc[8] = {vc0.x, vc0.y, vc0.z, vc0.w, vc1.x, vc1.y, vc1.z, vc1.w};
                    const float wc[8] = {wc0.x, wc0.y, wc0.z, wc0.w, wc1.x, wc1.y, wc1.z, wc1.w};
                    #pragma unroll
                    for (int q = 0; q < 8; q++) {
                        v[q].x = fmaf(-vr.x, wc[q], fmaf(-wr.x, vc[q], v[q].x));
                        v[q].y = fmaf(-vr.y, wc[q], fmaf(-wr.y, vc[q], v[q].y));
                        v[q].z = fmaf(-vr.z, wc[q], fmaf(-wr.z, vc[q], v[q].z));
                        v[q].w = fmaf(-vr.w, wc[q], fmaf(-wr.w, vc[q], v[q].w));
                    }
                }
                if (c0 >= p0 && r0 < n) {   // finished columns keep their reflectors
                    #pragma unroll
                    for (int q = 0; q < 8; q++) {
                        if (RES) *reinterpret_cast<float4 *>(tile_ptr(I, J) + 4 * g + 32 * (8 * h + q)) = v[q];
                        else if (c0 + q < n) __stcg(reinterpret_cast<float4 *>(A + (size_t)(c0 + q) * ld + r0), v[q]);
                    }
                }
            };
            auto mult = [&](const float4 (&v)[8], int I, int J) {
                const float4 xr = *reinterpret_cast<const float4 *>(X + 32 * I + 4 * g);
                const float4 xc0 = *reinterpret_cast<const float4 *>(X + 32 * J + 8 * h);
                const float4 xc1 = *reinterpret_cast<const float4 *>(X + 32 * J + 8 * h + 4);
                const float xc[8] = {xc0.x, xc0.y, xc0.z, xc0.w, xc1.x, xc1.y, xc1.z, xc1.w};
                float yr[4] = {0.f, 0.f, 0.f, 0.f};
                if (I != J) {
                    #pragma unroll
                    for (int q = 0; q < 8; q++) {
                        yr[0] = fmaf(v[q].x, xc[q], yr[0]);
                        yr[1] = fmaf(v[q].y, xc[q], yr[1]);
                        yr[2] = fmaf(v[q].z, xc[q], yr[2]);
                        yr[3] = fmaf(v[q].w, xc[q], yr[3]);
                        yc[q] = fmaf(v[q].x, xr.x, fmaf(v[q].y, xr.y, fmaf(v[q].z, xr.z, fmaf(v[q].w, xr.w, yc[q]))));
                    }
                } else {       // r >= c in the row sums, r > c in the column sums
                    #pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const int c = 8 * h + q - 4 * g;   // column less the lane's first row
                        const float e0 = c <= 0 ? v[q].x : 0.f, e1 = c <= 1 ? v[q].y : 0.f,
                                    e2 = c <= 2 ? v[q].z : 0.f, e3 = c <= 3 ? v[q].w : 0.f;
                        yr[0] = fmaf(e0, xc[q], yr[0]);
                        yr[1] = fmaf(e1, xc[q], yr[1]);
                        yr[2] = fmaf(e2, xc[q], yr[2]);
                        yr[3] = fmaf(e3, xc[q], yr[3]);
                        yc[q] = fmaf(c < 0 ? e0 : 0.f, xr.x, fmaf(c < 1 ? e1 : 0.f, xr.y,
                                fmaf(c < 2 ? e2 : 0.f, xr.z, fmaf(c < 3 ? e3 : 0.f, xr.w, yc[q]))));
                    }
                }
                cac = fmaf(yr[0], scale * xr.x, fmaf(yr[1], scale * xr.y, fmaf(yr[2], scale * xr.z, fmaf(yr[3], scale * xr.w, cac))));
                // row sums over h (lane bits 3-4): lane (g, h) keeps row 4g + h
                #pragma unroll
                for (int i = 0; i < 2; i++) {
                    const bool up = lane & 16;
                    const float send = up ? yr[i] : yr[i + 2], keep = up ? yr[i + 2] : yr[i];
                    yr[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
                }
                const bool up = lane & 8;
                const float send = up ? yr[0] : yr[1], keep = up ? yr[1] : yr[0];
                yrow[32 * I + 4 * g + h] += keep + __shfl_xor_sync(0xffffffffu, send, 8);
            };
            auto flush = [&](int J) {   // column sums over g (lane bits 0-2): lane g keeps column 8h + g
                #pragma unroll
                for (int i = 0; i < 4; i++) {
                    const bool up = lane & 4;
                    const float send = up ? yc[i] : yc[i + 4], keep = up ? yc[i + 4] : yc[i];
                    yc[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
                }
                #pragma unroll
                for (int i = 0; i < 2; i++) {
                    const bool up = lane & 2;
                    const float send = up ? yc[i] : yc[i + 2], keep = up ? yc[i + 2] : yc[i];
                    yc[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
                }
                const bool up = lane & 1;
                const float send = up ? yc[0] : yc[1], keep = up ? yc[1] : yc[0];
                const float y = keep + __shfl_xor_sync(0xffffffffu, send, 1);
                const int c = 32 * J + 8 * h + g;
                ycol[c] += y;
                cac = fmaf(y, scale * X[c], cac);
                #pragma unroll
                for (int t = 0; t < 8; t++) yc[t] = 0.f;
            };
            TqWalk w0, w1;
            bool more = w0.first(j0, tn, wa, wb, At, Bt, rev);
            if (upd || D == 1) {
                float4 v[8];
                while (more) {
                    load(v, w0.I, w0.J);
                    if (upd) update(v, w0.I, w0.J);
                    mult(v, w0.I, w0.J);
                    w1 = w0;
                    more = w1.next(j0, tn, wa, At, Bt, rev);
                    if (!more || w1.J != w0.J) flush(w0.J);
                    w0 = w1;
                }
            } else if (more) {
                float4 va[8], vb[8];
                load(va, w0.I, w0.J);
                for (;;) {
                    w1 = w0;
                    bool m1 = w1.next(j0, tn, wa, At, Bt, rev);
                    if (m1) load(vb, w1.I, w1.J);
                    mult(va, w0.I, w0.J);
                    if (!m1 || w1.J != w0.J) flush(w0.J);
                    if (!m1) break;
                    w0 = w1;
                    m1 = w0.next(j0, tn, wa, At, Bt, rev);
                    if (m1) load(va, w0.I, w0.J);
                    mult(vb, w1.I, w1.J);
                    if (!m1 || w0.J != w1.J) flush(w1.J);
                    if (!m1) break;
                }
            }
            cac = warp_sum(cac);
            if (lane == 0) red[16 + warp] = cac;
            mark(upd ? 17 : 14);
            // W^T c, V^T c over this block's rows (rows <= k: c is zero)
            for (int q = warp; q < 2 * kk; q += NW) {
                const float *col = q < kk ? WS + (size_t)q * R : VS + (size_t)(q - kk) * R;
                float s = 0.f, s2 = 0.f;
                for (int l = 4 * lane; l < R; l += 128) {
                    const int r = own_row(l);
                    if (r + 3 > k && r < n32) {
                        const float4 p = *reinterpret_cast<const float4 *>(col + l);
                        const float4 x = *reinterpret_cast<const float4 *>(X + r);
                        s = fmaf(p.x, x.x, fmaf(p.y, x.y, s));
                        s2 = fmaf(p.z, x.z, fmaf(p.w, x.w, s2));
                    }
                }
                s = warp_sum(s + s2);
                if (lane == 0) T[q < kk ? q : NB + q - kk] = s;
            }
        }
        __syncthreads();
        mark(15);
        if (CL) {   // y' to its rows' owners, the dot products to every block
            #pragma unroll
            for (int i = 0; i < RW; i++) {
                const int r = tid + i * NT;
                if (r > k && r < n) {
                    float s = 0.f;
                    #pragma unroll
                    for (int c = 0; c < GA + GB; c++) { s += YR[(size_t)c * n32 + r]; YR[(size_t)c * n32 + r] = 0.f; }
                    const int J = r >> 5;
                    cl_store(cl_map(smem + L.YIN + rank * R + (J / C) * 32 + (r & 31), J % C), s);
                    if (r <= p0 + NB)       // the rows of the panel's own window go to every block
                        for (int c = 0; c < C; c++) cl_store(cl_map(smem + L.YWIN + rank * NB + r - p0 - 1, c), s);
                }
            }
            for (int c = warp; c < C; c += NW) {     // a warp per destination
                const float cy = warp_sum(lane < NW ? red[16 + lane] : 0.f);
                if (lane < 2 * NB) cl_store(cl_map(smem + L.TIN + rank * (2 * NB + 1) + lane, c), T[lane]);
                if (lane == 0) cl_store(cl_map(smem + L.TIN + rank * (2 * NB + 1) + 2 * NB, c), cy);
            }
            cl_sync();
        }
        mark(12);
        // (2) w and column k + 1
        if (!RES && upd) fetch();
        if (RES) a11 = tile_ptr((k + 1) >> 5, (k + 1) >> 5)[33 * ((k + 1) & 31)];
        float half, wk1;
        {
            // per warp: lane j < kk the panel's dot products and rows k+1 of V and W
            float t1 = 0.f, t2 = 0.f, v1 = 0.f, w1 = 0.f, y1 = 0.f, cy = 0.f;
            if (CL) {
                float s = 0.f;
                if (lane < 2 * NB)
                    for (int c = 0; c < C; c++) s += smem[L.TIN + c * (2 * NB + 1) + lane];
                t1 = s;
                t2 = __shfl_sync(0xffffffffu, s, (lane + NB) & 31);
                if (lane < C) cy = smem[L.TIN + lane * (2 * NB + 1) + 2 * NB];
                if (lane < C) y1 = smem[L.YWIN + lane * NB + k - p0];
            } else {
                if (lane < NB) { t1 = T[lane]; t2 = T[NB + lane]; }
                if (lane < NW) cy = red[16 + lane];
                if (lane < GA + GB) y1 = YR[(size_t)lane * n32 + k + 1];
            }
            if (lane < kk) {
                v1 = CL ? smem[L.VW + lane * NB + k - p0] : VS[(size_t)lane * R + k + 1];
                w1 = CL ? smem[L.WW + lane * NB + k - p0] : WS[(size_t)lane * R + k + 1];
            }
            t1 = lane < kk ? scale * (t1 - beta * w1) : 0.f;
            t2 = lane < kk ? scale * (t2 - beta * v1) : 0.f;
            float tt = t1 * t2, wk = v1 * t1 + w1 * t2;
            #pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                tt += __shfl_xor_sync(0xffffffffu, tt, o);
                wk += __shfl_xor_sync(0xffffffffu, wk, o);
                y1 += __shfl_xor_sync(0xffffffffu, y1, o);
                cy += __shfl_xor_sync(0xffffffffu, cy, o);
            }
            if (lane < NB) Tq[lane] = make_float4(t1, t2, w1, v1);
            const float sb = scale * beta, vay = scale * cy - sb * (2.f * scale * y1 - sb * a11);
            half = -0.5f * tk * tk * (vay - 2.f * tt);
            wk1 = tk * (scale * (y1 - beta * a11) - wk) + half;
            __syncwarp();
        }
        float *Xn = CL ? smem + ((k & 1) ? L.X : L.X2) : X;
        if (CL && tid < 2) {   // the next column's buffer: zero up to row k + 1
            if (k + tid >= 0) Xn[k + tid] = 0.f;
        }
        float part2 = 0.f;
        #pragma unroll
        for (int i = 0; i < RS; i++) {
            const int l = tid + i * NT, r = own_row(l);
            if (l >= R || r <= k || r >= n) continue;
            float s = 0.f, c;
            if (CL) {
                for (int q = 0; q < C; q++) s += smem[L.YIN + q * R + l];
            } else {
                #pragma unroll
                for (int q = 0; q < GA + GB; q++) s += YR[(size_t)q * n32 + r];
                if (r > k + 1)      // (row k + 1 is read by every warp and never again)
                    #pragma unroll
                    for (int q = 0; q < GA + GB; q++) YR[(size_t)q * n32 + r] = 0.f;
            }
            c = RES ? tile_ptr(r >> 5, (k + 1) >> 5)[32 * ((k + 1) & 31) + (r & 31)] : creg[i];
            s = scale * (s - beta * c);
            const float v = r == k + 1 ? 1.f : scale * X[r];
            #pragma unroll 4
            for (int j = 0; j < kk; j++) {
                const float4 t = Tq[j];
                const float vj = VS[(size_t)j * R + l], wj = WS[(size_t)j * R + l];
                s -= vj * t.x + wj * t.y;
                c -= vj * t.z + wj * t.w;
            }
            const float w = fmaf(tk, s, half * v);
            VS[(size_t)kk * R + l] = v;
            WS[(size_t)kk * R + l] = w;
            A[(size_t)k * ld + r] = v;
            if (CL) Wg[(size_t)kk * ld + r] = w;
            c -= v * wk1 + w;
            if (r == k + 1) {
                dd[k + 1] = c;
                if (!CL) X[r] = 0.f;
            } else {
                if (CL) for (int q = 0; q < C; q++) cl_store(cl_map(Xn + r, q), c);
                else X[r] = c;
                if (r > k + 2) part2 += c * c;
            }
        }
        if (CL && tid < NB) {   // the panel window's v and w, in every block
            const int r = p0 + 1 + tid;
            float v = 0.f, w = 0.f;
            if (r > k && r < n) {
                float s = 0.f;
                for (int q = 0; q < C; q++) s += smem[L.YWIN + q * NB + tid];
                s = scale * (s - beta * awin);
                v = r == k + 1 ? 1.f : scale * X[r];
                for (int j = 0; j < kk; j++) {
                    const float4 t = Tq[j];
                    s -= smem[L.VW + j * NB + tid] * t.x + smem[L.WW + j * NB + tid] * t.y;
                }
                w = fmaf(tk, s, half * v);
            }
            // (read by every warp before the barrier: rows j < kk only)
            smem[L.VW + kk * NB + tid] = v;
            smem[L.WW + kk * NB + tid] = w;
        }
        part2 = warp_sum(part2);
        if (lane == 0) red[warp] = part2;
        __syncthreads();
        mark(16);
        if (CL) {
            if (tid < C) {
                float s = 0.f;
                for (int w = 0; w < NW; w++) s += red[w];
                cl_store(cl_map(smem + L.NIN + rank, tid), s);
            }
            cl_sync();
            X = Xn;
        }
    }
    // the last two columns: d[n-2] is written, column n-2 below it is e[n-2], and d[n-1] is the
    // corner less the last panel
    {
        const int cnt = klast % NB + 1;
        const int l = CL ? ((((n - 1) >> 5) / C) << 5) + ((n - 1) & 31) : n - 1;
        if (tid == 0 && (!CL || ((n - 1) >> 5) % C == rank)) {
            float c = RES ? tile_ptr((n - 1) >> 5, (n - 1) >> 5)[33 * ((n - 1) & 31)]
                          : __ldcg(A + (size_t)(n - 1) * ld + n - 1);
            for (int j = 0; j < cnt; j++) c -= 2.f * VS[(size_t)j * R + l] * WS[(size_t)j * R + l];
            dd[n - 1] = c;
            ee[n - 2] = X[n - 1];
            ee[n - 1] = 0.f;
            tau[n - 2] = 0.f;
            tau[n - 1] = 0.f;
        }
    }
    if (pt && tid == 0) pt[1] = tq_ns();
    if (CL) cl_sync();   // no block leaves while another may still write to it
}

template <int NT, int MINB, bool RES, bool CL, int D>
__global__ void __launch_bounds__(NT, MINB) k_tridiag(EighArgs a) {
    tridiag<NT, RES, CL, D, true>(a, CL ? blockIdx.x / cl_size() : blockIdx.x);
}

// Several batches in one launch, the longest matrices first, so that the shorter ones fill the
// last wave
struct TqPlan {
    EighArgs a[CIR_TQ_MAXP];
    int start[CIR_TQ_MAXP + 1];
    int np;
};

template <int NT, int MINB, int D>
__global__ void __launch_bounds__(NT, MINB) k_tridiag_multi(const __grid_constant__ TqPlan plan) {
    int p = 0;
    while (p + 1 < plan.np && (int)blockIdx.x >= plan.start[p + 1]) p++;
    tridiag<NT, false, false, D, false>(plan.a[p], (int)blockIdx.x - plan.start[p]);
}

template <class K>
cudaError_t launch(K kern, const EighArgs &a, int nmat, int nt, bool res, int C, int minb, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cudaError_t e;
    size_t smem = sizeof(float) * (size_t)TqSmem(a.n, nt, res, C).total;
    if (a.tq_blocks > 0 && a.tq_blocks < minb) {
        // fewer blocks per SM: ask for enough shared memory that only tq_blocks fit
        int dev = 0, per_sm = 0, reserved = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess ||
            (e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) != cudaSuccess)
            return e;
        smem = std::max(smem, (size_t)per_sm / (a.tq_blocks + 1) - (size_t)reserved + 1024);
    }
    if ((e = cir_allow_smem(kern, smem)) != cudaSuccess) return e;
    cfg.gridDim = dim3(nmat * C);
    cfg.blockDim = dim3(nt);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    if (C > 1) {
        if (C > 8 && (e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return e;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = C;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, kern, a);
}

// clusters of C blocks (one block per SM) that run at a time; a fact of the device, asked once
int cluster_slots(int C) {
    static std::mutex mu;
    static int known[64][17];   // 0: not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    std::lock_guard<std::mutex> lock(mu);
    if (known[dev][C]) return known[dev][C];
    auto kern = k_tridiag<512, 1, false, true, 2>;
    const size_t smem = sizeof(float) * (size_t)TqSmem(1024, 512, false, C).total;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int k = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cir_allow_smem(kern, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&k, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        k = 0;
    }
    return known[dev][C] = k > 0 ? k : -1;
}

// Blocks per matrix.  Measured (ms per wave of matrices that run at once, GB300):
//     n      C = 1    2     4     8    16
//     512     3.1     -    3.2   2.9   3.0
//     768     7.4     -    6.0   5.1   4.9
//     1024   14.6   14.0   9.6   7.8   7.1
//     2048     -     72    44    28    22
// that is about a n + b n^3 / C, a the barriers of a column and b the pass over the triangle.
// The order of least waves times that is taken; orders up to 512 gain nothing from a cluster,
// orders above 1024 need one (the panel of 1024 rows fills a block's shared memory).
int cluster_size(int n, int nmat, int sms) {
    if (n <= 512) return 1;
    const double n3 = (double)n * n * n;
    int best = 1;
    double t = n <= 1024 ? std::ceil((double)nmat / sms) * (3.3e-3 * n + 1.2e-8 * n3) : 1e300;
    for (int C = 2; C <= 16; C *= 2) {
        const int slots = cluster_slots(C);
        if (slots < 1) continue;
        const double x = std::ceil((double)nmat / slots) * (5.8e-3 * n + 1.7e-8 * n3 / C);
        if (x < t) { t = x; best = C; }
    }
    return best == 1 && n > 1024 ? 2 : best;
}

}  // namespace

int cir_tridiag_blocks(int n) { return n <= 128 ? 4 : (n <= 512 ? 2 : 1); }

cudaError_t cir_launch_tridiag(const EighArgs &a, int nmat, cudaStream_t s) {
    int dev = 0, sms = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    EighArgs b = a;
    b.tq_blocks = cir_tridiag_limit(a.tq_blocks, nmat, sms);
    switch (cir_tridiag_form(a.n, nmat, sms)) {
    case CIR_TRI_RES4: return launch(k_tridiag<128, 4, true, false, 1>, b, nmat, 128, true, 1, 4, s);
    case CIR_TRI_RES8: return launch(k_tridiag<256, 2, true, false, 1>, b, nmat, 256, true, 1, 2, s);
    case CIR_TRI_STREAM8: return launch(k_tridiag<256, 2, false, false, 1>, b, nmat, 256, false, 1, 2, s);
    case CIR_TRI_WIDE: break;
    }
    const int C = cluster_size(a.n, nmat, sms);
    if (C > 1) return launch(k_tridiag<512, 1, false, true, 2>, b, nmat, 512, false, C, 1, s);
    return launch(k_tridiag<512, 1, false, false, 2>, b, nmat, 512, false, 1, 1, s);
}

cudaError_t cir_launch_tridiag_multi(const EighArgs *a, const int *nmat, int np, cudaStream_t s, int *launches) {
    if (np < 1 || np > CIR_TQ_MAXP) return cudaErrorInvalidValue;
    int order[CIR_TQ_MAXP];
    for (int i = 0; i < np; i++) {
        const EighArgs &x = a[i];
        if (x.n <= 256 || x.n > 1024 || nmat[i] < 1 || nmat[i] > 65535 || (x.ld & 3) || x.ld < x.n || !x.DE ||
            (reinterpret_cast<uintptr_t>(x.A) & 15))
            return cudaErrorInvalidValue;
        order[i] = i;
    }
    std::sort(order, order + np, [&](int x, int y) { return a[x].n > a[y].n; });
    TqPlan plan;
    memset(&plan, 0, sizeof plan);
    plan.np = np;
    size_t smem = 0;
    int total = 0;
    for (int k = 0; k < np; k++) {
        plan.a[k] = a[order[k]];
        plan.start[k] = total;
        total += nmat[order[k]];
        smem = std::max(smem, sizeof(float) * (size_t)TqSmem(plan.a[k].n, 512, false, 1).total);
    }
    plan.start[np] = total;
    auto kern = k_tridiag_multi<512, 1, 2>;
    cudaError_t e = cir_allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    kern<<<total, 512, smem, s>>>(plan);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (launches) *launches += 1;
    return cudaSuccess;
}
