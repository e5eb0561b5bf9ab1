// Device-side helpers and the kernel entry points shared by the .cu files.
#ifndef CIR_DEVICE_CUH_
#define CIR_DEVICE_CUH_

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <float.h>
#include <atomic>
#include <map>
#include <mutex>
#include <utility>
#include "cir_internal.h"

// SMs of the current device (asked once per device)
inline int cir_sms() {
    static std::atomic<int> known[64];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
    if ((n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 152;
    known[dev].store(n, std::memory_order_relaxed);
    return n;
}

// Lets kern be launched with that much dynamic shared memory.  The limit belongs to the kernel, whichever
// thread or context launches it, so it is only ever set to the most the device gives a block: another
// thread's smaller launch must not take it back between this call and the launch.
template <class K>
inline cudaError_t cir_allow_smem(K kern, size_t bytes) {
    static std::mutex mu;
    static std::map<const void *, size_t> own;     // the kernels' static shared memory
    size_t fixed = 0;
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = own.find(reinterpret_cast<const void *>(kern));
        if (it == own.end()) {
            cudaFuncAttributes a;
            const cudaError_t e = cudaFuncGetAttributes(&a, kern);
            if (e != cudaSuccess) return e;
            it = own.emplace(reinterpret_cast<const void *>(kern), a.sharedSizeBytes).first;
        }
        fixed = it->second;
    }
    if (bytes + fixed <= 48 * 1024) return cudaSuccess;     // what every kernel may have unasked
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fixed);
}

// minImage (calcIR.cu:1459-1463): dx - L*round(dx/L), round half away from zero, evaluated
// as the reference's float expression is, one rounding per operation (no fused multiply-add),
// so that the image chosen at the box's half-width rounds as the reference rounds it.
__device__ __forceinline__ float cir_mi(float dx, float L) {
    return __fsub_rn(dx, __fmul_rn(L, roundf(__fdiv_rn(dx, L))));
}
// cir_mi of three components with the quotients' rounding taken from products with 1 / L.  The
// nearest integers are the same unless a quotient lies within the products' error of a half (or
// is large, or NaN): cir_mi3_quick says so and leaves the components, cir_mi3 asks cir_mi.
__device__ __forceinline__ bool cir_mi3_quick(float &dx, float &dy, float &dz, float bx, float by, float bz, float rx,
                                              float ry, float rz) {
    const float tx = dx * rx, ty = dy * ry, tz = dz * rz;
    constexpr float R = 12582912.f;   // 1.5 * 2^23: adding it leaves the nearest integer (|t| < 2^22)
    const float nx = __fsub_rn(__fadd_rn(tx, R), R), ny = __fsub_rn(__fadd_rn(ty, R), R), nz = __fsub_rn(__fadd_rn(tz, R), R);
    const float half = fmaxf(fmaxf(fabsf(tx - nx), fabsf(ty - ny)), fabsf(tz - nz));
    const float big = fmaxf(fmaxf(fabsf(nx), fabsf(ny)), fabsf(nz));
    if (!(half < 0.49999f && big < 32.f && tx == tx && ty == ty && tz == tz)) return false;
    dx = __fsub_rn(dx, __fmul_rn(bx, nx));
    dy = __fsub_rn(dy, __fmul_rn(by, ny));
    dz = __fsub_rn(dz, __fmul_rn(bz, nz));
    return true;
}
__device__ __forceinline__ void cir_mi3(float &dx, float &dy, float &dz, float bx, float by, float bz, float rx, float ry,
                                        float rz) {
    if (cir_mi3_quick(dx, dy, dz, bx, by, bz, rx, ry, rz)) return;
    dx = cir_mi(dx, bx);
    dy = cir_mi(dy, by);
    dz = cir_mi(dz, bz);
}
// 1 / sqrt(x), the hardware's approximation with one Newton step
__device__ __forceinline__ float cir_rsqrt(float x) {
    const float y = rsqrtf(x);
    return fmaf(__fmul_rn(0.5f, y), fmaf(__fmul_rn(-x, y), y, 1.f), y);
}
// exp(i ph) as FP32 cosine and sine and what they lack of length one: sincosf's pair is long by 8.4e-9
// on average (phases up to 0.75, 4M of them; 0.0e-9 for correctly rounded ones), which every
// propagation step would multiply into F, 2e-6 in 250.
struct CirPhase {
    float c, s, dc, ds;
};
__device__ __forceinline__ CirPhase cir_phase(float ph) {
    CirPhase p;
    sincosf(ph, &p.s, &p.c);
    // 1 - c^2 - s^2: the squares with their rounding errors, the larger one first
    const float cc = __fmul_rn(p.c, p.c), ss = __fmul_rn(p.s, p.s);
    const float d = __fsub_rn(__fsub_rn(__fsub_rn(1.f, fmaxf(cc, ss)), fminf(cc, ss)),
                              __fadd_rn(fmaf(p.c, p.c, -cc), fmaf(p.s, p.s, -ss)));
    p.dc = 0.5f * d * p.c;
    p.ds = 0.5f * d * p.s;
    return p;
}
// (re, im) times exp(i ph); infinite values without the corrections, which may have the other sign
__device__ __forceinline__ void cir_rotate(const CirPhase &p, float &re, float &im) {
    float x = fmaf(p.c, re, fmaf(-p.s, im, fmaf(p.dc, re, -p.ds * im)));
    float y = fmaf(p.s, re, fmaf(p.c, im, fmaf(p.ds, re, p.dc * im)));
    if (!(fabsf(x) <= FLT_MAX && fabsf(y) <= FLT_MAX)) {
        x = p.c * re - p.s * im;
        y = p.s * re + p.c * im;
    }
    re = x;
    im = y;
}
// mag3 (calcIR.cu:1464-1476): sqrt(x*x + y*y + z*z) with the reference's order of operations
// and one rounding each; the field's cutoff test compares it with 0.7831 nm, a discontinuous
// decision that a contracted evaluation would take differently for pairs within an ulp of it.
__device__ __forceinline__ float cir_mag3(float x, float y, float z) {
    return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z)));
}

__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_sum_d(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Strict total order on (value, index) with NaN after every number: ranks counted with it
// form a permutation whatever the values, so non-finite input can never turn a rank into an
// out-of-range index.  cir_lt / cir_le are x < v and x <= v in the same order (no index).
template <typename T>
__device__ __forceinline__ bool cir_before(T a, int i, T b, int j) {
    const bool na = a != a, nb = b != b;
    if (na || nb) return na && nb ? i < j : nb;
    return a < b || (a == b && i < j);
}
template <typename T>
__device__ __forceinline__ bool cir_lt(T x, T v) { return x == x && (v != v || x < v); }
template <typename T>
__device__ __forceinline__ bool cir_le(T x, T v) { return v != v || (x == x && x <= v); }

// Per-chromophore quantities produced by the field kernel, struct-of-arrays per frame:
// row r of a frame's [CT_NROW][ld] block.
enum {
    CT_E = 0,     // field projection (a.u.)
    CT_W,         // map frequency omega (cm^-1)
    CT_X,         // map x
    CT_P,         // map p
    CT_MUP,       // map mu'
    CT_UX, CT_UY, CT_UZ,   // OH unit vector
    CT_TX, CT_TY, CT_TZ,   // transition dipole position, wrapped by minImage
    CT_NROW
};

struct BuildArgs {
    const float *xyz;     // [nframes][natoms][3]
    const float *box;     // [nframes][3]
    float *ct;            // [nframes][CT_NROW][ld] chromophore table
    float *H;             // [nframes][n][ldh]
    float *eproj;         // [nframes][n]  or null
    float *dip;           // frame f: rows x,y,z at dip + f*dip_fstride + {0,1,2}*ldv, or null
    float *pol;           // frame f: rows xx,yy,zz,xy,yz,zx at pol + f*pol_fstride + r*ldv, or null
    long long dip_fstride, pol_fstride;
    int natoms, natom_mol, nchrom_mol, nmol, n;
    int ld;               // leading dimension of the chromophore table rows
    int ldh;              // row stride of H
    int ldv;              // row stride of dip/pol
    int imodel, ispecies;
    float avef;
    CirMaps maps;
};

constexpr int CIR_EIG_PROF_SLOTS = 20;

struct EighArgs {
    float *A;             // [nmat] matrices, column j of matrix m at A + m*mstride + j*ld
    float *W;             // [nmat][wstride] eigenvalues
    float *Z;             // scratch, same shape as A
    float2 *rot;          // scratch, cir_eigh_rot_bytes(n) per matrix
    float *DE;            // scratch, cir_eigh_de_bytes(ld) per matrix (tridiagonal d, e, tau)
    cudaEvent_t tq_done;  // recorded after the tridiagonalisation kernel when not null
    int precision;        // CIR_PREC_*: FP32, or the tensor-core form of the final V = Q_H Q_T product
    int *err;             // tensor-core kernels: set to 1 when a bounded wait gives up
    float *DC;            // divide-and-conquer scratch, cir_dc_bytes(n, ld) per matrix, laid out
                          // [3][nmat][mstride]; null selects the implicit-QR path (rot needed)
    long long mstride;
    int wstride;
    int n, ld;
    int *status;          // [nmat] 0 ok, 1 sweep cap reached
    unsigned long long *sweeps;   // accumulated QR sweeps (may be null)
    // frequency distribution (calcIR.cu:493-538); hist_count == null disables it
    int hist_group;       // matrices per histogram set (consecutive matrices; 0: one set for all);
                          // set g uses hist_*[g*nomega ..] and out_of_range[g]
    unsigned long long *hist_count;
    double *hist_ipr, *hist_mipr;
    const int *hist_weight;       // [nmat] times each matrix counts in the distributions (null: once)
    unsigned long long *out_of_range;
    int nomega, omegaStep, nchrom_mol;
    float avef, omegaStart;
    // optional [nmat][CIR_EIG_PROF_SLOTS]: %globaltimer at the start and end of the
    // tridiagonalisation, of forming Q, of the QR iteration and of the ordering (0-6), then the
    // chase and apply times (ns), rotations, the chase's block-search time (ns) and sweeps
    // (7-11; on the divide-and-conquer path: the merges' time in setup and deflation, secular
    // roots, z and norms, ranking and rotation, summed over a matrix's merges), then the
    // tridiagonalisation's time (ns) in its cluster exchange, reflector, symmetric matrix-vector
    // product, panel dot products, w and the products that update the matrix (12-17), then the
    // secular equation's iterations and roots (18-19)
    unsigned long long *phase_ns;
    // optional FP64 refinement of the eigenpairs on the divide-and-conquer path (k_refine.cu),
    // on when Href is not null: Href holds a copy of the input matrices (same strides as A), RW
    // is scratch of cir_refine_bytes(n, ld) per matrix for refine_chunk matrices at a time
    const float *Href;
    void *RW;
    int refine_iters, refine_chunk;
    // fault drills (tests only, 0 = off): the split-BF16 GEMMs' stall (SplitGemmArgs::test_stall)
    // and a cap on the QR sweeps of each divide-and-conquer leaf
    int test_stall, test_sweep_cap;
    // thread blocks of the tridiagonalisation per SM: 0 the kernel's own occupancy, or a
    // smaller count enforced through its shared-memory request (the autotuner's choice)
    int tq_blocks;
    // 1: cir_launch_eigh starts after the tridiagonalisation (d, e, tau already in DE and the
    // reflectors in A, as cir_launch_tridiag_multi leaves them)
    int skip_tridiag;
};

// kernel launchers (return cudaError_t of the launch)
cudaError_t cir_launch_build(const BuildArgs &a, int nframes, cudaStream_t s, int *launches);
cudaError_t cir_launch_eigh(const EighArgs &a, int nmat, cudaStream_t s, int *launches);
// the tridiagonalisation kernel alone (phase 1 of cir_launch_eigh), for the autotuner
cudaError_t cir_launch_tridiag(const EighArgs &a, int nmat, cudaStream_t s);
// thread blocks per SM the tridiagonalisation of order n runs with by default
int cir_tridiag_blocks(int n);
// The tridiagonalisations of up to CIR_TQ_MAXP batches of orders 257-1024 (boxes of different
// size) in one launch, the longest matrices first; a[i] as for cir_launch_tridiag (tq_blocks
// is not applied: the kernel's own occupancy).
constexpr int CIR_TQ_MAXP = 4;
cudaError_t cir_launch_tridiag_multi(const EighArgs *a, const int *nmat, int np, cudaStream_t s, int *launches);
size_t cir_eigh_rot_bytes(int n);
size_t cir_eigh_de_bytes(int ld);
size_t cir_dc_bytes(int n, int ld);
cudaError_t cir_launch_dc(const EighArgs &a, int nmat, cudaStream_t s, int *launches);
// V = Q_H Q into a.A by blocked compact-WY application of the tridiagonalisation's
// reflectors (in a.A) to Q; Q is overwritten, P and U are scratch (a.mstride floats per
// matrix), a.Z holds the blocks' T^T V^T.
cudaError_t cir_launch_backtransform(const EighArgs &a, float *Q, float *P, float *U, int nmat, cudaStream_t s,
                                     int *launches,
                                     bool q_split = false);
// FP64 refinement of eigenpairs (k_refine.cu): iters steps on the eigenvectors Z (row j =
// eigenvector j, mstride / ld as A) of the matrices H (same strides) with eigenvalues w
// (stride wstride), chunk matrices at a time in ws (cir_refine_bytes(n, ld) per matrix).
size_t cir_refine_bytes(int n, int ld);
cudaError_t cir_launch_refine(const float *H, float *Z, long long mstride, int ld, int n, float *w, long long wstride,
                              int nmat, int iters, void *ws, int chunk, cudaStream_t s, int *launches);
int cir_eigh_max_n();

// batched FP32 GEMM (k_gemm.cu), C = A * B (row-major B, C); A row- or column-major.
// epilogue 1: rotate column pairs (2q, 2q+1) of row i by exp(+i w[i] dt/hbar).
struct GemmArgs {
    const float *A, *B;
    float *C;
    int M, N, K;
    int lda, ldb, ldc;
    long long sA, sB, sC;  // batch strides (elements)
    bool a_colmajor;
    bool b_kmajor;         // B element (k, n) at B[n*ldb + k] instead of B[k*ldb + n]
    bool full_range;       // k_gemm: infinite, very large and very small values as exact as FFMAs (C is
                           // neither A nor B); the eigensolver's products, of vectors, go without
    int epilogue;          // 0 none, 1 phase rotation, 2 C = D - A B
    const float *D;        // epilogue 2 (may equal C)
    int ldd;
    long long sD;
    const float *w;        // [batch][wstride] for epilogue 1
    int wstride;
    float dt_over_hbar;
    int *err;              // tensor-core kernels: set to 1 when a bounded wait gives up
    // k_tc_gemm only, epilogue 0: when set, C is written as a BF16 hi/lo pair at the same
    // element offsets instead (batch stride 2 sC elements)
    __nv_bfloat16 *Chi, *Clo;
};
struct TcfArgs;
// tcf: the product is the propagated F whose contraction is wanted; *fused is set where the launch
// has done it (small products), and is otherwise left
cudaError_t cir_launch_gemm(const GemmArgs &g, int batch, cudaStream_t s, int *launches, const TcfArgs *tcf = nullptr,
                            bool *fused = nullptr);
// the same product in TF32 or two-term split BF16 (k_tc_gemm.cu)
cudaError_t cir_launch_tc_gemm(const GemmArgs &g, int batch, int precision, cudaStream_t s, int *launches);
size_t cir_tc_gemm_smem_bytes();

// ---- split-BF16 propagation on pre-split operands (k_tc_split.cu) ----
// A matrix held as two BF16 matrices, hi = bf16(x) and lo = bf16(x - hi).
struct SplitMat {
    __nv_bfloat16 *hi, *lo;
};
// C = A B (hi*hi + hi*lo + lo*hi, FP32 accumulation) with K-major operands:
// A(i, k) at A[i*lda + k], B(k, j) at B[j*ldb + k].  out_mode 0: C(i, j) written as a
// hi/lo pair at C[j*ldc + i]; 1: as a pair at C[i*ldc + j]; 2: in FP32 at Cf[i*ldc + j].
// lda, ldb and the batch strides are multiples of 8, the operand pointers 16-byte aligned.
// epilogue 1: columns (2q, 2q+1) of row i rotated by exp(+i w[i] dt/hbar) before the split;
// epilogue 2: C = D - A B, D a row-major pair (D[i*ldd + j], batch stride sD; may be C).
struct SplitGemmArgs {
    const __nv_bfloat16 *Ahi, *Alo, *Bhi, *Blo;
    __nv_bfloat16 *Chi, *Clo;
    float *Cf;
    int out_mode;
    const __nv_bfloat16 *Dhi, *Dlo;
    int ldd;
    long long sD;
    int M, N, K;
    int lda, ldb, ldc;
    long long sA, sB, sC;
    int epilogue;
    const float *w;
    int wstride;
    float dt_over_hbar;
    int *err;
    // fused correlation contraction for the propagation product F' = V G (out_mode 0): when
    // tcf_out is set, row r of the product contracts with m(0) over the tile's complex columns
    // and with m(k) at row r (the terms of k_tcf), and each block adds its six sums to
    // tcf_out[batch * tcf_sout ..]
    const float *tcf_m0, *tcf_mt;
    long long tcf_sm0, tcf_smt;
    int tcf_ldv;
    double *tcf_out;
    long long tcf_sout;
    int bz0;              // batch entry of blockIdx.z == 0 (set by the launcher when it splits a batch)
    int test_stall;       // fault drill (tests only): 1 withholds the first tile's completion and
                          // shortens the pipeline waits, so that they run out and raise err
    int tile_n;           // tile width: 0 picks by shape; 128 or 256 forces it (the autotuner's choice)
};
size_t cir_split_ld(int n);   // leading dimension of the split operands (n rounded up to 8)
cudaError_t cir_launch_split_gemm(const SplitGemmArgs &g, int batch, cudaStream_t s, int *launches);
// Several split-BF16 products in one persistent launch (the tiles of problem 0 first, then
// problem 1, ...): each problem a batch of one shape with its own operands, epilogue and
// tensor maps, all in the widest tile width any of them takes; bz0 must be 0.
constexpr int CIR_SPLIT_MAXP = 4;
cudaError_t cir_launch_split_gemm_multi(const SplitGemmArgs *g, const int *batch, int np, cudaStream_t s,
                                        int *launches);
// Vc = V (V[k][i] at A[i*ld + k]) and Vr = V^T, both as Vc[i*ldh + k]-style K-major pairs
cudaError_t cir_launch_split_v(const float *A, int ld, long long sA, int n, SplitMat Vc, SplitMat Vr, int ldh,
                               long long sV, int batch, cudaStream_t s, int *launches);
// Ft = I for the transposed complex F (real column c = 2q + {0: re, 1: im} at Ft[c*ldh ..])
cudaError_t cir_launch_identity_t(SplitMat F, int n, int ldh, long long sF, int batch, cudaStream_t s, int *launches);

// ---- two-stage reduction to tridiagonal form (k_sbr.cu): dense -> band on the split-BF16
// tcgen05 GEMM, band -> tridiagonal by bulge chasing; d and e only (no eigenvectors) ----
int cir_sbr_max_n();
size_t cir_sbr_bytes(int n, int ld);   // work area per matrix (ld a multiple of 8)
cudaError_t cir_launch_sbr(const float *H, long long sH, int nmat, int n, int ld, float *d, float *e, void *work,
                           int *err, cudaStream_t s, float *ms, int *launches);

// TCF terms: out[b][6] += (IR, VV, VH) for batch element b
struct TcfArgs {
    const float *F;        // [batch] complex row-major, row stride ldf floats (2 per element)
    long long sF;
    const float *m0;       // [batch][9][ldv] dip0 (3) then pol0 (6)
    const float *mt;       // [batch][9][ldv]
    long long sm0, smt;
    double *out;           // [batch][6]
    long long sout;
    int n, ldf, ldv;
    SplitMat Ft;           // when Ft.hi is set: F stored transposed as a split pair, F[r][c] at
    long long sFt;         // Ft[c*ldft + r], instead of F
    int ldft;
};
cudaError_t cir_launch_tcf(const TcfArgs &t, int batch, cudaStream_t s, int *launches);

// spectral density of S * sets frames (strides sV, sw, sdip; set q holds frames qS .. qS + S - 1):
// Sw[set][nomega] += the set's sum, or, when Swf is given (one set), Swf[nomega] += in FP32;
// mu2: scratch, n floats per frame
cudaError_t cir_launch_spectral(const float *V, int ld, long long sV, const float *w, long long sw, const float *dip, int ldv,
                                long long sdip, int n, int S, int sets, float *mu2, double *Sw, float *Swf, int nomega,
                                float omegaStart, int omegaStep, float t1, float avef, cudaStream_t s, int *launches);

// The printed rows of a lineshape: outputs i0 .. i0 + cnt1 - 1 of the transform of length n,
// then outputs 0 .. cnt2 - 1, each over norm (cir_api.cu ls_rows).
struct LsRows {
    int n, i0, cnt1, cnt2;
    float norm;
};
// rows [nq][cnt1 + cnt2] of nq damped TCFs X [nq][K] (complex double): the unnormalised inverse
// real DFT (cuFFT C2R convention) of the zero-padded TCFs; work: cir_lineshape_work_bytes (null
// when 0)
size_t cir_lineshape_work_bytes(int K, int n);
cudaError_t cir_launch_lineshape(const double *X, int nq, int K, const LsRows &r, void *work, float *out,
                                 cudaStream_t s, int *launches);
// L = sum (rows - target)^2 over two spectra and dL/dX [2][K] (complex) into g; dy: scratch
// [2][cnt1 + cnt2]
cudaError_t cir_launch_ls_adjoint(const float *rows, const float *target, int K, const LsRows &r, double *dy,
                                  double *loss, double *g, cudaStream_t s, int *launches);

// F = I for nprop complex matrices
cudaError_t cir_launch_identity(float *F, int n, int ldf, long long sF, int batch, cudaStream_t s, int *launches);


// ---- differentiation form (k_adjoint.cu) ----
constexpr int CIR_PSI_LD = 18;   // psi / lambda: n x 9 complex, row-major (re, im) pairs
struct DthetaArgs {       // matrix b = s*K + k: step k of origin s
    const float *ct;      // chromophore tables, CT_NROW * ld apart
    const float *box;     // boxes, 3 apart
    const float *G;       // dL/dH (symmetric, leading dimension ldg), sG apart; not read at step 0
    int ldg;
    long long sG;
    const float *psi;     // psi(k) of origin s at (k*S + s) * n * CIR_PSI_LD
    const float *lam0;    // lambda(0), n x CIR_PSI_LD per origin
    const double *g;      // dL/dTCF of the steps: (re, im) of IR and of VV, 4 a step
    CirMaps maps;
    int n, ld, K, nchrom_mol, ispecies;
    double *out;          // [13] accumulated
};
// the adjoint's source w(k): m(k) of origin 0 (origin s at M + s*sM) and dL/dTCF of the step
struct PsiSource {
    const float *M;
    long long sM;
    float gir_r, gir_i, gvv_r, gvv_i;
};
// one step out = V e^{i L dt/hbar} V^T in (+ the source, if any) of S origins (n x CIR_PSI_LD per
// origin each; in may be out); raw, if given, receives V^T in
cudaError_t cir_psi_step(const float *V, int ld, long long sV, int n, const float *w, long long sw, float dt_over_hbar,
                         const float *in, float *out, float *tmp, float *raw, const PsiSource *src, int S,
                         cudaStream_t s);
cudaError_t cir_adj_psi_init(const float *M, long long sM, int ld, int n, int S, float *psi, cudaStream_t s);
// K steps: psi(k) of all origins at psi + k * S * n * CIR_PSI_LD, m(k) at M + 9 k ld
cudaError_t cir_adj_tcf(const float *psi, const float *M, long long sM, int ld, int n, int S, int K, double *out,
                        long long sout, cudaStream_t s);
cudaError_t cir_adj_lambda_init(float *lam, const PsiSource &src, int ld, int n, int S, cudaStream_t s);
cudaError_t cir_adj_build_R(const float *a, const float *b, long long sab, const float *W, long long sW, int n, int batch,
                            float tau, float *R, int ldr, long long sR, cudaStream_t s);
cudaError_t cir_adj_dtheta(const DthetaArgs &d, int S, cudaStream_t s);

#endif
