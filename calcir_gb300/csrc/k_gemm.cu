// Batched FP32 GEMM on the tensor cores: C[b] = A[b] B[b], FP32 in and out and FP32 accuracy,
// for the plain form: the propagation step, the eigensolver's back-transform and upper merges,
// and the gradient.  The reference builds a dense diagonal propagator and multiplies three
// complex matrices per frame (Pinit + 3 x magma_cgemm, calcIR.cu:596-613, 24 N^3 real flops).
// Here the complex F is a real N x 2N matrix of interleaved (re, im) columns and one step is two
// real GEMMs, 8 N^3 flops:
//     G  = V^T F                  (epilogue: row j of G times exp(+i w_j dt/hbar))
//     F' = V G
//
// Each operand value is split into three BF16 terms, x = h + m + l, on grids common to the 32 values
// of a row (column) of a slice: h is x rounded to 2^(e-8), 2^e above the largest of them, m the rest
// rounded to 2^(e-16), l what is left (the error-free splitting of Ozaki, Ogita, Oishi and Rump,
// Numer. Algorithms 59, 2012).  The product is eight tcgen05.mma kind::f16 per 16 of K: h h into
// the accumulator H, and h m, m h, m m, h l, l h, m l, l m into a second accumulator L (l l, below
// 2^-34 of the slices' largest product, is left out).  The tensor core drops the bits that fall below the
// accumulator's last on every instruction, always toward zero.  In H there are none: h is at most
// 256 steps of its grid, 32 products at most 2^21 steps of theirs, so a slice's sum is exact; H
// is read out every slice and summed in FP32 registers with rounding to nearest.  L, 2^-8 of the sum
// and of no fixed sign against it, is read out once a tile.  (With h, m, l rounded value by value the
// sums of h h lost a part of a bit every instruction: F shrank by 1.3e-7 a step, 1.9e-5 in 146 steps of
// 244 chromophores.)
//
// BF16 numbers have FP32's range, but not all three terms of a value near its ends, and infinite
// terms do not add up.  Where the caller's values may be anything (full_range), the loaders watch the
// largest magnitude of every row and column of a tile, and a tile with one outside F_TINY .. F_HUGE
// is summed again by FFMAs in its epilogue.
//
// One CTA per SM walks 128 x 128 tiles (column tile fastest, then row tile, then matrix):
//   warps 0-7   copy FP32 slices 32 deep (0-3 A, 4-7 B) into shared memory, F_RAW slices ahead,
//               split them and store the three terms K-major (core matrices of 8 rows x 16 bytes,
//               (r/8, k/8) at (r/8)*SBO + (k/8)*LBO; SBO padded so that either orientation stores
//               without bank conflicts) into a ring;
//   warps 8-15  sum the slices (a thread a row and half of the columns), then the epilogue, while
//               the next tile is loaded and multiplied (two H and two L accumulators, all 512
//               columns of tensor memory);
//   warp 16     issues the MMAs.
// The splitting bounds it (with the two products of m and l left out 314-391 us below, without the
// slices' maxima 303-361).  1024 x 2048 x 1024 in ten matrices: 859-1044 us as SIMT FFMAs (50-41
// TFLOP/s), 323-386 so (133-111), error against 64 bits 5.7e-7 and 6e-8; with the terms rounded
// value by value and six products 283-331 us, 1.2e-7 and the drift above.  Not taken: 16 splitting
// warps (403-432: the copies of 8 bytes that rows contiguous then need).  Smaller products
// run on the SIMT kernels further down (cir_gemm_form).
// Every wait is bounded: a timeout raises the CTA's abort flag and the error flag, every role
// leaves its loop, and the MMAs issued are waited for before the tensor memory is freed.
#include "cir_device.cuh"
#include "cir_plan.h"
#include "cir_tcf.cuh"
#include "cir_tcgen05.cuh"

#include <cuda_bf16.h>
#include <algorithm>
#include <climits>

namespace {

constexpr int FM = 128, FN = 128, FK = 32;     // tile, K of a slice
constexpr int F_LBO = 128, F_SBO = 528;
constexpr int F_PART = (FM / 8) * F_SBO;       // bytes of one term of one operand's slice
constexpr int F_STAGE = 6 * F_PART, F_NS = 3, F_RAW = 2;
constexpr int F_LOAD = 8, F_ACC = 8;           // warps
constexpr int F_NT = 32 * (F_LOAD + F_ACC + 4);   // whole warpgroups: the register split is per group
// below F_TINY l reaches under BF16's smallest normal number; from F_HUGE the grids' constants would overflow
constexpr float F_TINY = 0x1p-100f, F_HUGE = 0x1p112f;
constexpr int F_ODD = 8;                       // tiles the loaders' notes reach back: they are at most 5 ahead of the epilogue
constexpr size_t F_RAWB = (size_t)F_LOAD * 32 * 128;   // bytes of an FP32 slice of both operands
constexpr size_t F_SMEM = (size_t)F_NS * F_STAGE + F_RAW * F_RAWB + 256;

// The warpgroups' registers: 640 threads launch with 96 each (61440); the idle three warps of
// the MMA group give theirs to the loads in flight and the sums: 2 * 128 * 120 + 2 * 128 * 104 +
// 128 * 24 = 60416
template <int R>
__device__ __forceinline__ void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

__device__ __forceinline__ void mbar_arrive1(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// The constants that round to the grids 2^(e-8) and 2^(e-16) by being added and taken away, 2^e the
// power of two above mx: 1.5 * 2^(e+15) and 1.5 * 2^(e+7).  Within e's range below the grids are BF16 numbers
// and the constants finite.
__device__ __forceinline__ float2 split_grids(float mx) {
    const uint32_t e = min(max(__float_as_uint(mx) & 0x7f800000u, 10u << 23), 238u << 23);
    return make_float2(__uint_as_float(e + ((16u << 23) | 0x400000u)), __uint_as_float(e + ((8u << 23) | 0x400000u)));
}

// two FP32 operations an instruction
__device__ __forceinline__ uint64_t pair_of(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {   // a - b
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(0xbf800000bf800000ull), "l"(a));
    return r;
}

// the three BF16 terms of eight values on the grids c, as 16-byte words
__device__ __forceinline__ void split3(const float (&x)[8], float2 c, uint4 &h, uint4 &m, uint4 &l) {
    const uint64_t ch = pair_of(c.x, c.x), chn = pair_of(-c.x, -c.x), cm = pair_of(c.y, c.y), cmn = pair_of(-c.y, -c.y);
    uint32_t wh[4], wm[4], wl[4];
    #pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint64_t v = pair_of(x[2 * q], x[2 * q + 1]);
        const uint64_t hv = add2(add2(v, ch), chn), r = sub2(v, hv);
        const uint64_t mv = add2(add2(r, cm), cmn), lv = sub2(r, mv);
        // h and m have eight significant bits: their upper halves are the BF16 numbers
        wh[q] = __byte_perm((uint32_t)hv, (uint32_t)(hv >> 32), 0x7632);
        wm[q] = __byte_perm((uint32_t)mv, (uint32_t)(mv >> 32), 0x7632);
        const __nv_bfloat162 pl = __floats2bfloat162_rn(__uint_as_float((uint32_t)lv), __uint_as_float((uint32_t)(lv >> 32)));
        wl[q] = *reinterpret_cast<const uint32_t *>(&pl);
    }
    h = make_uint4(wh[0], wh[1], wh[2], wh[3]);
    m = make_uint4(wm[0], wm[1], wm[2], wm[3]);
    l = make_uint4(wl[0], wl[1], wl[2], wl[3]);
}

// One thread's part of an operand slice (128 rows of the M or N dimension, 32 of K): four groups
// of eight consecutive K of one row.  KC: K contiguous in memory (element (r, k) at p[r*ld + k]),
// group i is row 32 i + 8 (warp & 3) + (lane & 7), K 8 (lane >> 3) ..; else rows contiguous
// (element (r, k) at p[k*ld + r]), group i is row 32 (warp & 3) + 4 (lane & 7) + i, K 8 (lane >> 3) ...
// Either way four lanes of a warp, 8 apart, hold the 32 values of a row.
// The values wait in shared memory, each thread's own eight 16-byte words (raw, RAW_ST apart),
// which no other thread reads: an asynchronous copy needs no register and no barrier.
constexpr int RAW_ST = F_LOAD * 32 * 16;

template <bool KC>
struct Part {
    // four values at q, of which the first `have` exist; the others are zero (p: any address of the
    // operand, for what is not read)
    __device__ __forceinline__ static void load4(unsigned char *raw, const float *q, int have, const float *p, bool vec) {
        const uint32_t dst = smem_addr(raw);
        if (vec) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(have > 0 ? q : p),
                         "r"(4 * max(0, min(have, 4))) : "memory");
            return;
        }
        #pragma unroll
        for (int e = 0; e < 4; e++)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * e), "l"(have > e ? q + e : p),
                         "r"(have > e ? 4 : 0) : "memory");
    }
    __device__ __forceinline__ static void load(unsigned char *raw, const float *p, int ld, int rdim, int kdim, int r0, int k0,
                                                int w4, int lane, bool vec) {
        if (vec && r0 + 128 <= rdim && k0 + 32 <= kdim) {   // the whole slice inside
            const float *q = KC ? p + (size_t)(r0 + 8 * w4 + (lane & 7)) * ld + k0 + 8 * (lane >> 3)
                                : p + (size_t)(k0 + 8 * (lane >> 3)) * ld + r0 + 32 * w4 + 4 * (lane & 7);
            const size_t st = KC ? (size_t)32 * ld : (size_t)ld;
            #pragma unroll
            for (int i = 0; i < 8; i++)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(raw + i * RAW_ST)),
                             "l"(KC ? q + (i >> 1) * st + 4 * (i & 1) : q + i * st)
                             : "memory");
        } else if (KC) {
            #pragma unroll
            for (int i = 0; i < 4; i++) {
                const int r = r0 + 32 * i + 8 * w4 + (lane & 7), k = k0 + 8 * (lane >> 3);
                const float *q = p + (size_t)r * ld + k;
                const int have = r < rdim ? kdim - k : 0;
                load4(raw + 2 * i * RAW_ST, q, have, p, vec);
                load4(raw + (2 * i + 1) * RAW_ST, q + 4, have - 4, p, vec);
            }
        } else {
            const int r = r0 + 32 * w4 + 4 * (lane & 7);
            #pragma unroll
            for (int i = 0; i < 8; i++) {
                const int k = k0 + 8 * (lane >> 3) + i;
                load4(raw + i * RAW_ST, p + (size_t)k * ld + r, k < kdim ? rdim - r : 0, p, vec);
            }
        }
    }
    // rmx: the largest magnitude so far of each group's row
    __device__ __forceinline__ static void store(const unsigned char *raw, unsigned char *base, int w4, int lane, float (&rmx)[4]) {
        float4 v[8];
        #pragma unroll
        for (int i = 0; i < 8; i++) v[i] = *reinterpret_cast<const float4 *>(raw + i * RAW_ST);
        #pragma unroll
        for (int i = 0; i < 4; i++) {
            float x[8];
            uint32_t o;
            if (KC) {
                x[0] = v[2 * i].x; x[1] = v[2 * i].y; x[2] = v[2 * i].z; x[3] = v[2 * i].w;
                x[4] = v[2 * i + 1].x; x[5] = v[2 * i + 1].y; x[6] = v[2 * i + 1].z; x[7] = v[2 * i + 1].w;
                o = (4 * i + w4) * F_SBO + (lane >> 3) * F_LBO + (lane & 7) * 16;
            } else {
                #pragma unroll
                for (int q = 0; q < 8; q++) x[q] = i == 0 ? v[q].x : i == 1 ? v[q].y : i == 2 ? v[q].z : v[q].w;
                const int r = 32 * w4 + 4 * (lane & 7) + i;
                o = (r >> 3) * F_SBO + (lane >> 3) * F_LBO + (r & 7) * 16;
            }
            float mx = 0.f;
            #pragma unroll
            for (int q = 0; q < 8; q++) mx = fmaxf(mx, fabsf(x[q]));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
            rmx[i] = fmaxf(rmx[i], mx);
            uint4 h, m, l;
            split3(x, split_grids(mx), h, m, l);
            *reinterpret_cast<uint4 *>(base + o) = h;
            *reinterpret_cast<uint4 *>(base + F_PART + o) = m;
            *reinterpret_cast<uint4 *>(base + 2 * F_PART + o) = l;
        }
    }
};

__device__ __forceinline__ uint64_t f_desc(uint32_t addr) { return smem_desc_kmajor(addr, F_LBO, F_SBO); }

// 64 columns from c0 of row r by FFMAs (out of line: no registers of the tile's sums held for it)
template <bool ACOL, bool BKC>
__device__ __noinline__ void f_row_again(const GemmArgs &g, int bz, int r, int c0) {
    const float *A = g.A + (size_t)bz * g.sA + (ACOL ? (size_t)r : (size_t)r * g.lda), *B = g.B + (size_t)bz * g.sB;
    const size_t as = ACOL ? g.lda : 1, bs = BKC ? 1 : g.ldb, bc = BKC ? g.ldb : 1;
    float *C = g.C + (size_t)bz * g.sC + (size_t)r * g.ldc;
    for (int c = c0; c < min(c0 + 64, g.N); c += 2) {
        const bool two = c + 1 < g.N;
        const float *b = B + c * bc;
        float re = 0.f, im = 0.f;
        for (int k = 0; k < g.K; k++, b += bs) {
            const float a = A[k * as];
            re = fmaf(a, b[0], re);
            if (two) im = fmaf(a, b[bc], im);
        }
        if (g.epilogue == 1) cir_rotate(cir_phase(g.w[(size_t)bz * g.wstride + r] * g.dt_over_hbar), re, im);
        C[c] = re;
        if (two) C[c + 1] = im;
    }
}

// vecA, vecB, vecC: every 16-byte access of the operand (C and D: both) is aligned (pointer,
// leading dimension, stride)
template <bool ACOL, bool BKC>
__global__ void __launch_bounds__(F_NT, 1) k_gemm(GemmArgs g, int tiles_n, int tiles_mn, int ntiles, bool vecA, bool vecB,
                                                   bool vecC, int *err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + (size_t)F_NS * F_STAGE + F_RAW * F_RAWB);   // [F_NS]
    uint64_t *empty = full + F_NS;                                                 // [F_NS]
    uint64_t *hfull = empty + F_NS;                                                // [2] slice in H
    uint64_t *hempty = hfull + 2;                                                  // [2]
    uint64_t *lempty = hempty + 2;                                                 // [2] L read out
    uint64_t *drain = lempty + 2;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(drain + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tslot + 1);
    volatile int *odd = abort_flag + 1;                                            // [F_ODD]: t + 1: the CTA's tile t is out of range
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == F_LOAD + F_ACC) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tslot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int s = 0; s < F_NS; s++) {
            mbar_init(&full[s], F_LOAD);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(&hfull[a], 1);
            mbar_init(&hempty[a], F_ACC);
            mbar_init(&lempty[a], F_ACC);
        }
        mbar_init(drain, 1);
        *abort_flag = 0;
        for (int i = 0; i < F_ODD; i++) odd[i] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tslot;
    const int KT = (g.K + FK - 1) / FK;      // slices of a tile
    auto fail = [&]() {
        *abort_flag = 1;
        if (err) atomicExch(err, 1);
    };
    auto tile = [&](int t, int &bz, int &m0, int &n0) {
        bz = t / tiles_mn;
        const int rem = t % tiles_mn;
        m0 = (rem / tiles_n) * FM;
        n0 = (rem % tiles_n) * FN;
    };

    if (warp < F_LOAD) {
        regs_up<120>();
        const bool isA = warp < 4;
        const int w4 = warp & 3;
        // (the operand's side: pointer, strides, extents)
        auto produce = [&](auto part, const float *base, long long sb, int ld, int rdim, bool vec) {
            // the load side runs F_RAW slices ahead of the store side
            int lt = blockIdx.x, lkt = 0, r0 = 0;
            const float *src = base;
            unsigned char *raw = smem + (size_t)F_NS * F_STAGE + 16 * tid;
            auto seek = [&] {
                if (lt >= ntiles) return;
                int bz, m0, n0;
                tile(lt, bz, m0, n0);
                src = base + (size_t)bz * sb;
                r0 = isA ? m0 : n0;
            };
            auto load = [&](uint32_t slot) {
                if (lt < ntiles) {
                    part.load(raw + slot * F_RAWB, src, ld, rdim, g.K, r0, lkt * FK, w4, lane, vec);
                    if (++lkt == KT) { lkt = 0; lt += gridDim.x; seek(); }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            seek();
            for (int i = 0; i < F_RAW; i++) load(i);
            uint32_t it = 0;
            const uint32_t total = (uint32_t)((ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * KT;
            bool ok = true;
            float rmx[4] = {};
            int skt = 0, sli = 0;                // slice and tile stored
            auto step = [&] {
                const int s = it % F_NS;
                if (it >= F_NS && !(ok = warp_agrees(mbar_wait(&empty[s], ((it / F_NS) & 1) ^ 1)))) return;
                if (!(ok = warp_agrees(!*abort_flag))) return;
                asm volatile("cp.async.wait_group %0;" ::"n"(F_RAW - 1) : "memory");
                part.store(raw + it % F_RAW * F_RAWB, smem + (size_t)s * F_STAGE + (isA ? 0 : 3 * F_PART), w4, lane, rmx);
                if (++skt == KT) {
                    if (g.full_range) {
                        bool out = false;
                        #pragma unroll
                        for (int i = 0; i < 4; i++) out |= rmx[i] >= F_HUGE || (rmx[i] > 0.f && rmx[i] < F_TINY);
                        if (out) odd[sli % F_ODD] = sli + 1;
                        __threadfence_block();
                    }
                    #pragma unroll
                    for (int i = 0; i < 4; i++) rmx[i] = 0.f;
                    skt = 0;
                    sli++;
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive1(&full[s]);
                load(it % F_RAW);
                it++;
            };
            while (it < total && ok) step();
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            if (!ok) fail();
        };
        if (isA) produce(Part<!ACOL>(), g.A, g.sA, g.lda, g.M, vecA);
        else produce(Part<BKC>(), g.B, g.sB, g.ldb, g.N, vecB);
    } else if (warp >= F_LOAD + F_ACC) {
        regs_down<24>();
        if (warp == F_LOAD + F_ACC && lane == 0) {
            constexpr uint32_t IDESC = make_idesc_mn(1u, FM, FN);
            uint32_t it = 0;              // slices issued
            bool ok = true, issued = false;
            int li = 0;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, li++) {
                const int a = li & 1;
                if (li >= 2 && !(ok = mbar_wait(&lempty[a], ((li >> 1) & 1) ^ 1))) break;
                const uint32_t dl = tmem + 256 + 128 * a;
                for (int kt = 0; kt < KT && ok; kt++, it++) {
                    const int s = it % F_NS, hb = it & 1;
                    const uint32_t dh = tmem + 128 * hb;
                    if (it >= 2 && !(ok = mbar_wait(&hempty[hb], ((it >> 1) & 1) ^ 1))) break;
                    if (!(ok = mbar_wait(&full[s], (it / F_NS) & 1))) break;
                    if (*abort_flag) { ok = false; break; }
                    fence_after();
                    const uint32_t st = smem_addr(smem) + s * F_STAGE;
                    #pragma unroll
                    for (int ks = 0; ks < FK / 16; ks++) {
                        const uint32_t o = st + 2 * ks * F_LBO;
                        const uint64_t ah = f_desc(o), am = f_desc(o + F_PART), al = f_desc(o + 2 * F_PART);
                        const uint64_t bh = f_desc(o + 3 * F_PART), bm = f_desc(o + 4 * F_PART), bl = f_desc(o + 5 * F_PART);
                        mma_f16(dh, ah, bh, IDESC, ks != 0);
                        mma_f16(dl, am, bl, IDESC, (kt | ks) != 0);
                        mma_f16(dl, al, bm, IDESC, 1u);
                        mma_f16(dl, ah, bl, IDESC, 1u);
                        mma_f16(dl, al, bh, IDESC, 1u);
                        mma_f16(dl, am, bm, IDESC, 1u);
                        mma_f16(dl, ah, bm, IDESC, 1u);
                        mma_f16(dl, am, bh, IDESC, 1u);
                    }
                    issued = true;
                    mma_commit(&empty[s]);
                    mma_commit(&hfull[hb]);
                }
            }
            if (!ok) fail();
            if (issued) {   // every MMA issued has completed before the accumulators are freed
                mma_commit(drain);
                mbar_wait(drain, 0);
            }
        }
        __syncwarp();
    } else {
        regs_up<104>();
        const int quarter = warp & 3, half = (warp - F_LOAD) >> 2, row = quarter * 32 + lane;
        const uint32_t tl = tmem + ((uint32_t)(quarter * 32) << 16) + 64 * half;
        uint32_t it = 0;
        int li = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, li++) {
            float acc[4][16];
            #pragma unroll
            for (int h = 0; h < 4; h++)
                #pragma unroll
                for (int q = 0; q < 16; q++) acc[h][q] = 0.f;
            int bz, m0, n0;
            tile(t, bz, m0, n0);
            const int r = m0 + row;
            const float *D = g.epilogue == 2 && r < g.M ? g.D + (size_t)bz * g.sD + (size_t)r * g.ldd : nullptr;
            if (D) {   // the row's 256 bytes of D into L2 while the tile is multiplied
                const int c = n0 + 64 * half;
                if (c < g.N) asm volatile("prefetch.global.L2 [%0];" ::"l"(D + c));
                if (c + 32 < g.N) asm volatile("prefetch.global.L2 [%0];" ::"l"(D + c + 32));
            }
            for (int kt = 0; kt < KT; kt++, it++) {
                const int hb = it & 1;
                if (!(ok = warp_agrees(mbar_wait(&hfull[hb], (it >> 1) & 1) && !*abort_flag))) break;
                fence_after();
                #pragma unroll
                for (int h = 0; h < 4; h++) {
                    float v[16];
                    tmem_ld16(tl + 128 * hb + 16 * h, v);
                    #pragma unroll
                    for (int q = 0; q < 16; q++) acc[h][q] += v[q];
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive1(&hempty[hb]);
            }
            if (!ok) { fail(); break; }
            #pragma unroll
            for (int h = 0; h < 4; h++) {
                float v[16];
                tmem_ld16(tl + 256 + 128 * (li & 1) + 16 * h, v);
                #pragma unroll
                for (int q = 0; q < 16; q++) acc[h][q] += v[q];
            }
            const bool again = g.full_range && odd[li % F_ODD] == li + 1;
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive1(&lempty[li & 1]);
            if (r >= g.M) continue;
            if (again) {
                f_row_again<ACOL, BKC>(g, bz, r, n0 + 64 * half);
                continue;
            }
            const CirPhase ph = g.epilogue == 1 ? cir_phase(g.w[(size_t)bz * g.wstride + r] * g.dt_over_hbar) : CirPhase{};
            float *C = g.C + (size_t)bz * g.sC + (size_t)r * g.ldc;
            const int cb = n0 + 64 * half;
            #pragma unroll
            for (int h = 0; h < 4; h++) {
                const int c0 = cb + 16 * h;
                if (g.epilogue == 1)   // (re, im) pairs times exp(+i ph)
                    #pragma unroll
                    for (int q = 0; q < 16; q += 2) cir_rotate(ph, acc[h][q], acc[h][q + 1]);
                if (vecC && c0 + 16 <= g.N) {
                    float4 d[4];
                    if (D)
                        #pragma unroll
                        for (int q = 0; q < 4; q++) d[q] = *reinterpret_cast<const float4 *>(D + c0 + 4 * q);
                    #pragma unroll
                    for (int q = 0; q < 4; q++) {
                        float4 x = make_float4(acc[h][4 * q], acc[h][4 * q + 1], acc[h][4 * q + 2], acc[h][4 * q + 3]);
                        if (D) x = make_float4(d[q].x - x.x, d[q].y - x.y, d[q].z - x.z, d[q].w - x.w);   // C = D - A B
                        *reinterpret_cast<float4 *>(C + c0 + 4 * q) = x;
                    }
                } else {
                    #pragma unroll
                    for (int q = 0; q < 16; q++)
                        if (c0 + q < g.N) C[c0 + q] = D ? D[c0 + q] - acc[h][q] : acc[h][q];
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == F_LOAD + F_ACC) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
}

// ---- smaller products: FP32 SIMT.  Where the 128 x 128 tiles above leave most SMs idle or K gives them
// little to do, their start-up and read-out are most of the time (cir_gemm_form).

// four values at q, of which the first `have` exist (one load where the address allows it: of rows that are
// not aligned some still start on 16 bytes)
__device__ __forceinline__ bool at16(const float *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
__device__ __forceinline__ float4 simt_load4(const float *q, int have) {
    if (have >= 4 && at16(q)) return __ldg(reinterpret_cast<const float4 *>(q));
    return make_float4(have > 0 ? __ldg(q) : 0.f, have > 1 ? __ldg(q + 1) : 0.f, have > 2 ? __ldg(q + 2) : 0.f,
                       have > 3 ? __ldg(q + 3) : 0.f);
}
// row r, columns c .. c + 3 of a product: the phase or C = D - A B, stored
__device__ __forceinline__ void simt_store(const GemmArgs &g, int bz, int r, int c, float4 v, const CirPhase &ph) {
    float x[4] = {v.x, v.y, v.z, v.w};
    if (g.epilogue == 1) {   // (re, im) pairs times exp(+i ph)
        cir_rotate(ph, x[0], x[1]);
        cir_rotate(ph, x[2], x[3]);
    }
    float *C = g.C + (size_t)bz * g.sC + (size_t)r * g.ldc + c;
    const float *D = g.epilogue == 2 ? g.D + (size_t)bz * g.sD + (size_t)r * g.ldd + c : nullptr;
    if (c + 3 < g.N && at16(C) && at16(D)) {
        if (D) {
            const float4 d = *reinterpret_cast<const float4 *>(D);
            x[0] = d.x - x[0]; x[1] = d.y - x[1]; x[2] = d.z - x[2]; x[3] = d.w - x[3];
        }
        *reinterpret_cast<float4 *>(C) = make_float4(x[0], x[1], x[2], x[3]);
        return;
    }
    #pragma unroll
    for (int q = 0; q < 4; q++)
        if (c + q < g.N) C[q] = D ? D[q] - x[q] : x[q];
}
__device__ __forceinline__ CirPhase simt_phase(const GemmArgs &g, int bz, int r) {
    return g.epilogue == 1 ? cir_phase(g.w[(size_t)bz * g.wstride + r] * g.dt_over_hbar) : CirPhase{};
}

// The correlation terms of the propagated F (interleaved complex columns) from the patches that a
// thread holds: m(0) at its two complex columns, and a row's four values added to the sums.  150
// steps at n = 128: 3050 us with a launch of k_tcf a step, 2820 so.
struct TcfCols {
    float a[9], b[9];
    TcfCols() = default;
    __device__ __forceinline__ TcfCols(const TcfArgs &tc, int bz, int c) {
        const float *m = tc.m0 + (size_t)bz * tc.sm0;
        const int q = c >> 1;
        #pragma unroll
        for (int u = 0; u < 9; u++) {
            a[u] = q < tc.n ? __ldg(m + (size_t)u * tc.ldv + q) : 0.f;
            b[u] = q + 1 < tc.n ? __ldg(m + (size_t)u * tc.ldv + q + 1) : 0.f;
        }
    }
};
__device__ __forceinline__ void tcf_row(const TcfArgs &tc, int bz, int r, const TcfCols &m0, float4 v, Pair (&sum)[8]) {
    float pr[9], pi[9], c[9];
    const float *m = tc.mt + (size_t)bz * tc.smt + r;
    #pragma unroll
    for (int u = 0; u < 9; u++) {
        pr[u] = fmaf(v.z, m0.b[u], v.x * m0.a[u]);
        pi[u] = fmaf(v.w, m0.b[u], v.y * m0.a[u]);
        c[u] = __ldg(m + (size_t)u * tc.ldv);
    }
    tcf_sums(pr, pi, c, sum);
}

// Few tiles, bound by the chain of loads and sums along K: 32 x 32 tiles, SK groups of 64 threads (4 x 4
// outputs each) take every SK-th slice of 32 of K and meet in shared memory.
constexpr int SB = 32, SLD = SB + 4, SK = 4;

template <bool KC>
__device__ __forceinline__ void small_load(const float *p, int ld, int rdim, int kdim, int r0, int k0, int t, float4 (&v)[4]) {
    #pragma unroll
    for (int i = 0; i < 4; i++) {
        const int idx = t + 64 * i, o = idx >> 3, c4 = 4 * (idx & 7);
        const int r = r0 + (KC ? o : c4), k = k0 + (KC ? c4 : o);
        v[i] = simt_load4(KC ? p + (size_t)r * ld + k : p + (size_t)k * ld + r, KC ? (r < rdim ? kdim - k : 0) : (k < kdim ? rdim - r : 0));
    }
}
template <bool KC>
__device__ __forceinline__ void small_store(float *s, int t, const float4 (&v)[4]) {
    #pragma unroll
    for (int i = 0; i < 4; i++) {
        const int idx = t + 64 * i, o = idx >> 3, c4 = 4 * (idx & 7);
        if (KC) {
            s[c4 * SLD + o] = v[i].x; s[(c4 + 1) * SLD + o] = v[i].y;
            s[(c4 + 2) * SLD + o] = v[i].z; s[(c4 + 3) * SLD + o] = v[i].w;
        } else *reinterpret_cast<float4 *>(s + o * SLD + c4) = v[i];
    }
}

template <bool ACOL, bool BKC, bool TCF>
__global__ void __launch_bounds__(64 * SK) k_gemm_small(GemmArgs g, TcfArgs tc) {
    __shared__ __align__(16) float sm[SK][2][SB * SLD];
    const int bz = blockIdx.z, m0 = blockIdx.y * SB, n0 = blockIdx.x * SB;
    const float *A = g.A + (size_t)bz * g.sA, *B = g.B + (size_t)bz * g.sB;
    const int t = threadIdx.x & 63, grp = threadIdx.x >> 6;
    const int tx = 4 * (t & 7), ty = 4 * (t >> 3);
    auto group_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(grp + 1) : "memory"); };
    float acc[4][4] = {};
    float4 ra[4], rb[4];
    small_load<!ACOL>(A, g.lda, g.M, g.K, m0, SB * grp, t, ra);
    small_load<BKC>(B, g.ldb, g.N, g.K, n0, SB * grp, t, rb);
    small_store<!ACOL>(sm[grp][0], t, ra);
    small_store<BKC>(sm[grp][1], t, rb);
    group_sync();
    for (int k0 = SB * grp; k0 < g.K; k0 += SB * SK) {
        const int kn = k0 + SB * SK;
        if (kn < g.K) {
            small_load<!ACOL>(A, g.lda, g.M, g.K, m0, kn, t, ra);
            small_load<BKC>(B, g.ldb, g.N, g.K, n0, kn, t, rb);
        }
        const float *as = sm[grp][0] + ty, *bs = sm[grp][1] + tx;
        #pragma unroll 8
        for (int k = 0; k < SB; k++) {
            const float4 a4 = *reinterpret_cast<const float4 *>(as + k * SLD);
            const float4 b4 = *reinterpret_cast<const float4 *>(bs + k * SLD);
            const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
            #pragma unroll
            for (int i = 0; i < 4; i++)
                #pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (kn < g.K) {
            group_sync();
            small_store<!ACOL>(sm[grp][0], t, ra);
            small_store<BKC>(sm[grp][1], t, rb);
        }
        group_sync();
    }
    // the first group adds the others' sums
    float *part = sm[grp][0];
    #pragma unroll
    for (int i = 0; i < 4; i++) *reinterpret_cast<float4 *>(part + (ty + i) * SLD + tx) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    __syncthreads();
    if (grp) return;
    #pragma unroll
    for (int q = 1; q < SK; q++)
        #pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 v = *reinterpret_cast<const float4 *>(sm[q][0] + (ty + i) * SLD + tx);
            acc[i][0] += v.x; acc[i][1] += v.y; acc[i][2] += v.z; acc[i][3] += v.w;
        }
    Pair sum[8] = {};
    const TcfCols mc = TCF ? TcfCols(tc, bz, n0 + tx) : TcfCols();
    #pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = m0 + ty + i;
        if (r >= g.M) continue;
        const float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        if (TCF) tcf_row(tc, bz, r, mc, v, sum);
        simt_store(g, bz, r, n0 + tx, v, simt_phase(g, bz, r));
    }
    if (TCF) {
        __shared__ double psum[8];
        const double v = tcf_reduce(sum);
        if (t >= 32 && (t & 3) == 0) psum[(t & 31) >> 2] = v;
        group_sync();
        if (t < 32) tcf_add(__shfl_sync(0xffffffffu, v, (4 * t) & 31) + (t < 8 ? psum[t] : 0.0), tc.out + (size_t)bz * tc.sout);
    }
}

// Many tiles: T x T tiles of 256 threads, 4 x 4 outputs in each quarter of 64, TK of K at a time, double
// buffered: 64 x 64 x 16 and 128 x 128 x 8.
template <int T, int TK, bool KC>
__device__ __forceinline__ float4 tile_load(const float *p, int ld, int rdim, int kdim, int r0, int k0) {
    constexpr int W = KC ? TK / 4 : T / 4;
    const int t = threadIdx.x, r = r0 + (KC ? t / W : 4 * (t % W)), k = k0 + (KC ? 4 * (t % W) : t / W);
    return simt_load4(KC ? p + (size_t)r * ld + k : p + (size_t)k * ld + r, KC ? (r < rdim ? kdim - k : 0) : (k < kdim ? rdim - r : 0));
}
template <int T, int TK, bool KC>
__device__ __forceinline__ void tile_store(float (*s)[T], float4 v) {
    constexpr int W = KC ? TK / 4 : T / 4;
    const int t = threadIdx.x;
    if (KC) {
        const int r = t / W, k = 4 * (t % W);
        s[k][r] = v.x; s[k + 1][r] = v.y; s[k + 2][r] = v.z; s[k + 3][r] = v.w;
    } else *reinterpret_cast<float4 *>(&s[t / W][4 * (t % W)]) = v;
}

template <int T, int TK, bool ACOL, bool BKC, bool TCF>
__global__ void __launch_bounds__(256) k_gemm_tile(GemmArgs g, TcfArgs tc) {
    static_assert(T * TK == 1024, "four values a thread");
    constexpr int Q = T / 64;
    __shared__ __align__(16) float As[2][TK][T], Bs[2][TK][T];
    const int bz = blockIdx.z, m0 = blockIdx.y * T, n0 = blockIdx.x * T;
    const float *A = g.A + (size_t)bz * g.sA, *B = g.B + (size_t)bz * g.sB;
    const int tx = 4 * (threadIdx.x % 16), ty = 4 * (threadIdx.x / 16);
    float acc[4 * Q][4 * Q] = {};
    float4 ra = tile_load<T, TK, !ACOL>(A, g.lda, g.M, g.K, m0, 0), rb = tile_load<T, TK, BKC>(B, g.ldb, g.N, g.K, n0, 0);
    tile_store<T, TK, !ACOL>(As[0], ra);
    tile_store<T, TK, BKC>(Bs[0], rb);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < g.K; k0 += TK) {
        const bool more = k0 + TK < g.K;
        if (more) {
            ra = tile_load<T, TK, !ACOL>(A, g.lda, g.M, g.K, m0, k0 + TK);
            rb = tile_load<T, TK, BKC>(B, g.ldb, g.N, g.K, n0, k0 + TK);
        }
        #pragma unroll
        for (int k = 0; k < TK; k++) {
            float a[4 * Q], b[4 * Q];
            #pragma unroll
            for (int q = 0; q < Q; q++) {
                *reinterpret_cast<float4 *>(a + 4 * q) = *reinterpret_cast<const float4 *>(&As[buf][k][ty + 64 * q]);
                *reinterpret_cast<float4 *>(b + 4 * q) = *reinterpret_cast<const float4 *>(&Bs[buf][k][tx + 64 * q]);
            }
            #pragma unroll
            for (int i = 0; i < 4 * Q; i++)
                #pragma unroll
                for (int j = 0; j < 4 * Q; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (more) {
            tile_store<T, TK, !ACOL>(As[buf ^ 1], ra);
            tile_store<T, TK, BKC>(Bs[buf ^ 1], rb);
        }
        __syncthreads();
        buf ^= 1;
    }
    Pair sum[8] = {};
    const TcfCols mc = TCF ? TcfCols(tc, bz, n0 + tx) : TcfCols();
    #pragma unroll
    for (int i = 0; i < 4 * Q; i++) {
        const int r = m0 + ty + 64 * (i / 4) + i % 4;
        if (r >= g.M) continue;
        const CirPhase ph = simt_phase(g, bz, r);
        #pragma unroll
        for (int q = 0; q < Q; q++) {
            const float4 v = make_float4(acc[i][4 * q], acc[i][4 * q + 1], acc[i][4 * q + 2], acc[i][4 * q + 3]);
            if (TCF) tcf_row(tc, bz, r, mc, v, sum);
            simt_store(g, bz, r, n0 + tx + 64 * q, v, ph);
        }
    }
    if (TCF) {
        static_assert(!TCF || Q == 1, "one column group a thread");
        __shared__ double psum[8][8];
        const int lane = threadIdx.x & 31;
        const double v = tcf_reduce(sum);
        if ((lane & 3) == 0) psum[threadIdx.x >> 5][lane >> 2] = v;
        __syncthreads();
        if (threadIdx.x < 32) {
            double s = 0.0;
            if (lane < 8)
                #pragma unroll
                for (int w = 0; w < 8; w++) s += psum[w][lane];
            tcf_add(s, tc.out + (size_t)bz * tc.sout);
        }
    }
}

__global__ void k_identity(float *F, int n, int ldf, long long sF) {
    float *f = F + (size_t)blockIdx.y * sF;
    const int r = blockIdx.x;
    for (int c = threadIdx.x; c < 2 * n; c += blockDim.x) f[(size_t)r * ldf + c] = (c == 2 * r) ? 1.f : 0.f;
}

}  // namespace

cudaError_t cir_launch_gemm(const GemmArgs &g, int batch, cudaStream_t s, int *launches, const TcfArgs *tcf, bool *fused) {
    if ((g.epilogue == 1 && (g.N & 1)) || (g.epilogue == 2 && !g.D) || (g.a_colmajor && g.b_kmajor)) return cudaErrorInvalidValue;
    if (batch < 1 || batch > 65535 || g.M < 1 || g.N < 1 || g.K < 1) return cudaErrorInvalidValue;
    const int tiles_n = (g.N + FN - 1) / FN;
    const long long mn = (long long)tiles_n * ((g.M + FM - 1) / FM), nt = mn * batch;
    if (nt > INT_MAX) return cudaErrorInvalidValue;
    auto vec = [&](const float *p, int ld, long long st) {
        return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && (ld & 3) == 0 && (batch == 1 || (st & 3) == 0);
    };
    const bool va = vec(g.A, g.lda, g.sA), vb = vec(g.B, g.ldb, g.sB),
               vc = vec(g.C, g.ldc, g.sC) && (g.epilogue != 2 || vec(g.D, g.ldd, g.sD));
    const int sms = cir_sms();
    const CirGemmForm form = cir_gemm_form(g.M, g.N, g.K, batch, g.epilogue, va && vb, vc, sms);
    if (form != CIR_GEMM_TC) {
        const bool fuse = tcf && g.a_colmajor && g.epilogue == 0 && form != CIR_GEMM_TILE128;
        const TcfArgs tc = tcf ? *tcf : TcfArgs{};
        const int T = form == CIR_GEMM_SMALL ? SB : form == CIR_GEMM_TILE64 ? 64 : 128;
        const dim3 grid((g.N + T - 1) / T, (g.M + T - 1) / T, batch);
        auto go = [&](auto small, auto t64, auto t128) {
            if (form == CIR_GEMM_SMALL) small<<<grid, 64 * SK, 0, s>>>(g, tc);
            else if (form == CIR_GEMM_TILE64) t64<<<grid, 256, 0, s>>>(g, tc);
            else t128<<<grid, 256, 0, s>>>(g, tc);
        };
        if (fuse) {
            go(k_gemm_small<true, false, true>, k_gemm_tile<64, 16, true, false, true>, k_gemm_tile<128, 8, true, false, false>);
            *fused = true;
        } else if (g.a_colmajor)
            go(k_gemm_small<true, false, false>, k_gemm_tile<64, 16, true, false, false>, k_gemm_tile<128, 8, true, false, false>);
        else if (g.b_kmajor)
            go(k_gemm_small<false, true, false>, k_gemm_tile<64, 16, false, true, false>, k_gemm_tile<128, 8, false, true, false>);
        else
            go(k_gemm_small<false, false, false>, k_gemm_tile<64, 16, false, false, false>, k_gemm_tile<128, 8, false, false, false>);
        if (launches) *launches += 1;
        return cudaGetLastError();
    }
    const int grid = (int)std::min<long long>(nt, sms);
    auto go = [&](auto kern) {
        cudaError_t e = cir_allow_smem(kern, F_SMEM);
        if (e != cudaSuccess) return e;
        kern<<<grid, F_NT, F_SMEM, s>>>(g, tiles_n, (int)mn, (int)nt, va, vb, vc, g.err);
        return cudaGetLastError();
    };
    const cudaError_t e = g.a_colmajor ? go(k_gemm<true, false>) : g.b_kmajor ? go(k_gemm<false, true>) : go(k_gemm<false, false>);
    if (e == cudaSuccess && launches) *launches += 1;
    return e;
}

cudaError_t cir_launch_identity(float *F, int n, int ldf, long long sF, int batch, cudaStream_t s, int *launches) {
    k_identity<<<dim3(n, batch), 256, 0, s>>>(F, n, ldf, sF);
    if (launches) *launches += 1;
    return cudaGetLastError();
}
