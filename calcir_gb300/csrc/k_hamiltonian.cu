// Field projection, spectroscopic maps and the exciton Hamiltonian of a batch of frames.
//
// k_chromophore: the field at H_c sums the H1/H2 (+0.52) and M (-1.04) charges of every other
// molecule whose O lies within 0.7831 nm of H_c (minimum image), projected on the OH unit vector
// (get_eproj_GPU, calcIR.cu:1020-1168); then the maps, the per-chromophore table, the dipole and
// the polarisability (calcIR.cu:1256-1304).  The frame's molecules are staged in shared memory.
// First a warp tests the molecules for each of its chromophores, a molecule per lane, and keeps
// the outcomes; then the charges of the molecules inside (a fifth of a 343-molecule box) are
// summed.  The terms nearly cancel; they are added in the molecules' order, as the reference's
// loop adds them.  Two forms, bound by instruction issue and by latency:
//   many chromophores (WIDE false): a thread per chromophore runs over its own set bits, so that
//     neighbours with different molecules inside work side by side;
//   few (WIDE): a warp per chromophore forms 32 molecules' terms at a time and adds them up
//     by shuffles.
// Testing and summing in one loop, a thread per chromophore, took the charges' path for every
// molecule that any of a warp's chromophores had inside: 472 us for 200 frames of 343 molecules
// against 273, and 56 us for one frame of 64 against 10 (38 by the form for many).
//
// k_hmatrix: 32x32 tiles of H (get_kappa_GPU, calcIR.cu:1306-1402).  A pair's value does not
// depend on the order of the two, so H is exactly symmetric; both triangles are written with
// coalesced stores.
#include "cir_device.cuh"
#include "cir_plan.h"

#include <cmath>

namespace {

constexpr int CHROM_NT = 64;        // threads of a block: 64 chromophores, or 2 (WIDE)
constexpr int MOL_F = 12;           // floats of a staged molecule: H1, H2, M, O

// (the roundings are written out wherever the compiler could contract two copies of the code
// differently: both forms of k_chromophore give the same bits)
__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz) {
    return fmaf(az, bz, fmaf(ax, bx, __fmul_rn(ay, by)));
}

// charge over distance cubed, and the distance vector (bohr) from a site to H
__device__ __forceinline__ float4 site_term(float hx, float hy, float hz, float sx, float sy, float sz, float q, float bx,
                                            float by, float bz, float rx, float ry, float rz) {
    float qx = hx - sx, qy = hy - sy, qz = hz - sz;
    cir_mi3(qx, qy, qz, bx, by, bz, rx, ry, rz);
    qx = qx * CIR_BOHR_NM;
    qy = qy * CIR_BOHR_NM;
    qz = qz * CIR_BOHR_NM;
    const float rr = sqrtf(dot3(qx, qy, qz, qx, qy, qz));
    return make_float4(q / (rr * rr * rr), qx, qy, qz);
}

// cut2: the largest float whose square root (rounded to nearest) is at most the cutoff, so the
// test on the sum of squares decides as cir_mag3 does
template <bool WIDE>
__global__ void __launch_bounds__(CHROM_NT) k_chromophore(BuildArgs a, float cut2) {
    constexpr int PW = WIDE ? 1 : 32;                   // chromophores of a warp
    extern __shared__ __align__(16) float sm_mol[];     // [nmol][MOL_F], then the bits
    const int W = (a.nmol + 31) / 32, WL = W | 1;       // words of a chromophore's bits (odd stride)
    unsigned *bits = reinterpret_cast<unsigned *>(sm_mol + (size_t)a.nmol * MOL_F);
    const int f = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *x = a.xyz + (size_t)f * a.natoms * 3;
    const float bx = a.box[3 * f], by = a.box[3 * f + 1], bz = a.box[3 * f + 2];
    const float rx = 1.f / bx, ry = 1.f / by, rz = 1.f / bz;
    const bool hasm = a.natom_mol >= 4;
    for (int m = tid; m < a.nmol; m += CHROM_NT) {
        const float *mo = x + (size_t)m * a.natom_mol * 3;
        float *o = sm_mol + m * MOL_F;
        #pragma unroll
        for (int q = 0; q < 6; q++) o[q] = mo[3 + q];
        float mx = 0.f, my = 0.f, mz = 0.f;
        if (hasm) {
            mx = mo[9]; my = mo[10]; mz = mo[11];
            if (a.imodel != 0) {   // move M to the TIP4P distance (calcIR.cu:1131-1146)
                const float dx = cir_mi(mx - mo[0], bx), dy = cir_mi(my - mo[1], by), dz = cir_mi(mz - mo[2], bz);
                const float r = sqrtf(dot3(dx, dy, dz, dx, dy, dz));
                mx = __fadd_rn(mo[0], CIR_OM_TIP4P * dx / r);
                my = __fadd_rn(mo[1], CIR_OM_TIP4P * dy / r);
                mz = __fadd_rn(mo[2], CIR_OM_TIP4P * dz / r);
            }
        }
        o[6] = mx; o[7] = my; o[8] = mz;
        o[9] = mo[0]; o[10] = mo[1]; o[11] = mo[2];
    }
    __syncthreads();
    const int c0 = (blockIdx.x * (CHROM_NT / 32) + warp) * PW, nc = min(PW, a.n - c0);   // the warp's chromophores
    if (nc <= 0) return;
    for (int m0 = 0; m0 < a.nmol; m0 += 32) {
        const int m = m0 + lane;
        float ox = 0.f, oy = 0.f, oz = 0.f;
        if (m < a.nmol) { ox = sm_mol[m * MOL_F + 9]; oy = sm_mol[m * MOL_F + 10]; oz = sm_mol[m * MOL_F + 11]; }
        unsigned mine = 0;
        #pragma unroll 4
        for (int q = 0; q < nc; q++) {
            const int n = (c0 + q) / a.nchrom_mol;
            const float *h = sm_mol + n * MOL_F + 3 * ((c0 + q) % 2);   // chrom%2 selects HW1/HW2 (calcIR.cu:1061-1072)
            float dx = ox - h[0], dy = oy - h[1], dz = oz - h[2];
            cir_mi3(dx, dy, dz, bx, by, bz, rx, ry, rz);
            // calcIR.cu:1106-1113 (a NaN distance is not beyond the cutoff)
            const bool in = !(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)) > cut2);
            const unsigned b = __ballot_sync(0xffffffffu, in && m < a.nmol && m != n);
            if (lane == q) mine = b;
        }
        if (lane < PW) bits[(warp * PW + lane) * WL + m0 / 32] = mine;
    }
    __syncwarp();
    const int c = WIDE ? c0 : c0 + lane;
    if (c >= a.n) return;
    const unsigned *my = bits + (WIDE ? warp : tid) * WL;
    const float *mo = sm_mol + (c / a.nchrom_mol) * MOL_F;
    const int hoff = 3 * (c % 2);
    const float hx = mo[hoff], hy = mo[hoff + 1], hz = mo[hoff + 2];
    const float ox = mo[9], oy = mo[10], oz = mo[11];
    float ex = 0.f, ey = 0.f, ez = 0.f;
    if (WIDE) {
        for (int w = 0; w < W; w++) {
            const unsigned set = my[w];
            if (set == 0) continue;
            float4 t[3];
            const int m = 32 * w + lane;
            #pragma unroll
            for (int s = 0; s < 3; s++) {
                t[s] = make_float4(0.f, 0.f, 0.f, 0.f);
                if ((set >> lane) & 1u && (s < 2 || hasm)) {
                    const float *q = sm_mol + m * MOL_F + 3 * s;
                    t[s] = site_term(hx, hy, hz, q[0], q[1], q[2], s < 2 ? CIR_QH : -CIR_QM, bx, by, bz, rx, ry, rz);
                }
            }
            for (unsigned b = set; b; b &= b - 1) {
                const int l = __ffs(b) - 1;
                #pragma unroll
                for (int s = 0; s < 3; s++) {
                    if (s == 2 && !hasm) break;
                    const float s3 = __shfl_sync(0xffffffffu, t[s].x, l);
                    ex = fmaf(s3, __shfl_sync(0xffffffffu, t[s].y, l), ex);
                    ey = fmaf(s3, __shfl_sync(0xffffffffu, t[s].z, l), ey);
                    ez = fmaf(s3, __shfl_sync(0xffffffffu, t[s].w, l), ez);
                }
            }
        }
        if (lane) return;
    } else {
        unsigned b = my[0];
        for (int w = 0;;) {
            while (b == 0 && ++w < W) b = my[w];
            if (b == 0) break;
            const float4 *q4 = reinterpret_cast<const float4 *>(sm_mol + (32 * w + __ffs(b) - 1) * MOL_F);
            b &= b - 1;
            const float4 s0 = q4[0], s1 = q4[1];
            const float site[9] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w, reinterpret_cast<const float *>(q4)[8]};
            #pragma unroll
            for (int s = 0; s < 3; s++) {
                if (s == 2 && !hasm) break;
                const float4 t = site_term(hx, hy, hz, site[3 * s], site[3 * s + 1], site[3 * s + 2],
                                           s < 2 ? CIR_QH : -CIR_QM, bx, by, bz, rx, ry, rz);
                ex = fmaf(t.x, t.y, ex);
                ey = fmaf(t.x, t.z, ey);
                ez = fmaf(t.x, t.w, ez);
            }
        }
    }
    float ux = cir_mi(hx - ox, bx), uy = cir_mi(hy - oy, by), uz = cir_mi(hz - oz, bz);
    {
        const float r = sqrtf(dot3(ux, uy, uz, ux, uy, uz));
        ux /= r; uy /= r; uz /= r;
    }
    const float E = dot3(ex, ey, ez, ux, uy, uz);
    const CirMaps &mp = a.maps;
    const float w = fmaf(__fmul_rn(mp.w[2], E), E, fmaf(mp.w[1], E, mp.w[0]));
    const float xm = fmaf(mp.x[1], w, mp.x[0]);
    const float pm = fmaf(mp.p[1], w, mp.p[0]);
    const float mup = fmaf(__fmul_rn(mp.mup[2], E), E, fmaf(mp.mup[1], E, mp.mup[0]));
    // transition dipole position, each coordinate wrapped by minImage (calcIR.cu:1288-1291)
    const float tx = cir_mi(fmaf(CIR_TDM_OFFSET, ux, ox), bx);
    const float ty = cir_mi(fmaf(CIR_TDM_OFFSET, uy, oy), by);
    const float tz = cir_mi(fmaf(CIR_TDM_OFFSET, uz, oz), bz);
    float *ct = a.ct + (size_t)f * CT_NROW * a.ld;
    ct[CT_E * a.ld + c] = E;
    ct[CT_W * a.ld + c] = w;
    ct[CT_X * a.ld + c] = xm;
    ct[CT_P * a.ld + c] = pm;
    ct[CT_MUP * a.ld + c] = mup;
    ct[CT_UX * a.ld + c] = ux; ct[CT_UY * a.ld + c] = uy; ct[CT_UZ * a.ld + c] = uz;
    ct[CT_TX * a.ld + c] = tx; ct[CT_TY * a.ld + c] = ty; ct[CT_TZ * a.ld + c] = tz;
    if (a.eproj) a.eproj[(size_t)f * a.n + c] = E;
    if (a.dip) {   // calcIR.cu:1294-1296
        float *d = a.dip + (size_t)f * a.dip_fstride;
        const float s = mup * xm;
        d[c] = ux * s; d[a.ldv + c] = uy * s; d[2 * a.ldv + c] = uz * s;
    }
    if (a.pol) {   // calcIR.cu:1299-1304
        float *p = a.pol + (size_t)f * a.pol_fstride;
        p[c] = fmaf(__fmul_rn(4.6f, ux), ux, 1.0f) * xm;
        p[a.ldv + c] = fmaf(__fmul_rn(4.6f, uy), uy, 1.0f) * xm;
        p[2 * a.ldv + c] = fmaf(__fmul_rn(4.6f, uz), uz, 1.0f) * xm;
        p[3 * a.ldv + c] = 4.6f * ux * uy * xm;
        p[4 * a.ldv + c] = 4.6f * uy * uz * xm;
        p[5 * a.ldv + c] = 4.6f * uz * ux * xm;
    }
}

struct Chrom {
    float E, w, x, p, xm, ux, uy, uz, tx, ty, tz;   // xm = x mu'
    int mol;
    float pad;      // an odd stride: neighbouring lanes read different banks
};

// Symmetric in its two chromophores to the last bit: every product and sum pairs them, and each
// rounding is written out, so that no two places in the code contract it differently.
__device__ __forceinline__ float pair_coupling(const Chrom &lo, const Chrom &hi, float bx, float by, float bz,
                                               float rx, float ry, float rz, const CirMaps &mp, int ispecies) {
    if (ispecies == 1 || ispecies == 2) return 0.f;       // HOD: no coupling (calcIR.cu:1334, 1348)
    if (lo.mol == hi.mol)                                   // intramolecular map (calcIR.cu:1339)
        return fmaf(fmaf(mp.wi[1], __fadd_rn(lo.E, hi.E), mp.wi[0]), __fmul_rn(lo.x, hi.x),
                    __fmul_rn(mp.wi[2], __fmul_rn(lo.p, hi.p)));
    // transition dipole coupling (calcIR.cu:1352-1399)
    float dx = lo.tx - hi.tx, dy = lo.ty - hi.ty, dz = lo.tz - hi.tz;
    cir_mi3(dx, dy, dz, bx, by, bz, rx, ry, rz);
    const float ri = cir_rsqrt(dot3(dx, dy, dz, dx, dy, dz));
    const float uu = dot3(lo.ux, lo.uy, lo.uz, hi.ux, hi.uy, hi.uz);
    const float un = __fmul_rn(dot3(lo.ux, lo.uy, lo.uz, dx, dy, dz), ri);
    const float vn = __fmul_rn(dot3(hi.ux, hi.uy, hi.uz, dx, dy, dz), ri);
    const float k = __fmul_rn(fmaf(-3.f, __fmul_rn(un, vn), uu), __fmul_rn(__fmul_rn(ri, ri), ri));
    return __fmul_rn(__fmul_rn(k, __fmul_rn(lo.xm, hi.xm)), CIR_TDC);
}

constexpr int HT = 32;   // tile edge

__device__ __forceinline__ void load_chrom(const BuildArgs &a, const float *ct, int i0, Chrom *out, int tid) {
    float *o = reinterpret_cast<float *>(out);
    for (int i = tid; i < HT * 11; i += HT * 8) {
        const int q = i / HT, l = i % HT, idx = i0 + l;
        // table row of the field (x mu' is formed below)
        const int row = q == 0 ? CT_E : q == 1 ? CT_W : q == 2 ? CT_X : q == 3 ? CT_P : q == 4 ? CT_MUP : CT_UX + q - 5;
        float v = idx < a.n ? ct[row * a.ld + idx] : 0.f;
        if (q == 4 && idx < a.n) v = ct[CT_X * a.ld + idx] * v;
        o[l * (sizeof(Chrom) / 4) + q] = v;
    }
    if (tid < HT) out[tid].mol = (i0 + tid) / a.nchrom_mol;
}

// A tile above the diagonal is computed once and written twice: directly and, through shared
// memory, transposed into its mirror tile.  Block (x, y): tile row y, tile columns y + per x ..
// (blocks past the last column return).
__global__ void __launch_bounds__(HT * 8) k_hmatrix(BuildArgs a, int per) {
    const int nt = (a.n + HT - 1) / HT, ty = blockIdx.y, tx0 = ty + per * blockIdx.x;
    if (tx0 >= nt) return;
    __shared__ Chrom rows[HT], cols[2][HT];
    __shared__ float tile[HT][HT + 1];
    const int f = blockIdx.z;
    const int r0 = ty * HT;
    const float *ct = a.ct + (size_t)f * CT_NROW * a.ld;
    const int tid = threadIdx.y * HT + threadIdx.x;
    load_chrom(a, ct, r0, rows, tid);
    load_chrom(a, ct, tx0 * HT, cols[0], tid);
    const float bx = a.box[3 * f], by = a.box[3 * f + 1], bz = a.box[3 * f + 2];
    const float rx = 1.f / bx, ry = 1.f / by, rz = 1.f / bz;
    float *H = a.H + (size_t)f * a.n * a.ldh;
    for (int t = 0; t < per && tx0 + t < nt; t++) {
        __syncthreads();      // this tile's columns are in, the last tile's mirror is out
        if (t + 1 < per && tx0 + t + 1 < nt) load_chrom(a, ct, (tx0 + t + 1) * HT, cols[(t + 1) & 1], tid);
        const int c0 = (tx0 + t) * HT, c = c0 + threadIdx.x;
        const bool mirror = tx0 + t > ty;
        const Chrom cc = cols[t & 1][threadIdx.x];
        #pragma unroll
        for (int i = 0; i < HT / 8; i++) {
            const int rl = threadIdx.y + 8 * i;
            const int r = r0 + rl;
            if (r >= a.n || c >= a.n) continue;
            float h;
            if (r == c) h = rows[rl].w - a.avef;               // calcIR.cu:1322-1328
            else h = pair_coupling(rows[rl], cc, bx, by, bz, rx, ry, rz, a.maps, a.ispecies);
            H[(size_t)r * a.ldh + c] = h;
            tile[rl][threadIdx.x] = h;
        }
        if (!mirror) continue;
        __syncthreads();
        // the mirror tile: H[c0 + j][r0 + l] = H[r0 + l][c0 + j], written along r0 + l
        const int rm = r0 + threadIdx.x;
        #pragma unroll
        for (int i = 0; i < HT / 8; i++) {
            const int jl = threadIdx.y + 8 * i, cm = c0 + jl;
            if (cm < a.n && rm < a.n) H[(size_t)cm * a.ldh + rm] = tile[threadIdx.x][jl];
        }
    }
}

}  // namespace

cudaError_t cir_launch_build(const BuildArgs &a, int nframes, cudaStream_t s, int *launches) {
    static const float cut2 = [] {
        float s = CIR_CUTOFF * CIR_CUTOFF;
        while (sqrtf(s) <= CIR_CUTOFF) s = nextafterf(s, 2.f);
        while (sqrtf(s) > CIR_CUTOFF) s = nextafterf(s, 0.f);
        return s;
    }();
    const bool wide = cir_build_wide(a.n, a.nmol, nframes, cir_sms());
    const int per_block = wide ? CHROM_NT / 32 : CHROM_NT;
    auto kern = wide ? k_chromophore<true> : k_chromophore<false>;
    const size_t smem = sizeof(float) * MOL_F * (size_t)a.nmol + sizeof(unsigned) * per_block * (size_t)(((a.nmol + 31) / 32) | 1);
    cudaError_t e = cir_allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    kern<<<dim3((a.n + per_block - 1) / per_block, nframes), CHROM_NT, smem, s>>>(a, cut2);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int nt = (a.n + HT - 1) / HT;
    // tiles of a block: four share the loads of their row where that leaves blocks enough, one
    // where latency counts (a frame of 64 molecules: 5 us against 10)
    const int per = (long long)nt * nt / 8 * nframes >= 2048 ? 4 : 1;
    dim3 g2((nt + per - 1) / per, nt, nframes);
    k_hmatrix<<<g2, dim3(HT, 8), 0, s>>>(a, per);
    if (launches) *launches += 2;
    return cudaGetLastError();
}
