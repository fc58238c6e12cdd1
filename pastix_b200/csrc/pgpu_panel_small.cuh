// Panels of cblks of at most 32 columns (kernels/core_zpotrfsp.c:68
// core_zpotf2sp and its LU / LDL kin, and the panel TRSM of their rows,
// kernels/core_ztrsmsp.c:71): one warp per cblk.
#pragma once

#include "pgpu_common.cuh"
#include "pgpu_panel.cuh"

namespace pgpu {

// 16-byte shared-memory load of consecutive elements.
template <typename T>
__device__ __forceinline__ void wp_lds16(const T *p, T (&v)[16 / sizeof(T)]) {
    const uint4 u = *reinterpret_cast<const uint4 *>(p);
    memcpy(v, &u, 16);
}

// Row solve against the factorized tile with the row in registers (fully
// unrolled, so x stays out of local memory):
//   x[j] = (x[j] - sum_{l<j} x[l] op(C[j][l])) * (UNIT ? 1 : rdiag[j])
// in increasing l, C row-major with 16-byte rows (ldc), read as broadcast
// vectors.  C = the tile's lower part (LL^h, LDL rows; LU row block, unit),
// or the transposed upper part (LU rows: x U = a).
template <typename T, bool CJ, bool UNIT>
__device__ __forceinline__ void wp_solve_rows(T (&x)[PB], const T *C, int ldc, const T *rdiag, int nb) {
    constexpr int VK = 16 / sizeof(T);
#pragma unroll
    for (int j = 0; j < PB; j++)
        if (j < nb) {
            T s = x[j];
#pragma unroll
            for (int l0 = 0; l0 < j; l0 += VK) {
                T c[VK];
                wp_lds16<T>(C + j * ldc + l0, c);
#pragma unroll
                for (int v = 0; v < VK; v++)
                    if (l0 + v < j) s -= x[l0 + v] * cj<CJ>(c[v]);
            }
            x[j] = UNIT ? s : s * rdiag[j];
        }
}

// ---------------------------------------------------------------------------
// Cblks of at most 32 columns (the leaves, ~10^5-10^6 of them in the
// batched 2D problems): one warp per cblk.  The w x w diagonal block is one
// tile, factorized by the warp in shared memory (warp_factor_tile_smem: with
// every warp of the SM in it, the fully unrolled register form misses in the
// instruction cache), and the panel rows below
// it are solved one lane per row with the row in registers -- the same
// operations as k_panel_factor for such a cblk, without a 256-thread CTA per
// leaf.
// Shared memory per warp: X [PB][PB + VK] (the tile with row length PBL
// while it is factorized, then TA, the tile as 16-byte rows for the row
// solves), TB [PB][PB + VK] for LU, 1 / op(diagonal) [PB].
// ---------------------------------------------------------------------------
constexpr int PS_WARPS = 8;
template <typename T>
__host__ __device__ constexpr int ps_warp_elems(bool lu) { return (lu ? 2 : 1) * PB * (PB + 16 / (int)sizeof(T)) + PB; }
template <typename T>
constexpr int ps_smem_bytes(bool lu) { return PS_WARPS * ps_warp_elems<T>(lu) * (int)sizeof(T); }

template <typename T, int MODE>
__global__ void __launch_bounds__(PS_WARPS * 32) k_panel_small(Meta m, const int2 *__restrict__ jobs, int njobs,
                                                               T *__restrict__ coefL, T *__restrict__ coefU,
                                                               const double *critp, int fuse_rows, Status *st) {
    typedef typename real_of<T>::type R;
    constexpr bool LU = (MODE == FM_GETRF);
    constexpr bool LDL = fm_ldl(MODE);
    constexpr bool CJ = fm_conj(MODE);
    constexpr int VK = 16 / sizeof(T), LDT = PB + VK;
    static_assert(LDT >= PBL, "the tile fits in TA");
    extern __shared__ __align__(16) unsigned char ps_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x * PS_WARPS + warp;
    if (q >= njobs) return;                        // whole warps; warp-level synchronization only
    T *TA = reinterpret_cast<T *>(ps_raw) + (size_t)warp * ps_warp_elems<T>(LU);
    T *tile = TA;
    T *TB = TA + PB * LDT;
    T *rdiag = TA + (LU ? 2 : 1) * PB * LDT;
    const int c = jobs[q].x;
    const int w = m.width[c], h = m.height[c], ld = m.ld[c];
    const int rows = (h <= fuse_rows) ? h : w;
    T *A = coefL + m.coefoff[c];
    T *AU = coefU + m.coefoff[c];
    const R crit = R(*critp);
    int npiv = 0, nneg = 0, nbad = 0;
    if (lane < w)
        for (int i = 0; i < w; i++) tile[i * PBL + lane] = A[(int64_t)i * ld + lane];
    __syncwarp();
    warp_factor_tile_smem<T, MODE>(tile, w, crit, npiv, nneg, nbad);
    __syncwarp();
    if (lane < w) {
        for (int i = 0; i < w; i++)
            if (LU || lane <= i) A[(int64_t)i * ld + lane] = tile[i * PBL + lane];
        const T d = tile[lane * PBL + lane];
        rdiag[lane] = T(1) / (MODE == FM_POTRF ? cj<CJ>(d) : d);
        if (LU)
            for (int j = 0; j < w; j++) TB[j * LDT + lane] = tile[j * PBL + lane];
    }
    {   // TA over the tile's storage: the whole tile goes through registers
        T v[PB];
#pragma unroll
        for (int j = 0; j < PB; j++)
            v[j] = (lane < w && j < w) ? (LU ? tile[lane * PBL + j] : tile[j * PBL + lane]) : T(0);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < PB; j++)
            if (lane < w && j < w) TA[j * LDT + lane] = v[j];
    }
    __syncwarp();
    for (int r = w + lane; r < rows; r += 32) {
        T x[PB];
        T *row = A + (int64_t)r * ld;
#pragma unroll
        for (int j = 0; j < PB; j++) x[j] = (j < w) ? row[j] : T(0);
        if (LU) wp_solve_rows<T, false, false>(x, TA, LDT, rdiag, w);
        else if (LDL) wp_solve_rows<T, CJ, true>(x, TA, LDT, rdiag, w);
        else wp_solve_rows<T, CJ, false>(x, TA, LDT, rdiag, w);
#pragma unroll
        for (int j = 0; j < PB; j++)
            if (j < w) row[j] = LDL ? x[j] * rdiag[j] : x[j];
        if constexpr (LU) {   // the U^t rows: x L^t = a (unit)
            T *urow = AU + (int64_t)r * ld;
#pragma unroll
            for (int j = 0; j < PB; j++) x[j] = (j < w) ? urow[j] : T(0);
            wp_solve_rows<T, false, true>(x, TB, LDT, rdiag, w);
#pragma unroll
            for (int j = 0; j < PB; j++)
                if (j < w) urow[j] = x[j];
        }
    }
    if (lane == 0) {
        if (npiv) atomicAdd(&st->nbpivots, npiv);
        if (nneg) atomicAdd(&st->negpivots, nneg);
        if (nbad) atomicAdd(&st->nonfinite, nbad);
    }
}

}  // namespace pgpu
