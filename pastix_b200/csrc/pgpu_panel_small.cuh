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
// tile, eliminated with lane = row and the row in registers (the active
// columns shifted down by one each step, as in k_panel_rows: a 32-fold
// unrolled body would miss in the instruction cache with every warp of the SM
// in it, a tile kept in shared memory costs a round trip per step), and the
// panel rows below it are solved one lane per row with the row in registers.
// What bounds it is the latency of the 32 dependent steps and of the row's
// substitution; a warp has no more work to hide it with than its own cblk.
// (501x389 2D, panels of all levels: 0.72 -> 0.65 ms with the tile eliminated
// in registers here and the pivot sent ahead in both panel kernels.)
// Shared memory per warp: TA [PB][PB + VK] (the coefficients of the row
// solves: the unit lower factor, LU: U transposed), TB alike for LU (its unit
// lower factor), two column buffers (LU: and two row buffers), d and 1 / d.
// ---------------------------------------------------------------------------
constexpr int PS_WARPS = 8;
template <typename T>
__host__ __device__ constexpr int ps_warp_elems(bool lu) { return (lu ? 2 : 1) * (PB * (PB + 16 / (int)sizeof(T)) + 2 * PB) + 3 * PB; }
template <typename T>
constexpr int ps_smem_bytes(bool lu) { return PS_WARPS * ps_warp_elems<T>(lu) * (int)sizeof(T); }

// Elimination steps PB - W .. PB - W + 7 (pr_factor_steps, without the publication): l_ik = a_ik / d_k to
// TL[i][k], LU: u_kj to TU[j][k], d_k and 1 / d_k to ds / rs.
template <typename T, int MODE, int W>
__device__ __forceinline__ void ps_factor_steps(T (&a)[PB], T &dn, int nb, typename real_of<T>::type crit, T *TL, T *TU,
                                                T *col, T *urow, T *ds, T *rs, int &npiv, int &nneg, int &nbad) {
    typedef typename real_of<T>::type R;
    constexpr bool LU = (MODE == FM_GETRF), CJ = fm_conj(MODE);
    constexpr int VK = 16 / sizeof(T), LDT = PB + VK;
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int k = PB - W; k < PB - W + 8; k++) {
        if (k >= nb) break;
        T d = dn;
        const T u1 = LU ? shfl_v(a[1], k) : T(0);
        if (!finite_v(d)) nbad++;
        d = static_pivot<T, MODE>(d, crit, npiv);
        if (CJ) d = T(real_v(d));   // (the diagonal of a Hermitian form is real)
        if (MODE == FM_POTRF && real_v(d) < R(0)) {
            nneg++;
            d = T(R(NAN));          // (as its square root would be)
        }
        const T r = T(1) / d;
        const bool below = lane > k && lane < nb;
        const T raw = below ? a[0] : T(0);
        const T l = raw * r;
        dn = shfl_v(LU ? fma_v(-l, u1, a[1]) : fma_v(-raw, cj<CJ>(l), a[1]), min(k + 1, 31));
        T *cb = col + (k & 1) * PB, *ub = urow + (k & 1) * PB;
        if (lane > k) {
            cb[lane - k - 1] = l;
            TL[lane * LDT + k] = l;
        }
        if (lane == k) {
            ds[k] = d;
            rs[k] = r;
            if (LU)
#pragma unroll
                for (int t = 0; t < W; t += VK) {
                    T v[VK];
#pragma unroll
                    for (int q = 0; q < VK; q++) v[q] = t + q + 1 < W ? a[t + q + 1] : T(0);
                    st16(ub + t, v);
                }
        }
        __syncwarp();
        if (LU && lane > k) TU[lane * LDT + k] = ub[lane - k - 1];
        const T x = LU ? l : raw;
        const T *cv = LU ? ub : cb;
#pragma unroll
        for (int t = 0; t < W; t += VK) {
            T c[VK];
            ld16(cv + t, c);
#pragma unroll
            for (int q = 0; q < VK; q++)
                if (t + q + 1 < W) a[t + q] = fma_v(-x, cj<CJ && !LU>(c[q]), a[t + q + 1]);
        }
    }
}

template <typename T, int MODE>
__global__ void __launch_bounds__(PS_WARPS * 32) k_panel_small(Meta m, const int2 *__restrict__ jobs, int njobs,
                                                               T *__restrict__ coefL, T *__restrict__ coefU,
                                                               const double *critp, int fuse_rows, Status *st) {
    typedef typename real_of<T>::type R;
    constexpr bool LU = (MODE == FM_GETRF);
    constexpr bool CJ = fm_conj(MODE);
    constexpr int VK = 16 / sizeof(T), LDT = PB + VK;
    extern __shared__ __align__(16) unsigned char ps_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x * PS_WARPS + warp;
    if (q >= njobs) return;                        // whole warps; warp-level synchronization only
    T *TA = reinterpret_cast<T *>(ps_raw) + (size_t)warp * ps_warp_elems<T>(LU);
    T *TB = TA + PB * LDT;                         // (LU)
    T *col = TA + (LU ? 2 : 1) * PB * LDT, *urow = col + (LU ? 2 * PB : 0);
    T *ds = col + (LU ? 4 : 2) * PB, *rs = ds + PB, *sc = rs + PB;
    const int c = jobs[q].x;
    const int w = m.width[c], h = m.height[c], ld = m.ld[c];
    const int rows = (h <= fuse_rows) ? h : w;
    T *A = coefL + m.coefoff[c];
    T *AU = coefU + m.coefoff[c];
    const R crit = R(*critp);
    int npiv = 0, nneg = 0, nbad = 0;
    // elements [0, w) of a panel row (16-byte loads / stores: rows are 16-byte aligned, padded to a multiple of 4)
    auto load_row = [&](const T *row, bool ok, T (&x)[PB]) {
#pragma unroll
        for (int j = 0; j < PB; j += VK) {
            uint4 u = make_uint4(0, 0, 0, 0);
            if (ok && j < w) u = *reinterpret_cast<const uint4 *>(row + j);
            memcpy(&x[j], &u, 16);
        }
#pragma unroll
        for (int j = 0; j < PB; j++)
            if (j >= w) x[j] = T(0);
    };
    auto store_row = [&](T *row, const T (&x)[PB]) {
#pragma unroll
        for (int j = 0; j < PB; j += VK)
            if (j < w) {
                uint4 u;
                memcpy(&u, &x[j], 16);
                *reinterpret_cast<uint4 *>(row + j) = u;
            }
    };
    {
        T a[PB];
        load_row(A + (int64_t)(lane < w ? lane : 0) * ld, lane < w, a);
        T *TL = LU ? TB : TA;
        T dn = shfl_v(a[0], 0);
        ps_factor_steps<T, MODE, 32>(a, dn, w, crit, TL, TA, col, urow, ds, rs, npiv, nneg, nbad);
        ps_factor_steps<T, MODE, 24>(a, dn, w, crit, TL, TA, col, urow, ds, rs, npiv, nneg, nbad);
        ps_factor_steps<T, MODE, 16>(a, dn, w, crit, TL, TA, col, urow, ds, rs, npiv, nneg, nbad);
        ps_factor_steps<T, MODE, 8>(a, dn, w, crit, TL, TA, col, urow, ds, rs, npiv, nneg, nbad);
    }
    __syncwarp();
    // sc: what the solved rows (and, inverted, the tile's columns) are scaled by -- 1 / sqrt(d) or 1 / d
    T sq = T(1);
    if (lane < w) {
        if (MODE == FM_POTRF) sq = sqrt_v(ds[lane]);
        sc[lane] = MODE == FM_POTRF ? T(1) / sq : rs[lane];
    }
    if (MODE == FM_POTRF && lane < w) ds[lane] = sq;
    __syncwarp();
    for (int i = 0; i < w; i++) {   // the factorized tile, row by row (coalesced): lower part, LU: all of it
        if (lane < i) {
            const T l = (LU ? TB : TA)[i * LDT + lane];
            A[(int64_t)i * ld + lane] = MODE == FM_POTRF ? l * ds[lane] : l;
        } else if (lane == i) {
            A[(int64_t)i * ld + lane] = ds[i];
        } else if (LU && lane < w) {
            A[(int64_t)i * ld + lane] = TA[lane * LDT + i];
        }
    }
    for (int r = w + lane; r < rows; r += 32) {
        T x[PB];
        T *row = A + (int64_t)r * ld;
        load_row(row, true, x);
        // LU: x U = a; else x (L D^(1/2 or 1)) op(L)^t = a: the unit solve, then the columns scaled
        if (LU) wp_solve_rows<T, false, false>(x, TA, LDT, rs, w);
        else wp_solve_rows<T, CJ, true>(x, TA, LDT, rs, w);
        if (!LU)
#pragma unroll
            for (int j = 0; j < PB; j++)
                if (j < w) x[j] = x[j] * sc[j];
        store_row(row, x);
        if constexpr (LU) {   // the U^t rows: x L^t = a (unit)
            T *ur = AU + (int64_t)r * ld;
            load_row(ur, true, x);
            wp_solve_rows<T, false, true>(x, TB, LDT, rs, w);
            store_row(ur, x);
        }
    }
    if (lane == 0) {
        if (npiv) atomicAdd(&st->nbpivots, npiv);
        if (nneg) atomicAdd(&st->negpivots, nneg);
        if (nbad) atomicAdd(&st->nonfinite, nbad);
    }
}

}  // namespace pgpu
