// Diagonal-block factorization of a cblk spread over the GPU: one CTA per
// 32-row block row (kernels/core_zpotrfsp.c:144 core_zpotrfsp,
// core_zgetrfsp.c:138, core_zsytrfsp.c:141, core_zhetrfsp.c:144), and one CTA
// per 32-column block of its inverse (the panel TRSM done as a GEMM and the
// solves read it).
//
// Tile (i, j) of the w x w block belongs to the CTA of row i, which holds its
// row in shared memory from the first load to the last store.  At step k it
//   1. waits for row k's diagonal tile (its inverse is published in `scr`),
//   2. X_ik = A_ik op(L_kk)^{-1} (LU: U_kk^{-1}) as a product with that inverse,
//      corrected once by its residual (solve_tile), stored into the panel and
//      published,
//   3. A_ij -= X_ik op(L_jk)^t for k < j <= i with the rows' X_jk read through
//      L2 as they are published (LU: U_kj^t in place of L_jk; the CTA holds
//      column i of U, transposed, beside row i of L, and updates it alike),
// and after step i - 1 factorizes its diagonal tile and publishes its inverse.
// prog[row] counts the row's published tiles (i + 1 once the diagonal one is):
// step k of row i waits only for prog[j] > k with j < i.  Rows below the
// diagonal block (a fused panel) are block rows without a diagonal tile.  An
// inverse CTA (column block j) waits row by row: Inv_ij = -T_i sum_m L_im
// Inv_mj with T_i the tile's inverse.  CTAs take their jobs from a ticket in an
// order where a job waits only for earlier ones, so whatever part of the
// launch is resident makes progress.  All waits are bounded (Status::panel_timeout).
//
// What bounds it: the chain of w / 32 steps, each one L2 round trip (poll and
// tiles), four 32^3 products, and the 32-column elimination of the tile on one
// warp; the other rows' updates run beside it.  With one CTA for the whole
// block the rank-32 updates of one SM bounded it.  Block and inverse of a
// root-chain cblk of ~320 columns on one B200, from 512-thread CTA + inverse
// kernel to this (without the products' correction): FP32 LL^t 300 -> 110 us,
// FP64 LL^t 750 -> 165, FP32 LU 380 -> 145, complex64 LDL^h 1150 -> 290; the
// 20^3 FP64 factor + solve 2.53 -> 1.54 ms (with it some 0.07 more).
#pragma once

#include "pgpu_common.cuh"
#include "pgpu_panel.cuh"

namespace pgpu {

constexpr int PR_THREADS = 256;
constexpr long long PR_WAIT_CYCLES = 4000000000ll;

// Tiles in shared memory: 32 rows, k contiguous, rows padded by one 16-byte
// vector (row r starts at bank group r mod 8: the products' 16-byte loads of
// consecutive rows are conflict-free).
template <typename T> constexpr int pr_vk() { return 16 / (int)sizeof(T); }
template <typename T> constexpr int pr_pitch() { return PB + pr_vk<T>(); }
template <typename T> constexpr int pr_tile() { return PB * pr_pitch<T>(); }
// Shared-memory tiles of a job on a block of width w: the row's tiles (LU: and
// the U column's), one of X D^-1 / the inverse jobs' T, and the staging slots.
__host__ __device__ constexpr int pr_row_tiles(int w, bool lu) { return ((w + PB - 1) / PB) * (lu ? 2 : 1); }
// Staging slots (4; complex128, whose tiles are 17 KB, 2 where 4 do not fit), 0: the block does not fit.
inline int pr_slots(int w, size_t esz, bool lu, size_t limit) {
    const size_t tile = (size_t)PB * (PB + 16 / esz) * esz;
    for (int ns = 4; ns >= (lu ? 4 : 2); ns -= 2)
        if ((size_t)(pr_row_tiles(w, lu) + 1 + ns) * tile <= limit) return ns;
    return 0;
}
inline size_t pr_smem_bytes(int w, size_t esz, bool lu, int slots) {
    return (size_t)(pr_row_tiles(w, lu) + 1 + slots) * PB * (PB + 16 / esz) * esz;
}
// Published per diagonal tile: T = L^{-1} and L (32 x 32 each), LU: V = (U^t)^{-1} and U^t, and 1/d.
__host__ __device__ constexpr int pr_scr_tile(bool lu) { return (lu ? 4 : 2) * PB * PB + PB; }

// Jobs {cblk, block row (inverse: column block) | kind << 16, counter of row 0,
// scratch tile of row 0}.
enum { PR_ROW = 0, PR_INV = 1, PR_INV2 = 2 };

template <typename T> __device__ __forceinline__ void ldcg16(const T *p, T (&v)[16 / sizeof(T)]) {
    const uint4 u = __ldcg(reinterpret_cast<const uint4 *>(p));
    memcpy(v, &u, 16);
}
template <typename T> __device__ __forceinline__ T ldcg_s(const T *p) {   // one element through L2
    if constexpr (is_cplx<T>::value) {
        if constexpr (sizeof(T) == 8) {
            const float2 v = __ldcg(reinterpret_cast<const float2 *>(p));
            return T(v.x, v.y);
        } else {
            const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
            return T(v.x, v.y);
        }
    } else {
        return __ldcg(p);
    }
}

// acc[p][q] += sum_k A[a0 + p S][k] op(B[b0 + q S][k]) over one 32-column tile.
template <int NP, int S, bool CB, typename T>
__device__ __forceinline__ void pr_mm(const T *A, const T *B, int a0, int b0, T (&acc)[NP][NP]) {
    constexpr int VK = pr_vk<T>(), P = pr_pitch<T>();
#pragma unroll(VK >= 4 ? 4 : 2)
    for (int k = 0; k < PB; k += VK) {
        T a[NP][VK], b[NP][VK];
#pragma unroll
        for (int p = 0; p < NP; p++) ld16(A + (a0 + p * S) * P + k, a[p]);
#pragma unroll
        for (int q = 0; q < NP; q++) ld16(B + (b0 + q * S) * P + k, b[q]);
#pragma unroll
        for (int v = 0; v < VK; v++)
#pragma unroll
            for (int p = 0; p < NP; p++)
#pragma unroll
                for (int q = 0; q < NP; q++) acc[p][q] = fma_v(a[p][v], cj<CB>(b[q][v]), acc[p][q]);
    }
}
template <int NP, typename T> __device__ __forceinline__ void pr_zero(T (&acc)[NP][NP]) {
#pragma unroll
    for (int p = 0; p < NP; p++)
#pragma unroll
        for (int q = 0; q < NP; q++) acc[p][q] = T(0);
}

__device__ __forceinline__ int pr_ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool pr_wait(const int *p, int need) {
    const long long t0 = clock64();
    while (pr_ld_acquire(p) < need)
        if (clock64() - t0 > PR_WAIT_CYCLES) return false;
    return true;
}

// Named barrier 1 + C: columns 8 C .. 8 C + 7 of the elimination are in shared memory (the eliminating
// warp arrives, the inverse warps, one or two, wait).
template <int C, int THREADS> __device__ __forceinline__ void pr_chunk_arrive() {
    asm volatile("bar.arrive %0, %1;" ::"n"(C + 1), "n"(THREADS) : "memory");
}
template <int C, int THREADS> __device__ __forceinline__ void pr_chunk_sync() {
    asm volatile("bar.sync %0, %1;" ::"n"(C + 1), "n"(THREADS) : "memory");
}

// Elimination of the nb x nb tile by one warp, lane = row, the row in
// registers: a_ij -= l_ik d_k op(l_jk) (LU: l_ik u_kj) with l_ik = a_ik / d_k.
// The active columns sit at a[0 ..]: each step shifts them down by one, so the
// step loop needs no unrolling (its 32-fold body would miss in the instruction
// cache) and the update no dynamic register index; after every 8 steps the
// unrolled width shrinks by 8.  The next pivot needs only its own row's l, so
// it goes to the other lanes (dn) before the column is exchanged: a step costs
// a reciprocal, two products and a shuffle, the rest runs beside it.  Column k
// of l goes to Lc[k][i - k - 1], row k of u (LU) to Ub[k][j - k - 1], d_k and
// 1/d_k to dsm / rsm.  A negative Cholesky pivot becomes NaN at once, as its
// square root would.
template <typename T, int MODE, int W>
__device__ __forceinline__ void pr_factor_steps(T (&a)[PB], T &dn, int nb, typename real_of<T>::type crit, T *Lc,
                                                T *Ub, T *dsm, T *rsm, int &npiv, int &nneg, int &nbad) {
    typedef typename real_of<T>::type R;
    constexpr bool LU = (MODE == FM_GETRF), CJ = fm_conj(MODE);
    constexpr int VK = pr_vk<T>();
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
            d = T(R(NAN));
        }
        const T r = T(1) / d;
        const bool below = lane > k && lane < nb;
        const T raw = below ? a[0] : T(0);
        const T l = raw * r;
        dn = shfl_v(LU ? fma_v(-l, u1, a[1]) : fma_v(-raw, cj<CJ>(l), a[1]), min(k + 1, 31));
        if (lane > k) Lc[k * PB + lane - k - 1] = l;
        if (lane == k) {
            dsm[k] = d;
            rsm[k] = r;
            if (LU)
#pragma unroll
                for (int t = 0; t < W; t += VK) {
                    T v[VK];
#pragma unroll
                    for (int q = 0; q < VK; q++) v[q] = t + q + 1 < W ? a[t + q + 1] : T(0);
                    st16(Ub + k * PB + t, v);
                }
        }
        __syncwarp();
        const T x = LU ? l : raw;
        const T *col = (LU ? Ub : Lc) + k * PB;
#pragma unroll
        for (int t = 0; t < W; t += VK) {
            T c[VK];
            ld16(col + t, c);
#pragma unroll
            for (int q = 0; q < VK; q++)
                if (t + q + 1 < W) a[t + q] = fma_v(-x, cj<CJ && !LU>(c[q]), a[t + q + 1]);
        }
    }
    if (PB - W < nb) pr_chunk_arrive<(PB - W) / 8, LU ? 96 : 64>();
}
template <typename T, int MODE>
__device__ __noinline__ void pr_factor_tile(const T *tile, int nb, typename real_of<T>::type crit, T *Lc, T *Ub,
                                            T *dsm, T *rsm, Status *st) {
    const int lane = threadIdx.x & 31;
    int npiv = 0, nneg = 0, nbad = 0;
    T a[PB];
#pragma unroll
    for (int j = 0; j < PB; j += pr_vk<T>()) {
        T v[pr_vk<T>()];
        ld16(tile + lane * pr_pitch<T>() + j, v);
#pragma unroll
        for (int q = 0; q < pr_vk<T>(); q++) a[j + q] = (lane < nb && j + q < nb) ? v[q] : T(0);
    }
    T dn = shfl_v(a[0], 0);
    pr_factor_steps<T, MODE, 32>(a, dn, nb, crit, Lc, Ub, dsm, rsm, npiv, nneg, nbad);
    pr_factor_steps<T, MODE, 24>(a, dn, nb, crit, Lc, Ub, dsm, rsm, npiv, nneg, nbad);
    pr_factor_steps<T, MODE, 16>(a, dn, nb, crit, Lc, Ub, dsm, rsm, npiv, nneg, nbad);
    pr_factor_steps<T, MODE, 8>(a, dn, nb, crit, Lc, Ub, dsm, rsm, npiv, nneg, nbad);
    if (lane == 0) {
        if (npiv) atomicAdd(&st->nbpivots, npiv);
        if (nneg) atomicAdd(&st->negpivots, nneg);
        if (nbad) atomicAdd(&st->nonfinite, nbad);
    }
}
// Inverse of the unit lower factor whose columns are col[k][i - k - 1] (with
// scale: of the lower factor with diagonal 1 / rsm[k], (U^t)^{-1}), one warp
// eight columns behind the elimination, lane = column: out[k][lane].
template <typename T, int THREADS, int W>
__device__ __forceinline__ void pr_inverse_steps(T (&x)[PB], int nb, const T *col, const T *rsm, bool scale, T *out) {
    constexpr int VK = pr_vk<T>();
    const int lane = threadIdx.x & 31;
    if (PB - W < nb) pr_chunk_sync<(PB - W) / 8, THREADS>();
#pragma unroll 1
    for (int k = PB - W; k < PB - W + 8; k++) {
        if (k >= nb) break;
        T v = x[0];
        if (scale) v = v * rsm[k];
        out[k * pr_pitch<T>() + lane] = v;
        const T *c = col + k * PB;
#pragma unroll
        for (int t = 0; t < W; t += VK) {
            T cv[VK];
            ld16(c + t, cv);
#pragma unroll
            for (int q = 0; q < VK; q++)
                if (t + q + 1 < W) x[t + q] = fma_v(-cv[q], v, x[t + q + 1]);
        }
    }
}
template <typename T, int THREADS>
__device__ __noinline__ void pr_inverse_tile(int nb, const T *col, const T *rsm, bool scale, T *out) {
    const int lane = threadIdx.x & 31;
    T x[PB];
#pragma unroll
    for (int i = 0; i < PB; i++) x[i] = T(i == lane ? 1 : 0);
    pr_inverse_steps<T, THREADS, 32>(x, nb, col, rsm, scale, out);
    pr_inverse_steps<T, THREADS, 24>(x, nb, col, rsm, scale, out);
    pr_inverse_steps<T, THREADS, 16>(x, nb, col, rsm, scale, out);
    pr_inverse_steps<T, THREADS, 8>(x, nb, col, rsm, scale, out);
    for (int k = nb; k < PB; k++) out[k * pr_pitch<T>() + lane] = T(0);   // (rows past a ragged tile)
}

template <typename T, int MODE>
__global__ void __launch_bounds__(PR_THREADS, sizeof(T) <= 8 ? 2 : 1) k_panel_rows(Meta m, const int4 *__restrict__ jobs, int *ticket,
                                                           int *prog, T *scr, T *coefL, T *coefU, T *inv,
                                                           const double *critp, int fuse_rows, int slots,
                                                           Status *st, const int *pos, int64_t *prof) {
    typedef typename real_of<T>::type R;
    constexpr bool LU = (MODE == FM_GETRF), LDL = fm_ldl(MODE), CJ = fm_conj(MODE);
    constexpr int VK = pr_vk<T>(), P = pr_pitch<T>(), TILE = pr_tile<T>(), NV = PB / VK;
    constexpr int SCR = pr_scr_tile(LU);
    extern __shared__ __align__(16) unsigned char pr_smem[];
    __shared__ __align__(16) T dsm[PB], rsm[PB], sqs[PB];
    __shared__ int job_s, fail_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        job_s = atomicAdd(ticket, 1);
        fail_s = 0;
    }
    __syncthreads();
    const int4 jb = jobs[job_s];
    const int c = jb.x, kind = jb.y >> 16, i = jb.y & 0xffff;
    const uint64_t t_start = prof ? global_ns() : 0;
    const int w = m.width[c], h = m.height[c], ld = m.ld[c];
    const int nt = (w + PB - 1) / PB;
    T *A = coefL + m.coefoff[c], *AU = coefU + m.coefoff[c];
    int *pc = prog + jb.z;
    T *sc = scr + (int64_t)jb.w * SCR;
    T *row = reinterpret_cast<T *>(pr_smem);            // the row's tiles (inverse jobs: its column's)
    // the products' thread grids: 16 x 16 threads of 2 x 2, four groups of 8 x 8 threads of 4 x 4
    const int x16 = tid & 15, y16 = tid >> 4;
    const int grp = tid >> 6, x8 = tid & 7, y8 = (tid >> 3) & 7;
    auto wait_for = [&](int r, int need) {              // one thread of the CTA; all see fail_s after a barrier
        if (!pr_wait(pc + r, need)) fail_s = 1;
    };
    // a dense 32 x 32 tile of the scratch into a slot
    auto load_scr = [&](const T *src, T *dst) {
        for (int e = tid; e < PB * NV; e += PR_THREADS) {
            T v[VK];
            ldcg16(src + e * VK, v);
            st16(dst + (e / NV) * P + (e % NV) * VK, v);
        }
    };
    // panel tile rows r0 .. r0 + nr, columns c0 .. (zero past nr and past column w) into a slot
    auto load_tile = [&](const T *base, int r0, int nr, int c0, T *dst, int t, int nthr) {
        for (int e = t; e < PB * NV; e += nthr) {
            const int r = e / NV, q = e % NV * VK;
            T v[VK];
#pragma unroll
            for (int u = 0; u < VK; u++) v[u] = T(0);
            if (r < nr && c0 + q < w) {
                ldcg16(base + (int64_t)(r0 + r) * ld + c0 + q, v);
#pragma unroll
                for (int u = 0; u < VK; u++)
                    if (c0 + q + u >= w) v[u] = T(0);
            }
            st16(dst + r * P + q, v);
        }
    };
    // the transposed tile: dst[r][q] = base[r0 + q][c0 + r] (q < nq, c0 + r < w)
    auto load_tile_t = [&](const T *base, int r0, int nq, int c0, T *dst, int t, int nthr) {
        for (int e = t; e < PB * PB; e += nthr) {
            const int q = e / PB, r = e % PB;
            dst[r * P + q] = (q < nq && c0 + r < w) ? ldcg_s(base + (int64_t)(r0 + q) * ld + c0 + r) : T(0);
        }
    };
    auto failed = [&]() { return *(volatile int *)&fail_s != 0; };
    // x = M op(Ti)^t, then once x += (M - x op(Lt)^t) op(Ti)^t, and with TWO y from N alike (x, y: this thread's
    // 2 x 2 entries; M and N are overwritten): the product with an inverse alone leaves a residual larger by the
    // tile's condition than a substitution's, the corrected one does not.  (Solves of shifted, indefinite grids of
    // some 9000 unknowns with the factor, error without and with: FP64 LDL^t 1.7e-11 -> 8.4e-12, by substitution
    // 8.0e-12; single precision 1.7e-2 -> 7.5e-3.  It costs 1 to 5 % of a call, the most where the panel chain
    // is the longest part: 60^3 complex LDL^h 23.0 -> 24.2 ms.)
    auto solve_tile = [&](auto cb, auto two, T *M, const T *Ti, const T *Lt, T (&x)[2][2], T *N, const T *Ni,
                          const T *Nt, T (&y)[2][2]) {
        constexpr bool CB = decltype(cb)::value, TWO = decltype(two)::value;
        auto own = [&](T *t, int p, int q) -> T & { return t[(y16 + 16 * p) * P + x16 + 16 * q]; };
        T m[2][2], n[2][2], z[2][2];
        auto put = [&](const T (&u)[2][2], const T (&v)[2][2]) {
            __syncthreads();
#pragma unroll
            for (int p = 0; p < 2; p++)
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    own(M, p, q) = u[p][q];
                    if (TWO) own(N, p, q) = v[p][q];
                }
            __syncthreads();
        };
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int q = 0; q < 2; q++) {
                m[p][q] = own(M, p, q);
                if (TWO) n[p][q] = own(N, p, q);
            }
        pr_zero(x);
        pr_mm<2, 16, CB>(M, Ti, y16, x16, x);
        if (TWO) {
            pr_zero(y);
            pr_mm<2, 16, false>(N, Ni, y16, x16, y);
        }
        put(x, y);
        auto residual = [&](T (&r)[2][2]) {
#pragma unroll
            for (int p = 0; p < 2; p++)
#pragma unroll
                for (int q = 0; q < 2; q++) r[p][q] -= z[p][q];
        };
        pr_zero(z);
        pr_mm<2, 16, CB>(M, Lt, y16, x16, z);
        residual(m);
        if (TWO) {
            pr_zero(z);
            pr_mm<2, 16, false>(N, Nt, y16, x16, z);
            residual(n);
        }
        put(m, n);
        pr_mm<2, 16, CB>(M, Ti, y16, x16, x);
        if (TWO) pr_mm<2, 16, false>(N, Ni, y16, x16, y);
        __syncthreads();
    };

    if (kind == PR_ROW) {
        const bool diag = i < nt;
        const int rows = (h <= fuse_rows) ? h : w;
        const int r0 = diag ? i * PB : w + (i - nt) * PB;
        const int nr = min(PB, (diag ? w : rows) - r0);
        const int nk = min(i, nt), ntile = diag ? i + 1 : nt;
        T *vrow = row + nt * TILE;                      // LU: column i of U, transposed
        T *P1 = row + pr_row_tiles(w, LU) * TILE;       // X D^{-1} (LDL)
        T *S = P1 + TILE;
        for (int j = 0; j < ntile; j++) load_tile(A, r0, nr, j * PB, row + j * TILE, tid, PR_THREADS);
        if (LU)
            for (int j = 0; j < nk; j++) {
                if (diag) load_tile_t(A, j * PB, PB, r0, vrow + j * TILE, tid, PR_THREADS);
                else load_tile(AU, r0, nr, j * PB, vrow + j * TILE, tid, PR_THREADS);
            }
        for (int k = 0; k < nk; k++) {
            T *Q = row + k * TILE, *V = vrow + k * TILE;
            const int nbk = min(PB, w - k * PB);
            if (tid == 0) wait_for(k, k + 1);
            __syncthreads();
            if (failed()) break;
            const T *sk = sc + (int64_t)k * SCR;
            load_scr(LU ? sk + PB * PB : sk, S);                      // T (LU: V)
            load_scr(sk + (LU ? 3 : 1) * PB * PB, S + TILE);          // L (LU: U^t)
            if (LU) {
                load_scr(sk, S + 2 * TILE);
                load_scr(sk + 2 * PB * PB, S + 3 * TILE);
            }
            if (LDL && tid < PB) rsm[tid] = ldcg_s(sk + 2 * PB * PB + tid);
            __syncthreads();
            T x[2][2], y[2][2];
            solve_tile(std::integral_constant<bool, CJ>{}, std::integral_constant<bool, LU>{}, Q, S, S + TILE, x, V,
                       S + 2 * TILE, S + 3 * TILE, y);
#pragma unroll
            for (int p = 0; p < 2; p++)
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int r = y16 + 16 * p, cc = x16 + 16 * q;
                    Q[r * P + cc] = x[p][q];
                    const T out = LDL ? x[p][q] * rsm[cc] : x[p][q];
                    if (LDL) P1[r * P + cc] = out;
                    if (LU) V[r * P + cc] = y[p][q];
                    if (r < nr && cc < nbk) {
                        A[(int64_t)(r0 + r) * ld + k * PB + cc] = out;
                        if (LU && !diag) AU[(int64_t)(r0 + r) * ld + k * PB + cc] = y[p][q];
                    }
                }
            __syncthreads();
            if (LU && diag) {
                for (int e = tid; e < PB * PB; e += PR_THREADS) {
                    const int q = e / PB, r = e % PB;
                    if (q < nbk && r < nr) A[(int64_t)(k * PB + q) * ld + r0 + r] = V[r * P + q];
                }
                __syncthreads();
            }
            if (diag && tid == PR_THREADS - 1) {        // (not the warp that factorizes the tile)
                __threadfence();
                atomicExch(pc + i, k + 1);
            }
            const T *own = LDL ? P1 : LU ? V : Q;
            if (diag && i == k + 1) {
                // the next tile to factorize: all threads on its update
                T z[2][2];
                T *D = row + i * TILE;
                pr_zero(z);
                pr_mm<2, 16, CJ>(Q, own, y16, x16, z);
#pragma unroll
                for (int p = 0; p < 2; p++)
#pragma unroll
                    for (int q = 0; q < 2; q++) D[(y16 + 16 * p) * P + x16 + 16 * q] -= z[p][q];
                continue;
            }
            const int jend = diag ? i + 1 : nt, step = LU ? 2 : slots;
            bool stop = false;
            for (int j0 = k + 1; j0 < jend; j0 += step) {
                const int nj = min(step, jend - j0);
                if (warp == 0 && lane < nj && j0 + lane < min(i, nt)) wait_for(j0 + lane, k + 1);
                __syncthreads();                        // (also: the previous chunk's slots are free)
                if (failed()) {
                    stop = true;
                    break;
                }
                for (int q = 0; q < nj; q++) {
                    const int j = j0 + q;
                    if (diag && j == i) continue;
                    const int nrj = min(PB, w - j * PB);
                    if (LU) {
                        load_tile_t(A, k * PB, nbk, j * PB, S + 2 * q * TILE, tid, PR_THREADS);
                        load_tile(A, j * PB, nrj, k * PB, S + (2 * q + 1) * TILE, tid, PR_THREADS);
                    } else {
                        load_tile(A, j * PB, nrj, k * PB, S + q * TILE, tid, PR_THREADS);
                    }
                }
                __syncthreads();
                T z[4][4];
                const int jq = LU ? grp >> 1 : grp, j = j0 + jq;
                const bool side = LU && (grp & 1);      // LU: the U column's half
                if (jq < nj && !(side && diag && j == i)) {
                    const T *B = (diag && j == i) ? own : S + grp * TILE;
                    T *D = (side ? vrow : row) + j * TILE;
                    pr_zero(z);
                    pr_mm<4, 8, CJ>(side ? V : Q, B, y8, x8, z);
#pragma unroll
                    for (int p = 0; p < 4; p++)
#pragma unroll
                        for (int q = 0; q < 4; q++) D[(y8 + 8 * p) * P + x8 + 8 * q] -= z[p][q];
                }
            }
            if (stop) break;
        }
        __syncthreads();
        if (diag && !failed()) {
            // the diagonal tile: elimination (warp 0), its inverse (warp 1; LU: U's on warp 2) behind it
            T *Lc = S, *To = S + TILE, *Ub = LU ? S + 2 * TILE : nullptr, *Vo = LU ? S + 3 * TILE : nullptr;
            const R crit = R(*critp);
            if (warp == 0) pr_factor_tile<T, MODE>(row + i * TILE, nr, crit, Lc, Ub, dsm, rsm, st);
            else if (warp == 1) pr_inverse_tile<T, LU ? 96 : 64>(nr, Lc, rsm, false, To);
            else if (LU && warp == 2) pr_inverse_tile<T, 96>(nr, Ub, rsm, true, Vo);
            __syncthreads();
            if (MODE == FM_POTRF) {
                if (tid < nr) sqs[tid] = sqrt_v(dsm[tid]);
                __syncthreads();
            }
            // what the other rows wait for first
            T *so = sc + (int64_t)i * SCR;
            for (int e = tid; e < PB * PB; e += PR_THREADS) {
                const int r = e / PB, q = e % PB;
                T t = To[r * P + q];
                if (MODE == FM_POTRF && r < nr) t = t * (T(1) / sqs[r]);
                so[e] = t;
                const bool in = r < nr && q <= r;
                T l = !in ? T(0) : q == r ? (MODE == FM_POTRF ? sqs[r] : T(1)) : Lc[q * PB + r - q - 1];
                if (MODE == FM_POTRF && in && q < r) l = l * sqs[q];
                so[(LU ? 2 : 1) * PB * PB + e] = l;
                if (LU) {
                    so[PB * PB + e] = Vo[r * P + q];
                    so[3 * PB * PB + e] = !in ? T(0) : q == r ? dsm[r] : Ub[q * PB + r - q - 1];
                }
            }
            if (tid < PB) so[(LU ? 4 : 2) * PB * PB + tid] = tid < nr ? rsm[tid] : T(0);
            __syncthreads();
            if (tid == 0) {
                __threadfence();
                atomicExch(pc + i, i + 1);
            }
            for (int e = tid; e < PB * PB; e += PR_THREADS) {
                const int r = e / PB, q = e % PB;
                if (r >= nr || q >= nr || (!LU && q > r)) continue;
                T v;
                if (q == r) v = MODE == FM_POTRF ? sqs[r] : dsm[r];
                else if (q < r) v = MODE == FM_POTRF ? Lc[q * PB + r - q - 1] * sqs[q] : Lc[q * PB + r - q - 1];
                else v = Ub[r * PB + q - r - 1];
                A[(int64_t)(r0 + r) * ld + r0 + q] = v;
            }
        }
    } else {
        // inverse, column block i; rows j = i .. nt - 1 (LU: kind PR_INV inverts U^t, PR_INV2 the unit L)
        const bool tr = LU && kind == PR_INV;
        const int64_t vo = tr ? PB * PB : 0;            // V or T in the scratch tile
        T *Inv = inv + m.invoff[c] + (LU && kind == PR_INV2 ? inv_span(w, ld) : 0);
        T *Tt = row + pr_row_tiles(w, LU) * TILE, *S = Tt + TILE;
        const int ncol = min(PB, w - i * PB);
        for (int j = i; j < nt; j++) {
            T *X = row + (j - i) * TILE;                // [column][row of the inverse]
            const int nrj = min(PB, w - j * PB);
            if (tid == 0) wait_for(j, j + 1);
            __syncthreads();
            if (failed()) break;
            const T *sj = sc + (int64_t)j * SCR;
            if (LDL && tid < PB) rsm[tid] = ldcg_s(sj + 2 * PB * PB + tid);
            load_scr(sj + vo, Tt);
            if (j == i) {
                __syncthreads();
                for (int e = tid; e < PB * PB; e += PR_THREADS) X[(e % PB) * P + e / PB] = Tt[e / PB * P + e % PB];
            } else {
                T z[4][4];
                pr_zero(z);
                for (int m0 = i; m0 < j; m0 += slots) {
                    const int nm = min(slots, j - m0);
                    if (m0 > i) __syncthreads();
                    for (int q = 0; q < nm; q++) {
                        if (tr) load_tile_t(A, (m0 + q) * PB, PB, j * PB, S + q * TILE, tid, PR_THREADS);
                        else load_tile(A, j * PB, nrj, (m0 + q) * PB, S + q * TILE, tid, PR_THREADS);
                    }
                    __syncthreads();
                    if (grp < nm) pr_mm<4, 8, false>(row + (m0 + grp - i) * TILE, S + grp * TILE, y8, x8, z);
                }
                __syncthreads();
                if (grp < slots) {
#pragma unroll
                    for (int p = 0; p < 4; p++)
#pragma unroll
                        for (int q = 0; q < 4; q++) S[grp * TILE + (y8 + 8 * p) * P + x8 + 8 * q] = z[p][q];
                }
                __syncthreads();
                for (int e = tid; e < PB * PB; e += PR_THREADS) {
                    const int o = e / PB * P + e % PB;
                    T s = S[o];
                    for (int g = 1; g < slots; g++) s += S[g * TILE + o];
                    X[o] = s;
                }
                __syncthreads();                        // (the slots are free: L or U^t of tile j into the first)
                load_scr(sj + vo + (LU ? 2 : 1) * PB * PB, S);
                __syncthreads();
                T x[2][2];
                solve_tile(std::false_type{}, std::false_type{}, X, Tt, S, x, X, Tt, S, x);
#pragma unroll
                for (int p = 0; p < 2; p++)
#pragma unroll
                    for (int q = 0; q < 2; q++) X[(y16 + 16 * p) * P + x16 + 16 * q] = -x[p][q];
            }
            __syncthreads();
            for (int e = tid; e < PB * PB; e += PR_THREADS) {
                const int r = e / PB, q = e % PB;
                if (r < nrj && q < ncol) {
                    T v = cj<CJ>(X[q * P + r]);
                    if (LDL) v = v * rsm[r];
                    Inv[(int64_t)(j * PB + r) * ld + i * PB + q] = v;
                }
            }
        }
    }
    if (tid == 0 && failed()) atomicAdd(&st->panel_timeout, 1);
    if (prof && kind == PR_ROW) {
        // the panel's task record: from the start of its first block row to the end of its last
        __syncthreads();
        if (tid == 0) {
            int64_t *t = prof + 2 * (int64_t)pos[c];
            if (i == 0) t[0] = (int64_t)t_start;
            atomicMax(reinterpret_cast<unsigned long long *>(t + 1), (unsigned long long)global_ns());
        }
    }
}

}  // namespace pgpu
