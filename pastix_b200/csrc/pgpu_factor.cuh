// Numerical factorization kernels: coeftab fill-in, diagonal-block
// factorization with static pivoting, panel TRSM and the update GEMM with its
// indexed scatter-add into the facing column block.
#pragma once

#include "pgpu_common.cuh"

namespace pgpu {

// ---------------------------------------------------------------------------
// Fill-in (kernels/cpucblk_zinit.c:393 cpucblk_zfillin_fr and, for the mixed
// factorization, kernels/cpucblk_zcinit.c:81 cpucblk_zcfillin_fr): every
// value of the user's matrix lands at its precomputed coeftab offset.  The
// coeftab was zeroed before.  A value that does not fit the factor type
// (single precision) is flagged, as cpucblk_zccheck_overflow does.
// ---------------------------------------------------------------------------
// dst[k] >= 0: coef[dst[k]] = v; dst[k] < 0: coef[~dst[k]] = conj(v) (a
// Hermitian entry stored in the other triangle after the permutation, the
// conjugation bcsc/bcsc_zinit.c applies through __fct_conj).
template <typename T, typename Tin>
__global__ void k_fillin(int64_t nnz, const Tin *__restrict__ vals,
                         const int64_t *__restrict__ dst, T *__restrict__ coef,
                         Status *st) {
    typedef typename real_of<T>::type R;
    int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (; k < nnz; k += stride) {
        Tin v = vals[k];
        int64_t d = dst[k];
        if (d < 0) {
            d = ~d;
            v = conj_v(v);
        }
        if (sizeof(R) == 4 && !(abs_v(v) <= 3.4028234663852886e38)) atomicAdd(&st->overflow, 1);
        coef[d] = T(v);
    }
}

// ---------------------------------------------------------------------------
// Update GEMM with indexed scatter-add (kernels/core_zgemmsp.c:104
// core_zgemmsp_1d1d: W = A B^T then core_zgeadd into the facing cblk).
// Task t: source cblk c, block b facing cblk f.  A = panel rows
// [arow0, arow0 + M) of c, B = the m_b rows of block b, K = w_c; C = A B^T is
// subtracted from f at (panel row of the source row in f, column
// frownum_b + j - fcolnum_f).  Different source cblks of one level may hit the
// same target entries, so the subtraction is an atomic reduction.
// One CTA computes one GEMM_TM x GEMM_TN tile with a 4x4 register block per
// thread.  tile = {task, tile_m, tile_n, 0};
// task = {c, b, f, arow0, M, flags} with flags: 1 A from U, 2 B from U,
// 4 target U, 8 lower-triangle-only target (symmetric diagonal block),
// 16 scale by the pivots of c (LDL: C -= A D op(B)^t, core_zgemdm),
// 32 conjugate B (Hermitian forms: op = conj),
// 64 panel TRSM as a GEMM: X = A B^t with A the off-diagonal rows of c
//    (arow0 = w_c, M = h_c - w_c), B the inverse of its diagonal block
//    (inv + invoff[c], N = K = w_c), X stored (not accumulated) at scr + out
//    with row stride ld_c; 128: B is the cblk's second inverse (LU U^t side).
// ---------------------------------------------------------------------------
constexpr int GEMM_TM = 64, GEMM_TN = 64, GEMM_TK = 16;

struct GemmTask {
    int c, b, f, arow0, M, flags;
    int64_t out;   // flags & 64 (panel TRSM as GEMM): element offset of X in the level's scratch
};

template <typename T>
__global__ void __launch_bounds__(256) k_gemm_scatter(Meta m, const int4 *__restrict__ tiles,
                                                      const GemmTask *__restrict__ tasks,
                                                      T *__restrict__ coefL, T *__restrict__ coefU,
                                                      const T *__restrict__ inv, T *__restrict__ scr,
                                                      int64_t *prof) {
    const uint64_t t_start = prof ? global_ns() : 0;
    __shared__ T As[GEMM_TK][GEMM_TM + 4];
    __shared__ T Bs[GEMM_TK][GEMM_TN + 4];
    __shared__ T Ds[GEMM_TK];
    __shared__ int trow_s[GEMM_TM];
    const int4 tl = tiles[blockIdx.x];
    const GemmTask t = tasks[tl.x];
    const int c = t.c, b = t.b, f = t.f;
    const int K = m.width[c], ld = m.ld[c];
    const bool trsm = (t.flags & 64) != 0;
    const int N = trsm ? K : m.blrow[b] - m.bfrow[b] + 1;
    const int i0 = tl.y * GEMM_TM, j0 = tl.z * GEMM_TN;
    const T *A = ((t.flags & 1) ? coefU : coefL) + m.coefoff[c] + (int64_t)(t.arow0 + i0) * ld;
    const T *B = trsm ? inv + m.invoff[c] + ((t.flags & 128) ? inv_span(K, ld) : 0) + (int64_t)j0 * ld
                      : ((t.flags & 2) ? coefU : coefL) + m.coefoff[c] + (int64_t)(m.browoff[b] + j0) * ld;
    const int mrows = min(GEMM_TM, t.M - i0), ncols = min(GEMM_TN, N - j0);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;

    // target panel row of each tile row (binary search in f's blocks)
    if (tid < GEMM_TM && !trsm) {
        int tr = -1;
        if (tid < mrows) {
            int grow = m.rowidx[m.rowbase[c] + t.arow0 + i0 + tid];
            tr = panel_row_of(m, f, grow);
        }
        trow_s[tid] = tr;
    }

    T acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[a][q] = T(0);

    const bool scale_d = (t.flags & 16) != 0, conj_b = (t.flags & 32) != 0;
    const T *Dg = coefL + m.coefoff[c];
    for (int k0 = 0; k0 < K; k0 += GEMM_TK) {
        if (scale_d) {
            if (tid < GEMM_TK) Ds[tid] = (k0 + tid < K) ? Dg[(int64_t)(k0 + tid) * ld + k0 + tid] : T(0);
            __syncthreads();
        }
#pragma unroll
        for (int s = 0; s < 4; s++) {
            int e = tid + s * 256;
            int r = e >> 4, kk = e & 15;
            int kg = k0 + kk;
            T av = (r < mrows && kg < K) ? A[(int64_t)r * ld + kg] : T(0);
            T bv = (r < ncols && kg < K) ? B[(int64_t)r * ld + kg] : T(0);
            if (scale_d) av = av * Ds[kk];
            if (conj_b) bv = conj_v(bv);
            As[kk][r] = av;
            Bs[kk][r] = bv;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GEMM_TK; kk++) {
            T a[4], bv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                a[q] = As[kk][ty * 4 + q];
                bv[q] = Bs[kk][tx * 4 + q];
            }
#pragma unroll
            for (int p = 0; p < 4; p++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[p][q] += a[p] * bv[q];
        }
        __syncthreads();
    }

    if (trsm) {
        T *O = scr + t.out + (int64_t)i0 * ld + j0;
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const int i = ty * 4 + p;
            if (i >= mrows) continue;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int j = tx * 4 + q;
                if (j < ncols) O[(int64_t)i * ld + j] = acc[p][q];
            }
        }
        if (prof) {
            __syncthreads();
            if (tid == 0) {
                prof[2 * blockIdx.x] = (int64_t)t_start;
                prof[2 * blockIdx.x + 1] = (int64_t)global_ns();
            }
        }
        return;
    }
    T *C = ((t.flags & 4) ? coefU : coefL) + m.coefoff[f];
    const int ldf = m.ld[f];
    const int tcol0 = m.bfrow[b] + j0 - m.fcol[f];
    const bool lower_only = (t.flags & 8) != 0;
    const int wf = m.width[f];
#pragma unroll
    for (int p = 0; p < 4; p++) {
        int i = ty * 4 + p;
        if (i >= mrows) continue;
        int tr = trow_s[i];
        if (tr < 0) continue;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            int j = tx * 4 + q;
            if (j >= ncols) continue;
            int tc = tcol0 + j;
            if (lower_only && tr < wf && tc > tr) continue;
            atomic_sub(&C[(int64_t)tr * ldf + tc], acc[p][q]);
        }
    }
    if (prof) {
        __syncthreads();
        if (tid == 0) {
            prof[2 * blockIdx.x] = (int64_t)t_start;
            prof[2 * blockIdx.x + 1] = (int64_t)global_ns();
        }
    }
}

// ---------------------------------------------------------------------------
// Narrow update tasks (N <= 32 rows in block b: the leaves of 2D problems and
// thin separators): one warp per 32-row slab of the task, lane i owning row
// i's N outputs in registers.  The slab's A rows and B rows are staged per
// 32-column chunk of K in the warp's shared memory by 16-byte loads (a row's
// chunk over 32 / VE lanes, several rows per load), then C[i][j] += A[i][k]
// op(B[j][k]) in increasing k with B read as 16-byte broadcasts; the same flags
// as k_gemm_scatter (U-side operands, D-scaled A for LDL, conjugated B,
// lower-triangle-only targets) and the same scatter-add into the facing cblk,
// in single precision 16 bytes of a target row per reduction.  Scalar loads
// of B and of the rows, and 4-byte reductions, bounded it before: the narrow
// updates of 128 2D systems 7.5 -> 6.8 ms, of the 20^3 FP64 factor 0.24 ->
// 0.21 ms on one B200.
// ---------------------------------------------------------------------------
constexpr int GS_TM = 32, GS_TN = 32, GS_WARPS = 8;
template <typename T> constexpr int gs_pitch_b() { return 32 + 16 / (int)sizeof(T); }   // rows start 16-byte aligned
template <typename T> constexpr int gs_warp_elems() { return 32 * 33 + 32 * gs_pitch_b<T>(); }
template <typename T>
constexpr int gs_smem_bytes() { return GS_WARPS * gs_warp_elems<T>() * (int)sizeof(T); }

template <typename T>
__global__ void __launch_bounds__(GS_WARPS * 32, sizeof(T) == 4 ? 3 : 2) k_gemm_scatter_small(Meta m, const int4 *__restrict__ tiles,
                                                                       int ntiles, const GemmTask *__restrict__ tasks,
                                                                       T *__restrict__ coefL, T *__restrict__ coefU) {
    constexpr int VE = 16 / sizeof(T), QL = 32 / VE, RL = 32 / QL;   // elements per load; lanes per row, rows per load
    constexpr int PBT = gs_pitch_b<T>();
    extern __shared__ __align__(16) unsigned char gs_smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T *As = reinterpret_cast<T *>(gs_smem_raw) + warp * gs_warp_elems<T>();   // [k][i], stride 33
    T *Bs = As + 32 * 33;                                                      // [k][j], stride PBT
    const int ti = blockIdx.x * GS_WARPS + warp;
    if (ti >= ntiles) return;                 // whole warps; only warp-level synchronization below
    const int4 tl = tiles[ti];
    const GemmTask t = tasks[tl.x];
    const int c = t.c, b = t.b, f = t.f;
    const int K = m.width[c], ld = m.ld[c];
    const int N = m.blrow[b] - m.bfrow[b] + 1;
    const int i0 = tl.y * GS_TM;
    const int mrows = min(GS_TM, t.M - i0), ncols = min(GS_TN, N);
    const T *A = ((t.flags & 1) ? coefU : coefL) + m.coefoff[c] + (int64_t)(t.arow0 + i0) * ld;
    const T *Bm = ((t.flags & 2) ? coefU : coefL) + m.coefoff[c] + (int64_t)m.browoff[b] * ld;
    const T *Dg = coefL + m.coefoff[c];
    const bool scale_d = (t.flags & 16) != 0, conj_b = (t.flags & 32) != 0;
    int tr = -1;
    if (lane < mrows) tr = panel_row_of(m, f, m.rowidx[m.rowbase[c] + t.arow0 + i0 + lane]);
    T acc[GS_TN];
#pragma unroll
    for (int j = 0; j < GS_TN; j++) acc[j] = T(0);
    const int kq = (lane % QL) * VE, rq = lane / QL;   // this lane's columns of a chunk, its row of a load
    for (int k0 = 0; k0 < K; k0 += 32) {
        const int kn = min(32, K - k0);
        // (ld is a multiple of 4: a vector that starts inside the row ends inside its padding)
        T d[VE];
        if (scale_d)
#pragma unroll
            for (int v = 0; v < VE; v++) {
                const int k = k0 + kq + v;
                d[v] = k < K ? Dg[(int64_t)k * ld + k] : T(0);
            }
#pragma unroll 1
        for (int h = 0; h < QL; h += 4) {   // up to four loads of A and of B in flight (QL >= 8 rows' groups)
            uint4 ua[4], ub[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int r = (h + u) * RL + rq;
                ua[u] = ub[u] = make_uint4(0, 0, 0, 0);
                if (r < mrows && kq < kn) ua[u] = *reinterpret_cast<const uint4 *>(A + (int64_t)r * ld + k0 + kq);
                if (r < ncols && kq < kn) ub[u] = *reinterpret_cast<const uint4 *>(Bm + (int64_t)r * ld + k0 + kq);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int r = (h + u) * RL + rq;
                T a[VE], bv[VE];
                memcpy(a, &ua[u], 16);
                memcpy(bv, &ub[u], 16);
#pragma unroll
                for (int v = 0; v < VE; v++) {
                    As[(kq + v) * 33 + r] = scale_d ? a[v] * d[v] : a[v];
                    Bs[(kq + v) * PBT + r] = conj_b ? conj_v(bv[v]) : bv[v];
                }
            }
        }
        __syncwarp();
        for (int kk = 0; kk < kn; kk++) {
            const T a = As[kk * 33 + lane];
#pragma unroll
            for (int j = 0; j < GS_TN; j += VE)
                if (j < ncols) {
                    T bv[VE];
                    const uint4 u4 = *reinterpret_cast<const uint4 *>(Bs + kk * PBT + j);
                    memcpy(bv, &u4, 16);
#pragma unroll
                    for (int v = 0; v < VE; v++) acc[j + v] = fma_v(a, bv[v], acc[j + v]);
                }
        }
        __syncwarp();
    }
    if (tr < 0) return;
    T *C = ((t.flags & 4) ? coefU : coefL) + m.coefoff[f] + (int64_t)tr * m.ld[f];
    const int tcol0 = m.bfrow[b] - m.fcol[f];
    // columns the row takes: on the diagonal block (symmetric forms) up to the diagonal
    const int nvalid = (t.flags & 8) && tr < m.width[f] ? min(ncols, tr - tcol0 + 1) : ncols;
    if constexpr (sizeof(typename real_of<T>::type) == 4) {
        // 16-byte groups of the target row: group g takes source columns VE g - O .. VE g - O + VE - 1,
        // the offset O = tcol0 mod VE a compile-time constant per branch; columns outside add zero
        auto reduce = [&](auto oc) {
            constexpr int O = decltype(oc)::value;
            float *Cg = reinterpret_cast<float *>(C + tcol0 - O);
#pragma unroll
            for (int g = 0; g * VE - O < GS_TN; g++) {
                if (g * VE - O >= nvalid) break;
                T a[VE];
#pragma unroll
                for (int v = 0; v < VE; v++) {
                    const int j = g * VE - O + v;
                    a[v] = (j >= 0 && j < GS_TN) ? (j < nvalid ? T(0) - acc[j < 0 ? 0 : j >= GS_TN ? 0 : j] : T(0)) : T(0);
                }
                float r[4];
                memcpy(r, a, 16);
                red_add_v4(Cg + 4 * g, r[0], r[1], r[2], r[3]);
            }
        };
        if constexpr (VE == 4) {
            switch (tcol0 & 3) {
                case 0: reduce(std::integral_constant<int, 0>{}); break;
                case 1: reduce(std::integral_constant<int, 1>{}); break;
                case 2: reduce(std::integral_constant<int, 2>{}); break;
                default: reduce(std::integral_constant<int, 3>{}); break;
            }
        } else {
            if (tcol0 & 1) reduce(std::integral_constant<int, 1>{});
            else reduce(std::integral_constant<int, 0>{});
        }
    } else {
#pragma unroll
        for (int j = 0; j < GS_TN; j++)
            if (j < nvalid) atomic_sub(&C[tcol0 + j], acc[j]);
    }
}

}  // namespace pgpu
