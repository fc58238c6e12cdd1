// Update GEMM on the tensor cores with operands brought in by TMA
// (cp.async.bulk.tensor) instead of producer warps: the same task, tile and
// epilogue as k_gemm_scatter_tc_persistent, C = A B^T scatter-added into the
// facing cblk (kernels/core_zgemmsp.c:104 core_zgemmsp_1d1d).
//
// Operands: for 3xTF32 (SPLIT) the finished panel rows are split once into
// hi = tf32(x) and lo = x - hi by the level's split / copy-back kernels, into
// a mirror of the coeftab laid out [2][ncoef] (hi, then lo), and the
// diagonal-block inverses alike.  One tensor map per (cblk, operand kind)
// covers the panel as a 3-D tensor {K = w_c, rows = h_c, 2} with row stride
// ld_c and the hi/lo stride ncoef, so one box {32, 128, 2} lands the hi tile
// and the lo tile of a k-block (2 x 16 KB, SWIZZLE_128B, the canonical
// K-major layout the MMA descriptors expect).  Without the split the maps
// cover the coeftab itself, {K, rows, 1}.  Rows and columns past the panel
// are zero-filled by the TMA unit.
//
// Roles (384 threads, one CTA per SM walking the level's tiles):
//   warps 0-7: epilogue (TMEM -> registers, summed over the tile's segments
//              -> a swizzled 32 x 32 shared buffer per warp -> 16-byte vector
//              reductions along the target rows);
//   warp 8, lane 0: TMA producer -- per k-block waits for a free stage,
//              announces the stage's bytes on its mbarrier and issues the A
//              and B box loads;
//   warp 9, lane 0: MMA issuer (tcgen05.mma into one of two TMEM
//              accumulators, commits to the stage / accumulator barriers).
// Every wait is bounded; after a time-out the producer waits (bounded) for
// the loads it issued and TMEM is freed after all roles met.  The tensor
// maps name only this GPU's memory and the loads carry no multicast.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <type_traits>

#include "pgpu_common.cuh"
#include "pgpu_factor.cuh"
#include "pgpu_gemm_tc.cuh"

namespace pgpu {

// warps 0-7 gather and write back the accumulators (two warps per TMEM lane
// quarter, each taking every other 32-column chunk), warp 8 loads, warp 9
// issues the MMAs.  The epilogue warps hold a pair's sums (128 registers), so
// the third warpgroup hands them registers: 2 x 208 + 88 = 3 x 168, the
// launch's own share of 384 threads.
constexpr int TMA_THREADS = 384, TMA_EPI_WARPS = 8;
constexpr int TMA_PROD_WARP = 8, TMA_MMA_WARP = 9;
constexpr int TMA_REGS_EPI = 208, TMA_REGS_REST = 88;
constexpr int TMA_REGS_LAUNCH = 168;
static_assert(2 * TMA_REGS_EPI + TMA_REGS_REST == 3 * TMA_REGS_LAUNCH, "register split");
constexpr int TMA_EPI_BYTES = TMA_EPI_WARPS * 32 * 32 * 4;   // a swizzled 32 x 32 float buffer per warp
// operand maps per cblk: L panel, U panel (LU; LDL: the L rows times D), first / second diagonal-block
// inverse, and in complex arithmetic the L / U panels as B operands (two real rows per row, see below)
enum { TMAP_L = 0, TMAP_U = 1, TMAP_I = 2, TMAP_I2 = 3, TMAP_BL = 4, TMAP_BU = 5, TMAP_KINDS = 6 };
constexpr int TC_FLAG_CPLX = 256;   // TcDesc::flags: real and imaginary parts are neighbouring columns

// A stage holds two A tiles (a pair of 128-row tiles of one task sharing the
// B tile) and the B tile; hi and lo planes each for 3xTF32.
template <bool SPLIT> struct TmaCfg;
template <> struct TmaCfg<false> { static constexpr int STAGES = 4, TILES = 3, PL = 1; };
template <> struct TmaCfg<true> { static constexpr int STAGES = 2, TILES = 6, PL = 2; };
constexpr int TMA_TMEM_COLS = 512;   // two accumulator buffers x (two 128-column halves)
template <bool SPLIT>
constexpr int tma_smem_bytes() {
    return TmaCfg<SPLIT>::STAGES * TmaCfg<SPLIT>::TILES * TC_TILE_BYTES + TMA_EPI_BYTES + 1024;
}


// 3-D tiled TMA load into this CTA's shared memory, completing on mbar.
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2,
                                            uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
            "r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(mbar)
        : "memory");
}

// Everything the three roles need for one tile, built on the host when the
// plan is made: the kernel reads one 64-byte record per tile and one 48-byte
// record per segment (loaded one or two ahead) instead of walking tile -> task
// -> cblk tables through chains of dependent loads.
//
// A tile sums nseg segments: update tasks of different source cblks with the
// same target rows and columns (the cblks of one separator chain), each a
// product of its own depth and row scales.  The epilogue warps gather the
// segments' accumulators in registers and scatter the sum once: the atomic
// reductions into the target panel, which bound the kernel when every source
// writes its own (100^3: 41 GB of them), shrink by the number of segments.  A
// tile of one segment goes chunk by chunk from the accumulator to the target
// (through the registers of a whole tile it took a third longer).
// A segment may also be a part of its source's columns: the tensor core's
// additions cut off what lies below the accumulator's last bits, always
// towards zero, so that the error of a sum grows with its length faster than
// that of an FMA chain; the additions in the epilogue round to nearest.  With the
// fan-in what bounds the kernel is the latency of its loads: on 72^3, tensor
// pipe 43 % of active cycles, L2 23 %, DRAM below 15 %.
struct __align__(16) TcSeg {
    int mapa, mapb, rowa, rowb;   // tensor maps (indices into maps), first row of the task in A and in B
    int nk, kb0, pad[2];          // k-blocks, the first of them
    int64_t sa, sb;               // 3xFP16: scale index of those rows
};
struct __align__(16) TcDesc {
    int seg0, nseg, ncols, pair;  // segments, valid columns, paired 128-row tiles
    int flags, mrows, ldo, wf;    // task flags (64: TRSM), rows from the tile's first; target (or output) row
                                  // stride, target cblk width (lower-triangle rule)
    int tcol, i0, j0, pad;        // first target column; the tile's first row and column in its task
    int64_t off;                  // target panel offset from coefL, or (TRSM) output offset in scr
    int64_t rmap;                 // row-map index of the tile's first row (update tiles)
};
static_assert(sizeof(TcSeg) == 48 && sizeof(TcDesc) == 64, "whole 16-byte vectors");

// 2^e, and e of 2^e, for normal floats.
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }
__device__ __forceinline__ int pow2_exp(float x) { return (__float_as_int(x) >> 23) - 127; }

template <typename R>
__device__ __forceinline__ R tc_rec_load(const R *p) {
    R d;
    const int4 *s = reinterpret_cast<const int4 *>(p);
    int4 *o = reinterpret_cast<int4 *>(&d);
#pragma unroll
    for (int k = 0; k < (int)(sizeof(R) / 16); k++) o[k] = __ldg(s + k);
    return d;
}

// F16 (with SPLIT): "3xFP16" operands -- every row r of a source matrix
// (panel rows, diagonal-block inverse rows) is scaled by a power of two
// 2^e_r that brings its largest magnitude into [2^14, 2^15), then split into
// hi = fp16(x 2^e_r) and lo = fp16(x 2^e_r - hi) (both round to nearest):
// 11 + 11 significant bits, the precision of the 3xTF32 split, in half the
// bytes, on the FP16 MMA rate (twice the TF32 rate).  The k-block is 64
// halves (128 bytes, the same SWIZZLE_128B tile as 32 floats) and each MMA
// covers K = 16.  The epilogue multiplies the accumulator by the rows'
// inverse scales 2^-e_a 2^-e_b (hscale, one float per source row; hsbase
// gives each operand map's first row there), exact powers of two.
//
// Complex C = A op(B)^t as a real product of twice the columns and depth: a
// row of A is its interleaved (re, im) pairs as they lie in the panel; a row
// of B becomes two, whose products with it are the real and the imaginary
// part -- (re, -im) and (im, re), or for op = conj (re, im) and (-im, re) --
// so that neighbouring columns of the accumulator are re and im, as in the
// target panel, and the epilogue is the real one.
template <bool SPLIT, bool F16 = false>
__global__ void __launch_bounds__(TMA_THREADS, 1)
    k_gemm_scatter_tc_tma(const TcDesc *__restrict__ desc, const TcSeg *__restrict__ segs, int ntiles,
                          float *__restrict__ coefL, Status *st,
                          float *__restrict__ scr, const CUtensorMap *__restrict__ maps,
                          const int *__restrict__ tmap, const float *__restrict__ hscale = nullptr) {
    static_assert(!F16 || SPLIT, "the FP16 operands are always split");
    constexpr int S = TmaCfg<SPLIT>::STAGES, NT = TmaCfg<SPLIT>::TILES, PL = TmaCfg<SPLIT>::PL;
    constexpr int BK = F16 ? 64 : TC_BK;                              // elements per k-block (128 B per row)
    constexpr uint32_t BOX_BYTES = (uint32_t)PL * TC_TILE_BYTES;   // one operand box (hi [+ lo])
    constexpr int QA1 = PL, QB = 2 * PL;                            // tile slots of A1 and B in a stage
    extern __shared__ __align__(16) unsigned char tc_smem_raw[];
    __shared__ __align__(8) uint64_t full[S], empty[S], accf[2], acce[2], drained;
    __shared__ uint32_t tmem_base_s;
    __shared__ int fail_s;

    const uint32_t raw = smem_u32(tc_smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char *sbase = tc_smem_raw + (base - raw);
    float *epi = reinterpret_cast<float *>(sbase + S * NT * TC_TILE_BYTES);   // [8][32][32]

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == TMA_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                     "r"(TMA_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(smem_u32(&accf[b]), 1);
            mbar_init(smem_u32(&acce[b]), TMA_EPI_WARPS);
        }
        mbar_init(smem_u32(&drained), 1);
        fail_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;
    auto tile_addr = [&](int s, int q) { return base + (uint32_t)(s * NT + q) * TC_TILE_BYTES; };
    auto failed = [&]() { return *(volatile int *)&fail_s != 0; };

    if (warp >= TMA_EPI_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TMA_REGS_REST));
    if (warp == TMA_PROD_WARP) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            int it = 0;
            TcDesc nx{};
            TcSeg ns{};
            if (blockIdx.x < ntiles) {
                nx = tc_rec_load(desc + blockIdx.x);
                ns = tc_rec_load(segs + nx.seg0);
            }
            bool ok = true;
            for (int ti = blockIdx.x; ti < ntiles && ok && !failed(); ti += gridDim.x) {
                const TcDesc o = nx;
                const bool more = ti + (int)gridDim.x < ntiles;
                if (more) nx = tc_rec_load(desc + ti + gridDim.x);   // for the next tile
                const uint32_t bytes = (o.pair ? 3u : 2u) * BOX_BYTES;
                for (int g = 0; g < o.nseg && ok; g++) {
                    const TcSeg sg = ns;
                    if (g + 1 < o.nseg) ns = tc_rec_load(segs + o.seg0 + g + 1);
                    else if (more) ns = tc_rec_load(segs + nx.seg0);
                    const CUtensorMap *ma = maps + sg.mapa, *mbm = maps + sg.mapb;
                    const int rowa = sg.rowa + o.i0, rowb = sg.rowb + o.j0;
                    for (int kb = 0; kb < sg.nk; kb++, it++) {
                        const int s = it % S;
                        if (it >= S && !mbar_wait(smem_u32(&empty[s]), (uint32_t)((it / S - 1) & 1))) {
                            ok = false;
                            break;
                        }
                        mbar_arrive_expect_tx(smem_u32(&full[s]), bytes);
                        tma_load_3d(tile_addr(s, 0), ma, (sg.kb0 + kb) * BK, rowa, 0, smem_u32(&full[s]));
                        if (o.pair) tma_load_3d(tile_addr(s, QA1), ma, (sg.kb0 + kb) * BK, rowa + TC_BM, 0, smem_u32(&full[s]));
                        tma_load_3d(tile_addr(s, QB), mbm, (sg.kb0 + kb) * BK, rowb, 0, smem_u32(&full[s]));
                    }
                }
                if (!ok) atomicExch(&fail_s, 1);
            }
            if (failed()) {
                // the loads still in flight land before the CTA leaves; if one
                // of these waits gives up as well, the CTA may leave with bulk
                // copies still writing its shared memory: recorded apart, and the
                // host treats the whole factorization as failed
                for (int j = 1; j <= S && it - j >= 0; j++) {
                    const int k = it - j;
                    if (!mbar_wait(smem_u32(&full[k % S]), (uint32_t)((k / S) & 1))) atomicAdd(&st->drain_timeout, 1);
                }
            }
        }
    } else if (warp == TMA_MMA_WARP) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            int it = 0, cnt = 0;   // k-blocks, segments
            TcDesc nx{};
            TcSeg ns{};
            if (blockIdx.x < ntiles) {
                nx = tc_rec_load(desc + blockIdx.x);
                ns = tc_rec_load(segs + nx.seg0);
            }
            bool ok = true;
            for (int ti = blockIdx.x; ti < ntiles && ok && !failed(); ti += gridDim.x) {
                const TcDesc v = nx;
                const bool more = ti + (int)gridDim.x < ntiles;
                if (more) nx = tc_rec_load(desc + ti + gridDim.x);   // for the next tile
                const uint32_t idesc = F16 ? tc_idesc_f16(tc_mma_n(v.ncols)) : tc_idesc(tc_mma_n(v.ncols));
                const bool pair = v.pair != 0;
                for (int g = 0; g < v.nseg && ok; g++, cnt++) {
                    const TcSeg sg = ns;
                    if (g + 1 < v.nseg) ns = tc_rec_load(segs + v.seg0 + g + 1);
                    else if (more) ns = tc_rec_load(segs + nx.seg0);
                    const int ab = cnt & 1;
                    const uint32_t acc = tmem + (uint32_t)(ab * 256), acc1 = acc + 128u;
                    if (cnt >= 2 && !mbar_wait(smem_u32(&acce[ab]), (uint32_t)((cnt / 2 - 1) & 1))) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (int kb = 0; kb < sg.nk; kb++, it++) {
                        const int s = it % S;
                        if (!mbar_wait(smem_u32(&full[s]), (uint32_t)((it / S) & 1))) {
                            ok = false;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    #pragma unroll
                        for (int kk = 0; kk < TC_BK / 8; kk++) {
                            const uint32_t first = (kb > 0 || kk > 0) ? 1u : 0u;
                            if (SPLIT) {
                                const uint64_t bh = tc_sdesc(tile_addr(s, QB) + kk * 32),
                                               bl = tc_sdesc(tile_addr(s, QB + 1) + kk * 32);
    #pragma unroll
                                for (int h = 0; h < 2; h++) {
                                    if (h == 1 && !pair) break;
                                    const uint64_t ah = tc_sdesc(tile_addr(s, h * QA1) + kk * 32),
                                                   al = tc_sdesc(tile_addr(s, h * QA1 + 1) + kk * 32);
                                    const uint32_t ac = h ? acc1 : acc;
                                    if (F16) {
                                        tc_mma_f16(ac, al, bh, idesc, first);
                                        tc_mma_f16(ac, ah, bl, idesc, 1u);
                                        tc_mma_f16(ac, ah, bh, idesc, 1u);
                                    } else {
                                        tc_mma(ac, al, bh, idesc, first);
                                        tc_mma(ac, ah, bl, idesc, 1u);
                                        tc_mma(ac, ah, bh, idesc, 1u);
                                    }
                                }
                            } else {
                                const uint64_t bd = tc_sdesc(tile_addr(s, QB) + kk * 32);
                                tc_mma(acc, tc_sdesc(tile_addr(s, 0) + kk * 32), bd, idesc, first);
                                if (pair) tc_mma(acc1, tc_sdesc(tile_addr(s, QA1) + kk * 32), bd, idesc, first);
                            }
                        }
                        tc_commit(smem_u32(&empty[s]));
                    }
                    if (ok) tc_commit(smem_u32(&accf[ab]));
                }
                if (!ok) atomicExch(&fail_s, 1);
            }
            tc_commit(smem_u32(&drained));
            if (!mbar_wait(smem_u32(&drained), 0u)) atomicExch(&fail_s, 1);
        }
    }
    } else {
        // ---------------- epilogue (warps 0-7) ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TMA_REGS_EPI));
        // The next segment's row and column scales (and the next tile's
        // descriptor and target rows) are loaded before the wait on the
        // current segment's accumulator: their load chains stay off the path
        // of the reductions.
        const int qw = warp & 3;                       // TMEM lane quarter (rows 32 qw .. 32 qw + 31)
        const int grp = warp >> 2;                     // column chunks 32 grp, 32 grp + 64
        float *E = epi + warp * 32 * 32;
        const int myrow = qw * 32 + lane;
        struct Scales {
            float rs[2], cs[2];   // this lane's row of each half; column 32 grp + 64 x + lane
        };
        auto scales = [&](const TcDesc &d, int g) {
            Scales e;
            e.rs[0] = e.rs[1] = e.cs[0] = e.cs[1] = 1.f;
            if (F16) {
                const TcSeg *sg = segs + d.seg0 + g;
                const int64_t sa = __ldg(&sg->sa) + d.i0, sb = __ldg(&sg->sb) + d.j0;
                for (int h = 0; h < 2; h++) {
                    const int r = h * TC_BM + myrow, col = 32 * grp + 64 * h + lane;
                    e.rs[h] = ((h == 0 || d.pair) && r < d.mrows) ? hscale[sa + r] : 1.f;
                    e.cs[h] = col < d.ncols ? hscale[sb + col] : 1.f;
                }
            }
            return e;
        };
        auto targets = [&](const TcDesc &d, int (&tr)[2]) {
            for (int h = 0; h < 2; h++) {
                const int r = h * TC_BM + myrow;
                tr[h] = ((d.flags & 64) == 0 && (h == 0 || d.pair) && r < d.mrows) ? tmap[d.rmap + r] : -1;
            }
        };
        TcDesc v{}, vn{};
        Scales sc{};
        int trn[2] = {-1, -1};
        if (blockIdx.x < ntiles) {
            v = tc_rec_load(desc + blockIdx.x);
            sc = scales(v, 0);
            targets(v, trn);
        }
        int cnt = 0;
        bool ok = true;
        for (int ti = blockIdx.x; ti < ntiles && ok && __all_sync(0xffffffffu, !failed()); ti += gridDim.x) {
            const bool more = ti + (int)gridDim.x < ntiles;
            const int trw[2] = {trn[0], trn[1]};   // each lane's row target, shuffled to the writers
            if (more) vn = tc_rec_load(desc + ti + gridDim.x);
            const bool trsm = (v.flags & 64) != 0;
            const int nh = v.pair ? 2 : 1;
            float *C = coefL + v.off;
            const int ldf = v.ldo, wf = v.wf;
            const int tcol0 = v.tcol;
            const bool lower_only = (v.flags & 8) != 0;
            const int csh = (v.flags & TC_FLAG_CPLX) ? 1 : 0;
            // one 32 x 32 chunk (half h, columns cb ..) into the target
            auto put = [&](int h, int cb, const float (&xx)[32]) {
                const int mrows = min(TC_BM, v.mrows - h * TC_BM);   // valid rows of this half
                // this lane's row (TMEM lane) as eight 16-byte groups, group g at
                // slot g ^ (row & 7): conflict-free both for the row-wise stores
                // here and for the loads along a row / down a column below
#pragma unroll
                for (int g = 0; g < 8; g++)
                    *reinterpret_cast<float4 *>(E + lane * 32 + ((g ^ (lane & 7)) << 2)) =
                        make_float4(xx[4 * g], xx[4 * g + 1], xx[4 * g + 2], xx[4 * g + 3]);
                __syncwarp();
                const int j = cb + lane;
                if (j < v.ncols && trsm) {
                    const int ldc = v.ldo;
                    float *O = scr + v.off + (int64_t)h * TC_BM * ldc;
                    for (int rr = 0; rr < 32; rr++) {
                        const int i = qw * 32 + rr;
                        if (i >= mrows) break;
                        O[(int64_t)i * ldc + j] = E[rr * 32 + ((((lane >> 2) ^ (rr & 7)) << 2) | (lane & 3))];
                    }
                } else if (!trsm && cb < v.ncols) {
                    const int nvalid = min(32, v.ncols - cb);
                    const int tcs = tcol0 + cb, a0 = tcs & ~3;
                    const int trh = h ? trw[1] : trw[0];
                    // target group g (columns a0 + 4 g ..) takes source columns 4 g - O ..
                    // 4 g + 3 - O: the tail of group g - 1 and the head of group g, the
                    // offset O = tcs mod 4 a compile-time constant per branch
                    auto reduce = [&](auto oc) {
                        constexpr int O = decltype(oc)::value;
                        for (int k = lane; k < 32 * 9; k += 32) {
                            const int rr = k / 9, g = k - rr * 9;
                            const int t2 = __shfl_sync(0xffffffffu, trh, rr);
                            if (t2 < 0 || (O == 0 && g == 8)) continue;
                            const float *Er = E + rr * 32;
                            const int sw = rr & 7;
                            float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
                            if (O > 0 && g >= 1) lo = *reinterpret_cast<const float4 *>(Er + (((g - 1) ^ sw) << 2));
                            if (g <= 7) hi = *reinterpret_cast<const float4 *>(Er + ((g ^ sw) << 2));
                            float a[4];
                            if (O == 0) { a[0] = hi.x; a[1] = hi.y; a[2] = hi.z; a[3] = hi.w; }
                            if (O == 1) { a[0] = lo.w; a[1] = hi.x; a[2] = hi.y; a[3] = hi.z; }
                            if (O == 2) { a[0] = lo.z; a[1] = lo.w; a[2] = hi.x; a[3] = hi.y; }
                            if (O == 3) { a[0] = lo.y; a[1] = lo.z; a[2] = lo.w; a[3] = hi.x; }
                            const int j0 = 4 * g - O;   // source column of a[0]
                            if (j0 < 0 || j0 + 3 >= nvalid || lower_only) {
                                bool any = false;
#pragma unroll
                                for (int u = 0; u < 4; u++) {
                                    const int jj = j0 + u, tc = a0 + 4 * g + u;
                                    const bool ok = jj >= 0 && jj < nvalid && !(lower_only && t2 < wf && (tc >> csh) > t2);
                                    a[u] = ok ? a[u] : 0.f;
                                    any |= ok;
                                }
                                if (!any) continue;
                            }
                            red_add_v4(&C[(int64_t)t2 * ldf + a0 + 4 * g], a[0], a[1], a[2], a[3]);
                        }
                    };
                    switch (tcs - a0) {
                        case 0: reduce(std::integral_constant<int, 0>{}); break;
                        case 1: reduce(std::integral_constant<int, 1>{}); break;
                        case 2: reduce(std::integral_constant<int, 2>{}); break;
                        default: reduce(std::integral_constant<int, 3>{}); break;
                    }
                }
                __syncwarp();
            };
            // the update subtracts: the sign rides on the row scale
            const float sgn = trsm ? 1.f : -1.f;
            // chunk (h, y) of the accumulator, scaled.  Every lane needs every column's scale: they go through
            // the warp's buffer, read back as 16-byte broadcasts
            auto take = [&](int ab, int h, int y, float (&xx)[32], bool more_sums) {
                if (F16) E[lane] = y ? sc.cs[1] : sc.cs[0];
                uint32_t r[32];
                tc_ld32(tmem + (uint32_t)(ab * 256 + h * 128) + ((uint32_t)(qw * 32) << 16) +
                            (uint32_t)(32 * grp + 64 * y), r);
                __syncwarp();
                const float rsh = (h ? sc.rs[1] : sc.rs[0]) * sgn;
#pragma unroll
                for (int q = 0; q < 32; q += 4) {
                    float4 c = make_float4(1.f, 1.f, 1.f, 1.f);
                    if (F16) c = *reinterpret_cast<const float4 *>(E + q);
                    const float cs[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const float p = __uint_as_float(r[q + u]) * rsh;
                        xx[q + u] = more_sums ? fmaf(p, cs[u], xx[q + u]) : p * cs[u];
                    }
                }
                __syncwarp();
            };
            // An accumulator reaches 2^40: a row scale above 2^60 hands what it has beyond to the columns', so that
            // the product with the row scale stays in range where the product with both does (powers of two:
            // exact but for rows 2^130 below others of their 32)
            auto balance = [&]() {
                if (!F16 || !__any_sync(0xffffffffu, fmaxf(sc.rs[0], sc.rs[1]) > 0x1p60f)) return;
                const int re = __reduce_max_sync(0xffffffffu, pow2_exp(fmaxf(sc.rs[0], sc.rs[1])));
                const int ce = __reduce_max_sync(0xffffffffu, pow2_exp(fmaxf(sc.cs[0], sc.cs[1])));
                const int t = max(0, min(re - 60, 120 - ce));
                for (int h = 0; h < 2; h++) {
                    sc.rs[h] *= pow2f(-t);
                    sc.cs[h] *= pow2f(t);
                }
            };
            auto release = [&](int ab) {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&acce[ab]));
            };
            auto landed = [&](int n) {
                if (!mbar_wait_warp(smem_u32(&accf[n & 1]), (uint32_t)((n / 2) & 1))) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                return true;
            };
            if (v.nseg == 1) {
                // a single product: chunk by chunk from the accumulator to the target
                Scales sn{};
                if (more) {
                    sn = scales(vn, 0);
                    targets(vn, trn);
                }
                if (!landed(cnt)) {
                    atomicExch(&fail_s, 1);
                    break;
                }
                balance();
                for (int h = 0; h < nh; h++)
#pragma unroll
                    for (int y = 0; y < 2; y++) {
                        const int cb = 32 * grp + 64 * y;
                        if (cb >= v.ncols) continue;
                        float xx[32];
                        take(cnt & 1, h, y, xx, false);
                        put(h, cb, xx);
                    }
                release(cnt & 1);
                sc = sn;
                cnt++;
            } else {
                float x[2][2][32];   // [half][column chunk][column]
                for (int g = 0; g < v.nseg; g++, cnt++) {
                    Scales sn{};
                    if (g + 1 < v.nseg) {
                        sn = scales(v, g + 1);
                    } else if (more) {
                        sn = scales(vn, 0);
                        targets(vn, trn);
                    }
                    if (!landed(cnt)) {
                        ok = false;
                        break;
                    }
                    balance();
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int y = 0; y < 2; y++)
                            if (h < nh && 32 * grp + 64 * y < v.ncols) take(cnt & 1, h, y, x[h][y], g > 0);
                    release(cnt & 1);
                    sc = sn;
                }
                if (!ok) {
                    atomicExch(&fail_s, 1);
                    break;
                }
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int y = 0; y < 2; y++)
                        if (h < nh && 32 * grp + 64 * y < v.ncols) put(h, 32 * grp + 64 * y, x[h][y]);
            }
            v = vn;
        }
    }
    if (tid == 0 && failed()) atomicAdd(&st->timeout, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == TMA_MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMA_TMEM_COLS)
                     : "memory");
    }
}

// hi / lo split of panel rows for the TMA operands: rows [r0, r0 + 32) of
// cblk c's panel (L, or U^t when the job's panel flag is set), w columns, into
// hilo[0][...] = tf32(x) and hilo[ncoef][...] = x - tf32(x), same offsets as
// the coeftab.  Jobs: {cblk, first row, panel, -}.
__global__ void k_split_rows(Meta m, const int4 *__restrict__ jobs, const float *__restrict__ coefL,
                             const float *__restrict__ coefU, float *__restrict__ hilo, int64_t ncoef,
                             int64_t coefnbr) {
    const int4 jb = jobs[blockIdx.x];
    const int c = jb.x, r0 = jb.y;
    const int w = m.width[c], h = m.height[c], ld = m.ld[c];
    const int nr = min(32, h - r0);
    const int64_t off = m.coefoff[c] + (jb.z ? coefnbr : 0) + (int64_t)r0 * ld;
    const float *src = (jb.z ? coefU : coefL) + m.coefoff[c] + (int64_t)r0 * ld;
    float *hi = hilo + off, *lo = hilo + ncoef + off;
    const int wv = (w + 3) >> 2;   // float4 per row (the panel's rows are 16-byte aligned, ld % 4 == 0)
    for (int e = threadIdx.x; e < nr * wv; e += blockDim.x) {
        const int i = e / wv, q = e - i * wv;
        const float4 x = reinterpret_cast<const float4 *>(src + (int64_t)i * ld)[q];
        float4 h4, l4;
        h4.x = tf32_hi(x.x); h4.y = tf32_hi(x.y); h4.z = tf32_hi(x.z); h4.w = tf32_hi(x.w);
        l4.x = x.x - h4.x; l4.y = x.y - h4.y; l4.z = x.z - h4.z; l4.w = x.w - h4.w;
        reinterpret_cast<float4 *>(hi + (int64_t)i * ld)[q] = h4;
        reinterpret_cast<float4 *>(lo + (int64_t)i * ld)[q] = l4;
    }
}

// ---------------------------------------------------------------------------
// 3xFP16 operands: per-row power-of-two scaling and hi / lo split.
//
// Row scale: the largest magnitude m of the row has binary exponent E
// (2^E <= m < 2^(E+1)); e = 14 - E puts it in [2^14, 2^15), below the FP16
// maximum 65504 and far above its normal minimum 2^-14.  e is clamped to
// [-126, 126] so that 2^e and 2^-e are normal floats (an all-zero row keeps
// e = 0).  The row's stored scale is 2^-e, which the GEMM epilogue applies.

// One warp splits one row of nf floats (complex: interleaved parts; src 16-byte
// aligned, padded to a multiple of 4): optionally times dsc (one factor per
// matrix column), an FP32 copy to dst, hi / lo halves at ha and ha + hplane
// (an A operand, or real B) with the inverse scale at *sa, and (complex) the
// two rows of a B operand at hb and hb + ldb with their scales at sb[0 .. 1].
template <typename T>
__device__ __forceinline__ void split_row_h16(const T *__restrict__ src_t, int nf, const T *dsc, T *__restrict__ dst_t,
                                              __half *__restrict__ ha, float *__restrict__ sa,
                                              __half *__restrict__ hb, int ldb, float *__restrict__ sb, bool conjb,
                                              int64_t hplane, int lane) {
    constexpr bool CX = is_cplx<T>::value;
    constexpr int RV = CX ? 8 : 4;   // the whole row in registers (at most 400 columns): read once, all loads in flight
    const float *src = reinterpret_cast<const float *>(src_t);
    float *dst = reinterpret_cast<float *>(dst_t);
    const int nq = (nf + 3) >> 2;
    float x[RV][4];
    float mx = 0.f;
#pragma unroll
    for (int u = 0; u < RV; u++) {
        const int q = lane + 32 * u;
        float4 v = q < nq ? __ldg(reinterpret_cast<const float4 *>(src) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[u][0] = v.x; x[u][1] = v.y; x[u][2] = v.z; x[u][3] = v.w;
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (4 * q + e >= nf) x[u][e] = 0.f;
    }
    if (dsc) {
#pragma unroll
        for (int u = 0; u < RV; u++) {
            const int q = lane + 32 * u;
            if (q >= nq) continue;
            if constexpr (CX) {
#pragma unroll
                for (int e = 0; e < 4; e += 2)
                    if (4 * q + e < nf) {
                        const T y = T(x[u][e], x[u][e + 1]) * dsc[2 * q + e / 2];
                        x[u][e] = y.re;
                        x[u][e + 1] = y.im;
                    }
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (4 * q + e < nf) x[u][e] *= dsc[4 * q + e];
            }
        }
    }
#pragma unroll
    for (int u = 0; u < RV; u++)
#pragma unroll
        for (int e = 0; e < 4; e++) mx = fmaxf(mx, fabsf(x[u][e]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    int ex = 0;
    if (mx > 0.f) {
        const int E = ((__float_as_int(mx) >> 23) & 0xff) - 127;
        ex = max(-126, min(126, 14 - E));
    }
    const float s = pow2f(ex);
    if (lane == 0) {
        if (ha) *sa = pow2f(-ex);
        if (CX && hb) sb[0] = sb[1] = pow2f(-ex);
    }
    auto put = [&](__half *row, int q, __half a, __half b, __half c, __half d) {
        __half2 v[2] = {__halves2half2(a, b), __halves2half2(c, d)};
        uint2 w;
        memcpy(&w, v, 8);
        reinterpret_cast<uint2 *>(row)[q] = w;
    };
#pragma unroll
    for (int u = 0; u < RV; u++) {
        const int q = lane + 32 * u;
        if (q < nq) {
            if (dst) reinterpret_cast<float4 *>(dst)[q] = make_float4(x[u][0], x[u][1], x[u][2], x[u][3]);
            __half h[4], l[4];
#pragma unroll
            for (int v = 0; v < 4; v++) {
                const float y = x[u][v] * s;
                h[v] = __float2half_rn(y);
                l[v] = __float2half_rn(y - __half2float(h[v]));
            }
            if (ha) {
                put(ha, q, h[0], h[1], h[2], h[3]);
                put(ha + hplane, q, l[0], l[1], l[2], l[3]);
            }
            if (CX && hb) {
                __half *b1 = hb + ldb;
                if (conjb) {
                    put(hb, q, h[0], h[1], h[2], h[3]);
                    put(hb + hplane, q, l[0], l[1], l[2], l[3]);
                    put(b1, q, __hneg(h[1]), h[0], __hneg(h[3]), h[2]);
                    put(b1 + hplane, q, __hneg(l[1]), l[0], __hneg(l[3]), l[2]);
                } else {
                    put(hb, q, h[0], __hneg(h[1]), h[2], __hneg(h[3]));
                    put(hb + hplane, q, l[0], __hneg(l[1]), l[2], __hneg(l[3]));
                    put(b1, q, h[1], h[0], h[3], h[2]);
                    put(b1 + hplane, q, l[1], l[0], l[3], l[2]);
                }
            }
        }
    }
}

// Target rows of the tensor-core update tasks, once per plan: for task
// tlist[blockIdx.x] and each row i of its M rows, the panel row of the facing
// cblk that source row arow0 + i lands in (kernels/core_zgemmsp.c:170-250
// walks the facing blocks for this).  tmap[taux[task] + i].
__global__ void k_task_rowmap(Meta m, const GemmTask *__restrict__ tasks, const int *__restrict__ tlist,
                              const int64_t *__restrict__ taux, int *__restrict__ tmap) {
    const int id = tlist[blockIdx.x];
    const GemmTask t = tasks[id];
    const int64_t base = taux[id];
    const int *rows = m.rowidx + m.rowbase[t.c] + t.arow0;
    for (int i = threadIdx.x; i < t.M; i += blockDim.x) tmap[base + i] = panel_row_of(m, t.f, rows[i]);
}

// Layout of the FP16 planes: per operand map (mapidx[c] + kind) the first
// element in the planes (hoff, rows of ld16 halves, a multiple of 64 that holds
// the row's floats, so that no 128-byte box row straddles two lines: 80^3 LU
// 39.1 -> 38.8 ms) and the first row in hscale (hsbase).
// pitch: 64 halves, whole 128-byte lines, one per box row; 8 (the alignment of a tensor map's rows) where memory is short
__host__ __device__ inline int ld16_of(int nf, int pitch) { return (nf + pitch - 1) & -pitch; }
constexpr int H16_MAXW = 400;   // widest cblk (pastix_gpu_structure)

// The pivots of cblk c (LDL: diagonal of its panel) into shared memory.
template <typename T>
__device__ __forceinline__ void load_pivots(const T *__restrict__ panel, int w, int ld, T *ds) {
    for (int j = threadIdx.x; j < w; j += blockDim.x) ds[j] = panel[(int64_t)j * ld + j];
}

// Split jobs {cblk, first row, kind (TMAP_*), -}: rows [r0, r0 + 32) of the
// source matrix of that kind (L / U panel rows, LDL: L times D for TMAP_U, or
// the rows of the first / second diagonal-block inverse), one warp per row.
template <typename T>
__global__ void __launch_bounds__(256) k_split_rows_h16(Meta m, const int4 *__restrict__ jobs,
                                                        const T *__restrict__ coefL, const T *__restrict__ coefU,
                                                        const T *__restrict__ inv, __half *__restrict__ h16,
                                                        int64_t hplane, float *__restrict__ hscale,
                                                        const int64_t *__restrict__ hoff,
                                                        const int64_t *__restrict__ hsbase,
                                                        const int *__restrict__ mapidx, int pitch, int ldl, int cj) {
    constexpr bool CX = is_cplx<T>::value;
    __shared__ __align__(16) unsigned char ds_raw[H16_MAXW * sizeof(T)];
    T *ds = reinterpret_cast<T *>(ds_raw);
    const int4 jb = jobs[blockIdx.x];
    const int c = jb.x, r0 = jb.y, kind = jb.z;
    const int w = m.width[c], ld = m.ld[c], nf = CX ? 2 * w : w, l16 = ld16_of(nf, pitch);
    const bool isinv = kind == TMAP_I || kind == TMAP_I2, upper = kind == TMAP_U || kind == TMAP_BU;
    const int rows = isinv ? w : m.height[c];
    const T *src = isinv ? inv + m.invoff[c] + (kind == TMAP_I2 ? inv_span(w, ld) : 0)
                         : ((upper && !ldl) ? coefU : coefL) + m.coefoff[c];
    const int mi = mapidx[c] + kind;
    const bool pair = CX && kind >= TMAP_I;   // a B operand of complex data
    const T *dsc = nullptr;
    if (ldl && kind == TMAP_U) {
        load_pivots(coefL + m.coefoff[c], w, ld, ds);
        __syncthreads();
        dsc = ds;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r1 = min(r0 + 32, rows);
    for (int i = r0 + warp; i < r1; i += blockDim.x >> 5) {
        const int row = pair ? 2 * i : i;
        __half *h = h16 + hoff[mi] + (int64_t)row * l16;
        float *sc = hscale + hsbase[mi] + row;
        split_row_h16<T>(src + (int64_t)i * ld, nf, dsc, nullptr, pair ? nullptr : h, sc, pair ? h : nullptr, l16, sc,
                         cj && !isinv, hplane, lane);
    }
}

// TRSM copy-back with the FP16 split: rows [r0, r0 + 32) of the level's
// TRSM output (chunks {cblk, r0, side, -} as k_trsm_copyback) into the panel
// and, when the cblk is a tensor-core source, into the FP16 planes its
// updates read.
template <typename T>
__global__ void __launch_bounds__(256) k_trsm_copyback_h16(Meta m, const int4 *__restrict__ chunks,
                                                           const int64_t *__restrict__ scroff,
                                                           const T *__restrict__ scr, T *__restrict__ coefL,
                                                           T *__restrict__ coefU, __half *__restrict__ h16,
                                                           int64_t hplane, float *__restrict__ hscale,
                                                           const int64_t *__restrict__ hoff,
                                                           const int64_t *__restrict__ hsbase,
                                                           const int *__restrict__ mapidx, int pitch, int ldl, int cj) {
    constexpr bool CX = is_cplx<T>::value;
    __shared__ __align__(16) unsigned char ds_raw[H16_MAXW * sizeof(T)];
    T *ds = reinterpret_cast<T *>(ds_raw);
    const int4 ch = chunks[blockIdx.x];
    const int c = ch.x, r0 = ch.y;
    const int w = m.width[c], h = m.height[c], ld = m.ld[c], nf = CX ? 2 * w : w, l16 = ld16_of(nf, pitch);
    const int nr = min(32, h - r0);
    const T *src = scr + scroff[c] + (ch.z ? inv_span(h - w, ld) : 0) + (int64_t)(r0 - w) * ld;
    T *dst = (ch.z ? coefU : coefL) + m.coefoff[c] + (int64_t)r0 * ld;
    const int mb = mapidx[c];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (mb < 0) {   // not a tensor-core source: the FP32 rows only
        for (int e = threadIdx.x; e < nr * w; e += blockDim.x) {
            const int i = e / w, j = e - i * w;
            dst[(int64_t)i * ld + j] = src[(int64_t)i * ld + j];
        }
        return;
    }
    if (ldl) {
        load_pivots(coefL + m.coefoff[c], w, ld, ds);
        __syncthreads();
    }
    const int ka = mb + (ch.z ? TMAP_U : TMAP_L), kb = mb + (ch.z ? TMAP_BU : TMAP_BL);
    const bool rowsa = !(CX && ldl);   // (complex LDL: the updates read L D and the B rows only)
    for (int i = warp; i < nr; i += blockDim.x >> 5) {
        const T *row = src + (int64_t)i * ld;
        split_row_h16<T>(row, nf, nullptr, dst + (int64_t)i * ld,
                         rowsa ? h16 + hoff[ka] + (int64_t)(r0 + i) * l16 : nullptr,
                         rowsa ? hscale + hsbase[ka] + r0 + i : nullptr,
                         CX ? h16 + hoff[kb] + (int64_t)(2 * (r0 + i)) * l16 : nullptr, l16,
                         CX ? hscale + hsbase[kb] + 2 * (r0 + i) : nullptr, cj, hplane, lane);
        if (ldl)
            split_row_h16<T>(row, nf, ds, nullptr, h16 + hoff[mb + TMAP_U] + (int64_t)(r0 + i) * l16,
                             hscale + hsbase[mb + TMAP_U] + r0 + i, nullptr, 0, nullptr, false, hplane, lane);
    }
}

}  // namespace pgpu
