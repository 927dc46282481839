// The face loops with an L2 prefetch of the tile one wave ahead, and the
// tile descriptors they read (built once per mesh).
//
// Cells are cut into tiles of TILE_CELLS = 256 consecutive internal cells
// (eight SELL slices). Because faces are numbered by owner slice, everything
// a tile reads in order is one contiguous range of device memory: its
// incidence entries, the records (and gface values) of the faces its cells
// own, and its cells' entries in every cell array (prefetch.cuh).
#pragma once

#include "kernels_adj.cuh"
#include "prefetch.cuh"

namespace cupcfd_gpu {

// Threads per block of each kernel, by list form. Measured on full lists: the
// FP32 step on a permuted 192^3 mesh 431 us in 64-thread blocks (gradient
// adjoint in 256), 425 in 128, 431 in 256, 464 in 512; FP64 forward and
// adjoint at 96^3 70 / 92 in 64, 72 / 87 in 128, 74 / 90 in 256.
template <int WF> constexpr int PF_BLOCK_FWD = 64;
template <int WF> constexpr int PF_BLOCK_ADJ = WF == 0 ? 256 : 64;
template <int WF> constexpr int PF_BLOCK_FWD_F64 = 64;
template <int WF> constexpr int PF_BLOCK_ADJ_F64 = 128;
template <int WF> constexpr int PF_BLOCK_FWD_MADJ = WF == -6 ? 64 : 128;
template <int WF> constexpr int PF_BLOCK_GADJ = WF == -6 ? 64 : 128;
template <int WF> constexpr int PF_BLOCK_MADJ = 256;
template <int WF> constexpr int PF_BLOCK_MADJ_F64 = 128;
template <int WF> constexpr int PF_BLOCK_GRAD = WF == 0 ? 64 : 128;
template <int WF> constexpr int PF_BLOCK_GRAD_ADJ = 128;

// Entries per chunk, whether the next chunk's entries load during the current
// chunk's arithmetic, and the tiles' worth of blocks per SM the registers
// allow. In run form the entries come from one cache line, so one face at a
// time with the next entry ahead leaves registers for more warps, which
// counts for more: FP32 forward at 256^3 382 us at 1 / ahead / 6 (455 at
// 3 / no / 4, 410 at 1 / ahead / 5, 424 at 1 / ahead / 7), FP32 adjoint 471 at
// 1 / ahead / 4 (493 at 2 / no / 4, 544 at 1 / ahead / 5), FP64 forward 604 at
// 1 / ahead / 4 (748 at 2 / no / 3; 1 / no / 4 613; five and six tiles spill),
// gradient adjoint 237 at 1 / ahead / 7 and 8 (247 at 2 / ahead / 6; gathered
// into shared memory like the forward+mass adjoint 240, and 848 against 841
// us a step under the power limit). The FP64 forward stays at 2 / 3 on full
// lists: 2 / 2 takes 68 against 72 at 96^3, but 15 against 13 at 48^3 and the
// same from 128^3 on.
// Lists of varying width (meshes of merged hexahedra, 6 to 26 faces a cell, at
// 5,220 / 136,991 / 632,627 cells): FP32 adjoint with the entries ahead in
// 256-thread blocks 14.5 / 24.9 / 103 us, in 64-thread blocks 12.6 / 26.9 /
// 106, without the entries ahead 14.7 / 26.9 / 112, plain kernel 14.7 / 25.0 /
// 108 (three entries spill: 206).
template <int WF> constexpr int PF_CHUNK_FWD = WF == -6 ? 1 : 3;
template <int WF> constexpr int PF_PIPE_FWD = WF == -6;
template <int WF> constexpr int PF_MINB_FWD = WF == -6 ? 6 : 4;
template <int WF> constexpr int PF_CHUNK_ADJ = WF == -6 ? 1 : 2;
template <int WF> constexpr int PF_PIPE_ADJ = WF != 6;
constexpr int PF_MINB_ADJ = 4;
template <int WF> constexpr int PF_CHUNK_FWD_F64 = WF == -6 ? 1 : 2;
template <int WF> constexpr int PF_PIPE_FWD_F64 = WF == -6;
template <int WF> constexpr int PF_MINB_FWD_F64 = WF == -6 ? 4 : 3;
// The FP64 adjoint in two forms (forms_setup in api.cu chooses): DEEP, more
// values in flight per thread, and more warps. Its mass part is as DEEP.
template <int WF, bool DEEP> constexpr int PF_CHUNK_ADJ_F64 = DEEP ? (WF == 6 ? 3 : 2) : 1;
template <int WF, bool DEEP> constexpr int PF_MINB_ADJ_F64 = DEEP ? 2 : WF == 0 ? 3 : 4;
template <int WF> constexpr int PF_CHUNK_GADJ = WF == -6 ? 1 : 2;
template <int WF> constexpr int PF_MINB_GADJ = WF == -6 ? 7 : 6;

// Entries per chunk of the gradient kernels, and the tiles' worth of blocks
// per SM the registers allow. At 128^3 (112^3 permuted for the correction),
// all in 128-thread blocks: one FP64 gradient 56 us at 2 / 4 (3 / 4 60, 1 / 6
// 59, 6 / 3 in 256-thread blocks 68), against 106 for the plain kernel. An
// iteration with the correction carries fourteen values per face: three
// iterations on the permuted mesh 352 us at 2 / 2 (110 registers; 1 / 3 374,
// 1 / 4 spilling 451) against 449 for the plain kernels with a copy after each
// iteration; on rows in run form 314 at 1 / 3, 333 at 2 / 2, against 527. The
// general adjoint 3 / 3: with the mass adjoint 154 us, 2 / 4 156, 1 / 4 160,
// against 241 (its plain kernel took the incidences one by one, with a
// division each). On lists of varying width (the meshes above) one FP32 gradient
// takes 8.6 / 15.7 / 61 us DEEP, 4 / 3 in 64-thread blocks, against 10.6 / 15.9
// / 74 at 2 / 4 in 128-thread blocks and 9.6 / 16.7 / 62 for the plain kernel;
// the FP64 one 10.6 / 24.6 / 90 DEEP, 12.6 / 18.9 / 96 at 2 / 4, 10.5 / 22.3 /
// 109 plain (forms_setup in api.cu chooses).
template <bool CORR, int WF, bool DEEP> constexpr int PF_CHUNK_GRAD = CORR ? (WF == -6 ? 1 : 2) : DEEP ? 4 : 2;
template <bool CORR, int WF, bool DEEP> constexpr int PF_MINB_GRAD = CORR ? (WF == -6 ? 3 : 2) : DEEP ? 3 : 4;
constexpr int PF_CHUNK_GRAD_ADJ = 3, PF_MINB_GRAD_ADJ = 3;

// ---------------------------------------------------------------------------
// L2 prefetch variant: the unstaged one-cell-per-thread kernels (the same
// per-cell bodies, so bit-identical results), where one lane per 256-cell
// block asks L2 to fetch the contiguous ranges of the tile `dist` blocks
// ahead (cp.async.bulk.prefetch.L2). Shared memory and L1 are untouched;
// the streamed loads of later blocks become L2 hits.
//
// WF: 0 for any mesh; -6 lists in run form (CellList in sell.cuh); 6 when every cell has exactly six incidences (all
// hexahedral meshes: every slice six entries wide, no padding). The cell
// loop then has a compile-time trip count: no padding checks, the chunks
// unrolled and their loads scheduled across chunks (same arithmetic in the
// same order, so the same bits).
// ---------------------------------------------------------------------------

// The separate forward and FP32 adjoint kernels run in blocks of 64 threads
// (TileBlock), the forwards with one loss
// partial per warp, folded per tile by k_group_partials before the fixed-
// order sum. At 256^3 on one box: FP32 forward 0.477-0.485 ms against
// 0.503-0.533 in 256-thread blocks, FP32 adjoint 0.518-0.529 against
// 0.543-0.583, FP64 forward 0.698-0.704 against 0.707-0.717.
template <int WF>
__global__ void __launch_bounds__(PF_BLOCK_FWD<WF>, PF_MINB_FWD<WF> *TILE_CELLS / PF_BLOCK_FWD<WF>)
    k_fwd_f32_pf(int nC, SellView sv, const float4 *__restrict__ fg, const float *__restrict__ phi,
                 const float *__restrict__ phiB, const double *__restrict__ vol, const float4 *__restrict__ st,
                 const float *__restrict__ gface, float *__restrict__ g, float *__restrict__ mflux,
                 double *__restrict__ lossPart, int64_t ldc, PrefetchArgs pf) {
    constexpr int T = TILE_CELLS;
    const TileBlock<PF_BLOCK_FWD<WF>> tb(pf);
    const int c = tb.c;
    __shared__ int4 s_rng;
    const void *const cellSrc[3] = {phi, st, vol};
    const int cellBytes[3] = {T * 4, T * 16, T * 8};
    if (tb.lead) fetch_ranges_async(&s_rng, pf.desc + tb.tp);
    double l = 0.0;
    if (c < nC) l = fwd_cell_f32<PF_CHUNK_FWD<WF>, PF_PIPE_FWD<WF>, WF>(c, sv, fg, phi, phiB, vol, st, gface, g, mflux, ldc);
    if (tb.lead) prefetch_tile<3>(pf, tb.tp, ranges_ready(&s_rng), fg, 16, gface, cellSrc, cellBytes);
    if (lossPart) warp_partial_store<PF_BLOCK_FWD<WF>>(l, c, lossPart);
}

template <int WF>
__global__ void __launch_bounds__(PF_BLOCK_ADJ<WF>, PF_MINB_ADJ *TILE_CELLS / PF_BLOCK_ADJ<WF>)
    k_adj_f32_pf(int nC, SellView sv, const float4 *__restrict__ fg, const float *__restrict__ g, float hscale,
                 const float4 *__restrict__ st, const float *__restrict__ gface, float *__restrict__ phibar,
                 float *__restrict__ phibBar, float4 *__restrict__ stbar, int64_t ldc, PrefetchArgs pf) {
    constexpr int T = TILE_CELLS;
    const TileBlock<PF_BLOCK_ADJ<WF>> tb(pf);
    const int c = tb.c;
    __shared__ int4 s_rng;
    const void *const cellSrc[4] = {g, g + ldc, g + 2 * ldc, st};
    const int cellBytes[4] = {T * 4, T * 4, T * 4, T * 16};
    if (tb.lead) fetch_ranges_async(&s_rng, pf.desc + tb.tp);
    if (c < nC) adj_cell_f32<false, PF_CHUNK_ADJ<WF>, PF_PIPE_ADJ<WF>, WF>(c, sv, fg, g, hscale, st, gface, phibar, phibBar, stbar, ldc);
    if (tb.lead) prefetch_tile<4>(pf, tb.tp, ranges_ready(&s_rng), fg, 16, gface, cellSrc, cellBytes);
}

// FP64 forward (fwd_cell_f64, exact reference arithmetic) with the same L2
// prefetch; the state's four component blocks are prefetched one by one.
template <int WF>
__global__ void __launch_bounds__(PF_BLOCK_FWD_F64<WF>, PF_MINB_FWD_F64<WF> *TILE_CELLS / PF_BLOCK_FWD_F64<WF>)
    k_fwd_f64_pf(int nC, SellView sv, const double4 *__restrict__ fg, const double *__restrict__ phi,
                 const double *__restrict__ phiB, const double *__restrict__ vol, const double *__restrict__ st,
                 const double *__restrict__ gface, double *__restrict__ g, double *__restrict__ mflux,
                 double *__restrict__ lossPart, int64_t ldc, PrefetchArgs pf) {
    constexpr int T = TILE_CELLS;
    const TileBlock<PF_BLOCK_FWD_F64<WF>> tb(pf);
    const int c = tb.c;
    __shared__ int4 s_rng;
    const void *const cellSrc[6] = {phi, vol, st, st + ldc, st + 2 * ldc, st + 3 * ldc};
    const int cellBytes[6] = {T * 8, T * 8, T * 8, T * 8, T * 8, T * 8};
    if (tb.lead) fetch_ranges_async(&s_rng, pf.desc + tb.tp);
    double l = 0.0;
    if (c < nC) l = fwd_cell_f64<PF_CHUNK_FWD_F64<WF>, PF_PIPE_FWD_F64<WF>, WF>(c, sv, fg, phi, phiB, vol, st, gface, g, mflux, ldc);
    if (tb.lead) prefetch_tile<6>(pf, tb.tp, ranges_ready(&s_rng), fg, 32, gface, cellSrc, cellBytes);
    if (lossPart) warp_partial_store<PF_BLOCK_FWD_F64<WF>>(l, c, lossPart);
}

// FP64 adjoint (adj_cell_f64) with the same L2 prefetch.
template <int WF, bool DEEP>
__global__ void __launch_bounds__(PF_BLOCK_ADJ_F64<WF>, PF_MINB_ADJ_F64<WF, DEEP> *TILE_CELLS / PF_BLOCK_ADJ_F64<WF>)
    k_adj_f64_pf(int nC, SellView sv, const double4 *__restrict__ fg, const double *__restrict__ g, double hscale,
                 const double *__restrict__ st, const double *__restrict__ gface, double *__restrict__ phibar,
                 double *__restrict__ phibBar, double *__restrict__ stbar, int64_t ldc, PrefetchArgs pf) {
    constexpr int T = TILE_CELLS;
    const TileBlock<PF_BLOCK_ADJ_F64<WF>> tb(pf);
    const int c = tb.c;
    __shared__ int4 s_rng;
    const void *const cellSrc[7] = {g, g + ldc, g + 2 * ldc, st, st + ldc, st + 2 * ldc, st + 3 * ldc};
    const int cellBytes[7] = {T * 8, T * 8, T * 8, T * 8, T * 8, T * 8, T * 8};
    if (tb.lead) fetch_ranges_async(&s_rng, pf.desc + tb.tp);
    if (c < nC) adj_cell_f64<false, PF_CHUNK_ADJ_F64<WF, DEEP>, WF>(c, sv, fg, g, hscale, st, gface, phibar, phibBar, stbar, ldc);
    if (tb.lead) prefetch_tile<7>(pf, tb.tp, ranges_ready(&s_rng), fg, 32, gface, cellSrc, cellBytes);
}

// Forward with the mass-flux adjoint (fwd_madj_cell_f32), L2 prefetch as
// k_fwd_f32_pf. With k_gadj_f32_pf it forms the two-launch forward+adjoint:
// the state and gface are then read by one pass only.
//
// It runs in blocks of PF_BLOCK_FWD_MADJ threads, several per tile, at
// the same registers and warps per SM as 256-thread blocks: a block's slot
// frees when its two warps end instead of its slowest of eight (measured at
// 256^3, 64 threads: 0.543 ms against 0.568 ms; 32-thread blocks 0.540). The last block
// of a tile prefetches for the tile. The loss partials are one per warp,
// warp k of tile t at lossPart[k nTiles + t]; k_reduce_partials<8> sums each
// tile's eight in order, which gives the per-tile value of
// block_sum_store<256> bit for bit.
//
// On lists in run form (WF -6) the faces past the first two are gathered into
// shared memory (fwd_madj_cell_staged; 10 KB a block, 160 KB an SM) at the same
// 64 registers and 32 warps per SM. At 256^3, 50-step runs on one box:
// 0.480-0.485 ms against 0.540 with the lists and gathers of two faces at a
// time; the run form alone 0.555, and roles known at compile time cut its
// instructions from 752 to about 620 a warp (0.83 against 0.86 ms for the
// step under the power limit). Five tiles a SM (48 registers) 0.567, three
// (24 warps) 0.54. It moves 2.04 GB; issue slots are 61% busy (at 128^3).
#ifndef CUPCFD_FWD_MADJ_CHUNK
#define CUPCFD_FWD_MADJ_CHUNK 2
#endif
#ifndef CUPCFD_MINB_FWD_MADJ
#define CUPCFD_MINB_FWD_MADJ 4  // in 256-cell tiles per SM
#endif
template <int WF>
__global__ void __launch_bounds__(PF_BLOCK_FWD_MADJ<WF>, CUPCFD_MINB_FWD_MADJ *TILE_CELLS / PF_BLOCK_FWD_MADJ<WF>)
    k_fwd_madj_f32_pf(int nC, SellView sv, const float4 *__restrict__ fg, const float *__restrict__ phi,
                      const float *__restrict__ phiB, const double *__restrict__ vol, const float4 *__restrict__ st,
                      const float *__restrict__ gface, float *__restrict__ g, float *__restrict__ mflux,
                      float4 *__restrict__ stbar, double *__restrict__ lossPart, int64_t ldc, PrefetchArgs pf) {
    constexpr int T = TILE_CELLS;
    const TileBlock<PF_BLOCK_FWD_MADJ<WF>> tb(pf);
    const int c = tb.c;
    __shared__ int4 s_rng;
    const void *const cellSrc[3] = {phi, st, vol};
    const int cellBytes[3] = {T * 4, T * 16, T * 8};
    if (tb.lead) fetch_ranges_async(&s_rng, pf.desc + tb.tp);
    double l = 0.0;
    if (c < nC) {
        if constexpr (WF == -6) {
            __shared__ FwdMadjStage<PF_BLOCK_FWD_MADJ<WF>> stage;
            const CellList<WF> e(sv, c);
            l = e.alternating == 2   ? fwd_madj_cell_staged<2>(c, e, stage, fg, phi, phiB, vol, st, gface, g, mflux, stbar, ldc)
                : e.alternating == 1 ? fwd_madj_cell_staged<1>(c, e, stage, fg, phi, phiB, vol, st, gface, g, mflux, stbar, ldc)
                                     : fwd_madj_cell_staged<0>(c, e, stage, fg, phi, phiB, vol, st, gface, g, mflux, stbar, ldc);
        } else
            l = fwd_madj_cell_f32<CUPCFD_FWD_MADJ_CHUNK, 0, WF>(c, sv, fg, phi, phiB, vol, st, gface, g, mflux, stbar, ldc);
    }
    if (tb.lead) prefetch_tile<3>(pf, tb.tp, ranges_ready(&s_rng), fg, 16, gface, cellSrc, cellBytes);
    if (lossPart) warp_partial_store<PF_BLOCK_FWD_MADJ<WF>>(l, c, lossPart);
}

// Gradient part of the adjoint only (adj_cell_f32 without the mass part):
// phibar and phibBar. The next chunk's entries load during the current
// chunk's arithmetic. 0.278 ms at 256^3 on full lists (1.86 GB of DRAM
// traffic), 0.237 in run form (1.14 GB).
template <int WF>
__global__ void __launch_bounds__(PF_BLOCK_GADJ<WF>, PF_MINB_GADJ<WF> *TILE_CELLS / PF_BLOCK_GADJ<WF>)
    k_gadj_f32_pf(int nC, SellView sv, const float4 *__restrict__ fg, const float *__restrict__ g, float hscale,
                  float *__restrict__ phibar, float *__restrict__ phibBar, int64_t ldc, PrefetchArgs pf) {
    constexpr int T = TILE_CELLS;
    const TileBlock<PF_BLOCK_GADJ<WF>> tb(pf);
    const int c = tb.c;
    __shared__ int4 s_rng;
    const void *const cellSrc[3] = {g, g + ldc, g + 2 * ldc};
    const int cellBytes[3] = {T * 4, T * 4, T * 4};
    if (tb.lead) fetch_ranges_async(&s_rng, pf.desc + tb.tp);
    if (c < nC)
        adj_cell_f32<false, PF_CHUNK_GADJ<WF>, 1, WF>(c, sv, fg, g, hscale, nullptr, nullptr, phibar, phibBar, nullptr, ldc);
    if (tb.lead) prefetch_tile<3>(pf, tb.tp, ranges_ready(&s_rng), fg, 16, (const float *) nullptr, cellSrc, cellBytes);
}

// Mass-flux part of the adjoint only (adj_cell_f32 with hscale 0): stbar
// from the state and gface, with the L2 prefetch of their tile ranges. The
// host forward+adjoint call runs it once gface is in; with k_gadj_f32_pf for
// the gradient part it forms the same sums as k_adj_f32_pf, so the same bits.
template <int WF>
__global__ void __launch_bounds__(PF_BLOCK_MADJ<WF>, CUPCFD_MINB_F32 *TILE_CELLS / PF_BLOCK_MADJ<WF>)
    k_madj_f32_pf(int nC, SellView sv, const float4 *__restrict__ fg, const float4 *__restrict__ st,
                  const float *__restrict__ gface, float4 *__restrict__ stbar, int64_t ldc, PrefetchArgs pf) {
    constexpr int T = TILE_CELLS;
    const TileBlock<PF_BLOCK_MADJ<WF>> tb(pf);
    const int c = tb.c;
    __shared__ int4 s_rng;
    const void *const cellSrc[1] = {st};
    const int cellBytes[1] = {T * 16};
    if (tb.lead) fetch_ranges_async(&s_rng, pf.desc + tb.tp);
    if (c < nC)
        adj_cell_f32<false, CUPCFD_ADJ_CHUNK, 0, WF>(c, sv, fg, nullptr, 0.f, st, gface, nullptr, nullptr, stbar, ldc);
    if (tb.lead) prefetch_tile<1>(pf, tb.tp, ranges_ready(&s_rng), fg, 16, gface, cellSrc, cellBytes);
}

// The mass-flux part of the adjoint only, FP64 (adj_cell_f64 with hscale 0).
template <int WF>
__global__ void __launch_bounds__(PF_BLOCK_MADJ_F64<WF>, PF_MINB_ADJ_F64<WF, WF != -6> *TILE_CELLS / PF_BLOCK_MADJ_F64<WF>)
    k_madj_f64_pf(int nC, SellView sv, const double4 *__restrict__ fg, const double *__restrict__ st,
                  const double *__restrict__ gface, double *__restrict__ stbar, int64_t ldc, PrefetchArgs pf) {
    constexpr int T = TILE_CELLS;
    const TileBlock<PF_BLOCK_MADJ_F64<WF>> tb(pf);
    const int c = tb.c;
    __shared__ int4 s_rng;
    const void *const cellSrc[4] = {st, st + ldc, st + 2 * ldc, st + 3 * ldc};
    const int cellBytes[4] = {T * 8, T * 8, T * 8, T * 8};
    if (tb.lead) fetch_ranges_async(&s_rng, pf.desc + tb.tp);
    if (c < nC)
        adj_cell_f64<false, PF_CHUNK_ADJ_F64<WF, WF != -6>, WF>(c, sv, fg, nullptr, 0.0, st, gface, nullptr, nullptr, stbar, ldc);
    if (tb.lead) prefetch_tile<4>(pf, tb.tp, ranges_ready(&s_rng), fg, 32, gface, cellSrc, cellBytes);
}

// The gradient by itself (grad_cell_*, reference sign), with the L2 prefetch;
// CORR: an iteration with the non-orthogonal correction, which reads the
// previous iterate go and the cells' and faces' centres as well.
template <class T, bool CORR, int WF, bool DEEP = false>
__global__ void __launch_bounds__(PF_BLOCK_GRAD<WF>, PF_MINB_GRAD<CORR, WF, DEEP> *TILE_CELLS / PF_BLOCK_GRAD<WF>)
    k_grad_pf(int nC, SellView sv, const typename Vec4<T>::type *__restrict__ fg, const typename Vec4<T>::type *__restrict__ fc,
              const typename Vec4<T>::type *__restrict__ cc, const T *__restrict__ phi, const T *__restrict__ phiB,
              const double *__restrict__ vol, const T *__restrict__ go, T *__restrict__ g, T *__restrict__ gcopy, int64_t ldc,
              PrefetchArgs pf) {
    constexpr int TC = TILE_CELLS, S = (int) sizeof(T), N = CORR ? 6 : 2;
    const TileBlock<PF_BLOCK_GRAD<WF>> tb(pf);
    const int c = tb.c;
    __shared__ int4 s_rng;
    if (tb.lead) fetch_ranges_async(&s_rng, pf.desc + tb.tp);
    if (c < nC) {
        if constexpr (S == 8)
            grad_cell_f64<CORR, false, PF_CHUNK_GRAD<CORR, WF, DEEP>, WF>(c, sv, fg, fc, cc, phi, phiB, vol, go, g, gcopy, ldc);
        else
            grad_cell_f32<CORR, false, PF_CHUNK_GRAD<CORR, WF, DEEP>, WF>(c, sv, fg, fc, cc, phi, phiB, vol, go, g, gcopy, ldc);
    }
    if (tb.lead) {
        const int4 r = ranges_ready(&s_rng);
        const void *const cellSrc[6] = {phi, vol, go, go + ldc, go + 2 * ldc, cc};
        const int cellBytes[6] = {TC * S, TC * 8, TC * S, TC * S, TC * S, TC * 4 * S};
        const void *src[N];
        int bytes[N];
#pragma unroll
        for (int i = 0; i < N; i++) { src[i] = cellSrc[i]; bytes[i] = cellBytes[i]; }
        prefetch_tile<N>(pf, tb.tp, r, fg, 4 * S, (const T *) nullptr, src, bytes);
        if (CORR && r.w > r.z) bulk_prefetch_l2(fc + r.z, (unsigned) (r.w - r.z) * (unsigned) (4 * S));
    }
}

// The general gradient adjoint (grad_adj_cell, reference sign), with the L2 prefetch.
template <class T, int WF>
__global__ void __launch_bounds__(PF_BLOCK_GRAD_ADJ<WF>, PF_MINB_GRAD_ADJ *TILE_CELLS / PF_BLOCK_GRAD_ADJ<WF>)
    k_grad_adj_pf(int nC, SellView sv, const typename Vec4<T>::type *__restrict__ fg, const double *__restrict__ ivol,
                  const T *__restrict__ gbar, T *__restrict__ phibar, T *__restrict__ phibBar, int64_t ldc, PrefetchArgs pf) {
    constexpr int TC = TILE_CELLS, S = (int) sizeof(T);
    const TileBlock<PF_BLOCK_GRAD_ADJ<WF>> tb(pf);
    const int c = tb.c;
    __shared__ int4 s_rng;
    const void *const cellSrc[4] = {gbar, gbar + ldc, gbar + 2 * ldc, ivol};
    const int cellBytes[4] = {TC * S, TC * S, TC * S, TC * 8};
    if (tb.lead) fetch_ranges_async(&s_rng, pf.desc + tb.tp);
    if (c < nC) grad_adj_cell<false, T, PF_CHUNK_GRAD_ADJ, WF>(c, sv, fg, ivol, gbar, phibar, phibBar, ldc);
    if (tb.lead) prefetch_tile<4>(pf, tb.tp, ranges_ready(&s_rng), fg, 4 * S, (const T *) nullptr, cellSrc, cellBytes);
}

// The mean number of 128-byte lines of an FP64 cell array that a warp's 32
// cells gather from for one of their entries: lines[0] lines over lines[1]
// gathers. 2.2 on generated meshes by rows, 3 to 5 in Morton or RCM order, 7
// to 10 on irregular meshes in those orders (each cell has its own order of
// faces), 31 on hexahedra numbered at random (16 on mixed cells).
__global__ void k_gather_lines(int nSlices, const int *__restrict__ slicePtr, const int2 *__restrict__ inc,
                               unsigned long long *__restrict__ lines) {
    const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
    unsigned n = 0, gathers = 0;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nSlices; s += warps)
        for (int k = slicePtr[s]; k < slicePtr[s + 1]; k += 32) {
            const int o = inc[k + lane].y, line = o >= 0 ? o >> 4 : -1;
            const unsigned same = __match_any_sync(0xffffffffu, line);
            const unsigned first = __ballot_sync(0xffffffffu, line >= 0 && __ffs((int) same) - 1 == lane);
            n += __popc(first);
            gathers += first != 0;
        }
    if (lane == 0) {
        atomicAdd(lines, (unsigned long long) n);
        atomicAdd(lines + 1, (unsigned long long) gathers);
    }
}

// Largest |c - neighbour| over the incidence lists (the numbering's bandwidth).
// Launched with whole warps (blockDim a multiple of 32), no early return.
__global__ void k_bandwidth(int nC, SellView sv, int *__restrict__ out) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    int bw = 0;
    if (c < nC) {
        int w;
        const int2 *e = cell_entries(sv, c, w);
        for (int k = 0; k < w; k++) {
            int2 en = e[32 * k];
            if (en.x < 0) break;
            if (en.y >= 0) bw = max(bw, abs(c - en.y));
        }
    }
    for (int s = 16; s > 0; s >>= 1) bw = max(bw, __shfl_xor_sync(0xffffffffu, bw, s));
    if ((threadIdx.x & 31) == 0) atomicMax(out, bw);
}

// ---------------------------------------------------------------------------
// Tile descriptors (mesh creation). Faces are numbered by owner slice, so
// the owner tile is non-decreasing in the face number; k_tile_face_start
// records where each tile's faces begin and flags any decrease.
// ---------------------------------------------------------------------------
__global__ void k_tile_face_start(int nF, int nTiles, const int2 *__restrict__ fcells, int *__restrict__ start,
                                  int *__restrict__ bad) {
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nF) return;
    int t = fcells[f].x / TILE_CELLS;
    int tp = f > 0 ? fcells[f - 1].x / TILE_CELLS : -1;
    if (t < tp) atomicOr(bad, 1);
    for (int u = tp + 1; u <= t; u++) start[u] = f;
    if (f == nF - 1)
        for (int u = t + 1; u <= nTiles; u++) start[u] = nF;
}

__global__ void k_tile_desc(int nTiles, int nSlices, const int *__restrict__ slicePtr, const int *__restrict__ start,
                            TileDesc *__restrict__ desc, int *__restrict__ maxima) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nTiles) return;
    int s0 = t * (TILE_CELLS / 32);
    TileDesc d;
    d.entStart = slicePtr[s0];
    d.entEnd = slicePtr[min(s0 + TILE_CELLS / 32, nSlices)];
    d.fs = start[t];
    d.fe = start[t + 1];
    unsigned w[2] = {0u, 0u};
    int wmax = 0;
    for (int i = 0; i < TILE_CELLS / 32; i++) {
        int s = s0 + i;
        int wi = s < nSlices ? (slicePtr[s + 1] - slicePtr[s]) >> 5 : 0;
        wmax = max(wmax, wi);
        w[i >> 2] |= (unsigned) min(wi, 255) << (8 * (i & 3));
    }
    d.w03 = w[0]; d.w47 = w[1];
    d.pad0 = 0; d.pad1 = 0;
    desc[t] = d;
    atomicMax(maxima + 0, d.entEnd - d.entStart);
    atomicMax(maxima + 1, d.fe - d.fs);
    atomicMax(maxima + 2, wmax);
}

// The descriptors of the run form: the same tiles, with the range of the
// tile's runs (six int2 each) in place of its SELL entries.
__global__ void k_tile_desc_runs(int nTiles, int nSlices, int nRuns, const RunHead *__restrict__ runHead,
                                 const TileDesc *__restrict__ desc, TileDesc *__restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nTiles) return;
    const int s0 = t * (TILE_CELLS / 32), s1 = s0 + TILE_CELLS / 32;
    TileDesc d = desc[t];
    d.entStart = 6 * runHead[s0].first;
    d.entEnd = 6 * (s1 < nSlices ? runHead[s1].first : nRuns);
    out[t] = d;
}

}  // namespace cupcfd_gpu
