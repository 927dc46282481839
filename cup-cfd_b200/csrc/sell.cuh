// SELL-32 incidence-list access shared by the kernels of every translation
// unit (inline device functions only): the cell's first entry and slice
// width, and chunked entry loads. Layout in internal.cuh (struct Sell).
#pragma once

#include "internal.cuh"

namespace cupcfd_gpu {

struct SellView {
    const int *slicePtr;
    const int2 *inc;
    int width;  // common slice width, or 0 when widths vary
    const RunHead *runHead;  // run form (struct Sell), null when the mesh has none
    const int4 *runs;
};

// The cell's first incidence entry and its slice width (entries per lane).
// With a common width (every hexahedral mesh) the position is arithmetic,
// which takes a dependent load off the head of every cell's load chain.
__device__ __forceinline__ const int2 *cell_entries(const SellView &sv, int c, int &w) {
    int s = c >> 5;
    if (sv.width) {
        w = sv.width;
        return sv.inc + (s * 32 * sv.width + (c & 31));  // entries fit in int (slicePtr is int)
    }
    int p0 = __ldg(sv.slicePtr + s);
    w = (__ldg(sv.slicePtr + s + 1) - p0) >> 5;
    return sv.inc + p0 + (c & 31);
}

// Read-only 8-byte load of an incidence entry. With CUPCFD_L2_PREFETCH the
// load asks L2 to fetch 256-byte blocks from DRAM (the incidence stream is
// read sequentially slice by slice).
__device__ __forceinline__ int2 ld_entry(const int2 *p) {
#ifdef CUPCFD_L2_PREFETCH
    int2 v;
    asm("ld.global.nc.L2::256B.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
#else
    return __ldg(p);
#endif
}

// Entries k0 .. k0+W-1 of the cell (padding {-1,-1} past its slice width).
template <int W>
__device__ __forceinline__ void load_entries(const int2 *e, int k0, int w, int2 (&en)[W]) {
#pragma unroll
    for (int j = 0; j < W; j++) en[j] = (k0 + j < w) ? ld_entry(e + 32 * (k0 + j)) : make_int2(-1, -1);
}

// A cell's incidence list as the L2-prefetch kernels read it. WF: 0 any mesh;
// 6 every cell has exactly six entries; -6 the same in run form (struct Sell
// in internal.cuh): the entries of the first cell of this cell's run, each
// advanced by the cell's distance d from it (the face code by 2 d, the other
// cell by d, a boundary id by d).
template <int WF>
struct CellList {
    const int2 *e;
    int w;
    __device__ __forceinline__ CellList(const SellView &sv, int c) {
        e = cell_entries(sv, c, w);
        if (WF) w = WF;
    }
    template <int W>
    __device__ __forceinline__ void load(int k0, int2 (&en)[W]) const {
        static_assert(!WF || 6 % W == 0, "the six-entry forms test for no padding: chunks divide six");
        load_entries(e, k0, w, en);
    }
    __device__ __forceinline__ int2 at(int k) const { return ld_entry(e + 32 * k); }  // k < w
};
template <>
struct CellList<-6> {
    const int2 *e;
    int d;
    int alternating;  // the same for the whole slice (RunHead)
    static constexpr int w = 6;
    __device__ __forceinline__ CellList(const SellView &sv, int c) {
        const int4 h = __ldg(reinterpret_cast<const int4 *>(sv.runHead + (c >> 5)));
        const int lane = c & 31;
        const unsigned m = (unsigned) h.x & (0xffffffffu >> (31 - lane));
        d = lane - (31 - __clz(m));
        e = reinterpret_cast<const int2 *>(sv.runs + 3 * (h.y + __popc(m) - 1));
        alternating = h.z;
    }
    template <int W>
    __device__ __forceinline__ void load(int k0, int2 (&en)[W]) const {
        static_assert(6 % W == 0, "no padding: chunks divide six");
#pragma unroll
        for (int j = 0; j < W; j++) {
            int2 b = make_int2(-1, -1);
            if (k0 + j < w) {
                if (W % 2 == 0) {  // two entries a load: a run's six start on a 16-byte boundary
                    if (j % 2 == 1) continue;
                    const int4 q = __ldg(reinterpret_cast<const int4 *>(e + k0 + j));
                    en[j] = advance(make_int2(q.x, q.y));
                    en[j + 1 < W ? j + 1 : j] = advance(make_int2(q.z, q.w));
                    continue;
                }
                b = advance(__ldg(e + k0 + j));
            }
            en[j] = b;
        }
    }
    __device__ __forceinline__ int2 at(int k) const { return advance(__ldg(e + k)); }
    __device__ __forceinline__ int2 advance(int2 b) const {
        return make_int2(b.x + 2 * d, b.y >= 0 ? b.y + d : b.y - d);
    }
    // All six entries of a cell of an alternating slice, with the face in
    // place of the code: interior faces, but for the first two with ALT 1.
    template <int ALT>
    __device__ __forceinline__ void load_alternating(int (&face)[6], int (&other)[6]) const {
#pragma unroll
        for (int j = 0; j < 6; j += 2) {
            const int4 q = __ldg(reinterpret_cast<const int4 *>(e + j));
            face[j] = (q.x >> 1) + d;
            face[j + 1] = (q.z >> 1) + d;
            other[j] = ALT == 1 && j == 0 && q.y < 0 ? q.y - d : q.y + d;
            other[j + 1] = ALT == 1 && j == 0 && q.w < 0 ? q.w - d : q.w + d;
        }
    }
};

// The entries of the cell's next chunk into en: with PIPE they were loaded
// into nx before the current chunk's arithmetic (so their latency overlaps
// it; two more registers per entry), else they are loaded now.
template <int PIPE, int WF, int W>
__device__ __forceinline__ void next_entries(const CellList<WF> &e, int k0, int2 (&en)[W], const int2 (&nx)[W]) {
    if (PIPE) {
#pragma unroll
        for (int j = 0; j < W; j++) en[j] = nx[j];
    } else {
        e.load(k0, en);
    }
}

}  // namespace cupcfd_gpu
