// Sums over the boundaries of one region type in boundary order, bit for bit
// the sums of a loop that walks ib = 0 .. nB-1 and adds each selected
// boundary's value into a running total and into its region's accumulator
// (FluxMassDolfynBoundaryLoop1-5, MassKernels.ipp:311-521;
// FluxUVWDolfynBndsLoop1, UVWKernels.ipp:527-544).
//
// IEEE addition is not associative, so each sum must round as its chain of
// additions in boundary order does. While the running sum stays between two
// powers of two, though, all its values are multiples of one unit u in the
// last place, and adding v rounds the real number acc + v to the nearest
// multiple: acc / u grows by the integer nearest to v / u, whatever acc is.
// Those integers are added in parallel, and the partial sums are the chain's
// own values, provided no addition on the way rounds. A stretch of consecutive
// integers adds up to the difference of two partial sums, both between the
// same powers of two (2^52 and 2^53 units), so to less than 2^52: exact. Sums
// of every second or fourth thread or warp, as a butterfly of exchanges forms
// them, have no such bound (values that rise through one thread's share and
// fall through the next pass 2^53) and serve only where the integers' sizes
// add up to less than 2^51. Only a tie (v / u an integer and a half) looks at acc:
// it goes to the even neighbour, which the parities of the integers since the
// tie before tell. Where a partial sum leaves the interval between the powers
// of two (or a value is not finite, or too large), the additions up to there
// count, a few more run one by one, and the rest starts again with the new
// unit. A sum of values of one sign changes its unit a dozen times; one that
// keeps crossing a power of two falls back to longer and longer stretches one
// by one.
//
// One block per sum: the total, and each region's accumulator (or each
// component of it). A pass over many blocks first gathers the type's values
// densely in boundary order, through lists that depend on the regions alone
// and are built when these are set (struct BndLists). At 192^3 (36,864 inlet
// and as many outlet boundaries) a sum takes 4 us to gather and 46 to add
// (three quarters of it the fifteen or so scans, the rest the additions one
// by one, 8 cycles each, and the loads), against 215 us for adding one value
// after another; the solver step's chain of five sums (13 launches) 267 us in
// short runs, 280 to 290 in calls from Python, against 1160. 512 threads with 8
// additions each: 1,024 with 4 take 322 us, 256 with 16 323.
//
// F32: the chains add in float (the reference's T = float instantiation);
// values and accumulators stay in double arrays, which hold the float values
// exactly.
//
// Kernels and helpers sit in an unnamed namespace (at file scope, as in
// perm.cuh): each translation unit that includes this header gets its own
// copies, so no kernel symbol is defined twice.
#pragma once

#include <algorithm>

#include "internal.cuh"

namespace {

using namespace cupcfd_gpu;

#ifndef CUPCFD_OS_T
#define CUPCFD_OS_T 512
#endif
#ifndef CUPCFD_OS_FIRST
#define CUPCFD_OS_FIRST 512
#endif
constexpr int OS_T = CUPCFD_OS_T;  // threads of a block
constexpr int OS_E = 4096 / OS_T;  // consecutive additions a thread takes
constexpr int OS_B = OS_T * OS_E;  // additions a block holds at a time
constexpr int OS_TIES = 16;        // ties a batch may have and still be taken at once
static_assert(OS_T % 32 == 0 && OS_T <= 1024 && OS_B == 4096 && OS_E % 2 == 0,
              "whole warps, at most one per lane of a warp; the values in pairs");
static_assert(CUPCFD_OS_FIRST > 0, "the additions one by one go on");

// The unit of acc's interval between powers of two, and its inverse; false
// where the scan does not apply (zero, subnormal, not finite, or powers
// whose unit or inverse would not be normal).
template <bool F32>
__device__ __forceinline__ bool unit_of(double acc, double &u, double &inv) {
    const int e = ((__double2hiint(acc) >> 20) & 0x7ff) - 1023;
    constexpr int P = F32 ? 23 : 52;
    if (e < (F32 ? -126 : -900) || e > (F32 ? 127 : 1000)) return false;
    u = __hiloint2double((e - P + 1023) << 20, 0);
    inv = __hiloint2double((P - e + 1023) << 20, 0);
    return true;
}

template <bool F32>
__device__ __forceinline__ double add_one(double a, double v) {
    return F32 ? (double) __fadd_rn((float) a, (float) v) : __dadd_rn(a, v);
}

// The values of a type's boundaries, densely in boundary order: component q
// of item k, vals[nv k + q] = base[item[k] * stride + offset + q]. Many blocks:
// the addresses are scattered, and the one block that adds the values would
// take longer to fetch them than to add them (74 us in all against 46).
__global__ void __launch_bounds__(256) k_gather_values(int n, const int *__restrict__ item, const double *__restrict__ base,
                                                       int stride, int offset, int nv, double *__restrict__ vals) {
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k >= n) return;
    const double *p = base + (size_t) item[k] * stride + offset;
    for (int q = 0; q < nv; q++) vals[(size_t) nv * k + q] = p[q];
}

struct OrderedSum {
    const double *vals;          // [nv n] the type's values (k_gather_values)
    int n, nv;
    const int *place;            // their places grouped by region, region r's from regionStart[r]
    const int *regionStart, *regionType;
    int type;
    const double *init;          // the total's start: *init, or initValue
    double initValue;
    double *out, *regionAcc;     // the total (nv 1) and the regions' accumulators; either may be null
};

template <bool F32>
__global__ void __launch_bounds__(OS_T) k_ordered_sum(const __grid_constant__ OrderedSum a) {
    constexpr int NW = OS_T / 32;
    __shared__ __align__(16) double sv[OS_B];
    __shared__ double2 warpSums[2][NW];
    __shared__ int warpOdd[2][NW];
    __shared__ double s_acc, s_seq[2];
    __shared__ int s_first, s_ties, s_tie[OS_TIES];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;

    const int *place = nullptr;  // null: all the type's values
    int n = a.n, q = 0;
    double *target = a.out;
    double acc;
    if (a.out && blockIdx.x == 0) {
        acc = a.init ? *a.init : a.initValue;
    } else {
        const int j = blockIdx.x - (a.out ? 1 : 0), r = j / a.nv;
        if (a.regionType[r] != a.type) return;
        q = j % a.nv;
        place = a.place + a.regionStart[r];
        n = a.regionStart[r + 1] - a.regionStart[r];
        target = a.regionAcc + j;
        acc = *target;
    }

    // the next batch's places and values are on their way while one is added
    int id[OS_E];
    double next[OS_E];
    auto load_ids = [&](int b0) {
#pragma unroll
        for (int k = 0; k < OS_E; k++) {
            const int i = b0 + k * OS_T + t;
            id[k] = i >= n ? -1 : place ? __ldg(place + i) : i;
        }
    };
    auto load_values = [&]() {
#pragma unroll
        for (int k = 0; k < OS_E; k++) next[k] = id[k] >= 0 ? a.vals[(size_t) id[k] * a.nv + q] : 0.0;
    };
    load_ids(0);
    load_values();
    load_ids(OS_B);

    // Additions one by one where a scan ended early. At first the sum is zero,
    // then doubles quickly: a few hundred additions cost less than the scans
    // that its changes of unit would take. Where more than three scans in a
    // row end early they go up to a whole batch: 98,304 values of random sign
    // then take 532 us, 695 with at most 1,024 between scans, 559 all one by one.
    int stretch = CUPCFD_OS_FIRST, shorts = 0, turn = 0, turnSums = 0;
    for (int b0 = 0; b0 < n; b0 += OS_B) {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < OS_E; k++) sv[k * OS_T + t] = next[k];
        __syncthreads();
        load_values();
        load_ids(b0 + 2 * OS_B);
        const int nb = min(OS_B, n - b0);
        double v[OS_E];
#pragma unroll
        for (int k = 0; k < OS_E; k += 2) {
            const double2 p = *reinterpret_cast<const double2 *>(sv + t * OS_E + k);
            v[k] = p.x;
            v[k + 1] = p.y;
        }
        for (int o = 0; o < nb;) {  // uniform: o, acc and stretch are the same in every thread
            double u, inv;
            if (unit_of<F32>(acc, u, inv)) {
                constexpr double MAGIC = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds |x| < 2^51 to an integer
                constexpr double LO = F32 ? 8388608.0 : 4503599627370496.0, HI = 2 * LO;  // 2^23, 2^52
                constexpr double MOST = 2251799813685248.0;                               // 2^51
                const double start = __dmul_rn(acc, inv);
                double step[OS_E];                    // the integer nearest v / u; of a tie the one below
                unsigned tie = 0, odd = 0;
                double sum = 0.0, size = 0.0;
#pragma unroll
                for (int k = 0; k < OS_E; k++) {
                    const int i = t * OS_E + k;
                    const double x = i >= o && i < nb ? __dmul_rn(v[k], inv) : 0.0;
                    const double m = __dadd_rn(x, MAGIC);
                    step[k] = __dsub_rn(m, MAGIC);
                    const double d = __dsub_rn(x, step[k]);
                    odd ^= (unsigned) __double2loint(m) & 1u;
                    if (fabs(d) == 0.5) {
                        tie |= 1u << k;
                        if (d < 0.0) {
                            step[k] = __dsub_rn(step[k], 1.0);
                            odd ^= 1u;
                        }
                    }
                    sum = __dadd_rn(sum, step[k]);
                    size = __dadd_rn(size, fabs(step[k]));
                }
                double at = sum;  // with the warp's threads before: consecutive, so exact up to where the scan ends
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const double p = __shfl_up_sync(0xffffffffu, at, d);
                    if (lane >= d) at = __dadd_rn(at, p);
                    size = __dadd_rn(size, __shfl_xor_sync(0xffffffffu, size, d));
                }
                const unsigned odds = __ballot_sync(0xffffffffu, odd);  // of the warp's threads
                turnSums ^= 1;
                if (lane == 31) {
                    warpSums[turnSums][wid] = make_double2(at, size);
                    warpOdd[turnSums][wid] = __popc(odds) & 1;
                }
                if (t == 0) {
                    s_first = OS_B;
                    s_ties = 0;
                }
                const bool ties = __syncthreads_or(tie);
                // Where even the increments' sizes together keep to the
                // interval no partial sum leaves it, and only the total is
                // needed (exact: below 2^53; every |x| is then below 2^51).
                const double2 w = lane < NW ? warpSums[turnSums][lane] : make_double2(0.0, 0.0);
                double total = w.x;
                size = w.y;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) {
                    total = __dadd_rn(total, __shfl_xor_sync(0xffffffffu, total, d));
                    size = __dadd_rn(size, __shfl_xor_sync(0xffffffffu, size, d));
                }
                bool whole = size < MOST && __dadd_rn(fabs(start), size) < HI - OS_B && __dsub_rn(fabs(start), size) > LO + OS_B;
                if (whole && ties) {
                    // Each tie adds one more where acc / u + step is odd, and
                    // leaves acc / u even. So it adds the parity of the steps
                    // since the tie before it (of all of them and the start
                    // for the first): the parities of acc / u without the
                    // ties' own additions, up to each tie, say it.
                    const unsigned wodds = __ballot_sync(0xffffffffu, lane < NW && warpOdd[turnSums][lane]);
                    unsigned p = ((unsigned) (long long) start + __popc(wodds & ((1u << wid) - 1u)) +
                                  __popc(odds & ((1u << lane) - 1u))) & 1u;
#pragma unroll
                    for (int k = 0; k < OS_E; k++) {
                        p ^= (unsigned) __double2loint(__dadd_rn(step[k], MAGIC)) & 1u;
                        if (tie >> k & 1) {
                            const int j = atomicAdd(&s_ties, 1);
                            if (j < OS_TIES) s_tie[j] = (t * OS_E + k) * 2 + (int) p;
                        }
                    }
                    __syncthreads();
                    const int nt = s_ties;
                    whole = nt <= OS_TIES;
                    if (whole) {
                        unsigned before = 0;
                        for (int j = 0, at = -1; j < nt; j++) {  // in order
                            int lowest = 0x7fffffff;
                            for (int i = 0; i < nt; i++)
                                if (s_tie[i] > at) lowest = min(lowest, s_tie[i]);
                            at = lowest;
                            total = __dadd_rn(total, ((unsigned) at & 1u) != before ? 1.0 : 0.0);
                            before = (unsigned) at & 1u;
                        }
                    }
                    __syncthreads();  // before s_ties starts over
                }
                if (whole) {
                    acc = __dmul_rn(__dadd_rn(start, total), u);
                    o = nb;
                    stretch = max(stretch / 2, 16);
                    continue;
                }
                // Else the partial sums themselves, up to the first that
                // leaves the interval, tie, or value too large or not finite.
                double warps = w.x;  // with the warps before
#pragma unroll
                for (int d = 1; d < NW; d <<= 1) {
                    const double p = __shfl_up_sync(0xffffffffu, warps, d);
                    if (lane >= d) warps = __dadd_rn(warps, p);
                }
                warps = __shfl_sync(0xffffffffu, warps, max(wid - 1, 0));
                at = __shfl_up_sync(0xffffffffu, at, 1);
                at = __dadd_rn(wid > 0 ? __dadd_rn(start, warps) : start, lane > 0 ? at : 0.0);
                int first = OS_B;
#pragma unroll
                for (int k = 0; k < OS_E; k++) {
                    if (first < OS_B) continue;
                    const int i = t * OS_E + k;
                    const double to = __dadd_rn(at, step[k]);
                    const bool fine = fabs(__dmul_rn(v[k], inv)) < MOST && !(tie >> k & 1) && fabs(to) > LO && fabs(to) < HI;
                    if (i >= o && i < nb && !fine) first = i;
                    else at = to;
                }
                const int wfirst = __reduce_min_sync(0xffffffffu, first);
                if (lane == 0 && wfirst < OS_B) atomicMin(&s_first, wfirst);
                __syncthreads();
                const int stop = s_first;
                if (t == min(stop / OS_E, OS_T - 1)) s_acc = __dmul_rn(at, u);
                __syncthreads();
                acc = s_acc;
                const int done = min(stop, nb) - o;
                o += done;
                shorts = done < 256 ? shorts + 1 : 0;
                stretch = shorts ? min(2 * stretch, shorts > 3 ? OS_B : 1024) : max(stretch / 2, 16);
            }
            if (o < nb) {
                const int end = min(nb, o + stretch);
                if (t == 0) {
                    double s = acc;
                    int i = o;
                    for (; i < end && i % 16; i++) s = add_one<F32>(s, sv[i]);
                    for (; i + 16 <= end; i += 16) {
                        double x[16];
#pragma unroll
                        for (int k = 0; k < 16; k++) x[k] = sv[i + k];
#pragma unroll
                        for (int k = 0; k < 16; k++) s = add_one<F32>(s, x[k]);
                    }
                    for (; i < end; i++) s = add_one<F32>(s, sv[i]);
                    s_seq[turn] = s;
                }
                __syncthreads();
                acc = s_seq[turn];
                turn ^= 1;
                o = end;
            }
        }
    }
    if (t == 0) *target = acc;
}

// *out = init + v_0 + v_1 + ... over the values of the boundaries of `type`
// (out not null) and regionAcc[nv r + q] += region r's values (regionAcc not
// null), each in boundary order. out may be init (the sum continues from it).
template <bool F32 = false>
int launch_ordered_sum(const cupcfd_gpu_mesh *m, int type, const double *vals, int nv, const double *init, double initValue,
                       double *out, double *regionAcc, cudaStream_t st) {
    OrderedSum a{};
    a.vals = vals;
    a.n = m->bndLists.count(type);
    a.nv = nv;
    a.place = m->bndLists.regionPlace;
    a.regionStart = m->bndLists.regionStart;
    a.regionType = m->regionType;
    a.type = type;
    a.init = init; a.initValue = initValue;
    a.out = out;
    a.regionAcc = a.n > 0 ? regionAcc : nullptr;  // without a boundary of the type no region changes
    const int64_t grid = (out ? 1 : 0) + (a.regionAcc ? (int64_t) m->nR * nv : 0);
    if (grid == 0) return CUPCFD_E_SUCCESS;
    k_ordered_sum<F32><<<(unsigned) grid, OS_T, 0, st>>>(a);
    CG_LAUNCHED();
    return CUPCFD_E_SUCCESS;
}

// The same of base[item[k] * stride + offset + q] for the type's items k (item
// [nB] grouped by type as BndLists); vals: scratch, [nv x the type's count].
template <bool F32 = false>
int launch_gathered_sum(const cupcfd_gpu_mesh *m, int type, const int *item, const double *base, int stride, int offset,
                        int nv, double *vals, double *out, double *regionAcc, cudaStream_t st) {
    const int n = m->bndLists.count(type);
    if (n > 0) {
        k_gather_values<<<grid_for(n, 256), 256, 0, st>>>(n, item + m->bndLists.typeStart[type], base, stride, offset, nv,
                                                          vals);
        CG_LAUNCHED();
    }
    return launch_ordered_sum<F32>(m, type, vals, nv, nullptr, 0.0, out, regionAcc, st);
}

}  // namespace
