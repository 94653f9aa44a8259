// Persistent pair-binning kernels of the batched path: CTAs pull
// (job, i-tile, j-tile) items from the culled queues that hbt_batch.cu
// builds and run the screened tile-pair bodies of hbt_tile.cuh on them.
// The kernel templates are instantiated in three translation units,
// compiled in parallel: hbt_persist_fast.cu (fast binning),
// hbt_persist_caps.cu (the two passes of ordered cap admission) and
// hbt_persist_qinv.cu (fast binning with the q_inv histograms).
#pragma once

#include <algorithm>

#include "hbt_batch.cuh"
#include "hbt_tile.cuh"

namespace hbt {

// Launchers, one family per translation unit (same-event items
// [base, end) of the queue; mixed-event items all at once).
cudaError_t persistent_same_fast(const Device &d, const BatchDev &b, unsigned base, unsigned end,
                                 int grid, cudaStream_t st);
cudaError_t persistent_mixed_fast(const Device &d, const BatchDev &b, int grid, cudaStream_t st);
cudaError_t persistent_same_ordered(const Device &d, const BatchDev &b, unsigned base,
                                    unsigned end, int grid, cudaStream_t st, int mode);
cudaError_t persistent_mixed_ordered(const Device &d, const BatchDev &b, int grid,
                                     cudaStream_t st, int mode);
cudaError_t persistent_same_qinv(const Device &d, const BatchDev &b, unsigned base, unsigned end,
                                 int grid, cudaStream_t st);
cudaError_t persistent_mixed_qinv(const Device &d, const BatchDev &b, int grid, cudaStream_t st);
// Dispatch on the admission mode and the q_inv histograms.
cudaError_t persistent_same(const Device &d, const BatchDev &b, unsigned base, unsigned end,
                            int grid, cudaStream_t st, int mode);
cudaError_t persistent_mixed(const Device &d, const BatchDev &b, int grid, cudaStream_t st,
                             int mode);

namespace persist {

using namespace tile;

// Serving many analyses in one launch (MANY): the job's engine descriptor,
// its entry of b.devs, copied into shared memory.  A launch of one analysis
// reads the descriptor from its kernel parameter instead: its fields are
// then constant-bank operands, where a reference that may point to either
// the parameter or shared memory made every field a generic load (the
// same-event kernel took 141 ms per central group that way, 121 ms
// without).
__device__ __forceinline__ void load_device(const BatchDev &b, const BatchJob &job, Device &dsm) {
    const int *src = reinterpret_cast<const int *>(b.devs + job.dev);
    int *dst = reinterpret_cast<int *>(&dsm);
    for (int k = threadIdx.x; k < (int)(sizeof(Device) / sizeof(int)); k += blockDim.x)
        dst[k] = src[k];
    __syncthreads();
}

// Resident CTAs per SM (register budget 65536 / (128 x CTAs)), measured on
// GB300 in whole kernels.  FP64 form, central group: 5 (51.0 ms; 53.5 at 4,
// 55.1 at 6).  FP32-weight form: 5 (46.2 ms; 50.6 at 3, 47.8 at 4, 48.1 at 6).
// With q_inv histograms, 45,000 pions: same-event 5, what shared memory holds
// (17.0 ms a call; 17.1 at 4), mixed-event 7 (2.9 ms; 3.1 at 6, 3.2 at 5).
// Mixed-event without them: 5 (uneven events 2.57 ms, small ones 0.34; 2.74 and
// 0.37 at 6, 3.03 and 0.41 at 8).
#ifndef HBT_FP64_SAME_CTAS
#define HBT_FP64_SAME_CTAS 5  // compile-time choices (-D to measure others)
#endif
#ifndef HBT_FP32W_SAME_CTAS
#define HBT_FP32W_SAME_CTAS 5
#endif
#ifndef HBT_QINV_SAME_CTAS
#define HBT_QINV_SAME_CTAS 5
#endif
#ifndef HBT_MIXED_CTAS
#define HBT_MIXED_CTAS 5
#endif
#ifndef HBT_QINV_MIXED_CTAS
#define HBT_QINV_MIXED_CTAS 7
#endif
template <int PREC, bool QINV>
struct SameCtas {
    static constexpr int value =
        QINV ? HBT_QINV_SAME_CTAS : (PREC == 1 ? HBT_FP32W_SAME_CTAS : HBT_FP64_SAME_CTAS);
};
template <bool QINV>
struct MixedCtas {
    static constexpr int value = QINV ? HBT_QINV_MIXED_CTAS : HBT_MIXED_CTAS;
};

// Parts of a tile pair (ranges of its j-tile) that its items are split into:
// with fewer items than CTAs, a pair's 64 steps on one CTA are the launch's
// whole time, so up to kMaxParts CTAs share it, as long as all have a resident
// slot: for a list of 1,000 (36 tile pairs) 31 us in 4 parts, 22 us in 16.
constexpr unsigned kMaxParts = 16;
__device__ __forceinline__ unsigned item_parts(unsigned n_items) {
    unsigned parts = kMaxParts;
    while (parts > 1u && n_items > gridDim.x / parts) parts >>= 1;
    return parts;
}

// A list of the batch as the tile kernels read it (c: its column pointers).
__device__ __forceinline__ ListRows rows_of(const BatchDev &b, const BatchList &l,
                                            const double *const *c) {
    return ListRows{c,           b.orig + l.off, b.fixed + l.fixed_off, b.terms4 + l.off,
                    b.terms2 + l.off, b.fixed_cap, l.n};
}

// Same-event items [base, min(end, queued)) pulled by persistent CTAs.
// MODE: fast binning, or one pass of ordered cap admission; MANY: the items
// of many analyses (b.devs), fast binning only.
template <bool AZ, bool BOOST, int PREC, int MODE, bool QINV, bool MANY>
__global__ void __launch_bounds__(FT, SameCtas<PREC, QINV>::value)
    k_persistent_same(Device d, BatchDev b, unsigned base, unsigned end) {
    __shared__ SameSmem<PREC, QINV> sm;
    __shared__ unsigned item;
    __shared__ double cs[PREC == 0 ? kCosEntries : 1];  // the form's cos table
    if (PREC == 0)
        for (int k = threadIdx.x; k < kCosEntries; k += FT) cs[k] = b.cos[k];
    const unsigned stop = min(end, min(b.n_items[0], b.same_cap));
    const unsigned parts = item_parts(stop > base ? stop - base : 0u), rows = FT / parts;
    for (;;) {
        if (threadIdx.x == 0) item = atomicAdd(b.item_next, 1u);
        __syncthreads();
        const unsigned k = base + item / parts;
        const int jb = (int)((item % parts) * rows), je = jb + (int)rows;
        if (k >= stop) break;
        const Item it = b.items[b.order_items ? b.item_pos_out[k] : k];
        const BatchJob &job = b.jobs[it.job];
        const BatchList &la = b.lists[job.la];
        const double *c[8];
#pragma unroll
        for (int f = 0; f < 8; f++) c[f] = b.table + (long long)f * b.cap + la.off;
        if constexpr (MANY) {
            __shared__ Device dsm;
            load_device(b, job, dsm);
            same_tile_pair<AZ, BOOST, PREC, MODE, QINV>(dsm, sm, cs, rows_of(b, la, c),
                                                        (long long)it.ti * FT,
                                                        (long long)it.tj * FT, jb, je);
        } else {
            same_tile_pair<AZ, BOOST, PREC, MODE, QINV>(d, sm, cs, rows_of(b, la, c),
                                                        (long long)it.ti * FT,
                                                        (long long)it.tj * FT, jb, je);
        }
        __syncthreads();
    }
}

// Mixed-event items, all in one launch.
template <bool AZ, bool BOOST, int MODE, bool QINV, bool MANY>
__global__ void __launch_bounds__(FT, MixedCtas<QINV>::value)
    k_persistent_mixed(Device d, BatchDev b) {
    __shared__ MixedSmem sm;
    __shared__ unsigned item;
    const unsigned stop = min(b.n_items[1], b.mixed_cap);
    const unsigned parts = item_parts(stop), rows = FT / parts;
    for (;;) {
        if (threadIdx.x == 0) item = atomicAdd(b.item_next + 1, 1u);
        __syncthreads();
        const unsigned k = item / parts;
        const int jb = (int)((item % parts) * rows), je = jb + (int)rows;
        if (k >= stop) break;
        const Item it = b.items[b.same_cap + k];
        const BatchJob &job = b.jobs[it.job];
        const BatchList &la = b.lists[job.la], &lb = b.lists[job.lb];
        const double *c1[4], *c2[4];
#pragma unroll
        for (int f = 0; f < 4; f++) {
            c1[f] = b.table + (long long)f * b.cap + la.off;
            c2[f] = b.table + (long long)f * b.cap + lb.off;
        }
        if constexpr (MANY) {
            __shared__ Device dsm;
            load_device(b, job, dsm);
            mixed_tile_pair<AZ, BOOST, MODE, QINV>(
                dsm, sm, rows_of(b, la, c1), rows_of(b, lb, c2), (long long)it.ti * FT,
                (long long)it.tj * FT, job.row_base, jb, je);
        } else {
            mixed_tile_pair<AZ, BOOST, MODE, QINV>(
                d, sm, rows_of(b, la, c1), rows_of(b, lb, c2), (long long)it.ti * FT,
                (long long)it.tj * FT, job.row_base, jb, je);
        }
        __syncthreads();
    }
}

inline int sm_count() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            sms = 152;
    }
    return sms;
}

// grid > 0: that many CTAs; otherwise one CTA per resident slot; never more
// than the candidate items make parts (item_parts).
template <class K>
int persistent_grid(K kernel, int grid, unsigned items) {
    if (grid <= 0) {
        int nb = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, FT, 0) != cudaSuccess ||
            nb < 1)
            nb = 4;
        grid = sm_count() * nb;
    }
    return (int)std::max(1ll, std::min((long long)grid, (long long)kMaxParts * items));
}

// The kernel for one analysis, or (b.devs, fast binning only) for many.
template <bool AZ, bool BOOST, int PREC, int MODE, bool QINV>
cudaError_t launch_same_items(const Device &d, const BatchDev &b, unsigned base, unsigned end,
                              int grid, cudaStream_t st) {
    if (b.devs) {
        if constexpr (MODE == MODE_FAST) {
            grid = persistent_grid(k_persistent_same<AZ, BOOST, PREC, MODE, QINV, true>, grid,
                                   b.same_cap);
            k_persistent_same<AZ, BOOST, PREC, MODE, QINV, true><<<grid, FT, 0, st>>>(d, b, base,
                                                                                     end);
            return cudaGetLastError();
        }
        return cudaErrorNotSupported;
    }
    grid = persistent_grid(k_persistent_same<AZ, BOOST, PREC, MODE, QINV, false>, grid,
                           b.same_cap);
    k_persistent_same<AZ, BOOST, PREC, MODE, QINV, false><<<grid, FT, 0, st>>>(d, b, base, end);
    return cudaGetLastError();
}

template <bool AZ, bool BOOST, int MODE, bool QINV>
cudaError_t launch_mixed_items(const Device &d, const BatchDev &b, int grid, cudaStream_t st) {
    if (b.devs) {
        if constexpr (MODE == MODE_FAST) {
            grid = persistent_grid(k_persistent_mixed<AZ, BOOST, MODE, QINV, true>, grid,
                                   b.mixed_cap);
            k_persistent_mixed<AZ, BOOST, MODE, QINV, true><<<grid, FT, 0, st>>>(d, b);
            return cudaGetLastError();
        }
        return cudaErrorNotSupported;
    }
    grid = persistent_grid(k_persistent_mixed<AZ, BOOST, MODE, QINV, false>, grid, b.mixed_cap);
    k_persistent_mixed<AZ, BOOST, MODE, QINV, false><<<grid, FT, 0, st>>>(d, b);
    return cudaGetLastError();
}

// The same-event kernel of the context's flags and precision form for one
// admission mode.  The COUNT pass only counts decided pairs per row, the
// same in every form, so it runs the FP64 form's kernel.
template <int MODE, bool QINV>
cudaError_t launch_same_mode(const Device &d, const BatchDev &b, unsigned base, unsigned end,
                             int grid, cudaStream_t st) {
    const bool az = d.g.azimuthal, boost = d.g.boost;
    // the COUNT pass runs the FP64 form's kernel, and so does the double-float
    // form: same bins, closer values, and faster than double-float arithmetic
    // (central group 50.8 against 79.7 ms)
    constexpr int P1 = MODE == MODE_COUNT ? 0 : 1;
    const int prec = MODE == MODE_COUNT || d.precision != 1 ? 0 : 1;
#define HBT_P(AZ_, BO_, PR_) \
    return launch_same_items<AZ_, BO_, PR_, MODE, QINV>(d, b, base, end, grid, st)
    if (prec == 0) {
        if (az && boost) HBT_P(true, true, 0);
        if (az) HBT_P(true, false, 0);
        if (boost) HBT_P(false, true, 0);
        HBT_P(false, false, 0);
    }
    if (az && boost) HBT_P(true, true, P1);
    if (az) HBT_P(true, false, P1);
    if (boost) HBT_P(false, true, P1);
    HBT_P(false, false, P1);
#undef HBT_P
}

template <int MODE, bool QINV>
cudaError_t launch_mixed_mode(const Device &d, const BatchDev &b, int grid, cudaStream_t st) {
    const bool az = d.g.azimuthal, boost = d.g.boost;
    if (az && boost) return launch_mixed_items<true, true, MODE, QINV>(d, b, grid, st);
    if (az) return launch_mixed_items<true, false, MODE, QINV>(d, b, grid, st);
    if (boost) return launch_mixed_items<false, true, MODE, QINV>(d, b, grid, st);
    return launch_mixed_items<false, false, MODE, QINV>(d, b, grid, st);
}

}  // namespace persist
}  // namespace hbt
