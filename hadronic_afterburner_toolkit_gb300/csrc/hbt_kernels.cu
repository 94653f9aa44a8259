// HBT pair-binning kernels for sm_103a (plain FP64 form).
//
// Every bin-deciding expression follows the reference's operand order
// (src/HBT_correlation.cpp:311-458 same-event, :574-687 mixed-event) and the
// translation unit is compiled with --fmad=false, so each FP64 add, multiply,
// divide and square root is the same IEEE-rounded operation the reference's
// CPU build performs.  Pair counts and bin indices are therefore bit-exact;
// only the order of the FP64 sums differs.
//
// Launch shapes
//  same-event : one CTA per (i-tile <= j-tile) pair of 128-particle tiles;
//               the j-tile is staged in shared memory, each thread owns one i.
//  mixed-event: one CTA per (list-1 tile, list-2 tile).
// Admission modes for the order-dependent pair caps (needed_number_of_pairs):
//  FAST  - no cap can bind in this launch: bin every survivor.
//  COUNT - count survivors per (stream bin, row) for the ordered pass.
//  ORDER - admit rows before each stream bin's cut row; the cut row itself
//          is admitted in pair order by the straddle kernel.
#include "hbt_engine.cuh"
#include <algorithm>

#include "hbt_chain.cuh"

namespace hbt {
namespace {

using namespace chain;

template <int MODE>
__global__ void __launch_bounds__(TILE) k_same(Device d, long long n, Cols8 c) {
    __shared__ double sj[8][TILE];
    long long ti, tj;
    tri_tile(blockIdx.x, ti, tj);
    const int tid = threadIdx.x;
    const long long j0 = tj * TILE;
    for (int f = 0; f < 8; f++) sj[f][tid] = (j0 + tid < n) ? c.p[f][j0 + tid] : 0.0;
    __syncthreads();
    const long long i = ti * TILE + tid;
    if (i >= n) return;
    const double apx = c.p[0][i], apy = c.p[1][i], apz = c.p[2][i], aE = c.p[3][i];
    const double ax[4] = {c.p[4][i], c.p[5][i], c.p[6][i], c.p[7][i]};
    const int jend = (int)min((long long)TILE, n - j0);
    for (int jj = 0; jj < jend; jj++) {
        const long long j = j0 + jj;
        if (j <= i) continue;
        const double bx[4] = {sj[4][jj], sj[5][jj], sj[6][jj], sj[7][jj]};
        const Chain ch = pair_chain<false>(d.g, apx, apy, apz, aE, sj[0][jj], sj[1][jj],
                                           sj[2][jj], sj[3][jj], ax, bx);
        consume<false, MODE>(d, i, j, n, n, ch);
    }
}

template <int MODE>
__global__ void __launch_bounds__(TILE) k_mixed(Device d, long long n1, Cols4 l1,
                                                long long n2, Cols4 l2, long long tiles1) {
    __shared__ double sj[4][TILE];
    const long long ti = blockIdx.x % tiles1;
    const long long tj = blockIdx.x / tiles1;
    const int tid = threadIdx.x;
    const long long j0 = tj * TILE;
    for (int f = 0; f < 4; f++) sj[f][tid] = (j0 + tid < n2) ? l2.p[f][j0 + tid] : 0.0;
    __syncthreads();
    const long long i = ti * TILE + tid;
    if (i >= n1) return;
    const double apx = l1.p[0][i], apy = l1.p[1][i], apz = l1.p[2][i], aE = l1.p[3][i];
    const int jend = (int)min((long long)TILE, n2 - j0);
    for (int jj = 0; jj < jend; jj++) {
        const Chain ch = pair_chain<true>(d.g, apx, apy, apz, aE, sj[0][jj], sj[1][jj],
                                          sj[2][jj], sj[3][jj], nullptr, nullptr);
        consume<true, MODE>(d, i, j0 + jj, n2, n1, ch);
    }
}

// Admission of a stream bin's cut row, pair by pair in column order, by many
// blocks: straddle_mark runs the reference chain on the row's pairs and
// leaves the survivors' bits and each block's count, straddle_admit bins the
// survivors whose rank is below the bin's quota (their chain again).  One
// warp per stream bin walking the row is bound by its serial chain of pairs: it
// took 9.6 ms for 60,000 columns (and 2.1 ms over mixed jobs); with the columns
// spread over blocks a capped run of that size went from 28.3 to 18.3 ms.

// The cut row of stream bin b: the first particle's columns and row, the row
// and column stride of the deferrals' keys, and the second particles.
struct CutRow {
    const double *const *a, *const *b;
    long long r, key_row, key_cols, first, cols;
};
template <bool MIXED>
__device__ __forceinline__ bool cut_row(const Device &d, int b, long long rows, long long cols,
                                        const double *const *a8, const double *const *b4,
                                        CutRow &t) {
    const long long r = d.caps.row_cut[b];
    if (r >= rows || d.caps.quota[b] == 0ull) return false;
    t = CutRow{a8, MIXED ? b4 : a8, r, r, cols, MIXED ? 0 : r + 1, cols};
    return true;
}
// The jobs' joint row order: row r belongs to the last job whose row_base is
// at most r.
__device__ __forceinline__ bool cut_row_jobs(const Device &d, int b, const StraddleJob *jobs,
                                             int n_jobs, long long rows, CutRow &t) {
    const long long r = d.caps.row_cut[b];
    if (r >= rows || d.caps.quota[b] == 0ull) return false;
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].row_base <= r)
            lo = mid;
        else
            hi = mid - 1;
    }
    const StraddleJob &job = jobs[lo];
    t = CutRow{job.a, job.b, r - job.row_base, r, d.caps.cols_key, 0, job.n2};
    return true;
}

// Does column j's pair fall in stream bin b (3-D slots first, then the q_inv
// K_T bins)?  Fills the chain and the slot.
template <bool MIXED>
__device__ __forceinline__ bool cut_pair(const Device &d, int b, const CutRow &t, long long j,
                                         Chain &c, int &slot) {
    if (j < t.first || j >= t.cols) return false;
    const int ns = d.g.n_slots;
    const double apx = t.a[0][t.r], apy = t.a[1][t.r], bpx = t.b[0][j], bpy = t.b[1][j];
    double ax[4] = {0, 0, 0, 0}, bx[4] = {0, 0, 0, 0};
    if (!MIXED)
        for (int f = 0; f < 4; f++) {
            ax[f] = t.a[4 + f][t.r];
            bx[f] = t.b[4 + f][j];
        }
    c = pair_chain<MIXED>(d.g, apx, apy, t.a[2][t.r], t.a[3][t.r], bpx, bpy, t.b[2][j], t.b[3][j],
                          ax, bx);
    if (c.iK < 0) return false;
    if (b >= ns) return c.qi_k >= 0 && ns + c.iK == b;
    slot = -1;
    if (c.ev3 == 1)
        slot = c.slot;
    else if (c.ev3 == 2)
        slot = resolved_slot(d, t.key_row * t.key_cols + j, c.iK);
    return slot == b;
}

template <bool MIXED>
__device__ __forceinline__ void straddle_mark(const Device &d, int b, const CutRow &t) {
    const int chunk = blockIdx.x % d.caps.straddle_chunks;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Chain c;
    int slot;
    const bool has =
        cut_pair<MIXED>(d, b, t, (long long)chunk * kStraddleCols + threadIdx.x, c, slot);
    const unsigned m = __ballot_sync(0xffffffffu, has);
    __shared__ unsigned cnt[kStraddleCols / 32];
    const long long at = (long long)b * d.caps.straddle_chunks + chunk;
    if (lane == 0) {
        d.caps.straddle_bits[at * (kStraddleCols / 32) + w] = m;
        cnt[w] = __popc(m);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned n = 0;
        for (int k = 0; k < kStraddleCols / 32; k++) n += cnt[k];
        d.caps.straddle_count[at] = n;
    }
}

template <bool MIXED>
__device__ __forceinline__ void straddle_admit(const Device &d, int b, const CutRow &t) {
    const int chunk = blockIdx.x % d.caps.straddle_chunks;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned *count = d.caps.straddle_count + (long long)b * d.caps.straddle_chunks;
    const unsigned long long quota = d.caps.quota[b];
    __shared__ unsigned long long before;
    if (threadIdx.x == 0) before = 0ull;
    __syncthreads();
    unsigned long long n = 0;
    for (int k = threadIdx.x; k < chunk; k += kStraddleCols) n += count[k];
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (lane == 0 && n) atomicAdd(&before, n);
    __syncthreads();
    if (before >= quota) return;
    const unsigned *bits = d.caps.straddle_bits +
                           ((long long)b * d.caps.straddle_chunks + chunk) * (kStraddleCols / 32);
    unsigned long long rank = before;
    for (int k = 0; k < w; k++) rank += __popc(bits[k]);
    rank += __popc(bits[w] & ((1u << lane) - 1u));
    if (!((bits[w] >> lane) & 1u) || rank >= quota) return;
    Chain c;
    int slot;
    if (!cut_pair<MIXED>(d, b, t, (long long)chunk * kStraddleCols + threadIdx.x, c, slot)) return;
    if (b >= d.g.n_slots) {
        if (MIXED)
            bin_den_qinv(d, c);
        else
            bin_num_qinv(d, c);
    } else {
        if (MIXED)
            bin_den3(d, slot, c.bin);
        else
            bin_num3(d, slot, c.bin, c);
    }
}

// One launch's cut rows (a block for each stream bin's chunk of columns).
template <bool MIXED, bool ADMIT>
__global__ void __launch_bounds__(kStraddleCols) k_straddle(Device d, long long rows,
                                                            long long cols, Cols8 a8, Cols4 b4) {
    const int b = blockIdx.x / d.caps.straddle_chunks;
    CutRow t;
    if (!cut_row<MIXED>(d, b, rows, cols, a8.p, b4.p, t)) return;
    if (ADMIT)
        straddle_admit<MIXED>(d, b, t);
    else
        straddle_mark<MIXED>(d, b, t);
}

// The cut rows of several mixed-event jobs admitted together.
template <bool ADMIT>
__global__ void __launch_bounds__(kStraddleCols) k_straddle_jobs(Device d, const StraddleJob *jobs,
                                                                 int n_jobs, long long rows) {
    const int b = blockIdx.x / d.caps.straddle_chunks;
    CutRow t;
    if (!cut_row_jobs(d, b, jobs, n_jobs, rows, t)) return;
    if (ADMIT)
        straddle_admit<true>(d, b, t);
    else
        straddle_mark<true>(d, b, t);
}

// Per stream bin: first row at which the running survivor count exceeds
// remaining[b]; everything before it is admitted, `quota` more inside it.
__global__ void __launch_bounds__(1024) k_cut(Device d, long long rows,
                                              const unsigned long long *remaining) {
    const int b = blockIdx.x;
    const unsigned long long rem = remaining[b];
    const unsigned *rc = d.caps.rowcnt + (long long)b * rows;
    __shared__ unsigned long long warp_tot[32];
    __shared__ long long found;
    __shared__ unsigned long long found_quota;
    if (threadIdx.x == 0) found = rows;
    unsigned long long running = 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (long long base = 0; base < rows; base += 1024) {
        const long long r = base + threadIdx.x;
        const unsigned long long v = r < rows ? rc[r] : 0;
        unsigned long long incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warp_tot[w] = incl;
        __syncthreads();
        unsigned long long before = 0;
        for (int k = 0; k < w; k++) before += warp_tot[k];
        incl += before;
        unsigned long long chunk = 0;
        for (int k = 0; k < 32; k++) chunk += warp_tot[k];
        const unsigned long long excl = running + incl - v;
        if (r < rows && running + incl > rem && excl <= rem) {
            // exactly one row satisfies this: the first that crosses rem
            found = r;
            found_quota = rem - excl;
        }
        __syncthreads();
        if (found < rows) break;
        running += chunk;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        d.caps.row_cut[b] = found;
        d.caps.quota[b] = found < rows ? found_quota : 0ull;
    }
}

// Bins deferred records with their host-resolved K_phi bins (fast mode).
__device__ __forceinline__ void apply_one(const Device &d, const Deferral *rec, const int *iphi,
                                          int k) {
    const int ip = iphi[k];
    if (ip < 0) return;
    const Deferral r = rec[k];
    const long long at = (long long)(r.iK * d.g.n_Kphi + ip) * d.g.q3 + r.bin;
    if (r.mixed) {
        atomicAdd(d.h.den + at, 1ull);
    } else {
        Sums *s = d.h.sums + at;
        atomicAdd(&s->qo, r.qo);
        atomicAdd(&s->qs, r.qs);
        atomicAdd(&s->ql, r.ql);
        atomicAdd(&s->w, r.cosw);
        atomicAdd(d.h.cnt + at, 1ull);
    }
}

__global__ void k_apply(Device d, const Deferral *rec, const int *iphi, int n) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) apply_one(d, rec, iphi, k);
}

// As k_apply, with the number of records read from device memory (decided
// by a host function queued on the same stream).
__global__ void k_apply_n(Device d, const Deferral *rec, const int *iphi, const int *count) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < *count) apply_one(d, rec, iphi, k);
}

// Adds host-resolved deferred pairs to the per-row survivor counts.
__global__ void k_defer_count(Device d, long long rows, long long cols, int n_res) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_res) return;
    const Resolved rv = d.caps.resolved[k];
    if (rv.iphi < 0) return;
    const long long i = rv.key / cols;
    const int slot = rv.iK * d.g.n_Kphi + rv.iphi;
    atomicAdd(d.caps.rowcnt + (long long)slot * rows + i, 1u);
}

// Pair counters = sums of the count histograms (each counter is
// incremented exactly when a pair is binned).  out: [num slots][den
// slots][num q_inv][den q_inv].
// kCounterParts blocks per counter, each adding its part of the bins (one
// block alone took 42 us for the 68,921 bins of a slot).
constexpr int kCounterParts = 16;
__global__ void __launch_bounds__(256) k_counters(Device d, unsigned long long *out) {
    const int ns = d.g.n_slots, nk = d.g.n_KT;
    const int b = blockIdx.x / kCounterParts, part = blockIdx.x % kCounterParts;
    const u64 *src;
    long long len;
    if (b < ns) {
        src = d.h.cnt + (long long)b * d.g.q3;
        len = d.g.q3;
    } else if (b < 2 * ns) {
        src = d.h.den + (long long)(b - ns) * d.g.q3;
        len = d.g.q3;
    } else if (b < 2 * ns + nk) {
        src = d.h.qi_cnt + (long long)(b - 2 * ns) * d.g.qnpts;
        len = d.g.qnpts;
    } else {
        src = d.h.qi_den + (long long)(b - 2 * ns - nk) * d.g.qnpts;
        len = d.g.qnpts;
    }
    unsigned long long s = 0;
    for (long long k = part * 256 + threadIdx.x; k < len; k += kCounterParts * 256) s += src[k];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    __shared__ unsigned long long ws[8];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int k = 0; k < 8; k++) t += ws[k];
        if (t) atomicAdd(out + b, t);
    }
}

Cols8 cols8(const double *const *c) {
    Cols8 r;
    for (int f = 0; f < 8; f++) r.p[f] = c ? c[f] : nullptr;
    return r;
}
Cols4 cols4(const double *const *c) {
    Cols4 r;
    for (int f = 0; f < 4; f++) r.p[f] = c ? c[f] : nullptr;
    return r;
}

}  // namespace

cudaError_t launch_same(const Device &d, int mode, long long n, const double *const *c8,
                        cudaStream_t st) {
    if (n < 2) return cudaSuccess;
    const long long nt = (n + TILE - 1) / TILE;
    const long long blocks = nt * (nt + 1) / 2;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    const Cols8 c = cols8(c8);
    if (mode == MODE_FAST)
        k_same<MODE_FAST><<<(unsigned)blocks, TILE, 0, st>>>(d, n, c);
    else if (mode == MODE_COUNT)
        k_same<MODE_COUNT><<<(unsigned)blocks, TILE, 0, st>>>(d, n, c);
    else
        k_same<MODE_ORDER><<<(unsigned)blocks, TILE, 0, st>>>(d, n, c);
    return cudaGetLastError();
}

cudaError_t launch_mixed(const Device &d, int mode, long long n1, const double *const *l1,
                         long long n2, const double *const *l2, cudaStream_t st) {
    if (n1 < 1 || n2 < 1) return cudaSuccess;
    const long long t1 = (n1 + TILE - 1) / TILE, t2 = (n2 + TILE - 1) / TILE;
    const long long blocks = t1 * t2;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    const Cols4 a = cols4(l1), b = cols4(l2);
    if (mode == MODE_FAST)
        k_mixed<MODE_FAST><<<(unsigned)blocks, TILE, 0, st>>>(d, n1, a, n2, b, t1);
    else if (mode == MODE_COUNT)
        k_mixed<MODE_COUNT><<<(unsigned)blocks, TILE, 0, st>>>(d, n1, a, n2, b, t1);
    else
        k_mixed<MODE_ORDER><<<(unsigned)blocks, TILE, 0, st>>>(d, n1, a, n2, b, t1);
    return cudaGetLastError();
}

cudaError_t launch_same_straddle(const Device &d, long long n, const double *const *c8,
                                 int n_stream, cudaStream_t st) {
    const long long grid = (long long)d.caps.straddle_chunks * n_stream;
    if (grid < 1) return cudaSuccess;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidValue;
    k_straddle<false, false><<<(unsigned)grid, kStraddleCols, 0, st>>>(d, n, n, cols8(c8), cols4(nullptr));
    k_straddle<false, true><<<(unsigned)grid, kStraddleCols, 0, st>>>(d, n, n, cols8(c8), cols4(nullptr));
    return cudaGetLastError();
}

cudaError_t launch_mixed_straddle(const Device &d, long long n1, const double *const *l1,
                                  long long n2, const double *const *l2, int n_stream,
                                  cudaStream_t st) {
    Cols8 a;
    for (int f = 0; f < 8; f++) a.p[f] = f < 4 ? l1[f] : nullptr;
    const long long grid = (long long)d.caps.straddle_chunks * n_stream;
    if (grid < 1) return cudaSuccess;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidValue;
    k_straddle<true, false><<<(unsigned)grid, kStraddleCols, 0, st>>>(d, n1, n2, a, cols4(l2));
    k_straddle<true, true><<<(unsigned)grid, kStraddleCols, 0, st>>>(d, n1, n2, a, cols4(l2));
    return cudaGetLastError();
}

cudaError_t launch_jobs_straddle(const Device &d, const StraddleJob *jobs, int n_jobs,
                                 long long rows, int n_stream, cudaStream_t st) {
    if (n_jobs < 1) return cudaSuccess;
    const long long grid = (long long)d.caps.straddle_chunks * n_stream;
    if (grid < 1) return cudaSuccess;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidValue;
    k_straddle_jobs<false><<<(unsigned)grid, kStraddleCols, 0, st>>>(d, jobs, n_jobs, rows);
    k_straddle_jobs<true><<<(unsigned)grid, kStraddleCols, 0, st>>>(d, jobs, n_jobs, rows);
    return cudaGetLastError();
}

cudaError_t launch_cut(const Device &d, long long rows, int n_stream,
                       const unsigned long long *remaining, cudaStream_t st) {
    k_cut<<<n_stream, 1024, 0, st>>>(d, rows, remaining);
    return cudaGetLastError();
}

cudaError_t launch_apply(const Device &d, const Deferral *rec, const int *iphi, int n,
                         cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_apply<<<(n + 127) / 128, 128, 0, st>>>(d, rec, iphi, n);
    return cudaGetLastError();
}

cudaError_t launch_apply_n(const Device &d, const Deferral *rec, const int *iphi, const int *count,
                           int cap, cudaStream_t st) {
    k_apply_n<<<(cap + 127) / 128, 128, 0, st>>>(d, rec, iphi, count);
    return cudaGetLastError();
}

cudaError_t launch_defer_count(const Device &d, long long rows, long long cols, int n_res,
                               cudaStream_t st) {
    if (n_res <= 0) return cudaSuccess;
    k_defer_count<<<(n_res + 127) / 128, 128, 0, st>>>(d, rows, cols, n_res);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(256) k_export(Device d, int field, double *out,
                                                long long nbins) {
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nbins;
         k += (long long)gridDim.x * blockDim.x) {
        double v;
        switch (field) {
            case 0: v = d.h.sums[k].qo; break;
            case 1: v = d.h.sums[k].qs; break;
            case 2: v = d.h.sums[k].ql; break;
            case 3: v = d.h.sums[k].w; break;
            case 4: v = (double)d.h.cnt[k]; break;
            default: v = (double)d.h.den[k]; break;
        }
        out[k] = v;
    }
}

// The six arrays of hbt_read_hist (any may be null) in one pass over the
// histograms, with the status words: into host memory where the GPU writes
// it.  Six kernels and copies took 127 us for the smallest histograms.
__global__ void __launch_bounds__(256) k_export_all(Device d, HistOut o, long long nbins) {
    if (blockIdx.x == 0 && threadIdx.x < STAT_N) o.stats[threadIdx.x] = d.stats[threadIdx.x];
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nbins;
         k += (long long)gridDim.x * blockDim.x) {
        const Sums s = d.h.sums[k];
        if (o.v[0]) o.v[0][k] = s.qo;
        if (o.v[1]) o.v[1][k] = s.qs;
        if (o.v[2]) o.v[2][k] = s.ql;
        if (o.v[3]) o.v[3][k] = s.w;
        if (o.v[4]) o.v[4][k] = (double)d.h.cnt[k];
        if (o.v[5]) o.v[5][k] = (double)d.h.den[k];
    }
}

// The four arrays of hbt_read_qinv (any may be null) and the status words.
__global__ void __launch_bounds__(256) k_export_qinv(Device d, HistOut o, long long nbins) {
    if (blockIdx.x == 0 && threadIdx.x < STAT_N) o.stats[threadIdx.x] = d.stats[threadIdx.x];
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nbins;
         k += (long long)gridDim.x * blockDim.x) {
        if (o.v[0]) o.v[0][k] = d.h.qi_sums[k].q;
        if (o.v[1]) o.v[1][k] = d.h.qi_sums[k].w;
        if (o.v[2]) o.v[2][k] = (double)d.h.qi_cnt[k];
        if (o.v[3]) o.v[3][k] = (double)d.h.qi_den[k];
    }
}

cudaError_t launch_export_all(const Device &d, const HistOut &o, long long nbins, bool qinv,
                              cudaStream_t st) {
    const unsigned blocks =
        (unsigned)std::max<long long>(1, std::min<long long>((nbins + 255) / 256, 152 * 8));
    if (qinv)
        k_export_qinv<<<blocks, 256, 0, st>>>(d, o, nbins);
    else
        k_export_all<<<blocks, 256, 0, st>>>(d, o, nbins);
    return cudaGetLastError();
}

// One warp per q_inv bin; the copies are added in lane order (the same sum on
// every run for the same copies).
__global__ void __launch_bounds__(256) k_qinv_merge(Device d, int nq) {
    const int bin = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (bin >= nq) return;
    QiPart s = {0.0, 0.0, 0.0, 0.0};
    for (int c = lane; c < kQiCopies; c += 32) {
        QiPart &p = d.h.qi_part[(long long)c * nq + bin];
        s.q += p.q;
        s.w += p.w;
        s.n += p.n;
        s.den += p.den;
        p = QiPart{0.0, 0.0, 0.0, 0.0};
    }
    for (int o = 16; o > 0; o >>= 1) {
        s.q += __shfl_down_sync(0xffffffffu, s.q, o);
        s.w += __shfl_down_sync(0xffffffffu, s.w, o);
        s.n += __shfl_down_sync(0xffffffffu, s.n, o);
        s.den += __shfl_down_sync(0xffffffffu, s.den, o);
    }
    if (lane == 0) {
        d.h.qi_sums[bin].q += s.q;
        d.h.qi_sums[bin].w += s.w;
        d.h.qi_cnt[bin] += (u64)s.n;
        d.h.qi_den[bin] += (u64)s.den;
    }
}

cudaError_t launch_qinv_merge(const Device &d, cudaStream_t st) {
    const int nq = d.g.n_KT * d.g.qnpts;
    k_qinv_merge<<<(nq * 32 + 255) / 256, 256, 0, st>>>(d, nq);
    return cudaGetLastError();
}

// One segment per block: read across the CPU link, whose latency (1 to 2 us)
// sets how much must be in flight.  One launch takes a batch's 880 columns
// (12.8 MB) over in 85 us, 150 GB/s, where one cudaMemcpyAsync per column
// took 1.9 ms, 2 us each.
__global__ void __launch_bounds__(256) k_copy_in(const CopySeg *segs, int n) {
    for (int s = blockIdx.x; s < n; s += gridDim.x) {
        const CopySeg g = segs[s];
#pragma unroll 4
        for (long long k = threadIdx.x; k < g.n; k += blockDim.x) g.dst[k] = g.src[k];
    }
}

cudaError_t launch_copy_in(const CopySeg *segs, int n, cudaStream_t st) {
    if (n < 1) return cudaSuccess;
    k_copy_in<<<std::min(n, 152 * 8), 256, 0, st>>>(segs, n);
    return cudaGetLastError();
}

cudaError_t launch_export(const Device &d, int field, double *out, long long nbins,
                          cudaStream_t st) {
    const long long blocks = std::min<long long>((nbins + 255) / 256, 152 * 16);
    k_export<<<(unsigned)std::max<long long>(blocks, 1), 256, 0, st>>>(d, field, out, nbins);
    return cudaGetLastError();
}

cudaError_t launch_counters(const Device &d, unsigned long long *out, cudaStream_t st) {
    const int n = 2 * d.g.n_slots + 2 * d.g.n_KT;
    const cudaError_t e = cudaMemsetAsync(out, 0, n * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    k_counters<<<n * kCounterParts, 256, 0, st>>>(d, out);
    return cudaGetLastError();
}

}  // namespace hbt
