// Batched Gaussian HBT radii fits (include/hbt_fit.h).
//
// The reference fits each correlation table with scipy's curve_fit, one
// table and one q_cut at a time (ebe_scripts/fit_HBT_radii.py:60-92).  Here
// all fits of a batch of tables advance together:
//
//  * k_fit_count and k_fit_select (a block for each 4096 rows of a table)
//    apply the script's preprocessing (numpy nan_to_num, C_err + 1e-15, weight
//    1 / sigma) and keep the rows with q_cut_min < |q| < the largest cut,
//    ordered by the smallest cut they pass, so the rows of cut k are a prefix
//    of the table's kept rows.  Per row they store the five q products of the
//    exponent (FP64 and FP32), C and the weight.
//  * Each fit's rows are cut into work items of up to 8192 rows, four units
//    each.  A pass (k_fit_pass, a block per unit) sums chi^2, J^T r and J^T J
//    of every active fit's units at its trial point; the block that finishes a
//    fit's last unit adds them and makes one Levenberg-Marquardt step: damped
//    6 x 6 system by Cholesky, accept or reject, next trial point.  Passes
//    repeat until no fit has a trial point; work is balanced over the GPU
//    whatever the fits' sizes, and finished fits are passed over.
//  * A last pass sums J^T J in FP64 at each minimum; k_fit_finish inverts
//    it for the errors sqrt(diag((J^T J)^-1)) (curve_fit, absolute_sigma).
//
// A pass reads 76 bytes per row against 32 FP64 operations (exp table-driven,
// hbt_math.cuh): the fits are bound by the FP64 pipe.  The order in which a
// fit's rows are added is fixed (lane, unit, item), so a fit's result does not
// depend on the other fits of the call.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/hbt_fit.h"
#include "hbt_math.cuh"

namespace {

constexpr double kHbarC = 0.19733;  // fit_HBT_radii.py:10
constexpr double kEps = 1e-15;      // fit_HBT_radii.py:11
constexpr int kMaxCuts = 16;
constexpr int kSelThreads = 512;
constexpr int kSelRows = 4096;  // a selection block's rows
constexpr int kFitThreads = 128;
constexpr int kSums = 28;  // chi2, J^T r (6), J^T J (21, packed lower)
// A work item: up to kItemRows consecutive kept rows of one fit, in kItemUnits
// units of 32 lanes: lane l of unit w takes every kItemStride-th row from
// 32 w + l on.
constexpr int kItemRows = 8192;
constexpr int kItemUnits = 4;
constexpr int kItemStride = 32 * kItemUnits;
constexpr int kItemWarps = kFitThreads / 32;  // warps to a unit

// Resident pass CTAs per SM the pass kernel is compiled for.
#ifndef HBT_FIT_MIN_BLOCKS
#define HBT_FIT_MIN_BLOCKS 4
#endif

struct FitConst {
    double cut_sorted[kMaxCuts];  // ascending
    // the cuts on |q|^2 as bits of doubles: sqrt(s) < cut_sorted[c] exactly
    // when s < cut_sq[c], sqrt(s) > q_cut_min exactly when s > min_sq
    long long cut_sq[kMaxCuts], min_sq;
    int rank[kMaxCuts];           // position of cut k in cut_sorted
    int n_cuts;
    double q_cut_min;
    double p0[6];
    int max_iter;
};

// Where a table's columns sit in the batch's input buffer: column k of row
// i at in[base + col[k] + i * stride].  An interleaved host table (all five
// columns in one row-major block) is copied as that block; other tables are
// packed column by column (stride 1).
struct TabDesc {
    long long base, stride, col[5];
};

// Device rows of a batch: the kept rows of table t start at row_off[t];
// cls[t * (n_cuts + 1) + c] = rows of t whose smallest passed cut is c.
// Column k of kept row o: d[k * ld + o] for the doubles (the five q
// products q_out^2, q_side^2, q_long^2, 2 q_out q_side, 2 q_out q_long, then
// C and the weight), f[k * ld + o] for the FP32 copies of the q products.
// One base pointer each keeps the fitting loop's registers for its sums.
struct Rows {
    double *d;
    float *f;
    long long ld;
};
constexpr int kColC = 5, kColW = 6;

__device__ __forceinline__ double nan_to_num(double v) {
    const int hi = __double2hiint(v);
    if ((hi & 0x7ff00000) != 0x7ff00000) return v;
    if ((hi & 0xfffff) | __double2loint(v)) return 0.0;
    return hi > 0 ? DBL_MAX : -DBL_MAX;
}

// The smallest cut that |q| = sqrt(q_out**2. + q_side**2. + q_long**2.)
// passes (numpy's sum, without contraction), -1 for none.  The cuts are
// compared on the sum itself, as integers (it is never negative or NaN).
__device__ __forceinline__ int cut_class(const FitConst &fc, double qo, double qs, double ql) {
    const long long s = __double_as_longlong(
        __dadd_rn(__dadd_rn(__dmul_rn(qo, qo), __dmul_rn(qs, qs)), __dmul_rn(ql, ql)));
    if (!(s > fc.min_sq)) return -1;
    for (int c = 0; c < fc.n_cuts; c++)
        if (s < fc.cut_sq[c]) return c;
    return -1;
}

// A selection block's rows: part p of table t.
struct SelPart {
    int t, p;
};

// Row selection, sweep 1: the rows of each cut class (the smallest cut a row
// passes) in each part of kSelRows rows, part_cls[block][c].
//
// Both sweeps read 24 or 40 bytes a row against the few FP64 operations of
// |q|^2; with one block for a whole table and square roots in FP64 they took
// 1.59 ms for 64 tables of 41^3 rows (64 of 152 SMs), now 65 + 190 us.
__global__ void __launch_bounds__(kSelThreads)
    k_fit_count(FitConst fc, const long long *tab_off, const TabDesc *desc, const double *in,
                const SelPart *parts, int *part_cls) {
    __shared__ int cnt[kMaxCuts];
    const SelPart P = parts[blockIdx.x];
    const TabDesc d = desc[P.t];
    const long long i0 = (long long)P.p * kSelRows;
    const long long i1 = min(i0 + kSelRows, tab_off[P.t + 1] - tab_off[P.t]);
    const double *qo_in = in + d.base + d.col[0], *qs_in = in + d.base + d.col[1],
                 *ql_in = in + d.base + d.col[2];
    if (threadIdx.x < kMaxCuts) cnt[threadIdx.x] = 0;
    __syncthreads();
    int mine[kMaxCuts];
#pragma unroll
    for (int c = 0; c < kMaxCuts; c++) mine[c] = 0;
    for (long long i = i0 + threadIdx.x; i < i1; i += kSelThreads) {
        const int c = cut_class(fc, nan_to_num(qo_in[i * d.stride]), nan_to_num(qs_in[i * d.stride]),
                                nan_to_num(ql_in[i * d.stride]));
#pragma unroll
        for (int k = 0; k < kMaxCuts; k++) mine[k] += (c == k);
    }
#pragma unroll
    for (int k = 0; k < kMaxCuts; k++) {
        if (k >= fc.n_cuts) break;
        const int v = __reduce_add_sync(0xffffffffu, mine[k]);
        if ((threadIdx.x & 31) == 0 && v) atomicAdd(&cnt[k], v);
    }
    __syncthreads();
    if (threadIdx.x < fc.n_cuts)
        part_cls[(long long)blockIdx.x * fc.n_cuts + threadIdx.x] = cnt[threadIdx.x];
}

// Sweep 2 writes every kept row at its class's running position: within a
// class, rows keep their table order (the same arrays and sums on every run).
// first[t] is table t's first part; part 0 leaves the table's class counts.
__global__ void __launch_bounds__(kSelThreads)
    k_fit_select(FitConst fc, const long long *tab_off, const TabDesc *desc, const double *in,
                 const SelPart *parts, const int *first, const int *part_cls, Rows out, int *cls) {
    __shared__ int cnt[kSelThreads / 32][kMaxCuts];
    __shared__ int base[kMaxCuts], total[kMaxCuts];
    const SelPart P = parts[blockIdx.x];
    const int t = P.t;
    const long long r0 = tab_off[t], n = tab_off[t + 1] - r0;
    const TabDesc d = desc[t];
    const double *qo_in = in + d.base + d.col[0], *qs_in = in + d.base + d.col[1],
                 *ql_in = in + d.base + d.col[2], *c_in = in + d.base + d.col[3],
                 *e_in = in + d.base + d.col[4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nc = fc.n_cuts;
    const unsigned below = (1u << lane) - 1u;
    // a class's rows in the parts before this one and in the whole table
    for (int c = warp; c < nc; c += kSelThreads / 32) {
        int before = 0, all = 0;
        for (int b = first[t] + lane; b < first[t + 1]; b += 32) {
            const int v = part_cls[(long long)b * nc + c];
            all += v;
            if (b < (int)blockIdx.x) before += v;
        }
        before = __reduce_add_sync(0xffffffffu, before);
        all = __reduce_add_sync(0xffffffffu, all);
        if (lane == 0) {
            base[c] = before;
            total[c] = all;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int c = 0; c < nc; c++) {
            base[c] += run;
            run += total[c];
            if (P.p == 0) cls[t * (nc + 1) + c] = total[c];
        }
        if (P.p == 0) cls[t * (nc + 1) + nc] = run;
    }
    __syncthreads();
    // chunk by chunk, rank each row among its class in row order
    const long long i1 = min(((long long)P.p + 1) * kSelRows, n);
    for (long long i0 = (long long)P.p * kSelRows; i0 < i1; i0 += kSelThreads) {
        const long long i = i0 + threadIdx.x;
        double qo = 0, qs = 0, ql = 0;
        int c = -1;
        if (i < i1) {
            qo = nan_to_num(qo_in[i * d.stride]);
            qs = nan_to_num(qs_in[i * d.stride]);
            ql = nan_to_num(ql_in[i * d.stride]);
            c = cut_class(fc, qo, qs, ql);
        }
        // this warp's rows per class: zeroed, then each class group's first
        // lane writes the group's size
        for (int k = lane; k < nc; k += 32) cnt[warp][k] = 0;
        __syncwarp();
        const unsigned same = __match_any_sync(0xffffffffu, c);
        if (c >= 0 && lane == __ffs(same) - 1) cnt[warp][c] = __popc(same);
        __syncthreads();
        if (c >= 0) {
            int off = base[c] + __popc(same & below);
            for (int w = 0; w < warp; w++) off += cnt[w][c];
            const long long o = r0 + off;
            const double cc = nan_to_num(c_in[i * d.stride]);
            const double sigma = nan_to_num(e_in[i * d.stride]) + kEps;
            const double q5[5] = {qo * qo, qs * qs, ql * ql, 2.0 * qo * qs, 2.0 * qo * ql};
            for (int k = 0; k < 5; k++) {
                out.d[k * out.ld + o] = q5[k];
                out.f[k * out.ld + o] = (float)q5[k];
            }
            out.d[kColC * out.ld + o] = cc;
            out.d[kColW * out.ld + o] = 1.0 / sigma;
        }
        __syncthreads();
        if (threadIdx.x < nc) {
            int tot = 0;
            for (int w = 0; w < kSelThreads / 32; w++) tot += cnt[w][threadIdx.x];
            base[threadIdx.x] += tot;
        }
        __syncthreads();
    }
}

// Sums each of v[0..7] over the warp's lanes: every halving exchanges the half
// a lane gives up, 9 adds instead of 5 for each value (and the same pairs as
// the tree of one value, so the same result).  Lane l returns sum l / 4.
__device__ __forceinline__ double warp_sums(double (&v)[8]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int h = 4, o = 16; h >= 1; h /= 2, o /= 2) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const double give = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    return v[0];
}

__device__ __forceinline__ double fma_rn(double a, double b, double c) {
    return __fma_rn(a, b, c);
}
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// A step's row of one lane, as the columns give it.
struct RowIn {
    double q[5], w, c;
    float f[5];
};
__device__ __forceinline__ void load_row(const Rows &rw, long long o, bool in, RowIn &x) {
#pragma unroll
    for (int k = 0; k < 5; k++) {
        x.q[k] = in ? rw.d[k * rw.ld + o] : 0.0;
        x.f[k] = in ? rw.f[k * rw.ld + o] : 0.f;
    }
    x.w = in ? rw.d[kColW * rw.ld + o] : 0.0;
    x.c = in ? rw.d[kColC * rw.ld + o] : 0.0;
}

// The steps of a batch in shared memory: v[0..5], r, and the FP32 J.
constexpr int kBatchSteps = 8;
struct StepBuf {
    double v[kBatchSteps][7][32];
    float j[kBatchSteps][6][32];
};

// The chains of warp G of a pass's block: s and sa by number.
template <int G>
struct Chains {
    static constexpr int s0 = 2 * G, ns = G == 3 ? 1 : 2;   // of chi^2, J^T r
    static constexpr int a0 = 5 * G, na = G == 3 ? 6 : 5;   // of J^T J
};
// J^T J's element m is the product of columns col_j(m) and col_k(m).
__host__ __device__ constexpr int col_j(int m) {
    int j = 0;
    while ((j + 1) * (j + 2) / 2 <= m) j++;
    return j;
}
__host__ __device__ constexpr int col_k(int m) { return m - col_j(m) * (col_j(m) + 1) / 2; }

template <int G, class AccT>
__device__ __forceinline__ void add_steps(const StepBuf &b, int lane, double (&s)[2],
                                          AccT (&sa)[6]) {
    using C = Chains<G>;
#pragma unroll
    for (int t = 0; t < kBatchSteps; t++) {
        const double r = b.v[t][6][lane];
#pragma unroll
        for (int k = 0; k < C::ns; k++) {
            const int n = C::s0 + k;
            s[k] = __fma_rn(n == 0 ? r : b.v[t][n == 0 ? 6 : n - 1][lane], r, s[k]);
        }
        AccT v[6];
#pragma unroll
        for (int k = 0; k < 6; k++) {
            if constexpr (std::is_same<AccT, double>::value)
                v[k] = b.v[t][k][lane];
            else
                v[k] = b.j[t][k][lane];
        }
#pragma unroll
        for (int k = 0; k < C::na; k++) {
            sa[k] = fma_rn(v[col_j(C::a0 + k)], v[col_k(C::a0 + k)], sa[k]);
        }
    }
}

// A trial point's constants: lambda, a_k^2 and the factors of the 28 sums.
struct PassConst {
    double lam, a2[5], factor[kSums];
};

// A warp's chains summed over its lanes, with J's constant factors: lane 4 k
// leaves its sum k.
template <int G, class AccT>
__device__ __forceinline__ void store_chains(const double (&s)[2], const AccT (&sa)[6],
                                             const PassConst &pc, double *out) {
    using C = Chains<G>;
    double tot[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < C::ns; k++) tot[k] = C::s0 + k == 0 ? s[k] : s[k] * pc.factor[C::s0 + k];
#pragma unroll
    for (int k = 0; k < C::na; k++) tot[C::ns + k] = (double)sa[k] * pc.factor[7 + C::a0 + k];
    const double x = warp_sums(tot);
    const int lane = threadIdx.x & 31, k = lane >> 2;
    if ((lane & 3) == 0 && k < C::ns + C::na)
        __stcg(out + (k < C::ns ? C::s0 + k : 7 + C::a0 + k - C::ns), x);
}

#define FIT_BY_WARP(g, call)      \
    switch (g) {                  \
        case 0: call(0); break;   \
        case 1: call(1); break;   \
        case 2: call(2); break;   \
        default: call(3); break;  \
    }

// One pass at parameters p: chi^2, J^T r, J^T J of the rows first, first +
// kItemStride, ... below n of an item, for 32 neighbouring `first` (a unit)
// by the block, to out[0..27].
// Residual r = w (f - C), J = w df/dp with f = lambda exp(-E),
// E = sum_k a_k^2 Q_k over the five q products Q_k (a_k = R_k / hbar c), so
// J_0 = w e and J_k = -w f (2 a_k / hbar c) Q_k: the constant factors
// 2 a_k / hbar c are applied after the sums.  chi^2 and J^T r, which fix
// where the minimum is, are summed in FP64.  J^T J only shapes the steps
// while iterating (kExact = false: FP32 products and sums over a lane's at
// most 64 rows, 1e-5 relative); the pass at the minimum that gives the
// covariance sums it in FP64 (kExact = true).
//
// A lane's rows add up in row order.  The block's four warps evaluate two
// steps each of eight (a step: one row a lane), then each adds the eight
// steps to its share of the 28 sums: an SM sub-partition gives one FP64 warp
// instruction in 64 clocks, so one warp alone needs 150 us for the 64 steps of
// a full unit, however few fits are still active, and four of them a quarter.
template <bool kExact>
__device__ __forceinline__ void fit_unit(const Rows &rw, long long r0, int first, int n,
                                         const PassConst &pc, const double *etab, StepBuf *buf,
                                         double *out) {
    using AccT = typename std::conditional<kExact, double, float>::type;
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    double a2[5];
#pragma unroll
    for (int k = 0; k < 5; k++) a2[k] = pc.a2[k];
    const double lam = pc.lam;
    double s[2] = {0.0, 0.0};
    AccT sa[6] = {0, 0, 0, 0, 0, 0};
    constexpr int kMine = kBatchSteps / kItemWarps;  // steps of a warp in a batch
    RowIn x[kMine];
    auto load = [&](int b) {
#pragma unroll
        for (int m = 0; m < kMine; m++) {
            const int i = first + lane + (b + g * kMine + m) * kItemStride;
            load_row(rw, r0 + i, i < n, x[m]);
        }
    };
    load(0);
    for (int b = 0, at = 0; first + b * kItemStride < n; b += kBatchSteps, at ^= 1) {
        StepBuf &sb = buf[at];
#pragma unroll
        for (int m = 0; m < kMine; m++) {
            const int t = g * kMine + m;
            const RowIn &y = x[m];
            double E = 0.0;
#pragma unroll
            for (int k = 0; k < 5; k++) E = __fma_rn(a2[k], y.q[k], E);
            const double e = table_exp(etab, -E);
            const double f = lam * e;
            // a lane past the item's end adds zeros
            const bool in = first + lane + (b + t) * kItemStride < n;
            const double r = in ? __dmul_rn(y.w, __dsub_rn(f, y.c)) : 0.0;
            const double u = in ? y.w * f : 0.0;
            const double v0 = in ? y.w * e : 0.0;
            sb.v[t][0][lane] = v0;
#pragma unroll
            for (int k = 0; k < 5; k++) sb.v[t][k + 1][lane] = u * y.q[k];
            sb.v[t][6][lane] = r;
            if (!kExact) {
                const float uf = to_float_rn(u);
                sb.j[t][0][lane] = to_float_rn(v0);
#pragma unroll
                for (int k = 0; k < 5; k++) sb.j[t][k + 1][lane] = uf * y.f[k];
            }
        }
        load(b + kBatchSteps);
        __syncthreads();
#define FIT_ADD(G) add_steps<G>(sb, lane, s, sa)
        FIT_BY_WARP(g, FIT_ADD)
#undef FIT_ADD
    }
#define FIT_STORE(G) store_chains<G>(s, sa, pc, out)
    FIT_BY_WARP(g, FIT_STORE)
#undef FIT_STORE
}
#undef FIT_BY_WARP

// Cholesky of the packed symmetric 6 x 6 matrix M (lower, row-major
// packed: M[j(j+1)/2 + k], k <= j) in place; false if not positive definite.
__device__ bool cholesky6(double *M) {
    for (int j = 0; j < 6; j++) {
        for (int k = 0; k <= j; k++) {
            double s = M[j * (j + 1) / 2 + k];
            for (int l = 0; l < k; l++) s -= M[j * (j + 1) / 2 + l] * M[k * (k + 1) / 2 + l];
            if (k == j) {
                if (!(s > 0.0)) return false;
                M[j * (j + 1) / 2 + j] = sqrt(s);
            } else {
                M[j * (j + 1) / 2 + k] = s / M[k * (k + 1) / 2 + k];
            }
        }
    }
    return true;
}

// Solves L L^T x = b with the factor of cholesky6.
__device__ void chol_solve6(const double *L, const double *b, double *x) {
    double y[6];
    for (int j = 0; j < 6; j++) {
        double s = b[j];
        for (int l = 0; l < j; l++) s -= L[j * (j + 1) / 2 + l] * y[l];
        y[j] = s / L[j * (j + 1) / 2 + j];
    }
    for (int j = 5; j >= 0; j--) {
        double s = y[j];
        for (int l = j + 1; l < 6; l++) s -= L[l * (l + 1) / 2 + j] * x[l];
        x[j] = s / L[j * (j + 1) / 2 + j];
    }
}

// Levenberg-Marquardt state of one fit, in device memory, advanced by one
// thread of the block that finishes the fit's last unit of a pass.
struct LmState {
    double x[6], trial[6];
    double S, g[6], A[21], D[6], mu, nu;
    int iter, status, stop, go;
    int use_x;  // the next pass evaluates x (the start point), not trial
    int done;   // units finished in the current pass
    long long passes;
};

// After the pass at the start point.
__device__ __noinline__ void lm_init(LmState &st, const double *red) {
    st.S = red[0];
    for (int j = 0; j < 6; j++) st.g[j] = red[1 + j];
    for (int j = 0; j < 21; j++) st.A[j] = red[7 + j];
    // Marquardt's scaling: the damping adds mu times the diagonal of J^T J
    // (dimensionless mu), so every parameter is damped on its own scale
    for (int j = 0; j < 6; j++) {
        const double d = st.A[j * (j + 1) / 2 + j];
        st.D[j] = d > 0 ? d : 1.0;
    }
    st.mu = 1e-3;
    st.nu = 2;
    st.iter = 0;
    st.status = HBT_FIT_CONVERGED;
    st.stop = 0;
    st.passes = 1;
}

// The next trial point: solve (A + mu D) delta = -g (D: the largest
// diagonal of J^T J seen, Marquardt's scaling), raising mu while the damped
// matrix is not positive definite.  go = 0 when the step no longer moves
// the point, the damping overflowed or the iterations ran out.
__device__ __noinline__ void lm_propose(LmState &st, int max_iter) {
    st.go = 0;
    while (!st.stop) {
        if (st.iter >= max_iter) {
            st.status = HBT_FIT_MAX_ITER;
            return;
        }
        st.iter++;
        double M[21], delta[6], mg[6];
        for (int j = 0; j < 21; j++) M[j] = st.A[j];
        for (int j = 0; j < 6; j++) {
            M[j * (j + 1) / 2 + j] += st.mu * st.D[j];
            mg[j] = -st.g[j];
        }
        if (!cholesky6(M)) {
            st.mu *= st.nu;
            st.nu *= 2;
            st.stop = !(st.mu < 1e300);
            continue;
        }
        chol_solve6(M, mg, delta);
        bool small = true;
        for (int j = 0; j < 6; j++) {
            st.trial[j] = st.x[j] + delta[j];
            if (fabs(delta[j]) > 1e-12 * (fabs(st.x[j]) + 1e-12)) small = false;
        }
        if (small) {
            st.stop = 1;
            return;
        }
        st.go = 1;
        return;
    }
}

// After the pass at the trial point: accept it when chi^2 fell (gain ratio
// rho > 0, Nielsen's update of mu), else raise mu.  Converged when an
// accepted step changed chi^2 by less than 1e-14 of it, predicted and
// actual.
__device__ __noinline__ void lm_update(LmState &st, const double *red) {
    st.passes++;
    const double Sn = red[0];
    double pred = 0;
    for (int j = 0; j < 6; j++) {
        const double dj = st.trial[j] - st.x[j];
        pred += dj * (st.mu * st.D[j] * dj - st.g[j]);
    }
    const double rho = (isfinite(Sn) && pred > 0) ? (st.S - Sn) / pred : -1.0;
    if (rho > 0) {
        const double drop = st.S - Sn;
        for (int j = 0; j < 6; j++) st.x[j] = st.trial[j];
        st.S = Sn;
        for (int j = 0; j < 6; j++) st.g[j] = red[1 + j];
        for (int j = 0; j < 21; j++) st.A[j] = red[7 + j];
        for (int j = 0; j < 6; j++) st.D[j] = fmax(st.D[j], st.A[j * (j + 1) / 2 + j]);
        const double q = 2 * rho - 1;
        st.mu *= fmax(1.0 / 3.0, 1.0 - q * q * q);
        st.nu = 2;
        st.stop = drop <= 1e-14 * st.S && pred <= 1e-14 * st.S;
    } else {
        st.mu *= st.nu;
        st.nu *= 2;
        st.stop = !(st.mu < 1e300);
    }
}

// A fit of a batch: table t, cut k, its n kept rows and its work items
// [item0, item1).
struct FitInfo {
    int t, k, n, item0, item1;
};

// A work item's fit, rows and place: unit w's sums are at
// partial[(kItemUnits slot + w) * kSums].
struct FitItem {
    int fit, rows, slot, pad;
    long long row0;
};

// Per pass of a check interval: the next (item, unit) to take, and whether any fit
// has another trial point.
struct PassCtl {
    int next, active;
};

__global__ void k_fit_init(FitConst fc, const FitInfo *fits, int n_fits, LmState *st) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_fits) return;
    LmState &s = st[f];
    s.done = 0;
    for (int j = 0; j < 6; j++) s.x[j] = s.trial[j] = fc.p0[j];
    s.use_x = 1;
    s.iter = 0;
    s.passes = 0;
    s.stop = 0;
    s.S = NAN;
    const bool enough = fits[f].n >= 6;
    s.go = enough;
    s.status = enough ? HBT_FIT_CONVERGED : HBT_FIT_TOO_FEW;
}

// Sum k of a fit: its items' units' partials in order.  They come from other
// SMs: read past L1.
__device__ __forceinline__ double fit_sum(const FitInfo &fi, const double *partial, int k) {
    double x = 0.0;
    for (int it = fi.item0; it < fi.item1; it++) {
        double y = 0.0;
#pragma unroll
        for (int w = 0; w < kItemUnits; w++)
            y += __ldcg(partial + ((long long)it * kItemUnits + w) * kSums + k);
        x += y;
    }
    return x;
}

// One pass over every active fit's rows: the chi^2, J^T r and J^T J of each
// item's units (at the fit's trial point, its start point on the first pass,
// or with kExact at its minimum for the covariance) into `partial`.
// Blocks take units in turn, the largest first; finished fits' are skipped.
// The block that finishes a fit's last unit of an iterating pass makes its
// Levenberg-Marquardt step, so the fit's state only changes once all its units
// of the pass are done; `active` is set while any fit has another trial point.
//
// Bound by the FP64 pipe (2 lanes a clock and SM): 32 operations a row, 36
// issued with a unit's constants and reduction, the conversions by the integer
// pipe.  The first pass over 64 tables of 41^3 rows, five cuts: 349 us, FP64
// pipe 82 % busy (474 us as a block per item with 39 operations a row); a late
// pass with few active fits 110 us (180 us with a warp per unit); over four
// tables 52 us (168 us).
template <bool kExact>
__global__ void __launch_bounds__(kFitThreads, HBT_FIT_MIN_BLOCKS)
    k_fit_pass(FitConst fc, const FitItem *items, int n_items, Rows rw, const FitInfo *fits,
               LmState *st, double *partial, PassCtl *ctl) {
    __shared__ double etab[EXP_TABLE];
    __shared__ StepBuf buf[2];
    __shared__ double red[kSums];
    __shared__ PassConst pc;
    __shared__ int next, last;
    const int n_units = n_items * kItemUnits;
    // warp 0 takes the next active unit; units of finished fits are passed
    // over up to 32 at a time
    auto take = [&] {
        const int lane = threadIdx.x;
        int u = 0;
        while (true) {
            if (lane == 0) u = atomicAdd(&ctl->next, 1);
            u = __shfl_sync(0xffffffffu, u, 0);
            if (u >= n_units) break;
            bool on = true;  // past the last unit: nothing to pass over
            if (u + lane < n_units) {
                const LmState &s = st[items[(u + lane) / kItemUnits].fit];
                on = kExact ? s.status != HBT_FIT_TOO_FEW : s.go;
            }
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (m & 1u) break;
            if (lane == 0) atomicMax(&ctl->next, u + (m ? __ffs(m) - 1 : 32));
        }
        if (lane == 0) next = u;
    };
    if (threadIdx.x < 32) take();
    fill_exp_table(etab);
    __syncthreads();
    while (next < n_units) {
        const FitItem I = items[next / kItemUnits];
        const int w = next % kItemUnits;
        LmState &s = st[I.fit];
        if (threadIdx.x < 32) {
            // lane k forms parameter k's constants, lane k the factor of sum k:
            // 1 + j carries J's column j, 7 + m the columns of element m
            const int k = threadIdx.x;
            const double pk = k < 6 ? ((kExact || s.use_x) ? s.x[k] : s.trial[k]) : 0.0;
            const double a = pk / kHbarC;
            const double cdf = k ? -2.0 * a / kHbarC : 1.0;
            if (k == 0) pc.lam = pk;
            if (k >= 1 && k < 6) pc.a2[k - 1] = a * a;
            int j = 0;
            while (k >= 7 && (j + 1) * (j + 2) / 2 <= k - 7) j++;
            const int l = k >= 7 ? k - 7 - j * (j + 1) / 2 : 0;
            const double cj = __shfl_sync(0xffffffffu, cdf, k >= 7 ? j : max(k - 1, 0));
            const double cl = __shfl_sync(0xffffffffu, cdf, l);
            if (k < kSums) pc.factor[k] = k >= 7 ? cj * cl : cj;
        }
        __syncthreads();
        fit_unit<kExact>(rw, I.row0, 32 * w, I.rows, pc, etab, buf,
                         partial + ((long long)I.slot * kItemUnits + w) * kSums);
        __threadfence();
        __syncthreads();
        if (!kExact) {
            const FitInfo fi = fits[I.fit];
            if (threadIdx.x == 0)
                last = atomicAdd(&s.done, 1) == (fi.item1 - fi.item0) * kItemUnits - 1;
            __syncthreads();
            if (last) {
                __threadfence();
                if (threadIdx.x < kSums) red[threadIdx.x] = fit_sum(fi, partial, threadIdx.x);
                __syncthreads();
                if (threadIdx.x == 0) {
                    s.done = 0;
                    if (s.use_x) {
                        lm_init(s, red);
                        s.use_x = 0;
                    } else {
                        lm_update(s, red);
                    }
                    lm_propose(s, fc.max_iter);
                    if (s.go) atomicOr(&ctl->active, 1);
                }
            }
        }
        if (threadIdx.x < 32) take();
        __syncthreads();
    }
}

// Results: the point, chi^2, the errors sqrt(diag((J^T J)^-1)) from the
// exact pass at the minimum (inf and the singular status when J^T J is not
// positive definite), rows, iterations, status.  One warp per fit: a lane per
// sum, then a lane per column of the inverse.
__global__ void __launch_bounds__(32) k_fit_finish(FitConst fc, int first_table, const FitInfo *fits, int n_fits,
                             const LmState *st, const double *partial, hbt_fit_result *res,
                             unsigned long long *n_passes) {
    const int f = blockIdx.x, j = threadIdx.x;
    if (f >= n_fits) return;
    const FitInfo fi = fits[f];
    const LmState &s = st[f];
    hbt_fit_result *out = res + (long long)(first_table + fi.t) * fc.n_cuts + fi.k;
    const bool few = s.status == HBT_FIT_TOO_FEW;
    if (j == 0) {
        out->q_cut = fc.cut_sorted[fc.rank[fi.k]];
        out->n_points = fi.n;
        out->iterations = s.iter;
        out->reserved = 0;
        out->chi2 = few ? NAN : s.S;
    }
    if (j < 6) out->p[j] = few ? NAN : s.x[j];
    if (few) {
        if (j < 6) out->err[j] = NAN;
        if (j == 0) out->status = HBT_FIT_TOO_FEW;
        return;
    }
    __shared__ double L[21];
    __shared__ int definite;
    if (j >= 7 && j < kSums) L[j - 7] = fit_sum(fi, partial, j);
    __syncwarp();
    if (j == 0) definite = cholesky6(L);
    __syncwarp();
    if (j < 6) {
        double e[6] = {0, 0, 0, 0, 0, 0}, col[6];
        e[j] = 1.0;
        chol_solve6(L, e, col);
        out->err[j] = definite ? sqrt(col[j]) : INFINITY;
    }
    if (j == 0) {
        out->status = !definite && s.status == HBT_FIT_CONVERGED ? HBT_FIT_SINGULAR : s.status;
        atomicAdd(n_passes, (unsigned long long)s.passes + 1);
    }
}

struct Buf {
    void *p = nullptr;
    size_t bytes = 0;
};

bool grow(Buf &b, size_t bytes) {
    if (b.p && b.bytes >= bytes) return true;
    if (b.p) cudaFree(b.p);
    b.p = nullptr;
    b.bytes = 0;
    if (bytes == 0) return true;
    if (cudaMalloc(&b.p, bytes + bytes / 8) != cudaSuccess) {
        b.p = nullptr;
        return false;
    }
    b.bytes = bytes + bytes / 8;
    return true;
}

// Per batch: at most 32 M table rows (7 doubles and 5 floats each once
// kept) and 256 M doubles of input, which bounds the device memory of a
// call to about 4.5 GB; a batch of 41^3-row tables holds 464 of them.
constexpr long long kBatchRows = 32LL << 20;
constexpr long long kBatchIn = 256LL << 20;
// Iterations launched between two reads of the any-fit-active flag.
constexpr int kStepsPerCheck = 4;

// The cuts on |q| as cuts on its square (FitConst): the square root is
// monotone, so each is the neighbour of the cut's square at which the
// comparison turns.
void set_cut_squares(FitConst &fc) {
    auto bits = [](double v) {
        long long b;
        std::memcpy(&b, &v, sizeof(b));
        return b;
    };
    for (int k = 0; k < fc.n_cuts; k++) {
        const double cut = fc.cut_sorted[k];
        double z = 0.0;  // nothing is below a cut that is 0, negative or NaN
        if (cut > 0.0) {
            z = cut * cut;
            while (std::sqrt(z) < cut) z = std::nextafter(z, HUGE_VAL);
            while (z > 0.0 && !(std::sqrt(std::nextafter(z, 0.0)) < cut)) z = std::nextafter(z, 0.0);
        }
        fc.cut_sq[k] = bits(z);
    }
    const double lo = fc.q_cut_min;
    if (std::isnan(lo)) {
        fc.min_sq = bits(HUGE_VAL);
    } else if (lo < 0.0) {
        fc.min_sq = -1;  // every row is above
    } else {
        double z = lo * lo;
        while (z > 0.0 && std::sqrt(z) > lo) z = std::nextafter(z, 0.0);
        while (std::sqrt(std::nextafter(z, HUGE_VAL)) <= lo && z < HUGE_VAL)
            z = std::nextafter(z, HUGE_VAL);
        fc.min_sq = bits(z);
    }
}

// The input doubles of a table and, for an interleaved one, where its
// block starts: the five columns within one row-major block of n rows.
long long table_span(const hbt_fit_table &T, const double **lo_out) {
    const double *col[5] = {T.q_out, T.q_side, T.q_long, T.C, T.C_err};
    const uintptr_t b0 = reinterpret_cast<uintptr_t>(col[0]);
    uintptr_t lo = b0, hi = b0;
    bool aligned = true;
    for (const double *c : col) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(c);
        lo = std::min(lo, a);
        hi = std::max(hi, a);
        aligned = aligned && (a - b0) % sizeof(double) == 0;
    }
    const long long width = (long long)((hi - lo) / sizeof(double)) + 1;
    if (T.stride > 1 && aligned && width <= T.stride && T.n_rows > 0) {
        *lo_out = reinterpret_cast<const double *>(lo);
        return (T.n_rows - 1) * T.stride + width;
    }
    *lo_out = nullptr;
    return 5 * T.n_rows;
}

}  // namespace

struct hbt_fit_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
    Buf in, rows, frows, tab_off, desc, parts, first, part_cls, cls, fits, items, state, partial,
        res, counter, ctl;
    int sms = 0;
    int *active_host = nullptr;  // pinned
    std::vector<double> packed;
    hbt_fit_stats stats{};
    std::string err;
};

namespace {

hbt_status fit_fail(hbt_fit_ctx *c, hbt_status s, const std::string &m) {
    if (c) c->err = m;
    return s;
}

}  // namespace

extern "C" {

hbt_status hbt_fit_create(int device, hbt_fit_ctx **out) {
    if (!out) return HBT_ERR_INVALID;
    *out = nullptr;
    hbt_fit_ctx *c = new hbt_fit_ctx();
    c->device = device;
    if (cudaSetDevice(device) != cudaSuccess ||
        cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&c->ev[0]) != cudaSuccess || cudaEventCreate(&c->ev[1]) != cudaSuccess ||
        cudaEventCreate(&c->ev[2]) != cudaSuccess || !grow(c->counter, 8) ||
        !grow(c->ctl, (kStepsPerCheck + 1) * sizeof(PassCtl)) ||
        cudaMallocHost(&c->active_host, sizeof(int)) != cudaSuccess) {
        hbt_fit_destroy(c);
        return HBT_ERR_CUDA;
    }
    if (cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        hbt_fit_destroy(c);
        return HBT_ERR_CUDA;
    }
    *out = c;
    return HBT_OK;
}

void hbt_fit_destroy(hbt_fit_ctx *c) {
    if (!c) return;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    for (Buf *b : {&c->in, &c->rows, &c->frows, &c->tab_off, &c->desc, &c->parts, &c->first,
                   &c->part_cls, &c->cls, &c->fits, &c->items, &c->state, &c->partial, &c->res,
                   &c->counter, &c->ctl})
        if (b->p) cudaFree(b->p);
    for (cudaEvent_t e : c->ev)
        if (e) cudaEventDestroy(e);
    if (c->active_host) cudaFreeHost(c->active_host);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
}

const char *hbt_fit_last_error(const hbt_fit_ctx *c) { return c ? c->err.c_str() : "null context"; }

hbt_status hbt_fit_get_stats(const hbt_fit_ctx *c, hbt_fit_stats *out) {
    if (!c || !out) return HBT_ERR_INVALID;
    *out = c->stats;
    return HBT_OK;
}

hbt_status hbt_fit_radii(hbt_fit_ctx *c, int32_t n_tables, const hbt_fit_table *tables,
                         const hbt_fit_options *opt, hbt_fit_result *out) {
    if (!c || n_tables < 0 || (n_tables > 0 && (!tables || !out)) || !opt)
        return HBT_ERR_INVALID;
    if (opt->n_cuts < 1 || opt->n_cuts > kMaxCuts || !opt->q_cut_max)
        return fit_fail(c, HBT_ERR_INVALID, "n_cuts must be 1..16");
    FitConst fc{};
    fc.n_cuts = opt->n_cuts;
    fc.q_cut_min = opt->q_cut_min;
    fc.max_iter = opt->max_iterations > 0 ? opt->max_iterations : 500;
    for (int j = 0; j < 6; j++) fc.p0[j] = opt->p0[j];
    std::vector<int> order(opt->n_cuts);
    for (int k = 0; k < opt->n_cuts; k++) order[k] = k;
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return opt->q_cut_max[a] < opt->q_cut_max[b]; });
    for (int s = 0; s < opt->n_cuts; s++) {
        fc.cut_sorted[s] = opt->q_cut_max[order[s]];
        fc.rank[order[s]] = s;
    }
    set_cut_squares(fc);
    for (int t = 0; t < n_tables; t++) {
        const hbt_fit_table &T = tables[t];
        if (T.n_rows < 0 || T.stride < 1 ||
            (T.n_rows > 0 && (!T.q_out || !T.q_side || !T.q_long || !T.C || !T.C_err)))
            return fit_fail(c, HBT_ERR_INVALID, "table " + std::to_string(t) + " is invalid");
        const double *lo = nullptr;
        if (T.n_rows > kBatchRows || table_span(T, &lo) > kBatchIn)
            return fit_fail(c, HBT_ERR_INVALID, "table larger than a launch's row budget");
    }
    if (cudaSetDevice(c->device) != cudaSuccess) return fit_fail(c, HBT_ERR_CUDA, "cudaSetDevice");
    c->stats = hbt_fit_stats{};
    c->stats.fits = (int64_t)n_tables * opt->n_cuts;
    if (n_tables == 0) return HBT_OK;
    const int nc = opt->n_cuts;
    if (!grow(c->res, (size_t)n_tables * nc * sizeof(hbt_fit_result)))
        return fit_fail(c, HBT_ERR_NOMEM, "device allocation failed");
    cudaStream_t st = c->stream;
    cudaError_t e = cudaMemsetAsync(c->counter.p, 0, 8, st);
    float up_ms = 0.f, fit_ms = 0.f;
    std::vector<long long> off;
    std::vector<TabDesc> desc;
    std::vector<const double *> block;
    std::vector<long long> packed_at;
    std::vector<int> cls_h, first;
    std::vector<SelPart> parts;
    std::vector<FitInfo> fits;
    std::vector<FitItem> items;
    for (int t0 = 0; t0 < n_tables && e == cudaSuccess;) {
        // the batch: tables [t0, t1) within the row and input budgets
        int t1 = t0;
        long long rows = 0, in_total = 0, n_packed = 0;
        off.assign(1, 0);
        desc.clear();
        block.clear();
        parts.clear();
        first.assign(1, 0);
        while (t1 < n_tables) {
            const hbt_fit_table &T = tables[t1];
            const double *lo = nullptr;
            const long long span = table_span(T, &lo);
            if (t1 > t0 && (rows + T.n_rows > kBatchRows || in_total + span > kBatchIn)) break;
            TabDesc d{};
            d.base = in_total;
            if (lo) {
                d.stride = T.stride;
                const double *col[5] = {T.q_out, T.q_side, T.q_long, T.C, T.C_err};
                for (int k = 0; k < 5; k++) d.col[k] = col[k] - lo;
            } else {
                d.stride = 1;
                for (int k = 0; k < 5; k++) d.col[k] = k * T.n_rows;
                n_packed += span;
            }
            desc.push_back(d);
            block.push_back(lo);
            in_total += span;
            rows += T.n_rows;
            off.push_back(rows);
            // a table without rows has one part, which leaves its counts
            const int np = (int)std::max<long long>(1, (T.n_rows + kSelRows - 1) / kSelRows);
            for (int p = 0; p < np; p++) parts.push_back(SelPart{t1 - t0, p});
            first.push_back((int)parts.size());
            t1++;
        }
        const int nt = t1 - t0;
        bool ok = grow(c->tab_off, (nt + 1) * sizeof(long long)) &&
                  grow(c->desc, nt * sizeof(TabDesc)) &&
                  grow(c->cls, (size_t)nt * (nc + 1) * sizeof(int)) &&
                  grow(c->parts, parts.size() * sizeof(SelPart)) &&
                  grow(c->first, first.size() * sizeof(int)) &&
                  grow(c->part_cls, parts.size() * nc * sizeof(int)) &&
                  grow(c->in, in_total * sizeof(double)) &&
                  grow(c->rows, 7 * rows * sizeof(double)) &&
                  grow(c->frows, 5 * rows * sizeof(float));
        if (!ok) return fit_fail(c, HBT_ERR_NOMEM, "device allocation failed");
        // tables that are not one interleaved block are packed on the host
        c->packed.resize((size_t)std::max<long long>(n_packed, 1));
        long long pk = 0;
        packed_at.assign(nt, -1);
        for (int t = t0; t < t1; t++) {
            if (block[t - t0]) continue;
            const hbt_fit_table &T = tables[t];
            const double *col[5] = {T.q_out, T.q_side, T.q_long, T.C, T.C_err};
            packed_at[t - t0] = pk;
            for (int k = 0; k < 5; k++)
                for (long long i = 0; i < T.n_rows; i++) c->packed[pk++] = col[k][i * T.stride];
        }
        double *din = static_cast<double *>(c->in.p);
        Rows rw{static_cast<double *>(c->rows.p), static_cast<float *>(c->frows.p), rows};
        const long long *d_off = static_cast<const long long *>(c->tab_off.p);
        if ((e = cudaEventRecord(c->ev[0], st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(c->tab_off.p, off.data(), off.size() * sizeof(long long),
                                 cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(c->desc.p, desc.data(), desc.size() * sizeof(TabDesc),
                                 cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(c->parts.p, parts.data(), parts.size() * sizeof(SelPart),
                                 cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (e = cudaMemcpyAsync(c->first.p, first.data(), first.size() * sizeof(int),
                                 cudaMemcpyHostToDevice, st)) != cudaSuccess)
            break;
        // all copies first (copies from pageable memory wait for the stream's
        // earlier work, so a kernel between them would serialise them), then
        // the row selection of every table
        for (int t = t0; t < t1 && e == cudaSuccess; t++) {
            const long long span =
                (t + 1 < t1 ? desc[t - t0 + 1].base : in_total) - desc[t - t0].base;
            if (span == 0) continue;
            const double *src = block[t - t0] ? block[t - t0] : c->packed.data() + packed_at[t - t0];
            e = cudaMemcpyAsync(din + desc[t - t0].base, src, span * sizeof(double),
                                cudaMemcpyHostToDevice, st);
        }
        if (e != cudaSuccess) break;
        const TabDesc *d_desc = static_cast<const TabDesc *>(c->desc.p);
        const SelPart *d_parts = static_cast<const SelPart *>(c->parts.p);
        const unsigned sb = (unsigned)parts.size();
        k_fit_count<<<sb, kSelThreads, 0, st>>>(fc, d_off, d_desc, din, d_parts,
                                                static_cast<int *>(c->part_cls.p));
        k_fit_select<<<sb, kSelThreads, 0, st>>>(
            fc, d_off, d_desc, din, d_parts, static_cast<const int *>(c->first.p),
            static_cast<const int *>(c->part_cls.p), rw, static_cast<int *>(c->cls.p));
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        // the fits and their work items, from the selected row counts
        cls_h.resize((size_t)nt * (nc + 1));
        if ((e = cudaMemcpyAsync(cls_h.data(), c->cls.p, cls_h.size() * sizeof(int),
                                 cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
            (e = cudaEventRecord(c->ev[1], st)) != cudaSuccess ||
            (e = cudaStreamSynchronize(st)) != cudaSuccess)
            break;
        fits.clear();
        items.clear();
        int slots = 0;
        for (int t = 0; t < nt; t++) {
            const int f0 = (int)fits.size();
            int most = 0;
            for (int k = 0; k < nc; k++) {
                FitInfo fi{t, k, 0, slots, 0};
                for (int r = 0; r <= fc.rank[k]; r++) fi.n += cls_h[(size_t)t * (nc + 1) + r];
                if (fi.n >= 6) {
                    slots += (fi.n + kItemRows - 1) / kItemRows;
                    most = std::max(most, fi.n);
                }
                fi.item1 = slots;
                fits.push_back(fi);
            }
            for (int r = 0; r < most; r += kItemRows)
                for (int k = 0; k < nc; k++) {
                    const FitInfo &fi = fits[f0 + k];
                    if (fi.n >= 6 && r < fi.n)
                        items.push_back(FitItem{f0 + k, std::min(kItemRows, fi.n - r),
                                                fi.item0 + r / kItemRows, 0, off[t] + r});
                }
        }
        // the largest items first (the blocks take their units in turn); items of the
        // same size stay in row order, so fits that share rows find them in L2
        std::stable_sort(items.begin(), items.end(),
                         [](const FitItem &a, const FitItem &b) { return a.rows > b.rows; });
        const int nf = (int)fits.size(), ni = (int)items.size();
        ok = grow(c->fits, nf * sizeof(FitInfo)) && grow(c->items, std::max(ni, 1) * sizeof(FitItem)) &&
             grow(c->state, nf * sizeof(LmState)) &&
             grow(c->partial, (size_t)std::max(slots, 1) * kItemUnits * kSums * sizeof(double));
        if (!ok) return fit_fail(c, HBT_ERR_NOMEM, "device allocation failed");
        if ((e = cudaMemcpyAsync(c->fits.p, fits.data(), nf * sizeof(FitInfo),
                                 cudaMemcpyHostToDevice, st)) != cudaSuccess ||
            (ni > 0 && (e = cudaMemcpyAsync(c->items.p, items.data(), ni * sizeof(FitItem),
                                            cudaMemcpyHostToDevice, st)) != cudaSuccess))
            break;
        const FitInfo *d_fits = static_cast<const FitInfo *>(c->fits.p);
        const FitItem *d_items = static_cast<const FitItem *>(c->items.p);
        LmState *d_state = static_cast<LmState *>(c->state.p);
        double *d_part = static_cast<double *>(c->partial.p);
        PassCtl *d_ctl = static_cast<PassCtl *>(c->ctl.p);
        // resident pass blocks: with few units two an SM, so that the small
        // units come after the large ones (16 tables of 23^3 rows: 2.15 ms a
        // call against 2.39 ms at four); with many four, which fill the FP64
        // pipe (64 tables of 41^3 rows: 9.4 ms against 9.9 ms at two)
        const int units = ni * kItemUnits;
        const int per_sm = units < 8 * c->sms ? 2 : HBT_FIT_MIN_BLOCKS;
        const unsigned pg = (unsigned)std::max(1, std::min(units, c->sms * per_sm));
        k_fit_init<<<(unsigned)((nf + 127) / 128), 128, 0, st>>>(fc, d_fits, nf, d_state);
        e = cudaGetLastError();
        // Levenberg-Marquardt passes over all active fits' rows, each with
        // the fits' steps; the flag is read every few passes
        for (int done = 0; e == cudaSuccess && ni > 0 && done <= fc.max_iter + 1;
             done += kStepsPerCheck) {
            if ((e = cudaMemsetAsync(d_ctl, 0, kStepsPerCheck * sizeof(PassCtl), st)) !=
                cudaSuccess)
                break;
            for (int r = 0; r < kStepsPerCheck; r++)
                k_fit_pass<false><<<pg, kFitThreads, 0, st>>>(fc, d_items, ni, rw, d_fits,
                                                              d_state, d_part, d_ctl + r);
            e = cudaGetLastError();
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(c->active_host, &d_ctl[kStepsPerCheck - 1].active, sizeof(int),
                                    cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess || *c->active_host == 0) break;
        }
        if (e != cudaSuccess) break;
        // J^T J in FP64 at each minimum, then the results
        if (ni > 0) {
            if ((e = cudaMemsetAsync(d_ctl, 0, sizeof(PassCtl), st)) != cudaSuccess) break;
            k_fit_pass<true><<<pg, kFitThreads, 0, st>>>(fc, d_items, ni, rw, d_fits,
                                                         d_state, d_part, d_ctl);
        }
        k_fit_finish<<<(unsigned)nf, 32, 0, st>>>(fc, t0, d_fits, nf, d_state, d_part,
                                                  static_cast<hbt_fit_result *>(c->res.p),
                                                  static_cast<unsigned long long *>(c->counter.p));
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        if ((e = cudaEventRecord(c->ev[2], st)) != cudaSuccess) break;
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess) break;
        float a = 0.f, b = 0.f;
        cudaEventElapsedTime(&a, c->ev[0], c->ev[1]);
        cudaEventElapsedTime(&b, c->ev[1], c->ev[2]);
        up_ms += a;
        fit_ms += b;
        c->stats.rows += rows;
        t0 = t1;
    }
    if (e != cudaSuccess) {
        cudaStreamSynchronize(st);
        return fit_fail(c, HBT_ERR_CUDA, cudaGetErrorString(e));
    }
    unsigned long long passes = 0;
    if ((e = cudaMemcpyAsync(out, c->res.p, (size_t)n_tables * nc * sizeof(hbt_fit_result),
                             cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaMemcpyAsync(&passes, c->counter.p, 8, cudaMemcpyDeviceToHost, st)) !=
            cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return fit_fail(c, HBT_ERR_CUDA, cudaGetErrorString(e));
    for (long long f = 0; f < (long long)n_tables * nc; f++) c->stats.points += out[f].n_points;
    c->stats.passes = (int64_t)passes;
    c->stats.upload_ms = up_ms;
    c->stats.kernel_ms = fit_ms;
    return HBT_OK;
}

}  // extern "C"
