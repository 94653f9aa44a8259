// Balance-function pair binning (include/hbt_bf.h).
//
// One CTA per event pair (job) and 128 particles of list A, in registers (one
// per thread); those of list B are staged through shared memory 256 at a time.
// Every pair is binned in FP32 with rigorous error bounds (decide); the pairs
// within those bounds of a bin edge or a cut run the reference's FP64
// expressions (bin_slow, src/BalanceFunction.cpp:136-160 and :183-204; this unit
// is compiled with --fmad=false), so every bin is the reference's.  Counts go to
// a shared-memory histogram of Bnpts x 40 (columns c and c + 20 are one bin),
// whose non-zero bins are added to the global histogram when the item is
// done.  The bins are few and every pair lands in one, so privatising the
// histogram in shared memory turns the pair rate's worth of global atomics
// into one per non-zero bin and job.
#include <algorithm>
#include <cmath>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/hbt_bf.h"
#include "hbt_engine.cuh"
#include "hbt_hostmem.h"
#include "hbt_screen.cuh"

namespace {

using hbt::tile::add2;
using hbt::tile::f2;
using hbt::tile::fma2;
using hbt::tile::pack2;
using hbt::tile::unpack2;

constexpr int kTile = 128;
#ifndef HBT_BF_STAGE
#define HBT_BF_STAGE 256
#endif
constexpr int kStage = HBT_BF_STAGE;  // particles of list B staged at a time
constexpr int kGroup = 4;  // pairs of a thread between two branches
constexpr int kNphi = HBT_BF_NPHI;
// bytes of the largest shared-memory histogram (Bnpts x 40 counts)
constexpr int kMaxSharedHist = 96 * 1024;

// Resident CTAs per SM the kernel is compiled for (register budget).
#ifndef HBT_BF_MIN_BLOCKS
#define HBT_BF_MIN_BLOCKS 8
#endif

// A job with its particle ranges resolved in the concatenated arrays.
struct BfJob {
    long long a0, a1, b0, b1;
    double rotation;
    int hist, mixed;
};

// The reference's binning constants (src/BalanceFunction.cpp:29-35) and
// the reciprocals the screen multiplies by.
struct BfConst {
    double drap, Brap_min, dphi, Bphi_min;
    double inv_drap, inv_dphi;
    double phi0;  // -Bphi_min / dphi, in [0, 20)
    int Bnpts;
};

// The reference's FP64 binning of one pair (src/BalanceFunction.cpp
// :183-204; the same-event loop :136-157 has no rotation term, and adding
// a zero rotation changes no value): the flat bin, or -1 when skipped.
__device__ __forceinline__ int bin64(const BfConst &c, double pa, double ya, double pb, double yb,
                                     int mixed, double rot) {
    const double d = mixed ? (pa - pb) + rot : pa - pb;
    int ip = static_cast<int>(floor((d - c.Bphi_min) / c.dphi)) % kNphi;
    if (ip < 0) ip += kNphi;
    const double dy = ya - yb;
    if (fabs(dy) < 1e-10) return -1;
    if (dy < c.Brap_min) return -1;
    const int iy = static_cast<int>((dy - c.Brap_min) / c.drap);
    if (iy >= 0 && iy < c.Bnpts) return iy * kNphi + ip;
    return -1;
}

// A pair the FP32 screen leaves undecided, from the particles' FP64 values
// in global memory: equal rapidities (a particle with itself, when the two
// lists hold the same species) give dy = 0, which the reference skips;
// everything else runs the reference's expressions.  Out of line: it runs
// for about one pair in a thousand and keeps the loop's registers free.
__device__ __noinline__ int bin_slow(const BfConst &c, const double *phi, const double *y,
                                     long long ia, long long ib, int mixed, double rot) {
    const double ya = y[ia], yb = y[ib];
    if (ya == yb && fabs(ya) < INFINITY) return -1;
    return bin64(c, phi[ia], ya, phi[ib], yb, mixed, rot);
}

// The screen.  A pair's bins are the floors of two quotients,
//   T_phi = (phi_a - phi_b + rot - Bphi_min) / dphi   (taken mod 20),
//   T_y   = (y_a - y_b - Brap_min) / drap              (T_y < 0 is the
//           reference's dy < Brap_min cut),
// each the difference of a term of particle a and a term of particle b.
// The terms are computed once per particle and call in FP64, the phi terms
// reduced mod 20 into [0, 20) (particle a's without the rotation, which a job
// adds to it in two floats), and rounded to FP32 (error <= u |term|, u =
// 2^-24), so a pair costs one FP32 subtraction per quotient (error <= u
// (|term a| + |term b|)).  Each term carries a bound: 2.0001 u |term| for
// those roundings, 2^-46 times the magnitudes it was made of for the FP64
// arithmetic here and in the reference's own quotient (and, 120 units of it,
// for the two floats), and on particle a 2e-7 for the FP32 rounding of 0.5 -
// bound.  When the fraction of both FP32 differences clears the summed
// bounds, their floors are the reference's.  A term of magnitude >= 5e8 (or
// NaN) becomes NaN: every pair of that particle then fails the screen and
// takes the FP64 path.
constexpr double kU64 = 0x1p-24;
constexpr float kU = 0x1p-24f;
constexpr double kTermMax = 5e8;

__device__ __forceinline__ double wrap20(double x) {
    double r = x - 20.0 * floor(x * 0.05);
    if (r < 0.0) r += 20.0;
    if (r >= 20.0) r -= 20.0;
    return r;
}

// Particle b's terms, negated (the pair loop adds): the terms of phi / dphi
// and y / drap, and their bounds.
__device__ __forceinline__ float4 terms_b(const BfConst &c, double wp, double xp, double xy) {
    if (!(fabs(xp) < kTermMax && fabs(xy) < kTermMax)) return make_float4(NAN, NAN, 0.f, 0.f);
    const float tp = (float)wp, ty = (float)xy;
    const float ep = (float)(2.0001 * kU64 * fabs((double)tp) + 0x1p-46 * (fabs(xp) + 40.0));
    const float ey = (float)(2.0001 * kU64 * fabs((double)ty) + 0x1p-46 * fabs(xy));
    return make_float4(-tp, -ty, -ep, -ey);
}

// Particle a's terms: of (phi - Bphi_min) / dphi, wrapped, in two floats (the
// job's rotation and 19.5 come on top, a_terms), then of (y - Brap_min) / drap
// less 0.5 (the shifts make rint of a pair's difference the floor of the
// unshifted one, plus 20 for the azimuth: a column in [0, 40) of a histogram
// whose columns c and c + 20 are the same bin), then the parts of the bounds:
// the azimuth's without 2 u |term|, and 0.5 - bound of the rapidity's.
struct TermsA {
    float ph, pl, ty, ep, gy, pad;
};
__device__ __forceinline__ TermsA terms_a(const BfConst &c, double wp, double xp, double y) {
    const double cp = c.Bphi_min * c.inv_dphi, xy = (y - c.Brap_min) * c.inv_drap;
    const double my = (fabs(y) + fabs(c.Brap_min)) * c.inv_drap;
    TermsA t = {NAN, 0.f, NAN, 0.f, 0.f, 0.f};
    if (!(fabs(xp) < kTermMax && fabs(xy) < kTermMax)) return t;
    double s = wp + c.phi0;
    if (s >= 20.0) s -= 20.0;
    t.ph = (float)s;
    t.pl = (float)(s - (double)t.ph);
    t.ty = (float)(xy - 0.5);
    t.ep = (float)(0x1p-46 * (fabs(xp) + fabs(cp) + 200.0) + 2e-7);
    t.gy = (float)(0.5 - (2.0001 * kU64 * fabs((double)t.ty) + 0x1p-46 * (my + 1.0) + 2e-7));
    return t;
}

// A job's rotation as the terms take it: wrapped, in two floats, and its part
// of the bound.
struct Rotation {
    float h, l, e;
};
__device__ __forceinline__ Rotation rotation_of(const BfConst &c, double rot) {
    const double x = rot * c.inv_dphi;
    if (!(fabs(x) < kTermMax)) return Rotation{NAN, 0.f, 0.f};
    const double w = wrap20(x);
    const float h = (float)w;
    return Rotation{h, (float)(w - (double)h), (float)(0x1p-46 * (fabs(x) + 1.0))};
}

// The |dy| < 1e-10 cut: |dy| from FP32 copies errs by at most u (|y_a| +
// |y_b| + |dy|); the pair certainly passes when |dy| exceeds 7 u per
// magnitude plus 1.0001e-10 (1e-10f itself rounds above 1e-10).
__device__ __forceinline__ float2 dy_terms(double y, float slack) {
    const float fy = (float)y;
    return make_float2(fy, 7.0f * kU * fabsf(fy) + slack);
}

// Particle a in a job, as the pair loop uses it: {t_phi, t_y}, {0.5 - bound of
// each}, {y, slack}.
struct ParticleA {
    f2 t, g, y;
};
__device__ __forceinline__ ParticleA a_terms(const TermsA &a, const float2 &yb,
                                             const Rotation &r) {
    // (ph + pl) + (h + l) + 19.5, less 20 from 20 on; two_sum each
    auto two_sum = [](float x, float y, float &err) {
        const float s = __fadd_rn(x, y), v = __fsub_rn(s, x);
        err = __fadd_rn(__fsub_rn(x, __fsub_rn(s, v)), __fsub_rn(y, v));
        return s;
    };
    float e1, e2;
    float s = two_sum(a.ph, r.h, e1);
    const float low = __fadd_rn(e1, __fadd_rn(a.pl, r.l));
    s = two_sum(s, s >= 20.f ? -0.5f : 19.5f, e2);
    const float tp = __fadd_rn(s, __fadd_rn(e2, low));
    const float ep = __fmaf_rn(2.0002f * kU, fabsf(tp), __fadd_rn(a.ep, r.e));
    return ParticleA{pack2(tp, a.ty), pack2(0.5f - ep, a.gy), pack2(yb.x, yb.y + 1.0001e-10f)};
}

// Every particle's terms, once per call: a dozen FP64 operations and the
// conversions a particle, which a job's every block made again before (57 us
// of FP64 for 1,600 jobs of 385 x 385 particles).
__global__ void k_bf_terms(long long n, const double *phi, const double *y, BfConst c,
                           float4 *tb, float2 *yb, TermsA *ta) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const double p = phi[i], yi = y[i], xp = p * c.inv_dphi;
        const double wp = wrap20(xp);
        tb[i] = terms_b(c, wp, xp, yi * c.inv_drap);
        ta[i] = terms_a(c, wp, xp, yi);
        const float2 d = dy_terms(yi, 0.f);
        yb[i] = make_float2(-d.x, d.y);
    }
}

// A pair's place in the shared histogram, and whether the screen is sure of it.
struct Decision {
    unsigned k;
    bool sure;
};
__device__ __forceinline__ Decision decide(const ParticleA &A, const float4 &B, const float2 &By) {
    constexpr float kMagic = 12582912.0f;  // 1.5 2^23
    constexpr unsigned kOff = 0x4b400000u * (2u * kNphi + 1u);
    // shifted differences: rint gives the floors (the azimuth + 20); certain
    // when their distance to the rint is below 0.5 - bound (which also keeps
    // |t| below 2^22)
    const f2 t = add2(A.t, pack2(B.x, B.y)), g = add2(A.g, pack2(B.z, B.w));
    const f2 m = add2(t, pack2(kMagic, kMagic));
    const f2 r = fma2(add2(m, pack2(-kMagic, -kMagic)), pack2(-1.f, -1.f), t);
    const f2 dy = add2(A.y, pack2(By.x, By.y));
    float mp, my, rp, ry, gp, gy, d, dmin;
    unpack2(m, mp, my);
    unpack2(r, rp, ry);
    unpack2(g, gp, gy);
    unpack2(dy, d, dmin);
    // t_phi in (-0.5, 39.5): column in [0, 39]; a row beyond [0, Bnpts) puts k
    // outside the histogram
    return Decision{__float_as_uint(my) * (2u * kNphi) + __float_as_uint(mp) - kOff,
                    bool((fabsf(rp) < gp) & (fabsf(ry) < gy) & (fabsf(d) > dmin))};
}

// Adds one to word k of the histogram at `at` when k < n, without a branch.
__device__ __forceinline__ void count_one(unsigned at, unsigned k, unsigned n) {
    asm volatile(
        "{\n .reg .pred p;\n setp.lt.u32 p, %0, %1;\n @p red.shared.add.u32 [%2], 1;\n}" ::"r"(k),
        "r"(n), "r"(at + 4u * k)
        : "memory");
}

// One work item per (job, tile of up to 128 particles of list A): a job of
// n_a particles is ceil(n_a / 128) items, so the grid holds several waves
// of similar items instead of one CTA per event pair.  A's terms sit in
// registers (one particle per thread), B's are staged through shared memory
// 256 at a time; the histogram is privatised in shared memory and its
// non-zero bins are added to the global one when the item is done.
//
// A pair costs two broadcast reads, six packed FP32 operations (rint by the
// addition of 1.5 2^23, whose low bits then are the bin), three comparisons
// and the shared-memory addition; four pairs share a branch for those the
// screen leaves open.  Bound by the issue of some 28 instructions a pair (62 %
// of the slots) next to the shared-memory pipe (58 %): 160 million pairs of
// 1,600 jobs in 188 us, 273 us with scalar operations, rint and a branch a
// pair.
__global__ void __launch_bounds__(kTile, HBT_BF_MIN_BLOCKS)
    k_bf(const BfJob *jobs, const int2 *items, long long n_items, const double *phi,
         const double *y, const float4 *tb, const float2 *yb, const TermsA *ta, BfConst c,
         unsigned long long *hist, unsigned long long *n_slow) {
    extern __shared__ unsigned sh[];  // [Bnpts][2 kNphi]: columns c and c + 20 are bin c
    __shared__ float4 sb[kStage];
    __shared__ float2 sd[kStage];
    __shared__ BfJob sj;
    __shared__ Rotation rot;
    const int nbins = c.Bnpts * kNphi, nsh = 2 * nbins;
    const unsigned sh_at = (unsigned)__cvta_generic_to_shared(sh);
    unsigned slow = 0;
    for (long long it = blockIdx.x; it < n_items; it += gridDim.x) {
        const int2 item = items[it];
        for (int k = threadIdx.x; k < nsh; k += blockDim.x) sh[k] = 0u;
        if (threadIdx.x == 0) {
            sj = jobs[item.x];
            rot = rotation_of(c, sj.mixed ? sj.rotation : 0.0);
        }
        __syncthreads();
        const long long ia = sj.a0 + item.y + threadIdx.x;
        const bool have = ia < sj.a1;
        ParticleA A = {};
        bool self_skips = false;
        if (have) {
            const float2 ya = yb[ia];
            A = a_terms(ta[ia], make_float2(-ya.x, ya.y), rot);
            self_skips = fabsf(ya.x) < INFINITY;
        }
        for (long long b = sj.b0; b < sj.b1; b += kStage) {
            // past the end: terms that leave every pair undecided
            for (int k = threadIdx.x; k < kStage; k += kTile) {
                const bool in = b + k < sj.b1;
                sb[k] = in ? tb[b + k] : make_float4(NAN, NAN, 0.f, 0.f);
                sd[k] = in ? yb[b + k] : make_float2(0.f, 0.f);
            }
            __syncthreads();
            const int nb = (int)min((long long)kStage, sj.b1 - b);
            if (have) {
                for (int j = 0; j < nb; j += kGroup) {
                    unsigned k[kGroup];
                    bool sure = true;
#pragma unroll
                    for (int q = 0; q < kGroup; q++) {
                        const Decision s = decide(A, sb[j + q], sd[j + q]);
                        k[q] = s.k;
                        sure = sure & s.sure;
                    }
                    if (!sure) {
#pragma unroll 1
                        for (int q = 0; q < kGroup; q++) {
                            if (decide(A, sb[j + q], sd[j + q]).sure) continue;
                            int f = -1;
                            if (j + q < nb) {
                                slow++;
                                // a particle with itself: dy = 0, skipped
                                if (!(ia == b + j + q && self_skips))
                                    f = bin_slow(c, phi, y, ia, b + j + q, sj.mixed, sj.rotation);
                            }
                            const unsigned to =
                                f < 0 ? ~0u : (unsigned)((f / kNphi) * (2 * kNphi) + f % kNphi);
#pragma unroll
                            for (int p = 0; p < kGroup; p++)
                                if (p == q) k[p] = to;
                        }
                    }
#pragma unroll
                    for (int q = 0; q < kGroup; q++)
                        count_one(sh_at, k[q], (unsigned)nsh);
                }
            }
            __syncthreads();
        }
        unsigned long long *h = hist + (long long)sj.hist * nbins;
        for (int k = threadIdx.x; k < nbins; k += blockDim.x) {
            const int r = k / kNphi, col = k - r * kNphi;
            const unsigned v = sh[r * 2 * kNphi + col] + sh[r * 2 * kNphi + col + kNphi];
            if (v) atomicAdd(h + k, (unsigned long long)v);
        }
        __syncthreads();
    }
    for (int o = 16; o > 0; o >>= 1) slow += __shfl_xor_sync(0xffffffffu, slow, o);
    if ((threadIdx.x & 31) == 0 && slow) atomicAdd(n_slow, (unsigned long long)slow);
}

// A histogram as doubles, to memory the GPU writes (host memory too).
__global__ void k_bf_export(const unsigned long long *h, int n, double *out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) out[k] = (double)h[k];
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

}  // namespace

struct hbt_bf_ctx {
    hbt_bf_params p;
    int device = 0;
    cudaStream_t stream = nullptr;
    BfConst c;
    Buf hist, jobs, items, phi, y, tb, yb, ta, counter;
    bool reads_host = false;  // the GPU reads and writes pageable host memory
    std::vector<hbt::CopySeg> segs;
    cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
    hbt_bf_stats stats{};
    std::string err;
};

namespace {

hbt_status bf_fail(hbt_bf_ctx *c, hbt_status s, const std::string &m) {
    if (c) c->err = m;
    return s;
}

}  // namespace

extern "C" {

hbt_status hbt_bf_create(const hbt_bf_params *p, int device, hbt_bf_ctx **out) {
    if (!p || !out) return HBT_ERR_INVALID;
    *out = nullptr;
    if (p->Bnpts < 2 || p->Bnpts > kMaxSharedHist / (2 * kNphi * (int)sizeof(unsigned)))
        return HBT_ERR_INVALID;
    hbt_bf_ctx *c = new hbt_bf_ctx();
    c->p = *p;
    c->device = device;
    // the reference's expressions (src/BalanceFunction.cpp:29-35)
    c->c.drap = 2. * std::abs(p->Brap_max) / (p->Bnpts - 1);
    c->c.Brap_min = -std::abs(p->Brap_max) - 0.5 * c->c.drap;
    c->c.dphi = 2. * M_PI / kNphi;
    c->c.Bphi_min = -M_PI / 2.;
    c->c.Bnpts = p->Bnpts;
    c->c.inv_drap = 1.0 / c->c.drap;
    c->c.inv_dphi = 1.0 / c->c.dphi;
    const double x0 = -c->c.Bphi_min * c->c.inv_dphi;
    c->c.phi0 = x0 - 20.0 * std::floor(x0 * 0.05);
    if (cudaSetDevice(device) != cudaSuccess ||
        cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&c->ev[0]) != cudaSuccess || cudaEventCreate(&c->ev[1]) != cudaSuccess ||
        cudaEventCreate(&c->ev[2]) != cudaSuccess ||
        !grow(c->hist, (size_t)8 * p->Bnpts * kNphi * sizeof(unsigned long long)) ||
        !grow(c->counter, sizeof(unsigned long long)) ||
        // the same for every context: the limit is the kernel's, not a launch's
        cudaFuncSetAttribute(k_bf, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSharedHist) !=
            cudaSuccess) {
        hbt_bf_destroy(c);
        return HBT_ERR_CUDA;
    }
    int pageable = 0, tables = 0;
    cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, device);
    cudaDeviceGetAttribute(&tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables, device);
    c->reads_host = pageable && tables;
    const hbt_status s = hbt_bf_reset(c);
    if (s != HBT_OK) {
        hbt_bf_destroy(c);
        return s;
    }
    *out = c;
    return HBT_OK;
}

void hbt_bf_destroy(hbt_bf_ctx *c) {
    if (!c) return;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    for (Buf *b : {&c->hist, &c->jobs, &c->items, &c->phi, &c->y, &c->tb, &c->yb, &c->ta, &c->counter})
        if (b->p) cudaFree(b->p);
    for (cudaEvent_t e : c->ev)
        if (e) cudaEventDestroy(e);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
}

const char *hbt_bf_last_error(const hbt_bf_ctx *c) { return c ? c->err.c_str() : "null context"; }

hbt_status hbt_bf_reset(hbt_bf_ctx *c) {
    if (!c) return HBT_ERR_INVALID;
    if (cudaSetDevice(c->device) != cudaSuccess ||
        cudaMemsetAsync(c->hist.p, 0, (size_t)8 * c->p.Bnpts * kNphi * 8, c->stream) != cudaSuccess)
        return bf_fail(c, HBT_ERR_CUDA, "clearing the histograms failed");
    return HBT_OK;
}

hbt_status hbt_bf_bin(hbt_bf_ctx *c, int32_t n_lists, const hbt_bf_list *lists, int32_t n_jobs,
                      const hbt_bf_job *jobs) {
    if (!c || n_lists < 0 || n_jobs < 0 || (n_lists > 0 && !lists) || (n_jobs > 0 && !jobs))
        return HBT_ERR_INVALID;
    if (n_jobs == 0) return HBT_OK;
    if (cudaSetDevice(c->device) != cudaSuccess) return bf_fail(c, HBT_ERR_CUDA, "cudaSetDevice");
    // concatenate the lists (a list passed again with the same arrays, as the
    // mixed-event pool is when it is the buffer itself, shares the first
    // copy), resolve every job's particle ranges
    std::vector<long long> base(n_lists, 0);
    std::vector<int> copy_of(n_lists, -1);
    std::map<std::tuple<const void *, const void *, const void *, int32_t>, int> first;
    long long total = 0;
    for (int l = 0; l < n_lists; l++) {
        const hbt_bf_list &L = lists[l];
        if (L.n_events < 0 || (L.n_events > 0 && !L.offsets))
            return bf_fail(c, HBT_ERR_INVALID, "list without offsets");
        const long long n = L.n_events > 0 ? L.offsets[L.n_events] : 0;
        if (n > 0 && (!L.phi || !L.y)) return bf_fail(c, HBT_ERR_INVALID, "list without columns");
        const auto key = std::make_tuple(static_cast<const void *>(L.offsets),
                                         static_cast<const void *>(L.phi),
                                         static_cast<const void *>(L.y), L.n_events);
        const auto seen = first.emplace(key, l);
        if (!seen.second) copy_of[l] = seen.first->second;
        if (copy_of[l] >= 0) {
            base[l] = base[copy_of[l]];
        } else {
            base[l] = total;
            total += n;
        }
    }
    long long pairs = 0;
    std::vector<BfJob> dj(n_jobs);
    for (int k = 0; k < n_jobs; k++) {
        const hbt_bf_job &J = jobs[k];
        if (J.hist < 0 || J.hist > 7 || J.la < 0 || J.la >= n_lists || J.lb < 0 ||
            J.lb >= n_lists || J.ea < 0 || J.ea >= lists[J.la].n_events || J.eb < 0 ||
            J.eb >= lists[J.lb].n_events)
            return bf_fail(c, HBT_ERR_INVALID, "job out of range");
        const int64_t *oa = lists[J.la].offsets, *ob = lists[J.lb].offsets;
        dj[k] = BfJob{base[J.la] + oa[J.ea], base[J.la] + oa[J.ea + 1], base[J.lb] + ob[J.eb],
                      base[J.lb] + ob[J.eb + 1], J.rotation, J.hist, J.mixed ? 1 : 0};
        pairs += (oa[J.ea + 1] - oa[J.ea]) * (ob[J.eb + 1] - ob[J.eb]);
    }
    std::vector<int2> items;
    for (int k = 0; k < n_jobs; k++)
        if (dj[k].b1 > dj[k].b0)
            for (long long a = 0; a < dj[k].a1 - dj[k].a0; a += kTile)
                items.push_back(make_int2(k, (int)a));
    if (items.empty()) {
        c->stats = hbt_bf_stats{};
        return HBT_OK;
    }
    if (!grow(c->jobs, dj.size() * sizeof(BfJob)) || !grow(c->items, items.size() * sizeof(int2)) ||
        !grow(c->phi, total * sizeof(double)) || !grow(c->y, total * sizeof(double)) ||
        !grow(c->tb, total * sizeof(float4)) || !grow(c->yb, total * sizeof(float2)) ||
        !grow(c->ta, total * sizeof(TermsA)))
        return bf_fail(c, HBT_ERR_NOMEM, "device allocation failed");
    cudaError_t e = cudaEventRecord(c->ev[0], c->stream);
    // where the GPU reads host memory itself, one kernel takes everything
    c->segs.clear();
    auto copy = [&](void *dst, const void *src, long long n_doubles) {
        if (e != cudaSuccess) return;
        if (!c->reads_host || hbt::host_route(src) != hbt::HostRoute::kKernel) {
            e = cudaMemcpyAsync(dst, src, n_doubles * sizeof(double), cudaMemcpyHostToDevice,
                                c->stream);
            return;
        }
        double *to = static_cast<double *>(dst);
        const double *from = static_cast<const double *>(src);
        // a bad pointer fails here, on the host
        const volatile char *v = static_cast<const volatile char *>(src);
        (void)v[0];
        (void)v[n_doubles * sizeof(double) - 1];
        for (long long k = 0; k < n_doubles; k += hbt::kCopyInChunk)
            c->segs.push_back(
                hbt::CopySeg{from + k, to + k, std::min(hbt::kCopyInChunk, n_doubles - k)});
    };
    static_assert(sizeof(BfJob) % 8 == 0 && sizeof(int2) == 8, "copied as doubles");
    copy(c->jobs.p, dj.data(), (long long)(dj.size() * sizeof(BfJob) / 8));
    copy(c->items.p, items.data(), (long long)items.size());
    if (e == cudaSuccess)
        e = cudaMemsetAsync(c->counter.p, 0, sizeof(unsigned long long), c->stream);
    for (int l = 0; l < n_lists; l++) {
        const long long n = lists[l].n_events > 0 ? lists[l].offsets[lists[l].n_events] : 0;
        if (n == 0 || copy_of[l] >= 0) continue;
        copy(static_cast<double *>(c->phi.p) + base[l], lists[l].phi, n);
        copy(static_cast<double *>(c->y.p) + base[l], lists[l].y, n);
    }
    if (e == cudaSuccess)
        e = hbt::launch_copy_in(c->segs.data(), (int)c->segs.size(), c->stream);
    if (e == cudaSuccess) e = cudaEventRecord(c->ev[1], c->stream);
    // a copy that was queued reads the host arrays: wait before giving up
    auto give_up = [&](const std::string &m) {
        cudaStreamSynchronize(c->stream);
        return bf_fail(c, HBT_ERR_CUDA, m);
    };
    if (e != cudaSuccess) return give_up("upload failed");
    const double *dphi_p = static_cast<const double *>(c->phi.p);
    const double *dy_p = static_cast<const double *>(c->y.p);
    if (total > 0)
        k_bf_terms<<<(unsigned)std::min<long long>((total + 255) / 256, 152LL * 16), 256, 0,
                     c->stream>>>(total, dphi_p, dy_p, c->c, static_cast<float4 *>(c->tb.p),
                                  static_cast<float2 *>(c->yb.p),
                                  static_cast<TermsA *>(c->ta.p));
    const long long n_items = (long long)items.size();
    const long long grid = std::min<long long>(n_items, 1LL << 30);
    k_bf<<<(unsigned)grid, kTile, (size_t)c->p.Bnpts * 2 * kNphi * sizeof(unsigned), c->stream>>>(
        static_cast<const BfJob *>(c->jobs.p), static_cast<const int2 *>(c->items.p), n_items,
        dphi_p, dy_p, static_cast<const float4 *>(c->tb.p), static_cast<const float2 *>(c->yb.p),
        static_cast<const TermsA *>(c->ta.p), c->c, static_cast<unsigned long long *>(c->hist.p),
        static_cast<unsigned long long *>(c->counter.p));
    if ((e = cudaGetLastError()) != cudaSuccess)
        return give_up(std::string("k_bf: ") + cudaGetErrorString(e));
    unsigned long long slow = 0;
    if ((e = cudaEventRecord(c->ev[2], c->stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(&slow, c->counter.p, sizeof slow, cudaMemcpyDeviceToHost,
                             c->stream)) != cudaSuccess)
        return bf_fail(c, HBT_ERR_CUDA, cudaGetErrorString(e));
    // the host arrays may be reused once the copies are done
    if ((e = cudaStreamSynchronize(c->stream)) != cudaSuccess)
        return bf_fail(c, HBT_ERR_CUDA, cudaGetErrorString(e));
    float up = 0.f, ker = 0.f;
    cudaEventElapsedTime(&up, c->ev[0], c->ev[1]);
    cudaEventElapsedTime(&ker, c->ev[1], c->ev[2]);
    c->stats.pairs = pairs;
    c->stats.bytes_uploaded = (int64_t)(dj.size() * sizeof(BfJob) + items.size() * sizeof(int2) +
                                        2 * total * sizeof(double));
    c->stats.fp64_pairs = (int64_t)slow;
    c->stats.upload_ms = up;
    c->stats.kernel_ms = ker;
    return HBT_OK;
}

hbt_status hbt_bf_get_stats(const hbt_bf_ctx *c, hbt_bf_stats *out) {
    if (!c || !out) return HBT_ERR_INVALID;
    *out = c->stats;
    return HBT_OK;
}

hbt_status hbt_bf_read(hbt_bf_ctx *c, int32_t hist, double *out) {
    if (!c || hist < 0 || hist > 7 || !out) return HBT_ERR_INVALID;
    const size_t nb = (size_t)c->p.Bnpts * kNphi;
    if (cudaSetDevice(c->device) != cudaSuccess) return bf_fail(c, HBT_ERR_CUDA, "cudaSetDevice");
    if (c->reads_host && hbt::host_route(out) == hbt::HostRoute::kKernel) {
        // the host maps the pages, one kernel writes them
        for (size_t k = 0; k < nb; k += 512) static_cast<volatile double *>(out)[k] = 0.0;
        static_cast<volatile double *>(out)[nb - 1] = 0.0;
        k_bf_export<<<(unsigned)((nb + 255) / 256), 256, 0, c->stream>>>(
            static_cast<unsigned long long *>(c->hist.p) + hist * nb, (int)nb, out);
        if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(c->stream) != cudaSuccess)
            return bf_fail(c, HBT_ERR_CUDA, "reading the histogram failed");
        return HBT_OK;
    }
    std::vector<unsigned long long> v(nb);
    if (
        cudaMemcpyAsync(v.data(), static_cast<unsigned long long *>(c->hist.p) + hist * nb,
                        nb * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                        c->stream) != cudaSuccess ||
        cudaStreamSynchronize(c->stream) != cudaSuccess)
        return bf_fail(c, HBT_ERR_CUDA, "reading the histogram failed");
    for (size_t k = 0; k < nb; k++) out[k] = (double)v[k];
    return HBT_OK;
}

}  // extern "C"
