// Device evaluation of the table-driven FP64 functions and of the
// double-float cos of the pair kernels (include/hbt_check.h).
#include "../../include/hbt_check.h"
#include "hbt_hostmem.h"
#include "hbt_math.cuh"
#include "hbt_tile.cuh"

namespace {

using namespace hbt::tile;

// Double-float cosine: 48 significant bits on the FP32 pipe alone.
//
// Table of cos(k / 64) and sin(k / 64), |k| <= 51, as split pairs
// (cos hi, cos lo, sin hi, sin lo), filled by each CTA of the double-float
// same-event kernels from the FP64 sincos.
constexpr int DF_TABLE_HALF = 51;
constexpr int DF_TABLE = 2 * DF_TABLE_HALF + 1;
__device__ __forceinline__ void fill_df_table(float4 *t) {
    for (int k = threadIdx.x; k < DF_TABLE; k += blockDim.x) {
        double s, c;
        sincos((k - DF_TABLE_HALF) / 64.0, &s, &c);
        const float2 cc = split(c), ss = split(s);
        t[k] = make_float4(cc.x, cc.y, ss.x, ss.y);
    }
}

// cos of a double-float phase, to about 5e-15 absolute (the table's 48-bit
// values), for |ph| < 3200 (|q.dx| / hbarC is a few hundred at most; beyond,
// the FP64 cos).  Cody-Waite reduction by quarter periods x = ph - j pi / 2
// with pi / 2 in four FP32 parts: the first two have 12 significant bits
// (j times them is exact for |j| < 2^11), the third goes through an FMA
// two-product and the fourth is below 2^-57, so x carries about 2^-48
// absolute error; |x| <= pi / 4.  Then the table point t = k / 64 nearest x
// (exact in FP32) and d = x - t, |d| <= 1 / 128:
//   cos(x + j pi / 2) = A cos d + B sin d,
// (A, B) = (C, -S), (-S, -C), (-C, S), (S, C) for j mod 4 = 0..3 with
// C = cos t, S = sin t; cos d - 1 = -d^2 / 2 + d^4 / 24 and
// sin d - d = d^3 (-1 / 6 + d^2 / 120) (truncations below 3.2e-16 and
// 4e-19), the d^2 and d^3 terms in double-float.
__device__ __forceinline__ double df_cos(const float4 *tab, FF ph) {
    const float j = rintf(ph.h * 0.63661977f);  // 2 / pi
    if (!(fabsf(j) < 2048.0f)) return cos((double)ph.h + (double)ph.l);
    const float t1 = __fmaf_rn(-j, 1.57080078125f, ph.h);  // exact
    const FF s1 = two_sum(t1, __fmul_rn(-j, -4.453584551811218e-06f));  // product exact
    const float p3 = __fmul_rn(-j, -8.705515752716053e-10f);
    const float e3 = __fmaf_rn(-j, -8.705515752716053e-10f, -p3);
    const FF s2 = two_sum(s1.h, p3);
    const FF u = two_sum(s2.h, ph.l);
    const float rest = __fadd_rn(__fadd_rn(s1.l, s2.l),
                                 __fadd_rn(e3, __fmul_rn(-j, 5.721188916458728e-18f)));
    const FF x = fast_two_sum(u.h, __fadd_rn(u.l, rest));
    const float k = rintf(x.h * 64.0f);
    const FF dd = two_sum(__fsub_rn(x.h, k * 0.015625f), x.l);  // x.h - k / 64 exact
    const FF d2 = ff_mul(dd, dd);
    const float c4 = __fmul_rn(__fmul_rn(d2.h, d2.h), 1.0f / 24.0f);
    const FF cm = {__fmul_rn(d2.h, -0.5f), __fadd_rn(__fmul_rn(d2.l, -0.5f), c4)};
    // -1 / 6 as a split pair, plus d^2 / 120
    const FF kq = fast_two_sum(-0.1666666716337204f,
                               __fadd_rn(4.967053879312289e-09f, d2.h * (1.0f / 120.0f)));
    const FF sd = ff_add(dd, ff_mul(ff_mul(d2, dd), kq));
    const float4 e = tab[(int)k + DF_TABLE_HALF];
    const int quad = ((int)j) & 3;
    FF A, B;
    if (quad == 0) {
        A = FF{e.x, e.y};
        B = FF{-e.z, -e.w};
    } else if (quad == 1) {
        A = FF{-e.z, -e.w};
        B = FF{-e.x, -e.y};
    } else if (quad == 2) {
        A = FF{-e.x, -e.y};
        B = FF{e.z, e.w};
    } else {
        A = FF{e.z, e.w};
        B = FF{e.x, e.y};
    }
    const FF r = ff_add(A, ff_add(ff_mul(A, cm), ff_mul(B, sd)));
    return (double)r.h + (double)r.l;
}

// df_cos of each argument split into (hi, lo) FP32 parts, as the
// double-float pair kernels split their columns.
__global__ void k_check_dfcos(long long n, const double *x, double *out) {
    __shared__ float4 t[DF_TABLE];
    fill_df_table(t);
    __syncthreads();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float2 s = split(x[i]);
        out[i] = df_cos(t, FF{s.x, s.y});
    }
}

__global__ void k_check_math(int which, CosScale k, long long n, const double *x, double *out) {
    __shared__ double2 cs[COS_TABLE];
    __shared__ double et[EXP_TABLE];
    fill_cos_table(cs);
    fill_exp_table(et);
    __syncthreads();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        double v;
        if (which == HBT_CHECK_COS || which == HBT_CHECK_COS_PHASE)
            v = table_cos(cs, k, x[i]);
        else
            v = table_exp(et, x[i]);
        out[i] = v;
    }
}

}  // namespace

extern "C" hbt_status hbt_check_math(int device, int32_t which, int64_t n, const double *x,
                                     double *out) {
    if (n < 0 || (n > 0 && (!x || !out)) ||
        which < HBT_CHECK_COS || which > HBT_CHECK_COS_PHASE)
        return HBT_ERR_INVALID;
    if (n == 0) return HBT_OK;
    if (cudaSetDevice(device) != cudaSuccess) return HBT_ERR_CUDA;
    double *d = nullptr;
    if (cudaMalloc(&d, 2 * n * sizeof(double)) != cudaSuccess) return HBT_ERR_NOMEM;
    cudaError_t e = cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        const long long blocks = (n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024;
        if (which == HBT_CHECK_DFCOS)
            k_check_dfcos<<<(unsigned)blocks, 256>>>(n, d, d + n);
        else
            k_check_math<<<(unsigned)blocks, 256>>>(
                which, make_cos_scale(which == HBT_CHECK_COS_PHASE ? 1.0 / hbt::kHbarC : 1.0), n,
                d, d + n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + n, n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? HBT_OK : HBT_ERR_CUDA;
}

extern "C" int32_t hbt_check_host_route(const void *p) {
    return static_cast<int32_t>(hbt::host_route(p));
}
