// Device evaluation of the kernels' table-driven FP64 functions
// (include/hbt_check.h).
#include "../../include/hbt_check.h"
#include "hbt_hostmem.h"
#include "hbt_internal.h"
#include "hbt_math.cuh"
#include "hbt_tile.cuh"

namespace {

// table: cos_entries.
__global__ void k_check_math(int which, CosScale k, const double *table, long long n,
                             const double *x, double *out) {
    __shared__ double cs[kCosEntries];
    __shared__ double et[EXP_TABLE];
    for (int e = threadIdx.x; e < kCosEntries; e += blockDim.x) cs[e] = table[e];
    fill_exp_table(et);
    __syncthreads();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        double v = x[i];
        if (which == HBT_CHECK_DFCOS) {
            const float2 s = hbt::tile::split(v);
            v = (double)s.x + (double)s.y;
        }
        out[i] = which == HBT_CHECK_EXP ? table_exp(et, v) : table_cos(cs, k, v);
    }
}

// cos_fixed of hh 2^-37 + hl 2^-67 steps of 2 pi / 512, in: n pairs (hh, hl).
__global__ void k_check_cos_fixed(hbt::Grid g, const double *table, long long n,
                                  const long long *in, double *out) {
    __shared__ double cs[kCosEntries];
    for (int e = threadIdx.x; e < kCosEntries; e += blockDim.x) cs[e] = table[e];
    __syncthreads();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = hbt::tile::cos_fixed(g, cs, in[2 * i], (unsigned)in[2 * i + 1]);
}

}  // namespace

extern "C" hbt_status hbt_check_cos_fixed(int device, int64_t n, const int64_t *steps, double *out) {
    if (n < 0 || (n > 0 && (!steps || !out))) return HBT_ERR_INVALID;
    if (n == 0) return HBT_OK;
    hbt_params p = {};
    p.qnpts = 11;
    p.q_min = -0.1;
    p.q_max = 0.1;
    p.n_KT = 2;
    p.KT_max = 1.0;
    p.n_Kphi = 1;
    hbt::Grid g;
    hbt::grid_from_params(p, g);
    double table[kCosEntries];
    cos_entries(table);
    if (cudaSetDevice(device) != cudaSuccess) return HBT_ERR_CUDA;
    const size_t in_bytes = (size_t)n * 2 * sizeof(long long), out_bytes = (size_t)n * sizeof(double);
    char *d = nullptr;
    if (cudaMalloc(&d, in_bytes + out_bytes + sizeof(table)) != cudaSuccess) return HBT_ERR_NOMEM;
    double *d_out = reinterpret_cast<double *>(d + in_bytes);
    double *d_table = reinterpret_cast<double *>(d + in_bytes + out_bytes);
    cudaError_t e = cudaMemcpy(d, steps, in_bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d_table, table, sizeof(table), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_check_cos_fixed<<<(unsigned)((n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024), 256>>>(
            g, d_table, n, reinterpret_cast<const long long *>(d), d_out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d_out, out_bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? HBT_OK : HBT_ERR_CUDA;
}

extern "C" hbt_status hbt_check_math(int device, int32_t which, int64_t n, const double *x,
                                     double *out) {
    if (n < 0 || (n > 0 && (!x || !out)) ||
        which < HBT_CHECK_COS || which > HBT_CHECK_COS_PHASE)
        return HBT_ERR_INVALID;
    if (n == 0) return HBT_OK;
    if (cudaSetDevice(device) != cudaSuccess) return HBT_ERR_CUDA;
    double *d = nullptr, table[kCosEntries];
    if (cudaMalloc(&d, (2 * n + kCosEntries) * sizeof(double)) != cudaSuccess) return HBT_ERR_NOMEM;
    cos_entries(table);
    cudaError_t e = cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(d + 2 * n, table, sizeof(table), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        const long long blocks = (n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024;
        k_check_math<<<(unsigned)blocks, 256>>>(
            which, make_cos_scale(which == HBT_CHECK_COS_PHASE ? 1.0 / hbt::kHbarC : 1.0),
            d + 2 * n, n, d, d + n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + n, n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? HBT_OK : HBT_ERR_CUDA;
}

extern "C" int32_t hbt_check_host_route(const void *p) {
    return static_cast<int32_t>(hbt::host_route(p));
}
