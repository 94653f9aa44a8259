// Batched, culled, persistent pair binning.
//
// A batch is a list of jobs: same-event jobs (all pairs i < j of one list)
// and mixed-event jobs (list 1 x list 2).  When no pair cap can bind, the
// order of the pairs does not matter, and the batch is run as:
//
//  1. k_keys + CUB radix sort, or k_order: every list is reordered by a
//     Morton key of (p_x, p_y, rapidity) cells into a sorted particle table,
//     so that 128-particle tiles are compact in momentum space;
//  2. k_tiles: per tile, the sorted rows with their screen terms and
//     fixed-point columns, and the tile's FP32 box: ranges of p_x, p_y,
//     rapidity y, p_z, and the smallest m_T = sqrt(E^2 - p_z^2);
//  3. k_cull: every tile pair of every job is kept unless no pair in it can
//     pass the q windows.  The test is rigorous: the reference's q_out and
//     q_side satisfy q_out^2 + q_side^2 = q_x^2 + q_y^2, and both lie within
//     Q = max(|lo|, |hi|) of the window, so a pair needs |q_T|^2 <= 2 Q^2;
//     with the longitudinal boost
//       q_long = 2 m_T1 m_T2 sinh(y1 - y2) / sqrt(m_T1^2 + m_T2^2 +
//                2 m_T1 m_T2 cosh(y1 - y2)),
//     which grows with m_T1, m_T2 and |y1 - y2|, so its smallest value over
//     two tiles bounds |q_long| from below; without the boost q_long = q_z.
//     With q_inv histograms the LCMS q_long bound alone also keeps a tile
//     pair (boxes_may_pair).  FP32, every step rounded outwards;
//  4. k_persistent_same / k_persistent_mixed (hbt_persist.cuh): persistent
//     CTAs (5 to 7 per SM) pull (job, i-tile, j-tile) items from the culled
//     same-event and mixed-event queues and run the screened tile-pair
//     bodies of hbt_tile.cuh.  The FP32-weight form runs the same-event
//     queue in chunks and merges the FP32 partials between them.
#include <cub/block/block_radix_sort.cuh>
#include <cub/device/device_radix_sort.cuh>

#include "hbt_batch.cuh"
#include "hbt_persist.cuh"
#include "hbt_tile.cuh"

namespace hbt {
namespace {

using namespace tile;

static_assert(kFixedCols == kFixedEntries, "row size of BatchDev::fixed");

// Morton interleave of three 10-bit cell coordinates.
__device__ __forceinline__ unsigned spread10(unsigned v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__device__ __forceinline__ int find_range(const long long *off, int n, long long g) {
    // largest k with off[k] <= g (off is non-decreasing, off[0] == 0)
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= g)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// Cell of v (in cells from the first one), 0 to `last`.
__device__ __forceinline__ unsigned cell(float v, float last) {
    return v > 0.0f ? (unsigned)fminf(v, last) : 0u;
}

// Morton code of a particle's (p_x, p_y, rapidity) cells, `half` cells either
// side of zero, the outermost taking what lies beyond.  FP32: the key only
// orders the list.
__device__ __forceinline__ unsigned morton_key(const BatchDev &b, const BatchList &l, long long k,
                                               float half, float last) {
    const float px = (float)l.src[0][k], py = (float)l.src[1][k];
    const double pz = l.src[2][k], E = l.src[3][k];
    const float y = 0.5f * __logf((float)(E + pz) / (float)(E - pz));
    return spread10(cell(fmaf(px, (float)b.inv_cell_pt, half), last)) |
           (spread10(cell(fmaf(py, (float)b.inv_cell_pt, half), last)) << 1) |
           (spread10(cell(fmaf(y == y ? y : 0.0f, (float)b.inv_cell_y, half), last)) << 2);
}

// The queues start empty (the first kernel of a batch clears their counters).
__device__ __forceinline__ void clear_queues(const BatchDev &b) {
    if (blockIdx.x == 0 && threadIdx.x < 2) {
        b.n_items[threadIdx.x] = 0u;
        b.item_next[threadIdx.x] = 0u;
    }
}

__global__ void k_keys(BatchDev b) {
    clear_queues(b);
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < b.total;
         g += (long long)gridDim.x * blockDim.x) {
        const int L = find_range(b.list_off, b.n_lists, g);
        const BatchList &l = b.lists[L];
        b.keys_in[g] = ((unsigned long long)L << 32) | morton_key(b, l, g - l.off, 512.0f, 1023.0f);
        b.vals_in[g] = (unsigned)g;
    }
}

// Order of one list of at most kThreads x kItems particles, by one block, for
// batches of short lists: one launch in the place of keys and the device-wide
// radix sort's 6 to 8, whose launches and gaps cost such a batch more than
// its pairs do.  The key has 8 bits to a dimension (2.56 GeV and 6.4 units of
// rapidity either side of zero at the default cells), which orders the list
// as 10 bits do: 6 passes of the block's sort.  (Cells scaled to the list's
// own ranges, which the few largest momenta set, made tiles wide in p_x, p_y
// and culled less.)
template <int kThreads, int kItems>
__global__ void __launch_bounds__(kThreads) k_order(BatchDev b) {
    typedef cub::BlockRadixSort<unsigned, kThreads, kItems, unsigned short> Sort;
    __shared__ typename Sort::TempStorage tmp;
    clear_queues(b);
    const BatchList &l = b.lists[blockIdx.x];
    const int n = (int)l.n;
    unsigned key[kItems];
    unsigned short row[kItems];
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const int k = i * kThreads + threadIdx.x;
        row[i] = (unsigned short)k;
        // past the end: behind every row (whose cells are 254 at most, so
        // that no key equals the padding's 24 bits)
        key[i] = k < n ? morton_key(b, l, k, 128.0f, 254.0f) : 0xffffffffu;
    }
    Sort(tmp).SortBlockedToStriped(key, row, 0, 24);
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const int s = i * kThreads + threadIdx.x;
        if (s < n) b.orig[l.off + s] = row[i];
    }
}

__device__ __forceinline__ float warp_min(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_min(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// One block per tile: its sorted rows (columns, screen terms, fixed-point
// columns: converted once per particle here, as a tile pair would convert its
// 256 particles again each time it is taken) and its box.  One tile to a
// block, so that the conversions' FP64 work, 2 instructions a cycle on an SM,
// spreads over the SMs: by one block per list it took 78 us for a list of
// 1000.  The box is FP32 where the cull's bounds allow (rapidity: logarithm
// of the light-cone terms' ratio, within 2e-6).
template <bool LC>
__global__ void __launch_bounds__(FT) k_tiles(BatchDev b, Grid g, bool split) {
    __shared__ float part[FT / 32][9];
    __shared__ double part2[FT / 32][2];
    const long long tile = blockIdx.x;
    const BatchList &l = b.lists[find_range(b.tile_off, b.n_lists, tile)];
    const long long t = tile - l.tile_off, r = t * FT + threadIdx.x, s = l.off + r;
    const float inf = __int_as_float(0x7f800000);
    // minima of x, y, Y, z, of their negatives, and of m_T
    float q[9];
#pragma unroll
    for (int k = 0; k < 9; k++) q[k] = inf;
    double mm0 = 1e300, mm1 = 1e300;
    if (r < l.n) {
        long long k;
        if (b.vals_out) {
            k = (long long)b.vals_out[s] - l.off;
            b.orig[s] = (unsigned)k;
        } else {
            k = b.orig[s];
        }
        double v[8];
#pragma unroll
        for (int f = 0; f < 8; f++)
            if (f < l.ncols) {
                v[f] = l.src[f][k];
                b.table[(long long)f * b.cap + s] = v[f];
            }
        const Terms w = screen_terms<LC>(v[0], v[1], v[2], v[3]);
        b.terms4[s] = make_float4(w.x, w.y, w.m, w.p);
        b.terms2[s] = make_float2(w.r2, w.t2);
        if (l.ncols == 8) {
            const FixedCols c = split ? split_cols(v) : fixed_cols(g, l.fixed_p, v);
#pragma unroll
            for (int f = 0; f < kFixedCols; f++)
                b.fixed[(long long)f * b.fixed_cap + l.fixed_off + r] = c.c[f];
        }
        q[0] = __double2float_rd(v[0]);
        q[1] = __double2float_rd(v[1]);
        q[3] = __double2float_rd(v[2]);
        q[4] = -__double2float_ru(v[0]);
        q[5] = -__double2float_ru(v[1]);
        q[7] = -__double2float_ru(v[2]);
        q[2] = q[6] = -inf;  // no sound rapidity: never cull on it
        q[8] = 0.0f;
        mm0 = mm1 = -1e300;  // never treated as one mass
        // up to rapidity 10.7 the reference's q_long stays within the cull's
        // margin (1e-6) of the bound: 3 2^-53 of gamma^2
        const float m = (float)(v[3] - v[2]), p = (float)(v[3] + v[2]);
        if (LC && m * 0x1p31f > p && p * 0x1p31f > m) {
            const float y = 0.5f * logf(p / m), e = 2e-6f + 1e-6f * fabsf(y);
            q[2] = y - e;
            q[6] = -(y + e);
            q[8] = sqrtf(m * p) * (1.0f - 1e-6f);
            if (g.qinv) {
                const double mm = (v[3] - v[2]) * (v[3] + v[2]) - (v[0] * v[0] + v[1] * v[1]);
                if (mm == mm) {
                    mm0 = mm;
                    mm1 = -mm;
                }
            }
        }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        q[k] = warp_min(q[k]);
        if (lane == 0) part[w][k] = q[k];
    }
    if (g.qinv) {
        mm0 = warp_min(mm0);
        mm1 = warp_min(mm1);
        if (lane == 0) {
            part2[w][0] = mm0;
            part2[w][1] = mm1;
        }
    }
    __syncthreads();
    if (threadIdx.x > 0) return;
    for (int o = 1; o < FT / 32; o++) {
#pragma unroll
        for (int k = 0; k < 9; k++) q[k] = fminf(q[k], part[o][k]);
        if (g.qinv) {
            mm0 = fmin(mm0, part2[o][0]);
            mm1 = fmin(mm1, part2[o][1]);
        }
    }
    b.boxes[tile] = Box{q[0], -q[4], q[1], -q[5], q[2], -q[6], q[8], q[3], -q[7], mm0, -mm1};
}

// Can a pair with one particle in box a and one in box b pass the windows?
// The 3-D windows bound q_x^2 + q_y^2 and |q_long|; the LCMS q_long of two
// particles with transverse masses m_1, m_2 and rapidity gap dy is
// 2 m_1 m_2 sinh(dy) / sqrt(m_1^2 + m_2^2 + 2 m_1 m_2 cosh(dy)), which
// grows with dy, m_1 and m_2, so the boxes' smallest m_T and gap bound it
// from below.  With q_inv histograms a pair may also pass the q_inv window:
// for two particles of one mass q.K = 0, so in the LCMS
// q_inv^2 = q_out^2 (1 - beta_T^2) + q_side^2 + q_long^2 >= q_long^2, and
// only the q_long bound culls (tiles whose masses differ keep every pair).
// In FP32 with every bound rounded so that it stays one: gaps and squares
// rounded down, sinh below 1 by its series cut (a lower bound), and 2e-5 taken
// off the quotient, far above the rounding of exp, the root and the products.
__device__ __forceinline__ bool boxes_may_pair(const BatchJob &b, const Box &a, const Box &c) {
    const float gY = fmaxf(0.0f, fmaxf(__fsub_rd(a.Y0, c.Y1), __fsub_rd(c.Y0, a.Y1)));
    float qlong = 0.0f;  // lower bound of |q_long| in the LCMS
    if (gY > 0.0f) {
        const float m1 = a.m0, m2 = c.m0, g = fminf(gY, 40.0f);
        const float e = expf(g), i = 1.0f / e;
        const float sh = g < 1.0f ? g * (1.0f + g * g * (1.0f / 6.0f)) : 0.5f * (e - i);
        const float ch = 0.5f * (e + i);
        qlong = (1.0f - 2e-5f) * 2.0f * m1 * m2 * sh *
                rsqrtf(m1 * m1 + m2 * m2 + 2.0f * m1 * m2 * ch);
        if (!(qlong == qlong)) qlong = 0.0f;  // both masses zero
    }
    const float gx = fmaxf(0.0f, fmaxf(__fsub_rd(a.x0, c.x1), __fsub_rd(c.x0, a.x1)));
    const float gy = fmaxf(0.0f, fmaxf(__fsub_rd(a.y0, c.y1), __fsub_rd(c.y0, a.y1)));
    bool pass3 = !((double)__fadd_rd(__fmul_rd(gx, gx), __fmul_rd(gy, gy)) > b.qt2_max);
    if (b.boost) {
        pass3 = pass3 && !((double)qlong > b.ql_max);
    } else {
        // q_long = q_z
        const float gz = fmaxf(0.0f, fmaxf(__fsub_rd(a.z0, c.z1), __fsub_rd(c.z0, a.z1)));
        pass3 = pass3 && !((double)gz > b.ql_max);
    }
    if (pass3 || !b.qinv) return pass3;
    const double lo = fmin(a.mm0, c.mm0), hi = fmax(a.mm1, c.mm1);
    if (!(hi - lo <= 1e-9 * fabs(hi))) return true;
    return !((double)qlong > b.ql_max);
}

// Momentum-space region of a tile pair's pairs: K = (p_1 + p_2) / 2 at the
// boxes' centres, in K_T cells of 1/32 GeV (up to 2 GeV) and 32 azimuthal
// sectors, above the analysis index (serving).  Items of one region update
// the same few histogram slots.
__device__ __forceinline__ unsigned region_key(const BatchJob &job, const Box &a, const Box &c) {
    const float kx = 0.25f * (a.x0 + a.x1 + c.x0 + c.x1);
    const float ky = 0.25f * (a.y0 + a.y1 + c.y0 + c.y1);
    const float kt = sqrtf(kx * kx + ky * ky);
    const unsigned kc = kt < 2.0f ? (unsigned)(kt * 32.0f) : 63u;
    const float ph = atan2f(ky, kx) * (16.0f / 3.14159265f) + 16.0f;  // [0, 32]
    const unsigned pc = ph >= 0.0f && ph < 32.0f ? (unsigned)ph : 0u;
    // (below 0x1FFFFF, so that no key equals the unused entries' 0xffffffff)
    const unsigned dev = job.dev < 0x1FFFFE ? (unsigned)job.dev : 0x1FFFFEu;
    return (dev << 11) | (kc << 5) | pc;
}

// Ordered cap admission: the 3-D slots already at their cap (of the pass's
// counter family) and the grid constants that map a tile pair to the slots
// its pairs can reach.  full == nullptr: no slot test.
struct SlotCull {
    const unsigned char *full;
    double KT_min, dKT, KT_min_sq, KT_max_sq, psi, dKphi, two_pi;
    int n_KT, n_Kphi, az;
};

// Can the pairs of boxes a and c reach only slots already at their cap?
// K = (p_1 + p_2) / 2 lies in the rectangle of the boxes' mean p_x, p_y
// ranges: its K_T range (nearest and farthest points) gives the K_T bins the
// reference can assign (K_perp^2 in [KT_min^2, KT_max^2], src/HBT_correlation.cpp
// :323-366), its angle range the K_phi bins (:408-422), each widened by a
// margin far above rounding.  A rectangle that holds the origin is never
// skipped (its pairs may have K_perp = 0, counted as anomalies).  Admission
// admits nothing more in a full slot, so such a tile pair needs neither the
// count nor the order pass.
__device__ bool slots_all_full(const SlotCull &sc, const Box &a, const Box &c) {
    const double x0 = 0.5 * ((double)a.x0 + c.x0), x1 = 0.5 * ((double)a.x1 + c.x1);
    const double y0 = 0.5 * ((double)a.y0 + c.y0), y1 = 0.5 * ((double)a.y1 + c.y1);
    if (x0 <= 0.0 && x1 >= 0.0 && y0 <= 0.0 && y1 >= 0.0) return false;
    const double nx = x0 > 0.0 ? x0 : (x1 < 0.0 ? x1 : 0.0);
    const double ny = y0 > 0.0 ? y0 : (y1 < 0.0 ? y1 : 0.0);
    const double fx = fmax(fabs(x0), fabs(x1)), fy = fmax(fabs(y0), fabs(y1));
    const double k2lo = (nx * nx + ny * ny) * (1.0 - 1e-9), k2hi = (fx * fx + fy * fy) * (1.0 + 1e-9);
    if (k2hi < sc.KT_min_sq || k2lo > sc.KT_max_sq) return true;  // no pair in the K_T window
    const double klo = sqrt(fmax(k2lo, sc.KT_min_sq)), khi = sqrt(fmin(k2hi, sc.KT_max_sq));
    const int i0 = max(0, (int)floor((klo - sc.KT_min) / sc.dKT - 1e-6));
    const int i1 = min(sc.n_KT - 1, (int)floor((khi - sc.KT_min) / sc.dKT + 1e-6));
    if (!sc.az) {
        for (int k = i0; k <= i1; k++)
            if (!sc.full[k]) return false;
        return true;
    }
    // the angle range around the centre's direction (under pi: the
    // rectangle does not hold the origin), as bins modulo n_Kphi
    const double cth = atan2(0.5 * (y0 + y1), 0.5 * (x0 + x1));
    const double cx[4] = {x0, x1, x0, x1}, cy[4] = {y0, y0, y1, y1};
    double lo = 0.0, hi = 0.0;
    for (int q = 0; q < 4; q++) {
        const double da = remainder(atan2(cy[q], cx[q]) - cth, sc.two_pi);
        lo = fmin(lo, da);
        hi = fmax(hi, da);
    }
    double u = cth + lo - 1e-6 - sc.psi;
    u -= sc.two_pi * floor(u / sc.two_pi);
    const int p0 = (int)floor(u / sc.dKphi);
    const int p1 = (int)floor((u + hi - lo + 2e-6) / sc.dKphi);
    const int np = min(sc.n_Kphi, p1 - p0 + 1);
    for (int k = i0; k <= i1; k++)
        for (int t = 0; t < np; t++) {
            const int ip = ((p0 + t) % sc.n_Kphi + sc.n_Kphi) % sc.n_Kphi;  // u may round below 0
            if (!sc.full[k * sc.n_Kphi + ip]) return false;
        }
    return true;
}

// Culled queues: same-event items at items[0, same_cap), mixed-event items
// at items[same_cap, same_cap + mixed_cap); n_items[0] / n_items[1] count them.
__global__ void k_cull(BatchDev b, SlotCull sc) {
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < b.total_pairs;
         p += (long long)gridDim.x * blockDim.x) {
        const int J = find_range(b.pair_off, b.n_jobs, p);
        const BatchJob &job = b.jobs[J];
        const long long k = p - job.pair_off;
        long long ti, tj;
        if (job.kind == 0) {
            tri_tile(k, ti, tj);
        } else {
            const long long ta = b.lists[job.la].tiles;
            ti = k % ta;
            tj = k / ta;
        }
        const Box &A = b.boxes[b.lists[job.la].tile_off + ti];
        const Box &B = b.boxes[b.lists[job.lb].tile_off + tj];
        if (boxes_may_pair(job, A, B) && !(sc.full && !job.qinv && slots_all_full(sc, A, B))) {
            const Item it = Item{(unsigned)J, (unsigned)ti, (unsigned)tj};
            if (job.kind == 0) {
                const unsigned slot = atomicAdd(b.n_items, 1u);
                if (slot < b.same_cap) {
                    b.items[slot] = it;
                    if (b.order_items) {
                        b.item_key_in[slot] = region_key(job, A, B);
                        b.item_pos_in[slot] = slot;
                    }
                }
            } else {
                const unsigned slot = atomicAdd(b.n_items + 1, 1u);
                if (slot < b.mixed_cap) b.items[b.same_cap + slot] = it;
            }
        }
    }
}

}  // namespace

cudaError_t persistent_same(const Device &d, const BatchDev &b, unsigned base, unsigned end,
                            int grid, cudaStream_t st, int mode) {
    if (d.g.qinv)
        return mode == MODE_FAST ? persistent_same_qinv(d, b, base, end, grid, st)
                                 : cudaErrorNotSupported;
    if (mode == MODE_FAST) return persistent_same_fast(d, b, base, end, grid, st);
    return persistent_same_ordered(d, b, base, end, grid, st, mode);
}

cudaError_t persistent_mixed(const Device &d, const BatchDev &b, int grid, cudaStream_t st,
                             int mode) {
    if (d.g.qinv)
        return mode == MODE_FAST ? persistent_mixed_qinv(d, b, grid, st) : cudaErrorNotSupported;
    if (mode == MODE_FAST) return persistent_mixed_fast(d, b, grid, st);
    return persistent_mixed_ordered(d, b, grid, st, mode);
}

size_t item_sort_temp_bytes(long long n) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const unsigned *)nullptr,
                                    (unsigned *)nullptr, (const unsigned *)nullptr,
                                    (unsigned *)nullptr, (int)n, 0, 32);
    return bytes;
}

size_t batch_sort_temp_bytes(long long cap) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const unsigned long long *)nullptr,
                                    (unsigned long long *)nullptr, (const unsigned *)nullptr,
                                    (unsigned *)nullptr, (int)cap, 0, 64);
    return bytes;
}

cudaError_t run_batch(const Device &d, const BatchDev &b, int grid, unsigned chunk,
                      const Device *host_devs, int n_host_devs, cudaStream_t st,
                      cudaEvent_t *marks, int mode) {
    cudaError_t e;
    const int gs = 152 * 8;
    const bool lc = d.g.boost || d.g.qinv;  // light-cone screen terms
    if (b.max_list <= kSmallList) {
        // the smallest block that holds the list: its sort's time grows with
        // the threads it synchronises and their items (10, 12, 18 and 24 us)
        if (b.max_list <= 1024)
            k_order<256, 4><<<b.n_lists, 256, 0, st>>>(b);
        else if (b.max_list <= 2048)
            k_order<512, 4><<<b.n_lists, 512, 0, st>>>(b);
        else if (b.max_list <= 4096)
            k_order<512, 8><<<b.n_lists, 512, 0, st>>>(b);
        else
            k_order<1024, 8><<<b.n_lists, 1024, 0, st>>>(b);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    } else {
        k_keys<<<gs, 256, 0, st>>>(b);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        int end_bit = 32;
        while (end_bit < 64 && (1LL << (end_bit - 32)) < b.n_lists) end_bit++;
        size_t bytes = b.sort_temp_bytes;
        e = cub::DeviceRadixSort::SortPairs(b.sort_temp, bytes, b.keys_in, b.keys_out, b.vals_in,
                                            b.vals_out, (int)b.total, 0, end_bit, st);
        if (e != cudaSuccess) return e;
    }
    const bool split = d.precision == 1;  // the FP32-weight form's columns
    if (lc)
        k_tiles<true><<<(unsigned)b.total_tiles, FT, 0, st>>>(b, d.g, split);
    else
        k_tiles<false><<<(unsigned)b.total_tiles, FT, 0, st>>>(b, d.g, split);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (b.order_items && b.same_cap > 0 &&
        (e = cudaMemsetAsync(b.item_key_in, 0xff, (size_t)b.same_cap * sizeof(unsigned), st)) !=
            cudaSuccess)
        return e;
    if (b.total_pairs > 0) {
        SlotCull sc = {};
        if (mode != MODE_FAST && d.caps.slot_full && !b.devs) {
            sc.full = d.caps.slot_full;
            sc.KT_min = d.g.KT_min;
            sc.dKT = d.g.dKT;
            sc.KT_min_sq = d.g.KT_min_sq;
            sc.KT_max_sq = d.g.KT_max_sq;
            sc.psi = d.g.psi_ref;
            sc.dKphi = d.g.dKphi;
            sc.two_pi = d.g.two_pi;
            sc.n_KT = d.g.n_KT;
            sc.n_Kphi = d.g.n_Kphi;
            sc.az = d.g.azimuthal;
        }
        k_cull<<<(unsigned)min((long long)gs, (b.total_pairs + 255) / 256), 256, 0, st>>>(b, sc);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (b.order_items && b.same_cap > 0) {
        // unused entries keep the key 0xffffffff and sort behind the queue
        size_t bytes = b.item_sort_temp_bytes;
        e = cub::DeviceRadixSort::SortPairs(b.item_sort_temp, bytes, b.item_key_in,
                                            b.item_key_out, b.item_pos_in, b.item_pos_out,
                                            (int)b.same_cap, 0, 32, st);
        if (e != cudaSuccess) return e;
    }
    // the COUNT pass bins nothing: no FP32 partials to merge
    const int prec = mode == MODE_COUNT ? 0 : d.precision;
    // same-event items (chunked for the FP32-weight form)
    const unsigned upper = b.same_cap;
    if (chunk == 0 || prec != 1) chunk = upper;
    if (marks && (e = cudaEventRecord(marks[0], st)) != cudaSuccess) return e;
    for (unsigned base = 0; base < upper; base += chunk) {
        const unsigned end =
            (unsigned)min((unsigned long long)base + chunk, (unsigned long long)upper);
        if (base > 0 && (e = cudaMemsetAsync(b.item_next, 0, sizeof(unsigned), st)) != cudaSuccess)
            return e;
        e = persistent_same(d, b, base, end, grid, st, mode);
        if (e != cudaSuccess) return e;
        if (prec == 1 && !b.devs) {
            if ((e = launch_merge(d, st, b.n_items, base)) != cudaSuccess) return e;
        } else if (prec == 1) {
            for (int k = 0; k < n_host_devs; k++)
                if ((e = launch_merge(host_devs[k], st, b.n_items, base)) != cudaSuccess) return e;
        }
    }
    if (marks && (e = cudaEventRecord(marks[1], st)) != cudaSuccess) return e;
    if (marks && (e = cudaEventRecord(marks[2], st)) != cudaSuccess) return e;
    // mixed-event items
    if (b.mixed_cap > 0) {
        e = persistent_mixed(d, b, grid, st, mode);
        if (e != cudaSuccess) return e;
    }
    if (d.g.qinv && mode == MODE_FAST) {
        for (int k = 0; k < (b.devs ? n_host_devs : 1); k++)
            if ((e = launch_qinv_merge(b.devs ? host_devs[k] : d, st)) != cudaSuccess) return e;
    }
    if (marks && (e = cudaEventRecord(marks[3], st)) != cudaSuccess) return e;
    return cudaSuccess;
}

}  // namespace hbt
