// Deterministic energy reductions and small device utilities.
//
//  item_reduce_kernel:   per triple, the compensated sum of its tile-pair items (fixed order) -> rec[t][4]
//  system_reduce_kernel: per system, the compensated total of emp4i + [i != k] emp4k and of
//                        emp5i + [i != k] emp5k over the triples (the accumulation of
//                        omp/ccsd_trpdrv_omp_cbody.c:133-142), as a double-double (hi, lo) pair,
//                        built with error-free TwoSum in a fixed order.
//  negate_kernel:        dst = -src (the occupied A operands are stored negated).
//  pack_rows_kernel:     rows of odd length copied to an even pitch (operands of the cp.async staging).

#include "device_common.cuh"
#include "launch.h"

namespace trpdrv {

__global__ void item_reduce_kernel(const double *__restrict__ partial, int npairs, long long ntriples,
                                   double *__restrict__ rec)
{
    const long long t = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= ntriples) return;
    const int nslot = npairs * TRPDRV_FUSED_SLOTS;
    const double *p = partial + 4 * t * (long long)nslot;
    // compensated per lane (error-free TwoSum, errors carried in lo), then the lanes' hi and lo sums
    double hi[4] = {0.0, 0.0, 0.0, 0.0}, lo[4] = {0.0, 0.0, 0.0, 0.0};
    for (int q = lane; q < nslot; q += 32) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            double s, e;
            two_sum(hi[c], p[4 * q + c], s, e);
            hi[c] = s;
            lo[c] += e;
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const double h = warp_sum(hi[c]), l = warp_sum(lo[c]);
        if (lane == 0) rec[4 * t + c] = h + l;
    }
}

__device__ __forceinline__ void dd_add(double &hi, double &lo, double x)
{
    double s, e;
    two_sum(hi, x, s, e);
    hi = s;
    lo += e;
}

constexpr int RED_THREADS = 1024;

__global__ void __launch_bounds__(RED_THREADS)
system_reduce_kernel(const double *__restrict__ rec, const int32_t *__restrict__ triples, long long n, long long nt,
                     double *__restrict__ out)
{
    __shared__ double sh[4][RED_THREADS];
    double h4 = 0.0, l4 = 0.0, h5 = 0.0, l5 = 0.0;
    for (long long t = threadIdx.x; t < n; t += RED_THREADS) {
        const int packed = triples[t % nt];  // records are [a][triple]
        const int i = packed & 1023, k = (packed >> 20) & 1023;
        dd_add(h4, l4, rec[4 * t + 0]);
        dd_add(h5, l5, rec[4 * t + 1]);
        if (i != k) {
            dd_add(h4, l4, rec[4 * t + 2]);
            dd_add(h5, l5, rec[4 * t + 3]);
        }
    }
    sh[0][threadIdx.x] = h4;
    sh[1][threadIdx.x] = l4;
    sh[2][threadIdx.x] = h5;
    sh[3][threadIdx.x] = l5;
    __syncthreads();
    for (int w = RED_THREADS / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            const int o = threadIdx.x + w;
            double s, e;
            two_sum(sh[0][threadIdx.x], sh[0][o], s, e);
            sh[0][threadIdx.x] = s;
            sh[1][threadIdx.x] += sh[1][o] + e;
            two_sum(sh[2][threadIdx.x], sh[2][o], s, e);
            sh[2][threadIdx.x] = s;
            sh[3][threadIdx.x] += sh[3][o] + e;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double s, e;
        two_sum(sh[0][0], sh[1][0], s, e);  // renormalise
        out[0] = s;
        out[1] = e;
        two_sum(sh[2][0], sh[3][0], s, e);
        out[2] = s;
        out[3] = e;
    }
}

__global__ void negate_kernel(const double *__restrict__ src, double *__restrict__ dst, size_t n)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = -src[i];
}

// One row of the grid per segment; a block copies whole rows, two destination elements per thread and step.
// HBM-bound (reads width, writes pitch doubles a row).
constexpr int PACK_PAIRS = 2048;  // destination pairs per block and pass
__global__ void pack_rows_kernel(const trpdrv_pack_list L)
{
    const auto &g = L.seg[blockIdx.y];
    const int ppr = g.pitch >> 1, rpb = ppr < PACK_PAIRS ? PACK_PAIRS / ppr : 1;
    const double sg = g.neg ? -1.0 : 1.0;
    for (long long row0 = (long long)blockIdx.x * rpb; row0 < g.rows; row0 += (long long)gridDim.x * rpb) {
        const int nr = g.rows - row0 < rpb ? (int)(g.rows - row0) : rpb;
        const double *src = g.src + row0 * g.width;
        double2 *dst = reinterpret_cast<double2 *>(g.dst + row0 * g.pitch);
        for (int e = threadIdx.x; e < nr * ppr; e += blockDim.x) {
            const int r = e / ppr, c = 2 * (e - r * ppr);
            const double *s = src + (long long)r * g.width + c;
            dst[e] = make_double2(sg * __ldg(s), c + 1 < g.width ? sg * __ldg(s + 1) : 0.0);
        }
    }
}

}  // namespace trpdrv

using namespace trpdrv;

extern "C" int trpdrv_launch_pack_rows(const trpdrv_pack_list *list, void *stream)
{
    if (!list || list->n <= 0) return 0;
    if (list->n > TRPDRV_PACK_LIST_MAX) return (int)cudaErrorInvalidValue;
    long long most = 1;
    for (int s = 0; s < list->n; ++s) {
        const long long b = (list->seg[s].rows * (list->seg[s].pitch / 2) + PACK_PAIRS - 1) / PACK_PAIRS;
        if (b > most) most = b;
    }
    pack_rows_kernel<<<dim3((unsigned)(most < 2048 ? most : 2048), (unsigned)list->n), 256, 0,
                       (cudaStream_t)stream>>>(*list);
    return (int)cudaGetLastError();
}

extern "C" int trpdrv_launch_item_reduce(const trpdrv_dev_system *h_sys, void *stream)
{
    if (h_sys->ntriples <= 0) return 0;
    const int warps = 8;
    const long long blocks = (h_sys->ntriples + warps - 1) / warps;
    item_reduce_kernel<<<(unsigned)blocks, warps * 32, 0, (cudaStream_t)stream>>>(h_sys->partial, h_sys->npairs,
                                                                                 h_sys->ntriples, h_sys->rec);
    return (int)cudaGetLastError();
}

extern "C" int trpdrv_launch_system_reduce(const double *rec, const int32_t *triples, int64_t ntriples, int64_t nt,
                                           double *out, void *stream)
{
    if (nt <= 0) return 0;
    system_reduce_kernel<<<1, RED_THREADS, 0, (cudaStream_t)stream>>>(rec, triples, (long long)ntriples, (long long)nt,
                                                                     out);
    return (int)cudaGetLastError();
}

extern "C" int trpdrv_launch_negate(const double *src, double *dst, size_t n, void *stream)
{
    if (n == 0) return 0;
    size_t blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    negate_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(src, dst, n);
    return (int)cudaGetLastError();
}
