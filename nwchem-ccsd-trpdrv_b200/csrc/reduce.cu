// Deterministic energy reductions and small device utilities.
//
//  records_kernel:       per triple, the compensated sum of its tile-pair items (fixed order) -> rec[t][4]
//  totals_kernel:        per system, the compensated total of emp4i + [i != k] emp4k and of
//                        emp5i + [i != k] emp5k over the triples (the accumulation of
//                        omp/ccsd_trpdrv_omp_cbody.c:133-142), as a double-double (hi, lo) pair, built with
//                        error-free TwoSum in a fixed order.
//  negate_kernel:        dst = -src (the occupied A operands are stored negated).
//  pack_rows_kernel:     rows of odd length copied to an even pitch (operands of the cp.async staging).

#include "device_common.cuh"
#include "launch.h"

namespace trpdrv {

__device__ __forceinline__ void dd_add(double &hi, double &lo, double x)
{
    double s, e;
    two_sum(hi, x, s, e);
    hi = s;
    lo += e;
}

struct DdPair {
    double h4, l4, h5, l5;
    __device__ __forceinline__ void add_record(const double (&rec)[4], int packed)
    {
        dd_add(h4, l4, rec[0]);
        dd_add(h5, l5, rec[1]);
        if ((packed & 1023) != ((packed >> 20) & 1023)) {  // i != k
            dd_add(h4, l4, rec[2]);
            dd_add(h5, l5, rec[3]);
        }
    }
};

constexpr int REC_WARPS = 8;       // records per block of records_kernel
constexpr int FIN_THREADS = 512;   // totals_kernel
constexpr int FIN_BLOCKS = 1024;   // its most blocks per system
constexpr int MAX_GRID_Y = 65535;  // rows of a grid

// The block's sum of every thread's pair in thread 0 (a fixed tree).
__device__ __forceinline__ DdPair block_dd(DdPair v, double (&sh)[4][FIN_THREADS])
{
    const int t = threadIdx.x;
    sh[0][t] = v.h4;
    sh[1][t] = v.l4;
    sh[2][t] = v.h5;
    sh[3][t] = v.l5;
    __syncthreads();
    for (int w = FIN_THREADS / 2; w > 0; w >>= 1) {
        if (t < w) {
            double s, e;
            two_sum(sh[0][t], sh[0][t + w], s, e);
            sh[0][t] = s;
            sh[1][t] += sh[1][t + w] + e;
            two_sum(sh[2][t], sh[2][t + w], s, e);
            sh[2][t] = s;
            sh[3][t] += sh[3][t + w] + e;
        }
        __syncthreads();
    }
    const DdPair r = {sh[0][0], sh[1][0], sh[2][0], sh[3][0]};
    __syncthreads();
    return r;
}

__host__ __device__ inline int total_blocks(long long ntriples)
{
    const long long n = (ntriples + FIN_THREADS - 1) / FIN_THREADS;
    return n < FIN_BLOCKS ? (int)n : FIN_BLOCKS;
}

// Rows of the grid take systems (more systems than MAX_GRID_Y share rows), one warp per record.
__global__ void __launch_bounds__(REC_WARPS * 32) records_kernel(const trpdrv_dev_system *__restrict__ sys, int nsys)
{
    const int lane = threadIdx.x & 31;
    for (int s = blockIdx.y; s < nsys; s += gridDim.y) {
        const trpdrv_dev_system &S = sys[s];
        const int nslot = S.npairs * TRPDRV_FUSED_SLOTS;
        for (long long t = (long long)blockIdx.x * REC_WARPS + (threadIdx.x >> 5); t < S.ntriples;
             t += (long long)gridDim.x * REC_WARPS) {
            const double *p = S.partial + 4 * t * (long long)nslot;
            // compensated per lane (error-free TwoSum, errors carried in lo), then the lanes' hi and lo sums
            double hi[4] = {0.0, 0.0, 0.0, 0.0}, lo[4] = {0.0, 0.0, 0.0, 0.0};
            for (int q = lane; q < nslot; q += 32) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    double v, e;
                    two_sum(hi[c], p[4 * q + c], v, e);
                    hi[c] = v;
                    lo[c] += e;
                }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const double h = warp_sum(hi[c]), l = warp_sum(lo[c]);
                if (lane == 0) S.rec[4 * t + c] = h + l;
            }
        }
    }
}

// One system: each block leaves its records' double-double sum; the system's last block adds those in block order and
// writes the totals and the execution's status word to pinned host memory, so that reading the energies needs
// no copy.
__device__ __forceinline__ void system_totals(const trpdrv_dev_system &S, double *__restrict__ bs,
                                              unsigned *__restrict__ done, double *__restrict__ out,
                                              double *__restrict__ status_out, const int *__restrict__ status,
                                              double (&sh)[4][FIN_THREADS], int &last)
{
    const long long n = S.ntriples;
    const int nblk = total_blocks(n), tid = threadIdx.x;
    if ((int)blockIdx.x >= nblk) return;
    DdPair v = {0.0, 0.0, 0.0, 0.0};
    for (long long t = (long long)blockIdx.x * FIN_THREADS + tid; t < n; t += (long long)nblk * FIN_THREADS) {
        const double rec[4] = {S.rec[4 * t], S.rec[4 * t + 1], S.rec[4 * t + 2], S.rec[4 * t + 3]};
        v.add_record(rec, S.triples[t % S.nt]);  // records are [a][triple]
    }
    v = block_dd(v, sh);
    if (nblk > 1) {
        if (tid == 0) {
            double *b = bs + 4 * blockIdx.x;
            b[0] = v.h4;
            b[1] = v.l4;
            b[2] = v.h5;
            b[3] = v.l5;
            __threadfence();
            last = atomicAdd(done, 1u) == (unsigned)nblk - 1;
        }
        __syncthreads();
        if (!last) return;
        __threadfence();
        v = {0.0, 0.0, 0.0, 0.0};
        for (int q = tid; q < nblk; q += FIN_THREADS) {
            const double *b = bs + 4 * q;
            double s, e;
            two_sum(v.h4, __ldcg(b), s, e);
            v.h4 = s;
            v.l4 += __ldcg(b + 1) + e;
            two_sum(v.h5, __ldcg(b + 2), s, e);
            v.h5 = s;
            v.l5 += __ldcg(b + 3) + e;
        }
        v = block_dd(v, sh);
        if (tid == 0) *done = 0u;
    }
    if (tid == 0) {
        double s, e;
        two_sum(v.h4, v.l4, s, e);  // renormalise
        out[0] = s;
        out[1] = e;
        two_sum(v.h5, v.l5, s, e);
        out[2] = s;
        out[3] = e;
        *status_out = (double)*status;
    }
}

// Rows of the grid take systems, as in records_kernel.
__global__ void __launch_bounds__(FIN_THREADS)
totals_kernel(const trpdrv_dev_system *__restrict__ sys, int nsys, double *__restrict__ bsum, unsigned *__restrict__ done,
              const int *__restrict__ status, double *__restrict__ res)
{
    __shared__ double sh[4][FIN_THREADS];
    __shared__ int last;
    for (int s = blockIdx.y; s < nsys; s += gridDim.y)
        system_totals(sys[s], bsum + 4 * (size_t)s * gridDim.x, done + s, res + 4 * (size_t)s,
                      res + 4 * (size_t)nsys, status, sh, last);
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

extern "C" int trpdrv_launch_records(const trpdrv_dev_system *h_sys, const trpdrv_dev_system *d_sys, int nsys,
                                     void *stream)
{
    long long blocks = 0;
    for (int q = 0; q < nsys; ++q) {
        const long long n = (h_sys[q].ntriples + REC_WARPS - 1) / REC_WARPS;
        if (n > blocks) blocks = n;
    }
    if (blocks == 0) return 0;
    if (blocks > 65535) blocks = 65535;
    records_kernel<<<dim3((unsigned)blocks, (unsigned)(nsys < MAX_GRID_Y ? nsys : MAX_GRID_Y)), REC_WARPS * 32, 0,
                     (cudaStream_t)stream>>>(d_sys, nsys);
    return (int)cudaGetLastError();
}

static int most_total_blocks(const trpdrv_dev_system *h_sys, int nsys)
{
    int blocks = 0;
    for (int q = 0; q < nsys; ++q) {
        const int n = total_blocks(h_sys[q].ntriples);
        if (n > blocks) blocks = n;
    }
    return blocks;
}

extern "C" size_t trpdrv_totals_doubles(const trpdrv_dev_system *h_sys, int nsys)
{
    return 4 * (size_t)nsys * (size_t)most_total_blocks(h_sys, nsys);
}

extern "C" int trpdrv_launch_totals(const trpdrv_dev_system *h_sys, const trpdrv_dev_system *d_sys, int nsys,
                                    double *bsum, unsigned *done, const int *status, double *res, void *stream)
{
    const int blocks = most_total_blocks(h_sys, nsys);
    if (blocks == 0) return 0;
    totals_kernel<<<dim3((unsigned)blocks, (unsigned)(nsys < MAX_GRID_Y ? nsys : MAX_GRID_Y)), FIN_THREADS, 0,
                    (cudaStream_t)stream>>>(d_sys, nsys, bsum, done, status, res);
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
