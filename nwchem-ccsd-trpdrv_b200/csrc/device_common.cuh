// Device-side building blocks shared by the triples kernels (sm_100a).
//
//  * FP64 tensor-core MMA (DMMA) wrappers: mma.sync ... .f64 (sm_100a has no tcgen05 kind for
//    f64, so FP64 contractions run on the mma.sync DMMA path).
//  * cp.async global->shared staging with zero fill for masked tails.
//  * The tengy (b,c) energy term of omp/ccsd_tengy_c99.c:65-111, written once and used by both the
//    fused epilogue and the standalone reduction kernel.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace trpdrv {

// ------------------------------------------------------------------------------------------------
// FP64 MMA.  Fragment layouts (PTX ISA, mma.m16n8k4 .f64):  g = lane>>2, t = lane&3
//   A 16x4 (row): a0 = A[g][t], a1 = A[g+8][t]
//   B 4x8  (col): b0 = B[t][g]
//   C 16x8      : c0 = C[g][2t], c1 = C[g][2t+1], c2 = C[g+8][2t], c3 = C[g+8][2t+1]
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void dmma_16x8x4(double (&d)[4], double a0, double a1, double b0)
{
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a0, double b0)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a0), "d"(b0));
}

__device__ __forceinline__ void dmma_16x8x8(double (&d)[4], const double (&a)[4], const double (&b)[2])
{
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

__device__ __forceinline__ void dmma_16x8x16(double (&d)[4], const double (&a)[8], const double (&b)[4])
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, "
        "{%4,%5,%6,%7,%8,%9,%10,%11}, {%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]),
          "d"(b[0]), "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

// ------------------------------------------------------------------------------------------------
// cp.async staging.  `valid == false` copies nothing from global and zero-fills the destination
// (src-size operand 0); the source address is still required to be a mapped address, so callers
// pass an in-bounds base pointer in that case.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async_16(void *smem, const void *gmem, bool valid)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}

__device__ __forceinline__ void cp_async_8(void *smem, const void *gmem, bool valid)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int n = valid ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }

template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// ------------------------------------------------------------------------------------------------
// Reductions
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Error-free transformation a + b = s + e (Knuth TwoSum).
__device__ __forceinline__ void two_sum(double a, double b, double &s, double &e)
{
    s = a + b;
    const double bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// ------------------------------------------------------------------------------------------------
// The tengy terms.  f index order used throughout the library:
//   0 f1n, 1 f2n, 2 f3n, 3 f4n, 4 f1t, 5 f2t, 6 f3t, 7 f4t
// bc[x] = f_x(b,c), cb[x] = f_x(c,b).  The four forms of omp/ccsd_tengy_c99.c:91-111 with the denominator
// denom = -1/(e_b + e_c + eaijk) factored out of each (equal up to floating-point reassociation).
// ------------------------------------------------------------------------------------------------
struct TengySums {
    double e4i, e5i, e4k, e5k;
};

// The terms of a position (b,c) and its mirror (c,b) together.  They share the
// denominator, and the sums t2 + t3, t1 + t4, n2 + n3, n1 + n4 of each position enter both positions' forms, so a
// pair costs about 135 FP64 instructions; the forms written out twice cost 200 (FP64 arithmetic
// is issued at half a warp instruction per clock per scheduler, on the same pipe as the MMAs).  vb, vc: the
// per-index vectors at b and at c.
struct TengyIdx {
    double t1v1, t1v2, dx1, dx2, dc1, dc2;
};

struct TengyPos {  // one position's eight f and the sums shared by both positions' forms
    double n1, n2, n3, n4, t1, t2, t3, t4, sn, un, st, ut;
    __device__ __forceinline__ explicit TengyPos(const double (&f)[8])
        : n1(f[0]), n2(f[1]), n3(f[2]), n4(f[3]), t1(f[4]), t2(f[5]), t3(f[6]), t4(f[7]), sn(n2 + n3), un(n1 + n4),
          st(t2 + t3), ut(t1 + t4)
    {
    }
};

__device__ __forceinline__ void tengy_forms(const TengyPos &p, const TengyPos &q, double &a4i, double &a4k, double &f5i,
                                            double &g5i, double &f5k, double &g5k)
{
    a4i = (p.t1 + q.un + (q.t2 + p.n3)) * (p.ut - 2 * p.st) - (p.n1 + q.t1 + q.sn) * (2 * p.ut - p.st)
        + 3 * (p.n1 * (p.n1 + q.n3 + 2 * q.t4) + p.n2 * q.t2 + p.n3 * p.t4);
    a4k = (p.n1 + q.ut + (q.n2 + p.t3)) * (p.un - 2 * p.sn) - (p.t1 + q.n1 + q.st) * (2 * p.un - p.sn)
        + 3 * (p.t1 * (p.t1 + q.t3 + 2 * q.n4) + p.t2 * q.n2 + p.t3 * p.n4);
    f5i = (p.t1 + p.n2 + q.n4) - 2 * (p.st + p.un + q.sn) + 4 * (p.n3 + p.t4 + q.n1);
    g5i = p.un + q.t1 - 2 * (p.sn + q.t2);
    f5k = (p.n1 + p.t2 + q.t4) - 2 * (p.sn + p.ut + q.st) + 4 * (p.t3 + p.n4 + q.t1);
    g5k = p.ut + q.n1 - 2 * (p.st + q.n2);
}

// The four terms but for the factor denom; both (of a whole warp): false for those of (b,c) alone.
struct TengyTerms {
    double a4i, a4k, e5i, e5k;
};

__device__ __forceinline__ TengyTerms tengy_terms(bool both, const double (&bc)[8], const double (&cb)[8],
                                                  const TengyIdx &vb, const TengyIdx &vc)
{
    const TengyPos p(bc), q(cb);
    TengyTerms r;
    double f5i, g5i, f5k, g5k;
    tengy_forms(p, q, r.a4i, r.a4k, f5i, g5i, f5k, g5k);
    r.e5i = vb.t1v1 * (vc.dx1 * f5i + vc.dc1 * g5i);
    r.e5k = vb.t1v2 * (vc.dx2 * f5k + vc.dc2 * g5k);
    if (both) {
        double b4i, b4k;
        tengy_forms(q, p, b4i, b4k, f5i, g5i, f5k, g5k);
        r.a4i += b4i;
        r.a4k += b4k;
        r.e5i += vc.t1v1 * (vb.dx1 * f5i + vb.dc1 * g5i);
        r.e5k += vc.t1v2 * (vb.dx2 * f5k + vb.dc2 * g5k);
    }
    return r;
}

__device__ __forceinline__ void tengy_pair(bool both, const double (&bc)[8], const double (&cb)[8], double denom,
                                           const TengyIdx &vb, const TengyIdx &vc, TengySums &s)
{
    const TengyTerms t = tengy_terms(both, bc, cb, vb, vc);
    s.e4i += denom * t.a4i;
    s.e4k += denom * t.a4k;
    s.e5i += denom * t.e5i;
    s.e5k += denom * t.e5k;
}

template <bool BOTH>
__device__ __forceinline__ void tengy_pair(const double (&bc)[8], const double (&cb)[8], double denom,
                                           const TengyIdx &vb, const TengyIdx &vc, TengySums &s)
{
    tengy_pair(BOTH, bc, cb, denom, vb, vc, s);
}

// The four sums of a warp, each as warp_sum adds it up; lanes 8 e .. 8 e + 7 return the e-th (e4i, e5i, e4k, e5k).  Two
// thirds of the shuffles of four warp_sums.
__device__ __forceinline__ double warp_sum4(const TengySums &s, int lane)
{
    const bool h = lane & 16, g = lane & 8;
    double a = h ? s.e4k : s.e4i, b = h ? s.e5k : s.e5i;  // kept
    a += __shfl_xor_sync(0xffffffffu, h ? s.e4i : s.e4k, 16);
    b += __shfl_xor_sync(0xffffffffu, h ? s.e5i : s.e5k, 16);
    double c = g ? b : a;
    c += __shfl_xor_sync(0xffffffffu, g ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    return c;
}

// Block-wide sum of the four partial energies; returns the totals in thread 0.  `scratch` must
// hold 4 * (blockDim.x / 32) doubles.  The summation order is fixed (deterministic).
__device__ __forceinline__ TengySums block_sum4(TengySums s, double *scratch)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const double sum = warp_sum4(s, lane);
    if ((lane & 7) == 0) scratch[4 * warp + (lane >> 3)] = sum;
    __syncthreads();
    TengySums r = {0.0, 0.0, 0.0, 0.0};
    if (threadIdx.x == 0) {
        for (int w = 0; w < nw; ++w) {
            r.e4i += scratch[4 * w + 0];
            r.e5i += scratch[4 * w + 1];
            r.e4k += scratch[4 * w + 2];
            r.e5k += scratch[4 * w + 3];
        }
    }
    return r;
}

}  // namespace trpdrv
