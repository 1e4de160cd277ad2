// The tengy reduction over one tile pair {B,C} whose f tiles are parked in shared memory, for the emulated form's
// energies.  For a diagonal pair (B == C) only the tiles of orientation (B, C) are used.  Follows
// omp/ccsd_tengy_c99.c:58-111: every (b,c) of BxC and CxB contributes one term with
// denom = -1/(e_b + e_c + eaijk).
#pragma once

#include "device_common.cuh"

namespace trpdrv {

struct TengyVecs {
    const double *eorb, *dintc1, *dintx1, *t1v1, *dintc2, *dintx2, *t1v2;
    double eaijk;
    int voff;  // ncor + nocc: index of the first virtual orbital energy
    int nvir;
    __device__ __forceinline__ TengyIdx idx(int x) const
    {
        return {__ldg(t1v1 + x), __ldg(t1v2 + x), __ldg(dintx1 + x), __ldg(dintx2 + x), __ldg(dintc1 + x),
                __ldg(dintc2 + x)};
    }
};

// Tengy terms of one tile pair {B, C} of width W from tiles parked in shared memory: park holds the
// eight f tiles of orientation (B, C) followed (off the diagonal) by the eight of (C, B), each tile
// W x (W + 1) doubles, element (row r, column q) at r * (W + 1) + q.  One thread per (b, c) of B x C: the 16
// values at (b, c) and (c, b) are loaded once for the terms of (b, c) and, off the diagonal, of (c, b).
template <int W>
__device__ __forceinline__ void tengy_tile_pair_factored(const double *park, int b0, int c0, bool diag,
                                                         const TengyVecs &v, int tid, int nthreads, TengySums &su)
{
    constexpr int P = W + 1, TILE = W * P;
    for (int idx = tid; idx < W * W; idx += nthreads) {
        const int r = idx / W, q = idx % W;
        const int b = b0 + r, c = c0 + q;
        if (b < v.nvir && c < v.nvir) {
            const double *bcT = park + r * P + q;                          // f_x(B + r, C + q)
            const double *cbT = park + (diag ? 0 : 8) * TILE + q * P + r;  // f_x(C + q, B + r)
            double fbc[8], fcb[8];
#pragma unroll
            for (int f = 0; f < 8; ++f) {
                fbc[f] = bcT[f * TILE];
                fcb[f] = cbT[f * TILE];
            }
            const double denom = -1.0 / (__ldg(v.eorb + v.voff + b) + __ldg(v.eorb + v.voff + c) + v.eaijk);
            const TengyIdx vb = v.idx(b), vc = v.idx(c);
            if (diag)
                tengy_pair<false>(fbc, fcb, denom, vb, vc, su);
            else
                tengy_pair<true>(fbc, fcb, denom, vb, vc, su);
        }
    }
}

// Element x of the 16-double row `col` in a box landed with the 128-byte swizzle: the 16-byte chunk
// index is XORed with col mod 8 (rows are 128 bytes, the box starts on a 1024-byte boundary).
__device__ __forceinline__ int swz128(int x, int col) { return (((x >> 1) ^ (col & 7)) << 1) | (x & 1); }

// The same sums over 16-wide tiles as TMA lands them: the (B, C) box, then off the diagonal the
// (C, B) box, each 8 planes (one per f) of 16 columns x 16 rows, row index contiguous and swizzled
// by swz128.  Each half-warp walks one diagonal q = (r + d) mod 16: both the (b, c) reads (row r of
// column q) and the (c, b) reads (row q of column r) then hit 16 different 8-byte bank pairs.  The per-index
// vectors come from a shared table (rows of 16: t1v(i), t1v(k), dintx(i), dintx(k), dintc(i), dintc(k), e_virt
// at b0 + r, then the same seven at c0 + q).
template <int NTHREAD>
__device__ __forceinline__ void tengy_tile_pair_swz16_sv(const double *park, const double *vsh, int b0, int c0,
                                                         bool diag, int nvir, double eaijk, int tid, TengySums &su)
{
    constexpr int PLANE = 16 * 16, BOX = 8 * PLANE, NDIAG = 16 / (NTHREAD / 16);
    static_assert(NTHREAD % 16 == 0 && NTHREAD <= 256 && 16 % (NTHREAD / 16) == 0, "half-warps walk the 16 diagonals");
    const int r = tid & 15;
    const double *vb = vsh, *vc = vsh + 7 * 16;  // row x of a side at [x * 16 + index]
#pragma unroll
    for (int k = 0; k < NDIAG; ++k) {
        const int d = (tid >> 4) + k * (NTHREAD / 16);
        const int q = (r + d) & 15;
        if (b0 + r < nvir && c0 + q < nvir) {
            const double *bcT = park + q * 16 + swz128(r, q);                       // f_x(B + r, C + q)
            const double *cbT = park + (diag ? 0 : BOX) + r * 16 + swz128(q, r);    // f_x(C + q, B + r)
            double fbc[8], fcb[8];
#pragma unroll
            for (int f = 0; f < 8; ++f) {
                fbc[f] = bcT[f * PLANE];
                fcb[f] = cbT[f * PLANE];
            }
            const double denom = -1.0 / (vb[6 * 16 + r] + vc[6 * 16 + q] + eaijk);
            const TengyIdx ib = {vb[r], vb[16 + r], vb[2 * 16 + r], vb[3 * 16 + r], vb[4 * 16 + r], vb[5 * 16 + r]};
            const TengyIdx ic = {vc[q], vc[16 + q], vc[2 * 16 + q], vc[3 * 16 + q], vc[4 * 16 + q], vc[5 * 16 + q]};
            if (diag)
                tengy_pair<false>(fbc, fcb, denom, ib, ic, su);
            else
                tengy_pair<true>(fbc, fcb, denom, ib, ic, su);
        }
    }
}

}  // namespace trpdrv
