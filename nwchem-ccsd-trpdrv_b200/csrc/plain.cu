// Plain path (sm_100a, FP64 DMMA): the reference body's structure on the GPU, f in HBM between two launches.
//
//  plain_gemm_kernel: one grouped launch computes the eight f of n triples into f[n][8][nvir][nvir] (the 16
//    DGEMMs of omp/ccsd_trpdrv_omp_cbody.c:70-117: each f is its K=nvir product followed by its K=nocc
//    product, here one contraction over the concatenated index).
//  tengy_kernel: the (b,c) reduction of omp/ccsd_tengy_c99.c:5-119 over f in HBM, one CTA per 16-wide tile
//    pair of a triple; a triple's last CTA sums the per-CTA partials in a fixed order.
//
// One triple is 8 (nvir/64)^2 tiles, less than one wave of the chip up to nvir = 300, so the plans run a batch
// of triples per launch; single-triple callers get 32-wide tiles where the 64-wide ones would leave SMs idle.

#include <type_traits>

#include "device_common.cuh"
#include "launch.h"

namespace trpdrv {
namespace plain {

constexpr int DK = 16;  // contraction indices per stage: two m16n8k8 steps, 128-byte X-major rows
constexpr int NTHREAD = 128;  // four warps, 2 x 2 over the tile

// Tile of BM x BM outputs.  K-major panels (rows of 16 contraction indices, BM + 2 doubles apart): the four lanes
// t of a group read rows 2t apart, and 2 (BM + 2) = 4 (mod 16) puts a half-warp's 64-bit reads in 16 different
// bank pairs.  X-major panels (one 128-byte row per column, 16-byte units XORed with the column mod 8): the
// quarter-warp's two columns are perm8(0) and perm8(1), ..., whose units never meet.
template <int BM> struct Tile {
    static constexpr int PK = BM + 2;
    static constexpr int APANEL = DK * PK;
    static constexpr int BPANEL = DK * PK > DK * BM ? DK * PK : DK * BM;
    static constexpr int STAGE = (APANEL + BPANEL + 15) / 16 * 16;
    static constexpr size_t smem(int stages) { return (size_t)stages * STAGE * sizeof(double); }
    static constexpr int MI = BM / 32, NI = BM / 16;  // m16 and n8 tiles per warp (BM / 2 square)
};

// Stages in flight: three where the CTAs of a batch share the SMs; four 32-wide ones for a single triple, six CTAs of
// which fit an SM, so that nvir = 300 (800 tiles) is one wave.
constexpr int BATCH_STAGES = 3;
template <int BM> constexpr int one_stages() { return BM == 32 ? 4 : 3; }

// Column that lane group g owns of its 8 (conflict-free X-major reads, see Tile).
__device__ __forceinline__ int perm8(int g) { return (0x53427160 >> (4 * g)) & 7; }

struct Src {
    const double *a, *b;
    int lda, ldb, bk, klim;  // bk: B is K-major (B(kk, c) = b[c + kk ldb]), else X-major (b[kk + c ldb])
};

template <int BM, int VEC>
__device__ __forceinline__ void load_stage(double *stage, const Src &s, int r0, int c0, int kk0, int nvir, int tid)
{
    using L = Tile<BM>;
    constexpr int CP = BM * DK / VEC;  // copies per panel
    static_assert(CP % NTHREAD == 0, "copies must split evenly over the CTA");
    auto kmajor = [&](double *panel, const double *src, int ld, int x0) {
#pragma unroll
        for (int u = 0; u < CP / NTHREAD; ++u) {
            const int q = tid + u * NTHREAD, kk = q / (BM / VEC), x = (q % (BM / VEC)) * VEC;
            const bool ok = (x0 + x < nvir) && (kk0 + kk < s.klim);
            const double *p = ok ? src + (x0 + x) + (size_t)(kk0 + kk) * ld : src;
            if (VEC == 2)
                cp_async_16(panel + kk * L::PK + x, p, ok);
            else
                cp_async_8(panel + kk * L::PK + x, p, ok);
        }
    };
    kmajor(stage, s.a, s.lda, r0);
    double *bst = stage + L::APANEL;
    if (s.bk) {
        kmajor(bst, s.b, s.ldb, c0);
        return;
    }
#pragma unroll
    for (int u = 0; u < CP / NTHREAD; ++u) {
        const int q = tid + u * NTHREAD, c = q / (DK / VEC), d = (q % (DK / VEC)) * VEC;
        const bool ok = (c0 + c < nvir) && (kk0 + d < s.klim);
        const double *p = ok ? s.b + (kk0 + d) + (size_t)(c0 + c) * s.ldb : s.b;
        double *w = bst + c * DK + (((d >> 1) ^ (c & 7)) << 1) + (d & 1);
        if (VEC == 2)
            cp_async_16(w, p, ok);
        else
            cp_async_8(w, p, ok);
    }
}

// A thread's copies of one panel over the chunks with DK valid contraction indices: the sources advance by a constant.
// Addresses and bounds worked out per copy were most of the loop's instructions beside the products (tensor pipe active
// 72 % of the time, L2 19 %, so neither traffic nor arithmetic bounds the loop).
template <int BM, int VEC>
struct Copies {
    static constexpr int U = BM * DK / VEC / NTHREAD;
    const double *p;  // the first copy's source; the others are `next` apart
    size_t next, advance;
    int dst, dnext, n;  // n: copies inside the tensor
    Copies() = default;
    // x0: first row (column) of the panel; there is at least one such chunk
    __device__ __forceinline__ Copies(const double *src, int ld, bool kmajor, int x0, int nvir, int tid)
    {
        const int W = kmajor ? BM / VEC : DK / VEC, lo = (tid % W) * VEC, hi = tid / W, step = NTHREAD / W;
        // K-major: lo a row, hi a contraction index; X-major: lo a contraction index, hi a column
        const int x = x0 + (kmajor ? lo : hi);
        n = kmajor ? (x < nvir ? U : 0) : (x < nvir ? min(U, (nvir - x + step - 1) / step) : 0);
        p = n > 0 ? src + (kmajor ? x + (size_t)hi * ld : lo + (size_t)x * ld) : src;
        next = (size_t)step * ld;
        advance = kmajor ? (size_t)DK * ld : DK;
        dst = kmajor ? hi * Tile<BM>::PK + lo : hi * DK + (((lo >> 1) ^ (hi & 7)) << 1) + (lo & 1);
        dnext = step * (kmajor ? Tile<BM>::PK : DK);  // X-major: columns a multiple of 8 apart, the same swizzle
    }
    __device__ __forceinline__ void issue(double *panel)
    {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const double *s = u < n ? p + u * next : p;
            if (VEC == 2)
                cp_async_16(panel + dst + u * dnext, s, u < n);
            else
                cp_async_8(panel + dst + u * dnext, s, u < n);
        }
        if (n > 0) p += advance;
    }
};

// One chunk's products.  FULL: every m16 and n8 tile of the warp has valid outputs; else only the first mi_n, ni_n.
template <int BM, bool BK, bool FULL>
__device__ __forceinline__ void chunk(const double *As, const double *Bs, int wm, int wn, int g, int t, int steps,
                                      bool neg, int mi_n, int ni_n, double (&acc)[Tile<BM>::MI][Tile<BM>::NI][4])
{
    using L = Tile<BM>;
    const int pc = perm8(g);
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
        if (ks == 1 && steps < 2) break;
        const int kk = ks * 8 + 2 * t;
        double a[L::MI][4], b[L::NI][2];
#pragma unroll
        for (int mi = 0; mi < L::MI; ++mi) {
            if (!FULL && mi >= mi_n) break;
            const double *p = As + kk * L::PK + wm + mi * 16 + g;
            a[mi][0] = p[0];
            a[mi][1] = p[8];
            a[mi][2] = p[L::PK];
            a[mi][3] = p[L::PK + 8];
            if (neg)
#pragma unroll
                for (int e = 0; e < 4; ++e) a[mi][e] = -a[mi][e];
        }
#pragma unroll
        for (int ni = 0; ni < L::NI; ++ni) {
            if (!FULL && ni >= ni_n) break;
            const int c = wn + ni * 8 + pc;
            if (BK) {
                b[ni][0] = Bs[kk * L::PK + c];
                b[ni][1] = Bs[(kk + 1) * L::PK + c];
            } else {
                const double2 v = *reinterpret_cast<const double2 *>(Bs + c * DK + (((kk >> 1) ^ (c & 7)) << 1));
                b[ni][0] = v.x;
                b[ni][1] = v.y;
            }
        }
#pragma unroll
        for (int mi = 0; mi < L::MI; ++mi)
#pragma unroll
            for (int ni = 0; ni < L::NI; ++ni) {
                if (!FULL && (mi >= mi_n || ni >= ni_n)) continue;
                dmma_16x8x8(acc[mi][ni], a[mi], b[ni]);
            }
    }
}

struct BatchArgs {
    trpdrv_dev_system S;  // by value: the kernels read the triple list and the tensors through it
    long long pos0;       // first record of the batch
    double *f;
    double *block_partial;  // [triple][pairs][4]
    unsigned *counter;      // [triple], zero
};

struct Triple {
    int i, j, k, ai;
    size_t vi, vk;  // offsets of the i and k vectors
};

__device__ __forceinline__ Triple batch_triple(const BatchArgs &B, int n)
{
    const long long r = B.pos0 + n, ai = r / B.S.nt;  // records are [a][triple]
    const int pk = B.S.triples[r - ai * B.S.nt];
    Triple t;
    t.i = pk & 1023;
    t.j = (pk >> 10) & 1023;
    t.k = (pk >> 20) & 1023;
    t.ai = (int)ai;
    t.vi = ((size_t)ai * B.S.nocc + t.i) * B.S.nvir;
    t.vk = ((size_t)ai * B.S.nocc + t.k) * B.S.nvir;
    return t;
}

// Operands of f_x of the batch's triple n; false where f_x is not computed (i == k: the t family is the n family).
__device__ __forceinline__ bool batch_sources(const BatchArgs &B, int n, int x, Src (&ph)[2])
{
    const trpdrv_dev_system &S = B.S;
    const Triple t = batch_triple(B, n);
    if (x >= 4 && t.i == t.k) return false;
    const size_t vv = (size_t)S.nvir * S.nvir, ov = (size_t)S.nocc * S.nvir;
    const int ia = x < 4 ? t.i : t.k, ib = x < 4 ? t.k : t.i;
    const size_t jb = (size_t)t.j * S.nocc + ib, ao = (size_t)t.ai * S.nocc + ia;
    const int two = (x >> 1) & 1;  // f3, f4
    ph[0].a = ((x & 1) ? S.kvv : S.jvv) + ao * vv;
    ph[0].b = S.t2 + jb * vv;
    ph[0].bk = !two;
    ph[1].a = ((x & 1) ? S.nxov : S.ntov) + (size_t)ia * ov;
    ph[1].b = (two ? S.jov : S.kov) + jb * ov;
    ph[0].lda = ph[0].ldb = ph[1].lda = S.nvir;
    ph[1].ldb = S.nocc;
    return true;
}

__device__ __forceinline__ bool one_sources(const trpdrv_plain_args &P, int x, Src (&ph)[2])
{
    ph[0].a = P.a1[x];
    ph[0].b = P.b1[x];
    ph[0].bk = P.b1_nt[x];
    ph[1].a = P.a2[x];
    ph[1].b = P.b2[x];
    ph[0].lda = P.lda1[x];
    ph[0].ldb = P.ldb1[x];
    ph[1].lda = P.lda2[x];
    ph[1].ldb = P.ldb2[x];
    return true;
}

template <int BM, int VEC, int STAGES, bool BATCH, bool FAST>
__device__ __forceinline__ void gemm_body(const trpdrv_plain_args *one, const BatchArgs *batch, int nvir, int nocc,
                                          double *fbase, bool neg)
{
    using L = Tile<BM>;
    extern __shared__ __align__(16) double smem[];
    const int x = blockIdx.z & 7, n = blockIdx.z >> 3;
    const int r0 = blockIdx.x * BM, c0 = blockIdx.y * BM;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp & 1) * (BM / 2), wn = (warp >> 1) * (BM / 2);
    const int g = lane >> 2, t = lane & 3;

    Src ph[2];
    if (!(BATCH ? batch_sources(*batch, n, x, ph) : one_sources(*one, x, ph))) return;
    ph[0].klim = nvir;
    ph[1].klim = nocc;
    ph[1].bk = 0;
    const int nV = (nvir + DK - 1) / DK, nO = (nocc + DK - 1) / DK, nch = nV + nO;
    const int nfull = FAST ? nvir / DK : 0;  // chunks copied by running pointers, their products without branches
    Copies<BM, VEC> ca, cb;
    if (FAST) {
        ca = Copies<BM, VEC>(ph[0].a, ph[0].lda, true, r0, nvir, tid);
        cb = Copies<BM, VEC>(ph[0].b, ph[0].ldb, ph[0].bk, c0, nvir, tid);
    }
    auto load = [&](int ch, double *st) {
        if (FAST && ch < nfull) {
            ca.issue(st);
            cb.issue(st + L::APANEL);
        } else if (ch < nch) {
            if (ch < nV)
                load_stage<BM, VEC>(st, ph[0], r0, c0, ch * DK, nvir, tid);
            else
                load_stage<BM, VEC>(st, ph[1], r0, c0, (ch - nV) * DK, nvir, tid);
        }
        cp_async_commit();
    };

    double acc[L::MI][L::NI][4];
#pragma unroll
    for (int mi = 0; mi < L::MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < L::NI; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[mi][ni][e] = 0.0;
    // m16 and n8 tiles of this warp that hold valid outputs
    const int mr = nvir - (r0 + wm), nc = nvir - (c0 + wn);
    int mi_n = mr <= 0 ? 0 : (mr + 15) >> 4, ni_n = nc <= 0 ? 0 : (nc + 7) >> 3;
    if (mi_n > L::MI) mi_n = L::MI;
    if (ni_n > L::NI) ni_n = L::NI;
    const bool whole = !FAST && mi_n == L::MI && ni_n == L::NI;

    double *ring = smem, *fill = smem;  // the stage to multiply and the stage to fill
    auto next = [&](double *st) { return st == smem + (STAGES - 1) * L::STAGE ? smem : st + L::STAGE; };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        load(s, fill);
        fill = next(fill);
    }
    int ch = 0;
    auto step = [&](auto products) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        load(ch + STAGES - 1, fill);
        fill = next(fill);
        products(ring, ring + L::APANEL);
        ring = next(ring);
        ++ch;
    };
    // the chunks of the K = nvir product without a branch among their products
    auto fast = [&](auto bk, auto full) {
#pragma unroll 1
        while (ch < nfull)
            step([&](const double *As, const double *Bs) {
                chunk<BM, decltype(bk)::value, decltype(full)::value>(As, Bs, wm, wn, g, t, 2, false, mi_n, ni_n, acc);
            });
    };
    if (FAST && r0 + BM <= nvir && c0 + BM <= nvir)  // the whole CTA: its warps take the same loop
        ph[0].bk ? fast(std::true_type{}, std::true_type{}) : fast(std::false_type{}, std::true_type{});
#pragma unroll 1
    while (ch < nch) {
        const bool virt = ch < nV;
        const int steps = (virt ? nvir - ch * DK : nocc - (ch - nV) * DK) > 8 ? 2 : 1;
        step([&](const double *As, const double *Bs) {
            if (mi_n <= 0 || ni_n <= 0) return;
            if (whole && virt && ph[0].bk)
                chunk<BM, true, true>(As, Bs, wm, wn, g, t, steps, false, 0, 0, acc);
            else if (whole)
                chunk<BM, false, true>(As, Bs, wm, wn, g, t, steps, neg && !virt, 0, 0, acc);
            else if (virt && ph[0].bk)
                chunk<BM, true, false>(As, Bs, wm, wn, g, t, steps, false, mi_n, ni_n, acc);
            else
                chunk<BM, false, false>(As, Bs, wm, wn, g, t, steps, neg && !virt, mi_n, ni_n, acc);
        });
    }
    cp_async_wait<0>();
    // a batch's products overlap the energies of the batch before; its f goes to the same buffer only after them
    if (BATCH) asm volatile("griddepcontrol.wait;" ::: "memory");

    double *f = fbase + ((size_t)n * 8 + x) * nvir * nvir;
#pragma unroll
    for (int mi = 0; mi < L::MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < L::NI; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = r0 + wm + mi * 16 + g + ((e & 2) ? 8 : 0), c = c0 + wn + ni * 8 + perm8(2 * t + (e & 1));
                if (r < nvir && c < nvir) f[r + (size_t)c * nvir] = acc[mi][ni][e];
            }
}

template <int BM, int VEC, bool FAST>
__global__ void __launch_bounds__(NTHREAD, BM == 64 ? 3 : 6) plain_gemm_kernel(const __grid_constant__ trpdrv_plain_args args)
{
    // the dependent tengy launch may start its prologue (it waits for this grid before reading f)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (args.counter && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x) == 0) *args.counter = 0u;
    gemm_body<BM, VEC, one_stages<BM>(), false, FAST>(&args, nullptr, args.nvir, args.nocc, args.f, args.neg2 != 0);
}

template <int BM, int VEC, bool FAST>
__global__ void __launch_bounds__(NTHREAD, BM == 64 ? 3 : 5) plain_batch_kernel(const __grid_constant__ BatchArgs args)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    gemm_body<BM, VEC, BATCH_STAGES, true, FAST>(nullptr, &args, args.S.nvir, args.S.nocc, args.f, false);
}

// ------------------------------------------------------------------------------------------------
// energies
// ------------------------------------------------------------------------------------------------
constexpr int TW = 16;  // tile width
constexpr int TNTHREAD = TW * TW;

struct TengyIn {
    const double *fn, *ft;  // the four f of the n and of the t family
    const double *ev;       // virtual orbital energies
    const double *dintc1, *dintx1, *t1v1, *dintc2, *dintx2, *t1v2;
    double eaijk;
    double *partial, *out;
    unsigned *counter;
};

// The per-index vectors of a tile pair, rows of 16 at b and then at c: loaded together with f.  Loaded by each thread
// after the exchange instead they cost a second round trip to L2 (20, 200: 30.8 against 30.3 ms for all triples, a
// single triple 19.8 against 18.7 us).
constexpr int TVROWS = 14;

__device__ __forceinline__ double vec_entry(const TengyIn &P, int row, int n)
{
    const int kind = row >= 7 ? row - 7 : row;
    const double *src = kind == 0 ? P.t1v1 : kind == 1 ? P.t1v2 : kind == 2 ? P.dintx1 : kind == 3 ? P.dintx2
                      : kind == 4 ? P.dintc1 : kind == 5 ? P.dintc2 : P.ev;
    return __ldg(src + n);
}

// One CTA: the terms of (b, c) and (c, b) over a 16-wide tile pair B <= C, one thread per (b, c).  Both tiles of all
// eight f are read with 128-byte coalesced loads, 16 independent ones per thread; the (c, b) values cross
// through shared memory.  A latency-bound kernel (a single triple has 91 CTAs at nvir = 200): 16-wide tiles give
// four times the CTAs of 32-wide ones and one round of loads each.
// CHAIN: lets the next batch's products start.
template <bool CHAIN>
__device__ __forceinline__ void tengy_body(const TengyIn &P, int nvir)
{
    __shared__ double xch[8][TW][TW + 1], vsh[TVROWS][TW];
    __shared__ double red[4 * (TNTHREAD / 32)];
    __shared__ int s_last;
    const int nb = (nvir + TW - 1) / TW, tid = threadIdx.x;
    int B = 0, rem = blockIdx.x;
    while (B < nb && rem >= nb - B) {
        rem -= nb - B;
        ++B;
    }
    const int C = B + rem, r = tid & (TW - 1), q = tid / TW;
    const bool diag = B == C;
    const int b = B * TW + r, c = C * TW + q;    // this thread's (b, c)
    const int cr = C * TW + r, bq = B * TW + q;  // the mirrored tile's element it loads
    const size_t vv = (size_t)nvir * nvir;
    const int vrow = tid / TW, vn = (vrow < 7 ? B : C) * TW + r;
    const double ve = vrow < TVROWS && vn < nvir ? vec_entry(P, vrow, vn) : 0.0;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // f (and a single triple's counter) come from the launch before
    if (CHAIN) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    double fbc[8], fcb[8];
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const double *f = (x < 4 ? P.fn + x * vv : P.ft + (x - 4) * vv);
        fbc[x] = b < nvir && c < nvir ? __ldcg(f + b + (size_t)c * nvir) : 0.0;
        fcb[x] = !diag && cr < nvir && bq < nvir ? __ldcg(f + cr + (size_t)bq * nvir) : 0.0;
    }
#pragma unroll
    for (int x = 0; x < 8; ++x) xch[x][q][r] = diag ? fbc[x] : fcb[x];
    if (vrow < TVROWS) vsh[vrow][r] = ve;
    __syncthreads();
    TengySums su = {0.0, 0.0, 0.0, 0.0};
    if (b < nvir && c < nvir) {
#pragma unroll
        for (int x = 0; x < 8; ++x) fcb[x] = xch[x][r][q];
        const double denom = -1.0 / (vsh[6][r] + vsh[13][q] + P.eaijk);
        const TengyIdx ib = {vsh[0][r], vsh[1][r], vsh[2][r], vsh[3][r], vsh[4][r], vsh[5][r]};
        const TengyIdx ic = {vsh[7][q], vsh[8][q], vsh[9][q], vsh[10][q], vsh[11][q], vsh[12][q]};
        tengy_pair(!diag, fbc, fcb, denom, ib, ic, su);
    }
    const TengySums tot = block_sum4(su, red);
    if (tid == 0) {
        double *bp = P.partial + 4 * (size_t)blockIdx.x;
        bp[0] = tot.e4i;
        bp[1] = tot.e5i;
        bp[2] = tot.e4k;
        bp[3] = tot.e5k;
        __threadfence();
        s_last = atomicAdd(P.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    TengySums all = {0.0, 0.0, 0.0, 0.0};
    for (unsigned blk = tid; blk < gridDim.x; blk += TNTHREAD) {
        const double *bp = P.partial + 4 * (size_t)blk;
        all.e4i += __ldcg(bp + 0);
        all.e5i += __ldcg(bp + 1);
        all.e4k += __ldcg(bp + 2);
        all.e5k += __ldcg(bp + 3);
    }
    const TengySums sum = block_sum4(all, red);
    if (tid == 0) {
        P.out[0] = sum.e4i;
        P.out[1] = sum.e5i;
        P.out[2] = sum.e4k;
        P.out[3] = sum.e5k;
        *P.counter = 0u;
    }
}

__global__ void __launch_bounds__(TNTHREAD) tengy_kernel(const __grid_constant__ trpdrv_tengy_args a)
{
    TengyIn P;
    P.fn = a.f;
    P.ft = a.f + 4 * (size_t)a.nvir * a.nvir;
    P.ev = a.eorb + a.ncor + a.nocc;
    P.dintc1 = a.dintc1;
    P.dintx1 = a.dintx1;
    P.t1v1 = a.t1v1;
    P.dintc2 = a.dintc2;
    P.dintx2 = a.dintx2;
    P.t1v2 = a.t1v2;
    // omp/ccsd_trpdrv_omp_cbody.c:126
    P.eaijk = a.use_eaijk ? a.eaijk
                          : a.eorb[a.a - 1] - (a.eorb[a.ncor + a.i - 1] + a.eorb[a.ncor + a.j - 1] +
                                               a.eorb[a.ncor + a.k - 1]);
    P.partial = a.block_partial;
    P.out = a.out4;
    P.counter = a.counter;
    tengy_body<false>(P, a.nvir);
}

// Four CTAs per SM (64 registers): a CTA waits on its 16 loads, a division and the sums more than it computes.  39 triples of
// nvir = 200 took 47 us with three, all triples of nocc = 20 30.3 against 29.6 ms.
__global__ void __launch_bounds__(TNTHREAD, 4) tengy_batch_kernel(const __grid_constant__ BatchArgs a)
{
    const trpdrv_dev_system &S = a.S;
    const int n = blockIdx.y;
    const Triple t = batch_triple(a, n);
    TengyIn P;
    P.fn = a.f + (size_t)n * 8 * S.nvir * S.nvir;
    P.ft = t.i == t.k ? P.fn : P.fn + 4 * (size_t)S.nvir * S.nvir;
    P.ev = S.eorb + S.ncor + S.nocc;
    P.dintc1 = S.dintc + t.vi;
    P.dintx1 = S.dintx + t.vi;
    P.t1v1 = S.t1v + t.vi;
    P.dintc2 = S.dintc + t.vk;
    P.dintx2 = S.dintx + t.vk;
    P.t1v2 = S.t1v + t.vk;
    P.eaijk = S.eorb[S.a - 1 + t.ai] - (S.eorb[S.ncor + t.i] + S.eorb[S.ncor + t.j] + S.eorb[S.ncor + t.k]);
    P.partial = a.block_partial + (size_t)n * gridDim.x * 4;
    P.out = S.rec + 4 * (a.pos0 + n);
    P.counter = a.counter + n;
    tengy_body<true>(P, S.nvir);
}

// 64-wide tiles where they fill the chip once over (two CTAs per SM) and cover not much more than 32-wide ones:
// at equal padding they are 4 to 12 % faster (nvir = 300, 250, 111), with 1.31 times the area 13 % slower
// (nvir = 200: 35.8 against 31.6 ms for all triples of nocc = 20).
constexpr int SMS = 148;  // of a B200
bool wide_tiles(int nvir, long long triples)
{
    const long long n64 = (nvir + 63) / 64, n32 = (nvir + 31) / 32;
    return n64 * n64 * 8 * triples >= 2 * SMS && 100 * 4 * n64 * n64 <= 115 * n32 * n32;
}

// Running pointers where their set-up pays, from eight copies a thread and panel of 32 rows on: nvir >= 64, or 32 if the
// copies are of 8 bytes.
// All triples, ms without and with: (20, 200) 29.63, 28.2; (8, 300) 5.15, 4.91; (17, 111) 4.40, 4.15; (30, 33) 3.67, 3.37;
// (12, 100) 1.21, 1.18, but (10, 60) 0.155, 0.161 and (16, 16) 0.100, 0.107.
bool fast_copies(int nvir, int vec2) { return nvir / DK * (vec2 ? 2 : 4) >= 8; }

// f(<BM, VEC, FAST>)
template <class F>
int with_variant(bool wide, int vec2, int nvir, F f)
{
    using W = std::integral_constant<int, 64>;
    using N = std::integral_constant<int, 32>;
    using V1 = std::integral_constant<int, 1>;
    using V2 = std::integral_constant<int, 2>;
    using Yes = std::true_type;
    using No = std::false_type;
    const bool fast = fast_copies(nvir, vec2);
    if (wide) return !vec2 ? f(W{}, V1{}, Yes{}) : fast ? f(W{}, V2{}, Yes{}) : f(W{}, V2{}, No{});  // nvir > 32
    if (fast) return vec2 ? f(N{}, V2{}, Yes{}) : f(N{}, V1{}, Yes{});
    return vec2 ? f(N{}, V2{}, No{}) : f(N{}, V1{}, No{});
}

template <int BM, int VEC, bool FAST>
int set_smem()
{
    cudaError_t e = cudaFuncSetAttribute(plain_gemm_kernel<BM, VEC, FAST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)Tile<BM>::smem(one_stages<BM>()));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(plain_batch_kernel<BM, VEC, FAST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Tile<BM>::smem(BATCH_STAGES));
    return (int)e;
}

template <int BM, int VEC, bool FAST>
int launch_one(const trpdrv_plain_args &a, cudaStream_t st)
{
    const unsigned nbt = (a.nvir + BM - 1) / BM;
    plain_gemm_kernel<BM, VEC, FAST><<<dim3(nbt, nbt, 8), NTHREAD, Tile<BM>::smem(one_stages<BM>()), st>>>(a);
    return (int)cudaGetLastError();
}

// dependent: a programmatic dependent launch, scheduled while the launch before it on the stream drains.
template <class A>
int launch(void (*kernel)(const A), dim3 grid, int threads, size_t smem, bool dependent, const A &args, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = dependent ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, kernel, args);
}

template <int BM, int VEC, bool FAST>
int launch_batch(const BatchArgs &a, int n, bool dependent, cudaStream_t st)
{
    const unsigned nbt = (a.S.nvir + BM - 1) / BM;
    return launch(plain_batch_kernel<BM, VEC, FAST>, dim3(nbt, nbt, 8 * n), NTHREAD, Tile<BM>::smem(BATCH_STAGES), dependent, a, st);
}

}  // namespace plain
}  // namespace trpdrv

using namespace trpdrv;

extern "C" int trpdrv_launch_plain_gemm(const trpdrv_plain_args *args, int vec2, void *stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    return plain::with_variant(plain::wide_tiles(args->nvir, 1), vec2, args->nvir, [&](auto bm, auto vec, auto fast) {
        return plain::launch_one<decltype(bm)::value, decltype(vec)::value, decltype(fast)::value>(*args, st);
    });
}

extern "C" int64_t trpdrv_tengy_pairs(int nvir)
{
    const int64_t nb = (nvir + plain::TW - 1) / plain::TW;
    return nb * (nb + 1) / 2;
}

extern "C" int trpdrv_launch_tengy(const trpdrv_tengy_args *args, void *stream)
{
    return plain::launch(plain::tengy_kernel, dim3((unsigned)trpdrv_tengy_pairs(args->nvir)), plain::TNTHREAD, 0, true,
                         *args, (cudaStream_t)stream);
}

// Enough triples for several waves of tiles, as long as their f (written by one launch, read by the next) stay in
// L2: 96 MB of its 126 MB, at least one triple.  (20, 200): 37.1 ms with 48 MB, 35.8 with 96 (64-wide tiles).
extern "C" int trpdrv_plain_batch(int nvir)
{
    const long long per = 8LL * nvir * nvir * 8, fit = (96LL << 20) / per;
    return (int)(fit < 1 ? 1 : fit > 256 ? 256 : fit);
}

extern "C" int trpdrv_launch_plain_batch(const trpdrv_dev_system *h_sys, int64_t pos0, int n, double *f,
                                         double *block_partial, unsigned *counter, int vec2, int chained,
                                         void *stream)
{
    if (n <= 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    plain::BatchArgs a;
    a.S = *h_sys;
    a.pos0 = pos0;
    a.f = f;
    a.block_partial = block_partial;
    a.counter = counter;
    const int e = plain::with_variant(plain::wide_tiles(h_sys->nvir, n), vec2, h_sys->nvir, [&](auto bm, auto vec, auto fast) {
        return plain::launch_batch<decltype(bm)::value, decltype(vec)::value, decltype(fast)::value>(a, n, chained, st);
    });
    if (e) return e;
    return plain::launch(plain::tengy_batch_kernel, dim3((unsigned)trpdrv_tengy_pairs(h_sys->nvir), (unsigned)n),
                         plain::TNTHREAD, 0, true, a, st);
}

extern "C" int trpdrv_plain_init(void)
{
    int e = plain::set_smem<64, 1, true>();
    if (!e) e = plain::set_smem<64, 2, true>();
    if (!e) e = plain::set_smem<64, 2, false>();
    if (!e) e = plain::set_smem<32, 1, true>();
    if (!e) e = plain::set_smem<32, 2, true>();
    if (!e) e = plain::set_smem<32, 1, false>();
    if (!e) e = plain::set_smem<32, 2, false>();
    return e;
}
