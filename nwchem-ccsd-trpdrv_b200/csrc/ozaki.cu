// Emulated-FP64 form of the triples body (sm_100a): Ozaki splitting of every contraction into int8
// digit slices on the 5th-generation tensor cores, exact int32 accumulation in tensor memory, FP64
// recombination; energy denominators and sums stay in native FP64.
//
// Each of the eight f of a triple is one contraction over d = [virtual | occupied]
// (omp/ccsd_trpdrv_omp_cbody.c:70-117 with the occupied A operand negated, as in the fused kernels).
// The emulation:
//  * every row of an A operand and every column of a B operand is scaled by a power of two 2^e chosen
//    so that its largest element has magnitude in [1/4, 1/2), then written as S signed base-128
//    digits x = 2^e * sum_{p=1..S} d_p 2^(-7p) with |d_p| <= 64 (each digit rounded to nearest, so the
//    remainder after S digits is at most 2^(e-7S-1));
//  * products of digit slices with p + q <= S + 1 are accumulated on the tensor cores
//    (tcgen05.mma kind::i8, int32 accumulators in TMEM).  Pairs with equal p + q carry the same
//    weight and share one accumulator; |sum| <= S * dp * 64 * 64 < 2^31, so the integer sums are exact;
//  * the S level sums are recombined in FP64: f = 2^(eA + eB) * sum_L 2^(-7L) C_L.
// f of a batch of triples go to a device buffer and become energies in FP64 (omp/ccsd_tengy_c99.c:5-119): for even nvir
// beside the next batch's products, in their launch, else in a launch of their own.
//
// Operand slices (int8, contraction index d contiguous, zero-padded to dp, a multiple of 32):
//   SA[x][p][r][d]:      r < V: [J(x) | -TOV(x)] row r;       r >= V: [K(x) | -XOV(x)] row r - V
//   SB[j*O+y][p][c][d]:  c < V: [T2[j][y]^T ; KOV[j][y]] col c; c >= V: [T2[j][y] ; JOV[j][y]] col c - V
// The n-group of triple (i, j, k) is SA[i] x SB[j,k] and its t-group SA[k] x SB[j,i]; the 2V x 2V
// product [A1; A2] [B1 | B3] holds the four f of the group in its quadrants:
//   f1n = A1 B1, f2n = A2 B1, f3n = A1 B3, f4n = A2 B3 (and f1t..f4t likewise).
//
// Contraction kernel: persistent, one CTA per SM walking 128 x 64 output tiles of the batch's products.
//   warp 0       TMA loads (64-byte swizzle) of all S digit slices of A and B, 64 contraction indices a stage; runs ahead
//                across tiles
//   warp 1       allocates tensor memory and issues every MMA (M=128, N=64, K=32) into S level accumulators (S*64
//                columns)
//   warp 2       the energies' operands: triples, per-index vectors, f by TMA
//   warps 4-11   wait for a tile's last MMA, join its levels, release the accumulators to the next tile, then
//                scale and store in FP64 while that tile's MMAs run
//   warps 12-15  energies
// Every wait is bounded (globaltimer) and reports through *status; tensor memory is released on every path.
//
// What bounds it: the int8 products take 32 cycles each at best and 35 as issued, 9.8 kclk of a tile of 7 slices and
// 320 contraction indices; a tile takes 15.6 (13.9 without the energies, 12 without the operands' loads as well).
// The accumulators fill tensor memory, so nothing overlaps their drain (1.7 kclk), and shared memory is nearly
// saturated: 84 KB read by the 28 products of a K step and 42 KB written, in 980 cycles.  7 slices, all
// triples, ms at (nocc, nvir) = (12, 300), (10, 400), (20, 200): 7.79, 9.17, 15.8 with each MMA issued under `lane == 0`;
// 7.28, 8.45, 14.4 under elect.sync; 6.55, 8.06, 13.0 with scales added to exponents and shorter code; 6.5, 7.9, 12.7 with
// the levels joined in integers; 5.8, 7.5, 11.8 with the energies' operands prepared by a warp of its own.

#include <cuda.h>
#include <cudaTypedefs.h>

#include "device_common.cuh"
#include "launch.h"
#include "tengy_tile.cuh"

namespace trpdrv {
namespace oz {

constexpr int BM = 128;         // output rows per tile (TMEM lanes)
constexpr int BN = 64;          // output columns per tile (TMEM columns per level)
constexpr int KC = 64;          // contraction bytes (= int8 indices) per stage
constexpr int KSTEP = 32;       // contraction indices per MMA
constexpr int NREC = 8;         // recombination warps: two per TMEM lane quadrant, 32 columns each
constexpr int NENG = 4;         // energy warps (energies fused into the launch)
// Warpgroup 0: warp 0 TMA, warp 1 MMA + TMEM, warp 2 the energies' operands (warp 3 idle); warpgroups 1, 2 (warps 4 .. 11)
// recombination; warpgroup 3 (warps 12 .. 15) energies.
constexpr int REC0 = 4, ENG0 = REC0 + NREC;
constexpr int NTHREAD = 32 * (ENG0 + NENG);
// Register split by setmaxnreg: launched at 65536 / 512 = 128 per thread, the recombination
// warpgroups rise to 168 (their drain spills below that), the others drop.
constexpr int REG_LAUNCH = 128, REG_CTRL = 72, REG_REC = 168, REG_ENG = 104;
static_assert(128 * REG_CTRL + 256 * REG_REC + 128 * REG_ENG <= NTHREAD * REG_LAUNCH, "register split exceeds the launch");
constexpr unsigned SLICE_A = BM * KC;
constexpr unsigned SLICE_B = BN * KC;
constexpr int SMEM_AVAIL = 227 * 1024 - 1024;  // less the alignment of the stages
constexpr unsigned long long WAIT_LIMIT_NS = 4000000000ull;

// fused energies: the f of half a tile pair (16 b x 8 c), both orientations of the eight f, 8 KB each
constexpr unsigned HALF_BYTES = 2u * 8u * 16u * 8u * 8u;

template <int S>
struct Cfg {
    static constexpr unsigned STAGE = S * (SLICE_A + SLICE_B);
    // two stages or more beside three half-pair buffers of the energies (and 4 KB of static variables), else, for 8
    // slices, beside two (and 2 KB)
    static constexpr int FIT3 = (SMEM_AVAIL - 4096 - 3 * (int)HALF_BYTES) / (int)STAGE;
    static constexpr int FIT2 = (SMEM_AVAIL - 2048 - 2 * (int)HALF_BYTES) / (int)STAGE;
    static constexpr int HALVES = FIT3 >= 2 ? 3 : 2;
    static constexpr int STAGES = FIT3 >= 2 ? (FIT3 > 4 ? 4 : FIT3) : FIT2;
    static constexpr size_t SMEM = (size_t)STAGES * STAGE + (size_t)HALVES * HALF_BYTES + 1024;
    static constexpr unsigned TMEM_COLS = S * BN <= 256 ? 256u : 512u;
    static_assert(STAGES >= 2, "fewer than two stages fit");
    static_assert(S * BN <= 512, "level accumulators exceed tensor memory");
};

// instruction descriptor, kind::i8: D s32 (bits 4-5 = 2), A and B signed (bits 7-9, 10-12 = 1),
// both K-major (bits 15, 16 = 0), N >> 3 at bits 17-22, M >> 4 at bits 24-28
constexpr unsigned IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(BN >> 3) << 17) |
                           ((unsigned)(BM >> 4) << 24);

struct GemmParams {
    CUtensorMap mapA, mapB;  // 64-byte aligned members first
    CUtensorMap fbc, fcb;    // fused energies: efbuf as {V rows (contiguous), V columns, 8 * enpos planes}, in
                             // boxes of 16 rows x 8 columns (at (b,c)) and 8 rows x 16 columns (at (c,b))
    trpdrv_dev_system sys;   // fused energies: vectors, triples and energy slots of the system
    const double *ea, *eb;   // power-of-two scales per A row / B column
    const int32_t *triples, *order;
    const int32_t *jobs;     // this batch's (position, group) products: position << 1 | group
    long long pos0, ntriples, nt;  // ntriples records = n_a * nt triples per a
    double *fbuf;            // [batch][8][V][ldf]
    // fused energies: the energies of positions epos0 .. epos0 + enpos - 1, whose f an earlier launch
    // stored (at the maps' base); unit u = tile pair u % np of position epos0 + u / np
    long long epos0;
    int enpos, np;
    int V, O, ldf, nks, mtiles, ntiles, tiles;  // tiles = jobs * mtiles * ntiles
    int *status;
};

// ------------------------------------------------------------------------------------------------
// PTX helpers
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned saddr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(unsigned long long *b, unsigned count)
{
    asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(saddr(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *b, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(saddr(b)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *b, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(saddr(b)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait; false (and status bit 1) when it runs out.
__device__ __forceinline__ bool mbar_wait_for(unsigned long long *b, unsigned parity, int *status,
                                              unsigned long long limit_ns)
{
    if (mbar_try_wait(b, parity)) return true;
    const unsigned long long t0 = globaltimer();
    for (;;) {
#pragma unroll 1
        for (int spin = 0; spin < 256; ++spin)
            if (mbar_try_wait(b, parity)) return true;
        if (globaltimer() - t0 > limit_ns) {
            atomicOr(status, 2);
            return false;
        }
    }
}

__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned parity, int *status)
{
    return mbar_wait_for(b, parity, status, WAIT_LIMIT_NS);
}

// The wait of a whole converged warp that goes on to instructions all of its lanes take part in (elect.sync,
// tcgen05.ld, __syncwarp): every lane polls by its own clock, so one may give up in the moment in which the phase
// completes for the others.  The same answer in all lanes, or part of the warp would wait at the CTA's last barrier
// and the rest, for it, inside the loop.
__device__ __forceinline__ bool mbar_wait_warp_for(unsigned long long *b, unsigned parity, int *status,
                                                   unsigned long long limit_ns)
{
    return __all_sync(0xffffffffu, mbar_wait_for(b, parity, status, limit_ns));
}

__device__ __forceinline__ bool mbar_wait_warp(unsigned long long *b, unsigned parity, int *status)
{
    return mbar_wait_warp_for(b, parity, status, WAIT_LIMIT_NS);
}

// L2 cache policies for loads and stores: evict_last for data read again soon (the digit planes, reused
// across the tiles and triples that share them), evict_first for data read once
__device__ __forceinline__ unsigned long long policy_evict_last()
{
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

__device__ __forceinline__ unsigned long long policy_evict_first()
{
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

__device__ __forceinline__ void tma_load_3d_hint(void *dst, const CUtensorMap *map, unsigned long long *bar, int x,
                                                 int y, int z, unsigned long long pol)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, "
        "%4, %5}], [%2], %6;" ::"r"(saddr(dst)),
        "l"(map), "r"(saddr(bar)), "r"(x), "r"(y), "r"(z), "l"(pol)
        : "memory");
}

__device__ __forceinline__ void tmem_alloc(unsigned *dst, unsigned ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(dst)), "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(unsigned taddr, unsigned ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major operand tile in shared memory with the 64-byte swizzle: rows of 64 bytes, 8-row atoms of
// 512 bytes (stride byte offset 512), leading byte offset unused (1), descriptor version 1.
__device__ __forceinline__ unsigned long long sdesc_sw64(const void *p)
{
    const unsigned a = saddr(p);
    return (unsigned long long)((a >> 4) & 0x3FFFu) | (1ull << 16) | ((unsigned long long)(512 >> 4) << 32) |
           (1ull << 46) | (4ull << 61);
}

// True in one lane of the converged warp.  The branch it guards is compiled with warp-uniform operands: a
// tcgen05.mma then takes its descriptors from uniform registers.  Under an ordinary `lane == 0` the compiler
// moves every operand there instruction by instruction, and one thread issues an MMA every 44.7 cycles whatever
// its N (16 to 80); under elect, every 22.6 (N = 32) and, at N = 64, every 35.1 against 32 of the tensor pipe.
__device__ __forceinline__ bool elect_one()
{
    unsigned r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
    return r != 0;
}

// A-operand collector buffer use of one MMA: the first MMA of a run that shares its A tile fills the
// buffer, the following ones read A from it instead of shared memory, the last one releases it.
enum { COL_DISCARD = 0, COL_FILL = 1, COL_USE = 2, COL_LASTUSE = 3 };

__device__ __forceinline__ void mma_i8(unsigned d, unsigned long long a, unsigned long long b, int accumulate,
                                       int col = COL_DISCARD)
{
#define OZ_MMA_I8(Q)                                                                                          \
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"                                                 \
                 " tcgen05.mma.cta_group::1.kind::i8" Q " [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n}\n" ::"r"(d), \
                 "l"(a), "l"(b), "r"(IDESC), "r"(accumulate), "r"(0), "r"(0), "r"(0), "r"(0)                 \
                 : "memory")
    if (col == COL_FILL)
        OZ_MMA_I8(".collector::a::fill");
    else if (col == COL_USE)
        OZ_MMA_I8(".collector::a::use");
    else if (col == COL_LASTUSE)
        OZ_MMA_I8(".collector::a::lastuse");
    else
        OZ_MMA_I8("");
#undef OZ_MMA_I8
}

// collector use of the q-th of n MMAs in a row that share one A tile
__host__ __device__ constexpr int collector_op(int q, int n)
{
    return n == 1 ? COL_DISCARD : q == 0 ? COL_FILL : q == n - 1 ? COL_LASTUSE : COL_USE;
}

__device__ __forceinline__ void mma_commit(unsigned long long *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar))
                 : "memory");
}

// 32 lanes x 16 columns of 32 bits into v (valid only after tmem_wait_ld and reg_fence16)
__device__ __forceinline__ void tmem_ld16_nowait(unsigned taddr, unsigned (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Orders every use of v after the preceding tcgen05.wait::ld (volatile asm keeps its place in
// program order, and the registers pass through it).
__device__ __forceinline__ void reg_fence16(unsigned (&v)[16])
{
    asm volatile(""
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]),
                   "+r"(v[15]));
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *b)
{
    asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(saddr(b)) : "memory");
}

// Self-test of mbar_wait_warp: warp 1 completes the phase after twice the limit that half of warp 0's lanes have; the
// others would wait on.  All lanes of warp 0 must give up together (status bit 3: they did not).
__global__ void warp_wait_selftest_kernel(unsigned long long limit_ns, int *status)
{
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int local;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        local = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x >= 32) {
        const unsigned long long t0 = globaltimer();
        while (globaltimer() - t0 < 2 * limit_ns) {
        }
        if (lane == 0) mbar_arrive(&bar);
        return;
    }
    const bool done = mbar_wait_warp_for(&bar, 0u, &local, lane < 16 ? limit_ns : 64 * limit_ns);
    if (done) atomicOr(status, 8);
}

// weight of level L (0-based, slices p + q = L + 2 in 1-based digits): 2^(-7 (L + 2)), exact
__device__ __forceinline__ double level_weight(int L)
{
    double w = 1.0 / 16384.0;
    for (int l = 0; l < L; ++l) w *= 1.0 / 128.0;
    return w;
}

// ------------------------------------------------------------------------------------------------
constexpr int TW = 16;
constexpr size_t TSMEM_BYTES = (size_t)16 * TW * (TW + 1) * sizeof(double);
// TMA form: the eight f tiles of one orientation arrive as one 16 x 16 x 8 box with the 128-byte swizzle; both
// orientations take 32 KB on a 1024-byte boundary.  Odd nvir too: f's columns are padded to an even length.
constexpr int TBOX = TW * TW * 8;  // doubles of one orientation
constexpr size_t TSMEM_TMA_BYTES = (size_t)2 * TBOX * sizeof(double) + 1024;
// Threads of a CTA of the separate energy launch (at most 96 registers, five CTAs per SM).  The energies of one batch
// are launched on a second stream after its contraction launch; since the contraction kernel holds every
// register of its SMs (512 threads x 128), they run on the SMs it has left, between its launches.
constexpr int TNTHREAD = 128;

struct TengyItem {
    int i, j, k, pairi, y, b0, c0;
    bool diag;
    unsigned ai;
    long long tt;
};

// Geometry of work item (16-wide tile pair, batch position y after pos0), from indices alone; false for
// positions past the end of the system.
__device__ __forceinline__ bool tengy_geom(const trpdrv_dev_system &S, long long pos0, int pairi, int y,
                                           TengyItem &it)
{
    if (pos0 + y >= S.ntriples || S.nt <= 0) return false;
    const int nb = (S.nvir + TW - 1) / TW;
    int B = 0, rem = pairi;
    while (B < nb && rem >= nb - B) {
        rem -= nb - B;
        ++B;
    }
    it.pairi = pairi;
    it.y = y;
    it.b0 = B * TW;
    it.c0 = (B + rem) * TW;
    it.diag = rem == 0;
    return true;
}

// The item's triple (its record and indices); false for a malformed queue entry.
__device__ __forceinline__ bool tengy_triple(const trpdrv_dev_system &S, long long pos0, TengyItem &it)
{
    const long long pos = pos0 + it.y;  // a position over the records ([a][triple])
    it.ai = pos >= S.nt ? (unsigned)pos / (unsigned)S.nt : 0u;  // records < 2^31
    const long long tpos = pos - (long long)it.ai * S.nt;
    it.tt = S.order ? (long long)S.order[tpos] : tpos;
    if (it.tt < 0 || it.tt >= S.nt) return false;
    const int packed = S.triples[it.tt];
    it.i = packed & 1023;
    it.j = (packed >> 10) & 1023;
    it.k = (packed >> 20) & 1023;
    return true;
}

__device__ __forceinline__ bool tengy_decode(const trpdrv_dev_system &S, long long pos0, int pairi, int y,
                                             TengyItem &it)
{
    return tengy_geom(S, pos0, pairi, y, it) && tengy_triple(S, pos0, it);
}

// The vectors and eaijk of an item's triple.
__device__ __forceinline__ TengyVecs tengy_vecs(const trpdrv_dev_system &S, const TengyItem &it)
{
    const int nvir = S.nvir;
    TengyVecs v;
    v.eorb = S.eorb;
    const size_t ao = (size_t)it.ai * S.nocc;  // the a block of the a-dependent vectors
    v.dintc1 = S.dintc + (ao + it.i) * nvir;
    v.dintx1 = S.dintx + (ao + it.i) * nvir;
    v.t1v1 = S.t1v + (ao + it.i) * nvir;
    v.dintc2 = S.dintc + (ao + it.k) * nvir;
    v.dintx2 = S.dintx + (ao + it.k) * nvir;
    v.t1v2 = S.t1v + (ao + it.k) * nvir;
    v.voff = S.ncor + S.nocc;
    v.nvir = nvir;
    // omp/ccsd_trpdrv_omp_cbody.c:126 (a is 1-based, i/j/k here 0-based)
    v.eaijk = S.eorb[S.a - 1 + it.ai] - (S.eorb[S.ncor + it.i] + S.eorb[S.ncor + it.j] + S.eorb[S.ncor + it.k]);
    return v;
}

// The per-index vectors of an item in shared memory, rows of 16: t1v(i), t1v(k), dintx(i), dintx(k),
// dintc(i), dintc(k), e_virt at b0 + r (rows 0 .. 6), then the same at c0 + q (rows 7 .. 13); zero
// past nvir.  Loaded by the CTA while the item's f tiles are in flight.
constexpr int TVROWS = 14;
__device__ __forceinline__ void tengy_stage_vecs(const TengyVecs &v, const TengyItem &it, double *vsh, int tid,
                                                 int nthreads)
{
    for (int idx = tid; idx < TVROWS * TW; idx += nthreads) {
        const int row = idx / TW, x = idx % TW, side = row / 7, kind = row % 7;
        const int n = (side ? it.c0 : it.b0) + x;
        const double *src = kind == 0 ? v.t1v1 : kind == 1 ? v.t1v2 : kind == 2 ? v.dintx1 : kind == 3 ? v.dintx2
                          : kind == 4 ? v.dintc1 : kind == 5 ? v.dintc2 : v.eorb + v.voff;
        vsh[idx] = n < v.nvir ? __ldg(src + n) : 0.0;
    }
}

// The item's four energy slots (e4i, e5i, e4k, e5k).
__device__ __forceinline__ double *tengy_slot(const trpdrv_dev_system &S, const TengyItem &it)
{
    return S.partial + ((size_t)((long long)it.ai * S.nt + it.tt) * S.npairs * TRPDRV_FUSED_SLOTS + it.pairi) * 4;
}

// number of 16-wide tile pairs (must fit in the npairs * TRPDRV_FUSED_SLOTS slots of a triple)
__host__ __device__ inline int tengy_pairs(int nvir)
{
    const int nb = (nvir + TW - 1) / TW;
    return nb * (nb + 1) / 2;
}


// ------------------------------------------------------------------------------------------------
// energies fused into the contraction kernel: those of the positions whose f the launch before stored, beside
// this launch's products
// ------------------------------------------------------------------------------------------------
constexpr int NENG_THREADS = 32 * NENG;

// named barrier 1 over the energy warps (barrier 0 is the CTA's)
__device__ __forceinline__ void eng_bar() { asm volatile("bar.sync 1, %0;" ::"n"(NENG_THREADS) : "memory"); }

// the energy barrier, true in every thread when p is true in any
__device__ __forceinline__ bool eng_bar_or(bool p)
{
    unsigned r;
    asm volatile("{\n .reg .pred a, b;\n setp.ne.u32 a, %1, 0;\n bar.red.or.pred b, 1, %2, a;\n selp.u32 %0, 1, 0, b;\n}\n"
                 : "=r"(r)
                 : "r"((unsigned)p), "n"(NENG_THREADS)
                 : "memory");
    return r != 0;
}

// The fused energies of a CTA: the contiguous range u0 .. u1 of the tile pairs B <= C (16-wide) of the positions
// whose f an earlier launch stored.  Warp 2 looks up each pair's triple, loads its per-index vectors and copies its f in
// two halves of 16 b x 8 c into a ring of NBUF buffers; the energy warps find everything in shared memory.
// Done by the energy warps themselves, the lookups (dependent loads) took 2.8 of the 9 kclk of a pair, and
// with one buffer of 32 KB nothing of the next pair could be in flight meanwhile.
struct EnergyUnit {  // of one tile pair
    double vec[TVROWS * TW];  // as tengy_stage_vecs
    double eaijk;
    double *slot;  // the pair's four energies; null: a malformed queue entry
    int b0, c0;
};

template <int NBUF>
struct EnergyRing {
    static constexpr int NUNIT = NBUF >= 3 ? 2 : 1;  // tables
    unsigned long long full[NBUF], empty[NBUF];
    EnergyUnit unit[NUNIT];
    double red[NUNIT][4 * (NENG - 1)];  // the sums of the energy warps but the first
    __device__ __forceinline__ void init()
    {
        for (int q = 0; q < NBUF; ++q) {
            mbar_init(&full[q], 32);     // every lane of warp 2, and the bytes
            mbar_init(&empty[q], NENG);  // one arrival per energy warp
        }
    }
};

__device__ __forceinline__ void energy_range(const GemmParams &P, unsigned &u0, unsigned &u1)
{
    const unsigned total = (unsigned)P.enpos * (unsigned)P.np, per = (total + gridDim.x - 1) / gridDim.x;
    u0 = min(total, blockIdx.x * per);
    u1 = min(total, u0 + per);
}

// Warp 2, all lanes.
template <int NBUF>
__device__ __forceinline__ void energy_operands(const GemmParams &P, char *bufs, EnergyRing<NBUF> &R, int lane)
{
    constexpr int PER = TVROWS * TW / 32;  // vector entries per lane
    static_assert(TVROWS * TW % 32 == 0, "vector entries per lane");
    const trpdrv_dev_system &S = P.sys;
    unsigned u0, u1;
    energy_range(P, u0, u1);
    if (u0 >= u1) return;
    const int nb = (S.nvir + TW - 1) / TW;
    const unsigned long long pol = policy_evict_first();
    TengyItem it;
    it.y = (int)(u0 / (unsigned)P.np);
    it.pairi = (int)(u0 % (unsigned)P.np);
    int B = 0, C = it.pairi;
    while (B < nb - 1 && C >= nb - B) C -= nb - B++;
    C += B;
    bool valid = false, fresh = true;  // of the triple; fresh: a position not looked up yet
    TengyVecs v;
    int q = 0;
    unsigned phase = 1;
    for (unsigned u = u0; u < u1; ++u) {
        if (fresh) {
            valid = P.epos0 + it.y < S.ntriples && S.nt > 0 && tengy_triple(S, P.epos0, it);
            if (valid) v = tengy_vecs(S, it);
            fresh = false;
        }
        const int b0 = B * TW, c0 = C * TW;
        double x[PER];
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int idx = lane + 32 * e, row = idx / TW, side = row / 7, kind = row % 7, n = (side ? c0 : b0) + idx % TW;
            const double *src = kind == 0 ? v.t1v1 : kind == 1 ? v.t1v2 : kind == 2 ? v.dintx1 : kind == 3 ? v.dintx2
                              : kind == 4 ? v.dintc1 : kind == 5 ? v.dintc2 : v.eorb + v.voff;
            x[e] = valid && n < S.nvir ? __ldg(src + n) : 0.0;
        }
#pragma unroll 1
        for (int hf = 0; hf < 2; ++hf) {
            if (!mbar_wait(&R.empty[q], phase, P.status)) return;
            if (hf == 0) {
                // The table's last readers are done: with three buffers, since this one was freed by the pair before
                // the last (both of whose halves lie before it); with two, once the pair before has freed the other.
                if (NBUF == 2 && !mbar_wait(&R.empty[1], phase, P.status)) return;
                EnergyUnit &t = R.unit[R.NUNIT == 2 ? (u - u0) & 1 : 0];
#pragma unroll
                for (int e = 0; e < PER; ++e) t.vec[lane + 32 * e] = x[e];
                if (lane == 0) {
                    t.eaijk = valid ? v.eaijk : 0.0;
                    t.slot = valid ? tengy_slot(S, it) : nullptr;
                    t.b0 = b0;
                    t.c0 = c0;
                }
            }
            if (lane == 0) {
                char *dst = bufs + (size_t)q * HALF_BYTES;
                // this buffer's previous reads (generic proxy) before the tensor-copy writes
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_arrive_expect_tx(&R.full[q], HALF_BYTES);
                tma_load_3d_hint(dst, &P.fbc, &R.full[q], b0, c0 + 8 * hf, it.y * 8, pol);
                tma_load_3d_hint(dst + HALF_BYTES / 2, &P.fcb, &R.full[q], c0 + 8 * hf, b0, it.y * 8, pol);
            } else
                mbar_arrive(&R.full[q]);
            if (++q == NBUF) {
                q = 0;
                phase ^= 1u;
            }
        }
        ++it.pairi;
        if (++C == nb) {
            if (++B == nb) {
                B = 0;
                ++it.y;
                it.pairi = 0;
                fresh = true;
            }
            C = B;
        }
    }
}

// The energy warps (te = 0 .. NENG_THREADS - 1), one (b, c) of a half a thread.  Every wait is bounded; one that runs
// out ends the loop in all threads.
template <int NBUF>
__device__ __forceinline__ void fused_energies(const GemmParams &P, const char *bufs, EnergyRing<NBUF> &R, int te)
{
    unsigned u0, u1;
    energy_range(P, u0, u1);
    const int V = P.sys.nvir, lane = te & 31, we = te >> 5;
    // (r, c) of this thread within a half: c = cc ^ (r >> 3) keeps the half-warp's reads of both boxes free of bank
    // conflicts (16 rows of 128 bytes, 128-byte swizzle; lines of 64 bytes, 64-byte swizzle)
    const int r = te & 15, c = (te >> 4) ^ (r >> 3);
    const int o1 = c * 128 + (((r >> 1) ^ c) << 4) + ((r & 1) << 3);
    const int o2 = (int)(HALF_BYTES / 2) + r * 64 + (((c >> 1) ^ ((r >> 1) & 3)) << 4) + ((c & 1) << 3);
    int q = 0;
    unsigned phase = 0;
    bool ok = true;
    for (unsigned u = u0; u < u1; ++u) {
        const EnergyUnit &t = R.unit[R.NUNIT == 2 ? (u - u0) & 1 : 0];
        TengySums su = {0.0, 0.0, 0.0, 0.0};
        double *slot = nullptr;
#pragma unroll 1
        for (int hf = 0; hf < 2; ++hf) {
            ok = ok && mbar_wait(&R.full[q], phase, P.status);
            if (ok) {
                slot = t.slot;
                const int cc = 8 * hf + c;
                if (slot && t.b0 + r < V && t.c0 + cc < V) {
                    const char *p = bufs + (size_t)q * HALF_BYTES;
                    double fbc[8], fcb[8];
#pragma unroll
                    for (int x = 0; x < 8; ++x) {
                        fbc[x] = *reinterpret_cast<const double *>(p + o1 + x * 1024);
                        fcb[x] = *reinterpret_cast<const double *>(p + o2 + x * 1024);
                    }
                    const double *vb = t.vec + r, *vc = t.vec + 7 * TW + cc;
                    const TengyIdx ib = {vb[0], vb[TW], vb[2 * TW], vb[3 * TW], vb[4 * TW], vb[5 * TW]};
                    const TengyIdx ic = {vc[0], vc[TW], vc[2 * TW], vc[3 * TW], vc[4 * TW], vc[5 * TW]};
                    const double denom = -1.0 / (vb[6 * TW] + vc[6 * TW] + t.eaijk);
                    tengy_pair(t.b0 != t.c0, fbc, fcb, denom, ib, ic, su);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&R.empty[q]);
            if (++q == NBUF) {
                q = 0;
                phase ^= 1u;
            }
        }
        double *red = R.red[R.NUNIT == 2 ? (u - u0) & 1 : 0];
        const double s = warp_sum4(su, lane), s0 = __shfl_sync(0xffffffffu, s, 8 * (lane & 3));
        if (we > 0 && (lane & 7) == 0) red[4 * (we - 1) + (lane >> 3)] = s;
        if (eng_bar_or(!ok)) return;  // also: the sums are in place
        if (te < 4 && slot) {  // fixed order: the sums do not depend on which CTA ran the pair
            double e = s0;
            for (int w = 0; w < NENG - 1; ++w) e += red[4 * w + te];
            slot[te] = e;
        }
        if (R.NUNIT == 1) eng_bar();  // else the next pair's sums go to the other half of red
    }
}

// ------------------------------------------------------------------------------------------------
// contraction kernel (persistent: CTA b takes tiles b, b + grid, ...)
// ------------------------------------------------------------------------------------------------
struct Tile {
    int ok, y, grp, same, planeA, planeB, m0, n0;  // y: batch position; same: i == k (the t group is the n group)
};

__device__ __forceinline__ Tile decode_tile(const GemmParams &P, int t)
{
    Tile d;
    const int per = P.mtiles * P.ntiles;
    const int job = t / per, rem = t - job * per;
    d.m0 = (rem % P.mtiles) * BM;
    d.n0 = (rem / P.mtiles) * BN;
    const int jb = P.jobs[job];
    d.grp = jb & 1;
    const long long pos = jb >> 1;  // a position over the records ([a][triple])
    d.y = (int)(pos - P.pos0);
    // records < 2^31 (the host checks): 32-bit division, none for a single a
    const unsigned ai = (P.nt > 0 && pos >= P.nt) ? (unsigned)pos / (unsigned)P.nt : 0u;
    const long long tpos = pos - (long long)ai * P.nt;
    const long long tt = (pos < P.ntriples) ? (P.order ? (long long)P.order[tpos] : tpos) : -1;
    const int packed = (tt >= 0 && tt < P.nt) ? P.triples[tt] : -1;
    const int i = packed & 1023, j = (packed >> 10) & 1023, k = (packed >> 20) & 1023;
    d.ok = packed >= 0 && i < P.O && j < P.O && k < P.O;
    d.same = i == k;
    d.planeA = (int)ai * P.O + (d.grp ? k : i);  // the A operands carry the a index
    d.planeB = j * P.O + (d.grp ? i : k);
    return d;
}

// Draining.  The next tile's products wait until the accumulators have been read, so as little as possible happens
// before they are released; and the roles' code together must stay within the instruction caches, beside
// which everything but the products ran at half its speed or less.  Two forms, by the width dp of the contraction
// (|C_l| <= (l + 1) dp 64^2):
//   SUM64:  all levels joined in int64, two adjacent ones in int32 first (128 C_l + C_{l+1}), converted after the
//           release (dp <= sum64_limit(S): 504 for 7 slices, no width for 8)
//   GROUPS: levels 0 .. 3 and 4 .. S - 1 joined in int64, the two sums added in FP64
// Both round once, so they give the same bits: the integer sums are exact, a group's is below 2^53 (group_max_dp) and so
// exact in FP64, and only the addition of the second group rounds.
enum DrainForm { SUM64, GROUPS };

// The widest contraction whose pairs of levels stay below 2^31.
__host__ __device__ constexpr int pair_limit(int S)
{
    const int l = (S - 1) & ~1;               // first level of the last pair (or the last level alone)
    const int first = l + 1 < S ? l : l - 2;  // first level of the last complete pair
    return (int)((0x7fffffffLL - 1) / ((long long)(first + 1) * 4096 * 128 + (long long)(first + 2) * 4096));
}

__host__ __device__ constexpr int sum64_limit(int S)
{
    unsigned long long unit = 0;  // the largest |sum| of dp = 1
    for (int l = 0; l < S; ++l) unit = unit * 128 + (unsigned long long)(l + 1) * 4096;
    const unsigned long long lim = 0x7fffffffffffffffull / unit;
    return lim < (unsigned long long)pair_limit(S) ? (int)lim : pair_limit(S);
}

// The widest contraction whose groups of four levels stay below 2^53.
__host__ __device__ constexpr long long group_max_dp()
{
    return (1LL << 53) / (4096LL * (5LL * 128 * 128 * 128 + 6LL * 128 * 128 + 7LL * 128 + 8LL));  // levels 4 .. 7
}
static_assert(TRPDRV_MAX_NOCC + TRPDRV_MAX_NVIR + 32 <= group_max_dp(), "a group of four levels exceeds 53 bits");

// 16 columns at TMEM address base: sum_L C_L 2^(-7 (L + 2)); SUM64: the bits of the integer 2^(7 (S + 1)) times that.
template <int S, DrainForm FORM>
__device__ __forceinline__ void drain16(unsigned base, double (&val)[16])
{
    constexpr int GROUP = 4;
#pragma unroll
    for (int u = 0; u < 16; ++u) val[u] = 0.0;
#pragma unroll
    for (int g = 0; g < S; g += GROUP) {
        const int n = S - g < GROUP ? S - g : GROUP;
        unsigned v[GROUP][16];
#pragma unroll
        for (int l = 0; l < GROUP; ++l)
            if (l < n) tmem_ld16_nowait(base + (unsigned)((g + l) * BN), v[l]);
        tmem_wait_ld();
#pragma unroll
        for (int l = 0; l < GROUP; ++l)
            if (l < n) reg_fence16(v[l]);
        if (FORM == SUM64) {
#pragma unroll
            for (int l = 0; l < GROUP; l += 2) {
                if (l >= n) break;
                const bool two = l + 1 < n;
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    const int x = two ? (int)v[l][u] * 128 + (int)v[two ? l + 1 : l][u] : (int)v[l][u];
                    val[u] = __longlong_as_double(
                        g + l == 0 ? (long long)x : __double_as_longlong(val[u]) * (two ? 16384 : 128) + x);
                }
            }
        } else {
            const double w = level_weight(g + n - 1);
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                long long sum = (int)v[0][u];
#pragma unroll
                for (int l = 1; l < GROUP; ++l)
                    if (l < n) sum = sum * 128 + (int)v[l][u];
                val[u] = fma((double)sum, w, val[u]);
            }
        }
    }
}

__device__ __forceinline__ int scale_exp(double s) { return (__double2hiint(s) >> 20) - 1023; }  // s = 2^e, normal

// x 2^e by the exponent bits: x zero or normal, and so the result
__device__ __forceinline__ double scale_by_exp(double x, int e)
{
    const int hi = __double2hiint(x);
    return __hiloint2double((hi & 0x7ff00000) ? hi + (e << 20) : hi, __double2loint(x));
}

template <int S>
__global__ void __launch_bounds__(NTHREAD, 1) oz_gemm_kernel(const __grid_constant__ GemmParams P)
{
    using C = Cfg<S>;
    extern __shared__ char smem_raw[];
    __shared__ __align__(8) unsigned long long full[C::STAGES], empty[C::STAGES], tfull[1], tempty[1], done[1];
    __shared__ EnergyRing<C::HALVES> ering;
    __shared__ unsigned tmem_sh;
    // aligned by an offset, not by integer arithmetic on the pointer: the compiler then still knows that they
    // are shared memory
    char *stages = smem_raw + ((1024u - (saddr(smem_raw) & 1023u)) & 1023u);
    char *halves = stages + (size_t)C::STAGES * C::STAGE;  // 1024-byte aligned

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nchunks = (P.nks * KSTEP + KC - 1) / KC;

    if (tid == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(tfull, 1);
        mbar_init(tempty, NREC);  // one arrival per recombination warp
        mbar_init(done, 1);
        ering.init();
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(&tmem_sh, C::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_sh;

    // each role's code sits in the branch of its warpgroup's register change
    if (warp < REC0) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_CTRL));
      if (warp == 0) {
        if (lane == 0) {  // TMA producer: runs ahead across tiles, bounded by the stage ring
            const unsigned long long pol = policy_evict_last();
            int stage = 0;
            unsigned phase = 0;
            bool alive = true;
            for (int t = blockIdx.x; alive && t < P.tiles; t += gridDim.x) {
                const Tile d = decode_tile(P, t);
                if (!d.ok) {
                    atomicOr(P.status, 1);
                    continue;
                }
                for (int kc = 0; kc < nchunks; ++kc) {
                    if (!mbar_wait(&empty[stage], phase ^ 1, P.status)) {
                        alive = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&full[stage], C::STAGE);
                    char *sA = stages + (size_t)stage * C::STAGE, *sB = sA + S * SLICE_A;
                    // the digit planes are reused by the tiles and triples that share them: evict_last
#pragma unroll
                    for (int p = 0; p < S; ++p)
                        tma_load_3d_hint(sA + p * SLICE_A, &P.mapA, &full[stage], kc * KC, d.m0, d.planeA * S + p, pol);
#pragma unroll
                    for (int q = 0; q < S; ++q)
                        tma_load_3d_hint(sB + q * SLICE_B, &P.mapB, &full[stage], kc * KC, d.n0, d.planeB * S + q, pol);
                    if (++stage == C::STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        const unsigned long long dA0 = sdesc_sw64(stages), dB0 = sdesc_sw64(stages + S * SLICE_A);
        {  // MMA issuer: level L = p + q (0-based) accumulates at columns L*BN..
            int stage = 0;
            unsigned phase = 0;
            bool alive = true;
            int it = 0;
            for (int t = blockIdx.x; alive && t < P.tiles; t += gridDim.x, ++it) {
                const Tile d = decode_tile(P, t);
                // the accumulators are free once the previous tile has been drained
                if (!mbar_wait_warp(tempty, (it & 1) ^ 1, P.status)) break;
                tc_fence_after();
                if (d.ok) {
                    for (int kc = 0; kc < nchunks; ++kc) {
                        if (!mbar_wait_warp(&full[stage], phase, P.status)) {
                            alive = false;
                            break;
                        }
                        tc_fence_after();
                        const unsigned long long so = (unsigned long long)(stage * (int)(C::STAGE >> 4));
                        const unsigned long long dA = dA0 + so, dB = dB0 + so;
                        if (elect_one()) {
#pragma unroll 1
                        for (int ks = 0; ks < KC / KSTEP; ++ks) {
                            const int kg = kc * (KC / KSTEP) + ks;
                            if (kg < P.nks) {
#pragma unroll
                                for (int p = 0; p < S; ++p)
#pragma unroll
                                    for (int q = 0; p + q < S; ++q)  // S - p MMAs share A slice p
                                        mma_i8(tmem + (unsigned)((p + q) * BN),
                                               dA + (unsigned long long)(p * (SLICE_A >> 4) + ks * (KSTEP >> 4)),
                                               dB + (unsigned long long)(q * (SLICE_B >> 4) + ks * (KSTEP >> 4)),
                                               (kg > 0 || p > 0) ? 1 : 0, collector_op(q, S - p));
                            }
                        }
                        mma_commit(&empty[stage]);  // the stage is free once these MMAs have read it
                        }
                        __syncwarp();
                        if (++stage == C::STAGES) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                }
                if (elect_one()) mma_commit(tfull);  // this tile's sums are complete (or the tile was skipped)
            }
            if (it > 0) {  // a CTA with no tiles (an energies-only launch) issued nothing to wait for
                if (elect_one()) mma_commit(done);  // every MMA issued by this thread has completed when `done` flips
                mbar_wait(done, 0, P.status);
            }
        }
        __syncwarp();
      } else if (warp == 2 && P.enpos > 0)
        energy_operands<C::HALVES>(P, halves, ering, lane);
    } else if (warp < ENG0) {  // recombination: TMEM lanes 32*(warp%4).., columns 32*half..
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REG_REC));
        const int qd = warp & 3, half = (warp - REC0) >> 2;
        constexpr int WC = BN / 2;  // columns per recombination warp
        constexpr bool SUM64_FITS = sum64_limit(S) >= KSTEP;  // the narrowest contraction; false for 8 slices
        const int V = P.V;
        const size_t vv = (size_t)V * P.ldf;
        int it = 0;
        for (int t = blockIdx.x; t < P.tiles; t += gridDim.x, ++it) {
            const Tile d = decode_tile(P, t);
            // the exponents of the tile's scales, before its products are complete: this lane's row, and this lane's
            // column of the 32
            const int r = d.m0 + qd * 32 + lane, lcol = d.n0 + half * WC + lane;
            int esa = d.ok && r < 2 * V ? scale_exp(P.ea[(size_t)d.planeA * 2 * V + r]) : 0;
            int esb = d.ok && lcol < 2 * V ? scale_exp(P.eb[(size_t)d.planeB * 2 * V + lcol]) : 0;
            if (!mbar_wait_warp(tfull, it & 1, P.status)) break;
            tc_fence_after();
            const int rh = r >= V ? 1 : 0, b = r - rh * V;
            double *fj = P.fbuf + (size_t)d.y * 8 * vv + (size_t)d.grp * 4 * vv + (size_t)rh * vv + b;
            const bool row_ok = d.ok && r < 2 * V;
            const unsigned base = tmem + ((unsigned)(qd * 32) << 16) + (unsigned)(half * WC);
            double val[WC / 16][16];
            const int dp = P.nks * KSTEP;
            const bool sum64 = SUM64_FITS && dp <= sum64_limit(S);
            if (sum64) {
#pragma unroll
                for (int cb = 0; cb < WC / 16; ++cb) drain16<S, SUM64>(base + (unsigned)(cb * 16), val[cb]);
            } else {
#pragma unroll
                for (int cb = 0; cb < WC / 16; ++cb) drain16<S, GROUPS>(base + (unsigned)(cb * 16), val[cb]);
            }
            // the accumulators may be overwritten by the next tile from here on
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty);
            if (!d.ok) continue;
            int e0 = 0;
            if (sum64) {
                e0 = -7 * (S + 1);
#pragma unroll
                for (int cb = 0; cb < WC / 16; ++cb)
#pragma unroll
                    for (int u = 0; u < 16; ++u) val[cb][u] = (double)__double_as_longlong(val[cb][u]);
            }
            // the scales as integer additions to the exponent: exact while every result is a normal number
            if (!__all_sync(0xffffffffu, esa >= -450 && esa <= 450 && esb >= -450 && esb <= 450)) {
                const double sa = row_ok ? P.ea[(size_t)d.planeA * 2 * V + r] : 0.0, w0 = e0 ? level_weight(S - 1) : 1.0;
#pragma unroll
                for (int c = 0; c < WC; ++c) {
                    const int col = d.n0 + half * WC + c;
                    val[c / 16][c % 16] = val[c / 16][c % 16] * w0 * sa;
                    if (col < 2 * V) val[c / 16][c % 16] *= P.eb[(size_t)d.planeB * 2 * V + col];
                }
                esa = esb = e0 = 0;
            }
            e0 += esa;
            double *dst = fj + (size_t)(d.n0 + half * WC) * P.ldf;
#pragma unroll
            for (int cb = 0; cb < WC / 16; ++cb)
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    const int c = cb * 16 + u, col = d.n0 + half * WC + c;
                    const double x = scale_by_exp(val[cb][u], e0 + __shfl_sync(0xffffffffu, esb, c));
                    if (row_ok && col < 2 * V) {
                        // column col - V of f3, f4 (two planes further) from column V on
                        double *q = dst + (col >= V ? 2 * vv - (size_t)V * P.ldf : 0);
                        __stcs(q, x);  // evict-first: read once, by a later launch; keeps the digits in L2
                        if (d.same) __stcs(q + 4 * vv, x);
                    }
                    dst += P.ldf;
                }
        }
    } else {  // energy warps: the units of the positions an earlier launch stored
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_ENG));
        if (P.enpos > 0) fused_energies<C::HALVES>(P, halves, ering, tid - 32 * ENG0);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, C::TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------------
// slicing: power-of-two scale per row and S base-128 digits per element
// ------------------------------------------------------------------------------------------------
struct SliceParams {
    const double *t2, *jvv, *kvv, *ntov, *nxov, *jov, *kov;
    signed char *out;  // [planes][S][2V][dp]
    double *scale;     // [planes][2V]
    int V, O, S, dp;
};

// One element of row r of plane `plane`; A side (SIDE 0) or B side (SIDE 1).
template <int SIDE>
__device__ __forceinline__ double slice_src(const SliceParams &P, int plane, int r, int d)
{
    const int V = P.V, O = P.O;
    const int h = r >= V ? 1 : 0, x = r - h * V;
    const size_t vv = (size_t)V * V, ov = (size_t)O * V;
    if (SIDE == 0) {
        if (d < V) return (h ? P.kvv : P.jvv)[plane * vv + x + (size_t)d * V];
        return (h ? P.nxov : P.ntov)[(size_t)(plane % O) * ov + x + (size_t)(d - V) * V];  // shared over a
    }
    if (d < V) return h ? P.t2[plane * vv + d + (size_t)x * V] : P.t2[plane * vv + x + (size_t)d * V];
    return (h ? P.jov : P.kov)[plane * ov + (d - V) + (size_t)x * O];
}

// whether row index is the contiguous one in memory for this tile (coalescing only)
template <int SIDE>
__device__ __forceinline__ bool slice_rows_contiguous(const SliceParams &P, int r0, int d0)
{
    if (SIDE == 0) return true;
    return r0 < P.V && d0 < P.V;
}

template <int SIDE>
__device__ __forceinline__ void slice_load(const SliceParams &P, int plane, int r0, int d0, double (*tile)[33],
                                           int tid)
{
    const int D = P.V + P.O, R = 2 * P.V;
    const bool rc = slice_rows_contiguous<SIDE>(P, r0, d0);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int idx = tid + 256 * e;
        const int rr = rc ? (idx & 31) : (idx >> 5), dd = rc ? (idx >> 5) : (idx & 31);
        const int r = r0 + rr, d = d0 + dd;
        tile[rr][dd] = (r < R && d < D) ? slice_src<SIDE>(P, plane, r, d) : 0.0;
    }
}

template <int SIDE>
__global__ void __launch_bounds__(256) oz_slice_kernel(const SliceParams P)
{
    __shared__ double tile[32][33];
    const int tid = threadIdx.x, row = tid >> 3, part = tid & 7;
    const int plane = blockIdx.y, r0 = blockIdx.x * 32;
    const int D = P.V + P.O, R = 2 * P.V;

    double mx = 0.0;
    for (int d0 = 0; d0 < D; d0 += 32) {
        slice_load<SIDE>(P, plane, r0, d0, tile, tid);
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 4; ++u) mx = fmax(mx, fabs(tile[row][part * 4 + u]));
        __syncthreads();
    }
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
    int e = 0;
    if (mx > 0.0) {
        frexp(mx, &e);  // mx = m 2^e, m in [1/2, 1)
        e += 1;         // mx 2^-e in [1/4, 1/2)
    }
    const double inv = ldexp(1.0, -e);
    const int r = r0 + row;
    if (part == 0 && r < R) P.scale[(size_t)plane * R + r] = ldexp(1.0, e);

    for (int d0 = 0; d0 < P.dp; d0 += 32) {
        slice_load<SIDE>(P, plane, r0, d0, tile, tid);
        __syncthreads();
        unsigned w[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            double x = tile[row][part * 4 + u] * inv;  // exact: power-of-two scaling
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                if (p < P.S) {
                    const double t = x * 128.0;
                    const double dg = rint(t);  // |dg| <= 64 since |x| <= 1/2
                    x = t - dg;                 // exact, |x| <= 1/2
                    w[p] |= ((unsigned)(int)dg & 0xffu) << (8 * u);
                }
            }
        }
        if (r < R) {
#pragma unroll
            for (int p = 0; p < 8; ++p)
                if (p < P.S)
                    *reinterpret_cast<unsigned *>(P.out + (((size_t)plane * P.S + p) * R + r) * P.dp + d0 + part * 4) =
                        w[p];
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------------
// batched tengy over the f of a batch: one CTA per (16-wide tile pair, triple), six or more CTAs per
// SM.  A CTA's four sums go to its own slot of the triple's items (slot index = tile-pair index; the
// 16-wide pairs fit in the 8 slots of each 32-wide item, and the slots no CTA writes are zero from
// plan creation), so records_kernel sums them in a fixed order.
struct TengyParams {
    CUtensorMap fmap;  // TMA form: fbuf as {nvir rows (contiguous), nvir columns, 8 * npos planes}
    trpdrv_dev_system sys;
    long long pos0;
    const double *fbuf;
    int *status;  // bit 1: a wait for the tiles ran out (the item's energies are not written)
};

// cp.async form: park f(B,C) (o = 0) and f(C,B) (o = 1) tiles of all eight f, W x (W + 1) doubles
// each; column q of a tile is contiguous in f.  Every copy of a thread is issued before any is
// waited for (zero fill outside nvir), so that a CTA keeps its whole 32 KB in flight.
__device__ __forceinline__ void tengy_park_cpasync(const TengyParams &P, const TengyItem &it, double *park)
{
    constexpr int TP = TW + 1, TILE = TW * TP;
    const int nvir = P.sys.nvir, ldf = trpdrv_oz_ldf(nvir);
    const size_t lnvv = (size_t)nvir * ldf;
    const double *f = P.fbuf + (size_t)it.y * 8 * lnvv;
    const int ntiles = it.diag ? 8 : 16;
    for (int idx = threadIdx.x; idx < ntiles * TW * TW; idx += TNTHREAD) {
        const int tile = idx / (TW * TW), q = (idx / TW) % TW, r = idx % TW;
        const int o = tile >> 3, xf = tile & 7;
        const int row = (o ? it.c0 : it.b0) + r, col = (o ? it.b0 : it.c0) + q;
        const bool ok = row < nvir && col < nvir;
        cp_async_8(park + tile * TILE + r * TP + q, ok ? f + (size_t)xf * lnvv + row + (size_t)col * ldf : f, ok);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
}

// Energies of one item from its tiles parked by cp.async, summed over the CTA into its slot.
__device__ __forceinline__ void tengy_finish(const TengyParams &P, const TengyItem &it, const double *park, double *red)
{
    const int tid = threadIdx.x;
    const TengyVecs v = tengy_vecs(P.sys, it);
    TengySums su = {0.0, 0.0, 0.0, 0.0};
    tengy_tile_pair_factored<TW>(park, it.b0, it.c0, it.diag, v, tid, TNTHREAD, su);
    const TengySums tot = block_sum4(su, red);
    if (tid == 0) {  // block_sum4's result is valid in thread 0
        double *out = tengy_slot(P.sys, it);
        out[0] = tot.e4i;
        out[1] = tot.e5i;
        out[2] = tot.e4k;
        out[3] = tot.e5k;
    }
    __syncthreads();  // the park and the reduction scratch are reused by the CTA's next item
}

// CTA b takes items b, b + grid, ... (the launches use one CTA per item).
template <bool TMA>
__global__ void __launch_bounds__(TNTHREAD, 5) oz_tengy_kernel(const __grid_constant__ TengyParams P, int np, int npos)
{
    extern __shared__ __align__(16) double tsmem[];
    __shared__ double red[4 * (TNTHREAD / 32)];
    __shared__ __align__(8) unsigned long long tbar[1];
    double *park = TMA ? tsmem + ((1024u - (saddr(tsmem) & 1023u)) & 1023u) / sizeof(double) : tsmem;
    if (TMA) {
        if (threadIdx.x == 0) {
            mbar_init(tbar, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
    }
    unsigned phase = 0;
    const long long items = (long long)np * npos;
    for (long long w = blockIdx.x; w < items; w += gridDim.x) {
        TengyItem it;
        if (TMA) {  // the tiles' coordinates need no loads: copies first, the triple and vectors meanwhile
            __shared__ double vsh[TVROWS * TW];
            if (!tengy_geom(P.sys, P.pos0, (int)(w % np), (int)(w / np), it)) continue;  // uniform over the CTA
            if (threadIdx.x == 0) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_arrive_expect_tx(tbar, (it.diag ? 1u : 2u) * (unsigned)(TBOX * sizeof(double)));
                const unsigned long long pol = policy_evict_first();
                tma_load_3d_hint(park, &P.fmap, tbar, it.b0, it.c0, it.y * 8, pol);
                if (!it.diag) tma_load_3d_hint(park + TBOX, &P.fmap, tbar, it.c0, it.b0, it.y * 8, pol);
            }
            const bool valid = tengy_triple(P.sys, P.pos0, it);  // the same in every thread
            TengyVecs v;
            if (valid) {
                v = tengy_vecs(P.sys, it);
                tengy_stage_vecs(v, it, vsh, threadIdx.x, TNTHREAD);
            }
            const bool ok = mbar_wait(tbar, phase, P.status);
            phase ^= 1;
            if (__syncthreads_or(!ok)) return;  // status bit 1 is set
            if (!valid) {
                __syncthreads();  // the park is free again
                continue;
            }
            TengySums su = {0.0, 0.0, 0.0, 0.0};
            tengy_tile_pair_swz16_sv<TNTHREAD>(park, vsh, it.b0, it.c0, it.diag, v.nvir, v.eaijk, threadIdx.x, su);
            const TengySums tot = block_sum4(su, red);
            if (threadIdx.x == 0) {
                double *out = tengy_slot(P.sys, it);
                out[0] = tot.e4i;
                out[1] = tot.e5i;
                out[2] = tot.e4k;
                out[3] = tot.e5k;
            }
            __syncthreads();  // the park, the vectors and the reduction scratch are reused by the next item
            continue;
        }
        // cp.async form: TRPDRV_OZ_TENGY_TMA=0, or where the tensor map cannot be encoded
        if (!tengy_decode(P.sys, P.pos0, (int)(w % np), (int)(w / np), it)) continue;  // uniform over the CTA
        tengy_park_cpasync(P, it, park);
        tengy_finish(P, it, park, red);
    }
}


// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// 3-D map over int8 digits: dims {dp (contiguous), 2V, planes*S}, box {KC, rows, 1}, 64-byte swizzle
static int make_map_i8(CUtensorMap *m, const signed char *base, unsigned long long dp, unsigned long long rows,
                       unsigned long long planes, unsigned box_rows)
{
    PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
    if (!fn) return 1;
    const cuuint64_t dims[3] = {dp, rows, planes};
    const cuuint64_t strides[2] = {dp, dp * rows};
    const cuuint32_t box[3] = {(cuuint32_t)KC, box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<signed char *>(base), dims, strides, box,
                          estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 2;
}

// 3-D map over the f of a batch for the TMA form of the energies: dims {nvir rows (contiguous), nvir
// columns, planes}, box {16, 16, 8} (the eight f of one triple), 128-byte swizzle, zero fill past nvir.
// Columns are trpdrv_oz_ldf(nvir) doubles apart (a multiple of 16 bytes); needs a 16-byte aligned base.
static int make_map_f64(CUtensorMap *m, const double *base, int nvir, unsigned long long planes, unsigned rows = TW,
                        unsigned cols = TW)
{
    PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
    if (!fn || (reinterpret_cast<uintptr_t>(base) & 15)) return 1;
    const cuuint64_t dims[3] = {(cuuint64_t)nvir, (cuuint64_t)nvir, planes};
    const cuuint64_t ldf = (cuuint64_t)trpdrv_oz_ldf(nvir);
    const cuuint64_t strides[2] = {ldf * sizeof(double), ldf * nvir * sizeof(double)};
    const cuuint32_t box[3] = {(cuuint32_t)rows, (cuuint32_t)cols, 8};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE,
                          rows * sizeof(double) == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 2;
}

// TRPDRV_OZ_TENGY_TMA=0 keeps the cp.async form of the energies for every nvir.
static bool tengy_tma_enabled()
{
    static int on = -1;
    if (on < 0) {
        const char *e = getenv("TRPDRV_OZ_TENGY_TMA");
        on = (e && e[0] == '0') ? 0 : 1;
    }
    return on != 0;
}

template <int S>
static int set_attr()
{
    return (int)cudaFuncSetAttribute(oz_gemm_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)Cfg<S>::SMEM);
}

template <int S>
static int launch_gemm(const GemmParams &P, dim3 grid, cudaStream_t st)
{
    oz_gemm_kernel<S><<<grid, NTHREAD, Cfg<S>::SMEM, st>>>(P);
    return (int)cudaGetLastError();
}

}  // namespace oz
}  // namespace trpdrv

using namespace trpdrv;

// Registers per thread the contraction kernels are launched with (read back at init): the setmaxnreg
// split is valid only when every instantiation has exactly REG_LAUNCH.
static int g_oz_launch_regs = 0;

extern "C" int trpdrv_oz_slices_supported(int slices) { return slices >= TRPDRV_OZ_MIN_SLICES && slices <= TRPDRV_OZ_MAX_SLICES; }

extern "C" int trpdrv_oz_dp(int nocc, int nvir) { return ((nvir + nocc) + 31) / 32 * 32; }

// Energies inside the contraction launch (the default for even nvir; the f tiles are read by TMA): the
// kernel's energy warps compute the previous batch's energies while the tensor cores run this batch's
// products.  Odd nvir, whose f TMA could read here too since its columns are padded, keeps the separate launch, which
// the tests hold it to.
// TRPDRV_OZ_FUSED_ENERGY=0 (read at each call) selects the separate launch for every nvir.
extern "C" int trpdrv_oz_fused_energy_supported(int nvir)
{
    const char *e = getenv("TRPDRV_OZ_FUSED_ENERGY");
    const int on = !(e && e[0] == '0');
    return on && nvir >= 2 && (nvir & 1) == 0 && oz::tengy_tma_enabled();
}

extern "C" size_t trpdrv_oz_maps_bytes(void) { return 2 * sizeof(CUtensorMap); }

extern "C" int trpdrv_oz_prepare(const trpdrv_oz_system *oz, void *maps_out)
{
    CUtensorMap *m = static_cast<CUtensorMap *>(maps_out);
    const unsigned long long R = 2ull * oz->nvir, O = (unsigned long long)oz->nocc, S = (unsigned long long)oz->slices;
    const unsigned long long NA = (unsigned long long)(oz->n_a > 0 ? oz->n_a : 1);
    int e = oz::make_map_i8(&m[0], oz->sa, (unsigned long long)oz->dp, R, NA * O * S, oz::BM);
    if (e) return e;
    return oz::make_map_i8(&m[1], oz->sb, (unsigned long long)oz->dp, R, O * O * S, oz::BN);
}

extern "C" int trpdrv_launch_oz_slices(const trpdrv_dev_system *h_sys, const trpdrv_oz_system *oz, void *stream)
{
    oz::SliceParams P;
    P.t2 = h_sys->t2;
    P.jvv = h_sys->jvv;
    P.kvv = h_sys->kvv;
    P.ntov = h_sys->ntov;
    P.nxov = h_sys->nxov;
    P.jov = h_sys->jov;
    P.kov = h_sys->kov;
    P.V = oz->nvir;
    P.O = oz->nocc;
    P.S = oz->slices;
    P.dp = oz->dp;
    const unsigned rb = (unsigned)((2 * oz->nvir + 31) / 32);
    cudaStream_t st = (cudaStream_t)stream;
    P.out = oz->sa;
    P.scale = oz->ea;
    oz::oz_slice_kernel<0><<<dim3(rb, (unsigned)(oz->nocc * (oz->n_a > 0 ? oz->n_a : 1))), 256, 0, st>>>(P);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    P.out = oz->sb;
    P.scale = oz->eb;
    oz::oz_slice_kernel<1><<<dim3(rb, (unsigned)(oz->nocc * oz->nocc)), 256, 0, st>>>(P);
    return (int)cudaGetLastError();
}

extern "C" int trpdrv_launch_oz_gemm(const trpdrv_dev_system *h_sys, const trpdrv_oz_system *oz, const void *maps,
                                     int64_t pos0, int64_t job0, int njobs, double *fbuf, int64_t epos0, int enpos,
                                     const double *efbuf, int *status, int grid, void *stream)
{
    if (njobs < 0 || enpos < 0 || (njobs == 0 && enpos == 0)) return 0;
    oz::GemmParams P;
    memset(&P, 0, sizeof(P));
    if (enpos > 0) {  // energies of an earlier launch's positions, fused into this one
        if (!trpdrv_oz_fused_energy_supported(h_sys->nvir)) return (int)cudaErrorInvalidValue;
        P.np = oz::tengy_pairs(h_sys->nvir);
        if (P.np > h_sys->npairs * TRPDRV_FUSED_SLOTS) return (int)cudaErrorInvalidValue;
        if ((long long)P.np * enpos > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
        if (oz::make_map_f64(&P.fbc, efbuf, h_sys->nvir, 8ull * enpos, 16, 8) != 0 ||
            oz::make_map_f64(&P.fcb, efbuf, h_sys->nvir, 8ull * enpos, 8, 16) != 0)
            return (int)cudaErrorInvalidValue;
        P.sys = *h_sys;
        P.epos0 = epos0;
        P.enpos = enpos;
    }
    memcpy(&P.mapA, maps, sizeof(CUtensorMap));
    memcpy(&P.mapB, static_cast<const char *>(maps) + sizeof(CUtensorMap), sizeof(CUtensorMap));
    P.ea = oz->ea;
    P.eb = oz->eb;
    P.triples = h_sys->triples;
    P.order = h_sys->order;
    P.jobs = oz->jobs + job0;
    P.pos0 = pos0;
    P.ntriples = h_sys->ntriples;
    P.nt = h_sys->nt;
    P.fbuf = fbuf;
    P.V = oz->nvir;
    P.O = oz->nocc;
    P.ldf = trpdrv_oz_ldf(oz->nvir);
    P.nks = oz->dp / oz::KSTEP;
    P.mtiles = (2 * oz->nvir + oz::BM - 1) / oz::BM;
    P.ntiles = (2 * oz->nvir + oz::BN - 1) / oz::BN;
    P.tiles = njobs * P.mtiles * P.ntiles;
    P.status = status;
    const long long work = P.tiles > 0 ? P.tiles : (long long)P.np * enpos;  // an energies-only launch
    if (grid < 1) grid = 1;
    if (grid > work) grid = (int)work;
    cudaStream_t st = (cudaStream_t)stream;
    if (g_oz_launch_regs != oz::REG_LAUNCH) return (int)cudaErrorInvalidConfiguration;  // split unusable
    switch (oz->slices) {
    case 4: return oz::launch_gemm<4>(P, dim3((unsigned)grid), st);
    case 5: return oz::launch_gemm<5>(P, dim3((unsigned)grid), st);
    case 6: return oz::launch_gemm<6>(P, dim3((unsigned)grid), st);
    case 7: return oz::launch_gemm<7>(P, dim3((unsigned)grid), st);
    case 8: return oz::launch_gemm<8>(P, dim3((unsigned)grid), st);
    default: return (int)cudaErrorInvalidValue;
    }
}

extern "C" int trpdrv_launch_oz_tengy(const trpdrv_dev_system *h_sys, int64_t pos0, int npos, const double *fbuf,
                                      int *status, void *stream)
{
    if (npos <= 0) return 0;
    const int np = oz::tengy_pairs(h_sys->nvir);
    if (np > h_sys->npairs * TRPDRV_FUSED_SLOTS) return (int)cudaErrorInvalidValue;
    const long long items = (long long)np * npos;
    if (items > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
    oz::TengyParams P;
    memset(&P, 0, sizeof(P));
    P.sys = *h_sys;
    P.pos0 = pos0;
    P.fbuf = fbuf;
    P.status = status;
    const bool tma = oz::tengy_tma_enabled() && oz::make_map_f64(&P.fmap, fbuf, h_sys->nvir, 8ull * npos) == 0;
    // one CTA per item: a launch of one CTA per SM (each CTA looping
    // over many items) was measured 30 % slower overall, too little memory parallelism per SM
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned grid = (unsigned)items;
    if (tma)
        oz::oz_tengy_kernel<true><<<grid, oz::TNTHREAD, oz::TSMEM_TMA_BYTES, st>>>(P, np, npos);
    else
        oz::oz_tengy_kernel<false><<<grid, oz::TNTHREAD, oz::TSMEM_BYTES, st>>>(P, np, npos);
    return (int)cudaGetLastError();
}

extern "C" int trpdrv_launch_warp_wait_selftest(unsigned long long limit_ns, int *status, void *stream)
{
    oz::warp_wait_selftest_kernel<<<1, 64, 0, (cudaStream_t)stream>>>(limit_ns, status);
    return (int)cudaGetLastError();
}

template <int S>
static int oz_regs(int *all_equal)
{
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, oz::oz_gemm_kernel<S>);
    if (e != cudaSuccess) return (int)e;
    if (a.numRegs != oz::REG_LAUNCH) *all_equal = 0;
    return 0;
}

extern "C" int trpdrv_oz_init(void)
{
    int e, regs_ok = 1;
    if ((e = oz_regs<4>(&regs_ok)) != 0 || (e = oz_regs<5>(&regs_ok)) != 0 || (e = oz_regs<6>(&regs_ok)) != 0 ||
        (e = oz_regs<7>(&regs_ok)) != 0 || (e = oz_regs<8>(&regs_ok)) != 0)
        return e;
    g_oz_launch_regs = regs_ok ? oz::REG_LAUNCH : 0;
    if ((e = oz::set_attr<4>()) != 0) return e;
    if ((e = oz::set_attr<5>()) != 0) return e;
    if ((e = oz::set_attr<6>()) != 0) return e;
    if ((e = oz::set_attr<7>()) != 0) return e;
    if ((e = oz::set_attr<8>()) != 0) return e;
    const cudaFuncAttribute dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if ((e = (int)cudaFuncSetAttribute(oz::oz_tengy_kernel<false>, dyn, (int)oz::TSMEM_BYTES)) != 0) return e;
    return (int)cudaFuncSetAttribute(oz::oz_tengy_kernel<true>, dyn, (int)oz::TSMEM_TMA_BYTES);
}
