// Fused persistent triples kernel (sm_100a, FP64 DMMA), operands staged by TMA or cp.async.
//
// A work item is (triple, tile pair {B,C}); each consumer warp owns a 16(b) x 8(c) sub-block and computes all eight
// f of omp/ccsd_trpdrv_omp_cbody.c:70-117 at (b,c) and, through the operand-swapped MMA, at (c,b), so that the
// energies are evaluated from registers.
//
//  * four producer warps: the first takes work tickets and writes each item's context to a ring in shared memory; all
//    of them fill, per chunk of DK contraction indices, the stage's panels, by cp.async.bulk.tensor loads or (odd or
//    unaligned tensors, more than eight systems) by cp.async, that complete on the stage's "full" mbarrier;
//  * eight consumer warps wait on "full", run the DMMAs straight from the staged panels and
//    release the stage through its "empty" mbarrier; no CTA-wide barrier in the main loop.
//
// What bounds it: the FP64 tensor pipe (37.1 TFLOP/s).  nocc 16, nvir 288: 34.9 TFLOP/s (27.8 with branches among a
// chunk's MMAs, generic loads and an epilogue with branches); 16, 300: 33.5; 20, 200: 29.9, where 8 of the 208 covered
// indices are padding and an item's epilogue and start-up are 12 % of it; 10, 60: 18.8; 13, 151 (cp.async): 23.8.
//
// Panel layouts in shared memory (4 KB per panel, 16 panels per stage, DK = 16):
//  * K-major panels (rows contiguous in HBM: Jia/Kia/Jka/Kka, -Tia/-Xia/-Tka/-Xka, T2 as T(c,d)):
//    two 16-row boxes of [DK][16] doubles written with the 128-byte swizzle, which makes the
//    k-permuted fragment reads bank-conflict free;
//  * X-major panels (contraction contiguous: T2 as T(d,c), Jkj/Kkj/Jij/Kij): one [32][DK] box, also
//    128-byte swizzled, read with 128-bit loads.
// Every box row is a full 128-byte line: with 64-byte rows (DK = 8) the TMA request rate, not L2
// bandwidth, bounded the staging at about half of this rate.
// Fragment row/column labels are permuted, lane group g owning row (and column) PERM[g] of its 8,
// PERM = {0,6,1,7,2,4,3,5}: the two rows a quarter-warp reads with one 128-bit load of an X-major
// panel then differ in bit 2 (disjoint bank sets under the 128-byte swizzle) and the rows of one
// 64-bit load of a K-major panel differ in bit 1 where they share bit 0, so no fragment read of a k8 or
// k16 step has a bank conflict.  (The k4 step of a last chunk, whose lanes hold other contraction indices,
// reads both kinds in two wavefronts.)  The permutation only relabels which (b, c) a register holds; the
// epilogue and the diagonal exchange use the permuted coordinates.
// The MMA shape is a template parameter: m16n8k8 (two k-steps per 16-index chunk) or m16n8k16,
// whose fragments are exactly the two k8 fragments of the chunk side by side (lane t holds logical
// k = t + 4q at physical index 2t + (q & 1) + 8 (q >> 1)).
// The 3-D tensor maps ([system block][contraction][row]) give every dimension its own bound, so the
// ragged tails in nvir and nocc are zero-filled by the TMA unit.
//
// Every wait is bounded (globaltimer); a wait that runs out sets bit 1 of *status and the CTA stops
// issuing work.  TMA staging requires even nvir and nocc and 16-byte aligned tensors (host checks).

#include <cuda.h>
#include <cudaTypedefs.h>

#include "device_common.cuh"
#include "launch.h"

namespace trpdrv {
namespace tma {

constexpr int T = TRPDRV_TILE;  // 32
constexpr int DK = 16;          // contraction indices per stage (two m16n8k8 steps; 128-byte box rows)
constexpr int STAGES = 3;
constexpr int NCW = TRPDRV_FUSED_SLOTS;  // consumer warps (8) = two warpgroups
constexpr int NTHREAD = (NCW + 4) * 32;  // + one producer warpgroup
// Register split by setmaxnreg: launched at 65536 / 384 = 168 per thread; the producer warpgroup drops to 88 and
// the two consumer warpgroups rise to 208 (2*128*208 + 128*88 = 384*168): at this split the MMA loops do not
// spill and the producers least (-Xptxas -v; 216 / 64 and 200 / 96 both spill more).
constexpr int REG_LAUNCH = 168, REG_CONSUMER = 208, REG_PRODUCER = 88;
static_assert(2 * 128 * REG_CONSUMER + 128 * REG_PRODUCER <= NTHREAD * REG_LAUNCH, "register split exceeds the launch");
constexpr int PANEL_BYTES = 4096;
constexpr int NPANEL = 16;
constexpr int STAGE_BYTES = NPANEL * PANEL_BYTES;
constexpr int RING = 16;
constexpr int TICKETS = 8;  // work tickets in flight between the producer warps (>= STAGES + 2)
constexpr int KBOX = PANEL_BYTES / 2;  // one 16-row K-major box
constexpr size_t SMEM_BYTES = (size_t)STAGES * STAGE_BYTES + 1024;  // + alignment slack
constexpr unsigned long long WAIT_LIMIT_NS = 4000000000ull;       // 4 s: far above any legitimate wait

static_assert(RING >= STAGES + 2 && TICKETS >= STAGES + 2, "context or ticket ring too small");

enum { M_J = 0, M_K, M_NT, M_NX, M_T2K, M_T2X, M_JOV, M_KOV, NMAP };

struct __align__(64) Maps {
    CUtensorMap m[TRPDRV_TMA_MAX_SYSTEMS][NMAP];
};

struct ItemCtx {
    const double *eorb, *dintc1, *dintx1, *t1v1, *dintc2, *dintx2, *t1v2;
    double *out, *out1;  // energy slots of the item's pair (and of the second pair of a packed item)
    double eaijk;
    int ncor, nocc, nvir, b0, c0, diag, same, nch, state;  // same: i == k; state: 1 work, 0 malformed, -1 end
    int packed, b1;      // packed edge item: pairs (b0, c0) and (b1, c0); b1 < 0 when the second is absent
    int pad;
};

// at 160 bytes the batched kernel measured 6 % slower
static_assert(sizeof(ItemCtx) == 128, "the item context is kept at 128 bytes");

// Packed edge items (systems with pack_edge: the last column tile E holds 1..16 valid indices).  The
// pairs (B, E) and (B + 1, E), B even, run as one item: each family of a chunk gets its own stage
// slot, in which the 4 KB panels are
//   0, 1: J (or -T) rows of B and B + 1      2, 3: K (or -X) rows of B and B + 1   (K-major, 2 boxes)
//   4: B_1 columns of E (1 K-major box, or 1 X-major box)   5: B_3 columns of E (X-major)
//   6, 7: J / K (or -T / -X) rows of E (1 K-major box each)
//   8, 9: B_1 columns of B and B + 1 (2 K-major boxes, or 1 X-major)   10, 11: B_3 columns (X-major)
// and warp w computes pair w >> 2, rows 16 ((w & 3) >> 1) and columns 8 (w & 1) of it: the work of one
// full pair over 8 warps instead of two half-idle pairs.
constexpr int PK_A = 0, PK_B1E = 4, PK_B3E = 5, PK_AE = 6, PK_B1B = 8, PK_B3B = 10;

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

__device__ __forceinline__ void mbar_arrive(unsigned long long *b)
{
    asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(saddr(b)) : "memory");
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

// Whether the phase with the given parity has completed, without waiting.
__device__ __forceinline__ bool mbar_test_wait(unsigned long long *b, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(saddr(b)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait for the phase with the given parity; false (and status bit 1) when it runs out.
// try_wait itself suspends the warp for a while in hardware; the clock is read only every 256
// failed polls so that waiting warps take few issue slots from the MMA warps of their scheduler.
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

// Self-test of the bounded waits: one thread waits, with the given limit, on an mbarrier that
// nothing completes; the wait must give up, set status bit 1 and return (elapsed_ns: how long it took).
__global__ void bounded_wait_selftest_kernel(unsigned long long limit_ns, int *status,
                                             unsigned long long *elapsed_ns)
{
    __shared__ __align__(8) unsigned long long bar;
    if (threadIdx.x != 0) return;
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const unsigned long long t0 = globaltimer();
    const bool completed = mbar_wait_for(&bar, 0u, status, limit_ns);
    *elapsed_ns = globaltimer() - t0;
    if (completed) atomicOr(status, 4);  // a phase nothing arrived on reported complete
}

// One arrival on the barrier once every cp.async of this thread has landed.
__device__ __forceinline__ void cp_async_arrive(unsigned long long *b)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(saddr(b)) : "memory");
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, unsigned long long *bar, int x, int y,
                                            int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(saddr(dst)), "l"(map), "r"(saddr(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// ------------------------------------------------------------------------------------------------
// fragments (m16n8k8, lane t holds logical k = t and t+4 at physical kk = 2t, 2t+1)
// ------------------------------------------------------------------------------------------------
// Byte offsets of one thread's fragment elements inside a staged panel.  They depend only on the
// thread's sub-block and lane, so they are computed once and every fragment read in the main loop is
// a single shared load at (panel base + constant offset).
// Row/column of its 8 that lane group g (0..7) owns (see the header): conflict-free fragment reads.
__device__ __forceinline__ int perm8(int g) { return (0x53427160 >> (4 * g)) & 7; }

__device__ __forceinline__ int kmajor_off(int kk, int x)
{
    const int h = x >> 4, xi = x & 15;
    return h * KBOX + kk * 128 + (((xi >> 1) ^ (kk & 7)) << 4) + ((xi & 1) << 3);
}

struct FragOffsets {
    int kA0, kA1, kA2, kA3;  // K-major A fragment: (2t, r), (2t, r+8), (2t+1, r), (2t+1, r+8)
    int kB0, kB1;            // K-major B fragment: (2t, c), (2t+1, c)
    int xA0;                 // X-major A fragment: rows r and (1024 bytes on) r+8 at contraction 2t (128-bit)
    int xB;                  // X-major B fragment: column c at contraction 2t (128-bit)
    __device__ __forceinline__ FragOffsets(int rx0, int cx0, int g, int t)
    {
        const int r = rx0 + perm8(g), c = cx0 + perm8(g);
        kA0 = kmajor_off(2 * t, r);
        kA1 = kmajor_off(2 * t, r + 8);
        kA2 = kmajor_off(2 * t + 1, r);
        kA3 = kmajor_off(2 * t + 1, r + 8);
        kB0 = kmajor_off(2 * t, c);
        kB1 = kmajor_off(2 * t + 1, c);
        xA0 = r * 128 + ((t ^ (r & 7)) << 4);
        xB = c * 128 + ((t ^ (c & 7)) << 4);
    }
    __device__ __forceinline__ static double ld(const char *p, int off) { return *reinterpret_cast<const double *>(p + off); }
    __device__ __forceinline__ static double2 ld2(const char *p, int off) { return *reinterpret_cast<const double2 *>(p + off); }
    __device__ __forceinline__ void ldA_K(double (&a)[4], const char *P) const
    {
        a[0] = ld(P, kA0);
        a[1] = ld(P, kA1);
        a[2] = ld(P, kA2);
        a[3] = ld(P, kA3);
    }
    __device__ __forceinline__ void ldB_K(double (&b)[2], const char *P) const
    {
        b[0] = ld(P, kB0);
        b[1] = ld(P, kB1);
    }
    __device__ __forceinline__ void ldA_X(double (&a)[4], const char *P, int kx) const
    {
        const double2 lo = ld2(P, xA0 ^ kx), hi = ld2(P, (xA0 ^ kx) + 1024);
        a[0] = lo.x;
        a[2] = lo.y;
        a[1] = hi.x;
        a[3] = hi.y;
    }
    __device__ __forceinline__ void ldB_X(double (&b)[2], const char *P, int kx) const
    {
        const double2 v = ld2(P, xB ^ kx);
        b[0] = v.x;
        b[1] = v.y;
    }
};

// m16n8k16 fragments: the k8 fragments of the chunk's two k-steps (K-major panels: the second
// k-step starts 8 rows = 1024 bytes further; X-major panels: 64 bytes further in each row).
__device__ __forceinline__ void ld_a16_K(const FragOffsets &fo, double (&a)[8], const char *P)
{
    fo.ldA_K(*reinterpret_cast<double(*)[4]>(&a[0]), P);
    fo.ldA_K(*reinterpret_cast<double(*)[4]>(&a[4]), P + 1024);
}
__device__ __forceinline__ void ld_b16_K(const FragOffsets &fo, double (&b)[4], const char *P)
{
    fo.ldB_K(*reinterpret_cast<double(*)[2]>(&b[0]), P);
    fo.ldB_K(*reinterpret_cast<double(*)[2]>(&b[2]), P + 1024);
}
__device__ __forceinline__ void ld_a16_X(const FragOffsets &fo, double (&a)[8], const char *P)
{
    fo.ldA_X(*reinterpret_cast<double(*)[4]>(&a[0]), P, 0);
    fo.ldA_X(*reinterpret_cast<double(*)[4]>(&a[4]), P, 64);
}
__device__ __forceinline__ void ld_b16_X(const FragOffsets &fo, double (&b)[4], const char *P)
{
    fo.ldB_X(*reinterpret_cast<double(*)[2]>(&b[0]), P, 0);
    fo.ldB_X(*reinterpret_cast<double(*)[2]>(&b[2]), P, 64);
}

// ------------------------------------------------------------------------------------------------
// products of one chunk
// ------------------------------------------------------------------------------------------------
// Fragments of one group of four m16n8k8: two A operands, two B operands.
struct Group {
    double a0[4], a1[4], b0[2], b1[2];
};

// Byte offsets of the panels that one family's groups read: the two A operands (K-major), B_1 (K-major, in the
// occupied phase X-major) and B_3 (X-major) of the products at (b, c) (o = 0) and of the transposes (o = 1).
struct Panels {
    int a0[2], a1[2], b0[2], b1[2];
};

// Ordinary items: panel 2 q + o of the family's eight holds operand q (A_J, A_K, B_1, B_3) of orientation o.
template <int FAM> __device__ __forceinline__ constexpr Panels item_panels()
{
    constexpr int P = FAM * 8 * PANEL_BYTES, S = PANEL_BYTES;
    return {{P, P + 5 * S}, {P + 2 * S, P + 7 * S}, {P + 4 * S, P + S}, {P + 6 * S, P + 3 * S}};
}

// Packed edge items (layout at PK_*): pair pp of the two that share the slot.
__device__ __forceinline__ Panels packed_panels(int pp)
{
    constexpr int S = PANEL_BYTES;
    return {{(PK_A + pp) * S, (PK_B1B + pp) * S},
            {(PK_A + 2 + pp) * S, (PK_B3B + pp) * S},
            {PK_B1E * S, PK_AE * S},
            {PK_B3E * S, (PK_AE + 1) * S}};
}

// Group O of k-step ks.  O = 0: A_J, A_K rows and B_1, B_3 columns; f1 = A_J B_1, f2 = A_K B_1, f3 = A_J B_3,
// f4 = A_K B_3 at (b, c).  O = 1: the transposes f_x(c,b) = sum_d B_x(d,b) A_x(c,d): a0, a1 = B_1, B_3 and
// b0, b1 = A_J, A_K of the C side.  PH1: the occupied phase, where B_1 is X-major.
template <bool PH1, int O>
__device__ __forceinline__ void load_group(const FragOffsets &fo, const char *st, const Panels &pn, int ks, Group &g)
{
    const int kk = ks * 1024, kx = ks * 64;  // K-major: 8 rows further; X-major: 64 bytes into each row
    if (O == 0) {
        fo.ldA_K(g.a0, st + pn.a0[0] + kk);
        fo.ldA_K(g.a1, st + pn.a1[0] + kk);
        fo.ldB_X(g.b1, st + pn.b1[0], kx);
        if (!PH1)
            fo.ldB_K(g.b0, st + pn.b0[0] + kk);
        else
            fo.ldB_X(g.b0, st + pn.b0[0], kx);
    } else {
        fo.ldB_K(g.b0, st + pn.b0[1] + kk);
        fo.ldB_K(g.b1, st + pn.b1[1] + kk);
        fo.ldA_X(g.a1, st + pn.a1[1], kx);
        if (!PH1)
            fo.ldA_K(g.a0, st + pn.a0[1] + kk);
        else
            fo.ldA_X(g.a0, st + pn.a0[1], kx);
    }
}

// m16n8k8, or (KS = 4) the two m16n8k4 it consists of: its fragments hold the contraction indices 2t and 2t + 1.
template <int KS>
__device__ __forceinline__ void mma8(double (&d)[4], const double (&a)[4], const double (&b)[2])
{
    if (KS == 4) {
        dmma_16x8x4(d, a[0], a[1], b[0]);
        dmma_16x8x4(d, a[2], a[3], b[1]);
    } else {
        dmma_16x8x8(d, a, b);
    }
}

template <int KS, int FAM, int O>
__device__ __forceinline__ void mma_group(const Group &g, double (&f)[8][4], double (&gT)[8][4])
{
    constexpr int x0 = FAM * 4;
    if (O == 0) {
        mma8<KS>(f[x0 + 0], g.a0, g.b0);
        mma8<KS>(f[x0 + 1], g.a1, g.b0);
        mma8<KS>(f[x0 + 2], g.a0, g.b1);
        mma8<KS>(f[x0 + 3], g.a1, g.b1);
    } else {
        mma8<KS>(gT[x0 + 0], g.a0, g.b0);
        mma8<KS>(gT[x0 + 1], g.a0, g.b1);
        mma8<KS>(gT[x0 + 2], g.a1, g.b0);
        mma8<KS>(gT[x0 + 3], g.a1, g.b1);
    }
}

// The same four products over both k-steps of a chunk with m16n8k16 (ordinary items).
template <bool PH1, int FAM, int O>
__device__ __forceinline__ void group16(const FragOffsets &fo, const char *st, double (&f)[8][4], double (&gT)[8][4])
{
    constexpr int x0 = FAM * 4;
    constexpr Panels pn = item_panels<FAM>();
    double a0[8], a1[8], b0[4], b1[4];
    if (O == 0) {
        ld_a16_K(fo, a0, st + pn.a0[0]);
        ld_a16_K(fo, a1, st + pn.a1[0]);
        ld_b16_X(fo, b1, st + pn.b1[0]);
        if (!PH1)
            ld_b16_K(fo, b0, st + pn.b0[0]);
        else
            ld_b16_X(fo, b0, st + pn.b0[0]);
        dmma_16x8x16(f[x0 + 0], a0, b0);
        dmma_16x8x16(f[x0 + 1], a1, b0);
        dmma_16x8x16(f[x0 + 2], a0, b1);
        dmma_16x8x16(f[x0 + 3], a1, b1);
    } else {
        ld_b16_K(fo, b0, st + pn.b0[1]);
        ld_b16_K(fo, b1, st + pn.b1[1]);
        ld_a16_X(fo, a1, st + pn.a1[1]);
        if (!PH1)
            ld_a16_K(fo, a0, st + pn.a0[1]);
        else
            ld_a16_X(fo, a0, st + pn.a0[1]);
        dmma_16x8x16(gT[x0 + 0], a0, b0);
        dmma_16x8x16(gT[x0 + 1], a0, b1);
        dmma_16x8x16(gT[x0 + 2], a1, b0);
        dmma_16x8x16(gT[x0 + 3], a1, b1);
    }
}

// A consumer warp's place in the stage ring.
struct RingPos {
    int stage;
    unsigned phase;
    bool ready;  // the stage's full barrier is known to have completed
    __device__ __forceinline__ void next()
    {
        if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
        }
    }
};

// What a consumer warp's chunk loops need besides the accumulators.
struct Pipe {
    const char *stages;
    unsigned long long *full, *empty;
    int *status;
    int lane;
    __device__ __forceinline__ bool wait(const RingPos &rp) const
    {
        return rp.ready || mbar_wait(&full[rp.stage], rp.phase, status);
    }
    // releases the stage and looks at the next one without waiting for it
    __device__ __forceinline__ void release(RingPos &rp) const
    {
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[rp.stage]);
        rp.next();
        rp.ready = mbar_test_wait(&full[rp.stage], rp.phase);
    }
};

// Products of family FAM with the k8 steps of a chunk, except (TAIL) the last group's MMAs, whose fragments are
// left in `tail`: the caller releases the stage and looks at the next one in between, so neither the barrier
// nor the first fragment loads of the next chunk leave the tensor pipe idle.  NKS: k8 steps of the chunk (1
// when the second lies entirely in the zero padding).  A diagonal pair (DIAG) gets f(c,b) from the other warps
// at the end of the item.
template <int KS, int NKS, bool PH1, bool DIAG, int FAM, bool TAIL>
__device__ __forceinline__ void family_products(const FragOffsets &fo, const char *st, const Panels &pn,
                                                double (&f)[8][4], double (&gT)[8][4], Group &tail)
{
    Group g;
#pragma unroll
    for (int ks = 0; ks < NKS; ++ks) {
        const bool last = TAIL && ks == NKS - 1;
        if (DIAG && last) {
            load_group<PH1, 0>(fo, st, pn, ks, tail);
            return;
        }
        load_group<PH1, 0>(fo, st, pn, ks, g);
        mma_group<KS, FAM, 0>(g, f, gT);
        if (DIAG) continue;
        if (last) {
            load_group<PH1, 1>(fo, st, pn, ks, tail);
            return;
        }
        load_group<PH1, 1>(fo, st, pn, ks, g);
        mma_group<KS, FAM, 1>(g, f, gT);
    }
}

// n chunks of one kind of an ordinary item.  Everything that differs between chunks (phase, diagonal pair,
// number of k-steps, SAME: i == k, where the t family equals the n family and is not computed) is a template
// parameter, so that a chunk is straight-line code and the fragment loads of one group are scheduled over the
// MMAs of the group before.  With the same choices as branches between the groups, and generic instead of
// shared-memory loads, the MMA loop ran at 76 % of the FP64 tensor pipe's rate (measured without epilogue).
template <int KS, int NKS, bool PH1, bool DIAG, bool SAME>
__device__ __forceinline__ bool run_chunks(int n, const FragOffsets &fo, const Pipe &pp, RingPos &rp, double (&f)[8][4],
                                           double (&gT)[8][4])
{
    constexpr bool K16 = KS == 16 && NKS == 2;
    constexpr int LAST = SAME ? 0 : 1;
#pragma unroll 1
    for (; n > 0; --n) {
        if (!pp.wait(rp)) return false;
        const char *st = pp.stages + (size_t)rp.stage * STAGE_BYTES;
        Group tail;
        if (K16) {
            group16<PH1, 0, 0>(fo, st, f, gT);
            if (!DIAG) group16<PH1, 0, 1>(fo, st, f, gT);
            if (!SAME) group16<PH1, 1, 0>(fo, st, f, gT);
            if (!SAME && !DIAG) group16<PH1, 1, 1>(fo, st, f, gT);
        } else {
            if (!SAME) family_products<KS, NKS, PH1, DIAG, 0, false>(fo, st, item_panels<0>(), f, gT, tail);
            family_products<KS, NKS, PH1, DIAG, LAST, true>(fo, st, item_panels<LAST>(), f, gT, tail);
        }
        pp.release(rp);
        if (!K16) mma_group<KS, LAST, DIAG ? 0 : 1>(tail, f, gT);
    }
    return true;
}

// n chunks of a packed edge item: one stage slot per (chunk, family), m16n8k8 in both kernels (the packed path's
// extra fragment registers would push the k16 kernel's MMA warps past their register budget).
template <int KS, int NKS, bool PH1, bool SAME>
__device__ __forceinline__ bool run_packed(int n, const FragOffsets &fo, const Panels &pn, const Pipe &pp, RingPos &rp,
                                           double (&f)[8][4], double (&gT)[8][4])
{
#pragma unroll 1
    for (; n > 0; --n) {
        Group tail;
        if (!pp.wait(rp)) return false;
        family_products<KS, NKS, PH1, false, 0, true>(fo, pp.stages + (size_t)rp.stage * STAGE_BYTES, pn, f, gT, tail);
        pp.release(rp);
        mma_group<KS, 0, 1>(tail, f, gT);
        if (SAME) continue;
        if (!pp.wait(rp)) return false;
        family_products<KS, NKS, PH1, false, 1, true>(fo, pp.stages + (size_t)rp.stage * STAGE_BYTES, pn, f, gT, tail);
        pp.release(rp);
        mma_group<KS, 1, 1>(tail, f, gT);
    }
    return true;
}

// The last chunk of either contraction, where four of its indices or fewer remain past a multiple of 8: one k4 step
// instead of a k8 step over zeros.  10, 60: 0.123 to 0.119 ms; 12, 100: 0.802 to 0.778; 16, 300: 29.70 to 29.55; 20, 200:
// 19.88 to 19.81.
//
// Products of family FAM with the four contraction indices 8 ks .. 8 ks + 3 of a chunk, m16n8k4: lane t holds index
// 8 ks + t (in a k8 step 2t and 2t + 1).  Its reads, of both panel kinds, take two wavefronts each; it runs once a
// contraction at most.
template <bool PH1, bool DIAG, int FAM>
__device__ __forceinline__ void quarter_products(const FragOffsets &fo, const char *st, const Panels &pn, int ks, int t,
                                                 double (&f)[8][4], double (&gT)[8][4])
{
    constexpr int x0 = FAM * 4;
    const int r = fo.xA0 >> 7, c = fo.xB >> 7, kk = ks * 1024, kx = ks * 64;
    auto ldK = [&](int panel, int x) { return FragOffsets::ld(st, panel + kk + kmajor_off(t, x)); };
    auto ldX = [&](int panel, int x) {
        return FragOffsets::ld(st, panel + x * 128 + ((((t >> 1) ^ (x & 7)) << 4) ^ kx) + ((t & 1) << 3));
    };
    {
        const double aj[2] = {ldK(pn.a0[0], r), ldK(pn.a0[0], r + 8)}, ak[2] = {ldK(pn.a1[0], r), ldK(pn.a1[0], r + 8)};
        const double b1 = PH1 ? ldX(pn.b0[0], c) : ldK(pn.b0[0], c), b3 = ldX(pn.b1[0], c);
        dmma_16x8x4(f[x0 + 0], aj[0], aj[1], b1);
        dmma_16x8x4(f[x0 + 1], ak[0], ak[1], b1);
        dmma_16x8x4(f[x0 + 2], aj[0], aj[1], b3);
        dmma_16x8x4(f[x0 + 3], ak[0], ak[1], b3);
    }
    if (DIAG) return;
    const double b1[2] = {PH1 ? ldX(pn.a0[1], r) : ldK(pn.a0[1], r), PH1 ? ldX(pn.a0[1], r + 8) : ldK(pn.a0[1], r + 8)};
    const double b3[2] = {ldX(pn.a1[1], r), ldX(pn.a1[1], r + 8)};
    const double aj = ldK(pn.b0[1], c), ak = ldK(pn.b1[1], c);
    dmma_16x8x4(gT[x0 + 0], b1[0], b1[1], aj);
    dmma_16x8x4(gT[x0 + 1], b1[0], b1[1], ak);
    dmma_16x8x4(gT[x0 + 2], b3[0], b3[1], aj);
    dmma_16x8x4(gT[x0 + 3], b3[0], b3[1], ak);
}

// The last chunk of a phase where its last 8 contraction indices hold 1 to 4 valid ones: kind 1, those alone, or 2, a
// k8 step before them; 0, no such chunk.
template <int KS, bool PH1, bool DIAG, bool SAME>
__device__ __forceinline__ bool run_quarter(int kind, const FragOffsets &fo, const Pipe &pp, RingPos &rp, double (&f)[8][4],
                                            double (&gT)[8][4])
{
    constexpr int LAST = SAME ? 0 : 1;
    if (kind == 0) return true;
    if (!pp.wait(rp)) return false;
    const char *st = pp.stages + (size_t)rp.stage * STAGE_BYTES;
    Group unused;
    if (kind == 2) {
        if (!SAME) family_products<KS, 1, PH1, DIAG, 0, false>(fo, st, item_panels<0>(), f, gT, unused);
        family_products<KS, 1, PH1, DIAG, LAST, false>(fo, st, item_panels<LAST>(), f, gT, unused);
    }
    const int t = pp.lane & 3;
    if (!SAME) quarter_products<PH1, DIAG, 0>(fo, st, item_panels<0>(), kind - 1, t, f, gT);
    quarter_products<PH1, DIAG, LAST>(fo, st, item_panels<LAST>(), kind - 1, t, f, gT);
    pp.release(rp);
    return true;
}

template <int KS, bool PH1, bool SAME>
__device__ __forceinline__ bool run_packed_quarter(int kind, const FragOffsets &fo, const Panels &pn, const Pipe &pp, RingPos &rp,
                                                   double (&f)[8][4], double (&gT)[8][4])
{
    if (kind == 0) return true;
    const int t = pp.lane & 3;
    Group unused;
    if (!pp.wait(rp)) return false;
    const char *st = pp.stages + (size_t)rp.stage * STAGE_BYTES;
    if (kind == 2) family_products<KS, 1, PH1, false, 0, false>(fo, st, pn, f, gT, unused);
    quarter_products<PH1, false, 0>(fo, st, pn, kind - 1, t, f, gT);
    pp.release(rp);
    if (SAME) return true;
    if (!pp.wait(rp)) return false;
    st = pp.stages + (size_t)rp.stage * STAGE_BYTES;
    if (kind == 2) family_products<KS, 1, PH1, false, 1, false>(fo, st, pn, f, gT, unused);
    quarter_products<PH1, false, 1>(fo, st, pn, kind - 1, t, f, gT);
    pp.release(rp);
    return true;
}

// The item's chunks by kind: full and one-k-step chunks of the virtual phase, then of the occupied one (the last
// chunk of a phase runs one k-step when the second lies entirely in the zero padding).
struct ChunkCounts {
    int v2, v1, vq, o2, o1, oq;
    __device__ __forceinline__ static void split(int n, int &n2, int &n1, int &nq)
    {
        const int chunks = (n + DK - 1) / DK, last = n - (chunks - 1) * DK;  // 1 .. 16 indices in the last one
        nq = last <= 4 ? 1 : last > 8 && last <= 12 ? 2 : 0;
        n1 = last > 4 && last <= 8;
        n2 = chunks - n1 - (nq > 0);
    }
    __device__ __forceinline__ ChunkCounts(int nvir, int nocc)
    {
        split(nvir, v2, v1, vq);
        split(nocc, o2, o1, oq);
    }
};

template <int KS, bool DIAG, bool SAME>
__device__ __forceinline__ bool run_item(const ChunkCounts &n, const FragOffsets &fo, const Pipe &pp, RingPos &rp,
                                         double (&f)[8][4], double (&gT)[8][4])
{
    return run_chunks<KS, 2, false, DIAG, SAME>(n.v2, fo, pp, rp, f, gT) &&
           run_chunks<KS, 1, false, DIAG, SAME>(n.v1, fo, pp, rp, f, gT) &&
           run_quarter<KS, false, DIAG, SAME>(n.vq, fo, pp, rp, f, gT) &&
           run_chunks<KS, 2, true, DIAG, SAME>(n.o2, fo, pp, rp, f, gT) &&
           run_chunks<KS, 1, true, DIAG, SAME>(n.o1, fo, pp, rp, f, gT) &&
           run_quarter<KS, true, DIAG, SAME>(n.oq, fo, pp, rp, f, gT);
}

template <int KS, bool SAME>
__device__ __forceinline__ bool run_packed_item(const ChunkCounts &n, const FragOffsets &fo, const Panels &pn,
                                                const Pipe &pp, RingPos &rp, double (&f)[8][4], double (&gT)[8][4])
{
    return run_packed<KS, 2, false, SAME>(n.v2, fo, pn, pp, rp, f, gT) &&
           run_packed<KS, 1, false, SAME>(n.v1, fo, pn, pp, rp, f, gT) &&
           run_packed_quarter<KS, false, SAME>(n.vq, fo, pn, pp, rp, f, gT) &&
           run_packed<KS, 2, true, SAME>(n.o2, fo, pn, pp, rp, f, gT) &&
           run_packed<KS, 1, true, SAME>(n.o1, fo, pn, pp, rp, f, gT) &&
           run_packed_quarter<KS, true, SAME>(n.oq, fo, pn, pp, rp, f, gT);
}

// Brings the 128-byte lines of the energy vectors the item's epilogue will read into L1 (lanes 0..27:
// 7 vectors x {B, C} block x 2 lines), so the register epilogue does not wait on L2.
__device__ __forceinline__ void prefetch_epilogue(const ItemCtx &cx, int lane)
{
    if (lane >= 28) return;
    const int v = lane >> 2, r = (lane >> 1) & 1, l = lane & 1;
    // the seven pointers at the head of the context (a switch over them would run as seven divergent branches)
    const double *base = (&cx.eorb)[v] + (v == 0 ? cx.ncor + cx.nocc : 0);
    const int idx = (r ? cx.c0 : cx.b0) + 16 * l;
    if (idx < cx.nvir) asm volatile("prefetch.global.L1 [%0];" ::"l"(base + idx));
}

// ------------------------------------------------------------------------------------------------
// energies of one warp's sub-block, in registers
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ TengyIdx load_idx(const ItemCtx &cx, int x)
{
    return {__ldg(cx.t1v1 + x), __ldg(cx.t1v2 + x), __ldg(cx.dintx1 + x), __ldg(cx.dintx2 + x), __ldg(cx.dintc1 + x),
            __ldg(cx.dintc2 + x)};
}

// DIAG: the pair's own mirror block is a block of the same tile (another warp, or this one, adds its terms).
// No branches: a position past nvir takes the vectors of the last one and adds 0, so that the four positions' chains
// (a division and some 130 FP64 instructions each) overlap.
template <bool DIAG>
__device__ __forceinline__ void warp_epilogue(const ItemCtx &cx, const double (&f)[8][4], const double (&gT)[8][4],
                                              int rb0, int cb0, int g, int t, int lane, double *out)
{
    TengySums su = {0.0, 0.0, 0.0, 0.0};
    const int V = cx.nvir;
    const double *ev = cx.eorb + cx.ncor + cx.nocc;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int b = rb0 + perm8(g) + 8 * h, bi = min(b, V - 1);
        const TengyIdx vb = load_idx(cx, bi);
        const double eb = __ldg(ev + bi);
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const int e = 2 * h + w, c = cb0 + perm8(2 * t + w), ci = min(c, V - 1);
            const bool valid = b < V && c < V;
            double fbc[8], fcb[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                fbc[x] = f[x][e];
                fcb[x] = gT[x][e];
            }
            // omp/ccsd_tengy_c99.c:65 denominator; e_b + e_c == e_c + e_b, so (b,c) and (c,b) share it
            const double denom = -1.0 / (valid ? eb + __ldg(ev + ci) + cx.eaijk : 1.0);
            const TengyTerms p = tengy_terms(!DIAG, fbc, fcb, vb, load_idx(cx, ci));
            su.e4i += denom * (valid ? p.a4i : 0.0);
            su.e4k += denom * (valid ? p.a4k : 0.0);
            su.e5i += denom * (valid ? p.e5i : 0.0);
            su.e5k += denom * (valid ? p.e5k : 0.0);
        }
    }
    const double sum = warp_sum4(su, lane);
    if ((lane & 7) == 0 && out) out[lane >> 3] = sum;
}

// ------------------------------------------------------------------------------------------------
// producer warps: tickets and item contexts (warp 0, lane 0), operand staging (all four)
// ------------------------------------------------------------------------------------------------
// Operand kinds of one family: A_J, A_K (K-major), B_1 (K-major in the virtual phase, X-major in the occupied
// one), B_3 (X-major).
enum { OP_AJ = 0, OP_AK, OP_B1, OP_B3 };

__device__ __forceinline__ bool op_kmajor(int kind, bool virt) { return kind < OP_B1 || (kind == OP_B1 && virt); }

// A work item, decoded from its ticket.  Every producer warp decodes it for itself.
struct Item {
    const trpdrv_dev_system *S;
    long long own;  // index of the item's energy slots
    int s, B, C, i, j, k, ai;
    int za0, za1, zb0, zb1;  // blocks of the A and B operands per family (n, t): A: i / k slot, B: [j][k] / [j][i]
    bool in_range, ok, pack, skip, same, diag;
    __device__ __forceinline__ int za(int fam) const { return fam ? za1 : za0; }
    __device__ __forceinline__ int zb(int fam) const { return fam ? zb1 : zb0; }
};

// pair_major: a system's items run pair by pair, those of two tiles (twice the products) before the diagonal ones, each
// over all triples: small launches then end with the small items on every SM.
__device__ __forceinline__ Item decode_item(const trpdrv_dev_system *__restrict__ sys, int nsys, long long item,
                                            int pair_major)
{
    Item it;
    int s = 0;
    while (s + 1 < nsys && item >= sys[s + 1].item_begin) ++s;
    const trpdrv_dev_system &S = sys[s];
    it.S = &S;
    it.s = s;
    const long long local = item - S.item_begin;
    long long qpos;  // processing position over the system's records
    int B = 0, C;
    if (pair_major && S.ntriples > 0) {
        int rem = (int)(local / S.ntriples);
        qpos = local - (long long)rem * S.ntriples;
        const int noff = S.npairs - S.nb;
        if (rem >= noff) {
            B = C = rem - noff;
        } else {
            while (B < S.nb && rem >= S.nb - 1 - B) rem -= S.nb - 1 - B++;
            C = B + 1 + rem;
        }
    } else {
        qpos = local / S.npairs;
        int rem = (int)(local - qpos * S.npairs);
        while (B < S.nb && rem >= S.nb - B) rem -= S.nb - B++;
        C = B + rem;
    }
    const int p = B * S.nb - B * (B - 1) / 2 + C - B;  // the pair's slot within the record
    // a index (records are [a][triple], fewer than 2^31: the host checks); no division for a single a
    const long long ai = (S.nt > 0 && qpos >= S.nt) ? (long long)((unsigned)qpos / (unsigned)S.nt) : 0;
    const long long tpos = qpos - ai * S.nt;
    const long long tt = (S.order && local >= 0 && qpos < S.ntriples) ? (long long)S.order[tpos] : tpos;
    it.own = (ai * S.nt + tt) * S.npairs + p;  // energies go to the record's own items
    const int O = S.nocc;
    it.B = B;
    it.C = C;
    it.ai = (int)ai;
    it.diag = B == C;
    // edge pairs (B, E) with B odd are computed by the packed item of B - 1
    it.pack = S.pack_edge && C == S.nb - 1 && B < C;
    it.skip = it.pack && (B & 1);
    it.in_range = local >= 0 && qpos < S.ntriples && tt >= 0 && tt < S.nt && ai < S.n_a;
    const int packed = it.in_range ? S.triples[tt] : 0;
    it.i = packed & 1023;
    it.j = (packed >> 10) & 1023;
    it.k = (packed >> 20) & 1023;
    it.za0 = it.i;
    it.za1 = it.k;
    it.zb0 = it.j * O + it.k;
    it.zb1 = it.j * O + it.i;
    it.ok = it.in_range && B < S.nb && C < S.nb && it.i < O && it.j < O && it.k <= it.i;
    it.same = it.i == it.k;  // both families read the same blocks
    return it;
}

__device__ __forceinline__ void write_ctx(ItemCtx &cx, const Item &it)
{
    const trpdrv_dev_system &S = *it.S;
    const int O = S.nocc, V = S.nvir, nV = (V + DK - 1) / DK, nO = (O + DK - 1) / DK;
    cx.eorb = S.eorb;
    const size_t vi = ((size_t)it.ai * O + it.za0) * V, vk = ((size_t)it.ai * O + it.za1) * V;
    cx.dintc1 = S.dintc + vi;
    cx.dintx1 = S.dintx + vi;
    cx.t1v1 = S.t1v + vi;
    cx.dintc2 = S.dintc + vk;
    cx.dintx2 = S.dintx + vk;
    cx.t1v2 = S.t1v + vk;
    cx.out = S.partial + (size_t)it.own * NCW * 4;
    // the second pair (B2, E) of a packed item: its own slots, at its triangular pair index
    // (B2 = B + 1: nb - B - 1 pairs further)
    const bool two = it.pack && it.B + 1 < it.C;
    cx.out1 = cx.out + (two ? (S.nb - it.B - 1) * NCW * 4 : 0);
    cx.packed = it.pack;
    cx.b1 = two ? (it.B + 1) * T : -1;
    // omp/ccsd_trpdrv_omp_cbody.c:126 (a is 1-based, i/j/k here 0-based)
    cx.eaijk = S.eorb[S.a - 1 + it.ai] - (S.eorb[S.ncor + it.i] + S.eorb[S.ncor + it.j] + S.eorb[S.ncor + it.k]);
    cx.ncor = S.ncor;
    cx.nocc = O;
    cx.nvir = V;
    cx.b0 = it.B * T;
    cx.c0 = it.C * T;
    cx.diag = it.diag;
    cx.same = it.same;
    cx.nch = nV + nO;
    cx.state = 1;
}

// The panels of producer warp pw: for an ordinary item the four operands of group (family pw >> 1, orientation
// pw & 1); for a packed item operand kind pw of the three tiles B, B + 1, E.  Spread over one warp per scheduler,
// the staging takes few issue slots from any one scheduler's MMA warps (with one warp issuing every TMA box,
// its scheduler's MMA warps ran 3 % behind the others).
struct Role {
    int npanel, fam, o;
    bool idle;
    __device__ __forceinline__ Role(const Item &it, int pw)
    {
        npanel = it.pack ? 3 : 4;
        fam = it.pack ? 0 : pw >> 1;
        o = it.pack ? 0 : pw & 1;
        idle = !it.pack && ((it.diag && o == 1) || (it.same && fam == 1));
    }
};

// Panel q of the role: its operand kind, the first virtual index of its tile (-1: absent) and its place.
__device__ __forceinline__ void role_panel(const Item &it, const Role &r, int pw, int q, int &kind, int &tile, int &off)
{
    if (!it.pack) {
        kind = q;
        // A rows: B for (B,C), C for (C,B); B columns: C for (B,C), B for (C,B)
        tile = ((q < OP_B1) == (r.o == 0) ? it.B : it.C) * T;
        off = (r.fam * 8 + 2 * q + r.o) * PANEL_BYTES;
    } else {
        kind = pw;
        tile = q == 2 ? it.C * T : q == 0 ? it.B * T : it.B + 1 < it.C ? (it.B + 1) * T : -1;
        const int base = pw < OP_B1 ? (q < 2 ? PK_A + 2 * pw : PK_AE + pw) : pw == OP_B1 ? (q < 2 ? PK_B1B : PK_B1E)
                                                                                        : (q < 2 ? PK_B3B : PK_B3E);
        off = (base + (q < 2 ? q : 0)) * PANEL_BYTES;
    }
}

// TMA staging: one box per lane (ordinary items: 7 per warp, packed ones: 5).
struct TmaStage {
    const Maps *maps;
    const CUtensorMap *mv, *mo;  // this lane's box in the virtual / occupied phase
    int kind, tile, half, off, zav;
    bool act_v, act_o;
    unsigned bytes_v, bytes_o;

    __device__ __forceinline__ void begin(const Item &it, const Role &r, int pw, int lane)
    {
        // K-major panels are two 16-row boxes, X-major ones a single box; the E tile of a packed item has at
        // most 16 valid rows
        const int q = lane >> 1;
        half = lane & 1;
        const bool mine = !r.idle && q < r.npanel;
        role_panel(it, r, pw, mine ? q : 0, kind, tile, off);
        off += half * KBOX;
        const bool box = mine && tile >= 0;
        const bool second = half == 1, e_tile = it.pack && q == 2;
        act_v = box && (!second || (op_kmajor(kind, true) && !e_tile));
        act_o = box && (!second || (op_kmajor(kind, false) && !e_tile));
        bytes_v = __reduce_add_sync(0xffffffffu, act_v ? (op_kmajor(kind, true) ? KBOX : PANEL_BYTES) : 0);
        bytes_o = __reduce_add_sync(0xffffffffu, act_o ? (op_kmajor(kind, false) ? KBOX : PANEL_BYTES) : 0);
        const CUtensorMap *mp = maps->m[it.s];
        mv = &mp[kind == OP_AJ ? M_J : kind == OP_AK ? M_K : kind == OP_B1 ? M_T2K : M_T2X];
        mo = &mp[kind == OP_AJ ? M_NT : kind == OP_AK ? M_NX : kind == OP_B1 ? M_KOV : M_JOV];
        zav = it.ai * it.S->nocc;  // J and K carry the a index, -T and -X do not
    }

    __device__ __forceinline__ void slot(const Item &it, const Role &, int, char *st, unsigned long long *full,
                                         bool virt, int kk0, int fam, int lane)
    {
        const unsigned bytes = virt ? bytes_v : bytes_o;
        if (lane == 0) {
            if (bytes)
                mbar_arrive_expect_tx(full, bytes);
            else
                mbar_arrive(full);
        }
        __syncwarp();
        if (virt ? act_v : act_o) {
            const bool km = op_kmajor(kind, virt);
            const int row = tile + 16 * half;
            const int z = kind < OP_B1 ? it.za(fam) + (virt ? zav : 0) : it.zb(fam);
            tma_load_3d(st + off, virt ? mv : mo, full, km ? row : kk0, km ? kk0 : tile, z);
        }
    }
    static constexpr unsigned FULL_COUNT = 4;  // one arrival (with its byte count) per producer warp
    __device__ __forceinline__ static void marker(unsigned long long *full, int, int lane)
    {
        if (lane == 0) mbar_arrive(full);
    }
};

// cp.async staging, into the same swizzled panels: any sizes and alignments (VEC = 1: 8-byte copies; VEC = 2:
// 16-byte copies, even row pitches and 16-byte aligned tensors) and any number of systems.  A pad element at the
// end of an odd row (VEC = 2) must be zero: in an X-major panel it stands at a contraction index.
template <int VEC>
struct CpStage {
    static constexpr unsigned FULL_COUNT = 129;  // every producer thread's copies, and the item context's writer

    __device__ __forceinline__ void begin(const Item &, const Role &, int, int) {}

    // One K-major panel: rows src[0 .. rows) of contraction indices 0 .. klim - 1 (ld apart), zeros elsewhere.
    __device__ __forceinline__ static void panel_k(char *dst, const double *src, int ld, int rows, int klim, int lane)
    {
        constexpr int KSTEP = VEC;  // 32 lanes cover 32 * VEC rows: VEC contraction indices per pass
        const int x = (lane * VEC) & 31, k0 = VEC == 2 ? lane >> 4 : 0;
        const bool row_ok = x < rows;
        const double *q = src + (row_ok ? x : 0) + (size_t)k0 * ld;
        char *d = dst + (x >> 4) * KBOX + ((x & 1) << 3);
        const int c = (x & 15) >> 1;
#pragma unroll 4
        for (int kk = k0; kk < DK; kk += KSTEP, q += (size_t)KSTEP * ld) {
            const bool ok = row_ok && kk < klim;
            char *w = d + kk * 128 + ((c ^ (kk & 7)) << 4);
            if (VEC == 2)
                cp_async_16(w, ok ? q : src, ok);
            else
                cp_async_8(w, ok ? q : src, ok);
        }
    }

    // One X-major panel: columns src + c ld, c < rows, of contraction indices 0 .. klim - 1 (contiguous).
    __device__ __forceinline__ static void panel_x(char *dst, const double *src, int ld, int rows, int klim, int lane)
    {
        constexpr int PER = DK / VEC, CSTEP = 32 / PER;  // copies per row, rows per pass
        const int dd = (lane & (PER - 1)) * VEC, r0 = lane / PER;
        const bool k_ok = dd < klim;
        const double *q = src + (k_ok ? dd : 0) + (size_t)r0 * ld;
#pragma unroll 4
        for (int r = r0; r < T; r += CSTEP, q += (size_t)CSTEP * ld) {
            const bool ok = k_ok && r < rows;
            char *w = dst + r * 128 + (((dd >> 1) ^ (r & 7)) << 4) + ((dd & 1) << 3);
            if (VEC == 2)
                cp_async_16(w, ok ? q : src, ok);
            else
                cp_async_8(w, ok ? q : src, ok);
        }
    }

    __device__ __forceinline__ void slot(const Item &it, const Role &r, int pw, char *st, unsigned long long *full,
                                         bool virt, int kk0, int fam, int lane)
    {
        const trpdrv_dev_system &S = *it.S;
        const int V = S.nvir, O = S.nocc, klim = (virt ? V : O) - kk0;
        const int ldv = S.ldv ? S.ldv : V, ldo = S.ldo ? S.ldo : O;
        if (!r.idle) {
#pragma unroll 1
            for (int q = 0; q < r.npanel; ++q) {
                int kind, tile, off;
                role_panel(it, r, pw, q, kind, tile, off);
                if (tile < 0) continue;
                // block of the operand's matrix
                const double *m;
                if (virt)
                    m = (kind == OP_AJ ? S.jvv : kind == OP_AK ? S.kvv : S.t2) +
                        (size_t)(kind < OP_B1 ? it.ai * O + it.za(fam) : it.zb(fam)) * ldv * V;
                else if (kind < OP_B1)
                    m = (kind == OP_AJ ? S.ntov : S.nxov) + (size_t)it.za(fam) * ldv * O;
                else
                    m = (kind == OP_B1 ? S.kov : S.jov) + (size_t)it.zb(fam) * ldo * V;
                const int ld = virt || kind < OP_B1 ? ldv : ldo;
                if (op_kmajor(kind, virt))
                    panel_k(st + off, m + tile + (size_t)kk0 * ld, ld, V - tile, klim, lane);
                else
                    panel_x(st + off, m + kk0 + (size_t)tile * ld, ld, V - tile, klim, lane);
            }
        }
        cp_async_arrive(full);
        if (pw == 0 && lane == 0) mbar_arrive(full);
    }
    __device__ __forceinline__ static void marker(unsigned long long *full, int pw, int lane)
    {
        cp_async_arrive(full);
        if (pw == 0 && lane == 0) mbar_arrive(full);
    }
};

template <class Stage>
__device__ __forceinline__ void producer(const trpdrv_dev_system *__restrict__ sys, int nsys, long long total, int pair_major,
                                         unsigned long long *counter, int *status, Stage &sg, char *stages,
                                         unsigned long long *full, unsigned long long *empty, ItemCtx *ring,
                                         long long *tickets, unsigned long long *tbar, int pw, int lane)
{
    const unsigned FULL = 0xffffffffu;
    int stage = 0;
    unsigned phase = 0;  // parity of the current pass over the stages
    long long next = 0;
    if (pw == 0) {
        if (lane == 0) next = (long long)atomicAdd(counter, 1ULL);
        next = __shfl_sync(FULL, next, 0);
    }
    for (long long n = 0;; ++n) {
        // warp 0 draws the tickets; the others read them from a ring (warp 0 is at most STAGES slots ahead: a stage
        // is released only after all four warps have filled it, and every ticket in the ring has a slot)
        const int tq = (int)(n % TICKETS);
        long long item;
        Item it;
        if (pw == 0) {
            for (;;) {
                item = next;
                if (item >= total) break;
                if (lane == 0) next = (long long)atomicAdd(counter, 1ULL);  // the following ticket, early
                next = __shfl_sync(FULL, next, 0);
                it = decode_item(sys, nsys, item, pair_major);
                if (!it.skip) break;
            }
            if (lane == 0) {
                tickets[tq] = item;
                mbar_arrive(&tbar[tq]);
            }
        } else {
            if (!mbar_wait(&tbar[tq], (unsigned)((n / TICKETS) & 1), status)) return;
            item = tickets[tq];
            if (item < total) it = decode_item(sys, nsys, item, pair_major);
        }
        ItemCtx &cx = ring[n % RING];
        if (item >= total || !it.ok) {
            if (!mbar_wait(&empty[stage], phase ^ 1, status)) return;
            if (pw == 0 && lane == 0) {
                cx.nch = 0;
                cx.packed = 0;
                if (item >= total) {
                    cx.state = -1;
                } else {
                    atomicOr(status, 1);
                    cx.state = 0;
                    cx.out = it.in_range ? it.S->partial + (size_t)it.own * NCW * 4 : nullptr;
                }
            }
            Stage::marker(&full[stage], pw, lane);
            if (item >= total) return;
            if (++stage == STAGES) {
                stage = 0;
                phase ^= 1;
            }
            continue;
        }
        if (pw == 0 && lane == 0) write_ctx(cx, it);
        const Role role(it, pw);
        sg.begin(it, role, pw, lane);
        const int nV = (it.S->nvir + DK - 1) / DK, nch = nV + (it.S->nocc + DK - 1) / DK;
        // packed items: one slot per (chunk, family)
        const int f0 = it.pack ? 0 : role.fam, f1 = it.pack ? (it.same ? 1 : 2) : role.fam + 1;
        for (int ch = 0; ch < nch; ++ch) {
            const bool virt = ch < nV;
            const int kk0 = (virt ? ch : ch - nV) * DK;
            for (int f = f0; f < f1; ++f) {
                if (!mbar_wait(&empty[stage], phase ^ 1, status)) return;
                sg.slot(it, role, pw, stages + (size_t)stage * STAGE_BYTES, &full[stage], virt, kk0, f, lane);
                if (++stage == STAGES) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        if (it.diag) {  // a slot for the consumers' exchange
            if (!mbar_wait(&empty[stage], phase ^ 1, status)) return;
            Stage::marker(&full[stage], pw, lane);
            if (++stage == STAGES) {
                stage = 0;
                phase ^= 1;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Releases the n stage slots of an item whose sub-block of this warp lies entirely in the padding.
__device__ __forceinline__ bool skip_slots(int n, const Pipe &pp, RingPos &rp)
{
    for (; n > 0; --n) {
        if (!pp.wait(rp)) return false;
        pp.release(rp);
    }
    return true;
}

// Place of (row, col) in a 32x32 exchange tile: the half-warp's four rows {0,6,1,7} or {2,4,3,5} (mod 8) and four
// columns, and the same with the roles swapped, fall in 16 different bank pairs.
__device__ __forceinline__ int xch_off(int row, int col) { return row * T + (col ^ ((row & 3) << 2)); }

// i == k: the t family's operands are the n family's, so its products are the same numbers.
__device__ __forceinline__ void copy_families(double (&f)[8][4], double (&gT)[8][4])
{
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            f[4 + x][e] = f[x][e];
            gT[4 + x][e] = gT[x][e];
        }
}

// ------------------------------------------------------------------------------------------------
// The tensor maps travel as a kernel parameter of the TMA instantiations only.
template <int STG> struct StageParam {
    Maps maps;
};
struct NoParam {
    int unused;
};
template <> struct StageParam<1> : NoParam {};
template <> struct StageParam<2> : NoParam {};

// STG: operand staging, 0 = TMA, 1 / 2 = cp.async with 8 / 16-byte copies.  KS: FP64 MMA shape.
template <int KS, int STG>
__global__ void __launch_bounds__(NTHREAD, 1)
fused_kernel(const trpdrv_dev_system *__restrict__ sys, int nsys, long long total, int pair_major,
             unsigned long long *counter, int *status, const __grid_constant__ StageParam<STG> param)
{
    extern __shared__ char smem_raw[];
    __shared__ __align__(8) unsigned long long full[STAGES], empty[STAGES], tbar[TICKETS];
    __shared__ ItemCtx ring[RING];
    __shared__ long long tickets[TICKETS];
    __shared__ __align__(8) unsigned long long xbar[1];     // diagonal-pair exchange
    // aligned by an offset, not by integer arithmetic on the pointer: the compiler then still knows that the
    // fragment reads are shared-memory loads (32-bit addresses)
    char *stages = smem_raw + ((1024u - (saddr(smem_raw) & 1023u)) & 1023u);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], STG ? CpStage<1>::FULL_COUNT : TmaStage::FULL_COUNT);
            mbar_init(&empty[s], NCW);
        }
        for (int q = 0; q < TICKETS; ++q) mbar_init(&tbar[q], 1);
        mbar_init(xbar, NCW);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp >= NCW) {  // producer warpgroup
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_PRODUCER));
        if constexpr (STG == 0) {
            TmaStage sg;
            sg.maps = &param.maps;
            producer(sys, nsys, total, pair_major, counter, status, sg, stages, full, empty, ring, tickets, tbar, warp - NCW,
                            lane);
        } else {
            CpStage<STG> sg;
            producer(sys, nsys, total, pair_major, counter, status, sg, stages, full, empty, ring, tickets, tbar, warp - NCW,
                            lane);
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REG_CONSUMER));

    const int g = lane >> 2, t = lane & 3;
    // sub-block: rows (b) rs*16.., columns (c) cs*8..; warps w and w+4 share a scheduler and differ in both
    const int rs = warp >> 2, cs = (warp & 3) ^ (rs << 1);
    const int rx0 = rs * 16, cx0 = cs * 8;
    const FragOffsets fo(rx0, cx0, g, t);

    double f[8][4], gT[8][4];
    const Pipe pipe = {stages, full, empty, status, lane};
    RingPos rp = {0, 0u, false};
    unsigned xphase = 0;
    for (long long n = 0;; ++n) {
        if (!pipe.wait(rp)) return;
        rp.ready = true;
        const ItemCtx &cx = ring[n % RING];
        const int state = cx.state;
        if (state < 0) return;
        if (state == 0) {
            if (lane == 0 && cx.out) {
                double *o = cx.out + warp * 4;
                o[0] = o[1] = o[2] = o[3] = 0.0;
            }
            pipe.release(rp);
            continue;
        }
#pragma unroll
        for (int x = 0; x < 8; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) f[x][e] = gT[x][e] = 0.0;
        const ChunkCounts nc(cx.nvir, cx.nocc);
        const bool same = cx.same != 0;
        prefetch_epilogue(cx, lane);
        if (cx.packed) {
            // two edge pairs (b0, c0) and (b1, c0): warp w takes pair w >> 2, sub-block w & 3 of it; each
            // (chunk, family) has its own stage slot
            const int pair = warp >> 2, sub = warp & 3, prs = sub >> 1, pcs = sub & 1;
            const int pb0 = pair ? cx.b1 : cx.b0;
            if (pb0 >= 0 && cx.c0 + pcs * 8 < cx.nvir) {
                const FragOffsets fp(prs * 16, pcs * 8, g, t);
                const Panels pn = packed_panels(pair);
                if (!(same ? run_packed_item<KS, true>(nc, fp, pn, pipe, rp, f, gT)
                           : run_packed_item<KS, false>(nc, fp, pn, pipe, rp, f, gT)))
                    return;
            } else if (!skip_slots(same ? cx.nch : 2 * cx.nch, pipe, rp)) {
                return;
            }
            if (same) copy_families(f, gT);
            if (pb0 >= 0) {  // this pair's slots: the 4 sub-blocks' sums, zeros in the other 4
                double *out = pair ? cx.out1 : cx.out;
                warp_epilogue<false>(cx, f, gT, pb0 + prs * 16, cx.c0 + pcs * 8, g, t, lane, out + sub * 4);
                if (lane == 0) {
                    double *z = out + (sub + 4) * 4;
                    z[0] = z[1] = z[2] = z[3] = 0.0;
                }
            }
            continue;
        }
        const bool diag = cx.diag != 0;
        if (cx.b0 + rx0 < cx.nvir && cx.c0 + cx0 < cx.nvir) {
            bool ok;
            if (!same)
                ok = diag ? run_item<KS, true, false>(nc, fo, pipe, rp, f, gT)
                          : run_item<KS, false, false>(nc, fo, pipe, rp, f, gT);
            else
                ok = diag ? run_item<KS, true, true>(nc, fo, pipe, rp, f, gT)
                          : run_item<KS, false, true>(nc, fo, pipe, rp, f, gT);
            if (!ok) return;
        } else if (!skip_slots(cx.nch, pipe, rp)) {  // only padding
            return;
        }
        if (diag) {
            // f(c,b) of a diagonal pair is f at the mirrored position of the same 32x32 block, held by another
            // warp.  The item has one more stage slot, which the producers leave empty: all tiles (8 KB each, rows
            // of 256 bytes with the columns XORed so that neither the writes nor the mirrored reads conflict)
            // are exchanged through it with one consumer-only mbarrier (bounded wait; no CTA-wide barrier).
            if (!pipe.wait(rp)) return;
            double *xt = reinterpret_cast<double *>(stages + (size_t)rp.stage * STAGE_BYTES);
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                if (x == 4 && same) break;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = rx0 + perm8(g) + ((e & 2) ? 8 : 0), col = cx0 + perm8(2 * t + (e & 1));
                    xt[x * T * T + xch_off(row, col)] = f[x][e];
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(xbar);
            if (!mbar_wait(xbar, xphase, status)) return;
            xphase ^= 1;
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                if (x == 4 && same) break;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = rx0 + perm8(g) + ((e & 2) ? 8 : 0), col = cx0 + perm8(2 * t + (e & 1));
                    gT[x][e] = xt[x * T * T + xch_off(col, row)];
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // before the slot's next TMA writes
            pipe.release(rp);
        }
        if (same) copy_families(f, gT);
        if (diag)
            warp_epilogue<true>(cx, f, gT, cx.b0 + rx0, cx.c0 + cx0, g, t, lane, cx.out + warp * 4);
        else
            warp_epilogue<false>(cx, f, gT, cx.b0 + rx0, cx.c0 + cx0, g, t, lane, cx.out + warp * 4);
    }
}

// ------------------------------------------------------------------------------------------------
// host side: tensor maps
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

// 3-D map over doubles: dims {d0 (contiguous), d1, d2}, box {b0, b1, 1}
static int make_map(CUtensorMap *m, const double *base, unsigned long long d0, unsigned long long d1,
                    unsigned long long d2, unsigned b0, unsigned b1, bool swizzle)
{
    PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
    if (!fn) return 1;
    const cuuint64_t dims[3] = {d0, d1, d2};
    const cuuint64_t strides[2] = {d0 * 8ull, d0 * d1 * 8ull};
    const cuuint32_t box[3] = {b0, b1, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE,
                          swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 2;
}

}  // namespace tma
}  // namespace trpdrv

using namespace trpdrv;

extern "C" size_t trpdrv_tma_maps_bytes(void) { return sizeof(tma::StageParam<0>); }

// Registers per thread the kernel is launched with (read back at init).  The setmaxnreg split is
// only valid when this equals REG_LAUNCH: with fewer, the consumers' increase could never be met.
static int g_launch_regs = -1;

extern "C" int trpdrv_tma_supported(const trpdrv_dev_system *h_sys, int nsys)
{
    if (g_launch_regs != tma::REG_LAUNCH) return 0;
    if (nsys > TRPDRV_TMA_MAX_SYSTEMS || !tma::encode_fn()) return 0;
    for (int s = 0; s < nsys; ++s) {
        const trpdrv_dev_system &S = h_sys[s];
        if ((S.nvir & 1) || (S.nocc & 1)) return 0;  // row strides must be multiples of 16 bytes
        const void *p[] = {S.t2, S.jvv, S.kvv, S.ntov, S.nxov, S.jov, S.kov};
        for (const void *q : p)
            if (((uintptr_t)q) & 15u) return 0;
    }
    return 1;
}

// Packing needs at least two edge pairs and an edge tile of at most 16 valid columns (two 8-wide
// column blocks per pair).  TRPDRV_TMA_PACK_EDGE=0 keeps the edge pairs as ordinary items.
extern "C" int trpdrv_tma_pack_edge(int nvir)
{
    const char *v = getenv("TRPDRV_TMA_PACK_EDGE");
    if (v && v[0] == '0') return 0;
    const int nb = (nvir + tma::T - 1) / tma::T, w = nvir - (nb - 1) * tma::T;
    return nb >= 3 && w >= 1 && w <= 16;
}

extern "C" int trpdrv_tma_prepare(const trpdrv_dev_system *h_sys, int nsys, void *maps_out)
{
    tma::Maps *M = static_cast<tma::Maps *>(maps_out);
    memset(M, 0, sizeof(*M));
    for (int s = 0; s < nsys && s < TRPDRV_TMA_MAX_SYSTEMS; ++s) {
        const trpdrv_dev_system &S = h_sys[s];
        const unsigned long long V = S.nvir, O = S.nocc;
        CUtensorMap *m = M->m[s];
        int e = 0;
        const unsigned long long OA = O * (unsigned long long)(S.n_a > 0 ? S.n_a : 1), O2 = O * O;
        e |= tma::make_map(&m[tma::M_J], S.jvv, V, V, OA, 16, tma::DK, true);    // [a][i][d][b]
        e |= tma::make_map(&m[tma::M_K], S.kvv, V, V, OA, 16, tma::DK, true);
        e |= tma::make_map(&m[tma::M_NT], S.ntov, V, O, O, 16, tma::DK, true);   // [i][m][b]
        e |= tma::make_map(&m[tma::M_NX], S.nxov, V, O, O, 16, tma::DK, true);
        e |= tma::make_map(&m[tma::M_T2K], S.t2, V, V, O2, 16, tma::DK, true);   // [jx][d][c]: T(c,d)
        e |= tma::make_map(&m[tma::M_T2X], S.t2, V, V, O2, tma::DK, 32, true);  // [jx][c][d]: T(d,c)
        e |= tma::make_map(&m[tma::M_JOV], S.jov, O, V, O2, tma::DK, 32, true);  // [jx][c][m]
        e |= tma::make_map(&m[tma::M_KOV], S.kov, O, V, O2, tma::DK, 32, true);
        if (e) return e;
    }
    return 0;
}

template <int KS, int STG>
static int launch_kernel(const trpdrv_dev_system *d_sys, int nsys, int64_t total, int pair_major,
                         unsigned long long *counter, int *status, int grid, const tma::StageParam<STG> &param, void *stream)
{
    tma::fused_kernel<KS, STG><<<grid, tma::NTHREAD, tma::SMEM_BYTES, (cudaStream_t)stream>>>(
        d_sys, nsys, total, pair_major, counter, status, param);
    return (int)cudaGetLastError();
}

extern "C" int trpdrv_launch_fused_tma(const trpdrv_dev_system *d_sys, int nsys, int64_t total_items,
                                       int pair_major, unsigned long long *counter, int *status, int grid, const void *maps,
                                       int mma_k, void *stream)
{
    if (grid <= 0 || total_items <= 0) return 0;
    if (g_launch_regs != tma::REG_LAUNCH) return (int)cudaErrorInvalidConfiguration;
    if (nsys > TRPDRV_TMA_MAX_SYSTEMS) return (int)cudaErrorInvalidValue;
    const tma::StageParam<0> &m = *static_cast<const tma::StageParam<0> *>(maps);
    if (mma_k == 16)
        return launch_kernel<16, 0>(d_sys, nsys, total_items, pair_major, counter, status, grid, m, stream);
    if (mma_k == 8)
        return launch_kernel<8, 0>(d_sys, nsys, total_items, pair_major, counter, status, grid, m, stream);
    return (int)cudaErrorInvalidValue;
}

extern "C" int trpdrv_launch_fused(const trpdrv_dev_system *d_sys, int nsys, int64_t total_items,
                                   int pair_major, unsigned long long *counter, int *status, int grid, int vec2, int mma_k,
                                   void *stream)
{
    if (grid <= 0 || total_items <= 0) return 0;
    if (g_launch_regs != tma::REG_LAUNCH) return (int)cudaErrorInvalidConfiguration;
    const tma::StageParam<1> p1 = {};
    const tma::StageParam<2> p2 = {};
    if (mma_k == 4)
        return vec2 ? launch_kernel<4, 2>(d_sys, nsys, total_items, pair_major, counter, status, grid, p2, stream)
                    : launch_kernel<4, 1>(d_sys, nsys, total_items, pair_major, counter, status, grid, p1, stream);
    return vec2 ? launch_kernel<8, 2>(d_sys, nsys, total_items, pair_major, counter, status, grid, p2, stream)
                : launch_kernel<8, 1>(d_sys, nsys, total_items, pair_major, counter, status, grid, p1, stream);
}

extern "C" int trpdrv_launch_wait_selftest(unsigned long long limit_ns, int *status, unsigned long long *elapsed_ns,
                                           void *stream)
{
    tma::bounded_wait_selftest_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(limit_ns, status, elapsed_ns);
    return (int)cudaGetLastError();
}

// Every instantiation must be launched with REG_LAUNCH registers per thread (the setmaxnreg split
// assumes it); g_launch_regs holds the common value, or 0 when they differ.
template <int KS, int STG>
static cudaError_t init_kernel(int *regs)
{
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, tma::fused_kernel<KS, STG>);
    if (e != cudaSuccess) return e;
    *regs = *regs < 0 || *regs == a.numRegs ? a.numRegs : 0;
    return cudaFuncSetAttribute(tma::fused_kernel<KS, STG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tma::SMEM_BYTES);
}

extern "C" int trpdrv_fused_tma_init(void)
{
    int regs = -1;
    cudaError_t e = init_kernel<8, 0>(&regs);
    if (e == cudaSuccess) e = init_kernel<16, 0>(&regs);
    if (e == cudaSuccess) e = init_kernel<8, 1>(&regs);
    if (e == cudaSuccess) e = init_kernel<8, 2>(&regs);
    if (e == cudaSuccess) e = init_kernel<4, 1>(&regs);
    if (e == cudaSuccess) e = init_kernel<4, 2>(&regs);
    if (e == cudaSuccess) g_launch_regs = regs;
    return (int)e;
}
