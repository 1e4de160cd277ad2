// FP32 parity form of the triples body: the single-precision variant of the reference
// (gpu-omp/ccsd_trpdrv_omp_cbody.c:38-226, 16 cblas_sgemm calls and the float tengy loop, and
// gpu-omp/ccsd_tengy_c99.c:5-119) on the GPU, built into its own library, libtrpdrv_b200_fp32.so,
// because its entry points keep the reference's names with float arguments
// (gpu-omp/test.c:24-62).  It exists to compare with that variant's numbers, not for speed:
//
//  * sgemm_group_kernel: the eight f = A1 op(B1) - A2 B2 of one triple in IEEE FP32 (FFMA, no TF32), 64 x 64 or
//    (few tiles) 32 x 32 outputs per CTA, 16-index contraction chunks staged by cp.async three deep, 4 x 4
//    outputs per thread;
//  * tengy_f32_kernel: the (b,c) sum of the reference's float energy forms over 16 x 16 tile pairs (the denominator
//    formed as the reference forms it: -1.0 / (float sum), a double division rounded to float), float partial
//    sums per tile pair, which the last CTA sums in a fixed order and writes to pinned host memory.
//
// A call is bound by the host: its slices are compared with a pinned mirror and sent in one or two pieces (stage.h).
// All arithmetic of the energies is float, like the reference's (its emp4i..emp5k are float).

#include <cuda_runtime.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "stage.h"
#include "trpdrv_fp32.h"

namespace trpdrv {
namespace f32 {

constexpr int KB = 16;     // contraction chunk
constexpr int STAGES = 3;
constexpr int TT = 16;     // tengy tile edge
constexpr int NT = TT * TT;

struct GemmArgs {
    int nocc, nvir, ldv, ldo;  // ldv, ldo: row lengths of nvir and nocc floats, multiples of 4 (zero pads)
    const float *a1[8], *b1[8], *a2[8], *b2[8];
    int b1_t[8];  // 1: B1 enters transposed (B1'(d, c) = B1[c + d ldv])
    float *f;     // [8][nvir][nvir]
    unsigned *counter;  // zeroed for the energy kernel that follows
};

__device__ __forceinline__ void cp16(float *smem, const float *gmem, bool ok)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}

// Threads of a CTA of BT x BT outputs, and one stage: A K-major [KB][BT + 4]; B K-major the same or X-major
// [BT][KB + 4] (pitch 20: eight columns' float4 fall in eight different 16-byte bank groups).
template <int BT> struct Tile {
    static constexpr int THREADS = (BT / 4) * (BT / 4);
    static constexpr int PK = BT + 4, PX = KB + 4;
    static constexpr int APANEL = KB * PK, BPANEL = APANEL > BT * PX ? APANEL : BT * PX;
    static constexpr int STAGE = APANEL + BPANEL;
};

// f_x(b, c) = sum_d A1(b, d) B1'(d, c) - sum_m A2(b, m) B2(m, c), column-major like the reference; each output one
// FFMA chain in the order d, then m.
template <int BT>
__global__ void __launch_bounds__(Tile<BT>::THREADS) sgemm_group_kernel(const __grid_constant__ GemmArgs P)
{
    using L = Tile<BT>;
    constexpr int W = BT / 4;  // threads along a tile edge
    __shared__ __align__(16) float sm[STAGES][L::STAGE];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if ((blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x) == 0) *P.counter = 0u;
    const int x = blockIdx.z, V = P.nvir, O = P.nocc, tid = threadIdx.x;
    const int b0 = blockIdx.x * BT, c0 = blockIdx.y * BT;
    const int tx = tid % W, ty = tid / W;
    const float *A1 = P.a1[x], *B1 = P.b1[x], *A2 = P.a2[x], *B2 = P.b2[x];
    const int bt = P.b1_t[x], nV = (V + KB - 1) / KB, nch = nV + (O + KB - 1) / KB;

    auto load = [&](int ch) {
        if (ch < nch) {
            const bool occ = ch >= nV;
            const int k0 = (occ ? ch - nV : ch) * KB, K = occ ? O : V;
            float *As = sm[ch % STAGES], *Bs = As + L::APANEL;
            const float *A = occ ? A2 : A1, *B = occ ? B2 : B1;
            for (int e = tid; e < KB * W; e += L::THREADS) {  // rows b contiguous
                const int k = e / W, r = (e % W) * 4;
                const bool ok = b0 + r < P.ldv && k0 + k < K;
                cp16(As + k * L::PK + r, ok ? A + (b0 + r) + (size_t)(k0 + k) * P.ldv : A, ok);
            }
            if (!occ && bt) {
                for (int e = tid; e < KB * W; e += L::THREADS) {
                    const int k = e / W, c = (e % W) * 4;
                    const bool ok = c0 + c < P.ldv && k0 + k < K;
                    cp16(Bs + k * L::PK + c, ok ? B + (c0 + c) + (size_t)(k0 + k) * P.ldv : B, ok);
                }
            } else {  // contraction contiguous; a row's pad holds zeros
                const int ld = occ ? P.ldo : P.ldv;
                for (int e = tid; e < BT * (KB / 4); e += L::THREADS) {
                    const int c = e / (KB / 4), k = (e % (KB / 4)) * 4;
                    const bool ok = c0 + c < V && k0 + k < ld;
                    cp16(Bs + c * L::PX + k, ok ? B + (k0 + k) + (size_t)(c0 + c) * ld : B, ok);
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };

    float acc[4][4] = {};
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) load(s);
    for (int ch = 0; ch < nch; ++ch) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
        __syncthreads();
        load(ch + STAGES - 1);
        const float *As = sm[ch % STAGES], *Bs = As + L::APANEL;
        const bool occ = ch >= nV;
        const float sg = occ ? -1.0f : 1.0f;
        const bool bk = !occ && bt;
#pragma unroll
        for (int k4 = 0; k4 < KB / 4; ++k4) {
            float bv[4][4];  // [kk][w]
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const int c = tx + W * w;
                if (bk) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) bv[q][w] = Bs[(4 * k4 + q) * L::PK + c];
                } else {
                    const float4 v = *reinterpret_cast<const float4 *>(Bs + c * L::PX + 4 * k4);
                    bv[0][w] = v.x;
                    bv[1][w] = v.y;
                    bv[2][w] = v.z;
                    bv[3][w] = v.w;
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 a = *reinterpret_cast<const float4 *>(As + (4 * k4 + q) * L::PK + 4 * ty);
                const float av[4] = {sg * a.x, sg * a.y, sg * a.z, sg * a.w};
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int w = 0; w < 4; ++w) acc[u][w] = fmaf(av[u], bv[q][w], acc[u][w]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    float *F = P.f + (size_t)x * V * V;
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const int b = b0 + 4 * ty + u, c = c0 + tx + W * w;
            if (b < V && c < V) F[b + (size_t)c * V] = acc[u][w];
        }
}

struct TengyArgs {
    int ncor, nocc, nvir;
    float eaijk;
    const float *f;  // f1n f2n f3n f4n f1t f2t f3t f4t
    const float *eorb, *dintc1, *dintx1, *t1v1, *dintc2, *dintx2, *t1v2;
    float *pair;     // [npairs][4]
    unsigned *counter;
    float *out;      // emp4i, emp5i, emp4k, emp5k
};

// the reference's float forms at one (b, c): gpu-omp/ccsd_trpdrv_omp_cbody.c:176-217
__device__ __forceinline__ void term(const TengyArgs &P, const float (&bc)[8], const float (&cb)[8], float denom, int b,
                                     int c, float (&s)[4])
{
    const float n1bc = bc[0], n2bc = bc[1], n3bc = bc[2], n4bc = bc[3];
    const float t1bc = bc[4], t2bc = bc[5], t3bc = bc[6], t4bc = bc[7];
    const float n1cb = cb[0], n2cb = cb[1], n3cb = cb[2], n4cb = cb[3];
    const float t1cb = cb[4], t2cb = cb[5], t3cb = cb[6], t4cb = cb[7];
    s[0] += denom * (t1bc + n1cb + t2cb + n3bc + n4cb) * (t1bc - t2bc * 2 - t3bc * 2 + t4bc)
          - denom * (n1bc + t1cb + n2cb + n3cb) * (t1bc * 2 - t2bc - t3bc + t4bc * 2)
          + denom * 3 * (n1bc * (n1bc + n3cb + t4cb * 2) + n2bc * t2cb + n3bc * t4bc);
    s[2] += denom * (n1bc + t1cb + n2cb + t3bc + t4cb) * (n1bc - n2bc * 2 - n3bc * 2 + n4bc)
          - denom * (t1bc + n1cb + t2cb + t3cb) * (n1bc * 2 - n2bc - n3bc + n4bc * 2)
          + denom * 3 * (t1bc * (t1bc + t3cb + n4cb * 2) + t2bc * n2cb + t3bc * n4bc);
    const float t1v1b = P.t1v1[b], t1v2b = P.t1v2[b];
    const float dx1c = P.dintx1[c], dx2c = P.dintx2[c], dc1c = P.dintc1[c], dc2c = P.dintc2[c];
    s[1] += denom * t1v1b * dx1c * (t1bc + n2bc + n4cb - (t3bc + n4bc + n2cb + n1bc + t2bc + n3cb) * 2
                                    + (n3bc + t4bc + n1cb) * 4)
          + denom * t1v1b * dc1c * (n1bc + n4bc + t1cb - (n2bc + n3bc + t2cb) * 2);
    s[3] += denom * t1v2b * dx2c * (n1bc + t2bc + t4cb - (n3bc + t4bc + t2cb + t1bc + n2bc + t3cb) * 2
                                    + (t3bc + n4bc + t1cb) * 4)
          + denom * t1v2b * dc2c * (t1bc + t4bc + n1cb - (t2bc + t3bc + n2cb) * 2);
}

// The CTA's sums of the four values, in thread q < 4's s[0] (a fixed order).
__device__ __forceinline__ float block_sum(const float (&s)[4], float (&red)[4][NT / 32])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float v = s[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[q][warp] = v;
    }
    __syncthreads();
    float v = 0.0f;
    if (threadIdx.x < 4)
        for (int w = 0; w < NT / 32; ++w) v += red[threadIdx.x][w];
    __syncthreads();
    return v;
}

// one CTA per 16 x 16 tile pair (B <= C), one thread per (b, c): the terms of (b, c) and, for B < C, of (c, b); the
// mirrored tile's values cross through shared memory, so every load is coalesced
__global__ void __launch_bounds__(NT) tengy_f32_kernel(const __grid_constant__ TengyArgs P)
{
    __shared__ float xch[8][TT][TT + 1];
    __shared__ float red[4][NT / 32];
    __shared__ int last;
    const int V = P.nvir, nb = (V + TT - 1) / TT, tid = threadIdx.x;
    int B = 0, rem = blockIdx.x;
    while (rem >= nb - B) {
        rem -= nb - B;
        ++B;
    }
    const int C = B + rem, r = tid & (TT - 1), q = tid / TT;
    const int b = B * TT + r, c = C * TT + q, cr = C * TT + r, bq = B * TT + q;
    const size_t vv = (size_t)V * V;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // f and the counter come from the launch before
    float fbc[8], fcb[8];
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        fbc[x] = b < V && c < V ? __ldcg(P.f + x * vv + b + (size_t)c * V) : 0.0f;
        fcb[x] = cr < V && bq < V ? __ldcg(P.f + x * vv + cr + (size_t)bq * V) : 0.0f;
    }
#pragma unroll
    for (int x = 0; x < 8; ++x) xch[x][q][r] = fcb[x];
    __syncthreads();
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (b < V && c < V) {
#pragma unroll
        for (int x = 0; x < 8; ++x) fcb[x] = xch[x][r][q];
        const float denom = (float)(-1.0 / (double)(P.eorb[P.ncor + P.nocc + b] + P.eorb[P.ncor + P.nocc + c] + P.eaijk));
        term(P, fbc, fcb, denom, b, c, s);
        if (B != C) term(P, fcb, fbc, denom, c, b, s);
    }
    const float v = block_sum(s, red);
    if (tid < 4) P.pair[4 * (size_t)blockIdx.x + tid] = v;
    if (tid < 4) __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(P.counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (unsigned p = tid; p < gridDim.x; p += NT)
#pragma unroll
        for (int u = 0; u < 4; ++u) t[u] += __ldcg(P.pair + 4 * (size_t)p + u);
    const float o = block_sum(t, red);
    if (tid < 4) P.out[tid] = o;
    if (tid == 0) *P.counter = 0u;
}

// ------------------------------------------------------------------------------------------------
// host state: one device, one stream, buffers grown to the largest shape seen
// ------------------------------------------------------------------------------------------------
// Staging layout as in the double-precision library (host.c): I = tij jia kia tia xia jij kij, K = the same blocks of
// the k role, then dintc1 dintx1 t1v1 dintc2 dintx2 t1v2 eorb.  Rows are padded to multiples of 4 floats.
enum { DS_I = 0, DS_K = 7, DS_VEC = 14, DS_N = 21 };
enum { DS_T = 0, DS_J, DS_KV, DS_TO, DS_XO, DS_JO, DS_KO };
constexpr size_t SEGMENT = (size_t)512 << 10;

struct State {
    int ready, ncor, nocc, nvir;
    cudaStream_t st;
    size_t off[DS_N + 1], cap_stage, cap_f, cap_pair, cap_vec;
    float *d_stage, *h_stage, *f, *pair, *vec;
    unsigned *counter;
    float *h_out;  // pinned, 4 floats: the energy kernel writes it
};
State g;
pthread_mutex_t g_mu = PTHREAD_MUTEX_INITIALIZER;
thread_local char t_msg[256];
thread_local int t_status;

int fail(int status, const char *msg)
{
    snprintf(t_msg, sizeof t_msg, "%s", msg);
    t_status = status;
    return status;
}

#define F32_TRY(call)                                                                   \
    do {                                                                                \
        const cudaError_t e_ = (call);                                                  \
        if (e_ != cudaSuccess) {                                                        \
            char m_[200];                                                               \
            cudaGetLastError(); /* reported here: the next launch's check must not find it */ \
            snprintf(m_, sizeof m_, "%s: %s", #call, cudaGetErrorString(e_));          \
            return fail(e_ == cudaErrorMemoryAllocation ? 3 : 2, m_);                   \
        }                                                                               \
    } while (0)

int dev_alloc(void **p, size_t bytes) { return (int)cudaMalloc(p, bytes); }
void dev_release(void *p) { cudaFree(p); }

// *cap in bytes
int grow(float **p, size_t *cap, size_t want)
{
    F32_TRY((cudaError_t)stage_grow((void **)p, cap, sizeof(float) * want, dev_alloc, dev_release));
    return 0;
}

int pitch4(int n) { return (n + 3) & ~3; }

int reserve(int nvir, int nbf)
{
    if (!g.ready) {
        int dev = 0, major = 0;
        F32_TRY(cudaGetDevice(&dev));
        F32_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
        if (major != 10) return fail(4, "the current device is not sm_100");
        F32_TRY(cudaStreamCreateWithFlags(&g.st, cudaStreamNonBlocking));
        F32_TRY(cudaMalloc((void **)&g.counter, sizeof(unsigned)));
        F32_TRY(cudaMemset(g.counter, 0, sizeof(unsigned)));
        F32_TRY(cudaMallocHost((void **)&g.h_out, sizeof(float) * 4));
        g.ready = 1;
    }
    const size_t vv = (size_t)nvir * nvir, nb = (size_t)(nvir + TT - 1) / TT;
    if (int rc = grow(&g.f, &g.cap_f, 8 * vv)) return rc;
    if (int rc = grow(&g.pair, &g.cap_pair, 4 * (nb * (nb + 1) / 2))) return rc;
    return grow(&g.vec, &g.cap_vec, 6 * (size_t)nvir + (size_t)nbf);
}

// Lays the staging block out for this shape and clears it (the pads must be zero, and mirror and device equal).
int layout(int ncor, int nocc, int nvir)
{
    if (g.cap_stage && g.ncor == ncor && g.nocc == nocc && g.nvir == nvir) return 0;
    g.nvir = 0;  // no valid layout until the end
    const size_t V = (size_t)nvir, O = (size_t)nocc, ldv = (size_t)pitch4(nvir), ldo = (size_t)pitch4(nocc);
    const size_t role[7] = {ldv * V, ldv * V, ldv * V, ldv * O, ldv * O, ldo * V, ldo * V};
    size_t o = 0;
    for (int q = 0; q < DS_N; ++q) {
        g.off[q] = o;
        const size_t n = q < DS_VEC ? role[q % 7] : q < DS_N - 1 ? V : (size_t)(ncor + nocc + nvir);
        o += (n + 31) & ~(size_t)31;
    }
    F32_TRY(cudaStreamSynchronize(g.st));  // no transfer of a failed call still reads the mirror
    if (o > g.cap_stage) {
        if (g.d_stage) cudaFree(g.d_stage);
        if (g.h_stage) cudaFreeHost(g.h_stage);
        g.d_stage = g.h_stage = nullptr;
        g.cap_stage = 0;
        F32_TRY(cudaMalloc((void **)&g.d_stage, sizeof(float) * o));
        F32_TRY(cudaMallocHost((void **)&g.h_stage, sizeof(float) * o));
        g.cap_stage = o;
    }
    memset(g.h_stage, 0, sizeof(float) * o);
    F32_TRY(cudaMemsetAsync(g.d_stage, 0, sizeof(float) * o, g.st));
    g.ncor = ncor;
    g.nocc = nocc;
    g.nvir = nvir;
    return 0;
}

int send(void *, char *lo, char *hi)
{
    const size_t a = (size_t)(lo - (char *)g.h_stage), n = (size_t)(hi - lo);
    F32_TRY(cudaMemcpyAsync((char *)g.d_stage + a, (char *)g.h_stage + a, n, cudaMemcpyHostToDevice, g.st));
    return 0;
}

int h2d(float *dst, const float *src, size_t n)
{
    F32_TRY(cudaMemcpyAsync(dst, src, sizeof(float) * n, cudaMemcpyHostToDevice, g.st));
    return 0;
}

// The energies of the f at g.f; a programmatic dependent of the launch before it on the stream.
int launch_tengy(int ncor, int nocc, int nvir, float eaijk, const float *const *vec, const float *eorb, float *out4)
{
    TengyArgs T;
    T.ncor = ncor;
    T.nocc = nocc;
    T.nvir = nvir;
    T.eaijk = eaijk;
    T.f = g.f;
    T.eorb = eorb;
    T.dintc1 = vec[0];
    T.dintx1 = vec[1];
    T.t1v1 = vec[2];
    T.dintc2 = vec[3];
    T.dintx2 = vec[4];
    T.t1v2 = vec[5];
    T.pair = g.pair;
    T.counter = g.counter;
    T.out = g.h_out;
    const unsigned nb = (unsigned)(nvir + TT - 1) / TT;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nb * (nb + 1) / 2);
    cfg.blockDim = dim3(NT);
    cfg.stream = g.st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    F32_TRY(cudaLaunchKernelEx(&cfg, tengy_f32_kernel, T));
    F32_TRY(cudaStreamSynchronize(g.st));
    for (int q = 0; q < 4; ++q) out4[q] = g.h_out[q];
    return 0;
}

int body(float *f1n, float *f1t, float *f2n, float *f2t, float *f3n, float *f3t, float *f4n, float *f4t,
         const float *eorb, const int *ncor_, const int *nocc_, const int *nvir_, float *emp4_, float *emp5_,
         const int *a_, const int *i_, const int *j_, const int *k_, const int *klo_, const float *tij,
         const float *tkj, const float *tia, const float *tka, const float *xia, const float *xka, const float *jia,
         const float *jka, const float *kia, const float *kka, const float *jij, const float *jkj, const float *kij,
         const float *kkj, const float *dintc1, const float *dintx1, const float *t1v1, const float *dintc2,
         const float *dintx2, const float *t1v2)
{
    if (!ncor_ || !nocc_ || !nvir_ || !a_ || !i_ || !j_ || !k_ || !klo_ || !emp4_ || !emp5_ || !eorb)
        return fail(1, "NULL argument");
    const int ncor = *ncor_, nocc = *nocc_, nvir = *nvir_, a = *a_, i = *i_, j = *j_, k = *k_, klo = *klo_;
    const float *arr[] = {tij, tkj, tia, tka, xia, xka, jia, jka, kia, kka, jij, jkj, kij, kkj,
                          dintc1, dintx1, t1v1, dintc2, dintx2, t1v2};
    for (const float *p : arr)
        if (!p) return fail(1, "NULL array argument");
    if (nocc < 1 || nvir < 1 || ncor < 0 || nocc > 1023 || nvir > 16384) return fail(1, "ncor/nocc/nvir out of range");
    const int nbf = ncor + nocc + nvir;
    if (a < 1 || a > nbf || i < 1 || i > nocc || j < 1 || j > nocc || k < 1 || k > nocc || klo < 1 || klo > k)
        return fail(1, "orbital index out of range");
    const char *wf = getenv("TRPDRV_WRITE_F");
    const int write_f = wf && strcmp(wf, "1") == 0;
    if (write_f && (!f1n || !f1t || !f2n || !f2t || !f3n || !f3t || !f4n || !f4t))
        return fail(1, "TRPDRV_WRITE_F=1 with a NULL f array");
    if (int rc = reserve(nvir, nbf)) return rc;
    if (int rc = layout(ncor, nocc, nvir)) return rc;
    const size_t V = (size_t)nvir, O = (size_t)nocc, vv = V * V, ov = O * V;
    const size_t kv = (size_t)(k - klo) * vv, ko = (size_t)(k - klo) * ov;
    // the reference's offsets of the k-chunk slices (gpu-omp/ccsd_trpdrv_omp_cbody.c:64-70)
    const float *in[DS_N] = {tij, jia, kia, tia, xia, jij, kij, tkj + kv, jka + kv, kka + kv, tka + ko, xka + ko,
                             jkj + ko, kkj + ko, dintc1, dintx1, t1v1, dintc2, dintx2, t1v2, eorb};
    const float *dev[DS_N];
    stage_piece pc[DS_N];
    for (int q = 0; q < DS_N; ++q) {
        const int b = q % 7, is_vec = q >= DS_VEC;
        const size_t width = is_vec ? (q < DS_N - 1 ? V : (size_t)nbf) : b < DS_JO ? V : O;
        const size_t rows = is_vec ? 1 : b < DS_TO || b >= DS_JO ? V : O;
        const size_t pitch = is_vec ? width : (size_t)pitch4((int)width);
        const bool flat = pitch == width;
        dev[q] = g.d_stage + g.off[q];
        pc[q].dst = (char *)(g.h_stage + g.off[q]);
        pc[q].src = (const char *)in[q];
        pc[q].rows = flat ? 1 : rows;
        pc[q].width = sizeof(float) * (flat ? rows * width : width);
        pc[q].pitch = sizeof(float) * (flat ? rows * width : pitch);
    }
    const int threads = stage_threads();
    int rc = stage_send(pc + DS_K, DS_N - DS_K, threads, SEGMENT, send, nullptr);
    if (!rc) rc = stage_send(pc, DS_K, threads, SEGMENT, send, nullptr);
    if (rc) {
        g.nvir = 0;  // mirror and device may differ now
        return rc;
    }

    // f1n f2n f3n f4n f1t f2t f3t f4t: gpu-omp/ccsd_trpdrv_omp_cbody.c:72-167
    GemmArgs G;
    G.nocc = nocc;
    G.nvir = nvir;
    G.ldv = pitch4(nvir);
    G.ldo = pitch4(nocc);
    G.f = g.f;
    G.counter = g.counter;
    for (int x = 0; x < 8; ++x) {
        const int A = x < 4 ? DS_I : DS_K, B = x < 4 ? DS_K : DS_I, two = (x >> 1) & 1;
        G.a1[x] = dev[A + (x & 1 ? DS_KV : DS_J)];
        G.b1[x] = dev[B + DS_T];
        G.b1_t[x] = !two;
        G.a2[x] = dev[A + (x & 1 ? DS_XO : DS_TO)];
        G.b2[x] = dev[B + (two ? DS_JO : DS_KO)];
    }
    // 64-wide tiles once they fill the chip's 148 SMs
    const unsigned n64 = (unsigned)(nvir + 63) / 64, n32 = (unsigned)(nvir + 31) / 32;
    if (n64 * n64 * 8 >= 148)
        sgemm_group_kernel<64><<<dim3(n64, n64, 8), Tile<64>::THREADS, 0, g.st>>>(G);
    else
        sgemm_group_kernel<32><<<dim3(n32, n32, 8), Tile<32>::THREADS, 0, g.st>>>(G);
    F32_TRY(cudaGetLastError());

    // gpu-omp/ccsd_trpdrv_omp_cbody.c:62
    const float eaijk = eorb[a - 1] - (eorb[ncor + i - 1] + eorb[ncor + j - 1] + eorb[ncor + k - 1]);
    float r[4];
    if (int rc2 = launch_tengy(ncor, nocc, nvir, eaijk, dev + DS_VEC, dev[DS_N - 1], r)) return rc2;
    if (write_f) {
        float *outs[8] = {f1n, f2n, f3n, f4n, f1t, f2t, f3t, f4t};
        for (int x = 0; x < 8; ++x)
            F32_TRY(cudaMemcpy(outs[x], g.f + (size_t)x * vv, sizeof(float) * vv, cudaMemcpyDeviceToHost));
    }
    // gpu-omp/ccsd_trpdrv_omp_cbody.c:220-228
    float emp4 = *emp4_, emp5 = *emp5_;
    emp4 += r[0];
    emp5 += r[1];
    if (*i_ != *k_) {
        emp4 += r[2];
        emp5 += r[3];
    }
    *emp4_ = emp4;
    *emp5_ = emp5;
    return 0;
}

int tengy(const float *const *f8, const float *const *vec, const float *eorb, float eaijk, float *out4, int ncor,
          int nocc, int nvir)
{
    for (int q = 0; q < 8; ++q)
        if (!f8[q]) return fail(1, "NULL f array");
    for (int q = 0; q < 6; ++q)
        if (!vec[q]) return fail(1, "NULL vector");
    if (!eorb || nocc < 1 || nvir < 1 || ncor < 0 || nvir > 16384) return fail(1, "bad tengy arguments");
    const int nbf = ncor + nocc + nvir;
    if (int rc = reserve(nvir, nbf)) return rc;
    const size_t vv = (size_t)nvir * nvir;
    // device order f1n f2n f3n f4n f1t f2t f3t f4t from the argument order f1n f1t f2n f2t ...
    for (int x = 0; x < 4; ++x) {
        if (int rc = h2d(g.f + (size_t)x * vv, f8[2 * x], vv)) return rc;
        if (int rc = h2d(g.f + (size_t)(4 + x) * vv, f8[2 * x + 1], vv)) return rc;
    }
    const float *dvec[6];
    for (int q = 0; q < 6; ++q) {
        dvec[q] = g.vec + (size_t)q * nvir;
        if (int rc = h2d(g.vec + (size_t)q * nvir, vec[q], (size_t)nvir)) return rc;
    }
    float *deorb = g.vec + 6 * (size_t)nvir;
    if (int rc = h2d(deorb, eorb, (size_t)nbf)) return rc;
    return launch_tengy(ncor, nocc, nvir, eaijk, dvec, deorb, out4);
}

void report(int rc, const char *who)
{
    if (!rc) return;
    const char *v = getenv("TRPDRV_ON_ERROR");
    if (v && strcmp(v, "return") == 0) return;
    fprintf(stderr, "%s: %s\n", who, t_msg);
    abort();
}

}  // namespace f32
}  // namespace trpdrv

using namespace trpdrv::f32;

#define F32_BODY_ARGS                                                                                       \
    float *f1n, float *f1t, float *f2n, float *f2t, float *f3n, float *f3t, float *f4n, float *f4t,        \
        float *eorb, int *ncor, int *nocc, int *nvir, float *emp4, float *emp5, int *a, int *i, int *j,    \
        int *k, int *klo, float *tij, float *tkj, float *tia, float *tka, float *xia, float *xka,           \
        float *jia, float *jka, float *kia, float *kka, float *jij, float *jkj, float *kij, float *kkj,     \
        float *dintc1, float *dintx1, float *t1v1, float *dintc2, float *dintx2, float *t1v2
#define F32_BODY_PASS                                                                                       \
    f1n, f1t, f2n, f2t, f3n, f3t, f4n, f4t, eorb, ncor, nocc, nvir, emp4, emp5, a, i, j, k, klo, tij, tkj,  \
        tia, tka, xia, xka, jia, jka, kia, kka, jij, jkj, kij, kkj, dintc1, dintx1, t1v1, dintc2, dintx2, t1v2

static void body_entry(const char *who, F32_BODY_ARGS)
{
    pthread_mutex_lock(&g_mu);
    t_status = 0;
    const int rc = body(F32_BODY_PASS);
    pthread_mutex_unlock(&g_mu);
    report(rc, who);
}

extern "C" void ccsd_trpdrv_omp_cbody_(F32_BODY_ARGS) { body_entry("ccsd_trpdrv_omp_cbody_", F32_BODY_PASS); }
extern "C" void ccsd_trpdrv_omp_fbody_(F32_BODY_ARGS) { body_entry("ccsd_trpdrv_omp_fbody_", F32_BODY_PASS); }

extern "C" void ccsd_tengy_omp(const float *f1n, const float *f1t, const float *f2n, const float *f2t,
                               const float *f3n, const float *f3t, const float *f4n, const float *f4t,
                               const float *dintc1, const float *dintx1, const float *t1v1, const float *dintc2,
                               const float *dintx2, const float *t1v2, const float *eorb, const float eaijk,
                               float *emp4i, float *emp5i, float *emp4k, float *emp5k, const int ncor,
                               const int nocc, const int nvir)
{
    pthread_mutex_lock(&g_mu);
    t_status = 0;
    int rc = (emp4i && emp5i && emp4k && emp5k) ? 0 : fail(1, "NULL output");
    const float *f8[8] = {f1n, f1t, f2n, f2t, f3n, f3t, f4n, f4t};
    const float *vec[6] = {dintc1, dintx1, t1v1, dintc2, dintx2, t1v2};
    float r[4];
    if (!rc) rc = tengy(f8, vec, eorb, eaijk, r, ncor, nocc, nvir);
    pthread_mutex_unlock(&g_mu);
    if (!rc) {  // outputs overwritten, gpu-omp/ccsd_tengy_c99.c:115-118
        *emp4i = r[0];
        *emp5i = r[1];
        *emp4k = r[2];
        *emp5k = r[3];
    }
    report(rc, "ccsd_tengy_omp");
}

extern "C" int trpdrv_fp32_last_error(void) { return t_status; }
extern "C" const char *trpdrv_fp32_last_error_message(void) { return t_msg; }
