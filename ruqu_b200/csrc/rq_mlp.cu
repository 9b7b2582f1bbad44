// rq_mlp.cu -- BF16 tensor-core (tcgen05) GEMMs and the warm-start MLP.
//
// The warm start for QAOA angles is a small MLP (325 -> 256 -> 256 -> 8, ReLU,
// BF16 weights and activations, FP32 accumulation).  It has no counterpart in
// the reference (whose run_qaoa always starts from gamma = beta = 0.5,
// qaoa.rs:221-222); it is trained on angles the batched simulator optimises.
//
// k_gemm_bf16 computes C[M x N] = A[M x K] * B[N x K]^T (+ epilogue) on the
// 5th-generation tensor cores: each CTA owns a tile of C of BM (128 or 64) rows
// and NT columns; K is consumed in chunks of KC through two shared-memory buffers, so
// a chunk loads while the previous one's MMAs run.  Operands sit in shared
// memory in the no-swizzle K-major "core matrix" layout (8 rows x 16 bytes per
// core matrix; element (r, k) of a tile at byte (r/8)*SBO + (k/8)*128 +
// (r%8)*16 + (k%8)*2, SBO = 16 KC); an operand stored the other way round
// (K rows of M or N values) is transposed in registers on the way in, one 8x8
// block per thread, so no transposed copies exist in memory.  One thread
// issues tcgen05.mma (kind::f16, BF16 inputs, FP32 accumulator in tensor
// memory), tcgen05.commit signals the buffer's mbarrier, and the epilogue reads
// the accumulator back with tcgen05.ld and applies the layer's elementwise work.
// Every wait on an mbarrier is bounded; on expiry the kernel records an error
// and returns after freeing its tensor memory.
#include "rq_internal.cuh"

#include <cuda_bf16.h>

#include <atomic>
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

namespace {

constexpr int GT = 256;      // threads per CTA
constexpr int LBO = 128;     // bytes between core matrices along K

__device__ int g_mma_timeout = 0;   // set when a bounded wait expires

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor, no swizzle, K-major (sm_100 version 1)
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)(LBO >> 4) << 16;
    d |= (uint64_t)(sbo >> 4) << 32;
    d |= (uint64_t)1 << 46;   // descriptor version for sm_100
    return d;                 // base offset 0, lbo mode 0, layout type 0 (no swizzle)
}

// instruction descriptor: BF16 x BF16 -> F32, A and B K-major, M = m (64 or 128), N = n
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
    return (1u << 4)               // D format F32
         | (1u << 7)               // A format BF16
         | (1u << 10)              // B format BF16
         | ((uint32_t)(n >> 3) << 17)
         | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// polls before a main-path wait counts as expired (rq_debug_set_wait_limit); the clean-up
// wait after an expiry always uses WAIT_POLLS
constexpr uint32_t WAIT_POLLS = 1u << 26;
__device__ uint32_t g_mma_wait_polls = WAIT_POLLS;

// bounded wait for the mbarrier phase `parity`; false on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t polls = WAIT_POLLS) {
    const uint32_t a = smem_u32(bar);
    for (uint32_t it = 0; it < polls; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

enum Epi : int {
    EPI_F32 = 0,         // C (f32) = acc
    EPI_BIAS_RELU = 1,   // H (bf16) = relu(acc + bias)
    EPI_BIAS = 2,        // C (f32) = acc + bias
    EPI_RELU_BACK = 3,   // F (f32) = acc where mask > 0 and row < valid, else 0; H (bf16) = F
    EPI_MSE = 4          // d = acc + bias - target: F (f32) = 2 d, H (bf16) = 2 d / (valid * out),
                         // losspart = sum of d^2
};

// Column sums of an f32 matrix, dst[c] = scale * sum over the rows, added in row order: the bias
// gradients, computed by extra CTAs (32 columns each) of a launch of products that is ready anyway.
struct ColSum {
    const float* src;
    int ld, cols, rows;
    float scale;
    float* dst;
};

struct GemmArgs {
    const __nv_bfloat16* A;   // [M x K] row-major, or [K x M] with at
    const __nv_bfloat16* B;   // [N x K] row-major, or [K x N] with bt
    int M, N, K;              // K % 16 == 0
    int lda, ldb;             // row strides (elements, multiples of 8)
    int at, bt;               // operand stored transposed (M / N then a multiple of 8)
    int arows;                // rows of A that exist (the rest of M reads as zeros); at: K rows of A and B
    float* C;                 // [M x N] f32 (row stride ldc)
    int ldc;
    const float* bias;        // [nbias]
    int nbias;
    __nv_bfloat16* H;         // [M x N] bf16 (row stride ldh)
    int ldh;
    int epi;
    const __nv_bfloat16* mask;   // EPI_RELU_BACK: [M x N] bf16 (row stride ldh)
    int valid;                   // EPI_RELU_BACK, EPI_MSE: rows that count
    const float* target;         // EPI_MSE: [valid x out] f32
    int out;                     // EPI_MSE: columns that count
    float* F;                    // EPI_RELU_BACK, EPI_MSE: [M x N] f32 (row stride ldh)
    float* losspart;             // EPI_MSE: [row tiles * column tiles]
    int early;                   // EARLY_A, EARLY_B: operands that the launch just before does not write
};
constexpr int EARLY_A = 1, EARLY_B = 2;

// Programmatic dependent launch: a kernel of the training chain starts while its predecessor
// drains, sets up its tensor memory and barriers, and waits here for the predecessor's results
// (griddepcontrol.wait returns once every earlier grid of the chain has finished and its writes are
// visible; it returns at once in a kernel launched without the attribute).  What a predecessor
// writes is read past the L1 cache (cp.async.cg, __ldcg): the reading kernel may have begun before
// the write, so the read-only path would be free to return or to fetch early a stale line.
// A kernel starts once every CTA of its predecessor is past its own wait, so what the launch before
// that one wrote, or an older one, is there already: such operands (GemmArgs::early) are read before
// the wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void gcp_async16(void* dst, const void* src, bool take) {
    const uint32_t n = take ? 16u : 0u;   // 0: the 16 bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n) : "memory");
}

// rows [row0, +R) x k [k0, +kw) of an operand stored [rows x K] into the core-matrix layout.
// Eight neighbouring threads fill one core matrix (128 contiguous bytes of shared memory, no
// bank conflicts); a warp reads 64 contiguous bytes of each of its eight rows.
template <int R, int KC>
__device__ __forceinline__ void load_k_major(unsigned char* dst, const __nv_bfloat16* src, int ld, int row0,
                                             int row_lim, int k0, int kw, int tid) {
    // core matrix (rg, kc) of this thread's eight, stepped by GT / 8 without further divisions
    const int kch = kw >> 3, sg = (GT / 8) / kch, sc = (GT / 8) - sg * kch;
    int rg = (tid >> 3) / kch, kc = (tid >> 3) - rg * kch;
#pragma unroll 4
    while (rg < R / 8) {
        const int r = row0 + rg * 8 + (tid & 7);
        const bool ok = r < row_lim;
        const __nv_bfloat16* g = src + (ok ? (size_t)r * ld + k0 + kc * 8 : 0);
        gcp_async16(dst + rg * (KC * 16) + kc * 128 + (tid & 7) * 16, g, ok);
        rg += sg;
        kc += sc;
        if (kc >= kch) {
            kc -= kch;
            ++rg;
        }
    }
}

// the same tile of an operand stored [K x rows]: 8x8 blocks transposed in registers, one core
// matrix per thread and step (eight 16-byte loads in flight, eight contiguous 16-byte stores)
template <int R, int KC>
__device__ __forceinline__ void load_mn_major(unsigned char* dst, const __nv_bfloat16* src, int ld, int row0,
                                              int row_lim, int k0, int kw, int k_lim, int tid) {
    const int kch = kw >> 3, total = (R / 8) * kch;
#pragma unroll 2
    for (int u = tid; u < total; u += GT) {
        const int kc = u / (R / 8), rg = u - kc * (R / 8);   // neighbouring threads: neighbouring 16 bytes of a row
        const bool ok = row0 + rg * 8 < row_lim;
        uint4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = k0 + kc * 8 + j;
            v[j] = ok && k < k_lim ? __ldcg(reinterpret_cast<const uint4*>(src + (size_t)k * ld + row0 + rg * 8))
                                   : make_uint4(0u, 0u, 0u, 0u);
        }
        unsigned char* d = dst + rg * (KC * 16) + kc * 128;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t* x = reinterpret_cast<const uint32_t*>(&v[2 * j]);
                const uint32_t* y = reinterpret_cast<const uint32_t*>(&v[2 * j + 1]);
                o[j] = __byte_perm(x[r >> 1], y[r >> 1], (r & 1) ? 0x7632 : 0x5410);
            }
            *reinterpret_cast<uint4*>(d + r * 16) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
}

// One thread's serial sum keeps the rounding of one long addition chain; the rows come in through
// shared memory, 256 at a time with every load of the block in flight (a chain of dependent
// global loads took 135 us for 256 rows).
__device__ void column_sums(const ColSum& s, int block, float* stage, int tid) {
    const int c0 = block * 32;
    float acc = 0.f;
    for (int r0 = 0; r0 < s.rows; r0 += 256) {
        const int nr = min(256, s.rows - r0);
#pragma unroll 8
        for (int k = tid; k < 256 * 8; k += GT) {   // 8 float4 per row (ld and c0 are multiples of 16)
            const int r = k >> 3, c = (k & 7) * 4;
            if (r < nr && c0 + c < s.ld)
                *reinterpret_cast<float4*>(stage + r * 32 + c) =
                    __ldcg(reinterpret_cast<const float4*>(s.src + (size_t)(r0 + r) * s.ld + c0 + c));
        }
        __syncthreads();
        if (tid < 32)
#pragma unroll 16
            for (int r = 0; r < nr; ++r) acc = fmaf(stage[r * 32 + tid], s.scale, acc);
        __syncthreads();
    }
    if (tid < 32 && c0 + tid < s.cols) s.dst[c0 + tid] = acc;
}

// One launch covers the tiles of g0 and, after them, those of g1 (independent products that
// become ready together; tiles0 and tiles1 = their tiles), then the column sums cs.  A tile is rows [BM i, +BM) x columns
// [NT j, +NT) of C (BM 128 or 64; the accumulator of 64 rows lies in the first 16 tensor-memory lanes of
// each warp).  The warm-start products are small (256 x 256 x 256-336): what bounds them is
// the latency of load -> MMA -> epilogue, so narrow tiles (more CTAs, each loading little) and the
// whole K in at most two chunks.  The operand that is older than the predecessor is read before the wait
// for it, both chunks are in flight at once, and the epilogue's operands come in beside them: a training
// step (batch 256, 336 -> 256 -> 256 -> 8, with Adam) takes 35 us.  Of a product's 4.5 us 1.3 are the
// hand-over between launches, 1.2 the late operand, 0.9 the MMAs, 0.6 the epilogue.
template <int BM, int NT, int KC>
__global__ void __launch_bounds__(GT, 1) k_gemm_bf16(const GemmArgs g0, const GemmArgs g1, const ColSum cs, int tiles0,
                                                     int tiles1) {
    static_assert(NT % 32 == 0 && NT >= 32 && NT <= 256, "tile N");
    constexpr int ABYTES = BM * KC * 2, BBYTES = NT * KC * 2;
    extern __shared__ __align__(1024) unsigned char smem[];   // two buffers of A | B
    __shared__ __align__(8) uint64_t mbar[2];
    __shared__ uint32_t tmem_base;
    __shared__ int timed_out;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int uwarp = __shfl_sync(0xffffffffu, warp, 0);
    const uint32_t leader = lane == 0 ? 1u : 0u;
    if ((int)blockIdx.x >= tiles0 + tiles1) {
        pdl_wait();
        pdl_go();
        column_sums(cs, blockIdx.x - tiles0 - tiles1, reinterpret_cast<float*>(smem), tid);
        return;
    }
    const GemmArgs g = (int)blockIdx.x < tiles0 ? g0 : g1;
    const int tile = (int)blockIdx.x < tiles0 ? blockIdx.x : blockIdx.x - tiles0;
    const int mt = (g.M + BM - 1) / BM;
    const int tm = tile % mt, tn = tile / mt;
    const int row0 = tm * BM, col0 = tn * NT;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(NT)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        mbar_init(&mbar[0], 1);
        mbar_init(&mbar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        timed_out = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    const int nk = (g.K + KC - 1) / KC;
    auto load_a = [&](int kc) {
        unsigned char* sA = smem + (kc & 1) * (ABYTES + BBYTES);
        const int k0 = kc * KC, kw = min(KC, g.K - k0);   // multiple of 16
        if (g.at) load_mn_major<BM, KC>(sA, g.A, g.lda, row0, g.M, k0, kw, g.arows, tid);
        else load_k_major<BM, KC>(sA, g.A, g.lda, row0, g.arows, k0, kw, tid);
    };
    auto load_b = [&](int kc) {
        unsigned char* sB = smem + (kc & 1) * (ABYTES + BBYTES) + ABYTES;
        const int k0 = kc * KC, kw = min(KC, g.K - k0);
        if (g.bt) load_mn_major<NT, KC>(sB, g.B, g.ldb, col0, g.N, k0, kw, g.at ? g.arows : g.K, tid);
        else load_k_major<NT, KC>(sB, g.B, g.ldb, col0, g.N, k0, kw, tid);
    };
    // what the epilogue adds, masks with or compares with, for 16 columns of this thread's row
    const int r = row0 + (warp & 3) * (BM / 4) + lane, half = warp >> 2;
    float eb = 0.f, et[16];   // eb: lanes 0-15 hold the columns' biases
    uint4 em[2];
    auto fetch = [&](int c) {
        if (g.epi == EPI_BIAS || g.epi == EPI_BIAS_RELU || g.epi == EPI_MSE) {
            const int b = c + (lane & 15);
            eb = b < g.nbias ? __ldcg(g.bias + b) : 0.f;
        }
        if (g.epi == EPI_MSE) {
#pragma unroll
            for (int j = 0; j < 16; ++j) et[j] = r < g.valid && c + j < g.out ? g.target[(size_t)r * g.out + c + j] : 0.f;
        }
        if (g.epi == EPI_RELU_BACK) {
            em[0] = em[1] = make_uint4(0u, 0u, 0u, 0u);
            if (r < g.M && c < g.N && r < g.valid) {   // N is a multiple of 16 here
                const uint4* mp = reinterpret_cast<const uint4*>(g.mask + (size_t)r * g.ldh + c);
                em[0] = __ldcg(mp);
                em[1] = __ldcg(mp + 1);
            }
        }
    };

    // the first two chunks into the two buffers: what the predecessor does not write, then the rest
    const int pre = min(nk, 2);
    for (int kc = 0; kc < pre; ++kc) {
        if (g.early & EARLY_A) load_a(kc);
        if (g.early & EARLY_B) load_b(kc);
    }
    pdl_wait();
    pdl_go();
    for (int kc = 0; kc < pre; ++kc) {
        if (!(g.early & EARLY_A)) load_a(kc);
        if (!(g.early & EARLY_B)) load_b(kc);
    }
    if (NT == 32) fetch(col0 + half * 16);   // lands while the operands do

    int issued = 0;                       // chunks whose MMAs have been issued
    for (int kc = 0; kc < nk; ++kc) {
        const int buf = kc & 1;
        if (kc >= 2) {                    // the MMAs of chunk kc - 2 read this buffer
            if (!mbar_wait(&mbar[buf], (uint32_t)((kc >> 1) - 1) & 1u, g_mma_wait_polls)) timed_out = 1;
            __syncthreads();
            if (timed_out) break;
            load_a(kc);
            load_b(kc);
        }
        if (kc != 1) {                    // chunk 1 landed with chunk 0
            asm volatile("cp.async.wait_all;" ::: "memory");
            // make the generic-proxy writes visible to the tensor core (async proxy)
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncthreads();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        // the whole of warp 0 steps the descriptors, so that they stay in uniform registers; one lane issues
        if (uwarp == 0) {
            const uint32_t a0 = smem_u32(smem + buf * (ABYTES + BBYTES));
            uint64_t ad = sdesc(a0, KC * 16), bd = sdesc(a0 + ABYTES, KC * 16);
            const int steps = min(KC, g.K - kc * KC) / 16;
            uint32_t acc = kc > 0 ? 1u : 0u;
#pragma unroll 4
            for (int ks = 0; ks < steps; ++ks) {
                asm volatile(
                    "{\n\t.reg .pred p, e;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "setp.ne.b32 e, %9, 0;\n\t"
                    "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                    ::"r"(tmem), "l"(ad), "l"(bd), "r"(idesc_bf16(BM, NT)), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u),
                    "r"(leader)
                    : "memory");
                ad += 2 * LBO >> 4;       // the address field: the next 16 of K
                bd += 2 * LBO >> 4;
                acc = 1u;
            }
            if (leader)
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&mbar[buf]))
                             : "memory");
        }
        issued = kc + 1;
    }
    // the last chunk's commit covers every earlier MMA of the issuing thread
    if (!timed_out) {
        if (!mbar_wait(&mbar[(nk - 1) & 1], (uint32_t)((nk - 1) >> 1) & 1u, g_mma_wait_polls)) timed_out = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    __syncthreads();
    if (timed_out) {
        // MMAs may still be in flight: let them land (bounded) before the shared and tensor memory
        // they use are released
        if (tid == 0) {
            mbar_wait(&mbar[(issued - 1) & 1], (uint32_t)((issued - 1) >> 1) & 1u);
            atomicExch(&g_mma_timeout, 1);
        }
    } else {
        // epilogue: warps w and w + 4 read the tensor-memory lanes 32 (w % 4).. (BM / 4 rows of the tile),
        // the lower four warps the first half of the columns, the upper four the second
        float loss = 0.f;
        const float inv = g.epi == EPI_MSE ? 1.f / (float)(g.valid * g.out) : 0.f;
        for (int c0 = half * (NT / 2); c0 < (half + 1) * (NT / 2); c0 += 16) {
            uint32_t v[16];
            const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            float x[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) x[j] = __uint_as_float(v[j]);
            const int c = col0 + c0;
            if (NT != 32) fetch(c);
            const bool row_ok = lane < BM / 4;
            const bool in = row_ok && r < g.M && c < g.N;
            const bool full = in && c + 16 <= g.N;
            if (g.epi == EPI_BIAS || g.epi == EPI_BIAS_RELU || g.epi == EPI_MSE) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float b = __shfl_sync(0xffffffffu, eb, j);
                    if (c + j < g.nbias) x[j] += b;
                }
            }
            if (g.epi == EPI_F32 || g.epi == EPI_BIAS) {
                float* o = g.C + (size_t)r * g.ldc + c;
                if (full && (g.ldc & 3) == 0) {
#pragma unroll
                    for (int j = 0; j < 16; j += 4)
                        *reinterpret_cast<float4*>(o + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
                } else if (in) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (c + j < g.N) o[j] = x[j];
                }
                continue;
            }
            if (g.epi == EPI_BIAS_RELU) {
#pragma unroll
                for (int j = 0; j < 16; ++j) x[j] = x[j] > 0.f ? x[j] : 0.f;
            } else if (g.epi == EPI_RELU_BACK) {
                const __nv_bfloat16* mb = reinterpret_cast<const __nv_bfloat16*>(em);
#pragma unroll
                for (int j = 0; j < 16; ++j) x[j] = __bfloat162float(mb[j]) > 0.f ? x[j] : 0.f;
            } else {   // EPI_MSE
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float gr = 0.f;
                    if (row_ok && r < g.valid && c + j < g.out) {
                        const float d = x[j] - et[j];
                        loss += d * d;
                        gr = 2.f * d;
                    }
                    x[j] = gr;
                }
            }
            if (row_ok && r < g.M && c + 16 <= g.ldh) {     // ldh is a multiple of 16: whole 16-column groups
                const size_t at = (size_t)r * g.ldh + c;
                if (g.epi != EPI_BIAS_RELU) {
#pragma unroll
                    for (int j = 0; j < 16; j += 4)
                        *reinterpret_cast<float4*>(g.F + at + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
                }
                const float f = g.epi == EPI_MSE ? inv : 1.f;
                __nv_bfloat16 h[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) h[j] = __float2bfloat16_rn(x[j] * f);
                reinterpret_cast<uint4*>(g.H + at)[0] = reinterpret_cast<const uint4*>(h)[0];
                reinterpret_cast<uint4*>(g.H + at)[1] = reinterpret_cast<const uint4*>(h)[1];
            }
        }
        if (g.epi == EPI_MSE) {
            __shared__ float lred[GT / 32];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
            if (lane == 0) lred[warp] = loss;
            __syncthreads();
            if (tid == 0) {
                float s = 0.f;
                for (int k = 0; k < GT / 32; ++k) s += lred[k];
                g.losspart[tile] = s;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NT) : "memory");
}

// launch with the programmatic-serialization attribute (see pdl_wait)
template <typename... KA, typename... A>
int launch_chained(cudaStream_t stream, void (*kern)(KA...), unsigned grid, unsigned threads, size_t smem, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    RQ_CUDA(cudaLaunchKernelEx(&cfg, kern, KA(args)...));
    return RQ_OK;
}

template <int BM, int NT, int KC>
int launch_gemm(cudaStream_t stream, const GemmArgs& g0, const GemmArgs* g1, const ColSum* cs) {
    auto tiles = [](const GemmArgs& g) { return ((g.M + BM - 1) / BM) * ((g.N + NT - 1) / NT); };
    constexpr int smem = 2 * (BM + NT) * KC * 2;
    const int t0 = tiles(g0), t1 = g1 ? tiles(*g1) : 0, tc = cs ? (cs->cols + 31) / 32 : 0;
    RQ_CUDA(cudaFuncSetAttribute(k_gemm_bf16<BM, NT, KC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return launch_chained(stream, k_gemm_bf16<BM, NT, KC>, t0 + t1 + tc, GT, smem, g0, g1 ? *g1 : g0,
                          cs ? *cs : ColSum{}, t0, t1);
}

// Tile of a single product by the number of CTAs it leaves: the widest whose grid still has a CTA for
// every SM (A is re-read once per column tile, so large products want wide tiles); where even 32 columns
// leave SMs idle, 64 rows by 32 columns, whose CTAs each load 48 KB instead of 80 (64 training steps of
// batch 256: 2.30 against 2.76 ms).  Two products in one launch, and the output layer, always take the
// small tile: they are made for the warm start's widths.  Wider networks re-read their operands by it (4096
// wide, batch 4096: 7.7 ms a step).
int gemm(cudaStream_t stream, const GemmArgs& g0, const GemmArgs* g1 = nullptr, const ColSum* cs = nullptr) {
    const long mt = (g0.M + 127) / 128;
    if (!g1 && mt * ((g0.N + 255) / 256) >= 148) return launch_gemm<128, 256, 128>(stream, g0, g1, cs);
    if (!g1 && mt * ((g0.N + 127) / 128) >= 148) return launch_gemm<128, 128, 192>(stream, g0, g1, cs);
    if (!g1 && mt * ((g0.N + 63) / 64) >= 148) return launch_gemm<128, 64, 192>(stream, g0, g1, cs);
    if (!g1 && mt * ((g0.N + 31) / 32) >= 148) return launch_gemm<128, 32, 256>(stream, g0, g1, cs);
    return launch_gemm<64, 32, 256>(stream, g0, g1, cs);
}

}  // namespace

namespace rq {

// C = A * B^T on `stream`.  Shapes are checked here.
int gemm_bf16(cudaStream_t stream, const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int M, int N,
              int K, float* C, int ldc) {
    if (M < 1 || N < 1 || K < 16 || K % 16)
        return fail(RQ_ERR_INVALID_ARGUMENT, "gemm_bf16: M, N >= 1 and K a positive multiple of 16");
    if (lda % 8 || ldb % 8) return fail(RQ_ERR_INVALID_ARGUMENT, "gemm_bf16: row strides must be multiples of 8");
    GemmArgs g{};
    g.A = A; g.lda = lda; g.B = B; g.ldb = ldb;
    g.M = M; g.N = N; g.K = K;
    g.arows = M;
    g.C = C; g.ldc = ldc;
    g.epi = EPI_F32;
    return gemm(stream, g);
}

int mma_timeout_flag(int* out) {
    int v = 0, zero = 0;
    RQ_CUDA(cudaMemcpyFromSymbol(&v, g_mma_timeout, sizeof(int)));
    if (v) {
        RQ_CUDA(cudaMemcpyToSymbol(g_mma_timeout, &zero, sizeof(int)));
        RQ_CUDA(cudaDeviceSynchronize());
    }
    *out = v;
    return RQ_OK;
}

int mma_set_wait_polls(uint32_t polls) {
    const uint32_t v = polls == RQ_WAIT_LIMIT_DEFAULT ? WAIT_POLLS : polls;
    RQ_CUDA(cudaMemcpyToSymbol(g_mma_wait_polls, &v, sizeof(v)));
    RQ_CUDA(cudaDeviceSynchronize());   // landed before any later launch, on any stream
    return RQ_OK;
}

}  // namespace rq

extern "C" {

// C (f32, M x N) = A (bf16, M x K) * B (bf16, N x K)^T on the tensor cores;
// host buffers in and out (test and benchmark entry point of the GEMM).
int rq_gemm_bf16(const uint16_t* A, const uint16_t* B, int32_t M, int32_t N, int32_t K, float* C) {
    if (!A || !B || !C) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "null pointer");
    __nv_bfloat16 *dA = nullptr, *dB = nullptr;
    float* dC = nullptr;
    RQ_CUDA(rq::device_malloc((void**)&dA, (size_t)M * K * 2));
    RQ_CUDA(rq::device_malloc((void**)&dB, (size_t)N * K * 2));
    RQ_CUDA(rq::device_malloc((void**)&dC, (size_t)M * N * 4));
    int rc = RQ_OK;
    cudaError_t e = cudaMemcpy(dA, A, (size_t)M * K * 2, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dB, B, (size_t)N * K * 2, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) rc = rq::cuda_fail(e, "cudaMemcpy");
    if (rc == RQ_OK) rc = rq::gemm_bf16(0, dA, K, dB, K, M, N, K, dC, N);
    if (rc == RQ_OK) {
        e = cudaMemcpy(C, dC, (size_t)M * N * 4, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) rc = rq::cuda_fail(e, "cudaMemcpy");
    }
    int to = 0;
    if (rc == RQ_OK && rq::mma_timeout_flag(&to) == RQ_OK && to)
        rc = rq::fail(RQ_ERR_TIMEOUT, "tensor-core wait expired");
    cudaFree(dA);
    cudaFree(dB);
    cudaFree(dC);
    return rc;
}

}  // extern "C"

// ===========================================================================
// The warm-start MLP: in -> h1 -> h2 -> out, ReLU after the two hidden layers,
// FP32 master parameters (row-major [out_features x in_features] weights and
// biases), BF16 copies for the tensor-core GEMMs, FP32 accumulation, mean
// squared error loss, Adam updates in FP32 on the device.
// ===========================================================================
namespace {

__global__ void k_pad_bf16(const float* __restrict__ src, int rows, int cols, int lds, __nv_bfloat16* __restrict__ dst,
                           int prow, int pcol, int ldd) {
    const long total = (long)prow * pcol;
    for (long w = (long)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (long)gridDim.x * blockDim.x) {
        const int r = (int)(w / pcol), c = (int)(w - (long)r * pcol);
        const float v = (r < rows && c < cols) ? src[(long)r * lds + c] : 0.f;
        dst[(long)r * ldd + c] = __float2bfloat16_rn(v);
    }
}

// Where the parameters, their gradients and their BF16 copies lie (flat parameter index order:
// W1, b1, W2, b2, W3, b3).
struct ParamMap {
    int in, h1, h2, out, inp, outp;
    long b1, w2, b2, w3, b3, total;       // first parameter of each later block
    const float *g1, *g2, *g3t;           // dW1 [h1 x inp], dW2 [h2 x h1], dW3^T [h2 x outp]
    const float *db1, *db2, *db3;         // [h1], [h2], [out]
    __nv_bfloat16 *W1b, *W2b, *W3b;
};

// where the gradient of parameter w lies; *copy = where its BF16 copy lives (null for a bias)
__device__ __forceinline__ const float* grad_of(const ParamMap& m, long w, __nv_bfloat16** copy) {
    *copy = nullptr;
    if (w < m.b1) {
        const int r = (int)(w / m.in), k = (int)(w - (long)r * m.in);
        *copy = m.W1b + (long)r * m.inp + k;
        return m.g1 + (long)r * m.inp + k;
    } else if (w < m.w2) {
        return m.db1 + (w - m.b1);
    } else if (w < m.b2) {
        *copy = m.W2b + (w - m.w2);
        return m.g2 + (w - m.w2);
    } else if (w < m.w3) {
        return m.db2 + (w - m.b2);
    } else if (w < m.b3) {
        const int r = (int)((w - m.w3) / m.h2), k = (int)((w - m.w3) - (long)r * m.h2);
        *copy = m.W3b + (long)r * m.h2 + k;
        return m.g3t + (long)k * m.outp + r;
    }
    return m.db3 + (w - m.b3);
}

// a warp's sum of the tiles' losses, added in tile order
__device__ __forceinline__ float loss_sum(const float* losspart, int nloss) {
    const int lane = threadIdx.x & 31;
    float s = 0.f;
    for (int k0 = 0; k0 < nloss; k0 += 32) {
        const float v = k0 + lane < nloss ? __ldcg(losspart + k0 + lane) : 0.f;
        for (int k = 0; k < min(32, nloss - k0); ++k) s += __shfl_sync(0xffffffffu, v, k);
    }
    return s;
}

// One Adam step over every parameter, and the BF16 copies the next step's products read, in one
// launch; the loss of the step from its per-tile sums by the last CTA.  Parameters, moments and the places
// of the gradients are older than the predecessor and come before the wait.
__global__ void k_adam(ParamMap map, float* p, float* m, float* v, float lr,
                       float b1, float b2, float eps, float c1, float c2, const float* losspart, int nloss,
                       float inv, float* loss) {
    const long w0 = (long)blockIdx.x * blockDim.x + threadIdx.x, step = (long)(gridDim.x - 1) * blockDim.x;
    if (blockIdx.x == gridDim.x - 1) {
        pdl_wait();
        pdl_go();
        if (threadIdx.x < 32) {
            const float s = loss_sum(losspart, nloss);
            if (threadIdx.x == 0) *loss = s * inv;
        }
        return;
    }
    bool waited = false;
    for (long w = w0; w < map.total; w += step) {
        __nv_bfloat16* copy;
        const float* grad = grad_of(map, w, &copy);
        const float mo = __ldcg(m + w), vo = __ldcg(v + w), po = __ldcg(p + w);
        if (!waited) {
            pdl_wait();
            pdl_go();
            waited = true;
        }
        const float gr = __ldcg(grad);
        // roundings spelled out: training amplifies a last-bit difference, so they must not move with the code
        const float mm = __fmaf_rn(1.f - b1, gr, __fmul_rn(b1, mo));
        const float vv = __fmaf_rn(__fmul_rn(1.f - b2, gr), gr, __fmul_rn(b2, vo));
        m[w] = mm;
        v[w] = vv;
        const float np = po - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
        p[w] = np;
        if (copy) *copy = __float2bfloat16_rn(np);
    }
    if (!waited) {
        pdl_wait();
        pdl_go();
    }
}

// gradients in the caller's flat layout, and the loss
__global__ void k_gather(ParamMap map, const float* __restrict__ losspart, int nloss, float inv, float* __restrict__ out,
                         float* __restrict__ loss) {
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        const float s = loss_sum(losspart, nloss);
        if (threadIdx.x == 0) *loss = s * inv;
    }
    for (long w = (long)blockIdx.x * blockDim.x + threadIdx.x; w < map.total; w += (long)gridDim.x * blockDim.x) {
        __nv_bfloat16* copy;
        out[w] = __ldcg(grad_of(map, w, &copy));
    }
}

inline int pad16(int x) { return (x + 15) & ~15; }

}  // namespace

struct rq_mlp {
    int device = 0;
    int in = 0, h1 = 0, h2 = 0, out = 0;
    int inp = 0, outp = 0;        // padded widths (K multiple of 16, N padded to 32)
    cudaStream_t stream = nullptr;
    // FP32 master parameters and Adam moments, one flat buffer each
    float *P = nullptr, *Mo = nullptr, *Vo = nullptr;
    long off_w1 = 0, off_b1 = 0, off_w2 = 0, off_b2 = 0, off_w3 = 0, off_b3 = 0, nparam = 0;
    long step = 0;
    // BF16 copies: W1b [h1 x inp], W2b [h2 x h1], W3b [outp x h2]
    __nv_bfloat16 *W1b = nullptr, *W2b = nullptr, *W3b = nullptr;
    // batch workspace
    int cap = 0;
    __nv_bfloat16 *X = nullptr, *H1 = nullptr, *H2 = nullptr, *dY = nullptr, *dZ2 = nullptr, *dZ1 = nullptr;
    float *Xf = nullptr, *Tf = nullptr, *Y = nullptr;
    float *F1 = nullptr, *F2 = nullptr, *F3 = nullptr;     // f32 dZ1, dZ2 and 2 (Y - T): summed over rows into
    float *db1 = nullptr, *db2 = nullptr, *db3 = nullptr;  // the bias gradients
    float* losspart = nullptr;                             // per-tile sums of squares
    // a training set on the device (kept between calls: keep_training_rows)
    float *tx = nullptr, *tt = nullptr;
    __nv_bfloat16* txb = nullptr;
    size_t train_rows = 0;
    size_t train_kept = 0;        // bytes of it counted in g_train_kept
    float* G = nullptr;           // gradients: dW1 [h1 x inp], dW2 [h2 x h1], dW3t [h2 x outp]
    long g_w1 = 0, g_w2 = 0, g_w3t = 0, g_total = 0;
    float* loss = nullptr;
};

namespace {

template <typename P>
int dalloc(P** p, size_t n) {
    cudaError_t e = rq::device_malloc((void**)p, std::max<size_t>(1, n) * sizeof(P));
    if (e != cudaSuccess) {
        cudaGetLastError();
        return rq::fail(RQ_ERR_MEMORY_ALLOCATION, "memory allocation failed: need " + std::to_string(n * sizeof(P)) + " bytes");
    }
    return RQ_OK;
}

constexpr size_t TRAIN_KEEP_BYTES = (size_t)256 << 20;   // training sets kept on the device, all networks together
std::atomic<size_t> g_train_kept{0};

int mlp_refresh_bf16(rq_mlp* m) {
    const int sms = rq::num_sms(m->device);
    const float* P = m->P;
    k_pad_bf16<<<rq::grid_for((uint64_t)m->h1 * m->inp, 256, sms), 256, 0, m->stream>>>(P + m->off_w1, m->h1, m->in, m->in,
                                                                                     m->W1b, m->h1, m->inp, m->inp);
    k_pad_bf16<<<rq::grid_for((uint64_t)m->h2 * m->h1, 256, sms), 256, 0, m->stream>>>(P + m->off_w2, m->h2, m->h1, m->h1,
                                                                                    m->W2b, m->h2, m->h1, m->h1);
    k_pad_bf16<<<rq::grid_for((uint64_t)m->outp * m->h2, 256, sms), 256, 0, m->stream>>>(P + m->off_w3, m->out, m->h2,
                                                                                      m->h2, m->W3b, m->outp, m->h2, m->h2);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

int mlp_reserve(rq_mlp* m, int B) {
    const int Bp = (B + 127) & ~127;
    if (Bp <= m->cap) return RQ_OK;
    m->cap = 0;
    auto regrow = [](auto** p, size_t n) {
        if (*p) cudaFree(*p);
        *p = nullptr;
        return dalloc(p, n);
    };
    const size_t b = (size_t)Bp, nt = b / 64;
    RQ_TRY(regrow(&m->X, b * m->inp));
    RQ_TRY(regrow(&m->H1, b * m->h1));
    RQ_TRY(regrow(&m->H2, b * m->h2));
    RQ_TRY(regrow(&m->dY, b * m->outp));
    RQ_TRY(regrow(&m->dZ2, b * m->h2));
    RQ_TRY(regrow(&m->dZ1, b * m->h1));
    RQ_TRY(regrow(&m->Xf, b * m->in));
    RQ_TRY(regrow(&m->Tf, b * m->out));
    RQ_TRY(regrow(&m->Y, b * m->outp));
    RQ_TRY(regrow(&m->F1, b * m->h1));
    RQ_TRY(regrow(&m->F2, b * m->h2));
    RQ_TRY(regrow(&m->F3, b * m->outp));
    RQ_TRY(regrow(&m->losspart, nt * (size_t)((m->outp + 31) / 32)));
    m->cap = Bp;
    return RQ_OK;
}

void train_release(rq_mlp* m) {
    void* bufs[] = {m->tx, m->tt, m->txb};
    for (void* b : bufs) if (b) cudaFree(b);
    m->tx = m->tt = nullptr;
    m->txb = nullptr;
    m->train_rows = 0;
    g_train_kept -= m->train_kept;
    m->train_kept = 0;
}

// after a call: the training set stays for the next one if there is room for it, else it is freed
void keep_training_rows(rq_mlp* m) {
    if (m->train_kept) return;
    const size_t bytes = m->train_rows * (m->in * sizeof(float) + m->out * sizeof(float) + m->inp * sizeof(__nv_bfloat16));
    size_t kept = g_train_kept.load();
    while (kept + bytes <= TRAIN_KEEP_BYTES)
        if (g_train_kept.compare_exchange_weak(kept, kept + bytes)) {
            m->train_kept = bytes;
            return;
        }
    train_release(m);
}

int train_reserve(rq_mlp* m, size_t n) {
    if (n <= m->train_rows) return RQ_OK;
    train_release(m);
    RQ_TRY(dalloc(&m->tx, n * m->in));
    RQ_TRY(dalloc(&m->tt, n * m->out));
    RQ_TRY(dalloc(&m->txb, n * m->inp));
    m->train_rows = n;
    return RQ_OK;
}

// rows of f32 inputs as padded BF16 rows
int mlp_pack_rows(rq_mlp* m, const float* src, size_t rows, __nv_bfloat16* dst) {
    k_pad_bf16<<<rq::grid_for((uint64_t)rows * m->inp, 256, rq::num_sms(m->device)), 256, 0, m->stream>>>(
        src, (int)rows, m->in, m->in, dst, (int)rows, m->inp, m->inp);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

// hidden layers on B packed rows X: H1, H2 (settled: X is older than the launch before)
int mlp_hidden(rq_mlp* m, const __nv_bfloat16* X, int B, bool settled) {
    const int Bp = (B + 127) & ~127;
    GemmArgs g{};
    g.A = X; g.lda = m->inp; g.arows = B;
    g.B = m->W1b; g.ldb = m->inp;
    g.M = Bp; g.N = m->h1; g.K = m->inp;
    g.bias = m->P + m->off_b1; g.nbias = m->h1;
    g.H = m->H1; g.ldh = m->h1;
    g.epi = EPI_BIAS_RELU;
    g.early = settled ? EARLY_A : 0;
    RQ_TRY(gemm(m->stream, g));
    g.early = EARLY_B;
    g.A = m->H1; g.lda = m->h1; g.arows = Bp;
    g.B = m->W2b; g.ldb = m->h1;
    g.N = m->h2; g.K = m->h1;
    g.bias = m->P + m->off_b2; g.nbias = m->h2;
    g.H = m->H2; g.ldh = m->h2;
    return gemm(m->stream, g);
}

GemmArgs output_layer(rq_mlp* m, int B) {
    GemmArgs g{};
    g.M = (B + 127) & ~127;
    g.A = m->H2; g.lda = m->h2; g.arows = g.M;
    g.B = m->W3b; g.ldb = m->h2;
    g.N = m->out; g.K = m->h2;
    g.bias = m->P + m->off_b3; g.nbias = m->out;
    g.C = m->Y; g.ldc = m->outp;
    g.epi = EPI_BIAS;
    g.early = EARLY_B;
    return g;
}

// forward and backward pass on B packed rows X with targets T (device): weight gradients into m->G,
// bias gradients into m->db1..3, the loss as per-tile sums
int mlp_gradients_dev(rq_mlp* m, const __nv_bfloat16* X, const float* T, int B, bool settled) {
    const int Bp = (B + 127) & ~127;
    RQ_TRY(mlp_hidden(m, X, B, settled));
    // output layer with the loss: dY = 2 (Y - T) / (B out)
    GemmArgs y = output_layer(m, B);
    y.N = m->outp;                     // W3b's padding rows are zero; columns past out become zero in dY
    y.H = m->dY; y.ldh = m->outp;
    y.epi = EPI_MSE;
    y.nbias = m->out;
    y.valid = B; y.out = m->out; y.target = T;
    y.F = m->F3; y.losspart = m->losspart;
    RQ_TRY((launch_gemm<64, 32, 256>(m->stream, y, nullptr, nullptr)));
    // dW3^T [h2 x outp] = H2^T dY, and dZ2 [Bp x h2] = (dY W3) where H2 > 0
    GemmArgs w{};
    w.A = m->H2; w.lda = m->h2; w.at = 1;
    w.B = m->dY; w.ldb = m->outp; w.bt = 1;
    w.M = m->h2; w.N = m->outp; w.K = Bp; w.arows = B;
    w.C = m->G + m->g_w3t; w.ldc = m->outp;
    w.epi = EPI_F32;
    w.early = EARLY_A;
    GemmArgs d{};
    d.A = m->dY; d.lda = m->outp; d.arows = Bp;
    d.B = m->W3b; d.ldb = m->h2; d.bt = 1;
    d.M = Bp; d.N = m->h2; d.K = m->outp;
    d.H = m->dZ2; d.ldh = m->h2; d.mask = m->H2;
    d.valid = B; d.F = m->F2;
    d.epi = EPI_RELU_BACK;
    d.early = EARLY_B;
    const ColSum b3{m->F3, m->outp, m->out, B, 1.f / (float)(B * m->out), m->db3};
    RQ_TRY(gemm(m->stream, w, &d, &b3));
    // dW2 [h2 x h1] = dZ2^T H1, and dZ1 [Bp x h1] = (dZ2 W2) where H1 > 0
    w.A = m->dZ2; w.lda = m->h2;
    w.B = m->H1; w.ldb = m->h1;
    w.M = m->h2; w.N = m->h1;
    w.early = EARLY_B;
    w.C = m->G + m->g_w2; w.ldc = m->h1;
    d.A = m->dZ2; d.lda = m->h2;
    d.B = m->W2b; d.ldb = m->h1;
    d.N = m->h1; d.K = m->h2;
    d.H = m->dZ1; d.ldh = m->h1; d.mask = m->H1;
    d.F = m->F1;
    const ColSum b2{m->F2, m->h2, m->h2, B, 1.f, m->db2};
    RQ_TRY(gemm(m->stream, w, &d, &b2));
    // dW1 [h1 x inp] = dZ1^T X
    w.A = m->dZ1; w.lda = m->h1;
    w.B = X; w.ldb = m->inp;
    w.M = m->h1; w.N = m->inp;
    w.C = m->G + m->g_w1; w.ldc = m->inp;
    const ColSum b1{m->F1, m->h1, m->h1, B, 1.f, m->db1};
    return gemm(m->stream, w, nullptr, &b1);
}

ParamMap param_map(const rq_mlp* m) {
    ParamMap k{};
    k.in = m->in; k.h1 = m->h1; k.h2 = m->h2; k.out = m->out; k.inp = m->inp; k.outp = m->outp;
    k.b1 = m->off_b1; k.w2 = m->off_w2; k.b2 = m->off_b2; k.w3 = m->off_w3; k.b3 = m->off_b3; k.total = m->nparam;
    k.g1 = m->G + m->g_w1; k.g2 = m->G + m->g_w2; k.g3t = m->G + m->g_w3t;
    k.db1 = m->db1; k.db2 = m->db2; k.db3 = m->db3;
    k.W1b = m->W1b; k.W2b = m->W2b; k.W3b = m->W3b;
    return k;
}

// tiles of the output layer (64 rows of the padded batch, 32 columns)
int loss_tiles(const rq_mlp* m, int B) { return ((B + 127) / 128 * 2) * ((m->outp + 31) / 32); }

// one Adam step over every parameter from the gradients of the last mlp_gradients_dev (B rows)
int mlp_adam(rq_mlp* m, int B, float lr, float b1, float b2, float eps) {
    m->step += 1;
    const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
    return launch_chained(m->stream, k_adam, rq::grid_for((uint64_t)m->nparam, 256, rq::num_sms(m->device)) + 1, 256, 0,
                          param_map(m), m->P, m->Mo, m->Vo, lr, b1, b2, eps, c1, c2, m->losspart, loss_tiles(m, B),
                          1.f / (float)(B * m->out), m->loss);
}

}  // namespace

extern "C" {

int rq_mlp_create(int32_t in, int32_t h1, int32_t h2, int32_t out, uint64_t seed, rq_mlp** res) {
    if (!res) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "null pointer");
    if (in < 1 || h1 < 16 || h2 < 16 || out < 1 || h1 % 16 || h2 % 16)
        return rq::fail(RQ_ERR_INVALID_ARGUMENT, "mlp: hidden widths must be positive multiples of 16");
    std::unique_ptr<rq_mlp> m(new rq_mlp());
    cudaGetDevice(&m->device);
    m->in = in; m->h1 = h1; m->h2 = h2; m->out = out;
    m->inp = pad16(in);
    m->outp = (out + 31) & ~31;
    m->off_w1 = 0;
    m->off_b1 = m->off_w1 + (long)h1 * in;
    m->off_w2 = m->off_b1 + h1;
    m->off_b2 = m->off_w2 + (long)h2 * h1;
    m->off_w3 = m->off_b2 + h2;
    m->off_b3 = m->off_w3 + (long)out * h2;
    m->nparam = m->off_b3 + out;
    m->g_w1 = 0;
    m->g_w2 = m->g_w1 + (long)h1 * m->inp;
    m->g_w3t = m->g_w2 + (long)h2 * h1;
    m->g_total = m->g_w3t + (long)h2 * m->outp;
    RQ_CUDA(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
    RQ_TRY(dalloc(&m->P, m->nparam));
    RQ_TRY(dalloc(&m->Mo, m->nparam));
    RQ_TRY(dalloc(&m->Vo, m->nparam));
    RQ_TRY(dalloc(&m->G, m->g_total));
    RQ_TRY(dalloc(&m->loss, 1));
    RQ_TRY(dalloc(&m->db1, h1));
    RQ_TRY(dalloc(&m->db2, h2));
    RQ_TRY(dalloc(&m->db3, out));
    RQ_TRY(dalloc(&m->W1b, (size_t)h1 * m->inp));
    RQ_TRY(dalloc(&m->W2b, (size_t)h2 * h1));
    RQ_TRY(dalloc(&m->W3b, (size_t)m->outp * h2));
    RQ_CUDA(cudaMemset(m->G, 0, m->g_total * sizeof(float)));
    RQ_CUDA(cudaMemset(m->Mo, 0, m->nparam * sizeof(float)));
    RQ_CUDA(cudaMemset(m->Vo, 0, m->nparam * sizeof(float)));
    // He-uniform weights from the documented Philox stream (stream 6), zero biases
    std::vector<float> P(m->nparam, 0.f);
    uint64_t draw = 0;
    auto fill = [&](long off, int rows, int cols) {
        const double lim = std::sqrt(6.0 / cols);
        for (long k = 0; k < (long)rows * cols; ++k) P[off + k] = (float)((2.0 * rqd::uniform(seed, 6, draw++) - 1.0) * lim);
    };
    fill(m->off_w1, h1, in);
    fill(m->off_w2, h2, h1);
    fill(m->off_w3, out, h2);
    // stream-ordered: the refresh below runs on the network's (non-blocking) stream
    RQ_CUDA(cudaMemcpyAsync(m->P, P.data(), m->nparam * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    RQ_TRY(mlp_refresh_bf16(m.get()));
    RQ_CUDA(cudaStreamSynchronize(m->stream));
    *res = m.release();
    return RQ_OK;
}

int rq_mlp_destroy(rq_mlp* m) {
    if (!m) return RQ_OK;
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    void* bufs[] = {m->P, m->Mo, m->Vo, m->G, m->loss, m->W1b, m->W2b, m->W3b, m->X, m->H1, m->H2, m->dY, m->dZ2,
                    m->dZ1, m->Xf, m->Tf, m->Y, m->F1, m->F2, m->F3, m->db1, m->db2, m->db3, m->losspart};
    for (void* b : bufs) if (b) cudaFree(b);
    train_release(m);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return RQ_OK;
}

int rq_mlp_num_params(const rq_mlp* m, int64_t* n) {
    if (!m || !n) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "null pointer");
    *n = m->nparam;
    return RQ_OK;
}

int rq_mlp_get_params(rq_mlp* m, float* params) {
    if (!m || !params) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "null pointer");
    RQ_CUDA(cudaSetDevice(m->device));
    RQ_CUDA(cudaMemcpyAsync(params, m->P, m->nparam * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    RQ_CUDA(cudaStreamSynchronize(m->stream));
    return RQ_OK;
}

int rq_mlp_set_params(rq_mlp* m, const float* params) {
    if (!m || !params) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "null pointer");
    RQ_CUDA(cudaSetDevice(m->device));
    RQ_CUDA(cudaMemcpyAsync(m->P, params, m->nparam * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    RQ_CUDA(cudaMemsetAsync(m->Mo, 0, m->nparam * sizeof(float), m->stream));
    RQ_CUDA(cudaMemsetAsync(m->Vo, 0, m->nparam * sizeof(float), m->stream));
    m->step = 0;
    RQ_TRY(mlp_refresh_bf16(m));
    RQ_CUDA(cudaStreamSynchronize(m->stream));
    return RQ_OK;
}

int rq_mlp_forward(rq_mlp* m, const float* x, int32_t B, float* y) {
    if (!m || !x || !y || B < 1) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "bad argument");
    RQ_CUDA(cudaSetDevice(m->device));
    RQ_TRY(mlp_reserve(m, B));
    RQ_CUDA(cudaMemcpyAsync(m->Xf, x, (size_t)B * m->in * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    RQ_TRY(mlp_pack_rows(m, m->Xf, B, m->X));
    RQ_TRY(mlp_hidden(m, m->X, B, false));
    RQ_TRY(gemm(m->stream, output_layer(m, B)));
    RQ_CUDA(cudaMemcpy2DAsync(y, m->out * sizeof(float), m->Y, m->outp * sizeof(float), m->out * sizeof(float), B,
                              cudaMemcpyDeviceToHost, m->stream));
    RQ_CUDA(cudaStreamSynchronize(m->stream));
    int to = 0;
    RQ_TRY(rq::mma_timeout_flag(&to));
    if (to) return rq::fail(RQ_ERR_TIMEOUT, "tensor-core wait expired");
    return RQ_OK;
}

// loss and flat gradients (same layout as the parameters) for x (B x in), targets (B x out)
int rq_mlp_gradients(rq_mlp* m, const float* x, const float* t, int32_t B, float* loss, float* grads) {
    if (!m || !x || !t || !loss || !grads || B < 1) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "bad argument");
    RQ_CUDA(cudaSetDevice(m->device));
    RQ_TRY(mlp_reserve(m, B));
    RQ_CUDA(cudaMemcpyAsync(m->Xf, x, (size_t)B * m->in * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    RQ_CUDA(cudaMemcpyAsync(m->Tf, t, (size_t)B * m->out * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    RQ_TRY(mlp_pack_rows(m, m->Xf, B, m->X));
    RQ_TRY(mlp_gradients_dev(m, m->X, m->Tf, B, false));
    float* dflat = nullptr;
    RQ_TRY(dalloc(&dflat, m->nparam));
    k_gather<<<rq::grid_for((uint64_t)m->nparam, 256, rq::num_sms(m->device)), 256, 0, m->stream>>>(
        param_map(m), m->losspart, loss_tiles(m, B), 1.f / (float)(B * m->out), dflat, m->loss);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(grads, dflat, m->nparam * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    cudaFree(dflat);
    RQ_CUDA(e);
    int to = 0;
    RQ_TRY(rq::mma_timeout_flag(&to));
    if (to) return rq::fail(RQ_ERR_TIMEOUT, "tensor-core wait expired");
    return RQ_OK;
}

// `steps` Adam steps over minibatches x (n x in), t (n x out): minibatch k uses rows
// [k*B mod n ...) wrapping; returns the mean loss of the last step
int rq_mlp_train(rq_mlp* m, const float* x, const float* t, int32_t n, int32_t B, int32_t steps, float lr,
                 float* last_loss) {
    if (!m || !x || !t || n < 1 || B < 1 || steps < 0) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "bad argument");
    RQ_CUDA(cudaSetDevice(m->device));
    RQ_TRY(mlp_reserve(m, B));
    RQ_TRY(train_reserve(m, n));
    int rc = RQ_OK;
    cudaError_t e = cudaMemcpyAsync(m->tx, x, (size_t)n * m->in * sizeof(float), cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(m->tt, t, (size_t)n * m->out * sizeof(float), cudaMemcpyHostToDevice, m->stream);
    if (e != cudaSuccess) rc = rq::cuda_fail(e, "cudaMemcpyAsync");
    // every row in BF16 once; a minibatch is a range of those rows
    if (rc == RQ_OK) rc = mlp_pack_rows(m, m->tx, n, m->txb);
    for (int s = 0; s < steps && rc == RQ_OK; ++s) {
        const long r0 = ((long)s * B) % n;
        const int take = (int)std::min<long>(B, n - r0);
        rc = mlp_gradients_dev(m, m->txb + r0 * m->inp, m->tt + r0 * m->out, take, s > 0);
        if (rc == RQ_OK) rc = mlp_adam(m, take, lr, 0.9f, 0.999f, 1e-8f);
    }
    if (rc == RQ_OK && last_loss) {
        e = cudaMemcpyAsync(last_loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream);
        if (e != cudaSuccess) rc = rq::cuda_fail(e, "cudaMemcpyAsync");
    }
    e = cudaStreamSynchronize(m->stream);
    keep_training_rows(m);
    RQ_TRY(rc);
    RQ_CUDA(e);
    int to = 0;
    RQ_TRY(rq::mma_timeout_flag(&to));
    if (to) return rq::fail(RQ_ERR_TIMEOUT, "tensor-core wait expired");
    return RQ_OK;
}

}  // extern "C"
