// rq_reduce.cu -- FP64-accumulated reductions over the state.
//
// Counterparts of probabilities / probability_of_qubit (state.rs:123-137),
// expectation_value / expectation_hamiltonian (state.rs:362-408), normalize
// and fidelity (state.rs:415-435).  Every reduction accumulates in FP64 (also
// for f32 states) and is deterministic: a fixed grid writes one partial per
// block and term, and a second kernel sums the partials in a fixed order.
#include "rq_internal.cuh"
#include "rq_pauli_plan.cuh"

#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

namespace {

using rqd::C2;
using rqd::insert0;
using namespace rqs;

constexpr int TPB = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// sum `v` over the block; result valid in thread 0
__device__ __forceinline__ double block_sum(double v, double* sh) {
    v = warp_sum(v);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
        r = warp_sum(r);
    }
    return r;
}

template <typename V>
__device__ __forceinline__ double norm2(V x) {
    double re = (double)x.x, im = (double)x.y;
    return re * re + im * im;
}

// sum of |a_i|^2 over i with bit q == want (q = 64: all i)
template <typename T>
__global__ void k_prob(const typename C2<T>::t* __restrict__ a, uint64_t count, uint32_t q, int want,
                       double* __restrict__ partials) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < count;
         p += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t i = q < 64 ? (insert0(p, q) | ((uint64_t)want << q)) : p;
        acc += norm2(a[i]);
    }
    double r = block_sum(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = r;
}

// ---- Pauli strings ------------------------------------------------------------
//
// A string is (x, z): x = XOR of its X/Y qubits, z = XOR of its Y/Z qubits.
//   x == 0: sum over i of (-1)^|i & z| |a_i|^2
//   x != 0: sum over the pairs {i, j = i ^ x} of (-1)^|i & z| times Re (|x & z| even) or Im (odd) of
//           conj(a_j) a_i, which is the same from either end of the pair.
// Products and sums in FP64 for either state type.  Three kernels:
//   k_pauli_small  a string per CTA (states of at most SMALL_QUBITS: latency, not bandwidth);
//   k_pauli_z      up to ZK strings with x == 0 per read of the state;
//   k_pauli_span   up to SK strings with x != 0 per read of the state.

constexpr int SMALL_STRINGS = 480;
struct SmallStrings {
    uint32_t x[SMALL_STRINGS], z[SMALL_STRINGS];
};

// One launch for all strings, each summed by one CTA straight into out[]: a launch takes as long as
// such a sum (3 us).
template <typename T>
__global__ void k_pauli_small(const typename C2<T>::t* __restrict__ a, uint32_t n, const __grid_constant__ SmallStrings ss,
                              double* __restrict__ out) {
    __shared__ double sh[32];
    const uint32_t x = ss.x[blockIdx.x], z = ss.z[blockIdx.x];
    const bool odd = __popc(x & z) & 1;
    const uint32_t h = x ? 31 - __clz(x) : 0, count = x ? 1u << (n - 1) : 1u << n;
    double acc = 0.0;
#pragma unroll 4
    for (uint32_t p = threadIdx.x; p < count; p += blockDim.x) {
        uint32_t i = p;
        double v;
        if (x == 0) {
            v = norm2(a[i]);
        } else {
            i = (uint32_t)insert0(p, h);
            const auto ai = a[i], aj = a[i ^ x];
            const double air = ai.x, aii = ai.y, ajr = aj.x, aji = aj.y;
            v = odd ? ajr * aii - aji * air : ajr * air + aji * aii;
        }
        acc += (__popc(i & z) & 1) ? -v : v;
    }
    const double r = block_sum(acc, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = r;
}

// Strings with x == 0.  A thread takes 16 amplitudes whose indices differ in four fixed bits (f32: bit
// 0 and bits 9-11, f64: bits 8-11 of a tile of 2^12), forms the 16 signed sums of their probabilities
// over those bits (a Walsh-Hadamard transform, 64 additions), and every string adds the one that its
// mask on those bits selects, with the sign of the other bits: five instructions per string and 16
// amplitudes.  The sums go through the thread's own column of shared memory, as a register cannot be
// selected at run time.  Bound by HBM: 30 single-Z strings of 30 qubits f32 in 1.43 ms (a copy-rate read takes
// 1.31 ms).
constexpr int ZK = 32, ZPASSES = 11, ZT = 256;
struct ZPass {
    uint64_t z[ZK];
    uint16_t col[ZK];   // offset of the selected sum in a thread's column of sums
    uint32_t k;
    uint32_t pad;
};
struct ZPasses {
    ZPass p[ZPASSES];
};

template <typename T> struct Vec16;
template <> struct Vec16<float> { using t = float4; };
template <> struct Vec16<double> { using t = double2; };

// 16 bytes of amplitudes (two f32, one f64).  PAIRS: a caller's f32 array that is only 8-byte aligned
// (rq_expectation_batch_noalloc), two loads of 8 bytes.
template <bool PAIRS>
__device__ __forceinline__ float4 load16(const float4* p) {
    if constexpr (PAIRS) {
        const float2 x = __ldcs(reinterpret_cast<const float2*>(p)), y = __ldcs(reinterpret_cast<const float2*>(p) + 1);
        return make_float4(x.x, x.y, y.x, y.y);
    }
    return __ldcs(p);
}
template <bool PAIRS>
__device__ __forceinline__ double2 load16(const double2* p) {
    return __ldcs(p);
}

template <typename T, int KT, bool PAIRS>
__global__ void __launch_bounds__(ZT, KT > 16 ? 2 : 3) k_pauli_z(const typename C2<T>::t* __restrict__ a, uint64_t ntiles,
                                                   const __grid_constant__ ZPasses zp, double* __restrict__ partials,
                                                   uint32_t stride) {
    using VV = typename Vec16<T>::t;
    constexpr bool F = sizeof(T) == 4;
    __shared__ double W[16 * ZT];
    const ZPass& P = zp.p[blockIdx.y];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, K = P.k;
    const uint32_t ebits = F ? tid << 1 : tid;          // this thread's part of the element index
    uint64_t zl = lane < K ? P.z[lane] : 0ull;          // lane k keeps string k's mask
    uint32_t tpar = 0;                                  // bit k: parity of ebits & z_k
    for (uint32_t k = 0; k < K; ++k) tpar |= (uint32_t)(__popc(ebits & (uint32_t)P.z[k]) & 1) << k;
    double acc[KT];   // strings past K have mask 0 and are not written
#pragma unroll
    for (int k = 0; k < KT; ++k) acc[k] = 0.0;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const VV* src = reinterpret_cast<const VV*>(a + (tile << 12));
        double p[16];
        if constexpr (F) {   // register bit 0 = element bit 0, register bits 1-3 = element bits 9-11
            VV v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = load16<PAIRS>(src + u * ZT + tid);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                p[2 * u] = (double)v[u].x * v[u].x + (double)v[u].y * v[u].y;
                p[2 * u + 1] = (double)v[u].z * v[u].z + (double)v[u].w * v[u].w;
            }
        } else {             // register bits 0-3 = element bits 8-11
            VV v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = load16<PAIRS>(src + u * ZT + tid);
#pragma unroll
            for (int u = 0; u < 16; ++u) p[u] = v[u].x * v[u].x + v[u].y * v[u].y;
        }
#pragma unroll
        for (int b = 1; b < 16; b <<= 1)
#pragma unroll
            for (int m = 0; m < 16; ++m)
                if (!(m & b)) {
                    const double s = p[m], d = p[m | b];
                    p[m] = s + d;
                    p[m | b] = s - d;
                }
#pragma unroll
        for (int m = 0; m < 16; ++m) W[m * ZT + tid] = p[m];
        const uint32_t sg = tpar ^ __ballot_sync(0xffffffffu, __popcll((tile << 12) & zl) & 1);
#pragma unroll
        for (int k0 = 0; k0 < KT; k0 += 8) {
            double w[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k] = W[P.col[k0 + k] + tid];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int flip = (int)((sg << (31 - k0 - k)) & 0x80000000u);
                acc[k0 + k] += __hiloint2double(__double2hiint(w[k]) ^ flip, __double2loint(w[k]));
            }
        }
    }
    double* red = W;   // [warp][string]
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KT; ++k) {
        const double r = warp_sum(acc[k]);
        if (lane == 0) red[(tid >> 5) * ZK + k] = r;
    }
    __syncthreads();
    if (tid < K) {
        double r = 0.0;
        for (int w = 0; w < ZT / 32; ++w) r += red[w * ZK + tid];
        partials[(size_t)(blockIdx.y * ZK + tid) * stride + blockIdx.x] = r;
    }
}

// Strings with x != 0.  A pass owns eight independent X patterns (of the bits above the contiguous
// low ones): a tile is a coset of their span, 2^8 runs of 256 bytes, so for every string whose x lies
// in the span both ends of each pair are in the tile, and one read of the state serves them all
// (at least eight strings of a Hamiltonian of unrelated patterns; the X fields of an Ising model).
// The basis is in reduced echelon form: index = rep ^ sum_k u_k basis_k with rep zero at the pivot bits,
// so a string's local X mask is its pivot bits, and its local sign mask the parities of basis_k & z.
// A thread keeps 16 / 8 elements in registers as doubles and reads the partners from shared memory; a
// pair is walked once, by a register bit of the local X mask held at 0 (all elements where it has none:
// the sum is then halved by the caller).  Sums per string and thread live in shared memory across the
// CTA's tiles.  Bound by the FP64 conversions (XU 60 %, issue 47 %): 64 random strings of 24 qubits
// f32 in 0.59 ms (one read of the state per string: 2.8 ms).
constexpr int SPASSES = 10, ST = 512;
static_assert(ST == 1 << STB, "a tile index is a thread and a register");
struct SpanPasses {
    SpanPass p[SPASSES];
};
template <typename T> struct SpanShape;
template <> struct SpanShape<float> { static constexpr int C = 5, RB = 4; };    // 2^13 elements of 8 bytes
template <> struct SpanShape<double> { static constexpr int C = 4, RB = 3; };   // 2^12 elements of 16 bytes

template <typename T, int RB, int BIT, bool ODD>
__device__ __forceinline__ double span_walk(const double* ar, const double* ai, const typename C2<T>::t* tile,
                                            uint32_t tid, const SpanString& s) {
    constexpr int NB = BIT >= 0 ? RB - 1 : RB, NW = 1 << NB, B0 = BIT < 0 ? 0 : BIT;
    const uint32_t P = tid ^ s.lx;
    double v[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        const int i = BIT < 0 ? w : ((w >> B0) << (B0 + 1)) | (w & ((1 << B0) - 1));
        const auto b = tile[P ^ ((uint32_t)i << STB)];
        const double br = b.x, bi = b.y;
        v[w] = ODD ? br * ai[i] - bi * ar[i] : br * ar[i] + bi * ai[i];
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int gb = BIT >= 0 && b >= BIT ? b + 1 : b;
        const double sg = ((s.lz >> (STB + gb)) & 1u) ? -1.0 : 1.0;
#pragma unroll
        for (int w = 0; w < NW; w += 2 << b) v[w] = fma(sg, v[w + (1 << b)], v[w]);
    }
    return v[0];
}

template <typename T, int RB, bool ODD>
__device__ __forceinline__ double span_string(const double* ar, const double* ai, const typename C2<T>::t* tile,
                                              uint32_t tid, const SpanString& s) {
    switch (s.mode) {
        case 0: return span_walk<T, RB, 0, ODD>(ar, ai, tile, tid, s);
        case 1: return span_walk<T, RB, 1, ODD>(ar, ai, tile, tid, s);
        case 2: return span_walk<T, RB, 2, ODD>(ar, ai, tile, tid, s);
        case 3: if constexpr (RB > 3) return span_walk<T, RB, 3, ODD>(ar, ai, tile, tid, s); break;
        default: break;
    }
    return span_walk<T, RB, -1, ODD>(ar, ai, tile, tid, s);
}

template <typename T, bool PAIRS>
__global__ void __launch_bounds__(ST, 1) k_pauli_span(const typename C2<T>::t* __restrict__ a, uint32_t tile_bits,
                                                      const __grid_constant__ SpanPasses sp,
                                                      double* __restrict__ partials, uint32_t stride) {
    using V = typename C2<T>::t;
    constexpr int C = SpanShape<T>::C, RB = SpanShape<T>::RB, NR = 1 << RB;
    constexpr uint32_t L = 1u << (C + 8), EPV = 16 / sizeof(V);   // elements of a tile, per 16 bytes
    extern __shared__ __align__(16) unsigned char smem[];
    V* buf = reinterpret_cast<V*>(smem);                           // two tiles
    double* sums = reinterpret_cast<double*>(smem + 2 * L * sizeof(V));   // [string][thread]
    const SpanPass& P = sp.p[blockIdx.y];
    const uint32_t tid = threadIdx.x;
    for (uint32_t k = 0; k < P.k; ++k) sums[k * ST + tid] = 0.0;
    // this thread's 16-byte piece of a run: runs u = (tid >> 4) + 32 j, the piece tid & 15
    const uint32_t piece = (tid & 15u) * EPV;
    uint64_t ut = 0;
#pragma unroll
    for (int b = 0; b < 5; ++b)
        if ((tid >> (4 + b)) & 1u) ut ^= P.basis[b];
    const uint64_t ntiles = 1ull << tile_bits;
    auto rep_of = [&](uint64_t t) {
        uint64_t r = 0;
        for (uint32_t b = 0; b < tile_bits; ++b) r |= ((t >> b) & 1ull) << P.free_bit[b];
        return r;
    };
    auto load = [&](uint64_t rep, V* dst) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            uint64_t g = rep ^ ut;
            if (j & 1) g ^= P.basis[5];
            if (j & 2) g ^= P.basis[6];
            if (j & 4) g ^= P.basis[7];
            const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + (((tid >> 4) + 32 * j) << C) + piece);
            const V* p = a + g + piece;
            if constexpr (PAIRS) {   // 8-byte aligned f32 (load16)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(p) : "memory");
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + 8), "l"(p + 1) : "memory");
            } else {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(p) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    uint64_t tile = blockIdx.x;
    uint64_t rep = rep_of(tile);
    uint32_t at = 0;
    if (tile < ntiles) load(rep, buf);
    while (tile < ntiles) {
        const uint64_t next = tile + gridDim.x;
        uint64_t nrep = 0;
        if (next < ntiles) {
            nrep = rep_of(next);
            load(nrep, buf + (at ^ 1u) * L);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const V* tl = buf + at * L;
        double ar[NR], ai[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const V v = tl[tid | ((uint32_t)i << STB)];
            ar[i] = v.x;
            ai[i] = v.y;
        }
        for (uint32_t k = 0; k < P.k; ++k) {
            const SpanString& s = P.s[k];
            const double v = s.odd ? span_string<T, RB, true>(ar, ai, tl, tid, s) : span_string<T, RB, false>(ar, ai, tl, tid, s);
            const bool neg = (__popcll(rep & s.z) + __popc(tid & s.lz)) & 1;
            sums[k * ST + tid] += neg ? -v : v;
        }
        __syncthreads();
        tile = next;
        rep = nrep;
        at ^= 1u;
    }
    // the CTA's sum of each string: a warp per string, fixed order
    __syncthreads();
    const uint32_t lane = tid & 31u;
    for (uint32_t k = tid >> 5; k < P.k; k += ST / 32) {
        double r = 0.0;
        for (uint32_t t = lane; t < ST; t += 32) r += sums[k * ST + t];
        r = warp_sum(r);
        if (lane == 0) partials[(size_t)(P.row0 + k) * stride + blockIdx.x] = r;
    }
}

// <a|b> = sum conj(a_i) b_i
template <typename TA, typename TB>
__global__ void k_inner(const typename C2<TA>::t* __restrict__ a, const typename C2<TB>::t* __restrict__ b,
                        uint64_t n, double* __restrict__ partials, uint32_t stride) {
    __shared__ double sh[32];
    double re = 0.0, im = 0.0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        auto x = a[i];
        auto y = b[i];
        double xr = x.x, xi = x.y, yr = y.x, yi = y.y;
        re += xr * yr + xi * yi;
        im += xr * yi - xi * yr;
    }
    double r = block_sum(re, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = r;
    r = block_sum(im, sh);
    if (threadIdx.x == 0) partials[stride + blockIdx.x] = r;
}

// out[k] = sum_b partials[k*stride + b] over the first na blocks for k < ka, nb for the others, in a
// fixed order.  out may be pinned host memory.
__global__ void k_finalize(const double* __restrict__ partials, uint32_t ka, uint32_t na, uint32_t nb, uint32_t stride,
                           double* __restrict__ out) {
    __shared__ double sh[32];
    const double* p = partials + (size_t)blockIdx.x * stride;
    const uint32_t nblocks = blockIdx.x < ka ? na : nb;
    double acc = 0.0;
    for (uint32_t b = threadIdx.x; b < nblocks; b += blockDim.x) acc += p[b];
    double r = block_sum(acc, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = r;
}

// p_i = re*re + im*im, rounded exactly as a host computation without FMA
template <typename T>
__global__ void k_probs(const typename C2<T>::t* __restrict__ a, uint64_t n, double* __restrict__ out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        auto x = a[i];
        double re = x.x, im = x.y;
        out[i] = __dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im));
    }
}

int reduction_grid(rq_state* s) { return rq::num_sms(s->device) * 4; }

// finalize `nout` partial rows into the pinned staging, read by the host after one synchronisation
int finish(rq_state* s, unsigned nblocks, unsigned stride, unsigned nout, double* host) {
    RQ_TRY(rq::ensure_hbuf(s, nout));
    k_finalize<<<nout, TPB, 0, s->stream>>>(s->partials, nout, nblocks, nblocks, stride, s->hbuf);
    RQ_CUDA(cudaGetLastError());
    RQ_TRY(rq::sync_checked(s));
    for (unsigned k = 0; k < nout; ++k) host[k] = s->hbuf[k];
    return RQ_OK;
}

template <typename T, bool PAIRS>
int launch_strings_t(const PauliPlan& P, const void* amps, uint32_t n, cudaStream_t st, double* partials, double* out) {
    using V = typename C2<T>::t;
    const V* a = (const V*)amps;
    if (P.small) {
        for (uint32_t k0 = 0; k0 < P.rows; k0 += SMALL_STRINGS) {
            SmallStrings ss{};
            const uint32_t k1 = std::min<uint32_t>(P.rows, k0 + SMALL_STRINGS);
            for (uint32_t k = k0; k < k1; ++k) {
                ss.x[k - k0] = (uint32_t)P.terms[k].xmask;
                ss.z[k - k0] = (uint32_t)P.terms[k].pmask;
            }
            k_pauli_small<T><<<k1 - k0, TPB, 0, st>>>(a, n, ss, out + k0);
            RQ_CUDA(cudaGetLastError());
        }
        return RQ_OK;
    }
    const uint32_t nz = (uint32_t)P.zs.size(), zpasses = (nz + ZK - 1) / ZK;
    for (uint32_t p0 = 0; p0 < zpasses; p0 += ZPASSES) {
        ZPasses zp{};
        const uint32_t np = std::min<uint32_t>(ZPASSES, zpasses - p0);
        for (uint32_t p = 0; p < np; ++p) {
            const uint32_t k0 = (p0 + p) * ZK;
            zp.p[p].k = std::min<uint32_t>(ZK, nz - k0);
            for (uint32_t k = 0; k < zp.p[p].k; ++k) {
                const uint64_t z = P.terms[P.zs[k0 + k]].pmask;
                zp.p[p].z[k] = z;
                zp.p[p].col[k] = (uint16_t)(ZT * (sizeof(T) == 4 ? (z & 1u) | ((z >> 8) & 14u) : (z >> 8) & 15u));
            }
        }
        double* part = partials + (size_t)p0 * ZK * P.stride;
        auto kern = nz <= 8 ? k_pauli_z<T, 8, PAIRS> : nz <= 16 ? k_pauli_z<T, 16, PAIRS> : k_pauli_z<T, ZK, PAIRS>;
        kern<<<dim3(P.zblocks, np), ZT, 0, st>>>(a, 1ull << (n - 12), zp, part, P.stride);
        RQ_CUDA(cudaGetLastError());
    }
    constexpr int smem = 2 * (1 << (SpanShape<T>::C + 8)) * (int)sizeof(V) + SK * ST * (int)sizeof(double);
    if (!P.spans.empty())
        RQ_CUDA(cudaFuncSetAttribute(k_pauli_span<T, PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    for (size_t p0 = 0; p0 < P.spans.size(); p0 += SPASSES) {
        SpanPasses sp{};
        const size_t np = std::min<size_t>(SPASSES, P.spans.size() - p0);
        for (size_t p = 0; p < np; ++p) sp.p[p] = P.spans[p0 + p];
        k_pauli_span<T, PAIRS><<<dim3(P.sblocks, (unsigned)np), ST, smem, st>>>(a, n - SpanShape<T>::C - 8, sp, partials,
                                                                              P.stride);
        RQ_CUDA(cudaGetLastError());
    }
    k_finalize<<<P.rows, TPB, 0, st>>>(partials, nz, P.zblocks, P.sblocks, P.stride, out);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

// the sums of every string on `st`: out[row] (device or pinned host memory), partials of
// P.rows * P.stride doubles
int launch_strings(const PauliPlan& P, const void* amps, uint32_t n, int32_t prec, cudaStream_t st, double* partials,
                   double* out) {
    if (prec != RQ_F32) return launch_strings_t<double, false>(P, amps, n, st, partials, out);
    return reinterpret_cast<uintptr_t>(amps) % 16 == 0 ? launch_strings_t<float, false>(P, amps, n, st, partials, out)
                                                       : launch_strings_t<float, true>(P, amps, n, st, partials, out);
}

}  // namespace

namespace rq {

int prob_bit(rq_state* s, uint32_t q, int want_one, double* out) {
    unsigned G = reduction_grid(s);
    uint64_t count = q < 64 ? s->n >> 1 : s->n;
    G = std::min<unsigned>(G, grid_for(count, TPB, num_sms(s->device), 4));
    RQ_TRY(ensure_partials(s, 2 * (size_t)G + 8));
    if (s->prec == RQ_F32)
        k_prob<float><<<G, TPB, 0, s->stream>>>((const float2*)s->amps, count, q, want_one, s->partials);
    else
        k_prob<double><<<G, TPB, 0, s->stream>>>((const double2*)s->amps, count, q, want_one, s->partials);
    RQ_CUDA(cudaGetLastError());
    return finish(s, G, G, 1, out);
}

int norm_sq(rq_state* s, double* out) { return prob_bit(s, 64, 0, out); }

int pauli_expect(rq_state* s, const PauliMask* terms, uint32_t nterms, double* out) {
    if (nterms == 0) return RQ_OK;
    PauliPlan plan;
    plan_strings(s->nq, s->prec, num_sms(s->device), terms, nterms, plan);
    RQ_TRY(ensure_partials(s, (size_t)plan.rows * plan.stride));
    RQ_TRY(ensure_hbuf(s, plan.rows));
    RQ_TRY(launch_strings(plan, s->amps, s->nq, s->prec, s->stream, s->partials, s->hbuf));
    RQ_TRY(sync_checked(s));
    for (uint32_t k = 0; k < nterms; ++k) out[k] = s->hbuf[plan.row_of[k]] * plan.factor[k];
    return RQ_OK;
}

int inner(rq_state* a, rq_state* b, double* re, double* im) {
    unsigned G = reduction_grid(a);
    RQ_TRY(ensure_partials(a, 2 * (size_t)G + 8));
    // b's pending work must be done before a's stream reads it
    RQ_TRY(sync_checked(b));
    if (a->prec == RQ_F32 && b->prec == RQ_F32)
        k_inner<float, float><<<G, TPB, 0, a->stream>>>((const float2*)a->amps, (const float2*)b->amps, a->n, a->partials, G);
    else if (a->prec == RQ_F32)
        k_inner<float, double><<<G, TPB, 0, a->stream>>>((const float2*)a->amps, (const double2*)b->amps, a->n, a->partials, G);
    else if (b->prec == RQ_F32)
        k_inner<double, float><<<G, TPB, 0, a->stream>>>((const double2*)a->amps, (const float2*)b->amps, a->n, a->partials, G);
    else
        k_inner<double, double><<<G, TPB, 0, a->stream>>>((const double2*)a->amps, (const double2*)b->amps, a->n, a->partials, G);
    RQ_CUDA(cudaGetLastError());
    double r[2];
    RQ_TRY(finish(a, G, G, 2, r));
    *re = r[0];
    *im = r[1];
    return RQ_OK;
}

int probabilities_dev(rq_state* s, double* dev_out) {
    unsigned g = grid_for(s->n, TPB, num_sms(s->device));
    if (s->prec == RQ_F32) k_probs<float><<<g, TPB, 0, s->stream>>>((const float2*)s->amps, s->n, dev_out);
    else k_probs<double><<<g, TPB, 0, s->stream>>>((const double2*)s->amps, s->n, dev_out);
    RQ_CUDA(cudaGetLastError());
    return RQ_OK;
}

}  // namespace rq

// ---------------------------------------------------------------------------
// Allocation-free expectation values (rq_expectation_batch_noalloc).
//
// Some callers cannot allocate device memory at all (their budget is fixed, or
// another framework owns the allocator).  For them the partial sums of the
// Pauli-string reduction live in this one static device array instead of the
// per-state buffer.  It is fixed in size, exists once per GPU that loads the
// library, and is shared by every call: two calls in flight at once on the GPU
// would overwrite each other's partials, so callers must serialise them.
// Nothing in it has to start at zero: every slot a call reads back was
// written by that same call's first kernel.
// ---------------------------------------------------------------------------
static __device__ __align__(256) double g_noalloc_scratch[RQ_NOALLOC_SCRATCH_DOUBLES];

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
double* g_noalloc_addr[kMaxDevices] = {nullptr};
unsigned long long g_noalloc_ctx[kMaxDevices] = {0};   // context the address belongs to

// Device address of g_noalloc_scratch on the current device.  In host code
// the array's name is only a host-side stand-in, so the address is looked up
// with that device current, once per device and context: the first call on a
// device (and the first call after its context was re-created, for example by
// cudaDeviceReset, which reloads the module and can move the array) looks it
// up; later calls reuse it.
int noalloc_scratch_address(int device, double** out) {
    if (device < 0 || device >= kMaxDevices) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "device index out of range");
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    const unsigned long long ctx = rq::current_context_id();
    if (!g_noalloc_addr[device] || ctx == 0 || ctx != g_noalloc_ctx[device]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return rq::cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
        g_noalloc_addr[device] = static_cast<double*>(p);
        g_noalloc_ctx[device] = ctx;
    }
    *out = g_noalloc_addr[device];
    return RQ_OK;
}

}  // namespace

extern "C" int rq_expectation_batch_noalloc(const void* device_amps, uint32_t num_qubits, int32_t precision,
                                            const rq_pauli_op* ops, const uint32_t* offsets, uint32_t nstrings,
                                            double* out, void* stream_handle) {
    if (!device_amps || (!out && nstrings) || (!offsets && nstrings))
        return rq::fail(RQ_ERR_INVALID_ARGUMENT, "null pointer");
    if (precision != RQ_F32 && precision != RQ_F64)
        return rq::fail(RQ_ERR_INVALID_ARGUMENT, "precision must be RQ_F32 or RQ_F64");
    uint32_t maxq = precision == RQ_F32 ? RQ_MAX_QUBITS_F32 : RQ_MAX_QUBITS_F64;
    if (num_qubits == 0 || num_qubits > maxq)
        return rq::fail(RQ_ERR_QUBIT_LIMIT_EXCEEDED, "num_qubits must be in 1.." + std::to_string(maxq));
    if (nstrings > RQ_NOALLOC_MAX_STRINGS)
        return rq::fail(RQ_ERR_INVALID_ARGUMENT, "rq_expectation_batch_noalloc takes at most " +
                                                     std::to_string(RQ_NOALLOC_MAX_STRINGS) + " Pauli strings per call, got " +
                                                     std::to_string(nstrings));
    if (nstrings == 0) return RQ_OK;
    const size_t align = precision == RQ_F32 ? sizeof(float2) : sizeof(double2);
    if (reinterpret_cast<uintptr_t>(device_amps) % align)   // a load would fault
        return rq::fail(RQ_ERR_INVALID_ARGUMENT, "device_amps must be aligned to an amplitude (" + std::to_string(align) + " bytes)");
    if (!ops && offsets[nstrings] > offsets[0]) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "null pointer");
    // Pauli strings in mask form (same rules as rq_state_expectation_batch)
    std::vector<rq::PauliMask> terms(nstrings);
    for (uint32_t k = 0; k < nstrings; ++k) {
        if (offsets[k + 1] < offsets[k]) return rq::fail(RQ_ERR_INVALID_ARGUMENT, "offsets must be non-decreasing");
        rq::PauliMask m{0, 0, 0};
        for (uint32_t j = offsets[k]; j < offsets[k + 1]; ++j) {
            uint32_t q = ops[j].qubit;
            int op = ops[j].op;
            if (op < RQ_PAULI_I || op > RQ_PAULI_Z)
                return rq::fail(RQ_ERR_INVALID_ARGUMENT, "invalid Pauli operator " + std::to_string(op));
            if (op == RQ_PAULI_I) continue;
            if (q >= num_qubits)
                return rq::fail(RQ_ERR_INVALID_QUBIT_INDEX, "invalid qubit index " + std::to_string(q) + " for " +
                                                                std::to_string(num_qubits) + "-qubit system");
            uint64_t b = 1ull << q;
            if (op == RQ_PAULI_X || op == RQ_PAULI_Y) m.xmask ^= b;
            if (op == RQ_PAULI_Y || op == RQ_PAULI_Z) m.pmask ^= b;
            if (op == RQ_PAULI_Y) m.ny += 1;
        }
        m.ny &= 3u;
        terms[k] = m;
    }
    int device = 0;
    RQ_CUDA(cudaGetDevice(&device));
    double* scratch = nullptr;
    RQ_TRY(noalloc_scratch_address(device, &scratch));
    cudaStream_t st = static_cast<cudaStream_t>(stream_handle);
    // partials occupy [0, nstrings * stride), at most RQ_NOALLOC_MAX_STRINGS * RQ_NOALLOC_MAX_BLOCKS;
    // the finalised sums follow
    PauliPlan plan;
    plan_strings(num_qubits, precision, rq::num_sms(device), terms.data(), nstrings, plan);
    if (plan.stride > RQ_NOALLOC_MAX_BLOCKS) {   // fewer CTAs take more tiles each
        plan.zblocks = std::min<uint32_t>(plan.zblocks, RQ_NOALLOC_MAX_BLOCKS);
        plan.sblocks = std::min<uint32_t>(plan.sblocks, RQ_NOALLOC_MAX_BLOCKS);
        plan.stride = RQ_NOALLOC_MAX_BLOCKS;
    }
    double* sums = scratch + (size_t)nstrings * plan.stride;
    RQ_TRY(launch_strings(plan, device_amps, num_qubits, precision, st, scratch, sums));
    std::vector<double> host(nstrings);
    RQ_CUDA(cudaMemcpyAsync(host.data(), sums, nstrings * sizeof(double), cudaMemcpyDeviceToHost, st));
    RQ_CUDA(cudaStreamSynchronize(st));
    for (uint32_t k = 0; k < nstrings; ++k) out[k] = host[plan.row_of[k]] * plan.factor[k];
    return RQ_OK;
}
