// rq_tree.cuh -- FP64 prefix trees over the probabilities of one or many states, shared by the
// single-state sampler (rq_sample.cu) and the batched QAOA engine (rq_batch.cu).
//
// A tree of n index bits lies at offsets 2^L - 1, levels L = 0 .. n-1: entry j of level L is the sum of
// |a_i|^2 over the i whose low L (permuted) bits are j, level n the probabilities themselves (not
// stored).  Every entry is the rounded sum of its two children, j and j + 2^L of level L + 1, without FMA,
// so a host fold of the same probabilities gives identical bits.
#pragma once

#include "rq_internal.cuh"

namespace rqt {

using rqd::C2;

struct Perm {
    uint8_t order[64];   // permuted bit position -> qubit
    uint8_t pos[64];     // qubit -> permuted bit position
    uint32_t n;
    int identity;
};

__device__ __forceinline__ uint64_t unpermute(uint64_t j, const Perm& P) {
    if (P.identity) return j;
    uint64_t i = 0;
    for (uint32_t b = 0; b < P.n; ++b) i |= ((j >> b) & 1ull) << P.order[b];
    return i;
}

template <typename T>
__device__ __forceinline__ double prob_at(const typename C2<T>::t* a, uint64_t i) {
    const auto x = a[i];
    const double re = x.x, im = x.y;
    return __dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im));
}

constexpr int TREE_TPB = 256;
constexpr int TREE_TAIL = 12;   // levels up to 2^TREE_TAIL entries are folded by one CTA

// three levels from the eight values v[m] = entry j + m 2^k of level k + 3, for one j < 2^k
__device__ __forceinline__ void store_three(double* __restrict__ tree, uint32_t k, uint64_t j, const double* v) {
    double* l2 = tree + ((4ull << k) - 1);
    double* l1 = tree + ((2ull << k) - 1);
    double* l0 = tree + ((1ull << k) - 1);
    double s[4], t[2];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        s[m] = __dadd_rn(v[m], v[m + 4]);
        l2[j + ((uint64_t)m << k)] = s[m];
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        t[m] = __dadd_rn(s[m], s[m + 2]);
        l1[j + ((uint64_t)m << k)] = t[m];
    }
    l0[j] = __dadd_rn(t[0], t[1]);
}

// Levels n-1, n-2 and n-3 from the amplitudes: eight probabilities of a thread, all loads in flight, and
// no level is read back.  A 23-qubit f64 state takes 5 kernels and 43 us (a copy-rate read of the
// amplitudes alone: 20 us); a launch a level, which reads every level again, 12 kernels and 62 us.
template <typename T>
__global__ void __launch_bounds__(TREE_TPB) k_tree_leaf(const typename C2<T>::t* __restrict__ amps, const Perm P,
                                                        double* __restrict__ tree) {
    const uint32_t n = P.n, k = n - 3;
    const typename C2<T>::t* a = amps + ((uint64_t)blockIdx.y << n);
    double* t = tree + ((uint64_t)blockIdx.y << n);
    uint64_t off[3] = {1ull << k, 2ull << k, 4ull << k};
    if (!P.identity)
        for (int b = 0; b < 3; ++b) off[b] = 1ull << P.order[k + b];
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < 1ull << k; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = unpermute(j, P);
        double v[8];
#pragma unroll
        for (int m = 0; m < 8; ++m)
            v[m] = prob_at<T>(a, i | (m & 1 ? off[0] : 0) | (m & 2 ? off[1] : 0) | (m & 4 ? off[2] : 0));
        store_three(t, k, j, v);
    }
}

// levels k+2, k+1 and k from level k+3
static __global__ void __launch_bounds__(TREE_TPB) k_tree_fold(double* __restrict__ tree, uint32_t n, uint32_t k) {
    double* t = tree + ((uint64_t)blockIdx.y << n);
    const double* up = t + ((8ull << k) - 1);
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < 1ull << k; j += (uint64_t)gridDim.x * blockDim.x) {
        double v[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = up[j + ((uint64_t)m << k)];
        store_three(t, k, j, v);
    }
}

// every level below `top` (2^top <= 2^TREE_TAIL entries); top == n: from the amplitudes
template <typename T>
__global__ void k_tree_tail(const typename C2<T>::t* __restrict__ amps, const Perm P, double* __restrict__ tree, uint32_t top) {
    double* t = tree + ((uint64_t)blockIdx.x << P.n);
    uint32_t k = top;
    if (top == P.n) {   // the state itself: level n-1 from the amplitudes
        const typename C2<T>::t* a = amps + ((uint64_t)blockIdx.x << P.n);
        const uint64_t half = 1ull << --k;
        for (uint64_t j = threadIdx.x; j < half; j += blockDim.x)
            t[half - 1 + j] = __dadd_rn(prob_at<T>(a, unpermute(j, P)), prob_at<T>(a, unpermute(j + half, P)));
        __syncthreads();
    }
    while (k-- > 0) {
        const double* up = t + ((2ull << k) - 1);
        double* dn = t + ((1ull << k) - 1);
        const uint64_t len = 1ull << k;
        for (uint64_t j = threadIdx.x; j < len; j += blockDim.x) dn[j] = __dadd_rn(up[j], up[j + len]);
        __syncthreads();
    }
}

// the trees of `count` states of P.n index bits, tree c at tree + c * 2^n, on `st`
template <typename T>
int build_trees(const typename C2<T>::t* amps, const Perm& P, uint64_t count, double* tree, int sms, cudaStream_t st) {
    const uint32_t n = P.n;
    uint32_t k = n;
    for (uint64_t c0 = 0; c0 < count; c0 += 65535) {   // grid.y
        const unsigned nc = (unsigned)(count - c0 < 65535 ? count - c0 : 65535);
        const typename C2<T>::t* a = amps + (c0 << n);
        double* t = tree + (c0 << n);
        auto grid = [&](uint32_t lev) {
            const uint64_t need = ((1ull << lev) + TREE_TPB - 1) / TREE_TPB, cap = ((uint64_t)sms * 8 + nc - 1) / nc;
            return dim3((unsigned)(need < cap ? need : cap), nc);
        };
        k = n;
        if (n > (uint32_t)TREE_TAIL) {
            k = n - 3;
            k_tree_leaf<T><<<grid(k), TREE_TPB, 0, st>>>(a, P, t);
            RQ_CUDA(cudaGetLastError());
            for (; k > (uint32_t)TREE_TAIL; k -= 3) {
                k_tree_fold<<<grid(k - 3), TREE_TPB, 0, st>>>(t, n, k - 3);
                RQ_CUDA(cudaGetLastError());
            }
        }
        if (k > 0) {
            const unsigned threads = k >= 11 ? 1024u : 256u;
            k_tree_tail<T><<<nc, threads, 0, st>>>(a, P, t, k);
            RQ_CUDA(cudaGetLastError());
        }
    }
    return RQ_OK;
}

}  // namespace rqt
