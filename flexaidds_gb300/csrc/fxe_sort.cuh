// fxe_sort.cuh — block-wide ascending sort of (64-bit key, index) pairs, ties by index.
//
// A bitonic network over kSortThreads threads, each holding kE pairs in registers (pair e of thread t
// is entry t + kSortThreads * e): strides below a warp's width exchange by shuffles, strides of a
// whole block inside a thread, and only the strides between go through shared memory with a block
// barrier — 20 of the 66 stages of 2,048 pairs. Bound by the latency of its stages: ordering a launch's
// 2,000 poses takes 28 us with it and took 98 with every stage in shared memory behind a barrier (4,096
// poses: 53 us).
#pragma once

#include <cstdint>

namespace fxe {

constexpr int kSortThreads = 1024;

// Keeps the smaller (up) or larger of the pairs at an exchange's two ends.
__device__ __forceinline__ void sort_keep(uint64_t& k, int& i, uint64_t k2, int i2, bool keep_min) {
    const bool less = k2 < k || (k2 == k && i2 < i);
    if (less == keep_min) {
        k = k2;
        i = i2;
    }
}

// Orders two pairs of one thread, ascending when up.
__device__ __forceinline__ void sort_pair(uint64_t& ka, int& ia, uint64_t& kb, int& ib, bool up) {
    const bool gt = ka > kb || (ka == kb && ia > ib);
    if (gt == up) {
        const uint64_t k = ka;
        ka = kb;
        kb = k;
        const int i = ia;
        ia = ib;
        ib = i;
    }
}

// key[e], idx[e]: the thread's pairs. buf_k, buf_i: kSortThreads * kE entries of shared memory,
// whose first n hold the sorted pairs at the end (every thread of the block calls; block barriers).
template <int kE>
__device__ __forceinline__ void block_sort_regs(uint64_t* key, int* idx, uint64_t* buf_k, int* buf_i) {
    const int t = threadIdx.x;
    constexpr int N = kSortThreads * kE;
    #pragma unroll 1
    for (int k = 2; k <= N; k <<= 1) {
        #pragma unroll 1
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j == kSortThreads) {
                if constexpr (kE >= 2) {
                    sort_pair(key[0], idx[0], key[1], idx[1], (t & k) == 0);
                    if constexpr (kE == 4) sort_pair(key[2], idx[2], key[3], idx[3], ((t + 2 * kSortThreads) & k) == 0);
                }
            } else if (j == 2 * kSortThreads) {
                if constexpr (kE == 4) {
                    sort_pair(key[0], idx[0], key[2], idx[2], (t & k) == 0);
                    sort_pair(key[1], idx[1], key[3], idx[3], ((t + kSortThreads) & k) == 0);
                }
            } else if (j >= 32) {
                __syncthreads();
#pragma unroll
                for (int e = 0; e < kE; ++e) {
                    buf_k[t + kSortThreads * e] = key[e];
                    buf_i[t + kSortThreads * e] = idx[e];
                }
                __syncthreads();
#pragma unroll
                for (int e = 0; e < kE; ++e) {
                    const int i = t + kSortThreads * e;
                    sort_keep(key[e], idx[e], buf_k[i ^ j], buf_i[i ^ j], ((i & k) == 0) == ((i & j) == 0));
                }
            } else {
#pragma unroll
                for (int e = 0; e < kE; ++e) {
                    const int i = t + kSortThreads * e;
                    const uint64_t k2 = __shfl_xor_sync(0xffffffffu, (unsigned long long)key[e], j);
                    const int i2 = __shfl_xor_sync(0xffffffffu, idx[e], j);
                    sort_keep(key[e], idx[e], k2, i2, ((i & k) == 0) == ((i & j) == 0));
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < kE; ++e) {
        buf_k[t + kSortThreads * e] = key[e];
        buf_i[t + kSortThreads * e] = idx[e];
    }
    __syncthreads();
}

// Sorts the first n pairs of buf_k / buf_i in place (n <= 4 * kSortThreads, which the buffers hold;
// entries past n are padding afterwards).
__device__ __forceinline__ void block_sort(uint64_t* buf_k, int* buf_i, int n) {
    const int t = threadIdx.x;
    __syncthreads();
    if (n <= kSortThreads) {
        uint64_t k[1] = {t < n ? buf_k[t] : ~0ull};
        int i[1] = {t < n ? buf_i[t] : 0x7fffffff};
        block_sort_regs<1>(k, i, buf_k, buf_i);
    } else if (n <= 2 * kSortThreads) {
        uint64_t k[2];
        int i[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int p = t + kSortThreads * e;
            k[e] = p < n ? buf_k[p] : ~0ull;
            i[e] = p < n ? buf_i[p] : 0x7fffffff;
        }
        block_sort_regs<2>(k, i, buf_k, buf_i);
    } else {
        uint64_t k[4];
        int i[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int p = t + kSortThreads * e;
            k[e] = p < n ? buf_k[p] : ~0ull;
            i[e] = p < n ? buf_i[p] : 0x7fffffff;
        }
        block_sort_regs<4>(k, i, buf_k, buf_i);
    }
}

}  // namespace fxe
