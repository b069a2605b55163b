// Grid-wide sums of the persistent solvers (sm_100a), two axes at a time.
#pragma once

#include "ktg_common.cuh"

namespace ktg {

constexpr int kSumGroups = 5;  // records a lane polls: at most 160 blocks
constexpr int kSumSets = 4;
constexpr int kSumWords = 4;   // words per axis of a record, at most
// A partial sum that has not been written yet. Arithmetic produces only the
// canonical NaN, and a sum that carries this pattern is replaced by it.
constexpr unsigned long long kUnset = ~0ull;

// K (1 to 4) words of a record (16-byte aligned, K rounded up to even).
template <bool Acquire>
__device__ __forceinline__ void ld_pair(const unsigned long long *p, unsigned long long &a,
                                        unsigned long long &b) {
    if constexpr (Acquire)
        asm volatile("ld.acquire.gpu.global.v2.u64 {%0, %1}, [%2];"
                     : "=l"(a), "=l"(b) : "l"(p) : "memory");
    else
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                     : "=l"(a), "=l"(b) : "l"(p) : "memory");
}

template <bool Acquire, int K>
__device__ __forceinline__ void ld_words(const unsigned long long *p, unsigned long long (&u)[K]) {
    if constexpr (K == 1) {
        if constexpr (Acquire)
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(u[0]) : "l"(p) : "memory");
        else
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(u[0]) : "l"(p) : "memory");
    } else if constexpr (K == 2) {
        ld_pair<Acquire>(p, u[0], u[1]);
    } else {
        unsigned long long last = 0ull;
        ld_pair<Acquire>(p, u[0], u[1]);
        ld_pair<Acquire>(p + 2, u[2], K == 4 ? u[K - 1] : last);
    }
}

__device__ __forceinline__ void st_relaxed_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void fence_acq_rel_gpu() {
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
}

// Warp totals of K values per lane: lane k < K returns the total of value k.
// While more than one value is left a step hands half of them to the partner
// lane instead of exchanging all, so K values cost P - 1 + (5 - log2 P)
// exchanges (P: K rounded up to a power of two) instead of 5 K.
template <int K>
__device__ __forceinline__ double warp_sums(const double (&v)[K]) {
    constexpr int P = K == 1 ? 1 : K == 2 ? 2 : K <= 4 ? 4 : 8;
    const int lane = threadIdx.x & 31;
    double t[P];
#pragma unroll
    for (int k = 0; k < P; ++k) t[k] = k < K ? v[k] : 0.0;
#pragma unroll
    for (int h = P / 2; h >= 1; h >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const double give = up ? t[k] : t[k + h];
            const double keep = up ? t[k + h] : t[k];
            t[k] = keep + __shfl_xor_sync(0xffffffffu, give, h);
        }
    }
#pragma unroll
    for (int o = P; o < 32; o <<= 1) t[0] += __shfl_xor_sync(0xffffffffu, t[0], o);
    return t[0];  // lane l: value l mod P
}

// Grid-wide sums that are also a grid barrier, one hop through L2: every block
// stores its partial sums in a record of its own and polls all blocks'
// records; the totals are added in a fixed order, the same in every block.
// Warp a does it all for axis a (a lane polls up to kSumGroups records) and goes
// straight on to that axis's scalars, so a reduction costs the block two
// __syncthreads. 211k cells, 148 blocks: 4.5k cycles after the last arrival;
// an arrival counter with a generation word, a read of the partials by all
// threads and the scalars in every thread took 7k.
//
// A word is written and later set back to kUnset by its owner. Set b % kSumSets
// serves reduction b: a block that has passed reduction b knows that every
// block has arrived at it and so has read all records of b - 1, and resets its
// own of that set. The reset is published by its next fence, at most two
// reductions later, and the set is used again three later. Reductions without
// Publish carry no fence, so they establish no order between blocks that the
// memory model would promise for accesses at large. Callers use them only to
// keep a later overwrite behind earlier reads, and only where every value read
// goes into a sum: the writer holds a total computed from it, and a load whose
// value has been used cannot return a later store. (The solves' gathers qualify;
// those of an axis that is done do not enter a sum, but nothing writes its
// entries any more.) Reads of what others wrote need Publish.
//
// A record holds W words of each axis.
template <int W>
struct AllReduce {
    static constexpr int kRecord = 2 * W;
    unsigned long long *slots;  // [kSumSets][grid][kRecord]: words W a ... of axis a
    int *status;
    unsigned round;
    uint64_t total_deadline;
    uint64_t barrier_timeout;

    // v: K values per thread and axis. In warp a every lane calls
    // finish(a, totals of axis a) before the block goes on. Publish: other
    // blocks read what this block wrote before the call. Returns false in every
    // thread when a wait gave up. scratch holds 2 K * 33 doubles.
    template <bool Publish, int K, class Finish>
    __device__ bool sum(const double (&v)[2 * K], double *scratch, Finish finish) {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const int nw = blockDim.x >> 5;
        const int grid = gridDim.x;
        const double wsum = warp_sums<2 * K>(v);
        if (lane < 2 * K) scratch[lane * 33 + wid] = wsum;
        __syncthreads();
        int bad = 0;
        if (wid < 2) {
            double t[K];
#pragma unroll
            for (int k = 0; k < K; ++k) t[k] = lane < nw ? scratch[(wid * K + k) * 33 + lane] : 0.0;
            double mine = warp_sums<K>(t);
            if (grid > 1) {
                unsigned long long *set =
                    slots + static_cast<size_t>(round % kSumSets) * grid * kRecord + W * wid;
                if (lane < K) {
                    unsigned long long u =
                        static_cast<unsigned long long>(__double_as_longlong(mine));
                    if (u == kUnset) u = 0x7ff8000000000000ull;
                    if (Publish) fence_acq_rel_gpu();
                    st_relaxed_u64(set + static_cast<size_t>(blockIdx.x) * kRecord + lane, u);
                }
                unsigned long long u[kSumGroups][K];
                unsigned wait = 0;
#pragma unroll
                for (int g = 0; g < kSumGroups; ++g) {
#pragma unroll
                    for (int k = 0; k < K; ++k) u[g][k] = 0ull;
                    if (g * 32 + lane < grid) wait |= 1u << g;
                }
                uint64_t deadline = 0;
                for (uint32_t spins = 1; wait; ++spins) {
#pragma unroll
                    for (int g = 0; g < kSumGroups; ++g)
                        if ((wait >> g) & 1u)
                            ld_words<Publish>(set + static_cast<size_t>(g * 32 + lane) * kRecord,
                                              u[g]);
#pragma unroll
                    for (int g = 0; g < kSumGroups; ++g) {
                        bool have = true;
#pragma unroll
                        for (int k = 0; k < K; ++k) have = have && u[g][k] != kUnset;
                        if (have) wait &= ~(1u << g);
                    }
                    if (wait && (spins & 63u) == 0u) {
                        const uint64_t now = global_timer_ns();
                        if (deadline == 0) deadline = min(now + barrier_timeout, total_deadline);
                        if (ld_relaxed_gpu(status) != kStatusOk || now > deadline) {
                            atomicCAS(status, kStatusOk, kStatusTimeout);
                            bad = 1;
                            break;
                        }
                    }
                }
                __syncwarp();
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    t[k] = __longlong_as_double(static_cast<long long>(u[0][k]));
#pragma unroll
                    for (int g = 1; g < kSumGroups; ++g)
                        t[k] += __longlong_as_double(static_cast<long long>(u[g][k]));
                }
                mine = warp_sums<K>(t);
                if (round > 0 && lane < W)
                    st_relaxed_u64(slots + (static_cast<size_t>((round - 1) % kSumSets) * grid +
                                            blockIdx.x) * kRecord + W * wid + lane,
                                   kUnset);
            }
#pragma unroll
            for (int k = 0; k < K; ++k) t[k] = __shfl_sync(0xffffffffu, mine, k);
            finish(wid, t);
        }
        ++round;
        return !__syncthreads_or(bad);
    }
};

}  // namespace ktg
