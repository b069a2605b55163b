// Batched Jacobi-PCG over many independent systems (sm_100a).
//
// The solves of solveBothAxes (globalPlacer/simpl/simpl_lss.cc:203-290) for
// many netlists at once -- x and y of each, of uneven sizes -- in one
// persistent launch of thread-block clusters:
//   * one cluster (2-16 CTAs on as many SMs) solves one system at a time; its
//     CTAs split the rows, meet at hardware cluster barriers, and combine
//     their dot-product partials through distributed shared memory in a
//     fixed order (deterministic, identical in every CTA);
//   * clusters take systems from an atomic work queue ordered largest first,
//     so uneven sizes balance without any grid-wide synchronisation;
//   * FP64 Jacobi-PCG (the reference's method), or FP32 Jacobi-PCG inside FP64
//     iterative refinement (true FP64 residual as the convergence test);
//     the latter on a renumbered FP32 copy of the system (Jagged), with the
//     search direction in every CTA's shared memory, where that pays (jagged_pays,
//     near_clusters), else on the system itself in warp tiles;
//   * per system the device records iterations, the final residual and the
//     solve latency (%globaltimer from dequeue to done).
// The launch only enqueues work, so the whole batch solve is captured once
// in a CUDA graph and replayed.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <functional>
#include <new>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include "ktg_common.cuh"
#include "ktg_context.h"
#include "ktg_spmv.cuh"
#include "ktplace_b200.h"

namespace cg = cooperative_groups;

namespace ktg {
namespace {

struct SysDesc {
    int64_t row_base;  // first row in the concatenated vectors
    int64_t nnz_base;  // first entry in col/val
    int32_t n;
    int32_t nnz;
};

struct BatchArgs {
    const SysDesc *sys;
    const int32_t *order;  // solve order (largest first)
    int32_t num_sys;
    const int32_t *rp;     // system k's row_ptr (local offsets) at row_base + k
    const int32_t *col;
    const double *val;
    const float *val32;
    const double *diag;
    const double *rhs;
    double *x;
    double *r;
    double *z;
    double *p;
    double *ap;
    float *d32;
    float *ri32;
    float *z32;
    float *p32;
    float *ap32;
    // the mixed solve's copy of the systems (Jagged)
    int32_t *jcol;
    float *jval;
    float *diag32;
    int32_t *perm, *inv, *len, *start, *next;
    unsigned *queue;
    ktg_batch_result *results;
    double tol;
    double inner_tol;
    int64_t max_iter;
    int32_t max_outer;
    uint64_t total_timeout_ns;
};

// Cluster-wide deterministic sum of K values per thread. Partials are double
// buffered in shared memory so one cluster barrier per reduction suffices. Every
// thread reads all of them, or (ByWarp) one warp reads each once for the others:
// 16 CTAs of 512 threads, 2,000 rows, 0.91 against 0.70 ms a solve; 4 CTAs, 52,000
// rows, 22.4 against 23.8.
constexpr int kPortable = 8;  // CTAs of a portable cluster

template <int K, bool ByWarp>
__device__ __forceinline__ void cluster_sum(double (&v)[K], double *part, int &buf,
                                            double *scratch, cg::cluster_group &cl) {
    block_sum_k<K>(v, scratch);
    double *mine = part + buf * 4;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) mine[k] = v[k];
    }
    cl.sync();
    const int nb = static_cast<int>(cl.num_blocks()), lane = threadIdx.x & 31;
    if constexpr (!ByWarp) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double t = 0.0;
            for (int q = 0; q < nb; ++q) t += *cl.map_shared_rank(mine + k, q);
            v[k] = t;
        }
    } else {
        if (threadIdx.x < 32) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const double q = lane < nb ? *cl.map_shared_rank(mine + k, lane) : 0.0;
                double t = 0.0;
                for (int r = 0; r < nb; ++r) t += __shfl_sync(0xffffffffu, q, r);
                if (lane == 0) scratch[k] = t;
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = scratch[k];
        __syncthreads();
    }
    buf ^= 1;
}

template <typename T, typename V>
__device__ __forceinline__ T row_dot(const int32_t *rp, const int32_t *col, const V *val,
                                     const T *in, int32_t i, T acc) {
    int32_t e = rp[i];
    const int32_t e1 = rp[i + 1];
    for (; e + 4 <= e1; e += 4) {
        const int32_t c0 = __ldg(col + e), c1 = __ldg(col + e + 1);
        const int32_t c2 = __ldg(col + e + 2), c3 = __ldg(col + e + 3);
        const T g0 = __ldcg(in + c0), g1 = __ldcg(in + c1);
        const T g2 = __ldcg(in + c2), g3 = __ldcg(in + c3);
        acc += static_cast<T>(__ldg(val + e)) * g0;
        acc += static_cast<T>(__ldg(val + e + 1)) * g1;
        acc += static_cast<T>(__ldg(val + e + 2)) * g2;
        acc += static_cast<T>(__ldg(val + e + 3)) * g3;
    }
    for (; e < e1; ++e) acc += static_cast<T>(__ldg(val + e)) * __ldcg(in + __ldg(col + e));
    return acc;
}

// Rows a thread handles at a time in the vector phases: their loads are issued
// together.
constexpr int kBatchRows = 4;

template <class Row>
__device__ __forceinline__ void each_rows(int32_t a, int32_t b, Row row) {
    const int32_t step = kBatchRows * blockDim.x, last = (kBatchRows - 1) * blockDim.x;
    int32_t i = a + static_cast<int32_t>(threadIdx.x);
    for (; i + last < b; i += step) row(i, std::integral_constant<int, kBatchRows>());
    for (; i < b; i += blockDim.x) row(i, std::integral_constant<int, 1>());
}

// Whether the renumbered copy and the direction in shared memory pay for a system.
// Few rows a CTA do not make up for building the copy (ms a solve, without and with:
// 300 rows 1 x 512 0.27 and 0.38, 1,000 rows 4 x 512 0.50 and 0.56, 2 x 512 0.58 and
// 0.58, 1 x 512 0.78 and 0.72; 5,000 rows 8 x 512 1.14 and 1.06), and in clusters of
// 16 storing every CTA's rows to all others takes what the gathers save (16 x 512:
// 10,000 rows 1.92 and 2.01, 48,000 rows 7.5 and 9.9).
constexpr int kJaggedRows = 600;  // of a CTA

__host__ __device__ inline bool jagged_pays(int64_t rows, int cluster) {
    return cluster <= kPortable && rows >= static_cast<int64_t>(kJaggedRows) * cluster;
}

// Whether they pay for a launch whose systems are all like this one; beside one for
// which they do, the rule above holds (the tiles are slower in the kernel that has
// both). With more than 512 threads the tiles are faster and the copy's warps have less
// each: it pays from 1,400 rows and 8,500 entries a CTA on, and not for chains (speed
// with the copy against without, 1,024 threads, clusters 1, 2, 4, 8: 800 rows a CTA of 3
// entries 0.83, 0.84, 0.72, 0.78, of 8 0.91, 0.88, 0.87, 0.97; 1,400 of 3 0.96, 0.90,
// 0.88, 1.07, of 8 1.02, 1.00, 1.10, 1.17; 3,000 of 2 0.95, 0.99, 0.93, 0.87, of 3 1.07,
// 1.04, 1.15, 1.12). With up to 512, rows of few entries pay later in clusters of 4 and
// more (512 threads: 800 rows of 3 1.06, 1.06, 0.86, 0.92, of 8 1.10, 1.05, 1.09, 1.10;
// 1,000 of 3 1.14, 1.14, 0.98, 0.99).
inline bool jagged_pays_alone(int64_t rows, int64_t nnz, int cluster, int threads) {
    if (!jagged_pays(rows, cluster)) return false;
    if (threads > 512)
        return rows >= 1400ll * cluster && nnz >= 8500ll * cluster && 2 * nnz >= 5 * rows;
    return cluster < 4 || rows >= 1000ll * cluster || nnz >= 6 * rows;
}

// The search direction p that its products gather lies whole in every CTA's shared
// memory; a CTA stores its rows into each. Random gathers from L2 run at 0.9 per clock and SM, those from
// shared memory at about 9, and they bound the solve.
// FP32 copy of a CTA's rows for the inner products of the mixed solve. The rows
// are renumbered by length (longest first, stable) and dealt to the warps in
// units: a long row (long_row) (its entries in order; the warp forms
// the products 128 at a time and every lane adds them in that order), or 32
// shorter rows, a lane each (entries step by step, those of the rows that have
// one next to each other, so nothing is padded). Either way a row's terms are
// added in storage order. The whole inner solve runs in this numbering. The
// warp tiles wait for a row pointer, a column and a value per 128
// entries and for the longest row of each 32: 66k cycles a product for 8,550
// rows, this 34k, bound by instruction issue (the copy costs 40k once). 24
// systems of 5k to 48k rows on clusters of 4 x 1,024: 11.5 -> 7.1 ms.
constexpr int kLenBuckets = 64;   // rows of 63 entries and more are one bucket
constexpr int kSliceCost = 4;     // a unit's own cost, in steps
// Rows taken by a whole warp. One lane needs a round trip to L2 per eight entries,
// a warp one per 128 but two instructions of every lane per entry: up to 128
// rows a warp the round trips count (5,016 rows on 4 CTAs: 17.4 us an iteration
// with long rows by lanes, 13.2 by warps), beyond that the instructions do
// (34,219 rows: 34k cycles a product with the longest rows alone by warps, 48k
// with all from 32 entries on).
__device__ __forceinline__ int long_row(int32_t rows, int warps) {
    return rows > 128 * warps ? kLenBuckets - 1 : 32;
}

struct Jagged {
    int32_t a, rows;      // first row of the CTA (in the renumbered system), rows
    int32_t *col;         // of the system
    float *val;
    float *diag, *ap;     // from here on by renumbered row of the system
    int32_t *perm, *inv;  // row of a number, number of a row
    int32_t *len, *start; // entries of a row; first entry of unit s at start[a + s]
    int32_t *next;        // the unit its warp takes after s (-1: none) at next[a + s]
    int32_t *first;       // shared memory: the first unit of each warp, then the
                          // number of long rows (units of one row, the first ones)

    __device__ static int bucket(int32_t n) {
        return kLenBuckets - 1 - (n < kLenBuckets ? n : kLenBuckets - 1);
    }

    // Row (from a on) of lane q in unit s; -1: none.
    __device__ int32_t row_of(int32_t s, int32_t longs, int q) const {
        if (s < longs) return q == 0 ? s : -1;
        const int32_t r = longs + 32 * (s - longs) + q;
        return r < rows ? r : -1;
    }

    // hist: [warps][kLenBuckets], tot: [kLenBuckets] in shared memory.
    __device__ __noinline__ void build(const int32_t *rp, const int32_t *scol, const double *sval,
                          const double *sdiag, int32_t *hist, int32_t *tot,
                          cg::cluster_group &cl) const {
        const int tid = threadIdx.x, nt = blockDim.x;
        const int lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
        const unsigned below = (1u << lane) - 1u;
        __syncthreads();
        for (int k = tid; k < nw * kLenBuckets; k += nt) hist[k] = 0;
        __syncthreads();
        const int32_t w0 = static_cast<int32_t>(static_cast<int64_t>(rows) * wid / nw);
        const int32_t w1 = static_cast<int32_t>(static_cast<int64_t>(rows) * (wid + 1) / nw);
        int32_t *mine = hist + wid * kLenBuckets;
        for (int32_t l = w0 + lane; l < w1; l += 32)
            atomicAdd(mine + bucket(rp[a + l + 1] - rp[a + l]), 1);
        __syncthreads();
        for (int k = tid; k < kLenBuckets; k += nt) {
            int32_t t = 0;
            for (int w = 0; w < nw; ++w) t += hist[w * kLenBuckets + k];
            tot[k] = t;
        }
        __syncthreads();
        if (wid == 0) {
            constexpr int kPer = kLenBuckets / 32;
            int32_t sum = 0;
            for (int q = 0; q < kPer; ++q) sum += tot[lane * kPer + q];
            int32_t incl = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            int32_t run = incl - sum;
            for (int q = 0; q < kPer; ++q) {
                const int32_t t = tot[lane * kPer + q];
                tot[lane * kPer + q] = run;
                run += t;
            }
            __syncwarp();
            if (lane == 0) first[32] = tot[bucket(long_row(rows, nw)) + 1];
        }
        __syncthreads();
        for (int k = tid; k < kLenBuckets; k += nt) {
            int32_t run = tot[k];
            for (int w = 0; w < nw; ++w) {
                const int32_t t = hist[w * kLenBuckets + k];
                hist[w * kLenBuckets + k] = run;
                run += t;
            }
        }
        __syncthreads();
        for (int32_t l0 = w0; l0 < w1; l0 += 32) {
            const int32_t l = l0 + lane;
            const bool in = l < w1;
            const int32_t n = in ? rp[a + l + 1] - rp[a + l] : 0;
            const int bk = in ? bucket(n) : -1;
            const unsigned same = __match_any_sync(0xffffffffu, bk);
            const int rank = __popc(same & below);
            const int32_t to = in ? a + mine[bk] + rank : 0;
            __syncwarp();
            if (in && rank == 0) mine[bk] += __popc(same);
            __syncwarp();
            if (in) {
                perm[to] = a + l;
                inv[a + l] = to;
                len[to] = n;
                diag[to] = static_cast<float>(sdiag[a + l]);
            }
        }
        __syncthreads();
        const int32_t longs = first[32], slices = longs + (rows - longs + 31) / 32;
        for (int32_t s = wid; s < slices; s += nw) {
            const int32_t r = row_of(s, longs, lane);
            const int32_t n = r >= 0 ? len[a + r] : 0;
            const int32_t t = __reduce_add_sync(0xffffffffu, n);
            if (lane == 0) start[a + s] = t;
        }
        __syncthreads();
        if (wid == 0) {
            int32_t run = rows > 0 ? rp[a] : 0;
            for (int32_t s0 = 0; s0 < slices; s0 += 32) {
                const int32_t t = s0 + lane < slices ? start[a + s0 + lane] : 0;
                int32_t incl = t;
                for (int o = 1; o < 32; o <<= 1) {
                    const int32_t u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
                if (s0 + lane < slices) start[a + s0 + lane] = run + incl - t;
                run += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
        // slices, longest first, to the warp with least to do (lane w: warp w)
        if (wid == nw - 1) {
            uint32_t load = 0;
            int32_t last = -1;
            if (lane < nw) first[lane] = -1;
            for (int32_t s0 = 0; s0 < slices; s0 += 32) {
                const int32_t u = s0 + lane;
                const int32_t longest = u >= slices ? 0
                                        : u < longs ? len[a + u] / 4
                                                    : len[a + row_of(u, longs, 0)];
                const int32_t here = slices - s0 < 32 ? slices - s0 : 32;
                for (int32_t q = 0; q < here; ++q) {
                    const uint32_t cost = __shfl_sync(0xffffffffu, longest, q) + kSliceCost;
                    // (loads stay below 2^26 steps: 2^31 entries of 32 a step)
                    const uint32_t least =
                        __reduce_min_sync(0xffffffffu, lane < nw ? load << 5 | lane : ~0u);
                    if (lane == (least & 31u)) {
                        if (last < 0) first[lane] = s0 + q;
                        else next[a + last] = s0 + q;
                        last = s0 + q;
                        load += cost;
                    }
                }
            }
            if (last >= 0) next[a + last] = -1;
        }
        cl.sync();  // every CTA's inv
        for (int32_t s = wid; s < slices; s += nw) {
            if (s < longs) {
                const int32_t n = len[a + s], e = rp[perm[a + s]], at = start[a + s];
                for (int32_t j = lane; j < n; j += 32) {
                    col[at + j] = __ldcg(inv + scol[e + j]);
                    val[at + j] = static_cast<float>(sval[e + j]);
                }
                continue;
            }
            const int32_t r = row_of(s, longs, lane);
            const int32_t n = r >= 0 ? len[a + r] : 0, e = r >= 0 ? rp[perm[a + r]] : 0;
            const int32_t most = __reduce_max_sync(0xffffffffu, n);
            int32_t at = start[a + s];
#pragma unroll 4
            for (int32_t j = 0; j < most; ++j) {
                const unsigned m = __ballot_sync(0xffffffffu, j < n);
                if (j < n) {
                    const int32_t to = at + __popc(m & below);
                    col[to] = __ldcg(inv + scol[e + j]);
                    val[to] = static_cast<float>(sval[e + j]);
                }
                at += __popc(m);
            }
        }
        __syncthreads();
    }

    // ap = A p for the CTA's rows; returns the thread's part of p^T A p. p is in
    // shared memory. A lane's entries are loaded kDeep at a
    // time, one group ahead, across slices: L2's latency is what there is to
    // hide. Not inlined: it needs the registers to itself.
    __device__ __noinline__ double product() const {
        extern __shared__ __align__(16) double near_mem[];
        const float *near_p = reinterpret_cast<const float *>(near_mem);
        auto gather = [&](int32_t k) { return near_p[k]; };
        double w = 0.0;
        constexpr int kDeep = 8;
        const int lane = threadIdx.x & 31;
        const unsigned below = (1u << lane) - 1u;
        int32_t c[kDeep];
        float v[kDeep];
        const int32_t longs = first[32];
        auto head = [&](int32_t s, int32_t &n, int32_t &at, int32_t &after) {
            const int32_t r = s >= 0 ? row_of(s, longs, lane) : -1;
            n = r >= 0 ? len[a + r] : 0;
            at = s >= 0 ? start[a + s] : 0;
            after = s >= 0 ? next[a + s] : -1;
        };
        // entries j, j + 1, ... of slice rows of n entries each from `at` on, or
        // of rows of one length (even): then step j lies at at + 32 j
        auto load = [&](int32_t j, int32_t n, int32_t &at, bool even) {
            if (even) {
                const int32_t *ce = col + at + 32 * j + lane;
                const float *ve = val + at + 32 * j + lane;
#pragma unroll
                for (int k = 0; k < kDeep; ++k) {
                    c[k] = j + k < n ? __ldcg(ce + 32 * k) : -1;
                    v[k] = j + k < n ? __ldcg(ve + 32 * k) : 0.0f;
                }
                return;
            }
#pragma unroll
            for (int k = 0; k < kDeep; ++k) {
                const bool has = j + k < n;
                const unsigned m = __ballot_sync(0xffffffffu, has);
                const int32_t e = at + __popc(m & below);
                c[k] = has ? __ldcg(col + e) : -1;
                v[k] = has ? __ldcg(val + e) : 0.0f;
                at += __popc(m);
            }
        };
        auto same = [&](int32_t n) {
            return __reduce_max_sync(0xffffffffu, n) == __reduce_min_sync(0xffffffffu, n);
        };
        int32_t s = first[threadIdx.x >> 5], n, at, after;
        head(s, n, at, after);
        while (s >= 0 && s < longs) {  // a warp's long rows come first
            const int32_t many = __shfl_sync(0xffffffffu, n, 0);
            const float p = gather(a + s);
            float sum = diag[a + s] * p;
            for (int32_t j = 0; j < many; j += 128) {
                float t[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int32_t e = j + 32 * k + lane;
                    c[k] = e < many ? __ldcg(col + at + e) : -1;
                    t[k] = e < many ? __ldcg(val + at + e) : 0.0f;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (c[k] >= 0) t[k] = t[k] * gather(c[k]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int32_t here = min(32, many - j - 32 * k);
                    for (int32_t q = 0; q < here; ++q) sum += __shfl_sync(0xffffffffu, t[k], q);
                }
            }
            if (lane == 0) {
                ap[a + s] = sum;
                w += static_cast<double>(p) * sum;
            }
            s = after;
            head(s, n, at, after);
        }
        bool even = same(n);
        load(0, n, at, even);
        while (s >= 0) {
            int32_t next_n, next_at, next_after;
            head(after, next_n, next_at, next_after);
            const int32_t r = row_of(s, longs, lane), i = a + r;
            const bool on = r >= 0;
            const int32_t most = __reduce_max_sync(0xffffffffu, n);
            const float p = on ? gather(i) : 0.0f;
            float sum = on ? diag[i] * p : 0.0f;
            for (int32_t j = 0; j < most; j += kDeep) {
#pragma unroll
                for (int k = 0; k < kDeep; ++k)
                    if (c[k] >= 0) sum += v[k] * gather(c[k]);
                if (j + kDeep < most) {
                    load(j + kDeep, n, at, even);
                } else {
                    even = same(next_n);
                    load(0, next_n, next_at, even);
                }
            }
            if (on) {
                ap[i] = sum;
                w += static_cast<double>(p) * sum;
            }
            s = after;
            n = next_n;
            at = next_at;
            after = next_after;
        }
        return w;
    }
};

// kNear: the mixed solve where some system's p is kept in shared memory; apart from
// kTiles, whose registers it does not fit (52,000 rows, 4 x 512: 22.4 ms, with the
// code for both 23.1). kTilesWide: kTiles for clusters beyond kPortable.
enum Solve { kFp64 = 0, kTiles = 1, kTilesWide = 2, kNear = 3 };

template <int Kind>
__global__ void __launch_bounds__(1024) k_batch_pcg(BatchArgs A) {
    constexpr bool kByWarp = Kind != kTiles;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) double near_mem[];
    __shared__ double scratch[33 * 4];
    __shared__ double part[2 * 4];
    __shared__ __align__(16) double tilebuf[32 * kTileChunk];  // warp tiles, <= 32 warps
    __shared__ int32_t wb[32 + 1];
    __shared__ int32_t first_slice[33];
    __shared__ Jagged J;
    __shared__ float *peers[16];  // p of every CTA of the cluster
    __shared__ int s_job;
    __shared__ int s_stop;
    int buf = 0;
    const unsigned rank = cl.block_rank();
    const unsigned nb = cl.num_blocks();
    const uint64_t deadline = global_timer_ns() + A.total_timeout_ns;
    cl.sync();  // every CTA of the cluster is running before DSMEM is touched

    for (;;) {
        if (rank == 0 && threadIdx.x == 0) {
            s_job = static_cast<int>(atomicAdd(A.queue, 1u));
            s_stop = global_timer_ns() > deadline ? 1 : 0;
        }
        cl.sync();
        const int job = *cl.map_shared_rank(&s_job, 0);
        const bool late = *cl.map_shared_rank(&s_stop, 0) != 0;
        if (job >= A.num_sys) break;
        const int sid = A.order[job];
        const SysDesc S = A.sys[sid];
        const uint64_t t0 = global_timer_ns();
        const int32_t n = S.n;
        // the CTA's rows (from a multiple of four on: p is stored by fours)
        auto split = [&](unsigned q) {
            return q == nb ? n : static_cast<int32_t>(static_cast<int64_t>(n) * q / nb) & ~3;
        };
        const int32_t a = split(rank), b = split(rank + 1);
        const int32_t *rp = A.rp + S.row_base + sid;
        const int32_t *col = A.col + S.nnz_base;
        const double *val = A.val + S.nnz_base;
        const double *dg = A.diag + S.row_base;
        const double *rhs = A.rhs + S.row_base;
        double *x = A.x + S.row_base;
        double *r = A.r + S.row_base;

        // per-warp row ranges of the warp tiles, balanced by nonzeros
        warp_row_bounds(b - a, wb, [&](int32_t l) {
            return int64_t(__ldg(rp + a + l)) - __ldg(rp + a) + int64_t(kRowCost) * l;
        });

        ktg_batch_result res;
        res.iters = 0;
        res.outer = 0;
        res.status = late ? KTG_ERR_TIMEOUT : KTG_OK;
        double resid = 0.0;

        if constexpr (Kind == kFp64) {
            double *z = A.z + S.row_base;
            double *p = A.p + S.row_base;
            double *ap = A.ap + S.row_base;
            double v[3] = {0.0, 0.0, 0.0};  // bb, rz, rr
            for (int32_t i = a + threadIdx.x; i < b; i += blockDim.x) {
                const double s = row_dot<double, double>(rp, col, val, x, i, dg[i] * x[i]);
                const double bi = rhs[i];
                const double ri = bi - s;
                const double zi = ri / dg[i];
                r[i] = ri;
                z[i] = zi;
                __stcg(p + i, zi);
                v[0] += bi * bi;
                v[1] += ri * zi;
                v[2] += ri * ri;
            }
            cluster_sum<3, kByWarp>(v, part, buf, scratch, cl);
            const double bnorm = sqrt(v[0]);
            bool active = bnorm > 0.0 && !late;
            double rho = v[1];
            resid = bnorm > 0.0 ? sqrt(v[2]) / bnorm : 0.0;
            int64_t it = 0;
            for (;;) {
                if (!(active && resid > A.tol && it < A.max_iter)) break;
                if (rank == 0 && threadIdx.x == 0) s_stop = global_timer_ns() > deadline ? 1 : 0;
                double w[1] = {0.0};
                double pcur = 0.0;
                warp_tile_spmv<double, true>(
                    a, INT32_MAX, b - a, kAllAxes, wb, tilebuf,
                    [&](int, const int32_t *&trp, const int32_t *&tcol, const double *&tval,
                        const double *&tin) {
                        trp = rp;
                        tcol = col;
                        tval = val;
                        tin = p;
                    },
                    [&](int32_t, int, int32_t i) {
                        pcur = __ldcg(p + i);
                        return dg[i] * pcur;
                    },
                    [&](int32_t, int, int32_t i, double s) {
                        ap[i] = s;
                        w[0] += pcur * s;
                    });
                cluster_sum<1, kByWarp>(w, part, buf, scratch, cl);
                if (*cl.map_shared_rank(&s_stop, 0)) {
                    res.status = KTG_ERR_TIMEOUT;
                    break;
                }
                const bool ok = w[0] > 0.0;
                const double alpha = ok ? rho / w[0] : 0.0;
                double u[2] = {0.0, 0.0};  // rr, rz
                if (ok) {
                    for (int32_t i = a + threadIdx.x; i < b; i += blockDim.x) {
                        x[i] += alpha * __ldcg(p + i);
                        const double ri = r[i] - alpha * ap[i];
                        const double zi = ri / dg[i];
                        r[i] = ri;
                        z[i] = zi;
                        u[0] += ri * ri;
                        u[1] += ri * zi;
                    }
                }
                cluster_sum<2, kByWarp>(u, part, buf, scratch, cl);
                ++it;
                if (!ok) {
                    active = false;
                    continue;
                }
                resid = sqrt(u[0]) / bnorm;
                if (!(u[1] > 0.0)) {
                    active = false;
                    continue;
                }
                const double beta = u[1] / rho;
                rho = u[1];
                for (int32_t i = a + threadIdx.x; i < b; i += blockDim.x)
                    __stcg(p + i, z[i] + beta * __ldcg(p + i));
                cl.sync();
            }
            res.iters = it;
        } else {
            // r = b - A x for the CTA's rows
            auto residual = [&](auto emit) {
                warp_tile_spmv<double, true>(
                    a, INT32_MAX, b - a, kAllAxes, wb, tilebuf,
                    [&](int, const int32_t *&trp, const int32_t *&tcol, const double *&tval,
                        const double *&tin) {
                        trp = rp;
                        tcol = col;
                        tval = val;
                        tin = x;
                    },
                    [&](int32_t, int, int32_t i) { return dg[i] * __ldcg(x + i); },
                    [&](int32_t, int, int32_t i, double s) { emit(i, rhs[i], rhs[i] - s); });
            };
            int64_t inner = 0;
            int32_t outer = 0;
            // A copy of the solve for each place of p, so that neither has the
            // other's pointers in registers.
            auto solve = [&](auto place) {
                constexpr bool Near = decltype(place)::value;
                float *d = A.d32 + S.row_base;
                float *ri = A.ri32 + S.row_base;
                float *z = A.z32 + S.row_base;
                float *p = A.p32 + S.row_base;
                float *ap = A.ap32 + S.row_base;
                const float *val32 = A.val32 + S.nnz_base;
                float *const near_p = reinterpret_cast<float *>(near_mem);
                if constexpr (Near) {
                    if (threadIdx.x == 0)
                        J = Jagged{a, b - a, A.jcol + S.nnz_base, A.jval + S.nnz_base,
                                   A.diag32 + S.row_base, ap, A.perm + S.row_base,
                                   A.inv + S.row_base, A.len + S.row_base, A.start + S.row_base,
                                   A.next + S.row_base, first_slice};
                    if (threadIdx.x < nb)
                        peers[threadIdx.x] = cl.map_shared_rank(near_p, threadIdx.x);
                    __syncthreads();
                }
                auto put = [&](int32_t i, float t) {
                    if constexpr (Near)
                        for (unsigned q = 0; q < nb; ++q) peers[q][i] = t;
                    else
                        __stcg(p + i, t);
                };
                auto own = [&](int32_t i) {
                    if constexpr (Near) return near_p[i];
                    else return __ldcg(p + i);
                };
                auto row = [&](int32_t i) {
                    if constexpr (Near) return J.perm[i];
                    else return i;
                };
                auto diagonal = [&](int32_t i) {
                    if constexpr (Near) return J.diag[i];
                    else return static_cast<float>(dg[i]);
                };
                double bnorm = 0.0, prev = 0.0;
                for (int round = 0;; ++round) {
                    double v[2] = {0.0, 0.0};  // rr, bb
                    residual([&](int32_t i, double bi, double rr) {
                        r[i] = rr;
                        v[0] += rr * rr;
                        v[1] += bi * bi;
                    });
                    cluster_sum<2, kByWarp>(v, part, buf, scratch, cl);
                    if (round == 0) bnorm = sqrt(v[1]);
                    const double rnorm = sqrt(v[0]);
                    prev = resid;
                    resid = bnorm > 0.0 ? rnorm / bnorm : 0.0;
                    const bool stalled = round > 0 && !(resid < 0.5 * prev);
                    if (!(bnorm > 0.0) || late || resid <= A.tol || outer >= A.max_outer ||
                        inner >= A.max_iter || stalled) {
                        // stalled: caller may retry in FP64
                        if (stalled && resid > A.tol) res.status = 1;
                        break;
                    }
                    if constexpr (Near)
                        if (round == 0)
                            J.build(rp, col, val, dg, reinterpret_cast<int32_t *>(tilebuf),
                                    reinterpret_cast<int32_t *>(scratch), cl);
                    double q[2] = {0.0, 0.0};  // rz, rr (inner)
                    for (int32_t i = a + threadIdx.x; i < b; i += blockDim.x) {
                        const float rf = static_cast<float>(r[row(i)]);
                        const float zf = rf / diagonal(i);
                        ri[i] = rf;
                        d[i] = 0.0f;
                        z[i] = zf;
                        put(i, zf);
                        q[0] += static_cast<double>(rf) * zf;
                        q[1] += static_cast<double>(rf) * rf;
                    }
                    cluster_sum<2, kByWarp>(q, part, buf, scratch, cl);
                    double rho = q[0];
                    double iresid = sqrt(q[1]);
                    const double target = A.inner_tol * rnorm;
                    bool live = rho > 0.0;
                    while (live && iresid > target && inner < A.max_iter) {
                        double w[1] = {0.0};
                        if constexpr (Near) {
                            w[0] = J.product();
                        } else {
                            float pcur = 0.0f;
                            warp_tile_spmv<float>(
                                a, INT32_MAX, b - a, kAllAxes, wb,
                                reinterpret_cast<float *>(tilebuf),
                                [&](int, const int32_t *&trp, const int32_t *&tcol,
                                    const float *&tval, const float *&tin) {
                                    trp = rp;
                                    tcol = col;
                                    tval = val32;
                                    tin = p;
                                },
                                [&](int32_t, int, int32_t i) {
                                    pcur = __ldcg(p + i);
                                    return diagonal(i) * pcur;
                                },
                                [&](int32_t, int, int32_t i, float s) {
                                    ap[i] = s;
                                    w[0] += static_cast<double>(pcur) * s;
                                });
                        }
                        cluster_sum<1, kByWarp>(w, part, buf, scratch, cl);
                        ++inner;
                        if (!(w[0] > 0.0)) break;
                        const float alpha = static_cast<float>(rho / w[0]);
                        double u[2] = {0.0, 0.0};
                        each_rows(a, b, [&](int32_t i0, auto count) {
                            float xv[kBatchRows], rv[kBatchRows], av[kBatchRows], dv[kBatchRows];
#pragma unroll
                            for (int k = 0; k < count(); ++k) {
                                const int32_t i = i0 + k * blockDim.x;
                                xv[k] = d[i];
                                rv[k] = ri[i];
                                av[k] = ap[i];
                                dv[k] = diagonal(i);
                            }
#pragma unroll
                            for (int k = 0; k < count(); ++k) {
                                const int32_t i = i0 + k * blockDim.x;
                                d[i] = xv[k] + alpha * own(i);
                                const float rr = rv[k] - alpha * av[k];
                                const float zz = rr / dv[k];
                                ri[i] = rr;
                                z[i] = zz;
                                u[0] += static_cast<double>(rr) * rr;
                                u[1] += static_cast<double>(rr) * zz;
                            }
                        });
                        cluster_sum<2, kByWarp>(u, part, buf, scratch, cl);
                        iresid = sqrt(u[0]);
                        if (!(u[1] > 0.0)) break;
                        const float beta = static_cast<float>(u[1] / rho);
                        rho = u[1];
                        int32_t first = a;
                        if constexpr (Near) {
                            first = a + (b - a) / 4 * 4;
                            for (int32_t i = a + 4 * static_cast<int32_t>(threadIdx.x); i < first;
                                 i += 4 * blockDim.x) {
                                float4 t = *reinterpret_cast<const float4 *>(near_p + i);
                                t.x = z[i] + beta * t.x;
                                t.y = z[i + 1] + beta * t.y;
                                t.z = z[i + 2] + beta * t.z;
                                t.w = z[i + 3] + beta * t.w;
                                for (unsigned q = 0; q < nb; ++q)
                                    *reinterpret_cast<float4 *>(peers[q] + i) = t;
                            }
                        }
                        for (int32_t i = first + static_cast<int32_t>(threadIdx.x); i < b;
                             i += blockDim.x)
                            put(i, z[i] + beta * own(i));
                        cl.sync();
                    }
                    for (int32_t i = a + threadIdx.x; i < b; i += blockDim.x) x[row(i)] += d[i];
                    ++outer;
                    cl.sync();
                }
            };
            if constexpr (Kind == kNear) {
                if (jagged_pays(n, static_cast<int>(nb))) solve(std::true_type());
                else solve(std::false_type());
            } else {
                solve(std::false_type());
            }
            res.iters = inner;
            res.outer = outer;
        }
        if (rank == 0 && threadIdx.x == 0) {
            res.resid = resid;
            res.latency_ns = static_cast<int64_t>(global_timer_ns() - t0);
            A.results[sid] = res;
        }
        cl.sync();  // the job word may be rewritten only after every CTA read it
    }
    cl.sync();  // no CTA leaves while another may still read its shared memory
}

}  // namespace
}  // namespace ktg

struct ktg_batch {
    int device = 0;
    int num_sms = 0;
    int near_limit = 0;         // dynamic shared memory a CTA of the mixed solve can have
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    std::string err;
    int64_t launches = 0;       // kernels launched by solves (graph replays included)
    int graph_kernels = 0;      // kernels in the captured graph
    // host mirror of the descriptors
    std::vector<ktg::SysDesc> sys;
    std::vector<int64_t> cost;
    int64_t rows = 0, nnz = 0;     // used
    int64_t cap_rows = 0, cap_nnz = 0, cap_sys = 0, cap_rp = 0;
    // device arrays
    ktg::SysDesc *d_sys = nullptr;
    int32_t *d_order = nullptr;
    int32_t *rp = nullptr;  // rows + num_sys entries
    int32_t *col = nullptr;
    double *val = nullptr;
    float *val32 = nullptr;   // values for the mixed solve on the CSR system
    // the mixed solve's copies, built by it: one allocation for so many rows, entries
    char *jagged = nullptr;
    int64_t jagged_rows = 0, jagged_nnz = 0;
    int32_t *jcol = nullptr;
    float *jval = nullptr, *diag32 = nullptr;
    int32_t *perm = nullptr, *inv = nullptr, *len = nullptr, *start = nullptr,
            *next = nullptr;
    double *diag = nullptr, *rhs = nullptr, *x = nullptr, *x0 = nullptr;
    double *r = nullptr, *z = nullptr, *p = nullptr, *ap = nullptr;
    float *d32 = nullptr, *ri32 = nullptr, *z32 = nullptr, *p32 = nullptr, *ap32 = nullptr;
    unsigned *queue = nullptr;
    ktg_batch_result *results = nullptr;
    bool dirty = true;  // descriptors / order need upload
    // launch shape
    int cluster = 8;
    int threads = 512;
    // size classes: systems of at least split_rows rows (0: none) are solved
    // by a second, concurrent launch of split_clusters clusters of
    // split_cluster CTAs of split_threads threads, with their own queue
    int64_t split_rows = 0;
    int split_cluster = 16, split_threads = 1024, split_clusters = 1;
    int num_large = 0;           // systems in the large class (first in d_order)
    unsigned *queue2 = nullptr;  // the large class's work queue
    int64_t order_split_rows = -1;  // split the uploaded order was built for
    int num_queued = 0;             // systems the cluster launches take (in d_order)
    // whole-GPU path: pairs of consecutive systems of equal size >=
    // offload_rows (the x and y systems of one netlist) are solved one pair
    // after another by an internal context (aggregation-preconditioned mixed
    // solve, or the FP64 solve), before the cluster launches take the rest
    int64_t offload_rows = 0;
    int offload_precond = 2, offload_coarse = 0;
    int64_t order_offload_rows = -1;
    std::vector<int32_t> off_first;  // first system of each offloaded pair
    ktg_ctx *octx = nullptr;
    int64_t octx_launches = 0;
    ktg_mixed_info *d_minfo = nullptr;
    ktg_solve_info *d_sinfo = nullptr;
    unsigned long long *d_stamp = nullptr;
    // graph cache
    cudaGraphExec_t graph = nullptr;
    double g_tol = -1, g_inner = -1;
    int64_t g_max_iter = -1;
    int g_mixed = -1, g_cluster = -1, g_threads = -1;
    int64_t g_split_rows = -1;
    int g_split_cluster = -1, g_split_threads = -1, g_split_clusters = -1;
};

namespace {

int berr(ktg_batch *b, int code, const std::string &m) {
    if (b) b->err = m;
    return code;
}

#define KTG_BCUDA(b, call)                                                          \
    do {                                                                            \
        cudaError_t e_ = (call);                                                    \
        if (e_ != cudaSuccess)                                                      \
            return berr((b), KTG_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

template <typename T>
int grow(ktg_batch *b, T **ptr, int64_t used, int64_t cap) {
    T *np = nullptr;
    KTG_BCUDA(b, cudaMalloc(reinterpret_cast<void **>(&np), sizeof(T) * std::max<int64_t>(cap, 1)));
    if (*ptr && used > 0)
        KTG_BCUDA(b, cudaMemcpyAsync(np, *ptr, sizeof(T) * used, cudaMemcpyDeviceToDevice, b->stream));
    KTG_BCUDA(b, cudaStreamSynchronize(b->stream));
    if (*ptr) cudaFree(*ptr);
    *ptr = np;
    return KTG_OK;
}

// Room for `rows` vector rows, `nnz` entries and `nsys` systems in total.
int reserve(ktg_batch *b, int64_t rows, int64_t nnz, int64_t nsys) {
    int rc;
    if (rows > b->cap_rows) {
        const int64_t cap = std::max(rows, 2 * b->cap_rows);
        const int64_t used = b->rows;
        if ((rc = grow(b, &b->diag, used, cap)) || (rc = grow(b, &b->rhs, used, cap)) ||
            (rc = grow(b, &b->x, used, cap)) || (rc = grow(b, &b->x0, used, cap)) ||
            (rc = grow(b, &b->r, 0, cap)) || (rc = grow(b, &b->z, 0, cap)) ||
            (rc = grow(b, &b->p, 0, cap)) || (rc = grow(b, &b->ap, 0, cap)) ||
            (rc = grow(b, &b->d32, 0, cap)) || (rc = grow(b, &b->ri32, 0, cap)) ||
            (rc = grow(b, &b->z32, 0, cap)) || (rc = grow(b, &b->p32, 0, cap)) ||
            (rc = grow(b, &b->ap32, 0, cap)))
            return rc;
        b->cap_rows = cap;
    }
    if (rows + nsys > b->cap_rp) {
        const int64_t cap = std::max(rows + nsys, 2 * b->cap_rp);
        if ((rc = grow(b, &b->rp, b->rows + static_cast<int64_t>(b->sys.size()), cap))) return rc;
        b->cap_rp = cap;
    }
    if (nsys > b->cap_sys) {
        const int64_t cap = std::max<int64_t>(nsys, 2 * b->cap_sys);
        if ((rc = grow(b, &b->d_sys, 0, cap)) || (rc = grow(b, &b->d_order, 0, cap)) ||
            (rc = grow(b, &b->results, static_cast<int64_t>(b->sys.size()), cap)))
            return rc;
        b->cap_sys = cap;
    }
    if (nnz > b->cap_nnz) {
        const int64_t cap = std::max(nnz, 2 * b->cap_nnz);
        if ((rc = grow(b, &b->col, b->nnz, cap)) || (rc = grow(b, &b->val, b->nnz, cap)) ||
            (rc = grow(b, &b->val32, b->nnz, cap)))
            return rc;
        b->cap_nnz = cap;
    }
    return KTG_OK;
}

// The arrays of the renumbered copies, in one allocation when a mixed solve first
// wants them (grown with every system that was added they took a fifth of the time
// of adding 24).
int reserve_jagged(ktg_batch *b) {
    if (b->cap_rows <= b->jagged_rows && b->cap_nnz <= b->jagged_nnz) return KTG_OK;
    if (b->jagged) cudaFree(b->jagged);
    b->jagged = nullptr;
    b->jagged_rows = b->jagged_nnz = 0;
    const int64_t per_row = (b->cap_rows * 4 + 255) / 256 * 256;
    const int64_t per_entry = (b->cap_nnz * 4 + 255) / 256 * 256;
    KTG_BCUDA(b, cudaMalloc(&b->jagged, 6 * per_row + 2 * per_entry + 256));
    char *at = b->jagged;
    auto take = [&](auto **p, int64_t bytes) {
        *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(at);
        at += bytes;
    };
    take(&b->jcol, per_entry);
    take(&b->jval, per_entry);
    take(&b->diag32, per_row);
    take(&b->perm, per_row);
    take(&b->inv, per_row);
    take(&b->len, per_row);
    take(&b->start, per_row);
    take(&b->next, per_row);
    b->jagged_rows = b->cap_rows;
    b->jagged_nnz = b->cap_nnz;
    return KTG_OK;
}

__global__ void k_batch_f32(const double *a, float *b, int64_t n) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        b[i] = static_cast<float>(a[i]);
}

__global__ void k_stamp(unsigned long long *t) { *t = ktg::global_timer_ns(); }

// Results of an offloaded pair (systems sx, sy) from its solve's info: the
// mixed solve's inner iterations, rounds and final true residuals (the FP64
// pass's when it ran), or the FP64 solve's iterations and residuals; status
// the solve's error, else 0 when the residual meets tol and 1 when not.
__global__ void k_offload_results(const ktg_mixed_info *mi, const ktg_solve_info *si, int mixed,
                                  double tol, int32_t sx, int32_t sy,
                                  const unsigned long long *t0, ktg_batch_result *res) {
    const int64_t lat = static_cast<int64_t>(ktg::global_timer_ns() - *t0);
    for (int a = 0; a < 2; ++a) {
        ktg_batch_result r;
        if (mixed) {
            r.iters = a ? mi->inner_y : mi->inner_x;
            r.outer = a ? mi->outer_y : mi->outer_x;
            r.resid = a ? mi->resid_y : mi->resid_x;
            r.status = mi->status != 0 ? mi->status : (r.resid <= tol ? 0 : 1);
        } else {
            r.iters = a ? si->iters_y : si->iters_x;
            r.outer = 0;
            r.resid = a ? si->resid_y : si->resid_x;
            r.status = si->status != 0 ? si->status : (r.resid <= tol ? 0 : 1);
        }
        r.latency_ns = lat;
        res[a ? sy : sx] = r;
    }
}

}  // namespace

// Systems that leave the queues for the whole GPU at the current offload
// threshold: consecutive systems of equal size (an x/y pair) of at least
// offload_rows rows, paired from the front.
static std::vector<char> offloaded(const ktg_batch *b, std::vector<int32_t> *first = nullptr) {
    const int32_t ns = static_cast<int32_t>(b->sys.size());
    std::vector<char> off(ns, 0);
    if (first) first->clear();
    if (b->offload_rows > 0) {
        for (int32_t k = 0; k + 1 < ns;) {
            if (b->sys[k].n >= b->offload_rows && b->sys[k + 1].n == b->sys[k].n) {
                if (first) first->push_back(k);
                off[k] = off[k + 1] = 1;
                k += 2;
            } else {
                ++k;
            }
        }
    }
    return off;
}

extern "C" {

int ktg_batch_create(int device, ktg_batch **out) {
    if (!out) return KTG_ERR_ARG;
    *out = nullptr;
    ktg_batch *b = new (std::nothrow) ktg_batch();
    if (!b) return KTG_ERR_NOMEM;
    b->device = device;
    if (cudaSetDevice(device) != cudaSuccess ||
        cudaDeviceGetAttribute(&b->num_sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaStreamCreateWithFlags(&b->own_stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc(&b->queue, sizeof(unsigned)) != cudaSuccess ||
        cudaMalloc(&b->queue2, sizeof(unsigned)) != cudaSuccess) {
        ktg_batch_destroy(b);
        return KTG_ERR_CUDA;
    }
    b->stream = b->own_stream;
    *out = b;
    return KTG_OK;
}

void ktg_batch_destroy(ktg_batch *b) {
    if (!b) return;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    if (b->graph) cudaGraphExecDestroy(b->graph);
    void *ptrs[] = {b->d_sys, b->d_order, b->rp, b->col, b->val, b->val32, b->jagged,
                    b->diag, b->rhs, b->x, b->x0, b->r, b->z, b->p, b->ap, b->d32, b->ri32, b->z32,
                    b->p32, b->ap32, b->queue, b->queue2, b->results, b->d_minfo, b->d_sinfo,
                    b->d_stamp};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (b->octx) ktg_destroy(b->octx);
    if (b->own_stream) cudaStreamDestroy(b->own_stream);
    delete b;
}

const char *ktg_batch_last_error(const ktg_batch *b) { return b ? b->err.c_str() : "null batch"; }

int ktg_batch_set_stream(ktg_batch *b, void *stream) {
    if (!b) return KTG_ERR_ARG;
    b->stream = stream ? static_cast<cudaStream_t>(stream) : b->own_stream;
    return KTG_OK;
}

int64_t ktg_batch_size(const ktg_batch *b) { return b ? static_cast<int64_t>(b->sys.size()) : 0; }

int ktg_batch_add_system(ktg_batch *b, int64_t n, const int64_t *row_ptr, const int32_t *col,
                         const double *val, const double *diag, const double *rhs,
                         const double *x0, int64_t *id) {
    if (!b || n < 0 || !row_ptr || (n > 0 && (!diag || !rhs || !x0))) return KTG_ERR_ARG;
    const int64_t m = row_ptr[n];
    if (m < 0 || (m > 0 && (!col || !val))) return KTG_ERR_ARG;
    if (n > 0x3fffffffll || m > 0x7fffffffll || b->rows + n > 0x7fffffffll ||
        b->nnz + m > 0x7fffffffll)
        return berr(b, KTG_ERR_RANGE, "batch exceeds 32-bit indices");
    std::vector<int32_t> rp(n + 1);
    for (int64_t i = 0; i <= n; ++i) {
        if (row_ptr[i] < 0 || (i > 0 && row_ptr[i] < row_ptr[i - 1]))
            return berr(b, KTG_ERR_ARG, "row_ptr not monotone");
        rp[i] = static_cast<int32_t>(row_ptr[i]);
    }
    for (int64_t e = 0; e < m; ++e)
        if (col[e] < 0 || col[e] >= n) return berr(b, KTG_ERR_ARG, "col out of range");
    if (cudaSetDevice(b->device) != cudaSuccess) return KTG_ERR_CUDA;
    const int64_t nsys = static_cast<int64_t>(b->sys.size()) + 1;
    int rc = reserve(b, b->rows + n, b->nnz + m, nsys);
    if (rc) return rc;
    const int64_t base = b->rows, ebase = b->nnz, k = nsys - 1;
    KTG_BCUDA(b, cudaMemcpyAsync(b->rp + base + k, rp.data(), sizeof(int32_t) * (n + 1),
                                 cudaMemcpyHostToDevice, b->stream));
    if (m) {
        KTG_BCUDA(b, cudaMemcpyAsync(b->col + ebase, col, sizeof(int32_t) * m, cudaMemcpyHostToDevice, b->stream));
        KTG_BCUDA(b, cudaMemcpyAsync(b->val + ebase, val, sizeof(double) * m, cudaMemcpyHostToDevice, b->stream));
    }
    if (n) {
        KTG_BCUDA(b, cudaMemcpyAsync(b->diag + base, diag, sizeof(double) * n, cudaMemcpyHostToDevice, b->stream));
        KTG_BCUDA(b, cudaMemcpyAsync(b->rhs + base, rhs, sizeof(double) * n, cudaMemcpyHostToDevice, b->stream));
        KTG_BCUDA(b, cudaMemcpyAsync(b->x + base, x0, sizeof(double) * n, cudaMemcpyHostToDevice, b->stream));
        KTG_BCUDA(b, cudaMemcpyAsync(b->x0 + base, x0, sizeof(double) * n, cudaMemcpyHostToDevice, b->stream));
    }
    if (m) {
        k_batch_f32<<<static_cast<int>(std::min<int64_t>((m + 255) / 256, 4096)), 256, 0, b->stream>>>(
            b->val + ebase, b->val32 + ebase, m);
        ++b->launches;
    }
    KTG_BCUDA(b, cudaStreamSynchronize(b->stream));
    b->sys.push_back(ktg::SysDesc{base, ebase, static_cast<int32_t>(n), static_cast<int32_t>(m)});
    b->cost.push_back(m + n);
    b->rows += n;
    b->nnz += m;
    b->dirty = true;
    if (id) *id = k;
    return KTG_OK;
}

int ktg_batch_add_from_context(ktg_batch *b, ktg_ctx *c, const double *x0, const double *y0,
                               int64_t *first_id) {
    if (!b || !c || !x0 || !y0) return KTG_ERR_ARG;
    if (!c->have_system) return berr(b, KTG_ERR_STATE, "context has no systems");
    int64_t first = -1;
    for (int axis = 0; axis < 2; ++axis) {
        int64_t n = 0, m = 0;
        int rc = ktg_system_info(c, axis, &n, &m);
        if (rc) return berr(b, rc, "ktg_system_info failed");
        std::vector<int64_t> rp(n + 1);
        std::vector<int32_t> col(m);
        std::vector<double> val(m), dg(n), rhs(n);
        if ((rc = ktg_download_system(c, axis, rp.data(), col.data(), val.data(), dg.data(), rhs.data())))
            return berr(b, rc, "ktg_download_system failed");
        int64_t id = -1;
        if ((rc = ktg_batch_add_system(b, n, rp.data(), col.data(), val.data(), dg.data(), rhs.data(),
                                       axis ? y0 : x0, &id)))
            return rc;
        if (axis == 0) first = id;
    }
    if (first_id) *first_id = first;
    return KTG_OK;
}

int ktg_batch_set_shape(ktg_batch *b, int cluster, int threads) {
    if (!b) return KTG_ERR_ARG;
    if (!(cluster == 1 || cluster == 2 || cluster == 4 || cluster == 8 || cluster == 16))
        return berr(b, KTG_ERR_ARG, "cluster must be 1, 2, 4, 8 or 16");
    if (!(threads == 128 || threads == 256 || threads == 512 || threads == 1024))
        return berr(b, KTG_ERR_ARG, "threads must be 128, 256, 512 or 1024");
    b->cluster = cluster;
    b->threads = threads;
    return KTG_OK;
}

int ktg_batch_get_shape(const ktg_batch *b, int *cluster, int *threads) {
    if (!b) return KTG_ERR_ARG;
    if (cluster) *cluster = b->cluster;
    if (threads) *threads = b->threads;
    return KTG_OK;
}

int ktg_batch_set_split(ktg_batch *b, int64_t rows, int cluster, int threads, int clusters) {
    if (!b) return KTG_ERR_ARG;
    if (rows < 0) return berr(b, KTG_ERR_ARG, "negative split rows");
    if (rows > 0) {
        if (!(cluster == 1 || cluster == 2 || cluster == 4 || cluster == 8 || cluster == 16))
            return berr(b, KTG_ERR_ARG, "cluster must be 1, 2, 4, 8 or 16");
        if (!(threads == 128 || threads == 256 || threads == 512 || threads == 1024))
            return berr(b, KTG_ERR_ARG, "threads must be 128, 256, 512 or 1024");
        if (clusters < 1) return berr(b, KTG_ERR_ARG, "clusters must be >= 1");
        b->split_cluster = cluster;
        b->split_threads = threads;
        b->split_clusters = clusters;
    }
    b->split_rows = rows;
    return KTG_OK;
}

int ktg_batch_set_offload(ktg_batch *b, int64_t rows, int precond, int coarse) {
    if (!b) return KTG_ERR_ARG;
    if (rows < 0) return berr(b, KTG_ERR_ARG, "negative offload rows");
    if (precond < 0 || precond > 2) return berr(b, KTG_ERR_ARG, "precond must be 0, 1 or 2");
    if (coarse < 0 || coarse > 2) return berr(b, KTG_ERR_ARG, "coarse must be 0, 1 or 2");
    if (precond == 1) return berr(b, KTG_ERR_ARG, "the learned inverse needs a prepared network");
    b->offload_rows = rows;
    b->offload_precond = precond;
    b->offload_coarse = coarse;
    return KTG_OK;
}

int ktg_batch_get_offload(const ktg_batch *b, int64_t *rows, int *pairs) {
    if (!b) return KTG_ERR_ARG;
    if (rows) *rows = b->offload_rows;
    if (pairs) {
        int k = 0;
        const int32_t ns = static_cast<int32_t>(b->sys.size());
        if (b->offload_rows > 0)
            for (int32_t i = 0; i + 1 < ns;) {
                if (b->sys[i].n >= b->offload_rows && b->sys[i + 1].n == b->sys[i].n) {
                    ++k;
                    i += 2;
                } else {
                    ++i;
                }
            }
        *pairs = k;
    }
    return KTG_OK;
}

int ktg_batch_get_split(const ktg_batch *b, int64_t *rows, int *cluster, int *threads,
                        int *clusters, int *num_large) {
    if (!b) return KTG_ERR_ARG;
    if (rows) *rows = b->split_rows;
    if (cluster) *cluster = b->split_cluster;
    if (threads) *threads = b->split_threads;
    if (clusters) *clusters = b->split_clusters;
    if (num_large) {
        // systems of the queues only: offloaded pairs are in no class
        const std::vector<char> off = offloaded(b);
        int64_t k = 0;
        if (b->split_rows > 0)
            for (size_t i = 0; i < b->sys.size(); ++i) k += !off[i] && b->sys[i].n >= b->split_rows;
        *num_large = static_cast<int>(k);
    }
    return KTG_OK;
}

int ktg_batch_reset_x(ktg_batch *b) {
    if (!b) return KTG_ERR_ARG;
    if (b->rows)
        KTG_BCUDA(b, cudaMemcpyAsync(b->x, b->x0, sizeof(double) * b->rows, cudaMemcpyDeviceToDevice,
                                     b->stream));
    return KTG_OK;
}

static void (*batch_kernel(int mixed, int cluster, int near_bytes))(ktg::BatchArgs) {
    return !mixed                      ? ktg::k_batch_pcg<ktg::kFp64>
           : near_bytes > 0            ? ktg::k_batch_pcg<ktg::kNear>
           : cluster <= ktg::kPortable ? ktg::k_batch_pcg<ktg::kTiles>
                                       : ktg::k_batch_pcg<ktg::kTilesWide>;
}

// What a class would keep in shared memory: the search directions of its mixed
// solves, room for the largest that pays (bytes; none where a system's direction does
// not fit, since that one decides the class's time), and its systems in rows.
struct NearPlan {
    int bytes = 0;
    int64_t most = 0;          // rows of the largest system
    int64_t all = 0, big = 0;  // rows of all, and of those of at least half as many
};

// A system's own cost, in rows: a solve of 300 rows takes as long as 1,000 more do
// (8 x 512: 0.3 ms, and 0.2 us a row).
constexpr int64_t kSystemRows = 1000;

// The FP64 solve keeps nothing there: 8 bytes a row leave it too little L1 (24
// systems of 5k to 48k rows on 4 x 1,024: 20.7 ms with, 13.7 without).
static int near_room(ktg_batch *b, int mixed, NearPlan *plan) {
    if (!mixed) return KTG_OK;
    int &near_limit = b->near_limit;
    if (near_limit == 0) {
        const auto kernel = ktg::k_batch_pcg<ktg::kNear>;
        cudaFuncAttributes fa;
        int most = 0;
        KTG_BCUDA(b, cudaFuncGetAttributes(&fa, kernel));
        KTG_BCUDA(b, cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                            b->device));
        const int limit = (most - static_cast<int>(fa.sharedSizeBytes)) / 256 * 256;
        KTG_BCUDA(b, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          limit));
        near_limit = limit;
    }
    const std::vector<char> off = offloaded(b);
    auto in_class = [&](size_t i) { return b->split_rows > 0 && b->sys[i].n >= b->split_rows; };
    int64_t near[2] = {0, 0};
    bool alone[2] = {false, false};
    for (size_t i = 0; i < b->sys.size(); ++i) {
        if (off[i]) continue;
        const int k = in_class(i) ? 1 : 0;
        const int64_t n = b->sys[i].n;
        plan[k].most = std::max(plan[k].most, n);
        const int cluster = k ? b->split_cluster : b->cluster;
        if (ktg::jagged_pays(n, cluster)) near[k] = std::max(near[k], n);
        alone[k] = alone[k] || ktg::jagged_pays_alone(n, b->sys[i].nnz, cluster,
                                                      k ? b->split_threads : b->threads);
    }
    for (size_t i = 0; i < b->sys.size(); ++i) {
        if (off[i]) continue;
        NearPlan &p = plan[in_class(i) ? 1 : 0];
        const int64_t rows = b->sys[i].n + kSystemRows;
        p.all += rows;
        if (2 * static_cast<int64_t>(b->sys[i].n) >= p.most) p.big += rows;
    }
    for (int k = 0; k < 2; ++k)
        if (alone[k] && plan[k].most * 4 <= near_limit)
            plan[k].bytes = static_cast<int>((near[k] * 4 + 255) / 256 * 256);
    return KTG_OK;
}

// How many clusters of `cluster` CTAs of `threads` threads can be resident
// at once on the whole device.
static int resident_clusters(ktg_batch *b, int mixed, int cluster, int threads, int near_bytes,
                             int *out) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(threads);
    cfg.gridDim = dim3(cluster);
    cfg.dynamicSmemBytes = near_bytes;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cluster > 8)
        KTG_BCUDA(b, cudaFuncSetAttribute(batch_kernel(mixed, cluster, near_bytes),
                                          cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    KTG_BCUDA(b, cudaOccupancyMaxActiveClusters(out, batch_kernel(mixed, cluster, near_bytes), &cfg));
    if (*out < 1) return berr(b, KTG_ERR_CUDA, "cluster shape cannot be resident");
    return KTG_OK;
}

// The same for a class's plan: with the search directions in shared memory, or
// without (*near_bytes 0) where the shape is then not resident, or where fewer
// clusters are and that costs more than it gives: the class is mostly systems much
// smaller than its largest, which gain little, and they would take well longer than
// the largest does (8 x 512: 2 systems of 45k rows and 200 of 5k 8.4 ms without, 13.1
// with; 200 of 40k rows 30.7 and 28.3; 4 x 512: the first 14.3 and 8.6).
static int near_clusters(ktg_batch *b, int mixed, int cluster, int threads, const NearPlan &plan,
                         int *near_bytes, int *out) {
    *near_bytes = 0;
    if (plan.bytes > 0) {
        int with = 0, without = 0;
        if (resident_clusters(b, mixed, cluster, threads, plan.bytes, &with) == KTG_OK &&
            (resident_clusters(b, mixed, cluster, threads, 0, &without) != KTG_OK ||
             with >= without || 2 * plan.big >= plan.all || 4 * plan.all <= 5 * with * plan.most)) {
            b->err.clear();
            *near_bytes = plan.bytes;
            *out = with;
            return KTG_OK;
        }
        (void)cudaGetLastError();
        b->err.clear();
    }
    return resident_clusters(b, mixed, cluster, threads, 0, out);
}

// One persistent launch over the systems order[first, first + count): `clusters`
// clusters of `cluster` CTAs of `threads` threads draining `queue`.
static int enqueue_class(ktg_batch *b, int first, int count, unsigned *queue, int cluster,
                         int threads, int clusters, int near_bytes, double tol, int64_t max_iter,
                         int mixed, double inner_tol, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = near_bytes;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(std::max(1, std::min(clusters, count)) * cluster);
    ktg::BatchArgs A{b->d_sys, b->d_order + first, count, b->rp, b->col, b->val, b->val32,
                     b->diag, b->rhs, b->x, b->r, b->z, b->p, b->ap, b->d32, b->ri32, b->z32,
                     b->p32, b->ap32, b->jcol, b->jval, b->diag32, b->perm, b->inv, b->len,
                     b->start, b->next, queue, b->results, tol, inner_tol, max_iter, 50,
                     120000000000ull};
    KTG_BCUDA(b, cudaMemsetAsync(queue, 0, sizeof(unsigned), st));
    KTG_BCUDA(b, cudaLaunchKernelEx(&cfg, batch_kernel(mixed, cluster, near_bytes), A));
    return KTG_OK;
}

// Enqueues the whole batch solve on `st`. Without a size split it is one
// launch of the batch shape sized to the device. With one, the large class
// runs on a forked stream as its own launch while the small class's grid is
// cut to the SMs the large clusters leave free; the two launches share no
// state besides the solution arrays of disjoint systems, so neither waits on
// the other and the fork is joined back into `st` at the end.
static int batch_enqueue(ktg_batch *b, double tol, int64_t max_iter, int mixed, double inner_tol,
                         cudaStream_t st) {
    const int ns = b->num_queued;
    const int nl = b->num_large;
    int res_small = 0, near_small = 0, near_large = 0;
    NearPlan plan[2];  // of the systems below the split, and from it on
    int rc = near_room(b, mixed, plan);
    if (rc) return rc;
    if (nl < ns &&
        (rc = near_clusters(b, mixed, b->cluster, b->threads, plan[0], &near_small, &res_small)))
        return rc;
    if (nl == 0) {
        rc = enqueue_class(b, 0, ns, b->queue, b->cluster, b->threads, res_small, near_small, tol,
                           max_iter, mixed, inner_tol, st);
        b->graph_kernels = 1;
        return rc;
    }
    int res_large = 0;
    if ((rc = near_clusters(b, mixed, b->split_cluster, b->split_threads, plan[1], &near_large,
                            &res_large)))
        return rc;
    const int large_clusters = std::min({b->split_clusters, res_large, nl});
    if (nl == ns) {
        rc = enqueue_class(b, 0, ns, b->queue2, b->split_cluster, b->split_threads, large_clusters,
                           near_large, tol, max_iter, mixed, inner_tol, st);
        b->graph_kernels = 1;
        return rc;
    }
    // SMs held by the large class, from its CTAs per SM when the device is full.
    const int sms = std::max(1, b->num_sms);
    const int large_per_sm = std::max(1, res_large * b->split_cluster / sms);
    const int large_sms = (large_clusters * b->split_cluster + large_per_sm - 1) / large_per_sm;
    const int small_per_sm = std::max(1, res_small * b->cluster / sms);
    const int free_sms = std::max(b->cluster, sms - large_sms);
    const int small_clusters = std::max(1, std::min(res_small, free_sms * small_per_sm / b->cluster));
    cudaEvent_t fork = nullptr, join = nullptr;
    cudaStream_t side = nullptr;
    KTG_BCUDA(b, cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    if (cudaEventCreateWithFlags(&join, cudaEventDisableTiming) != cudaSuccess ||
        cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking) != cudaSuccess) {
        cudaEventDestroy(fork);
        if (join) cudaEventDestroy(join);
        return berr(b, KTG_ERR_CUDA, "fork stream creation failed");
    }
    if (cudaEventRecord(fork, st) != cudaSuccess || cudaStreamWaitEvent(side, fork, 0) != cudaSuccess)
        rc = berr(b, KTG_ERR_CUDA, "stream fork failed");
    if (!rc)
        rc = enqueue_class(b, 0, nl, b->queue2, b->split_cluster, b->split_threads, large_clusters,
                           near_large, tol, max_iter, mixed, inner_tol, side);
    if (!rc)
        rc = enqueue_class(b, nl, ns - nl, b->queue, b->cluster, b->threads, small_clusters,
                           near_small, tol, max_iter, mixed, inner_tol, st);
    if (!rc && (cudaEventRecord(join, side) != cudaSuccess ||
                cudaStreamWaitEvent(st, join, 0) != cudaSuccess))
        rc = berr(b, KTG_ERR_CUDA, "stream join failed");
    cudaEventDestroy(fork);
    cudaEventDestroy(join);
    cudaStreamDestroy(side);
    b->graph_kernels = 2;
    return rc;
}

// The offloaded pairs, one after another on the batch's stream, each through
// the internal context: its x and y systems copied in (device to device),
// then the whole-GPU solve on the batch's own solution slices, then the
// pair's results.
static int solve_offloaded(ktg_batch *b, double tol, int64_t max_iter, int precision,
                           double inner_tol) {
    int rc;
    if (!b->octx) {
        if ((rc = ktg_create(b->device, &b->octx))) return berr(b, rc, "internal context");
        if (cudaMalloc(&b->d_minfo, sizeof(ktg_mixed_info)) != cudaSuccess ||
            cudaMalloc(&b->d_sinfo, sizeof(ktg_solve_info)) != cudaSuccess ||
            cudaMalloc(&b->d_stamp, sizeof(unsigned long long)) != cudaSuccess)
            return berr(b, KTG_ERR_NOMEM, "offload buffers");
    }
    ktg_ctx *c = b->octx;
    const int64_t launches0 = c->launches;
    if ((rc = ktg_set_stream(c, b->stream)) || (rc = ktg_set_pointer_mode(c, KTG_PTR_DEVICE)) ||
        (rc = ktg_set_option(c, "precond", b->offload_precond)) ||
        (rc = ktg_set_option(c, "coarse", b->offload_coarse)))
        return berr(b, rc, std::string("internal context: ") + c->err);
    for (int32_t f : b->off_first) {
        const ktg::SysDesc &X = b->sys[f], &Y = b->sys[f + 1];
        k_stamp<<<1, 1, 0, b->stream>>>(b->d_stamp);
        ++b->launches;
        const int64_t mx = b->cost[f] - X.n, my = b->cost[f + 1] - Y.n;
        // room for both axes at once (one growth at most)
        if ((rc = ktg::reserve_system_arrays(c, X.n, std::max(mx, my))) ||
            (rc = ktg::load_system_device(c, 0, X.n, mx, b->rp + X.row_base + f,
                                          b->col + X.nnz_base, b->val + X.nnz_base,
                                          b->diag + X.row_base, b->rhs + X.row_base)) ||
            (rc = ktg::load_system_device(c, 1, Y.n, my, b->rp + Y.row_base + f + 1,
                                          b->col + Y.nnz_base, b->val + Y.nnz_base,
                                          b->diag + Y.row_base, b->rhs + Y.row_base)))
            return berr(b, rc, std::string("offload load: ") + c->err);
        if (!c->have_system) return berr(b, KTG_ERR_STATE, "offload load: pair not complete");
        double *x = b->x + X.row_base, *y = b->x + Y.row_base;
        rc = precision == 1 ? ktg_solve_mixed(c, x, y, tol, inner_tol, max_iter, 50, b->d_minfo,
                                              nullptr, nullptr, 0)
                            : ktg_solve(c, x, y, tol, max_iter, b->d_sinfo, nullptr, nullptr, 0);
        if (rc) return berr(b, rc, std::string("offload solve: ") + c->err);
        k_offload_results<<<1, 1, 0, b->stream>>>(b->d_minfo, b->d_sinfo, precision, tol, f,
                                                        f + 1, b->d_stamp, b->results);
        ++b->launches;
        KTG_BCUDA(b, cudaGetLastError());
    }
    b->launches += c->launches - launches0;
    return KTG_OK;
}

int ktg_batch_solve(ktg_batch *b, double tol, int64_t max_iter, int precision, double inner_tol) {
    if (!b) return KTG_ERR_ARG;
    if (precision != 0 && precision != 1) return berr(b, KTG_ERR_ARG, "precision must be 0 or 1");
    if (precision == 1 && !(inner_tol > 0.0 && inner_tol < 1.0))
        return berr(b, KTG_ERR_ARG, "inner_tol must be in (0, 1)");
    if (max_iter < 0) return berr(b, KTG_ERR_ARG, "negative max_iter");
    if (b->sys.empty()) return KTG_OK;
    if (cudaSetDevice(b->device) != cudaSuccess) return KTG_ERR_CUDA;
    if (b->dirty || b->order_split_rows != b->split_rows ||
        b->order_offload_rows != b->offload_rows) {
        // Offloaded pairs first leave the queues; then largest first within
        // each class, the large class (rows >= split_rows) at the front.
        const int32_t ns = static_cast<int32_t>(b->sys.size());
        const std::vector<char> off = offloaded(b, &b->off_first);
        std::vector<int32_t> order;
        for (int32_t k = 0; k < ns; ++k)
            if (!off[k]) order.push_back(k);
        b->num_queued = static_cast<int>(order.size());
        auto large = [&](int32_t p) { return b->split_rows > 0 && b->sys[p].n >= b->split_rows; };
        std::stable_sort(order.begin(), order.end(), [&](int32_t p, int32_t q) {
            if (large(p) != large(q)) return large(p);
            return b->cost[p] > b->cost[q];
        });
        b->num_large = static_cast<int>(std::count_if(order.begin(), order.end(), large));
        KTG_BCUDA(b, cudaMemcpyAsync(b->d_sys, b->sys.data(), sizeof(ktg::SysDesc) * b->sys.size(),
                                     cudaMemcpyHostToDevice, b->stream));
        if (!order.empty())
            KTG_BCUDA(b, cudaMemcpyAsync(b->d_order, order.data(), sizeof(int32_t) * order.size(),
                                         cudaMemcpyHostToDevice, b->stream));
        KTG_BCUDA(b, cudaStreamSynchronize(b->stream));
        b->dirty = false;
        b->order_split_rows = b->split_rows;
        b->order_offload_rows = b->offload_rows;
        if (b->graph) {
            cudaGraphExecDestroy(b->graph);
            b->graph = nullptr;
        }
    }
    if (!b->off_first.empty()) {
        int rc = solve_offloaded(b, tol, max_iter, precision, inner_tol);
        if (rc) return rc;
    }
    if (b->num_queued == 0) return KTG_OK;
    const bool same = b->graph && b->g_tol == tol && b->g_max_iter == max_iter &&
                      b->g_mixed == precision && b->g_inner == inner_tol &&
                      b->g_cluster == b->cluster && b->g_threads == b->threads &&
                      b->g_split_rows == b->split_rows && b->g_split_cluster == b->split_cluster &&
                      b->g_split_threads == b->split_threads &&
                      b->g_split_clusters == b->split_clusters;
    if (!same) {
        if (b->graph) {
            cudaGraphExecDestroy(b->graph);
            b->graph = nullptr;
        }
        NearPlan plan[2];
        int rc = near_room(b, precision, plan);
        if (!rc && plan[0].bytes + plan[1].bytes > 0) rc = reserve_jagged(b);
        if (rc) return rc;
        // Capture the whole batch solve once on a private stream.
        cudaStream_t cap;
        KTG_BCUDA(b, cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
        cudaGraph_t g = nullptr;
        if (cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaStreamDestroy(cap);
            return berr(b, KTG_ERR_CUDA, "stream capture failed to start");
        }
        rc = batch_enqueue(b, tol, max_iter, precision, inner_tol, cap);
        const cudaError_t ec = cudaStreamEndCapture(cap, &g);
        cudaStreamDestroy(cap);
        if (rc) {
            if (g) cudaGraphDestroy(g);
            return rc;
        }
        if (ec != cudaSuccess) return berr(b, KTG_ERR_CUDA, "stream capture failed");
        const cudaError_t ei = cudaGraphInstantiate(&b->graph, g, 0);
        cudaGraphDestroy(g);
        if (ei != cudaSuccess) return berr(b, KTG_ERR_CUDA, "graph instantiation failed");
        b->g_tol = tol;
        b->g_max_iter = max_iter;
        b->g_mixed = precision;
        b->g_inner = inner_tol;
        b->g_cluster = b->cluster;
        b->g_threads = b->threads;
        b->g_split_rows = b->split_rows;
        b->g_split_cluster = b->split_cluster;
        b->g_split_threads = b->split_threads;
        b->g_split_clusters = b->split_clusters;
    }
    KTG_BCUDA(b, cudaGraphLaunch(b->graph, b->stream));
    b->launches += b->graph_kernels;
    return KTG_OK;
}

int ktg_batch_results(ktg_batch *b, ktg_batch_result *out) {
    if (!b || !out) return KTG_ERR_ARG;
    if (b->sys.empty()) return KTG_OK;
    KTG_BCUDA(b, cudaMemcpyAsync(out, b->results, sizeof(ktg_batch_result) * b->sys.size(),
                                 cudaMemcpyDeviceToHost, b->stream));
    KTG_BCUDA(b, cudaStreamSynchronize(b->stream));
    return KTG_OK;
}

int ktg_batch_get_x(ktg_batch *b, int64_t id, double *x) {
    if (!b || !x || id < 0 || id >= static_cast<int64_t>(b->sys.size())) return KTG_ERR_ARG;
    const ktg::SysDesc &s = b->sys[id];
    KTG_BCUDA(b, cudaMemcpyAsync(x, b->x + s.row_base, sizeof(double) * s.n, cudaMemcpyDeviceToHost,
                                 b->stream));
    KTG_BCUDA(b, cudaStreamSynchronize(b->stream));
    return KTG_OK;
}

int64_t ktg_batch_launch_count(const ktg_batch *b) { return b ? b->launches : 0; }

int ktg_batch_autotune(ktg_batch *b, double tol, int precision, double inner_tol,
                       int64_t probe_iter, int *cluster, int *threads, float *best_ms) {
    if (!b || probe_iter <= 0) return KTG_ERR_ARG;
    if (b->sys.empty()) return berr(b, KTG_ERR_STATE, "empty batch");
    static const int kClusters[] = {2, 4, 8, 16};
    static const int kThreads[] = {256, 512, 1024};
    cudaEvent_t e0, e1;
    KTG_BCUDA(b, cudaEventCreate(&e0));
    KTG_BCUDA(b, cudaEventCreate(&e1));
    float best = 1e30f;
    int bc = b->cluster, bt = b->threads;
    int rc = KTG_OK;
    for (int c : kClusters) {
        for (int t : kThreads) {
            if ((rc = ktg_batch_set_shape(b, c, t))) break;
            int resident = 0;
            if (resident_clusters(b, precision, c, t, 0, &resident) != KTG_OK) {
                b->err.clear();
                continue;  // shape not launchable on this device
            }
            float ms = 0.0f;
            for (int rep = 0; rep < 2 && rc == KTG_OK; ++rep) {
                if ((rc = ktg_batch_reset_x(b))) break;
                if (cudaEventRecord(e0, b->stream) != cudaSuccess) rc = KTG_ERR_CUDA;
                if (!rc) rc = ktg_batch_solve(b, tol, probe_iter, precision, inner_tol);
                if (!rc && cudaEventRecord(e1, b->stream) != cudaSuccess) rc = KTG_ERR_CUDA;
                if (!rc && cudaEventSynchronize(e1) != cudaSuccess) rc = KTG_ERR_CUDA;
                if (!rc) cudaEventElapsedTime(&ms, e0, e1);
            }
            if (rc) break;
            if (ms < best) {
                best = ms;
                bc = c;
                bt = t;
            }
        }
        if (rc) break;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    ktg_batch_set_shape(b, bc, bt);
    if ((rc = ktg_batch_reset_x(b))) return rc;
    if (cluster) *cluster = bc;
    if (threads) *threads = bt;
    if (best_ms) *best_ms = best;
    return KTG_OK;
}

// Times one full solve (from reset x) of the current configuration.
static int time_solve(ktg_batch *b, double tol, int64_t max_iter, int precision, double inner_tol,
                      cudaEvent_t e0, cudaEvent_t e1, float *ms) {
    int rc;
    if ((rc = ktg_batch_reset_x(b))) return rc;
    KTG_BCUDA(b, cudaEventRecord(e0, b->stream));
    if ((rc = ktg_batch_solve(b, tol, max_iter, precision, inner_tol))) return rc;
    KTG_BCUDA(b, cudaEventRecord(e1, b->stream));
    KTG_BCUDA(b, cudaEventSynchronize(e1));
    KTG_BCUDA(b, cudaEventElapsedTime(ms, e0, e1));
    return KTG_OK;
}

int ktg_batch_autotune_split(ktg_batch *b, double tol, int precision, double inner_tol,
                             int64_t max_iter, float *base_ms, float *best_ms) {
    if (!b || max_iter <= 0) return KTG_ERR_ARG;
    if (b->sys.empty()) return berr(b, KTG_ERR_STATE, "empty batch");
    // Thresholds that put the 1, 2, 4, 8 or 16 largest queued systems (ties
    // included) in the large class; offloaded pairs are in no class.
    std::vector<int64_t> sizes;
    const std::vector<char> off = offloaded(b);
    for (size_t i = 0; i < b->sys.size(); ++i)
        if (!off[i]) sizes.push_back(b->sys[i].n);
    if (sizes.empty()) {  // every system is offloaded: nothing to split
        if (base_ms) *base_ms = 0.0f;
        if (best_ms) *best_ms = 0.0f;
        return ktg_batch_set_split(b, 0, 0, 0, 0);
    }
    std::sort(sizes.begin(), sizes.end(), std::greater<int64_t>());
    std::vector<int64_t> cuts;
    for (size_t k : {1, 2, 4, 8, 16}) {
        if (k >= sizes.size()) break;
        const int64_t t = sizes[k - 1];
        if (t > sizes.back() && (cuts.empty() || cuts.back() != t)) cuts.push_back(t);
    }
    static const int kShapes[][2] = {{16, 1024}, {8, 1024}, {16, 512}};
    static const int kCount[] = {1, 2, 4, 8};
    cudaEvent_t e0, e1;
    KTG_BCUDA(b, cudaEventCreate(&e0));
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return berr(b, KTG_ERR_CUDA, "event creation failed");
    }
    int rc = ktg_batch_set_split(b, 0, 0, 0, 0);
    float none = 0.0f, ms = 0.0f;
    for (int rep = 0; rep < 2 && !rc; ++rep) rc = time_solve(b, tol, max_iter, precision, inner_tol, e0, e1, &none);
    float best = none;
    int64_t br = 0;
    int bc = b->split_cluster, bt = b->split_threads, bn = b->split_clusters;
    for (int64_t cut : cuts) {
        if (rc) break;
        for (const auto &sh : kShapes) {
            if (rc) break;
            int resident = 0;
            if (resident_clusters(b, precision, sh[0], sh[1], 0, &resident) != KTG_OK) {
                b->err.clear();
                continue;  // shape not launchable on this device
            }
            for (int n : kCount) {
                if (n > resident) break;
                if ((rc = ktg_batch_set_split(b, cut, sh[0], sh[1], n))) break;
                int nl = 0;
                ktg_batch_get_split(b, nullptr, nullptr, nullptr, nullptr, &nl);
                if (n > nl) break;
                float t = 1e30f;
                for (int rep = 0; rep < 2 && !rc; ++rep) {
                    rc = time_solve(b, tol, max_iter, precision, inner_tol, e0, e1, &ms);
                    t = std::min(t, ms);
                }
                if (!rc && t < best) {
                    best = t;
                    br = cut;
                    bc = sh[0];
                    bt = sh[1];
                    bn = n;
                }
            }
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if ((rc = ktg_batch_set_split(b, br, bc, bt, bn))) return rc;
    if ((rc = ktg_batch_reset_x(b))) return rc;
    if (base_ms) *base_ms = none;
    if (best_ms) *best_ms = best;
    return KTG_OK;
}

int ktg_batch_autotune_offload(ktg_batch *b, double tol, int precision, double inner_tol,
                               int64_t max_iter, float *base_ms, float *best_ms) {
    if (!b || max_iter <= 0) return KTG_ERR_ARG;
    if (b->sys.empty()) return berr(b, KTG_ERR_STATE, "empty batch");
    std::vector<int64_t> sizes;
    for (const ktg::SysDesc &d : b->sys) sizes.push_back(d.n);
    std::sort(sizes.begin(), sizes.end(), std::greater<int64_t>());
    std::vector<int64_t> cuts;  // the 2, 4, ... 64 largest systems (pairs of them)
    for (size_t k : {2, 4, 8, 16, 24, 32, 48, 64}) {
        if (k > sizes.size()) break;
        const int64_t t = sizes[k - 1];
        if (t > 0 && (cuts.empty() || cuts.back() != t)) cuts.push_back(t);
    }
    cudaEvent_t e0, e1;
    KTG_BCUDA(b, cudaEventCreate(&e0));
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return berr(b, KTG_ERR_CUDA, "event creation failed");
    }
    const int64_t split0 = b->split_rows;
    int rc = ktg_batch_set_split(b, 0, 0, 0, 0);
    const int pre = b->offload_precond, co = b->offload_coarse;
    if (!rc) rc = ktg_batch_set_offload(b, 0, pre, co);
    float none = 1e30f, ms = 0.0f;
    for (int rep = 0; rep < 2 && !rc; ++rep) {
        rc = time_solve(b, tol, max_iter, precision, inner_tol, e0, e1, &ms);
        none = std::min(none, ms);
    }
    float best = none;
    int64_t br = 0;
    for (int64_t cut : cuts) {
        if (rc) break;
        if ((rc = ktg_batch_set_offload(b, cut, pre, co))) break;
        int pairs = 0;
        ktg_batch_get_offload(b, nullptr, &pairs);
        if (pairs == 0) continue;
        float t = 1e30f;
        for (int rep = 0; rep < 2 && !rc; ++rep) {
            rc = time_solve(b, tol, max_iter, precision, inner_tol, e0, e1, &ms);
            t = std::min(t, ms);
        }
        if (!rc && t < best) {
            best = t;
            br = cut;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if ((rc = ktg_batch_set_offload(b, br, pre, co))) return rc;
    b->split_rows = split0;
    if ((rc = ktg_batch_reset_x(b))) return rc;
    if (base_ms) *base_ms = none;
    if (best_ms) *best_ms = best;
    return KTG_OK;
}

}  // extern "C"
