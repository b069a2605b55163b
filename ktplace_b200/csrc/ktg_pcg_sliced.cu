// The default FP64 solve: Jacobi-PCG for the x and y systems in one
// persistent cooperative launch over a sliced copy of the systems (sm_100a).
//
// Same iteration as form 3 of ktg_pcg.cu (solveBothAxes, simpl_lss.cc:203-290,
// with A p = A z + beta A p_prev: two grid-wide reductions per iteration).
// What differs is how the SpMV is fed:
//
//  * Sliced rows. Every block sorts the rows of its slice of the combined row
//    space [x rows | y rows] by length (stable counting sort, longest first)
//    and copies them into slices of 32 rows, entry k of a slice's rows side by
//    side: a warp takes a slice, a lane takes a row, column and value loads
//    are coalesced and each lane adds its row's products in storage order in a
//    register. The staged form (warp tiles of ktg_spmv.cuh) moves every
//    product through shared memory; on the 211k system that is as many L1TEX
//    wavefronts again as the gathers themselves, and the gathers (one
//    wavefront each, random columns) are what bounds an SpMV here: 28.2k per
//    SM and pass = 15 us. Sorting keeps the padding at 3% of the entries.
//  * Rows renumbered by position. The gathered vector lives in sorted order,
//    so the update phase publishes it with coalesced stores, and the other
//    vectors are in that order too.
//  * Slices are dealt to the warps once per solve by longest-processing-time
//    (widths are known), so the summation order is fixed by the pattern alone
//    and results are the same from run to run.
//  * A row longer than `width` entries takes 2, 4, ... 32 lanes, so that no
//    warp's slices outlast the others' (a 48-entry row on one lane did).
//  * The two reductions per iteration are the barriers (ktg_allreduce.cuh), and
//    the iteration's scalars are advanced by one lane per axis.
//
// The copy costs one pass over the CSR system and doubles as the solve's first
// product A x; with the sort it takes 85 us at 211k cells, three steps.
//
// Measured against the warp-tile form it replaced, us per step of both axes
// (same iterations): 300 cells 13.6 -> 5.1, 1k 18.9 -> 7.0, 12k 20.1 -> 9.7,
// 47k 21.0 -> 13.6, 100k 23.9 -> 17.0, 211k 34.4 -> 28.8, 300k 57.9 -> 38.6,
// 600k 99.8 -> 70.2, 1M 158 -> 114. What bounds a step at 211k: 32k cycles of
// gathers in the average block (28k wavefronts) and 38k in the slowest, 7k for
// each reduction, 3k for the update.
#include "ktg_allreduce.cuh"
#include "ktg_common.cuh"
#include "ktg_context.h"

#include <algorithm>

namespace ktg {
namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxWidth = 24;              // entries per lane, at most (a warp per row aside)
constexpr int kMinWidth = 8;               // even, as all widths
constexpr int kBuckets = 2 + 3 * kMaxWidth;
constexpr int kSmallRows = 256;            // rows a block of a small system owns, at least
constexpr int kSmallBlocks = 48;           // and blocks it has, at most
constexpr size_t kSmemBudget = 124 * 1024;

struct SlicedAxis {
    const int32_t *rp;
    const int32_t *col;
    const double *val;
    const double *diag;
    const double *rhs;
    double *x;
};

// The iteration's scalars, per axis (masks: bit a = axis a). Kept in shared
// memory and advanced by two lanes of warp 0: in every thread's registers,
// their divisions and square roots took 3.8k cycles of FP64 issue a step.
struct SlicedState {
    double b_norm[2], rr[2], rho[2], alpha[2], beta[2];
    unsigned active[2], live[2], ok[2];
    unsigned first[2];  // no step taken yet: p = z, A p = w
    unsigned owed[2];   // x += alpha p is left to the next product phase (or the
                        // end), which reads p anyway
    int64_t steps[2];
};

struct SlicedArgs {
    SlicedAxis ax[2];
    int32_t n;               // rows per axis
    int32_t rows_per_block;
    int32_t slices_per_block;
    int32_t width;           // entries per lane before a row takes more lanes
    double tol;
    int64_t max_iter;
    SlicedSystem S;
    int *status;
    ktg_solve_info *info;
    double *hist_x;
    double *hist_y;
    int64_t hist_cap;
    uint64_t barrier_timeout_ns;
    uint64_t total_timeout_ns;
    const ktg_mixed_info *gate;  // see launch_solve
};

// Entry loads of the sliced copy: read once per iteration, so they bypass L1
// (which serves the gathers) and leave L2 first.
__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

__device__ __forceinline__ int32_t ld_stream(const int32_t *p, uint64_t pol) {
    int32_t v;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.s32 %0, [%1], %2;"
                 : "=r"(v) : "l"(p), "l"(pol));
    return v;
}

__device__ __forceinline__ double ld_stream(const double *p, uint64_t pol) {
    double v;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;"
                 : "=d"(v) : "l"(p), "l"(pol));
    return v;
}

// Lanes per row: the fewest (a power of two) that leave each at most `kw`
// entries, at most a warp. log2 of it.
__device__ __forceinline__ int lane_shift(int32_t len, int32_t kw) {
    int sh = 0;
    while (sh < 5 && len > (kw << sh)) ++sh;
    return sh;
}

// First entry of block b's region in the sliced copy, in units of 32 entries.
// Rows of a class (lanes per row) come widest first, so each slice but its
// class's first is no wider than the rows of the one before it are long; the
// rounding of a row to its lanes adds at most a quarter, and each class one
// slice of the widest rows at most.
__host__ __device__ __forceinline__ int64_t region_base(int64_t entries_before, int64_t block) {
    return (entries_before + entries_before / 4 + 31) / 32 + block * (6 * kMaxWidth + 7);
}

// NV of the vectors r, x, p, A p (in this order) live in shared memory, the rest
// in global memory; the gathered z is always global.
template <int NV>
__global__ void __launch_bounds__(kThreads, 1) k_pcg_sliced(SlicedArgs A) {
    if (A.gate) {
        // FP64 pass after a mixed solve: nothing left to do when that converged
        const ktg_mixed_info g = *A.gate;
        if (g.status == 0 && g.stalled == 0 && g.resid_x <= A.tol && g.resid_y <= A.tol) {
            if (blockIdx.x == 0 && threadIdx.x == 0)
                *A.info = ktg_solve_info{g.resid_x, g.resid_y, 0, 0, 0, 0, 0};
            return;
        }
    }
    extern __shared__ __align__(16) double dyn[];
    __shared__ double scratch[4 * 33];
    __shared__ SlicedState st;
    __shared__ int32_t hist[kBuckets + 1];
    __shared__ uint16_t wcnt[kWarps * kBuckets];
    __shared__ SlicedAxis sax[2];
    __shared__ int32_t s_class[7];  // first position of each class, 32 lanes per row first
    __shared__ int32_t s_wbeg[kWarps + 1];
    if (threadIdx.x < 2) sax[threadIdx.x] = A.ax[threadIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int32_t n = A.n, total = 2 * n, kw = A.width;
    const int32_t r0 = min(static_cast<int64_t>(blockIdx.x) * A.rows_per_block,
                           static_cast<int64_t>(total));
    const int32_t R = min(A.rows_per_block, total - r0);
    const int32_t cap = A.rows_per_block;
    const int32_t cap_slices = A.slices_per_block;
    // Positions [0, R) of the block; vectors at position j: shared memory, or
    // the block's part of the global arrays.
    double *vr = NV > 0 ? dyn : A.S.r + r0;
    double *vx = NV > 1 ? dyn + cap : A.S.x + r0;
    double *vp = NV > 2 ? dyn + 2 * cap : A.S.p + r0;
    double *vap = NV > 3 ? dyn + 3 * cap : A.S.ap + r0;
    double *vz = A.S.z + r0;
    const double *vd = A.S.diag + r0;
    uint8_t *vax = NV > 0 ? reinterpret_cast<uint8_t *>(dyn + NV * cap) : A.S.axis + r0;
    // Per slice (in the order the warps take them): first entry / 32, and the
    // first position with the lane shift in the top bits.
    const size_t moff = static_cast<size_t>(blockIdx.x) * cap_slices;
    uint2 *const slices = A.S.slices + moff;
    uint2 *const mine = A.S.dealt + moff;
    AllReduce<2> red{A.S.slots, A.status, 0u, global_timer_ns() + A.total_timeout_ns,
                  A.barrier_timeout_ns};
    const uint64_t stream = evict_first_policy();
    __syncthreads();

    // ---- rows by class and width, widest first (stable counting sort) -----------
    auto row_of = [&](int32_t c, int &axis) {  // combined row -> axis, row
        axis = c >= n ? 1 : 0;
        return c - (axis ? n : 0);
    };
    auto row_len = [&](int32_t c) -> int32_t {
        int axis;
        const int32_t i = row_of(c, axis);
        return __ldg(sax[axis].rp + i + 1) - __ldg(sax[axis].rp + i);
    };
    const int32_t half = kw / 2;
    auto bucket = [&](int32_t len) -> int {
        const int sh = lane_shift(len, kw);
        if (sh == 5) return 0;
        const int32_t w = (len + (1 << sh) - 1) >> sh;
        return sh ? 1 + (4 - sh) * half + (kw - w) : 1 + 4 * half + (kw - len);
    };
    const int nb = 2 + 4 * half + kw;  // buckets
    for (int k = threadIdx.x; k <= nb; k += blockDim.x) hist[k] = 0;
    __syncthreads();
    for (int32_t l = threadIdx.x; l < R; l += blockDim.x)
        atomicAdd(hist + bucket(row_len(r0 + l)), 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        int32_t at = 0;
        for (int k = 0; k < nb; ++k) {
            const int32_t c = hist[k];
            hist[k] = at;
            at += c;
        }
        s_class[0] = 0;
        for (int k = 1; k <= 5; ++k) s_class[k] = hist[1 + (k - 1) * half];
        s_class[6] = R;
    }
    __syncthreads();
    for (int32_t l0 = 0; l0 < R; l0 += blockDim.x) {
        for (int k = threadIdx.x; k < nw * nb; k += blockDim.x) wcnt[k] = 0;
        __syncthreads();
        const int32_t l = l0 + threadIdx.x;
        const int b = l < R ? bucket(row_len(r0 + l)) : nb;
        const unsigned same = __match_any_sync(0xffffffffu, b);
        const int rank = __popc(same & ((1u << lane) - 1u));
        if (l < R && rank == 0) wcnt[warp * nb + b] = static_cast<uint16_t>(__popc(same));
        __syncthreads();
        if (threadIdx.x < nb) {  // exclusive over the warps; warp 0's entry: the total
            int32_t at = 0;
            for (int w = 0; w < nw; ++w) {
                const int32_t c = wcnt[w * nb + threadIdx.x];
                wcnt[w * nb + threadIdx.x] = static_cast<uint16_t>(at);
                at += c;
            }
            wcnt[threadIdx.x] = static_cast<uint16_t>(at);
        }
        __syncthreads();
        if (l < R) {
            const int32_t j = hist[b] + (warp ? wcnt[warp * nb + b] : 0) + rank;
            int axis;
            const int32_t i = row_of(r0 + l, axis);
            A.S.perm[r0 + j] = r0 + l;
            vax[j] = static_cast<uint8_t>(axis);
            A.S.diag[r0 + j] = __ldg(sax[axis].diag + i);
            const double x = sax[axis].x[i];
            A.S.start[r0 + l] = Start{x, r0 + j};  // gathered by the first product
            vx[j] = x;
        }
        __syncthreads();
        if (threadIdx.x < nb) hist[threadIdx.x] += wcnt[threadIdx.x];
        __syncthreads();
    }
    // ---- slices, their widths and offsets, and their warps ----------------------
    if (warp == 0) {
        int32_t ns = 0;
        uint32_t at = 0;
        // longest-processing-time: the next slice goes to the warp with the
        // least work so far (lane = warp)
        uint32_t load = 0, count = 0;
        for (int k = 0; k < 6; ++k) {
            const int sh = 5 - k;
            const int32_t per = 32 >> sh;
            for (int32_t f = s_class[k]; f < s_class[k + 1]; f += 32 * per) {
                // lane: one slice of up to 32
                const int32_t first = f + lane * per;
                const bool on = first < s_class[k + 1];
                const int32_t len = on ? row_len(A.S.perm[r0 + first]) : 0;
                const uint32_t w = static_cast<uint32_t>((len + (1 << sh) - 1) >> sh);
                uint32_t inc = w;
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += t;
                }
                const int cnt = __popc(__ballot_sync(0xffffffffu, on));
                const uint2 d = make_uint2(at + inc - w, static_cast<uint32_t>(first) |
                                                             static_cast<uint32_t>(sh) << 29);
                int own = 0;
                for (int q = 0; q < cnt; ++q) {
                    const uint32_t key = lane < nw ? (min(load, (1u << 26) - 1u) << 5 | lane) : ~0u;
                    const uint32_t best = __reduce_min_sync(0xffffffffu, key) & 31u;
                    const uint32_t wq = __shfl_sync(0xffffffffu, w, q);
                    if (static_cast<uint32_t>(lane) == best) {
                        load += wq + 2 + sh;
                        ++count;
                    }
                    if (lane == q) own = static_cast<int>(best);
                }
                if (on) {
                    slices[ns + lane] = d;
                    A.S.owner[moff + ns + lane] = static_cast<uint8_t>(own);
                }
                ns += cnt;
                at += __shfl_sync(0xffffffffu, inc, 31);
            }
        }
        uint32_t inc = count;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        s_wbeg[lane] = static_cast<int32_t>(inc - count);
        if (lane == 31) s_wbeg[32] = static_cast<int32_t>(inc);
        if (lane == 0) slices[ns] = make_uint2(at, 0u);  // the last slice's end
        hist[0] = ns;
    }
    __syncthreads();
    const int32_t q0 = s_wbeg[warp], q1 = s_wbeg[warp + 1];
    // each warp's slices, in order: entry offset | first position and shift,
    // widths apart
    {
        const int32_t ns = hist[0];
        uint32_t *const wid = A.S.widths + moff;
        int32_t at = q0;
        for (int32_t s0 = 0; s0 < ns; s0 += 32) {
            const int32_t s = s0 + lane;
            const bool take = s < ns && A.S.owner[moff + s] == static_cast<uint8_t>(warp);
            const unsigned m = __ballot_sync(0xffffffffu, take);
            if (take) {
                const int32_t q = at + __popc(m & ((1u << lane) - 1u));
                mine[q] = slices[s];
                wid[q] = slices[s + 1].x - slices[s].x;
            }
            at += __popc(m);
        }
    }
    __syncwarp();
    int64_t base;
    {
        const int64_t e = r0 <= n ? static_cast<int64_t>(__ldg(sax[0].rp + r0))
                                  : static_cast<int64_t>(__ldg(sax[0].rp + n)) +
                                        __ldg(sax[1].rp + (r0 - n));
        base = region_base(e, blockIdx.x) * 32;
    }
    int32_t *const ecol = A.S.col + base;
    double *const eval = A.S.val + base;
    const uint32_t *const widths = A.S.widths + moff;
    // Slice q of this warp: lane's row position j (sub-lane sub of 1 << sh; j
    // is past the class's end for lanes without a row), entries and width.
    auto slice = [&](int32_t q, int32_t &j, int &sh, int &sub, size_t &o, int32_t &w) {
        const uint2 d = mine[q];
        w = static_cast<int32_t>(widths[q]);
        sh = static_cast<int>(d.y >> 29);
        sub = lane & ((1 << sh) - 1);
        j = static_cast<int32_t>(d.y & 0x1fffffffu) + (lane >> sh);
        o = static_cast<size_t>(d.x) * 32 + lane;
        return j < s_class[6 - sh];
    };
    auto row_sum = [&](double s, int sh) {  // over the row's lanes
        for (int d = 1; d < (1 << sh); d <<= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        return s;
    };
    const double none[2] = {0.0, 0.0};
    if (!red.sum<true, 1>(none, scratch, [](int, const double (&)[1]) {})) return;

    // ---- start: Ap = A x, r = b - Ap, z = r / diag, and the sliced copy ---------
    // Vectors much larger than L1 are gathered past it (1M cells: 113.6 us a
    // step instead of 120; 211k cells: 31.8 instead of 30).
    auto gather = [](const double *p) { return NV > 1 ? *p : __ldcg(p); };
    // ||r|| / ||b|| > tol; the squares decide unless they are close (the exact
    // form's square root and division are on every step's critical path). A
    // negative tolerance, which nothing meets, has no square to compare with.
    auto resid = [](double rr, double bn) { return sqrt(rr) / bn; };
    auto above_tol = [&](double rr, double bn) {
        const double lim = A.tol * bn, q = lim * lim;
        if (lim > 0.0 && q > 1e-280 && q < 1e280) {
            if (rr > q * (1.0 + 1e-10)) return true;
            if (rr < q * (1.0 - 1e-10)) return false;
        }
        return resid(rr, bn) > A.tol;
    };
    double bb[2] = {0.0, 0.0}, acc0[4] = {0.0, 0.0, 0.0, 0.0};  // b.b; rr x, rz x, rr y, rz y
    for (int32_t q = q0; q < q1; ++q) {
        int32_t j, w;
        int sh, sub, axis = 0;
        size_t o;
        const bool on = slice(q, j, sh, sub, o, w);
        // the lane's entries of the row: [eb, ee), read four at a time aligned
        int32_t i = 0, eb = 0, ee = 0;
        if (on) {
            i = row_of(A.S.perm[r0 + j], axis);
            const int32_t e0 = __ldg(sax[axis].rp + i), e1 = __ldg(sax[axis].rp + i + 1);
            const int32_t per = (e1 - e0 + (1 << sh) - 1) >> sh;
            eb = min(e0 + sub * per, e1);
            ee = min(eb + per, e1);
        }
        const Start *from = A.S.start + (axis ? n : 0);
        const int4 *cols = reinterpret_cast<const int4 *>(sax[axis].col);
        const double2 *vals = reinterpret_cast<const double2 *>(sax[axis].val);
        double sum = 0.0;
        for (int32_t e = eb & ~3; e < ee; e += 4) {
            const int4 c4 = __ldg(cols + (e >> 2));
            const double2 va = __ldg(vals + (e >> 1)), vb = __ldg(vals + (e >> 1) + 1);
            const int32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
            const double v[4] = {va.x, va.y, vb.x, vb.y};
            Start g[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (e + u >= eb && e + u < ee) g[u] = from[c[u]];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (e + u >= eb && e + u < ee) {
                    sum += v[u] * g[u].x;
                    const size_t q = o + static_cast<size_t>(e + u - eb) * 32;
                    ecol[q] = static_cast<int32_t>(g[u].pos);
                    eval[q] = v[u];
                }
        }
        for (int32_t k = ee - eb; k < w; ++k) ecol[o + static_cast<size_t>(k) * 32] = -1;
        sum = row_sum(sum, sh);
        if (on && sub == 0) {
            const double b = __ldg(sax[axis].rhs + i);
            const double d = vd[j];
            const double r = b - (d * vx[j] + sum);
            const double z = r / d;
            vr[j] = r;
            vz[j] = z;
            if (axis) {
                bb[1] += b * b;
                acc0[2] += r * r;
                acc0[3] += r * z;
            } else {
                bb[0] += b * b;
                acc0[0] += r * r;
                acc0[1] += r * z;
            }
        }
    }
    if (!red.sum<false, 1>(bb, scratch, [&](int a, const double (&t)[1]) {
            if (lane == 0) st.b_norm[a] = sqrt(t[0]);
        }))
        return;
    if (!red.sum<true, 2>(acc0, scratch, [&](int a, const double (&t)[2]) {
            if (lane != 0) return;
            const bool act = st.b_norm[a] > 0.0;
            st.rr[a] = t[0];
            st.rho[a] = act ? t[1] : 0.0;
            st.active[a] = act;
            st.live[a] = act && above_tol(t[0], st.b_norm[a]);
            st.alpha[a] = st.beta[a] = 0.0;
            st.ok[a] = st.owed[a] = 0u;
            st.first[a] = 1u;
            st.steps[a] = 0;
        }))
        return;

    auto final_resid = [&](int a) {
        return st.b_norm[a] > 0.0 ? resid(st.rr[a], st.b_norm[a]) : 0.0;
    };
    int64_t it = 0;
    for (;;) {
        const unsigned mask = st.live[0] | st.live[1] << 1;
        if (it >= A.max_iter || !mask) break;

        // ---- A: w = A z; p = z + beta p, Ap = w + beta Ap; p.Ap ---------------
        double pap[2] = {0.0, 0.0};
        for (int32_t q = q0; q < q1; ++q) {
            int32_t j, w;
            int sh, sub;
            size_t o;
            const bool in = slice(q, j, sh, sub, o, w);
            const int axis = in ? vax[j] : 0;
            const bool on = in && ((mask >> axis) & 1u);
            if (mask != 3u && !__any_sync(0xffffffffu, on)) continue;
            const int32_t *cp = ecol + o;
            const double *ep = eval + o;
            const bool lead = on && sub == 0;
            const bool fresh = st.first[axis] != 0u;
            double zi = 0.0, dz = 0.0, p0 = 0.0, ap0 = 0.0;
            if (lead) {  // in flight behind the gathers
                zi = vz[j];
                dz = vd[j];
                if (!fresh) {
                    p0 = vp[j];
                    ap0 = vap[j];
                }
            }
            double sum = 0.0;
            for (int32_t k = 0; k < w; k += 4, cp += 128, ep += 128) {
                int32_t c[4];
                double v[4], g[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) c[u] = k + u < w ? ld_stream(cp + 32 * u, stream) : -1;
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = k + u < w ? ld_stream(ep + 32 * u, stream) : 0.0;
#pragma unroll
                for (int u = 0; u < 4; ++u) g[u] = c[u] >= 0 ? gather(A.S.z + c[u]) : 0.0;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (c[u] >= 0) sum += v[u] * g[u];
            }
            sum = row_sum(sum, sh);
            if (lead) {
                double pn = zi, apn = dz * zi + sum;
                if (!fresh) {
                    const double be = st.beta[axis];
                    if (st.owed[axis]) vx[j] += st.alpha[axis] * p0;
                    pn = zi + be * p0;
                    apn = apn + be * ap0;
                }
                vp[j] = pn;
                vap[j] = apn;
                if (axis)
                    pap[1] += pn * apn;
                else
                    pap[0] += pn * apn;
            }
        }
        if (!red.sum<false, 1>(pap, scratch, [&](int a, const double (&t)[1]) {
                if (lane != 0 || !st.live[a]) return;
                const bool ok = t[0] > 0.0;
                st.ok[a] = st.owed[a] = ok;
                if (ok) st.alpha[a] = st.rho[a] / t[0];
            }))
            return;

        // ---- B: r, z update, r.r and r.z ---------------------------------------
        double acc[4] = {0.0, 0.0, 0.0, 0.0};  // rr x, rz x, rr y, rz y
#pragma unroll 2
        for (int32_t j = threadIdx.x; j < R; j += blockDim.x) {
            const int axis = vax[j];
            const bool on = st.ok[axis] != 0u;
            const double a = st.alpha[axis];
            const double apv = vap[j], d = vd[j], ri = vr[j];
            if (!on) continue;
            const double r = ri - a * apv;
            const double z = r / d;
            vr[j] = r;
            vz[j] = z;  // gathered by the next product
            if (axis) {
                acc[2] += r * r;
                acc[3] += r * z;
            } else {
                acc[0] += r * r;
                acc[1] += r * z;
            }
        }
        if (!red.sum<true, 2>(acc, scratch, [&](int a, const double (&t)[2]) {
                // lane 0: rho and beta; lane 1: residual and the stopping test
                const bool live = st.live[a] != 0u;
                const bool ok = st.ok[a] != 0u, go = ok && t[1] > 0.0;
                __syncwarp();
                if (!live || lane >= 2) return;
                if (lane == 0) {
                    st.beta[a] = go ? t[1] / st.rho[a] : 0.0;
                    if (go) st.rho[a] = t[1];
                    st.first[a] = 0u;
                    ++st.steps[a];
                } else {
                    const bool more = go && above_tol(t[0], st.b_norm[a]);
                    if (ok) st.rr[a] = t[0];
                    st.active[a] = go;
                    st.live[a] = more;
                    if (!more) st.ok[a] = 0u;  // its rows are left alone from here on
                }
            }))
            return;
        if (blockIdx.x == 0 && threadIdx.x < 2 && it < A.hist_cap) {
            double *h = threadIdx.x ? A.hist_y : A.hist_x;
            if (h) h[it] = final_resid(threadIdx.x);
        }
        ++it;
    }

    for (int32_t j = threadIdx.x; j < R; j += blockDim.x) {
        int axis;
        const int32_t i = row_of(A.S.perm[r0 + j], axis);
        double x = vx[j];
        if (st.owed[axis]) x += st.alpha[axis] * vp[j];
        sax[axis].x[i] = x;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ktg_solve_info inf;
        inf.resid_x = final_resid(0);
        inf.resid_y = final_resid(1);
        inf.iters = it;
        inf.iters_x = st.steps[0];
        inf.iters_y = st.steps[1];
        inf.status = kStatusOk;
        inf.live = static_cast<int32_t>(st.live[0] | st.live[1] << 1);
        *A.info = inf;
    }
}

size_t sliced_smem(int nv, int64_t rows_per_block) {
    return nv ? (sizeof(double) * nv + 1) * rows_per_block : 0;
}

}  // namespace

// Blocks of a solve over `rows` rows of both axes.
static int sliced_grid(int64_t rows, int num_sms) {
    // One up to kThreads rows (its sums need no barrier: 5.1 us a step at 600
    // rows, 7.5 us on three blocks). Then kSmallBlocks of kSmallRows to kThreads
    // rows (2,000 rows: 7.0 us a step with 256 rows a block, 9.4 with 1,024;
    // 24,000 rows: 9.7 and 10.1), and beyond that kThreads rows a block: a third of
    // the SMs serves a small system as well as all of them, and leaves room for
    // solves on other streams.
    const int64_t per =
        rows <= kThreads
            ? kThreads
            : std::min<int64_t>(kThreads, std::max<int64_t>(kSmallRows,
                                                            (rows + kSmallBlocks - 1) / kSmallBlocks));
    const int64_t most = std::min(num_sms, 32 * kSumGroups);
    return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(most, (rows + per - 1) / per)));
}

// The most blocks of a solve over up to `rows` rows (sliced_grid can fall by one
// where the rows of a block grow).
int sliced_blocks(int64_t rows, int num_sms) {
    const int64_t small = std::min<int64_t>(kSmallBlocks, (rows + kSmallRows - 1) / kSmallRows);
    const int64_t blocks = rows <= kThreads ? 1 : std::max(small, (rows + kThreads - 1) / kThreads);
    return static_cast<int>(std::min<int64_t>(std::min(num_sms, 32 * kSumGroups), blocks));
}

int64_t sliced_entries(int64_t nnz_both, int blocks) { return 32 * region_base(nnz_both, blocks); }

// Slices of a block of `rows` rows: a warp per row at worst, and one end mark.
int64_t sliced_slices(int64_t rows, int num_sms) { return rows + 2 * num_sms; }

int64_t sliced_slots(int num_sms) { return int64_t(kSumSets) * 2 * kSumWords * num_sms; }

int launch_solve_sliced(ktg_ctx *c, double *x, double *y, double tol, int64_t max_iter,
                        ktg_solve_info *info_dev, double *hist_x, double *hist_y,
                        int64_t hist_cap) {
    SlicedArgs A;
    for (int a = 0; a < 2; ++a) {
        AxisSystem &s = c->sys[a];
        A.ax[a] = SlicedAxis{s.row_ptr, s.col, s.val, s.diag, s.rhs, a ? y : x};
    }
    A.n = static_cast<int32_t>(c->sys_n);
    const int64_t total = 2 * c->sys_n;
    const int grid = sliced_grid(total, c->num_sms);
    A.rows_per_block = static_cast<int32_t>(std::max<int64_t>(1, (total + grid - 1) / grid));
    A.slices_per_block = A.rows_per_block + 1;
    const int threads = grid > 1 && A.rows_per_block <= kSmallRows ? kThreads / 2 : kThreads;
    // Entries per lane: a block with few slices waits for its widest, one with
    // many is bound by the gathers and pays for partly filled slices (12k cells:
    // 10.5 / 10.1 / 11.3 us a step with 8 / 16 / 24 at 1,024 rows a block; 1M:
    // 129 / 119 / 118).
    A.width = A.rows_per_block <= kSmallRows || grid == 1 ? kMinWidth
              : A.rows_per_block < 2048                   ? 2 * kMinWidth
                                                          : kMaxWidth;
    // Vectors in shared memory: as many as leave half the SM's memory to L1.
    // 300k cells: 42.2 / 39.7 / 41.1 us a step with 4 (134 KB) / 2 (69 KB) / 0;
    // 400k: 66.4 / 50.3 / 52.2; 1M: 118 with 1 (121 KB), 126 with 0.
    using Kernel = void (*)(SlicedArgs);
    const Kernel kernels[] = {k_pcg_sliced<0>, k_pcg_sliced<1>, k_pcg_sliced<2>, k_pcg_sliced<4>};
    const int vecs[] = {0, 1, 2, 4};
    int pick = 3;
    while (sliced_smem(vecs[pick], A.rows_per_block) > kSmemBudget) --pick;
    const Kernel fn = kernels[pick];
    const size_t bytes = sliced_smem(vecs[pick], A.rows_per_block);
    // per variant, as it comes up: the attribute loads the kernel
    if (!(c->attr_bits & (kAttrSliced << pick))) {
        KTG_CUDA(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kSmemBudget)));
        c->attr_bits |= kAttrSliced << pick;
    }
    A.tol = tol;
    A.max_iter = max_iter;
    A.S = c->sliced;
    A.status = c->status;
    A.info = info_dev;
    A.gate = c->pcg_gate;
    A.hist_x = hist_x;
    A.hist_y = hist_y;
    A.hist_cap = hist_cap;
    A.barrier_timeout_ns = 2000000000ull;   // 2 s for any single barrier
    A.total_timeout_ns = 120000000000ull;   // 120 s for the whole solve
    KTG_CUDA(c, cudaMemsetAsync(c->status, 0, sizeof(int), c->stream));
    KTG_CUDA(c, cudaMemsetAsync(c->sliced.slots, 0xff,
                                sizeof(unsigned long long) * kSumSets * 4 * grid, c->stream));
    void *args[] = {&A};
    KTG_CUDA(c, cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(fn), dim3(grid),
                                            dim3(threads), args, bytes, c->stream));
    c->launches += 1;
    return KTG_OK;
}

}  // namespace ktg
