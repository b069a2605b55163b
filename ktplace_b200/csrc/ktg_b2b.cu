// B2B net-model assembly and HPWL (sm_100a).
//
// Replaces LinearSystems::buildB2B / buildB2BAxis (globalPlacer/simpl/
// simpl_lss.cc:11-114) and simplPlacer::Impl::getHpwl (simpl_placer.cc:
// 256-275). Four launches build both axes at once:
//
//   k_bound_pins  one lane per net, pins staged by the warp: first-index
//                 argmin/argmax of the pin coordinate for x and y
//                 (simpl_lss.cc:32-45) and, from the same pass, the net's
//                 half perimeter (HPWL of the inputs).
//   k_row_count   four lanes per (axis, movable cell): number of movable
//                 other ends of its B2B edges (simpl_lss.cc:75-83), plus a
//                 per-block total.
//   k_scan_blocks one block: exclusive scan of the block totals -> the first
//                 CSR slot of every block and nnz per axis.
//   k_fill        a CTA per (axis, 64 movable cells): row_ptr, then the rows'
//                 edges in the reference's order (simpl_lss.cc:47-73, 89-113),
//                 computed a thread each and summed in order, so that diag and
//                 rhs are rounded exactly as the reference rounds them.
//
// Bit-exactness: the library is compiled with -fmad=false (no FMA
// contraction, like the reference's -ffp-contract=off) and CUDA's IEEE
// double division, so every w, val, diag and rhs equals the reference's.
//
// The same kernels also build Kraftwerk2's systems
// (Kraftwerk2Placer::Impl::buildSystem, globalPlacer/kraftwerk2/
// kraftwerk2_placer.cc:328-410) under its own rules (Rules = kKraftwerk2):
// the high bound pin is the last maximum (>=), the edge weight base is
// 2 w / (p - 1), nets may list a cell twice and edges to the row's own cell
// are skipped, the right-hand side uses the raw pin offsets, and there is
// neither an anchor term nor a diagonal floor (the caller applies them).
#include "ktg_common.cuh"
#include "ktg_context.h"

namespace ktg {
namespace {

constexpr int kBuildThreads = 256;
enum Rules { kSimpl = 0, kKraftwerk2 = 1 };

struct NetlistDev {
    const int32_t *var_of_vertex;
    const double *fixed_x;
    const double *fixed_y;
    const int32_t *net_start;
    const int32_t *pin_cell;
    const int32_t *pin_var;
    const double *off_x;
    const double *off_y;
    const double *net_base;
    const int32_t *net_mov;
    const int32_t *pin_start;
    const int2 *pin_ref;
    int32_t n;
    int32_t N;
};

NetlistDev view_of(const ktg_ctx *c) {
    return NetlistDev{c->var_of_vertex, c->fixed_x, c->fixed_y, c->net_start, c->pin_cell,
                      c->pin_var,       c->off_x,   c->off_y,   c->net_base,  c->net_mov,
                      c->pin_start,     c->pin_ref, static_cast<int32_t>(c->n),
                      static_cast<int32_t>(c->N)};
}

// Position of a pin's cell: movable cells read the variable vector, fixed
// cells their fixed coordinate (simpl_lss.cc:14-19).
__device__ __forceinline__ double cell_pos(const double *pos, const double *fixed, int32_t var,
                                           int32_t cell) {
    return var >= 0 ? pos[var] : fixed[cell];
}

// Pins staged per warp and round by k_bound_pins (two per lane).
constexpr int kPinChunk = 64;

// One lane per net, the pins staged by the warp. Each warp owns 32
// consecutive nets, whose pins are contiguous; the warp walks that pin range
// in chunks of kPinChunk, every lane loading and positioning pins of the
// chunk (coalesced pin reads, independent position gathers), and then each
// lane scans the part of its own net that falls in the chunk from shared
// memory, in pin order, carrying its running bounds across chunks. The scan
// order and the comparisons are the reference's, so the bound pins (first
// index wins on ties) and the half perimeters are the sequential ones; a
// net's term lands in the same thread as with one thread per net, so the
// block sums are too. WithBounds: also choose the bound pins of both axes.
template <bool WithBounds, int R = kSimpl>
__global__ void __launch_bounds__(kBuildThreads)
    k_bound_pins(NetlistDev nl, const double *__restrict__ x, const double *__restrict__ y,
                 int4 *__restrict__ bound_x, int4 *__restrict__ bound_y,
                 double *__restrict__ partials, unsigned *__restrict__ ticket,
                 double *__restrict__ hpwl_out, double *__restrict__ terms = nullptr) {
    __shared__ double scratch[40];
    __shared__ double spx[kBuildThreads / 32][kPinChunk];
    __shared__ double spy[kBuildThreads / 32][kPinChunk];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int kw0 = blockIdx.x * blockDim.x + (wid << 5);  // the warp's first net
    int32_t s = 0, e = 0, p0 = 0, p1 = 0;
    if (k < nl.N) {
        s = nl.net_start[k];
        e = nl.net_start[k + 1];
    }
    if (kw0 < nl.N) {  // warp-uniform pin range of nets [kw0, kw0 + 32)
        p0 = nl.net_start[kw0];
        p1 = nl.net_start[min(kw0 + 32, nl.N)];
    }
    uint32_t lx = 0, hx = 0, ly = 0, hy = 0;
    double vlx = 0.0, vhx = 0.0, vly = 0.0, vhy = 0.0;
    // BBox::getEmpty then BBox::extend (geometry/kt_geometry.cc:70-75)
    double bx0 = __longlong_as_double(0x7ff0000000000000ll);  // +inf
    double by0 = bx0;
    double bx1 = -bx0;
    double by1 = -bx0;
    for (int32_t cb = p0; cb < p1; cb += kPinChunk) {
        for (int j = lane; j < kPinChunk; j += 32) {
            const int32_t p = cb + j;
            if (p < p1) {
                const int32_t cell = nl.pin_cell[p];
                const int32_t var = nl.pin_var[p];
                spx[wid][j] = cell_pos(x, nl.fixed_x, var, cell) + nl.off_x[p];
                spy[wid][j] = cell_pos(y, nl.fixed_y, var, cell) + nl.off_y[p];
            }
        }
        __syncwarp();
        const int32_t qa = max(s, cb), qb = min(e, cb + kPinChunk);
        for (int32_t p = qa; p < qb; ++p) {
            const int32_t q = p - s;
            const double px = spx[wid][p - cb];
            const double py = spy[wid][p - cb];
            if (WithBounds) {
                if (q == 0) {
                    vlx = vhx = px;
                    vly = vhy = py;
                } else {
                    // lo = pinAt(q) < pinAt(lo) ? q : lo (simpl_lss.cc:41-42);
                    // Kraftwerk2: hi = at[q] >= at[hi] ? q : hi (kraftwerk2_placer.cc:341-342)
                    if (px < vlx) { lx = q; vlx = px; }
                    if (R == kKraftwerk2 ? px >= vhx : px > vhx) { hx = q; vhx = px; }
                    if (py < vly) { ly = q; vly = py; }
                    if (R == kKraftwerk2 ? py >= vhy : py > vhy) { hy = q; vhy = py; }
                }
            }
            bx0 = ref_min(bx0, px);
            by0 = ref_min(by0, py);
            bx1 = ref_max(bx1, px);
            by1 = ref_max(by1, py);
        }
        __syncwarp();
    }
    double term = 0.0;
    if (k < nl.N) {
        if (WithBounds) {
            bound_x[k] = make_int4(s, static_cast<int32_t>(lx), static_cast<int32_t>(hx), e - s);
            bound_y[k] = make_int4(s, static_cast<int32_t>(ly), static_cast<int32_t>(hy), e - s);
        }
        // getHalfPerimeter: 0 for an empty box; nets with < 2 pins add 0.
        if (e - s >= 2 && !(bx0 > bx1 || by0 > by1)) term = (bx1 - bx0) + (by1 - by0);
        if (terms) terms[k] = term;
    }
    if (terms) return;  // summed in the reference's order by k_hpwl_ref_order
    const double bs = block_sum(term, scratch);
    if (threadIdx.x == 0) __stcg(partials + blockIdx.x, bs);
    if (last_block_done(ticket)) {
        const double total = sum_partials(partials, gridDim.x, scratch);
        if (threadIdx.x == 0) *hpwl_out = total;
    }
}

// HPWL in the reference's summation order (getDeterministicSum,
// simpl_parallel.h:35-51): the per-net terms in chunks of kGrain nets, each
// chunk summed left to right by one thread, then the chunk sums in order.
constexpr int64_t kGrain = 4096;
__global__ void __launch_bounds__(1024)
    k_hpwl_ref_order(const double *__restrict__ terms, int64_t N, double *__restrict__ out) {
    __shared__ double chunk[1024];
    const int64_t chunks = (N + kGrain - 1) / kGrain;
    double total = 0.0;
    for (int64_t c0 = 0; c0 < chunks; c0 += blockDim.x) {
        const int64_t c = c0 + threadIdx.x;
        double s = 0.0;
        if (c < chunks) {
            const int64_t e = min(N, (c + 1) * kGrain);
            for (int64_t i = c * kGrain; i < e; ++i) s += terms[i];
        }
        chunk[threadIdx.x] = s;
        __syncthreads();
        const int64_t here = chunks - c0 < blockDim.x ? chunks - c0 : blockDim.x;
        if (threadIdx.x == 0)
            for (int64_t k = 0; k < here; ++k) total += chunk[k];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = total;
}

struct AxisArgs {
    const double *pos;
    const double *fixed;
    const double *off;
    const int4 *bound;
    double floor_len;
    const double *anchor;
    int32_t *row_ptr;
    int32_t *col;
    double *val;
    double *diag;
    double *rhs;
};

// Count of movable other ends per row; per-block totals for the scan. Chains of
// dependent gathers (pin, bound pins, net) bound it, so a row's pins are split
// over kCountLanes lanes and one 16-byte record per net and axis answers for its
// first pin, bound pins and degree: 45 -> 31 us at 211k cells, 14 -> 8 at 12k.
constexpr int kCountLanes = 4;

template <int R = kSimpl>
__global__ void __launch_bounds__(kBuildThreads *kCountLanes)
    k_row_count(NetlistDev nl, AxisArgs ax, AxisArgs ay, int32_t blocks_per_axis,
                int32_t *__restrict__ row_cnt, int64_t *__restrict__ block_sum_out) {
    __shared__ int32_t warp_tot[kBuildThreads * kCountLanes / kWarp];
    const int axis = blockIdx.x >= blocks_per_axis ? 1 : 0;
    const AxisArgs &a = axis ? ay : ax;
    const int32_t i = (blockIdx.x - axis * blocks_per_axis) * kBuildThreads +
                      static_cast<int32_t>(threadIdx.x) / kCountLanes;
    const int sub = threadIdx.x % kCountLanes;
    int32_t cnt = 0;
    if (i < nl.n) {
        const int32_t e0 = nl.pin_start[i];
        const int32_t e1 = nl.pin_start[i + 1];
        for (int32_t e = e0 + sub; e < e1; e += kCountLanes) {
            const int2 ref = nl.pin_ref[e];
            const int32_t k = ref.x;
            const int32_t q = ref.y;
            const int4 net = a.bound[k];
            const int32_t s = net.x, l = net.y, h = net.z;
            if (l == h) continue;
            if (R == kKraftwerk2) {
                // movable other ends that are not the row's own cell
                const auto other = [&](int32_t t) {
                    const int32_t v = nl.pin_var[s + t];
                    return v >= 0 && v != i ? 1 : 0;
                };
                if (q == l || q == h) {
                    for (int32_t t = 0; t < net.w; ++t)
                        if (t != q) cnt += other(t);
                } else {
                    cnt += other(l) + other(h);
                }
            } else if (q == l || q == h) {
                cnt += nl.net_mov[k] - 1;  // every other movable pin of the net
            } else {
                cnt += (nl.pin_var[s + l] >= 0 ? 1 : 0) + (nl.pin_var[s + h] >= 0 ? 1 : 0);
            }
        }
    }
    int32_t v = cnt;
#pragma unroll
    for (int o = 1; o < kCountLanes; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (i < nl.n && sub == 0) row_cnt[axis * nl.n + i] = v;
#pragma unroll
    for (int o = kCountLanes; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t t = 0;
        for (int w = 0; w < kBuildThreads * kCountLanes / kWarp; ++w) t += warp_tot[w];
        block_sum_out[blockIdx.x] = t;
    }
}

// Exclusive scan of the per-block totals of both axes (one block). Writes the
// first slot of every block in place, nnz per axis, row_ptr[n] and flags a
// capacity overflow.
__global__ void __launch_bounds__(1024)
    k_scan_blocks(int64_t *__restrict__ block_sum, int32_t blocks_per_axis, int32_t n,
                  int64_t cap, int32_t *__restrict__ row_ptr_x, int32_t *__restrict__ row_ptr_y,
                  int64_t *__restrict__ nnz_out, int *__restrict__ status) {
    __shared__ int64_t warp_tot[32];
    __shared__ int64_t carry;
    for (int axis = 0; axis < 2; ++axis) {
        int64_t *bs = block_sum + axis * blocks_per_axis;
        const int per = (blocks_per_axis + blockDim.x - 1) / blockDim.x;
        const int b0 = threadIdx.x * per;
        const int b1 = min(b0 + per, blocks_per_axis);
        int64_t local = 0;
        for (int b = b0; b < b1; ++b) local += bs[b];
        // block exclusive scan of `local`
        int64_t incl = local;
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warp_tot[threadIdx.x >> 5] = incl;
        __syncthreads();
        if (threadIdx.x < 32) {
            int64_t w = warp_tot[threadIdx.x];
            int64_t wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t t = __shfl_up_sync(0xffffffffu, wi, o);
                if (threadIdx.x >= o) wi += t;
            }
            warp_tot[threadIdx.x] = wi - w;  // exclusive warp offsets
            if (threadIdx.x == 31) carry = wi;
        }
        __syncthreads();
        int64_t run = warp_tot[threadIdx.x >> 5] + incl - local;
        for (int b = b0; b < b1; ++b) {
            const int64_t v = bs[b];
            bs[b] = run;
            run += v;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const int64_t total = carry;
            nnz_out[axis] = total;
            if (total > cap) {
                atomicCAS(status, kStatusOk, kStatusCapacity);
                (axis ? row_ptr_y : row_ptr_x)[n] = 0;
            } else {
                (axis ? row_ptr_y : row_ptr_x)[n] = static_cast<int32_t>(total);
            }
        }
        __syncthreads();
    }
}

// Exclusive scan over the CTA (kBuildThreads threads); the total goes to *total.
__device__ __forceinline__ int32_t block_excl(int32_t v, int32_t *warp_tot, int32_t *total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[wid] = incl;
    __syncthreads();
    int32_t before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kBuildThreads / kWarp; ++w) {
        const int32_t t = warp_tot[w];
        if (w < wid) before += t;
        all += t;
    }
    __syncthreads();
    *total = all;
    return before + incl - v;
}

// Row pointers from a block scan of the counts, then the rows' entries, for
// kFillRows rows a CTA. Gathers bound it: four dependent ones per edge, all
// through L1/L2. A thread takes a pin of the rows (its bound pins, its weight,
// how many edges it has), then an edge; edge numbers come from a scan of the
// counts, so neighbouring threads read neighbouring pins of a net and write
// neighbouring entries, whatever the rows' lengths. The weights and right-hand
// terms go to shared memory, from where one thread per row and sum adds them in
// edge order. Both axes take 148 us at 211k cells (47% of the issue slots, a
// third of the stalls on gathers; six CTAs per SM instead of five cost spills
// and gained nothing), 19 at 12k and 15 at 300; one thread per row (a warp for
// rows of 32 ends and more) took 218 + 75 and 79 + 29.
// Kraftwerk2: alpha < 0 leaves the right-hand side at zero (withRhs false).
constexpr int kFillRows = 64;
constexpr int kFillEdges = 4 * kBuildThreads;  // edges in shared memory at once
static_assert(kBuildThreads % kFillRows == 0 && 2 * kFillRows <= kBuildThreads, "");

template <int R = kSimpl>
__global__ void __launch_bounds__(kBuildThreads, 5)
    k_fill(NetlistDev nl, AxisArgs ax, AxisArgs ay, int32_t blocks_per_axis,
           int32_t groups_per_axis, double alpha, const int32_t *__restrict__ row_cnt,
           const int64_t *__restrict__ block_first, int64_t cap, const int *__restrict__ status) {
    constexpr int kWarps = kBuildThreads / kWarp;
    constexpr int kPer = kFillEdges / kBuildThreads;
    __shared__ double s_w[kFillEdges], s_term[kFillEdges];
    __shared__ double s_own[kBuildThreads], s_off[kBuildThreads], s_base[kBuildThreads];
    __shared__ double s_pos[kFillRows];
    __shared__ int32_t s_first[kBuildThreads];                  // the net's first pin
    __shared__ int32_t s_lo[kBuildThreads], s_hi[kBuildThreads];  // hi < 0: every pin but lo
    __shared__ int32_t s_edge[kBuildThreads + 1];
    __shared__ uint8_t s_row[kBuildThreads];
    __shared__ int32_t s_pin[kFillRows + 1];
    __shared__ int32_t s_cnt[kPer * kWarps];
    __shared__ int32_t warp_tot[kWarps];
    __shared__ int64_t s_slot;
    static_assert(kPer * kWarps == kWarp, "one lane per count below");
    if (*status != kStatusOk) return;  // capacity exceeded: leave the buffers alone
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int axis = blockIdx.x >= groups_per_axis ? 1 : 0;
    const AxisArgs &a = axis ? ay : ax;
    const int32_t g = blockIdx.x - axis * groups_per_axis;
    const int32_t i0 = g * kFillRows;
    const int rows = min(kFillRows, nl.n - i0);
    {
        const int32_t b = i0 / kBuildThreads;
        const int32_t i = b * kBuildThreads + tid;
        int32_t all;
        const int32_t before =
            block_excl(i < nl.n ? row_cnt[axis * nl.n + i] : 0, warp_tot, &all);
        const int64_t slot = block_first[axis * blocks_per_axis + b] + before;
        if (i == i0) s_slot = slot;
        if (i >= i0 && i < i0 + rows) a.row_ptr[i] = static_cast<int32_t>(slot);
    }
    if (tid <= rows) s_pin[tid] = nl.pin_start[i0 + tid];
    if (tid < rows) s_pos[tid] = a.pos[i0 + tid];
    __syncthreads();
    int64_t slot = s_slot;
    // thread r sums row r's weights, thread kFillRows + r its right-hand terms
    const int row = tid % kFillRows;
    const bool adds = tid < 2 * kFillRows && row < rows;
    double sum = 0.0;
    for (int32_t pc = s_pin[0]; pc < s_pin[rows]; pc += kBuildThreads) {
        const int pins = min(kBuildThreads, s_pin[rows] - pc);
        int32_t ne = 0;
        if (tid < pins) {
            const int2 ref = nl.pin_ref[pc + tid];
            const int32_t k = ref.x, q = ref.y;
            const int4 net = a.bound[k];
            const int32_t s = net.x, l = net.y, h = net.z, deg = net.w;
            // Kraftwerk2's base, w * 2 / (p - 1), is exactly twice w / (p - 1)
            const double base = R == kKraftwerk2 ? 2.0 * nl.net_base[k] : nl.net_base[k];
            const double own_raw = a.off[s + q];
            int lo = 0, hi = rows;  // last row starting at or before the pin
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (s_pin[mid] <= pc + tid) lo = mid;
                else hi = mid;
            }
            const double own_pos = s_pos[lo];
            const double own = own_pos + own_raw;
            const bool bound = q == l || q == h;
            ne = l == h ? 0 : bound ? deg - 1 : 2;
            s_first[tid] = s;
            s_lo[tid] = bound ? q : l;
            s_hi[tid] = bound ? -1 : h;
            s_base[tid] = base;
            s_own[tid] = own;
            s_off[tid] = R == kKraftwerk2 ? own_raw : own - own_pos;
            if (R == kKraftwerk2) s_row[tid] = static_cast<uint8_t>(lo);
        }
        int32_t edges;
        const int32_t first = block_excl(ne, warp_tot, &edges);
        s_edge[tid] = first;
        if (tid == 0) s_edge[kBuildThreads] = edges;
        __syncthreads();
        for (int32_t c0 = 0; c0 < edges; c0 += kFillEdges) {
            int32_t var[kPer];
            double w[kPer];
            unsigned entry[kPer];
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                const int32_t j = c0 + u * kBuildThreads + tid;
                var[u] = -1;
                w[u] = 0.0;
                double term = 0.0;
                bool has = j < edges;
                if (has) {
                    int lo = 0, hi = pins;  // the pin of edge j
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if (s_edge[mid] <= j) lo = mid;
                        else hi = mid;
                    }
                    const int32_t at = j - s_edge[lo], lq = s_lo[lo], hq = s_hi[lo];
                    const int32_t t = hq < 0 ? at + (at >= lq ? 1 : 0) : at == 0 ? lq : hq;
                    const int32_t p = s_first[lo] + t;
                    var[u] = nl.pin_var[p];
                    // a second pin of the row's own cell is no edge
                    if (R == kKraftwerk2) has = var[u] != i0 + s_row[lo];
                    if (has) {
                        const double cp = var[u] >= 0 ? a.pos[var[u]] : a.fixed[nl.pin_cell[p]];
                        const double other_raw = a.off[p];
                        const double there = cp + other_raw;
                        w[u] = s_base[lo] / ref_max(fabs(s_own[lo] - there), a.floor_len);
                        // Kraftwerk2: w * (otherOffset - ownOffset), w * (at[other] - ownOffset)
                        term = var[u] < 0          ? w[u] * (there - s_off[lo])
                               : R == kKraftwerk2 ? w[u] * (other_raw - s_off[lo])
                                                  : w[u] * ((there - cp) - s_off[lo]);
                    }
                }
                // (an edge left out adds 0 below, which changes no sum)
                s_w[u * kBuildThreads + tid] = w[u];
                s_term[u * kBuildThreads + tid] = term;
                entry[u] = __ballot_sync(0xffffffffu, has && var[u] >= 0);
                if (lane == 0) s_cnt[u * kWarps + wid] = __popc(entry[u]);
            }
            __syncthreads();
            int32_t incl = s_cnt[lane];
            const int32_t mine = incl;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                const int32_t before = __shfl_sync(0xffffffffu, incl - mine, u * kWarps + wid);
                if (!((entry[u] >> lane) & 1u)) continue;
                const int64_t to = slot + before + __popc(entry[u] & ((1u << lane) - 1u));
                if (to < cap) {
                    a.col[to] = var[u];
                    a.val[to] = -w[u];
                }
            }
            slot += __shfl_sync(0xffffffffu, incl, 31);
            if (adds) {
                const int p0 = max(s_pin[row], pc) - pc, p1 = min(s_pin[row + 1], pc + pins) - pc;
                if (p0 < p1) {
                    const int j0 = max(s_edge[p0], c0) - c0;
                    const int j1 = min(p1 < pins ? s_edge[p1] : edges, c0 + kFillEdges) - c0;
                    const double *src = tid < kFillRows ? s_w : s_term;
                    for (int j = j0; j < j1; ++j) sum += src[j];
                }
            }
            __syncthreads();
        }
        __syncthreads();
    }
    if (!adds) return;
    const int32_t i = i0 + row;
    const bool diag = tid < kFillRows;
    if (R == kKraftwerk2) {
        if (diag) a.diag[i] = sum;
        else a.rhs[i] = alpha < 0.0 ? 0.0 : sum;
        return;
    }
    if (alpha > 0.0) {
        const double w = alpha / ref_max(fabs(s_pos[row] - a.anchor[i]), a.floor_len);
        sum += diag ? w : w * a.anchor[i];
    }
    if (diag) a.diag[i] = ref_max(sum, 1e-12);
    else a.rhs[i] = sum;
}

// Kraftwerk2's adjustments after buildSystem: diag += move_weight and
// rhs = -move_weight * toward (kraftwerk2_placer.cc:716-721) when
// move_weight is given, then diag = max(diag, floor) when floor > 0
// (kraftwerk2_placer.cc:433-437).
__global__ void k_kw2_adjust(int32_t n, double *dx, double *rx, double *dy, double *ry,
                             const double *mw, const double *tx, const double *ty, double floor) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double a = dx[i], b = dy[i];
    if (mw) {
        a += mw[i];
        b += mw[i];
        rx[i] = -mw[i] * tx[i];
        ry[i] = -mw[i] * ty[i];
    }
    if (floor > 0.0) {
        a = ref_max(a, floor);
        b = ref_max(b, floor);
    }
    dx[i] = a;
    dy[i] = b;
}


template <int R>
int launch_build(ktg_ctx *c, const double *x, const double *y, double alpha, const double *ax,
                 const double *ay, double floor_x, double floor_y) {
    const NetlistDev nl = view_of(c);
    const int32_t n = static_cast<int32_t>(c->n);
    const int net_blocks = static_cast<int>((c->N + kBuildThreads - 1) / kBuildThreads);
    const int32_t bpa = static_cast<int32_t>((c->n + kBuildThreads - 1) / kBuildThreads);
    KTG_CUDA(c, cudaMemsetAsync(c->status, 0, sizeof(int), c->stream));
    if (c->N > 0) {
        k_bound_pins<true, R><<<net_blocks, kBuildThreads, 0, c->stream>>>(
            nl, x, y, c->sys[0].bound, c->sys[1].bound, c->partials,
            c->counters + 0, c->scalars + 0);
        ++c->launches;
    } else {
        KTG_CUDA(c, cudaMemsetAsync(c->scalars + 0, 0, sizeof(double), c->stream));
    }
    AxisArgs a[2];
    for (int axis = 0; axis < 2; ++axis) {
        ktg::AxisSystem &s = c->sys[axis];
        a[axis] = AxisArgs{axis ? y : x, axis ? c->fixed_y : c->fixed_x, axis ? c->off_y : c->off_x,
                           s.bound, axis ? floor_y : floor_x, axis ? ay : ax,
                           s.row_ptr, s.col, s.val, s.diag, s.rhs};
    }
    if (n > 0) {
        k_row_count<R><<<2 * bpa, kBuildThreads * kCountLanes, 0, c->stream>>>(
            nl, a[0], a[1], bpa, c->row_cnt, c->block_sum);
        k_scan_blocks<<<1, 1024, 0, c->stream>>>(c->block_sum, bpa, n, c->cap_nnz,
                                                 c->sys[0].row_ptr, c->sys[1].row_ptr,
                                                 c->nnz_dev, c->status);
        const int32_t gpa = (n + kFillRows - 1) / kFillRows;
        k_fill<R><<<2 * gpa, kBuildThreads, 0, c->stream>>>(nl, a[0], a[1], bpa, gpa, alpha,
                                                            c->row_cnt, c->block_sum, c->cap_nnz,
                                                            c->status);
        c->launches += 3;
    } else {
        KTG_CUDA(c, cudaMemsetAsync(c->sys[0].row_ptr, 0, sizeof(int32_t), c->stream));
        KTG_CUDA(c, cudaMemsetAsync(c->sys[1].row_ptr, 0, sizeof(int32_t), c->stream));
        KTG_CUDA(c, cudaMemsetAsync(c->nnz_dev, 0, 2 * sizeof(int64_t), c->stream));
    }
    KTG_CUDA(c, cudaGetLastError());
    return KTG_OK;
}

}  // namespace

int launch_build_b2b(ktg_ctx *c, const double *x, const double *y, double alpha,
                     const double *ax, const double *ay, double floor_x, double floor_y) {
    return launch_build<kSimpl>(c, x, y, alpha, ax, ay, floor_x, floor_y);
}

int launch_build_kraftwerk2(ktg_ctx *c, const double *x, const double *y, bool with_rhs,
                            double floor_x, double floor_y) {
    return launch_build<kKraftwerk2>(c, x, y, with_rhs ? 0.0 : -1.0, nullptr, nullptr, floor_x,
                                     floor_y);
}

int launch_kraftwerk2_adjust(ktg_ctx *c, const double *move_weight, const double *toward_x,
                             const double *toward_y, double diag_floor) {
    const int32_t n = static_cast<int32_t>(c->sys_n);
    if (n == 0) return KTG_OK;
    k_kw2_adjust<<<(n + 255) / 256, 256, 0, c->stream>>>(n, c->sys[0].diag, c->sys[0].rhs,
                                                        c->sys[1].diag, c->sys[1].rhs,
                                                        move_weight, toward_x, toward_y,
                                                        diag_floor);
    ++c->launches;
    KTG_CUDA(c, cudaGetLastError());
    return KTG_OK;
}

int launch_hpwl(ktg_ctx *c, const double *x, const double *y, double *out_dev) {
    if (c->N == 0) {
        KTG_CUDA(c, cudaMemsetAsync(out_dev, 0, sizeof(double), c->stream));
        return KTG_OK;
    }
    const NetlistDev nl = view_of(c);
    const int net_blocks = static_cast<int>((c->N + kBuildThreads - 1) / kBuildThreads);
    if (c->hpwl_order == 2) {
        if (c->hpwl_terms_cap < c->N) {
            if (c->hpwl_terms) cudaFree(c->hpwl_terms);
            c->hpwl_terms = nullptr;
            KTG_CUDA(c, cudaMalloc(&c->hpwl_terms, sizeof(double) * c->N));
            c->hpwl_terms_cap = c->N;
        }
        k_bound_pins<false><<<net_blocks, kBuildThreads, 0, c->stream>>>(
            nl, x, y, nullptr, nullptr, c->partials, c->counters + 0, out_dev,
            c->hpwl_terms);
        k_hpwl_ref_order<<<1, 1024, 0, c->stream>>>(c->hpwl_terms, c->N, out_dev);
        c->launches += 2;
        KTG_CUDA(c, cudaGetLastError());
        return KTG_OK;
    }
    k_bound_pins<false><<<net_blocks, kBuildThreads, 0, c->stream>>>(
        nl, x, y, nullptr, nullptr, c->partials, c->counters + 0, out_dev);
    ++c->launches;
    KTG_CUDA(c, cudaGetLastError());
    return KTG_OK;
}

}  // namespace ktg
