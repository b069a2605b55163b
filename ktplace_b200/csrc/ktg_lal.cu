// Look-ahead legalization on the GPU (sm_100a).
//
// Replaces LookAheadLegalizer::legalize (globalPlacer/simpl/simpl_lal.cc:
// 43-372) with the BinGrid / FreeSpace / AxisProfile arithmetic of
// globalPlacer/simpl/simpl_grid.h, bit for bit:
//
//   host   the cluster loop, which is sequential in the reference: bins of
//          the cell centres and their occupancy (ktg's fixed-point occupancy
//          kernel, exact for the integer site areas of row-based designs),
//          overfilled clusters (4-neighbour flood fill from the lowest bin),
//          growth by the least dense of four one-bin extensions, batches of
//          regions whose one-bin reaches do not touch -- all with the
//          reference's summation order over the host copy of the grid;
//   device each batch: the regions' cells, then the recursive bisection
//          level by level over every block of the batch at once:
//            * cells sorted by (centre, index): tiles of 2048 keys in
//              shared memory, then merge passes;
//            * per block: cell area and the area median m (from an exact
//              prefix), the free-space profile of the box (vertical: row
//              spans as sorted (x, +-h) steps, running sums), the cutline and
//              the two half boxes;
//            * per half: its profile, the stripes (obstacle edges, unique,
//              midpoint splits above stripeAreaFraction of the region's room)
//              in the reference's distance-from-cut order;
//            * cells by (-distance from the cut, index): the centre order, or
//              its reverse; stripes filled greedily in that order;
//            * per stripe the lowest / highest centre, then every cell's new
//              position;
//            * children: the low and high cells, next axis.
//            The host knows the boxes and the free space, so it bounds the
//            profiles and stripes itself: one copy in and one wait per level
//            (0.25 to 0.35 ms; it took 0.8 with six waits, 15 copies, a bitonic
//            sort of 70 us and a second sort for the fill order).
//          then the bins and occupancy of all cells again for the host.
//
// The sorts are key-only over 16-byte keys: (order bits of a double, index)
// for cells and (order bits of x, order bits of dh) for profile steps; tiles of
// kSub keys are sorted by one CTA each in shared memory, longer segments by
// merge passes over them.
#include "ktg_common.cuh"
#include "ktg_context.h"

#include <algorithm>
#include <array>
#include <chrono>
#include <cmath>
#include <cstring>
#include <limits>
#include <utility>
#include <vector>

namespace ktg {

namespace {

constexpr int kT = 256;

struct Key {
    unsigned long long a, b;
};

__device__ __forceinline__ bool key_lt(const Key &x, const Key &y) {
    return x.a < y.a || (x.a == y.a && x.b < y.b);
}

// Order-preserving bits of a double; -0.0 counts as +0.0 (the reference's
// comparisons treat them as equal).
__device__ __forceinline__ unsigned long long ord(double v) {
    const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v + 0.0));
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

__device__ __forceinline__ double unord(unsigned long long u) {
    const unsigned long long r = (u >> 63) ? (u & 0x7fffffffffffffffull) : ~u;
    return __longlong_as_double(static_cast<long long>(r));
}

// ---- segmented key sort ---------------------------------------------------------

int blocks_for(int64_t items, int threads = kT) {
    return static_cast<int>(std::max<int64_t>(1, (items + threads - 1) / threads));
}

template <typename T>
struct DevBuf {
    T *p = nullptr;
    int64_t cap = 0;
    int ensure(ktg_ctx *c, int64_t n) {
        if (n <= cap) return KTG_OK;
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
        const int64_t want = std::max<int64_t>(n + n / 4, 64);
        if (cudaMalloc(&p, sizeof(T) * want) != cudaSuccess)
            return set_error(c, KTG_ERR_NOMEM, "out of device memory (legalization)");
        cap = want;
        return KTG_OK;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    }
};

// ---- free space -----------------------------------------------------------------

struct Free {
    const double *rowy;      // [2R] y start, y end (rows sorted by y start)
    const int64_t *rowspan;  // [R+1]
    const double *spans;     // [2S] x start, x end
    const double *obst;      // [4K] lx ly ux uy
    int32_t R, K;
};

// First row with ly < y.end (std::upper_bound with v < r.y.end).
__device__ __forceinline__ int32_t first_row(const Free &F, double ly) {
    int32_t lo = 0, hi = F.R;
    while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if (ly < F.rowy[2 * mid + 1]) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// First span of row r ending after x (spans of a row ascend and are
// disjoint, FreeSpace::build).
__device__ __forceinline__ int64_t first_span(const Free &F, int32_t r, double x) {
    int64_t lo = F.rowspan[r], hi = F.rowspan[r + 1];
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (F.spans[2 * mid + 1] > x) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// Rows [r0, r1) a box's row loops visit (rows sorted by y start).
__device__ __forceinline__ void box_rows(const Free &F, const double *box, int32_t &r0,
                                         int32_t &r1) {
    r0 = first_row(F, box[1]);
    int32_t lo = r0, hi = F.R;
    while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if (F.rowy[2 * mid] < box[3]) lo = mid + 1;
        else hi = mid;
    }
    r1 = lo;
}

// Steps of row r inside box (emit_steps restricted to one row), written
// through sink(k + i, x, dh); returns their count.
template <typename Sink>
__device__ __forceinline__ int64_t row_steps(const Free &F, int32_t r, const double *box, Sink sink,
                                             int64_t k) {
    const double lx = box[0], ly = box[1], ux = box[2], uy = box[3];
    const double h = ref_min(uy, F.rowy[2 * r + 1]) - ref_max(ly, F.rowy[2 * r]);
    if (!(h > 0.0)) return 0;
    const int64_t end = F.rowspan[r + 1];
    int64_t c = 0;
    for (int64_t s = first_span(F, r, lx); s < end && F.spans[2 * s] < ux; ++s) {
        const double a = ref_max(F.spans[2 * s], lx);
        const double z = ref_min(F.spans[2 * s + 1], ux);
        if (z > a) {
            sink(k + c, a, h);
            sink(k + c + 1, z, -h);
            c += 2;
        }
    }
    return c;
}

// AxisProfile (simpl_grid.h:29-65, getProfile :179-232) stored as edges /
// prefix arrays of `n` entries.
struct Prof {
    const double *e;
    const double *p;
    int64_t n;
    __device__ double total() const { return p[n - 1]; }
    __device__ double before(double c) const {
        if (c <= e[0]) return 0.0;
        if (c >= e[n - 1]) return total();
        int64_t lo = 0, hi = n;  // upper_bound
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (c < e[mid]) hi = mid;
            else lo = mid + 1;
        }
        const int64_t k = lo - 1;
        const double f = (c - e[k]) / (e[k + 1] - e[k]);
        return p[k] + f * (p[k + 1] - p[k]);
    }
    __device__ double coordinate_at(double target) const {
        if (target <= 0.0) return e[0];
        if (target >= total()) return e[n - 1];
        int64_t lo = 0, hi = n;  // lower_bound on prefix
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (p[mid] < target) lo = mid + 1;
            else hi = mid;
        }
        const int64_t k = lo;
        const double step = p[k] - p[k - 1];
        const double f = step > 0.0 ? (target - p[k - 1]) / step : 1.0;
        return e[k - 1] + f * (e[k] - e[k - 1]);
    }
};

// Builds the profile of `box` into e/p from its sorted steps (vertical;
// step(k, at, dh) reads the k-th) or the rows (horizontal); returns the
// number of edges.
template <typename Step>
__device__ int64_t build_profile_from(const Free &F, const double *box, bool vertical, Step step,
                                      int64_t nsteps, double *e, double *p) {
    const double lx = box[0], ly = box[1], ux = box[2], uy = box[3];
    const double lo = vertical ? lx : ly, hi = vertical ? ux : uy;
    int64_t n = 1;
    e[0] = lo;
    p[0] = 0.0;
    auto extend = [&](double to, double area) {
        if (to > e[n - 1]) {
            e[n] = to;
            p[n] = p[n - 1] + area;
            ++n;
        }
    };
    if (vertical) {
        double height = 0.0;
        for (int64_t k = 0; k < nsteps; ++k) {
            double at, dh;
            step(k, at, dh);
            extend(at, height * (at - e[n - 1]));
            height += dh;
        }
    } else {
        for (int32_t r = first_row(F, ly); r < F.R && F.rowy[2 * r] < uy; ++r) {
            const double a = ref_max(lo, F.rowy[2 * r]);
            const double z = ref_min(hi, F.rowy[2 * r + 1]);
            if (z > a) {
                extend(a, 0.0);
                // Row::getLength(b.getX()); spans outside [lx, ux] add +0.0
                double total = 0.0;
                const int64_t end = F.rowspan[r + 1];
                for (int64_t s = first_span(F, r, lx); s < end && F.spans[2 * s] < ux; ++s)
                    total += ref_max(0.0, ref_min(ux, F.spans[2 * s + 1]) - ref_max(lx, F.spans[2 * s]));
                extend(z, total * (z - a));
            }
        }
    }
    extend(hi, 0.0);
    if (n == 1) {
        e[1] = hi;
        p[1] = 0.0;
        n = 2;
    }
    return n;
}

// getStripes (simpl_lal.cc:266-312) for one half box, then the stable sort
// of nonlinearScale (:325-328) by distance from the cutline, farthest first.
// The reference inserts each midpoint split into its cut list and steps on;
// that visits the intervals depth first, which a small stack does here with
// the same operations (room.getBetween(a, b) = before(b) - before(a), each
// before() computed once). The stripes come out in ascending position, so
// their distance from the cut is monotone: below the cut the stable
// descending order is the order itself, above it the runs of equal distance
// in reverse with each run kept in order. `cuts` is scratch of `cap` doubles;
// the stripes' spans and capacities go to sa/sb/scap. Returns the number of
// stripes, or -1 when `cap` (or the split depth) is exceeded.
__device__ int64_t make_stripes(const Prof &room, const double *box, bool v, double cell_area,
                                double region_room, double frac, double limit_density,
                                const double *obst, int32_t K, double cutline, bool below,
                                double *cuts, int64_t cap, double *sa, double *sb, double *scap) {
    constexpr int kLocalCuts = 64;
    constexpr int kDepth = 64;
    const double lo = v ? box[0] : box[1], hi = v ? box[2] : box[3];
    double lc[kLocalCuts];  // small cut lists are sorted in (L1-resident) local memory
    int64_t nc = 0;
    bool local = true;
    auto put = [&](double x) {
        if (local && nc < kLocalCuts) {
            lc[nc++] = x;
            return;
        }
        if (local) {
            for (int64_t i = 0; i < nc; ++i) cuts[i] = lc[i];
            local = false;
        }
        cuts[nc++] = x;
    };
    put(lo);
    put(hi);
    for (int32_t o = 0; o < K; ++o) {
        const double *ob = obst + 4 * o;
        if (ob[2] <= box[0] || ob[0] >= box[2] || ob[3] <= box[1] || ob[1] >= box[3]) continue;
        const double e0 = v ? ob[0] : ob[1], e1 = v ? ob[2] : ob[3];
        if (nc + 2 > cap) return -1;
        if (e0 > lo && e0 < hi) put(e0);
        if (e1 > lo && e1 < hi) put(e1);
    }
    double *c = local ? lc : cuts;
    for (int64_t i = 1; i < nc; ++i) {  // insertion sort (stable)
        const double t = c[i];
        int64_t j = i - 1;
        while (j >= 0 && t < c[j]) {
            c[j + 1] = c[j];
            --j;
        }
        c[j + 1] = t;
    }
    int64_t u = 0;
    for (int64_t i = 0; i < nc; ++i)
        if (u == 0 || !(c[u - 1] == c[i])) c[u++] = c[i];
    nc = u;
    const double limit = frac * (region_room > 0.0 ? region_room : room.total());
    const double fill = room.total() > 0.0 ? ref_min(limit_density, cell_area / room.total())
                                           : limit_density;
    int64_t ns = 0;
    double a = c[0], ba = room.before(a);
    double stk[kDepth], stkb[kDepth];
    for (int64_t i = 1; i < nc; ++i) {
        int top = 0;
        stk[top] = c[i];
        stkb[top] = room.before(c[i]);
        ++top;
        while (top > 0) {
            const double b = stk[top - 1], bb = stkb[top - 1];
            const double here = bb - ba;
            const double mid = room.coordinate_at(ba + 0.5 * here);
            if (here > limit && mid > a && mid < b) {
                if (top == kDepth || ns + top + 1 > cap) return -1;
                stk[top] = mid;
                stkb[top] = room.before(mid);
                ++top;
            } else {
                if (ns >= cap) return -1;
                sa[ns] = a;
                sb[ns] = b;
                scap[ns] = fill * here;
                ++ns;
                --top;
                a = b;
                ba = bb;
            }
        }
    }
    if (!below) {
        auto swap_at = [&](int64_t i, int64_t j) {
            double t = sa[i]; sa[i] = sa[j]; sa[j] = t;
            t = sb[i]; sb[i] = sb[j]; sb[j] = t;
            t = scap[i]; scap[i] = scap[j]; scap[j] = t;
        };
        for (int64_t i = 0, j = ns - 1; i < j; ++i, --j) swap_at(i, j);
        for (int64_t r = 0; r < ns;) {  // restore the original order inside each run
            const double f = 0.5 * (sa[r] + sb[r]) - cutline;
            int64_t e = r + 1;
            while (e < ns && 0.5 * (sa[e] + sb[e]) - cutline == f) ++e;
            for (int64_t i = r, j = e - 1; i < j; ++i, --j) swap_at(i, j);
            r = e;
        }
    }
    return ns;
}

// ---- sorting -------------------------------------------------------------------------

constexpr int kSub = 2048;         // entries a CTA sorts in shared memory
constexpr int kSubThreads = 512;

// Where entry i of a buffer of 8- or 4-byte entries lies while it is merged: a
// thread's four outputs are consecutive, and unswizzled its 8-byte accesses
// would meet seven other lanes' banks.
template <typename V>
__device__ __forceinline__ int swizzled(int i) {
    return sizeof(V) == 8 ? i ^ ((i >> 4) & 15) : i ^ ((i >> 5) & 31);
}

// Sorts positions [0, tot), tot <= kSub, by (tag, key, val) with the whole CTA:
// four entries per thread sorted in registers, then merges of sorted runs, each
// thread finding its four outputs by a binary search along the merge path. tag
// ascends with the position, so entries move only among equal tags and every
// position keeps its tag; without Tags it is one segment. load(p, key, val)
// gives the entries; key and val have room for 2 kSub and end with the sorted
// ones in [0, tot).
template <bool Tags, typename V, class Load>
__device__ void merge_sort(unsigned long long *key, V *val, uint32_t *tag, int tot, Load load) {
    int P = 4, levels = 0;
    while (P < tot) P <<= 1, ++levels;
    int buf = levels & 1;
    const int p0 = 4 * threadIdx.x;
    const bool on = p0 < P;
    auto less_eq = [&](uint32_t ti, unsigned long long ki, V vi, uint32_t tj, unsigned long long kj,
                       V vj) {
        const bool le = (ki < kj) | ((ki == kj) & (vi <= vj));
        return Tags ? (ti < tj) | ((ti == tj) & le) : le;
    };
    unsigned long long k[4];
    V v[4];
    uint32_t t[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        k[u] = ~0ull;
        v[u] = static_cast<V>(~0ull);
        t[u] = 0u;
        if (p0 + u < tot) load(p0 + u, k[u], v[u]);
        else if (Tags && on) tag[p0 + u] = ~0u;
        if (Tags && on) t[u] = tag[p0 + u];
    }
    __syncwarp();  // all loaded before the first is stored: load may read key and val
    if (on) {
        auto cas = [&](int i, int j) {
            if (t[i] == t[j] && (k[j] < k[i] || (k[j] == k[i] && v[j] < v[i]))) {
                const unsigned long long x = k[i];
                k[i] = k[j];
                k[j] = x;
                const V y = v[i];
                v[i] = v[j];
                v[j] = y;
            }
        };
        cas(0, 1);
        cas(2, 3);
        cas(0, 2);
        cas(1, 3);
        cas(1, 2);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = p0 + u;
            key[buf * kSub + (levels ? swizzled<unsigned long long>(i) : i)] = k[u];
            val[buf * kSub + (levels ? swizzled<V>(i) : i)] = v[u];
        }
    }
    for (int w = 4; w < P; w <<= 1, buf ^= 1) {
        if (w >= 128) __syncthreads();  // up to there a warp merges its own entries
        else __syncwarp();
        if (!on) continue;
        const unsigned long long *sk = key + buf * kSub;
        const V *sv = val + buf * kSub;
        unsigned long long *dk = key + (buf ^ 1) * kSub;
        V *dv = val + (buf ^ 1) * kSub;
        auto kat = [&](int i) { return sk[swizzled<unsigned long long>(i)]; };
        auto vat = [&](int i) { return sv[swizzled<V>(i)]; };
        auto tat = [&](int i) { return Tags ? tag[i] : 0u; };
        const int base = p0 & ~(2 * w - 1), d = p0 - base;
        int lo = max(0, d - w), hi = min(d, w);
        while (lo < hi) {
            const int mid = (lo + hi) >> 1, i = base + mid, j = base + w + d - 1 - mid;
            if (less_eq(tat(i), kat(i), vat(i), tat(j), kat(j), vat(j))) lo = mid + 1;
            else hi = mid;
        }
        int i = base + lo, j = base + w + d - lo;
        const int ei = base + w, ej = base + 2 * w;
        unsigned long long ki = 0, kj = 0;
        V vi = 0, vj = 0;
        uint32_t ti = 0u, tj = 0u;
        if (i < ei) ki = kat(i), vi = vat(i), ti = tat(i);
        if (j < ej) kj = kat(j), vj = vat(j), tj = tat(j);
        const bool last = 2 * w == P;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool left = j >= ej || (i < ei && less_eq(ti, ki, vi, tj, kj, vj));
            const int q = p0 + u;
            dk[last ? q : swizzled<unsigned long long>(q)] = left ? ki : kj;
            dv[last ? q : swizzled<V>(q)] = left ? vi : vj;
            if (left) {
                if (++i < ei) ki = kat(i), vi = vat(i), ti = tat(i);
            } else {
                if (++j < ej) kj = kat(j), vj = vat(j), tj = tat(j);
            }
        }
    }
    __syncthreads();
}

// The segments of a sort: positions [b, e) (cells) or n entries from off.
struct Segs {
    const int32_t *b, *e;
    const int64_t *off, *n;
    __device__ int64_t begin(int i) const { return b ? b[i] : off[i]; }
    __device__ int64_t size(int i) const { return b ? e[i] - b[i] : n[i]; }
};

constexpr size_t kTileSmem = sizeof(unsigned long long) * 4 * kSub;

// Sorts tiles of kSub keys of every segment, in place: 17 us a tile (a bitonic
// network over 16-byte keys took 70).
__global__ void __launch_bounds__(kSubThreads) k_sort_tiles(Key *keys, Segs sg, int nseg) {
    extern __shared__ __align__(16) unsigned long long tile[];
    for (int i = blockIdx.y; i < nseg; i += gridDim.y) {
        const int64_t c0 = static_cast<int64_t>(blockIdx.x) * kSub, n = sg.size(i);
        if (c0 >= n) continue;
        Key *k = keys + sg.begin(i) + c0;
        const int tot = static_cast<int>(n - c0 < kSub ? n - c0 : kSub);
        unsigned long long *sa = tile, *sb = tile + 2 * kSub;
        merge_sort<false>(sa, sb, nullptr, tot,
                          [&](int p, unsigned long long &a, unsigned long long &b) {
                              a = k[p].a;
                              b = k[p].b;
                          });
        for (int p = threadIdx.x; p < tot; p += blockDim.x) k[p] = Key{sa[p], sb[p]};
        __syncthreads();
    }
}

// Entries that the first d of the merged runs A (la) and B (lb) take from A;
// a warp, 32 probes a round.
__device__ int64_t warp_merge_path(const Key *A, int64_t la, const Key *B, int64_t lb, int64_t d) {
    const int lane = threadIdx.x & 31;
    int64_t lo = d > lb ? d - lb : 0, hi = d < la ? d : la;
    while (lo < hi) {
        const int64_t step = (hi - lo + 31) / 32, i = lo + lane * step;
        const int c = __popc(__ballot_sync(0xffffffffu, i < hi && !key_lt(B[d - 1 - i], A[i])));
        const int64_t end = lo + c * step;
        if (c < 32 && end < hi) hi = end;
        if (c > 0) lo += (c - 1) * step + 1;
    }
    return lo;
}

// One merge pass: runs of `run` keys of every segment merged pairwise, kSub
// outputs per CTA through shared memory.
__global__ void __launch_bounds__(kSubThreads) k_merge_tiles(const Key *src, Key *dst, Segs sg,
                                                             int nseg, int64_t run) {
    extern __shared__ __align__(16) unsigned long long tile[];
    __shared__ int64_t s_split[2];
    unsigned long long *sa = tile, *sb = tile + kSub;
    for (int i = blockIdx.y; i < nseg; i += gridDim.y) {
        const int64_t c0 = static_cast<int64_t>(blockIdx.x) * kSub, n = sg.size(i);
        if (c0 >= n) continue;
        const int64_t base = c0 / (2 * run) * (2 * run);
        const int64_t la = n - base < run ? n - base : run;
        const int64_t lb = n - base - la < run ? n - base - la : run;
        const Key *A = src + sg.begin(i) + base, *B = A + la;
        Key *out = dst + sg.begin(i) + c0;
        const int64_t d0 = c0 - base, d1 = d0 + kSub < la + lb ? d0 + kSub : la + lb;
        const int warp = threadIdx.x >> 5;
        if (warp < 2) {
            const int64_t x = warp_merge_path(A, la, B, lb, warp ? d1 : d0);
            if ((threadIdx.x & 31) == 0) s_split[warp] = x;
        }
        __syncthreads();
        const int64_t i0 = s_split[0], j0 = d0 - i0;
        const int na = static_cast<int>(s_split[1] - i0), tot = static_cast<int>(d1 - d0);
        auto at = [](int q) { return swizzled<unsigned long long>(q); };
        for (int q = threadIdx.x; q < tot; q += blockDim.x) {
            const Key k = q < na ? A[i0 + q] : B[j0 + q - na];
            sa[at(q)] = k.a;
            sb[at(q)] = k.b;
        }
        __syncthreads();
        const int nb = tot - na, d = 4 * threadIdx.x;
        auto key = [&](int q) { return Key{sa[at(q)], sb[at(q)]}; };
        if (d < tot) {
            int lo = max(0, d - nb), hi = min(d, na);
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (!key_lt(key(na + d - 1 - mid), key(mid))) lo = mid + 1;
                else hi = mid;
            }
            int x = lo, y = na + d - lo;
            Key kx = x < na ? key(x) : Key{0ull, 0ull}, ky = y < tot ? key(y) : Key{0ull, 0ull};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (d + u >= tot) break;
                const bool left = y >= tot || (x < na && !key_lt(ky, kx));
                out[d + u] = left ? kx : ky;
                if (left) {
                    if (++x < na) kx = key(x);
                } else {
                    if (++y < tot) ky = key(y);
                }
            }
        }
        __syncthreads();
    }
}

// Sorts the segments (the longest of at most `maxlen` keys); the sorted keys
// are in *sorted, keys or tmp.
int sort_segs(ktg_ctx *c, Key *keys, Key *tmp, const Segs &sg, int nseg, int64_t maxlen,
              Key **sorted) {
    *sorted = keys;
    if (nseg == 0 || maxlen <= 1) return KTG_OK;
    const dim3 grid(static_cast<unsigned>((maxlen + kSub - 1) / kSub), std::min(nseg, 65535));
    k_sort_tiles<<<grid, kSubThreads, kTileSmem, c->stream>>>(keys, sg, nseg);
    ++c->launches;
    Key *src = keys, *dst = tmp;
    for (int64_t run = kSub; run < maxlen; run *= 2) {
        k_merge_tiles<<<grid, kSubThreads, kTileSmem / 2, c->stream>>>(src, dst, sg, nseg, run);
        ++c->launches;
        std::swap(src, dst);
    }
    *sorted = src;
    KTG_CUDA(c, cudaGetLastError());
    return KTG_OK;
}

// ---- per-level kernels --------------------------------------------------------------

struct CellsDev {
    double *x, *y;
    const double *w, *h, *area;
};

__device__ __forceinline__ double centre(const CellsDev &C, int32_t i, bool vertical) {
    return vertical ? C.x[i] + 0.5 * C.w[i] : C.y[i] + 0.5 * C.h[i];
}

struct Level {
    int32_t na;
    const int32_t *b, *e;  // cell ranges of the active blocks
    const double *box;     // [4 na]
    const int32_t *vert;
    const double *room;
    // results
    int32_t *m;
    double *low_area, *high_area, *cut;
    double *half_box;      // [8 na]: low box, high box
    int32_t *redo;         // set by k_fill_order: nothing filled or placed yet
};

// The per-cell kernels below run on a 2-D grid: y strides over the active
// blocks, x over the cells of one block.
__global__ void k_centre_keys(Level L, CellsDev C, const int32_t *cells, Key *keys) {
    for (int32_t blk = blockIdx.y; blk < L.na; blk += gridDim.y) {
        const int32_t b = L.b[blk], e = L.e[blk];
        const bool v = L.vert[blk] != 0;
        for (int32_t p = b + blockIdx.x * blockDim.x + threadIdx.x; p < e; p += gridDim.x * blockDim.x) {
            const int32_t i = cells[p];
            keys[p] = Key{ord(centre(C, i, v)), static_cast<unsigned long long>(i)};
        }
    }
}

__global__ void k_keys_to_cells(Level L, const Key *keys, int32_t *cells) {
    for (int32_t blk = blockIdx.y; blk < L.na; blk += gridDim.y)
        for (int32_t p = L.b[blk] + blockIdx.x * blockDim.x + threadIdx.x; p < L.e[blk];
             p += gridDim.x * blockDim.x)
            cells[p] = static_cast<int32_t>(keys[p].b);
}

// ---- exact area sums ------------------------------------------------------------
//
// When every cell area is a multiple of 2^-q and the total times 2^q stays
// below 2^52, every partial sum the reference forms (cellArea, lowArea, a
// stripe's used area) is exact in double, whatever the order. The sums are
// then read off an integer prefix over the positions: pre[p] = fixed-point
// area of positions [0, p).

constexpr int kScanTile = 2048;  // positions per tile: kT threads x 8

__device__ __forceinline__ long long area_fx(const double *area, int32_t i, double scale) {
    return __double2ll_rn(area[i] * scale);
}

__device__ __forceinline__ long long warp_incl64(long long v) {
    const int lane = threadIdx.x & 31;
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive block scan of one value per thread (blockDim.x == kT); returns
// the exclusive prefix and sets `total`.
__device__ long long block_excl64(long long v, long long &total) {
    __shared__ long long ws[kT / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long inc = warp_incl64(v);
    if (lane == 31) ws[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        long long w = lane < kT / 32 ? ws[lane] : 0;
        w = warp_incl64(w);
        if (lane < kT / 32) ws[lane] = w;
    }
    __syncthreads();
    const long long out = inc - v + (wid > 0 ? ws[wid - 1] : 0);
    total = ws[kT / 32 - 1];
    __syncthreads();
    return out;
}

__global__ void __launch_bounds__(kT) k_fx_tile_sums(const int32_t *cells, const double *area,
                                                     int32_t n, double scale, long long *tile) {
    const int32_t base = blockIdx.x * kScanTile;
    long long v = 0;
    for (int k = threadIdx.x; k < kScanTile; k += kT)
        if (base + k < n) v += area_fx(area, cells[base + k], scale);
    long long total;
    block_excl64(v, total);
    if (threadIdx.x == 0) tile[blockIdx.x] = total;
}

// Exclusive scan of the tile sums in place (one block).
__global__ void __launch_bounds__(kT) k_fx_tile_scan(long long *tile, int32_t ntiles) {
    const int per = (ntiles + kT - 1) / kT;
    const int beg = threadIdx.x * per, end = min(beg + per, ntiles);
    long long v = 0;
    for (int i = beg; i < end; ++i) v += tile[i];
    long long total;
    long long run = block_excl64(v, total);
    for (int i = beg; i < end; ++i) {
        const long long t = tile[i];
        tile[i] = run;
        run += t;
    }
}

// pre[p + 1] = fixed-point area of positions [0, p]; pre[0] = 0.
__global__ void __launch_bounds__(kT) k_fx_prefix(const int32_t *cells, const double *area,
                                                  int32_t n, double scale, const long long *tile,
                                                  long long *pre) {
    const int32_t base = blockIdx.x * kScanTile + threadIdx.x * (kScanTile / kT);
    long long v[kScanTile / kT];
    long long sum = 0;
#pragma unroll
    for (int k = 0; k < kScanTile / kT; ++k) {
        v[k] = base + k < n ? area_fx(area, cells[base + k], scale) : 0;
        sum += v[k];
    }
    long long total;
    long long run = block_excl64(sum, total) + tile[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanTile / kT; ++k) {
        run += v[k];
        if (base + k < n) pre[base + k + 1] = run;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) pre[0] = 0;
}

// Median split from the prefix: the least m >= 1 with 2 * low(m) >= total,
// at most size - 1 (the loop of split, simpl_lal.cc:230-233).
__device__ __forceinline__ int32_t median_fx(const long long *pre, int32_t b, int32_t size) {
    if (size <= 1) return 0;
    const long long tot = pre[b + size] - pre[b];
    int32_t lo = 1, hi = size - 1;  // answer in [lo, hi]
    while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if (2 * (pre[b + mid] - pre[b]) >= tot) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// median_fx by a warp.
__device__ int32_t warp_median_fx(const long long *pre, int32_t b, int32_t size) {
    if (size <= 1) return 0;
    const int lane = threadIdx.x & 31;
    const long long first = pre[b], tot = pre[b + size] - first;
    int32_t lo = 1, hi = size - 1;  // answer in [lo, hi]
    while (lo < hi) {
        const int32_t step = (hi - lo + 31) / 32, i = lo + lane * step;
        const bool below = i < hi && 2 * (pre[b + i] - first) < tot;  // answer past i
        const int c = __popc(__ballot_sync(0xffffffffu, below));
        const int32_t end = lo + c * step;
        if (c < 32 && end < hi) hi = end;
        if (c > 0) lo += (c - 1) * step + 1;
    }
    return lo;
}

// Areas and median of every block: from the exact prefix by a warp (32 probes a
// round), or in the reference's order by one thread.
__global__ void k_block_split(Level L, CellsDev C, const int32_t *cells, const long long *pre,
                              double inv_scale) {
    const int32_t blk = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (blk >= L.na) return;
    const int32_t b = L.b[blk], e = L.e[blk];
    const int32_t size = e - b;
    double cell_area = 0.0, low = 0.0, high = 0.0;
    int32_t m = 0;
    if (pre) {
        m = warp_median_fx(pre, b, size);
        cell_area = static_cast<double>(pre[e] - pre[b]) * inv_scale;
        low = static_cast<double>(pre[b + m] - pre[b]) * inv_scale;
        high = static_cast<double>(pre[e] - pre[b + m]) * inv_scale;
    } else if (lane == 0) {
        for (int32_t p = b; p < e; ++p) cell_area += C.area[cells[p]];
        while (m + 1 < size && (m == 0 || low < 0.5 * cell_area)) low += C.area[cells[b + m++]];
        for (int32_t p = b + m; p < e; ++p) high += C.area[cells[p]];
    }
    if (lane != 0) return;
    if (blk == 0) *L.redo = 0;
    L.m[blk] = m;
    L.low_area[blk] = low;
    L.high_area[blk] = high;
    L.cut[blk] = cell_area;  // kept until the cutline replaces it
}

struct Stripes {
    int64_t *off;    // [2 na] first stripe of the half (into the arrays below)
    int32_t *count;  // [2 na]
    double *a, *b, *cap, *used;
    unsigned long long *lo, *hi;
};

// ---- one CTA per block (or half) for the level-by-level path ------------------------
//
// Blocks too large for the one-CTA subtree have die-sized boxes: tens of
// thousands of profile steps and hundreds of obstacles. Latency bounds these
// kernels (a level has one or a few blocks), so everything that may run in any
// order runs on all threads; what keeps the reference's order is one addition
// per profile edge, a chain of thread 0 through shared memory. With the whole
// walk (heights, edge tests, stores to global memory), the obstacle list and
// the stripe loop on thread 0, the two kernels took 470 + 140 us a level on the
// 211k-cell design.

constexpr int kWideT = 512;                   // threads of the per-block kernels
constexpr int kPer = 8;                       // profile steps per thread and round
constexpr int kRound = kWideT * kPer;         // and so edges per round at most
constexpr int kProfSmem = 6144;               // profile edges kept in shared memory
constexpr int kCutSmem = 4096;                // obstacle cuts sorted there
// profile (edges, prefix), and a round's stage (three arrays) or the cuts, their
// input order, their prefix and the stripe counts
constexpr size_t kCtaStage = sizeof(double) * 3 * kRound;
constexpr size_t kHalfStripesSmem = sizeof(double) * 2 * kProfSmem + kCtaStage;
static_assert(kCtaStage >= (2 * sizeof(double) + 2 * sizeof(int32_t)) * kCutSmem, "");

template <typename T, class Op>
__device__ T cta_excl(T v, T zero, T &total, Op op) {
    __shared__ T ws[kWideT / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    T inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const T t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc = op(t, inc);
    }
    T exc = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) exc = zero;
    if (lane == 31) ws[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        T w = lane < nw ? ws[lane] : zero;
        for (int o = 1; o < 32; o <<= 1) {
            const T t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w = op(t, w);
        }
        if (lane < nw) ws[lane] = w;
    }
    __syncthreads();
    total = ws[nw - 1];
    const T before = wid > 0 ? ws[wid - 1] : zero;
    __syncthreads();
    return op(before, exc);
}

// Running sums of area[0, cnt) onto sum in order, in place; one thread. The
// next eight terms load behind the additions.
__device__ double chain_sums(double *area, int cnt, double sum) {
    double2 *v = reinterpret_cast<double2 *>(area);  // 16-byte aligned
    const int whole = cnt >> 3;
    double2 n0, n1, n2, n3;
    if (whole) n0 = v[0], n1 = v[1], n2 = v[2], n3 = v[3];
    for (int i = 0; i < whole; ++i, v += 4) {
        double2 c0 = n0, c1 = n1, c2 = n2, c3 = n3;
        if (i + 1 < whole) n0 = v[4], n1 = v[5], n2 = v[6], n3 = v[7];
        c0.x = sum = sum + c0.x;
        c0.y = sum = sum + c0.y;
        c1.x = sum = sum + c1.x;
        c1.y = sum = sum + c1.y;
        c2.x = sum = sum + c2.x;
        c2.y = sum = sum + c2.y;
        c3.x = sum = sum + c3.x;
        c3.y = sum = sum + c3.y;
        v[0] = c0, v[1] = c1, v[2] = c2, v[3] = c3;
    }
    for (int i = whole * 8; i < cnt; ++i) area[i] = sum = sum + area[i];
    return sum;
}

// Exponent of the lowest set bit of a nonzero finite double.
__device__ __forceinline__ int low_bit(double v) {
    const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
    const int ex = static_cast<int>((u >> 52) & 0x7ff);
    const unsigned long long m = (u & 0xfffffffffffffull) | (ex ? 0x10000000000000ull : 0ull);
    return (ex ? ex : 1) - 1075 + __ffsll(static_cast<long long>(m)) - 1;
}

// Edges and areas of a round, staged; writes them out with running prefixes.
// n: edges so far; plast: the last prefix (thread 0).
__device__ void cta_flush_edges(const double *se, double *sa, int cnt, int64_t &n, double &plast,
                                double *e, double *p) {
    __syncthreads();
    if (threadIdx.x == 0) plast = chain_sums(sa, cnt, plast);
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
        e[n + i] = se[i];
        p[n + i] = sa[i];
    }
    n += cnt;
    __syncthreads();
}

// Vertical profile: the heights before each step are prefix sums of the dh.
// Exact: every dh is a multiple of 2^g and no partial sum needs more than 53
// bits above 2^g, so the reference's sequential double sums round nowhere and
// 64-bit integer sums, in any order, are the same values; checked on every
// partial sum. False (nothing usable written) when the check fails; with
// Exact = false thread 0 adds the heights in order.
template <bool Exact>
__device__ bool cta_profile_steps(double lo, const Key *steps, int64_t nsteps, int g, double *stage,
                                  int64_t &n, double &plast, double &elast, double *e, double *p) {
    double *se = stage, *sa = stage + kRound, *sh = stage + 2 * kRound;
    const double scale = Exact ? ldexp(1.0, -g) : 1.0, unit = Exact ? ldexp(1.0, g) : 1.0;
    long long carry = 0;
    double height = 0.0;  // Exact = false, thread 0
    for (int64_t c0 = 0; c0 < nsteps; c0 += kRound) {
        const int64_t k0 = c0 + static_cast<int64_t>(threadIdx.x) * kPer;
        double at[kPer], dh[kPer];
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const Key q = k0 + u < nsteps ? steps[k0 + u] : Key{0ull, 0ull};
            at[u] = unord(q.a);
            dh[u] = k0 + u < nsteps ? unord(q.b) : 0.0;
        }
        double prev = k0 > 0 && k0 < nsteps ? unord(steps[k0 - 1].a) : lo;
        bool bad = false;
        long long run = 0;
        if constexpr (Exact) {
            long long local = 0, total;
#pragma unroll
            for (int u = 0; u < kPer; ++u) local += __double2ll_rn(dh[u] * scale);
            run = carry + cta_excl<long long>(local, 0ll, total,
                                              [](long long x, long long y) { return x + y; });
            carry += total;
        } else {
#pragma unroll
            for (int u = 0; u < kPer; ++u) sh[threadIdx.x * kPer + u] = dh[u];
            __syncthreads();
            if (threadIdx.x == 0)
                for (int i = 0; i < kRound; ++i) {
                    const double d = sh[i];
                    sh[i] = height;
                    height += d;
                }
            __syncthreads();
        }
        int cnt = 0;
        double ar[kPer];
        unsigned take = 0;
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            if (k0 + u < nsteps) {
                const double h = Exact ? static_cast<double>(run) * unit : sh[threadIdx.x * kPer + u];
                if (at[u] > prev) {
                    ar[u] = h * (at[u] - prev);
                    take |= 1u << u;
                    ++cnt;
                }
                prev = at[u];
                if constexpr (Exact) {
                    run += __double2ll_rn(dh[u] * scale);
                    bad = bad || run > (1ll << 53) || run < -(1ll << 53);
                }
            }
        }
        int total_cnt;
        int at_edge = cta_excl<int>(cnt, 0, total_cnt, [](int x, int y) { return x + y; });
        if (Exact && __syncthreads_or(bad)) return false;
#pragma unroll
        for (int u = 0; u < kPer; ++u)
            if ((take >> u) & 1u) {
                se[at_edge] = at[u];
                sa[at_edge] = ar[u];
                ++at_edge;
            }
        cta_flush_edges(se, sa, total_cnt, n, plast, e, p);
    }
    if (nsteps > 0) elast = ref_max(lo, unord(steps[nsteps - 1].a));
    return true;
}

// Builds the profile of `box` into e/p (global), as build_profile_from does.
// Returns the edge count to every thread.
__device__ int64_t cta_build_profile(const Free &F, const double *box, bool v, const Key *steps,
                                     int64_t nsteps, double *e, double *p, double *stage) {
    const double lx = box[0], ly = box[1], ux = box[2], uy = box[3];
    const double lo = v ? lx : ly, hi = v ? ux : uy;
    const int tid = threadIdx.x, nt = blockDim.x;
    int64_t n = 1;
    double elast = lo, plast = 0.0;
    if (tid == 0) {
        e[0] = lo;
        p[0] = 0.0;
    }
    if (v) {
        // the steps' granularity and size
        int g = 2000;
        double big = 0.0;
        for (int64_t k = tid; k < nsteps; k += nt) {
            const double dh = unord(steps[k].b);
            if (dh != 0.0) g = min(g, low_bit(dh));
            big = fmax(big, fabs(dh));
        }
        cta_excl<int>(g, 2000, g, [](int x, int y) { return min(x, y); });
        cta_excl<double>(big, 0.0, big, [](double x, double y) { return fmax(x, y); });
        bool done = false;
        if (g > -1000 && g < 1000 && ldexp(big, -g) * static_cast<double>(nsteps) < 4.0e18)
            done = cta_profile_steps<true>(lo, steps, nsteps, g, stage, n, plast, elast, e, p);
        if (!done) {
            n = 1;
            plast = 0.0;
            cta_profile_steps<false>(lo, steps, nsteps, 0, stage, n, plast, elast, e, p);
        }
    } else {
        double *se = stage, *sa = stage + kRound;
        int32_t r0, r1;
        box_rows(F, box, r0, r1);
        for (int32_t c0 = r0; c0 < r1; c0 += nt) {
            const int32_t r = c0 + tid;
            bool on = false;
            double a = 0.0, z = 0.0, total = 0.0;
            if (r < r1) {
                a = ref_max(lo, F.rowy[2 * r]);
                z = ref_min(hi, F.rowy[2 * r + 1]);
                on = z > a;
                // Row::getLength(b.getX())
                const int64_t end = F.rowspan[r + 1];
                if (on)
                    for (int64_t q = first_span(F, r, lx); q < end && F.spans[2 * q] < ux; ++q)
                        total += ref_max(0.0, ref_min(ux, F.spans[2 * q + 1]) -
                                                  ref_max(lx, F.spans[2 * q]));
            }
            // a row extends the profile where it lies above all before it
            double top;
            double last = cta_excl<double>(on ? z : elast, elast, top,
                                           [](double x, double y) { return y > x ? y : x; });
            last = last > elast ? last : elast;
            const bool ta = on && a > last;
            if (ta) last = a;
            const bool tz = on && z > last;
            int cnt;
            int at = cta_excl<int>((ta ? 1 : 0) + (tz ? 1 : 0), 0, cnt,
                                   [](int x, int y) { return x + y; });
            if (ta) {
                se[at] = a;
                sa[at++] = 0.0;
            }
            if (tz) {
                se[at] = z;
                sa[at] = total * (z - a);
            }
            if (top > elast) elast = top;
            cta_flush_edges(se, sa, cnt, n, plast, e, p);
        }
    }
    const bool more = hi > elast;
    if (tid == 0) {
        if (more) {
            e[n] = hi;
            p[n] = plast + 0.0;
        } else if (n == 1) {
            e[1] = hi;
            p[1] = 0.0;
        }
    }
    if (more || n == 1) ++n;
    __syncthreads();
    return n;
}

// make_stripes with a CTA: the cuts gathered and sorted by all threads, each
// interval between two cuts (independent of the others) split by one thread,
// once to count its stripes and once to write them. Up to kCutSmem cuts.
// Returns the number of stripes, or -1 as make_stripes does; -2 for too many
// cuts (the caller runs make_stripes).
__device__ int64_t cta_make_stripes(const Prof &room, const double *box, bool v, double cell_area,
                                    double region_room, double frac, double limit_density,
                                    const double *obst, int32_t K, double cutline, bool below,
                                    double *stage, int64_t cap, double *sa, double *sb,
                                    double *scap) {
    constexpr int kDepth = 64;
    __shared__ int s_nc;
    double *c = stage, *before = stage + kCutSmem;
    int32_t *idx = reinterpret_cast<int32_t *>(before + kCutSmem);
    const int tid = threadIdx.x, nt = blockDim.x;
    const double lo = v ? box[0] : box[1], hi = v ? box[2] : box[3];
    __syncthreads();
    if (tid == 0) {
        c[0] = lo;
        c[1] = hi;
        idx[0] = 0;
        idx[1] = 1;
        s_nc = 2;
    }
    __syncthreads();
    for (int32_t o = tid; o < K; o += nt) {
        const double *ob = obst + 4 * o;
        if (ob[2] <= box[0] || ob[0] >= box[2] || ob[3] <= box[1] || ob[1] >= box[3]) continue;
        for (int k = 0; k < 2; ++k) {
            const double x = ob[(v ? 0 : 1) + 2 * k];
            if (!(x > lo && x < hi)) continue;
            const int q = atomicAdd(&s_nc, 1);
            if (q < kCutSmem) {
                c[q] = x;
                idx[q] = 2 + 2 * o + k;
            }
        }
    }
    __syncthreads();
    int nc = s_nc;
    if (nc > kCutSmem) return -2;
    // sort by (value, input order), as the stable insertion sort leaves them
    int P = 2;
    while (P < nc) P <<= 1;
    for (int i = nc + tid; i < P; i += nt) {
        c[i] = INFINITY;
        idx[i] = 0x7fffffff;
    }
    __syncthreads();
    for (int k = 2; k <= P; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int t = tid; t < (P >> 1); t += nt) {
                const int i = 2 * j * (t / j) + (t % j), q = i + j;
                const double x = c[i], y = c[q];
                const int32_t xi = idx[i], yi = idx[q];
                const bool gt = y < x || (y == x && yi < xi);
                if (gt == ((i & k) == 0)) {
                    c[i] = y;
                    c[q] = x;
                    idx[i] = yi;
                    idx[q] = xi;
                }
            }
            __syncthreads();
        }
    // unique, in place: kPer consecutive entries per thread
    {
        const int per = (nc + nt - 1) / nt;
        const int b = min(tid * per, nc), e = min(b + per, nc);
        double keep[kCutSmem / kWideT];
        int cnt = 0;
        for (int i = b; i < e; ++i)
            if (i == 0 || !(c[i - 1] == c[i])) keep[cnt++] = c[i];
        int total;
        const int at = cta_excl<int>(cnt, 0, total, [](int x, int y) { return x + y; });
        for (int i = 0; i < cnt; ++i) c[at + i] = keep[i];
        nc = total;
        __syncthreads();
    }
    for (int i = tid; i < nc; i += nt) before[i] = room.before(c[i]);
    const double whole = room.total();
    const double limit = frac * (region_room > 0.0 ? region_room : whole);
    const double fill = whole > 0.0 ? ref_min(limit_density, cell_area / whole) : limit_density;
    __syncthreads();
    // The stripes of interval i (between cuts i - 1 and i), in order, to
    // put(index, start, end, room); the count, or -1 when cap is exceeded
    // with `first` stripes before them.
    auto interval = [&](int i, int64_t first, auto put) -> int64_t {
        double a = c[i - 1], ba = before[i - 1];
        double stk[kDepth], stkb[kDepth];
        int top = 0;
        int64_t ns = first;
        stk[top] = c[i];
        stkb[top] = before[i];
        ++top;
        while (top > 0) {
            const double b = stk[top - 1], bb = stkb[top - 1];
            const double here = bb - ba;
            double mid = 0.0;
            bool cut = here > limit;
            if (cut) {
                mid = room.coordinate_at(ba + 0.5 * here);
                cut = mid > a && mid < b;
            }
            if (cut) {
                if (top == kDepth || ns + top + 1 > cap) return -1;
                stk[top] = mid;
                stkb[top] = room.before(mid);
                ++top;
            } else {
                if (ns >= cap) return -1;
                put(ns, a, b, here);
                ++ns;
                --top;
                a = b;
                ba = bb;
            }
        }
        return ns - first;
    };
    const int per = (nc - 1 + nt - 1) / nt;
    const int b = 1 + min(tid * per, nc - 1), e = min(b + per, nc);
    int cnt = 0;
    bool bad = false;
    for (int i = b; i < e && !bad; ++i) {
        const int64_t k = interval(i, 0, [](int64_t, double, double, double) {});
        if (k < 0) bad = true;
        else cnt += static_cast<int>(k);
    }
    int total;
    int64_t at = cta_excl<int>(cnt, 0, total, [](int x, int y) { return x + y; });
    if (!bad)
        for (int i = b; i < e && !bad; ++i) {
            const int64_t k = interval(i, at, [&](int64_t q, double x, double y, double here) {
                sa[q] = x;
                sb[q] = y;
                scap[q] = fill * here;
            });
            if (k < 0) bad = true;
            else at += k;
        }
    if (__syncthreads_or(bad)) return -1;
    const int64_t ns = total;
    if (!below) {
        auto swap_at = [&](int64_t i, int64_t j) {
            double t = sa[i]; sa[i] = sa[j]; sa[j] = t;
            t = sb[i]; sb[i] = sb[j]; sb[j] = t;
            t = scap[i]; scap[i] = scap[j]; scap[j] = t;
        };
        for (int64_t i = tid; i < ns / 2; i += nt) swap_at(i, ns - 1 - i);
        __syncthreads();
        // restore the original order inside each run of equal distance
        auto from = [&](int64_t i) { return 0.5 * (sa[i] + sb[i]) - cutline; };
        bool run = false;
        for (int64_t i = tid; i + 1 < ns; i += nt) run = run || from(i) == from(i + 1);
        if (__syncthreads_or(run) && tid == 0)
            for (int64_t r = 0; r < ns;) {
                const double f = from(r);
                int64_t q = r + 1;
                while (q < ns && from(q) == f) ++q;
                for (int64_t i = r, j = q - 1; i < j; ++i, --j) swap_at(i, j);
                r = q;
            }
        __syncthreads();
    }
    return ns;
}

// Profile steps of each block (half = 0) or half box (half = 1), one CTA each,
// a warp per row; in any order (they are sorted next).
__global__ void __launch_bounds__(1024) k_steps_cta(Level L, Free F, int half, const int64_t *soff,
                                                    Key *steps, int64_t *nsteps) {
    __shared__ int32_t s_rows[2];
    __shared__ unsigned s_n;
    const int item = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int blk = half ? item >> 1 : item;
    const double *box = half ? L.half_box + 4 * item : L.box + 4 * item;
    if (!L.vert[blk]) {
        if (threadIdx.x == 0) nsteps[item] = 0;
        return;
    }
    if (threadIdx.x == 0) {
        box_rows(F, box, s_rows[0], s_rows[1]);
        s_n = 0;
    }
    __syncthreads();
    const int32_t r1 = s_rows[1];
    const double lx = box[0], ly = box[1], ux = box[2], uy = box[3];
    Key *out = steps + soff[item];
    for (int32_t r = s_rows[0] + warp; r < r1; r += blockDim.x >> 5) {
        const double h = ref_min(uy, F.rowy[2 * r + 1]) - ref_max(ly, F.rowy[2 * r]);
        if (!(h > 0.0)) continue;
        const int64_t end = F.rowspan[r + 1];
        for (int64_t s0 = first_span(F, r, lx); s0 < end; s0 += 32) {
            const int64_t s = s0 + lane;
            const bool in = s < end && F.spans[2 * s] < ux;
            double a = 0.0, z = 0.0;
            if (in) {
                a = ref_max(F.spans[2 * s], lx);
                z = ref_min(F.spans[2 * s + 1], ux);
            }
            const bool on = in && z > a;
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (!__any_sync(0xffffffffu, in)) break;
            if (!m) continue;
            unsigned at = 0;
            if (lane == 0) at = atomicAdd(&s_n, 2u * __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0) + 2u * __popc(m & ((1u << lane) - 1u));
            if (on) {
                out[at] = Key{ord(a), ord(h)};
                out[at + 1] = Key{ord(z), ord(-h)};
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) nsteps[item] = s_n;
}

// One CTA per block: profile, cutline, half boxes.
__global__ void __launch_bounds__(kWideT) k_block_cut_cta(Level L, Free F, const int64_t *soff,
                                                         const Key *steps, const int64_t *nsteps,
                                                         const int64_t *eoff, double *pe,
                                                         double *pp) {
    extern __shared__ __align__(16) double wide_smem[];
    const int blk = blockIdx.x;
    const bool v = L.vert[blk] != 0;
    const double *box = L.box + 4 * blk;
    double *e = pe + eoff[blk], *p = pp + eoff[blk];
    const int64_t n =
        cta_build_profile(F, box, v, steps + soff[blk], nsteps[blk], e, p, wide_smem);
    if (threadIdx.x != 0) return;
    const Prof room{e, p, n};
    const double cell_area = L.cut[blk];
    const double share = cell_area > 0.0 ? L.low_area[blk] / cell_area : 0.5;
    const double lo = v ? box[0] : box[1], hi = v ? box[2] : box[3];
    const double cut = room.total() > 0.0 ? room.coordinate_at(share * room.total())
                                          : lo + share * (hi - lo);
    L.cut[blk] = cut;
    double *lb = L.half_box + 8 * blk, *hb = lb + 4;
    for (int k = 0; k < 4; ++k) lb[k] = hb[k] = box[k];
    (v ? lb[2] : lb[3]) = cut;
    (v ? hb[0] : hb[1]) = cut;
}

// One CTA per half: profile, stripes (getStripes), fill state. A profile of
// up to kProfSmem edges is copied to shared memory before the stripes are cut,
// whose profile lookups are then shared-memory binary searches.
__global__ void __launch_bounds__(kWideT) k_half_stripes_cta(Level L, Free F, const int64_t *soff,
                                                            const Key *steps, const int64_t *nsteps,
                                                            const int64_t *eoff, double *pe,
                                                            double *pp, const int64_t *cap_over,
                                                            double frac, double limit_density,
                                                            Stripes S, int *status) {
    extern __shared__ __align__(16) double wide_smem[];
    __shared__ long long s_ns;
    double *prof = wide_smem, *stage = wide_smem + 2 * kProfSmem;
    const int h = blockIdx.x;
    const int blk = h >> 1, side = h & 1;
    const bool v = L.vert[blk] != 0;
    const double *box = L.half_box + 4 * h;
    double *e = pe + eoff[h], *p = pp + eoff[h];
    const int64_t n = cta_build_profile(F, box, v, steps + soff[h], nsteps[h], e, p, stage);
    const bool local = n <= kProfSmem;
    if (local) {
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
            prof[i] = e[i];
            prof[kProfSmem + i] = p[i];
        }
        __syncthreads();
    }
    const int64_t so = S.off[h];
    const Prof room{local ? prof : e, local ? prof + kProfSmem : p, n};
    const double cell_area = side ? L.high_area[blk] : L.low_area[blk];
    int64_t ns = cta_make_stripes(room, box, v, cell_area, L.room[blk], frac, limit_density, F.obst,
                                  F.K, L.cut[blk], side == 0, stage, cap_over[h], S.a + so,
                                  S.b + so, S.cap + so);
    if (ns == -2) {  // more cuts than shared memory holds
        if (threadIdx.x == 0)
            // cuts live after the profile in the global scratch
            s_ns = make_stripes(room, box, v, cell_area, L.room[blk], frac, limit_density, F.obst,
                                F.K, L.cut[blk], side == 0, p + n, cap_over[h], S.a + so, S.b + so,
                                S.cap + so);
        __syncthreads();
        ns = s_ns;
    }
    if (ns < 0) {
        if (threadIdx.x == 0) atomicCAS(status, kStatusOk, kStatusCapacity);
        ns = 0;
    }
    if (threadIdx.x == 0) S.count[h] = static_cast<int32_t>(ns);
    for (int64_t q = threadIdx.x; q < ns; q += blockDim.x) {
        S.used[so + q] = 0.0;
        S.lo[so + q] = ~0ull;
        S.hi[so + q] = 0ull;
    }
}

// Cells of each half by (-distance from the cut, id), from the keys sorted by
// (centre, id): the distance is monotone in that order, so the low half keeps
// it, the high half reverses it, and cells at the same (rounded) distance go by
// id. A run of one centre is in id order already; a run of several centres is
// ranked by counting, which costs the square of its length: past kMixedRun cells
// the level is left unfilled, and the host sorts by (distance, id) and fills it
// (150k cells within 60 ulp of one x: 5.6 ms in all, 12.9 with ranks by counting;
// 5.4 with one x for all of them).
constexpr int kMixedRun = 256;

__global__ void k_fill_order(Level L, const Key *keys, int32_t *cells) {
    for (int32_t blk = blockIdx.y; blk < L.na; blk += gridDim.y) {
        const int32_t b = L.b[blk], e = L.e[blk], mid = b + L.m[blk];
        const double cut = L.cut[blk];
        for (int32_t p = b + blockIdx.x * blockDim.x + threadIdx.x; p < e;
             p += gridDim.x * blockDim.x) {
            const bool low = p < mid;
            const int32_t hb = low ? b : mid, he = low ? mid : e;
            auto dist = [&](int32_t q) {
                const double c = unord(keys[q].a);
                return ord(-(low ? cut - c : c - cut));
            };
            const unsigned long long d = dist(p);
            int32_t rs = p, re = p + 1;
            while (rs > hb && p - rs < 32 && dist(rs - 1) == d) --rs;
            while (re < he && re - p < 32 && dist(re) == d) ++re;
            if (p - rs == 32) {
                int32_t lo = hb, hi = rs;
                while (lo < hi) {
                    const int32_t q = (lo + hi) >> 1;
                    if (dist(q) == d) hi = q;
                    else lo = q + 1;
                }
                rs = lo;
            }
            if (re - p == 32) {
                int32_t lo = re, hi = he;
                while (lo < hi) {
                    const int32_t q = (lo + hi) >> 1;
                    if (dist(q) == d) lo = q + 1;
                    else hi = q;
                }
                re = lo;
            }
            const unsigned long long id = keys[p].b;
            int32_t rank = p - rs;
            if (re - rs > 1 && keys[rs].a != keys[re - 1].a) {
                if (re - rs > kMixedRun) {
                    *L.redo = 1;
                    continue;
                }
                rank = 0;
                for (int32_t q = rs; q < re; ++q) rank += keys[q].b < id ? 1 : 0;
            }
            cells[low ? rs + rank : mid + (he - re) + rank] = static_cast<int32_t>(id);
        }
    }
}

// The keys of that order, from the keys sorted by (centre, id).
__global__ void k_distance_keys(Level L, const Key *keys, Key *out) {
    for (int32_t blk = blockIdx.y; blk < L.na; blk += gridDim.y) {
        const int32_t b = L.b[blk], e = L.e[blk], mid = b + L.m[blk];
        const double cut = L.cut[blk];
        for (int32_t p = b + blockIdx.x * blockDim.x + threadIdx.x; p < e;
             p += gridDim.x * blockDim.x) {
            const double c = unord(keys[p].a);
            out[p] = Key{ord(-(p < mid ? cut - c : c - cut)), keys[p].b};
        }
    }
}

// One thread per half: greedy fill in the sorted order (nonlinearScale,
// simpl_lal.cc:332-340).
__global__ void k_fill(Level L, CellsDev C, const int32_t *cells, Stripes S, int32_t *stripe_of) {
    if (*L.redo) return;
    const int32_t h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= 2 * L.na) return;
    const int32_t blk = h >> 1;
    const int32_t b = L.b[blk], e = L.e[blk], mid = b + L.m[blk];
    const int32_t p0 = (h & 1) ? mid : b, p1 = (h & 1) ? e : mid;
    const int64_t so = S.off[h];
    const int32_t ns = S.count[h];
    if (ns == 0) {  // a half of zero width: its cells stay where they are
        for (int32_t p = p0; p < p1; ++p) stripe_of[cells[p]] = -1;
        return;
    }
    int32_t s = 0;
    for (int32_t p = p0; p < p1; ++p) {
        while (s + 1 < ns && S.used[so + s] >= S.cap[so + s]) ++s;
        const int32_t i = cells[p];
        stripe_of[i] = static_cast<int32_t>(so + s);
        S.used[so + s] += C.area[i];
    }
}

// Greedy fill from the exact prefix (fill order): stripe s of a half takes
// positions [start_s, start_{s+1}), start_{s+1} the least position whose
// preceding area in the stripe reaches its capacity; the starts go to `sbeg`.
// The starts form a chain, so latency bounds this: one CTA per half loads the
// prefix a window at a time and a warp finds the starts in shared memory, 32
// probes a round, comparing integers (the area scale is a power of two, so
// used >= cap is prefix >= base + ceil(cap x scale)). 55 us a level at 211k
// cells (84 with every probe in global memory).
constexpr int kFillWindow = 16384;
constexpr size_t kFillSmem = sizeof(long long) * kFillWindow;

__global__ void __launch_bounds__(1024) k_fill_fx(Level L, Stripes S, const long long *pre,
                                                  double scale, int32_t *sbeg) {
    extern __shared__ long long win[];
    __shared__ int32_t s_done;
    if (*L.redo) return;
    const int lane = threadIdx.x & 31;
    const int32_t h = blockIdx.x;
    const int32_t blk = h >> 1;
    const int32_t b = L.b[blk], e = L.e[blk], mid = b + L.m[blk];
    const int32_t p0 = (h & 1) ? mid : b, p1 = (h & 1) ? e : mid;
    const int64_t so = S.off[h];
    const int32_t ns = S.count[h];
    if (ns == 0) return;
    int32_t s = 0, at = p0;
    long long base = pre[p0];
    auto need = [&](int32_t q) {  // area that fills stripe q (none reaches it: 2^62)
        const double cap = q < ns ? S.cap[so + q] : 0.0;
        return cap * scale < 0x1p62 ? __double2ll_ru(cap * scale) : 1ll << 62;
    };
    long long mine = need(lane);  // of stripe s - s % 32 + lane
    if (threadIdx.x == 0) {
        sbeg[so] = p0;
        s_done = ns == 1 ? 1 : 0;
    }
    __syncthreads();
    for (int32_t w0 = p0; !s_done; w0 += kFillWindow) {
        const int32_t w1 = min(w0 + kFillWindow, p1);  // positions [w0, w1)
        for (int32_t k = w0 + threadIdx.x; k < w1; k += blockDim.x) win[k - w0] = pre[k];
        __syncthreads();
        if (threadIdx.x < 32) {
            for (;;) {
                const long long full = base + __shfl_sync(0xffffffffu, mine, s & 31);
                int32_t lo = max(at, w0), hi = max(w1, lo);  // first hit in [lo, hi), or hi
                while (lo < hi) {
                    const int32_t step = (hi - lo + 31) / 32, k = lo + lane * step;
                    const int c =
                        __popc(__ballot_sync(0xffffffffu, k < hi && win[k - w0] < full));
                    const int32_t end = lo + c * step;
                    if (c < 32 && end < hi) hi = end;
                    if (c > 0) lo += (c - 1) * step + 1;
                }
                if (lo >= w1 && w1 < p1) break;  // not in this window
                at = min(lo, p1);
                base = at < w1 ? win[at - w0] : pre[at];
                ++s;
                if ((s & 31) == 0) mine = need(s + lane);
                if (lane == 0) sbeg[so + s] = at;
                if (s + 1 == ns) {
                    if (lane == 0) s_done = 1;
                    break;
                }
            }
        }
        __syncthreads();
    }
}

// Lowest and highest centre of each stripe, a warp per stripe: the centres are
// monotone along the fill order but for cells at one rounded distance, so only
// the runs at a stripe's ends can hold them.
__global__ void k_stripe_ends(Level L, CellsDev C, const int32_t *cells, Stripes S,
                              const int32_t *sbeg) {
    if (*L.redo) return;
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int32_t h = blockIdx.y; h < 2 * L.na; h += gridDim.y) {
        const int32_t blk = h >> 1;
        const int32_t p1 = (h & 1) ? L.e[blk] : L.b[blk] + L.m[blk];
        const int64_t so = S.off[h];
        const int32_t ns = S.count[h];
        const bool v = L.vert[blk] != 0;
        const double cut = L.cut[blk];
        for (int32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < ns; q += warps) {
            const int32_t f = sbeg[so + q], l = q + 1 < ns ? sbeg[so + q + 1] : p1;
            if (f >= l) continue;
            auto cen = [&](int32_t k) { return centre(C, cells[k], v); };
            auto dist = [&](double c) { return ord(-((h & 1) ? c - cut : cut - c)); };
            const double cf = cen(f), cl = cen(l - 1);
            unsigned long long mn = min(ord(cf), ord(cl)), mx = max(ord(cf), ord(cl));
            const unsigned long long ends[2] = {dist(cf), dist(cl)};
            for (int side = 0; side < (ends[0] == ends[1] ? 1 : 2); ++side) {
                for (int32_t k0 = 0; k0 < l - f; k0 += 32) {
                    const int32_t k = side ? l - 1 - k0 - lane : f + k0 + lane;
                    bool in = k >= f && k < l;
                    const double c = in ? cen(k) : 0.0;
                    in = in && dist(c) == ends[side];
                    if (in) {
                        mn = min(mn, ord(c));
                        mx = max(mx, ord(c));
                    }
                    if (!__all_sync(0xffffffffu, in)) break;
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            if (lane == 0) {
                S.lo[so + q] = mn;
                S.hi[so + q] = mx;
            }
        }
    }
}

// New position of cell i in stripe s.
__device__ __forceinline__ void place_cell(const CellsDev &C, const Stripes &S, int32_t i, int64_t s,
                                           bool v) {
    const double lo = unord(S.lo[s]), hi = unord(S.hi[s]);
    const double c0 = centre(C, i, v);
    const double t = hi > lo ? (c0 - lo) / (hi - lo) : 0.5;
    const double size = v ? C.w[i] : C.h[i];
    const double a = S.a[s], bb = S.b[s];
    const double c = a + t * (bb - a);
    const double lim = ref_max(a, bb - size);
    double np = c - 0.5 * size;
    np = np < a ? a : (lim < np ? lim : np);  // std::clamp
    (v ? C.x : C.y)[i] = np;
}

// Stripe of every position (the last of its half starting at or before it) and
// the cell's new position.
__global__ void k_place_fx(Level L, CellsDev C, const int32_t *cells, Stripes S,
                           const int32_t *sbeg) {
    if (*L.redo) return;
    for (int32_t blk = blockIdx.y; blk < L.na; blk += gridDim.y) {
        const int32_t b = L.b[blk], e = L.e[blk], mid = b + L.m[blk];
        const bool v = L.vert[blk] != 0;
        for (int32_t p = b + blockIdx.x * blockDim.x + threadIdx.x; p < e; p += gridDim.x * blockDim.x) {
            const int32_t h = 2 * blk + (p < mid ? 0 : 1);
            const int64_t so = S.off[h];
            const int32_t ns = S.count[h];
            if (ns == 0) continue;  // a half of zero width: its cells stay where they are
            int32_t lo = 0, hi = ns - 1;  // last s with sbeg[s] <= p (sbeg[0] <= p)
            while (lo < hi) {
                const int32_t k = (lo + hi + 1) >> 1;
                if (sbeg[so + k] <= p) lo = k;
                else hi = k - 1;
            }
            place_cell(C, S, cells[p], so + lo, v);
        }
    }
}

__global__ void k_stripe_minmax(Level L, CellsDev C, const int32_t *cells, Stripes S,
                                const int32_t *stripe_of) {
    if (*L.redo) return;
    for (int32_t blk = blockIdx.y; blk < L.na; blk += gridDim.y) {
        const int32_t b = L.b[blk], e = L.e[blk];
        const bool v = L.vert[blk] != 0;
        for (int32_t p = b + blockIdx.x * blockDim.x + threadIdx.x; p < e; p += gridDim.x * blockDim.x) {
            const int32_t i = cells[p];
            const int32_t s = stripe_of[i];
            if (s < 0) continue;
            const unsigned long long o = ord(centre(C, i, v));
            atomicMin(S.lo + s, o);
            atomicMax(S.hi + s, o);
        }
    }
}

__global__ void k_new_pos(Level L, CellsDev C, const int32_t *cells, Stripes S,
                          const int32_t *stripe_of) {
    if (*L.redo) return;
    for (int32_t blk = blockIdx.y; blk < L.na; blk += gridDim.y) {
        const int32_t b = L.b[blk], e = L.e[blk];
        const bool v = L.vert[blk] != 0;
        for (int32_t p = b + blockIdx.x * blockDim.x + threadIdx.x; p < e; p += gridDim.x * blockDim.x) {
            const int32_t i = cells[p];
            if (stripe_of[i] >= 0) place_cell(C, S, i, stripe_of[i], v);
        }
    }
}

// ---- small blocks: one CTA finishes a block's whole subtree ------------------------
//
// A block of at most kSub cells is handed to one CTA, which runs every
// remaining level of its bisection out of shared memory: the cells' ids,
// positions, sizes and areas, the CTA-wide sort buffer (three key words per
// entry, compared as (k2, k0, k1)) and the per-level scans. The level's
// sub-blocks, their profiles and stripes live in a per-CTA slice of global
// scratch. A block whose needs exceed a capacity (sort buffer, profile or
// stripe slots, sub-blocks per level, local obstacles) is left untouched
// and flagged; the caller runs it level by level instead.

constexpr int kSortCap = 4096;      // entries of the sort buffer (steps and profiles)
constexpr int kMaxSub = 1024;       // sub-blocks of one level
constexpr int kObstLocal = 256;     // obstacles overlapping the block
constexpr int64_t kStripeCap = 8192;
constexpr int kNearDesc = 12;       // sub-blocks of a level described in shared memory
constexpr int kRowsLocal = 512;     // free-space rows staged in shared memory
constexpr int kSpansLocal = 1280;   // and their spans
constexpr size_t kSubSmem = sizeof(unsigned long long) * 2 * kSortCap +
                            sizeof(uint32_t) * kSortCap + sizeof(long long) * (kSub + 2) +
                            sizeof(double) * (3 * kSub + 4 * kObstLocal) +
                            sizeof(double) * (2 * kRowsLocal + 2 * kSpansLocal) +
                            sizeof(int64_t) * (kRowsLocal + 2) +
                            sizeof(int32_t) * (3 * kSub + 2 * kMaxSub + 2) + sizeof(int16_t) * kSub;

struct SubTask {
    double box[4];
    double room;
    int32_t b, e, level, vert;
    int32_t r0, r1;  // rows its box can meet (r1 < 0: all, to be searched)
};

// Work queue of one launch. A block of more than kHandOff cells is split once
// and its halves go back to the queue, where idle CTAs pick them up: a batch
// has a few blocks of up to 2,048 cells, and finishing each in one CTA left
// the other SMs idle for ten levels. CTAs draw tickets; a ticket past the tail
// waits (with a time limit) until its slot is filled or nothing is pending.
struct SubQueue {
    int32_t head, tail, pending, nfail, timeout;
};
constexpr int64_t kQueueHead = 64;              // bytes before the tasks
constexpr int kHandSlots = 48;                  // queue slots per block handed in
constexpr int kHandOff = 160;
constexpr uint64_t kQueueTimeoutNs = 2000000000ull;
constexpr int kLongRun = 32;                    // cells at one distance ranked by counting

struct SubDesc {
    double box[4];
    double hbox[8];
    double cell_area, low_area, high_area, cut;
    int32_t b, e, level, vert, m, act, rank;
    int32_t soff, scnt, slen;                     // block profile region in the sort buffer
    int32_t hsoff[2], hscnt[2], hslen[2];         // the halves' regions
    int32_t stoff[2], stcap[2], stcnt[2];         // the halves' stripes
};

constexpr int64_t kDescBytes = 2 * kMaxSub * sizeof(SubDesc);  // of a CTA
static_assert(sizeof(SubDesc) % 8 == 0, "");

struct SubArgs {
    SubTask *tasks;          // [cap], the first ntasks filled in
    int32_t ntasks, cap;
    SubQueue *queue;
    unsigned *ready;         // [cap] == epoch: slot filled
    unsigned epoch;
    int2 *failed;            // [cap] (task, reason) of tasks left for the level-by-level path
    int32_t *cells;          // position -> cell id
    CellsDev C;
    Free F;
    SubDesc *desc;           // [grid * 2 * kMaxSub]
    double *strp;            // [grid * 4 * kStripeCap] cuts, start, end, capacity
    unsigned long long *strlh;  // [grid * 2 * kStripeCap] lowest / highest centre
    int32_t max_level, min_cells, stripe_extra;
    double frac, limit_density;
    int32_t exact;           // areas sum exactly: prefix sums and binary searches
    double scale, inv_scale; // 2^q, 2^-q
    int32_t rows_local;      // a block with more rows reads them where they are (-1: all do)
};

__device__ __forceinline__ bool sub_less(uint32_t a2, unsigned long long a0, unsigned long long a1,
                                         uint32_t b2, unsigned long long b0, unsigned long long b1) {
    return a2 < b2 || (a2 == b2 && (a0 < b0 || (a0 == b0 && a1 < b1)));
}

// In-place sort of entries [b, b + n) by `nthreads` cooperating threads
// (index `me`), for any n: every merge of two sorted halves starts with the
// mirrored comparators (i, k - 1 - i) and continues with half-cleaners, all
// ascending, so positions past n act as +inf and their comparators are
// skipped. `sync` separates the steps (a warp or the whole block).
template <typename Sync>
__device__ void net_sort(unsigned long long *k0, unsigned long long *k1, uint32_t *k2, int b, int n,
                         int me, int nthreads, Sync sync) {
    if (n <= 1) return;
    int P = 1;
    while (P < n) P <<= 1;
    auto cas = [&](int i, int q) {
        const uint32_t a2 = k2[b + i], b2 = k2[b + q];
        const unsigned long long a0 = k0[b + i], b0 = k0[b + q], a1 = k1[b + i], b1 = k1[b + q];
        if (sub_less(b2, b0, b1, a2, a0, a1)) {
            k2[b + i] = b2; k0[b + i] = b0; k1[b + i] = b1;
            k2[b + q] = a2; k0[b + q] = a0; k1[b + q] = a1;
        }
    };
    for (int k = 2; k <= P; k <<= 1) {
        const int h = k >> 1;
        for (int t = me; t < (P >> 1); t += nthreads) {
            const int base = (t / h) * k, off = t % h;
            const int q = base + k - 1 - off;
            if (q < n) cas(base + off, q);
        }
        sync();
        for (int j = k >> 2; j > 0; j >>= 1) {
            for (int t = me; t < (P >> 1); t += nthreads) {
                const int i = 2 * j * (t / j) + (t % j);
                if (i + j < n) cas(i, i + j);
            }
            sync();
        }
    }
}

__device__ __forceinline__ void named_barrier(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Sorts each segment [b, e) = seg(g) of g < nseg (none longer than maxlen):
// the whole block for one segment, equal groups of warps (each on its own
// named barrier) for a few long ones, else teams of lanes sized to the
// longest segment (one lane for up to 3 keys, up to a warp), each team
// taking segments in turn. Ends with a block barrier.
template <typename Seg>
__device__ void sort_segments(unsigned long long *k0, unsigned long long *k1, uint32_t *k2, int nseg,
                              int maxlen, Seg seg) {
    const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (nseg <= 0 || maxlen <= 1) {
        __syncthreads();
        return;
    }
    if (nseg == 1) {
        int b, e;
        seg(0, b, e);
        net_sort(k0, k1, k2, b, e - b, threadIdx.x, blockDim.x, [] { __syncthreads(); });
    } else if (nseg < 16 && nw / nseg >= 2 && maxlen > 256) {
        const int W = nw / nseg;  // warps per group
        const int g = w / W;
        if (g < nseg) {
            int b, e;
            seg(g, b, e);
            const int me = (w - g * W) * 32 + lane, n = W * 32;
            net_sort(k0, k1, k2, b, e - b, me, n, [g, n] { named_barrier(1 + g, n); });
        }
    } else {
        int T = 1;  // lanes per team: about half the longest segment, at most a warp
        while (T < 32 && 2 * T < maxlen) T <<= 1;
        const int me = threadIdx.x & (T - 1), team = threadIdx.x / T, nteams = blockDim.x / T;
        const unsigned mask = T == 32 ? 0xffffffffu : (((1u << T) - 1u) << (lane & ~(T - 1)));
        for (int g = team; g < nseg; g += nteams) {
            int b, e;
            seg(g, b, e);
            net_sort(k0, k1, k2, b, e - b, me, T, [mask] { __syncwarp(mask); });
        }
    }
    __syncthreads();
}

// Ranks of positions [0, tot), tot <= kSubThreads, inside their segments by
// counting: `per` threads share a position and each compares every per-th entry
// of its segment, so short segments cost little (160 cells: 3k cycles against
// 19k for the merges above, whose steps are chains of shared-memory reads).
// seg(p, b, e): the segment of p, empty for positions that stay; entry q is
// (key(q), val(q)), ties by the position. Returns the new position of *p, in
// the first of its threads; -1 in the others.
template <class Seg, class KeyOf, class ValOf>
__device__ int counted_position(int tot, int &p, Seg seg, KeyOf key, ValOf val) {
    int per = 1;
    while (per < 32 && 2 * per * tot <= kSubThreads) per <<= 1;
    p = threadIdx.x / per;
    const int sub = threadIdx.x & (per - 1);
    int b = 0, e = 0, rank = 0;
    if (p < tot) seg(p, b, e);
    if (e > b) {
        const unsigned long long k = key(p);
        const auto v = val(p);
#pragma unroll 4
        for (int q = b + sub; q < e; q += per) {
            const unsigned long long kq = key(q);
            const auto vq = val(q);
            rank += static_cast<int>((kq < k) | ((kq == k) & ((vq < v) | ((vq == v) & (q < p)))));
        }
    }
    for (int d = per >> 1; d > 0; d >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, d);
    return p < tot && sub == 0 ? (e > b ? b + rank : p) : -1;
}

// Exclusive scan of buf[0, n) in place; returns the total to every thread.
__device__ int32_t cta_scan(int32_t *buf, int n, int32_t *warp_tmp) {
    const int nt = blockDim.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int per = (n + nt - 1) / nt;
    const int beg = min(tid * per, n), end = min(beg + per, n);
    int32_t local = 0;
    for (int i = beg; i < end; ++i) local += buf[i];
    int32_t v = local;
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) warp_tmp[wid] = v;
    __syncthreads();
    const int nw = nt >> 5;
    if (wid == 0) {
        int32_t w = lane < nw ? warp_tmp[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < nw) warp_tmp[lane] = w;
    }
    __syncthreads();
    int32_t run = v - local + (wid > 0 ? warp_tmp[wid - 1] : 0);
    const int32_t total = warp_tmp[nw - 1];
    for (int i = beg; i < end; ++i) {
        const int32_t t = buf[i];
        buf[i] = run;
        run += t;
    }
    __syncthreads();
    return total;
}

// pre[p + 1] = fixed-point area of positions [0, p] (cell at[p], area sa);
// pre[0] = 0.
__device__ void cta_prefix64(const int32_t *at, const double *sa, int n, double scale,
                             long long *pre, long long *w64) {
    const int nt = blockDim.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int per = (n + nt - 1) / nt;
    const int beg = min(tid * per, n), end = min(beg + per, n);
    long long local = 0;
    for (int p = beg; p < end; ++p) local += __double2ll_rn(sa[at[p]] * scale);
    long long v = local;
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) w64[wid] = v;
    __syncthreads();
    const int nw = nt >> 5;
    if (wid == 0) {
        long long w = lane < nw ? w64[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < nw) w64[lane] = w;
    }
    __syncthreads();
    long long run = v - local + (wid > 0 ? w64[wid - 1] : 0);
    for (int p = beg; p < end; ++p) {
        run += __double2ll_rn(sa[at[p]] * scale);
        pre[p + 1] = run;
    }
    if (tid == 0) pre[0] = 0;
    __syncthreads();
}

// A region of the sort buffer holding a profile: two leading pads, then the
// sorted steps (vertical) or nothing (horizontal); the profile is written
// over it in place (edge n lands at slot n, the step read last sits at slot
// >= n + 1).
__device__ int64_t build_profile_inplace(const Free &F, const double *box, bool v,
                                         unsigned long long *k0, unsigned long long *k1, int o,
                                         int nsteps) {
    double *e = reinterpret_cast<double *>(k0 + o);
    double *p = reinterpret_cast<double *>(k1 + o);
    return build_profile_from(
        F, box, v,
        [&](int64_t k, double &x, double &dh) {
            x = unord(k0[o + 2 + k]);
            dh = unord(k1[o + 2 + k]);
        },
        nsteps, e, p);
}

// A team of T lanes (a power of two up to 32, aligned inside a warp) that
// works on one sub-block: few sub-blocks at a level get wide teams, many get
// one thread each. Row loops are split over the lanes; everything whose
// floating-point order matters runs on lane 0.
struct Team {
    int T, lane, team, nteams;
    unsigned mask;
    __device__ explicit Team(int items) {
        const int per = kSubThreads / max(items, 1);
        T = per >= 32 ? 32 : per >= 16 ? 16 : per >= 8 ? 8 : per >= 4 ? 4 : per >= 2 ? 2 : 1;
        lane = threadIdx.x & (T - 1);
        team = threadIdx.x / T;
        nteams = blockDim.x / T;
        const int wl = threadIdx.x & 31;
        mask = T == 32 ? 0xffffffffu : (((1u << T) - 1u) << (wl & ~(T - 1)));
    }
    template <typename V>
    __device__ V sum(V v) const {
        for (int o = T >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
        return v;
    }
    template <typename V>
    __device__ V excl(V v) const {
        V inc = v;
        for (int o = 1; o < T; o <<= 1) {
            const V t = __shfl_up_sync(mask, inc, o, T);
            if (lane >= o) inc += t;
        }
        return inc - v;
    }
    template <typename V>
    __device__ V bcast(V v) const { return __shfl_sync(mask, v, 0, T); }
    __device__ void sync() const { __syncwarp(mask); }
};

__device__ int32_t team_count_steps(const Team &tm, const Free &F, const double *box) {
    int32_t r0, r1;
    box_rows(F, box, r0, r1);
    int32_t c = 0;
    for (int32_t r = r0 + tm.lane; r < r1; r += tm.T)
        c += static_cast<int32_t>(row_steps(F, r, box, [](int64_t, double, double) {}, 0));
    return tm.sum(c);
}

__device__ int32_t team_count_obstacles(const Team &tm, const Free &F, const double *bx) {
    int32_t k = 0;
    for (int32_t ob = tm.lane; ob < F.K; ob += tm.T) {
        const double *q = F.obst + 4 * ob;
        if (q[2] <= bx[0] || q[0] >= bx[2] || q[3] <= bx[1] || q[1] >= bx[3]) continue;
        ++k;
    }
    return tm.sum(k);
}

// Writes a profile region: pads over [o, o + len), then (vertical) the box's
// steps from o + 2, the rows split over the team (step order inside the
// region does not matter: it is sorted next).
__device__ void team_emit_region(const Team &tm, const Free &F, const double *box, bool v,
                                 uint32_t tag, unsigned long long *k0, unsigned long long *k1,
                                 uint32_t *k2, int o, int len) {
    for (int q = tm.lane; q < len; q += tm.T) {
        k2[o + q] = tag;
        k0[o + q] = 0ull;
        k1[o + q] = 0ull;
    }
    tm.sync();
    if (!v) return;
    int32_t r0, r1;
    box_rows(F, box, r0, r1);
    int32_t c = 0;
    for (int32_t r = r0 + tm.lane; r < r1; r += tm.T)
        c += static_cast<int32_t>(row_steps(F, r, box, [](int64_t, double, double) {}, 0));
    int64_t k = o + 2 + tm.excl(c);
    auto sink = [&](int64_t q, double x, double dh) {
        k0[q] = ord(x);
        k1[q] = ord(dh);
    };
    for (int32_t r = r0 + tm.lane; r < r1; r += tm.T) k += row_steps(F, r, box, sink, k);
    tm.sync();
}

// build_profile_inplace with a team: horizontal boxes get their per-row
// lengths (Row::getLength, each row's spans summed in order by one lane)
// from the lanes first, parked at the top of the region (slots the profile
// reaches only after it has read them); the profile itself is built by lane
// 0. Returns the edge count to every lane.
__device__ int64_t team_build_profile(const Team &tm, const Free &F, const double *box, bool v,
                                      unsigned long long *k0, unsigned long long *k1, int o,
                                      int nsteps, int len) {
    int64_t n = 0;
    if (v) {
        if (tm.lane == 0) n = build_profile_inplace(F, box, v, k0, k1, o, nsteps);
        return tm.bcast(n);
    }
    const double lx = box[0], ly = box[1], ux = box[2], uy = box[3];
    int32_t r0, r1;
    box_rows(F, box, r0, r1);
    const int32_t nr = r1 - r0;
    double *tot = reinterpret_cast<double *>(k1 + o + len - nr);
    for (int32_t i = tm.lane; i < nr; i += tm.T) {
        const int32_t r = r0 + i;
        double total = 0.0;
        const int64_t end = F.rowspan[r + 1];
        for (int64_t s = first_span(F, r, lx); s < end && F.spans[2 * s] < ux; ++s)
            total += ref_max(0.0, ref_min(ux, F.spans[2 * s + 1]) - ref_max(lx, F.spans[2 * s]));
        tot[i] = total;
    }
    tm.sync();
    if (tm.lane == 0) {
        double *e = reinterpret_cast<double *>(k0 + o);
        double *p = reinterpret_cast<double *>(k1 + o);
        n = 1;
        e[0] = ly;
        p[0] = 0.0;
        auto extend = [&](double to, double area) {
            if (to > e[n - 1]) {
                e[n] = to;
                p[n] = p[n - 1] + area;
                ++n;
            }
        };
        for (int32_t i = 0; i < nr; ++i) {
            const int32_t r = r0 + i;
            const double a = ref_max(ly, F.rowy[2 * r]);
            const double z = ref_min(uy, F.rowy[2 * r + 1]);
            if (z > a) {
                const double total = tot[i];
                extend(a, 0.0);
                extend(z, total * (z - a));
            }
        }
        extend(uy, 0.0);
        if (n == 1) {
            e[1] = uy;
            p[1] = 0.0;
            n = 2;
        }
    }
    n = tm.bcast(n);
    tm.sync();
    return n;
}

// The prefix of a profile whose edges' areas are in p[1, n): one lane, the next
// eight areas loading behind the additions.
__device__ __forceinline__ void chain_prefix(double *p, int64_t n) {
    double sum = 0.0, next[8];
    int64_t i = 1;
#pragma unroll
    for (int u = 0; u < 8; ++u) next[u] = i + u < n ? p[i + u] : 0.0;
    for (; i < n; i += 8) {
        double cur[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) cur[u] = next[u];
#pragma unroll
        for (int u = 0; u < 8; ++u) next[u] = i + 8 + u < n ? p[i + 8 + u] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            sum = sum + cur[u];
            if (i + u < n) p[i + u] = sum;
        }
    }
}

// team_build_profile by a whole warp: 32 steps or rows at a time, edges packed
// by ballots, and only the prefix chained by one lane. Heights are exact
// integer sums as in cta_profile_steps (checked before anything is
// overwritten), else the team version takes over.
__device__ int64_t warp_build_profile(const Team &tm, const Free &F, const double *box, bool v,
                                      unsigned long long *k0, unsigned long long *k1, int o,
                                      int nsteps, int len) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    double *e = reinterpret_cast<double *>(k0 + o), *p = reinterpret_cast<double *>(k1 + o);
    const double lo = v ? box[0] : box[1], hi = v ? box[2] : box[3];
    int64_t n = 1;
    double elast = lo;
    if (v) {
        int g = 2000;
        double big = 0.0;
        for (int k = lane; k < nsteps; k += 32) {
            const double dh = unord(k1[o + 2 + k]);
            if (dh != 0.0) g = min(g, low_bit(dh));
            big = fmax(big, fabs(dh));
        }
        for (int d = 16; d > 0; d >>= 1) {
            g = min(g, __shfl_xor_sync(0xffffffffu, g, d));
            big = fmax(big, __shfl_xor_sync(0xffffffffu, big, d));
        }
        bool ok = nsteps == 0 || (g > -1000 && g < 1000 &&
                                  ldexp(big, -g) * static_cast<double>(nsteps) < 4.0e18);
        const double scale = ok ? ldexp(1.0, -g) : 0.0, unit = ok ? ldexp(1.0, g) : 0.0;
        auto incl = [&](long long x) {
            for (int d = 1; d < 32; d <<= 1) {
                const long long t = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= d) x += t;
            }
            return x;
        };
        long long carry = 0;
        for (int c0 = 0; ok && c0 < nsteps; c0 += 32) {
            const int k = c0 + lane;
            const long long s =
                carry + incl(k < nsteps ? __double2ll_rn(unord(k1[o + 2 + k]) * scale) : 0);
            ok = !__any_sync(0xffffffffu, s > (1ll << 53) || s < -(1ll << 53));
            carry = __shfl_sync(0xffffffffu, s, 31);
        }
        if (!ok) return team_build_profile(tm, F, box, v, k0, k1, o, nsteps, len);
        carry = 0;
        double prev_last = lo;
        for (int c0 = 0; c0 < nsteps; c0 += 32) {
            const int k = c0 + lane;
            const bool on = k < nsteps;
            const double at = on ? unord(k0[o + 2 + k]) : 0.0;
            const long long h = on ? __double2ll_rn(unord(k1[o + 2 + k]) * scale) : 0;
            const long long inc = incl(h);
            double prev = __shfl_up_sync(0xffffffffu, at, 1);
            if (lane == 0) prev = prev_last;
            const double area = static_cast<double>(carry + inc - h) * unit * (at - prev);
            const unsigned m = __ballot_sync(0xffffffffu, on && at > prev);
            if ((m >> lane) & 1u) {
                e[n + __popc(m & below)] = at;
                p[n + __popc(m & below)] = area;
            }
            n += __popc(m);
            carry += __shfl_sync(0xffffffffu, inc, 31);
            prev_last = __shfl_sync(0xffffffffu, at, min(31, nsteps - 1 - c0));
            __syncwarp();
        }
        elast = ref_max(lo, prev_last);
    } else {
        const double lx = box[0], ux = box[2];
        int32_t r0, r1;
        box_rows(F, box, r0, r1);
        for (int32_t c0 = r0; c0 < r1; c0 += 32) {
            const int32_t r = c0 + lane;
            bool on = false;
            double a = 0.0, z = 0.0, total = 0.0;
            if (r < r1) {
                a = ref_max(lo, F.rowy[2 * r]);
                z = ref_min(hi, F.rowy[2 * r + 1]);
                on = z > a;
                const int64_t end = F.rowspan[r + 1];
                if (on)
                    for (int64_t q = first_span(F, r, lx); q < end && F.spans[2 * q] < ux; ++q)
                        total += ref_max(0.0, ref_min(ux, F.spans[2 * q + 1]) -
                                                  ref_max(lx, F.spans[2 * q]));
            }
            double top = on ? z : elast;  // running maximum of the row tops
            for (int d = 1; d < 32; d <<= 1) {
                const double t = __shfl_up_sync(0xffffffffu, top, d);
                if (lane >= d && t > top) top = t;
            }
            double last = __shfl_up_sync(0xffffffffu, top, 1);
            if (lane == 0 || !(last > elast)) last = elast;
            const bool ta = on && a > last;
            if (ta) last = a;
            const bool tz = on && z > last;
            const unsigned ma = __ballot_sync(0xffffffffu, ta), mz = __ballot_sync(0xffffffffu, tz);
            int64_t at = n + __popc(ma & below) + __popc(mz & below);
            if (ta) {
                e[at] = a;
                p[at++] = 0.0;
            }
            if (tz) {
                e[at] = z;
                p[at] = total * (z - a);
            }
            n += __popc(ma) + __popc(mz);
            const double t = __shfl_sync(0xffffffffu, top, 31);
            if (t > elast) elast = t;
        }
    }
    const bool more = hi > elast;
    if (lane == 0) {
        e[0] = lo;
        p[0] = 0.0;
        if (more || n == 1) {
            e[n] = hi;
            p[n] = 0.0;
        }
    }
    if (more || n == 1) ++n;
    __syncwarp();
    if (lane == 0) chain_prefix(p, n);
    __syncwarp();
    return n;
}

// make_stripes by a warp for at most 32 cuts and stripes (-2: more): cuts
// ranked, all intervals halved at once until none is above the limit. `buf`
// holds 128 doubles of shared memory.
__device__ int64_t warp_make_stripes(const Prof &room, const double *box, bool v, double cell_area,
                                     double region_room, double frac, double limit_density,
                                     const double *obst, int32_t K, double cutline, bool below,
                                     int64_t cap, double *sa, double *sb, double *scap,
                                     double *buf) {
    const int lane = threadIdx.x & 31;
    const unsigned before_me = (1u << lane) - 1u;
    const double lo = v ? box[0] : box[1], hi = v ? box[2] : box[3];
    int32_t *order = reinterpret_cast<int32_t *>(buf + 32);
    int nc = 2;
    if (lane < 2) {
        buf[lane] = lane ? hi : lo;
        order[lane] = lane;
    }
    for (int32_t o0 = 0; o0 < K; o0 += 32) {
        const int32_t o = o0 + lane;
        bool in = o < K;
        const double *ob = obst + 4 * (in ? o : 0);
        in = in && !(ob[2] <= box[0] || ob[0] >= box[2] || ob[3] <= box[1] || ob[1] >= box[3]);
        for (int k = 0; k < 2; ++k) {
            const double x = ob[(v ? 0 : 1) + 2 * k];
            const bool put = in && x > lo && x < hi;
            const unsigned m = __ballot_sync(0xffffffffu, put);
            if (nc + __popc(m) > 32) return -2;
            if (put) {
                buf[nc + __popc(m & before_me)] = x;
                order[nc + __popc(m & before_me)] = 2 + 2 * o + k;
            }
            nc += __popc(m);
        }
    }
    __syncwarp();
    // rank by (value, input order), drop repeats
    double c = lane < nc ? buf[lane] : 0.0;
    const int32_t ord_me = lane < nc ? order[lane] : 0;
    int rank = 0;
    for (int j = 0; j < nc; ++j) {
        const double cj = __shfl_sync(0xffffffffu, c, j);
        const int32_t oj = __shfl_sync(0xffffffffu, ord_me, j);
        if (cj < c || (cj == c && oj < ord_me)) ++rank;
    }
    __syncwarp();
    if (lane < nc) buf[rank] = c;
    __syncwarp();
    c = lane < nc ? buf[lane] : 0.0;
    const double left = __shfl_up_sync(0xffffffffu, c, 1);
    const unsigned keep = __ballot_sync(0xffffffffu, lane < nc && (lane == 0 || !(left == c)));
    __syncwarp();
    if ((keep >> lane) & 1u) buf[__popc(keep & before_me)] = c;
    nc = __popc(keep);
    __syncwarp();
    c = lane < nc ? buf[lane] : 0.0;
    const double at = lane < nc ? room.before(c) : 0.0;
    const double whole = room.total();
    const double limit = frac * (region_room > 0.0 ? region_room : whole);
    const double fill = whole > 0.0 ? ref_min(limit_density, cell_area / whole) : limit_density;
    // interval of this lane, in ascending order
    int count = nc - 1;
    double a = c, b = __shfl_down_sync(0xffffffffu, c, 1);
    double ba = at, bb = __shfl_down_sync(0xffffffffu, at, 1);
    unsigned done = 0u;
    double *wa = buf, *wb = buf + 32, *wba = buf + 64, *wbb = buf + 96;
    for (;;) {
        const double here = bb - ba;
        bool cut = lane < count && !((done >> lane) & 1u) && here > limit;
        double mid = 0.0;
        if (cut) {
            mid = room.coordinate_at(ba + 0.5 * here);
            cut = mid > a && mid < b;
        }
        const unsigned m = __ballot_sync(0xffffffffu, cut);
        if (!m) break;
        if (count + __popc(m) > 32) return -2;
        const int to = lane + __popc(m & before_me);
        __syncwarp();
        if (lane < count) {
            wa[to] = a;
            wba[to] = ba;
            if (cut) {
                const double bm = room.before(mid);
                wb[to] = wa[to + 1] = mid;
                wbb[to] = wba[to + 1] = bm;
                wb[to + 1] = b;
                wbb[to + 1] = bb;
            } else {
                wb[to] = b;
                wbb[to] = bb;
            }
        }
        done = __reduce_or_sync(0xffffffffu, lane < count && !cut ? 1u << to : 0u);
        count += __popc(m);
        __syncwarp();
        if (lane < count) {
            a = wa[lane];
            b = wb[lane];
            ba = wba[lane];
            bb = wbb[lane];
        }
    }
    if (count > cap) return -1;
    int to = lane;
    if (!below) {  // farthest first: reversed, runs of equal distance in order
        const double f = 0.5 * (a + b) - cutline;
        const double pf = __shfl_up_sync(0xffffffffu, f, 1);
        const unsigned same = __ballot_sync(0xffffffffu, lane > 0 && lane < count && pf == f);
        const unsigned upto = 0xffffffffu >> (31 - lane);
        const int rs = 31 - __clz(~same & upto);
        const unsigned next = ~same & ~upto;
        const int re = next ? min(__ffs(next) - 1, count) : count;
        to = (count - re) + (lane - rs);
    }
    if (lane < count) {
        sa[to] = a;
        sb[to] = b;
        scap[to] = fill * (bb - ba);
    }
    __syncwarp();
    return count;
}

__global__ void __launch_bounds__(kSubThreads, 1) k_subtree(SubArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned long long *k0 = reinterpret_cast<unsigned long long *>(smem);
    unsigned long long *k1 = k0 + kSortCap;
    long long *pre = reinterpret_cast<long long *>(k1 + kSortCap);  // [kSub + 1]
    double *sx = reinterpret_cast<double *>(pre + kSub + 2);
    double *sy = sx + kSub, *sa = sy + kSub;
    double *obst = sa + kSub;
    double *lrowy = obst + 4 * kObstLocal, *lspans = lrowy + 2 * kRowsLocal;
    int64_t *lrowspan = reinterpret_cast<int64_t *>(lspans + 2 * kSpansLocal);
    uint32_t *k2 = reinterpret_cast<uint32_t *>(lrowspan + kRowsLocal + 2);
    uint32_t *v1 = reinterpret_cast<uint32_t *>(k1);  // local indices of sorted cells
    int32_t *gid = reinterpret_cast<int32_t *>(k2 + kSortCap);
    int32_t *at = gid + kSub, *sof = at + kSub, *scan = sof + kSub;
    int16_t *dof = reinterpret_cast<int16_t *>(scan + 2 * kMaxSub + 2);
    __shared__ int32_t warp_tmp[32];
    __shared__ long long w64[32];
    __shared__ int s_fail, s_nobst, s_ncur, s_maxsteps, s_c1;
    const int tid = threadIdx.x, nt = blockDim.x;
    __shared__ SubDesc near_desc[2][kNearDesc];  // levels of a few sub-blocks
    __shared__ int s_task, s_slot;
    SubDesc *const far_desc = A.desc + static_cast<size_t>(blockIdx.x) * 2 * kMaxSub;
    double *const scut = A.strp + static_cast<size_t>(blockIdx.x) * 4 * kStripeCap;
    double *const sta = scut + kStripeCap, *const stb = sta + kStripeCap;
    double *const stc = stb + kStripeCap;
    unsigned long long *const glo = A.strlh + static_cast<size_t>(blockIdx.x) * 2 * kStripeCap;
    unsigned long long *const ghi = glo + kStripeCap;
    const CellsDev &C = A.C;
    // a block of at most half the capacity keeps its cells' sizes behind their
    // positions
    bool near_sizes = false;
    auto extent = [&](int j, bool v) {
        return near_sizes ? (v ? sx : sy)[kSub / 2 + j] : v ? C.w[gid[j]] : C.h[gid[j]];
    };
    auto centre = [&](int j, bool v) { return (v ? sx : sy)[j] + 0.5 * extent(j, v); };
    // the steps of regions [0, tot) by (x, dh), in place; span: a tag's steps
    auto sort_steps = [&](int tot, auto span) {
        int p;
        const int to = counted_position(
            tot, p,
            [&](int q, int &b, int &e) {
                span(k2[q], b, e);
                if (q < b) b = e = 0;  // a pad stays
            },
            [&](int q) { return k0[q]; }, [&](int q) { return k1[q]; });
        const unsigned long long x = to >= 0 ? k0[p] : 0ull, dh = to >= 0 ? k1[p] : 0ull;
        __syncthreads();
        if (to >= 0) {
            k0[to] = x;
            k1[to] = dh;
        }
        __syncthreads();
    };
    // profile steps in the sort buffer; a region's pads (0, 0) sort first
    auto step_entry = [&](int p, unsigned long long &k, unsigned long long &v) {
        k = k0[p];
        v = k1[p];
    };

    for (;;) {
        __syncthreads();
        if (tid == 0) {
            int got = -1;
            const int t = atomicAdd(&A.queue->head, 1);
            if (t < A.ntasks) {
                got = t;
            } else if (t < A.cap) {
                const uint64_t deadline = global_timer_ns() + kQueueTimeoutNs;
                for (;;) {
                    if (ld_acquire_gpu(A.ready + t) == A.epoch) {
                        got = t;
                        break;
                    }
                    // nothing pending: no more slots will be filled
                    if (ld_acquire_gpu(reinterpret_cast<unsigned *>(&A.queue->pending)) == 0u ||
                        ld_relaxed_gpu(&A.queue->timeout) != 0)
                        break;
                    if (global_timer_ns() > deadline) {
                        atomicExch(&A.queue->timeout, 1);
                        break;
                    }
                    __nanosleep(100);
                }
            }
            s_task = got;
            s_fail = 0;
            s_slot = -1;
            s_nobst = 0;
            s_maxsteps = 0;
        }
        __syncthreads();
        const int task = s_task;
        if (task < 0) return;
        const SubTask T = A.tasks[task];
        const int size = T.e - T.b;
        if (size > kSub) {  // left alone
            if (tid == 0) {
                A.failed[atomicAdd(&A.queue->nfail, 1)] = make_int2(task, 1);
                __threadfence();
                atomicSub(&A.queue->pending, 1);
            }
            continue;
        }
        near_sizes = size <= kSub / 2;
        // cells by id, so that the sorts below break ties by the local index
        // (handed-off blocks come that way)
        if (task < A.ntasks) {
            merge_sort<false>(k0, v1, k2, size, [&](int p, unsigned long long &k, uint32_t &v) {
                k = static_cast<unsigned long long>(A.cells[T.b + p]);
                v = 0u;
            });
        }
        for (int j = tid; j < size; j += nt) {
            const int32_t g = task < A.ntasks ? static_cast<int32_t>(k0[j]) : A.cells[T.b + j];
            gid[j] = g;
            sx[j] = C.x[g];
            sy[j] = C.y[g];
            sa[j] = C.area[g];
            at[j] = j;
            if (near_sizes) {
                sx[kSub / 2 + j] = C.w[g];
                sy[kSub / 2 + j] = C.h[g];
            }
        }
        for (int o = tid; o < A.F.K; o += nt) {
            const double *ob = A.F.obst + 4 * o;
            if (ob[2] <= T.box[0] || ob[0] >= T.box[2] || ob[3] <= T.box[1] || ob[1] >= T.box[3])
                continue;
            const int k = atomicAdd(&s_nobst, 1);
            if (k < kObstLocal)
                for (int q = 0; q < 4; ++q) obst[4 * k + q] = ob[q];
        }
        if (tid == 0) {
            SubDesc &d = near_desc[0][0];
            for (int q = 0; q < 4; ++q) d.box[q] = T.box[q];
            d.b = 0;
            d.e = size;
            d.level = T.level;
            d.vert = T.vert;
            s_ncur = 1;
        }
        Free FL = A.F;
        int32_t row0 = T.r0, rows = T.r1 - T.r0;
        {  // the rows overlapping the block, with their spans overlapping its x
           // range, into shared memory (the only spans its sub-boxes can meet);
           // a handed-off block takes the rows of the block it came from
            if (T.r1 < 0) {
                int32_t r1;
                box_rows(A.F, T.box, row0, r1);
                rows = r1 - row0;
            }
            if (rows <= A.rows_local) {
                for (int i = tid; i < rows; i += nt) {
                    const int64_t f = first_span(A.F, row0 + i, T.box[0]);
                    int64_t e = f, hi = A.F.rowspan[row0 + i + 1];
                    while (e < hi) {  // first span from f that starts at or past the box
                        const int64_t mid = (e + hi) >> 1;
                        if (A.F.spans[2 * mid] < T.box[2]) e = mid + 1;
                        else hi = mid;
                    }
                    scan[i] = static_cast<int32_t>(e - f);
                    lrowspan[i] = f;  // first span, global index (rebased below)
                }
                __syncthreads();
                const int32_t ns = cta_scan(scan, rows, warp_tmp);
                if (ns <= kSpansLocal) {
                    for (int i = tid; i < rows; i += nt) {
                        const int64_t f = lrowspan[i];
                        const int32_t o = scan[i];
                        const int32_t cnt = (i + 1 < rows ? scan[i + 1] : ns) - o;
                        for (int32_t q = 0; q < cnt; ++q) {
                            lspans[2 * (o + q)] = A.F.spans[2 * (f + q)];
                            lspans[2 * (o + q) + 1] = A.F.spans[2 * (f + q) + 1];
                        }
                        lrowy[2 * i] = A.F.rowy[2 * (row0 + i)];
                        lrowy[2 * i + 1] = A.F.rowy[2 * (row0 + i) + 1];
                    }
                    __syncthreads();
                    for (int i = tid; i <= rows; i += nt) lrowspan[i] = i < rows ? scan[i] : ns;
                    FL.rowy = lrowy;
                    FL.rowspan = lrowspan;
                    FL.spans = lspans;
                    FL.R = rows;
                }
            }
        }
        __syncthreads();
        if (tid == 0 && s_nobst > kObstLocal) s_fail = 1;  // too many obstacles
        FL.obst = obst;
        FL.K = min(s_nobst, kObstLocal);
        SubDesc *cur = near_desc[0], *nxt = near_desc[1];
        for (int depth = 0;; ++depth) {
            __syncthreads();
            const int ncur = s_ncur;
            if (s_fail || ncur == 0) break;
            // A. which sub-blocks split at this level, and their rank
            for (int i = tid; i < ncur; i += nt) {
                const int len = cur[i].e - cur[i].b;
                const int act = cur[i].level < A.max_level && len > A.min_cells;
                cur[i].act = act;
                scan[i] = act;
            }
            __syncthreads();
            const int nact = cta_scan(scan, ncur, warp_tmp);
            if (nact == 0) break;
            if (2 * nact > kMaxSub) {
                if (tid == 0) s_fail = 2;  // too many sub-blocks
                break;
            }
            int drawn = 0, filled = 0;
            if (tid == 0) {
                drawn = ld_relaxed_gpu(&A.queue->head);
                filled = ld_relaxed_gpu(&A.queue->tail);
            }
            nxt = 2 * nact <= kNearDesc ? near_desc[(depth + 1) & 1]
                                        : far_desc + ((depth + 1) & 1) * kMaxSub;
            for (int i = tid; i < ncur; i += nt) cur[i].rank = scan[i];
            __syncthreads();
            // the sub-blocks' starts, and ends with the split and axis flags,
            // in shared memory for the position lookups
            for (int i = tid; i < ncur; i += nt) {
                scan[i] = cur[i].b;
                scan[kMaxSub + i] = cur[i].e | (cur[i].act << 30) | (cur[i].vert << 29);
            }
            __syncthreads();
            // B. each position's sub-block; cells of each splitting sub-block by
            // (centre, id), ties by cell id as the reference's sortCells
            for (int p = tid; p < size; p += nt) {
                int lo = 0, hi = ncur;  // last sub-block with b <= p
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (scan[mid] <= p) lo = mid;
                    else hi = mid;
                }
                const int i = lo;
                const int ev = scan[kMaxSub + i];
                const bool in = p >= scan[i] && p < (ev & 0x1fffffff) && ((ev >> 30) & 1);
                dof[p] = static_cast<int16_t>(in ? i : -1);
                k2[p] = static_cast<uint32_t>(in ? scan[i] : p);
            }
            __syncthreads();
            auto centre_key = [&](int p) {
                const int i = dof[p];
                return i >= 0 ? ord(centre(at[p], ((scan[kMaxSub + i] >> 29) & 1) != 0)) : 0ull;
            };
            if (size <= kSubThreads) {
                for (int p = tid; p < size; p += nt) k0[p] = centre_key(p);
                __syncthreads();
                int p;
                const int to = counted_position(
                    size, p,
                    [&](int q, int &b, int &e) {
                        const int i = dof[q];
                        if (i < 0) return;
                        b = scan[i];
                        e = scan[kMaxSub + i] & 0x1fffffff;
                    },
                    [&](int q) { return k0[q]; }, [&](int q) { return at[q]; });
                if (to >= 0) v1[to] = static_cast<uint32_t>(at[p]);
                __syncthreads();
            } else {
                auto entry = [&](int p, unsigned long long &k, uint32_t &v) {
                    k = centre_key(p);
                    v = static_cast<uint32_t>(at[p]);
                };
                if (ncur == 1) merge_sort<false>(k0, v1, k2, size, entry);
                else merge_sort<true>(k0, v1, k2, size, entry);
            }
            for (int p = tid; p < size; p += nt) at[p] = static_cast<int32_t>(v1[p]);
            __syncthreads();
            if (A.exact) cta_prefix64(at, sa, size, A.scale, pre, w64);
            // C. areas and median in sorted order; the block profile's region
            {
                const Team tm(nact);
                for (int i = tm.team; i < ncur; i += tm.nteams) {
                    SubDesc &d = cur[i];
                    int32_t steps = 0, len = 0;
                    if (d.act) {
                        const bool v = d.vert != 0;
                        steps = v ? team_count_steps(tm, FL, d.box) : 0;
                        int32_t r0, r1;
                        box_rows(FL, d.box, r0, r1);
                        len = (v ? steps : 2 * (r1 - r0)) + 2;
                        if (tm.lane == 0) {
                            const int b = d.b, e = d.e, n = e - b;
                            double cell_area = 0.0, low = 0.0, high = 0.0;
                            int m = 0;
                            if (A.exact) {
                                m = median_fx(pre, b, n);
                                cell_area = static_cast<double>(pre[e] - pre[b]) * A.inv_scale;
                                low = static_cast<double>(pre[b + m] - pre[b]) * A.inv_scale;
                                high = static_cast<double>(pre[e] - pre[b + m]) * A.inv_scale;
                            } else {
                                for (int p = b; p < e; ++p) cell_area += sa[at[p]];
                                while (m + 1 < n && (m == 0 || low < 0.5 * cell_area))
                                    low += sa[at[b + m++]];
                                for (int p = b + m; p < e; ++p) high += sa[at[p]];
                            }
                            d.m = m;
                            d.cell_area = cell_area;
                            d.low_area = low;
                            d.high_area = high;
                            atomicMax(&s_maxsteps, steps);
                        }
                    }
                    if (tm.lane == 0) {
                        d.scnt = steps;
                        d.slen = len;
                        scan[i] = len;
                    }
                }
            }
            __syncthreads();
            const int tot = cta_scan(scan, ncur, warp_tmp);
            const int maxsteps = s_maxsteps;
            for (int i = tid; i < ncur; i += nt) cur[i].soff = scan[i];
            __syncthreads();  // every thread has read s_maxsteps before it is reset
            if (tid == 0) {
                s_maxsteps = 0;
                scan[ncur] = tot;
            }
            // D + E, in chunks of consecutive sub-blocks whose profile regions fit
            // the sort buffer together (scan[] holds the regions' offsets)
            for (int c0 = 0; c0 < ncur;) {
                if (tid == 0) {
                    int lo = c0 + 1, hi = ncur;  // the last end offset within reach
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (scan[mid] - scan[c0] <= kSortCap) lo = mid;
                        else hi = mid - 1;
                    }
                    int c1 = lo;
                    if (scan[c1] - scan[c0] > kSortCap) c1 = c0;  // one region too long
                    if (c1 == c0) s_fail = 3;  // sort buffer
                    s_c1 = c1;
                }
                __syncthreads();
                if (s_fail) break;
                const int c1 = s_c1, base = scan[c0];
                // D. the block profiles' regions: pads, then the steps sorted by (x, dh)
                {
                    const Team tm(nact);
                    for (int i = c0 + tm.team; i < c1; i += tm.nteams) {
                        const SubDesc &d = cur[i];
                        if (!d.act) continue;
                        const int o = d.soff - base;
                        team_emit_region(tm, FL, d.box, d.vert != 0, static_cast<uint32_t>(i), k0,
                                         k1, k2, o, d.slen);
                    }
                }
                __syncthreads();
                if (maxsteps > 1 && scan[c1] - base <= kSubThreads)
                    sort_steps(scan[c1] - base, [&](uint32_t tag, int &b, int &e) {
                        const SubDesc &d = cur[tag];
                        b = d.soff - base + 2;
                        e = b + d.scnt;
                    });
                else if (maxsteps > 1 && scan[c1] - base <= kSub)
                    merge_sort<true>(k0, k1, k2, scan[c1] - base, step_entry);
                else
                    sort_segments(k0, k1, k2, c1 - c0, maxsteps, [&](int g, int &b, int &e) {
                        const SubDesc &d = cur[c0 + g];
                        const bool on = d.act && d.vert;
                        b = on ? d.soff - base + 2 : 0;
                        e = on ? d.soff - base + 2 + d.scnt : 0;
                    });
                // E. profile, cutline, half boxes, the halves' regions and stripe room
                {
                    const Team tm(nact);
                    for (int i = c0 + tm.team; i < c1; i += tm.nteams) {
                        SubDesc &d = cur[i];
                        if (!d.act) {
                            if (tm.lane == 0)
                                for (int side = 0; side < 2; ++side) d.hslen[side] = d.stcap[side] = 0;
                            continue;
                        }
                        const bool v = d.vert != 0;
                        const int o = d.soff - base;
                        const int64_t n =
                            tm.T == 32 ? warp_build_profile(tm, FL, d.box, v, k0, k1, o, d.scnt, d.slen)
                                       : team_build_profile(tm, FL, d.box, v, k0, k1, o, d.scnt, d.slen);
                        const Prof room{reinterpret_cast<const double *>(k0 + o),
                                        reinterpret_cast<const double *>(k1 + o), n};
                        const double share = d.cell_area > 0.0 ? d.low_area / d.cell_area : 0.5;
                        const double lo = v ? d.box[0] : d.box[1], hi = v ? d.box[2] : d.box[3];
                        const double cut = room.total() > 0.0 ? room.coordinate_at(share * room.total())
                                                              : lo + share * (hi - lo);
                        double hb[8];
                        for (int q = 0; q < 4; ++q) hb[q] = hb[4 + q] = d.box[q];
                        hb[v ? 2 : 3] = cut;
                        hb[4 + (v ? 0 : 1)] = cut;
                        const double r_lo = room.before(cut);
                        int32_t hsc[2], hsl[2], cap[2];
                        for (int side = 0; side < 2; ++side) {
                            const double *bx = hb + 4 * side;
                            hsc[side] = v ? team_count_steps(tm, FL, bx) : 0;
                            int32_t r0, r1;
                            box_rows(FL, bx, r0, r1);
                            hsl[side] = (v ? hsc[side] : 2 * (r1 - r0)) + 2;
                            const int32_t k = team_count_obstacles(tm, FL, bx);
                            // stripes from midpoint splits hold more than half the split
                            // limit each: at most 2 room / limit of them (+ margin)
                            const double r_h = side ? ref_max(0.0, room.total() - r_lo) : r_lo;
                            const double lim = A.frac * (T.room > 0.0 ? T.room : r_h);
                            int32_t extra = A.stripe_extra;
                            if (T.room > 0.0 && lim > 0.0)
                                extra = static_cast<int32_t>(ref_min(static_cast<double>(A.stripe_extra),
                                                                     ceil(2.02 * r_h / lim) + 4.0));
                            cap[side] = 2 * k + 2 + extra;
                        }
                        tm.sync();  // every lane has read the profile and the box
                        if (tm.lane == 0) {
                            d.cut = cut;
                            for (int q = 0; q < 8; ++q) d.hbox[q] = hb[q];
                            for (int side = 0; side < 2; ++side) {
                                d.hscnt[side] = hsc[side];
                                d.hslen[side] = hsl[side];
                                d.stcap[side] = cap[side];
                                atomicMax(&s_maxsteps, hsc[side]);
                            }
                        }
                    }
                }
                __syncthreads();
                c0 = c1;
            }
            if (s_fail) break;
            // the halves' stripe offsets, then their profile regions' offsets
            for (int h = tid; h < 2 * ncur; h += nt) scan[h] = cur[h >> 1].stcap[h & 1];
            __syncthreads();
            const int stot = cta_scan(scan, 2 * ncur, warp_tmp);
            if (stot > kStripeCap) {
                if (tid == 0) s_fail = 4;  // stripes
                break;
            }
            for (int h = tid; h < 2 * ncur; h += nt) {
                cur[h >> 1].stoff[h & 1] = scan[h];
                scan[h] = cur[h >> 1].hslen[h & 1];
            }
            __syncthreads();
            const int htot = cta_scan(scan, 2 * ncur, warp_tmp);
            const int maxhsteps = s_maxsteps;
            for (int h = tid; h < 2 * ncur; h += nt) cur[h >> 1].hsoff[h & 1] = scan[h];
            __syncthreads();
            if (tid == 0) {
                s_maxsteps = 0;
                scan[2 * ncur] = htot;
            }
            // F + G, in chunks of consecutive halves
            for (int c0 = 0; c0 < 2 * ncur;) {
                if (tid == 0) {
                    const int nh = 2 * ncur;
                    int lo = c0 + 1, hi = nh;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (scan[mid] - scan[c0] <= kSortCap) lo = mid;
                        else hi = mid - 1;
                    }
                    int c1 = lo;
                    if (scan[c1] - scan[c0] > kSortCap) c1 = c0;  // one region too long
                    if (c1 == c0) s_fail = 3;  // sort buffer
                    s_c1 = c1;
                }
                __syncthreads();
                if (s_fail) break;
                const int c1 = s_c1, base = scan[c0];
                // F. the halves' profile regions
                {
                    const Team tm(2 * nact);
                    for (int h = c0 + tm.team; h < c1; h += tm.nteams) {
                        const SubDesc &d = cur[h >> 1];
                        const int side = h & 1;
                        if (!d.act) continue;
                        const int o = d.hsoff[side] - base;
                        team_emit_region(tm, FL, d.hbox + 4 * side, d.vert != 0, static_cast<uint32_t>(h),
                                         k0, k1, k2, o, d.hslen[side]);
                    }
                }
                __syncthreads();
                if (maxhsteps > 1 && scan[c1] - base <= kSubThreads)
                    sort_steps(scan[c1] - base, [&](uint32_t tag, int &b, int &e) {
                        const SubDesc &d = cur[tag >> 1];
                        b = d.hsoff[tag & 1] - base + 2;
                        e = b + d.hscnt[tag & 1];
                    });
                else if (maxhsteps > 1 && scan[c1] - base <= kSub)
                    merge_sort<true>(k0, k1, k2, scan[c1] - base, step_entry);
                else
                    sort_segments(k0, k1, k2, c1 - c0, maxhsteps, [&](int g, int &b, int &e) {
                        const int h = c0 + g;
                        const SubDesc &d = cur[h >> 1];
                        const bool on = d.act && d.vert;
                        b = on ? d.hsoff[h & 1] - base + 2 : 0;
                        e = on ? d.hsoff[h & 1] - base + 2 + d.hscnt[h & 1] : 0;
                    });
                // G. the halves' profiles and stripes
                {
                    const Team tm(2 * nact);
                    for (int h = c0 + tm.team; h < c1; h += tm.nteams) {
                        SubDesc &d = cur[h >> 1];
                        const int side = h & 1;
                        if (!d.act) continue;
                        const bool v = d.vert != 0;
                        const int o = d.hsoff[side] - base;
                        const double *bx = d.hbox + 4 * side;
                        const int len = d.hslen[side], cnt = d.hscnt[side];
                        const int64_t n = tm.T == 32
                                              ? warp_build_profile(tm, FL, bx, v, k0, k1, o, cnt, len)
                                              : team_build_profile(tm, FL, bx, v, k0, k1, o, cnt, len);
                        const int so = d.stoff[side];
                        const double area = side ? d.high_area : d.low_area;
                        const Prof room{reinterpret_cast<const double *>(k0 + o),
                                        reinterpret_cast<const double *>(k1 + o), n};
                        int64_t ns = -2;
                        if (tm.T == 32)  // the tags of the step sort are used up
                            ns = warp_make_stripes(room, bx, v, area, T.room, A.frac, A.limit_density,
                                                   FL.obst, FL.K, d.cut, side == 0, d.stcap[side],
                                                   sta + so, stb + so, stc + so,
                                                   reinterpret_cast<double *>(k2) + 128 * (tid >> 5));
                        if (ns == -2 && tm.lane == 0)
                            ns = make_stripes(room, bx, v, area, T.room, A.frac, A.limit_density,
                                              FL.obst, FL.K, d.cut, side == 0, scut + so,
                                              d.stcap[side], sta + so, stb + so, stc + so);
                        if (tm.lane == 0) {
                            if (ns < 0) atomicExch(&s_fail, 4);
                            d.stcnt[side] = static_cast<int32_t>(ns < 0 ? 0 : ns);
                        }
                    }
                }
                __syncthreads();
                if (s_fail) break;
                c0 = c1;
            }
            if (s_fail) break;
            // H. cells of each half by (-distance from the cut, id). The cells
            // are in centre order, in which the distance is monotone: the low
            // half keeps the order, the high half is reversed, and cells at
            // the same distance go by id
            for (int p = tid; p < size; p += nt) {
                const int i = dof[p];
                if (i < 0) continue;
                const SubDesc &d = cur[i];
                const double c = centre(at[p], d.vert != 0);
                const double from = p < d.b + d.m ? d.cut - c : c - d.cut;
                k0[p] = ord(-from);
            }
            __syncthreads();
            bool unsorted = false;  // a long run out of id order
            for (int p = tid; p < size; p += nt) {
                const int i = dof[p];
                int to = p;
                if (i >= 0) {
                    const SubDesc &d = cur[i];
                    const int mid = d.b + d.m;
                    const int b = p < mid ? d.b : mid, e = p < mid ? mid : d.e;
                    const unsigned long long k = k0[p];
                    int rs = p, re = p + 1, rank = 0;
                    while (rs > b && k0[rs - 1] == k && p - rs < kLongRun) --rs;
                    while (re < e && k0[re] == k && re - p < kLongRun) ++re;
                    if (p - rs == kLongRun || re - p == kLongRun) {  // all of it, by binary search
                        int lo = b, hi = rs;
                        while (lo < hi) {
                            const int q = (lo + hi) >> 1;
                            if (k0[q] == k) hi = q;
                            else lo = q + 1;
                        }
                        rs = lo;
                        hi = e;
                        lo = re;
                        while (lo < hi) {
                            const int q = (lo + hi) >> 1;
                            if (k0[q] == k) lo = q + 1;
                            else hi = q;
                        }
                        re = lo;
                    }
                    if (re - rs > kLongRun) {
                        rank = p - rs;
                        unsorted = unsorted || (p > rs && at[p - 1] > at[p]);
                    } else {
                        for (int q = rs; q < re; ++q) rank += at[q] < at[p];
                    }
                    to = p < mid ? rs + rank : mid + (d.e - re) + rank;
                }
                v1[to] = static_cast<uint32_t>(at[p]);
            }
            if (__syncthreads_or(unsorted)) {
                for (int p = tid; p < size; p += nt) {
                    const int i = dof[p];
                    k2[p] = static_cast<uint32_t>(
                        i < 0 ? p : (p < cur[i].b + cur[i].m ? cur[i].b : cur[i].b + cur[i].m));
                }
                __syncthreads();
                merge_sort<true>(k0, v1, k2, size, [&](int p, unsigned long long &k, uint32_t &v) {
                    k = dof[p] < 0 ? 0ull : k0[p];
                    v = static_cast<uint32_t>(at[p]);
                });
            }
            for (int p = tid; p < size; p += nt) at[p] = static_cast<int32_t>(v1[p]);
            __syncthreads();
            // the stripes' starts and extreme centres, in the sort buffer when
            // they fit (the sorted entries are used up)
            const bool fits = stot <= kSortCap;
            unsigned long long *const slo = fits ? k0 : glo, *const shi = fits ? k1 : ghi;
            uint32_t *const starts = fits ? k2 : reinterpret_cast<uint32_t *>(scut);
            for (int q = tid; q < stot; q += nt) {
                slo[q] = ~0ull;
                shi[q] = 0ull;
            }
            // I. greedy fill (exact areas: stripe starts by binary search on the
            // prefix, then each position looks its stripe up; else one thread
            // per half in the reference's order)
            if (A.exact) {
                cta_prefix64(at, sa, size, A.scale, pre, w64);
                for (int h = tid; h < 2 * ncur; h += nt) {
                    const SubDesc &d = cur[h >> 1];
                    if (!d.act) continue;
                    const int side = h & 1;
                    const int mid = d.b + d.m;
                    const int p0 = side ? mid : d.b, p1 = side ? d.e : mid;
                    const int ns = d.stcnt[side], so = d.stoff[side];
                    int q0 = p0;
                    for (int q = 0; q < ns; ++q) {
                        starts[so + q] = static_cast<uint32_t>(q0);
                        if (q + 1 == ns) break;
                        const double cap = stc[so + q];
                        int lo = q0, hi = p1;
                        while (lo < hi) {
                            const int k = (lo + hi) >> 1;
                            if (static_cast<double>(pre[k] - pre[q0]) * A.inv_scale >= cap) hi = k;
                            else lo = k + 1;
                        }
                        q0 = lo;
                    }
                }
                __syncthreads();
                for (int p = tid; p < size; p += nt) {
                    const int i = dof[p];
                    if (i < 0) continue;
                    const SubDesc &d = cur[i];
                    const int side = p < d.b + d.m ? 0 : 1;
                    const int ns = d.stcnt[side], so = d.stoff[side];
                    int q = -1;
                    if (ns > 0) {
                        int lo = 0, hi = ns - 1;
                        while (lo < hi) {
                            const int k = (lo + hi + 1) >> 1;
                            if (starts[so + k] <= static_cast<uint32_t>(p)) lo = k;
                            else hi = k - 1;
                        }
                        q = so + lo;
                    }
                    sof[at[p]] = q;
                }
            } else {
                for (int h = tid; h < 2 * ncur; h += nt) {
                    const SubDesc &d = cur[h >> 1];
                    if (!d.act) continue;
                    const int side = h & 1;
                    const int mid = d.b + d.m;
                    const int p0 = side ? mid : d.b, p1 = side ? d.e : mid;
                    const int ns = d.stcnt[side], so = d.stoff[side];
                    if (ns == 0) {
                        for (int p = p0; p < p1; ++p) sof[at[p]] = -1;
                        continue;
                    }
                    int q = 0;
                    double used = 0.0;
                    for (int p = p0; p < p1; ++p) {
                        while (q + 1 < ns && used >= stc[so + q]) {
                            ++q;
                            used = 0.0;
                        }
                        const int j = at[p];
                        sof[j] = so + q;
                        used += sa[j];
                    }
                }
            }
            __syncthreads();
            // J. lowest and highest centre per stripe
            for (int p = tid; p < size; p += nt) {
                const int i = dof[p];
                if (i < 0) continue;
                const int j = at[p];
                const int q = sof[j];
                if (q < 0) continue;
                const unsigned long long o = ord(centre(j, cur[i].vert != 0));
                atomicMin(slo + q, o);
                atomicMax(shi + q, o);
            }
            __syncthreads();
            // K. new positions
            for (int p = tid; p < size; p += nt) {
                const int i = dof[p];
                if (i < 0) continue;
                const int j = at[p];
                const int q = sof[j];
                if (q < 0) continue;
                const bool v = cur[i].vert != 0;
                const double lo = unord(slo[q]), hi = unord(shi[q]);
                const double c0 = centre(j, v);
                const double t = hi > lo ? (c0 - lo) / (hi - lo) : 0.5;
                const double sz = extent(j, v);
                const double a = sta[q], bb = stb[q];
                const double c = a + t * (bb - a);
                const double lim = ref_max(a, bb - sz);
                double np = c - 0.5 * sz;
                np = np < a ? a : (lim < np ? lim : np);
                (v ? sx : sy)[j] = np;
            }
            __syncthreads();
            // L. children: low and high halves, next axis
            for (int i = tid; i < ncur; i += nt) {
                const SubDesc &d = cur[i];
                if (!d.act) continue;
                for (int side = 0; side < 2; ++side) {
                    SubDesc &c = nxt[2 * d.rank + side];
                    for (int q = 0; q < 4; ++q) c.box[q] = d.hbox[4 * side + q];
                    c.b = side ? d.b + d.m : d.b;
                    c.e = side ? d.e : d.b + d.m;
                    c.level = d.level + 1;
                    c.vert = d.vert ? 0 : 1;
                }
            }
            if (tid == 0) {
                s_ncur = 2 * nact;
                s_maxsteps = 0;
                // CTAs waiting (as of the level's start), and room for two
                // blocks? Only the whole block's halves are handed off: beside a
                // half that is done already they would not fill its positions
                if (size > kHandOff && ncur == 1 && drawn > filled) {
                    int t = filled;
                    while (t + 2 <= A.cap) {
                        const int was = atomicCAS(&A.queue->tail, t, t + 2);
                        if (was == t) {
                            s_slot = t;
                            break;
                        }
                        t = was;
                    }
                }
            }
            cur = nxt;
            __syncthreads();
            if (s_slot >= 0) break;
        }
        __syncthreads();
        if (!s_fail) {
            for (int j = tid; j < size; j += nt) {
                C.x[gid[j]] = sx[j];
                C.y[gid[j]] = sy[j];
            }
            if (s_slot >= 0) {  // the halves' cells, by id each
                const int m = cur[0].e;
                for (int p = tid; p < size; p += nt) scan[at[p]] = p < m ? 1 : 0;
                __syncthreads();
                for (int j = tid; j < size; j += nt) sof[j] = scan[j];
                cta_scan(scan, size, warp_tmp);
                for (int j = tid; j < size; j += nt)
                    A.cells[T.b + (sof[j] ? scan[j] : m + j - scan[j])] = gid[j];
            }
        }
        __syncthreads();
        if (tid == 0) {
            if (s_fail) A.failed[atomicAdd(&A.queue->nfail, 1)] = make_int2(task, s_fail);
            if (s_slot >= 0) {
                atomicAdd(&A.queue->pending, 2);
                for (int q = 0; q < 2; ++q) {
                    const SubDesc &d = cur[q];
                    SubTask &h = A.tasks[s_slot + q];
                    for (int k = 0; k < 4; ++k) h.box[k] = d.box[k];
                    h.room = T.room;
                    h.b = T.b + d.b;
                    h.e = T.b + d.e;
                    h.level = d.level;
                    h.vert = d.vert;
                    h.r0 = row0;
                    h.r1 = rows <= A.rows_local ? row0 + rows : -1;
                }
                __threadfence();
                for (int q = 0; q < 2; ++q) atomicExch(A.ready + s_slot + q, A.epoch);
            }
            __threadfence();
            atomicSub(&A.queue->pending, 1);
        }
    }
}

// ---- batch set-up and bins ---------------------------------------------------------

struct GridDev {
    double ox, oy, dx, dy;
    int32_t nx, ny;
};

__device__ __forceinline__ int32_t clamp_index(double f, int32_t n) {
    const double hi = static_cast<double>(n) - 1e-9;
    const double c = f < 0.0 ? 0.0 : (hi < f ? hi : f);
    return static_cast<int32_t>(c);
}

__global__ void k_bins(CellsDev C, int32_t n, GridDev G, int32_t *binof) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t ix = clamp_index((C.x[i] + 0.5 * C.w[i] - G.ox) / G.dx, G.nx);
    const int32_t iy = clamp_index((C.y[i] + 0.5 * C.h[i] - G.oy) / G.dy, G.ny);
    binof[i] = iy * G.nx + ix;
}

__global__ void k_region_map(const int32_t *rects, int32_t nreg, int32_t nx, int32_t *map) {
    for (int32_t r = blockIdx.y; r < nreg; r += gridDim.y) {
        const int32_t x0 = rects[4 * r], x1 = rects[4 * r + 1], y0 = rects[4 * r + 2],
                      y1 = rects[4 * r + 3];
        const int64_t w = x1 - x0 + 1, cnt = w * (y1 - y0 + 1);
        for (int64_t k = blockIdx.x * blockDim.x + threadIdx.x; k < cnt; k += gridDim.x * blockDim.x)
            map[(y0 + k / w) * nx + x0 + k % w] = r;
    }
}

__global__ void k_region_count(const int32_t *binof, int32_t n, const int32_t *map, int32_t *cnt) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t r = map[binof[i]];
    if (r >= 0) atomicAdd(cnt + r, 1);
}

__global__ void k_region_place(const int32_t *binof, int32_t n, const int32_t *map, int32_t *cursor,
                               int32_t *cells) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t r = map[binof[i]];
    if (r >= 0) cells[atomicAdd(cursor + r, 1)] = i;
}

__global__ void k_clamp_die(CellsDev C, int32_t n, double lx, double ly, double ux, double uy) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double mx = ref_max(lx, ux - C.w[i]), my = ref_max(ly, uy - C.h[i]);
    double x = C.x[i], y = C.y[i];
    x = x < lx ? lx : (mx < x ? mx : x);
    y = y < ly ? ly : (my < y ? my : y);
    C.x[i] = x;
    C.y[i] = y;
}

}  // namespace

// Free space, obstacles and die for the legalizer, and its scratch.
struct LalState {
    std::vector<double> rowy, spans, obst;
    std::vector<double> side[4];  // obstacles' lx, ly, ux, uy, each sorted
    int64_t odd = 0;              // obstacles that are in none of the four
    std::vector<int64_t> rowspan;
    bool rows_sorted = true;  // by y start, which are all numbers
    // The row ends ascend, and in each row the spans' starts and ends: a search
    // among a block's own rows and spans then finds what one among all of them
    // finds. Rows that overlap may break the order, and a binary search over
    // another window then ends at another row, so blocks read all rows in place.
    bool windows = true;
    double die[4] = {0, 0, 0, 0};
    DevBuf<double> d_rowy, d_spans, d_obst;
    DevBuf<int64_t> d_rowspan;
    DevBuf<int32_t> binof, map, cells, cnt, stripe_of, rects;
    DevBuf<double> occ;
    DevBuf<char> level;      // everything of the level in work (launch_lal)
    DevBuf<Key> keys, keys_tmp;
    DevBuf<double> overflow;
    DevBuf<long long> pre, tile;
    DevBuf<char> tasks;      // SubQueue (kQueueHead bytes), then the tasks
    DevBuf<unsigned> ready;
    unsigned epoch = 0;
    DevBuf<int2> tfail;
    DevBuf<char> swork;      // the subtree CTAs' sub-blocks and stripes
    bool subtree_attr = false;
    bool wide_attr = false;
    // Upper bound on the obstacles that overlap `box`: the lesser of those that
    // meet its x range and those that meet its y range. An obstacle whose sides
    // are not in order passes the kernels' overlap test where its upper side lies
    // above the box's lower and its lower side below the box's upper, so every
    // box counts all of these; a box without extent counts all obstacles.
    int64_t obstacle_bound(const double *box) const {
        auto meet = [&](int k) -> int64_t {
            if (!(box[k] < box[k + 2])) return static_cast<int64_t>(side[k].size());
            const auto past = std::lower_bound(side[k].begin(), side[k].end(), box[k + 2]);
            const auto before = std::upper_bound(side[k + 2].begin(), side[k + 2].end(), box[k]);
            return (past - side[k].begin()) - (before - side[k + 2].begin());
        };
        return odd + std::min(meet(0), meet(1));
    }
    // Upper bound on the profile's steps and edges of `box` and of its halves: the
    // rows it can meet (as box_rows) and their spans. Where rows start at no
    // number, box_rows finds others for a half than for the box: all of them then.
    void profile_bound(const double *box, bool vertical, int64_t &steps, int64_t &edges) const {
        const int64_t R = static_cast<int64_t>(rowy.size() / 2);
        int64_t lo = 0, hi = R;  // first row with box.ly < y end
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (box[1] < rowy[2 * mid + 1]) hi = mid;
            else lo = mid + 1;
        }
        int64_t r0 = lo;
        hi = R;  // first row from r0 with y start >= box.uy
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (rowy[2 * mid] < box[3]) lo = mid + 1;
            else hi = mid;
        }
        if (!rows_sorted) r0 = 0, lo = R;
        const int64_t sp = R ? rowspan[lo] - rowspan[r0] : 0;
        steps = vertical ? 2 * sp : 0;
        edges = (vertical ? 2 * sp : 2 * (lo - r0)) + 2;
    }
    // counters of the last ktg_lal call (ktg_lal_stats)
    double stats[16] = {};
};

void free_lal(ktg_ctx *c) {
    LalState *s = c->lal;
    if (!s) return;
    for (auto *b : {&s->binof, &s->map, &s->cells, &s->cnt, &s->stripe_of, &s->rects})
        b->release();
    for (auto *b : {&s->d_rowy, &s->d_spans, &s->d_obst, &s->occ, &s->overflow}) b->release();
    s->d_rowspan.release();
    s->level.release();
    s->keys.release();
    s->keys_tmp.release();
    s->pre.release();
    s->tile.release();
    s->tasks.release();
    s->tfail.release();
    s->ready.release();
    s->swork.release();
    delete s;
    c->lal = nullptr;
}

int set_free_space(ktg_ctx *c, int64_t nrows, const double *rowy, const int64_t *rowspan,
                   const double *spans, int64_t nobst, const double *obst, const double *die4) {
    if (!c->lal) c->lal = new LalState();
    LalState *s = c->lal;
    const int64_t S = nrows > 0 ? rowspan[nrows] : 0;
    s->rowy.assign(rowy, rowy + 2 * nrows);
    s->rowspan.assign(rowspan, rowspan + nrows + 1);
    s->rows_sorted = true;
    s->windows = true;
    for (int64_t r = 0; r < nrows; ++r) {
        s->rows_sorted = s->rows_sorted && !std::isnan(rowy[2 * r]);
        s->windows = s->windows && rowy[2 * std::max<int64_t>(r - 1, 0) + 1] <= rowy[2 * r + 1];
        for (int64_t k = rowspan[r]; k < rowspan[r + 1]; ++k)
            for (int q = 0; q < 2; ++q)
                s->windows = s->windows && spans[2 * std::max(k - 1, rowspan[r]) + q] <= spans[2 * k + q];
    }
    s->spans.assign(spans, spans + 2 * S);
    s->obst.assign(obst, obst + 4 * nobst);
    for (int k = 0; k < 4; ++k) s->side[k].clear();
    s->odd = 0;
    for (int64_t o = 0; o < nobst; ++o) {
        const double *q = obst + 4 * o;
        if (!(q[0] <= q[2]) || !(q[1] <= q[3])) {
            ++s->odd;
            continue;
        }
        for (int k = 0; k < 4; ++k) s->side[k].push_back(q[k]);
    }
    for (int k = 0; k < 4; ++k) std::sort(s->side[k].begin(), s->side[k].end());
    std::copy(die4, die4 + 4, s->die);
    int rc;
    if ((rc = s->d_rowy.ensure(c, 2 * nrows + 2)) || (rc = s->d_rowspan.ensure(c, nrows + 2)) ||
        (rc = s->d_spans.ensure(c, 2 * S + 2)) || (rc = s->d_obst.ensure(c, 4 * nobst + 4)))
        return rc;
    KTG_CUDA(c, cudaMemcpyAsync(s->d_rowy.p, s->rowy.data(), sizeof(double) * s->rowy.size(),
                                cudaMemcpyHostToDevice, c->stream));
    KTG_CUDA(c, cudaMemcpyAsync(s->d_rowspan.p, s->rowspan.data(),
                                sizeof(int64_t) * s->rowspan.size(), cudaMemcpyHostToDevice, c->stream));
    if (S > 0)
        KTG_CUDA(c, cudaMemcpyAsync(s->d_spans.p, s->spans.data(), sizeof(double) * s->spans.size(),
                                    cudaMemcpyHostToDevice, c->stream));
    if (nobst > 0)
        KTG_CUDA(c, cudaMemcpyAsync(s->d_obst.p, s->obst.data(), sizeof(double) * s->obst.size(),
                                    cudaMemcpyHostToDevice, c->stream));
    KTG_CUDA(c, cudaStreamSynchronize(c->stream));
    return KTG_OK;
}

namespace {

cudaError_t lal_sync(ktg_ctx *c) {
    c->lal->stats[3] += 1;
    return cudaStreamSynchronize(c->stream);
}

double now_ms() {
    return std::chrono::duration<double, std::milli>(
               std::chrono::steady_clock::now().time_since_epoch()).count();
}

// ---- host side: clusters and growth exactly as the reference sums them ---------------

struct HostGrid {
    int32_t nx, ny;
    const std::vector<double> *avail;
    double limit;
    double rect_sum(const std::vector<double> &f, const int32_t *r) const {
        double t = 0.0;
        for (int32_t iy = r[2]; iy <= r[3]; ++iy)
            for (int32_t ix = r[0]; ix <= r[1]; ++ix) t += f[static_cast<size_t>(iy) * nx + ix];
        return t;
    }
    double density(const std::vector<double> &occ, const int32_t *r) const {
        const double cells = rect_sum(occ, r);
        const double room = rect_sum(*avail, r);
        if (room > 0.0) return cells / room;
        return cells > 0.0 ? std::numeric_limits<double>::infinity() : 0.0;
    }
    std::vector<std::array<int32_t, 4>> clusters(const std::vector<double> &occ) const {
        const int64_t N = static_cast<int64_t>(nx) * ny;
        std::vector<char> over(N);
        for (int64_t k = 0; k < N; ++k) over[k] = occ[k] > limit * (*avail)[k] ? 1 : 0;
        std::vector<std::array<int32_t, 4>> out;
        std::vector<int64_t> frontier;
        for (int64_t seed = 0; seed < N; ++seed) {
            if (!over[seed]) continue;
            over[seed] = 0;
            frontier.assign(1, seed);
            std::array<int32_t, 4> r{static_cast<int32_t>(seed % nx), static_cast<int32_t>(seed % nx),
                                     static_cast<int32_t>(seed / nx), static_cast<int32_t>(seed / nx)};
            while (!frontier.empty()) {
                const int64_t k = frontier.back();
                frontier.pop_back();
                const int32_t ix = static_cast<int32_t>(k % nx), iy = static_cast<int32_t>(k / nx);
                r[0] = std::min(r[0], ix);
                r[1] = std::max(r[1], ix);
                r[2] = std::min(r[2], iy);
                r[3] = std::max(r[3], iy);
                const int32_t st[4][2] = {{1, 0}, {-1, 0}, {0, 1}, {0, -1}};
                for (const auto &d : st) {
                    const int64_t px = ix + d[0], py = iy + d[1];
                    if (px < 0 || py < 0 || px >= nx || py >= ny) continue;
                    const int64_t kk = py * nx + px;
                    if (over[kk]) {
                        over[kk] = 0;
                        frontier.push_back(kk);
                    }
                }
            }
            out.push_back(r);
        }
        return out;
    }
    std::array<int32_t, 4> grown(std::array<int32_t, 4> r, const std::vector<double> &occ) const {
        while (density(occ, r.data()) > limit) {
            const std::array<std::array<int32_t, 4>, 4> wider{{
                {r[0] > 0 ? r[0] - 1 : r[0], r[1], r[2], r[3]},
                {r[0], r[1] + 1 < nx ? r[1] + 1 : r[1], r[2], r[3]},
                {r[0], r[1], r[2] > 0 ? r[2] - 1 : r[2], r[3]},
                {r[0], r[1], r[2], r[3] + 1 < ny ? r[3] + 1 : r[3]},
            }};
            const int64_t bins = static_cast<int64_t>(r[1] - r[0] + 1) * (r[3] - r[2] + 1);
            int best = -1;
            double best_d = std::numeric_limits<double>::infinity();
            for (int k = 0; k < 4; ++k) {
                const auto &w = wider[k];
                if (static_cast<int64_t>(w[1] - w[0] + 1) * (w[3] - w[2] + 1) == bins) continue;
                const double d = density(occ, w.data());
                if (best < 0 || d < best_d) {
                    best = k;
                    best_d = d;
                }
            }
            if (best < 0) break;
            r = wider[best];
        }
        return r;
    }
};

}  // namespace

// Runs the legalizer on positions x, y (device, n values) in place.
int launch_lal(ktg_ctx *c, double *x, double *y, int32_t max_level, int32_t min_cells,
               double frac) {
    LalState *s = c->lal;
    const int32_t n = static_cast<int32_t>(c->n);
    const int32_t nx = static_cast<int32_t>(c->nx), ny = static_cast<int32_t>(c->ny);
    const int64_t nbins = static_cast<int64_t>(nx) * ny;
    int rc;
    if ((rc = s->binof.ensure(c, n + 1)) || (rc = s->map.ensure(c, nbins)) ||
        (rc = s->cells.ensure(c, n + 1)) ||
        (rc = s->occ.ensure(c, nbins)) || (rc = s->overflow.ensure(c, 1)) ||
        (rc = s->keys.ensure(c, n + 1)) || (rc = s->keys_tmp.ensure(c, n + 1)))
        return rc;
    KTG_CUDA(c, cudaMemsetAsync(c->status, 0, sizeof(int), c->stream));
    std::fill(s->stats, s->stats + 16, 0.0);
    const double t_start = now_ms();
    CellsDev C{x, y, c->width, c->height, c->area};
    const GridDev G{c->origin_x, c->origin_y, c->dx, c->dy, nx, ny};
    Free F{s->d_rowy.p, s->d_rowspan.p, s->d_spans.p, s->d_obst.p,
           static_cast<int32_t>(s->rowy.size() / 2), static_cast<int32_t>(s->obst.size() / 4)};
    const HostGrid HG{nx, ny, &c->avail_host, c->density_limit};
    std::vector<double> occ(nbins);
    auto refresh = [&]() -> int {  // bins and occupancy of the current positions
        const double t0 = now_ms();
        if (n > 0) {
            k_bins<<<blocks_for(n), kT, 0, c->stream>>>(C, n, G, s->binof.p);
            ++c->launches;
        }
        int r2 = launch_occupancy(c, x, y, s->occ.p, s->overflow.p);
        if (r2) return r2;
        KTG_CUDA(c, cudaMemcpyAsync(occ.data(), s->occ.p, sizeof(double) * nbins,
                                    cudaMemcpyDeviceToHost, c->stream));
        KTG_CUDA(c, lal_sync(c));
        s->stats[6] += now_ms() - t0;
        return KTG_OK;
    };
    if ((rc = refresh())) return rc;

    auto reach = [&](const std::array<int32_t, 4> &r) {
        return std::array<int32_t, 4>{r[0] > 0 ? r[0] - 1 : 0, std::min(r[1] + 1, nx - 1),
                                      r[2] > 0 ? r[2] - 1 : 0, std::min(r[3] + 1, ny - 1)};
    };
    auto touches = [](const std::array<int32_t, 4> &a, const std::array<int32_t, 4> &b) {
        return a[0] <= b[1] && b[0] <= a[1] && a[2] <= b[3] && b[2] <= a[3];
    };
    std::vector<std::array<int32_t, 4>> batch, batch_reach;
    const int32_t stripe_extra =
        64 + static_cast<int32_t>(std::min(1048576.0, std::ceil(4.0 / frac)));
    const bool exact = c->area_shift >= 0 && c->lal_exact_sums != 0;
    const double scale = exact ? std::ldexp(1.0, c->area_shift) : 1.0;
    const double inv_scale = exact ? std::ldexp(1.0, -c->area_shift) : 1.0;

    // pre[p] = fixed-point area of cell positions [0, p), p <= count.
    auto fx_prefix = [&](int32_t count) -> int {
        const int32_t tiles = std::max(1, (count + kScanTile - 1) / kScanTile);
        int r2;
        if ((r2 = s->pre.ensure(c, static_cast<int64_t>(count) + 1)) ||
            (r2 = s->tile.ensure(c, tiles)))
            return r2;
        k_fx_tile_sums<<<tiles, kT, 0, c->stream>>>(s->cells.p, c->area, count, scale, s->tile.p);
        k_fx_tile_scan<<<1, kT, 0, c->stream>>>(s->tile.p, tiles);
        k_fx_prefix<<<tiles, kT, 0, c->stream>>>(s->cells.p, c->area, count, scale, s->tile.p,
                                                 s->pre.p);
        c->launches += 3;
        KTG_CUDA(c, cudaGetLastError());
        return KTG_OK;
    };

    // Blocks of at most kSub cells: the subtree kernel runs the rest of the
    // bisection; left: the blocks (given or handed off) that remain for the
    // level-by-level path.
    auto run_subtree = [&](const std::vector<SubTask> &tasks, std::vector<SubTask> &left) -> int {
        const int32_t nt = static_cast<int32_t>(tasks.size());
        const int32_t cap = nt * kHandSlots;
        // CTAs: as many as the queue can keep busy, one for every part of at most
        // kHandOff cells that the blocks halve into; the rest would hold their SMs
        // waiting, and other streams' work out (a block of 100 cells: 1, not 48)
        int64_t parts = 0;
        for (const SubTask &t : tasks) {
            int64_t k = 1;
            for (int32_t size = t.e - t.b; size > kHandOff; size = (size + 1) / 2) k *= 2;
            parts += k;
        }
        const int grid = static_cast<int>(std::min<int64_t>(c->num_sms, parts));
        // scratch for them, and for what a larger batch of this design may take
        const int64_t room = std::max<int64_t>(
            grid, std::min<int64_t>(c->num_sms, 2 * static_cast<int64_t>(n) / kHandOff + 1));
        const double t0 = now_ms();
        int r2;
        const bool grow = s->ready.cap < cap;
        if ((r2 = s->tasks.ensure(c, kQueueHead + sizeof(SubTask) * static_cast<int64_t>(cap))) ||
            (r2 = s->ready.ensure(c, cap)) || (r2 = s->tfail.ensure(c, cap)) ||
            (r2 = s->swork.ensure(c, room * (kDescBytes + 6 * 8 * kStripeCap))))
            return r2;
        double *const strp = reinterpret_cast<double *>(s->swork.p + grid * kDescBytes);
        auto *const strlh =
            reinterpret_cast<unsigned long long *>(strp + grid * 4 * kStripeCap);
        if (grow || s->epoch == 0xffffffffu) {
            KTG_CUDA(c, cudaMemsetAsync(s->ready.p, 0, sizeof(unsigned) * s->ready.cap, c->stream));
            s->epoch = 0;
        }
        if (!s->subtree_attr) {
            KTG_CUDA(c, cudaFuncSetAttribute(k_subtree, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(kSubSmem)));
            s->subtree_attr = true;
        }
        std::vector<char> head(kQueueHead + sizeof(SubTask) * nt);
        SubQueue q{0, nt, nt, 0, 0};
        std::memcpy(head.data(), &q, sizeof(q));
        std::memcpy(head.data() + kQueueHead, tasks.data(), sizeof(SubTask) * nt);
        KTG_CUDA(c, cudaMemcpyAsync(s->tasks.p, head.data(), head.size(), cudaMemcpyHostToDevice,
                                    c->stream));
        SubTask *slots = reinterpret_cast<SubTask *>(s->tasks.p + kQueueHead);
        SubArgs A{slots, nt, cap, reinterpret_cast<SubQueue *>(s->tasks.p), s->ready.p, ++s->epoch,
                  s->tfail.p, s->cells.p, C, F, reinterpret_cast<SubDesc *>(s->swork.p), strp,
                  strlh, max_level, min_cells, stripe_extra, frac, c->density_limit,
                  exact ? 1 : 0, scale, inv_scale, s->windows ? kRowsLocal : -1};
        k_subtree<<<grid, kSubThreads, kSubSmem, c->stream>>>(A);
        ++c->launches;
        KTG_CUDA(c, cudaGetLastError());
        KTG_CUDA(c, cudaMemcpyAsync(&q, s->tasks.p, sizeof(q), cudaMemcpyDeviceToHost, c->stream));
        KTG_CUDA(c, lal_sync(c));
        if (q.timeout) return set_error(c, KTG_ERR_TIMEOUT, "legalizer: the block queue timed out");
        left.clear();
        if (q.nfail > 0) {
            std::vector<int2> fl(q.nfail);
            std::vector<SubTask> all(q.tail);
            KTG_CUDA(c, cudaMemcpyAsync(fl.data(), s->tfail.p, sizeof(int2) * q.nfail,
                                        cudaMemcpyDeviceToHost, c->stream));
            KTG_CUDA(c, cudaMemcpyAsync(all.data(), slots, sizeof(SubTask) * q.tail,
                                        cudaMemcpyDeviceToHost, c->stream));
            KTG_CUDA(c, lal_sync(c));
            for (const int2 &f : fl) {
                left.push_back(all[f.x]);
                s->stats[11] += 1;
                if (f.y >= 1 && f.y <= 4) s->stats[11 + f.y] += 1;
            }
            // disjoint position ranges: the level-by-level path takes them in order
            std::sort(left.begin(), left.end(),
                      [](const SubTask &a, const SubTask &b) { return a.b < b.b; });
        }
        s->stats[2] += 1;
        s->stats[4] += q.tail;
        s->stats[8] += now_ms() - t0;
        s->stats[10] += q.tail;
        return KTG_OK;
    };

    auto run_batch = [&]() -> int {
        const int32_t nreg = static_cast<int32_t>(batch.size());
        if (nreg == 0) return KTG_OK;
        const double t0 = now_ms();
        s->stats[0] += 1;
        s->stats[1] += nreg;
        int r2;
        std::vector<int32_t> rects(4 * nreg);
        std::vector<double> box(4 * nreg), room(nreg);
        for (int32_t r = 0; r < nreg; ++r) {
            for (int k = 0; k < 4; ++k) rects[4 * r + k] = batch[r][k];
            box[4 * r + 0] = c->origin_x + static_cast<double>(batch[r][0]) * c->dx;
            box[4 * r + 1] = c->origin_y + static_cast<double>(batch[r][2]) * c->dy;
            box[4 * r + 2] = c->origin_x + static_cast<double>(batch[r][1] + 1) * c->dx;
            box[4 * r + 3] = c->origin_y + static_cast<double>(batch[r][3] + 1) * c->dy;
            room[r] = HG.rect_sum(c->avail_host, batch[r].data());
        }
        if ((r2 = s->rects.ensure(c, 4 * nreg)) || (r2 = s->cnt.ensure(c, nreg + 1))) return r2;
        KTG_CUDA(c, cudaMemcpyAsync(s->rects.p, rects.data(), sizeof(int32_t) * rects.size(),
                                    cudaMemcpyHostToDevice, c->stream));
        KTG_CUDA(c, cudaMemsetAsync(s->map.p, 0xff, sizeof(int32_t) * nbins, c->stream));
        KTG_CUDA(c, cudaMemsetAsync(s->cnt.p, 0, sizeof(int32_t) * (nreg + 1), c->stream));
        k_region_map<<<dim3(64, std::min(nreg, 65535)), kT, 0, c->stream>>>(s->rects.p, nreg, nx, s->map.p);
        k_region_count<<<blocks_for(n), kT, 0, c->stream>>>(s->binof.p, n, s->map.p, s->cnt.p);
        c->launches += 2;
        std::vector<int32_t> cnt(nreg);
        KTG_CUDA(c, cudaMemcpyAsync(cnt.data(), s->cnt.p, sizeof(int32_t) * nreg,
                                    cudaMemcpyDeviceToHost, c->stream));
        KTG_CUDA(c, lal_sync(c));
        // level-1 blocks: one per region
        std::vector<int32_t> hb(nreg), he(nreg), hv(nreg, 1), hl(nreg, 1);
        int32_t run = 0;
        for (int32_t r = 0; r < nreg; ++r) {
            hb[r] = run;
            run += cnt[r];
            he[r] = run;
        }
        KTG_CUDA(c, cudaMemcpyAsync(s->cnt.p, hb.data(), sizeof(int32_t) * nreg,
                                    cudaMemcpyHostToDevice, c->stream));
        k_region_place<<<blocks_for(n), kT, 0, c->stream>>>(s->binof.p, n, s->map.p, s->cnt.p,
                                                             s->cells.p);
        ++c->launches;
        // host copies of the current level's blocks
        std::vector<double> hbox = box, hroom = room;
        for (;;) {
            // blocks that split: more than min_cells cells, below max_level;
            // small ones finish in the subtree kernel, the rest go level by level
            std::vector<int32_t> ab, ae, av, al;
            std::vector<double> abox, aroom;
            std::vector<SubTask> tasks;
            auto take = [&](size_t k) {
                ab.push_back(hb[k]);
                ae.push_back(he[k]);
                av.push_back(hv[k]);
                al.push_back(hl[k]);
                for (int q = 0; q < 4; ++q) abox.push_back(hbox[4 * k + q]);
                aroom.push_back(hroom[k]);
            };
            for (size_t k = 0; k < hb.size(); ++k) {
                if (he[k] - hb[k] <= min_cells || hl[k] >= max_level) continue;
                if (he[k] - hb[k] <= c->lal_subtree_cells) {
                    SubTask t;
                    for (int q = 0; q < 4; ++q) t.box[q] = hbox[4 * k + q];
                    t.room = hroom[k];
                    t.b = hb[k];
                    t.e = he[k];
                    t.level = hl[k];
                    t.vert = hv[k];
                    t.r0 = 0;
                    t.r1 = -1;
                    tasks.push_back(t);
                } else {
                    take(k);
                }
            }
            if (!tasks.empty()) {
                std::vector<SubTask> left;
                if ((r2 = run_subtree(tasks, left))) return r2;
                for (const SubTask &t : left) {
                    ab.push_back(t.b);
                    ae.push_back(t.e);
                    av.push_back(t.vert);
                    al.push_back(t.level);
                    for (int q = 0; q < 4; ++q) abox.push_back(t.box[q]);
                    aroom.push_back(t.room);
                }
            }
            const int32_t na = static_cast<int32_t>(ab.size());
            if (na == 0) break;
            s->stats[2] += 1;
            s->stats[4] += na;
            s->stats[9] += 1;
            // Room for the profiles and stripes of the blocks (steps, edges) and
            // of their halves, which have no more each; one copy takes the
            // level's descriptors to the device, one brings the halves back.
            std::vector<int64_t> soff(na), eoff(na), hsoff(2 * na), heoff(2 * na), stoff(2 * na),
                hcap(2 * na);
            int64_t st = 0, ed = 0, hst = 0, hed = 0, stripes = 0, max_steps = 0;
            int32_t maxlen = 0;
            for (int32_t k = 0; k < na; ++k) {
                int64_t ks, ke;
                s->profile_bound(&abox[4 * k], av[k] != 0, ks, ke);
                const int64_t ko = s->obstacle_bound(&abox[4 * k]);
                soff[k] = st;
                eoff[k] = ed;
                st += ks;
                ed += ke;
                max_steps = std::max(max_steps, ks);
                maxlen = std::max(maxlen, ae[k] - ab[k]);
                for (int side = 0; side < 2; ++side) {
                    // pe: the profile edges; pp: the prefix, then up to `edges` cuts
                    const int64_t edges = ke + 2 * ko + 2 + stripe_extra;
                    hsoff[2 * k + side] = hst;
                    heoff[2 * k + side] = hed;
                    hcap[2 * k + side] = edges;
                    stoff[2 * k + side] = stripes;
                    hst += ks;
                    hed += 2 * edges;
                    stripes += edges;
                }
            }
            std::vector<char> blob;
            auto pack = [&](const void *v, size_t bytes) {
                const size_t at = blob.size();
                blob.resize(at + (bytes + 7) / 8 * 8);
                std::memcpy(blob.data() + at, v, bytes);
                return at;
            };
            const size_t i32 = sizeof(int32_t) * na, i64 = sizeof(int64_t) * na;
            const size_t o_b = pack(ab.data(), i32), o_e = pack(ae.data(), i32),
                         o_v = pack(av.data(), i32), o_box = pack(abox.data(), 4 * i64),
                         o_room = pack(aroom.data(), i64), o_soff = pack(soff.data(), i64),
                         o_eoff = pack(eoff.data(), i64), o_hsoff = pack(hsoff.data(), 2 * i64),
                         o_heoff = pack(heoff.data(), 2 * i64), o_st = pack(stoff.data(), 2 * i64),
                         o_cap = pack(hcap.data(), 2 * i64);
            // the level's scratch, one allocation (a new context's first call at 12k
            // cells takes 2.5 ms; with one per array it took 5.2)
            size_t need = 0;
            auto carve = [&](size_t bytes) {
                const size_t at = need;
                need += (bytes + 255) / 256 * 256;
                return at;
            };
            const size_t n_steps = std::max(st, hst) + 1, n_edges = std::max(ed, hed) + 1,
                         n_st = stripes + 1;
            const size_t a_blob = carve(blob.size()), a_halves = carve(8 * i64 + i32 + 4),
                         a_low = carve(i64), a_high = carve(i64), a_cut = carve(i64),
                         a_nsteps = carve(2 * i64), a_count = carve(2 * i32),
                         a_steps = carve(sizeof(Key) * n_steps),
                         a_tmp = carve(sizeof(Key) * n_steps), a_pe = carve(8 * n_edges),
                         a_pp = carve(8 * n_edges), a_sa = carve(8 * n_st), a_sb = carve(8 * n_st),
                         a_cap = carve(8 * n_st), a_used = carve(8 * n_st), a_lo = carve(8 * n_st),
                         a_hi = carve(8 * n_st), a_beg = carve(4 * n_st),
                         a_ranges = carve(4 * i32);
            if ((r2 = s->level.ensure(c, static_cast<int64_t>(need)))) return r2;
            char *const slab = s->level.p;
            auto dbl = [&](size_t at) { return reinterpret_cast<double *>(slab + at); };
            auto i32p = [&](size_t at) { return reinterpret_cast<int32_t *>(slab + at); };
            auto i64p = [&](size_t at) { return reinterpret_cast<int64_t *>(slab + at); };
            auto d32 = [&](size_t o) { return i32p(a_blob + o); };
            auto d64 = [&](size_t o) { return i64p(a_blob + o); };
            Key *const steps = reinterpret_cast<Key *>(slab + a_steps);
            Key *const steps_tmp = reinterpret_cast<Key *>(slab + a_tmp);
            int64_t *const nsteps = i64p(a_nsteps);
            int32_t *const sbeg = i32p(a_beg);
            if (!s->wide_attr) {
                const std::pair<const void *, size_t> attrs[] = {
                    {reinterpret_cast<const void *>(k_block_cut_cta), kCtaStage},
                    {reinterpret_cast<const void *>(k_half_stripes_cta), kHalfStripesSmem},
                    {reinterpret_cast<const void *>(k_fill_fx), kFillSmem},
                    {reinterpret_cast<const void *>(k_sort_tiles), kTileSmem}};
                for (const auto &a : attrs)
                    KTG_CUDA(c, cudaFuncSetAttribute(a.first,
                                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     static_cast<int>(a.second)));
                s->wide_attr = true;
            }
            KTG_CUDA(c, cudaMemcpyAsync(slab + a_blob, blob.data(), blob.size(),
                                        cudaMemcpyHostToDevice, c->stream));
            Level L{na, d32(o_b), d32(o_e), dbl(a_blob + o_box), d32(o_v), dbl(a_blob + o_room),
                    i32p(a_halves + 8 * i64), dbl(a_low), dbl(a_high), dbl(a_cut), dbl(a_halves),
                    i32p(a_halves + 8 * i64 + i32)};
            const dim3 gcell(std::min(64, blocks_for(maxlen)), std::min(na, 65535));
            // 1. cells by centre
            Key *order, *sorted;
            k_centre_keys<<<gcell, kT, 0, c->stream>>>(L, C, s->cells.p, s->keys.p);
            if ((r2 = sort_segs(c, s->keys.p, s->keys_tmp.p, Segs{L.b, L.e, nullptr, nullptr}, na,
                                maxlen, &order)))
                return r2;
            k_keys_to_cells<<<gcell, kT, 0, c->stream>>>(L, order, s->cells.p);
            // 2. areas and median
            if (exact && (r2 = fx_prefix(run))) return r2;
            k_block_split<<<blocks_for(32 * static_cast<int64_t>(na)), kT, 0, c->stream>>>(
                L, C, s->cells.p, exact ? s->pre.p : nullptr, inv_scale);
            // 3. profile, cutline, half boxes
            k_steps_cta<<<na, 1024, 0, c->stream>>>(L, F, 0, d64(o_soff), steps, nsteps);
            c->launches += 4;
            if ((r2 = sort_segs(c, steps, steps_tmp,
                                Segs{nullptr, nullptr, d64(o_soff), nsteps}, na, max_steps,
                                &sorted)))
                return r2;
            k_block_cut_cta<<<na, kWideT, kCtaStage, c->stream>>>(
                L, F, d64(o_soff), sorted, nsteps, d64(o_eoff), dbl(a_pe), dbl(a_pp));
            // 4. stripes per half (profile arrays: e in pe, p and the cuts in pp)
            k_steps_cta<<<2 * na, 1024, 0, c->stream>>>(L, F, 1, d64(o_hsoff), steps,
                                                        nsteps);
            c->launches += 2;
            if ((r2 = sort_segs(c, steps, steps_tmp,
                                Segs{nullptr, nullptr, d64(o_hsoff), nsteps}, 2 * na, max_steps,
                                &sorted)))
                return r2;
            Stripes S{d64(o_st), i32p(a_count), dbl(a_sa), dbl(a_sb), dbl(a_cap), dbl(a_used),
                      reinterpret_cast<unsigned long long *>(slab + a_lo),
                      reinterpret_cast<unsigned long long *>(slab + a_hi)};
            k_half_stripes_cta<<<2 * na, kWideT, kHalfStripesSmem, c->stream>>>(
                L, F, d64(o_hsoff), sorted, nsteps, d64(o_heoff), dbl(a_pe), dbl(a_pp),
                d64(o_cap), frac, c->density_limit, S, c->status);
            // 5. fill order, fill, stripe ranges, positions
            auto fill = [&]() -> int {
                int r3;
                if (exact) {
                    if ((r3 = fx_prefix(run))) return r3;
                    k_fill_fx<<<2 * na, 1024, kFillSmem, c->stream>>>(L, S, s->pre.p, scale, sbeg);
                    k_stripe_ends<<<dim3(16, std::min(2 * na, 65535)), kT, 0, c->stream>>>(
                        L, C, s->cells.p, S, sbeg);
                    k_place_fx<<<gcell, kT, 0, c->stream>>>(L, C, s->cells.p, S, sbeg);
                } else {
                    if ((r3 = s->stripe_of.ensure(c, n + 1))) return r3;
                    k_fill<<<blocks_for(2 * na), kT, 0, c->stream>>>(L, C, s->cells.p, S,
                                                                     s->stripe_of.p);
                    k_stripe_minmax<<<gcell, kT, 0, c->stream>>>(L, C, s->cells.p, S,
                                                                 s->stripe_of.p);
                    k_new_pos<<<gcell, kT, 0, c->stream>>>(L, C, s->cells.p, S, s->stripe_of.p);
                }
                c->launches += 3;
                KTG_CUDA(c, cudaGetLastError());
                return KTG_OK;
            };
            k_fill_order<<<gcell, kT, 0, c->stream>>>(L, order, s->cells.p);
            c->launches += 2;
            if ((r2 = fill())) return r2;
            // children
            std::vector<char> back(8 * i64 + i32 + 4);
            KTG_CUDA(c, cudaMemcpyAsync(back.data(), slab + a_halves, back.size(),
                                        cudaMemcpyDeviceToHost, c->stream));
            KTG_CUDA(c, lal_sync(c));
            const double *halfbox = reinterpret_cast<const double *>(back.data());
            const int32_t *mh = reinterpret_cast<const int32_t *>(back.data() + 8 * i64);
            if (mh[na]) {  // long runs of one distance: the halves sorted, then filled
                std::vector<int32_t> ranges(4 * na);  // of the halves: first, end
                for (int32_t k = 0; k < na; ++k) {
                    ranges[2 * k] = ab[k];
                    ranges[2 * k + 1] = ranges[2 * na + 2 * k] = ab[k] + mh[k];
                    ranges[2 * na + 2 * k + 1] = ae[k];
                }
                KTG_CUDA(c, cudaMemcpyAsync(slab + a_ranges, ranges.data(), 4 * i32,
                                            cudaMemcpyHostToDevice, c->stream));
                KTG_CUDA(c, cudaMemsetAsync(L.redo, 0, sizeof(int32_t), c->stream));
                Key *const by = order == s->keys.p ? s->keys_tmp.p : s->keys.p;
                k_distance_keys<<<gcell, kT, 0, c->stream>>>(L, order, by);
                if ((r2 = sort_segs(c, by, order,
                                    Segs{i32p(a_ranges), i32p(a_ranges) + 2 * na, nullptr, nullptr},
                                    2 * na, maxlen, &order)))
                    return r2;
                k_keys_to_cells<<<gcell, kT, 0, c->stream>>>(L, order, s->cells.p);
                c->launches += 2;
                if ((r2 = fill())) return r2;
            }
            hb.clear();
            he.clear();
            hv.clear();
            hl.clear();
            hbox.clear();
            hroom.clear();
            for (int32_t k = 0; k < na; ++k) {
                for (int side = 0; side < 2; ++side) {
                    hb.push_back(side ? ab[k] + mh[k] : ab[k]);
                    he.push_back(side ? ae[k] : ab[k] + mh[k]);
                    hv.push_back(av[k] ? 0 : 1);
                    hl.push_back(al[k] + 1);
                    for (int q = 0; q < 4; ++q) hbox.push_back(halfbox[8 * k + 4 * side + q]);
                    hroom.push_back(aroom[k]);
                }
            }
        }
        batch.clear();
        batch_reach.clear();
        s->stats[5] += now_ms() - t0;
        return refresh();
    };

    for (const auto &cl : HG.clusters(occ)) {
        auto bins = HG.grown(cl, occ);
        bool clash = false;
        const auto rb = reach(bins);
        for (const auto &t : batch_reach)
            if (touches(t, rb)) clash = true;
        if (clash) {
            if ((rc = run_batch())) return rc;
            bins = HG.grown(cl, occ);
        }
        batch.push_back(bins);
        batch_reach.push_back(reach(bins));
    }
    if ((rc = run_batch())) return rc;
    if (n > 0) {
        k_clamp_die<<<blocks_for(n), kT, 0, c->stream>>>(C, n, s->die[0], s->die[1], s->die[2],
                                                         s->die[3]);
        ++c->launches;
    }
    KTG_CUDA(c, cudaGetLastError());
    s->stats[7] = now_ms() - t_start;
    return KTG_OK;
}

int lal_stats(ktg_ctx *c, double *out, int count) {
    for (int k = 0; k < count && k < 16; ++k) out[k] = c->lal ? c->lal->stats[k] : 0.0;
    return KTG_OK;
}

}  // namespace ktg
