// batch.cu -- batched exact k-NN over many independent point clouds.
//
// Build: every point gets the key (cloud id << 3B) | Morton_B(point in its
// cloud's box), B bits per axis; one radix sort of all keys puts each
// cloud's points together in Morton order, and one Karras tree over the
// whole key array is a forest whose node covering a cloud's key range is
// that cloud's LBVH (keys sharing the cloud prefix form a subtree of a
// binary radix tree).  Search: work items of <= 32 Morton-ordered queries of
// one cloud, taken from device counters by two persistent launches.  Lists
// of more than 8 are collected by a warp per query (knn_collect.cuh) on a
// side stream, longest first; shorter lists run a thread per query from the
// query's Morton neighbours (knn_traverse.cuh) in the second launch, whose
// blocks take the SMs as the first one's leave.  The second launch also
// holds the warp-per-query lists of passes with partial_results and the
// memory lists of more than 512 entries.  256 clouds, 9M points, 2.2M
// queries, k from {1, 5, 16, 64}: 25.0 ms with radius rounds and merged
// warp lists, now 6.4 ms; bound by instruction issue (0.85 of the slots).
// The whole pass is launch-only (no host synchronisation), so it can be
// captured as one CUDA graph and replayed.
#include <algorithm>
#include <new>
#include <vector>

#include "knn_backward.cuh"
#include "knn_collect.cuh"
#include "knn_traverse.cuh"

struct rtd_batch;

namespace rtd {
namespace {

constexpr int BLOCK = 256;
constexpr int SWARPS = 4;   // warps per block of the search kernel

struct CloudDesc {
    uint32_t pt_begin, n_pts, q_begin, n_q;
    uint32_t k, root, root_count, box[6];
    float r0sq;
    uint64_t out_off;
};

struct WorkItem {
    uint32_t cloud, start, count, cls;   // cls: k class (k_class), the search it runs
};

__global__ void batch_reset_kernel(CloudDesc *cd, uint32_t n_clouds) {
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n_clouds; c += gridDim.x * blockDim.x) {
        for (int a = 0; a < 3; ++a) {
            cd[c].box[a] = 0xFFFFFFFFu;
            cd[c].box[3 + a] = 0u;
        }
        cd[c].root = cd[c].n_pts == 0 ? CHILD_NONE : (CHILD_LEAF | cd[c].pt_begin);
        cd[c].root_count = cd[c].n_pts;
    }
}

// Cloud id of every point and every query (one block per cloud).
__global__ void batch_cloud_of_kernel(const CloudDesc *__restrict__ cd, uint32_t *__restrict__ pcloud,
                                      uint32_t *__restrict__ qcloud) {
    const uint32_t c = blockIdx.x;
    const CloudDesc d = cd[c];
    for (uint32_t i = threadIdx.x; i < d.n_pts; i += blockDim.x) pcloud[d.pt_begin + i] = c;
    for (uint32_t i = threadIdx.x; i < d.n_q; i += blockDim.x) qcloud[d.q_begin + i] = c;
}

// Per-cloud bounding boxes (NaN-ignoring).  A warp walks a run of consecutive
// points and keeps their box until the cloud changes, so that a cloud's six
// words take an atomic each a warp and cloud, not one every 32 points (8 M
// points: 192 us, now 58).
__global__ void __launch_bounds__(BLOCK) batch_bbox_kernel(const float *__restrict__ xyz, uint64_t n,
                                                           const uint32_t *__restrict__ pcloud,
                                                           CloudDesc *cd) {
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (BLOCK / 32), w = ((uint64_t)blockIdx.x * BLOCK + threadIdx.x) >> 5;
    const uint64_t run = ((n + warps - 1) / warps + 31) & ~31ull;
    const uint64_t first = w * run, last = first + run < n ? first + run : n;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    uint32_t cur = 0xFFFFFFFFu;   // the cloud of lo, hi; the same in every lane
    auto flush = [&]() {
        if (cur == 0xFFFFFFFFu) return;
        for (int a = 0; a < 3; ++a) {
            for (int o = 16; o > 0; o >>= 1) {
                lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
                hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
            }
            if (lane == 0 && lo[a] <= hi[a]) {   // (some coordinate was a number)
                atomicMin(&cd[cur].box[a], float_flip(lo[a]));
                atomicMax(&cd[cur].box[3 + a], float_flip(hi[a]));
            }
            lo[a] = INFINITY;
            hi[a] = -INFINITY;
        }
    };
    for (uint64_t base = first; base < last; base += 32) {
        const uint64_t i = base + lane;
        const bool ok = i < last;
        const uint32_t c = ok ? pcloud[i] : 0xFFFFFFFFu;
        float v[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) v[a] = ok ? xyz[3 * i + a] : NAN;
        // the clouds of these points, in order
        uint32_t left = __ballot_sync(0xffffffffu, ok);
        while (left) {
            const uint32_t c0 = __shfl_sync(0xffffffffu, c, __ffs(left) - 1);
            if (c0 != cur) {
                flush();
                cur = c0;
            }
            const bool mine = ok && c == c0;
            if (mine) {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    lo[a] = fminf(lo[a], v[a]);
                    hi[a] = fmaxf(hi[a], v[a]);
                }
            }
            left &= ~__ballot_sync(0xffffffffu, mine);
        }
    }
    flush();
}

// Initial radius of a cloud: `fixed` when > 0, else `mult` x the radius of
// a ball expected to hold k points at the cloud's mean density,
// (3 k V / 4 pi n)^(1/3).  Box extents are clamped to >= max extent /
// sqrt(n), which makes the estimate the mean spacing of a flat (2-D) cloud;
// an estimate that is too large only costs pruning, one that is too small
// costs extra rounds.
__global__ void batch_seed_kernel(CloudDesc *cd, uint32_t n_clouds, float fixed, float mult) {
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n_clouds; c += gridDim.x * blockDim.x) {
        float r = fixed;
        if (!(r > 0.0f)) {
            const float n = (float)(cd[c].n_pts > 0 ? cd[c].n_pts : 1);
            float e[3], emax = 0.0f;
            for (int a = 0; a < 3; ++a) {
                const float lo = float_unflip(cd[c].box[a]), hi = float_unflip(cd[c].box[3 + a]);
                e[a] = hi - lo;
                if (!isfinite(e[a]) || !(e[a] > 0.0f)) e[a] = 0.0f;
                emax = fmaxf(emax, e[a]);
            }
            const float emin = fmaxf(emax / sqrtf(n), 1e-20f);
            const float v = fmaxf(e[0], emin) * fmaxf(e[1], emin) * fmaxf(e[2], emin);
            r = mult * cbrtf(3.0f * (float)cd[c].k * v / (4.0f * 3.14159265f * n));
        }
        if (!(r > 0.0f) || !(r < INFINITY)) r = 1.0f;
        cd[c].r0sq = r * r;
    }
}

__global__ void __launch_bounds__(BLOCK) batch_keys_kernel(const float *__restrict__ xyz, uint64_t n,
                                                           const uint32_t *__restrict__ cloud_of,
                                                           const CloudDesc *__restrict__ cd,
                                                           int bpa, uint64_t *__restrict__ keys) {
    const float scale = (float)((1u << bpa) - 1u);
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * BLOCK) {
        const uint32_t c = cloud_of[i];
        // one cubic extent per cloud (the largest axis), as for single indexes
        float lo[3], ext = 1e-6f;
        for (int a = 0; a < 3; ++a) {
            const float hi = float_unflip(cd[c].box[3 + a]);
            lo[a] = float_unflip(cd[c].box[a]);
            ext = fmaxf(ext, __fsub_rn(hi, lo[a]));
        }
        uint32_t u[3];
        for (int a = 0; a < 3; ++a) u[a] = quantize(xyz[3 * i + a], lo[a], ext, scale);
        keys[i] = ((uint64_t)c << (3 * bpa)) | morton63(u[0], u[1], u[2]);
    }
}

// The points in key order.  Clouds lie in the same order as their keys, so
// the cloud of sorted position i is that of input point i.  Bound by the
// scattered reads of the points (8 M points: 139 us with the cloud read by
// input point as well, now 90).
__global__ void __launch_bounds__(BLOCK) batch_gather_kernel(const float *__restrict__ xyz,
                                                             const uint32_t *__restrict__ perm,
                                                             const uint32_t *__restrict__ pcloud,
                                                             const CloudDesc *__restrict__ cd,
                                                             uint64_t n, int vec4, float4 *__restrict__ pts) {
    const uint64_t stride = (uint64_t)gridDim.x * BLOCK;
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < n; i += stride) {
        const uint32_t o = perm[i];
        float x, y, z;
        load_point(xyz, o, n, vec4, x, y, z);
        pts[i] = make_float4(x, y, z, __uint_as_float(o - cd[pcloud[i]].pt_begin));
    }
}

// The kept forest node whose range is exactly a cloud's points is that
// cloud's root.
__global__ void __launch_bounds__(BLOCK) batch_roots_kernel(
    const uint64_t *__restrict__ skeys, uint64_t n, int shift, const uint32_t *__restrict__ kfirst,
    const uint32_t *__restrict__ klast, const KeptNodes kept, CloudDesc *cd) {
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i + 1 < n;
         i += (uint64_t)gridDim.x * BLOCK) {
        // only kept nodes carry their range; a cloud of <= leaf_size points
        // keeps the leaf root batch_reset_kernel gave it
        if (!kept.has((uint32_t)i)) continue;
        const uint32_t f = kfirst[i], l = klast[i];
        const uint32_t c = (uint32_t)(skeys[f] >> shift);
        const CloudDesc d = cd[c];
        if (f == d.pt_begin && l + 1 == d.pt_begin + d.n_pts) {
            cd[c].root = kept.number((uint32_t)i);
            cd[c].root_count = d.n_pts;
        }
    }
}

struct BatchArgs {
    const float4 *pts;
    const BvhNode *nodes;
    const IndexHeader *hdr;
    const CloudDesc *cd;
    const WorkItem *items;
    uint32_t n_items;
    uint32_t *counter;
    const uint32_t *qperm;
    const float *q;
    uint32_t *ids;
    float *d2;
    float mult2;
    uint32_t max_rounds;
    uint32_t partial;   // the reference's round cap (rtd_schedule.partial_results)
    uint32_t *err;
    uint2 *wide;        // per-warp list slabs of the widest class
    uint32_t wide_kk;   // entries per slab: the largest min(k, points) of that class
    // exact passes: the sorted keys of the points and of the queries (in item
    // order), and the box pyramid over the sorted points
    const uint64_t *skeys, *qskeys;
    const float4 *pyr;
    uint32_t n_points;
    uint32_t collect_kk, collect_n;   // largest min(k, points) and points of the collecting clouds
};

// Position of the queries of an item among their cloud's sorted keys.
__device__ __forceinline__ uint32_t cloud_position(const BatchArgs &a, const CloudDesc &c, uint64_t key) {
    uint32_t lo = c.pt_begin, hi = c.pt_begin + c.n_pts;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&a.skeys[mid]) < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

template <int KC>
__device__ __forceinline__ void item_thread(const BatchArgs &a, const TreeRef &t,
                                            const RoundSpec &rs, const CloudDesc &c,
                                            const WorkItem &w, uint2 *s_col, uint2 *l_stack) {
    const int lane = threadIdx.x & 31;
    if ((uint32_t)lane >= w.count) return;
    const uint32_t qi = a.qperm[w.start + lane];
    const float qx = a.q[3 * (uint64_t)qi], qy = a.q[3 * (uint64_t)qi + 1], qz = a.q[3 * (uint64_t)qi + 2];
    const int kk = (int)c.k;
    float bk[KC];
    uint32_t bi[KC];
    if (a.skeys) {
        // one unbounded round from the 4k points around the query in the
        // cloud's Morton order
        list_init<KC>(bk, bi, kk);
        const uint32_t pos = cloud_position(a, c, a.qskeys[w.start + lane]);
        const uint32_t n = 4u * (uint32_t)kk < c.n_pts ? 4u * (uint32_t)kk : c.n_pts;
        uint32_t w0 = pos - c.pt_begin > n / 2u ? pos - n / 2u : c.pt_begin;
        if (w0 + n > c.pt_begin + c.n_pts) w0 = c.pt_begin + c.n_pts - n;
        for (uint32_t j = w0; j < w0 + n; ++j) {
            const float4 pt = __ldg(&t.pts[j]);
            const float key = exact_key(qx, qy, qz, pt.x, pt.y, pt.z);
            const uint32_t id = __float_as_uint(pt.w);
            if (key_less(key, id, bk[KC - 1], bi[KC - 1])) list_insert<KC>(bk, bi, key, id);
        }
        const RoundSpec one{rs.r0sq, rs.mult2, 1u, 0u};
        knn_query_thread<KC, true>(t, one, qx, qy, qz, kk, s_col, 32, l_stack, a.err, bk, bi, w0, w0 + n);
    } else {
        knn_query_thread<KC>(t, rs, qx, qy, qz, kk, s_col, 32, l_stack, a.err, bk, bi);
    }
    const uint64_t ob = c.out_off + (uint64_t)(qi - c.q_begin) * kk;
#pragma unroll
    for (int j = 0; j < KC; ++j)
        if (j >= KC - kk) {
            a.ids[ob + j - (KC - kk)] = bi[j];
            if (a.d2) a.d2[ob + j - (KC - kk)] = bk[j];
        }
}

template <int S>
__device__ __forceinline__ void item_warp(const BatchArgs &a, const TreeRef &t, const RoundSpec &rs,
                                          const CloudDesc &c, const WorkItem &w, uint2 *stk,
                                          uint2 *ls) {
    const int lane = threadIdx.x & 31;
    for (uint32_t j = 0; j < w.count; ++j) {
        const uint32_t qi = a.qperm[w.start + j];
        const float qx = a.q[3 * (uint64_t)qi], qy = a.q[3 * (uint64_t)qi + 1], qz = a.q[3 * (uint64_t)qi + 2];
        float lk[S];
        uint32_t li[S];
        knn_query_warp<S>(t, rs, qx, qy, qz, c.k, stk, ls, a.err, lk, li);
        const uint64_t ob = c.out_off + (uint64_t)(qi - c.q_begin) * c.k;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const uint32_t slot = (uint32_t)(s * 32 + lane);
            if (slot < c.k) {
                a.ids[ob + slot] = li[s];
                if (a.d2) a.d2[ob + slot] = lk[s];
            }
        }
    }
}

__device__ __forceinline__ void item_wide(const BatchArgs &a, const TreeRef &t, const RoundSpec &rs,
                                          const CloudDesc &c, const WorkItem &w, uint2 *stk,
                                          uint32_t *s_r, uint2 *slab) {
    WideList list;
    list.L = slab;
    list.s_r = s_r;
    list.kk = c.k < c.n_pts ? c.k : (c.n_pts ? c.n_pts : 1u);
    for (uint32_t j = 0; j < w.count; ++j) {
        const uint32_t qi = a.qperm[w.start + j];
        const float qx = a.q[3 * (uint64_t)qi], qy = a.q[3 * (uint64_t)qi + 1], qz = a.q[3 * (uint64_t)qi + 2];
        knn_query_warp_list(t, rs, qx, qy, qz, stk, a.err, list);
        const uint64_t ob = c.out_off + (uint64_t)(qi - c.q_begin) * c.k;
        wide_list_store(list, c.k, a.ids + ob, a.d2 ? a.d2 + ob : nullptr);
        __syncwarp();
    }
}

// k classes of the search: register lists (thread per query), warp lists
// of 32, 64 or 256 slots (warp per query; passes with partial_results),
// memory list (warp per query), and collected lists (knn_collect.cuh, warp
// per query, in a launch of their own).
enum : uint32_t { CLS_T1, CLS_T5, CLS_T8, CLS_T16, CLS_W32, CLS_W64, CLS_W256, CLS_WIDE, CLS_COLLECT, N_CLASSES };
// Lists above this are collected: all 256 clouds of 1,000 to 200,000 points
// with k = 16, a thread / a warp per query: 11.1 / 10.2 ms, of up to 8,000
// points 1.20 / 0.93 ms; with k = 5 the thread's list is far shorter.
constexpr uint32_t COLLECT_ABOVE = 8;
constexpr uint32_t BATCH_COLLECT_MAX = 512;     // entries: 11 KB of shared memory a warp
inline uint32_t k_class(uint32_t k, uint32_t n, bool exact, bool warp) {
    const uint32_t kk = k < n ? k : n;
    if (exact && (k > COLLECT_ABOVE || warp) && kk <= BATCH_COLLECT_MAX) return CLS_COLLECT;
    if (k <= 16 && !warp) return k <= 1 ? CLS_T1 : k <= 5 ? CLS_T5 : k <= 8 ? CLS_T8 : CLS_T16;
    return k <= 32 ? CLS_W32 : k <= 64 ? CLS_W64 : k <= 256 ? CLS_W256 : CLS_WIDE;
}

// Shared memory of one warp, reused by whichever class its current item
// has: the thread classes' short stacks (SHORT_STACK x 32 entries, one
// column per lane) or the warp classes' stack, list scratch and rank words.
constexpr int WARP_SMEM = SHORT_STACK * 32;   // uint2 entries (3 KB)
static_assert(STACK_MAX + 256 + 16 <= WARP_SMEM, "warp classes fit the thread stacks' space");

__global__ void __launch_bounds__(SWARPS * 32) batch_knn_kernel(const BatchArgs a) {
    __shared__ uint2 s_warp[SWARPS][WARP_SMEM];
    uint2 l_stack[STACK_MAX - SHORT_STACK];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint2 *const sw = s_warp[warp];
    uint2 *const stk = sw;                       // warp classes: STACK_MAX entries
    uint2 *const ls = sw + STACK_MAX;            // list scratch (256 entries)
    uint32_t *const s_r = reinterpret_cast<uint32_t *>(sw + STACK_MAX + 256);   // 32 words
    uint2 *const slab = a.wide ? a.wide + ((size_t)blockIdx.x * SWARPS + warp) * a.wide_kk : nullptr;
    const uint32_t visit_cap = 2u * a.hdr->n_internal + 4u;
    while (true) {
        uint32_t it = 0;
        if (lane == 0) it = atomicAdd(a.counter, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= a.n_items) break;
        const WorkItem w = a.items[it];
        const CloudDesc c = a.cd[w.cloud];
        const TreeRef t{a.pts, a.nodes, nullptr, c.root, c.root_count, visit_cap};
        const RoundSpec rs{c.r0sq, a.mult2, a.max_rounds, a.partial};
        switch (w.cls) {
        case CLS_T1: item_thread<1>(a, t, rs, c, w, sw + lane, l_stack); break;
        case CLS_T5: item_thread<5>(a, t, rs, c, w, sw + lane, l_stack); break;
        case CLS_T8: item_thread<8>(a, t, rs, c, w, sw + lane, l_stack); break;
        case CLS_T16: item_thread<16>(a, t, rs, c, w, sw + lane, l_stack); break;
        case CLS_W32: item_warp<1>(a, t, rs, c, w, stk, ls); break;
        case CLS_W64: item_warp<2>(a, t, rs, c, w, stk, ls); break;
        case CLS_W256: item_warp<8>(a, t, rs, c, w, stk, ls); break;
        default: item_wide(a, t, rs, c, w, stk, s_r, slab); break;
        }
        __syncwarp();
    }
}

// The collected lists: a persistent launch over their items, a quarter of
// an item (8 queries) at a time, so that the last ones end close together.
constexpr uint32_t COLLECT_PART = 8;
__global__ void __launch_bounds__(SWARPS * 32, 10) batch_collect_kernel(const BatchArgs a) {
    extern __shared__ uint2 s_dyn[];
    __shared__ uint32_t s_off[12];
    if (threadIdx.x == 0) collect_offsets(a.n_points, s_off);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    char *base = reinterpret_cast<char *>(s_dyn) + (size_t)warp * collect_warp_bytes(a.collect_kk, a.collect_n);
    while (true) {
        uint32_t it = 0;
        if (lane == 0) it = atomicAdd(a.counter, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it / (32 / COLLECT_PART) >= a.n_items) break;
        const WorkItem w = a.items[it / (32 / COLLECT_PART)];
        const CloudDesc c = a.cd[w.cloud];
        const uint32_t kk = c.k < c.n_pts ? c.k : (c.n_pts ? c.n_pts : 1u);
        const CollectScratch s = collect_scratch(base, kk, c.n_pts);
        const CollectTree tree{a.pts, a.pyr, s_off, c.pt_begin, c.pt_begin + c.n_pts};
        // the positions of the part's queries, one a lane
        const uint32_t j0 = it % (32 / COLLECT_PART) * COLLECT_PART;
        const uint32_t have = w.count > j0 ? min(w.count - j0, COLLECT_PART) : 0u;
        uint32_t my_pos = 0;
        if ((uint32_t)lane < have) my_pos = cloud_position(a, c, a.qskeys[w.start + j0 + lane]);
        __syncwarp();
        for (uint32_t j = 0; j < have; ++j) {
            const uint32_t qi = a.qperm[w.start + j0 + j], pos = __shfl_sync(0xffffffffu, my_pos, j);
            const float qx = a.q[3 * (uint64_t)qi], qy = a.q[3 * (uint64_t)qi + 1], qz = a.q[3 * (uint64_t)qi + 2];
            const Collected got = collect_query<false>(tree, s, qx, qy, qz, kk, pos);
            const uint64_t ob = c.out_off + (uint64_t)(qi - c.q_begin) * c.k;
            collect_store(s, got, kk, c.k, a.ids + ob, a.d2 ? a.d2 + ob : nullptr);
        }
    }
}

__global__ void __launch_bounds__(256) batch_backward_kernel(const float *__restrict__ q, uint64_t nq,
                                                             const float *__restrict__ pts,
                                                             const uint32_t *__restrict__ qcloud,
                                                             const CloudDesc *__restrict__ cd,
                                                             const uint32_t *__restrict__ ids,
                                                             const float *__restrict__ g, float *__restrict__ gq,
                                                             float *__restrict__ gp) {
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < nq; i += (uint64_t)gridDim.x * 256) {
        const CloudDesc &c = cd[qcloud[i]];
        const uint64_t ob = c.out_off + (uint64_t)(i - c.q_begin) * c.k;
        // (a cloud's rows may start at an odd point, 4 bytes off)
        float *const cgp = gp ? gp + 3 * (uint64_t)c.pt_begin : nullptr;
        backward_query(q, pts + 3 * (uint64_t)c.pt_begin, c.n_pts, c.k, ids + ob, g + ob, gq, cgp, i,
                       backward_pairs(cgp));
    }
}

}  // namespace
}  // namespace rtd

using namespace rtd;

struct rtd_batch {
    std::vector<rtd_cloud> clouds;
    uint32_t n_clouds = 0, n_items = 0;
    uint32_t n_collect = 0;     // items of the collected lists, ahead of the others
    uint32_t collect_kk = 0, collect_n = 0;
    int blocks = 0, collect_blocks = 0;   // grids of the persistent searches
    uint32_t wide_kk = 0;       // list slab entries per warp (0: no k > 256 cloud)
    uint64_t n_points = 0, n_queries = 0;
    int cbits = 0, bpa = 21;
    rtd_schedule sched;
    rtd_index forest;
    DevBuf cd, items, pcloud, qcloud, qkeys, qkeys_alt, qvals, qvals_alt, counter, wide;
    // captured graph and the pointers it was captured with
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    const void *g_pts = nullptr, *g_q = nullptr;
    void *g_ids = nullptr, *g_d2 = nullptr;
    cudaStream_t g_stream = nullptr;
    void drop_graph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
    }
    ~rtd_batch() { drop_graph(); }
};

namespace rtd {

rtd_status check_index_errors(rtd_index *idx, cudaStream_t st);

static rtd_status batch_pass(rtd_batch *b, const float *d_pts, const float *d_q, uint32_t *d_ids,
                             float *d_d2, cudaStream_t st) {
    rtd_index &f = b->forest;
    const uint64_t n = b->n_points, nq = b->n_queries;
    CloudDesc *cd = b->cd.as<CloudDesc>();
    IndexHeader *h = f.hdr.as<IndexHeader>();
    RTD_CUDA(cudaMemsetAsync(h, 0, sizeof(IndexHeader), st));
    RTD_CUDA(cudaMemsetAsync(b->counter.ptr, 0, 2 * sizeof(uint32_t), st));
    batch_reset_kernel<<<grid_for(b->n_clouds, 128, 1024), 128, 0, st>>>(cd, b->n_clouds);
    RTD_LAUNCH_CHECK();
    batch_cloud_of_kernel<<<b->n_clouds, 256, 0, st>>>(cd, b->pcloud.as<uint32_t>(),
                                                        b->qcloud.as<uint32_t>());
    RTD_LAUNCH_CHECK();
    const int g = grid_for(n, BLOCK, 148 * 8);
    if (n) {
        batch_bbox_kernel<<<grid_for(n, BLOCK, 148 * 4), BLOCK, 0, st>>>(d_pts, n, b->pcloud.as<uint32_t>(), cd);
        RTD_LAUNCH_CHECK();
    }
    batch_seed_kernel<<<grid_for(b->n_clouds, 128, 1024), 128, 0, st>>>(
        cd, b->n_clouds, b->sched.radius_heuristic == RTD_RADIUS_FIXED ? b->sched.radius_param : 0.0f,
        b->sched.radius_param);
    RTD_LAUNCH_CHECK();
    const int kbits = 3 * b->bpa + b->cbits;
    const uint64_t *skeys = nullptr;
    if (n) {
        batch_keys_kernel<<<g, BLOCK, 0, st>>>(d_pts, n, b->pcloud.as<uint32_t>(), cd, b->bpa,
                                              f.keys.as<uint64_t>());
        RTD_LAUNCH_CHECK();
        bool alt = false;
        RTD_TRY(radix_sort_pairs<uint64_t>(f.keys.as<uint64_t>(), f.keys_alt.as<uint64_t>(),
                                           f.vals.as<uint32_t>(), f.vals_alt.as<uint32_t>(), true, n,
                                           0, kbits, f.sort, &h->err, st, &alt));
        const uint64_t *sk = alt ? f.keys_alt.as<uint64_t>() : f.keys.as<uint64_t>();
        skeys = sk;
        const uint32_t *perm = alt ? f.vals_alt.as<uint32_t>() : f.vals.as<uint32_t>();
        batch_gather_kernel<<<g, BLOCK, 0, st>>>(d_pts, perm, b->pcloud.as<uint32_t>(), cd, n,
                                                 ((uintptr_t)d_pts & 15u) == 0 ? 1 : 0, f.pts.as<float4>());
        RTD_LAUNCH_CHECK();
        RTD_TRY(build_tree_sorted<uint64_t>(&f, sk, n, st, true));
        if (n >= 2 && n > f.leaf_size) {
            batch_roots_kernel<<<grid_for(n, BLOCK, 148 * 8), BLOCK, 0, st>>>(
                sk, n, 3 * b->bpa, f.kfirst.as<uint32_t>(), f.klast.as<uint32_t>(),
                KeptNodes{f.kept_bits.as<uint32_t>(), f.kept_before.as<uint32_t>()}, cd);
            RTD_LAUNCH_CHECK();
        }
    }
    if (nq) {
        batch_keys_kernel<<<grid_for(nq, BLOCK, 148 * 8), BLOCK, 0, st>>>(
            d_q, nq, b->qcloud.as<uint32_t>(), cd, b->bpa, b->qkeys.as<uint64_t>());
        RTD_LAUNCH_CHECK();
        bool alt = false;
        RTD_TRY(radix_sort_pairs<uint64_t>(b->qkeys.as<uint64_t>(), b->qkeys_alt.as<uint64_t>(),
                                           b->qvals.as<uint32_t>(), b->qvals_alt.as<uint32_t>(),
                                           true, nq, 0, kbits, f.sort, &h->err, st, &alt));
        BatchArgs a;
        a.pts = f.pts.as<float4>();
        a.nodes = f.nodes.as<BvhNode>();
        a.hdr = h;
        a.cd = cd;
        a.items = nullptr;
        a.n_items = 0;
        a.counter = nullptr;
        a.qperm = alt ? b->qvals_alt.as<uint32_t>() : b->qvals.as<uint32_t>();
        a.q = d_q;
        a.ids = d_ids;
        a.d2 = d_d2;
        const float m = b->sched.radius_increment_mult;
        a.mult2 = m * m;
        a.max_rounds = b->sched.max_rounds;
        a.partial = b->sched.partial_results ? 1u : 0u;
        a.err = &h->err;
        a.wide = b->wide_kk ? b->wide.as<uint2>() : nullptr;
        a.wide_kk = b->wide_kk;
        // (without points no key is read: every window is empty)
        a.skeys = a.partial ? nullptr : n ? skeys : b->qkeys.as<uint64_t>();
        a.qskeys = alt ? b->qkeys_alt.as<uint64_t>() : b->qkeys.as<uint64_t>();
        a.pyr = f.pyramid.as<float4>();
        a.n_points = (uint32_t)n;
        a.collect_kk = b->collect_kk;
        a.collect_n = b->collect_n;
        // The collected lists run on the side stream; the other classes'
        // blocks take the SMs as theirs leave.
        const bool both = b->n_collect && b->n_items;
        cudaStream_t cs = st;
        if (both) {
            RTD_TRY(ensure_side_stream(&f));
            cs = f.side_stream;
            RTD_CUDA(cudaEventRecord(f.ev_fork, st));
            RTD_CUDA(cudaStreamWaitEvent(cs, f.ev_fork, 0));
        }
        cudaError_t ce = cudaSuccess;
        if (b->n_collect) {
            a.items = b->items.as<WorkItem>();
            a.n_items = b->n_collect;
            a.counter = b->counter.as<uint32_t>() + 1;
            batch_collect_kernel<<<b->collect_blocks, SWARPS * 32,
                                   SWARPS * collect_warp_bytes(b->collect_kk, b->collect_n), cs>>>(a);
            note_launch();
            ce = cudaGetLastError();
        }
        if (both) RTD_CUDA(cudaEventRecord(f.ev_join, cs));
        cudaError_t te = cudaSuccess;
        if (b->n_items) {
            a.items = b->items.as<WorkItem>() + b->n_collect;
            a.n_items = b->n_items;
            a.counter = b->counter.as<uint32_t>();
            batch_knn_kernel<<<b->blocks, SWARPS * 32, 0, st>>>(a);
            note_launch();
            te = cudaGetLastError();
        }
        if (both) RTD_CUDA(cudaStreamWaitEvent(st, f.ev_join, 0));   // also on the error paths
        if (ce != cudaSuccess) return cuda_fail(ce, "batch_collect_kernel launch");
        if (te != cudaSuccess) return cuda_fail(te, "batch_knn_kernel launch");
    }
    return RTD_OK;
}

}  // namespace rtd

extern "C" {

void rtd_batch_schedule_default(rtd_schedule *s) {
    if (!s) return;
    rtd_schedule_default(s);
    s->radius_param = 1.0f;
}

rtd_status rtd_batch_create(rtd_batch **out) {
    if (!out) return fail(RTD_ERR_INVALID_ARGUMENT, "out is NULL");
    *out = new (std::nothrow) rtd_batch();
    if (!*out) return fail(RTD_ERR_OUT_OF_MEMORY, "host allocation failed");
    rtd_batch_schedule_default(&(*out)->sched);
    return RTD_OK;
}

rtd_status rtd_batch_destroy(rtd_batch *b) {
    delete b;
    return RTD_OK;
}

rtd_status rtd_batch_plan(rtd_batch *b, const rtd_cloud *clouds, uint32_t n_clouds,
                          const rtd_schedule *sched) {
    if (!b || (n_clouds && !clouds)) return fail(RTD_ERR_INVALID_ARGUMENT, "NULL argument");
    rtd_schedule s;
    rtd_batch_schedule_default(&s);
    if (sched) s = *sched;
    if (!(s.radius_increment_mult > 1.0f)) return fail(RTD_ERR_INVALID_ARGUMENT, "radius_increment_mult must be > 1");
    if (s.max_rounds < 1) return fail(RTD_ERR_INVALID_ARGUMENT, "max_rounds must be >= 1");
    if (s.leaf_size < 1 || s.leaf_size > 64) return fail(RTD_ERR_INVALID_ARGUMENT, "leaf_size must be in [1, 64]");
    uint64_t np = 0, nq = 0;
    uint32_t wide_kk = 0, collect_kk = 0, collect_n = 0;
    std::vector<CloudDesc> cd(n_clouds);
    std::vector<WorkItem> cls_items[N_CLASSES];
    for (uint32_t c = 0; c < n_clouds; ++c) {
        const rtd_cloud &x = clouds[c];
        if (x.point_offset != np || x.query_offset != nq)
            return fail(RTD_ERR_INVALID_ARGUMENT, "clouds must be packed in order");
        if (x.k < 1) return fail(RTD_ERR_INVALID_ARGUMENT, "k must be >= 1");
        cd[c] = CloudDesc{(uint32_t)np, x.n_points, (uint32_t)nq, x.n_queries, x.k, 0u, 0u, {}, 0.f,
                          x.out_offset};
        const uint32_t cls = k_class(x.k, x.n_points, !s.partial_results, s.lanes_per_query == 32);
        const uint32_t kk = x.k < x.n_points ? x.k : (x.n_points ? x.n_points : 1u);
        if (cls == CLS_WIDE && x.n_queries && kk > wide_kk) wide_kk = kk;
        if (cls == CLS_COLLECT && x.n_queries) {
            if (kk > collect_kk) collect_kk = kk;
            if (x.n_points > collect_n) collect_n = x.n_points;
        }
        for (uint32_t s0 = 0; s0 < x.n_queries; s0 += 32)
            cls_items[cls].push_back(WorkItem{c, (uint32_t)nq + s0,
                                              x.n_queries - s0 < 32u ? x.n_queries - s0 : 32u, cls});
        np += x.n_points;
        nq += x.n_queries;
    }
    if (np >= (1ull << 30) - 1 || nq >= (1ull << 30)) return fail(RTD_ERR_INVALID_ARGUMENT, "batch too large");
    // the collected lists' queue, longest lists first, then the others',
    // heaviest class first
    std::stable_sort(cls_items[CLS_COLLECT].begin(), cls_items[CLS_COLLECT].end(),
                     [&](const WorkItem &x, const WorkItem &y) { return clouds[x.cloud].k > clouds[y.cloud].k; });
    std::vector<WorkItem> items;
    for (int c = N_CLASSES - 1; c >= 0; --c) items.insert(items.end(), cls_items[c].begin(), cls_items[c].end());
    b->drop_graph();
    b->clouds.assign(clouds, clouds + n_clouds);
    b->n_clouds = n_clouds;
    b->n_points = np;
    b->n_queries = nq;
    b->n_collect = (uint32_t)cls_items[CLS_COLLECT].size();
    b->n_items = (uint32_t)items.size() - b->n_collect;
    b->collect_kk = collect_kk;
    b->collect_n = collect_n;
    b->wide_kk = wide_kk;
    b->sched = s;
    int cb = 0;
    while (cb < 32 && (1ull << cb) < n_clouds) ++cb;
    b->cbits = cb;
    // bits per axis: the schedule's key width (auto 48 = 16 per axis), within what the
    // 63-bit key leaves beside the cloud id
    const int want = s.morton_bits ? (int)s.morton_bits / 3 : 16;
    b->bpa = (63 - cb) / 3 < want ? (63 - cb) / 3 : want;
    if (b->bpa < 8) return fail(RTD_ERR_INVALID_ARGUMENT, "too many clouds");
    rtd_index &f = b->forest;
    f.n = np;
    f.leaf_size = s.leaf_size;
    f.morton_bits = 63;
    RTD_CUDA(cudaGetDevice(&f.device));
    RTD_TRY(f.hdr.reserve(sizeof(IndexHeader)));
    RTD_TRY(f.pts.reserve((np ? np : 1) * sizeof(float4)));
    RTD_TRY(f.nodes.reserve((np > 1 ? np - 1 : 1) * sizeof(BvhNode)));
    RTD_TRY(f.keys.reserve(np * 8 + 8));
    RTD_TRY(f.keys_alt.reserve(np * 8 + 8));
    RTD_TRY(f.vals.reserve(np * 4 + 4));
    RTD_TRY(f.vals_alt.reserve(np * 4 + 4));
    RTD_TRY(b->cd.reserve(n_clouds * sizeof(CloudDesc) + 8));
    RTD_TRY(b->items.reserve(items.size() * sizeof(WorkItem) + 8));
    RTD_TRY(b->pcloud.reserve(np * 4 + 4));
    RTD_TRY(b->qcloud.reserve(nq * 4 + 4));
    RTD_TRY(b->qkeys.reserve(nq * 8 + 8));
    RTD_TRY(b->qkeys_alt.reserve(nq * 8 + 8));
    RTD_TRY(b->qvals.reserve(nq * 4 + 4));
    RTD_TRY(b->qvals_alt.reserve(nq * 4 + 4));
    RTD_TRY(b->counter.reserve(2 * sizeof(uint32_t)));
    if (n_clouds)
        RTD_CUDA(cudaMemcpy(b->cd.ptr, cd.data(), n_clouds * sizeof(CloudDesc), cudaMemcpyHostToDevice));
    if (!items.empty())
        RTD_CUDA(cudaMemcpy(b->items.ptr, items.data(), items.size() * sizeof(WorkItem), cudaMemcpyHostToDevice));
    int sms = 148;
    RTD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, f.device));
    // persistent grid: every resident warp, no more blocks than items need,
    // and (with k > 256 clouds) at most 1 GiB of list slabs
    int per_sm = 1;
    RTD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_knn_kernel, SWARPS * 32, 0));
    if (per_sm < 1) per_sm = 1;
    uint64_t blocks = (uint64_t)sms * per_sm;
    const uint64_t need = ((uint64_t)b->n_items + SWARPS - 1) / SWARPS;
    if (blocks > need) blocks = need ? need : 1;
    if (wide_kk) {
        const uint64_t per_block = (uint64_t)SWARPS * wide_kk * sizeof(uint2);
        const uint64_t cap = (1ull << 30) / per_block;
        if (blocks > cap) blocks = cap ? cap : 1;
        RTD_TRY(b->wide.reserve(blocks * per_block));
    }
    b->blocks = (int)blocks;
    if (b->n_collect) {
        const size_t smem = SWARPS * collect_warp_bytes(collect_kk, collect_n);
        RTD_CUDA(cudaFuncSetAttribute(batch_collect_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(SWARPS * collect_warp_bytes(BATCH_COLLECT_MAX, 1ull << 30))));
        RTD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_collect_kernel, SWARPS * 32, smem));
        if (per_sm < 1) per_sm = 1;
        const uint64_t most = ((uint64_t)b->n_collect * (32 / COLLECT_PART) + SWARPS - 1) / SWARPS;
        blocks = (uint64_t)sms * per_sm;
        b->collect_blocks = (int)(blocks < most ? blocks : most);
    }
    return RTD_OK;
}

rtd_status rtd_knn_batched(rtd_batch *b, const float *d_points, const float *d_queries,
                           uint32_t *d_ids, float *d_d2, int use_graph, rtd_stream stream) {
    if (!b) return fail(RTD_ERR_INVALID_ARGUMENT, "batch is NULL");
    if ((b->n_points && !d_points) || (b->n_queries && (!d_queries || !d_ids)))
        return fail(RTD_ERR_INVALID_ARGUMENT, "NULL device buffer");
    cudaStream_t st = (cudaStream_t)stream;
    if (!use_graph || st == nullptr) {
        RTD_TRY(batch_pass(b, d_points, d_queries, d_ids, d_d2, st));
        return check_index_errors(&b->forest, st);
    }
    const bool same = b->exec && b->g_pts == d_points && b->g_q == d_queries && b->g_ids == d_ids &&
                      b->g_d2 == d_d2 && b->g_stream == st;
    if (!same) {
        b->drop_graph();
        // an eager pass first sizes every scratch buffer (no allocation may
        // happen while capturing)
        RTD_TRY(batch_pass(b, d_points, d_queries, d_ids, d_d2, st));
        RTD_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeRelaxed));
        rtd_status s = batch_pass(b, d_points, d_queries, d_ids, d_d2, st);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(st, &g);
        if (s != RTD_OK) {
            if (g) cudaGraphDestroy(g);
            return s;
        }
        if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
        b->graph = g;
        e = cudaGraphInstantiate(&b->exec, g, 0);
        if (e != cudaSuccess) {
            b->drop_graph();
            return cuda_fail(e, "cudaGraphInstantiate");
        }
        b->g_pts = d_points;
        b->g_q = d_queries;
        b->g_ids = d_ids;
        b->g_d2 = d_d2;
        b->g_stream = st;
        return RTD_OK;   // the captured pass ran eagerly just before
    }
    RTD_CUDA(cudaGraphLaunch(b->exec, st));
    note_launch();
    return RTD_OK;
}

rtd_status rtd_knn_batched_backward(rtd_batch *b, const float *d_points, const float *d_queries,
                                    const uint32_t *d_ids, const float *d_grad_d2,
                                    float *d_grad_q, float *d_grad_p, rtd_stream stream) {
    if (!b) return fail(RTD_ERR_INVALID_ARGUMENT, "batch is NULL");
    if (b->n_queries == 0) return RTD_OK;
    if (!d_points || !d_queries || !d_ids || !d_grad_d2)
        return fail(RTD_ERR_INVALID_ARGUMENT, "NULL device buffer");
    cudaStream_t st = (cudaStream_t)stream;
    batch_backward_kernel<<<grid_for(b->n_queries, 256, 148 * 16), 256, 0, st>>>(
        d_queries, b->n_queries, d_points, b->qcloud.as<uint32_t>(), b->cd.as<CloudDesc>(), d_ids,
        d_grad_d2, d_grad_q, d_grad_p);
    RTD_LAUNCH_CHECK();
    return RTD_OK;
}

}  // extern "C"
