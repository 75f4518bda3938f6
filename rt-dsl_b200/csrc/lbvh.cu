// lbvh.cu -- LBVH builder: scene box -> Morton codes -> LSD radix sort
// -> Karras radix tree -> leaf collapse with every child box taken from a
// pyramid of run boxes over the sorted points -> top-level staging.
// Replaces the OptiX GAS build/refit of
// gprt-optix/host/main.cpp:200-292 and the sphere-AABB kernel of
// gprt-optix/host/kernels.cu:3-16: the tree holds point boxes only and the
// search radius is applied inside the search kernels.
#include "index.cuh"
#include "scan.cuh"

namespace rtd {
namespace {

constexpr int BLOCK = 256;

// Whether a device array can be read as float4.
inline int aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0 ? 1 : 0; }

__device__ __forceinline__ void hdr_init(IndexHeader *h) {
    h->root = CHILD_NONE;
    h->root_count = 0;
    h->n_internal = 0;
    h->n_top = 0;
    for (int a = 0; a < 3; ++a) {
        h->box[a] = 0xFFFFFFFFu;   // flip(+inf) side: any atomicMin lowers it
        h->box[3 + a] = 0u;
    }
    h->err = 0;
    h->r0sq = 0.0f;
    h->total = 0;
    h->nn95_key = -1.0f;   // "no sample": the seed falls back to radius 1
    h->n_sample = 0;
}

// Also zeroes the words that the kernels of a build add into: the sort's
// count rows and the tree's counts.
__global__ void __launch_bounds__(256) hdr_init_kernel(IndexHeader *h, uint32_t *rows, uint64_t n_rows, uint32_t *counts,
                                                       uint32_t n_counts) {
    chain_wait();
    const uint64_t t = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    if (t == 0) hdr_init(h);
    for (uint64_t i = t; i < n_rows; i += (uint64_t)gridDim.x * 256) rows[i] = 0u;
    for (uint64_t i = t; i < n_counts; i += (uint64_t)gridDim.x * 256) counts[i] = 0u;
}

// Points 4g .. 4g+3 of a 16-byte aligned xyz array: three float4 loads.
__device__ __forceinline__ void load_point4(const float *__restrict__ xyz, uint64_t g,
                                            float (&x)[4], float (&y)[4], float (&z)[4]) {
    const float4 *p = reinterpret_cast<const float4 *>(xyz) + 3 * g;
    const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
    x[0] = a.x; y[0] = a.y; z[0] = a.z;
    x[1] = a.w; y[1] = b.x; z[1] = b.y;
    x[2] = b.z; y[2] = b.w; z[2] = c.x;
    x[3] = c.y; y[3] = c.z; z[3] = c.w;
}

// Scene box, NaN-ignoring (fminf/fmaxf), as order-preserving atomics.  With
// vec4 (a 16-byte aligned array) whole groups of 4 points are read as three
// float4 each; the last n % 4 points, or all of them without vec4, one
// coordinate at a time.
__global__ void __launch_bounds__(BLOCK) bbox_kernel(const float *__restrict__ xyz, uint64_t n,
                                                     IndexHeader *h, int vec4) {
    chain_wait();
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    const uint64_t t0 = (uint64_t)blockIdx.x * BLOCK + threadIdx.x, stride = (uint64_t)gridDim.x * BLOCK;
    const uint64_t groups = vec4 ? n / 4 : 0;
    for (uint64_t g = t0; g < groups; g += stride) {
        float x[4], y[4], z[4];
        load_point4(xyz, g, x, y, z);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            lo[0] = fminf(lo[0], x[u]); hi[0] = fmaxf(hi[0], x[u]);
            lo[1] = fminf(lo[1], y[u]); hi[1] = fmaxf(hi[1], y[u]);
            lo[2] = fminf(lo[2], z[u]); hi[2] = fmaxf(hi[2], z[u]);
        }
    }
    for (uint64_t i = 4 * groups + t0; i < n; i += stride) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            float v = xyz[3 * i + a];
            lo[a] = fminf(lo[a], v);
            hi[a] = fmaxf(hi[a], v);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    __shared__ float s[BLOCK / 32][6];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        for (int a = 0; a < 3; ++a) { s[warp][a] = lo[a]; s[warp][3 + a] = hi[a]; }
    __syncthreads();
    if (threadIdx.x < 3) {
        int a = threadIdx.x;
        float l = INFINITY, u = -INFINITY;
        for (int w = 0; w < BLOCK / 32; ++w) { l = fminf(l, s[w][a]); u = fmaxf(u, s[w][3 + a]); }
        atomicMin(&h->box[a], float_flip(l));
        atomicMax(&h->box[3 + a], float_flip(u));
    }
}

// Keys of the points; with vec4 (as bbox_kernel) whole groups of 4 points
// are read as three float4 each.
template <typename K>
__global__ void __launch_bounds__(BLOCK) morton_kernel(const float *__restrict__ xyz, uint64_t n,
                                                       const IndexHeader *h, float scale,
                                                       K *__restrict__ keys, int vec4) {
    chain_wait();
    const SceneNorm s = sizeof(K) == 4 ? scene_norm(h) : scene_norm_cubic(h);
    const uint64_t t0 = (uint64_t)blockIdx.x * BLOCK + threadIdx.x, stride = (uint64_t)gridDim.x * BLOCK;
    const uint64_t groups = vec4 ? n / 4 : 0;
    for (uint64_t g = t0; g < groups; g += stride) {
        float x[4], y[4], z[4];
        load_point4(xyz, g, x, y, z);
#pragma unroll
        for (int u = 0; u < 4; ++u) keys[4 * g + u] = morton_key<K>(s, scale, x[u], y[u], z[u]);
    }
    for (uint64_t i = 4 * groups + t0; i < n; i += stride)
        keys[i] = morton_key<K>(s, scale, xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]);
}

// Common-prefix length of sorted keys i and j (ki = keys[i]), ties broken
// by index (Karras 2012, "Maximizing parallelism in the construction of
// BVHs"); -1 when j is outside [0, n).
template <typename K>
__device__ __forceinline__ int delta(const K *__restrict__ keys, int64_t n, K ki, int64_t i,
                                     int64_t j) {
    if (j < 0 || j >= n) return -1;
    const K b = keys[j];
    if (ki == b) return (int)(8 * sizeof(K)) + __clz((uint32_t)(i ^ j));
    return sizeof(K) == 8 ? __clzll((unsigned long long)(ki ^ b)) : __clz((uint32_t)(ki ^ b));
}

// Direction of Karras node i and the lower bound on its common prefix (the
// prefix shared with the neighbour away from the direction).
template <typename K>
__device__ __forceinline__ void karras_dir(const K *__restrict__ keys, int64_t n, K ki, int64_t i,
                                           int &dir, int &dmin) {
    const int dp = delta(keys, n, ki, i, i + 1), dm = delta(keys, n, ki, i, i - 1);
    dir = (dp - dm) >= 0 ? 1 : -1;
    dmin = dir > 0 ? dm : dp;
}

// Karras nodes.  Only nodes with more than leaf_size points are kept (the
// rest collapse into leaves), and a node's point count exceeds leaf_size
// exactly when the key leaf_size steps away in its direction still shares
// more than the node's lower bound on the common prefix: the prefix length
// of the (key, position) pairs, which are strictly increasing, cannot grow
// with distance.  keeps_node makes that one test on keys staged in shared
// memory with a halo of leaf_size + 1 on each side (s_k[0] is the key of
// position base).
constexpr int NODE_TILE = 1024;   // sorted points (and Karras nodes) of a tile
constexpr int FLAG_HALO = 65;     // leaf_size (<= 64) + 1
// Prefixes are compared without counting zeros: of two differences from the
// node's key the one with the lower top bit shares the longer prefix.  Equal
// keys (ties by position) take the counts.
template <typename K>
__device__ __forceinline__ bool shares_more(K x, K y) { return x < y && x < (x ^ y); }

template <typename K>
__device__ __forceinline__ bool keeps_node(const K *s_k, int64_t base, int64_t n, int64_t i, uint32_t leaf_size) {
    if (i == 0) return leaf_size < n;   // the root
    const K *k = s_k + (i - base);
    const K ki = *k, xp = ki ^ k[1], xm = ki ^ k[-1];   // (i < n - 1)
    if (xp == 0 || xm == 0) {
        auto dl = [&](int64_t j) -> int { return delta(s_k - base, n, ki, i, j); };
        const int dp = dl(i + 1), dm = dl(i - 1), dir = (dp - dm) >= 0 ? 1 : -1;
        return dl(i + (int64_t)leaf_size * dir) > (dir > 0 ? dm : dp);
    }
    const bool up = !shares_more(xm, xp);
    const int64_t j = up ? i + leaf_size : i - leaf_size;
    if (j < 0 || j >= n) return false;
    return shares_more<K>(ki ^ k[up ? (int)leaf_size : -(int)leaf_size], up ? xm : xp);
}

// Whether the keys of a node's direction share more than its lower bound:
// their differences from its key then have no bit of the bound's prefix or
// the one after it.  A bound inside the ties (dmin >= the key's width) takes
// the counts.
template <typename K>
struct PrefixTest {
    K lim;
    int dmin;
    __device__ __forceinline__ explicit PrefixTest(int d)
        : lim(d < 0 ? ~K(0) : d + 1 < (int)(8 * sizeof(K)) ? ~K(0) >> (d + 1) : K(0)), dmin(d) {}
    // x: the difference of the keys at positions i and j
    __device__ __forceinline__ bool operator()(K x, uint32_t i, uint32_t j) const {
        if (dmin < (int)(8 * sizeof(K))) return x <= lim;
        return x == 0 && (int)(8 * sizeof(K)) + __clz(i ^ j) > dmin;
    }
};

// The keys at positions base .. base + COUNT - 1 that exist, all loads in
// flight together.
template <int COUNT, typename K>
__device__ __forceinline__ void stage_keys(const K *__restrict__ keys, int64_t n, int64_t base, K *s_k) {
    constexpr int U = (COUNT + BLOCK - 1) / BLOCK;
    K k[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int t = u * BLOCK + (int)threadIdx.x;
        const int64_t j = base + t;
        if (t < COUNT && j >= 0 && j < n) k[u] = keys[j];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int t = u * BLOCK + (int)threadIdx.x;
        const int64_t j = base + t;
        if (t < COUNT && j >= 0 && j < n) s_k[t] = k[u];
    }
}

// Kept nodes of every tile, added into the sums of its group (32 tiles) and
// super group (32 groups), from which tile_nodes_kernel numbers them: the
// numbers follow the Karras index.
struct TreeCounts {
    uint32_t *tiles, *groups, *supers;
    uint32_t *cross, *done;   // nodes listed for cross_nodes_kernel; its finished blocks
};
template <typename K>
__global__ void __launch_bounds__(BLOCK) karras_count_kernel(const K *__restrict__ keys, int64_t n, uint32_t leaf_size,
                                                             const TreeCounts tc) {
    chain_wait();
    __shared__ K s_k[NODE_TILE + 2 * FLAG_HALO];
    __shared__ uint32_t s_cnt[BLOCK / 32];
    const uint32_t tile = blockIdx.x;
    const int64_t b0 = (int64_t)tile * NODE_TILE, base = b0 - FLAG_HALO;
    stage_keys<NODE_TILE + 2 * FLAG_HALO>(keys, n, base, s_k);
    __syncthreads();
    uint32_t c = 0;
#pragma unroll
    for (int t = 0; t < NODE_TILE; t += BLOCK) {
        const int64_t i = b0 + t + (int)threadIdx.x;
        c += __popc(__ballot_sync(0xffffffffu, i < n - 1 && keeps_node<K>(s_k, base, n, i, leaf_size)));
    }
    if ((threadIdx.x & 31) == 0) s_cnt[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        c = 0;
        for (int w = 0; w < BLOCK / 32; ++w) c += s_cnt[w];
        tc.tiles[tile] = c;
        if (c) {
            atomicAdd(&tc.groups[tile / GROUP_TILES], c);
            atomicAdd(&tc.supers[tile / SUPER_TILES], c);
        }
    }
}

// Point range [first, last] and split of the kept Karras node at position i,
// whose range holds at most `room` points after i in direction dir: the
// children hold [first, split] and [split + 1, last].  k: the keys, at
// positions base and up.  REACH: a power of two above the longest range.
template <int REACH, typename K>
__device__ __forceinline__ void karras_range(const K *k, uint32_t base, int i, int dir, int dmin, int room,
                                             uint32_t &first, uint32_t &last, uint32_t &split) {
    const K ki = k[i];
    auto more = [&](int j, const PrefixTest<K> &t) { return t(ki ^ k[j], base + i, base + j); };
    const PrefixTest<K> in(dmin);
    int l = 0;
#pragma unroll 1
    for (int t = REACH / 2; t >= 1; t >>= 1)
        if (l + t <= room && more(i + (l + t) * dir, in)) l += t;
    const K x = ki ^ k[i + l * dir];
    const PrefixTest<K> left(x == 0 ? (int)(8 * sizeof(K)) + __clz((base + i) ^ (base + i + l * dir))
                                    : sizeof(K) == 8 ? __clzll((unsigned long long)x) : __clz((uint32_t)x));
    int s = 0, t = l;
#pragma unroll 1
    do {
        t = (t + 1) >> 1;
        if (s + t < l && more(i + (s + t) * dir, left)) s += t;
    } while (t > 1);
    split = (uint32_t)(i + s * dir + (dir < 0 ? -1 : 0));
    first = (uint32_t)(dir > 0 ? i : i - l);
    last = (uint32_t)(dir > 0 ? i + l : i);
}

// ---------------------------------------------------- box pyramid
// Boxes of aligned runs of the sorted points: level j entry e covers points
// [e * 8^j, (e+1) * 8^j) as (lo.xyz, -) (hi.xyz, -).  A run holding a
// point with a NaN coordinate gets an unbounded box: such a point is never
// a neighbour, but no finite box holds it, so no search may treat a
// subtree containing it as lying wholly inside a ball.  Base 8 keeps the
// walk of a range short: at most 7 entries per end and level.
constexpr int PYR_SH = 3;                  // log2 of the base
constexpr uint32_t PYR_B = 1u << PYR_SH;   // 8 entries of a level per entry of the next
constexpr int PYR_MAX = 10;                // levels 1..10 cover 8^10 = 2^30 points
// Levels 1..nlev lie back to back in pyr (2 float4 per entry), level j
// holding ceil(n / 8^j) entries; nlev is the first level of <= 8 entries.
struct Pyramid {
    const float4 *pts;
    const float4 *pyr;
    uint32_t n;
    int nlev;
};

struct Box {
    float lo[3], hi[3];
};

__device__ __forceinline__ void box_empty(Box &b) {
    for (int a = 0; a < 3; ++a) { b.lo[a] = INFINITY; b.hi[a] = -INFINITY; }
}
__device__ __forceinline__ void box_add_point(Box &b, bool &nan, const float4 p) {
    b.lo[0] = fminf(b.lo[0], p.x); b.hi[0] = fmaxf(b.hi[0], p.x);
    b.lo[1] = fminf(b.lo[1], p.y); b.hi[1] = fmaxf(b.hi[1], p.y);
    b.lo[2] = fminf(b.lo[2], p.z); b.hi[2] = fmaxf(b.hi[2], p.z);
    nan |= isnan(p.x) || isnan(p.y) || isnan(p.z);
}
__device__ __forceinline__ void box_add(Box &b, const float4 lo, const float4 hi) {
    b.lo[0] = fminf(b.lo[0], lo.x); b.hi[0] = fmaxf(b.hi[0], hi.x);
    b.lo[1] = fminf(b.lo[1], lo.y); b.hi[1] = fmaxf(b.hi[1], hi.y);
    b.lo[2] = fminf(b.lo[2], lo.z); b.hi[2] = fmaxf(b.hi[2], hi.z);
}
__device__ __forceinline__ void box_unbounded(Box &b) {
    for (int a = 0; a < 3; ++a) { b.lo[a] = -INFINITY; b.hi[a] = INFINITY; }
}

// One step of a butterfly min / max over the lanes at xor distance o.
__device__ __forceinline__ void box_xor(Box &b, int o) {
    for (int a = 0; a < 3; ++a) {
        b.lo[a] = fminf(b.lo[a], __shfl_xor_sync(0xffffffffu, b.lo[a], o));
        b.hi[a] = fmaxf(b.hi[a], __shfl_xor_sync(0xffffffffu, b.hi[a], o));
    }
}

__device__ __forceinline__ void box_store(float4 *out, uint64_t e, const Box &b) {
    out[2 * e] = make_float4(b.lo[0], b.lo[1], b.lo[2], 0.f);
    out[2 * e + 1] = make_float4(b.hi[0], b.hi[1], b.hi[2], 0.f);
}

// Three levels of the pyramid from the `count` boxes of the level below o1
// (levels 1 to 3 come from tile_nodes_kernel): a 512-thread block per 512
// inputs, one input a thread.  Lanes fold 8 inputs into an o1 entry and a
// warp's 32 into half an o2 entry; warp 0 folds the block's 16 warp boxes
// into its 8 o2 entries and its o3 entry.  Inputs past count hold the empty
// box; a null output is a level above the top and is not written.
__global__ void __launch_bounds__(512) pyramid_fold_kernel(const float4 *__restrict__ in,
                                                           uint64_t count, float4 *o1, float4 *o2,
                                                           float4 *o3) {
    chain_wait();
    __shared__ float4 s_lo[16], s_hi[16];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t i = (uint64_t)blockIdx.x * 512 + threadIdx.x;
    Box b;
    box_empty(b);
    if (i < count) box_add(b, in[2 * i], in[2 * i + 1]);
    box_xor(b, 1);
    box_xor(b, 2);
    box_xor(b, 4);
    if ((lane & 7) == 0 && (i >> 3) * 8 < count) box_store(o1, i >> 3, b);
    box_xor(b, 8);
    box_xor(b, 16);
    if (lane == 0) {
        s_lo[warp] = make_float4(b.lo[0], b.lo[1], b.lo[2], 0.f);
        s_hi[warp] = make_float4(b.hi[0], b.hi[1], b.hi[2], 0.f);
    }
    __syncthreads();
    if (warp == 0 && o2) {
        Box c;
        box_empty(c);
        if (lane < 16) box_add(c, s_lo[lane], s_hi[lane]);
        box_xor(c, 1);   // lanes 2m, 2m + 1: the 64 inputs of o2 entry m
        const uint64_t e2 = (uint64_t)blockIdx.x * 8 + (lane >> 1);
        if (lane < 16 && (lane & 1) == 0 && e2 * 64 < count) box_store(o2, e2, c);
        box_xor(c, 2);
        box_xor(c, 4);
        box_xor(c, 8);   // lane 0: the block's 512 inputs
        if (lane == 0 && o3) box_store(o3, blockIdx.x, c);
    }
}

// Adds entries [a, b) of one level (the points when PTS) to a box, loading
// BATCH entries at a time so that their loads are in flight together.  The
// last batch repeats entry b - 1 in place of entries past b: a min / max
// does not change when an entry is added twice.
template <bool PTS>
__device__ __forceinline__ void add_run(Box &bx, bool &nan, const float4 *base,
                                        uint32_t a, uint32_t b) {
    constexpr int BATCH = PTS ? 4 : 2;
#pragma unroll 1
    for (uint32_t t = a; t < b; t += BATCH) {
        float4 lo[BATCH], hi[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const uint32_t e = t + u < b ? t + u : b - 1;
            if (PTS) {
                lo[u] = base[e];
            } else {
                lo[u] = base[2 * (uint64_t)e];
                hi[u] = base[2 * (uint64_t)e + 1];
            }
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            if (PTS) box_add_point(bx, nan, lo[u]);
            else box_add(bx, lo[u], hi[u]);
        }
    }
}

// Box of the sorted points [first, first + count): partial runs at both
// ends point by point, then whole runs from the pyramid level by level (at
// most 7 entries per end and level); the highest level is taken whole.
// The level offsets follow from n as the walk goes up, so the pyramid is
// passed as scalars (a struct taken by reference would be copied to local
// memory).
__device__ __noinline__ Box range_box(const float4 *pts, const float4 *pyr, uint32_t n, int nlev,
                                      uint32_t first, uint32_t count) {
    Box b;
    box_empty(b);
    bool nan = false;
    uint32_t l = first, r = first + count;   // n < 2^30: no overflow
    uint32_t size = n;                       // entries of the current level
    const float4 *lvl = pyr;                 // level j >= 1 (2 float4 per entry)
#pragma unroll 1
    for (int j = 0; j <= PYR_MAX; ++j) {
        if (l >= r) break;
        if (j == nlev) {
            if (j == 0) add_run<true>(b, nan, pts, l, r);
            else add_run<false>(b, nan, lvl, l, r);
            break;
        }
        uint32_t head = (l + PYR_B - 1) & ~(PYR_B - 1);
        if (head > r) head = r;
        uint32_t tail = r & ~(PYR_B - 1);
        if (tail < head) tail = head;
        if (j == 0) {
            add_run<true>(b, nan, pts, l, head);
            add_run<true>(b, nan, pts, tail, r);
        } else {
            add_run<false>(b, nan, lvl, l, head);
            add_run<false>(b, nan, lvl, tail, r);
            lvl += 2 * (uint64_t)size;
        }
        l = head >> PYR_SH;
        r = tail >> PYR_SH;
        size = (size + PYR_B - 1) >> PYR_SH;
    }
    if (nan) box_unbounded(b);
    return b;
}

// The node of the points [f0, last] with children [f0, sp] and [sp + 1, last]:
// Karras nodes sp and sp + 1 when they keep more than leaf_size points, else
// leaves.  The positions count from base; number(i) is the index of kept
// Karras node i.
template <typename Number>
__device__ __forceinline__ BvhNode pack_node(const Number &number, uint32_t leaf_size, uint32_t f0, uint32_t last,
                                             uint32_t sp, uint32_t base, const Box &b0, const Box &b1) {
    const uint32_t c0 = sp - f0 + 1, c1 = last - sp;
    BvhNode nd;
    // layout: [lo.x0 lo.y0 lo.z0 hi.x0] [hi.y0 hi.z0 lo.x1 lo.y1] [lo.z1 hi.x1 hi.y1 hi.z1]
    nd.a = make_float4(b0.lo[0], b0.lo[1], b0.lo[2], b0.hi[0]);
    nd.b = make_float4(b0.hi[1], b0.hi[2], b1.lo[0], b1.lo[1]);
    nd.c = make_float4(b1.lo[2], b1.hi[0], b1.hi[1], b1.hi[2]);
    nd.d = make_uint4(c0 > leaf_size ? number(base + sp) : (CHILD_LEAF | (base + f0)),
                      c1 > leaf_size ? number(base + sp + 1) : (CHILD_LEAF | (base + sp + 1)), c0, c1);
    return nd;
}
template <typename Number>
__device__ __forceinline__ BvhNode make_node(const Pyramid &P, const Number &number, uint32_t leaf_size, uint32_t f0,
                                             uint32_t last, uint32_t sp, uint32_t base) {
    const Box b0 = range_box(P.pts, P.pyr, P.n, P.nlev, f0, sp - f0 + 1);
    const Box b1 = range_box(P.pts, P.pyr, P.n, P.nlev, sp + 1, last - sp);
    return pack_node(number, leaf_size, f0, last, sp, base, b0, b1);
}

// Compact nodes: children become leaves when their subtree has <= leaf_size
// points.  Every child carries the number of points below it (a subtree's
// points are contiguous in sorted order, starting at the parent's first point
// for the left child and after the left child's points for the right one),
// and its box: the box of its contiguous points, from the pyramid.  Every
// node is computed independently, so no bottom-up pass over the tree follows.
// With kfirst non-null the range is also stored by Karras index.
//
// tile_nodes_kernel: a block takes NODE_TILE sorted points.  It stages their
// keys and points in shared memory, folds levels 1 to 3 of the pyramid there
// (and writes them out), numbers its kept nodes, and makes those whose points
// all lie in the tile, a thread a node: all but about one in ten.  The
// searches for a node's range and split and the walk of its boxes are chains
// of dependent reads, which is why they run on shared memory.  A node's prefix
// with the keys of its direction cannot grow with distance, so its range ends
// inside the tile exactly when the first key past the tile no longer exceeds
// its lower bound; the others are listed in `cross` for cross_nodes_kernel.
// Bound by the issue slots of the searches and box walks.  With flags, their
// scan, a list of the kept nodes and global searches a thread a node, the tree
// of 100 K points took 50 us (51 dependent reads at the root), now 37; that of
// 10 M 575 us besides the pyramid's 79, now 495 with it (counts 50, tiles 347,
// crossing nodes 95).
constexpr int NODE_DEPTH = 96;   // prefix lengths of (key, position) pairs: nodes that share a tile boundary are nested
template <typename K>
__global__ void __launch_bounds__(BLOCK, 6) tile_nodes_kernel(
    const K *__restrict__ keys, uint64_t n, IndexHeader *h, const TreeCounts tc, uint32_t *bits, uint32_t *before,
    uint32_t leaf_size, const float4 *__restrict__ pts, float4 *lv1, float4 *lv2, float4 *lv3, BvhNode *nodes,
    uint32_t *kfirst, uint32_t *klast, uint32_t *cross, uint32_t cross_cap) {
    chain_wait();
    __shared__ K s_k[NODE_TILE + 2 * FLAG_HALO];
    __shared__ float4 s_p[NODE_TILE];
    __shared__ float4 s_pyr[2 * (NODE_TILE / 8 + NODE_TILE / 64 + NODE_TILE / 512)];
    __shared__ uint32_t s_bits[NODE_TILE / 32], s_before[NODE_TILE / 32], s_kept, s_prefix;
    __shared__ uint16_t s_list[NODE_TILE];
    static_assert(NODE_TILE == 32 * 32, "a warp numbers the words of a tile");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t tile = blockIdx.x;
    const int64_t b0 = (int64_t)tile * NODE_TILE, base_k = b0 - FLAG_HALO;
    const uint32_t m = (uint32_t)(n - b0 < NODE_TILE ? n - b0 : NODE_TILE);
    const uint32_t n1 = (m + 7) / 8, n2 = (n1 + 7) / 8, n3 = (n2 + 7) / 8;
    float4 pt[NODE_TILE / BLOCK];   // (in flight with the keys)
#pragma unroll
    for (int u = 0; u < NODE_TILE / BLOCK; ++u) {
        const uint32_t t = u * BLOCK + threadIdx.x;
        if (t < m) pt[u] = pts[b0 + t];
    }
    stage_keys<NODE_TILE + 2 * FLAG_HALO>(keys, (int64_t)n, base_k, s_k);
    // level 1: the 8 lanes of an entry
#pragma unroll
    for (int u = 0; u < NODE_TILE / BLOCK; ++u) {
        const uint32_t t = u * BLOCK + threadIdx.x;
        Box b;
        box_empty(b);
        if (t < m) {
            const float4 p = pt[u];
            s_p[t] = p;
            bool nan = false;
            box_add_point(b, nan, p);
            if (nan) box_unbounded(b);
        }
        box_xor(b, 1);
        box_xor(b, 2);
        box_xor(b, 4);
        if ((t & 7) == 0 && t < m) {
            box_store(s_pyr, t / 8, b);
            if (lv1) box_store(lv1, b0 / 8 + t / 8, b);
        }
    }
    __syncthreads();
    // which nodes are kept
#pragma unroll
    for (int t = 0; t < NODE_TILE; t += BLOCK) {
        const int li = t + (int)threadIdx.x;
        const uint32_t w = __ballot_sync(
            0xffffffffu, b0 + li < (int64_t)n - 1 && keeps_node<K>(s_k, base_k, (int64_t)n, b0 + li, leaf_size));
        if (lane == 0) s_bits[li >> 5] = w;
    }
    // levels 2 and 3
    for (int lev = 2; lev <= 3; ++lev) {
        const float4 *in = lev == 2 ? s_pyr : s_pyr + 2 * n1;
        float4 *out = lev == 2 ? s_pyr + 2 * n1 : s_pyr + 2 * (n1 + n2), *g = lev == 2 ? lv2 : lv3;
        const uint32_t cnt_in = lev == 2 ? n1 : n2, cnt = lev == 2 ? n2 : n3;
        for (uint32_t e = threadIdx.x; e < cnt; e += BLOCK) {
            Box b;
            box_empty(b);
            for (uint32_t u = 8 * e; u < 8 * e + 8 && u < cnt_in; ++u) box_add(b, in[2 * u], in[2 * u + 1]);
            box_store(out, e, b);
            if (g) box_store(g, (uint64_t)(lev == 2 ? b0 / 64 : b0 / 512) + e, b);
        }
        __syncthreads();
    }
    Pyramid P;
    P.pts = s_p;
    P.pyr = s_pyr;
    P.n = m;
    P.nlev = 3;
    // their numbers: those of the earlier tiles, then a scan over the words
    if (warp == 0) {
        const uint32_t c = __popc(s_bits[lane]);
        uint32_t x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        s_before[lane] = x - c;
        if (lane == 31) s_kept = x;
    } else if (warp == 1) {
        const uint32_t g = tile / GROUP_TILES, sg = tile / SUPER_TILES;
        uint32_t v = 0;
        if ((uint32_t)lane < tile % GROUP_TILES) v += tc.tiles[g * GROUP_TILES + lane];
        if ((uint32_t)lane < g % 32) v += tc.groups[sg * 32 + lane];
        for (uint32_t j = lane; j < sg; j += 32) v += tc.supers[j];
        v = __reduce_add_sync(0xffffffffu, v);
        if (lane == 0) s_prefix = v;
    }
    __syncthreads();
    const uint32_t prefix = s_prefix, kept = s_kept;
    if (warp == 0) {
        const uint64_t w = (uint64_t)b0 / 32 + lane;
        if (w * 32 < n) {
            bits[w] = s_bits[lane];
            before[w] = prefix + s_before[lane];
        }
        if (lane == 0 && (uint64_t)b0 + NODE_TILE >= n) h->n_internal = prefix + kept;
    }
#pragma unroll
    for (int t = 0; t < NODE_TILE; t += BLOCK) {
        const uint32_t li = t + threadIdx.x, w = s_bits[li >> 5];
        if (w >> lane & 1u) s_list[s_before[li >> 5] + __popc(w & ((1u << lane) - 1u))] = (uint16_t)li;
    }
    __syncthreads();
    const uint32_t base = (uint32_t)b0;
    auto number = [&](uint32_t i) {   // (a node of the tile)
        const uint32_t w = (i - base) >> 5;
        return prefix + s_before[w] + __popc(s_bits[w] & ((1u << (i & 31)) - 1u));
    };
    for (uint32_t c = threadIdx.x; c < kept; c += BLOCK) {
        const int li = s_list[c];
        const uint32_t i = base + li;
        const K ki = s_k[li + FLAG_HALO];
        auto dl = [&](int lj) -> int {   // lj in [-1, NODE_TILE]
            const int64_t j = b0 + lj;
            if (j < 0 || j >= (int64_t)n) return -1;
            const K b = s_k[lj + FLAG_HALO];
            if (ki == b) return (int)(8 * sizeof(K)) + __clz(i ^ (uint32_t)j);
            return sizeof(K) == 8 ? __clzll((unsigned long long)(ki ^ b)) : __clz((uint32_t)(ki ^ b));
        };
        const int dp = dl(li + 1), dm = dl(li - 1), dir = (dp - dm) >= 0 ? 1 : -1, dmin = dir > 0 ? dm : dp;
        if (dl(dir > 0 ? NODE_TILE : -1) > dmin) {
            const uint32_t at = atomicAdd(tc.cross, 1u);
            if (at < cross_cap) cross[at] = i;
            else atomicOr(&h->err, DEVERR_OVERFLOW);
            continue;
        }
        uint32_t f0, last, sp;
        karras_range<NODE_TILE>(s_k + FLAG_HALO, base, li, dir, dmin,
                                dir > 0 ? (int)m - 1 - li : li, f0, last, sp);
        if (kfirst) {
            kfirst[i] = base + f0;
            klast[i] = base + last;
        }
        nodes[prefix + c] = make_node(P, number, leaf_size, f0, last, sp, base);
    }
}

// Root word and the breadth-first top levels, copied into `top`.  One warp:
// each level's nodes are loaded in parallel (level TOP_LEVELS-1 has at most
// 32 nodes) and their internal children are placed by a warp prefix sum.
// s_q: TOP_MAX words of shared memory.
__device__ __forceinline__ void stage_top(IndexHeader *h, const BvhNode *nodes, BvhNode *top, uint64_t n,
                                          uint32_t leaf_size, uint32_t *s_q) {
    const int lane = threadIdx.x & 31;
    if (n == 0 || n == 1 || n <= leaf_size) {
        if (lane == 0) {
            h->root = n == 0 ? CHILD_NONE : (CHILD_LEAF | 0u);
            h->root_count = (uint32_t)n;
            h->n_top = 0;
        }
        return;
    }
    if (lane == 0) s_q[0] = 0;
    __syncwarp();
    int begin = 0, end = 1;
    for (int depth = 0; depth < TOP_LEVELS; ++depth) {
        const int i = begin + lane;
        const bool has = i < end;
        BvhNode nd;
        if (has) nd = nodes[s_q[i]];
        const bool deeper = depth + 1 < TOP_LEVELS;
        const bool c0 = has && deeper && !(nd.d.x & CHILD_LEAF);
        const bool c1 = has && deeper && !(nd.d.y & CHILD_LEAF);
        const uint32_t cnt = (uint32_t)c0 + (uint32_t)c1;
        uint32_t incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        const uint32_t pos = (uint32_t)end + incl - cnt;
        if (c0) s_q[pos] = nd.d.x;
        if (c1) s_q[pos + (c0 ? 1u : 0u)] = nd.d.y;
        if (has) {
            if (c0) nd.d.x = CHILD_TOP | pos;
            if (c1) nd.d.y = CHILD_TOP | (pos + (c0 ? 1u : 0u));
            top[i] = nd;
        }
        __syncwarp();
        begin = end;
        end += (int)total;
        if (total == 0) break;
    }
    if (lane == 0) {
        h->root = CHILD_TOP | 0u;
        h->n_top = (uint32_t)end;
    }
}

// The nodes whose points lie in more than one tile, a warp a node: the range
// and the split are found 32 probes at a time (an end among n keys takes
// log32 n dependent reads), and the lanes of a half warp read the entries of
// one child's box at each level of the pyramid together.  The last block
// stages the top levels (with top non-null).
template <typename K>
__global__ void __launch_bounds__(BLOCK) cross_nodes_kernel(
    const K *__restrict__ keys, uint64_t n, IndexHeader *h, const TreeCounts tc, const KeptNodes kept,
    uint32_t leaf_size, const Pyramid P, BvhNode *nodes, uint32_t *kfirst, uint32_t *klast,
    const uint32_t *__restrict__ cross, uint32_t cross_cap, BvhNode *top) {
    chain_wait();
    const uint32_t count = *tc.cross < cross_cap ? *tc.cross : cross_cap;
    const int lane = threadIdx.x & 31;
    for (uint32_t w = (blockIdx.x * BLOCK + threadIdx.x) >> 5; w < count; w += (gridDim.x * BLOCK) >> 5) {
        const int64_t i = cross[w];
        const K ki = keys[i];
        int dir, dmin;
        karras_dir(keys, (int64_t)n, ki, i, dir, dmin);
        // 2^up <= length < 2^(up + 1)
        const int up =
            __popc(__ballot_sync(0xffffffffu, lane < 31 && delta(keys, (int64_t)n, ki, i, i + ((int64_t)1 << lane) * dir) > dmin)) - 1;
        // largest x of [lo, lo + width) whose key still shares more than d
        auto furthest = [&](int64_t lo, int64_t width, int d) {
            while (width > 1) {
                const int64_t step = width > 32 ? width >> 5 : 1, x = lo + lane * step;
                const bool ok = lane == 0 || (lane * step < width && delta(keys, (int64_t)n, ki, i, i + x * dir) > d);
                lo += (__popc(__ballot_sync(0xffffffffu, ok)) - 1) * step;
                width = step;
            }
            return lo;
        };
        const int64_t l = furthest((int64_t)1 << up, (int64_t)1 << up, dmin);
        const int64_t s = furthest(0, (int64_t)2 << up, delta(keys, (int64_t)n, ki, i, i + l * dir));
        const uint32_t f0 = (uint32_t)(dir > 0 ? i : i - l), last = (uint32_t)(dir > 0 ? i + l : i);
        const uint32_t sp = (uint32_t)(i + s * dir + (dir < 0 ? -1 : 0));
        // numbers of the node and its children (read beside the boxes)
        const uint32_t num = lane < 3 ? kept.number(lane == 0 ? (uint32_t)i : sp + lane - 1) : 0u;
        // boxes: lanes 0-15 the left child, 16-31 the right one; of 16 lanes
        // 8 take the partial run at the start of a level, 8 that at its end
        Box b;
        box_empty(b);
        const uint32_t e = lane & 7;
        const bool tail_lane = lane & 8;
        uint32_t a = lane < 16 ? f0 : sp + 1, r = lane < 16 ? sp + 1 : last + 1, size = P.n;
        const float4 *lvl = P.pyr;
#pragma unroll 1
        for (int j = 0; j <= P.nlev && a < r; ++j) {
            uint32_t head = (a + PYR_B - 1) & ~(PYR_B - 1);
            if (head > r) head = r;
            uint32_t tail = r & ~(PYR_B - 1);
            if (tail < head) tail = head;
            if (j == P.nlev) head = tail = r;   // (at most 8 entries: whole)
            const uint32_t x = tail_lane ? tail + e : a + e;
            if (x < (tail_lane ? r : head)) {
                if (j == 0) {
                    bool nan = false;
                    box_add_point(b, nan, P.pts[x]);
                    if (nan) box_unbounded(b);
                } else {
                    box_add(b, lvl[2 * (uint64_t)x], lvl[2 * (uint64_t)x + 1]);
                }
            }
            if (j) lvl += 2 * (uint64_t)size;
            size = (size + PYR_B - 1) >> PYR_SH;
            a = head >> PYR_SH;
            r = tail >> PYR_SH;
        }
        __syncwarp();
        for (int o = 1; o < 16; o <<= 1) box_xor(b, o);
        Box b1;
        for (int x = 0; x < 3; ++x) {
            b1.lo[x] = __shfl_sync(0xffffffffu, b.lo[x], 16);
            b1.hi[x] = __shfl_sync(0xffffffffu, b.hi[x], 16);
        }
        const uint32_t left = __shfl_sync(0xffffffffu, num, 1), right = __shfl_sync(0xffffffffu, num, 2);
        if (lane == 0) {
            nodes[num] = pack_node([&](uint32_t j) { return j == sp ? left : right; }, leaf_size, f0, last, sp, 0u, b,
                                   b1);
            if (kfirst) {
                kfirst[i] = f0;
                klast[i] = last;
            }
        }
    }
    if (!top) return;
    __shared__ bool s_last;
    __shared__ uint32_t s_q[TOP_MAX];
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();   // (cumulative over the block's stores, ordered by the barrier)
        s_last = atomicAdd(tc.done, 1u) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (s_last && threadIdx.x < 32) stage_top(h, nodes, top, n, leaf_size, s_q);
}

// ------------------------------------------------ radius-seed sample data
// Two stride samples of the points in input order, kept with the index:
// <= 1000 points (sample[0..n_sample)) for the k_nn! sampled-percentile seed
// (gprt-macros/src/lib.rs:433-434), and S = min(n, 4096) points, index
// b*n/S (sample[SEED_PCT_POINTS + b]), for the sampled 1-NN seed, which is
// computed from them on the first search that needs it (ensure_nn_seed).
__device__ __forceinline__ void seed_sample(const float *__restrict__ xyz, uint64_t n, float4 *sample, IndexHeader *h,
                                            uint32_t t0, uint32_t stride) {
    uint64_t pstep = n / SEED_PCT_POINTS > 1 ? n / SEED_PCT_POINTS : 1;
    uint64_t cnt = (n + pstep - 1) / pstep;
    if (cnt > SEED_PCT_POINTS) cnt = SEED_PCT_POINTS;
    for (uint64_t t = t0; t < cnt; t += stride) {
        uint64_t i = t * pstep;
        sample[t] = make_float4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], 0.0f);
    }
    const uint32_t S = n < SEED_NN_SAMPLE ? (uint32_t)n : (uint32_t)SEED_NN_SAMPLE;
    for (uint32_t b = t0; b < S; b += stride) {
        const uint64_t i = (uint64_t)b * n / S;
        sample[SEED_PCT_POINTS + b] = make_float4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], 0.0f);
    }
    if (t0 == 0) h->n_sample = (uint32_t)cnt;
}

__global__ void seed_sample_kernel(const float *__restrict__ xyz, uint64_t n, float4 *sample, IndexHeader *h) {
    seed_sample(xyz, n, sample, h, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// Squared 1-NN distance of each of the S sample points p[a] among the other
// sample points.  Grid (a-tiles x b-chunks); each thread folds its chunk's
// minimum into out[a] (order-preserving u32, pre-set to 0xFFFFFFFF).  The
// minimum does not depend on the order.
constexpr int SEED_CHUNK = 256;
__global__ void __launch_bounds__(128) seed_nn_kernel(const float4 *__restrict__ p, uint32_t S,
                                                      uint32_t *__restrict__ out) {
    __shared__ float3 s_p[SEED_CHUNK];
    const uint32_t a = blockIdx.x * 128 + threadIdx.x;
    const uint32_t b0 = blockIdx.y * SEED_CHUNK;
    for (uint32_t t = threadIdx.x; t < SEED_CHUNK; t += 128) {
        uint32_t b = b0 + t;
        if (b < S) {
            const float4 v = p[b];
            s_p[t] = make_float3(v.x, v.y, v.z);
        }
    }
    __syncthreads();
    if (a >= S) return;
    const float4 va = p[a];
    const float ax = va.x, ay = va.y, az = va.z;
    const uint32_t lim = S - b0 < (uint32_t)SEED_CHUNK ? S - b0 : (uint32_t)SEED_CHUNK;
    float best = INFINITY;
    for (uint32_t j = 0; j < lim; ++j) {
        if (b0 + j == a) continue;
        float key = exact_key(ax, ay, az, s_p[j].x, s_p[j].y, s_p[j].z);
        if (key < best) best = key;
    }
    if (best < INFINITY) atomicMin(&out[a], float_flip(best));
}

// rank-th smallest of S <= 4096 order-preserving u32 values: an 8-bit
// radix select in one 1024-thread block (4 histogram passes).
__global__ void __launch_bounds__(1024) seed_nn_select_kernel(const uint32_t *__restrict__ keys,
                                                              uint32_t S, IndexHeader *h) {
    __shared__ uint32_t s_hist[256];
    __shared__ uint32_t s_sel[2];   // prefix chosen so far, remaining rank
    uint32_t v[4];
    for (int j = 0; j < 4; ++j) {
        uint32_t i = threadIdx.x + 1024u * j;
        v[j] = i < S ? keys[i] : 0xFFFFFFFFu;
    }
    uint32_t rank = (uint32_t)(0.95f * (float)S);
    if (rank > S - 1) rank = S - 1;
    uint32_t prefix = 0;
    for (int pass = 3; pass >= 0; --pass) {
        const int shift = 8 * pass;
        const uint32_t hi_mask = pass == 3 ? 0u : (0xFFFFFFFFu << (shift + 8));
        if (threadIdx.x < 256) s_hist[threadIdx.x] = 0;
        __syncthreads();
        for (int j = 0; j < 4; ++j) {
            uint32_t i = threadIdx.x + 1024u * j;
            if (i < S && (v[j] & hi_mask) == prefix) atomicAdd(&s_hist[(v[j] >> shift) & 255u], 1u);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t acc = 0, d = 0;
            for (; d < 255; ++d) {
                if (acc + s_hist[d] > rank) break;
                acc += s_hist[d];
            }
            s_sel[0] = prefix | (d << shift);
            s_sel[1] = rank - acc;
        }
        __syncthreads();
        prefix = s_sel[0];
        rank = s_sel[1];
        __syncthreads();
    }
    if (threadIdx.x == 0) h->nn95_key = float_unflip(prefix);
}

rtd_status build_seed(rtd_index *idx, const float *d_xyz, uint64_t n, cudaStream_t st) {
    IndexHeader *h = idx->hdr.as<IndexHeader>();
    RTD_TRY(idx->sample.reserve((SEED_PCT_POINTS + SEED_NN_SAMPLE) * sizeof(float4)));
    RTD_TRY(idx->seed.reserve(SEED_NN_SAMPLE * sizeof(float)));
    seed_sample_kernel<<<(SEED_NN_SAMPLE + 255) / 256, 256, 0, st>>>(d_xyz, n,
                                                                    idx->sample.as<float4>(), h);
    RTD_LAUNCH_CHECK();
    idx->nn_seeded = false;
    return RTD_OK;
}

}  // namespace

rtd_status ensure_nn_seed(rtd_index *idx, cudaStream_t st) {
    if (idx->nn_seeded || idx->n < 2) return RTD_OK;
    IndexHeader *h = idx->hdr.as<IndexHeader>();
    const uint32_t S = idx->n < SEED_NN_SAMPLE ? (uint32_t)idx->n : (uint32_t)SEED_NN_SAMPLE;
    RTD_CUDA(cudaMemsetAsync(idx->seed.ptr, 0xFF, S * sizeof(uint32_t), st));
    dim3 grid((S + 127) / 128, (S + SEED_CHUNK - 1) / SEED_CHUNK);
    seed_nn_kernel<<<grid, 128, 0, st>>>(idx->sample.as<float4>() + SEED_PCT_POINTS, S,
                                         idx->seed.as<uint32_t>());
    RTD_LAUNCH_CHECK();
    seed_nn_select_kernel<<<1, 1024, 0, st>>>(idx->seed.as<uint32_t>(), S, h);
    RTD_LAUNCH_CHECK();
    // Inside a stream capture the kernels run at each launch of the graph,
    // not now: an eager search afterwards must still compute the seed.
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    RTD_CUDA(cudaStreamIsCapturing(st, &cs));
    if (cs == cudaStreamCaptureStatusNone) idx->nn_seeded = true;
    return RTD_OK;
}

namespace {

// The smallest clouds: the whole build in one block and one launch.  The
// chain of two dozen launches that builds larger indexes takes about 75 us
// for 2,000 points on the GPU and 100 us on the host, almost none of it work;
// this kernel 38 us.  Same index: keys sorted by (key, input position),
// the same Karras nodes, boxes and top copy.  Keys, points, pyramid and the
// kept nodes' indices stay in shared memory (40 B a point).  Bound by
// barriers and dependent shared-memory loads.
constexpr uint32_t SMALL_MAX = 4096;
constexpr int SMALL_THREADS = 1024;
struct SmallSmem {
    uint64_t *key;      // P
    float4 *pts;        // n
    float4 *pyr;        // 2 per entry
    uint32_t *idx, *cidx, *sel;   // P each
};
__host__ __device__ inline uint32_t small_pow2(uint32_t n) {
    uint32_t P = SMALL_THREADS;
    while (P < n) P <<= 1;
    return P;
}
__host__ __device__ inline uint32_t pyramid_entries(uint32_t n) {
    uint32_t total = 0;
    while (n > PYR_B) {
        n = (n + PYR_B - 1) / PYR_B;
        total += n;
    }
    return total ? total : 1;
}
__host__ __device__ inline size_t small_smem(uint32_t n) {
    const size_t P = small_pow2(n);
    return P * (sizeof(uint64_t) + sizeof(float4) + 3 * sizeof(uint32_t)) + 2 * pyramid_entries(n) * sizeof(float4);
}

// E elements a thread: element u * 1024 + thread in register u.
template <typename K, int E>
__global__ void __launch_bounds__(SMALL_THREADS) small_build_kernel(const float *__restrict__ xyz, uint32_t n,
                                                                    IndexHeader *h, float scale, uint32_t leaf_size,
                                                                    K *out_keys, float4 *out_pts, float4 *out_pyr,
                                                                    BvhNode *nodes, BvhNode *top, float4 *sample) {
    chain_wait();
    extern __shared__ float4 s_dyn[];
    __shared__ float s_box[32][6];
    __shared__ uint32_t s_cnt[33 * E], s_q[TOP_MAX];
    constexpr uint32_t P = E * SMALL_THREADS;
    SmallSmem s;
    s.pts = s_dyn;
    s.pyr = s.pts + P;
    s.key = reinterpret_cast<uint64_t *>(s.pyr + 2 * pyramid_entries(n));
    s.idx = reinterpret_cast<uint32_t *>(s.key + P);
    s.cidx = s.idx + P;
    s.sel = s.cidx + P;
    const uint32_t tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    if (tid == 0) hdr_init(h);
    // scene box, NaN-ignoring
    float x[E], y[E], z[E], lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const uint32_t i = u * SMALL_THREADS + tid;
        x[u] = y[u] = z[u] = NAN;
        if (i < n) {
            x[u] = xyz[3 * i];
            y[u] = xyz[3 * i + 1];
            z[u] = xyz[3 * i + 2];
        }
        lo[0] = fminf(lo[0], x[u]); hi[0] = fmaxf(hi[0], x[u]);
        lo[1] = fminf(lo[1], y[u]); hi[1] = fmaxf(hi[1], y[u]);
        lo[2] = fminf(lo[2], z[u]); hi[2] = fmaxf(hi[2], z[u]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
        if (lane == 0) {
            s_box[warp][a] = lo[a];
            s_box[warp][3 + a] = hi[a];
        }
    }
    __syncthreads();
    if (warp < 6) {
        float v = s_box[lane][warp];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float w = __shfl_xor_sync(0xffffffffu, v, o);
            v = warp < 3 ? fminf(v, w) : fmaxf(v, w);
        }
        if (lane == 0) h->box[warp] = float_flip(v);
        __syncwarp();
        if (lane == 0) s_box[0][warp] = v;   // (column `warp` is this warp's alone)
    }
    __syncthreads();
    SceneNorm nm;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        nm.lo[a] = s_box[0][a];
        nm.ext[a] = fmaxf(__fsub_rn(s_box[0][3 + a], nm.lo[a]), 1e-6f);
    }
    if (sizeof(K) == 8) nm.ext[0] = nm.ext[1] = nm.ext[2] = fmaxf(nm.ext[0], fmaxf(nm.ext[1], nm.ext[2]));
    // (key, position) pairs, sorted: runs of 32 by shuffles, merges at
    // distance 32 and more in shared memory (all-ascending bitonic sort)
    uint64_t k[E];
    uint32_t v[E];
#pragma unroll
    for (int u = 0; u < E; ++u) {
        v[u] = u * SMALL_THREADS + tid;
        k[u] = v[u] < n ? (uint64_t)morton_key<K>(nm, scale, x[u], y[u], z[u]) : ~0ull;   // padding: last
    }
    auto lanes = [&](int mask, bool lower) {
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const uint64_t ok = __shfl_xor_sync(0xffffffffu, k[u], mask);
            const uint32_t ov = __shfl_xor_sync(0xffffffffu, v[u], mask);
            if ((ok < k[u] || (ok == k[u] && ov < v[u])) == lower) {
                k[u] = ok;
                v[u] = ov;
            }
        }
    };
#pragma unroll 1
    for (int kb = 2; kb <= 32; kb <<= 1) {
        int mask = kb - 1;
#pragma unroll 1
        for (int j = kb >> 1; j > 0; j >>= 1) {
            lanes(mask, (lane & j) == 0);
            mask = j >> 1;
        }
    }
#pragma unroll 1
    for (uint32_t kb = 64; kb <= P; kb <<= 1) {
#pragma unroll
        for (int u = 0; u < E; ++u) {
            s.key[u * SMALL_THREADS + tid] = k[u];
            s.idx[u * SMALL_THREADS + tid] = v[u];
        }
        __syncthreads();
#pragma unroll 1
        for (uint32_t j = kb >> 1; j >= 32; j >>= 1) {
            for (uint32_t t = tid; t < P / 2; t += SMALL_THREADS) {
                const uint32_t r = t & (j - 1), a = (t - r) * 2 + r, b = j == kb >> 1 ? (t - r) * 2 + 2 * j - 1 - r : a + j;
                const uint64_t ka = s.key[a], kc = s.key[b];
                const uint32_t va = s.idx[a], vc = s.idx[b];
                if (kc < ka || (kc == ka && vc < va)) {
                    s.key[a] = kc;
                    s.key[b] = ka;
                    s.idx[a] = vc;
                    s.idx[b] = va;
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int u = 0; u < E; ++u) {
            k[u] = s.key[u * SMALL_THREADS + tid];
            v[u] = s.idx[u * SMALL_THREADS + tid];
        }
#pragma unroll 1
        for (int j = 16; j > 0; j >>= 1) lanes(j, (lane & j) == 0);
    }
    // sorted keys and points, in shared memory and out
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const uint32_t i = u * SMALL_THREADS + tid;
        s.key[i] = k[u];   // (each thread's own elements)
        if (i < n) {
            const float4 p = make_float4(xyz[3 * v[u]], xyz[3 * v[u] + 1], xyz[3 * v[u] + 2], __uint_as_float(v[u]));
            s.pts[i] = p;
            out_pts[i] = p;
            out_keys[i] = (K)k[u];
        }
    }
    seed_sample(xyz, n, sample, h, tid, SMALL_THREADS);
    __syncthreads();
    if (n >= 2 && n > leaf_size) {
        // box pyramid
        Pyramid Py;
        Py.pts = s.pts;
        Py.pyr = s.pyr;
        Py.n = n;
        Py.nlev = 0;
        uint32_t size = n, off = 0, below = 0;
        while (size > PYR_B) {
            const uint32_t up = (size + PYR_B - 1) / PYR_B;
            for (uint32_t e = tid; e < up; e += SMALL_THREADS) {
                Box b;
                bool nan = false;
                box_empty(b);
                const uint32_t end = min(size, (e + 1) * PYR_B);
                for (uint32_t i = e * PYR_B; i < end; ++i) {
                    if (Py.nlev == 0) box_add_point(b, nan, s.pts[i]);
                    else box_add(b, s.pyr[2 * (below + i)], s.pyr[2 * (below + i) + 1]);
                }
                if (nan) box_unbounded(b);
                box_store(s.pyr, off + e, b);
                box_store(out_pyr, off + e, b);
            }
            below = off;
            off += up;
            size = up;
            ++Py.nlev;
            __syncthreads();
        }
        // kept nodes (keeps_node's test), numbered in order
        bool keep[E];
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int64_t i = u * SMALL_THREADS + tid;
            keep[u] = false;
            if (i + 1 < (int64_t)n) {
                int dir, dmin;
                karras_dir<uint64_t>(s.key, n, s.key[i], i, dir, dmin);
                keep[u] = delta<uint64_t>(s.key, n, s.key[i], i, i + (int64_t)leaf_size * dir) > dmin;
            }
            const uint32_t m = __ballot_sync(0xffffffffu, keep[u]);
            if (lane == 0) s_cnt[u * 32 + warp] = __popc(m);
        }
        __syncthreads();
        if (warp == 0) {
            uint32_t run = 0;
#pragma unroll
            for (int u = 0; u < E; ++u) {
                const uint32_t c = s_cnt[u * 32 + lane];
                uint32_t incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t w = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += w;
                }
                s_cnt[u * 32 + lane] = run + incl - c;
                run += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) {
                s_cnt[32 * E] = run;
                h->n_internal = run;
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const uint32_t i = u * SMALL_THREADS + tid, m = __ballot_sync(0xffffffffu, keep[u]);
            const uint32_t at = s_cnt[u * 32 + warp] + __popc(m & ((1u << lane) - 1u));
            s.cidx[i] = at;
            if (keep[u]) s.sel[at] = i;
        }
        __syncthreads();
        for (uint32_t c = tid; c < s_cnt[32 * E]; c += SMALL_THREADS) {
            uint32_t f0, last, sp;
            const int i = (int)s.sel[c];
            const uint64_t ki = s.key[i];
            int dir, dmin;
            karras_dir(s.key, (int64_t)n, ki, i, dir, dmin);
            karras_range<SMALL_MAX>(s.key, 0u, i, dir, dmin, dir > 0 ? (int)n - 1 - i : i, f0, last, sp);
            nodes[c] = make_node(Py, [&](uint32_t j) { return s.cidx[j]; }, leaf_size, f0, last, sp, 0u);
        }
        __syncthreads();
    }
    if (warp == 0) stage_top(h, nodes, top, n, leaf_size, s_q);
}

template <typename K, int E>
rtd_status launch_small(rtd_index *idx, const float *d_xyz, uint32_t n, float scale, cudaStream_t st) {
    RTD_CUDA(cudaFuncSetAttribute(small_build_kernel<K, E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)small_smem(E * SMALL_THREADS)));
    RTD_LAUNCH_CHAINED((small_build_kernel<K, E>), dim3(1), dim3(SMALL_THREADS), small_smem(n), st, d_xyz, n,
                       idx->hdr.as<IndexHeader>(), scale, idx->leaf_size, idx->keys.as<K>(), idx->pts.as<float4>(),
                       idx->pyramid.as<float4>(), idx->nodes.as<BvhNode>(), idx->top.as<BvhNode>(),
                       idx->sample.as<float4>());
    return RTD_OK;
}

template <typename K>
rtd_status build_small(rtd_index *idx, const float *d_xyz, uint32_t n, cudaStream_t st) {
    const int kbits = sizeof(K) == 4 ? 30 : idx->morton_bits;
    const float scale = sizeof(K) == 4 ? 1023.0f : (float)((1u << (kbits / 3)) - 1u);
    RTD_TRY(idx->keys.reserve(n * sizeof(K)));
    RTD_TRY(idx->pyramid.reserve(2 * pyramid_entries(n) * sizeof(float4)));
    RTD_TRY(idx->sample.reserve((SEED_PCT_POINTS + SEED_NN_SAMPLE) * sizeof(float4)));
    RTD_TRY(idx->seed.reserve(SEED_NN_SAMPLE * sizeof(float)));
    idx->nn_seeded = false;
    if (n <= SMALL_THREADS) RTD_TRY((launch_small<K, 1>(idx, d_xyz, n, scale, st)));
    else if (n <= 2 * SMALL_THREADS) RTD_TRY((launch_small<K, 2>(idx, d_xyz, n, scale, st)));
    else RTD_TRY((launch_small<K, 4>(idx, d_xyz, n, scale, st)));
    idx->skeys = idx->keys.ptr;
    idx->mark(EV_BUILD_SORTED, st);
    if (idx->ev_sorted) RTD_CUDA(cudaEventRecord(idx->ev_sorted, st));
    idx->mark(EV_BUILD1, st);
    return RTD_OK;
}

template <typename K>
rtd_status build_typed(rtd_index *idx, const float *d_xyz, uint64_t n, cudaStream_t st) {
    IndexHeader *h = idx->hdr.as<IndexHeader>();
    uint32_t *d_err = &h->err;
    const int kbits = sizeof(K) == 4 ? 30 : idx->morton_bits;
    const float scale = sizeof(K) == 4 ? 1023.0f : (float)((1u << (kbits / 3)) - 1u);
    RTD_TRY(idx->keys.reserve(n * sizeof(K)));
    RTD_TRY(idx->keys_alt.reserve(n * sizeof(K)));
    RTD_TRY(idx->vals.reserve(n * sizeof(uint32_t)));
    RTD_TRY(idx->vals_alt.reserve(n * sizeof(uint32_t)));
    const int g = grid_for(n, BLOCK, 148 * 8);
    RTD_LAUNCH_CHAINED(morton_kernel<K>, dim3(g), dim3(BLOCK), 0, st, d_xyz, n,
                       (const IndexHeader *)h, scale, idx->keys.as<K>(), aligned16(d_xyz));
    // the last pass gathers the points into idx->pts in key order
    K *skeys;
    if (sizeof(K) == 8 && kbits > 32 && kbits <= 48) {
        // 64-bit keys of up to 48 bits: the low bits as 64-bit keys, then
        // four passes over the top 32 bits as 32-bit keys
        RTD_TRY(idx->k32a.reserve(n * sizeof(uint32_t)));
        RTD_TRY(idx->k32b.reserve(n * sizeof(uint32_t)));
        RTD_TRY(radix_sort_split64(reinterpret_cast<const uint64_t *>(idx->keys.ptr),
                                   idx->keys_alt.as<uint64_t>(), idx->k32a.as<uint32_t>(),
                                   idx->k32b.as<uint32_t>(), idx->vals.as<uint32_t>(),
                                   idx->vals_alt.as<uint32_t>(), n, kbits, idx->sort, st, d_xyz,
                                   idx->pts.as<float4>(), idx->keys_alt.as<uint64_t>(), nullptr, true,
                                   SceneKeys{h, scale}));
        skeys = idx->keys_alt.as<K>();
    } else {
        bool in_alt = false;
        RTD_TRY(radix_sort_pairs<K>(idx->keys.as<K>(), idx->keys_alt.as<K>(),
                                    idx->vals.as<uint32_t>(), idx->vals_alt.as<uint32_t>(), true, n,
                                    0, kbits, idx->sort, d_err, st, &in_alt, d_xyz,
                                    idx->pts.as<float4>(), true));
        skeys = in_alt ? idx->keys_alt.as<K>() : idx->keys.as<K>();
    }
    idx->skeys = skeys;
    idx->mark(EV_BUILD_SORTED, st);
    // the sorted keys are ready: side-stream work may wait on this
    if (idx->ev_sorted) RTD_CUDA(cudaEventRecord(idx->ev_sorted, st));
    return build_tree_sorted<K>(idx, skeys, n, st, false, true);
}

}  // namespace

// The counts of the kept nodes: the words before the tiles' are added into
// and must be zero when the build of the tree starts.
static rtd_status tree_counts(rtd_index *idx, uint64_t n, TreeCounts &tc, uint32_t &n_zero) {
    const Levels L(ceil_div(n, (uint64_t)NODE_TILE));
    RTD_TRY(idx->kept_counts.reserve((2 + L.groups + L.supers + L.tiles) * sizeof(uint32_t)));
    tc.cross = idx->kept_counts.as<uint32_t>();
    tc.done = tc.cross + 1;
    tc.groups = tc.cross + 2;
    tc.supers = tc.groups + L.groups;
    tc.tiles = tc.supers + L.supers;
    n_zero = (uint32_t)(2 + L.groups + L.supers);
    return RTD_OK;
}

// Karras tree, leaf collapse and child boxes over keys already sorted, with
// idx->pts holding the points in key order.  top: stages the top levels too,
// and the counts are zero already (index_build).
template <typename K>
rtd_status build_tree_sorted(rtd_index *idx, const K *skeys, uint64_t n, cudaStream_t st,
                             bool ranges, bool top) {
    IndexHeader *h = idx->hdr.as<IndexHeader>();
    if (n < 2 || n <= idx->leaf_size) return RTD_OK;
    const uint64_t ni = n - 1;
    TreeCounts tc;
    uint32_t n_zero;
    RTD_TRY(tree_counts(idx, n, tc, n_zero));
    if (!top) RTD_TRY(zero_words(tc.cross, n_zero, st));
    for (rtd::DevBuf *b : {&idx->kept_bits, &idx->kept_before}) RTD_TRY(b->reserve(ceil_div(n, 32) * sizeof(uint32_t)));
    if (ranges)
        for (rtd::DevBuf *b : {&idx->kfirst, &idx->klast}) RTD_TRY(b->reserve(ni * sizeof(uint32_t)));
    // box pyramid over the sorted points (levels until one has <= 8 entries)
    Pyramid P;
    P.pts = idx->pts.as<float4>();
    uint64_t sizes[PYR_MAX + 1] = {n}, offs[PYR_MAX + 1] = {0}, total = 0;
    int nlev = 0;
    while (sizes[nlev] > PYR_B && nlev < PYR_MAX) {
        ++nlev;
        sizes[nlev] = ceil_div(sizes[nlev - 1], PYR_B);
        offs[nlev] = total;
        total += sizes[nlev];
    }
    P.nlev = nlev;
    P.n = (uint32_t)n;
    RTD_TRY(idx->pyramid.reserve((total ? total : 1) * 2 * sizeof(float4)));
    float4 *pyr = idx->pyramid.as<float4>();
    P.pyr = pyr;
    float4 *lv[PYR_MAX + 1] = {};
    for (int j = 1; j <= nlev; ++j) lv[j] = pyr + 2 * offs[j];
    const uint64_t tiles = ceil_div(n, (uint64_t)NODE_TILE);
    const uint32_t cross_cap = (uint32_t)(ni < NODE_DEPTH * tiles ? ni : NODE_DEPTH * tiles);
    RTD_TRY(idx->cross.reserve(cross_cap * sizeof(uint32_t)));
    RTD_LAUNCH_CHAINED(karras_count_kernel<K>, dim3((unsigned)tiles), dim3(BLOCK), 0, st, skeys, (int64_t)n,
                       idx->leaf_size, tc);
    uint32_t *kf = ranges ? idx->kfirst.as<uint32_t>() : nullptr, *kl = ranges ? idx->klast.as<uint32_t>() : nullptr;
    uint32_t *bits = idx->kept_bits.as<uint32_t>(), *before = idx->kept_before.as<uint32_t>();
    RTD_LAUNCH_CHAINED(tile_nodes_kernel<K>, dim3((unsigned)tiles), dim3(BLOCK), 0, st, skeys, n, h, tc, bits, before,
                       idx->leaf_size, (const float4 *)P.pts, lv[1], lv[2], lv[3], idx->nodes.as<BvhNode>(), kf, kl,
                       idx->cross.as<uint32_t>(), cross_cap);
    // three levels of the pyramid per launch: 4-6 from level 3, ...
    for (int j = 4; j <= nlev; j += 3)
        RTD_LAUNCH_CHAINED(pyramid_fold_kernel, dim3((unsigned)ceil_div(sizes[j - 1], 512)), dim3(512), 0, st,
                           (const float4 *)lv[j - 1], sizes[j - 1], lv[j], j + 1 <= nlev ? lv[j + 1] : nullptr,
                           j + 2 <= nlev ? lv[j + 2] : nullptr);
    // (a warp a node, for about 8 nodes a tile)
    RTD_LAUNCH_CHAINED(cross_nodes_kernel<K>, dim3((unsigned)(tiles < 148 * 8 ? tiles : 148 * 8)), dim3(BLOCK), 0, st,
                       skeys, n, h, tc, KeptNodes{bits, before}, idx->leaf_size, P, idx->nodes.as<BvhNode>(), kf, kl,
                       (const uint32_t *)idx->cross.as<uint32_t>(), cross_cap,
                       top ? idx->top.as<BvhNode>() : nullptr);
    return RTD_OK;
}

template rtd_status build_tree_sorted<uint32_t>(rtd_index *, const uint32_t *, uint64_t,
                                                cudaStream_t, bool, bool);
template rtd_status build_tree_sorted<uint64_t>(rtd_index *, const uint64_t *, uint64_t,
                                                cudaStream_t, bool, bool);

rtd_status ensure_side_stream(rtd_index *idx) {
    if (idx->side_stream) return RTD_OK;
    for (cudaEvent_t *e : {&idx->ev_fork, &idx->ev_join, &idx->ev_seed_fork, &idx->ev_seed_join,
                           &idx->ev_sorted})
        RTD_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    // created last: its presence means every stream and event exists
    RTD_CUDA(cudaStreamCreateWithFlags(&idx->side_stream, cudaStreamNonBlocking));
    return RTD_OK;
}

rtd_status index_build(rtd_index *idx, const float *d_xyz, uint64_t n, const rtd_schedule *s,
                       cudaStream_t st) {
    if (!idx) return fail(RTD_ERR_INVALID_ARGUMENT, "index is NULL");
    if (n > 0 && !d_xyz) return fail(RTD_ERR_INVALID_ARGUMENT, "points pointer is NULL");
    if (n >= (1ull << 30) - 1) return fail(RTD_ERR_INVALID_ARGUMENT, "at most 2^30-2 points");
    rtd_schedule def;
    rtd_schedule_default(&def);
    if (!s) s = &def;
    if (s->leaf_size < 1 || s->leaf_size > 64)
        return fail(RTD_ERR_INVALID_ARGUMENT, "leaf_size must be in [1, 64]");
    int mb = (int)s->morton_bits;
    // auto: 48-bit cubic keys (16 bits per axis); measured as fast to search as
    // 63-bit keys on the clustered and sheet workloads, with two fewer sort passes
    if (mb == 0) mb = 48;
    if (mb != 30 && (mb < 33 || mb > 63 || mb % 3 != 0))
        return fail(RTD_ERR_INVALID_ARGUMENT, "morton_bits must be 30 or a multiple of 3 in [33, 63]");
    RTD_CUDA(cudaGetDevice(&idx->device));
    idx->rtoken.valid = false;
    idx->skeys = nullptr;
    idx->n = n;
    idx->leaf_size = s->leaf_size;
    idx->morton_bits = mb;
    RTD_TRY(idx->hdr.reserve(sizeof(IndexHeader)));
    RTD_TRY(idx->pts.reserve((n ? n : 1) * sizeof(float4)));
    RTD_TRY(idx->nodes.reserve((n > 1 ? n - 1 : 1) * sizeof(BvhNode)));
    RTD_TRY(idx->top.reserve(TOP_MAX * sizeof(BvhNode)));
    IndexHeader *h = idx->hdr.as<IndexHeader>();
    for (bool &e : idx->ev_set) e = false;
    idx->mark(EV_BUILD0, st);
    if (n > 0 && n <= SMALL_MAX)
        return mb == 30 ? build_small<uint32_t>(idx, d_xyz, (uint32_t)n, st)
                        : build_small<uint64_t>(idx, d_xyz, (uint32_t)n, st);
    uint32_t *rows = nullptr, n_counts = 0;
    uint64_t n_rows = 0;
    TreeCounts tc{};
    if (n > 0) {
        RTD_TRY(radix_sort_sums(n, mb, idx->sort, &rows, &n_rows));
        RTD_TRY(tree_counts(idx, n, tc, n_counts));
    }
    RTD_LAUNCH_CHAINED(hdr_init_kernel, dim3(n_rows ? grid_for(n_rows, 256, 148 * 4) : 1), dim3(256), 0, st, h, rows,
                       n_rows, tc.cross, n_counts);
    if (n > 0) {
        RTD_LAUNCH_CHAINED(bbox_kernel, dim3(grid_for(n, BLOCK, 148 * 4)), dim3(BLOCK), 0, st, d_xyz,
                           n, h, aligned16(d_xyz));
        // the radius-seed sample reads only the input points: it runs on the
        // side stream while the keys are made and sorted
        RTD_TRY(ensure_side_stream(idx));
        RTD_CUDA(cudaEventRecord(idx->ev_seed_fork, st));
        RTD_CUDA(cudaStreamWaitEvent(idx->side_stream, idx->ev_seed_fork, 0));
        const rtd_status rs = build_seed(idx, d_xyz, n, idx->side_stream);
        RTD_CUDA(cudaEventRecord(idx->ev_seed_join, idx->side_stream));
        const rtd_status rb = mb == 30 ? build_typed<uint32_t>(idx, d_xyz, n, st)
                                       : build_typed<uint64_t>(idx, d_xyz, n, st);
        RTD_CUDA(cudaStreamWaitEvent(st, idx->ev_seed_join, 0));   // also on the error paths
        RTD_TRY(rs);
        RTD_TRY(rb);
    }
    idx->mark(EV_BUILD1, st);
    return RTD_OK;
}

// ------------------------------------------------------- query ordering
namespace {
// Processing-order keys of the queries: 30-bit Morton codes; with chunks > 1
// the query's chunk (i * chunks / nq) takes the top cbits bits of a 32-bit
// key and the code loses its cbits - 2 lowest bits if it must.
__global__ void __launch_bounds__(BLOCK) query_morton_kernel(const float *__restrict__ q,
                                                             uint64_t nq, const IndexHeader *h,
                                                             uint32_t chunks, int cbits,
                                                             uint32_t *__restrict__ keys) {
    const SceneNorm s = scene_norm_cubic(h);   // processing order only
    const int drop = cbits > 2 ? cbits - 2 : 0;
    for (uint64_t i = (uint64_t)blockIdx.x * BLOCK + threadIdx.x; i < nq;
         i += (uint64_t)gridDim.x * BLOCK) {
        const uint32_t code = morton30(quantize(q[3 * i], s.lo[0], s.ext[0], 1023.0f),
                                       quantize(q[3 * i + 1], s.lo[1], s.ext[1], 1023.0f),
                                       quantize(q[3 * i + 2], s.lo[2], s.ext[2], 1023.0f));
        keys[i] = cbits ? ((uint32_t)(i * chunks / nq) << (32 - cbits)) | (code >> drop) : code;
    }
}
}  // namespace

rtd_status order_queries(rtd_index *idx, const float *d_q, uint64_t nq, bool morton,
                         const uint32_t **perm, cudaStream_t st) {
    *perm = nullptr;
    idx->rtoken.valid = false;   // the query-order buffers are about to change
    if (!morton || nq < 2) return RTD_OK;
    if (nq >= (1ull << 30)) return fail(RTD_ERR_INVALID_ARGUMENT, "at most 2^30-1 queries");
    RTD_TRY(idx->qkeys.reserve(nq * 4));
    RTD_TRY(idx->qkeys_alt.reserve(nq * 4));
    RTD_TRY(idx->qperm.reserve(nq * 4));
    RTD_TRY(idx->qperm_alt.reserve(nq * 4));
    IndexHeader *h = idx->hdr.as<IndexHeader>();
    query_morton_kernel<<<grid_for(nq, BLOCK, 148 * 8), BLOCK, 0, st>>>(d_q, nq, h, 1u, 0,
                                                                        idx->qkeys.as<uint32_t>());
    RTD_LAUNCH_CHECK();
    bool in_alt = false;
    RTD_TRY(radix_sort_pairs<uint32_t>(idx->qkeys.as<uint32_t>(), idx->qkeys_alt.as<uint32_t>(),
                                       idx->qperm.as<uint32_t>(), idx->qperm_alt.as<uint32_t>(),
                                       true, nq, 0, 30, idx->sort, &h->err, st, &in_alt));
    *perm = in_alt ? idx->qperm_alt.as<uint32_t>() : idx->qperm.as<uint32_t>();
    return RTD_OK;
}

rtd_status order_queries_own(QueryOrderScratch &qs, const float *d_q, uint64_t nq,
                             const uint32_t **perm, cudaStream_t st, uint32_t chunks) {
    *perm = nullptr;
    if (nq < 2) return RTD_OK;
    if (nq >= (1ull << 30)) return fail(RTD_ERR_INVALID_ARGUMENT, "at most 2^30-1 queries");
    if (chunks < 1 || chunks > (uint32_t)MAX_CHUNKS) return fail(RTD_ERR_INVALID_ARGUMENT, "bad chunk count");
    RTD_TRY(qs.hdr.reserve(sizeof(IndexHeader)));
    RTD_TRY(qs.keys.reserve(nq * 4));
    RTD_TRY(qs.keys_alt.reserve(nq * 4));
    RTD_TRY(qs.perm.reserve(nq * 4));
    RTD_TRY(qs.perm_alt.reserve(nq * 4));
    IndexHeader *h = qs.hdr.as<IndexHeader>();
    hdr_init_kernel<<<1, 256, 0, st>>>(h, nullptr, 0, nullptr, 0);
    RTD_LAUNCH_CHECK();
    bbox_kernel<<<grid_for(nq, BLOCK, 148 * 4), BLOCK, 0, st>>>(d_q, nq, h, aligned16(d_q));
    RTD_LAUNCH_CHECK();
    int cbits = 0;
    while ((1u << cbits) < chunks) ++cbits;
    query_morton_kernel<<<grid_for(nq, BLOCK, 148 * 8), BLOCK, 0, st>>>(d_q, nq, h, chunks, cbits,
                                                                        qs.keys.as<uint32_t>());
    RTD_LAUNCH_CHECK();
    bool in_alt = false;
    RTD_TRY(radix_sort_pairs<uint32_t>(qs.keys.as<uint32_t>(), qs.keys_alt.as<uint32_t>(),
                                       qs.perm.as<uint32_t>(), qs.perm_alt.as<uint32_t>(), true,
                                       nq, 0, cbits ? 32 : 30, qs.sort, &h->err, st, &in_alt));
    *perm = in_alt ? qs.perm_alt.as<uint32_t>() : qs.perm.as<uint32_t>();
    return RTD_OK;
}

}  // namespace rtd
