// knn_collect.cuh -- one query's exact k-NN by a warp that collects
// candidates and selects, shared by the single-cloud search (knn.cu) and the
// batched many-cloud search (batch.cu).
//
//   1. The points around the query's position in the index's Morton order
//      fill a buffer in shared memory; their k-th smallest key bounds the
//      search radius from the start.
//   2. The boxes of the pyramid over the sorted points (an implicit 8-ary
//      tree: level j entry e covers the points [e 8^j, (e + 1) 8^j)) are
//      walked 32 at a time, four popped nodes' eight children each; points
//      of passing runs of 8 are tested 64 at a time and appended when they
//      beat the bound.  A full buffer is cut back to its k best, which
//      tightens the bound.
//   3. The k best are sorted in registers and written.
//
// The k best (FP32 key, id) pairs do not depend on the order of the walk or
// on the bound it starts from, so no radius rounds are needed for an exact
// result.
#pragma once

#include "index.cuh"

namespace rtd {

// Points of a cloud in sorted order with the pyramid over all sorted points.
struct CollectTree {
    const float4 *pts;
    const float4 *pyr;
    const uint32_t *off;   // off[j]: first pyramid entry of level j >= 1
    uint32_t begin, end;   // the cloud's sorted points
};

// Shared memory of one warp.
struct CollectScratch {
    float *key;       // cap candidate keys
    uint32_t *id;     // and their ids
    uint2 *stack;     // (level << 28 | entry, bits of the box's smallest key)
    uint2 *leaf;      // COLLECT_LEAFQ runs of 8 points, the same fields
    uint32_t cap;
};
constexpr uint32_t COLLECT_LEAFQ = 48;    // a node step leaves at most 7 + 32
constexpr uint32_t COLLECT_MAX_K = 2048;

// Candidate slots for lists of kk: the window, and k more before a cut.
__host__ __device__ constexpr uint32_t collect_cap(uint32_t kk) { return (2 * kk + 64 + 31) / 32 * 32; }
// Stack entries for n sorted points: LIFO groups of at most 32 entries, the
// highest level in a group one below the highest in the group under it.
__host__ __device__ inline uint32_t collect_stack(uint64_t n) {
    uint32_t levels = 1;
    while (n > 32) { n = (n + 7) / 8; ++levels; }
    return 32 * levels;
}
__host__ __device__ inline size_t collect_warp_bytes(uint32_t kk, uint64_t n) {
    return (size_t)(collect_cap(kk) + collect_stack(n) + COLLECT_LEAFQ) * sizeof(uint2);
}
__device__ __forceinline__ CollectScratch collect_scratch(void *base, uint32_t kk, uint32_t n) {
    CollectScratch s;
    s.cap = collect_cap(kk);
    s.stack = static_cast<uint2 *>(base);
    s.leaf = s.stack + collect_stack(n);
    s.key = reinterpret_cast<float *>(s.leaf + COLLECT_LEAFQ);
    s.id = reinterpret_cast<uint32_t *>(s.key + s.cap);
    return s;
}

// Pyramid level offsets of n points (the layout of build_tree_sorted).
__device__ __forceinline__ void collect_offsets(uint32_t n, uint32_t *off) {
    uint32_t acc = 0, size = n;
    off[0] = 0;
    for (int j = 1; j <= 11; ++j) {
        off[j] = acc;
        size = (size + 7) / 8;
        acc += size;
    }
}

// First position in [lo, hi) of sorted keys whose key is not below `key`,
// 33-way by a warp.
template <typename K>
__device__ __forceinline__ uint32_t warp_lower_bound(const K *__restrict__ sk, uint32_t lo, uint32_t hi, K key) {
    const int lane = threadIdx.x & 31;
    while (hi - lo > 32) {
        const uint32_t step = (hi - lo) / 33 + 1, at = lo + (lane + 1) * step - 1;
        const uint32_t less = __popc(__ballot_sync(0xffffffffu, at < hi && __ldg(&sk[at]) < key));
        const uint32_t next = lo + (less + 1) * step - 1;   // the first probe not below the key
        lo += less * step;
        if (less < 32 && next < hi) hi = next;
    }
    return lo + __popc(__ballot_sync(0xffffffffu, lo + lane < hi && __ldg(&sk[lo + lane]) < key));
}

// The candidates of a warp: key[0 .. cnt) in no order, and the exclusive
// bound (tk, ti) below which a (key, id) pair still matters.
struct Collected {
    uint32_t cnt;
    float tk;
    uint32_t ti;
};

// Cuts the cnt > kk candidates back to between kk and kk + slack of the
// smallest (exactly kk when keys tie across the cut) and sets the bound.
// The kk-th smallest key is found bit by bit from the highest bit in which
// the keys differ (keys are >= +0, so their bits order as they do), stopping
// at the first threshold that keeps few enough.  Up to 192 keys (k <= 64)
// stay in registers meanwhile: a cut of 64 then takes about 150 instructions
// instead of 450.  (Not inlined: its four call sites would not fit the
// instruction cache.)
constexpr int CUT_REGS = 6;
template <bool small>
static __device__ __noinline__ Collected collect_cut_sized(float *key, uint32_t *ids, Collected c, uint32_t kk,
                                                           uint32_t slack) {
    constexpr int REGS = small ? CUT_REGS : 1;
    const int lane = threadIdx.x & 31;
    const uint32_t *kb = reinterpret_cast<const uint32_t *>(key);
    __syncwarp();
    uint32_t v[REGS];   // missing ones as the largest value, which is no key
    uint32_t mn = 0xFFFFFFFFu, mx = 0;
    if (small) {
#pragma unroll
        for (int u = 0; u < REGS; ++u) {
            v[u] = 0xFFFFFFFFu;
            if (u * 32 < c.cnt) {
                if (u * 32 + lane < c.cnt) {
                    v[u] = kb[u * 32 + lane];
                    mx = max(mx, v[u]);
                }
                mn = min(mn, v[u]);
            }
        }
    } else {
        for (uint32_t j = lane; j < c.cnt; j += 32) {
            const uint32_t x = kb[j];
            mn = min(mn, x);
            mx = max(mx, x);
        }
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    uint32_t lo = mx, below = 0;   // keys below lo
    bool found = false;
    if (mn != mx) {
        int b = 31 - __clz(mn ^ mx);
        lo = mx >> b >> 1 << b << 1;
        for (; b >= 0; --b) {
            const uint32_t test = lo | (1u << b);
            uint32_t n = 0;
            if (small) {
#pragma unroll
                for (int u = 0; u < REGS; ++u)
                    if (u * 32 < c.cnt) n += v[u] < test;
            } else {
                for (uint32_t j = lane; j < c.cnt; j += 32) n += kb[j] < test;
            }
            n = __reduce_add_sync(0xffffffffu, n);
            if (n < kk) {
                lo = test;
                below = n;
            } else if (n <= kk + slack) {
                // (a threshold past +inf keeps every key)
                c.tk = test > 0x7F800000u ? INFINITY : __uint_as_float(test);
                c.ti = test > 0x7F800000u ? EMPTY_ID : 0u;
                found = true;
                break;
            }
        }
    }
    if (!found) {   // lo is the kk-th key, and too many share it: the lowest ids stay
        const uint32_t r = kk - below;
        uint32_t id = 0;
        for (int b = 31; b >= 0; --b) {
            const uint32_t test = id | (1u << b);
            uint32_t n = 0;
            for (uint32_t j = lane; j < c.cnt; j += 32) n += kb[j] == lo && ids[j] < test;
            if (__reduce_add_sync(0xffffffffu, n) < r) id = test;
        }
        c.tk = __uint_as_float(lo);
        c.ti = id + 1;
    }
    uint32_t out = 0;
    auto chunk = [&](uint32_t j, float k) {
        uint32_t i = 0;
        bool keep = false;
        if (j < c.cnt) {
            i = ids[j];
            keep = key_less(k, i, c.tk, c.ti);
        }
        const uint32_t m = __ballot_sync(0xffffffffu, keep);
        __syncwarp();
        if (keep) {
            const uint32_t at = out + __popc(m & ((1u << lane) - 1u));
            key[at] = k;
            ids[at] = i;
        }
        out += __popc(m);
    };
    if (small) {
#pragma unroll
        for (int u = 0; u < REGS; ++u)
            if (u * 32 < c.cnt) chunk(u * 32 + lane, __uint_as_float(v[u]));
    } else {
        for (uint32_t base = 0; base < c.cnt; base += 32) {
            const uint32_t j = base + lane;
            chunk(j, j < c.cnt ? key[j] : 0.f);
        }
    }
    c.cnt = out;
    __syncwarp();
    return c;
}
__device__ __forceinline__ Collected collect_cut(float *key, uint32_t *ids, Collected c, uint32_t kk, uint32_t slack) {
    return c.cnt <= 32 * CUT_REGS ? collect_cut_sized<true>(key, ids, c, kk, slack)
                                  : collect_cut_sized<false>(key, ids, c, kk, slack);
}

// The candidates of one query: on return at least min(kk, finite-key points)
// of them, the kk best among them.  pos: the query's Morton position in
// [begin, end].  All arguments are warp-uniform.
// WHOLE: the cloud is the whole index.
template <bool WHOLE>
__device__ __forceinline__ Collected collect_query(const CollectTree &t, const CollectScratch &s, float qx, float qy,
                                                   float qz, uint32_t kk, uint32_t pos) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    Collected c{0, INFINITY, EMPTY_ID};
    if (isnan(qx) || isnan(qy) || isnan(qz) || t.begin >= t.end) return c;
    auto append = [&](bool ok, float key, uint32_t id) {
        ok = ok && key_less(key, id, c.tk, c.ti);
        const uint32_t m = __ballot_sync(0xffffffffu, ok);
        if (ok) {
            const uint32_t at = c.cnt + __popc(m & lt);
            s.key[at] = key;
            s.id[at] = id;
        }
        c.cnt += __popc(m);
    };
    const uint32_t slack = kk / 8 + 4;
    // the window: as many points as the buffer takes up to 2k (at least 64)
    const uint32_t n = t.end - t.begin;
    uint32_t w = 2 * kk > 64 ? 2 * kk : 64u;
    if (w > n) w = n;
    uint32_t w0 = pos > t.begin + w / 2 ? pos - w / 2 : t.begin;
    if (w0 + w > t.end) w0 = t.end - w;
    for (uint32_t j0 = 0; j0 < w; j0 += 32) {
        const bool ok = j0 + lane < w;
        const float4 p = ok ? __ldg(&t.pts[w0 + j0 + lane]) : make_float4(0.f, 0.f, 0.f, 0.f);
        append(ok, exact_key(qx, qy, qz, p.x, p.y, p.z), __float_as_uint(p.w));
    }
    if (w == n) return c;
    if (c.cnt > kk) c = collect_cut(s.key, s.id, c, kk, slack);

    // boxes of `level`: the start level's entries over the cloud, then the
    // children of popped nodes
    uint32_t sp = 0, lq = 0;
    auto visit = [&](bool ok, uint32_t level, uint32_t e) {
        float bk = 0.f;
        if (ok) {
            const float4 *b = t.pyr + 2 * (uint64_t)(t.off[level] + e);
            const float4 lo = __ldg(b), hi = __ldg(b + 1);
            bk = box_min_key(qx, qy, qz, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z);
            ok = !(bk > c.tk);
        }
        // far boxes go under the near ones, which are then popped first: when
        // the window lay far from the query, the bound shrinks before a
        // dense cluster inside it is walked
        const bool near = bk * 16.0f <= c.tk;
        const uint32_t mo = __ballot_sync(0xffffffffu, ok), ml = mo & __ballot_sync(0xffffffffu, level == 1);
        const uint32_t mnear = __ballot_sync(0xffffffffu, near);
        const uint32_t same = level == 1 ? ml : mo & ~ml, nl = __popc(ml), nn = __popc(mo & ~ml);
        const uint32_t at = __popc(same & (near ? mnear : ~mnear) & lt);
        uint2 *to = level == 1 ? s.leaf + lq : s.stack + sp;
        if (ok) to[near ? (level == 1 ? nl : nn) - 1 - at : at] = make_uint2(level << 28 | e, __float_as_uint(bk));
        lq += nl;
        sp += nn;
        __syncwarp();
    };
    uint32_t top = 1;
    while (((t.end - 1) >> (3 * top)) - (t.begin >> (3 * top)) >= 32) ++top;
    {
        const uint32_t e = (t.begin >> (3 * top)) + lane;
        visit(e <= (t.end - 1) >> (3 * top), top, e);
    }
    while (sp | lq) {
        if (lq >= 8 || sp == 0) {
            // up to 8 runs of 8 points, two points a lane
            const uint32_t take = lq < 8 ? lq : 8u;
            lq -= take;
            float4 p[2];
            bool ok[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t r = 4 * u + (lane >> 3);
                ok[u] = false;
                p[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < take) {
                    const uint2 e = s.leaf[lq + r];
                    const uint32_t at = (e.x & 0x0FFFFFFFu) * 8 + (lane & 7);
                    ok[u] = !(__uint_as_float(e.y) > c.tk) && (WHOLE || at >= t.begin) && at < t.end && at - w0 >= w;
                    if (ok[u]) p[u] = __ldg(&t.pts[at]);
                }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (c.cnt + 32 > s.cap) c = collect_cut(s.key, s.id, c, kk, slack);
                append(ok[u], exact_key(qx, qy, qz, p[u].x, p[u].y, p[u].z), __float_as_uint(p[u].w));
            }
            __syncwarp();
        } else {
            const uint32_t take = sp < 4 ? sp : 4u;
            sp -= take;
            const uint32_t r = lane >> 3;
            bool ok = r < take;
            uint32_t level = 2, e = 0;
            if (ok) {
                const uint2 node = s.stack[sp + r];
                level = node.x >> 28;
                e = (node.x & 0x0FFFFFFFu) * 8 + (lane & 7);
                ok = !(__uint_as_float(node.y) > c.tk);
            }
            --level;
            // children that hold points of the cloud
            ok = ok && e <= (t.end - 1) >> (3 * level) && (WHOLE || e >= t.begin >> (3 * level));
            __syncwarp();
            visit(ok, level, e);
        }
    }
    return c;
}

// One compare-exchange of every register's 32 elements with the lane at
// xor distance `mask`; the lanes marked `lower` keep the smaller pair.
template <int E>
__device__ __forceinline__ void collect_lane_exchange(float (&key)[E], uint32_t (&id)[E], int mask, bool lower) {
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const float ok = __shfl_xor_sync(0xffffffffu, key[u], mask);
        const uint32_t oi = __shfl_xor_sync(0xffffffffu, id[u], mask);
        const bool sw = key_less(ok, oi, key[u], id[u]) == lower;
        key[u] = sw ? ok : key[u];
        id[u] = sw ? oi : id[u];
    }
}

// Sorts the candidates and writes the first k; slots past them get the
// empty pair.  A bitonic sort in its all-ascending form (the first exchange
// of a merge mirrors the upper half): the padding at the end never moves, so
// only runs of 32 that hold candidates take part.  Exchanges at distance 32
// and more go through shared memory, the others through shuffles, two runs
// at a time; everything loops (sorts unrolled in registers, E = 12 for k =
// 300, spent more time on instruction fetches than on anything else).
static __device__ __noinline__ void collect_sort_store(float *key, uint32_t *id, uint32_t cnt, uint32_t k, uint32_t *ids,
                                                float *d2) {
    const int lane = threadIdx.x & 31;
    const uint32_t runs = cnt ? (cnt + 31) / 32 : 1u, n = runs * 32;
    auto store = [&](uint32_t j, float kv, uint32_t iv) {
        if (j < k) {
            ids[j] = iv;
            if (d2) d2[j] = kv;
        }
    };
    for (uint32_t j = n + lane; j < k; j += 32) store(j, INFINITY, EMPTY_ID);
    auto sort_lanes = [&](auto &x, auto &y) {   // every register's 32 elements
        constexpr int E = sizeof(x) / sizeof(x[0]);
#pragma unroll 1
        for (int kb = 2; kb <= 32; kb <<= 1) {
            int mask = kb - 1;
#pragma unroll 1
            for (int j = kb >> 1; j > 0; j >>= 1) {
                collect_lane_exchange<E>(x, y, mask, (lane & j) == 0);
                mask = j >> 1;
            }
        }
    };
    if (runs == 1) {
        float x[1] = {(uint32_t)lane < cnt ? key[lane] : INFINITY};
        uint32_t y[1] = {(uint32_t)lane < cnt ? id[lane] : EMPTY_ID};
        sort_lanes(x, y);
        store(lane, x[0], y[0]);
        return;
    }
    for (uint32_t r = 0; r < runs; r += 2) {
        float x[2];
        uint32_t y[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t j = (r + u) * 32 + lane;
            x[u] = j < cnt ? key[j] : INFINITY;
            y[u] = j < cnt ? id[j] : EMPTY_ID;
        }
        sort_lanes(x, y);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t j = (r + u) * 32 + lane;
            if (j < n) {
                key[j] = x[u];
                id[j] = y[u];
            }
        }
    }
    __syncwarp();
    auto exchange = [&](uint32_t a, uint32_t b) {
        if (b >= n) return;
        const float ka = key[a], kc = key[b];
        const uint32_t ia = id[a], ic = id[b];
        if (key_less(kc, ic, ka, ia)) {
            key[a] = kc;
            key[b] = ka;
            id[a] = ic;
            id[b] = ia;
        }
    };
    for (uint32_t m = 2; m < 2 * runs; m <<= 1) {   // merges of m / 2 runs with m / 2 runs
        const uint32_t half = m * 16, pairs = (runs + m - 1) / m * half;
        for (uint32_t p = lane; p < pairs; p += 32) {
            const uint32_t x = p & (half - 1), blk = (p - x) * 2;
            exchange(blk + x, blk + 2 * half - 1 - x);
        }
        __syncwarp();
        for (uint32_t j = half >> 1; j >= 32; j >>= 1) {
            for (uint32_t p = lane; p < pairs; p += 32) {
                const uint32_t x = p & (j - 1), a = (p - x) * 2 + x;
                exchange(a, a + j);
            }
            __syncwarp();
        }
        const bool last = m >= runs;
        for (uint32_t r = 0; r < runs; r += 2) {
            float x[2];
            uint32_t y[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t j = (r + u) * 32 + lane;
                x[u] = j < n ? key[j] : INFINITY;
                y[u] = j < n ? id[j] : EMPTY_ID;
            }
#pragma unroll 1
            for (int j = 16; j > 0; j >>= 1) collect_lane_exchange<2>(x, y, j, (lane & j) == 0);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t j = (r + u) * 32 + lane;
                if (last) {
                    if (j < n) store(j, x[u], y[u]);
                } else if (j < n) {
                    key[j] = x[u];
                    id[j] = y[u];
                }
            }
        }
        __syncwarp();
    }
}

// Writes the k best of the candidates (kk = min(k, the cloud's points)).
// The sort takes up to a quarter more than kk, unless that needs one merge
// more, which costs more than cutting the candidates closer.
__device__ __forceinline__ void collect_store(const CollectScratch &s, Collected c, uint32_t kk, uint32_t k,
                                              uint32_t *ids, float *d2) {
    uint32_t most = 32;
    while (most < kk) most <<= 1;
    const uint32_t want = (kk + kk / 4 + 4 + 31) / 32 * 32;
    if (want < most) most = want;
    if (c.cnt > most) c = collect_cut(s.key, s.id, c, kk, most - kk);
    __syncwarp();
    collect_sort_store(s.key, s.id, c.cnt, k, ids, d2);
    __syncwarp();
}

}  // namespace rtd
