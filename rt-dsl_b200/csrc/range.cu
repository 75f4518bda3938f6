// range.cu -- fixed-radius range query: a count pass sizes the output, a
// fill pass writes (query, id) pairs into it.  Replaces the reference's
// global-push programs (gprt-macros/src/lib.rs:276-295), where every
// any-hit does atomicAdd(&lens[q], 1) into a capped per-query slab that the
// host then copies back and filters (lib.rs:538-583).  Here the buffer is
// exactly sized by the count pass.  A fill that follows the count of the
// same queries writes every query's hits into its own segment of the
// buffer, at the offsets the count's exclusive scan left on the index (no
// atomics; pairs come out grouped by query in the caller's order).  Any
// other fill stages hits per warp in shared memory and pushes them with one
// global atomicAdd per flush (warp-aggregated compaction).  Membership:
// exact FP32 key <= RN(r*r), as the intersection program tests
// dist_sq <= r_val*r_val (lib.rs:283, 341).
#include "knn_backward.cuh"
#include "knn_collect.cuh"

namespace rtd {
namespace {

constexpr int RBLOCK = 128;
constexpr int RWARPS = RBLOCK / 32;
constexpr uint32_t WBUF = 256;     // staged pairs per warp (2 KB)
constexpr uint32_t WRECS = 64;     // staged records per warp (1 KB)

// Kernel modes: count hits, push pairs through warp staging and a global
// cursor, write pairs into per-query segments at known offsets, or count
// hits and push them at once (a count whose pairs the next fill scatters).
// MODE_SAMPLE counts a sample of the queries for launch_pass.
enum : int { MODE_COUNT = 0, MODE_PUSH = 1, MODE_SEG = 2, MODE_CPUSH = 3, MODE_SAMPLE = 4 };

struct RangeArgs {
    IndexView ix;
    const float4 *pyr;         // box pyramid over the sorted points
    const float *q;
    uint64_t nq;
    const uint32_t *perm;
    float r2;
    uint32_t *counts;
    uint32_t *most;            // counts and MODE_SAMPLE: the largest count
    int by_sample;             // the sample of the queries says which kernel runs (warp_walks)
    int small_leaves;          // the tree's leaves hold fewer than 6 points
    uint64_t sample_step;      // MODE_SAMPLE: every sample_step-th query
    uint32_t *sample_sum;      // MODE_SAMPLE: the sum of the counts
    uint2 *pairs;
    uint64_t capacity;
    unsigned long long *cursor;
    const uint64_t *offsets;   // MODE_SEG: exclusive offsets of the count pass
    uint64_t total;            // MODE_SEG: end of the last segment
    int skip_if_same;          // MODE_SEG: do nothing when the header's two query
                               // fingerprints agree (the scatter fills instead)
    // MODE_CPUSH: every box of 64 or more points inside the ball becomes a
    // record (query, first sorted point, points) that the fill's expansion
    // writes out; cursor[1] counts records, cursor[2] the points they cover
    uint4 *recs;
    uint64_t rec_cap;
    uint32_t *err;
};

// Whether a warp per query is ahead of a thread per query, by the hits of
// SAMPLE of the nq queries (launch_pass says why the lines lie here).
constexpr uint64_t SAMPLE = 1024;
template <int MODE>
__device__ __forceinline__ bool warp_walks(const IndexHeader *h, uint64_t nq, int small_leaves) {
    const uint64_t sum = h->sample_sum, most = h->sample_most;
    if (sum >= 64 * SAMPLE || most * SAMPLE >= nq) return true;
    return MODE == MODE_CPUSH && small_leaves && sum * sum * 2800 >= nq * SAMPLE * SAMPLE;
}

// Shared memory of one warp: the boxes to visit (level << 28 | entry), runs
// of 8 points to test, staged pairs and records.
__host__ __device__ inline size_t range_warp_bytes(int mode, uint64_t n) {
    const size_t lists = (collect_stack(n) + COLLECT_LEAFQ) * sizeof(uint32_t);
    const size_t pairs = mode == MODE_PUSH || mode == MODE_CPUSH ? WBUF * sizeof(uint2) : 0;
    return pairs + (mode == MODE_CPUSH ? WRECS * sizeof(uint4) : 0) + lists;
}

// A warp per query (grid-stride).  The boxes of the pyramid over the sorted
// points are walked 32 at a time, the eight children of four popped entries
// (knn_collect.cuh describes the walk); a box of 64 or more points wholly
// inside the ball (farthest-corner key <= r^2, a bound on every point's key)
// contributes all its points without a test: its count in the count pass,
// its contiguous ids in the fills; the points of the other runs of 8 are
// tested 64 at a time, and one ballot gives every hit its rank.  MODE_SEG
// writes them at the next slots of the query's segment and checks that the
// query fills it exactly; the pushing modes compact them into the warp's
// staging buffer, which outlives the query and is pushed with one global
// atomic when it fills.
//
// Bound by instruction issue.  It replaced a thread per query over the binary
// tree with the candidates of a step spread over the warp, in which the
// longest walk of 32 queries held the others: 1.8M clustered points, 400,000
// queries, 50 hits a query: pushing count 2.40 -> 0.96 ms; 200,000 points,
// 20 hits: 0.87 -> 0.34 ms.
template <int MODE>
__global__ void __launch_bounds__(RBLOCK, 10) range_kernel(const RangeArgs p) {
    constexpr bool PUSH = MODE == MODE_PUSH || MODE == MODE_CPUSH;   // through warp staging
    constexpr bool SEG = MODE == MODE_SEG;
    constexpr bool COUNTS = MODE == MODE_COUNT || MODE == MODE_CPUSH;
    if (SEG && p.skip_if_same && p.ix.hdr->qfp[0] == p.ix.hdr->qfp[1]) return;
    if (MODE != MODE_SAMPLE && p.by_sample && !warp_walks<MODE>(p.ix.hdr, p.nq, p.small_leaves)) return;
    extern __shared__ uint4 s_dyn[];
    __shared__ uint32_t s_off[12];
    const uint32_t n = (uint32_t)p.ix.n;
    if (threadIdx.x == 0) collect_offsets(n, s_off);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    char *base = reinterpret_cast<char *>(s_dyn) + warp * range_warp_bytes(MODE, n);
    uint4 *const recs = reinterpret_cast<uint4 *>(base);
    uint2 *const buf = reinterpret_cast<uint2 *>(base + (MODE == MODE_CPUSH ? WRECS * sizeof(uint4) : 0));
    uint32_t *const leaf = reinterpret_cast<uint32_t *>(buf + (PUSH ? WBUF : 0));
    uint32_t *const stack = leaf + COLLECT_LEAFQ;
    const float4 *__restrict__ pts = p.ix.pts;
    const float r2 = p.r2;
    uint32_t fill = 0, nrec = 0;             // staged pairs and records (warp-uniform)
    unsigned long long covered = 0;          // points of this warp's records
    uint32_t most = 0;                       // the largest count of this warp's queries

    // pushes the staged pairs / records with one reservation on the cursor
    auto flush = [&]() {
        if (fill == 0) return;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(p.cursor, (unsigned long long)fill);
        at = __shfl_sync(0xffffffffu, at, 0);
        __syncwarp();
        for (uint32_t j = lane; j < fill; j += 32)
            if (at + j < p.capacity) p.pairs[at + j] = buf[j];
        // (the count's own pushes are speculative: a short buffer only
        // means the fill runs its own traversal)
        if (MODE == MODE_PUSH && lane == 0 && at + fill > p.capacity) atomicOr(p.err, DEVERR_OVERFLOW);
        __syncwarp();
        fill = 0;
    };
    auto flush_recs = [&]() {
        if (nrec == 0) return;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&p.cursor[1], (unsigned long long)nrec);
        at = __shfl_sync(0xffffffffu, at, 0);
        __syncwarp();
        for (uint32_t j = lane; j < nrec; j += 32)
            if (at + j < p.rec_cap) p.recs[at + j] = recs[j];
        __syncwarp();
        nrec = 0;
    };

    uint32_t top = 1;
    while (n > 64 && (n - 1) >> (3 * top) >= 32) ++top;

    for (uint64_t t = (uint64_t)blockIdx.x * RWARPS + warp; t < p.nq; t += (uint64_t)gridDim.x * RWARPS) {
        const uint32_t qi = MODE == MODE_SAMPLE ? (uint32_t)(t * p.sample_step) : p.perm ? p.perm[t] : (uint32_t)t;
        const float qx = p.q[3 * (uint64_t)qi], qy = p.q[3 * (uint64_t)qi + 1], qz = p.q[3 * (uint64_t)qi + 2];
        uint64_t wb = 0;      // MODE_SEG: this query's segment of the pair buffer
        uint32_t wlen = 0;
        if (SEG) {
            wb = p.offsets[qi];
            wlen = (uint32_t)((qi + 1 < p.nq ? p.offsets[qi + 1] : p.total) - wb);
        }
        uint32_t cnt = 0, sp = 0, lq = 0;
        bool seg_bad = false;
        // the ids of `c` sorted points from f on, all of them hits
        auto copy_run = [&](uint32_t f, uint32_t c) {
            for (uint32_t j0 = 0; j0 < c; j0 += 32) {
                const uint32_t take = c - j0 < 32 ? c - j0 : 32u;
                const bool ok = (uint32_t)lane < take;
                const uint2 pair = make_uint2(qi, ok ? __float_as_uint(__ldg(&pts[f + j0 + lane].w)) : 0u);
                if (SEG) {
                    if (ok && cnt + lane < wlen) p.pairs[wb + cnt + lane] = pair;
                } else {
                    if (ok) buf[fill + lane] = pair;
                    fill += take;
                    __syncwarp();
                    if (fill > WBUF - 32) flush();
                }
                cnt += take;
            }
            if (SEG && cnt > wlen) seg_bad = true;
        };
        auto visit = [&](bool ok, uint32_t level, uint32_t e) {
            bool inside = false;
            if (ok) {
                const float4 *b = p.pyr + 2 * (uint64_t)(s_off[level] + e);
                const float4 lo = __ldg(b), hi = __ldg(b + 1);
                ok = !(box_min_key(qx, qy, qz, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z) > r2);
                const float far = box_max_key(qx, qy, qz, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z);
                // (an unbounded box holds a NaN point, which no ball holds)
                inside = ok && level > 1 && far <= r2 && far < INFINITY;
            }
            uint32_t mi = __ballot_sync(0xffffffffu, inside);
            if (mi) {
                uint32_t f = 0, c = 0;
                if (inside) {
                    f = e << (3 * level);
                    c = n - f < 1u << (3 * level) ? n - f : 1u << (3 * level);
                    ok = false;
                }
                if (COUNTS || MODE == MODE_SAMPLE) {
                    const uint32_t sum = __reduce_add_sync(0xffffffffu, c);
                    cnt += sum;
                    if (MODE == MODE_CPUSH) {
                        if (inside) recs[nrec + __popc(mi & lt)] = make_uint4(qi, f, c, 0u);
                        nrec += __popc(mi);
                        covered += sum;
                        __syncwarp();
                        if (nrec > WRECS - 32) flush_recs();
                    }
                } else {
                    for (; mi; mi &= mi - 1) {
                        const int src = __ffs(mi) - 1;
                        copy_run(__shfl_sync(0xffffffffu, f, src), __shfl_sync(0xffffffffu, c, src));
                    }
                }
            }
            const uint32_t mo = __ballot_sync(0xffffffffu, ok), ml = mo & __ballot_sync(0xffffffffu, level == 1);
            const uint32_t at = __popc((level == 1 ? ml : mo & ~ml) & lt);
            if (ok) (level == 1 ? leaf + lq : stack + sp)[at] = level << 28 | e;
            lq += __popc(ml);
            sp += __popc(mo & ~ml);
            __syncwarp();
        };
        // a query with a NaN coordinate has no neighbours (its keys are NaN)
        if (n > 0 && !isnan(qx) && !isnan(qy) && !isnan(qz)) {
            if (n <= 64) {   // no pyramid: every run
                lq = (n + 7) / 8;
                if ((uint32_t)lane < lq) leaf[lane] = lane;
                __syncwarp();
            } else {
                visit((uint32_t)lane <= (n - 1) >> (3 * top), top, lane);
            }
        }
        while (sp | lq) {
            if (lq >= 8 || sp == 0) {
                // up to 8 runs of 8 points, two points a lane
                const uint32_t take = lq < 8 ? lq : 8u;
                lq -= take;
                float4 pt[2];
                bool ok[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t r = 4 * u + (lane >> 3);
                    const uint32_t at = r < take ? (leaf[lq + r] & 0x0FFFFFFFu) * 8 + (lane & 7) : n;
                    ok[u] = at < n;
                    pt[u] = ok[u] ? __ldg(&pts[at]) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const bool hit = ok[u] && exact_key(qx, qy, qz, pt[u].x, pt[u].y, pt[u].z) <= r2;
                    const uint32_t hm = __ballot_sync(0xffffffffu, hit);
                    const uint2 pair = make_uint2(qi, __float_as_uint(pt[u].w));
                    if (SEG) {
                        const uint32_t at = cnt + __popc(hm & lt);
                        if (hit && at < wlen) p.pairs[wb + at] = pair;
                        seg_bad |= hit && at >= wlen;
                    } else if (PUSH) {
                        if (hit) buf[fill + __popc(hm & lt)] = pair;
                        fill += __popc(hm);
                        __syncwarp();
                        if (fill > WBUF - 32) flush();
                    }
                    cnt += __popc(hm);
                }
                __syncwarp();
            } else {
                const uint32_t take = sp < 4 ? sp : 4u;
                sp -= take;
                const uint32_t r = lane >> 3;
                const uint32_t node = r < take ? stack[sp + r] : 2u << 28;
                const uint32_t level = (node >> 28) - 1, e = (node & 0x0FFFFFFFu) * 8 + (lane & 7);
                __syncwarp();
                visit(r < take && e <= (n - 1) >> (3 * level), level, e);
            }
        }
        if (COUNTS && lane == 0) p.counts[qi] = cnt;
        if (COUNTS) most = cnt > most ? cnt : most;
        if (MODE == MODE_SAMPLE) {
            most = cnt > most ? cnt : most;
            if (lane == 0) atomicAdd(p.sample_sum, cnt < 64 * SAMPLE ? cnt : (uint32_t)(64 * SAMPLE));
        }
        // a segment left short or overrun: the queries changed since the count
        if (SEG && (seg_bad || cnt != wlen)) atomicOr(p.err, DEVERR_MISMATCH);
    }
    if (PUSH) flush();
    if (MODE == MODE_CPUSH) {
        flush_recs();
        if (lane == 0 && covered) atomicAdd(&p.cursor[2], covered);
    }
    if ((COUNTS || MODE == MODE_SAMPLE) && lane == 0 && most) atomicMax(p.most, most);
}

constexpr int SHORT_DEPTH = 12;  // stack entries per thread in shared memory
constexpr int STACK_DEPTH = 104; // >= maximal tree depth

__device__ __forceinline__ void load_node_r(const BvhNode *__restrict__ s_top,
                                            const BvhNode *__restrict__ g, uint32_t w, float4 &a,
                                            float4 &b, float4 &c, uint4 &d) {
    if (w & CHILD_TOP) {
        const BvhNode &n = s_top[w & CHILD_INDEX];
        a = n.a; b = n.b; c = n.c; d = n.d;
    } else {
        const BvhNode *n = g + (w & CHILD_INDEX);
        a = __ldg(&n->a); b = __ldg(&n->b); c = __ldg(&n->c); d = __ldg(&n->d);
    }
}

// Fields of the per-lane work a traversal step stages for the warp (one
// 32-word row per field, so lanes reading different owners hit different
// banks): the counts need the first, the fills the others too.
enum : int { F_QX = 0, F_QY, F_QZ, F_QI, F_F0, F_C0, F_F1, F_DONE, F_COUNT,
             F_T = F_COUNT, F_G0, F_N0, F_G1, F_PUSH, F_WLEN = F_PUSH, F_WBLO, F_WBHI, F_SEG };
constexpr uint32_t BIG_SUB = 32;  // contained subtrees of this size or more: copied by the warp

// A thread per query over the binary tree: where many queries have few hits
// each, its tighter boxes and 32 walks a warp need less than half the
// instructions of range_kernel (launch_pass says when).  Threads of a warp
// advance their own traversals one node per iteration of a warp-converged
// loop; a stack entry carries the node and the first sorted point below it.  A
// child whose whole box lies inside the ball contributes its points without a
// test: their number in the counts (MODE_CPUSH: a record), their ids in the
// fills, by the whole warp for BIG_SUB points and more.  After each step the
// lanes' other work, points of the leaves that straddle the sphere and (fills)
// of small contained subtrees, is flattened over the warp by a prefix sum and
// handled 32 points at a time: a lane finds its candidate's owner by a binary
// search over the prefix (shuffles) and reads the owner's query and ranges
// from shared memory.  MODE_SEG writes an owner's hits at the next slots of
// its segment and checks that the query fills it exactly; the pushing modes
// compact them into the warp's staging buffer.
template <int MODE>
__global__ void __launch_bounds__(RBLOCK, MODE == MODE_COUNT ? 10 : 8) range_thread_kernel(const RangeArgs p) {
    constexpr bool PUSH = MODE == MODE_PUSH || MODE == MODE_CPUSH;   // through warp staging
    constexpr bool COUNTS = MODE == MODE_COUNT || MODE == MODE_CPUSH;
    constexpr bool SEG = MODE == MODE_SEG, FILL = !COUNTS;
    constexpr int NF = SEG ? F_SEG : FILL ? F_PUSH : F_COUNT;
    if (warp_walks<MODE>(p.ix.hdr, p.nq, p.small_leaves)) return;
    __shared__ BvhNode s_top[TOP_MAX];
    __shared__ uint2 s_stack[SHORT_DEPTH][RBLOCK];
    __shared__ uint2 s_buf[PUSH ? RWARPS : 1][PUSH ? WBUF : 1];
    __shared__ uint32_t s_work[RWARPS][NF][32];
    const IndexHeader *h = p.ix.hdr;
    const uint32_t ntop = h->n_top;
    for (uint32_t i = threadIdx.x; i < ntop; i += RBLOCK) s_top[i] = p.ix.top[i];
    __syncthreads();
    const uint32_t root = h->root, root_count = h->root_count;
    const float4 *__restrict__ pts = p.ix.pts;
    const BvhNode *__restrict__ gn = p.ix.nodes;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const float r2 = p.r2;
    const uint32_t visit_cap = 2u * h->n_internal + 4u;
    uint2 l_stack[STACK_DEPTH - SHORT_DEPTH];
    uint2 *buf = s_buf[PUSH ? warp : 0];
    uint32_t (*W)[32] = s_work[warp];
    uint32_t fill = 0, most = 0;
    auto flush = [&]() {
        if (!PUSH || fill == 0) return;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(p.cursor, (unsigned long long)fill);
        base = __shfl_sync(0xffffffffu, base, 0);
        __syncwarp();
        for (uint32_t j = lane; j < fill; j += 32)
            if (base + j < p.capacity) p.pairs[base + j] = buf[j];
        if (MODE == MODE_PUSH && lane == 0 && base + fill > p.capacity) atomicOr(p.err, DEVERR_OVERFLOW);
        __syncwarp();
        fill = 0;
    };
    const uint64_t stride = (uint64_t)gridDim.x * RBLOCK;
    for (uint64_t tb = (uint64_t)blockIdx.x * RBLOCK + warp * 32; tb < p.nq; tb += stride) {
        const uint64_t t = tb + lane;
        const bool have = t < p.nq;
        uint64_t qi = 0;
        float qx = 0.f, qy = 0.f, qz = 0.f;
        if (have) {
            qi = p.perm ? p.perm[t] : t;
            qx = p.q[3 * qi]; qy = p.q[3 * qi + 1]; qz = p.q[3 * qi + 2];
        }
        __syncwarp();   // the previous batch's readers of W are done
        W[F_QX][lane] = __float_as_uint(qx);
        W[F_QY][lane] = __float_as_uint(qy);
        W[F_QZ][lane] = __float_as_uint(qz);
        W[F_QI][lane] = (uint32_t)qi;
        W[F_DONE][lane] = 0;
        if (SEG) {   // this query's segment of the pair buffer
            uint64_t wb = 0, wend = 0;
            if (have) {
                wb = p.offsets[qi];
                wend = qi + 1 < p.nq ? p.offsets[qi + 1] : p.total;
            }
            W[F_WLEN][lane] = (uint32_t)(wend - wb);
            W[F_WBLO][lane] = (uint32_t)wb;
            W[F_WBHI][lane] = (uint32_t)(wb >> 32);
        }
        bool seg_bad = false;
        // a query with a NaN coordinate has no neighbours (its keys are NaN)
        const bool live = have && !isnan(qx) && !isnan(qy) && !isnan(qz);
        uint32_t node = (live && root != CHILD_NONE) ? root : CHILD_NONE;
        uint32_t first = 0;   // first sorted point below `node`
        int sp = 0;
        uint32_t cnt = 0;     // points of contained subtrees
        uint32_t visits = 0;
        while (__any_sync(0xffffffffu, node != CHILD_NONE)) {
            if (node != CHILD_NONE && ++visits > visit_cap) {   // broken tree: give up
                atomicOr(p.err, DEVERR_STACK);
                node = CHILD_NONE;
                sp = 0;
            }
            uint32_t f0 = 0, c0 = 0, f1 = 0, c1 = 0;   // leaves to test
            uint32_t g0 = 0, n0 = 0, g1 = 0, n1 = 0;   // subtrees inside the ball
            if (node != CHILD_NONE) {
                uint32_t next = CHILD_NONE, next_first = 0;
                if (node & CHILD_LEAF) {
                    f0 = node & CHILD_INDEX;
                    c0 = root_count;
                } else {
                    float4 a, b, c;
                    uint4 d;
                    load_node_r(s_top, gn, node, a, b, c, d);
                    const uint32_t fl = first, fr = first + d.z;
                    bool v0 = !(box_min_key(qx, qy, qz, a.x, a.y, a.z, a.w, b.x, b.y) > r2);
                    bool v1 = !(box_min_key(qx, qy, qz, b.z, b.w, c.x, c.y, c.z, c.w) > r2);
                    const float far0 = box_max_key(qx, qy, qz, a.x, a.y, a.z, a.w, b.x, b.y);
                    const float far1 = box_max_key(qx, qy, qz, b.z, b.w, c.x, c.y, c.z, c.w);
                    // (an unbounded box holds a NaN point, as in range_kernel)
                    if (v0 && far0 <= r2 && far0 < INFINITY) {
                        g0 = fl; n0 = d.z; v0 = false;
                    }
                    if (v1 && far1 <= r2 && far1 < INFINITY) {
                        g1 = fr; n1 = d.w; v1 = false;
                    }
                    if (v0 && (d.x & CHILD_LEAF)) { f0 = fl; c0 = d.z; v0 = false; }
                    if (v1 && (d.y & CHILD_LEAF)) {
                        if (c0) { f1 = fr; c1 = d.w; }
                        else { f0 = fr; c0 = d.w; }
                        v1 = false;
                    }
                    if (v0 && v1) {
                        next = d.x;
                        next_first = fl;
                        const uint2 e = make_uint2(d.y, fr);
                        if (sp < SHORT_DEPTH) s_stack[sp++][threadIdx.x] = e;
                        else if (sp < STACK_DEPTH) { l_stack[sp - SHORT_DEPTH] = e; ++sp; }
                        else atomicOr(p.err, DEVERR_STACK);
                    } else if (v0) {
                        next = d.x;
                        next_first = fl;
                    } else if (v1) {
                        next = d.y;
                        next_first = fr;
                    }
                }
                if (next == CHILD_NONE && sp > 0) {
                    --sp;
                    const uint2 e = sp < SHORT_DEPTH ? s_stack[sp][threadIdx.x] : l_stack[sp - SHORT_DEPTH];
                    next = e.x;
                    next_first = e.y;
                }
                node = next;
                first = next_first;
            }
            if (COUNTS) cnt += n0 + n1;
            if (MODE == MODE_CPUSH) {
                const uint32_t rm0 = __ballot_sync(0xffffffffu, n0 != 0);
                const uint32_t rm1 = __ballot_sync(0xffffffffu, n1 != 0);
                const uint32_t nr = __popc(rm0) + __popc(rm1);
                if (nr) {
                    uint32_t covered = n0 + n1;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) covered += __shfl_xor_sync(0xffffffffu, covered, o);
                    unsigned long long base = 0;
                    if (lane == 0) {
                        base = atomicAdd(&p.cursor[1], (unsigned long long)nr);
                        atomicAdd(&p.cursor[2], (unsigned long long)covered);
                    }
                    base = __shfl_sync(0xffffffffu, base, 0);
                    // slots: the lanes' first records in lane order, then their second ones
                    uint64_t r = base + __popc(rm0 & lt);
                    if (n0 && r < p.rec_cap) p.recs[r] = make_uint4((uint32_t)qi, g0, n0, 0u);
                    r = base + __popc(rm0) + __popc(rm1 & lt);
                    if (n1 && r < p.rec_cap) p.recs[r] = make_uint4((uint32_t)qi, g1, n1, 0u);
                }
            }
            if (FILL) {
                // contained subtrees of BIG_SUB points or more: their
                // contiguous ids, one pair per lane
                const uint32_t b0 = n0 >= BIG_SUB ? n0 : 0u, b1 = n1 >= BIG_SUB ? n1 : 0u;
                if (b0) n0 = 0;
                if (b1) n1 = 0;
                for (uint32_t m = __ballot_sync(0xffffffffu, (b0 | b1) != 0); m; m &= m - 1) {
                    const int src = __ffs(m) - 1;
                    const uint32_t sq = W[F_QI][src];
                    for (int r = 0; r < 2; ++r) {
                        const uint32_t gs = __shfl_sync(0xffffffffu, r ? g1 : g0, src);
                        const uint32_t ns = __shfl_sync(0xffffffffu, r ? b1 : b0, src);
                        if (ns == 0) continue;
                        if (SEG) {
                            const uint32_t done = W[F_DONE][src];
                            if ((uint64_t)done + ns <= W[F_WLEN][src]) {
                                const uint64_t dst = ((uint64_t)W[F_WBHI][src] << 32 | W[F_WBLO][src]) + done;
                                for (uint32_t k = lane; k < ns; k += 32)
                                    p.pairs[dst + k] = make_uint2(sq, __float_as_uint(__ldg(&pts[gs + k].w)));
                            } else {
                                seg_bad = true;
                            }
                            __syncwarp();
                            if (lane == src) W[F_DONE][src] = done + ns;
                            __syncwarp();
                        } else {
                            for (uint32_t k = 0; k < ns; k += 32) {
                                const uint32_t take = ns - k < 32u ? ns - k : 32u;
                                if ((uint32_t)lane < take)
                                    buf[fill + lane] = make_uint2(sq, __float_as_uint(__ldg(&pts[gs + k + lane].w)));
                                fill += take;
                                __syncwarp();
                                if (fill > WBUF - 32) flush();
                            }
                        }
                    }
                }
            }
            // flatten this step's candidates over the warp
            const uint32_t tl = c0 + c1, items = tl + (FILL ? n0 + n1 : 0u);
            uint32_t incl = items;
#pragma unroll
            for (int dlt = 1; dlt < 32; dlt <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, dlt);
                if (lane >= dlt) incl += v;
            }
            const uint32_t excl = incl - items;
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            if (total == 0) continue;
            W[F_F0][lane] = f0;
            W[F_C0][lane] = c0;
            W[F_F1][lane] = f1;
            if (FILL) {
                W[F_T][lane] = tl;
                W[F_G0][lane] = g0;
                W[F_N0][lane] = n0;
                W[F_G1][lane] = g1;
            }
            __syncwarp();
            for (uint32_t base = 0; base < total; base += 32) {
                const uint32_t ci = base + lane;
                const bool valid = ci < total;
                // owner: the last lane whose prefix is <= ci
                int o = 0;
#pragma unroll
                for (int step = 16; step >= 1; step >>= 1) {
                    const uint32_t pv = __shfl_sync(0xffffffffu, excl, o + step);
                    if (pv <= ci) o += step;
                }
                const uint32_t oexcl = __shfl_sync(0xffffffffu, excl, o);
                const uint32_t oitems = __shfl_sync(0xffffffffu, items, o);
                bool hit = false;
                uint32_t id = 0;
                if (FILL && valid && ci - oexcl >= W[F_T][o]) {   // a point of a contained subtree
                    const uint32_t j = ci - oexcl - W[F_T][o], on0 = W[F_N0][o];
                    id = __float_as_uint(__ldg(&pts[j < on0 ? W[F_G0][o] + j : W[F_G1][o] + (j - on0)].w));
                    hit = true;
                } else if (valid) {
                    const uint32_t j = ci - oexcl, oc0 = W[F_C0][o];
                    const uint32_t pi = j < oc0 ? W[F_F0][o] + j : W[F_F1][o] + (j - oc0);
                    const float4 pt = __ldg(&pts[pi]);
                    hit = exact_key(__uint_as_float(W[F_QX][o]), __uint_as_float(W[F_QY][o]),
                                    __uint_as_float(W[F_QZ][o]), pt.x, pt.y, pt.z) <= r2;
                    id = __float_as_uint(pt.w);
                }
                const uint32_t hm = __ballot_sync(0xffffffffu, hit);
                // this owner's lanes in the batch: [rs, re]
                const int rs = oexcl > base ? (int)(oexcl - base) : 0;
                const uint32_t rend = oexcl + oitems - base;
                const int re = (int)(rend < 32u ? rend : 32u) - 1;
                const uint32_t below_rs = (1u << rs) - 1u;
                const uint32_t upto_re = re >= 31 ? 0xffffffffu : ((1u << (re + 1)) - 1u);
                if (PUSH && hm) {
                    if (hit) buf[fill + __popc(hm & lt)] = make_uint2(W[F_QI][o], id);
                    fill += __popc(hm);
                    if (fill > WBUF - 32) flush();
                }
                const uint32_t done = SEG ? W[F_DONE][o] : 0u;
                if (SEG) {
                    const uint32_t at = done + __popc(hm & lt & ~below_rs);
                    if (hit && at < W[F_WLEN][o])
                        p.pairs[((uint64_t)W[F_WBHI][o] << 32 | W[F_WBLO][o]) + at] = make_uint2(W[F_QI][o], id);
                    seg_bad |= hit && at >= W[F_WLEN][o];
                    __syncwarp();
                }
                if (valid && lane == re)
                    W[F_DONE][o] = (SEG ? done : W[F_DONE][o]) + __popc(hm & upto_re & ~below_rs);
                __syncwarp();
            }
        }
        __syncwarp();
        // a segment left short or overrun: the queries changed since the count
        if (SEG && (seg_bad || (have && W[F_DONE][lane] != W[F_WLEN][lane]))) atomicOr(p.err, DEVERR_MISMATCH);
        if (COUNTS && have) {
            const uint32_t c = cnt + W[F_DONE][lane];
            p.counts[qi] = c;
            most = c > most ? c : most;
        }
    }
    flush();
    if (COUNTS) {
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0 && most) atomicMax(p.most, most);
    }
}

// Order-free 64-bit fingerprint of a query array (wrapping sum of mixed
// per-query words, splitmix64 finalizer), added into *out.
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x ^= x >> 30;
    x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27;
    x *= 0x94d049bb133111ebull;
    x ^= x >> 31;
    return x;
}

__global__ void __launch_bounds__(256) query_fingerprint_kernel(const float *__restrict__ q,
                                                                uint64_t nq,
                                                                unsigned long long *out) {
    uint64_t acc = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < nq;
         i += (uint64_t)gridDim.x * 256) {
        const uint64_t xy = (uint64_t)__float_as_uint(q[3 * i]) |
                            ((uint64_t)__float_as_uint(q[3 * i + 1]) << 32);
        const uint64_t z = __float_as_uint(q[3 * i + 2]);
        acc += mix64(xy ^ mix64(z + (i + 1) * 0x9e3779b97f4a7c15ull));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, (unsigned long long)acc);
}

// The count's records into their queries' segments: LANES lanes per record,
// its slots reserved with one atomic, the ids read from the sorted points.
// Skipped like range_scatter_kernel.  The warp count's records hold 64 points
// or more and take a warp each; the thread count's are mostly leaves, of which
// a warp takes four (LANES = 8): 1.8M uniform points, 400,000 queries, 50 hits
// a query, count and fill 3.01 ms with a warp each, 2.70 with 8 lanes.
template <int LANES>
__global__ void __launch_bounds__(256) range_expand_kernel(const uint4 *__restrict__ recs,
                                                           uint64_t n_recs,
                                                           const uint64_t *__restrict__ offsets,
                                                           uint32_t *__restrict__ qcur,
                                                           const float4 *__restrict__ pts,
                                                           uint2 *__restrict__ out,
                                                           const IndexHeader *h) {
    if (h->qfp[0] != h->qfp[1]) return;
    constexpr int EACH = 32 / LANES;   // records of a warp
    const int lane = threadIdx.x & 31, sub = lane % LANES;
    for (uint64_t wb = (((uint64_t)blockIdx.x * 256 + threadIdx.x) >> 5) * EACH; wb < n_recs;
         wb += (((uint64_t)gridDim.x * 256) >> 5) * EACH) {
        const uint64_t w = wb + lane / LANES;
        const bool ok = w < n_recs;
        const uint4 rc = ok ? recs[w] : make_uint4(0u, 0u, 0u, 0u);
        uint32_t base = 0;
        if (ok && sub == 0) base = atomicAdd(&qcur[rc.x], rc.z);
        base = __shfl_sync(0xffffffffu, base, lane - sub);
        if (ok) {
            const uint64_t dst = offsets[rc.x] + base;
            for (uint32_t j = sub; j < rc.z; j += LANES)
                out[dst + j] = make_uint2(rc.x, __float_as_uint(__ldg(&pts[rc.y + j].w)));
        }
    }
}

// The count's pairs into their queries' segments (order within a segment
// unspecified), unless the queries changed since the count (fingerprints
// differ), in which case the segment fill that follows runs instead.  A
// query's pairs were pushed together, so the lanes of a warp mostly share
// queries: one atomic per query and warp reserves their slots.
__global__ void __launch_bounds__(256) range_scatter_kernel(const uint2 *__restrict__ spec,
                                                            uint64_t n_pairs,
                                                            const uint64_t *__restrict__ offsets,
                                                            uint32_t *__restrict__ qcur,
                                                            uint2 *__restrict__ out,
                                                            const IndexHeader *h) {
    if (h->qfp[0] != h->qfp[1]) return;
    const int lane = threadIdx.x & 31;
    uint32_t lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    for (uint64_t w = (uint64_t)blockIdx.x * 256 + (threadIdx.x & ~31u); w < n_pairs;
         w += (uint64_t)gridDim.x * 256) {
        const uint64_t t = w + lane;
        const bool ok = t < n_pairs;
        const uint2 pr = ok ? spec[t] : make_uint2(0xFFFFFFFFu, 0u);
        const uint32_t peers = __match_any_sync(0xffffffffu, pr.x);
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if (ok && lane == leader) base = atomicAdd(&qcur[pr.x], (uint32_t)__popc(peers));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (ok) out[offsets[pr.x] + base + __popc(peers & lt)] = pr;
    }
}

// Sorts every query's segment of the pair buffer by id.  A warp takes
// segments of up to WSORT pairs, ids in registers (element u 32 + lane in
// register u), by a bitonic sort in its all-ascending form; longer ones are
// listed for a block each (segment_sort_block_kernel).
constexpr uint32_t WSORT = 256;

// Compare-exchange of every register's 32 ids with the lane at xor distance
// `mask`.
template <int E>
__device__ __forceinline__ void id_lanes(uint32_t (&v)[E], int mask, bool lower) {
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const uint32_t o = __shfl_xor_sync(0xffffffffu, v[u], mask);
        v[u] = lower ? min(v[u], o) : max(v[u], o);
    }
}
// The exchanges at distances 16 E down to 1 of a merge.
template <int E>
__device__ __forceinline__ void id_merge(uint32_t (&v)[E], int from) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = E / 2; j > 0; j >>= 1)
        if (j <= from)
#pragma unroll
            for (int u = 0; u < E; ++u) {
                const int o = u ^ j;
                if (o > u) {
                    const uint32_t a = v[u], b = v[o];
                    v[u] = min(a, b);
                    v[o] = max(a, b);
                }
            }
#pragma unroll 1
    for (int j = 16; j > 0; j >>= 1) id_lanes(v, j, (lane & j) == 0);
}
template <int E>
__device__ __forceinline__ void id_sort(uint32_t (&v)[E]) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int kb = 2; kb <= 32; kb <<= 1) {
        int mask = kb - 1;
#pragma unroll 1
        for (int j = kb >> 1; j > 0; j >>= 1) {
            id_lanes(v, mask, (lane & j) == 0);
            mask = j >> 1;
        }
    }
#pragma unroll
    for (int m = 2; m <= E; m <<= 1) {   // merges of runs of m / 2 registers
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int o = u ^ (m - 1);
            if (o > u) {
                const uint32_t a = v[u], b = __shfl_xor_sync(0xffffffffu, v[o], 31);
                v[u] = min(a, b);
                v[o] = __shfl_xor_sync(0xffffffffu, max(a, b), 31);
            }
        }
        id_merge(v, m >> 2);
    }
}
template <int E>
__device__ __forceinline__ void segment_sort_warp(uint2 *__restrict__ seg, uint32_t c, uint32_t qi) {
    const int lane = threadIdx.x & 31;
    uint32_t v[E];
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const uint32_t j = u * 32 + lane;
        v[u] = j < c ? seg[j].y : 0xFFFFFFFFu;
    }
    id_sort(v);
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const uint32_t j = u * 32 + lane;
        if (j < c) seg[j] = make_uint2(qi, v[u]);
    }
}

__global__ void __launch_bounds__(256) segment_sort_kernel(uint2 *__restrict__ pairs,
                                                           const uint64_t *__restrict__ offsets, uint64_t nq,
                                                           uint64_t total, uint32_t *__restrict__ longer) {
    const int lane = threadIdx.x & 31;
    for (uint64_t q = ((uint64_t)blockIdx.x * 256 + threadIdx.x) >> 5; q < nq; q += ((uint64_t)gridDim.x * 256) >> 5) {
        const uint64_t b = offsets[q], e = q + 1 < nq ? offsets[q + 1] : total;
        const uint32_t c = (uint32_t)(e - b);
        if (c < 2) continue;
        uint2 *seg = pairs + b;
        if (c <= 32) segment_sort_warp<1>(seg, c, (uint32_t)q);
        else if (c <= 64) segment_sort_warp<2>(seg, c, (uint32_t)q);
        else if (c <= 128) segment_sort_warp<4>(seg, c, (uint32_t)q);
        else if (c <= WSORT) segment_sort_warp<8>(seg, c, (uint32_t)q);
        else if (lane == 0) longer[1 + atomicAdd(longer, 1u)] = (uint32_t)q;
    }
}

// The longer segments, up to BSORT pairs: a block each.  Its warps sort
// chunks of 256 ids in registers; the exchanges of the merges at distance
// 256 and more go through shared memory, the others through registers again.
constexpr uint32_t BSORT = 16384;
constexpr int BSORT_WARPS = 4;
__global__ void __launch_bounds__(BSORT_WARPS * 32) segment_sort_block_kernel(
    uint2 *__restrict__ pairs, const uint64_t *__restrict__ offsets, uint64_t nq, uint64_t total,
    const uint32_t *__restrict__ longer) {
    extern __shared__ uint32_t s_id[];
    constexpr int E = WSORT / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nl = longer[0];
    for (uint32_t k = blockIdx.x; k < nl; k += gridDim.x) {
        const uint32_t q = longer[1 + k];
        const uint64_t b = offsets[q], e = q + 1 < nq ? offsets[q + 1] : total;
        const uint32_t c = (uint32_t)(e - b), n = (c + WSORT - 1) / WSORT * WSORT;   // whole chunks
        uint32_t v[E];
        __syncthreads();   // the previous segment's readers are done
        for (uint32_t at = warp * WSORT; at < n; at += BSORT_WARPS * WSORT) {
#pragma unroll
            for (int u = 0; u < E; ++u) {
                const uint32_t j = at + u * 32 + lane;
                v[u] = j < c ? pairs[b + j].y : 0xFFFFFFFFu;
            }
            id_sort(v);
#pragma unroll
            for (int u = 0; u < E; ++u) s_id[at + u * 32 + lane] = v[u];
        }
        __syncthreads();
        // (ids past the whole chunks would be the largest: they never move)
        for (uint32_t kb = 2 * WSORT; kb < 2 * n; kb <<= 1) {
            for (uint32_t j = kb >> 1; j >= WSORT; j >>= 1) {
                for (uint32_t t = threadIdx.x; t < (n + kb - 1) / kb * (kb / 2); t += BSORT_WARPS * 32) {
                    const uint32_t x = t & (j - 1), lo = (t - x) * 2 + x;
                    const uint32_t hi = j == kb >> 1 ? (t - x) * 2 + 2 * j - 1 - x : lo + j;
                    if (hi < n) {
                        const uint32_t u = s_id[lo], w = s_id[hi];
                        if (w < u) {
                            s_id[lo] = w;
                            s_id[hi] = u;
                        }
                    }
                }
                __syncthreads();
            }
            for (uint32_t at = warp * WSORT; at < n; at += BSORT_WARPS * WSORT) {
#pragma unroll
                for (int u = 0; u < E; ++u) v[u] = s_id[at + u * 32 + lane];
                id_merge(v, E / 2);
#pragma unroll
                for (int u = 0; u < E; ++u) s_id[at + u * 32 + lane] = v[u];
            }
            __syncthreads();
        }
        for (uint32_t j = threadIdx.x; j < c; j += BSORT_WARPS * 32) pairs[b + j] = make_uint2(q, s_id[j]);
    }
}

__global__ void pairs_from_keys_kernel(const uint64_t *__restrict__ keys, uint64_t n,
                                       uint2 *__restrict__ out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t k = keys[i];
        out[i] = make_uint2((uint32_t)(k >> 32), (uint32_t)k);
    }
}

__global__ void keys_from_pairs_kernel(const uint2 *__restrict__ pairs, uint64_t n,
                                       uint64_t *__restrict__ keys) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint2 p = pairs[i];
        keys[i] = ((uint64_t)p.x << 32) | p.y;
    }
}

// The points' ids in Morton order.
__global__ void own_order_kernel(const float4 *__restrict__ pts, uint64_t n, uint32_t *__restrict__ perm) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        perm[i] = __float_as_uint(__ldg(&pts[i].w));
}

constexpr uint64_t RANGE_ORDER_MIN = 49152, RANGE_ORDER_POINTS = 2ull << 20;
constexpr uint64_t THREAD_QUERIES = 131072;   // see launch_pass
rtd_status launch_sample(rtd_index *idx, const float *d_q, uint64_t nq, float r, cudaStream_t st);

rtd_status range_args(rtd_index *idx, const float *d_q, uint64_t nq, float r,
                      const rtd_schedule *sched, RangeArgs &a, cudaStream_t st, bool own_points = false) {
    if (!idx || !idx->hdr.ptr) return fail(RTD_ERR_INVALID_ARGUMENT, "index not built");
    if (nq && !d_q) return fail(RTD_ERR_INVALID_ARGUMENT, "NULL queries");
    if (!(r >= 0.0f)) return fail(RTD_ERR_INVALID_ARGUMENT, "radius must be >= 0");
    if (idx->leaf_size > 64) return fail(RTD_ERR_UNSUPPORTED, "leaf_size > 64");
    rtd_schedule def;
    rtd_schedule_default(&def);
    const rtd_schedule &s = sched ? *sched : def;
    const uint32_t *perm = nullptr;
    for (int e = EV_SEARCH0; e <= EV_SEARCH1; ++e) idx->ev_set[e] = false;
    idx->mark(EV_SEARCH0, st);
    idx->mark(EV_SEEDED, st);
    // A thread's walk needs its warp's queries to be neighbours; a warp's
    // gains from the order only as the k-NN warp search does (knn.cu).
    const bool sample = nq >= THREAD_QUERIES;
    const bool wants_order = nq >= THREAD_QUERIES || (nq >= RANGE_ORDER_MIN && idx->n >= RANGE_ORDER_POINTS);
    if (sample) RTD_TRY(launch_sample(idx, d_q, nq, r, st));
    rtd_status os;
    if (own_points) {   // the queries are the index's points: its own order
        os = order_queries(idx, d_q, nq, false, &perm, st);
        if (os == RTD_OK && wants_order) os = idx->qperm.reserve(nq * sizeof(uint32_t));
        if (os == RTD_OK && wants_order) {
            own_order_kernel<<<grid_for(nq, 256, 148 * 8), 256, 0, st>>>(idx->pts.as<float4>(), nq,
                                                                        idx->qperm.as<uint32_t>());
            note_launch();
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) os = cuda_fail(e, "own_order_kernel launch");
            perm = idx->qperm.as<uint32_t>();
        }
    } else {
        os = order_queries(idx, d_q, nq, s.use_morton_lbv && wants_order, &perm, st);
    }
    if (sample) RTD_CUDA(cudaStreamWaitEvent(st, idx->ev_join, 0));   // also on the error path
    RTD_TRY(os);
    idx->mark(EV_ORDERED, st);
    a.ix = view_of(idx);
    a.pyr = idx->pyramid.as<float4>();
    a.q = d_q;
    a.nq = nq;
    a.perm = perm;
    a.r2 = r * r;
    a.counts = nullptr;
    a.most = &idx->hdr.as<IndexHeader>()->most;
    a.pairs = nullptr;
    a.capacity = 0;
    a.cursor = nullptr;
    a.offsets = nullptr;
    a.total = 0;
    a.skip_if_same = 0;
    a.recs = nullptr;
    a.rec_cap = 0;
    a.err = &idx->hdr.as<IndexHeader>()->err;
    return RTD_OK;
}

// Largest buffer kept for the count's own pairs (2^28 pairs, 2 GiB).
constexpr uint64_t RSPEC_MAX = 1ull << 28;

rtd_status query_fingerprint(const float *d_q, uint64_t nq, unsigned long long *out,
                             cudaStream_t st) {
    RTD_CUDA(cudaMemsetAsync(out, 0, sizeof(unsigned long long), st));
    query_fingerprint_kernel<<<grid_for(nq, 256, 148 * 4), 256, 0, st>>>(d_q, nq, out);
    RTD_LAUNCH_CHECK();
    return RTD_OK;
}

template <int MODE>
rtd_status launch_range(RangeArgs &a, cudaStream_t st) {
    // a persistent grid: staging outlives a query
    const size_t smem = RWARPS * range_warp_bytes(MODE, a.ix.n);
    range_kernel<MODE><<<grid_for(a.nq, RWARPS, NUM_SMS_HINT * 10), RBLOCK, smem, st>>>(a);
    RTD_LAUNCH_CHECK();
    return RTD_OK;
}

// Which kernel counts or fills.  A thread per query costs less where the hits
// are few: the warp kernel takes about 1.8 ns a query besides the hits.  The
// warp kernel is ahead from some 64 hits a query on, and earlier where a few
// queries find most: a warp of 32 threads takes as long as its longest walk,
// some 1.1 us for each of that query's hits, and the last such warp ends the
// launch, which shows with fewer than 500 to 1,000 queries for every hit of
// the largest query (1,024 for the largest of a sample, which misses the top).
// Pushing counts over leaves of 4 points change over earlier: a record for
// every such leaf inside the ball takes two reservations a step of a warp, and
// these queue up on the cursors; the line grows as the root of the number of
// queries.  Measured, thread / warp, us; 1.5M points, 400,000 queries:
//                             count  segment fill  pushing count, leaves of 4 / 12
//   uniform     4 hits    267 / 596     297 / 646     373 / 633     317 / 637
//               16        424 / 725     490 / 796    1016 / 787     518 / 784
//               50        677 / 905    794 / 1013   2213 / 1008    860 / 1000
//               62        750 / 960    893 / 1079   2554 / 1074    996 / 1071
//   clustered   8         395 / 750     512 / 802     625 / 803     512 / 797
//               24        724 / 813    1072 / 884    1302 / 884     995 / 879
//               50       1036 / 891    1672 / 975    2064 / 985    1429 / 973
//   the points as queries, 24 hits:
//   uniform             1416 / 2787   1757 / 3106   4556 / 3048   1855 / 3037
//   clustered           1208 / 2930   1621 / 3213   3411 / 3181   1572 / 3170
//   140,000 queries:
//   uniform     8         157 / 237     165 / 260     297 / 262     217 / 264
//               50        269 / 335     313 / 375     876 / 379     450 / 377
//   clustered   4         254 / 260     303 / 276     350 / 282     315 / 281
// The queries have to be in order for the threads' walks (50 us), before the
// sample can say which kernel runs, which decides below THREAD_QUERIES: count
// and first fill of 100,000 queries on 1.8M uniform points with it, 1 hit 200
// / 280 us, 8 hits 330 / 370, and count and fill with pushes, 8 hits 330 (in
// order, then a warp a query) / 270; 50,000 queries, 1 hit 180 / 163, 8 hits
// 289 / 205.  The sample runs on the side stream beside the ordering.
template <int MODE>
rtd_status launch_pass(const rtd_index *idx, RangeArgs &a, cudaStream_t st) {
    a.small_leaves = idx->leaf_size < 6;
    a.by_sample = a.nq >= THREAD_QUERIES;
    if (a.by_sample) {
        range_thread_kernel<MODE><<<grid_for(a.nq, RBLOCK, 1 << 20), RBLOCK, 0, st>>>(a);
        RTD_LAUNCH_CHECK();
    }
    return launch_range<MODE>(a, st);
}

// Starts the sample of launch_pass on the side stream.
rtd_status launch_sample(rtd_index *idx, const float *d_q, uint64_t nq, float r, cudaStream_t st) {
    RTD_TRY(ensure_side_stream(idx));
    cudaStream_t side = idx->side_stream;
    IndexHeader *h = idx->hdr.as<IndexHeader>();
    RTD_CUDA(cudaEventRecord(idx->ev_fork, st));
    RTD_CUDA(cudaStreamWaitEvent(side, idx->ev_fork, 0));
    RangeArgs a = {};
    a.ix = view_of(idx);
    a.pyr = idx->pyramid.as<float4>();
    a.q = d_q;
    a.nq = SAMPLE;
    a.sample_step = nq / SAMPLE;
    a.r2 = r * r;
    a.sample_sum = &h->sample_sum;
    a.most = &h->sample_most;
    a.err = &h->err;
    const cudaError_t me = cudaMemsetAsync(&h->sample_sum, 0, 2 * sizeof(uint32_t), side);
    const rtd_status s = launch_range<MODE_SAMPLE>(a, side);
    RTD_CUDA(cudaEventRecord(idx->ev_join, side));
    if (me != cudaSuccess || s != RTD_OK) {
        RTD_CUDA(cudaStreamWaitEvent(st, idx->ev_join, 0));
        return me != cudaSuccess ? cuda_fail(me, "cudaMemsetAsync") : s;
    }
    return RTD_OK;
}

}  // namespace

rtd_status check_index_errors(rtd_index *idx, cudaStream_t st);

// own_points: the queries are the points the index was built over.
rtd_status range_count(rtd_index *idx, const float *d_q, uint64_t nq, float r,
                       const rtd_schedule *s, uint32_t *d_counts, uint64_t *h_total,
                       cudaStream_t st, bool own_points) {
    if (!d_counts && nq) return fail(RTD_ERR_INVALID_ARGUMENT, "NULL counts");
    RangeArgs a = {};
    RTD_TRY(range_args(idx, d_q, nq, r, s, a, st, own_points));
    a.counts = d_counts;
    IndexHeader *h = idx->hdr.as<IndexHeader>();
    // With a buffer left by an earlier count, this count also pushes its
    // pairs there (and fingerprints the queries), so that a fill of the same
    // queries only scatters them into their segments.
    const bool spec = nq > 0 && idx->rspec_cap > 0;
    RTD_CUDA(cudaMemsetAsync(h->rcur, 0, offsetof(IndexHeader, most) + sizeof(uint32_t) - offsetof(IndexHeader, rcur), st));
    if (nq) {
        if (spec) {
            a.pairs = idx->rspec.as<uint2>();
            a.capacity = idx->rspec_cap;
            a.cursor = h->rcur;
            a.recs = idx->rrec.as<uint4>();
            a.rec_cap = idx->rrec_cap;
            RTD_TRY(query_fingerprint(d_q, nq, &h->qfp[0], st));
            RTD_TRY(launch_pass<MODE_CPUSH>(idx, a, st));
        } else {
            RTD_TRY(launch_pass<MODE_COUNT>(idx, a, st));
        }
        idx->mark(EV_SEARCH1, st);
        RTD_TRY(idx->roffsets.reserve(nq * sizeof(uint64_t)));
        RTD_TRY(exclusive_scan_u32(d_counts, idx->roffsets.as<uint64_t>(), nq, &h->total,
                                   idx->scan, &h->err, st));
    } else {
        RTD_CUDA(cudaMemsetAsync(&h->total, 0, sizeof(uint64_t), st));
    }
    // everything the host needs in one copy: total, cursors, largest count, errors
    IndexHeader now;
    RTD_CUDA(cudaMemcpyAsync(&now, h, sizeof(now), cudaMemcpyDeviceToHost, st));
    RTD_CUDA(cudaStreamSynchronize(st));
    if (now.err) {
        RTD_CUDA(cudaMemsetAsync(&h->err, 0, sizeof(uint32_t), st));
        return status_from_deverr(now.err);
    }
    const uint64_t total = now.total;
    const unsigned long long *cur = now.rcur;
    const uint32_t most = now.most;
    if (h_total) *h_total = total;
    const bool spec_ok = spec && cur[0] + cur[2] == total && cur[0] <= idx->rspec_cap &&
                         cur[1] <= idx->rrec_cap;
    if (!spec_ok && total > 0 && total < RSPEC_MAX) {
        // room for the next count's pairs and records (grown only; a
        // record covers at least one pair)
        uint64_t want = total + total / 8 + 4096;
        if (want > RSPEC_MAX) want = RSPEC_MAX;
        if (want > idx->rspec_cap) {
            RTD_TRY(idx->rspec.reserve(want * sizeof(uint2)));
            idx->rspec_cap = want;
        }
        const uint64_t want_r = (spec ? cur[1] + cur[1] / 8 : want / 4) + 4096;
        if (want_r > idx->rrec_cap) {
            RTD_TRY(idx->rrec.reserve(want_r * sizeof(uint4)));
            idx->rrec_cap = want_r;
        }
    }
    // a fill of the same queries can write straight into per-query segments
    idx->rtoken.valid = true;
    idx->rtoken.q = d_q;
    idx->rtoken.nq = nq;
    idx->rtoken.radius = r;
    idx->rtoken.total = total;
    idx->rtoken.most = most;
    idx->rtoken.perm = a.perm;
    idx->rtoken.spec = spec_ok;
    idx->rtoken.spec_pairs = spec_ok ? cur[0] : 0;
    idx->rtoken.spec_recs = spec_ok ? cur[1] : 0;
    return RTD_OK;
}

rtd_status range_fill(rtd_index *idx, const float *d_q, uint64_t nq, float r,
                      const rtd_schedule *s, uint32_t *d_pairs, uint64_t capacity, int sort_pairs,
                      uint64_t *h_written, cudaStream_t st, bool check) {
    if (capacity && !d_pairs) return fail(RTD_ERR_INVALID_ARGUMENT, "NULL pairs");
    // Segment mode: the last count pass on this index was over these queries
    // at this radius, its offsets and query order are still on the index,
    // and the buffer holds every pair.
    const auto &tk = idx->rtoken;
    const bool seg = tk.valid && tk.q == d_q && tk.nq == nq && tk.radius == r && nq > 0 &&
                     capacity >= tk.total;
    RangeArgs a = {};
    if (seg) {
        if (!idx->hdr.ptr) return fail(RTD_ERR_INVALID_ARGUMENT, "index not built");
        for (int e = EV_SEARCH0; e <= EV_SEARCH1; ++e) idx->ev_set[e] = false;
        idx->mark(EV_SEARCH0, st);
        idx->mark(EV_SEEDED, st);
        idx->mark(EV_ORDERED, st);
        a.ix = view_of(idx);
        a.pyr = idx->pyramid.as<float4>();
        a.q = d_q;
        a.nq = nq;
        a.perm = tk.perm;
        a.r2 = r * r;
        a.counts = nullptr;
        a.most = nullptr;
        a.recs = nullptr;
        a.rec_cap = 0;
        a.cursor = nullptr;
        a.offsets = idx->roffsets.as<uint64_t>();
        a.total = tk.total;
        a.skip_if_same = 0;
        a.err = &idx->hdr.as<IndexHeader>()->err;
    } else {
        RTD_TRY(range_args(idx, d_q, nq, r, s, a, st));
        IndexHeader *h = idx->hdr.as<IndexHeader>();
        RTD_CUDA(cudaMemsetAsync(h->rcur, 0, sizeof(unsigned long long), st));
        a.cursor = h->rcur;
    }
    a.pairs = reinterpret_cast<uint2 *>(d_pairs);
    a.capacity = capacity;
    if (seg && tk.spec) {
        // the count's own pairs, scattered into the segments; the segment
        // fill runs only if the queries changed since the count
        IndexHeader *h = idx->hdr.as<IndexHeader>();
        RTD_TRY(query_fingerprint(d_q, nq, &h->qfp[1], st));
        RTD_TRY(idx->rqcur.reserve((nq + 1) * sizeof(uint32_t)));
        RTD_CUDA(cudaMemsetAsync(idx->rqcur.ptr, 0, nq * sizeof(uint32_t), st));
        if (tk.spec_pairs) {
            range_scatter_kernel<<<grid_for(tk.spec_pairs, 256, 148 * 16), 256, 0, st>>>(
                idx->rspec.as<uint2>(), tk.spec_pairs, a.offsets, idx->rqcur.as<uint32_t>(), a.pairs, h);
            RTD_LAUNCH_CHECK();
        }
        if (tk.spec_recs) {
            if (tk.total - tk.spec_pairs >= 64 * tk.spec_recs)
                range_expand_kernel<32><<<grid_for(tk.spec_recs * 32, 256, 148 * 16), 256, 0, st>>>(
                    idx->rrec.as<uint4>(), tk.spec_recs, a.offsets, idx->rqcur.as<uint32_t>(), a.ix.pts, a.pairs, h);
            else
                range_expand_kernel<8><<<grid_for(tk.spec_recs * 8, 256, 148 * 16), 256, 0, st>>>(
                    idx->rrec.as<uint4>(), tk.spec_recs, a.offsets, idx->rqcur.as<uint32_t>(), a.ix.pts, a.pairs, h);
            RTD_LAUNCH_CHECK();
        }
        a.skip_if_same = 1;
        RTD_TRY(launch_range<MODE_SEG>(a, st));
        idx->mark(EV_SEARCH1, st);
    } else if (seg) {   // (the count's sample of the queries still stands)
        RTD_TRY(launch_pass<MODE_SEG>(idx, a, st));
        idx->mark(EV_SEARCH1, st);
    } else if (nq) {
        RTD_TRY(launch_pass<MODE_PUSH>(idx, a, st));
        idx->mark(EV_SEARCH1, st);
    }
    unsigned long long total = 0;
    if (seg) {
        total = tk.total;
    } else {
        RTD_CUDA(cudaMemcpyAsync(&total, a.cursor, sizeof(total), cudaMemcpyDeviceToHost, st));
        RTD_CUDA(cudaStreamSynchronize(st));
    }
    if (h_written) *h_written = total;
    if (total > capacity) {
        IndexHeader *h = idx->hdr.as<IndexHeader>();
        RTD_CUDA(cudaMemsetAsync(&h->err, 0, sizeof(uint32_t), st));
        return fail(RTD_ERR_OVERFLOW, "pair buffer smaller than the pair count");
    }
    if (sort_pairs && seg && tk.most <= BSORT) {
        // The pairs are grouped by query: each segment is sorted by itself,
        // the longest in shared memory (19.6M pairs, 50 a query: 0.37 ms;
        // the radix sort of all pairs, which longer segments and unmatched
        // fills still take, 1.73 ms).
        if (tk.most > 1) {
            RTD_TRY(idx->rqcur.reserve((nq + 1) * sizeof(uint32_t)));
            uint32_t *longer = idx->rqcur.as<uint32_t>();
            RTD_CUDA(cudaMemsetAsync(longer, 0, sizeof(uint32_t), st));
            segment_sort_kernel<<<grid_for(nq * 32, 256, 148 * 32), 256, 0, st>>>(a.pairs, a.offsets, nq, total,
                                                                                  longer);
            RTD_LAUNCH_CHECK();
            if (tk.most > WSORT) {
                const uint32_t P = (tk.most + WSORT - 1) / WSORT * WSORT;
                RTD_CUDA(cudaFuncSetAttribute(segment_sort_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)(BSORT * sizeof(uint32_t))));
                segment_sort_block_kernel<<<NUM_SMS_HINT * 16, BSORT_WARPS * 32, P * sizeof(uint32_t), st>>>(
                    a.pairs, a.offsets, nq, total, longer);
                RTD_LAUNCH_CHECK();
            }
        }
    } else if (sort_pairs && total > 1) {
        if (total >= (1ull << 30)) return fail(RTD_ERR_UNSUPPORTED, "sorting >= 2^30 pairs");
        RTD_TRY(idx->rkeys.reserve(total * 8));
        RTD_TRY(idx->rkeys_alt.reserve(total * 8));
        RTD_TRY(idx->rpairs_alt.reserve(total * 8));   // dummy values, ping-pong halves
        uint32_t *v0 = idx->rpairs_alt.as<uint32_t>();
        uint32_t *v1 = v0 + total;
        const int g = grid_for(total, 256, 148 * 8);
        keys_from_pairs_kernel<<<g, 256, 0, st>>>(a.pairs, total, idx->rkeys.as<uint64_t>());
        RTD_LAUNCH_CHECK();
        int qbits = 1;
        while (qbits < 32 && (1ull << qbits) < nq) ++qbits;
        bool in_alt = false;
        IndexHeader *h = idx->hdr.as<IndexHeader>();
        RTD_TRY(radix_sort_pairs<uint64_t>(idx->rkeys.as<uint64_t>(), idx->rkeys_alt.as<uint64_t>(),
                                           v0, v1, true, total, 0, 32 + qbits, idx->sort, &h->err,
                                           st, &in_alt));
        const uint64_t *sk = in_alt ? idx->rkeys_alt.as<uint64_t>() : idx->rkeys.as<uint64_t>();
        pairs_from_keys_kernel<<<g, 256, 0, st>>>(sk, total, a.pairs);
        RTD_LAUNCH_CHECK();
    }
    return check ? check_index_errors(idx, st) : RTD_OK;   // synchronises
}

// ------------------------------------------------------- kNN backward
namespace {
__global__ void __launch_bounds__(256) knn_backward_kernel(const float *__restrict__ q, uint64_t nq,
                                                           const float *__restrict__ pts, uint64_t n, uint32_t k,
                                                           const uint32_t *__restrict__ ids,
                                                           const float *__restrict__ g, float *__restrict__ gq,
                                                           float *__restrict__ gp) {
    const bool pairs = backward_pairs(gp);
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < nq; i += (uint64_t)gridDim.x * 256)
        backward_query(q, pts, n, k, ids + i * k, g + i * k, gq, gp, i, pairs);
}
}  // namespace

rtd_status knn_backward(const float *q, uint64_t nq, const float *pts, uint64_t n, uint32_t k,
                        const uint32_t *ids, const float *g, float *gq, float *gp, cudaStream_t st) {
    if (nq == 0 || k == 0) return RTD_OK;
    if (!q || !pts || !ids || !g) return fail(RTD_ERR_INVALID_ARGUMENT, "NULL input");
    knn_backward_kernel<<<grid_for(nq, 256, 148 * 16), 256, 0, st>>>(q, nq, pts, n, k, ids, g, gq, gp);
    RTD_LAUNCH_CHECK();
    return RTD_OK;
}

}  // namespace rtd
