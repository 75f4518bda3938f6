// bh_ref.cu -- the reference-law Barnes-Hut walk over the octree of
// bh_tree.cu: the intended walk of the reference's OptiX programs
// (gprt-macros/src/lib.rs:760-806), a warp per few neighbouring bodies,
// stackless over next = p + 1 / autorope, every operation rounded
// separately so the forces are bit-identical to the CPU restatement.
//
// Bound by instruction issue: about 45,000 body pairs per body at 1M bodies
// (a reached leaf of up to 128 bodies is always summed), some 70
// instructions a pair, half of them the two correctly rounded operations.
// With a thread per body the lanes of a warp each stood at another node and
// another body of a leaf: 50,000 bodies took 18.6 ms, now 4.1 ms; theta 0.5.
#include <rtdsl.h>

#include "bh.cuh"

namespace rtd {
namespace {

// ----------------------------------------------------- reference law
__device__ __forceinline__ float dot3_rn(float x, float y, float z) {
    float s = __fmul_rn(x, x);
    s = __fadd_rn(s, __fmul_rn(y, y));
    s = __fadd_rn(s, __fmul_rn(z, z));
    return s;
}

// A warp walks the tree once for B consecutive bodies of the flat order
// (neighbours in space).  Every body visits its nodes in pre-order, so the
// warp steps through the nodes in order of the smallest index any of its
// bodies wants next, and the bodies that want it take it together: node and
// body loads are one broadcast, and leaf sums run converged.  Each body has
// R = 32 / B lanes.  With R > 1 its lanes evaluate R bodies of a leaf at
// once, hand the terms over in shared memory, and lane c of the body adds
// component c in the leaf's order, so every sum keeps the sequential order
// of the CPU walk and its bits.  A skipped term is added as +0, which
// changes nothing: a sum that starts at +0 is never -0.
template <int B>
__global__ void __launch_bounds__(128) bh_ref_walk_kernel(const BhView v, float theta, float G,
                                                          float *__restrict__ out) {
    constexpr int R = 32 / B;
    static_assert(R == 1 || R % 4 == 0, "terms are read back four at a time");
    __shared__ float4 s_terms[R > 1 ? 4 : 1][2][3][B][R > 1 ? R / 4 : 1];
    const uint32_t n_nodes = v.hdr->n_nodes;
    const int lane = threadIdx.x & 31, slot = lane % B, sub = lane / B, comp = sub < 2 ? sub : 2;
    auto *terms = s_terms[R > 1 ? threadIdx.x >> 5 : 0];
    const uint64_t warps = (uint64_t)gridDim.x * 4;
    for (uint64_t w = (uint64_t)blockIdx.x * 4 + (threadIdx.x >> 5); w * B < v.n; w += warps) {
        const uint64_t i = w * B + slot;
        const bool have = i < v.n;
        const float4 me = have ? v.fbody[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float px = me.x, py = me.y, pz = me.z;
        const float gm = __fmul_rn(G, me.w);
        float s[R > 1 ? 1 : 3] = {};   // R > 1: this lane's component; else x, y, z
        uint32_t next = have ? 0u : n_nodes;
        while (true) {
            const uint32_t p = __reduce_min_sync(0xffffffffu, next);
            if (p >= n_nodes) break;
            const bool act = next == p;
            const float4 a = __ldg(&v.node_a[p]);
            const uint4 b = __ldg(&v.node_b[p]);
            const float dx = __fsub_rn(a.x, px), dy = __fsub_rn(a.y, py), dz = __fsub_rn(a.z, pz);
            const float dist_sq = dot3_rn(dx, dy, dz);
            const float d = __fsqrt_rn(dist_sq);
            const float tmax = __fadd_rn(fmaxf(1e-6f, __fmul_rn(theta, d)), 1e-5f);
            const bool hit = __uint_as_float(b.w) < tmax;
            if (b.z & BH_LEAF_BIT) {
                const float4 *__restrict__ src = v.fbody + b.y;
                const uint32_t c = b.z & ~BH_LEAF_BIT;
                int buf = 0;
#pragma unroll 2
                for (uint32_t j0 = 0; j0 < c; j0 += R) {
                    const uint32_t j = j0 + sub;
                    float tx = 0.f, ty = 0.f, tz = 0.f;
                    if (j < c && act) {
                        const float4 o = __ldg(&src[j]);
                        const float ex = __fsub_rn(o.x, px), ey = __fsub_rn(o.y, py), ez = __fsub_rn(o.z, pz);
                        const float d2 = dot3_rn(ex, ey, ez);
                        if (d2 > 1e-10f) {
                            const float denom = __fmul_rn(d2, __fsqrt_rn(__fadd_rn(d2, 1e-6f)));
                            const float fm = __fdiv_rn(__fmul_rn(gm, o.w), denom);
                            tx = __fmul_rn(ex, fm);
                            ty = __fmul_rn(ey, fm);
                            tz = __fmul_rn(ez, fm);
                        }
                    }
                    if (R == 1) {
                        s[0] = __fadd_rn(s[0], tx);
                        s[1] = __fadd_rn(s[1], ty);
                        s[2] = __fadd_rn(s[2], tz);
                    } else {
                        // two buffers: a lane may write the next terms while
                        // others still read these
                        reinterpret_cast<float *>(&terms[buf][0][slot])[sub] = tx;
                        reinterpret_cast<float *>(&terms[buf][1][slot])[sub] = ty;
                        reinterpret_cast<float *>(&terms[buf][2][slot])[sub] = tz;
                        __syncwarp();
#pragma unroll
                        for (int r = 0; r < R / 4; ++r) {
                            const float4 t = terms[buf][comp][slot][r];
                            s[0] = __fadd_rn(s[0], t.x);
                            s[0] = __fadd_rn(s[0], t.y);
                            s[0] = __fadd_rn(s[0], t.z);
                            s[0] = __fadd_rn(s[0], t.w);
                        }
                        buf ^= 1;
                    }
                }
                if (R > 1) __syncwarp();
                if (act) next = hit ? b.x : p + 1;
            } else if (act) {
                if (hit) {
                    if (dist_sq > 1e-10f) {
                        const float denom = __fmul_rn(dist_sq, __fsqrt_rn(__fadd_rn(dist_sq, 1e-6f)));
                        const float fm = __fdiv_rn(__fmul_rn(gm, a.w), denom);
                        if (R == 1) {
                            s[0] = __fadd_rn(s[0], __fmul_rn(dx, fm));
                            s[1] = __fadd_rn(s[1], __fmul_rn(dy, fm));
                            s[2] = __fadd_rn(s[2], __fmul_rn(dz, fm));
                        } else {
                            s[0] = __fadd_rn(s[0], __fmul_rn(comp == 0 ? dx : comp == 1 ? dy : dz, fm));
                        }
                    }
                    next = b.x;
                } else {
                    next = p + 1;
                }
            }
        }
        if (have && sub < 3) {
            float *o = out + 3 * (uint64_t)v.order[i];
            if (R == 1) {
                o[0] = s[0];
                o[1] = s[1];
                o[2] = s[2];
            } else {
                o[sub] = s[0];
            }
        }
    }
}

}  // namespace

// Bodies a warp takes.  The walk of a body is serial, so the fewer bodies
// the lanes are spread over, the shorter a warp's walk; but R > 1 adds the
// hand-over of the terms to every pair and walks the nodes once per B
// bodies.  The line lies where the warps stop filling the SMs (about 42 of
// them on each): measured at theta 0.5 for B = 2 / 4 / 8 / 32, ms: 2,000
// bodies 0.10 / 0.12 / 0.18 / 0.42; 20,000: 1.51 / 1.10 / 1.52 / 4.1;
// 50,000: 5.5 / 4.10 / 4.06 / 8.3; 200,000: 36 / 24 / 21.4 / 23.2; 1M:
// 230 / 150 / 124 / 100.
template <int B>
static rtd_status launch_ref_walk(const BhView &v, const rtd_bh_params *p, float *d_out, cudaStream_t st) {
    bh_ref_walk_kernel<B><<<grid_for(ceil_div(v.n, B), 4, 1 << 20), 128, 0, st>>>(v, p->theta, p->G, d_out);
    RTD_LAUNCH_CHECK();
    return RTD_OK;
}

rtd_status bh_ref_forward(rtd_bh *b, const rtd_bh_params *p, float *d_out, cudaStream_t st) {
    const BhView v = bh_view(b);
    constexpr uint64_t full = NUM_SMS_HINT * 42;   // warps that fill the SMs
    if (v.n <= 2 * full) return launch_ref_walk<2>(v, p, d_out, st);
    if (v.n <= 4 * full) return launch_ref_walk<4>(v, p, d_out, st);
    if (v.n <= 32 * full) return launch_ref_walk<8>(v, p, d_out, st);
    return launch_ref_walk<32>(v, p, d_out, st);
}

}  // namespace rtd
