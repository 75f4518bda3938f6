// bh_plummer.cu -- Plummer-law Barnes-Hut walks (forward and adjoint).
//
// Physics: phi_i = -G sum_j m_j / sqrt(|x_i - x_j|^2 + eps^2), a_i =
// -grad phi_i; accepted cells act as monopole + traceless quadrupole about
// their COM with the same softened distance.  A cell is accepted for body
// i when width^2 < theta^2 |COM - x_i|^2 (each operation rounded, so the
// CPU oracle makes identical decisions); rejected leaves are summed
// directly, rejected internal cells opened.
//
// Execution: a warp takes a group of 32 bodies (consecutive in flat order,
// so spatially compact) and walks the tree once for all of them.  Stack
// entries carry the mask of lanes that still need the node; up to 32 are
// taken per step, one per lane, and each lane decides its node for the whole
// group from the group's box where the box settles it (every operation of
// the per-body test is monotone in the distance, so a box decision equals
// every body's); only nodes it leaves open are tested body by body.
// Accepted cells and the bodies of rejected leaves go to four per-warp
// lists: those every body of the group interacts with, and those with a lane
// mask.  32 entries of a list form a tile, staged in shared memory as pairs
// and evaluated by all lanes (lane = body) two interactions at a time in
// packed FP32 (f32x2), which halves the instructions issued.
//
// Adjoint (dL/dx, dL/dm for upstream dL/da, dL/dphi): lane = body evaluates
// each (body, source) pair once, adds the body's derivative up and leaves
// three to five coefficients in shared memory; then lane = source sums the
// source's derivative over the bodies from the coefficients (replayed from
// the log at 1M bodies: 18.8 ms; a table of the derivatives themselves,
// summed row by row: 33.8 ms) and adds it with one vector atomic per source
// and part.  Cell derivatives (COM, mass,
// quadrupole) are then pushed to the bodies by a top-down pass: with Q
// about the COM the first moment vanishes, so for a cell C holding body j
//     dL/dx_j += m_j (g_c/M - 2 B c + 2 B x_j)
//     dL/dm_j += g_M + g_c.(x_j - c)/M + (x_j - c)^T B (x_j - c)
// with B = 3 sym(G_Q) - tr(G_Q) I; both split into per-node constants that
// add up along root-to-leaf paths.
#include <rtdsl.h>

#include "bh.cuh"

namespace rtd {
namespace {

constexpr int WW = 4;   // warps per block

// Lists of a warp, and the kinds of its tiles: what every body of the group
// takes, and what only the lanes of a mask take.
enum : int { L_CELLS = 0, L_CELLS_MASKED = 1, L_BODIES = 2, L_BODIES_MASKED = 3 };

struct WarpTile {
    float4 pair[16][5];   // sources 2p, 2p + 1 interleaved: (-x -x -y -y) (-z -z -M -M)
                          // (xx xx yy yy) (zz zz xy xy) (xz xz yz yz)
    uint32_t mask[32];
    uint2 list[4][64];    // (cell or body, lane mask)
    uint4 leaf[32];       // rejected leaves not yet listed: first body, bodies, lane mask
    uint32_t lost;        // the lanes that take a body without a place (forward)
};

// Adjoint: what the bodies' side of an interaction leaves for the source's
// side, for up to ADJ_SOURCES sources at a time: the coefficients of each
// (body, source) pair, a row a body (18 words apart: both sides read and
// write 64-bit pairs without bank conflicts), and the bodies' positions and
// upstream gradients, each value twice.
constexpr int ADJ_SOURCES = 16;
struct WarpAdj {
    float coef[5][32][ADJ_SOURCES + 2];
    float4 body[32][3];   // (x x y y) (z z vx vx) (vy vy vz vz)
};

// ------------------------------------------------------- packed FP32 pairs
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f2 pk(float a) { return pk(a, a); }
__device__ __forceinline__ float lo(f2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
    return x;
}
__device__ __forceinline__ float hi(f2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
    return y;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 rsqrt2(f2 a) { return pk(rsqrtf(lo(a)), rsqrtf(hi(a))); }
// The halves that are wanted, else 0.
__device__ __forceinline__ f2 keep2(f2 a, bool k0, bool k1) { return pk(k0 ? lo(a) : 0.f, k1 ? hi(a) : 0.f); }
__device__ __forceinline__ f2 xy(const float4 &v) { return pk(v.x, v.y); }
__device__ __forceinline__ f2 zw(const float4 &v) { return pk(v.z, v.w); }

__device__ __forceinline__ float dot3_rn(float x, float y, float z) {
    float s = __fmul_rn(x, x);
    s = __fadd_rn(s, __fmul_rn(y, y));
    s = __fadd_rn(s, __fmul_rn(z, z));
    return s;
}

// Per-body MAC: accept when width^2 < theta^2 * |COM - x|^2.
__device__ __forceinline__ bool body_accept(float x, float y, float z, float cx, float cy, float cz,
                                            float width, float theta2) {
    const float d2 = dot3_rn(__fsub_rn(cx, x), __fsub_rn(cy, y), __fsub_rn(cz, z));
    return __fmul_rn(width, width) < __fmul_rn(theta2, d2);
}

__device__ __forceinline__ uint32_t lane_lt() {
    uint32_t m;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Forward interaction of a field point with a pair of cells (r = x - c, G
// omitted, nM = -M): what it adds to phi and a.
template <bool QUAD>
__device__ __forceinline__ void cells_fwd(const float4 *c, f2 x, f2 y, f2 z, f2 eps2, f2 &phi, f2 &ax, f2 &ay, f2 &az) {
    const float4 c0 = c[0], c1 = c[1];
    const f2 rx = add2(x, xy(c0)), ry = add2(y, zw(c0)), rz = add2(z, xy(c1)), nM = zw(c1);
    const f2 i1 = rsqrt2(fma2(rx, rx, fma2(ry, ry, fma2(rz, rz, eps2))));
    const f2 i2 = mul2(i1, i1), i3 = mul2(i1, i2);
    phi = fma2(nM, i1, phi);
    if (!QUAD) {
        const f2 k = mul2(nM, i3);
        ax = fma2(k, rx, ax);
        ay = fma2(k, ry, ay);
        az = fma2(k, rz, az);
    } else {
        const float4 q0 = c[2], q1 = c[3], q2 = c[4];
        const f2 xx = xy(q0), yy = zw(q0), zz = xy(q1), cxy = zw(q1), cxz = xy(q2), cyz = zw(q2);
        const f2 qx = fma2(xx, rx, fma2(cxy, ry, mul2(cxz, rz)));
        const f2 qy = fma2(cxy, rx, fma2(yy, ry, mul2(cyz, rz)));
        const f2 qz = fma2(cxz, rx, fma2(cyz, ry, mul2(zz, rz)));
        const f2 i5 = mul2(i3, i2);
        const f2 t = mul2(fma2(rx, qx, fma2(ry, qy, mul2(rz, qz))), i5);   // r.Q.r / r^5
        phi = fma2(pk(-0.5f), t, phi);
        const f2 k = fma2(mul2(pk(-2.5f), t), i2, mul2(nM, i3));
        ax = fma2(k, rx, fma2(qx, i5, ax));
        ay = fma2(k, ry, fma2(qy, i5, ay));
        az = fma2(k, rz, fma2(qz, i5, az));
    }
}

// Body side of the derivatives of L = u*phi + v.a for a pair of sources (r =
// x - c, G omitted): d/dx added to g, and the coefficients
//   A, B, H, I, N:  dL/dr = A r + B v + Q (2 H r + I v),  dL/dM = N,
//                   dL/dQ = sym(r (H r + I v)^T)
// zeroed for the sources this lane does not take.
template <bool QUAD, bool MASKED>
__device__ __forceinline__ void sources_adj(const float4 *c, f2 x, f2 y, f2 z, f2 eps2, f2 u, f2 vx, f2 vy, f2 vz,
                                            bool k0, bool k1, f2 &gx, f2 &gy, f2 &gz, f2 (&coef)[5]) {
    const float4 c0 = c[0], c1 = c[1];
    const f2 rx = add2(x, xy(c0)), ry = add2(y, zw(c0)), rz = add2(z, xy(c1)), nM = zw(c1);
    const f2 i1 = rsqrt2(fma2(rx, rx, fma2(ry, ry, fma2(rz, rz, eps2))));
    const f2 i2 = mul2(i1, i1), i3 = mul2(i1, i2), i5 = mul2(i3, i2);
    const f2 nvr = mul2(pk(-1.f), fma2(vx, rx, fma2(vy, ry, mul2(vz, rz)))), nu = mul2(pk(-1.f), u);
    f2 N = fma2(nvr, i3, mul2(nu, i1));
    // monopole: dL/dr = M ((u i3 + 3 vr i5) r - i3 v)
    f2 A = mul2(nM, fma2(mul2(nvr, pk(3.f)), i5, mul2(nu, i3))), B = mul2(nM, i3);
    if (!QUAD) {
        if (MASKED) {
            A = keep2(A, k0, k1);
            B = keep2(B, k0, k1);
            N = keep2(N, k0, k1);
        }
        gx = fma2(A, rx, fma2(B, vx, gx));
        gy = fma2(A, ry, fma2(B, vy, gy));
        gz = fma2(A, rz, fma2(B, vz, gz));
    } else {
        const float4 q0 = c[2], q1 = c[3], q2 = c[4];
        const f2 xx = xy(q0), yy = zw(q0), zz = xy(q1), cxy = zw(q1), cxz = xy(q2), cyz = zw(q2);
        const f2 qrx = fma2(xx, rx, fma2(cxy, ry, mul2(cxz, rz)));
        const f2 qry = fma2(cxy, rx, fma2(yy, ry, mul2(cyz, rz)));
        const f2 qrz = fma2(cxz, rx, fma2(cyz, ry, mul2(zz, rz)));
        const f2 i7 = mul2(i5, i2);
        const f2 nk1 = mul2(mul2(fma2(rx, qrx, fma2(ry, qry, mul2(rz, qrz))), pk(-2.5f)), i7);   // -2.5 rQr i7
        const f2 vqr = fma2(vx, qrx, fma2(vy, qry, mul2(vz, qrz)));
        // u phi_Q + v.a_Q adds (u k1 - 5 vQr i7 + 7 k1 vr i2) r - k1 v
        // - (u i5 + 5 vr i7) Qr + i5 Qv
        const f2 n5i7 = mul2(pk(-5.f), i7);
        A = fma2(nu, nk1, fma2(vqr, n5i7, fma2(mul2(nk1, pk(7.f)), mul2(nvr, i2), A)));
        B = add2(B, nk1);
        f2 H = mul2(pk(0.5f), fma2(nu, i5, mul2(nvr, mul2(pk(5.f), i7)))), I = i5;
        if (MASKED) {
            A = keep2(A, k0, k1);
            B = keep2(B, k0, k1);
            H = keep2(H, k0, k1);
            I = keep2(I, k0, k1);
            N = keep2(N, k0, k1);
        }
        const f2 C = add2(H, H);
        // Q (C r + I v): Q applied to one vector
        const f2 tx = fma2(C, rx, mul2(I, vx)), ty = fma2(C, ry, mul2(I, vy)), tz = fma2(C, rz, mul2(I, vz));
        gx = fma2(xx, tx, fma2(cxy, ty, fma2(cxz, tz, fma2(A, rx, fma2(B, vx, gx)))));
        gy = fma2(cxy, tx, fma2(yy, ty, fma2(cyz, tz, fma2(A, ry, fma2(B, vy, gy)))));
        gz = fma2(cxz, tx, fma2(cyz, ty, fma2(zz, tz, fma2(A, rz, fma2(B, vz, gz)))));
        coef[3] = H;
        coef[4] = I;
    }
    coef[0] = A;
    coef[1] = B;
    coef[2] = N;
}

// Sum of a pair over the lanes whose numbers differ in bits 3 and 4.
__device__ __forceinline__ f2 quarter_sum(f2 a) {
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1)
        a = add2(a, pk(__shfl_xor_sync(0xffffffffu, lo(a), o), __shfl_xor_sync(0xffffffffu, hi(a), o)));
    return a;
}

// Source side: lane l + 8 h takes the pair of sources l of a chunk of 8 and
// every 4th body from h on, and adds up dL/dc (= -dL/dr), dL/dM and dL/dQ
// from the coefficients; the four lanes of a pair then add theirs, and two
// of them write one source each.
template <bool QUAD>
__device__ __forceinline__ void sources_sum(const WarpAdj &J, const float4 *c, uint32_t rows, bool have0, bool have1,
                                            uint32_t id0, uint32_t id1, bool cells, float G, float4 *cell_grad,
                                            float4 *body_grad) {
    const int lane = threadIdx.x & 31, l = lane & 7, h = lane >> 3;
    const f2 z = pk(0.f);
    const float4 c0 = c[0], c1 = c[1];
    const f2 nx = xy(c0), ny = zw(c0), nz = xy(c1);
    f2 sx = z, sy = z, sz = z, N = z, tx = z, ty = z, tz = z, gq[6] = {z, z, z, z, z, z};
    auto coef = [&](int k, uint32_t i) { return *reinterpret_cast<const f2 *>(&J.coef[k][i][2 * l]); };
#pragma unroll 1
    for (uint32_t i = h; i < rows; i += 4) {
        const float4 b0 = J.body[i][0], b1 = J.body[i][1], b2 = J.body[i][2];
        const f2 rx = add2(xy(b0), nx), ry = add2(zw(b0), ny), rz = add2(xy(b1), nz);
        const f2 vx = zw(b1), vy = xy(b2), vz = zw(b2);
        const f2 A = coef(0, i), B = coef(1, i);
        N = add2(N, coef(2, i));
        sx = fma2(A, rx, fma2(B, vx, sx));
        sy = fma2(A, ry, fma2(B, vy, sy));
        sz = fma2(A, rz, fma2(B, vz, sz));
        if (QUAD) {
            const f2 H = coef(3, i), I = coef(4, i);
            const f2 hx = mul2(H, rx), hy = mul2(H, ry), hz = mul2(H, rz);
            const f2 wx = fma2(I, vx, hx), wy = fma2(I, vy, hy), wz = fma2(I, vz, hz);
            tx = add2(tx, add2(wx, hx));
            ty = add2(ty, add2(wy, hy));
            tz = add2(tz, add2(wz, hz));
            gq[0] = fma2(rx, wx, gq[0]);
            gq[1] = fma2(ry, wy, gq[1]);
            gq[2] = fma2(rz, wz, gq[2]);
            gq[3] = fma2(rx, wy, fma2(ry, wx, gq[3]));
            gq[4] = fma2(rx, wz, fma2(rz, wx, gq[4]));
            gq[5] = fma2(ry, wz, fma2(rz, wy, gq[5]));
        }
    }
    if (QUAD) {
        const float4 q0 = c[2], q1 = c[3], q2 = c[4];
        sx = fma2(xy(q0), tx, fma2(zw(q1), ty, fma2(xy(q2), tz, sx)));
        sy = fma2(zw(q1), tx, fma2(zw(q0), ty, fma2(zw(q2), tz, sy)));
        sz = fma2(xy(q2), tx, fma2(zw(q2), ty, fma2(xy(q1), tz, sz)));
    }
    sx = quarter_sum(sx);
    sy = quarter_sum(sy);
    sz = quarter_sum(sz);
    N = quarter_sum(N);
    if (QUAD)
#pragma unroll
        for (int k = 0; k < 6; ++k) gq[k] = quarter_sum(gq[k]);
    if (h == 0 ? have0 : h == 1 && have1) {
        auto half = [&](f2 a) { return G * (h ? hi(a) : lo(a)); };
        const uint32_t id = h ? id1 : id0;
        float4 *to = cells ? &cell_grad[3 * (uint64_t)id] : &body_grad[id];
        atomicAdd(to, make_float4(-half(sx), -half(sy), -half(sz), half(N)));
        if (QUAD) {
            atomicAdd(to + 1, make_float4(half(gq[0]), half(gq[1]), half(gq[2]), 0.5f * half(gq[3])));
            atomicAdd(reinterpret_cast<float2 *>(to + 2), make_float2(0.5f * half(gq[4]), 0.5f * half(gq[5])));
        }
    }
}

template <bool V>
struct Flag {
    static constexpr bool value = V;
};

// The adjoint holds more state, and its coefficients leave room for 3 blocks
// of 4 warps per SM.
// SPLIT = 1: a warp per group.  SPLIT = WW: the warps of a block share a
// group, each the subtrees of every WW-th entry of the stack once it holds
// SPLIT_AT of them.
constexpr int SPLIT_AT = 64;
template <bool QUAD, bool ADJ, int SPLIT>
__global__ void __launch_bounds__(WW * 32, ADJ ? 3 : 6) bh_walk_kernel(
    const BhView v, float theta2, float eps2, float G, const float *__restrict__ g_acc,
    const float *__restrict__ g_phi, float *__restrict__ acc_out, float *__restrict__ phi_out,
    float4 *__restrict__ cell_grad, float4 *__restrict__ body_grad, uint2 *__restrict__ stack,
    uint32_t stack_entries, const IlogView lg, BhHeader *hm) {
    __shared__ WarpTile tiles[WW];
    extern __shared__ WarpAdj adjs[];   // the adjoint's: one a warp
    __shared__ uint32_t s_group;        // SPLIT: the block's group
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    WarpTile &T = tiles[warp];
    WarpAdj &J = adjs[ADJ ? warp : 0];
    const uint64_t gw = (uint64_t)blockIdx.x * WW + warp;
    uint2 *stk = stack + gw * BH_STACK_CAP_MAX;   // this warp's slice
    const uint32_t ngroups = (uint32_t)((v.n + BH_GROUP - 1) / BH_GROUP), n_nodes = v.hdr->n_nodes;
    const uint32_t lt = lane_lt(), mine = 1u << lane;
    const f2 e2 = pk(eps2);
    uint32_t max_sp = 0;
    while (true) {
        uint32_t g = 0;
        if (SPLIT == 1) {
            if (lane == 0) g = atomicAdd(&hm->group_counter, 1u);
            g = __shfl_sync(0xffffffffu, g, 0);
        } else {
            if (threadIdx.x == 0) s_group = atomicAdd(&hm->group_counter, 1u);
            __syncthreads();
            g = s_group;
        }
        if (g >= ngroups) break;
        const uint32_t part = SPLIT == 1 ? 0u : (uint32_t)warp, slot_g = g * SPLIT + part;   // the log's entry
        bool shared = SPLIT > 1;   // still the part of the walk that every warp makes
        const uint32_t gs = g * BH_GROUP, gc = (uint32_t)(v.n - gs < BH_GROUP ? v.n - gs : BH_GROUP);
        const uint32_t i = gs + lane;
        const bool valid = (uint32_t)lane < gc;
        // spare lanes stand at the first body, with no upstream gradient
        const float4 me = v.fbody[valid ? i : gs];
        const f2 px = pk(me.x), py = pk(me.y), pz = pk(me.z);
        f2 ax = pk(0.f), ay = pk(0.f), az = pk(0.f), phi = pk(0.f);   // forward sums / adjoint d/dx_i
        f2 vx = pk(0.f), vy = pk(0.f), vz = pk(0.f), u = pk(0.f);
        if (ADJ && valid) {
            const uint32_t o = v.order[i];
            vx = pk(g_acc[3 * (uint64_t)o]);
            vy = pk(g_acc[3 * (uint64_t)o + 1]);
            vz = pk(g_acc[3 * (uint64_t)o + 2]);
            u = pk(g_phi ? g_phi[o] : 0.f);
        }
        if (ADJ) {
            J.body[lane][0] = make_float4(me.x, me.x, me.y, me.y);
            J.body[lane][1] = make_float4(me.z, me.z, lo(vx), lo(vx));
            J.body[lane][2] = make_float4(lo(vy), lo(vy), lo(vz), lo(vz));
        }
        const uint32_t all = __ballot_sync(0xffffffffu, valid);
        // the group's box; a body with a NaN coordinate accepts no cell, so
        // no box speaks for it
        float blo[3] = {me.x, me.y, me.z}, bhi[3] = {me.x, me.y, me.z};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                blo[a] = fminf(blo[a], __shfl_xor_sync(0xffffffffu, blo[a], o));
                bhi[a] = fmaxf(bhi[a], __shfl_xor_sync(0xffffffffu, bhi[a], o));
            }
        const bool boxed = !__any_sync(0xffffffffu, isnan(me.x) || isnan(me.y) || isnan(me.z));
        int n_list[4] = {0, 0, 0, 0};   // (constant indices only)
        if (!ADJ && lane == 0) T.lost = 0;
        int n_leaf = 0, sp = 0;
        // The adjoint replays the group's tiles from the forward's log when
        // the log holds them all; otherwise it walks the tree.
        const uint2 lgg = (ADJ && lg.group) ? lg.group[slot_g] : make_uint2(ILOG_NONE, ILOG_NONE);
        const bool replay = ADJ && lgg.y != ILOG_NONE;
        const uint32_t logged = replay ? lgg.y : 0u;
        if (n_nodes > 0 && !replay) {
            if (lane == 0) stk[0] = make_uint2(0u, all);
            sp = 1;
        }
        __syncwarp();
        // replay: a page's tile counts come in one load (lane l: tile l) with
        // the next page's id, and each tile's entries are loaded while the
        // tile before it is evaluated
        uint32_t rt = 0, rpg = lgg.x, rpg_next = ILOG_NONE, rcounts = 0;
        uint2 rentry = make_uint2(0u, 0u);
        if (logged > 0) {
            rcounts = lane < (int)ILOG_PAGE ? lg.counts[(uint64_t)rpg * ILOG_PAGE + lane] : 0u;
            rpg_next = logged > ILOG_PAGE ? lg.next[rpg] : ILOG_NONE;
            rentry = lg.entries[(uint64_t)rpg * ILOG_PAGE * 32 + lane];
        }
        // forward: every evaluated tile appended to the group's chain of log
        // pages, while the pool has pages (all warp-uniform)
        uint32_t nt = 0, page = ILOG_NONE, first = ILOG_NONE;
        bool lok = !ADJ && lg.group != nullptr;

        // One step of the walk: up to 32 stack entries, one a lane.
        auto step = [&]() {
            const int t = sp < 32 ? sp : 32;
            sp -= t;
            uint2 e = make_uint2(0u, 0u);
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            uint4 b = make_uint4(0u, 0u, 0u, 0u);
            bool open = lane < t;
            uint32_t A = 0;
            if (open) {
                e = stk[sp + lane];
                a = __ldg(&v.node_a[e.x]);
                b = __ldg(&v.node_b[e.x]);
                // nearest and farthest squared distance from the COM to the
                // box, rounded as the per-body distance is
                const float w2 = __fmul_rn(__uint_as_float(b.w), __uint_as_float(b.w));
                const float c[3] = {a.x, a.y, a.z};
                float dn[3], df[3];
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const float l = __fsub_rn(blo[q], c[q]), h = __fsub_rn(c[q], bhi[q]);
                    dn[q] = fmaxf(fmaxf(l, h), 0.f);
                    df[q] = fmaxf(fabsf(l), fabsf(h));
                }
                const bool far = w2 < __fmul_rn(theta2, dot3_rn(dn[0], dn[1], dn[2]));
                const bool near = !(w2 < __fmul_rn(theta2, dot3_rn(df[0], df[1], df[2])));
                // (A centre with a NaN, from products that overflowed to inf -
                // inf, is accepted by no body: then near holds, and far may
                // too, since fmaxf drops the NaN.)
                if (boxed && (far || near)) {
                    if (!near) A = e.y;
                    open = false;
                }
            }
            __syncwarp();
            for (uint32_t m = __ballot_sync(0xffffffffu, open); m; m &= m - 1) {
                const int k = __ffs(m) - 1;
                const float cx = __shfl_sync(0xffffffffu, a.x, k);
                const float cy = __shfl_sync(0xffffffffu, a.y, k);
                const float cz = __shfl_sync(0xffffffffu, a.z, k);
                const float w = __uint_as_float(__shfl_sync(0xffffffffu, b.w, k));
                const uint32_t acc = __ballot_sync(0xffffffffu, body_accept(me.x, me.y, me.z, cx, cy, cz, w, theta2));
                if (lane == k) A = acc & e.y;
            }
            const uint32_t rest = lane < t ? e.y & ~A : 0u;   // lanes that open the node
            uint32_t m = __ballot_sync(0xffffffffu, A == all);
            if (A == all) T.list[L_CELLS][n_list[L_CELLS] + __popc(m & lt)] = make_uint2(e.x, A);
            n_list[L_CELLS] += __popc(m);
            m = __ballot_sync(0xffffffffu, A != all && A != 0);
            if (A != all && A != 0) T.list[L_CELLS_MASKED][n_list[L_CELLS_MASKED] + __popc(m & lt)] = make_uint2(e.x, A);
            n_list[L_CELLS_MASKED] += __popc(m);
            const bool leaf = b.z & BH_LEAF_BIT;
            m = __ballot_sync(0xffffffffu, rest && leaf);
            if (rest && leaf) T.leaf[__popc(m & lt)] = make_uint4(b.y, b.z & ~BH_LEAF_BIT, rest, 0u);
            n_leaf = __popc(m);
            // children of the opened cells
            uint32_t c[8];
            uint32_t np = 0;
            if (rest && !leaf) {
                const uint4 c0 = __ldg(&v.child8[2 * (uint64_t)e.x]), c1 = __ldg(&v.child8[2 * (uint64_t)e.x + 1]);
                c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w;
                c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
#pragma unroll
                for (int q = 0; q < 8; ++q) np += c[q] != 0xFFFFFFFFu;
            }
            uint32_t incl = np;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            if ((uint32_t)sp + total <= stack_entries) {
                uint2 *to = stk + sp + (incl - np);
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                    if (q < np) to[q] = make_uint2(c[q], rest);
                sp += (int)total;
            } else if (lane == 0) {
                atomicOr(&hm->err, DEVERR_STACK);
            }
            max_sp = max(max_sp, (uint32_t)sp);
            __syncwarp();
        };
        // Keeps this warp's share of the stack.
        auto share_out = [&]() {
            const int had = sp;
            for (int base = 0; base < had; base += 32) {
                const int j = base + lane;
                const uint2 e = j < had ? stk[j] : make_uint2(0u, 0u);
                __syncwarp();
                if (j < had && j % SPLIT == (int)part) stk[j / SPLIT] = e;
                __syncwarp();
            }
            sp = (had - (int)part + SPLIT - 1) / SPLIT;
        };
        // Up to 32 bodies of the last waiting leaf into a list.  A leaf that
        // holds bodies of the group goes to the masked list, each body
        // without its own lane.
        auto list_leaf = [&]() {
            const uint4 lf = T.leaf[n_leaf - 1];
            const uint32_t take = lf.y < 32u ? lf.y : 32u, id = lf.x + lane;
            const bool own = lf.x < gs + gc && lf.x + take > gs, plain = lf.z == all && !own;
            const int at = plain ? n_list[L_BODIES] : n_list[L_BODIES_MASKED];
            __syncwarp();
            if ((uint32_t)lane < take)
                T.list[plain ? L_BODIES : L_BODIES_MASKED][at + lane] =
                    make_uint2(id, id - gs < gc ? lf.z & ~(1u << (id - gs)) : lf.z);
            if (plain) n_list[L_BODIES] += (int)take;
            else n_list[L_BODIES_MASKED] += (int)take;
            if (lf.y > 32u) {
                if (lane == 0) T.leaf[n_leaf - 1] = make_uint4(lf.x + 32, lf.y - 32, lf.z, 0u);
            } else {
                --n_leaf;
            }
            __syncwarp();
        };

        while (true) {
            // the next tile: its kind and entries, in list[kind][0 .. cnt)
            int kind = -1, cnt = 32;
            if (ADJ && replay) {
                if (rt >= logged) break;
                const uint32_t pos = rt % ILOG_PAGE;
                if (pos == 0 && rt > 0) {
                    rpg = rpg_next;
                    rcounts = lane < (int)ILOG_PAGE ? lg.counts[(uint64_t)rpg * ILOG_PAGE + lane] : 0u;
                    rpg_next = rt + ILOG_PAGE < logged ? lg.next[rpg] : ILOG_NONE;
                }
                const uint32_t c = __shfl_sync(0xffffffffu, rcounts, (int)pos);
                kind = (int)(c >> 6);
                cnt = (int)(c & 0x3F);
                if (lane < cnt) T.list[kind][lane] = rentry;
                if (++rt < logged) {
                    const uint32_t pos1 = rt % ILOG_PAGE;
                    rentry = lg.entries[((uint64_t)(pos1 == 0 ? rpg_next : rpg) * ILOG_PAGE + pos1) * 32 + lane];
                }
                __syncwarp();
            } else {
                while (n_list[0] < 32 && n_list[1] < 32 && n_list[2] < 32 && n_list[3] < 32) {
                    if (n_leaf > 0) {
                        list_leaf();
                    } else if (sp > 0) {
                        step();
                        if (SPLIT > 1 && shared) {
                            if (part != 0) n_list[0] = n_list[1] = n_leaf = 0;   // the first warp's
                            if (sp >= SPLIT_AT) {
                                share_out();
                                shared = false;
                            }
                        }
                    } else {
                        break;
                    }
                }
                if (n_list[0] >= 32) kind = 0;
                else if (n_list[1] >= 32) kind = 1;
                else if (n_list[2] >= 32) kind = 2;
                else if (n_list[3] >= 32) kind = 3;
                else if (n_list[0] > 0) { kind = 0; cnt = n_list[0]; }
                else if (n_list[1] > 0) { kind = 1; cnt = n_list[1]; }
                else if (n_list[2] > 0) { kind = 2; cnt = n_list[2]; }
                else if (n_list[3] > 0) { kind = 3; cnt = n_list[3]; }
                else break;
                if (!ADJ && lg.group) {
                    const uint32_t pos = nt % ILOG_PAGE;
                    if (pos == 0 && lok) {
                        uint32_t pg = 0;
                        if (lane == 0) pg = atomicAdd(&hm->ilog_used, 1u);
                        pg = __shfl_sync(0xffffffffu, pg, 0);
                        if (pg >= lg.pages) {
                            lok = false;
                        } else {
                            if (page == ILOG_NONE) first = pg;
                            else if (lane == 0) lg.next[page] = pg;
                            page = pg;
                        }
                    }
                    if (lok) {
                        const uint64_t slot = (uint64_t)page * ILOG_PAGE + pos;
                        if (lane < cnt) lg.entries[slot * 32 + lane] = T.list[kind][lane];
                        if (lane == 0) lg.counts[slot] = (uint8_t)(cnt | kind << 6);
                    }
                    ++nt;
                }
            }
            // Stage the tile.  An odd last pair repeats its source with no
            // mass and no lanes.
            const bool cells = kind < L_BODIES, masked = (kind | cnt) & 1;
            const int pairs = (cnt + 1) / 2;
            if (lane < 2 * pairs) {
                const uint2 en = T.list[kind][lane < cnt ? lane : cnt - 1];
                bool pad = lane >= cnt;
                float *w = reinterpret_cast<float *>(T.pair[lane >> 1]) + (lane & 1);
                float4 a = cells ? __ldg(&v.node_a[en.x]) : __ldg(&v.fbody[en.x]);
                if (!ADJ && masked && !cells && (isnan(a.x) || isnan(a.y) || isnan(a.z))) {
                    // 1 / r masked to 0 times an r that is no number would be
                    // no number: such a body reaches its lanes at the end
                    if (!pad) atomicOr(&T.lost, en.y);
                    pad = true;
                    a = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                w[0] = -a.x;
                w[2] = -a.y;
                w[4] = -a.z;
                w[6] = pad ? 0.f : -a.w;
                if (QUAD && cells) {
                    const float4 q0 = __ldg(&v.node_q[2 * en.x]), q1 = __ldg(&v.node_q[2 * en.x + 1]);
                    w[8] = pad ? 0.f : q0.x;
                    w[10] = pad ? 0.f : q0.y;
                    w[12] = pad ? 0.f : q0.z;
                    w[14] = pad ? 0.f : q0.w;
                    w[16] = pad ? 0.f : q1.x;
                    w[18] = pad ? 0.f : q1.y;
                }
                T.mask[lane] = pad ? 0u : en.y;
            }
            __syncwarp();
            if (!ADJ) {
                if (cells && !masked) {
#pragma unroll 2
                    for (int p = 0; p < pairs; ++p) cells_fwd<QUAD>(T.pair[p], px, py, pz, e2, phi, ax, ay, az);
                } else if (cells) {
                    for (int p = 0; p < pairs; ++p) {
                        const bool k0 = T.mask[2 * p] & mine, k1 = T.mask[2 * p + 1] & mine;
                        f2 dp = pk(0.f), dx = pk(0.f), dy = pk(0.f), dz = pk(0.f);
                        cells_fwd<QUAD>(T.pair[p], px, py, pz, e2, dp, dx, dy, dz);
                        phi = add2(phi, keep2(dp, k0, k1));
                        ax = add2(ax, keep2(dx, k0, k1));
                        ay = add2(ay, keep2(dy, k0, k1));
                        az = add2(az, keep2(dz, k0, k1));
                    }
                } else {
#pragma unroll 2
                    for (int p = 0; p < pairs; ++p) {
                        const float4 c0 = T.pair[p][0], c1 = T.pair[p][1];
                        const f2 rx = add2(px, xy(c0)), ry = add2(py, zw(c0)), rz = add2(pz, xy(c1)), nm = zw(c1);
                        f2 i1 = rsqrt2(fma2(rx, rx, fma2(ry, ry, fma2(rz, rz, e2))));
                        if (masked) i1 = keep2(i1, T.mask[2 * p] & mine, T.mask[2 * p + 1] & mine);
                        const f2 mi = mul2(nm, i1), k = mul2(mi, mul2(i1, i1));
                        phi = add2(phi, mi);
                        ax = fma2(k, rx, ax);
                        ay = fma2(k, ry, ay);
                        az = fma2(k, rz, az);
                    }
                }
            } else {
                // lane = body, then lane = source (rows past the group's
                // bodies are spare lanes', which leave zeros)
#pragma unroll 1
                for (int p0 = 0; p0 < pairs; p0 += ADJ_SOURCES / 2) {
                    const int pn = pairs - p0 < ADJ_SOURCES / 2 ? pairs - p0 : ADJ_SOURCES / 2;
                    auto bodies_side = [&](auto quad, auto msk) {
#pragma unroll 2
                        for (int q = 0; q < pn; ++q) {
                            const int p = p0 + q;
                            f2 w[5];
                            sources_adj<quad.value, msk.value>(
                                T.pair[p], px, py, pz, e2, u, vx, vy, vz, msk.value && T.mask[2 * p] & mine,
                                msk.value && T.mask[2 * p + 1] & mine, ax, ay, az, w);
#pragma unroll
                            for (int k = 0; k < (quad.value ? 5 : 3); ++k)
                                *reinterpret_cast<f2 *>(&J.coef[k][lane][2 * q]) = w[k];
                        }
                    };
                    if (QUAD && cells) {
                        if (masked) bodies_side(Flag<QUAD>(), Flag<true>());
                        else bodies_side(Flag<QUAD>(), Flag<false>());
                    } else {
                        bodies_side(Flag<false>(), Flag<true>());
                    }
                    __syncwarp();
                    const int p = p0 + (lane & 7), s0 = 2 * p, s1 = s0 + 1;
                    const float4 *src = T.pair[p < 16 ? p : 15];
                    const uint32_t id0 = s0 < cnt ? T.list[kind][s0].x : 0u, id1 = s1 < cnt ? T.list[kind][s1].x : 0u;
                    if (QUAD && cells)
                        sources_sum<QUAD>(J, src, gc, s0 < cnt, s1 < cnt, id0, id1, true, G, cell_grad, body_grad);
                    else
                        sources_sum<false>(J, src, gc, s0 < cnt, s1 < cnt, id0, id1, cells, G, cell_grad, body_grad);
                    __syncwarp();
                }
            }
            __syncwarp();
            if (!replay) {   // the entries past the tile move to the front
                int left = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (q == kind) {
                        n_list[q] -= cnt;
                        left = n_list[q];
                    }
                if (left > 0) {
                    const uint2 en = T.list[kind][32 + lane];
                    if (lane < left) T.list[kind][lane] = en;
                    __syncwarp();
                }
            }
        }
        if (!ADJ && lg.group && lane == 0) {
            lg.group[slot_g] = make_uint2(first, lok ? nt : ILOG_NONE);
            atomicAdd(&hm->ilog_need, (nt + ILOG_PAGE - 1) / ILOG_PAGE);
        }
        float4 sum = make_float4(lo(ax) + hi(ax), lo(ay) + hi(ay), lo(az) + hi(az), lo(phi) + hi(phi));
        if (!ADJ && (T.lost & mine)) sum = make_float4(NAN, NAN, NAN, NAN);
        if (!ADJ && SPLIT > 1) {   // the first warp adds up the others' sums
            float4 *sums = T.pair[0];
            sums[lane] = sum;
            __syncthreads();
            if (part == 0)
                for (int w = 1; w < SPLIT; ++w) {
                    const float4 o = tiles[w].pair[0][lane];
                    sum = make_float4(sum.x + o.x, sum.y + o.y, sum.z + o.z, sum.w + o.w);
                }
        }
        if (valid && (ADJ || part == 0)) {
            if (!ADJ) {
                const uint32_t o = v.order[i];
                acc_out[3 * (uint64_t)o] = G * sum.x;
                acc_out[3 * (uint64_t)o + 1] = G * sum.y;
                acc_out[3 * (uint64_t)o + 2] = G * sum.z;
                if (phi_out) phi_out[o] = G * sum.w;
            } else {
                atomicAdd(&body_grad[i], make_float4(G * sum.x, G * sum.y, G * sum.z, 0.f));
            }
        }
        if (SPLIT > 1) __syncthreads();
        else __syncwarp();
    }
    if (lane == 0) atomicMax(&hm->max_stack, max_sp);
}

// Per-node constants of the cell-to-body rule (Pvec.xyz, Pconst | Pmat xx
// yy zz xy | xz yz) from the cell's derivatives (g_c, g_M | G_Q).
__device__ __forceinline__ void cell_constants(const float4 a, const float4 *cg, float out[10]) {
    const float4 g0 = cg[0], g1 = cg[1], g2 = cg[2];
    const float M = a.w, cx = a.x, cy = a.y, cz = a.z;
    const float Gxx = g1.x, Gyy = g1.y, Gzz = g1.z, Gxy = g1.w, Gxz = g2.x, Gyz = g2.y;
    const float tr = Gxx + Gyy + Gzz;
    const float Bxx = 3.f * Gxx - tr, Byy = 3.f * Gyy - tr, Bzz = 3.f * Gzz - tr;
    const float Bxy = 3.f * Gxy, Bxz = 3.f * Gxz, Byz = 3.f * Gyz;
    const float Bcx = Bxx * cx + Bxy * cy + Bxz * cz;
    const float Bcy = Bxy * cx + Byy * cy + Byz * cz;
    const float Bcz = Bxz * cx + Byz * cy + Bzz * cz;
    const float invM = M > 0.f ? 1.f / M : 0.f;
    out[0] = g0.x * invM - 2.f * Bcx;
    out[1] = g0.y * invM - 2.f * Bcy;
    out[2] = g0.z * invM - 2.f * Bcz;
    out[3] = g0.w - (g0.x * cx + g0.y * cy + g0.z * cz) * invM + (cx * Bcx + cy * Bcy + cz * Bcz);
    out[4] = Bxx; out[5] = Byy; out[6] = Bzz; out[7] = Bxy; out[8] = Bxz; out[9] = Byz;
}

// Each node's constants in place of its derivatives (10 of 12 words).
__global__ void __launch_bounds__(256) bh_constants_kernel(const BhView v, float4 *cell_grad) {
    const uint32_t n_nodes = v.hdr->n_nodes;
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n_nodes; i += gridDim.x * 256) {
        float own[10];
        float4 *c = cell_grad + 3 * (uint64_t)i;
        cell_constants(v.node_a[i], c, own);
        c[0] = make_float4(own[0], own[1], own[2], own[3]);
        c[1] = make_float4(own[4], own[5], own[6], own[7]);
        c[2] = make_float4(own[8], own[9], 0.f, 0.f);
    }
}

// The bodies' gradients, a warp per leaf: the constants added up along the
// path to the root (a word a lane; going through the levels in one block
// took 0.96 ms at 1M bodies, this 0.05 ms), then applied to the leaf's
// bodies.
__global__ void __launch_bounds__(128) bh_finish_grad_kernel(const BhView v, const float *__restrict__ constants,
                                                             const float4 *__restrict__ body_grad,
                                                             float *__restrict__ g_pos, float *__restrict__ g_mass) {
    const uint32_t n_nodes = v.hdr->n_nodes;
    const int lane = threadIdx.x & 31;
    for (uint32_t leaf = blockIdx.x * 4 + (threadIdx.x >> 5); leaf < n_nodes; leaf += gridDim.x * 4) {
        const uint4 b = v.node_b[leaf];
        if (!(b.z & BH_LEAF_BIT)) continue;
        float sum = 0.f;
        for (uint32_t i = leaf; i != 0xFFFFFFFFu; i = v.parent[i])
            if (lane < 10) sum += constants[12 * (uint64_t)i + lane];
        float P[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) P[k] = __shfl_sync(0xffffffffu, sum, k);
        const uint32_t s0 = b.y, c = b.z & ~BH_LEAF_BIT;
        for (uint32_t k = lane; k < c; k += 32) {
            const float4 o = v.fbody[s0 + k];
            const float Px = P[4] * o.x + P[7] * o.y + P[8] * o.z;
            const float Py = P[7] * o.x + P[5] * o.y + P[9] * o.z;
            const float Pz = P[8] * o.x + P[9] * o.y + P[6] * o.z;
            const float4 bg = body_grad[s0 + k];
            const uint32_t orig = v.order[s0 + k];
            g_pos[3 * (uint64_t)orig] = bg.x + o.w * (P[0] + 2.f * Px);
            g_pos[3 * (uint64_t)orig + 1] = bg.y + o.w * (P[1] + 2.f * Py);
            g_pos[3 * (uint64_t)orig + 2] = bg.z + o.w * (P[2] + 2.f * Pz);
            if (g_mass)
                g_mass[orig] = bg.w + P[3] + (P[0] * o.x + P[1] * o.y + P[2] * o.z) +
                               (o.x * Px + o.y * Py + o.z * Pz);
        }
    }
}

// Whether the warps of a block share a group: only where there are fewer
// groups than five warps an SM, so that the walk of one group is what the
// call takes.  Sharing repeats the first steps of the walk and leaves more
// tiles part empty.  Measured, a warp / a block per group, ms (forward;
// adjoint): 10,000 bodies 0.45 / 0.34; 0.58 / 0.42, 16,000: 0.51 / 0.33; 0.67
// / 0.51, 30,000: 0.62 / 0.54; 0.90 / 0.95, 100,000: 0.97 / 1.25; 2.1 / 3.2.
// rtd_bh_forward_noalloc, whose results are the same bits, follows the same
// rule, although its 148 blocks then take several groups in turn (whole call
// 4,000: 0.32 / 0.14, 10,000: 0.44 / 0.42, 16,000: 0.49 / 0.63, 23,600: 0.68 /
// 1.03; 1.5 ms before groups were shared or walked by their box).
inline bool split_groups(uint64_t n) { return n <= (uint64_t)NUM_SMS_HINT * 5 * BH_GROUP; }

template <bool QUAD, bool ADJ, int SPLIT>
rtd_status launch_walk(rtd_bh *b, const rtd_bh_params *p, const float *g_acc, const float *g_phi,
                       float *acc, float *phi, const IlogView &lg, cudaStream_t st) {
    int dev = 0, sms = 148, per_sm = 4;
    RTD_CUDA(cudaGetDevice(&dev));
    RTD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const size_t smem = ADJ ? WW * sizeof(WarpAdj) : 0;
    if (ADJ)
        RTD_CUDA(cudaFuncSetAttribute(bh_walk_kernel<QUAD, ADJ, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    RTD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bh_walk_kernel<QUAD, ADJ, SPLIT>,
                                                           WW * 32, smem));
    if (per_sm < 1) per_sm = 1;
    uint64_t blocks = (uint64_t)sms * (uint64_t)per_sm;
    const uint64_t need = ceil_div(ceil_div(b->n, BH_GROUP) * SPLIT, WW);
    if (blocks > need) blocks = need;
    if (blocks < 1) blocks = 1;
    const uint64_t warps = blocks * WW;
    if (b->stack_warps < warps) {
        RTD_TRY(b->stack.reserve(warps * BH_STACK_CAP_MAX * sizeof(uint2)));
        b->stack_warps = warps;
    }
    BhHeader *h = b->hdr.as<BhHeader>();
    RTD_CUDA(cudaMemsetAsync(&h->group_counter, 0, sizeof(uint32_t), st));
    const BhView v = bh_view(b);
    bh_walk_kernel<QUAD, ADJ, SPLIT><<<(unsigned)blocks, WW * 32, smem, st>>>(
        v, p->theta * p->theta, p->eps * p->eps, p->G, g_acc, g_phi, acc, phi,
        b->cell_grad.as<float4>(), b->gpos_flat.as<float4>(), b->stack.as<uint2>(),
        bh_stack_entries(), lg, h);
    RTD_LAUNCH_CHECK();
    return RTD_OK;
}

template <bool QUAD, bool ADJ>
rtd_status launch_walk(rtd_bh *b, const rtd_bh_params *p, const float *g_acc, const float *g_phi,
                       float *acc, float *phi, const IlogView &lg, cudaStream_t st) {
    return split_groups(b->n) ? launch_walk<QUAD, ADJ, WW>(b, p, g_acc, g_phi, acc, phi, lg, st)
                              : launch_walk<QUAD, ADJ, 1>(b, p, g_acc, g_phi, acc, phi, lg, st);
}

}  // namespace

rtd_status bh_ref_forward(rtd_bh *b, const rtd_bh_params *p, float *d_out, cudaStream_t st);

// The interaction log for a forward: pinned hint and event on first use,
// the pool grown to the last logging forward's need once its copy has
// landed (grown only), the per-group array for up to n groups, and the
// page counters cleared.
static rtd_status ilog_prepare(rtd_bh *b, cudaStream_t st, IlogView &lg) {
    if (!b->ilog_hint) {
        RTD_CUDA(cudaHostAlloc(reinterpret_cast<void **>(&b->ilog_hint), sizeof(uint32_t),
                               cudaHostAllocDefault));
        *b->ilog_hint = 0;
    }
    if (!b->ilog_ev) RTD_CUDA(cudaEventCreateWithFlags(&b->ilog_ev, cudaEventDisableTiming));
    const cudaError_t q = cudaEventQuery(b->ilog_ev);
    if (q == cudaSuccess && *b->ilog_hint > b->ilog_pages) {
        const uint64_t want = (uint64_t)*b->ilog_hint + *b->ilog_hint / 16 + 64;
        RTD_TRY(b->ilog_entries.reserve(want * ILOG_PAGE * 32 * sizeof(uint2)));
        RTD_TRY(b->ilog_counts.reserve(want * ILOG_PAGE));
        RTD_TRY(b->ilog_next.reserve(want * sizeof(uint32_t)));
        b->ilog_pages = (uint32_t)want;
    } else if (q != cudaSuccess && q != cudaErrorNotReady) {
        return cuda_fail(q, "cudaEventQuery");
    }
    cudaGetLastError();   // a not-ready query leaves no error behind
    RTD_TRY(b->ilog_group.reserve(b->n * sizeof(uint2) + 64));
    BhHeader *h = b->hdr.as<BhHeader>();
    RTD_CUDA(cudaMemsetAsync(&h->ilog_used, 0, 2 * sizeof(uint32_t), st));
    lg.entries = b->ilog_entries.as<uint2>();
    lg.counts = b->ilog_counts.as<uint8_t>();
    lg.next = b->ilog_next.as<uint32_t>();
    lg.group = b->ilog_group.as<uint2>();
    lg.pages = b->ilog_pages;
    return RTD_OK;
}

rtd_status bh_forward(rtd_bh *b, const rtd_bh_params *p, float *d_out, float *d_phi,
                      cudaStream_t st) {
    if (!b || !b->built) return fail(RTD_ERR_INVALID_ARGUMENT, "bh tree not built");
    if (b->n && !d_out) return fail(RTD_ERR_INVALID_ARGUMENT, "NULL output");
    rtd_bh_params def;
    rtd_bh_params_default(&def);
    if (!p) p = &def;
    if (b->n == 0) return RTD_OK;
    if (p->law == RTD_BH_LAW_REFERENCE) return bh_ref_forward(b, p, d_out, st);
    if (p->law != RTD_BH_LAW_PLUMMER) return fail(RTD_ERR_INVALID_ARGUMENT, "unknown law");
    if (!b->plummer_ready)
        return fail(RTD_ERR_INVALID_ARGUMENT, "tree was not built for the Plummer law");
    if (p->quadrupole && !b->has_quad)
        return fail(RTD_ERR_INVALID_ARGUMENT, "tree was built without quadrupoles");
    IlogView lg{};
    if (b->backward_seen) RTD_TRY(ilog_prepare(b, st, lg));
    b->ilog_valid = false;
    if (p->quadrupole) RTD_TRY((launch_walk<true, false>(b, p, nullptr, nullptr, d_out, d_phi, lg, st)));
    else RTD_TRY((launch_walk<false, false>(b, p, nullptr, nullptr, d_out, d_phi, lg, st)));
    if (lg.group) {
        // the pages this forward needed, for sizing the next one's pool
        RTD_CUDA(cudaMemcpyAsync(b->ilog_hint, &b->hdr.as<BhHeader>()->ilog_need, sizeof(uint32_t),
                                 cudaMemcpyDeviceToHost, st));
        RTD_CUDA(cudaEventRecord(b->ilog_ev, st));
        b->ilog_valid = lg.pages > 0;
        b->ilog_theta = p->theta;
        b->ilog_quad = p->quadrupole;
    }
    return RTD_OK;
}

rtd_status bh_backward(rtd_bh *b, const rtd_bh_params *p, const float *g_acc, const float *g_phi,
                       float *g_pos, float *g_mass, cudaStream_t st) {
    if (!b || !b->built) return fail(RTD_ERR_INVALID_ARGUMENT, "bh tree not built");
    rtd_bh_params def;
    rtd_bh_params_default(&def);
    if (!p) p = &def;
    if (p->law != RTD_BH_LAW_PLUMMER)
        return fail(RTD_ERR_UNSUPPORTED, "the adjoint is defined for the Plummer law");
    if (b->n == 0) return RTD_OK;
    if (!g_acc || !g_pos) return fail(RTD_ERR_INVALID_ARGUMENT, "NULL gradient buffer");
    if (!b->plummer_ready)
        return fail(RTD_ERR_INVALID_ARGUMENT, "tree was not built for the Plummer law");
    if (p->quadrupole && !b->has_quad)
        return fail(RTD_ERR_INVALID_ARGUMENT, "tree was built without quadrupoles");
    const uint64_t n = b->n;
    const uint64_t cells = b->node_cap;
    RTD_TRY(b->cell_grad.reserve(cells * 3 * sizeof(float4) + 64 * sizeof(uint32_t)));
    RTD_TRY(b->gpos_flat.reserve(n * sizeof(float4)));
    RTD_CUDA(cudaMemsetAsync(b->cell_grad.ptr, 0, cells * 3 * sizeof(float4), st));
    RTD_CUDA(cudaMemsetAsync(b->gpos_flat.ptr, 0, n * sizeof(float4), st));
    // replay the last forward's interaction log when it was taken on this
    // tree with these parameters; otherwise walk
    IlogView lg{};
    if (b->ilog_valid && b->ilog_theta == p->theta && b->ilog_quad == p->quadrupole) {
        lg.entries = b->ilog_entries.as<uint2>();
        lg.counts = b->ilog_counts.as<uint8_t>();
        lg.next = b->ilog_next.as<uint32_t>();
        lg.group = b->ilog_group.as<uint2>();
        lg.pages = b->ilog_pages;
    }
    b->backward_seen = true;
    if (p->quadrupole) RTD_TRY((launch_walk<true, true>(b, p, g_acc, g_phi, nullptr, nullptr, lg, st)));
    else RTD_TRY((launch_walk<false, true>(b, p, g_acc, g_phi, nullptr, nullptr, lg, st)));
    const BhView v = bh_view(b);
    bh_constants_kernel<<<grid_for(n, 256, 148 * 8), 256, 0, st>>>(v, b->cell_grad.as<float4>());
    RTD_LAUNCH_CHECK();
    bh_finish_grad_kernel<<<grid_for(cells, 4, 148 * 64), 128, 0, st>>>(
        v, b->cell_grad.as<float>(), b->gpos_flat.as<float4>(), g_pos, g_mass);
    RTD_LAUNCH_CHECK();
    return RTD_OK;
}

namespace {

// Forward walk on a traversal stack supplied by the caller: `stack` holds
// max_warps slices of BH_STACK_CAP_MAX entries and the launch is capped to that
// many warps.  Nothing is allocated.
template <bool QUAD, int SPLIT>
rtd_status launch_walk_on_stack(rtd_bh *b, const rtd_bh_params *p, float *acc, float *phi,
                                uint2 *stack, uint64_t max_warps, cudaStream_t st) {
    int dev = 0, sms = 148, per_sm = 4;
    RTD_CUDA(cudaGetDevice(&dev));
    RTD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    RTD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bh_walk_kernel<QUAD, false, SPLIT>,
                                                           WW * 32, 0));
    if (per_sm < 1) per_sm = 1;
    uint64_t blocks = (uint64_t)sms * (uint64_t)per_sm;
    const uint64_t need = ceil_div(ceil_div(b->n, BH_GROUP) * SPLIT, WW);
    if (blocks > need) blocks = need;
    if (blocks > max_warps / WW) blocks = max_warps / WW;
    if (blocks < 1) return fail(RTD_ERR_INVALID_ARGUMENT, "stack holds less than one block of warps");
    BhHeader *h = b->hdr.as<BhHeader>();
    RTD_CUDA(cudaMemsetAsync(&h->group_counter, 0, sizeof(uint32_t), st));
    const BhView v = bh_view(b);
    bh_walk_kernel<QUAD, false, SPLIT><<<(unsigned)blocks, WW * 32, 0, st>>>(
        v, p->theta * p->theta, p->eps * p->eps, p->G, nullptr, nullptr, acc, phi, nullptr,
        nullptr, stack, bh_stack_entries(), IlogView{}, h);
    RTD_LAUNCH_CHECK();
    return RTD_OK;
}

}  // namespace

// Plummer-law forward walk with the traversal stack given by the caller
// (max_warps slices of BH_STACK_CAP_MAX uint2 entries); same checks and results
// as bh_forward for the Plummer law.
rtd_status bh_forward_on_stack(rtd_bh *b, const rtd_bh_params *p, float *d_out, float *d_phi,
                               uint2 *stack, uint64_t max_warps, cudaStream_t st) {
    if (!b || !b->built) return fail(RTD_ERR_INVALID_ARGUMENT, "bh tree not built");
    if (b->n && !d_out) return fail(RTD_ERR_INVALID_ARGUMENT, "NULL output");
    if (!stack) return fail(RTD_ERR_INVALID_ARGUMENT, "NULL stack");
    rtd_bh_params def;
    rtd_bh_params_default(&def);
    if (!p) p = &def;
    if (p->law != RTD_BH_LAW_PLUMMER)
        return fail(RTD_ERR_UNSUPPORTED, "this walk implements the Plummer law only");
    if (b->n == 0) return RTD_OK;
    if (!b->plummer_ready)
        return fail(RTD_ERR_INVALID_ARGUMENT, "tree was not built for the Plummer law");
    if (p->quadrupole && !b->has_quad)
        return fail(RTD_ERR_INVALID_ARGUMENT, "tree was built without quadrupoles");
    if (split_groups(b->n))
        return p->quadrupole ? launch_walk_on_stack<true, WW>(b, p, d_out, d_phi, stack, max_warps, st)
                             : launch_walk_on_stack<false, WW>(b, p, d_out, d_phi, stack, max_warps, st);
    return p->quadrupole ? launch_walk_on_stack<true, 1>(b, p, d_out, d_phi, stack, max_warps, st)
                         : launch_walk_on_stack<false, 1>(b, p, d_out, d_phi, stack, max_warps, st);
}

}  // namespace rtd

namespace rtd {
namespace {

// Interaction counts of the Plummer walk for every stride-th flat body: the
// same per-body MAC over the pre-order tree (autoropes), counting accepted
// cells and the bodies of opened leaves.  out[0] += cells, out[1] += bodies.
__global__ void bh_count_kernel(const BhView v, float theta2, uint64_t stride,
                                unsigned long long *out) {
    const uint32_t n_nodes = v.hdr->n_nodes;
    unsigned long long cells = 0, bodies = 0;
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s * stride < v.n;
         s += (uint64_t)gridDim.x * blockDim.x) {
        const float4 me = v.fbody[s * stride];
        uint32_t p = 0;
        while (p < n_nodes) {
            const float4 a = __ldg(&v.node_a[p]);
            const uint4 b = __ldg(&v.node_b[p]);
            if (body_accept(me.x, me.y, me.z, a.x, a.y, a.z, __uint_as_float(b.w), theta2)) {
                ++cells;
                p = b.x;
            } else {
                if (b.z & BH_LEAF_BIT) bodies += b.z & ~BH_LEAF_BIT;
                ++p;
            }
        }
    }
    atomicAdd(&out[0], cells);
    atomicAdd(&out[1], bodies);
}

}  // namespace

rtd_status bh_interaction_counts(rtd_bh *b, float theta, uint64_t stride, uint64_t *h_cells,
                                 uint64_t *h_bodies, uint64_t *h_sampled, cudaStream_t st) {
    if (!b || !b->built) return fail(RTD_ERR_INVALID_ARGUMENT, "bh tree not built");
    if (stride < 1) return fail(RTD_ERR_INVALID_ARGUMENT, "stride must be >= 1");
    RTD_TRY(b->cell_grad.reserve(2 * sizeof(unsigned long long)));
    unsigned long long *d = b->cell_grad.as<unsigned long long>();
    RTD_CUDA(cudaMemsetAsync(d, 0, 2 * sizeof(unsigned long long), st));
    const uint64_t ns = b->n ? (b->n + stride - 1) / stride : 0;
    if (ns) {
        bh_count_kernel<<<grid_for(ns, 128, 148 * 8), 128, 0, st>>>(bh_view(b), theta * theta,
                                                                     stride, d);
        RTD_LAUNCH_CHECK();
    }
    unsigned long long h[2] = {0, 0};
    RTD_CUDA(cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, st));
    RTD_CUDA(cudaStreamSynchronize(st));
    if (h_cells) *h_cells = h[0];
    if (h_bodies) *h_bodies = h[1];
    if (h_sampled) *h_sampled = ns;
    return RTD_OK;
}

}  // namespace rtd
