// knn_backward.cuh -- gradient of the squared distances of one query's
// neighbours, shared by the single-cloud and the batched backward passes.
//
// d2_j = |q - p_j|^2: dL/dq = sum_j 2 g_j (q - p_j), dL/dp_j -= 2 g_j (q - p_j).
// T lanes take a query (T = k rounded up to a power of two, at most 32), so
// ids and upstream gradients are read in order, and sum dL/dq in FP64 by
// shuffles (in FP32, a tree of rounded products was less exact than one
// lane's chain of FMAs; the FP64 sums cost nothing beside the atomics).
// Bound by the atomics on dL/dp, one row of three floats a neighbour at a
// random place: two components that share an aligned 8 bytes go in one.
#pragma once

#include "index.cuh"

namespace rtd {

__host__ __device__ inline uint32_t backward_lanes(uint32_t k) {
    uint32_t T = 1;
    while (T < k && T < 32) T <<= 1;
    return T;
}

// Whether pairs of components of the rows of gp can be added together.
__device__ __forceinline__ bool backward_pairs(const float *gp) {
    return (reinterpret_cast<uintptr_t>(gp) & 7u) == 0;
}

// The T lanes of query i (all lanes of the warp take part; have: whether
// this lane's query exists).  ids, g: the query's rows; n: points.
__device__ __forceinline__ void backward_query(bool have, const float *__restrict__ q, const float *__restrict__ pts,
                                               uint64_t n, uint32_t k, const uint32_t *__restrict__ ids,
                                               const float *__restrict__ g, float *__restrict__ gq,
                                               float *__restrict__ gp, uint64_t i, uint32_t T, bool pairs) {
    const uint32_t sub = (threadIdx.x & 31) % T;
    double ax = 0.0, ay = 0.0, az = 0.0;
    if (have) {
        const float qx = q[3 * i], qy = q[3 * i + 1], qz = q[3 * i + 2];
        for (uint32_t j = sub; j < k; j += T) {
            const uint64_t id = ids[j];
            if (id == EMPTY_ID || id >= n) continue;
            const float w = 2.0f * g[j];
            const float dx = qx - pts[3 * id], dy = qy - pts[3 * id + 1], dz = qz - pts[3 * id + 2];
            ax += (double)w * dx; ay += (double)w * dy; az += (double)w * dz;
            if (gp) {
                float *to = gp + 3 * id;
                if (!pairs) {
                    atomicAdd(to, -w * dx);
                    atomicAdd(to + 1, -w * dy);
                    atomicAdd(to + 2, -w * dz);
                } else if (id & 1) {   // the row starts 4 bytes past an aligned 8
                    atomicAdd(to, -w * dx);
                    atomicAdd(reinterpret_cast<float2 *>(to + 1), make_float2(-w * dy, -w * dz));
                } else {
                    atomicAdd(reinterpret_cast<float2 *>(to), make_float2(-w * dx, -w * dy));
                    atomicAdd(to + 2, -w * dz);
                }
            }
        }
    }
    for (uint32_t o = T / 2; o > 0; o >>= 1) {
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
        ay += __shfl_xor_sync(0xffffffffu, ay, o);
        az += __shfl_xor_sync(0xffffffffu, az, o);
    }
    if (have && sub == 0 && gq) {
        gq[3 * i] = (float)ax;
        gq[3 * i + 1] = (float)ay;
        gq[3 * i + 2] = (float)az;
    }
}

}  // namespace rtd
