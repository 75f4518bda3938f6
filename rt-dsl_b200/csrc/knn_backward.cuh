// knn_backward.cuh -- gradient of the squared distances of one query's
// neighbours, shared by the single-cloud and the batched backward passes.
//
// d2_j = |q - p_j|^2: dL/dq = sum_j 2 g_j (q - p_j), dL/dp_j -= 2 g_j (q - p_j).
// A thread takes a query and its neighbours in order: the near ones, whose
// terms are small, are then added to dL/dp first.  With lanes across the
// neighbours all ranks arrive mixed, which is faster (50,000 queries, k = 16:
// 15 us; 256 clouds 1.18 ms for 1.57) but leaves dL/dp with a tenth more
// rounding error (7.9e-8 for 7.1e-8).  dL/dq is summed
// in FP64 (error 6.4e-8 -> 2.6e-8; it costs nothing beside the atomics).
// Bound by the atomics on dL/dp, one row of three floats a neighbour at a
// random place: two components that share an aligned 8 bytes go in one (24 ->
// 21 us).
#pragma once

#include "index.cuh"

namespace rtd {

// Whether pairs of components of the rows of gp can be added together.
__device__ __forceinline__ bool backward_pairs(const float *gp) {
    return (reinterpret_cast<uintptr_t>(gp) & 7u) == 0;
}

// Query i.  ids, g: the query's rows; n: points.
__device__ __forceinline__ void backward_query(const float *__restrict__ q, const float *__restrict__ pts, uint64_t n,
                                               uint32_t k, const uint32_t *__restrict__ ids,
                                               const float *__restrict__ g, float *__restrict__ gq,
                                               float *__restrict__ gp, uint64_t i, bool pairs) {
    double ax = 0.0, ay = 0.0, az = 0.0;
    const float qx = q[3 * i], qy = q[3 * i + 1], qz = q[3 * i + 2];
    for (uint32_t j = 0; j < k; ++j) {
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
    if (gq) {
        gq[3 * i] = (float)ax;
        gq[3 * i + 1] = (float)ay;
        gq[3 * i + 2] = (float)az;
    }
}

}  // namespace rtd
