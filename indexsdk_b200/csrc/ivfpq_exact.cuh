// Canonical distance of a stored vector to a query: the arithmetic of the CPU oracle.  Args: a scan's
// arguments (codes, rotated, M, d, dsub, codebooks, centroids, xq, by_residual).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace b200 {

constexpr int kPqCodes = 256;

// Byte offset of sub-quantizer m inside the stored code of the vector at `pos`.
__device__ __forceinline__ int code_byte(bool rotated, int m, int64_t pos) {
    return rotated ? ((m & ~15) | ((m - static_cast<int>(pos & 15)) & 15)) : m;
}

// The 16 bytes of a group of stored codes, turned back to canonical order: canonical byte m is stored byte
// (m - position) mod 16, so word j starts at stored byte (4 j - position) mod 16.
__device__ __forceinline__ uint4 unrotate_group(uint4 v, uint32_t pos) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const uint32_t first = (16u - (pos & 15u)) & 15u, a = first >> 2, sh = 8u * (first & 3u);
    uint32_t r[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t x = (a + j) & 3u, y = (a + j + 1u) & 3u;
        const uint32_t lo = x == 0u ? w[0] : x == 1u ? w[1] : x == 2u ? w[2] : w[3];
        const uint32_t hi = y == 0u ? w[0] : y == 1u ? w[1] : y == 2u ? w[2] : w[3];
        r[j] = __funnelshift_r(lo, hi, sh);
    }
    return make_uint4(r[0], r[1], r[2], r[3]);
}

// exact_distance for rotated codes and short sub-vectors: a group's codes are one 16-byte load, and the
// codewords of four sub-quantizers are on their way together (one after the other, code byte then
// codeword, the loop is a chain of 2 M memory latencies).  Sub-vectors of 8 keep the plain loop: 96 floats
// on their way cost the warp kernel the occupancy that hides its latency (69 -> 76 us at M = 16).
template <int DS, typename Args>
__device__ __forceinline__ float exact_distance_rotated(const Args& a, const float* qv, const float* cen, int64_t pos,
                                                        bool resid) {
    using V = typename std::conditional<DS == 2, float2, float4>::type;
    constexpr int E = DS == 2 ? 2 : 4, NV = DS / E;   // floats per load, loads per sub-vector
    float acc = 0.f;
    for (int g = 0; g < a.M / 16; ++g) {
        const uint4 c = unrotate_group(__ldg(reinterpret_cast<const uint4*>(a.codes + pos * a.M) + g), static_cast<uint32_t>(pos));
        const uint32_t cw[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            V w[4][NV], q[4][NV], r[4][NV];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int m = g * 16 + b * 4 + u;
                const uint32_t code = (cw[b] >> (8 * u)) & 255u;
                const V* src = reinterpret_cast<const V*>(a.codebooks + (static_cast<size_t>(m) * kPqCodes + code) * DS);
#pragma unroll
                for (int t = 0; t < NV; ++t) {
                    w[u][t] = __ldg(src + t);
                    q[u][t] = __ldg(reinterpret_cast<const V*>(qv + m * DS) + t);
                    if (resid) r[u][t] = __ldg(reinterpret_cast<const V*>(cen + m * DS) + t);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float e = 0.f;
#pragma unroll
                for (int t = 0; t < NV; ++t) {
                    const float* wf = reinterpret_cast<const float*>(&w[u][t]);
                    const float* qf = reinterpret_cast<const float*>(&q[u][t]);
                    const float* rf = reinterpret_cast<const float*>(&r[u][t]);
#pragma unroll
                    for (int x = 0; x < E; ++x) {
                        float v = qf[x];
                        if (resid) v -= rf[x];
                        const float df = v - wf[x];
                        e = fmaf(df, df, e);
                    }
                }
                acc = acc + e;
            }
        }
    }
    return acc;
}

// Canonical distance of the vector at `pos` (probed through list `list`): sum over m, in
// ascending m, of |(q - c_list)_m - cb[m][code_m]|^2 accumulated with sequential fmaf over the
// sub-vector (c_list = 0 for raw encoding).  Rows are read as float4 where the sub-vector length
// allows: the survivors of a query live in unrelated lists, so every lane streams its own
// centroid row and codewords, and wide loads keep the number of cache transactions down.
template <typename Args>
__device__ __forceinline__ float exact_distance(const Args& a, int64_t q, int64_t pos, int64_t list) {
    const uint8_t* code = a.codes + pos * a.M;
    const float* qv = a.xq + q * a.d;
    const float* cen = a.centroids + list * a.d;
    const bool resid = a.by_residual != 0;
    float acc = 0.f;
    if (a.rotated) {
        switch (a.dsub) {
            case 2: return exact_distance_rotated<2>(a, qv, cen, pos, resid);
            case 4: return exact_distance_rotated<4>(a, qv, cen, pos, resid);
            default: break;
        }
    }
    if ((a.dsub & 3) == 0) {
        const int d4 = a.dsub >> 2;
        const float4* q4 = reinterpret_cast<const float4*>(qv);
        const float4* c4 = reinterpret_cast<const float4*>(cen);
        for (int m = 0; m < a.M; ++m) {
            const float4* w4 = reinterpret_cast<const float4*>(
                a.codebooks + (static_cast<int64_t>(m) * kPqCodes + code[code_byte(a.rotated != 0, m, pos)]) * a.dsub);
            float e = 0.f;
            for (int t = 0; t < d4; ++t) {
                float4 r = __ldg(q4 + m * d4 + t);
                if (resid) {
                    const float4 c = __ldg(c4 + m * d4 + t);
                    r.x -= c.x; r.y -= c.y; r.z -= c.z; r.w -= c.w;
                }
                const float4 w = __ldg(w4 + t);
                float df;
                df = r.x - w.x; e = fmaf(df, df, e);
                df = r.y - w.y; e = fmaf(df, df, e);
                df = r.z - w.z; e = fmaf(df, df, e);
                df = r.w - w.w; e = fmaf(df, df, e);
            }
            acc = acc + e;
        }
        return acc;
    }
    for (int m = 0; m < a.M; ++m) {
        const float* cw = a.codebooks +
                          (static_cast<int64_t>(m) * kPqCodes + code[code_byte(a.rotated != 0, m, pos)]) * a.dsub;
        float e = 0.f;
        for (int t = 0; t < a.dsub; ++t) {
            float r = qv[m * a.dsub + t];
            if (resid) r -= cen[m * a.dsub + t];
            const float df = r - cw[t];
            e = fmaf(df, df, e);
        }
        acc = acc + e;
    }
    return acc;
}

}  // namespace b200
