// One block a row whose values stay in registers between the passes of a norm: NV groups of four neighbouring columns a thread.
// What bounds such a kernel in a decode step is a chain of latencies, so it is kept short: weights, which no kernel
// writes, are asked for before the kernel ahead is waited for (between two steps the layers' matrices have driven them out of L2),
// the row's operands come together in 16-byte loads, and a sum over the block takes one barrier.  Rows in shared memory, weights
// loaded behind the sums and three barriers a sum took, for 4 to 8 rows of 2,048, 3.8 us (RMS norm behind a scaled sum), 5.2 (a layer norm
// added, a second behind it) and 8.4 us (layer norm with token shift) of a recorded step; now 2.1, 3.2 and 2.9.
#pragma once
#include "common.cuh"

constexpr int kRowMaxWarps = 16;

// Threads and groups a thread for ``rows`` rows of ``hidden`` columns; nv 0: not for these kernels.  In bf16 many wide rows are bound by memory
// and want more of them on an SM than the registers of these kernels leave room for (2,048 rows of 4,096: 21.0 against 20.4 us
// with the row in shared memory, of 2,048 11.7 against 10.9; of 1,024 6.1 against 6.3; 512 of 8,192 8.9 against 7.3).  In 32-bit the
// width alone decides, so that a row's sum runs in one order whatever else is in the step.
struct RowShape { int threads, nv; };
static inline RowShape row_shape(int64_t rows, int hidden, int most_nv, bool f32) {
    if (hidden < 4 || hidden % 4 || hidden > 4 * 32 * kRowMaxWarps * most_nv) return {0, 0};
    if (f32 ? hidden > 4096 : (rows > 512 && hidden >= 2048) || (rows > 200 && hidden > 4096)) return {0, 0};
    const int quads = hidden / 4, warps = (quads + 31) / 32, threads = 32 * (warps < kRowMaxWarps ? warps : kRowMaxWarps);
    const int nv = (quads + threads - 1) / threads;
    return {threads, nv == 3 ? 4 : nv};
}

// Sums over the block, one barrier; ``scratch`` (16 floats a sum) is not to be used again before another barrier.
__device__ __forceinline__ float row_sum(float v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    return warp_sum(lane < (int)(blockDim.x >> 5) ? scratch[lane] : 0.f);
}
__device__ __forceinline__ float2 row_sum2(float2 v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v.x = warp_sum(v.x);
    v.y = warp_sum(v.y);
    if (lane == 0) {
        scratch[warp] = v.x;
        scratch[kRowMaxWarps + warp] = v.y;
    }
    __syncthreads();
    const bool in = lane < (int)(blockDim.x >> 5);
    return make_float2(warp_sum(in ? scratch[lane] : 0.f), warp_sum(in ? scratch[kRowMaxWarps + lane] : 0.f));
}

// Column of a thread's i-th group; a group past the row's end is skipped by row_in.
__device__ __forceinline__ int row_col(int i) { return 4 * (threadIdx.x + i * blockDim.x); }

template <int NV, typename P>
__device__ __forceinline__ void row_load(float4 (&v)[NV], const P* p, int hidden) {
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = p != nullptr && row_col(i) < hidden ? load4(p + row_col(i)) : make_float4(0.f, 0.f, 0.f, 0.f);
}
template <int NV, typename P>
__device__ __forceinline__ void row_store(P* p, const float4 (&v)[NV], int hidden) {
#pragma unroll
    for (int i = 0; i < NV; ++i)
        if (row_col(i) < hidden) store4(p + row_col(i), v[i]);
}
__device__ __forceinline__ float quad_sum(float4 v) { return (v.x + v.y) + (v.z + v.w); }
__device__ __forceinline__ float quad_squares(float4 v, float s) { return fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, s)))); }
__device__ __forceinline__ float4 quad_fma(float a, float4 x, float4 y) {
    return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}
// (v * r) * w (+ b)
__device__ __forceinline__ float4 quad_scaled(float4 v, float r, float4 w) { return make_float4(v.x * r * w.x, v.y * r * w.y, v.z * r * w.z, v.w * r * w.w); }
__device__ __forceinline__ float4 quad_add(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// The row minus its mean, in place; returns 1 / sqrt(mean of the squared deviations + eps).  scratch: 32 floats.
template <int NV>
__device__ __forceinline__ float row_centre(float4 (&v)[NV], int hidden, float eps, float* scratch) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) s += quad_sum(v[i]);
    const float mean = row_sum(s, scratch) / (float)hidden;
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        v[i] = make_float4(v[i].x - mean, v[i].y - mean, v[i].z - mean, v[i].w - mean);
        if (row_col(i) < hidden) q = quad_squares(v[i], q);
    }
    return 1.0f / sqrtf(row_sum(q, scratch + kRowMaxWarps) / (float)hidden + eps);
}

