// C[M,N] = alpha * A[M,K] * W[N,K]^T in true fp32: fp32 operands, fp32 FMA, no
// tensor cores and no reduced-precision matrix mode.  It is the matrix product of
// the 32-bit path (the reference has only 16-bit instantiations and cuBLAS,
// src/model/linear.cuh:8-37).
//
// The sum over K runs in one order for every output, whatever M and N are and whichever kernel takes the shape: K is cut
// into slices of 64, a slice is summed by FMAs in rising k from zero, and the slices' sums are added in rising order.  A
// row's result therefore does not depend on what else is in the batch.  The slices are what lets the two kernels share the
// work of an output among threads (few rows) or not (many) and still agree to the last bit.
//
// Two kernels, by rows:
//   up to 16 rows (decode): bound by streaming the weights; a block owns 8 weight rows, a thread one slice of one of them for
//     all token rows.  Weight pieces of 1,024 columns come by 16-byte cp.async three stages deep, each slice padded by four
//     floats so that the 16-byte reads of a quarter warp (8 rows) fall into 8 different bank groups.
//   more rows: 64 x 64 tiles, 128 threads with 8 x 4 outputs each.  Both operands stay K-major in shared memory as they lie
//     in global memory (rows padded to 36 floats: conflict-free 16-byte reads along K, no transposition), 32 columns a stage,
//     three stages by cp.async.  12 shared reads of 16 bytes per 128 FMAs a thread.
// Where K is no multiple of 4 or a pointer is not 16-byte aligned the same kernels load element by element.
//
// Measured on one B200 at the 0.5B layer sizes, 24 layers, three prompts of 453 tokens together and four decoded tokens:
// all products 19.1 ms (a decode step's 0.79 ms, the output head's 300 MB included; the prompts' 15.9 ms, 21 TFLOP/s) against
// 106 ms with one 64 x 64 tile kernel of scalar loads for every shape, which kept 16 of its 64 rows busy at most in a
// decode step and summed all of K in one chain (its error against 64 bits was three times as large).
#include "common.cuh"

constexpr int kSliceK = 64;

__device__ __forceinline__ void f32_cp_async_16(float* dst, const float* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void f32_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void f32_cp_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// Four columns [k, k+4) of a row into shared memory, zeros beyond the row's end or where ``row_ok`` is false.
template <bool VEC>
__device__ __forceinline__ void f32_stage4(float* dst, const float* row, int k, int K, bool row_ok) {
    if (VEC) {
        const bool ok = row_ok && k < K;                       // K is a multiple of 4
        f32_cp_async_16(dst, ok ? row + k : row, ok);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = (row_ok && k + i < K) ? row[k + i] : 0.f;
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// up to 16 rows
// ---------------------------------------------------------------------------------------------------------------------
constexpr int kFewRowsN = 8, kFewSlices = 16, kFewPad = kSliceK + 4, kFewStages = 3;
constexpr int kFewChunk = kFewSlices * kSliceK;                       // columns a stage
constexpr int kFewRowStride = kFewSlices * kFewPad + 4;               // floats between weight rows: 4 mod 32
constexpr int kFewThreads = kFewRowsN * kFewSlices;

// token rows that are staged beside the weights (MT: rows a thread sums, M rounded up to 1, 2, 4, 8 or 16)
template <int MT> constexpr int few_stage_floats() { return kFewRowsN * kFewRowStride + MT * kFewSlices * kFewPad; }
template <int MT> constexpr int few_stages() { return MT > 8 ? 2 : kFewStages; }
template <int MT> constexpr int few_red_floats() { return kFewSlices * kFewRowsN * (MT + 1); }
template <int MT> constexpr size_t few_smem(int stages) {
    return ((size_t)stages * few_stage_floats<MT>() + few_red_floats<MT>()) * sizeof(float);
}

template <int MT, bool VEC>
__global__ void __launch_bounds__(kFewThreads)
gemm_f32_few_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                         int64_t lda, int64_t ldw, int64_t ldc, float alpha) {
    extern __shared__ float red[];                                    // [slice][row][MT + 1], then the stages
    constexpr int STAGES = few_stages<MT>();
    float* stages = red + few_red_floats<MT>();
    const int tid = threadIdx.x, row = tid & 7, slice = tid >> 3;
    const int n0 = blockIdx.x * kFewRowsN;
    const int chunks = (K + kFewChunk - 1) / kFewChunk;

    auto stage = [&](int c) {
        float* ws = stages + (c % STAGES) * few_stage_floats<MT>();
        float* xs = ws + kFewRowsN * kFewRowStride;
        const int k0 = c * kFewChunk;
        for (int i = tid; i < kFewRowsN * (kFewChunk / 4); i += kFewThreads) {       // a row's 4,096 bytes by 256 neighbours
            const int r = i / (kFewChunk / 4), k = 4 * (i % (kFewChunk / 4));
            f32_stage4<VEC>(ws + r * kFewRowStride + (k / kSliceK) * kFewPad + k % kSliceK,
                            W + (int64_t)min(n0 + r, N - 1) * ldw, k0 + k, K, n0 + r < N);
        }
        for (int i = tid; i < MT * (kFewChunk / 4); i += kFewThreads) {
            const int m = i / (kFewChunk / 4), k = 4 * (i % (kFewChunk / 4));
            f32_stage4<VEC>(xs + (m * kFewSlices + k / kSliceK) * kFewPad + k % kSliceK,
                            A + (int64_t)min(m, M - 1) * lda, k0 + k, K, m < M);
        }
    };
#pragma unroll
    for (int c = 0; c < STAGES - 1; ++c) {
        if (c < chunks) stage(c);
        f32_cp_commit();
    }
    float total = 0.f;                                                // of output (row, m), by thread row + 8 * m
    for (int c = 0; c < chunks; ++c) {
        f32_cp_wait<STAGES - 2>();
        __syncthreads();                                              // stage c has arrived for all; stage c - 1 is free
        if (c + STAGES - 1 < chunks) stage(c + STAGES - 1);
        f32_cp_commit();
        const float* ws = stages + (c % STAGES) * few_stage_floats<MT>() + row * kFewRowStride + slice * kFewPad;
        const float* xs = stages + (c % STAGES) * few_stage_floats<MT>() + kFewRowsN * kFewRowStride + slice * kFewPad;
        float acc[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[m] = 0.f;
#pragma unroll 4
        for (int k = 0; k < kSliceK; k += 4) {
            const float4 w = *reinterpret_cast<const float4*>(ws + k);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4 x = *reinterpret_cast<const float4*>(xs + m * kFewSlices * kFewPad + k);
                acc[m] = fmaf(x.x, w.x, acc[m]);
                acc[m] = fmaf(x.y, w.y, acc[m]);
                acc[m] = fmaf(x.z, w.z, acc[m]);
                acc[m] = fmaf(x.w, w.w, acc[m]);
            }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m) red[(slice * kFewRowsN + row) * (MT + 1) + m] = acc[m];
        __syncthreads();
        // 8 x 16 outputs at most: one a thread, slices in rising order
        const int n_slices = min(kFewSlices, (K - c * kFewChunk + kSliceK - 1) / kSliceK);
        if (tid < kFewRowsN * MT)
            for (int s = 0; s < n_slices; ++s) total += red[(s * kFewRowsN + row) * (MT + 1) + (tid >> 3)];
    }
    const int m = tid >> 3;
    if (m < M && m < MT && n0 + row < N) C[(int64_t)m * ldc + n0 + row] = alpha * total;
}

// ---------------------------------------------------------------------------------------------------------------------
// more rows
// ---------------------------------------------------------------------------------------------------------------------
constexpr int BM = 64, BN = 64, BK = 32, kTilePad = BK + 4, kTileStages = 3, kTileThreads = 128;
constexpr size_t kTileSmem = (size_t)kTileStages * (BM + BN) * kTilePad * sizeof(float);

template <bool VEC>
__global__ void __launch_bounds__(kTileThreads)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                     int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc, float alpha) {
    extern __shared__ float tile_smem[];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;          // outputs (ty + 8 i, tx + 16 j)
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int steps = (K + BK - 1) / BK;
    auto stage = [&](int s) {
        float* as = tile_smem + (s % kTileStages) * (BM + BN) * kTilePad;
        float* bs = as + BM * kTilePad;
        const int k0 = s * BK;
#pragma unroll
        for (int i = 0; i < BM * (BK / 4) / kTileThreads; ++i) {
            const int e = tid + kTileThreads * i, r = e / (BK / 4), k = 4 * (e % (BK / 4));
            f32_stage4<VEC>(as + r * kTilePad + k, A + (int64_t)min(m0 + r, M - 1) * lda, k0 + k, K, m0 + r < M);
            f32_stage4<VEC>(bs + r * kTilePad + k, W + (int64_t)min(n0 + r, N - 1) * ldw, k0 + k, K, n0 + r < N);
        }
    };
#pragma unroll
    for (int s = 0; s < kTileStages - 1; ++s) {
        if (s < steps) stage(s);
        f32_cp_commit();
    }
    float total[8][4], acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) total[i][j] = acc[i][j] = 0.f;
    for (int s = 0; s < steps; ++s) {
        f32_cp_wait<kTileStages - 2>();
        __syncthreads();
        if (s + kTileStages - 1 < steps) stage(s + kTileStages - 1);
        f32_cp_commit();
        const float* as = tile_smem + (s % kTileStages) * (BM + BN) * kTilePad + ty * kTilePad;
        const float* bs = tile_smem + (s % kTileStages) * (BM + BN) * kTilePad + BM * kTilePad + tx * kTilePad;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(bs + 16 * j * kTilePad + k);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(as + 8 * i * kTilePad + k);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
                    acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
                    acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
                    acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
                }
            }
        }
        if ((s + 1) % (kSliceK / BK) == 0 || s + 1 == steps) {           // a slice is complete
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    total[i][j] += acc[i][j];
                    acc[i][j] = 0.f;
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty + 8 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx + 16 * j;
            if (n < N) C[(int64_t)m * ldc + n] = alpha * total[i][j];
        }
    }
}

template <int MT, bool VEC>
static int launch_few_rows(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc,
                           float alpha, cudaStream_t stream) {
    static bool done[kMaxDevices];
    const int rc = ensure_dynamic_smem(gemm_f32_few_rows_kernel<MT, VEC>, (int)few_smem<MT>(few_stages<MT>()), done);
    if (rc != CPM_OK) return rc;
    // a short K needs no more stages than it has pieces, and several blocks then fit an SM
    const int chunks = (K + kFewChunk - 1) / kFewChunk, stages = chunks < few_stages<MT>() ? chunks : few_stages<MT>();
    gemm_f32_few_rows_kernel<MT, VEC><<<(N + kFewRowsN - 1) / kFewRowsN, kFewThreads, few_smem<MT>(stages), stream>>>(
        A, W, C, M, N, K, lda, ldw, ldc, alpha);
    return launch_status();
}

template <bool VEC>
static int launch_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc,
                           float alpha, cudaStream_t stream) {
    if (M <= 1) return launch_few_rows<1, VEC>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
    if (M <= 2) return launch_few_rows<2, VEC>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
    if (M <= 4) return launch_few_rows<4, VEC>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
    if (M <= 8) return launch_few_rows<8, VEC>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
    if (M <= 16) return launch_few_rows<16, VEC>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
    static bool done[kMaxDevices];
    const int rc = ensure_dynamic_smem(gemm_f32_tile_kernel<VEC>, (int)kTileSmem, done);
    if (rc != CPM_OK) return rc;
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return CPM_BAD_ARGUMENT;
    gemm_f32_tile_kernel<VEC><<<grid, kTileThreads, kTileSmem, stream>>>(A, W, C, M, N, K, lda, ldw, ldc, alpha);
    return launch_status();
}

CPM_API int cpm_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda,
                         int64_t ldw, int64_t ldc, float alpha, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return CPM_OK;
    if (K <= 0) return CPM_BAD_ARGUMENT;
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    return vec ? launch_gemm_f32<true>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream)
               : launch_gemm_f32<false>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
}
