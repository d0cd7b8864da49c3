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
// Two kernels, by rows (and K):
//   up to 16 rows (decode): bound by streaming the weights; a block owns 8 weight rows, a thread one slice of one of them for
//     all token rows.  Weight pieces of 1,024 columns come by 16-byte cp.async three stages deep, each slice padded by four
//     floats so that the 16-byte reads of a quarter warp (8 rows) fall into 8 different bank groups.
//   more rows: tiles of 64, 80 or 96 rows times 64 columns, one block of four groups of 64 threads an SM.  A group sums every fourth
//     slice of the whole tile, a thread 8, 10 or 12 rows of 8 columns: a shared read of 16 bytes takes an SM as long as 16
//     FMAs of a thread, so 8 x 8 outputs (16 reads per 256 FMAs) are the least that does not wait for them.  Both operands stay K-major in
//     shared memory as they lie in global memory (rows padded to 20 floats: conflict-free 16-byte reads along K, no
//     transposition), 16 columns a stage, two stages a group by cp.async.  After each round of four slices the groups trade: each
//     keeps the totals of two of a thread's columns and adds the four groups' sums of them in the order of the slices.
//     The number of rows is the one whose tiles fill the SMs' rounds best.  Where K is one or two slices, from 9 rows on, a block is one such
//     group and takes 64 or 32 rows.
// Where K is no multiple of 4 or a pointer is not 16-byte aligned the same kernels load element by element.
//
// Measured on one B200 at the 0.5B layer sizes, 24 layers, prompts of 400, 141 and 50 tokens together and four decoded tokens:
// all products 16.9 ms (a decode step's 0.79 ms, the output head's 300 MB included; the prompts' 13.6 ms, about half of what the
// FMA units give; the down product of 591 rows 168 us).  One 64 x 64 tile kernel of scalar loads for every shape took 106 ms, kept
// 16 of its 64 rows busy at most in a decode step and summed all of K in one chain (its error against 64 bits was three times
// as large).  Tiles of 64 x 64 with one group of 128 threads, 8 x 4 outputs each, took 15.9 ms for the prompts (the down product
// 257 us: 160 tiles of one warp a scheduler, 12 shared reads per 128 FMAs).
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
constexpr int BN = 64, BK = 16, kTilePad = BK + 4, kGroups = 4, kGroupThreads = 64;
template <int RI> constexpr int tile_stage_floats() { return (8 * RI + BN) * kTilePad; }
template <int NG> constexpr int tile_stages() { return NG == 1 ? 4 : 2; }
template <int RI, int NG> constexpr size_t tile_smem_bytes() {
    return (size_t)(NG * tile_stages<NG>() * tile_stage_floats<RI>() + (NG == 1 ? 0 : NG * RI * 8 * kGroupThreads)) * sizeof(float);
}

template <bool VEC, int RI, int NG>
__global__ void __launch_bounds__(NG * kGroupThreads, 1)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                     int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc, float alpha) {
    extern __shared__ float tile_smem[];
    constexpr int BM = 8 * RI, kStage = tile_stage_floats<RI>(), kStages = tile_stages<NG>(), kSteps = kSliceK / BK, kOwn = 8 / NG;
    const int group = threadIdx.x / kGroupThreads, tid = threadIdx.x % kGroupThreads;
    const int tx = tid & 7, ty = tid >> 3;                              // outputs (ty + 8 i, tx + 8 j)
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    // (a group alone need not go on to the end of the last slice: what follows K is zeros)
    const int slices = (K + kSliceK - 1) / kSliceK, steps = NG == 1 ? (K + BK - 1) / BK : (slices + NG - 1) / NG * kSteps;
    float* ring = tile_smem + group * kStages * kStage;
    float* trade = tile_smem + NG * kStages * kStage;                   // [group][RI * 8][64]
    auto stage = [&](int s) {                                           // columns past K are zeros
        if (s < steps) {
            float* as = ring + (s % kStages) * kStage;
            float* bs = as + BM * kTilePad;
            const int k = ((s / kSteps) * NG + group) * kSliceK + (s % kSteps) * BK + 4 * (tid & 3);
#pragma unroll
            for (int i = 0; i < BM / 16; ++i) {
                const int r = (tid >> 2) + 16 * i;
                f32_stage4<VEC>(as + r * kTilePad + 4 * (tid & 3), A + (int64_t)min(m0 + r, M - 1) * lda, k, K, m0 + r < M);
            }
#pragma unroll
            for (int i = 0; i < BN / 16; ++i) {
                const int r = (tid >> 2) + 16 * i;
                f32_stage4<VEC>(bs + r * kTilePad + 4 * (tid & 3), W + (int64_t)min(n0 + r, N - 1) * ldw, k, K, n0 + r < N);
            }
        }
        f32_cp_commit();
    };
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) stage(s);
    float total[RI][kOwn], acc[RI][8];
#pragma unroll
    for (int i = 0; i < RI; ++i) {
#pragma unroll
        for (int j = 0; j < kOwn; ++j) total[i][j] = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    }
    for (int s = 0; s < steps; ++s) {
        f32_cp_wait<kStages - 2>();
        asm volatile("bar.sync %0, 64;" :: "r"(group + 1) : "memory");      // the stage has arrived; the one before it has been used
        stage(s + kStages - 1);
        const float* as = ring + (s % kStages) * kStage + ty * kTilePad;
        const float* bs = ring + (s % kStages) * kStage + (BM + tx) * kTilePad;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 b[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) b[j] = *reinterpret_cast<const float4*>(bs + 8 * j * kTilePad + k);
#pragma unroll
            for (int i = 0; i < RI; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(as + 8 * i * kTilePad + k);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
            }
        }
        if ((s + 1) % kSteps != 0 && (NG > 1 || s + 1 < steps)) continue;
        // a round's slices are complete (those past the last are zeros)
        if constexpr (NG == 1) {
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    total[i][j] += acc[i][j];
                    acc[i][j] = 0.f;
                }
        } else {
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    trade[((group * RI + i) * 8 + j) * kGroupThreads + tid] = acc[i][j];
                    acc[i][j] = 0.f;
                }
            __syncthreads();
#pragma unroll
            for (int g = 0; g < NG; ++g)
#pragma unroll
                for (int i = 0; i < RI; ++i)
#pragma unroll
                    for (int j = 0; j < kOwn; ++j) total[i][j] += trade[((g * RI + i) * 8 + group * kOwn + j) * kGroupThreads + tid];
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const int m = m0 + ty + 8 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < kOwn; ++j) {
            const int n = n0 + tx + 8 * (group * kOwn + j);
            if (n < N) C[(int64_t)m * ldc + n] = alpha * total[i][j];
        }
    }
}

template <bool VEC, int RI, int NG = kGroups>
static int launch_tile(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc, float alpha,
                       cudaStream_t stream) {
    static bool done[kMaxDevices];
    const int rc = ensure_dynamic_smem(gemm_f32_tile_kernel<VEC, RI, NG>, (int)tile_smem_bytes<RI, NG>(), done);
    if (rc != CPM_OK) return rc;
    const dim3 grid((N + BN - 1) / BN, (M + 8 * RI - 1) / (8 * RI));
    if (grid.y > 65535) return CPM_BAD_ARGUMENT;
    gemm_f32_tile_kernel<VEC, RI, NG><<<grid, NG * kGroupThreads, tile_smem_bytes<RI, NG>(), stream>>>(A, W, C, M, N, K, lda, ldw, ldc, alpha);
    return launch_status();
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
    const bool short_k = K <= 2 * kSliceK;               // (of which the kernel for few rows has little to share among its threads)
    if (M <= 16 && !short_k) return launch_few_rows<16, VEC>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
    const int sms = device_sms();
    if (sms < 1) return CPM_BAD_ARGUMENT;
    // One or two slices leave three or two of four groups idle (N 1,000, K 64: 17 rows 10.0 us, 2,048 rows 33.0): a group alone sums them,
    // several blocks an SM, of half the rows where there are not two of them for every SM (4.5 and 12.2).
    if (short_k)
        return (int64_t)((M + 63) / 64) * ((N + BN - 1) / BN) >= 2 * sms ? launch_tile<VEC, 8, 1>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream)
                                                                       : launch_tile<VEC, 4, 1>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
    // rounds of one block an SM, times the rows of a block
    auto cost = [&](int ri) {
        const int64_t tiles = (int64_t)((M + 8 * ri - 1) / (8 * ri)) * ((N + BN - 1) / BN);
        return (tiles + sms - 1) / sms * ri;
    };
    if (cost(12) < cost(10) && cost(12) < cost(8)) return launch_tile<VEC, 12>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
    if (cost(10) < cost(8)) return launch_tile<VEC, 10>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
    return launch_tile<VEC, 8>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
}

CPM_API int cpm_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda,
                         int64_t ldw, int64_t ldc, float alpha, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return CPM_OK;
    if (K <= 0) return CPM_BAD_ARGUMENT;
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    return vec ? launch_gemm_f32<true>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream)
               : launch_gemm_f32<false>(A, W, C, M, N, K, lda, ldw, ldc, alpha, stream);
}
