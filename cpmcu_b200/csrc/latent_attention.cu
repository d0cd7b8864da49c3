// Attention over a cached latent: every token leaves one vector c of ``rank`` values in the cache, and the keys
// and values of all heads are linear maps of it, k_h = Uk_h c and v_h = Uv_h c.  With the key map moved to the query
// side and the value map behind the weighted sum,
//
//   score_h(i, j) = scale * (Uk_h^T q_h(i)) . c_j          o_h(i) = Uv_h (sum_j p_h(i, j) c_j)
//
// the attention runs on the cached latents themselves: one shared "key = value" row per token for all heads.
// A query at position p sees the keys j with 0 <= p - j < window (window 0: every j <= p).
//
//   latent_norm_store   RMS-norms the two parts of the fused down projection [tokens, q_rank + rank (+ rot_dim)] (fp32):
//                       the query latent goes on as an activation, the key-value latent into the cache pages, followed
//                       there by the rotated key part that all heads share (when the design has one)
//   rotate_heads        turns a range of channels of every head by the token's position
//   latent_prepare      both of these in one kernel where queries have no latent: the fused projection's rows hold
//                       [heads x (dim + rot_dim) | rank | rot_dim] (or the queries alone), a token's angles are worked out once
//   head_project        out[t, h, :] = in[t, h, :] @ w[h]   (w [heads][k][n]; fp32 accumulation), the per-head
//                       maps Uk^T (queries into the latent space) and Uv (weighted latents into values)
//   latent_attention    softmax attention of [tokens, heads, rank] fp32 queries over the latent pages (rank up to 1,024); scores,
//                       softmax and the weighted sum are fp32; a block is one token and up to 16 heads, which share
//                       every tile of 32 latent rows through shared memory
//
// A latent page is [token_in_page][rank] (the key page layout with one key-value head).
#include "rownorm.cuh"
#include <type_traits>

// ---------------------------------------------------------------------------
// proj rows (fp32, ``stride`` floats) begin [q_rank | rank | rot_dim]: the first two parts are RMS-normed; the third (rot_dim
// may be 0) is one key part shared by all heads that is turned by the token's position, pairs (c, c + rot_dim/2) or with
// ``adjacent`` (2c, 2c + 1), angle position * inv_freq[c], cosine and sine times ``magnitude``, and not normed.  The cache
// row of the token is [rank | rot_dim].
template <typename T>
__global__ void latent_norm_store_kernel(const float* __restrict__ proj, int64_t stride, const float* __restrict__ wq,
                                         const float* __restrict__ wkv, T* __restrict__ cq, T* __restrict__ cache,
                                         const int* __restrict__ positions, const int* __restrict__ token_seq,
                                         const int* __restrict__ slots, const int* __restrict__ page_table, int max_pages,
                                         int q_rank, int rank, int rot_dim, const float* __restrict__ inv_freq, float magnitude,
                                         int adjacent, float eps) {
    __shared__ float scratch[2 * kRowMaxWarps];
    pdl_launch_dependents();
    // what needs the position alone, and the weights' way into L2, comes before the wait for the projections; both sums share a barrier
    const int t = blockIdx.x, p = positions[t];
    prefetch_l2(wq, (int64_t)q_rank * 4);
    if (cache != nullptr) prefetch_l2(wkv, (int64_t)rank * 4);
    int page = 0;
    if (cache != nullptr) page = CPM_PAGE(page_table + (int64_t)slots[token_seq[t]] * max_pages, p / kPageTokens, max_pages);
    float sn0 = 0.f, cs0 = 1.f;                          // this thread's first pair
    if (threadIdx.x < (rot_dim >> 1) && inv_freq != nullptr) sincosf((float)p * inv_freq[threadIdx.x], &sn0, &cs0);
    pdl_wait();
    const float* row = proj + (int64_t)t * stride;
    float2 s = make_float2(0.f, 0.f);
    for (int c = threadIdx.x; c < q_rank; c += blockDim.x) s.x = fmaf(row[c], row[c], s.x);
    for (int c = threadIdx.x; c < rank; c += blockDim.x) s.y = fmaf(row[q_rank + c], row[q_rank + c], s.y);
    s = row_sum2(s, scratch);
    float r = 1.0f / sqrtf(s.x / (float)q_rank + eps);
    for (int c = threadIdx.x; c < q_rank; c += blockDim.x) cq[(int64_t)t * q_rank + c] = from_f32<T>(row[c] * r * wq[c]);
    row += q_rank;
    r = 1.0f / sqrtf(s.y / (float)rank + eps);
    if (cache == nullptr) return;
    T* dst = cache + page_row_offset(page, 0, p % kPageTokens, 1, rank + rot_dim);
    for (int c = threadIdx.x; c < rank; c += blockDim.x) dst[c] = from_f32<T>(row[c] * r * wkv[c]);
    row += rank;
    dst += rank;
    const int half = rot_dim >> 1;
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        const int a = adjacent ? 2 * i : i, b = adjacent ? 2 * i + 1 : i + half;
        float sn = sn0, cs = cs0;
        if (i != (int)threadIdx.x && inv_freq != nullptr) sincosf((float)p * inv_freq[i], &sn, &cs);
        sn *= magnitude;
        cs *= magnitude;
        const float u = row[a], v = row[b];
        dst[a] = from_f32<T>(u * cs - v * sn);
        dst[b] = from_f32<T>(v * cs + u * sn);
    }
}

CPM_API int cpm_latent_norm_store(const float* proj, int64_t stride, const float* wq, const float* wkv, void* cq, void* cache,
                                  const int* positions, const int* token_seq, const int* slots, const int* page_table,
                                  int max_pages, int n_tokens, int q_rank, int rank, int rot_dim, const float* inv_freq,
                                  float magnitude, int adjacent, float eps, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0) return CPM_OK;
    if (q_rank <= 0 || rank <= 0 || rot_dim < 0 || (rot_dim & 1) || stride < q_rank + rank + rot_dim) return CPM_BAD_ARGUMENT;
    const int threads = (q_rank + rank) >= 1024 ? 256 : 128;
    if (dtype == CPM_BF16)
        cpm_launch(kLaunchRope, latent_norm_store_kernel<bf16>, n_tokens, threads, 0, stream, proj, stride, wq, wkv, (bf16*)cq,
                   (bf16*)cache, positions, token_seq, slots, page_table, max_pages, q_rank, rank, rot_dim, inv_freq, magnitude, adjacent,
                   eps);
    else
        cpm_launch(kLaunchRope, latent_norm_store_kernel<float>, n_tokens, threads, 0, stream, proj, stride, wq, wkv, (float*)cq,
                   (float*)cache, positions, token_seq, slots, page_table, max_pages, q_rank, rank, rot_dim, inv_freq, magnitude, adjacent,
                   eps);
    return launch_status();
}

// out[t][h][:] = in[t][h][:] (fp32 in, storage type out; heads of ``dh`` channels) with the channels [first, first + rot_dim)
// of every head turned by the token's position: pairs (c, c + rot_dim/2) or with ``adjacent`` (2c, 2c + 1) counted from
// ``first``, angle position * inv_freq[c], cosine and sine times ``magnitude``.  One thread per pair or per channel outside
// the turned part.
template <typename T>
__global__ void rotate_heads_kernel(const float* __restrict__ in, T* __restrict__ out, const int* __restrict__ positions,
                                    const float* __restrict__ inv_freq, float magnitude, int64_t n_units, int n_heads, int dh,
                                    int first, int rot_dim, int adjacent) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_units) return;
    const int per_head = dh - rot_dim / 2;                  // plain channels and pairs of a head
    const int64_t th = i / per_head;
    const int u = (int)(i % per_head);
    const int64_t base = th * dh;
    const int plain = dh - rot_dim;
    if (u < plain) {
        const int c = u < first ? u : u + rot_dim;
        out[base + c] = from_f32<T>(in[base + c]);
        return;
    }
    const int k = u - plain, half = rot_dim >> 1;
    const int a = first + (adjacent ? 2 * k : k), b = first + (adjacent ? 2 * k + 1 : k + half);
    float sn, cs;
    sincosf((float)positions[th / n_heads] * inv_freq[k], &sn, &cs);
    sn *= magnitude;
    cs *= magnitude;
    const float x = in[base + a], y = in[base + b];
    out[base + a] = from_f32<T>(x * cs - y * sn);
    out[base + b] = from_f32<T>(y * cs + x * sn);
}

CPM_API int cpm_rotate_heads(const float* in, void* out, const int* positions, const float* inv_freq, float magnitude,
                             int n_tokens, int n_heads, int dh, int first, int rot_dim, int adjacent, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0) return CPM_OK;
    if (n_heads < 1 || dh < 1 || first < 0 || rot_dim < 0 || (rot_dim & 1) || first + rot_dim > dh || (rot_dim && !inv_freq))
        return CPM_BAD_ARGUMENT;
    const int64_t n = (int64_t)n_tokens * n_heads * (dh - rot_dim / 2);
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (dtype == CPM_BF16)
        cpm_launch(kLaunchRope, rotate_heads_kernel<bf16>, dim3(blocks), dim3(256), 0, stream, in, (bf16*)out, positions, inv_freq, magnitude, n,
                   n_heads, dh, first, rot_dim, adjacent);
    else
        cpm_launch(kLaunchRope, rotate_heads_kernel<float>, dim3(blocks), dim3(256), 0, stream, in, (float*)out, positions, inv_freq,
                   magnitude, n, n_heads, dh, first, rot_dim, adjacent);
    return launch_status();
}

// Queries without a latent: proj rows (fp32, ``stride`` floats) begin [heads x (dim + rot_dim)] and, when ``cache`` is given,
// go on [rank | rot_dim].  The queries' last rot_dim channels of every head are turned (pairs, angle and magnitude as above)
// and leave in the storage type; the latent is RMS-normed and stored with the turned key part behind it.  One block a
// token: its cosines and sines are worked out once and serve all heads and the key part.
template <typename T>
__global__ void latent_prepare_kernel(const float* __restrict__ proj, int64_t stride, const float* __restrict__ wkv,
                                      T* __restrict__ q, T* __restrict__ cache, const int* __restrict__ positions,
                                      const int* __restrict__ token_seq, const int* __restrict__ slots,
                                      const int* __restrict__ page_table, int max_pages, int n_heads, int dim, int rank, int rot_dim,
                                      const float* __restrict__ inv_freq, float magnitude, int adjacent, float eps) {
    extern __shared__ float lp_smem[];                                   // [half][2] cosine, sine
    __shared__ float scratch[kRowMaxWarps];
    pdl_launch_dependents();
    // (before the wait: see latent_norm_store_kernel)
    const int t = blockIdx.x, half = rot_dim >> 1, dh = dim + rot_dim;
    const int p = positions[t];
    if (cache != nullptr) prefetch_l2(wkv, (int64_t)rank * 4);
    int page = 0;
    if (cache != nullptr) page = CPM_PAGE(page_table + (int64_t)slots[token_seq[t]] * max_pages, p / kPageTokens, max_pages);
    float2* cs = reinterpret_cast<float2*>(lp_smem);
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        float sn, cn;
        sincosf((float)p * inv_freq[i], &sn, &cn);
        cs[i] = make_float2(cn * magnitude, sn * magnitude);
    }
    pdl_wait();
    __syncthreads();
    const float* row = proj + (int64_t)t * stride;
    float s = 0.f;
    if (cache != nullptr) {
        const float* lat = row + (int64_t)n_heads * dh;
        for (int c = threadIdx.x; c < rank; c += blockDim.x) s = fmaf(lat[c], lat[c], s);
    }
    T* qrow = q + (int64_t)t * n_heads * dh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    const bool vec = ((dim | rot_dim) & 3) == 0 && (stride & 3) == 0;
    for (int h = warp; h < n_heads; h += n_warps) {
        const float* src = row + (int64_t)h * dh;
        T* dst = qrow + (int64_t)h * dh;
        if (vec) for (int c = 4 * lane; c < dim; c += 128) store4(dst + c, load4(src + c));
        else for (int c = lane; c < dim; c += 32) dst[c] = from_f32<T>(src[c]);
        for (int i = lane; i < half; i += 32) {
            const int a = dim + (adjacent ? 2 * i : i), b = dim + (adjacent ? 2 * i + 1 : i + half);
            const float u = src[a], v = src[b];
            dst[a] = from_f32<T>(u * cs[i].x - v * cs[i].y);
            dst[b] = from_f32<T>(v * cs[i].x + u * cs[i].y);
        }
    }
    if (cache == nullptr) return;
    row += (int64_t)n_heads * dh;
    const float r = 1.0f / sqrtf(row_sum(s, scratch) / (float)rank + eps);
    T* dst = cache + page_row_offset(page, 0, p % kPageTokens, 1, rank + rot_dim);
    for (int c = threadIdx.x; c < rank; c += blockDim.x) dst[c] = from_f32<T>(row[c] * r * wkv[c]);
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        const int a = rank + (adjacent ? 2 * i : i), b = rank + (adjacent ? 2 * i + 1 : i + half);
        const float u = row[a], v = row[b];
        dst[a] = from_f32<T>(u * cs[i].x - v * cs[i].y);
        dst[b] = from_f32<T>(v * cs[i].x + u * cs[i].y);
    }
}

CPM_API int cpm_latent_prepare(const float* proj, int64_t stride, const float* wkv, void* q, void* cache, const int* positions,
                               const int* token_seq, const int* slots, const int* page_table, int max_pages, int n_tokens,
                               int n_heads, int dim, int rank, int rot_dim, const float* inv_freq, float magnitude, int adjacent,
                               float eps, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0) return CPM_OK;
    if (n_heads < 1 || dim < 1 || rank < 1 || rot_dim < 0 || (rot_dim & 1) || rot_dim > 4096 || (rot_dim && !inv_freq)) return CPM_BAD_ARGUMENT;
    if (stride < (int64_t)n_heads * (dim + rot_dim) + (cache ? rank + rot_dim : 0) || ((uintptr_t)proj & 15)) return CPM_BAD_ARGUMENT;
    const int threads = (int64_t)n_heads * (dim + rot_dim) >= 1024 ? 256 : 128;
    const size_t smem = (size_t)rot_dim * sizeof(float) + 16;
    if (dtype == CPM_BF16)
        cpm_launch(kLaunchRope, latent_prepare_kernel<bf16>, n_tokens, threads, smem, stream, proj, stride, wkv, (bf16*)q, (bf16*)cache,
                   positions, token_seq, slots, page_table, max_pages, n_heads, dim, rank, rot_dim, inv_freq, magnitude, adjacent, eps);
    else
        cpm_launch(kLaunchRope, latent_prepare_kernel<float>, n_tokens, threads, smem, stream, proj, stride, wkv, (float*)q, (float*)cache,
                   positions, token_seq, slots, page_table, max_pages, n_heads, dim, rank, rot_dim, inv_freq, magnitude, adjacent, eps);
    return launch_status();
}

// ---------------------------------------------------------------------------
constexpr int kProjectTokens = 8;      // tokens of one head that share a pass over the head's matrix
constexpr int kProjectCols = 32;       // output columns of a block
constexpr int kProjectParts = 8;       // parts of the sum over k, one per warp
constexpr int kProjectFlight = 16;     // rows of the matrix a thread asks for before it uses the first

// A block is 8 tokens x one head x 32 output columns; its eight warps split the sum over k (a warp reads 32
// consecutive columns of every eighth row of the head's matrix, sixteen rows in flight) and add up through shared memory.
template <typename In, typename Wt, typename Out>
__global__ void __launch_bounds__(kProjectCols * kProjectParts)
head_project_kernel(const In* __restrict__ in, const Wt* __restrict__ w, Out* __restrict__ out,
                    int n_tokens, int n_heads, int K, int N) {
    extern __shared__ float hp_smem[];      // [kProjectTokens][K] inputs, then [parts][tokens][cols] partial sums
    float* part = hp_smem + kProjectTokens * K;
    pdl_launch_dependents();
    pdl_wait();
    const int h = blockIdx.y;
    const int t0 = blockIdx.x * kProjectTokens;
    const int nt = min(kProjectTokens, n_tokens - t0);
    for (int i = threadIdx.x; i < kProjectTokens * K; i += blockDim.x) {
        const int tt = i / K, k = i % K;
        hp_smem[i] = tt < nt ? to_f32(in[((int64_t)(t0 + tt) * n_heads + h) * K + k]) : 0.f;
    }
    __syncthreads();
    const int col = threadIdx.x % kProjectCols, kp = threadIdx.x / kProjectCols;
    const int n = blockIdx.z * kProjectCols + col;
    const Wt* wh = w + (int64_t)h * K * N + (n < N ? n : 0);
    float acc[kProjectTokens];
#pragma unroll
    for (int tt = 0; tt < kProjectTokens; ++tt) acc[tt] = 0.f;
    int k = kp;
    for (; k + (kProjectFlight - 1) * kProjectParts < K; k += kProjectFlight * kProjectParts) {
        float wv[kProjectFlight];
#pragma unroll
        for (int u = 0; u < kProjectFlight; ++u) wv[u] = to_f32(wh[(int64_t)(k + u * kProjectParts) * N]);
#pragma unroll
        for (int u = 0; u < kProjectFlight; ++u)
#pragma unroll
            for (int tt = 0; tt < kProjectTokens; ++tt) acc[tt] = fmaf(hp_smem[tt * K + k + u * kProjectParts], wv[u], acc[tt]);
    }
    for (; k < K; k += kProjectParts) {
        const float wv = to_f32(wh[(int64_t)k * N]);
#pragma unroll
        for (int tt = 0; tt < kProjectTokens; ++tt) acc[tt] = fmaf(hp_smem[tt * K + k], wv, acc[tt]);
    }
#pragma unroll
    for (int tt = 0; tt < kProjectTokens; ++tt) part[(kp * kProjectTokens + tt) * kProjectCols + col] = acc[tt];
    __syncthreads();
    const int tt = threadIdx.x / kProjectCols;            // 8 tokens x 32 columns = the block's 256 threads
    if (tt < nt && n < N) {
        float sum = 0.f;
#pragma unroll
        for (int p = 0; p < kProjectParts; ++p) sum += part[(p * kProjectTokens + tt) * kProjectCols + col];
        out[((int64_t)(t0 + tt) * n_heads + h) * N + n] = from_f32<Out>(sum);
    }
}

// The same product for the bf16 matrices of a decode step (N a multiple of 8, so that a row's pieces of 8 columns are 16 bytes):
// TOK tokens x one head x 32 columns a block, a thread 8 columns of every 64th row.  The first eight rows of a
// thread, all of them at ranks up to 512, are asked for before the kernel ahead is waited for (no kernel writes weights),
// so that what is left behind the wait is one trip for the inputs, the sums and two reductions.  Bound by that chain of latencies: 2.4 MB of
// matrices are read in less than a microsecond.  One column a thread, in rounds of sixteen rows behind the wait, took 21 us a launch in a
// decode step of 8 tokens (16 heads, 512 -> 128) and 8.4 us (128 -> 512).
template <int TOK, typename In, typename Out>
__global__ void __launch_bounds__(256)
head_project_few_kernel(const In* __restrict__ in, const bf16* __restrict__ w, Out* __restrict__ out, int n_tokens, int n_heads, int K, int N) {
    extern __shared__ __align__(16) float hf_smem[];                 // [K][TOK] inputs
    __shared__ float red[8][TOK][32];
    constexpr int kAhead = 8;
    const int h = blockIdx.y, t0 = blockIdx.x * TOK, nt = min(TOK, n_tokens - t0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.z * 32 + 8 * (threadIdx.x & 3), kp = threadIdx.x >> 2;
    const bf16* wh = w + (int64_t)h * K * N + (n < N ? n : 0);       // columns past N: the row's first, never stored
    uint4 ahead[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
        const int k = kp + 64 * u;
        ahead[u] = k < K ? __ldg(reinterpret_cast<const uint4*>(wh + (int64_t)k * N)) : make_uint4(0, 0, 0, 0);
    }
    pdl_launch_dependents();
    pdl_wait();
    for (int k = threadIdx.x; k < K; k += 256)
#pragma unroll
        for (int tt = 0; tt < TOK; ++tt) hf_smem[k * TOK + tt] = tt < nt ? to_f32(in[((int64_t)(t0 + tt) * n_heads + h) * K + k]) : 0.f;
    __syncthreads();
    float acc[8 * TOK];                                                // [column][token]
#pragma unroll
    for (int i = 0; i < 8 * TOK; ++i) acc[i] = 0.f;
    auto add = [&](const uint4& raw, int k) {
        float x[TOK];
#pragma unroll
        for (int tt = 0; tt < TOK; ++tt) x[tt] = hf_smem[k * TOK + tt];
        const __nv_bfloat162* pr = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(pr[i]);
#pragma unroll
            for (int tt = 0; tt < TOK; ++tt) {
                acc[2 * i * TOK + tt] = fmaf(x[tt], f.x, acc[2 * i * TOK + tt]);
                acc[(2 * i + 1) * TOK + tt] = fmaf(x[tt], f.y, acc[(2 * i + 1) * TOK + tt]);
            }
        }
    };
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
        if (kp + 64 * u < K) add(ahead[u], kp + 64 * u);
#pragma unroll 4
    for (int k = kp + 64 * kAhead; k < K; k += 64) add(__ldg(reinterpret_cast<const uint4*>(wh + (int64_t)k * N)), k);
    // the warp's eight partial sums of a column: lanes trade halves, so that each ends up with one column's tokens
#pragma unroll
    for (int step = 0; step < 3; ++step) {
        const int mask = 16 >> step, half = (4 * TOK) >> step;
        const bool upper = lane & mask;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float give = upper ? acc[i] : acc[i + half], keep = upper ? acc[i + half] : acc[i];
            acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, mask);
        }
    }
    const int col = 8 * (lane & 3) + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
#pragma unroll
    for (int tt = 0; tt < TOK; ++tt) red[warp][tt][col] = acc[tt];
    __syncthreads();
    const int c = threadIdx.x & 31, tt = threadIdx.x >> 5, nn = blockIdx.z * 32 + c;
    if (tt < nt && nn < N) {
        float sum = 0.f;
#pragma unroll
        for (int v = 0; v < 8; ++v) sum += red[v][tt][c];
        out[((int64_t)(t0 + tt) * n_heads + h) * N + nn] = from_f32<Out>(sum);
    }
}

template <int TOK, typename In, typename Out>
static int launch_head_project_few(const void* in, const void* w, void* out, int n_tokens, int n_heads, int K, int N, cudaStream_t stream) {
    cpm_launch(kLaunchProduct, head_project_few_kernel<TOK, In, Out>, dim3((n_tokens + TOK - 1) / TOK, n_heads, (N + 31) / 32), dim3(256),
               (size_t)K * TOK * sizeof(float), stream, (const In*)in, (const bf16*)w, (Out*)out, n_tokens, n_heads, K, N);
    return launch_status();
}

template <typename In, typename Wt, typename Out>
static int launch_head_project(const void* in, const void* w, void* out, int n_tokens, int n_heads, int K, int N,
                               cudaStream_t stream) {
    // Short sums over many columns (the map into the latents) are worth it for few tokens: K 128, N 512, 16 heads, this kernel and the
    // one below: 12 tokens 5.5 and 7.7 us, 20 7.9 and 8.0, 63 17.6 and 15.8.  (What the inputs take of shared memory is kept
    // to what a launch has without asking.)
    if ((K >= 256 || n_tokens <= 16) && sizeof(Wt) == 2 && N % 8 == 0 && ((uintptr_t)w & 15) == 0 && (size_t)K * 8 * sizeof(float) <= 36 * 1024) {
        if (n_tokens == 1) return launch_head_project_few<1, In, Out>(in, w, out, n_tokens, n_heads, K, N, stream);
        if (n_tokens == 2) return launch_head_project_few<2, In, Out>(in, w, out, n_tokens, n_heads, K, N, stream);
        if (n_tokens <= 4) return launch_head_project_few<4, In, Out>(in, w, out, n_tokens, n_heads, K, N, stream);
        return launch_head_project_few<8, In, Out>(in, w, out, n_tokens, n_heads, K, N, stream);
    }
    const size_t smem = (size_t)kProjectTokens * (K + kProjectParts * kProjectCols) * sizeof(float);
    auto kern = head_project_kernel<In, Wt, Out>;
    if (smem > 227 * 1024) return CPM_BAD_ARGUMENT;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    dim3 grid((n_tokens + kProjectTokens - 1) / kProjectTokens, n_heads, (N + kProjectCols - 1) / kProjectCols);
    const int threads = kProjectCols * kProjectParts;
    cpm_launch(kLaunchProduct, kern, grid, threads, smem, stream, (const In*)in, (const Wt*)w, (Out*)out, n_tokens, n_heads, K, N);
    return launch_status();
}

// in_f32 / out_f32: whether the activations on that side are fp32 (else the storage type ``dtype``); the matrix
// always has the storage type.
CPM_API int cpm_head_project(const void* in, const void* w, void* out, int n_tokens, int n_heads, int K, int N, int in_f32,
                             int out_f32, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0) return CPM_OK;
    if (n_heads <= 0 || n_heads > 65535 || K <= 0 || N <= 0 || (N + kProjectCols - 1) / kProjectCols > 65535) return CPM_BAD_ARGUMENT;
    if (dtype == CPM_F32) return launch_head_project<float, float, float>(in, w, out, n_tokens, n_heads, K, N, stream);
    if (in_f32 && out_f32) return launch_head_project<float, bf16, float>(in, w, out, n_tokens, n_heads, K, N, stream);
    if (in_f32) return launch_head_project<float, bf16, bf16>(in, w, out, n_tokens, n_heads, K, N, stream);
    if (out_f32) return launch_head_project<bf16, bf16, float>(in, w, out, n_tokens, n_heads, K, N, stream);
    return launch_head_project<bf16, bf16, bf16>(in, w, out, n_tokens, n_heads, K, N, stream);
}

// ---------------------------------------------------------------------------
constexpr int kLatentTile = 32;        // latent rows per shared-memory tile (one per lane in the scores)
constexpr int kLatentMaxWarps = 16;    // heads per block

// RL = ceil(rank / 32): what a lane keeps of a head's weighted sum.
template <typename T, int RL>
__global__ void latent_attention_kernel(const float* __restrict__ q /* [tokens, heads, rank] */, const T* __restrict__ cache,
                                        float* __restrict__ out /* [tokens, heads, rank] */, const int* __restrict__ positions,
                                        const int* __restrict__ token_seq, const int* __restrict__ slots,
                                        const int* __restrict__ page_table, int max_pages, int window, int n_heads, int rank,
                                        float scale) {
    extern __shared__ float la_smem[];
    const int n_warps = blockDim.x >> 5;
    const int pitch = rank + 1;                       // odd pitch: lane j reads row j without bank conflicts
    float* qs = la_smem;                              // [warps][rank]
    float* tile = la_smem + n_warps * rank;           // [kLatentTile][pitch]
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int h = blockIdx.y * n_warps + warp;
    const bool live = h < n_heads;
    const int p = positions[t];
    const int* pages = page_table + (int64_t)slots[token_seq[t]] * max_pages;
    if (live) {
        const float* qrow = q + ((int64_t)t * n_heads + h) * rank;
        for (int c = lane; c < rank; c += 32) qs[warp * rank + c] = qrow[c] * scale;
    }
    float m = -INFINITY, l = 0.f;
    float acc[RL];
#pragma unroll
    for (int i = 0; i < RL; ++i) acc[i] = 0.f;

    const int lo = window > 0 ? max(0, p - window + 1) : 0;
    for (int j0 = lo; j0 <= p; j0 += kLatentTile) {
        const int n_here = min(kLatentTile, p + 1 - j0);
        __syncthreads();                              // the tile of the previous iteration is no longer read
        for (int r = warp; r < n_here; r += n_warps) {
            const int j = j0 + r;
            const int page = CPM_PAGE(pages, j / kPageTokens, max_pages);
            const T* src = cache + page_row_offset(page, 0, j % kPageTokens, 1, rank);
            for (int c = lane; c < rank; c += 32) tile[r * pitch + c] = to_f32(src[c]);
        }
        __syncthreads();
        if (!live) continue;
        float s = -INFINITY;
        if (lane < n_here) {
            const float* row = tile + lane * pitch;
            const float* qh = qs + warp * rank;
            float dot = 0.f;
            for (int c = 0; c < rank; ++c) dot = fmaf(qh[c], row[c], dot);
            s = dot;
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        const float pr = lane < n_here ? expf(s - m_new) : 0.f;
        l = l * corr + warp_sum(pr);
#pragma unroll
        for (int i = 0; i < RL; ++i) acc[i] *= corr;
        m = m_new;
        for (int jj = 0; jj < n_here; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, pr, jj);
            const float* row = tile + jj * pitch;
#pragma unroll
            for (int i = 0; i < RL; ++i) {
                const int c = lane + 32 * i;
                if (c < rank) acc[i] = fmaf(pj, row[c], acc[i]);
            }
        }
    }
    if (!live) return;
    const float inv = l > 0.f ? 1.f / l : 0.f;
    float* orow = out + ((int64_t)t * n_heads + h) * rank;
#pragma unroll
    for (int i = 0; i < RL; ++i) {
        const int c = lane + 32 * i;
        if (c < rank) orow[c] = acc[i] * inv;
    }
}

template <typename T, int RL>
static int launch_latent_attention(const float* q, const void* cache, float* out, const int* positions, const int* token_seq,
                                   const int* slots, const int* page_table, int max_pages, int window, int n_tokens,
                                   int n_heads, int rank, float scale, cudaStream_t stream) {
    const int warps = n_heads < kLatentMaxWarps ? n_heads : kLatentMaxWarps;
    const size_t smem = ((size_t)warps * rank + (size_t)kLatentTile * (rank + 1)) * sizeof(float);
    auto kern = latent_attention_kernel<T, RL>;
    if (smem > 227 * 1024) return CPM_BAD_ARGUMENT;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    dim3 grid(n_tokens, (n_heads + warps - 1) / warps);
    cpm_launch(kLaunchOther, kern, grid, warps * 32, smem, stream, q, (const T*)cache, out, positions, token_seq, slots, page_table,
               max_pages, window, n_heads, rank, scale);
    return launch_status();
}

CPM_API int cpm_latent_attention(const float* q, const void* cache, float* out, const int* positions, const int* token_seq,
                                 const int* slots, const int* page_table, int max_pages, int window, int n_tokens, int n_heads,
                                 int rank, float scale, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0) return CPM_OK;
    if (n_heads <= 0 || rank <= 0 || rank > 1024 || window < 0) return CPM_BAD_ARGUMENT;
#define CPM_LATENT(RL)                                                                                                        \
    return dtype == CPM_BF16                                                                                                  \
        ? launch_latent_attention<bf16, RL>(q, cache, out, positions, token_seq, slots, page_table, max_pages, window,       \
                                            n_tokens, n_heads, rank, scale, stream)                                           \
        : launch_latent_attention<float, RL>(q, cache, out, positions, token_seq, slots, page_table, max_pages, window,      \
                                             n_tokens, n_heads, rank, scale, stream)
    if (rank <= 64) { CPM_LATENT(2); }
    if (rank <= 128) { CPM_LATENT(4); }
    if (rank <= 256) { CPM_LATENT(8); }
    if (rank <= 512) { CPM_LATENT(16); }
    CPM_LATENT(32);
#undef CPM_LATENT
}

// ---------------------------------------------------------------------------
// The same attention on the tensor cores, for bf16 latents (mma.sync m16n8k16, fp32 accumulation).  A block is one
// token, up to 16 heads (the 16 rows of the tile) and one share of the token's keys; its four warps split the work
// of every tile of 32 latent rows twice: for the scores each warp takes 8 of the 32 keys over the whole rank, for the
// weighted sum each warp takes every fourth group of 8 latent columns over all 32 keys, the latent tile being read
// as the "key" operand straight from its rows and as the "value" operand through ldmatrix.trans.  Scores go through
// shared memory in fp32; the softmax statistics are kept by every warp alike.  With more than one share a block
// leaves (max, sum, unnormalised output) in scratch and a second kernel merges the shares.
constexpr int kMmaKeys = 32;
constexpr int kMmaRows = 16;

__device__ __forceinline__ void mma_bf16_16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float fast_exp2(float x) {      // 2^x, about two units in the last place; 0 for x = -inf
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

constexpr int kPageSlots = 256;       // page numbers of a block's keys kept in shared memory (beyond: read from the table);
                                      // 1 KiB, so that three blocks of the rank-512 kernel fit one SM's shared memory

__device__ __forceinline__ void cp_async_16(void* smem, const void* gmem, bool real) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
    const int bytes = real ? 16 : 0;                                     // 0: the 16 bytes are filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// NT: column groups of 8 a warp may own in the weighted sum (rank <= 32 * NT); the same number bounds the 16-wide steps
// of the rank a warp owns in the scores (rank / 64, rounded up, <= NT / 2).  Per tile of 32 latent rows: the four warps
// split the rank for the scores (each keeps its part of the 16 query rows in registers for the whole kernel and leaves a
// partial 16 x 32 score tile in shared memory), every warp adds the four partials and keeps the softmax statistics, and
// the warps split the latent columns for the weighted sum.  Tiles arrive by cp.async one tile ahead, in two buffers.
// scratch per (token, head group, share): 16 * (rank + 2) floats.
// Blocks without keys leave at once.  one_token: no sequence brings more than one token, so that all cached rows but its own are older than the
// step, and pages and the first tiles without that row are asked for before the wait (a recorded decode step of Reravik 2k, four
// sequences of 90 to 1,900 tokens, 698 -> 677 us, of Dinutar 2k, eight of 100 to 700, 391 -> 381, of Lukelorn 2k 527 -> 520).  The blocks of a
// token as a cluster that adds up its shares out of shared memory instead of a kernel that follows: 728, 459 and 519 (a share is
// 33 KB here, which blocks read out of each other slower than out of L2).
template <int NT>
__global__ void __launch_bounds__(128)
latent_attention_mma_kernel(const float* __restrict__ q, const bf16* __restrict__ cache, void* __restrict__ out_any, int out_bf16,
                            float* __restrict__ scratch, const int* __restrict__ positions, const int* __restrict__ token_seq,
                            const int* __restrict__ slots, const int* __restrict__ page_table, int max_pages, int window,
                            int n_heads, int rank, float scale, int n_splits, int one_token) {
    constexpr int KS = NT / 2;                                           // 16-wide steps of the rank per warp, at most
    extern __shared__ __align__(16) unsigned char lm_smem[];
    __shared__ int page_s[kPageSlots];
    const int pitch = rank + 8;                                          // bf16 elements per latent row in shared memory
    bf16* Ks = reinterpret_cast<bf16*>(lm_smem);                         // [2][32][pitch]
    float* Ss = reinterpret_cast<float*>(Ks + 2 * kMmaKeys * pitch);     // [4 warps][16 values][32 lanes]
    pdl_launch_dependents();
    // (positions, slots and page tables were written before this step's kernels began)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
    const int t = blockIdx.x, h0 = blockIdx.y * kMmaRows, split = blockIdx.z;
    const int p = positions[t];
    const int* pages = page_table + (int64_t)slots[token_seq[t]] * max_pages;
    const int lo = window > 0 ? max(0, p - window + 1) : 0;
    const int tiles_total = (p + 1 - lo + kMmaKeys - 1) / kMmaKeys;
    const int per = (tiles_total + n_splits - 1) / n_splits, used = (tiles_total + per - 1) / per;
    const int tile0 = split * per, tile1 = min(tiles_total, tile0 + per);
    if (split >= used) return;                                           // (the merge reads the shares that had keys alone)
    const int k_steps = rank / 16;
    const int first_page = (lo + tile0 * kMmaKeys) / kPageTokens;
    const int last_key = min(p, lo + tile1 * kMmaKeys - 1);
    const int n_block_pages = last_key / kPageTokens - first_page + 1;
    const bool pages_in_smem = n_block_pages <= kPageSlots;
    if (pages_in_smem)
        for (int i = threadIdx.x; i < n_block_pages; i += blockDim.x) page_s[i] = CPM_PAGE(pages, first_page + i, max_pages);
    __syncthreads();

    const int vec_per_row = rank / 8;                                    // 16-byte pieces of a latent row
    // a warp brings every fourth row of a tile (the row's address worked out once), its lanes the row's 16-byte pieces
    auto fetch = [&](int tile) {
        const int j0 = lo + tile * kMmaKeys;
        bf16* dst = Ks + ((tile - tile0) & 1) * kMmaKeys * pitch;
#pragma unroll
        for (int rr = 0; rr < kMmaKeys / 4; ++rr) {
            const int r = warp + 4 * rr;
            const int j = j0 + r;
            const bool real = j <= p;
            const bf16* src = cache;
            if (real) {
                const int lp = j / kPageTokens;
                const int page = pages_in_smem ? page_s[lp - first_page] : CPM_PAGE(pages, lp, max_pages);
                src = cache + page_row_offset(page, 0, j % kPageTokens, 1, rank);
            }
            for (int v = lane; v < vec_per_row; v += 32) cp_async_16(dst + r * pitch + 8 * v, real ? src + 8 * v : src, real);
        }
        cp_async_commit();
    };
    int asked = tile0;                                                   // the next tile to ask for
    if (one_token)
        while (asked < min(tile0 + 2, tile1) && asked != tiles_total - 1) fetch(asked++);      // (the last tile has the token's own row)
    pdl_wait();
    if (asked == tile0) fetch(asked++);

    // this warp's part of the queries, as A fragments: 16-wide steps warp, warp + 4, ... of the rank
    uint32_t qa[KS][4];
#pragma unroll
    for (int i = 0; i < KS; ++i) {
        const int ks = warp + 4 * i;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int h = h0 + g + 8 * (e & 1);
            const int c = ks * 16 + 2 * tg + 8 * (e >> 1);
            float2 v = make_float2(0.f, 0.f);
            if (ks < k_steps && h < n_heads) v = *reinterpret_cast<const float2*>(q + ((int64_t)t * n_heads + h) * rank + c);
            qa[i][e] = pack_bf16(v.x, v.y);
        }
    }
    // softmax statistics in the base-2 domain: scores are multiplied by scale * log2(e) and weights are exp2
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};             // rows g and g + 8
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const float scale2 = scale * 1.4426950408889634f;
    // this lane's row addresses of the ldmatrix loads, relative to a tile: four 8 x 8 pieces at once.
    // scores (keys as the n side): pieces (keys 0-7, k 0-7), (keys 0-7, k 8-15), (keys 8-15, k 0-7), (keys 8-15, k 8-15)
    const int s_off = ((lane >> 4) * 8 + (lane & 7)) * pitch + 8 * ((lane >> 3) & 1);
    // weighted sum (keys as the k side, transposed on the way): pieces keys 0-7, 8-15, 16-23, 24-31 of 8 columns
    const int v_off = lane * pitch + 8 * warp;
    float* mine = Ss + warp * 16 * 32;                                   // [16 values][32 lanes] of this warp's partial scores

    for (int tile = tile0; tile < tile1; ++tile) {
        const int buf = (tile - tile0) & 1;
        const int j0 = lo + tile * kMmaKeys;
        if (tile + 1 < tile1) {
            if (asked == tile + 1) fetch(asked++);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();                                                 // the tile is there for every warp
        const bf16* Kt = Ks + buf * kMmaKeys * pitch;
        // partial scores of all 32 keys over this warp's part of the rank: c[n] is the 16 x 8 piece of keys 8n .. 8n + 7
        float c[4][4];
#pragma unroll
        for (int n = 0; n < 4; ++n) c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0.f;
        {
            const uint32_t s_base = (uint32_t)__cvta_generic_to_shared(Kt + s_off);
#pragma unroll
            for (int i = 0; i < KS; ++i) {
                const int ks = warp + 4 * i;
                if (ks < k_steps) {
#pragma unroll
                    for (int np = 0; np < 2; ++np) {
                        uint32_t b[4];
                        const uint32_t addr = s_base + (uint32_t)((16 * np * pitch + ks * 16) * sizeof(bf16));
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                                     : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(addr));
                        mma_bf16_16816(c[2 * np], qa[i], b[0], b[1]);
                        mma_bf16_16816(c[2 * np + 1], qa[i], b[2], b[3]);
                    }
                }
            }
        }
        // the four warps' partial scores are added lane by lane: every warp ends up with the whole 16 x 32 tile in the
        // layout of its own accumulators, which is also the layout of the A fragments of the weighted sum
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) mine[(4 * n + e) * 32 + lane] = c[n][e];
        __syncthreads();
        // (in the same order in every warp, so that all warps hold the very same sums and statistics)
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float* cell = Ss + (4 * n + e) * 32 + lane;
                c[n][e] = (cell[0] + cell[16 * 32]) + (cell[2 * 16 * 32] + cell[3 * 16 * 32]);
            }
        // c[n][0], c[n][1]: row g, keys 8n + 2tg, + 1;  c[n][2], c[n][3]: row g + 8
        const bool ragged = j0 + kMmaKeys - 1 > p;                       // the block's last tile may reach past the query
        if (ragged) {
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (j0 + 8 * n + 2 * tg + (e & 1) > p) c[n][e] = -INFINITY;
        }
        float corr[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float mx = -INFINITY;
#pragma unroll
            for (int n = 0; n < 4; ++n) mx = fmaxf(mx, fmaxf(c[n][2 * r], c[n][2 * r + 1]));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float m_new = fmaxf(m[r], mx * scale2);                // finite: a tile holds at least one visible key
            corr[r] = fast_exp2(m[r] - m_new);                           // 0 at the first tile (m = -inf)
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                c[n][2 * r] = fast_exp2(fmaf(c[n][2 * r], scale2, -m_new));
                c[n][2 * r + 1] = fast_exp2(fmaf(c[n][2 * r + 1], scale2, -m_new));
                sum += c[n][2 * r] + c[n][2 * r + 1];
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            l[r] = l[r] * corr[r] + sum;
            m[r] = m_new;
        }
        if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                acc[i][0] *= corr[0]; acc[i][1] *= corr[0];
                acc[i][2] *= corr[1]; acc[i][3] *= corr[1];
            }
        }
        uint32_t pa[2][4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            pa[half][0] = pack_bf16(c[2 * half][0], c[2 * half][1]);          // row g,     keys 16 half + 2tg, + 1
            pa[half][1] = pack_bf16(c[2 * half][2], c[2 * half][3]);          // row g + 8
            pa[half][2] = pack_bf16(c[2 * half + 1][0], c[2 * half + 1][1]);  // row g,     keys 16 half + 8 + 2tg, + 1
            pa[half][3] = pack_bf16(c[2 * half + 1][2], c[2 * half + 1][3]);  // row g + 8
        }
        {
            const uint32_t v_base = (uint32_t)__cvta_generic_to_shared(Kt + v_off);
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                if (8 * (warp + 4 * i) < rank) {
                    uint32_t b[4];
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(v_base + (uint32_t)(32 * i * sizeof(bf16))));
                    mma_bf16_16816(acc[i], pa[0], b[0], b[1]);
                    mma_bf16_16816(acc[i], pa[1], b[2], b[3]);
                }
            }
        }
        __syncthreads();                                                 // this buffer and the scores may be overwritten
    }
    // rows g and g + 8 are heads h0 + g and h0 + g + 8; a thread holds columns col0 + 2tg, + 1 of its column groups
    if (n_splits == 1) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int h = h0 + g + 8 * r;
            if (h >= n_heads) continue;
            const float inv = l[r] > 0.f ? 1.f / l[r] : 0.f;
            const int64_t o = ((int64_t)t * n_heads + h) * rank;
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int c = 8 * (warp + 4 * i) + 2 * tg;
                if (c >= rank) continue;
                if (out_bf16) *reinterpret_cast<uint32_t*>(static_cast<bf16*>(out_any) + o + c) = pack_bf16(acc[i][2 * r] * inv, acc[i][2 * r + 1] * inv);
                else *reinterpret_cast<float2*>(static_cast<float*>(out_any) + o + c) = make_float2(acc[i][2 * r] * inv, acc[i][2 * r + 1] * inv);
            }
        }
        return;
    }
    float* part = scratch + (((int64_t)t * gridDim.y + blockIdx.y) * n_splits + split) * kMmaRows * (rank + 2);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        float* prow = part + (g + 8 * r) * (rank + 2);
        if (warp == 0 && tg == 0) { prow[rank] = m[r]; prow[rank + 1] = l[r]; }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int c = 8 * (warp + 4 * i) + 2 * tg;
            if (c < rank) { prow[c] = acc[i][2 * r]; prow[c + 1] = acc[i][2 * r + 1]; }
        }
    }
}

// One block per (token, head group, row of the tile): the weights of the shares that had keys are worked out once, then a thread
// adds up two columns of all of them, sixteen shares in flight.  Bound by the latency of two dependent trips to L2 (one column at a
// time in rounds of eight shares, empty ones too: 14.5 us a launch for 8 tokens of 16 heads, rank 512, 32 shares).
__global__ void __launch_bounds__(288)
latent_attention_merge_kernel(const float* __restrict__ scratch, void* __restrict__ out_any, int out_bf16, const int* __restrict__ positions,
                              int window, int n_heads, int rank, int n_splits) {
    __shared__ float weight[64];
    __shared__ float inv_l;
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, hg = blockIdx.y, r = blockIdx.z;
    const int h = hg * kMmaRows + r;
    if (h >= n_heads) return;
    // the shares that had keys come first (the same arithmetic as in the kernel that wrote them)
    const int p = positions[t];
    const int lo = window > 0 ? max(0, p - window + 1) : 0;
    const int tiles = (p + 1 - lo + kMmaKeys - 1) / kMmaKeys, per = (tiles + n_splits - 1) / n_splits;
    const int used = (tiles + per - 1) / per;
    const float* base = scratch + (((int64_t)t * gridDim.y + hg) * n_splits * kMmaRows + r) * (rank + 2);
    const int64_t share = (int64_t)kMmaRows * (rank + 2);
    if (threadIdx.x < 32) {
        float ms[2], ls[2], mx = -INFINITY;                          // at most 64 shares
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int s = threadIdx.x + 32 * i;
            ms[i] = s < used ? base[s * share + rank] : -INFINITY;
            ls[i] = s < used ? base[s * share + rank + 1] : 0.f;
            mx = fmaxf(mx, ms[i]);
        }
        mx = warp_max(mx);
        float l = 0.f;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float w = ms[i] == -INFINITY ? 0.f : exp2f(ms[i] - mx);      // the shares' maxima are base-2 logarithms
            weight[threadIdx.x + 32 * i] = w;
            l = fmaf(ls[i], w, l);
        }
        l = warp_sum(l);
        if (threadIdx.x == 0) inv_l = l > 0.f ? 1.f / l : 0.f;
    }
    __syncthreads();
    const int64_t o = ((int64_t)t * n_heads + h) * rank;
    for (int c = 2 * threadIdx.x; c < rank; c += 2 * blockDim.x) {       // the rank is even, a share's row 8-byte aligned
        float2 acc = make_float2(0.f, 0.f);
        for (int s0 = 0; s0 < used; s0 += 16) {
            float2 v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = s0 + u < used ? *reinterpret_cast<const float2*>(base + (s0 + u) * share + c) : make_float2(0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 16; ++u)
                if (s0 + u < used) {
                    acc.x = fmaf(v[u].x, weight[s0 + u], acc.x);
                    acc.y = fmaf(v[u].y, weight[s0 + u], acc.y);
                }
        }
        acc.x *= inv_l;
        acc.y *= inv_l;
        if (out_bf16) *reinterpret_cast<uint32_t*>(static_cast<bf16*>(out_any) + o + c) = pack_bf16(acc.x, acc.y);
        else *reinterpret_cast<float2*>(static_cast<float*>(out_any) + o + c) = acc;
    }
}

CPM_API int64_t cpm_latent_attention_scratch_floats(int n_tokens, int n_heads, int rank, int n_splits) {
    if (n_splits <= 1) return 0;
    return (int64_t)n_tokens * ((n_heads + kMmaRows - 1) / kMmaRows) * n_splits * kMmaRows * (rank + 2);
}

template <int NT>
static int launch_latent_mma(const float* q, const void* cache, void* out, int out_bf16, float* scratch, const int* positions,
                             const int* token_seq, const int* slots, const int* page_table, int max_pages, int window,
                             int n_tokens, int n_heads, int rank, float scale, int n_splits, int one_token, cudaStream_t stream) {
    static bool smem_done[kMaxDevices];
    const size_t smem = (size_t)2 * kMmaKeys * (rank + 8) * sizeof(bf16) + (size_t)4 * 16 * 32 * sizeof(float);
    auto kern = latent_attention_mma_kernel<NT>;
    if (smem > 48 * 1024) {
        int dev = 0;
        cudaGetDevice(&dev);
        const bool first = dev >= 0 && dev < kMaxDevices && !smem_done[dev];
        // (of the template's largest rank: the attribute is set once, whatever rank comes first)
        if (int e = ensure_dynamic_smem(kern, (int)(2 * kMmaKeys * (32 * NT + 8) * sizeof(bf16) + 4 * 16 * 32 * sizeof(float)), smem_done)) return e;
        // all of the SM's unified memory as shared memory: three blocks of the rank-512 kernel then fit one SM
        if (first) cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
    const int groups = (n_heads + kMmaRows - 1) / kMmaRows;
    dim3 grid(n_tokens, groups, n_splits);
    cpm_launch(kLaunchAttention, kern, grid, 128, smem, stream, q, (const bf16*)cache, out, out_bf16, scratch, positions, token_seq, slots,
               page_table, max_pages, window, n_heads, rank, scale, n_splits, one_token);
    if (n_splits > 1)
        cpm_launch(kLaunchCombine, latent_attention_merge_kernel, dim3(n_tokens, groups, kMmaRows), rank > 512 ? 288 : rank > 256 ? 256 : 128, 0, stream,
                   (const float*)scratch, out, out_bf16, positions, window, n_heads, rank, n_splits);
    return launch_status();
}

// bf16 latents, rank a multiple of 16 up to 576; ``out`` fp32, or bf16 with ``out_bf16``; ``scratch``: cpm_latent_attention_scratch_floats floats
// when n_splits > 1.  ``one_token``: no sequence brings more than one token.
CPM_API int cpm_latent_attention_mma(const float* q, const void* cache, void* out, int out_bf16, float* scratch, const int* positions,
                                     const int* token_seq, const int* slots, const int* page_table, int max_pages, int window,
                                     int n_tokens, int n_heads, int rank, float scale, int n_splits, int one_token, cudaStream_t stream) {
    if (n_tokens <= 0) return CPM_OK;
    if (n_heads <= 0 || rank <= 0 || rank > 576 || rank % 16 || window < 0 || n_splits < 1 || n_splits > 64) return CPM_BAD_ARGUMENT;
    if (n_splits > 1 && scratch == nullptr) return CPM_BAD_ARGUMENT;
    if ((n_heads + kMmaRows - 1) / kMmaRows > 65535) return CPM_BAD_ARGUMENT;
    if (rank <= 128) return launch_latent_mma<4>(q, cache, out, out_bf16, scratch, positions, token_seq, slots, page_table, max_pages, window,
                                                  n_tokens, n_heads, rank, scale, n_splits, one_token, stream);
    if (rank <= 256) return launch_latent_mma<8>(q, cache, out, out_bf16, scratch, positions, token_seq, slots, page_table, max_pages, window,
                                                  n_tokens, n_heads, rank, scale, n_splits, one_token, stream);
    if (rank <= 512) return launch_latent_mma<16>(q, cache, out, out_bf16, scratch, positions, token_seq, slots, page_table, max_pages, window,
                                                  n_tokens, n_heads, rank, scale, n_splits, one_token, stream);
    return launch_latent_mma<18>(q, cache, out, out_bf16, scratch, positions, token_seq, slots, page_table, max_pages, window, n_tokens,
                                 n_heads, rank, scale, n_splits, one_token, stream);
}

// ---------------------------------------------------------------------------
// Prompt tokens: a block takes two neighbouring tokens of a sequence (the query tiles of 64 rows list them) and up to 16 heads, so that
// a page of 64 latents, brought once into shared memory, serves 32 rows.  Warps 0-3 are the first token's, 4-7 the second's.  A
// warp forms the scores of 16 of the page's keys over the whole rank (no partial scores to trade: the queries lie in shared memory
// too), the four warps of a token trade their rows' maxima, leave their weights in shared memory as the next product's operand
// and then split the latent columns for the weighted sum.  Two blocks an SM: one's page arrives while the other's is worked on.
// A latent that a token does not see never meets a weight of zero (0 * NaN is NaN): rows that neither token of a pair sees come as zeros, and
// the row that only the other one sees (the second token itself; behind a window, the first one's first key) is cleared from the operand.
// Bound by the operands' way out of shared memory.  The kernel above, one token a block and the rank split over its warps, spent
// 1,245 instructions a warp and tile on 64 tensor-core ones: 576 us for 2,048 tokens of two prompts, 16 heads, rank 512; this one 317.
constexpr int kPromptKeys = 64, kPromptTokens = 2;

template <int NT>
__global__ void __launch_bounds__(256, NT <= 16 ? 2 : 1)
latent_prompt_mma_kernel(const float* __restrict__ q, const bf16* __restrict__ cache, void* __restrict__ out_any, int out_bf16,
                         const int* __restrict__ positions, const int* __restrict__ slots, const int* __restrict__ page_table, int max_pages,
                         const int* __restrict__ tile_seq, const int* __restrict__ tile_row, const int* __restrict__ cu_q, int n_tiles, int window,
                         int n_heads, int rank, float scale2) {
    extern __shared__ __align__(16) unsigned char lp_raw[];
    const int pitch = rank + 8;                                          // bf16 elements per row in shared memory
    bf16* Ks = reinterpret_cast<bf16*>(lp_raw);                          // [64][pitch]
    bf16* Qs = Ks + kPromptKeys * pitch;                                 // [2][16][pitch]
    constexpr int kPPitch = kPromptKeys + 8;
    __shared__ __align__(16) bf16 Ps[kPromptTokens][16][kPPitch];
    __shared__ float row_max[kPromptTokens][4][16], row_sums[kPromptTokens][4][16];
    pdl_launch_dependents();
    constexpr int kPairs = 64 / kPromptTokens;                           // pairs of a query tile
    const int tile_no = n_tiles - 1 - blockIdx.x / kPairs;               // later tiles of a sequence have more keys: they go first
    const int seq = tile_seq[tile_no], row0 = tile_row[tile_no] + kPromptTokens * (blockIdx.x % kPairs);
    const int q_begin = cu_q[seq], q_len = cu_q[seq + 1] - q_begin;
    if (row0 >= q_len) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
    const int rt = warp >> 2, cw = warp & 3, h0 = blockIdx.y * kMmaRows;
    const int t = q_begin + row0 + rt;
    const bool live = row0 + rt < q_len;                                 // an odd portion's last pair has one token
    const int first_p = positions[q_begin + row0], last_p = first_p + (row0 + 1 < q_len ? 1 : 0);
    const int p = live ? first_p + rt : -1;
    const int lo = window > 0 ? max(0, p - window + 1) : 0;
    const int first_key = window > 0 ? max(0, first_p - window + 1) : 0;
    const int page0 = first_key / kPageTokens, page1 = last_p / kPageTokens;
    // the key between first_key and last_p that this warp's token does not see (at most one; -1: none)
    const int hidden_key = rt == 0 ? (last_p > first_p ? last_p : -1) : (live && lo > first_key ? first_key : -1);
    const int* pages = page_table + (int64_t)slots[seq] * max_pages;
    pdl_wait();
    // the queries as bf16, rows past the last head or token zeros
    for (int i = threadIdx.x; i < kPromptTokens * 16 * (rank / 4); i += 256) {
        const int row = i / (rank / 4), c = 4 * (i % (rank / 4)), tok = row >> 4, h = h0 + (row & 15);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (h < n_heads && row0 + tok < q_len) v = *reinterpret_cast<const float4*>(q + ((int64_t)(q_begin + row0 + tok) * n_heads + h) * rank + c);
        store4(Qs + row * pitch + c, v);
    }
    const int vec_per_row = rank / 8;
    auto ldsm = [](uint32_t (&r)[4], uint32_t addr) {
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
    };
    auto ldsm_t = [](uint32_t (&r)[4], uint32_t addr) {
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
    };
    auto token_barrier = [&]() { asm volatile("bar.sync %0, 128;" :: "r"(1 + rt) : "memory"); };
    const uint32_t q_addr = (uint32_t)__cvta_generic_to_shared(Qs + (rt * 16 + (lane & 15)) * pitch + 8 * (lane >> 4));
    const uint32_t k_addr = (uint32_t)__cvta_generic_to_shared(Ks + (16 * cw + (lane >> 4) * 8 + (lane & 7)) * pitch + 8 * ((lane >> 3) & 1));
    const uint32_t p_addr = (uint32_t)__cvta_generic_to_shared(&Ps[rt][lane & 15][8 * (lane >> 4)]);
    const uint32_t v_addr = (uint32_t)__cvta_generic_to_shared(Ks + lane * pitch + 8 * cw);
    const uint32_t half_page = (uint32_t)(32 * pitch * sizeof(bf16));
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};             // rows g and g + 8; l: this warp's keys only
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    for (int page = page0; page <= page1; ++page) {
        const bf16* src = cache + page_row_offset(CPM_PAGE(pages, page, max_pages), 0, 0, 1, rank);
        for (int r = warp; r < kPromptKeys; r += 8)
            for (int v = lane; v < vec_per_row; v += 32) {
                const int key = page * kPageTokens + r;
                cp_async_16(Ks + r * pitch + 8 * v, src + (int64_t)r * rank + 8 * v, key >= first_key && key <= last_p);
            }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();                                                 // the page (and the queries) are there
        float c[2][4] = {};
        const int k_steps = rank / 16;
#pragma unroll 4
        for (int ks = 0; ks < k_steps; ++ks) {
            uint32_t a[4], b[4];
            ldsm(a, q_addr + 32 * ks);
            ldsm(b, k_addr + 32 * ks);
            mma_bf16_16816(c[0], a, b[0], b[1]);
            mma_bf16_16816(c[1], a, b[2], b[3]);
        }
        // c[n][e]: row g (e < 2) or g + 8, key 16 cw + 8 n + 2 tg + (e & 1) of the page
        const int key0 = page * kPageTokens + 16 * cw + 2 * tg;
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int key = key0 + 8 * n + (e & 1);
                const float x = key <= p && key >= lo ? c[n][e] * scale2 : -INFINITY;
                c[n][e] = x;
                mx[e >> 1] = fmaxf(mx[e >> 1], x);
            }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
            if (tg == 0) row_max[rt][cw][g + 8 * r] = mx[r];
        }
        token_barrier();
        float corr[2], use[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int row = g + 8 * r;
            const float mn = fmaxf(fmaxf(m[r], fmaxf(row_max[rt][0][row], row_max[rt][1][row])), fmaxf(row_max[rt][2][row], row_max[rt][3][row]));
            use[r] = mn == -INFINITY ? 0.f : mn;
            corr[r] = fast_exp2(m[r] - use[r]);                          // 0 at the first visible key
            m[r] = mn;
            l[r] *= corr[r];
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                c[n][e] = fast_exp2(c[n][e] - use[e >> 1]);
                l[e >> 1] += c[n][e];
            }
            *reinterpret_cast<uint32_t*>(&Ps[rt][g][16 * cw + 8 * n + 2 * tg]) = pack_bf16(c[n][0], c[n][1]);
            *reinterpret_cast<uint32_t*>(&Ps[rt][g + 8][16 * cw + 8 * n + 2 * tg]) = pack_bf16(c[n][2], c[n][3]);
        }
        if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                acc[i][0] *= corr[0]; acc[i][1] *= corr[0];
                acc[i][2] *= corr[1]; acc[i][3] *= corr[1];
            }
        }
        token_barrier();                                                 // the token's weights are there
        uint32_t pa[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) ldsm(pa[k], p_addr + 32 * k);
        // a register of the values holds keys 8 j + 2 tg and the next: the half of the hidden key, if it lies in this page, is masked
        const int hidden = hidden_key - page * kPageTokens;
        uint32_t keep[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) keep[j] = hidden >> 1 != 4 * j + tg ? 0xffffffffu : hidden & 1 ? 0x0000ffffu : 0xffff0000u;
        auto add_values = [&](auto masked) {
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                if (8 * (cw + 4 * i) < rank) {
                    uint32_t b[2][4];
                    ldsm_t(b[0], v_addr + (uint32_t)(32 * i * sizeof(bf16)));
                    ldsm_t(b[1], v_addr + half_page + (uint32_t)(32 * i * sizeof(bf16)));
                    if (decltype(masked)::value)
#pragma unroll
                        for (int j = 0; j < 8; ++j) b[j >> 2][j & 3] &= keep[j];
                    mma_bf16_16816(acc[i], pa[0], b[0][0], b[0][1]);
                    mma_bf16_16816(acc[i], pa[1], b[0][2], b[0][3]);
                    mma_bf16_16816(acc[i], pa[2], b[1][0], b[1][1]);
                    mma_bf16_16816(acc[i], pa[3], b[1][2], b[1][3]);
                }
            }
        };
        if (hidden >= 0 && hidden < kPromptKeys) add_values(std::true_type{}); else add_values(std::false_type{});
        __syncthreads();                                                 // the page has been used
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
        if (tg == 0) row_sums[rt][cw][g + 8 * r] = l[r];
    }
    token_barrier();
    if (!live) return;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = g + 8 * r, h = h0 + row;
        if (h >= n_heads) continue;
        const float sum = (row_sums[rt][0][row] + row_sums[rt][1][row]) + (row_sums[rt][2][row] + row_sums[rt][3][row]);
        const float inv = sum > 0.f ? 1.f / sum : 0.f;
        const int64_t o = ((int64_t)t * n_heads + h) * rank;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int col = 8 * (cw + 4 * i) + 2 * tg;
            if (col >= rank) continue;
            if (out_bf16) *reinterpret_cast<uint32_t*>(static_cast<bf16*>(out_any) + o + col) = pack_bf16(acc[i][2 * r] * inv, acc[i][2 * r + 1] * inv);
            else *reinterpret_cast<float2*>(static_cast<float*>(out_any) + o + col) = make_float2(acc[i][2 * r] * inv, acc[i][2 * r + 1] * inv);
        }
    }
}

template <int NT>
static int launch_latent_prompt(const float* q, const void* cache, void* out, int out_bf16, const int* positions, const int* slots,
                                const int* page_table, int max_pages, const int* tile_seq, const int* tile_row, const int* cu_q, int n_tiles,
                                int window, int n_heads, int rank, float scale, cudaStream_t stream) {
    static bool done[kMaxDevices];
    const size_t smem = (size_t)(kPromptKeys + 16 * kPromptTokens) * (rank + 8) * sizeof(bf16);
    auto kern = latent_prompt_mma_kernel<NT>;
    if (int e = ensure_dynamic_smem(kern, (kPromptKeys + 16 * kPromptTokens) * (32 * NT + 8) * (int)sizeof(bf16), done)) return e;
    const dim3 grid(n_tiles * (64 / kPromptTokens), (n_heads + kMmaRows - 1) / kMmaRows);
    cpm_launch(kLaunchAttention, kern, grid, 256, smem, stream, q, (const bf16*)cache, out, out_bf16, positions, slots, page_table, max_pages,
               tile_seq, tile_row, cu_q, n_tiles, window, n_heads, rank, scale * 1.4426950408889634f);
    return launch_status();
}

// The same attention for the tokens of prompts, packed by sequence: cu_q, slots by sequence; tile_seq, tile_row: tiles of 64 rows that cover
// every sequence's tokens (tiles past a sequence's end hold none); a sequence's tokens have consecutive positions.
CPM_API int cpm_latent_attention_prompt(const float* q, const void* cache, void* out, int out_bf16, const int* positions, const int* slots,
                                        const int* page_table, int max_pages, const int* tile_seq, const int* tile_row, const int* cu_q,
                                        int n_tiles, int window, int n_heads, int rank, float scale, cudaStream_t stream) {
    if (n_tiles <= 0) return CPM_OK;
    if (n_heads <= 0 || rank <= 0 || rank > 576 || rank % 16 || window < 0 || n_tiles > (1 << 24) || (n_heads + kMmaRows - 1) / kMmaRows > 65535 ||
        (((uintptr_t)q | (uintptr_t)cache) & 15))
        return CPM_BAD_ARGUMENT;
#define CPM_LATENT_PROMPT(N) return launch_latent_prompt<N>(q, cache, out, out_bf16, positions, slots, page_table, max_pages, tile_seq, tile_row, cu_q, \
                                                            n_tiles, window, n_heads, rank, scale, stream)
    if (rank <= 128) CPM_LATENT_PROMPT(4);
    if (rank <= 256) CPM_LATENT_PROMPT(8);
    if (rank <= 512) CPM_LATENT_PROMPT(16);
    CPM_LATENT_PROMPT(18);
#undef CPM_LATENT_PROMPT
}

CPM_BOUNDS_TU(latent_attention)
