// Attention over the paged cache in fp32 arithmetic throughout.  This is the kernel of the true 32-bit path and the plain
// twin the tensor-core kernels are checked against; it takes every head size up to 256, group size, window and block
// selection.
//
// A query at absolute position p of its sequence sees keys j <= p (the rule of
// the reference's causal mask, src/flash_attn/src/mask.h:185-211), further limited to
// j > p - window when a window is given, or to the key blocks listed for it when a
// block list is given (the reference's block mask, src/flash_attn/src/flash_blockmask.h:15-93).
// Scores are scaled by ``scale`` before the softmax (src/model/attn.cuh:218).
//
// One block per (query token, up to NH heads of one key/value head): the heads share every key and value that is read.  The
// keys go in pieces of 32 to the block's warps in turn; in a warp a lane scores one key against all heads (queries in shared
// memory), the weights meet in shared memory, and a lane then adds up values of its channels (four tokens a load: value
// pages are stored transposed).  Each warp keeps a running maximum and sum per head; they are joined at the end.  How the
// keys are shared out depends on the query's position alone, so a row does not depend on what else is in the batch.
// Bound by latency: one warp per (token, head) that walked all its keys alone, loading a key row element by element, took
// 309 us a layer on average at 16 heads of 64, 2 kv heads (prompts and decode steps of three sequences of 50 to 400 keys);
// this form takes 32.
#include "common.cuh"
#include <math.h>

constexpr int kMaxDimsPerLane = 8;   // head_dim <= 256

// floats of shared memory: queries, weights, and the warps' results (which take the place of both at the end)
__host__ __device__ constexpr int generic_smem_floats(int warps, int nh, int d) {
    const int work = nh * d + warps * nh * 32, join = warps * nh * (d + 2);
    return work > join ? work : join;
}

template <typename T, int NH, int DPL, bool VEC>
__global__ void __launch_bounds__(256) attention_generic_kernel(
    const T* __restrict__ q,            // [tokens, heads, d]
    const T* __restrict__ k_cache, const T* __restrict__ v_cache,
    T* __restrict__ out,                // [tokens, heads, d]
    const int* __restrict__ positions, const int* __restrict__ token_seq, const int* __restrict__ slots,
    const int* __restrict__ page_table, int max_pages,
    const int* __restrict__ block_list, // [tokens, kv_heads, list_cap] or nullptr
    int list_cap, int block_size, int window,
    int n_heads, int n_kv, int d, float scale, int parts /* blocks a kv head's group is cut into */) {
    extern __shared__ __align__(16) float generic_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int t = blockIdx.x;
    const int group = n_heads / n_kv;
    const int kvh = blockIdx.y / parts;
    const int h0 = kvh * group + (blockIdx.y % parts) * NH;              // the block's heads: h0 .. h0 + nh - 1
    const int nh = min(NH, (kvh + 1) * group - h0);
    const int p = positions[t];
    const int slot = slots[token_seq[t]];
    const int* pages = page_table + (int64_t)slot * max_pages;

    float* qs = generic_smem;                                           // [NH][d]
    float* ps = generic_smem + NH * d + warp * NH * 32;                 // [NH][32]
    for (int i = threadIdx.x; i < NH * d; i += blockDim.x)
        qs[i] = i < nh * d ? to_f32(q[((int64_t)t * n_heads + h0) * d + i]) : 0.f;
    __syncthreads();

    float m[NH], l[NH], acc[NH][DPL];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
        m[h] = -INFINITY;
        l[h] = 0.f;
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[h][i] = 0.f;
    }
    const int* list = block_list ? block_list + ((int64_t)t * n_kv + kvh) * list_cap : nullptr;
    const bool listed = list != nullptr && list[0] != -2;
    int turn = 0;                                                       // pieces of 32 keys seen so far: piece i is warp (i mod warps)'s
    for (int seg_index = 0;; ++seg_index) {
        int seg_lo, seg_hi;                // keys [seg_lo, seg_hi)
        if (listed) {
            if (seg_index >= list_cap) break;
            const int b = list[seg_index];
            if (b < 0) break;
            seg_lo = b * block_size;
            seg_hi = min(seg_lo + block_size, p + 1);
        } else {
            if (seg_index > 0) break;
            seg_lo = window > 0 ? max(0, p - window + 1) : 0;
            seg_hi = p + 1;
        }
        for (int j0 = seg_lo; j0 < seg_hi; j0 += 32, ++turn) {
            if (turn % warps != warp) continue;
            const int j = j0 + lane;
            const bool valid = j < seg_hi;
            float s[NH];
#pragma unroll
            for (int h = 0; h < NH; ++h) s[h] = 0.f;
            if (valid) {
                const int page = CPM_PAGE(pages, j / kPageTokens, max_pages);
                const T* krow = k_cache + page_row_offset(page, kvh, j % kPageTokens, n_kv, d);
                if (VEC) {
#pragma unroll 4
                    for (int c = 0; c < d; c += 4) {
                        const float4 kk = load4(krow + c);
#pragma unroll
                        for (int h = 0; h < NH; ++h) {
                            const float4 qq = *reinterpret_cast<const float4*>(qs + h * d + c);
                            s[h] = fmaf(qq.x, kk.x, s[h]);
                            s[h] = fmaf(qq.y, kk.y, s[h]);
                            s[h] = fmaf(qq.z, kk.z, s[h]);
                            s[h] = fmaf(qq.w, kk.w, s[h]);
                        }
                    }
                } else {
                    for (int c = 0; c < d; ++c) {
                        const float kk = to_f32(krow[c]);
#pragma unroll
                        for (int h = 0; h < NH; ++h) s[h] = fmaf(qs[h * d + c], kk, s[h]);
                    }
                }
            }
            __syncwarp();                                               // the last piece's weights have been used
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                const float sc = valid ? s[h] * scale : -INFINITY;
                const float m_new = fmaxf(m[h], warp_max(sc));
                const float corr = (m[h] == -INFINITY) ? 0.f : expf(m[h] - m_new);
                const float pr = valid ? expf(sc - m_new) : 0.f;
                l[h] = l[h] * corr + warp_sum(pr);
#pragma unroll
                for (int i = 0; i < DPL; ++i) acc[h][i] *= corr;
                m[h] = m_new;
                ps[h * 32 + lane] = pr;
            }
            __syncwarp();
            // values: a piece that begins on a multiple of four lies in groups of four tokens of one page
            const int n_here = min(32, seg_hi - j0);
            if (VEC && (j0 & 3) == 0) {
                for (int jj = 0; jj < n_here; jj += 4) {
                    const int key = j0 + jj;
                    const int page = CPM_PAGE(pages, key / kPageTokens, max_pages);
                    const T* vcol = v_cache + value_offset(page, kvh, 0, key % kPageTokens, n_kv, d);
                    float4 pj[NH];
#pragma unroll
                    for (int h = 0; h < NH; ++h) pj[h] = *reinterpret_cast<const float4*>(ps + h * 32 + jj);
#pragma unroll
                    for (int i = 0; i < DPL; ++i) {
                        const int c = lane + 32 * i;
                        if (c >= d) continue;
                        const T* vp = vcol + (int64_t)c * kPageTokens;
                        float4 vv;
                        if (jj + 4 <= n_here) {
                            vv = load4(vp);
                        } else {                                        // what a page holds behind the last key is never read
                            vv.x = to_f32(vp[0]);
                            vv.y = jj + 1 < n_here ? to_f32(vp[1]) : 0.f;
                            vv.z = jj + 2 < n_here ? to_f32(vp[2]) : 0.f;
                            vv.w = 0.f;
                        }
#pragma unroll
                        for (int h = 0; h < NH; ++h) {
                            acc[h][i] = fmaf(pj[h].x, vv.x, acc[h][i]);
                            acc[h][i] = fmaf(pj[h].y, vv.y, acc[h][i]);
                            acc[h][i] = fmaf(pj[h].z, vv.z, acc[h][i]);
                            acc[h][i] = fmaf(pj[h].w, vv.w, acc[h][i]);
                        }
                    }
                }
            } else {
                for (int jj = 0; jj < n_here; ++jj) {
                    const int key = j0 + jj;
                    const int page = CPM_PAGE(pages, key / kPageTokens, max_pages);
                    const T* vcol = v_cache + value_offset(page, kvh, 0, key % kPageTokens, n_kv, d);
#pragma unroll
                    for (int i = 0; i < DPL; ++i) {
                        const int c = lane + 32 * i;
                        if (c >= d) continue;
                        const float vv = to_f32(vcol[(int64_t)c * kPageTokens]);
#pragma unroll
                        for (int h = 0; h < NH; ++h) acc[h][i] = fmaf(ps[h * 32 + jj], vv, acc[h][i]);
                    }
                }
            }
        }
    }
    __syncthreads();                                                    // queries and weights are no longer needed
    float* mine = generic_smem + warp * NH * (d + 2);                   // [NH][d + 2]: channels, maximum, sum
#pragma unroll
    for (int h = 0; h < NH; ++h) {
#pragma unroll
        for (int i = 0; i < DPL; ++i)
            if (lane + 32 * i < d) mine[h * (d + 2) + lane + 32 * i] = acc[h][i];
        if (lane == 0) {
            mine[h * (d + 2) + d] = m[h];
            mine[h * (d + 2) + d + 1] = l[h];
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nh * d; i += blockDim.x) {
        const int h = i / d, c = i % d;
        float top = -INFINITY;
        for (int w = 0; w < warps; ++w) top = fmaxf(top, generic_smem[(w * NH + h) * (d + 2) + d]);
        float sum = 0.f, v = 0.f;
        for (int w = 0; w < warps; ++w) {
            const float* from = generic_smem + (w * NH + h) * (d + 2);
            const float f = from[d] == -INFINITY ? 0.f : expf(from[d] - top);
            sum = fmaf(f, from[d + 1], sum);
            v = fmaf(f, from[c], v);
        }
        out[((int64_t)t * n_heads + h0) * d + i] = from_f32<T>(sum > 0.f ? v * (1.f / sum) : 0.f);
    }
}

template <typename T, int NH, int DPL>
static int launch_generic(const void* q, const void* k_cache, const void* v_cache, void* out, const int* positions,
                          const int* token_seq, const int* slots, const int* page_table, int max_pages, const int* block_list,
                          int list_cap, int block_size, int window, int n_tokens, int n_heads, int n_kv, int d, float scale,
                          cudaStream_t stream) {
    const int group = n_heads / n_kv, parts = (group + NH - 1) / NH;
    const dim3 grid(n_tokens, n_kv * parts);
    if (grid.y > 65535) return CPM_BAD_ARGUMENT;
    const int warps = d > 128 ? 4 : 8;                                  // the join needs warps * NH * (d + 2) floats
    const size_t smem = (size_t)generic_smem_floats(warps, NH, d) * sizeof(float);
    const bool vec = d % 4 == 0 && (((uintptr_t)k_cache | (uintptr_t)v_cache) & 15) == 0;      // key rows and groups of four tokens then begin on whole loads
#define CPM_GENERIC(V) attention_generic_kernel<T, NH, DPL, V><<<grid, warps * 32, smem, stream>>>((const T*)q, (const T*)k_cache,    \
        (const T*)v_cache, (T*)out, positions, token_seq, slots, page_table, max_pages, block_list, list_cap, block_size, window,    \
        n_heads, n_kv, d, scale, parts)
    if (vec) CPM_GENERIC(true); else CPM_GENERIC(false);
#undef CPM_GENERIC
    return launch_status();
}

template <typename T, int NH, typename... Args>
static int launch_generic_dims(int d, Args... args) {
    if (d <= 64) return launch_generic<T, NH, 2>(args...);
    if (d <= 128) return launch_generic<T, NH, 4>(args...);
    return launch_generic<T, NH, kMaxDimsPerLane>(args...);
}

// Heads a block takes: the whole group where it is small, at most four of them at large head sizes (registers)
template <typename T, typename... Args>
static int launch_generic_heads(int group, int d, Args... args) {
    if (group == 1) return launch_generic_dims<T, 1>(d, args...);
    if (group == 2) return launch_generic_dims<T, 2>(d, args...);
    if (group <= 4 || d > 128) return launch_generic_dims<T, 4>(d, args...);
    return launch_generic_dims<T, 8>(d, args...);
}

CPM_API int cpm_attention_generic(const void* q, const void* k_cache, const void* v_cache, void* out,
                                  const int* positions, const int* token_seq, const int* slots,
                                  const int* page_table, int max_pages, const int* block_list, int list_cap,
                                  int block_size, int window, int n_tokens, int n_heads, int n_kv, int d,
                                  float scale, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0) return CPM_OK;
    if (d <= 0 || d > 32 * kMaxDimsPerLane || n_kv <= 0 || n_heads % n_kv != 0) return CPM_BAD_ARGUMENT;
    if (block_list && (block_size <= 0 || list_cap <= 0)) return CPM_BAD_ARGUMENT;
    return dtype == CPM_BF16
        ? launch_generic_heads<bf16>(n_heads / n_kv, d, q, k_cache, v_cache, out, positions, token_seq, slots, page_table, max_pages,
                                     block_list, list_cap, block_size, window, n_tokens, n_heads, n_kv, d, scale, stream)
        : launch_generic_heads<float>(n_heads / n_kv, d, q, k_cache, v_cache, out, positions, token_seq, slots, page_table, max_pages,
                                      block_list, list_cap, block_size, window, n_tokens, n_heads, n_kv, d, scale, stream);
}

CPM_BOUNDS_TU(attention_generic)
