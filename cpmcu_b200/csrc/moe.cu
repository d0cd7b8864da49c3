// Routed experts: choice of experts per token, and the experts' products over the tokens that chose them.
//
// Routing (fp32): scores s = softmax(z) over all experts; choice scores c = s + correction; experts form
// ``n_groups`` equal groups of neighbours, a group's score is its largest choice score, and only experts of the
// ``keep`` best groups can be chosen (the others count as minus infinity); the ``top`` largest choice scores are
// chosen, and their weights are the plain scores s, not renormalised.  Ties go to the lower index.
// A second rule (``top_first`` 1): the choice scores are the logits plus a bias, the ``top`` largest are chosen, and
// their weights are the softmax over the chosen logits only.  A third (``top_first`` 2): the scores are the sigmoids of
// the logits, which are the choice scores too, chosen within the kept groups, and their weights are those scores.
// Two switches for the first and third rule: a group's score may be the sum of its two largest choice scores
// (``group_top2``), and the chosen scores may be divided by their sum + 1e-20 and multiplied by a constant (``normalize``,
// ``route_scale``).
//
// Products: the (token, choice) pairs are grouped by expert (counts, offsets, a list of pairs in expert order),
// and tiles of one expert's pairs times some output features are shared out among the blocks of one launch, whose number
// depends on no count that the device holds, so nothing is read back on the host:
//   gated (mode 1):  H[r] = silu(x[token(r)] Wg_e^T) * (x[token(r)] Wu_e^T)     r: place in expert order
//   bounded gate (mode 3): the same two products joined by the gate of GluClamp (common.cuh)
//   up (mode 2):     H[r] = relu(s[pair(r)] * (x[token(r)] Wu_e^T))^2           s: a number per pair (null: 1), which is
//                    the expert of the input times s, since the product is linear in its input
//   down (mode 0):   Y[pair(r)] = H[r] Wd_e^T
// and a last kernel adds up a token's pairs with their weights and the shared expert's output times its gate.
// Accumulation is fp32: on the CUDA cores for 32-bit storage (and where K is no multiple of 8 or there are more than 512
// experts), on the tensor cores for bf16 (moe_tcgen05.cu).
#include "common.cuh"

// moe_tcgen05.cu: bf16, A with a row per pair in expert order, K a multiple of 8, 16-byte aligned operands, at most 512 experts
int moe_product_tcgen05(const void* A, const void* B0, const void* B1, void* C, const int* offsets, const int* order, int n_pairs, int E,
                        int N, int K, int mode, const float* in_scale, const GluClamp& clamp, cudaStream_t stream);

constexpr int kRouteMaxPerLane = 16;      // experts <= 512

__device__ __forceinline__ ArgMax warp_argmax(ArgMax a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ArgMax b;
        b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
        b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
        a = better(a, b);
    }
    return a;
}

// A float as an unsigned number of the same order; 0 is left for "absent" (NaN is), and both zeros are the same number.
__device__ __forceinline__ uint32_t order_key(float v) {
    if (isnan(v)) return 0u;
    const uint32_t b = __float_as_uint(v + 0.0f);
    return (b & 0x80000000u) ? ~b : b | 0x80000000u;
}

// The place of the largest key over the warp, the lowest among equals, or -1 if all are absent; the one found becomes absent.  A lane
// holds the keys of places lane + 32 i.  Two warp-wide reductions a choice; with the scores in shared memory and the
// comparison of (value, place) carried through five shuffles, the routing of 4 tokens took 7.3 us, 6 chosen of 64 in 3 of 8 groups.
template <int PER>
__device__ __forceinline__ int take_largest(uint32_t (&key)[PER], int lane) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) m = max(m, key[i]);
    m = __reduce_max_sync(0xffffffffu, m);
    if (m == 0u) return -1;
    uint32_t at = 0xffffffffu;
#pragma unroll
    for (int i = PER - 1; i >= 0; --i)
        if (key[i] == m) at = (uint32_t)(lane + 32 * i);
    at = __reduce_min_sync(0xffffffffu, at);
#pragma unroll
    for (int i = 0; i < PER; ++i)
        if (at == (uint32_t)(lane + 32 * i)) key[i] = 0u;
    return (int)at;
}

// One warp per token.  logits rows of ``ld`` floats: the first E are the router's, column ``gate_col`` (if >= 0) is the
// shared expert's raw gate.
// The next kernel is let in behind the wait, not before it: the products ahead let this one in at their start, and the experts' blocks
// (by pair: hundreds, four an SM, which hold their place while they wait) would be placed around the blocks of up to four kernels that
// still run, unevenly over the SMs.  Rabadra 1k, four tokens: the first product 13.4 us behind the kernel ahead of it, 6.6 so.  us of a
// recorded decode step before and now: Rabadra 1k one, four, eight, 16 tokens 310, 404,
// 431, 502 and 308, 343, 384, 471; Kipizen 1k 252, 312, 349, 423 and 250, 282, 321, 405; Lukelorn 1k 275, 304, 350,
// 416 and 274, 295, 322, 391.
template <int PER>
__global__ void moe_route_kernel(const float* __restrict__ logits, int ld, const float* __restrict__ correction,
                                 int* __restrict__ chosen, float* __restrict__ weights, float* __restrict__ shared_gate,
                                 int gate_col, int n_tokens, int E, int top, int n_groups, int keep,
                                 const float* __restrict__ bias, int top_first, int group_top2, int normalize,
                                 float route_scale) {
    extern __shared__ float route_smem[];
    pdl_wait();
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= n_tokens) return;
    float* s = route_smem + (size_t)warp * (2 * E + n_groups);      // scores
    float* c = s + E;                                                 // choice scores
    float* gs = c + E;                                                // group scores
    const float* z = logits + (int64_t)t * ld;
    if (top_first == 1) {
        // choice scores: logits + bias; weights: softmax over the chosen scores (the largest is the first chosen)
        uint32_t key[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int e = lane + 32 * i;
            const float v = e < E ? z[e] + (bias ? bias[e] : 0.f) : NAN;
            if (e < E) c[e] = v;
            key[i] = order_key(v);
        }
        __syncwarp();
        float first = 0.f, sum = 0.f;
        for (int r = 0; r < top; ++r) {
            const int found = take_largest<PER>(key, lane), e = max(found, 0);
            const float v = found < 0 ? -INFINITY : c[e];
            if (r == 0) first = v;
            const float ex = expf(v - first);
            sum += ex;
            if (lane == 0) {
                chosen[(int64_t)t * top + r] = e;
                weights[(int64_t)t * top + r] = ex;
            }
        }
        if (lane == 0)
            for (int r = 0; r < top; ++r) weights[(int64_t)t * top + r] /= sum;
        if (gate_col >= 0 && lane == 0) shared_gate[t] = 1.0f / (1.0f + expf(-z[gate_col]));
        return;
    }
    if (top_first == 2) {
        for (int e = lane; e < E; e += 32) {
            const float v = 1.0f / (1.0f + expf(-(z[e] + (bias ? bias[e] : 0.f))));
            s[e] = v;
            c[e] = v;
        }
    } else {
        float m = -INFINITY;
        for (int e = lane; e < E; e += 32) m = fmaxf(m, z[e]);
        m = warp_max(m);
        float sum = 0.f;
        for (int e = lane; e < E; e += 32) {
            const float ex = expf(z[e] - m);
            s[e] = ex;
            sum += ex;
        }
        sum = warp_sum(sum);
        const float inv = 1.0f / sum;
        for (int e = lane; e < E; e += 32) {
            const float v = s[e] * inv;
            s[e] = v;
            c[e] = v + correction[e];
        }
    }
    __syncwarp();
    const int per = E / n_groups;
    if (n_groups > 1 && keep < n_groups) {
        for (int g = lane; g < n_groups; g += 32) {
            float best = -INFINITY, second = -INFINITY;
            for (int i = 0; i < per; ++i) {
                const float v = c[g * per + i];
                second = fmaxf(second, fminf(best, v));
                best = fmaxf(best, v);
            }
            gs[g] = (group_top2 && per > 1) ? best + second : best;
        }
        __syncwarp();
        // a kept group, one of the ``keep`` best, is marked by a score of +inf (one that is +inf already is kept by that)
        if (n_groups <= 32) {
            uint32_t key[1] = {lane < n_groups && gs[lane] != INFINITY ? order_key(gs[lane]) : 0u};
            for (int r = 0; r < keep; ++r) {
                const int found = take_largest<1>(key, lane);
                if (found >= 0 && lane == 0) gs[found] = INFINITY;
            }
        } else {
            for (int r = 0; r < keep; ++r) {
                ArgMax a{-INFINITY, 0x7fffffff};
                for (int g = lane; g < n_groups; g += 32) {
                    const float v = gs[g];
                    if (v != INFINITY) a = better(a, ArgMax{v, g});
                }
                a = warp_argmax(a);
                if (lane == 0 && a.i < n_groups) gs[a.i] = INFINITY;
                __syncwarp();
            }
        }
        __syncwarp();
        for (int e = lane; e < E; e += 32)
            if (gs[e / per] != INFINITY) c[e] = -INFINITY;
        __syncwarp();
    }
    uint32_t key[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) key[i] = lane + 32 * i < E ? order_key(c[lane + 32 * i]) : 0u;
    float total = 0.f;
    for (int r = 0; r < top; ++r) {
        const int e = max(take_largest<PER>(key, lane), 0);
        total += s[e];
        if (lane == 0) {
            chosen[(int64_t)t * top + r] = e;
            weights[(int64_t)t * top + r] = s[e];
        }
    }
    __syncwarp();
    if (normalize) {
        const float den = total + 1e-20f;
        for (int r = lane; r < top; r += 32) weights[(int64_t)t * top + r] = weights[(int64_t)t * top + r] / den * route_scale;
    }
    if (gate_col >= 0 && lane == 0) shared_gate[t] = 1.0f / (1.0f + expf(-z[gate_col]));
}

// One block: pairs per expert, offsets, and the pairs listed in expert order.  A pair's place among its expert's is what the
// counting returned; a thread holds those of its first kHeldPairs pairs, only pairs beyond that are counted off a second
// time.  (All of them twice, and the offsets summed up by one thread: 15.5 us for 12,288 pairs of 64 experts.)
constexpr int kHeldPairs = 16;

__global__ void __launch_bounds__(1024)
moe_group_kernel(const int* __restrict__ chosen, int n_pairs, int E, int* __restrict__ offsets /* [E+1] */,
                 int* __restrict__ order /* [pairs] */) {
    extern __shared__ int group_smem[];      // counts [E], places of the pairs that are not held [E]
    int* counts = group_smem;
    int* cursor = counts + E;
    pdl_launch_dependents();
    pdl_wait();
    for (int e = threadIdx.x; e < E; e += blockDim.x) counts[e] = 0;
    int expert[kHeldPairs], place[kHeldPairs];
#pragma unroll
    for (int h = 0; h < kHeldPairs; ++h) {
        const int i = threadIdx.x + h * 1024;
        expert[h] = i < n_pairs ? chosen[i] : -1;
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < kHeldPairs; ++h)
        if (expert[h] >= 0) place[h] = atomicAdd(&counts[expert[h]], 1);
    __syncthreads();
    if (n_pairs > kHeldPairs * 1024) {
        for (int e = threadIdx.x; e < E; e += blockDim.x) cursor[e] = counts[e];
        __syncthreads();
        for (int i = threadIdx.x + kHeldPairs * 1024; i < n_pairs; i += 1024) atomicAdd(&counts[chosen[i]], 1);
        __syncthreads();
    }
    if (threadIdx.x < 32) {
        int sum = 0;
        for (int base = 0; base < E; base += 32) {
            const int e = base + threadIdx.x, own = e < E ? counts[e] : 0;
            int incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o) incl += v;
            }
            if (e < E) {
                offsets[e] = sum + incl - own;
                counts[e] = sum + incl - own;
            }
            sum += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (threadIdx.x == 0) offsets[E] = sum;
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < kHeldPairs; ++h)
        if (expert[h] >= 0) order[counts[expert[h]] + place[h]] = threadIdx.x + h * 1024;
    for (int i = threadIdx.x + kHeldPairs * 1024; i < n_pairs; i += 1024) {
        const int e = chosen[i];
        order[counts[e] + atomicAdd(&cursor[e], 1)] = i;
    }
}

// The tokens' rows in expert order, a warp a row: out[r] = x[order[r] / top], rows of ``pieces`` 16-byte pieces.
__global__ void __launch_bounds__(256)
moe_gather_kernel(const uint4* __restrict__ x, const int* __restrict__ order, uint4* __restrict__ out, int n_pairs, int top, int pieces) {
    pdl_launch_dependents();
    pdl_wait();
    const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= n_pairs) return;
    const uint4* src = x + (int64_t)(order[r] / top) * pieces;
    uint4* dst = out + (int64_t)r * pieces;
#pragma unroll 4
    for (int i = lane; i < pieces; i += 32) dst[i] = src[i];
}

// What joins an expert's two products: silu(gate) * up, or the gate of two bounded products.
template <int MODE>
__device__ __forceinline__ float expert_gate(float g, float u, const GluClamp& clamp) {
    return MODE == 3 ? clamped_glu(g, u, clamp) : g / (1.0f + expf(-g)) * u;
}

constexpr int kTileM = 32, kTileN = 64, kTileK = 32;

// C[row_out(r)][n] = sum_k A[row_in(r)][k] * B_e[n][k] for the places r of expert e, tile by tile.
// GATED: A rows are tokens (pair / top), two weight stacks (gate, up) and the result is silu(gate) * up, written at
// row r.  Otherwise A rows are the places r themselves and the result goes to row pair(r).
template <typename T, int MODE>
__global__ void __launch_bounds__(256)
moe_tile_kernel(const T* __restrict__ A, const T* __restrict__ B0, const T* __restrict__ B1, T* __restrict__ C,
                const int* __restrict__ offsets, const int* __restrict__ order, int E, int top, int N, int K,
                const float* __restrict__ in_scale, GluClamp clamp) {
    constexpr bool GATED = MODE == 1 || MODE == 3, BY_TOKEN = MODE != 0;
    __shared__ float As[kTileM][kTileK + 1], Bs0[kTileN][kTileK + 1], Bs1[GATED ? kTileN : 1][kTileK + 1];
    __shared__ int s_tile[3];
    pdl_launch_dependents();
    pdl_wait();
    if (threadIdx.x == 0) {
        int tile = blockIdx.x, e = 0, found = -1, first = 0;
        for (; e < E; ++e) {
            const int n = offsets[e + 1] - offsets[e];
            const int tiles = (n + kTileM - 1) / kTileM;
            if (tile < tiles) { found = e; first = offsets[e] + tile * kTileM; break; }
            tile -= tiles;
        }
        s_tile[0] = found;
        s_tile[1] = first;
        s_tile[2] = found >= 0 ? min(kTileM, offsets[found + 1] - first) : 0;
    }
    __syncthreads();
    const int e = s_tile[0], r0 = s_tile[1], rows = s_tile[2];
    if (e < 0) return;
    const int n0 = blockIdx.y * kTileN;
    const T* W0 = B0 + (int64_t)e * N * K;
    const T* W1 = GATED ? B1 + (int64_t)e * N * K : nullptr;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;      // 4 columns, 2 rows a thread
    float acc0[2][4] = {}, acc1[2][4] = {};
    for (int k0 = 0; k0 < K; k0 += kTileK) {
        for (int i = threadIdx.x; i < kTileM * kTileK; i += 256) {
            const int r = i / kTileK, kk = i % kTileK;
            float v = 0.f;
            if (r < rows && k0 + kk < K) {
                const int64_t src = BY_TOKEN ? (int64_t)(order[r0 + r] / top) : (int64_t)(r0 + r);
                v = to_f32(A[src * K + k0 + kk]);
            }
            As[r][kk] = v;
        }
        for (int i = threadIdx.x; i < kTileN * kTileK; i += 256) {
            const int n = i / kTileK, kk = i % kTileK;
            const bool ok = n0 + n < N && k0 + kk < K;
            Bs0[n][kk] = ok ? to_f32(W0[(int64_t)(n0 + n) * K + k0 + kk]) : 0.f;
            if (GATED) Bs1[n][kk] = ok ? to_f32(W1[(int64_t)(n0 + n) * K + k0 + kk]) : 0.f;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < kTileK; ++kk) {
            const float a0 = As[ty * 2][kk], a1 = As[ty * 2 + 1][kk];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float b = Bs0[tx * 4 + j][kk];
                acc0[0][j] = fmaf(a0, b, acc0[0][j]);
                acc0[1][j] = fmaf(a1, b, acc0[1][j]);
                if (GATED) {
                    const float b1 = Bs1[tx * 4 + j][kk];
                    acc1[0][j] = fmaf(a0, b1, acc1[0][j]);
                    acc1[1][j] = fmaf(a1, b1, acc1[1][j]);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = ty * 2 + i;
        if (r >= rows) continue;
        const int64_t dst = BY_TOKEN ? (int64_t)(r0 + r) : (int64_t)order[r0 + r];
        const float sc = (MODE == 2 && in_scale != nullptr) ? in_scale[order[r0 + r]] : 1.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float v = acc0[i][j];
            if (GATED) v = expert_gate<MODE>(v, acc1[i][j], clamp);
            if (MODE == 2) { v = fmaxf(v * sc, 0.f); v *= v; }
            C[dst * N + n] = from_f32<T>(v);
        }
    }
}


// Few pairs (a decode step): a product that streams the weights of every chosen expert once, whatever the number of pairs
// that chose it.  A block belongs to a pair and 32 weight rows (32 features; 16 of gate and 16 of up where there are
// two stacks) and works for all pairs of its expert if no earlier pair chose that expert, else it leaves at once: no grouping
// kernel runs ahead of it, and H and Y are indexed by pair.  The pairs are the 8 columns of mma.sync m16n8k16 (fp32
// accumulation), the weights its 16 rows, straight from memory in 16-byte loads; the 8 warps take turns at 32-wide slices of K
// and meet in shared memory.  A weight row of another pair with the same expert costs a column that is there anyway.
// Bound by the weights' way from memory.  Before, every pair was a matrix-vector product of its own over an input row in
// shared memory, whose reads met eight to a bank: in decode steps 16 tokens of 4 choices among 32 experts of 512 x 1024 took 25.4 us for
// gate and up and 17.9 us for down, now 14.5 and 8.7; 4 tokens of 6 choices among 64 experts of 768 x 2048 27.9 and 17.6 us, now 22.4 and
// 14.6.  Four blocks an SM, two slices of K a warp in flight, hide a block's start and its sums behind the others' loads (two blocks of
// four slices: 20.0 and 12.2 us at the first of these sizes).
constexpr int kFewRows = 32;

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// weights are used once: keep them out of L1
__device__ __forceinline__ uint4 load_once(const bf16* p) {
    uint4 v;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

template <int MODE>
__global__ void __launch_bounds__(256, 4)
moe_few_pairs_kernel(const bf16* __restrict__ A, const bf16* __restrict__ B0, const bf16* __restrict__ B1, bf16* __restrict__ C,
                     const int* __restrict__ chosen, int n_pairs, int top, int N, int K, const float* __restrict__ in_scale, GluClamp clamp) {
    constexpr bool GATED = MODE == 1 || MODE == 3, BY_TOKEN = MODE != 0;
    constexpr int kFeatures = GATED ? kFewRows / 2 : kFewRows;
    extern __shared__ int same[];                              // the pairs that chose this expert, in order
    __shared__ float red[8][kFewRows][8 + 1];
    __shared__ int s_count;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
    const int pair = blockIdx.x, n0 = blockIdx.y * kFeatures;
    if (BY_TOKEN) pdl_wait();
    const int e = chosen[pair];
    if (warp == 0) {
        int count = 0;
        for (int base = 0; base < n_pairs; base += 32) {
            const bool mine = base + lane < n_pairs && chosen[base + lane] == e;
            const unsigned all = __ballot_sync(0xffffffffu, mine);
            if (mine) same[count + __popc(all & ((1u << lane) - 1u))] = base + lane;
            count += __popc(all);
        }
        if (lane == 0) s_count = count;
    }
    __syncthreads();
    if (same[0] != pair) return;                               // an earlier pair's blocks do this expert
    const int count = s_count;
    if (!BY_TOKEN) {
        // The kernel ahead is the first product, which lets this one start only once it has itself seen the choice of experts:
        // the choice may be read, and the weights asked for, before its rows are waited for.
        const int lines = (K * 2 + 127) / 128;
        const bf16* first = B0 + ((int64_t)e * N + n0) * K;
        for (int i = threadIdx.x; i < min(kFeatures, N - n0) * lines; i += 256) {
            const int r = i / lines, l = i - r * lines;
            asm volatile("prefetch.global.L2 [%0];" :: "l"(first + (int64_t)r * K + l * 64));
        }
        pdl_wait();
    }
    // fragment rows g and g + 8 of two 16-row tiles; rows past the last feature read the last one and are never stored
    const bf16* w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bf16* stack = GATED && i >= 2 ? B1 : B0;
        const int f = GATED ? n0 + g + 8 * (i & 1) : n0 + g + 8 * i;
        w[i] = stack + ((int64_t)e * N + min(f, N - 1)) * K + 8 * j;
    }
    const int slices = (K + 31) / 32;
    for (int c0 = 0; c0 < count; c0 += 8) {
        const int mine = same[min(c0 + g, count - 1)];
        const bf16* x = A + (int64_t)(BY_TOKEN ? mine / top : mine) * K + 8 * j;
        float acc[2][4] = {};
#pragma unroll 2
        for (int s = warp; s < slices; s += 8) {
            uint4 a[4] = {}, b = make_uint4(0, 0, 0, 0);
            if (32 * s + 8 * j < K) {                          // K is a multiple of 8: a lane's piece is whole or absent
                b = __ldg(reinterpret_cast<const uint4*>(x + 32 * s));
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = load_once(w[i] + 32 * s);
            }
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                mma_bf16_16816(acc[m], a[2 * m].x, a[2 * m + 1].x, a[2 * m].y, a[2 * m + 1].y, b.x, b.y);
                mma_bf16_16816(acc[m], a[2 * m].z, a[2 * m + 1].z, a[2 * m].w, a[2 * m + 1].w, b.z, b.w);
            }
        }
        if (c0 + 8 >= count) pdl_launch_dependents();
        if (c0) __syncthreads();                               // the last group's sums have been read
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int q = 0; q < 4; ++q) red[warp][16 * m + g + 8 * (q >> 1)][2 * j + (q & 1)] = acc[m][q];
        __syncthreads();
        const int f = threadIdx.x % kFeatures, col = threadIdx.x / kFeatures;
        if (col < 8 && c0 + col < count && n0 + f < N) {
            const int dst = same[c0 + col];
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                s0 += red[v][f][col];
                if (GATED) s1 += red[v][(f + kFeatures) & (kFewRows - 1)][col];
            }
            if (MODE == 2) { s0 = fmaxf(s0 * (in_scale != nullptr ? in_scale[dst] : 1.f), 0.f); s0 *= s0; }
            C[(int64_t)dst * N + n0 + f] = __float2bfloat16_rn(GATED ? expert_gate<MODE>(s0, s1, clamp) : s0);
        }
    }
}

// The same two products for few pairs, by pair: gated: C = H [pairs, N] by pair from x [tokens, K]; else C = Y [pairs, N]
// from H [pairs, K] by pair.  bf16, K a multiple of 8, at most 8192 pairs.  Mode 0 is to be launched right behind one of the others
// with the same choice of experts (or behind a kernel that has run to its end): it reads ``chosen`` before it waits.
// mode 1: gated; 3: the gate of two bounded products (limit, slope, offset); 2: one stack, relu(in_scale[pair] * product)^2, from x by pair; 0: the down product.
CPM_API int cpm_moe_pair_product(const void* A, const void* B0, const void* B1, void* C, const int* chosen, int n_pairs, int top,
                                 int N, int K, int mode, const float* in_scale, float limit, float slope, float offset,
                                 cudaStream_t stream) {
    if (n_pairs <= 0) return CPM_OK;
    if (top < 1 || N < 1 || K < 8 || K % 8 || ((uintptr_t)A & 15) || ((uintptr_t)B0 & 15) || ((uintptr_t)B1 & 15) || n_pairs > 8192)
        return CPM_BAD_ARGUMENT;
    if (mode < 0 || mode > 3) return CPM_BAD_ARGUMENT;
    const int features = mode == 1 || mode == 3 ? kFewRows / 2 : kFewRows;
    const dim3 grid(n_pairs, (N + features - 1) / features);
    if (grid.y > 65535) return CPM_BAD_ARGUMENT;
    const GluClamp clamp{limit, slope, offset};
#define CPM_FEW(M) cpm_launch(kLaunchProduct, moe_few_pairs_kernel<M>, grid, dim3(256), (size_t)n_pairs * sizeof(int), stream,      \
                              (const bf16*)A, (const bf16*)B0, (const bf16*)B1, (bf16*)C, chosen, n_pairs, top, N, K, in_scale, clamp)
    if (mode == 1) CPM_FEW(1); else if (mode == 2) CPM_FEW(2); else if (mode == 3) CPM_FEW(3); else CPM_FEW(0);
#undef CPM_FEW
    return launch_status();
}

// out[t] = sum_k weights[t][k] * Y[t * top + k] + gate[t] * shared[t]   (weights null: all 1)
template <typename T>
__global__ void moe_combine_kernel(const T* __restrict__ Y, const float* __restrict__ weights, const T* __restrict__ shared,
                                   const float* __restrict__ gate, T* __restrict__ out, int top, int W) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = blockIdx.x;
    for (int c = threadIdx.x; c < W; c += blockDim.x) {
        float v = 0.f;
        for (int k = 0; k < top; ++k) v = fmaf(weights ? weights[t * top + k] : 1.f, to_f32(Y[(t * top + k) * W + c]), v);
        if (shared) v = fmaf(gate ? gate[t] : 1.f, to_f32(shared[t * W + c]), v);
        out[t * W + c] = from_f32<T>(v);
    }
}

// The same sums in the same order for rows of whole 16-byte pieces: a thread takes 8 columns of a token, its loads of
// all choices in flight together.  One column a thread and load: 4 tokens of 6 choices and 2048 columns 11.0 us, 2048 tokens 31 us.
__global__ void __launch_bounds__(128)
moe_combine_wide_kernel(const bf16* __restrict__ Y, const float* __restrict__ weights, const bf16* __restrict__ shared,
                        const float* __restrict__ gate, bf16* __restrict__ out, int top, int W) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = blockIdx.y;
    const int c = (blockIdx.x * 128 + threadIdx.x) * 8;
    if (c >= W) return;
    float v[8] = {};
    auto add = [&](const bf16* row, float weight) {
        const uint4 raw = *reinterpret_cast<const uint4*>(row + c);
        const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(p[i]);
            v[2 * i] = fmaf(weight, f.x, v[2 * i]);
            v[2 * i + 1] = fmaf(weight, f.y, v[2 * i + 1]);
        }
    };
#pragma unroll 8
    for (int k = 0; k < top; ++k) add(Y + (t * top + k) * W, weights ? weights[t * top + k] : 1.f);
    if (shared) add(shared + t * W, gate ? gate[t] : 1.f);
    store4(out + t * W + c, make_float4(v[0], v[1], v[2], v[3]));
    store4(out + t * W + c + 4, make_float4(v[4], v[5], v[6], v[7]));
}

static int g_moe_tensor_cores = 1;
// 0: the bf16 products stay on the CUDA cores too (for comparisons and tests)
CPM_API int cpm_set_moe_tensor_cores(int on) {
    g_moe_tensor_cores = on;
    return CPM_OK;
}

CPM_API int cpm_moe_route(const float* logits, int ld, const float* correction, int* chosen, float* weights, float* shared_gate,
                          int gate_col, int n_tokens, int E, int top, int n_groups, int keep, const float* bias, int top_first,
                          int group_top2, int normalize, float route_scale, cudaStream_t stream) {
    if (n_tokens <= 0) return CPM_OK;
    if (top_first < 0 || top_first > 2 || (!top_first && !correction)) return CPM_BAD_ARGUMENT;
    if (top_first == 1 && (n_groups != 1 || normalize)) return CPM_BAD_ARGUMENT;
    if (E < 1 || E > 32 * kRouteMaxPerLane || top < 1 || top > E || n_groups < 1 || E % n_groups || keep < 1 || keep > n_groups ||
        top > keep * (E / n_groups))
        return CPM_BAD_ARGUMENT;
    const int warps = 4;
    const size_t smem = (size_t)warps * (2 * E + n_groups) * sizeof(float);
#define CPM_ROUTE(PER) cpm_launch(kLaunchNorm, moe_route_kernel<PER>, dim3((n_tokens + warps - 1) / warps), dim3(warps * 32), smem, stream,   \
                                  logits, ld, correction, chosen, weights, shared_gate, gate_col, n_tokens, E, top, n_groups, keep, bias,     \
                                  top_first, group_top2, normalize, route_scale)
    if (E <= 32) CPM_ROUTE(1); else if (E <= 64) CPM_ROUTE(2); else if (E <= 128) CPM_ROUTE(4); else CPM_ROUTE(kRouteMaxPerLane);
#undef CPM_ROUTE
    return launch_status();
}

CPM_API int cpm_moe_group(const int* chosen, int n_pairs, int E, int* offsets, int* order, cudaStream_t stream) {
    if (n_pairs <= 0) return CPM_OK;
    if (E < 1 || E > 4096) return CPM_BAD_ARGUMENT;
    cpm_launch(kLaunchNorm, moe_group_kernel, dim3(1), dim3(1024), (size_t)2 * E * sizeof(int), stream, chosen, n_pairs, E, offsets,
               order);
    return launch_status();
}

// Whether a product of many pairs goes to the tensor cores.
static bool expert_tiles(const void* A, const void* B0, const void* B1, const void* rows, int E, int N, int K, int mode, int dtype) {
    return dtype == CPM_BF16 && K % 8 == 0 && !(((uintptr_t)A | (uintptr_t)B0 | (uintptr_t)B1) & 15) && E <= 512 && (int64_t)E * N < (1 << 30) &&
           g_moe_tensor_cores && (mode == 0 || (rows != nullptr && ((uintptr_t)rows & 15) == 0));
}

// Kernels that cpm_moe_expert_product launches for these arguments.
CPM_API int cpm_moe_expert_product_kernels(const void* A, const void* B0, const void* B1, const void* rows, int E, int N, int K, int mode, int dtype) {
    return mode != 0 && expert_tiles(A, B0, B1, rows, E, N, K, mode, dtype) ? 2 : 1;      // the rows in expert order, then the product
}

// mode 1: A = x [tokens, K], B0 = gate stack [E, N, K], B1 = up stack, C = H [pairs, N] in expert order.
// mode 3: the same with the gate of two bounded products (limit, slope, offset).
// mode 2: A = x, B0 = up stack, C = H = relu(in_scale[pair] * product)^2 in expert order (in_scale null: 1).
// mode 0: A = H [pairs, K] in expert order, B0 = down stack [E, N, K], C = Y [pairs, N] by pair.
// rows: room for the tokens' rows in expert order, [pairs, K], which the tensor cores need in modes 1 to 3 (without it, null, these run
// on the CUDA cores); it may be memory that a later product of the same call writes.
CPM_API int cpm_moe_expert_product(const void* A, const void* B0, const void* B1, void* C, const int* offsets, const int* order, void* rows,
                                   int n_pairs, int E, int top, int N, int K, int mode, const float* in_scale, float limit,
                                   float slope, float offset, int dtype, cudaStream_t stream) {
    if (n_pairs <= 0) return CPM_OK;
    if (E < 1 || top < 1 || N < 1 || K < 1 || mode < 0 || mode > 3) return CPM_BAD_ARGUMENT;
    const GluClamp clamp{limit, slope, offset};
    if (expert_tiles(A, B0, B1, rows, E, N, K, mode, dtype)) {
        if (mode != 0)
            cpm_launch(kLaunchNorm, moe_gather_kernel, dim3((n_pairs + 7) / 8), dim3(256), 0, stream, (const uint4*)A, order, (uint4*)rows,
                       n_pairs, top, K / 8);
        return moe_product_tcgen05(mode == 0 ? A : rows, B0, B1, C, offsets, order, n_pairs, E, N, K, mode, in_scale, clamp, stream);
    }
    const dim3 grid((n_pairs + kTileM - 1) / kTileM + E, (N + kTileN - 1) / kTileN);
    if (grid.y > 65535) return CPM_BAD_ARGUMENT;
#define CPM_MOE(TT, G) cpm_launch(kLaunchProduct, moe_tile_kernel<TT, G>, grid, dim3(256), 0, stream, (const TT*)A, (const TT*)B0, \
                                  (const TT*)B1, (TT*)C, offsets, order, E, top, N, K, in_scale, clamp)
    if (dtype == CPM_BF16) { if (mode == 1) CPM_MOE(bf16, 1); else if (mode == 2) CPM_MOE(bf16, 2); else if (mode == 3) CPM_MOE(bf16, 3); else CPM_MOE(bf16, 0); }
    else { if (mode == 1) CPM_MOE(float, 1); else if (mode == 2) CPM_MOE(float, 2); else if (mode == 3) CPM_MOE(float, 3); else CPM_MOE(float, 0); }
#undef CPM_MOE
    return launch_status();
}

CPM_API int cpm_moe_combine(const void* Y, const float* weights, const void* shared, const float* gate, void* out, int n_tokens,
                            int top, int W, int dtype, cudaStream_t stream) {
    if (n_tokens <= 0) return CPM_OK;
    const dim3 block(W >= 1024 ? 256 : 128);
    if (dtype == CPM_BF16 && W % 8 == 0 && n_tokens <= 65535 && !(((uintptr_t)Y | (uintptr_t)shared | (uintptr_t)out) & 15))
        cpm_launch(kLaunchNorm, moe_combine_wide_kernel, dim3((W / 8 + 127) / 128, n_tokens), dim3(128), 0, stream, (const bf16*)Y, weights,
                   (const bf16*)shared, gate, (bf16*)out, top, W);
    else if (dtype == CPM_BF16)
        cpm_launch(kLaunchNorm, moe_combine_kernel<bf16>, dim3(n_tokens), block, 0, stream, (const bf16*)Y, weights, (const bf16*)shared,
                   gate, (bf16*)out, top, W);
    else
        cpm_launch(kLaunchNorm, moe_combine_kernel<float>, dim3(n_tokens), block, 0, stream, (const float*)Y, weights,
                   (const float*)shared, gate, (float*)out, top, W);
    return launch_status();
}
