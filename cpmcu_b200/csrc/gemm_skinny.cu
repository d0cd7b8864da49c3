// C[M,N] = alpha * X[M,K] * W[N,K]^T for a handful of rows (decode: M = tokens of the
// step, up to 16): a weight-streaming kernel.  The weights are read exactly once, with
// 16-byte loads along K straight into tensor-core fragments; the activations are tiny and
// come from the caches.
//
// A block owns 16 weight rows (one m16 tile of mma.sync m16n8k16, the weight as the A
// operand, the tokens as the n8 columns) and its 8 warps take interleaved 32-element
// slices of K, so that together they walk each row contiguously; the warps' partial sums
// meet in shared memory.  A thread's 8 consecutive K elements stand for the k-slots of two
// mma instructions; the sum over K does not care about the order as long as both operands
// use the same assignment.
//
// Epilogues: bf16 output; fp32 output times alpha (the output head); SiLU(gate)*up for a
// gate_up matrix whose rows are interleaved in blocks of 8 (8 gate rows, then the 8 up
// rows of the same features), so that gate and up of a feature meet in one tile; other gates of two values in the same
// layout; relu(x)^2 for a feed-forward without a gate; fp32 output capped by c * tanh(x / c).
// The reference calls cublasGemmEx for every product (src/model/linear.cuh:8-37) and runs
// the gated activation as a kernel of its own (src/model/activation.cuh:6-18).
#include "common.cuh"

// 2, 3: act(gate) * up with SiLU, with the tanh form of GELU; 4: relu(x)^2; 5: the gate of two bounded products
// (GluClamp); 6: fp32 output c * tanh(x / c), c = clamp.limit
enum : int { EPI_BF16 = 0, EPI_F32 = 1, EPI_SILU = 2, EPI_GELU = 3, EPI_RELU2 = 4, EPI_GLU_CLAMP = 5, EPI_F32_CAP = 6 };
__host__ __device__ constexpr bool skinny_gated(int epi) { return epi == EPI_SILU || epi == EPI_GELU || epi == EPI_GLU_CLAMP; }

// 128-byte lines of each weight row a block asks L2 for at its start (and, under programmatic dependent
// launch, before it waits for the kernel ahead of it).  Eight lines bring the first loads of the main loop
// forward and were worth 0.6 to 3.7 % of a decode step, depending on the machine; 16 and more cost time.
static int g_skinny_prefetch_lines = 8;

CPM_API void cpm_set_skinny_prefetch_lines(int n) { g_skinny_prefetch_lines = n < 0 ? 0 : n; }

__device__ __forceinline__ void mma_16816_s(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                            uint32_t b0, uint32_t b1) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// What the kernel ahead has written.  Not __ldg: memory that this kernel's lifetime sees written is not read-only, and the compiler may move
// such a load in front of the wait.
__device__ __forceinline__ uint4 ld_written16(const void* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
// weights are used once: keep them out of L1
__device__ __forceinline__ uint4 ld_stream16(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// The second launch bound (one block per SM suffices) matters: it lets the compiler spend registers on
// keeping the loads of eight K steps in flight instead of saving them for occupancy; with it the kernel
// went from 4.5 to 6.1 TB/s on the down projection.  With two tiles of token columns (9 to 16 rows) the
// kernel would take 166 registers and lose the second block per SM, so there the bound is two blocks (53
// instead of 59 us on the gate_up shape, which is what cuBLAS with the activation kernel takes).  Every block
// reads all the activations from L1 and L2, so the engine hands it 9 to 16 rows only for the products whose
// blocks * rows * K stays small (QKV, O and down of the 8B sizes, not gate_up or the head).
// kShort (K up to kShortK): a warp has at most four steps (kFlight: one up to K 256, two up to 512), whose loads take few registers, and a
// block lives for little more than their latency; four blocks an SM (three with two tiles of columns) hide one's start and sums behind the others' loads.  Whole calls with K
// of 1024 in most products: 17.6 -> 15.5 to 16.4 ms (one row), 29.4 -> 27.6 (16 rows).  At 2048 eight steps in flight are worth more than
// the other two blocks (24.1 against 24.8 ms for four rows), at 4096 27.7 against 29.8.
// A block asks for kFlight steps a warp whether K has them or not (steps beyond the last are its again), so the number follows K: with four
// for all of these, a product of K 64 to 256 took up to twice as long.  us a product in a row of independent ones, four steps and as it is, eight
// rows: 2,048 x 64 2.90 and 1.24, 4,096 x 128 3.16 and 1.35, 6,144 x 256 3.33 and 1.66, 2,048 x 512 2.82 and 2.03; sixteen rows of 2,048 x 128 3.24 and
// 1.39.  (Steps left out by a branch, four for all: 1.79, 2.09, 2.47, 2.30, 2.26, and 1,024 x 1,024 2.64 instead of 2.43.)
constexpr int kShortK = 1024;
// Long rows in blocks for at most half of the SMs: sixteen warps a block instead of eight, since no second block comes to keep more of
// the weights in flight.  One row, inputs cold, eight and sixteen warps: 1,024 weight rows of K 4,096 4.4 and 3.7 us, of 8,192 7.5 and 6.4, 256 of
// 16,384 11.4 and 8.6.  Such a block takes an SM's whole register file and cannot be placed before the kernel ahead has left it, and at K of
// 2,560 and 3,072 that costs more than it gives: 3.6 and 4.5, 4.9 and 5.3 us.
constexpr int kManyWarpsK = 4096;
// In a decode step's chain a product of a few MB lives for little more than latencies: of its launch, of its weights, of its activations.  So
// the first kFlight steps' weights (all of them up to K 1,024 and, with eight steps, 2,048) are on their way into registers before the kernel
// ahead has ended (kAhead), and a grid whose blocks the SMs hold all at once (``let_go``) lets the next kernel's blocks in at its start, so that
// these do the same; a grid of several waves would lose slots on the SMs to blocks that do nothing but wait, and lets them in
// after its main loop.  us of a recorded decode step before, with let_go alone, with both: 0.5B one row 585, 577, 549, 16 rows
// 862, 821, 787; 8B eight rows 3,305, 3,259, 3,244; Mufevik 1k 16 rows 647, 620, 597; Rabadra 2k four rows 707, 684, 671.
// With two tiles of columns and K from 2,048 on the registers do not hold a step's activations beside eight steps' weights: the loop that asks
// for both step by step is faster (us of a recorded step of 16 rows with the weights ahead and without: Dinutar 2k 444 and 428, Kipizen
// 2k 908 and 892, Lukelorn 2k 743 and 728, Rabadra 2k 1,010 and 991, Reravik 2k 822 and 808, the 8B sizes 3,708 and 3,707).
// Below 2,048 that loop has less than a round of eight steps a warp and asks for one after the other: 16 rows of 2,048 x 1,536 4.61 us with the weights
// ahead and 5.55 without, 2,048 x 1,056 4.01 and 4.3.
template <int NT, int EPI, int kSkinnyWarps, int kFlight, bool kAhead>
__global__ void __launch_bounds__(kSkinnyWarps * 32, kFlight < 8 ? (NT == 1 ? 4 : 3) : (NT == 1 || kSkinnyWarps > 8 ? 1 : 2))
skinny_gemm_kernel(const bf16* __restrict__ W, const bf16* __restrict__ X, void* __restrict__ out, int M, int N, int K,
                   float alpha, int prefetch_lines, int let_go, GluClamp clamp) {
    constexpr int MT = NT * 8;                          // token columns
    __shared__ float red[kSkinnyWarps][16][MT + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, j = lane & 3;
    const int n0 = blockIdx.x * 16;
    if (let_go) pdl_launch_dependents();
    // Before the kernel ahead of this one in the stream has finished, this block already asks for its
    // 16 weight rows to be brought into L2: weights are never written, and the tail of one product then
    // overlaps with the start of the next.
    {
        const int lines = min(prefetch_lines, (K * 2 + 127) / 128);      // 128-byte lines per row
        for (int i = threadIdx.x; i < 16 * lines; i += kSkinnyWarps * 32) {
            const int r = i / lines, l = i - r * lines;
            const char* p = reinterpret_cast<const char*>(W + (int64_t)min(n0 + r, N - 1) * K) + l * 128;
            asm volatile("prefetch.global.L2 [%0];" :: "l"(p));
        }
    }
    // Rows beyond N and token columns beyond M read a valid row instead and their results are never
    // stored: rows of the product are independent, so no load needs a predicate.
    const bf16* w0 = W + (int64_t)min(n0 + g, N - 1) * K + 8 * j;
    const bf16* w1 = W + (int64_t)min(n0 + g + 8, N - 1) * K + 8 * j;
    const int steps = K / 32;
    // the first steps' weights are on their way into registers before the wait
    constexpr bool kShort = kFlight < 8;
    const bool any = kFlight > 1 || warp < steps;
    auto step_of = [&](int i) { return min(warp + i * kSkinnyWarps, steps - 1); };
    uint4 lo[kFlight], hi[kFlight];
    if constexpr (kAhead) {
#pragma unroll
        for (int i = 0; i < kFlight; ++i) {
            const int s = step_of(i);
            if (!any) break;
            lo[i] = ld_stream16(w0 + 32 * s);
            hi[i] = ld_stream16(w1 + 32 * s);
        }
    }
    pdl_wait();
    const bf16* xp[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) xp[nt] = X + (int64_t)min(nt * 8 + g, M - 1) * K + 8 * j;
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    if constexpr (kAhead) {
        constexpr int kAtOnce = NT == 1 || kShort ? kFlight : kFlight / 2;       // steps whose activations are asked for together
#pragma unroll
        for (int i0 = 0; i0 < kFlight; i0 += kAtOnce) {
            uint4 b[kAtOnce][NT];
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
                    if (any) b[i][nt] = ld_written16(xp[nt] + 32 * step_of(i0 + i));
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i)
                if (warp + (i0 + i) * kSkinnyWarps < steps) {
                    const uint4 l = lo[i0 + i], h = hi[i0 + i];
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        mma_16816_s(acc[nt], l.x, h.x, l.y, h.y, b[i][nt].x, b[i][nt].y);
                        mma_16816_s(acc[nt], l.z, h.z, l.w, h.w, b[i][nt].z, b[i][nt].w);
                    }
                }
        }
    }
    if constexpr (!kShort) {
#pragma unroll kFlight
        for (int s = warp + (kAhead ? kFlight * kSkinnyWarps : 0); s < steps; s += kSkinnyWarps) {
            const uint4 l = ld_stream16(w0 + 32 * s);
            const uint4 h = ld_stream16(w1 + 32 * s);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const uint4 b = ld_written16(xp[nt] + 32 * s);
                mma_16816_s(acc[nt], l.x, h.x, l.y, h.y, b.x, b.y);
                mma_16816_s(acc[nt], l.z, h.z, l.w, h.w, b.z, b.w);
            }
        }
    }
    if (!let_go) pdl_launch_dependents();
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        red[warp][g][nt * 8 + 2 * j] = acc[nt][0];
        red[warp][g][nt * 8 + 2 * j + 1] = acc[nt][1];
        red[warp][g + 8][nt * 8 + 2 * j] = acc[nt][2];
        red[warp][g + 8][nt * 8 + 2 * j + 1] = acc[nt][3];
    }
    __syncthreads();
    if (skinny_gated(EPI)) {
        // rows 0..7 are gate, rows 8..15 up, of features (n0 / 2) + 0..7
        for (int o = threadIdx.x; o < 8 * MT; o += kSkinnyWarps * 32) {
            const int f = o & 7, tok = o >> 3;
            if (tok >= M) continue;
            float gate = 0.f, up = 0.f;
#pragma unroll
            for (int w = 0; w < kSkinnyWarps; ++w) {
                gate += red[w][f][tok];
                up += red[w][f + 8][tok];
            }
            const int feature = (n0 >> 1) + f;
            if (feature < (N >> 1)) {
                float h;
                if (EPI == EPI_GLU_CLAMP) {
                    h = clamped_glu(gate, up, clamp);
                } else if (EPI == EPI_GELU) {
                    h = 0.5f * gate * (1.0f + tanhf(0.7978845608028654f * (gate + 0.044715f * gate * gate * gate))) * up;
                } else {
                    const float s = 1.0f / (1.0f + expf(-gate));
                    h = gate * s * up;
                }
                reinterpret_cast<bf16*>(out)[(int64_t)tok * (N >> 1) + feature] = __float2bfloat16_rn(h);
            }
        }
    } else {
        for (int o = threadIdx.x; o < 16 * MT; o += kSkinnyWarps * 32) {
            const int row = o & 15, tok = o >> 4;
            if (tok >= M || n0 + row >= N) continue;
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < kSkinnyWarps; ++w) sum += red[w][row][tok];
            if (EPI == EPI_RELU2) {
                sum = fmaxf(sum, 0.f);
                sum *= sum;
            }
            if (EPI == EPI_F32_CAP) {
                const float cap = clamp.limit;
                reinterpret_cast<float*>(out)[(int64_t)tok * N + n0 + row] = cap * tanhf(alpha * sum / cap);
            } else if (EPI == EPI_F32) reinterpret_cast<float*>(out)[(int64_t)tok * N + n0 + row] = alpha * sum;
            else reinterpret_cast<bf16*>(out)[(int64_t)tok * N + n0 + row] = __float2bfloat16_rn(alpha * sum);
        }
    }
}

template <int NT, int EPI>
static int launch_skinny_epi(const void* W, const void* X, void* out, int M, int N, int K, float alpha,
                             const GluClamp& clamp, cudaStream_t stream) {
    const unsigned blocks = (unsigned)((N + 15) / 16), sms = (unsigned)device_sms();
    // per_sm: blocks an SM holds by their registers (128 a thread beyond K 1,024, 64 and 80 with four steps)
    auto start = [&](auto kern, int warps, unsigned per_sm) {
        cpm_launch(kLaunchProduct, kern, blocks, warps * 32, 0, stream, (const bf16*)W, (const bf16*)X, out, M, N, K, alpha,
                   g_skinny_prefetch_lines, (int)(blocks <= per_sm * sms), clamp);
    };
    if (K >= kManyWarpsK && 2 * blocks <= sms)
        start(skinny_gemm_kernel<NT, EPI, 16, 8, NT == 1>, 16, 1u);
    else if (K <= kShortK / 4)
        start(skinny_gemm_kernel<NT, EPI, 8, 1, true>, 8, NT == 1 ? 4u : 3u);
    else if (K <= kShortK / 2)
        start(skinny_gemm_kernel<NT, EPI, 8, 2, true>, 8, NT == 1 ? 4u : 3u);
    else if (K <= kShortK)
        start(skinny_gemm_kernel<NT, EPI, 8, 4, true>, 8, NT == 1 ? 4u : 3u);
    else
        start(NT == 1 || K < 2 * kShortK ? skinny_gemm_kernel<NT, EPI, 8, 8, true> : skinny_gemm_kernel<NT, EPI, 8, 8, NT == 1>, 8, 2u);
    return launch_status();
}

template <int NT>
static int launch_skinny(const void* W, const void* X, void* out, int M, int N, int K, float alpha, int epilogue,
                         const GluClamp& clamp, cudaStream_t stream) {
    if (epilogue == EPI_BF16) return launch_skinny_epi<NT, EPI_BF16>(W, X, out, M, N, K, alpha, clamp, stream);
    if (epilogue == EPI_F32) return launch_skinny_epi<NT, EPI_F32>(W, X, out, M, N, K, alpha, clamp, stream);
    if (epilogue == EPI_SILU) return launch_skinny_epi<NT, EPI_SILU>(W, X, out, M, N, K, alpha, clamp, stream);
    if (epilogue == EPI_GELU) return launch_skinny_epi<NT, EPI_GELU>(W, X, out, M, N, K, alpha, clamp, stream);
    if (epilogue == EPI_RELU2) return launch_skinny_epi<NT, EPI_RELU2>(W, X, out, M, N, K, alpha, clamp, stream);
    if (epilogue == EPI_GLU_CLAMP) return launch_skinny_epi<NT, EPI_GLU_CLAMP>(W, X, out, M, N, K, alpha, clamp, stream);
    if (epilogue == EPI_F32_CAP) return launch_skinny_epi<NT, EPI_F32_CAP>(W, X, out, M, N, K, alpha, clamp, stream);
    return CPM_BAD_ARGUMENT;
}

// W [N,K] bf16, X [M,K] bf16 (both contiguous); out [M,N] bf16 or fp32, or [M,N/2] bf16 for the gated
// epilogues.  Takes M <= 16 and K a multiple of 32; N is free (for the gated epilogues a multiple of 16).  limit, slope and
// offset belong to the bounded gate; the capped epilogue reads its cap from ``limit``.
CPM_API int cpm_gemm_skinny_bf16(const void* W, const void* X, void* out, int M, int N, int K, float alpha,
                                 int epilogue, float limit, float slope, float offset, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return CPM_OK;
    if (M > 16 || K <= 0 || K % 32 != 0) return CPM_BAD_ARGUMENT;
    if (skinny_gated(epilogue) && N % 16 != 0) return CPM_BAD_ARGUMENT;
    if (epilogue == EPI_F32_CAP && !(limit > 0.f)) return CPM_BAD_ARGUMENT;
    const GluClamp clamp{limit, slope, offset};
    if (M <= 8) return launch_skinny<1>(W, X, out, M, N, K, alpha, epilogue, clamp, stream);
    return launch_skinny<2>(W, X, out, M, N, K, alpha, epilogue, clamp, stream);
}
