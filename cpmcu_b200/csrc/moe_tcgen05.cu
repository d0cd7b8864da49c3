// The experts' products of many (token, choice) pairs on the fifth-generation tensor cores (bf16, fp32 accumulation).
//
// The weights are the rows of the product here and the pairs its columns:  D[feature, place] = W_e[feature, :] . x[place, :].
// What bounds these products is the reading of the experts' weights (2048 tokens of 6 choices among 64 experts of 768 x 2048:
// 403 MB for gate and up, 192 pairs an expert), so a tile takes 128 features of one expert and ALL its pairs, up to 256 (the
// widest instruction): every weight is then read from memory once, and an expert of few pairs pays for 16 columns at least,
// not for 128 rows.  An expert of more pairs is cut into equal chunks, which are neighbours in the order of the tiles
// and share the weights in L2.  Tiles of 128 pairs x 64 features on mma.sync took 404 us for gate and up and 352 us for
// down at that size, a fifth of what the memory gives.
//
// The pairs' rows lie in expert order: the down product reads what the first wrote so, and for the first a copy kernel lays
// the tokens' rows out (19 us for 12,288 rows of 2048; gathering them in this kernel, four rows to a TMA instruction, took 112 us
// of its 241).  At that size gate and up take 123 us and down 60 us; the weights alone 62 and 31 us.
//
// A block is persistent, one an SM.  Warp 0 is the TMA producer: 128 weight rows by 64 of K (two such tiles, gate and up,
// where there are two stacks) and the chunk's rows.  Warp 1 allocates tensor memory and issues
// the MMAs; the instruction's N is the chunk's size, rounded up to 16.  Warps 2 to 9 are the epilogue, two for each quarter
// of the 128 TMEM lanes; a lane is a feature and a column a pair, so gate and up of one value meet in one thread;
// 32 pairs x 128 features at a time pass through shared memory, and every output row is written in pieces of 256 bytes.
// With two stacks the two accumulators of 256 columns fill the tensor memory; with one there are two to take turns.
//
// Every wait is bounded: where a bound is hit the block records an error code, stops taking work, waits for its copies in
// flight, frees its tensor memory and returns.  No multicast and no clusters are used.
#include "tcgen05.cuh"

namespace moe5 {

using namespace tc5;

constexpr int kFeatures = 128, kMaxPairs = 256, kBlockK = 64;
constexpr int kWeightBytes = kFeatures * kBlockK * 2;           // 16 KiB
constexpr int kPairBytes = kMaxPairs * kBlockK * 2;             // 32 KiB
constexpr int kThreads = 320, kEpilogueWarps = 8;
constexpr int kStagingBytes = 2 * 32 * 256;                     // per group of four epilogue warps: 32 pairs x 128 features
constexpr int kMaxExperts = 512;
constexpr int kBoxRows = 32;                                    // rows of a box of neighbouring pairs
template <bool GATED> struct Ring {
    static constexpr int kStages = GATED ? 3 : 4;
    static constexpr int kStageBytes = (GATED ? 2 : 1) * kWeightBytes + kPairBytes;
    static constexpr int kSmem = kStages * kStageBytes + kStagingBytes + 1024;
};

__device__ int g_error = 0;      // first error code any block has recorded since the last reset
enum : int { ERR_FULL_WAIT = 1, ERR_EMPTY_WAIT = 2, ERR_ACC_FULL_WAIT = 3, ERR_ACC_EMPTY_WAIT = 4 };

__device__ __forceinline__ void group_barrier(int id) { asm volatile("bar.sync %0, 128;" :: "r"(id) : "memory"); }

struct Tile { int e, n0, r0, pairs; };      // expert, first feature, first place, places

// Tiles run over experts, inside an expert over its feature tiles, inside those over its chunks.
// first_chunk[e]: chunks of the experts before e; offsets[e]: places before expert e.
__device__ __forceinline__ Tile find_tile(int tile, const int* first_chunk, const int* offsets, int E, int tiles_n) {
    int lo = 0, hi = E;                     // the last expert whose first tile is not behind this one
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first_chunk[mid] * tiles_n <= tile) lo = mid; else hi = mid;
    }
    const int chunks = first_chunk[lo + 1] - first_chunk[lo], rem = tile - first_chunk[lo] * tiles_n;
    const int n = rem / chunks, c = rem - n * chunks, places = offsets[lo + 1] - offsets[lo];
    const int size = (places + chunks - 1) / chunks;
    Tile t;
    t.e = lo;
    t.n0 = n * kFeatures;
    t.r0 = offsets[lo] + c * size;
    t.pairs = min(size, places - c * size);
    return t;
}

template <int MODE>
__device__ __forceinline__ float joined(float g, float u, const GluClamp& clamp) {
    return MODE == 3 ? clamped_glu(g, u, clamp) : g / (1.0f + expf(-g)) * u;
}

template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
moe_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0,
                   const __grid_constant__ CUtensorMap map_w1, bf16* __restrict__ out, const int* __restrict__ offsets_in,
                   const int* __restrict__ order, int E, int N, int K, const float* __restrict__ in_scale, GluClamp clamp) {
    constexpr bool GATED = MODE == 1 || MODE == 3;
    constexpr int kStages = Ring<GATED>::kStages, kStageBytes = Ring<GATED>::kStageBytes;
    constexpr int kX = (GATED ? 2 : 1) * kWeightBytes;             // where the pairs' rows lie in a stage
    constexpr int kAccs = GATED ? 1 : 2;                            // accumulators that take turns
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kStages], empty_bar[kStages], acc_full_bar[2], acc_empty_bar[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    __shared__ int offsets[kMaxExperts + 1], first_chunk[kMaxExperts + 1];
    __shared__ int s_row[2][kMaxPairs];                             // per group of epilogue warps: the tile's output rows
    __shared__ float s_scale[MODE == 2 ? 2 : 1][MODE == 2 ? kMaxPairs : 1];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t stages = (smem_u32(smem_raw) + 1023u) & ~1023u;  // swizzled tiles want 1 KiB alignment
    unsigned char* staging = smem_raw + (stages - smem_u32(smem_raw)) + kStages * kStageBytes;
    const int tiles_n = (N + kFeatures - 1) / kFeatures, k_blocks = (K + kBlockK - 1) / kBlockK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full_bar[b]), 1);
            mbar_init(smem_u32(&acc_empty_bar[b]), kEpilogueWarps);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();                                                     // offsets, order and the rows come from kernels ahead
    for (int e = threadIdx.x; e <= E; e += kThreads) offsets[e] = offsets_in[e];
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    if (warp == 0) {                                                // chunks of an expert, summed up over the experts before it
        int sum = 0;
        for (int base = 0; base < E; base += 32) {
            const int e = base + lane;
            const int own = e < E ? (offsets[e + 1] - offsets[e] + kMaxPairs - 1) / kMaxPairs : 0;
            int incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (e < E) first_chunk[e] = sum + incl - own;
            sum += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) first_chunk[E] = sum;
    }
    __syncthreads();
    const int n_tiles = first_chunk[E] * tiles_n;
    const uint32_t tmem_base = tmem_base_slot;

    auto fail = [&](int code) {
        atomicCAS(&g_error, 0, code);
        atomicExch(&abort_flag, 1);
    };

    if (warp == 0) {
        // ---- TMA producer: lane 0 waits and loads the weights, all lanes load the pairs' rows, 32 to a lane ----
        uint32_t phase = 0, used = 0;               // per stage: parity of its next use; whether it has been filled before
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const Tile t = find_tile(tile, first_chunk, offsets, E, tiles_n);
            const int wrow = t.e * N + t.n0;
            const uint32_t x_bytes = (uint32_t)((t.pairs + kBoxRows - 1) / kBoxRows) * (kBoxRows * 128u);
            for (int first = 0; first < k_blocks && ok; first += kStages) {
#pragma unroll
                for (int s = 0; s < kStages; ++s) {
                    const int kb = first + s;
                    if (kb >= k_blocks) break;
                    const uint32_t bar = smem_u32(&full_bar[s]), at = stages + s * kStageBytes;
                    if ((used >> s) & 1u) {
                        // one lane's verdict for all, so that a stage is filled as a whole or not at all
                        bool got = true;
                        if (lane == 0) got = mbar_wait_bounded(smem_u32(&empty_bar[s]), ((phase >> s) & 1u) ^ 1u) && !*(volatile int*)&abort_flag;
                        if (!__shfl_sync(0xffffffffu, (int)got, 0)) {
                            if (lane == 0) fail(ERR_EMPTY_WAIT);
                            ok = false;
                            break;
                        }
                    }
                    if (lane == 0) {
                        mbar_expect_tx(bar, kX + x_bytes);
                        tma_load_2d(at, &map_w0, bar, kb * kBlockK, wrow);
                        if (GATED) tma_load_2d(at + kWeightBytes, &map_w1, bar, kb * kBlockK, wrow);
                    }
                    __syncwarp();
                    if (lane * kBoxRows < t.pairs) {
                        tma_load_2d(at + kX + lane * (kBoxRows * 128), &map_x, bar, kb * kBlockK, t.r0 + lane * kBoxRows);
                    }
                    phase ^= 1u << s;
                    used |= 1u << s;
                }
            }
            if (__shfl_sync(0xffffffffu, *(volatile int*)&abort_flag, 0)) ok = false;
        }
        if (lane == 0 && *(volatile int*)&abort_flag) {             // copies that were asked for must land before the block ends
            for (int s = 0; s < kStages; ++s)
                if ((used >> s) & 1u) mbar_wait_bounded(smem_u32(&full_bar[s]), ((phase >> s) & 1u) ^ 1u);
        }
    } else if (warp == 1) {
        // ---- MMA issuer (one elected lane) ----
        if (lane == 0) {
            uint32_t phase = 0, local = 0;
            bool ok = true;
            const uint64_t dw = smem_desc_sw128(stages), dx = smem_desc_sw128(stages + kX);
            constexpr uint64_t kStep = (uint64_t)(kStageBytes >> 4), kUp = (uint64_t)(kWeightBytes >> 4);
            for (int tile = blockIdx.x; tile < n_tiles && ok && !*(volatile int*)&abort_flag; tile += gridDim.x, ++local) {
                const Tile t = find_tile(tile, first_chunk, offsets, E, tiles_n);
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((t.pairs + 15) >> 4) << 18) |
                                       ((uint32_t)(kFeatures >> 4) << 24);
                const int acc = kAccs == 2 ? (local & 1) : 0;
                const uint32_t turn = kAccs == 2 ? local >> 1 : local;
                if (!mbar_wait_bounded(smem_u32(&acc_empty_bar[acc]), (turn & 1) ^ 1)) { fail(ERR_ACC_EMPTY_WAIT); break; }
                tcgen05_fence_after();
                const uint32_t d0 = tmem_base + acc * kMaxPairs, d1 = tmem_base + kMaxPairs;
                for (int first = 0; first < k_blocks && ok; first += kStages) {
#pragma unroll
                    for (int s = 0; s < kStages; ++s) {
                        const int kb = first + s;
                        if (kb >= k_blocks) break;
                        if (!mbar_wait_bounded(smem_u32(&full_bar[s]), (phase >> s) & 1u)) { fail(ERR_FULL_WAIT); ok = false; break; }
                        phase ^= 1u << s;
                        tcgen05_fence_after();
#pragma unroll
                        for (int k = 0; k < kBlockK / 16; ++k) {
                            tcgen05_mma_f16(d0, dw + s * kStep + 2 * k, dx + s * kStep + 2 * k, idesc, (kb | k) != 0);
                            if (GATED) tcgen05_mma_f16(d1, dw + s * kStep + kUp + 2 * k, dx + s * kStep + 2 * k, idesc, (kb | k) != 0);
                        }
                        tcgen05_commit(smem_u32(&empty_bar[s]));
                    }
                }
                if (!ok) break;
                tcgen05_commit(smem_u32(&acc_full_bar[acc]));
            }
        }
    } else {
        // ---- epilogue: a warp may touch TMEM lanes 32 * (warp % 4) .. + 31 only; warps 2..5 take the even groups of 32
        // pairs, warps 6..9 the odd ones ----
        const int quarter = warp & 3, group = warp >= 6, ethread = (warp - 2 - 4 * group) * 32 + lane;
        unsigned char* stage = staging + group * (32 * 256);
        const bool wide = (N & 7) == 0 && ((uintptr_t)out & 15) == 0;       // rows of whole 16-byte pieces
        uint32_t local = 0;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++local) {
            const Tile t = find_tile(tile, first_chunk, offsets, E, tiles_n);
            group_barrier(1 + group);                                // the last tile's rows have been used
            for (int i = ethread; i < t.pairs; i += 128) {
                const int pair = GATED ? 0 : order[t.r0 + i];
                s_row[group][i] = MODE == 0 ? pair : t.r0 + i;
                if (MODE == 2) s_scale[group][i] = in_scale != nullptr ? in_scale[pair] : 1.f;
            }
            group_barrier(1 + group);
            const int acc = kAccs == 2 ? (local & 1) : 0;
            const uint32_t turn = kAccs == 2 ? local >> 1 : local;
            // (the warps of a group meet at barriers: all of them go through the loop below, whatever they were told)
            const bool got = mbar_wait_bounded(smem_u32(&acc_full_bar[acc]), turn & 1);
            if (!got) fail(ERR_ACC_FULL_WAIT);
            tcgen05_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * kMaxPairs;
            for (int c0 = group * 32; c0 < t.pairs; c0 += 64) {
                uint32_t v[32], u[GATED ? 32 : 1];
                tmem_load_32cols(taddr + c0, v);
                if constexpr (GATED) tmem_load_32cols(taddr + kMaxPairs + c0, u);
                tmem_load_wait();
                // staging: pair c at 256 bytes, its 16-byte pieces turned by the pair
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    float x = __uint_as_float(v[c]);
                    if constexpr (GATED) x = joined<MODE>(x, __uint_as_float(u[c]), clamp);
                    if (MODE == 2) {
                        x = fmaxf(x * s_scale[MODE == 2 ? group : 0][MODE == 2 ? c0 + c : 0], 0.f);
                        x *= x;
                    }
                    const int f = quarter * 32 + lane;
                    *reinterpret_cast<bf16*>(stage + c * 256 + ((((f >> 3) ^ c) & 15) << 4) + (f & 7) * 2) = __float2bfloat16_rn(x);
                }
                group_barrier(1 + group);
                const int piece = ethread & 15, f0 = t.n0 + piece * 8;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = (ethread >> 4) + 8 * i;
                    if (c0 + c < t.pairs && f0 < N) {
                        const uint4 val = *reinterpret_cast<const uint4*>(stage + c * 256 + (((piece ^ c) & 15) << 4));
                        bf16* dst = out + (int64_t)s_row[group][c0 + c] * N + f0;
                        if (wide) *reinterpret_cast<uint4*>(dst) = val;
                        else {
                            const bf16* p = reinterpret_cast<const bf16*>(&val);
                            for (int q = 0; q < 8 && f0 + q < N; ++q) dst[q] = p[q];
                        }
                    }
                }
                group_barrier(1 + group);
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty_bar[acc]));
            // a tile whose accumulator never came ends the group's work: one answer for its four warps
            if (ethread == 0) *reinterpret_cast<volatile int*>(stage) = *(volatile int*)&abort_flag;
            group_barrier(1 + group);
            if (*reinterpret_cast<volatile int*>(stage)) break;
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(512u) : "memory");
    }
}

template <int MODE>
static int launch(const void* A, const void* B0, const void* B1, void* C, const int* offsets, const int* order, int n_pairs,
                  int E, int N, int K, const float* in_scale, const GluClamp& clamp, cudaStream_t stream) {
    constexpr bool GATED = MODE == 1 || MODE == 3;
    CUtensorMap map_x, map_w0, map_w1;
    if (!make_map_2d_bf16(&map_x, A, (uint64_t)n_pairs, (uint64_t)K, (uint64_t)K * 2, kBlockK, kBoxRows) ||
        !make_map_2d_bf16(&map_w0, B0, (uint64_t)E * N, (uint64_t)K, (uint64_t)K * 2, kBlockK, kFeatures) ||
        !make_map_2d_bf16(&map_w1, GATED ? B1 : B0, (uint64_t)E * N, (uint64_t)K, (uint64_t)K * 2, kBlockK, kFeatures))
        return CPM_BAD_ARGUMENT;
    auto kern = moe_tcgen05_kernel<MODE>;
    static bool configured[kMaxDevices] = {};
    if (int st = ensure_dynamic_smem(kern, Ring<GATED>::kSmem, configured)) return st;
    const int sms = device_sms();
    if (sms < 1) return CPM_BAD_ARGUMENT;
    const int64_t most = ((int64_t)(n_pairs + kMaxPairs - 1) / kMaxPairs + (E < n_pairs ? E : n_pairs)) * ((N + kFeatures - 1) / kFeatures);
    cpm_launch(kLaunchProduct, kern, dim3((unsigned)(most < sms ? most : sms)), dim3(kThreads), (size_t)Ring<GATED>::kSmem, stream,
               map_x, map_w0, map_w1, (bf16*)C, offsets, order, E, N, K, in_scale, clamp);
    return launch_status();
}

}  // namespace moe5

// The products of cpm_moe_expert_product (same arguments, but A holds a row per pair, in expert order, in every mode) for bf16
// storage, K a multiple of 8 (16-byte rows), 16-byte aligned operands, at most 512 experts and fewer than 2^30 weight rows.
int moe_product_tcgen05(const void* A, const void* B0, const void* B1, void* C, const int* offsets, const int* order, int n_pairs, int E,
                        int N, int K, int mode, const float* in_scale, const GluClamp& clamp, cudaStream_t stream) {
    if (E > moe5::kMaxExperts || K % 8) return CPM_BAD_ARGUMENT;
    if (mode == 0) return moe5::launch<0>(A, B0, B1, C, offsets, order, n_pairs, E, N, K, in_scale, clamp, stream);
    if (mode == 1) return moe5::launch<1>(A, B0, B1, C, offsets, order, n_pairs, E, N, K, in_scale, clamp, stream);
    if (mode == 2) return moe5::launch<2>(A, B0, B1, C, offsets, order, n_pairs, E, N, K, in_scale, clamp, stream);
    return moe5::launch<3>(A, B0, B1, C, offsets, order, n_pairs, E, N, K, in_scale, clamp, stream);
}

// Error code recorded by the kernel since the last call (0 = none), and reset.  Synchronises the device.
CPM_API int cpm_moe_tcgen05_error() {
    int code = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&code, moe5::g_error, sizeof(int)) != cudaSuccess) return -1;
    cudaMemcpyToSymbol(moe5::g_error, &zero, sizeof(int));
    return code;
}
