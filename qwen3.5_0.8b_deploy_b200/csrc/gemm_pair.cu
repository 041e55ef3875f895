// Prompt-sized products with what follows them in their epilogue: Y = f(X[rows, K] W[N, K]^T) on tcgen05 over pairs of CTAs.
//   kPairGlu    act = silu(gate) * up or gelu(gate) * up, gate and up columns of one product (fp16 hybrid stack, bf16 layer-described stacks)
// The library product in front of an element-wise kernel writes what that kernel reads straight back: for 65536 rows of 2 x 3584 columns that is
// 0.94 GB each way.  Here the accumulators go through the function on their way out of TMEM while the tensor cores work on the next tile: 613 us (1.57
// PFLOP/s, bound by the tensor cores' 512 cycles a slice and, over seconds, by the power limit) in place of 682 + 285 us.  fp16 products reach the function
// unrounded; bf16 ones are rounded first, as the two kernels did: outputs of the layer-described stacks stay the same bit for bit.
//
// A cluster of two CTAs owns a 256 x 256 tile (cta_group::2, M = 256): each CTA fetches its 128 rows of both operands and holds 128 rows of the
// result, so that an operand byte in shared memory serves twice the products that it would in a tile of one CTA.  Two accumulators of 256 columns
// fill TMEM; eight warps empty one while the other is being filled.  Persistent: one CTA per SM, tiles in a fixed order.
#include "elem.cuh"
#include "gemm_pair.cuh"
#include "kernels.cuh"
#include "la_math.cuh"
#include "tc05.cuh"

#include <algorithm>
#include <type_traits>

namespace b200 {
namespace {

constexpr int kStages = 6;                              // ring of 64-deep slices, 32 KB each per CTA
constexpr uint32_t kOperand = 128 * 128;                // 128 rows of 64 two-byte elements
constexpr uint32_t kStage = 2 * kOperand;
constexpr int kEpiWarps = 16;
constexpr uint32_t kOutBytes = kEpiWarps * 2048;
constexpr uint32_t kBars = kStages * kStage + kOutBytes;
constexpr uint32_t kSmem = kBars + 256 + 1024;
constexpr int kThreads = 32 * (kEpiWarps + 2);          // epilogue warps, one for loads, one for products (CTA 0) or the hand-over of slices (CTA 1)

enum { kPairGlu = 0 };

struct PairArgs {
    int row_tiles, col_tiles;      // tiles of X rows and of W rows
    int whole, split_log2;         // of the tiles in their order, `whole` are done as such, each one behind them in 1 << split_log2 narrower parts
    int items;
    int k_steps;
    int rows, cols;                // of the result
    int up;                        // kPairGlu: W row of the first up column (0: groups of 32 gate and 32 up rows)
    int* error;
};

// One unit of work: a tile, or a part of it `width` columns of the product wide.
struct PairItem {
    int row, col, width;           // tile row; first column and number of columns of the product
    __device__ PairItem(const PairArgs& p, int t) {
        const int behind = t - p.whole, shift = behind < 0 ? 0 : p.split_log2;
        const int tile = behind < 0 ? t : p.whole + (behind >> shift), sub = behind & ((1 << shift) - 1);
        width = 256 >> shift;
        row = tile / p.col_tiles;
        col = (tile - row * p.col_tiles) * 256 + sub * width;
    }
};

__device__ __forceinline__ float glu_silu(float g, __half) { return g / (1.0f + expf(-g)); }
__device__ __forceinline__ float glu_silu(float g, __nv_bfloat16) { return times_sigmoid<__nv_bfloat16>(g, g); }
__device__ __forceinline__ float through(float v, __half) { return v; }
__device__ __forceinline__ float through(float v, __nv_bfloat16) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ uint32_t pack2(float a, float b, __half) { return pack_half2(a, b); }
__device__ __forceinline__ uint32_t pack2(float a, float b, __nv_bfloat16) { return pack_bf16x2(a, b); }

// 32 rows of 32 outputs: through shared memory (64-byte rows, swizzled as the tensor map expects) and out by TMA, which clips what lies beyond the
// matrix.  gate, up: TMEM columns of the two.
template <typename T, int kAct>
__device__ __forceinline__ void glu_part(const PairArgs& p, const CUtensorMap* map_y, uint32_t gate, uint32_t up_at, uint32_t out_smem, unsigned char* out,
                                         int row, int col, int lane) {
    if (row >= p.rows || col >= p.cols) return;
    const bool live = row + lane < p.rows;               // rows beyond the matrix are zeros, and the exact quotient of a zero takes a slow path
    if (lane == 0) bulk_wait_group_read0();              // the last part has left this place
    __syncwarp();
    uint32_t gt[32], up[32];
    tmem_ld32(gate, gt);
    tmem_ld32(up_at, up);
    tmem_wait_ld();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float v[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float a = through(live ? __uint_as_float(gt[8 * j + 2 * e + i]) : 1.0f, T{}), b = through(__uint_as_float(up[8 * j + 2 * e + i]), T{});
                if constexpr (kAct == B200ATTN_ACT_SILU) v[i] = glu_silu(a, T{}) * b;
                else v[i] = gelu_tanh<T>(a) * b;
            }
            o[e] = pack2(v[0], v[1], T{});
        }
        *reinterpret_cast<uint4*>(out + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
        tma_store_2d(map_y, out_smem, col, row);
        bulk_commit_group();
    }
}

// grid 2 x pairs, clusters of two.  Rank 0 of a pair issues the products once its own slice and its neighbour's have landed; the neighbour's
// product warp passes that on (its loads signal its own barrier).  map_w32: boxes of 32 rows, for the narrower parts.
template <int EPI, typename T, int kAct>
__global__ void __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w32,
                 const __grid_constant__ CUtensorMap map_y, const PairArgs p) {
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* sm = smem_raw + (base - raw);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + kBars + 248);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kBars + 252);
    const uint32_t bar0 = base + kBars;
    auto full = [&](int s) { return bar0 + 8u * s; };                          // this CTA's slice has landed, in rank 0 the neighbour's too
    auto empty = [&](int s) { return bar0 + 8u * (kStages + s); };             // the products that read it are done
    auto acc_full = [&](int b) { return bar0 + 8u * (2 * kStages + b); };
    auto acc_empty = [&](int b) { return bar0 + 8u * (2 * kStages + 2 + b); }; // rank 0: the epilogue warps of both CTAs have read it

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(full(i), 2 - rank);
            mbar_init(empty(i), 1);
        }
        mbar_init(acc_full(0), 1);
        mbar_init(acc_full(1), 1);
        mbar_init(acc_empty(0), 2 * kEpiWarps);
        mbar_init(acc_empty(1), 2 * kEpiWarps);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == kEpiWarps + 1) {
        tmem_alloc_pair(smem_u32(tmem_slot), 512);
        tmem_relinquish_pair();
    }
    if (warp == kEpiWarps && lane == 0) { tma_prefetch_desc(&map_x); tma_prefetch_desc(&map_w); tma_prefetch_desc(&map_w32); tma_prefetch_desc(&map_y); }
    const PairItem first(p, pair);
    tc_fence_before();
    __syncthreads();
    cluster_meet_all();                   // the barriers of both CTAs are in place
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();

    // Tiles are numbered along W first: W stays in L2, X passes through once.  The warps that issue loads and products carry stage and parity along
    // and walk their loops whole, with one lane elected for the issue: the chain of instructions of a slice has to stay shorter than its four
    // products (512 cycles; 670 with descriptors made anew by a single thread).
    if (warp == kEpiWarps) {
        int s = 0, issued = 0;
        uint32_t parity = 1;
        bool ok = true;
        PairItem w = first;
        for (int t = pair; t < p.items && ok; t += pairs) {
            if (t != pair) w = PairItem(p, t);
            const int x_row = w.row * 256 + rank * 128;
            const int w_row = p.up ? w.col / 2 + rank * p.up : w.col + rank * w.width / 2;
            const uint32_t bytes = kOperand + w.width * 64;
            for (int k = 0; k < 64 * p.k_steps; k += 64) {
                if (!mbar_wait_warp(empty(s), parity, abort_flag)) { ok = false; break; }
                const uint32_t dst = base + s * kStage, bar = full(s);
                if (elect_one()) {
                    mbar_arrive_expect_tx(bar, bytes);
                    tma_load_2d(dst, &map_x, bar, k, x_row);
                    if (w.width == 256) tma_load_2d(dst + kOperand, &map_w, bar, k, w_row);
                    else
                        for (int r = 0; r < w.width / 2; r += 32) tma_load_2d(dst + kOperand + r * 128, &map_w32, bar, k, w_row + r);
                }
                ++issued;
                if (++s == kStages) { s = 0; parity ^= 1; }
            }
        }
        if (!ok && lane == 0)
            for (int j = max(0, issued - kStages); j < issued; ++j) mbar_drain(full(j % kStages), (j / kStages) & 1);
    } else if (warp == kEpiWarps + 1) {
        int s = 0;
        uint32_t parity = 0;
        if (rank == 0) {
            constexpr uint32_t fmt = std::is_same<T, __half>::value ? kFmtF16 : kFmtBF16;
            const uint64_t a0 = umma_smem_desc(base, 16, 1024), w0 = umma_smem_desc(base + kOperand, 16, 1024);
            int i = 0;
            bool ok = true;
            PairItem w = first;
            for (int t = pair; t < p.items && ok; t += pairs, ++i) {
                const int b = i & 1;
                if (t != pair) w = PairItem(p, t);
                const uint32_t idesc = umma_idesc(fmt, 256, w.width, 0, 0);
                if (!mbar_wait_warp(acc_empty(b), ((i >> 1) & 1) ^ 1, abort_flag)) break;
                tc_fence_after();
                const uint32_t d = tmem + b * 256;
                for (int ks = 0; ks < p.k_steps; ++ks) {
                    if (!mbar_wait_warp(full(s), parity, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t a = a0 + s * (kStage >> 4), wd = w0 + s * (kStage >> 4);
                    const uint32_t done = empty(s);
                    if (elect_one()) {
                        umma_f16_pair(d, a, wd, idesc, ks > 0);
#pragma unroll
                        for (int kk = 1; kk < 4; ++kk) umma_f16_pair(d, a + 2 * kk, wd + 2 * kk, idesc, 1u);
                        umma_commit_pair(done);
                    }
                    if (++s == kStages) { s = 0; parity ^= 1; }
                }
                if (ok && elect_one()) umma_commit_pair(acc_full(b));
            }
        } else {
            const uint32_t theirs = cluster_smem_addr(full(0), 0);
            for (int left = (p.items - pair + pairs - 1) / pairs * p.k_steps; left > 0; --left) {
                if (!mbar_wait_warp(full(s), parity, abort_flag)) break;
                if (elect_one()) mbar_arrive_cluster(theirs + 8u * s);
                if (++s == kStages) { s = 0; parity ^= 1; }
            }
        }
    } else {
        const int q = warp & 3, part = warp >> 2;          // TMEM lanes 32 q .. 32 q + 31, a quarter of the columns
        unsigned char* out = sm + kStages * kStage + warp * 2048;
        const uint32_t out_smem = base + kStages * kStage + warp * 2048;
        int i = 0;
        for (int t = pair; t < p.items; t += pairs, ++i) {
            const int b = i & 1;
            const PairItem w = t == pair ? first : PairItem(p, t);
            if (!mbar_wait_warp(acc_full(b), (i >> 1) & 1, abort_flag)) break;
            tc_fence_after();
            const uint32_t acc = tmem + b * 256 + ((uint32_t)(32 * q) << 16);
            if (64 * part < w.width)
                glu_part<T, kAct>(p, &map_y, acc + (p.up ? 32 : 64) * part, acc + (p.up ? 32 * part + w.width / 2 : 64 * part + 32), out_smem, out,
                                  w.row * 256 + rank * 128 + 32 * q, w.col / 2 + 32 * part, lane);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_smem_addr(acc_empty(b), 0));
        }
        if (lane == 0) bulk_wait_group0();
    }
    tc_fence_before();
    __syncthreads();
    cluster_meet_all();                   // neither CTA reads the other's shared memory, arrives on its barriers or works on its TMEM any more
    if (warp == kEpiWarps + 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem, 512);
    }
    if (threadIdx.x == 0 && *abort_flag) atomicExch(p.error, 7);
}

template <int EPI, typename T, int kAct>
int launch_pair(const CUtensorMap& mx, const CUtensorMap& mw, const CUtensorMap& mw32, const CUtensorMap& my, PairArgs p, cudaStream_t s) {
    static PerDeviceOnce once;
    B2_PER_DEVICE_ONCE(once, B2_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<EPI, T, kAct>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem)));
    int sms = 0;
    B2_TRY(device_sm_count(&sms));
    cudaLaunchConfig_t cfg = {};
    // Whole rounds of tiles, then the rest in parts as narrow as it takes to give every pair one (at least 64 columns).
    const int tiles = p.row_tiles * p.col_tiles, pairs = sms / 2, rest = tiles % pairs;
    p.split_log2 = rest == 0 ? 0 : rest * 4 <= pairs ? 2 : rest * 2 <= pairs ? 1 : 0;
    p.whole = tiles - rest;
    p.items = p.whole + (rest << p.split_log2);
    cfg.gridDim = dim3(2 * std::min(p.items, pairs));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_flags.pdl ? 2 : 1;
    B2_CUDA(cudaLaunchKernelEx(&cfg, gemm_pair_kernel<EPI, T, kAct>, mx, mw, mw32, my, p));
    count_launch();
    return 0;
}

// [rows, cols] of two-byte elements, row pitch = cols, in boxes of 64 or (results) 32 columns
int map_rows(CUtensorMap* m, ElemType t, const void* p, long long rows, int cols, int box_cols, int box_rows) {
    const uint64_t dims[2] = {(uint64_t)cols, (uint64_t)rows}, str[1] = {(uint64_t)cols * 2};
    const uint32_t box[2] = {(uint32_t)box_cols, (uint32_t)box_rows};
    return make_tensor_map(m, t == ELEM_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p, dims, str, box, box_cols * 2);
}
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

// Up to 128 rows the library's smaller tiles and the activation behind them are faster: 8.3 us at 128 rows of 1024 and 2 x 3584 columns (bf16)
// against 8.9 here; 9.7 / 9.0 at 256, 21.8 / 17.1 at 999, 53.7 / 39.9 at 3855, 130 / 78 at 8192 (the product alone 92).
bool gemm_glu_takes(ElemType t, const void* x, const void* w, const void* act, int rows, int ff, int K) {
    return rows > 128 && t != ELEM_F32 && K % 8 == 0 && ff % 8 == 0 && aligned16(x) && aligned16(w) && aligned16(act);
}

int gemm_glu(cudaStream_t s, ElemType t, int act_kind, const void* x, const void* w, void* act, int rows, int ff, int K, bool split, int* error) {
    CUtensorMap mx, mw, mw32, my;
    B2_TRY(map_rows(&mx, t, x, rows, K, 64, 128));
    B2_TRY(map_rows(&mw, t, w, 2LL * ff, K, 64, 128));
    B2_TRY(map_rows(&mw32, t, w, 2LL * ff, K, 64, 32));
    B2_TRY(map_rows(&my, t, act, rows, ff, 32, 32));
    PairArgs p{};
    p.row_tiles = ceil_div(rows, 256);
    p.col_tiles = ceil_div(ff, 128);
    p.k_steps = ceil_div(K, 64);
    p.rows = rows;
    p.cols = ff;
    p.up = split ? ff : 0;
    p.error = error;
    if (t == ELEM_F16) return launch_pair<kPairGlu, __half, B200ATTN_ACT_SILU>(mx, mw, mw32, my, p, s);
    if (act_kind == B200ATTN_ACT_SILU) return launch_pair<kPairGlu, __nv_bfloat16, B200ATTN_ACT_SILU>(mx, mw, mw32, my, p, s);
    return launch_pair<kPairGlu, __nv_bfloat16, B200ATTN_ACT_GELU_TANH>(mx, mw, mw32, my, p, s);
}

}  // namespace b200
