// Prompt-sized products with what follows them in their epilogue: Y = f(X[rows, K] W[N, K]^T) on tcgen05 over pairs of CTAs.
//   kPairGlu    act = silu(gate) * up or gelu(gate) * up, gate and up columns of one product (fp16 hybrid stack, bf16 layer-described stacks)
// The library product in front of an element-wise kernel writes what that kernel reads straight back: for 65536 rows of 2 x 3584 columns that is
// 0.94 GB each way.  Here the accumulators go through the function on their way out of TMEM while the tensor cores work on the next tile: 613 us (1.57
// PFLOP/s, bound by the tensor cores' 512 cycles a slice and, over seconds, by the power limit) in place of 682 + 285 us.  fp16 products reach the function
// unrounded; bf16 ones are rounded first, as the two kernels did: outputs of the layer-described stacks stay the same bit for bit.
//   kPairStore16, kPairStore32   the product alone, as bf16 or fp32 values (large products, gemm_typed)
//   kPairConv   the DeltaNet input projection with the causal convolution, SiLU, L2 norms and gates behind it (fp16).  Here the channels of W are the
//               rows of the product and the tokens its columns: a thread holds one channel and finds the taps of a token in its own registers.
//               65536 rows 950 us (projection 878 and convolution 502 before, 3.2 GB between them), 3 x 333 23 (33), 9 x 466 67 (111).
//
// A cluster of two CTAs owns a 256 x 256 tile (cta_group::2, M = 256): each CTA fetches its 128 rows of both operands and holds 128 rows of the
// result, so that an operand byte in shared memory serves twice the products that it would in a tile of one CTA.  Two accumulators of 256 columns
// fill TMEM; sixteen warps (kPairConv: eight, in turns) empty one while the other is being filled.  Persistent: one CTA per SM, tiles in a fixed order.
#include "elem.cuh"
#include "gemm_pair.cuh"
#include "kernels.cuh"
#include "la_math.cuh"
#include "tc05.cuh"

#include <algorithm>
#include <type_traits>

namespace b200 {
namespace {

constexpr uint32_t kOperand = 128 * 128;                // 128 rows of 64 two-byte elements
constexpr uint32_t kStage = 2 * kOperand;
constexpr int kEpiWarps = 16;
constexpr int kThreads = 32 * (kEpiWarps + 2);          // epilogue warps, one for loads, one for TMEM and (CTA 0) the products

enum { kPairGlu = 0, kPairConv, kPairStore16, kPairStore32 };
constexpr int kConvTokens = 253;                        // of a tile of 256 columns: the first three are the taps of the fourth
constexpr int kMaxSeqRows = 512;                        // first rows and slots of the sequences kept in shared memory, up to so many sequences

template <int EPI>
struct PairSmem {
    static constexpr int kStages = EPI == kPairConv ? 5 : 6;               // ring of 64-deep slices, 32 KB each per CTA
    static constexpr uint32_t kOut = kStages * kStage;                     // 2 KB per epilogue warp
    static constexpr uint32_t kExtra = kOut + kEpiWarps * 2048;            // kPairConv: the tables of conv_part
    static constexpr uint32_t kBars = kExtra + (EPI == kPairConv ? 4096 + 4096 + 2048 + 8 * kMaxSeqRows : 0);
    static constexpr int kReaders = EPI == kPairConv ? kEpiWarps / 2 : kEpiWarps;     // epilogue warps of one tile
    static constexpr uint32_t kBytes = kBars + 256 + 1024;
};
struct PairMaps {
    CUtensorMap a, b, b32;         // operands: rows of the product, its columns, those in boxes of 32 rows
    CUtensorMap out[4];            // results: kPairGlu one, kPairConv q, k, v, mixed
};

struct PairArgs {
    int row_tiles, col_tiles;      // tiles of X rows and of W rows
    int whole, split_log2;         // of the tiles in their order, `whole` are done as such, each one behind them in 1 << split_log2 narrower parts
    int items;
    int k_steps;
    int rows, cols;                // of the result
    int up;                        // kPairGlu: W row of the first up column (0: groups of 32 gate and 32 up rows)
    int* error;
    LaConvArgs la;                 // kPairConv
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
    __syncwarp();
}

// 32 rows of up to 64 columns as they are, 16-bit or fp32 rows of 64 bytes at a time.
template <typename T, int EPI>
__device__ __forceinline__ void plain_part(const PairArgs& p, const CUtensorMap* map_y, uint32_t acc, uint32_t out_smem, unsigned char* out, int row, int col, int lane) {
    constexpr int kCols = EPI == kPairStore16 ? 32 : 16;
    if (row >= p.rows) return;
#pragma unroll 1
    for (int c = 0; c < 64 && col + c < p.cols; c += kCols) {
        uint32_t o[16];
        if constexpr (EPI == kPairStore16) {
            uint32_t v[32];
            tmem_ld32(acc + c, v);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) o[j] = pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]), T{});
        } else {
            tmem_ld16(acc + c, o);
            tmem_wait_ld();
        }
        if (lane == 0) bulk_wait_group_read0();          // the last rows have left this place
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<uint4*>(out + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
            tma_store_2d(map_y, out_smem, col + c, row);
            bulk_commit_group();
        }
        __syncwarp();
    }
}

// What the convolution has to know of a token: place in its sequence's rows of this call, up to 3, and rows behind it, up to 3.
constexpr int kTokenNone = 16;
__device__ __forceinline__ int sequence_of(const LaConvArgs& a, const int* first_rows, int t) {
    int lo = 0, hi = a.n_seqs - 1;                       // the last sequence that starts at or before row t (empty ones start where the next does)
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((a.n_seqs <= kMaxSeqRows ? first_rows[mid] : a.seqs[mid].row0) <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ int slot_of(const LaConvArgs& a, const int* first_rows, int t) {
    const int i = sequence_of(a, first_rows, t);
    return a.n_seqs <= kMaxSeqRows ? first_rows[kMaxSeqRows + i] : a.seqs[i].slot;
}
__device__ __forceinline__ int token_info(const LaConvArgs& a, const int* first_rows, int rows, int t) {
    if (t < 0 || t >= rows) return kTokenNone;
    const int i = sequence_of(a, first_rows, t), row0 = a.n_seqs <= kMaxSeqRows ? first_rows[i] : a.seqs[i].row0;
    const int next = i + 1 == a.n_seqs ? rows : a.n_seqs <= kMaxSeqRows ? first_rows[i + 1] : a.seqs[i + 1].row0;
    return min(next - 1 - t, 3) << 2 | min(t - row0, 3);
}

__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// Taps of four tokens, the newest one's weight last in the reference's order, and SiLU.
__device__ __forceinline__ float conv_tap(const float4& w, float x0, float x1, float x2, float x3) {
    float y = w.w * x0;
    y += w.x * x1;
    y += w.y * x2;
    y += w.z * x3;
    return silu_sfu(y);
}

// Sum over the lanes of v[j]^2, token j's in lane j: every step halves the tokens that a lane still carries.
__device__ __forceinline__ float squares_by_token(const float (&v)[32], int lane) {
    float s[16];
    const bool up16 = lane & 16;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const float keep = up16 ? v[j + 16] : v[j], give = up16 ? v[j] : v[j + 16];
        s[j] = keep * keep + __shfl_xor_sync(0xffffffffu, give * give, 16);
    }
#pragma unroll
    for (int n = 8; n > 0; n >>= 1) {
        const bool up = lane & n;
#pragma unroll
        for (int j = 0; j < n; ++j) {
            const float keep = up ? s[j + n] : s[j], give = up ? s[j] : s[j + n];
            s[j] = keep + __shfl_xor_sync(0xffffffffu, give, n);
        }
    }
    return s[0];
}

// This warp's 32 channels and 128 tokens of a tile, 32 tokens at a time.  `info`: of the tile's 256 tokens; `sums`: 2 x 4 x 32 floats shared by the
// four warps of these tokens (all 128 channels of a head), which meet at barrier `bar`; `scale`: 32 floats of this warp; `stage`: its 2 KB, from where TMA
// writes the results (stores of 2 bytes a lane straight to memory took 4.4 cycles each of the SM's one load / store unit).  Without `ok` it only keeps
// its place at the barriers.
template <typename Release>
__device__ __forceinline__ void conv_part(const LaConvArgs& a, const PairMaps& maps, bool ok, uint32_t acc, int tile, int t_tile, int rows, int rank, int q, int part,
                                          int lane, const int* info, const int* first_rows, float* sums, int bar, float* scale, unsigned char* stage,
                                          Release&& release) {
    const int ch = tile * 256 + rank * 128 + 32 * q + lane, kind = min(tile >> 3, 3);       // 0 q, 1 k, 2 v, 3 z and (tile 32) the gates' inputs
    const bool wanted = ok && ch - lane < kLaProjCols;
    float* raw = reinterpret_cast<float*>(stage);
    if (kind == 3) {
#pragma unroll 1
        for (int c = 0; c < 8; ++c) {
            const int col = 128 * part + 16 * c, t0 = t_tile + col;
            const bool live = wanted && t0 < rows;
            uint32_t r[16];
            if (live) {
                tmem_ld16(acc + col, r);
                tmem_wait_ld();
            }
            if (c == 7) release();
            if (!live) continue;
            if (col == 0) {                              // its first three tokens are the tile's before
                float* dst = a.mixed + (long long)t0 * kLaProjCols + ch;
#pragma unroll
                for (int j = 3; j < 16; ++j)
                    if (t0 + j < rows) dst[(long long)j * kLaProjCols] = __uint_as_float(r[j]);
                continue;
            }
            if (lane == 0) bulk_wait_group_read0();
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 16; ++j) raw[32 * j + lane] = __uint_as_float(r[j]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                tma_store_2d(&maps.out[3], smem_u32(stage), ch, t0);
                bulk_commit_group();
            }
            __syncwarp();
        }
        return;
    }
    const float4 w = *reinterpret_cast<const float4*>(a.conv_w + (size_t)ch * kLaConvK);
    float h[3] = {0.f, 0.f, 0.f};                        // the three tokens in front, oldest first
    if (ok && part > 0) {
        uint32_t r[4];
        tmem_ld4(acc + 128 * part - 4, r);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 3; ++i) h[i] = __uint_as_float(r[i + 1]);
    }
    const int out_ch = (tile & 7) * 256 + rank * 128 + 32 * q;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
        const int col = 128 * part + 32 * c, t0 = t_tile + col;
        const bool live = wanted && t0 < rows;           // the same for all warps of these tokens
        float v[32];
        if (live) {
            uint32_t r[32];
            tmem_ld32(acc + col, r);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        }
        if (c == 3) release();
        if (live) {
            const float last[3] = {v[29], v[30], v[31]};
            const int f = info[col + lane];
            const unsigned tails = __ballot_sync(0xffffffffu, f < 12 && col + lane >= 3);               // of their sequence's last three rows
            const unsigned starts = __ballot_sync(0xffffffffu, f < kTokenNone && (f & 3) < 3);          // of its first three
            if (tails) {
                float* dst = a.mixed + (long long)t0 * kLaProjCols + ch;
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (tails >> j & 1) dst[(long long)j * kLaProjCols] = v[j];
            }
            if (starts == 0) {
#pragma unroll
                for (int j = 31; j >= 3; --j) v[j] = conv_tap(w, v[j], v[j - 1], v[j - 2], v[j - 3]);
                v[2] = conv_tap(w, v[2], v[1], v[0], h[2]);
                v[1] = conv_tap(w, v[1], v[0], h[2], h[1]);
                v[0] = conv_tap(w, v[0], h[2], h[1], h[0]);
            } else {
                int of = -1;                             // first row of the sequence whose last inputs are in s0 (oldest) .. s2
                float s0 = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll
                for (int j = 31; j >= 0; --j) {
                    float x1 = j >= 1 ? v[j >= 1 ? j - 1 : 0] : h[2], x2 = j >= 2 ? v[j >= 2 ? j - 2 : 0] : h[j == 1 ? 2 : 1];
                    float x3 = j >= 3 ? v[j >= 3 ? j - 3 : 0] : h[j < 3 ? j : 0];
                    if (starts >> j & 1) {
                        const int pos = info[col + j] & 3, first = t0 + j - pos;
                        if (first != of) {
                            of = first;
                            const float* st = a.conv_state + (size_t)slot_of(a, first_rows, t0 + j) * a.conv_stride + ch;
                            s0 = st[0]; s1 = st[kLaConvDim]; s2 = st[2 * kLaConvDim];
                        }
                        x3 = pos == 0 ? s0 : pos == 1 ? s1 : s2;
                        if (pos < 2) x2 = pos == 0 ? s1 : s2;
                        if (pos < 1) x1 = s2;
                    }
                    v[j] = conv_tap(w, v[j], x1, x2, x3);
                }
            }
            h[0] = last[0]; h[1] = last[1]; h[2] = last[2];
        }
        if (kind < 2) {
            float* sum = sums + (c & 1) * 128;
            if (live) sum[32 * q + lane] = squares_by_token(v, lane);
            bar_sync(bar, 128);
            if (live) {
                const float ss = (sum[lane] + sum[32 + lane]) + (sum[64 + lane] + sum[96 + lane]);
                scale[lane] = (kind == 0 ? 1.0f / sqrtf((float)kLaKd) : 1.0f) / sqrtf(ss + 1e-6f);
                __syncwarp();
#pragma unroll
                for (int j4 = 0; j4 < 8; ++j4) {
                    const float4 s4 = *reinterpret_cast<const float4*>(scale + 4 * j4);
                    v[4 * j4] *= s4.x; v[4 * j4 + 1] *= s4.y; v[4 * j4 + 2] *= s4.z; v[4 * j4 + 3] *= s4.w;
                }
            }
        }
        if (!live) continue;
        if (col == 0) {                                  // without the tile's first three tokens, which are the tile's before
            __half* dst = (kind == 0 ? a.q : kind == 1 ? a.k : a.v) + (long long)t0 * (kLaHeads * kLaKd) + out_ch + lane;
#pragma unroll
            for (int j = 3; j < 32; ++j)
                if (t0 + j < rows) dst[j * (kLaHeads * kLaKd)] = __float2half_rn(v[j]);
            continue;
        }
        if (lane == 0) bulk_wait_group_read0();
        __syncwarp();
        __half* out = reinterpret_cast<__half*>(stage);
#pragma unroll
        for (int j = 0; j < 32; ++j) out[32 * j + lane] = __float2half_rn(v[j]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
            tma_store_2d(&maps.out[kind], smem_u32(stage), out_ch, t0);
            bulk_commit_group();
        }
        __syncwarp();
    }
}

// grid 2 x pairs, clusters of two.  Rank 0 of a pair issues the products once its own slice and its neighbour's have landed: the copies of both CTAs
// complete on its barrier.  Every barrier here is signalled from the other CTA too, so all waits are of cluster scope.  Operand a gives the rows of
// the product (X, kPairConv: W), b its columns.
template <int EPI, typename T, int kAct>
__global__ void __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ PairMaps maps, const PairArgs p) {
    using Smem = PairSmem<EPI>;
    constexpr int kStages = Smem::kStages;
    constexpr uint32_t kBars = Smem::kBars;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* sm = smem_raw + (base - raw);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + kBars + 248);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kBars + 252);
    const uint32_t bar0 = base + kBars;
    auto full = [&](int s) { return bar0 + 8u * s; };                          // rank 0: the slices of both CTAs have landed
    auto empty = [&](int s) { return bar0 + 8u * (kStages + s); };             // the products that read it are done
    auto acc_full = [&](int b) { return bar0 + 8u * (2 * kStages + b); };
    auto acc_empty = [&](int b) { return bar0 + 8u * (2 * kStages + 2 + b); }; // rank 0: the epilogue warps of both CTAs have read it
    const uint32_t halted = bar0 + 8u * (2 * kStages + 4);                     // rank 0, after a wait that ran out: no product is under way any more

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(full(i), 1);
            mbar_init(empty(i), 1);
        }
        mbar_init(acc_full(0), 1);
        mbar_init(acc_full(1), 1);
        mbar_init(acc_empty(0), 2 * Smem::kReaders);
        mbar_init(acc_empty(1), 2 * Smem::kReaders);
        mbar_init(halted, 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == kEpiWarps + 1) {
        tmem_alloc_pair(smem_u32(tmem_slot), 512);
        tmem_relinquish_pair();
    }
    if (warp == kEpiWarps && lane == 0) {
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.b);
        tma_prefetch_desc(&maps.out[0]);
    }
    const PairItem first(p, pair);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                   // the barriers and the TMEM of both CTAs are in place
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();

    // Tiles are numbered along W first: W stays in L2, X passes through once.  The warps that issue loads and products carry stage and parity along
    // and walk their loops whole, with one lane elected for the issue: the chain of instructions of a slice has to stay shorter than its four
    // products (512 cycles; 670 with descriptors made anew by a single thread).
    if (warp == kEpiWarps) {
        int s = 0, issued = 0;
        uint32_t parity = 1;
        const uint32_t landed = cluster_smem_addr(full(0), 0);
        bool ok = true;
        PairItem w = first;
        for (int t = pair; t < p.items && ok; t += pairs) {
            if (t != pair) w = PairItem(p, t);
            const int a_row = (EPI == kPairConv ? w.col : w.row * 256) + rank * 128;
            const int b_row = EPI == kPairConv ? w.row * kConvTokens - 3 + rank * 128 : p.up ? w.col / 2 + rank * p.up : w.col + rank * w.width / 2;
            const uint32_t bytes = 2 * (kOperand + w.width * 64);              // of both CTAs
            for (int k = 0; k < 64 * p.k_steps; k += 64) {
                if (!mbar_wait_warp<kClusterScope>(empty(s), parity, abort_flag)) { ok = false; break; }
                const uint32_t dst = base + s * kStage, bar = landed + 8u * s;
                if (elect_one()) {
                    if (rank == 0) mbar_arrive_expect_tx(full(s), bytes);          // the neighbour's bytes may come in first: the phase waits for this arrival
                    tma_load_2d_pair(dst, &maps.a, bar, k, a_row);
                    if (w.width == 256) tma_load_2d_pair(dst + kOperand, &maps.b, bar, k, b_row);
                    else
                        for (int r = 0; r < w.width / 2; r += 32) tma_load_2d_pair(dst + kOperand + r * 128, &maps.b32, bar, k, b_row + r);
                }
                ++issued;
                if (++s == kStages) { s = 0; parity ^= 1; }
            }
        }
        // A copy or an arrival of the neighbour's that is still under way must not find this CTA gone.  When a wait has run out, rank 0 waits for the
        // copies of both, then for as long again (a phase that nothing completes) for what the neighbour may have asked for beyond.
        if (lane == 0) {
            if (ok)
                for (int j = max(0, issued - kStages); j < issued; ++j) mbar_wait<kClusterScope>(empty(j % kStages), (j / kStages) & 1, abort_flag);
            else if (rank == 0)
                for (int j = max(0, issued - kStages); j <= issued; ++j) mbar_drain(full(j % kStages), (j / kStages) & 1);
        }
    } else if (warp == kEpiWarps + 1) {
        if (rank == 0) {
            int s = 0;
            uint32_t parity = 0;
            constexpr uint32_t fmt = std::is_same<T, __half>::value ? kFmtF16 : kFmtBF16;
            const uint64_t a0 = umma_smem_desc(base, 16, 1024), w0 = umma_smem_desc(base + kOperand, 16, 1024);
            int i = 0;
            bool ok = true;
            PairItem w = first;
            for (int t = pair; t < p.items && ok; t += pairs, ++i) {
                const int b = i & 1;
                if (t != pair) w = PairItem(p, t);
                const uint32_t idesc = umma_idesc(fmt, 256, w.width, 0, 0);
                if (!mbar_wait_warp<kClusterScope>(acc_empty(b), ((i >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d = tmem + b * 256;
                for (int ks = 0; ks < p.k_steps; ++ks) {
                    if (!mbar_wait_warp<kClusterScope>(full(s), parity, abort_flag)) { ok = false; break; }
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
            for (int j = max(0, i - 2); ok && j < i; ++j) ok = mbar_wait_warp<kClusterScope>(acc_empty(j & 1), (j >> 1) & 1, abort_flag);     // the neighbour's arrivals
            if (!ok) {                    // products under way read shared memory and write TMEM that others are given when these CTAs leave
                if (elect_one()) umma_commit_pair(halted, 1);
                mbar_drain(halted, 0);
            }
        }
    } else {
        const int q = warp & 3, part = warp >> 2;          // TMEM lanes 32 q .. 32 q + 31, a quarter of the columns
        unsigned char* out = sm + Smem::kOut + warp * 2048;
        const uint32_t out_smem = base + Smem::kOut + warp * 2048;
        // kPairConv: the two halves of these warps take turns at the tiles.  One half's special functions then run beside the other's shuffles, loads
        // and stores; all on one tile went through them in step.
        int i = EPI == kPairConv ? warp >> 3 : 0;
        bool ok = true;
        if constexpr (EPI == kPairConv) {
            int* first_rows = reinterpret_cast<int*>(sm + Smem::kExtra + 10240);
            for (int j = threadIdx.x; j < min(p.la.n_seqs, kMaxSeqRows); j += 32 * kEpiWarps) {
                first_rows[j] = p.la.seqs[j].row0;
                first_rows[kMaxSeqRows + j] = p.la.seqs[j].slot;
            }
            __syncwarp();
            bar_sync(1, 32 * kEpiWarps);
        }
        for (int t = pair + i * pairs; t < p.items; t += EPI == kPairConv ? 2 * pairs : pairs, i += EPI == kPairConv ? 2 : 1) {
            const int b = i & 1;
            const PairItem w = t == pair ? first : PairItem(p, t);
            auto release = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(cluster_smem_addr(acc_empty(b), 0));
            };
            const uint32_t acc = tmem + b * 256 + ((uint32_t)(32 * q) << 16);
            if constexpr (EPI == kPairConv) {
                const int half = b, side = part & 1;                           // these warps' half, and their half of the tokens
                int* info = reinterpret_cast<int*>(sm + Smem::kExtra) + (2 * half + (i >> 1 & 1)) * 256;
                float* sums = reinterpret_cast<float*>(sm + Smem::kExtra + 4096) + (2 * half + side) * 256;
                float* scale = reinterpret_cast<float*>(sm + Smem::kExtra + 8192) + 32 * warp;
                const int* first_rows = reinterpret_cast<const int*>(sm + Smem::kExtra + 10240);
                const int t_tile = w.row * kConvTokens - 3, mine = threadIdx.x & 255;
                info[mine] = token_info(p.la, first_rows, p.rows, t_tile + mine);
                __syncwarp();
                bar_sync(2 + half, 256);
                ok = ok && mbar_wait_warp<kClusterScope>(acc_full(b), (i >> 1) & 1, abort_flag);
                tc_fence_after();
                conv_part(p.la, maps, ok, acc, w.col >> 8, t_tile, p.rows, rank, q, side, lane, info, first_rows, sums, 4 + 2 * half + side, scale, out, release);
            } else {
                if (!mbar_wait_warp<kClusterScope>(acc_full(b), (i >> 1) & 1, abort_flag)) break;
                tc_fence_after();
                if constexpr (EPI != kPairGlu) {
                    if (64 * part < w.width)
                        plain_part<T, EPI>(p, &maps.out[0], acc + 64 * part, out_smem, out, w.row * 256 + rank * 128 + 32 * q, w.col + 64 * part, lane);
                } else if (64 * part < w.width)
                    glu_part<T, kAct>(p, &maps.out[0], acc + (p.up ? 32 : 64) * part, acc + (p.up ? 32 * part + w.width / 2 : 64 * part + 32), out_smem, out,
                                      w.row * 256 + rank * 128 + 32 * q, w.col / 2 + 32 * part, lane);
                release();
            }
        }
        if (lane == 0) bulk_wait_group0();
    }
    tc_fence_before();
    __syncthreads();
    // Neither CTA reads the other's shared memory, arrives on its barriers or works on its TMEM any more: each has waited for what it started there.  Nothing
    // is handed over here, so the arrival need not wait for this CTA's stores (475 us for 3 x 333 tokens through four layers with, 473 without that).
    cluster_stay();
    if (warp == kEpiWarps + 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem, 512);
    }
    if (threadIdx.x == 0 && *abort_flag) atomicExch(p.error, 7);
}

template <int EPI, typename T, int kAct>
int launch_pair(const PairMaps& maps, PairArgs p, cudaStream_t s) {
    static PerDeviceOnce once;
    B2_PER_DEVICE_ONCE(once, B2_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<EPI, T, kAct>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem<EPI>::kBytes)));
    int sms = 0;
    B2_TRY(device_sm_count(&sms));
    cudaLaunchConfig_t cfg = {};
    // Whole rounds of tiles, then the rest in parts as narrow as it takes to give every pair one (at least 64 columns).
    const int tiles = p.row_tiles * p.col_tiles, pairs = sms / 2, rest = tiles % pairs;
    p.split_log2 = rest == 0 || EPI == kPairConv ? 0 : rest * 4 <= pairs ? 2 : rest * 2 <= pairs ? 1 : 0;
    p.whole = tiles - rest;
    p.items = p.whole + (rest << p.split_log2);
    cfg.gridDim = dim3(2 * std::min(p.items, pairs));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = PairSmem<EPI>::kBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_flags.pdl ? 2 : 1;
    B2_CUDA(cudaLaunchKernelEx(&cfg, gemm_pair_kernel<EPI, T, kAct>, maps, p));
    count_launch();
    return 0;
}

// [rows, cols] row-major, in boxes of so many columns and rows; a swizzle as wide as the box for operands and (64 bytes) results but those of kPairConv
int map_rows(CUtensorMap* m, ElemType t, const void* p, long long rows, int cols, int box_cols, int box_rows, bool swizzle = true, int pitch = 0) {
    const uint64_t dims[2] = {(uint64_t)cols, (uint64_t)rows}, str[1] = {(uint64_t)(pitch ? pitch : cols) * elem_bytes(t)};
    const uint32_t box[2] = {(uint32_t)box_cols, (uint32_t)box_rows};
    return make_tensor_map(m, t == ELEM_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : t == ELEM_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                           p, dims, str, box, swizzle ? (int)(box_cols * elem_bytes(t)) : 0);
}
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

// Up to 128 rows the library's smaller tiles and the activation behind them are faster: 8.3 us at 128 rows of 1024 and 2 x 3584 columns (bf16)
// against 8.9 here; 9.7 / 9.0 at 256, 21.8 / 17.1 at 999, 53.7 / 39.9 at 3855, 130 / 78 at 8192 (the product alone 92).  The deeper the product, the less the
// activation weighs and the more the library's rate, the higher one in deep products: a prompt pass of three layers of width 2048 and 5632 outputs takes 351 / 346
// us at 400 rows, 538 / 482 at 1000, 806 / 768 at 2000; of 4096 and 11008 656 / 673, 1022 / 1092 and 1842 / 2035; of 4096 and 1024 at 200 341 / 357.
bool gemm_glu_takes(ElemType t, const void* x, const void* w, const void* act, int rows, int ff, int K) {
    return rows > 128 && K <= 2048 && t != ELEM_F32 && K % 8 == 0 && ff % 8 == 0 && aligned16(x) && aligned16(w) && aligned16(act);
}

int gemm_glu(cudaStream_t s, ElemType t, int act_kind, const void* x, const void* w, void* act, int rows, int ff, int K, bool split, int* error) {
    PairMaps m{};
    B2_TRY(map_rows(&m.a, t, x, rows, K, 64, 128));
    B2_TRY(map_rows(&m.b, t, w, 2LL * ff, K, 64, 128));
    B2_TRY(map_rows(&m.b32, t, w, 2LL * ff, K, 64, 32));
    B2_TRY(map_rows(&m.out[0], t, act, rows, ff, 32, 32));
    PairArgs p{};
    p.row_tiles = ceil_div(rows, 256);
    p.col_tiles = ceil_div(ff, 128);
    p.k_steps = ceil_div(K, 64);
    p.rows = rows;
    p.cols = ff;
    p.up = split ? ff : 0;
    p.error = error;
    if (t == ELEM_F16) return launch_pair<kPairGlu, __half, B200ATTN_ACT_SILU>(m, p, s);
    if (act_kind == B200ATTN_ACT_SILU) return launch_pair<kPairGlu, __nv_bfloat16, B200ATTN_ACT_SILU>(m, p, s);
    return launch_pair<kPairGlu, __nv_bfloat16, B200ATTN_ACT_GELU_TANH>(m, p, s);
}

// A tile goes through all its weights whatever its rows, and a start of a sequence costs its chunk of 32 tokens a look-up of the state that nothing
// hides; the library's product with la_conv_seq_kernel behind it pays for neither.  A prompt pass of three such layers and an attention layer, in parts
// / fused in us: 1 x 1000 622 / 591; 4 x 100 406 / 413, 4 x 140 460 / 459, 4 x 220 515 / 501; 8 x 60 396 / 417, 8 x 100 491 / 483; 32 x 40 615 / 631, 32
// x 50 674 / 668; 64 x 40 952 / 954, 64 x 48 1044 / 1007; 128 x 20 1159 / 1169, 128 x 26 1308 / 1275, 128 x 64 2263 / 2045 (around the line, of 3 and 4
// tiles of rows in 6 or 8 sequences, up to 2.7 % either way).  The projection and convolution alone with sequences of 16 tokens: 256 x 16 122 / 128, 512
// x 16 225 / 243, 1024 x 16 431 / 553; of 32: 256 x 32 213 / 197.  One sequence of 4 to 128 rows takes 19 to 23 us against 15 to 19 in parts, but a user
// who waits for every call is served sooner without the parts' run table (a prompt and two tokens, in parts / fused: 9 tokens 714 / 691 us, 77 786 /
// 771, 128 770 / 770, 253 804 / 800).
bool gemm_la_conv_takes(const void* x, const void* w, long long rows, int n_seqs) {
    const bool long_enough = n_seqs == 1 || (rows >= std::min(300 + 36LL * n_seqs, 3000LL) && rows >= 24LL * n_seqs);
    return long_enough && aligned16(x) && aligned16(w);
}

int gemm_la_conv(cudaStream_t s, const __half* x, const __half* w, int rows, const LaConvArgs& la, int* error) {
    PairMaps m{};
    B2_TRY(map_rows(&m.a, ELEM_F16, w, kLaProjCols, kHidden, 64, 128));
    B2_TRY(map_rows(&m.b, ELEM_F16, x, rows, kHidden, 64, 128));
    __half* const out[3] = {la.q, la.k, la.v};
    for (int i = 0; i < 3; ++i) B2_TRY(map_rows(&m.out[i], ELEM_F16, out[i], rows, kLaHeads * kLaKd, 32, 32, false));
    B2_TRY(map_rows(&m.out[3], ELEM_F32, la.mixed, rows, kLaProjCols, 32, 16, false));
    PairArgs p{};
    p.row_tiles = ceil_div(rows, kConvTokens);
    p.col_tiles = ceil_div(kLaProjCols, 256);
    p.k_steps = kHidden / 64;
    p.rows = rows;
    p.cols = kLaProjCols;
    p.error = error;
    p.la = la;
    return launch_pair<kPairConv, __half, B200ATTN_ACT_SILU>(m, p, s);
}

// From four rounds of tiles over the device's pairs on, and of depths at which neither the stores (below 512) nor the products alone (above 3584) decide.
// Pairs / library (cuBLAS 12.8, which a process with PyTorch has) in us back to back, fp32 results: 5120 x 1024 of 3855 / 8192 / 65536 rows 42 / 45, 77 / 98, 599 /
// 754; 8192 x 2048 of 8192 rows 216 / 246; 1024 x 2048 of 65536 rows 213 / 245; 5120 x 512 of 3855 / 65536 rows 30 / 31, 399 / 479; bf16 results: 5120 x 1024 of 3855 /
// 65536 rows 32 / 34, 460 / 539; 8192 x 512 of 16384 rows 116 / 133.  Depth 128, bf16 results: 5120 outputs of 3855 / 65536 rows 14.9 / 12.5, 180 / 143, 1024 of 65536 rows
// 43 / 32 (fp32 results even); depth 3584, 1024 outputs of 40960 rows 202 / 222; depth 4096, 8192 x 8192 376 / 359.  An attention layer of 16384 rows takes
// 506 us with and 520 without them, of 65536 rows 1676 / 1710.  cuBLAS 12.9 alone (a program without PyTorch) is up to 13 % ahead of the pairs instead.
// Products that are added to Y stay with the library: 1024 x 3584 at 3855 / 8192 / 16384 rows 26.3 / 22.0, 49.6 / 47.6, 97.3 / 96.6.
bool gemm_pair_takes(const void* x, int ldx, const void* w, const void* y, int ldy, ElemType in_type, ElemType out_type, int rows, int out, int in) {
    if (in_type == ELEM_F32 || !(out_type == ELEM_F32 || (in_type == ELEM_BF16 && out_type == ELEM_BF16)) || in < 512 || in > 3584) return false;
    if (ldx % 8 != 0 || in % 8 != 0 || ldy * elem_bytes(out_type) % 16 != 0 || !aligned16(x) || !aligned16(w) || !aligned16(y)) return false;
    int sms = 0;
    return device_sm_count(&sms) == 0 && (long long)ceil_div(rows, 256) * ceil_div(out, 256) > 4 * (sms / 2);
}

int gemm_pair(cudaStream_t s, const void* x, int ldx, const void* w, void* y, int ldy, ElemType in_type, ElemType out_type, int rows, int out, int in, int* error) {
    PairMaps m{};
    B2_TRY(map_rows(&m.a, in_type, x, rows, in, 64, 128, true, ldx));
    B2_TRY(map_rows(&m.b, in_type, w, out, in, 64, 128));
    B2_TRY(map_rows(&m.b32, in_type, w, out, in, 64, 32));
    B2_TRY(map_rows(&m.out[0], out_type, y, rows, out, out_type == ELEM_F32 ? 16 : 32, 32, true, ldy));
    PairArgs p{};
    p.row_tiles = ceil_div(rows, 256);
    p.col_tiles = ceil_div(out, 256);
    p.k_steps = ceil_div(in, 64);
    p.rows = rows;
    p.cols = out;
    p.error = error;
    constexpr int kNone = B200ATTN_ACT_SILU;
    if (in_type == ELEM_F16) return launch_pair<kPairStore32, __half, kNone>(m, p, s);
    return out_type == ELEM_F32 ? launch_pair<kPairStore32, __nv_bfloat16, kNone>(m, p, s) : launch_pair<kPairStore16, __nv_bfloat16, kNone>(m, p, s);
}

}  // namespace b200
