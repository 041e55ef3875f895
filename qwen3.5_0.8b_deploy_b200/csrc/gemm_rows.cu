// Y = X W^T for the few rows of a decode step (M <= 16) on mma.sync, 16-bit operands, fp32 sums.
//
// At a few rows a projection is one pass over its weights: the 17 MB of an input projection take 2.5 us at the memory rate.  A library
// GEMM of this shape takes 5.5 to 8 us, because it starts to read them only after the kernel in front of it has finished, and the norm
// in front of it and the SwiGLU behind it are launches of 2 to 3 us each.  So
//   * a CTA owns 8 to 64 output columns with their whole K.  Its weight rows come in by bulk copies that are issued BEFORE the wait on the
//     preceding kernel (no kernel of a step writes weights), and the next launch is let in at once, so that it fetches its own
//     meanwhile.  The slabs of two neighbouring launches of a layer fit an SM together (see launch_pdl_split);
//   * the warps split K, and a warp's partial sums go where its own slice of the weights lay, which no other warp reads.  The
//     reduction over warps needs no shared memory of its own, and its order is fixed;
//   * the fp32 residual rows are normalised on the way in (the rounding point is the norm kernel's: one rounding of the normalised value), and
//     SwiGLU and the residual addition sit in the epilogue.  A layer of a step is five launches in place of eight or nine.
// Measured in a captured step of 8 rows, one CTA's stamps from the dependency wait on: input projection (8224 x 1024) 4.0 us, gate / up with SwiGLU
// (7168 x 1024) 3.7 us, output projections (1024 x 2048 and 1024 x 3584) 2.5 and 3.8 us; the step of four layers and the head 191 us on library GEMMs, 128 us
// here (fp16 cache, 50 tokens).  A Gutenex step of 1 / 16 rows takes 131 / 172 us (165 / 205 with the norms' weights read behind the wait).
// Taken back: X in registers with one column tile at a time (eight warps through 2000 instructions each: 8.6, 9.5 and 4.1 us); asking L2 for the
// weights of the launch after next (no change: the copies are not what a launch waits for).
// Why 16 rows: a step of the hybrid stack at 1 / 8 / 16 rows took 126 / 138 / 163 us (before the copies were shared out) against 194 / 191 / 200 us on library GEMMs.  Two row tiles (17 to 32
// rows) need 203 KB beside the widest slab, so the next launch no longer fits an SM, and 64 registers no longer hold them: at 17 / 24 / 32 rows 228 / 241 /
// 272 us against 193 / 204 / 221 (bf16 stacks 256 to 337 against 206 to 256), the head 25 to 29 us against 18; layers called alone gained 7 % at best.
// Taken out: the library GEMMs serve those steps.  tcgen05 would pad the rows to 64 or 128 and pay for a TMEM round trip (gemm_tc.cu: 9.0, 10.8 and 10.5 us).
#include "gemm_rows.cuh"
#include "elem.cuh"
#include "kernels.cuh"
#include "ptx_utils.cuh"

#include <type_traits>

namespace b200 {
namespace {

template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) { return pack_half2(lo, hi); }
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) { return pack_bf16x2(lo, hi); }
template <typename T> __device__ __forceinline__ void mma_rows(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma_rows<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    mma_16816(d, a0, a1, a2, a3, b0, b1);
}
template <> __device__ __forceinline__ void mma_rows<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <typename YT> __device__ __forceinline__ YT to_out(float v);
template <> __device__ __forceinline__ float to_out<float>(float v) { return v; }
template <> __device__ __forceinline__ __half to_out<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 to_out<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ unsigned long long pack_max(float v, int idx) {
    uint32_t u = __float_as_uint(v);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);                        // order-preserving map of fp32 to uint32
    return ((unsigned long long)u << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)idx);   // ties: smallest index wins
}

// k is assigned to lanes in runs of eight (lane % 4), the same for both operands of a product, so every load is 16 bytes.  Rows of
// operands in shared memory are 64 bytes modulo 128 apart: the two rows that eight lanes read together fill the 32 banks.  A weight row is a bulk
// copy of its own: few large ones (8 rows each, unpadded) arrived later, 158 us a step in place of 149.
__device__ __host__ __forceinline__ int rows_pitch(int k) { return (k * 2 + 127) / 128 * 128 + 64; }

// The items of a launch, cut evenly: part i of n gets [i items / n, (i + 1) items / n).  A launch has one CTA per SM: with fewer, the next
// launch put two CTAs on each idle SM and left no registers there for the one behind it, which then came late.
__device__ __forceinline__ int part_begin(int i, int n, int items) { return (int)((long long)i * items / n); }

// K in slices of `per` chunks of 32, one per warp.  A tile's partial sums of one warp, 16 x 8 floats, lie in the eight weight rows they came
// from, in the slice that this warp alone has read: row m % 8, with the halves m / 8 swapped in every other pair of rows against bank conflicts.
struct Slices {
    int chunks, per, active;      // active slices
    __device__ __forceinline__ Slices(int k, int warps) : chunks(k / 32) {
        per = (chunks + warps - 1) / warps;
        active = (chunks + per - 1) / per;
    }
    __device__ __forceinline__ int begin(int w) const { return min(chunks, w * per); }
    __device__ __forceinline__ static int at(int m, int pitch) { return (m & 7) * pitch + (((m >> 3) ^ ((m >> 1) & 1)) * 32); }
    __device__ __forceinline__ void store(unsigned char* tile, int pitch, int w, int r, int c, const float (&acc)[4]) const {
        unsigned char* slice = tile + w * per * 64 + 8 * c;
        *reinterpret_cast<float2*>(slice + at(r, pitch)) = make_float2(acc[0], acc[1]);
        *reinterpret_cast<float2*>(slice + at(8 + r, pitch)) = make_float2(acc[2], acc[3]);
    }
    __device__ __forceinline__ float total(const unsigned char* tile, int pitch, int m, int n) const {
        const unsigned char* p = tile + at(m, pitch) + 4 * n;
        float v = 0.f;
#pragma unroll 8
        for (int w = 0; w < active; ++w) v += *reinterpret_cast<const float*>(p + w * per * 64);
        return v;
    }
};

// The gate's activation: library functions in fp16 stacks (swiglu_kernel), the forms of act_mul_kernel where the result is rounded to bf16.
template <typename T, int EPI>
__device__ __forceinline__ float rows_act(float g) {
    using A = std::conditional_t<std::is_same_v<T, __nv_bfloat16>, __nv_bfloat16, float>;
    if constexpr (EPI == kRowsGeglu) return times_sigmoid<A>(g, 1.5957691216057308f * (g + 0.044715f * g * g * g));
    else return times_sigmoid<A>(g, g);
}

// The next kernel of the stream may take its place at once.  If it is one of these it fetches weights and waits; any other waits before it touches
// what a step writes, or reads recurrent state that was written before the step's embedding launch, which waits first (la_decode_kernel).  Where no
// such launch lies between two calls (RowsGemm::late) this one waits first, whichever of the kernels the shape takes.
__device__ __forceinline__ void rows_enter(bool late) {
    if (!late) pdl_launch_dependents();
    pdl_wait();
    if (late) pdl_launch_dependents();
}

constexpr int kRowsThreads = 512, kRowsWarps = 16, kRows = kRowsGemmMax;
static_assert(kRows == 16, "one row tile of mma.m16n8k16");

// The norm's weights, which no kernel of a step writes, come into shared memory by a copy that is issued with those of the product's weights.  Read from L2
// behind the dependency wait (which empties L1), one load after the other between the stores of the normalised row, they took 3.5 us of a launch.
template <int LOAD>
__device__ __forceinline__ bool norms_with_weights(const RowsGemm& a) { return (LOAD == kLoadNorm || LOAD == kLoadAddNorm) && a.norm_w; }
inline size_t norm_bytes(const RowsGemm& a) { return a.norm_w ? (size_t)a.K * 4 : 0; }

// X into shared memory as 16-bit rows, a warp per row.  s_norm: the norm's weights, there once norm_bar's first phase is over.  False: they did not come.
template <typename T, int LOAD, int WARPS>
__device__ __forceinline__ bool load_rows(const RowsGemm& a, unsigned char* sx, int pitch, int warp, int lane, const float* s_norm, uint32_t norm_bar,
                                          volatile int* abort_flag) {
    bool ok = true;
#pragma unroll 1
    for (int m = warp; m < a.M; m += WARPS) {
        const size_t at = (size_t)(a.row_index ? a.row_index[m] : m) * a.ldx;
        unsigned char* dst = sx + m * pitch;
        if constexpr (LOAD == kLoadAsIs) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int k = 8 * (32 * i + lane);
                if (k < a.K) *reinterpret_cast<uint4*>(dst + 2 * k) = __ldcg(reinterpret_cast<const uint4*>(static_cast<const T*>(a.x) + at + k));
            }
        } else {
            const float* xr = static_cast<const float*>(a.x) + at;
            const float* src = LOAD == kLoadAddNorm ? a.add + (size_t)m * a.K : xr;
            float4 v[8];
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int k = 4 * (32 * i + lane);
                v[i] = k < a.K ? __ldcg(reinterpret_cast<const float4*>(src + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            float rs = 1.0f;
            if constexpr (LOAD < kLoadF32) {
#pragma unroll
                for (int i = 0; i < 8; ++i) ss += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                rs = 1.0f / sqrtf(ss / (float)a.K + a.eps);
                if (norms_with_weights<LOAD>(a) && ok) ok = mbar_wait_warp(norm_bar, 0, abort_flag);
            }
            float4 h[4];                         // kLoadAddNorm: what is added to, half a row at a time
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int k = 4 * (32 * i + lane);
                if constexpr (LOAD == kLoadAddNorm) {
                    if ((i & 3) == 0) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int kj = k + 128 * j;
                            h[j] = kj < a.K ? __ldcg(reinterpret_cast<const float4*>(xr + kj)) : make_float4(0.f, 0.f, 0.f, 0.f);
                        }
                    }
                }
                if (k < a.K) {
                    float4 w = make_float4(rs, rs, rs, rs);
                    if (LOAD < kLoadF32 && a.norm_w) {
                        const float4 f = *reinterpret_cast<const float4*>(s_norm + k);
                        w = make_float4(rs * (a.norm_base + f.x), rs * (a.norm_base + f.y), rs * (a.norm_base + f.z), rs * (a.norm_base + f.w));
                    }
                    float4 n = make_float4(v[i].x * w.x, v[i].y * w.y, v[i].z * w.z, v[i].w * w.w);
                    if constexpr (LOAD == kLoadF32Lo)
                        n = make_float4((n.x - __half2float(__float2half_rn(n.x))) * kLoScale, (n.y - __half2float(__float2half_rn(n.y))) * kLoScale,
                                        (n.z - __half2float(__float2half_rn(n.z))) * kLoScale, (n.w - __half2float(__float2half_rn(n.w))) * kLoScale);
                    if constexpr (LOAD == kLoadAddNorm) {
                        n = make_float4(h[i & 3].x + n.x, h[i & 3].y + n.y, h[i & 3].z + n.z, h[i & 3].w + n.w);
                        if (blockIdx.x == m % gridDim.x) *reinterpret_cast<float4*>(a.x_out + (size_t)m * a.K + k) = n;
                    }
                    *reinterpret_cast<uint2*>(dst + 2 * k) = make_uint2(pack2<T>(n.x, n.y), pack2<T>(n.z, n.w));
                }
            }
        }
    }
    if (!ok) mbar_drain(norm_bar, 0);
    return ok;
}

// Many columns, K <= 1024: X in shared memory, up to eight column tiles per CTA.  A warp multiplies four tiles (two groups of eight warps when a
// launch has CTAs with more than four) over its slice of K.  Gated: units of two tiles, 8 gate rows of the weights and the 8 up rows that
// belong to them; the slab holds all gate rows, then all up rows.
template <typename T, int LOAD, int EPI, typename YT>
__global__ void __launch_bounds__(kRowsThreads, 2)
rows_wide_kernel(const RowsGemm a, unsigned long long* stamp) {
    constexpr bool kGated = EPI == kRowsSwiglu || EPI == kRowsGeglu;
    extern __shared__ __align__(128) unsigned char smem[];
    const int pitch = rows_pitch(a.K), row_bytes = a.K * 2;
    unsigned char* sx = smem + 8 * a.tiles * pitch;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sx + kRows * pitch);                          // of the weights, of the norm's
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bar + 2);
    float* s_norm = reinterpret_cast<float*>(sx + kRows * pitch + 32);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    const int cols = kGated ? a.N / 2 : a.N, units = (cols + 7) / 8;                         // output columns, and eights of them
    const int u0 = part_begin(blockIdx.x, gridDim.x, units), u1 = part_begin(blockIdx.x + 1, gridDim.x, units);
    const int col0 = 8 * u0, n_cols = min(cols, 8 * u1) - col0, half = 8 * (u1 - u0) * pitch;      // gated: the up rows' place
    const int tiles = (kGated ? 2 : 1) * (u1 - u0);

    if (tid == 0) {
        mbar_init(smem_u32(bar), 1);
        mbar_init(smem_u32(bar + 1), 1);
        *abort_flag = 0;
        mbar_fence_init();
        if (n_cols > 0) mbar_arrive_expect_tx(smem_u32(bar), (uint32_t)((kGated ? 2 : 1) * n_cols * row_bytes));
        if (norms_with_weights<LOAD>(a)) {
            mbar_arrive_expect_tx(smem_u32(bar + 1), (uint32_t)a.K * 4);
            bulk_g2s(smem_u32(s_norm), a.norm_w, (uint32_t)a.K * 4, smem_u32(bar + 1));
        }
    }
    __syncthreads();
    // A lane's copy takes 45 ns to issue, whoever of the warp is next: all warps share them.
    for (int i = warp + kRowsWarps * lane; i < n_cols; i += 32 * kRowsWarps) {
        const int n = col0 + i, from = kGated ? n + n / a.group * a.group : n;
        bulk_g2s(smem_u32(smem) + i * pitch, static_cast<const T*>(a.w) + (size_t)from * a.K, (uint32_t)row_bytes, smem_u32(bar));
        if (kGated)
            bulk_g2s(smem_u32(smem) + half + i * pitch, static_cast<const T*>(a.w) + (size_t)(from + a.group) * a.K, (uint32_t)row_bytes, smem_u32(bar));
    }
    __syncwarp();
    const int wide_log2 = a.tiles > 4 ? 3 : 4, splits = 1 << wide_log2, split = warp & (splits - 1), tile0 = (warp >> wide_log2) * 4;
    const Slices sl(a.K, splits);
    const int c0 = sl.begin(split), c1 = sl.begin(split + 1);
    const bool high = a.M > 8;
    rows_enter(a.late);
    stamp_begin(stamp);
    const bool rows_ok = load_rows<T, LOAD, kRowsWarps>(a, sx, pitch, warp, lane, s_norm, smem_u32(bar + 1), abort_flag);
    __syncthreads();
    if (n_cols <= 0) return;

    // ---- products --------------------------------------------------------------------------------------------------------
    auto tile_at = [&](int t) { return smem + (kGated ? (t & 1) * half + 8 * (t >> 1) * pitch : 8 * t * pitch); };
    const bool ok = mbar_wait(smem_u32(bar), 0, abort_flag) && rows_ok;
    if (!ok) mbar_drain(smem_u32(bar), 0);
    float acc[4][4] = {};
    const unsigned char* xp = sx + r * pitch + c * 16;
    // These two as functions: written out in the loop, ptxas spilled in the variants on 16-bit rows, 1.5 us more a step of the bf16 stacks.
    auto x_frag = [&](int ch, uint4& lo, uint4& hi) {
        lo = *reinterpret_cast<const uint4*>(xp + ch * 64);
        hi = make_uint4(0u, 0u, 0u, 0u);
        if (high) hi = *reinterpret_cast<const uint4*>(xp + 8 * pitch + ch * 64);
    };
    auto multiply = [&](float (&d)[4], const uint4& lo, const uint4& hi, const uint4& b) {
        mma_rows<T>(d, lo.x, hi.x, lo.y, hi.y, b.x, b.y);
        mma_rows<T>(d, lo.z, hi.z, lo.w, hi.w, b.z, b.w);
    };
#pragma unroll 2
    for (int ch = c0; ch < c1; ++ch) {
        uint4 lo, hi;
        x_frag(ch, lo, hi);
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (tile0 + t < tiles) {
                const uint4 b = *reinterpret_cast<const uint4*>(tile_at(tile0 + t) + r * pitch + c * 16 + ch * 64);
                multiply(acc[t], lo, hi, b);
            }
    }
    __syncwarp();                                // every lane has read the slice: it may be overwritten
    if (c0 < c1) {
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (tile0 + t < tiles) sl.store(tile_at(tile0 + t), pitch, split, r, c, acc[t]);
    }
    __syncthreads();
    const int n8 = tid & 7, em = (tid >> 3) % kRows;
    unsigned long long best = pack_max(-INFINITY, 0);      // a row without a number above -inf gives token 0
    if (em < a.M && ok) {
        for (int u = tid / (8 * kRows); u < u1 - u0; u += kRowsThreads / (8 * kRows)) {
            const int n = col0 + 8 * u + n8;
            if (n >= cols) break;
            if constexpr (kGated) {
                const float g = sl.total(tile_at(2 * u), pitch, em, n8), up = sl.total(tile_at(2 * u + 1), pitch, em, n8);
                static_cast<YT*>(a.y)[(size_t)em * a.ldy + n] = to_out<YT>(rows_act<T, EPI>(g) * up);
            } else {
                float v = sl.total(tile_at(u), pitch, em, n8) * a.scale;
                if (a.cap > 0.f) v = a.cap * tanhf(v / a.cap);
                if constexpr (EPI == kRowsStore && std::is_same_v<YT, float>) {
                    if (a.accumulate) v += __ldcg(static_cast<const float*>(a.y) + (size_t)em * a.ldy + n);
                }
                if constexpr (EPI == kRowsStore) static_cast<YT*>(a.y)[(size_t)em * a.ldy + n] = to_out<YT>(v);
                else if (v > -INFINITY) best = max(best, pack_max(v, n));
            }
        }
    }
    if constexpr (EPI == kRowsArgmax) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
        if (n8 == 0 && em < a.M) atomicMax(a.packed + em, best);
    }
    if (stamp) {
        __syncthreads();
        stamp_end(stamp);
    }
    if (tid == 0 && *abort_flag && a.error) atomicExch(a.error, 7);
}

// More columns than a wave of CTAs holds at eight tiles each (the LM head), K <= 1024: the warps work on tiles of their own.  A warp streams
// its tiles' weights through one slab in two halves of K, each refilled as soon as it has been multiplied, so that most of the 135 KB are
// in flight all the time, and no barrier of the CTA and no reduction stands between two tiles.
// From the dependency wait on, this / gemm_tc.cu's kernel, which needs a norm launch in front: 32768 columns at 8 rows 16.4 / 18.3 us (67 MB), 248320 at 1 / 8 / 16 rows
// 78 / 81 / 89 against 104 / 111 / 111 us (509 MB).  A ring at whose batches of tiles all warps met took 19.4 us at 32768.
constexpr int kStreamWarps = 8;
template <typename T, int LOAD, int EPI>
__global__ void __launch_bounds__(kStreamWarps * 32)
rows_stream_kernel(const RowsGemm a, unsigned long long* stamp) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int pitch = rows_pitch(a.K), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    unsigned char* sw = smem + warp * 8 * pitch;
    unsigned char* sx = smem + kStreamWarps * 8 * pitch;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sx + kRows * pitch);                // two per warp
    unsigned long long* s_best = reinterpret_cast<unsigned long long*>(bars + 2 * kStreamWarps);     // [kRows]
    uint64_t* norm_bar = reinterpret_cast<uint64_t*>(s_best + kRows);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(norm_bar + 1);
    float* s_norm = reinterpret_cast<float*>(norm_bar + 2);
    const uint32_t bar = smem_u32(bars + 2 * warp);
    const int chunks = a.K / 32, mid = (chunks + 1) / 2, n_tiles = (a.N + 7) / 8, step = gridDim.x * kStreamWarps;
    const int first = blockIdx.x + gridDim.x * warp;
    auto fetch = [&](int tile, int half) {
        const int k0 = half ? mid * 32 : 0, n = (half ? chunks - mid : mid) * 32, rows = min(8, a.N - 8 * tile);
        if (n == 0) return;
        if (lane == 0) mbar_arrive_expect_tx(bar + 8 * half, (uint32_t)(rows * n * 2));
        __syncwarp();
        if (lane < rows)
            bulk_g2s(smem_u32(sw) + lane * pitch + 2 * k0, static_cast<const T*>(a.w) + (size_t)(8 * tile + lane) * a.K + k0, (uint32_t)n * 2, bar + 8 * half);
    };
    if (lane == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 8, 1);
        if (warp == 0) *abort_flag = 0;
        mbar_fence_init();
    }
    if (tid == 0) {
        mbar_init(smem_u32(norm_bar), 1);
        mbar_fence_init();
        if (norms_with_weights<LOAD>(a)) {
            mbar_arrive_expect_tx(smem_u32(norm_bar), (uint32_t)a.K * 4);
            bulk_g2s(smem_u32(s_norm), a.norm_w, (uint32_t)a.K * 4, smem_u32(norm_bar));
        }
    }
    if (tid < kRows) s_best[tid] = 0ull;
    __syncthreads();
    if (first < n_tiles) { fetch(first, 0); fetch(first, 1); }
    rows_enter(a.late);
    stamp_begin(stamp);
    const bool rows_ok = load_rows<T, LOAD, kStreamWarps>(a, sx, pitch, warp, lane, s_norm, smem_u32(norm_bar), abort_flag);
    __syncthreads();

    const bool high = a.M > 8;
    unsigned long long best[2] = {pack_max(-INFINITY, 0), pack_max(-INFINITY, 0)};       // a row without a number above -inf gives token 0
    const unsigned char* xp = sx + r * pitch + c * 16;
    const unsigned char* wp = sw + r * pitch + c * 16;
    uint32_t parity = 0;
    bool ok = true;
    if (!rows_ok && first < n_tiles) {           // its first copies are on their way
        mbar_drain(bar, 0);
        if (mid < chunks) mbar_drain(bar + 8, 0);
    }
    for (int tile = first; ok && rows_ok && tile < n_tiles; tile += step, parity ^= 1u) {
        float acc[2][4] = {};                    // two chains
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            const int c0 = half ? mid : 0, c1 = half ? chunks : mid;
            if (c0 == c1) continue;
            ok = mbar_wait_warp(bar + 8 * half, parity, abort_flag);
            if (!ok) {                           // this half's copies, and the other half's: of this tile behind it, or of the next
                mbar_drain(bar + 8 * half, parity);
                if (half ? tile + step < n_tiles : mid < chunks) mbar_drain(bar + 8 * (half ^ 1), parity ^ half);
                break;
            }
#pragma unroll 4
            for (int ch = c0; ch < c1; ++ch) {
                const uint4 b = *reinterpret_cast<const uint4*>(wp + ch * 64);
                const uint4 lo = *reinterpret_cast<const uint4*>(xp + ch * 64);
                uint4 hi = make_uint4(0u, 0u, 0u, 0u);
                if (high) hi = *reinterpret_cast<const uint4*>(xp + 8 * pitch + ch * 64);
                mma_rows<T>(acc[0], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
                mma_rows<T>(acc[1], lo.z, hi.z, lo.w, hi.w, b.z, b.w);
            }
            __syncwarp();                        // every lane has read the half
            if (tile + step < n_tiles) {
                fence_proxy_async_smem();        // it was read by ordinary loads, the next copy into it is not one
                fetch(tile + step, half);
            }
        }
        if (!ok) break;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int m = 8 * (i >> 1) + r, n = 8 * tile + 2 * c + (i & 1);
            float v = (acc[0][i] + acc[1][i]) * a.scale;
            if (m >= a.M || n >= a.N) continue;
            if constexpr (EPI == kRowsStore) {
                if (a.cap > 0.f) v = a.cap * tanhf(v / a.cap);
                static_cast<float*>(a.y)[(size_t)m * a.ldy + n] = v;
            } else if (v > -INFINITY) {
                best[i >> 1] = max(best[i >> 1], pack_max(v, n));
            }
        }
    }
    if constexpr (EPI == kRowsArgmax) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            best[i] = max(best[i], __shfl_xor_sync(0xffffffffu, best[i], 1));
            best[i] = max(best[i], __shfl_xor_sync(0xffffffffu, best[i], 2));
            if (c == 0) atomicMax(s_best + 8 * i + r, best[i]);
        }
        __syncthreads();
        if (tid < a.M) atomicMax(a.packed + tid, s_best[tid]);
    }
    __syncthreads();
    stamp_end(stamp);
    if (tid == 0 && *abort_flag && a.error) atomicExch(a.error, 7);
}

// Few columns, deep K <= 4096: fp32 Y[M, N] = X W^T, added to what is there with ADD.  Up to eight columns per CTA (six or seven of 1024 on 148
// SMs), the 16 warps split K, X goes from L2 straight into the registers of the warp that multiplies it, kAhead chunks at a time: all that a warp has
// for up to eight rows, in two round trips to L2 for more rows (HIGH) and K above 2048.
template <typename T, bool ADD, bool HIGH>
__global__ void __launch_bounds__(kRowsThreads, 2)
rows_deep_kernel(const RowsGemm a, unsigned long long* stamp) {
    constexpr int kHalves = HIGH ? 2 : 1, kAhead = HIGH ? 4 : 8;
    extern __shared__ __align__(128) unsigned char smem[];
    const int pitch = rows_pitch(a.K);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 8 * pitch);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    const int n0 = part_begin(blockIdx.x, gridDim.x, a.N), cols = part_begin(blockIdx.x + 1, gridDim.x, a.N) - n0;
    const int n8 = tid & 7, em = (tid >> 3) % kRows;
    if (warp == 0) {
        if (lane == 0) {
            mbar_init(smem_u32(bar), 1);
            *abort_flag = 0;
            mbar_fence_init();
            mbar_arrive_expect_tx(smem_u32(bar), (uint32_t)(cols * a.K * 2));
        }
        __syncwarp();
        if (lane < cols)
            bulk_g2s(smem_u32(smem) + lane * pitch, static_cast<const T*>(a.w) + (size_t)(n0 + lane) * a.K, (uint32_t)a.K * 2, smem_u32(bar));
    }
    const Slices sl(a.K, kRowsWarps);
    const int c0 = sl.begin(warp), c1 = sl.begin(warp + 1);
    rows_enter(a.late);
    stamp_begin(stamp);
    const bool writes = tid < 8 * kRows && em < a.M && n8 < cols;
    float res = 0.f;
    if (ADD && writes) res = __ldcg(static_cast<const float*>(a.y) + (size_t)em * a.ldy + n0 + n8);
    const T* xp = static_cast<const T*>(a.x) + (size_t)r * a.ldx + 8 * c;
    auto load = [&](int i, int ch) {             // rows 8 i + r, chunk ch
        return 8 * i + r < a.M && ch < c1 ? __ldcg(reinterpret_cast<const uint4*>(xp + (size_t)8 * i * a.ldx + 32 * ch)) : make_uint4(0u, 0u, 0u, 0u);
    };
    uint4 x[kAhead][kHalves];
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
#pragma unroll
        for (int i = 0; i < kHalves; ++i) x[j][i] = load(i, c0 + j);
    __syncthreads();                             // the barrier is initialised
    const bool ok = mbar_wait(smem_u32(bar), 0, abort_flag);
    if (!ok) mbar_drain(smem_u32(bar), 0);
    float acc[2][4] = {};                        // two chains
    const unsigned char* wp = smem + r * pitch + c * 16;
#pragma unroll 1
    for (int g = c0; g < c1; g += kAhead) {
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            if (g + j >= c1) break;
            const uint4 b = *reinterpret_cast<const uint4*>(wp + (g + j) * 64);
            const uint4 lo = x[j][0], hi = HIGH ? x[j][kHalves - 1] : make_uint4(0u, 0u, 0u, 0u);
            mma_rows<T>(acc[0], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
            mma_rows<T>(acc[1], lo.z, hi.z, lo.w, hi.w, b.z, b.w);
#pragma unroll
            for (int i = 0; i < kHalves; ++i) x[j][i] = load(i, g + j + kAhead);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[0][i] += acc[1][i];
    __syncwarp();
    if (c0 < c1) sl.store(smem, pitch, warp, r, c, acc[0]);
    __syncthreads();
    if (writes && ok) static_cast<float*>(a.y)[(size_t)em * a.ldy + n0 + n8] = res + sl.total(smem, pitch, em, n8);
    if (stamp) {
        __syncthreads();
        stamp_end(stamp);
    }
    if (tid == 0 && *abort_flag && a.error) atomicExch(a.error, 7);
}

// Most shared memory of a launch: 64 weight rows, 16 of X, the norm's weights.  A layer's launches fit side by side: 153 and 34 KB, 169 and 57 KB (of 228
// with 1 KB reserved for each, so that the norm's 4 KB just fit).
constexpr int kSharedMost = 176 * 1024;

template <typename K>
int prepare(PerDeviceOnce& once, K kernel) {
    B2_PER_DEVICE_ONCE(once, B2_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedMost)));
    return 0;
}

template <typename T, int LOAD, int EPI, typename YT>
int launch_wide(RowsGemm a, cudaStream_t s, ProfKind kind) {
    static PerDeviceOnce once;
    B2_TRY(prepare(once, rows_wide_kernel<T, LOAD, EPI, YT>));
    int sms = 0;
    B2_TRY(device_sm_count(&sms));
    const int unit = EPI == kRowsSwiglu || EPI == kRowsGeglu ? 2 : 1, units = ceil_div(a.N / unit, 8);
    const int waves = ceil_div(units * unit, 8 * sms), grid = std::min(units, waves * sms);     // one CTA per SM where eight tiles each are enough
    a.tiles = ceil_div(units, grid) * unit;
    const size_t smem = (size_t)(8 * a.tiles + kRows) * rows_pitch(a.K) + 32 + norm_bytes(a);
    unsigned long long* stamp = prof_stamp_slot(kind);
    launch_pdl_split(true, true, rows_wide_kernel<T, LOAD, EPI, YT>, dim3(grid), dim3(kRowsThreads), smem, s, a, stamp);
    B2_LAUNCH_CHECK();
    return 0;
}

template <typename T, int LOAD, int EPI>
int launch_stream(const RowsGemm& a, int sms, cudaStream_t s, ProfKind kind) {
    static PerDeviceOnce once;
    B2_TRY(prepare(once, rows_stream_kernel<T, LOAD, EPI>));
    const size_t smem = (size_t)(8 * kStreamWarps + kRows) * rows_pitch(a.K) + 8 * (2 * kStreamWarps + kRows) + 16 + norm_bytes(a);
    unsigned long long* stamp = prof_stamp_slot(kind);
    launch_pdl_split(true, true, rows_stream_kernel<T, LOAD, EPI>, dim3(sms), dim3(kStreamWarps * 32), smem, s, a, stamp);
    B2_LAUNCH_CHECK();
    return 0;
}

template <typename T, bool ADD, bool HIGH>
int launch_deep_rows(const RowsGemm& a, cudaStream_t s) {
    static PerDeviceOnce once;
    B2_TRY(prepare(once, rows_deep_kernel<T, ADD, HIGH>));
    unsigned long long* stamp = prof_stamp_slot(PROF_GEMM_RES);
    int sms = 0;
    B2_TRY(device_sm_count(&sms));
    const int grid = std::max(ceil_div(a.N, 8), std::min(a.N, sms));      // up to eight columns a CTA
    launch_pdl_split(true, true, rows_deep_kernel<T, ADD, HIGH>, dim3(grid), dim3(kRowsThreads), (size_t)8 * rows_pitch(a.K) + 16, s, a, stamp);
    B2_LAUNCH_CHECK();
    return 0;
}
template <typename T, bool ADD>
int launch_deep(const RowsGemm& a, cudaStream_t s) {
    return a.M > 8 ? launch_deep_rows<T, ADD, true>(a, s) : launch_deep_rows<T, ADD, false>(a, s);
}

template <typename T, int LOAD, int EPI, typename YT>
int wide(const RowsGemm& a, cudaStream_t s, ProfKind kind) {
    // Above eight tiles a CTA: the streaming form, for the outputs that such products have.  At 9472 columns and fewer (148 SMs) a CTA holds its
    // whole slab, which is fetched before the wait, and splitting K over the warps ends sooner.
    if constexpr ((EPI == kRowsStore && std::is_same_v<YT, float>) || EPI == kRowsArgmax) {
        int sms = 0;
        B2_TRY(device_sm_count(&sms));
        if (a.N > 64 * sms && !a.accumulate) return launch_stream<T, LOAD, EPI>(a, sms, s, kind);
    }
    return launch_wide<T, LOAD, EPI, YT>(a, s, kind);
}

}  // namespace

bool gemm_rows_takes(const RowsGemm& a, int epi) {
    const bool deep = epi == kRowsResidual || epi == kRowsDeepStore;
    return a.M > 0 && a.M <= kRowsGemmMax && a.N > 0 && a.K > 0 && a.K % 32 == 0 && a.K <= (deep ? 4096 : 1024) && a.ldx % 8 == 0 &&
           ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.norm_w)) & 15) == 0;
}

int gemm_rows(cudaStream_t s, const RowsGemm& a, ElemType type, int epi, int load, ElemType out) {
    if (!gemm_rows_takes(a, epi)) B2_FAIL(B200ATTN_ERR_UNSUPPORTED, "gemm_rows: unsupported shape %d x %d x %d", a.M, a.N, a.K);
    using B = __nv_bfloat16;
    const bool norm = load == kLoadNorm;
    if (type == ELEM_F16) {
        if (epi == kRowsStore && out == ELEM_F32 && load == kLoadF32Lo) return wide<__half, kLoadF32Lo, kRowsStore, float>(a, s, PROF_GEMM_IN);
        if (epi == kRowsStore && out == ELEM_F32 && load == kLoadF32) return wide<__half, kLoadF32, kRowsStore, float>(a, s, PROF_GEMM_IN);
        if (epi == kRowsStore && out == ELEM_F32 && norm) return wide<__half, kLoadNorm, kRowsStore, float>(a, s, PROF_GEMM_IN);
        if (epi == kRowsSwiglu && out == ELEM_F16 && norm) return wide<__half, kLoadNorm, kRowsSwiglu, __half>(a, s, PROF_GEMM_FFN);
        if (epi == kRowsResidual) return launch_deep<__half, true>(a, s);
        if (epi == kRowsDeepStore) return launch_deep<__half, false>(a, s);
        if (epi == kRowsArgmax)
            return norm ? wide<__half, kLoadNorm, kRowsArgmax, float>(a, s, PROF_LM_HEAD) : wide<__half, kLoadAsIs, kRowsArgmax, float>(a, s, PROF_LM_HEAD);
    }
    if (type == ELEM_BF16) {
#define ROWS_LOADS(EPI, YT, PROF)                                                                                                     \
    return a.add ? wide<B, kLoadAddNorm, EPI, YT>(a, s, PROF) : norm ? wide<B, kLoadNorm, EPI, YT>(a, s, PROF) : wide<B, kLoadAsIs, EPI, YT>(a, s, PROF)
        if (epi == kRowsStore && out == ELEM_F32) ROWS_LOADS(kRowsStore, float, PROF_GEMM_IN);
        if (epi == kRowsSwiglu) ROWS_LOADS(kRowsSwiglu, B, PROF_GEMM_FFN);
        if (epi == kRowsGeglu) ROWS_LOADS(kRowsGeglu, B, PROF_GEMM_FFN);
#undef ROWS_LOADS
        if (epi == kRowsStore && out == ELEM_BF16 && !a.add)
            return norm ? wide<B, kLoadNorm, kRowsStore, B>(a, s, PROF_GEMM_IN) : wide<B, kLoadAsIs, kRowsStore, B>(a, s, PROF_GEMM_IN);
        if (epi == kRowsResidual) return launch_deep<B, true>(a, s);
        if (epi == kRowsDeepStore) return launch_deep<B, false>(a, s);
    }
    B2_FAIL(B200ATTN_ERR_UNSUPPORTED, "gemm_rows: unsupported types");
}

}  // namespace b200
