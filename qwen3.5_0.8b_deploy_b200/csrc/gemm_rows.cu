// Y = X W^T for the few rows of a decode step (M <= 32) on mma.sync, 16-bit operands, fp32 sums.
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
// Measured in a captured step of 8 rows, from the dependency wait on: input projection (8224 x 1024) 5.4 us, gate / up with SwiGLU (7168 x 1024)
// 4.6 us, output projections (1024 x 2048 and 1024 x 3584) 3.8 us; the step of four layers and the head 237 -> 149 us.  The first form, with X
// in registers and one column tile at a time, ran eight warps through 2000 instructions each and took 8.6, 9.5 and 4.1 us.
// tcgen05 would pad the rows to 64 or 128 and pay for a TMEM round trip (the kernels of gemm_tc.cu: 9.0, 10.8 and 10.5 us).  From 33 rows on X no
// longer fits beside the slabs, and the library GEMMs serve the step.
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
// operands in shared memory are 64 bytes modulo 128 apart: the two rows that eight lanes read together fill the 32 banks.
__device__ __forceinline__ int rows_pitch(int k) { return (k * 2 + 127) / 128 * 128 + 64; }

// A tile's partial sums of one warp, 16 MT x 8 floats, lie in the eight weight rows they came from, in the slice [64 k0, 64 (k0 + chunks))
// that this warp alone has read: row m % 8, with the halves m / 8 swapped in every other pair of rows against bank conflicts.
__device__ __forceinline__ uint32_t part_at(int m, int pitch) {
    return (uint32_t)((m & 7) * pitch + (((m >> 3) ^ ((m >> 1) & 1)) * 32));
}
template <int MT>
__device__ __forceinline__ void store_part(unsigned char* slice, int pitch, int r, int c, const float (&acc)[MT][4]) {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        *reinterpret_cast<float2*>(slice + part_at(16 * mt + r, pitch) + 8 * c) = make_float2(acc[mt][0], acc[mt][1]);
        *reinterpret_cast<float2*>(slice + part_at(16 * mt + 8 + r, pitch) + 8 * c) = make_float2(acc[mt][2], acc[mt][3]);
    }
}

// The gate's activation: library functions in fp16 stacks (swiglu_kernel), the forms of act_mul_kernel where the result is rounded to bf16.
template <typename T, int EPI>
__device__ __forceinline__ float rows_act(float g) {
    using A = std::conditional_t<std::is_same_v<T, __nv_bfloat16>, __nv_bfloat16, float>;
    if constexpr (EPI == kRowsGeglu) return times_sigmoid<A>(g, 1.5957691216057308f * (g + 0.044715f * g * g * g));
    else return times_sigmoid<A>(g, g);
}

constexpr int kRowsThreads = 512, kRowsWarps = 16;

// Many columns, K <= 1024: X in shared memory as 16-bit rows, `tiles` column tiles at a time.  A warp multiplies four tiles (two groups
// of eight warps when there are more than four) over its part of K.  grid: CTAs walk batches of `tiles` tiles; `buffers` slabs of
// weights in a ring.  LOAD: X comes in as 16-bit rows, as fp32 rows to normalise, or as
// fp32 rows to which normalised rows `add` are added first; the sums then also go to x_out, row m from CTA m.
enum { kLoadAsIs = 0, kLoadNorm, kLoadAddNorm };
template <typename T, int MT, int LOAD, int EPI, typename YT>
__global__ void __launch_bounds__(kRowsThreads, 2)
rows_wide_kernel(const RowsGemm a, unsigned long long* stamp) {
    constexpr int kRows = 16 * MT;
    constexpr bool kGated = EPI == kRowsSwiglu || EPI == kRowsGeglu;
    extern __shared__ __align__(128) unsigned char smem[];
    const int pitch = rows_pitch(a.K), batch_rows = 8 * a.tiles;
    const uint32_t slab = (uint32_t)(batch_rows * pitch);
    unsigned char* sx = smem + a.buffers * slab;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sx + kRows * pitch);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + a.buffers);
    const uint32_t base = smem_u32(smem), bar0 = smem_u32(bars);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    const int batches = (a.N + batch_rows - 1) / batch_rows;

    // Weight row behind row j of a batch.  SwiGLU: pairs of tiles, 8 gate rows then the 8 matching up rows.
    auto weight_row = [&](int batch, int j) {
        if constexpr (kGated) {
            const int ch = batch * (batch_rows / 2) + (j >> 4) * 8 + (j & 7);
            return 2 * ch < a.N ? (ch / a.group) * 2 * a.group + ch % a.group + ((j & 8) ? a.group : 0) : -1;
        } else {
            const int n = batch * batch_rows + j;
            return n < a.N ? n : -1;
        }
    };
    auto fetch = [&](int batch, int buf) {      // warp 0: one bulk copy per row; the barrier first learns the number of bytes
        const uint32_t bytes = (uint32_t)a.K * 2;
        int have = 0;
        for (int j = lane; j < batch_rows; j += 32) have += weight_row(batch, j) >= 0;
        have = __reduce_add_sync(0xffffffffu, have);
        if (lane == 0) mbar_arrive_expect_tx(bar0 + 8u * buf, (uint32_t)have * bytes);
        __syncwarp();
        for (int j = lane; j < batch_rows; j += 32) {
            const int n = weight_row(batch, j);
            if (n >= 0) bulk_g2s(base + buf * slab + j * pitch, static_cast<const T*>(a.w) + (size_t)n * a.K, bytes, bar0 + 8u * buf);
        }
    };
    int next = blockIdx.x;                       // warp 0's next batch to fetch
    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < a.buffers; ++i) mbar_init(bar0 + 8u * i, 1);
            *abort_flag = 0;
            mbar_fence_init();
        }
        __syncwarp();
        for (int i = 0; i < a.buffers && next < batches; ++i, next += gridDim.x) fetch(next, i);
    }
    // The next kernel of the stream may take its place now.  If it is one of these it fetches weights and waits; any other waits before
    // it touches what a step writes, or reads recurrent state that a kernel writes only after a wait of its own (la_decode_kernel).
    pdl_launch_dependents();
    pdl_wait();
    stamp_begin(stamp);

    // ---- X: a warp per row ---------------------------------------------------------------------------------------------
#pragma unroll 1
    for (int m = warp; m < a.M; m += kRowsWarps) {
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
#pragma unroll
            for (int i = 0; i < 8; ++i) ss += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            const float rs = 1.0f / sqrtf(ss / (float)a.K + a.eps);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int k = 4 * (32 * i + lane);
                if (k < a.K) {
                    float4 w = make_float4(rs, rs, rs, rs);
                    if (a.norm_w) {
                        const float4 f = __ldg(reinterpret_cast<const float4*>(a.norm_w + k));
                        w = make_float4(rs * (a.norm_base + f.x), rs * (a.norm_base + f.y), rs * (a.norm_base + f.z), rs * (a.norm_base + f.w));
                    }
                    float4 n = make_float4(v[i].x * w.x, v[i].y * w.y, v[i].z * w.z, v[i].w * w.w);
                    if constexpr (LOAD == kLoadAddNorm) {
                        const float4 h = __ldcg(reinterpret_cast<const float4*>(xr + k));
                        n = make_float4(h.x + n.x, h.y + n.y, h.z + n.z, h.w + n.w);
                        if (blockIdx.x == m % gridDim.x) *reinterpret_cast<float4*>(a.x_out + (size_t)m * a.K + k) = n;
                    }
                    *reinterpret_cast<uint2*>(dst + 2 * k) = make_uint2(pack2<T>(n.x, n.y), pack2<T>(n.z, n.w));
                }
            }
        }
    }
    __syncthreads();

    // ---- products --------------------------------------------------------------------------------------------------------
    const int groups = a.tiles > 4 ? 2 : 1, splits = kRowsWarps / groups, split = warp % splits, tile0 = (warp / splits) * 4;
    const int chunks = a.K / 32, per = max(MT, (chunks + splits - 1) / splits), c0 = split * per, c1 = min(c0 + per, chunks);
    const int active = (chunks + per - 1) / per;
    const bool high = a.M > 8;
    unsigned long long best = pack_max(-INFINITY, 0);      // a row without a number above -inf gives token 0
    int buf = 0;
    uint32_t parity = 0;
    for (int batch = blockIdx.x; batch < batches; batch += gridDim.x) {
        if (!mbar_wait(bar0 + 8u * buf, parity, abort_flag)) break;
        unsigned char* sw = smem + buf * slab;
        float acc[4][MT][4] = {};
        const unsigned char* xp = sx + r * pitch + c * 16;
        const unsigned char* wp = sw + (8 * tile0 + r) * pitch + c * 16;
#pragma unroll(MT == 1 ? 2 : 1)
        for (int ch = c0; ch < c1; ++ch) {
            uint4 lo[MT], hi[MT];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                lo[mt] = *reinterpret_cast<const uint4*>(xp + 16 * mt * pitch + ch * 64);
                hi[mt] = make_uint4(0u, 0u, 0u, 0u);
                if (high) hi[mt] = *reinterpret_cast<const uint4*>(xp + (16 * mt + 8) * pitch + ch * 64);
            }
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (tile0 + t < a.tiles) {
                    const uint4 b = *reinterpret_cast<const uint4*>(wp + 8 * t * pitch + ch * 64);
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        mma_rows<T>(acc[t][mt], lo[mt].x, hi[mt].x, lo[mt].y, hi[mt].y, b.x, b.y);
                        mma_rows<T>(acc[t][mt], lo[mt].z, hi[mt].z, lo[mt].w, hi[mt].w, b.z, b.w);
                    }
                }
        }
        __syncwarp();                            // every lane has read the slice: it may be overwritten
        if (c0 < chunks) {
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (tile0 + t < a.tiles) store_part<MT>(sw + 8 * (tile0 + t) * pitch + c0 * 64, pitch, r, c, acc[t]);
        }
        __syncthreads();
        auto total = [&](int t, int m, int n) {
            const unsigned char* p = sw + 8 * t * pitch + part_at(m, pitch) + 4 * n;
            float v = 0.f;
#pragma unroll 8
            for (int w = 0; w < active; ++w) v += *reinterpret_cast<const float*>(p + w * per * 64);
            return v;
        };
        const int n8 = tid & 7, em = (tid >> 3) % kRows;
        if (em < a.M) {
            if constexpr (kGated) {
                for (int p = tid / (8 * kRows); p < a.tiles / 2; p += kRowsThreads / (8 * kRows)) {
                    const int ch = batch * (batch_rows / 2) + 8 * p + n8;
                    if (2 * ch >= a.N) break;
                    const float g = total(2 * p, em, n8), u = total(2 * p + 1, em, n8);
                    static_cast<YT*>(a.y)[(size_t)em * a.ldy + ch] = to_out<YT>(rows_act<T, EPI>(g) * u);
                }
            } else {
                for (int t = tid / (8 * kRows); t < a.tiles; t += kRowsThreads / (8 * kRows)) {
                    const int n = batch * batch_rows + 8 * t + n8;
                    if (n >= a.N) break;
                    float v = total(t, em, n8);
                    if (a.scale != 1.0f) v *= a.scale;
                    if (a.cap > 0.f) v = a.cap * tanhf(v / a.cap);
                    if constexpr (EPI == kRowsStore) static_cast<YT*>(a.y)[(size_t)em * a.ldy + n] = to_out<YT>(v);
                    else if (v > -INFINITY) best = max(best, pack_max(v, n));
                }
            }
        }
        if (batch + (int)gridDim.x < batches) {
            fence_proxy_async_smem();            // the slab was read and written by ordinary accesses, the next copy into it is not one
            __syncthreads();
            if (warp == 0 && next < batches) { fetch(next, buf); next += gridDim.x; }
        }
        if (++buf == a.buffers) { buf = 0; parity ^= 1u; }
    }
    if constexpr (EPI == kRowsArgmax) {
        const int em = (tid >> 3) % kRows;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
        if ((tid & 7) == 0 && em < a.M) atomicMax(a.packed + em, best);
    }
    if (stamp) {
        __syncthreads();
        stamp_end(stamp);
    }
    if (tid == 0 && *abort_flag && a.error) atomicExch(a.error, 7);
}

// Few columns, deep K <= 4096: fp32 Y[M, N] = X W^T, added to what is there with ADD.  One column tile per CTA, the 16 warps split K, X goes from L2 straight into the
// registers of the warp that multiplies it, kAhead chunks at a time.
template <typename T, int MT, bool ADD>
__global__ void __launch_bounds__(kRowsThreads, 2)
rows_deep_kernel(const RowsGemm a, unsigned long long* stamp) {
    constexpr int kRows = 16 * MT, kAhead = MT == 1 ? 4 : 2;
    extern __shared__ __align__(128) unsigned char smem[];
    const int pitch = rows_pitch(a.K);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 8 * pitch);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    const int n0 = blockIdx.x * 8, n = n0 + (tid & 7), em = (tid >> 3) % kRows;
    if (warp == 0) {
        if (lane == 0) {
            mbar_init(smem_u32(bar), 1);
            *abort_flag = 0;
            mbar_fence_init();
            mbar_arrive_expect_tx(smem_u32(bar), (uint32_t)(min(8, a.N - n0) * a.K * 2));
        }
        __syncwarp();
        if (lane < 8 && n0 + lane < a.N)
            bulk_g2s(smem_u32(smem) + lane * pitch, static_cast<const T*>(a.w) + (size_t)(n0 + lane) * a.K, (uint32_t)a.K * 2, smem_u32(bar));
    }
    pdl_launch_dependents();                     // see rows_wide_kernel
    pdl_wait();
    stamp_begin(stamp);
    const int chunks = a.K / 32, per = max(MT, (chunks + kRowsWarps - 1) / kRowsWarps), c0 = warp * per, c1 = min(c0 + per, chunks);
    const int active = (chunks + per - 1) / per;
    const bool writes = tid < 8 * kRows && em < a.M && n < a.N;
    float res = 0.f;
    if (ADD && writes) res = __ldcg(static_cast<const float*>(a.y) + (size_t)em * a.ldy + n);
    const T* xp = static_cast<const T*>(a.x) + (size_t)r * a.ldx + 8 * c;
    auto load = [&](int i, int ch) {             // rows 8 i + r, chunk ch
        return 8 * i + r < a.M && ch < c1 ? __ldcg(reinterpret_cast<const uint4*>(xp + (size_t)8 * i * a.ldx + 32 * ch)) : make_uint4(0u, 0u, 0u, 0u);
    };
    uint4 x[kAhead][2 * MT];
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
#pragma unroll
        for (int i = 0; i < 2 * MT; ++i) x[j][i] = load(i, c0 + j);
    __syncthreads();                             // the barrier is initialised
    bool ok = mbar_wait(smem_u32(bar), 0, abort_flag);
    float acc[2][MT][4] = {};                    // two chains
    const unsigned char* wp = smem + r * pitch + c * 16;
#pragma unroll 1
    for (int g = c0; g < c1; g += kAhead) {
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            if (g + j < c1) {
                const uint4 b = *reinterpret_cast<const uint4*>(wp + (g + j) * 64);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    const uint4 lo = x[j][2 * mt], hi = x[j][2 * mt + 1];
                    mma_rows<T>(acc[0][mt], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
                    mma_rows<T>(acc[1][mt], lo.z, hi.z, lo.w, hi.w, b.z, b.w);
                }
#pragma unroll
                for (int i = 0; i < 2 * MT; ++i) x[j][i] = load(i, g + j + kAhead);
            }
        }
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[0][mt][i] += acc[1][mt][i];
    __syncwarp();
    if (c0 < chunks) store_part<MT>(smem + c0 * 64, pitch, r, c, acc[0]);
    __syncthreads();
    if (writes && ok) {
        const unsigned char* p = smem + part_at(em, pitch) + 4 * (tid & 7);
        float v = 0.f;
#pragma unroll 8
        for (int w = 0; w < active; ++w) v += *reinterpret_cast<const float*>(p + w * per * 64);
        static_cast<float*>(a.y)[(size_t)em * a.ldy + n] = res + v;
    }
    if (stamp) {
        __syncthreads();
        stamp_end(stamp);
    }
    if (tid == 0 && *abort_flag && a.error) atomicExch(a.error, 7);
}

int host_pitch(int k) { return (k * 2 + 127) / 128 * 128 + 64; }

// Most shared memory of a launch: what a layer's launches need side by side (152 and 33 KB, 169 and 59 KB), and what a ring may take.
constexpr int kSharedMost = 172 * 1024;

template <typename K>
int prepare(PerDeviceOnce& once, K kernel) {
    B2_PER_DEVICE_ONCE(once, B2_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedMost)));
    return 0;
}

template <typename T, int MT, int LOAD, int EPI, typename YT>
int launch_wide(RowsGemm a, cudaStream_t s, ProfKind kind) {
    static PerDeviceOnce once;
    B2_TRY(prepare(once, rows_wide_kernel<T, MT, LOAD, EPI, YT>));
    int sms = 0;
    B2_TRY(device_sm_count(&sms));
    const int unit = EPI == kRowsSwiglu || EPI == kRowsGeglu ? 2 : 1, n_tiles = ceil_div(a.N, 8), tile = 8 * host_pitch(a.K);
    const int room = kSharedMost - 16 * MT * host_pitch(a.K) - 128;
    a.tiles = ceil_div(ceil_div(n_tiles, unit), sms) * unit;      // one batch per CTA, one CTA per SM ...
    a.buffers = 1;
    if (a.tiles > 8 || a.tiles * tile > room) {                   // ... or, for more columns than a wave holds, batches of four tiles through a ring
        a.tiles = 4;
        a.buffers = std::min(4, room / (4 * tile));
    }
    const int grid = std::min(sms, ceil_div(n_tiles, a.tiles));
    const size_t smem = (size_t)a.buffers * a.tiles * tile + 16 * MT * host_pitch(a.K) + 8 * a.buffers + 16;
    unsigned long long* stamp = prof_stamp_slot(kind);
    launch_pdl_split(true, true, rows_wide_kernel<T, MT, LOAD, EPI, YT>, dim3(grid), dim3(kRowsThreads), smem, s, a, stamp);
    B2_LAUNCH_CHECK();
    return 0;
}

template <typename T, int MT, bool ADD>
int launch_deep(const RowsGemm& a, cudaStream_t s) {
    static PerDeviceOnce once;
    B2_TRY(prepare(once, rows_deep_kernel<T, MT, ADD>));
    unsigned long long* stamp = prof_stamp_slot(PROF_GEMM_RES);
    launch_pdl_split(true, true, rows_deep_kernel<T, MT, ADD>, dim3(ceil_div(a.N, 8)), dim3(kRowsThreads), (size_t)8 * host_pitch(a.K) + 16, s, a, stamp);
    B2_LAUNCH_CHECK();
    return 0;
}

template <typename T, int LOAD, int EPI, typename YT>
int wide(const RowsGemm& a, cudaStream_t s, ProfKind kind) {
    return a.M <= 16 ? launch_wide<T, 1, LOAD, EPI, YT>(a, s, kind) : launch_wide<T, 2, LOAD, EPI, YT>(a, s, kind);
}
template <typename T, bool ADD>
int deep(const RowsGemm& a, cudaStream_t s) {
    return a.M <= 16 ? launch_deep<T, 1, ADD>(a, s) : launch_deep<T, 2, ADD>(a, s);
}

}  // namespace

bool gemm_rows_takes(const RowsGemm& a, int epi) {
    const bool deep = epi == kRowsResidual || epi == kRowsDeepStore;
    return a.M > 0 && a.M <= kRowsGemmMax && a.N > 0 && a.K > 0 && a.K % 32 == 0 && a.K <= (deep ? 4096 : 1024) && a.ldx % 8 == 0 &&
           (reinterpret_cast<uintptr_t>(a.x) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.w) & 15) == 0;
}

int gemm_rows(cudaStream_t s, const RowsGemm& a, ElemType type, int epi, bool norm, ElemType out) {
    if (!gemm_rows_takes(a, epi)) B2_FAIL(B200ATTN_ERR_UNSUPPORTED, "gemm_rows: unsupported shape %d x %d x %d", a.M, a.N, a.K);
    using B = __nv_bfloat16;
    if (type == ELEM_F16) {
        if (epi == kRowsStore && out == ELEM_F32)
            return norm ? wide<__half, kLoadNorm, kRowsStore, float>(a, s, PROF_GEMM_IN) : wide<__half, kLoadAsIs, kRowsStore, float>(a, s, PROF_GEMM_IN);
        if (epi == kRowsSwiglu && out == ELEM_F16 && norm) return wide<__half, kLoadNorm, kRowsSwiglu, __half>(a, s, PROF_GEMM_FFN);
        if (epi == kRowsResidual) return deep<__half, true>(a, s);
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
        if (epi == kRowsResidual) return deep<B, true>(a, s);
        if (epi == kRowsDeepStore) return deep<B, false>(a, s);
    }
    B2_FAIL(B200ATTN_ERR_UNSUPPORTED, "gemm_rows: unsupported types");
}

}  // namespace b200
