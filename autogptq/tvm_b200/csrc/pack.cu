// Packing of integer fields into GPTQ int32 words on the GPU (load-time path, HBM-bound).
//
//   vals  int32 [R, C]  (R a multiple of 32): one field per element, packed along R
//   out   int32 [R / 32 * bits, C]
//
// 2/4/8 bits: field j of a word sits at bit bits*j.  3 bits: the 32 fields of a row block form one
// 96-bit little-endian stream over three words.  Values wider than `bits` are NOT masked: they spill
// into the neighbouring fields exactly as the reference's un-masked `|=` does
// (auto_gptq/nn_modules/qlinear.py:111-134 for qweight, :140-170 for qzeros), with the arithmetic done
// on the value as an unsigned 32-bit number, as numpy does there.
//
// One thread packs one row block of one column: its 32 reads are strided by C, so the threads of a warp
// (consecutive columns) read and write consecutive addresses.
#include <cuda_bf16.h>

#include <mutex>

#include "common.cuh"

namespace b200gptq {

namespace {

template <int BITS>
__global__ void __launch_bounds__(256)
pack_fields_kernel(const int32_t* __restrict__ vals, int R, int C, int32_t* __restrict__ out) {
    const int c = blockIdx.x * 32 + threadIdx.x;
    const int rb = blockIdx.y * blockDim.y + threadIdx.y;
    if (c >= C || rb * kRowsPerBlock >= R) return;
    const int32_t* src = vals + (size_t)rb * kRowsPerBlock * C + c;
    uint32_t w[BITS];
#pragma unroll
    for (int i = 0; i < BITS; ++i) w[i] = 0u;
#pragma unroll
    for (int j = 0; j < kRowsPerBlock; ++j) {
        const uint32_t v = (uint32_t)src[(size_t)j * C];
        if constexpr (BITS == 3) {
            const int bit = 3 * j, wi = bit >> 5, sh = bit & 31;
            w[wi] |= v << sh;
            if (sh > 29) w[wi + 1] |= (v >> (32 - sh)) & ((1u << (sh + 3 - 32)) - 1u);
        } else {
            constexpr int PF = 32 / BITS;
            w[j / PF] |= v << (BITS * (j % PF));
        }
    }
    int32_t* dst = out + (size_t)rb * BITS * C + c;
#pragma unroll
    for (int i = 0; i < BITS; ++i) dst[(size_t)i * C] = (int32_t)w[i];
}

template <int BITS>
int launch_pack(const int32_t* vals, int R, int C, int32_t* out, cudaStream_t stream) {
    dim3 block(32, 8);
    dim3 grid((C + 31) / 32, (R / kRowsPerBlock + 7) / 8);
    pack_fields_kernel<BITS><<<grid, block, 0, stream>>>(vals, R, C, out);
    B200GPTQ_CUDA_TRY(cudaGetLastError());
    return B200GPTQ_OK;
}

// ---- whole QuantLinear.pack in one launch ------------------------------------------------------------------------
// weight [N, K] (fp16 / bf16 / fp32), scales and zeros fp32 [N, G], g_idx int32 [K]  ->
//   qweight int32 [K/32*bits, N]    field = round((w + zero * scale) / float(fp16(scale))), all in fp32
//   qzeros  int32 [G, N/32*bits]    zero - 1
//   scales  fp16  [G, N]
// (auto_gptq/nn_modules/qlinear.py:77-175 of the reference, which loops over the rows on the CPU).
//
// As a chain of framework kernels this was eleven launches with five fp32 [K, N] intermediates: 1.0 ms for
// 4096 x 11008; the bound is one read of the weight and one write of the words, 17 us there.  A CTA takes 32 output
// columns (rows of `weight`) and a part of K: 256 k of every row are loaded with coalesced 16-byte reads into shared
// memory, a thread then owns one column and one 32-row block (128-bit reads, rows 16 bytes apart in banks) and writes
// its words, 128 bytes per warp and word-row.  (zero * scale, 1 / scale) of the 32 columns x all groups sit in shared
// memory, column fastest, so that a look-up by any g_idx is one conflict-free 8-byte read.
//
// An IEEE division per element would be most of the arithmetic.  t = a * (1 / s) is within |t| * 2^-22 of the rounded
// quotient (two roundings of 2^-24 and the quotient's own), so rounding t gives the same integer unless t lies that
// close to a half; a 32-row block with such an element (or with a NaN, an infinity, |t| >= 2^20) is redone with the
// division.  Quantised weights are integer multiples of the scale up to rounding, so that is rare.
constexpr int kPackCols = 32, kPackChunk = 256, kPackThreads = 256;
constexpr int kPackTableMax = 128 * 1024;     // bytes of the table; more groups are read from global memory

template <typename T> struct PackIn;
template <> struct PackIn<__half> { __device__ static float get(__half v) { return __half2float(v); } };
template <> struct PackIn<__nv_bfloat16> { __device__ static float get(__nv_bfloat16 v) { return __bfloat162float(v); } };
template <> struct PackIn<float> { __device__ static float get(float v) { return v; } };

template <int BITS>
__device__ __forceinline__ void pack_insert(uint32_t (&w)[BITS], int j, uint32_t v) {   // unmasked, as pack_fields
    if constexpr (BITS == 3) {
        const int bit = 3 * j, wi = bit >> 5, sh = bit & 31;
        w[wi] |= v << sh;
        if (sh > 29) w[wi + 1] |= (v >> (32 - sh)) & ((1u << (sh + 3 - 32)) - 1u);
    } else {
        constexpr int PF = 32 / BITS;
        w[j / PF] |= v << (BITS * (j % PF));
    }
}

template <int BITS, typename T>
__global__ void __launch_bounds__(kPackThreads)
pack_linear_kernel(const T* __restrict__ weight, const float* __restrict__ scales, const float* __restrict__ zeros,
                   const int32_t* __restrict__ g_idx, int K, int N, int G, int chunks_per_cta, int use_table,
                   int32_t* __restrict__ qweight, int32_t* __restrict__ qzeros, __half* __restrict__ scales_out) {
    constexpr int VEC = 16 / (int)sizeof(T);                       // elements of one 16-byte read
    constexpr int PITCH = kPackChunk + VEC;                        // elements of a tile row: 16 bytes of padding
    extern __shared__ __align__(16) unsigned char pack_smem[];
    T* tile = reinterpret_cast<T*>(pack_smem);                     // [32][PITCH]
    int* gs = reinterpret_cast<int*>(pack_smem + sizeof(T) * kPackCols * PITCH);   // groups of the chunk's rows
    float2* table = reinterpret_cast<float2*>(gs + kPackChunk);    // [G][32] (zero * scale, 1 / scale)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * kPackCols, n = n0 + lane;
    auto entry = [&](int g, float& s) {
        const float sf = scales[(size_t)n * G + g];
        s = __half2float(__float2half_rn(sf));
        return make_float2(__fmul_rn(zeros[(size_t)n * G + g], sf), __frcp_rn(s));
    };
    if (use_table)
        for (int g = warp; g < G; g += kPackThreads / 32) { float s; table[g * kPackCols + lane] = entry(g, s); }
    if (blockIdx.y == 0) {
        for (int g = warp; g < G; g += kPackThreads / 32)
            scales_out[(size_t)g * N + n] = __float2half_rn(scales[(size_t)n * G + g]);
        for (int g = threadIdx.x; g < G; g += kPackThreads) {
            uint32_t w[BITS];
#pragma unroll
            for (int i = 0; i < BITS; ++i) w[i] = 0u;
#pragma unroll
            for (int j = 0; j < 32; ++j)
                pack_insert<BITS>(w, j, (uint32_t)(long long)(zeros[(size_t)(n0 + j) * G + g] - 1.f));
#pragma unroll
            for (int i = 0; i < BITS; ++i) qzeros[(size_t)g * (N / 32 * BITS) + blockIdx.x * BITS + i] = (int32_t)w[i];
        }
    }
    const int c_end = min((K + kPackChunk - 1) / kPackChunk, (int)(blockIdx.y + 1) * chunks_per_cta);
    for (int c = blockIdx.y * chunks_per_cta; c < c_end; ++c) {
        const int k0 = c * kPackChunk;
        __syncthreads();                                           // the previous chunk has been read (and: the table is there)
#pragma unroll
        for (int i = threadIdx.x; i < kPackCols * kPackChunk / VEC; i += kPackThreads) {
            const int r = i / (kPackChunk / VEC), e = (i % (kPackChunk / VEC)) * VEC;
            if (k0 + e < K)
                *reinterpret_cast<uint4*>(tile + r * PITCH + e) =
                    __ldcs(reinterpret_cast<const uint4*>(weight + (size_t)(n0 + r) * K + k0 + e));
        }
        if (k0 + (int)threadIdx.x < K)      // an index outside the groups is refused by the host when the layer is used
            gs[threadIdx.x] = min(max(__ldg(g_idx + k0 + threadIdx.x), 0), G - 1);
        __syncthreads();
        const int rb = k0 / kRowsPerBlock + warp;
        if (rb * kRowsPerBlock >= K) continue;
        const T* row = tile + lane * PITCH + warp * kRowsPerBlock;
        const int* gr = gs + warp * kRowsPerBlock;
        uint32_t w[BITS];
#pragma unroll
        for (int i = 0; i < BITS; ++i) w[i] = 0u;
        bool close = false;                                        // some quotient is too close to a half, or not finite
#pragma unroll
        for (int j0 = 0; j0 < kRowsPerBlock; j0 += VEC) {
            const uint4 raw = *reinterpret_cast<const uint4*>(row + j0);
            const T* v = reinterpret_cast<const T*>(&raw);
#pragma unroll
            for (int i = 0; i < VEC; ++i) {
                const int g = gr[j0 + i];
                float s;
                const float2 e = use_table ? table[g * kPackCols + lane] : entry(g, s);
                const float t = __fadd_rn(PackIn<T>::get(v[i]), e.x) * e.y;
                const float u = __fadd_rn(t, 12582912.f);          // 1.5 * 2^23: rounds t to an integer, ties to even
                const float d = fabsf(t - __fadd_rn(u, -12582912.f));
                close |= !(d < fmaf(fabsf(t), -4.76837158203125e-7f, 0.5f));   // |t| * 2^-21
                pack_insert<BITS>(w, j0 + i, (uint32_t)(__float_as_int(u) - 0x4B400000));
            }
        }
        if (close) {
#pragma unroll
            for (int i = 0; i < BITS; ++i) w[i] = 0u;
#pragma unroll
            for (int j = 0; j < kRowsPerBlock; ++j) {
                float s;
                const float2 e = entry(gr[j], s);
                pack_insert<BITS>(w, j, (uint32_t)(int)rintf(__fdiv_rn(__fadd_rn(PackIn<T>::get(row[j]), e.x), s)));
            }
        }
#pragma unroll
        for (int i = 0; i < BITS; ++i) qweight[(size_t)(rb * BITS + i) * N + n] = (int32_t)w[i];
    }
}

template <int BITS, typename T>
int launch_pack_linear(const void* weight, const float* scales, const float* zeros, const int32_t* g_idx, int K, int N,
                       int G, int32_t* qweight, int32_t* qzeros, __half* scales_out, cudaStream_t stream) {
    const int chunks = (K + kPackChunk - 1) / kPackChunk, strips = N / kPackCols;
    const long long table = (long long)G * kPackCols * sizeof(float2);
    const int use_table = table <= kPackTableMax;
    const size_t smem = sizeof(T) * kPackCols * (kPackChunk + 16 / sizeof(T)) + kPackChunk * sizeof(int) + (use_table ? table : 0);
    static std::once_flag once[64];
    static int result[64];
    int dev = 0;
    B200GPTQ_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return B200GPTQ_ERR_TOO_LARGE;
    std::call_once(once[dev], [dev] {
        result[dev] = (int)cudaFuncSetAttribute(pack_linear_kernel<BITS, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                200 * 1024);
    });
    if (result[dev] != 0) { set_last_cuda_error(result[dev]); return B200GPTQ_ERR_CUDA; }
    // K is cut until the grid fills the device about four times over: every cut builds the table of its columns again
    int parts = (8 * sm_count() + strips - 1) / strips;
    if (parts > chunks) parts = chunks;
    const int per = (chunks + parts - 1) / parts;
    dim3 grid(strips, (chunks + per - 1) / per);
    pack_linear_kernel<BITS, T><<<grid, kPackThreads, smem, stream>>>(static_cast<const T*>(weight), scales, zeros, g_idx, K, N,
                                                                      G, per, use_table, qweight, qzeros, scales_out);
    B200GPTQ_CUDA_TRY(cudaGetLastError());
    return B200GPTQ_OK;
}

}  // namespace

int pack_linear_dispatch(const void* weight, int dtype, const float* scales, const float* zeros, const int32_t* g_idx,
                         int K, int N, int G, int bits, int32_t* qweight, int32_t* qzeros, __half* scales_out,
                         cudaStream_t stream) {
#define B200GPTQ_PACK(B)                                                                                               \
    (dtype == B200GPTQ_F16    ? launch_pack_linear<B, __half>(weight, scales, zeros, g_idx, K, N, G, qweight, qzeros,  \
                                                              scales_out, stream)                                      \
     : dtype == B200GPTQ_BF16 ? launch_pack_linear<B, __nv_bfloat16>(weight, scales, zeros, g_idx, K, N, G, qweight,   \
                                                                     qzeros, scales_out, stream)                       \
                              : launch_pack_linear<B, float>(weight, scales, zeros, g_idx, K, N, G, qweight, qzeros,   \
                                                             scales_out, stream))
    switch (bits) {
        case 2: return B200GPTQ_PACK(2);
        case 3: return B200GPTQ_PACK(3);
        case 4: return B200GPTQ_PACK(4);
        case 8: return B200GPTQ_PACK(8);
    }
#undef B200GPTQ_PACK
    return B200GPTQ_ERR_BITS;
}

int pack_fields_dispatch(const int32_t* vals, int R, int C, int bits, int32_t* out, cudaStream_t stream) {
    switch (bits) {
        case 2: return launch_pack<2>(vals, R, C, out, stream);
        case 3: return launch_pack<3>(vals, R, C, out, stream);
        case 4: return launch_pack<4>(vals, R, C, out, stream);
        case 8: return launch_pack<8>(vals, R, C, out, stream);
    }
    return B200GPTQ_ERR_BITS;
}

}  // namespace b200gptq
