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
#include <type_traits>

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
// columns (rows of `weight`) and a part of K: 256 k of every row come into shared memory with coalesced 16-byte
// asynchronous copies, the next 256 while these are packed (57 us for 4096 x 11008 when a chunk's copy and its packing
// took turns).  A thread then owns one column and one 32-row block (128-bit reads, rows 16 bytes apart in banks) and
// writes its words, 128 bytes per warp and word-row.  (zero * scale, 1 / scale) of the 32 columns x all groups sit in
// shared memory, column fastest, so that a look-up by any g_idx is one conflict-free 8-byte read; the rows are one entry
// longer than the columns, so that the table is written without conflicts from coalesced reads of [N, G] too.  scales and
// qzeros are left to CTAs of their own.  4096 x 11008, 4 bits, groups of 128 in act-order: 35 us from fp16; in
// order, where a row block is one group and needs no look-ups, 30 us.  fp16 weights of 2 to 4 bits have pack_pairs_kernel (26 and 25 us)
// unless its table is too large; this kernel packs 8 bits, bf16 and fp32.
//
// What remains is the start of a CTA (its table) and the instructions of an element, 20 of them once (25 us at full issue):
// - No IEEE division.  With r = 1 / s rounded, a * r is within a relative 2^-24 of a / s and the rounded quotient within
//   another, so for 0 <= q < 2^bits rounding a * r gives the integer that rounding the quotient gives unless a * r lies within
//   2^bits * 2^-22 of a half.  u = a * r + 1.5 * 2^23 in one fma is that integer in the low bits of a float; d, also one fma,
//   the rest.
// - A field is added to its word as (bits of u) << position, what 1.5 * 2^23 leaves there is a constant of the word.  That
//   takes 0 <= q < 2^bits: the upper bits of all u's or'ed and and'ed are then those of 1.5 * 2^23.  (So a NaN or an
//   infinity is seen too.)
// A 32-row block with an element close to a half or out of range is redone with the division and the unmasked insert.
// Quantised weights are multiples of the scale within the range up to rounding, so that is rare.
constexpr int kPackCols = 32, kPackChunk = 256, kPackThreads = 256, kPackPitch = kPackCols + 1;
constexpr int kPackCtas = 5;                  // per SM: what the registers and two tiles of fp16 allow
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

constexpr float kRound = 12582912.f;           // 1.5 * 2^23: adding it rounds to an integer, ties to even
constexpr uint32_t kRoundBits = 0x4B400000u;   // (its bits)
// What kRound's bits add up to in word i of a block (fields that lie in two words are added without them).
template <int BITS>
__device__ constexpr uint32_t pack_bias(int i) {
    uint32_t c = 0u;
    for (int j = 0; j < kRowsPerBlock; ++j) {
        const int bit = BITS * j, sh = bit & 31;
        if ((bit >> 5) == i && sh + BITS <= 32) c += kRoundBits << sh;
    }
    return c;
}

// A 32-row block with the division.  A call of its own: inlined, its loads in flight took the registers of the usual path.
template <int BITS, typename T>
__device__ __noinline__ void pack_divided(const T* row, const int* gr, const float* scales, const float* zeros, int32_t* out,
                                          int N) {
    uint32_t w[BITS];
#pragma unroll
    for (int i = 0; i < BITS; ++i) w[i] = 0u;
#pragma unroll
    for (int j = 0; j < kRowsPerBlock; ++j) {
        const float sf = scales[gr[j]], s = __half2float(__float2half_rn(sf));
        const float a = __fadd_rn(PackIn<T>::get(row[j]), __fmul_rn(zeros[gr[j]], sf));
        pack_insert<BITS>(w, j, (uint32_t)(int)rintf(__fdiv_rn(a, s)));
    }
#pragma unroll
    for (int i = 0; i < BITS; ++i) out[(size_t)i * N] = (int32_t)w[i];
}

// The group of row k (an index outside the groups is refused by the host when the layer is used).  The CTAs of the first strip, which read
// every row's, leave the copy of g_idx.  (By the few CTAs that write the constants of a narrow layer it was a serial loop: 10720 x 320 7.9 us
// instead of 5.8.)
__device__ __forceinline__ int pack_group(const int32_t* __restrict__ g_idx, int k, int G, int32_t* __restrict__ g_idx_out) {
    const int g = __ldg(g_idx + k);
    if (g_idx_out && blockIdx.x == 0) g_idx_out[k] = g;
    return min(max(g, 0), G - 1);
}

// scales_out and qzeros of one strip of 32 columns.  smem: 2 * 128 * kPackPitch floats
template <int BITS, int THREADS>
__device__ __forceinline__ void pack_constants(const float* __restrict__ scales, const float* __restrict__ zeros, int G, int N, int strip,
                                               int32_t* __restrict__ qzeros, __half* __restrict__ scales_out, unsigned char* smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n0 = strip * kPackCols, n = n0 + lane;
    // scales and zero-points of the strip, 128 groups at a time: read along the groups, written along the columns
    constexpr int GT = 128;
    float* st = reinterpret_cast<float*>(smem);
    float* zt = st + GT * kPackPitch;
    for (int g0 = 0; g0 < G; g0 += GT) {
        const int count = min(GT, G - g0);
        for (int g = lane; g < count; g += 32)
#pragma unroll
            for (int r = 0; r < kPackCols; r += THREADS / 32) {
                const size_t at = (size_t)(n0 + r + warp) * G + g0 + g;
                st[g * kPackPitch + r + warp] = scales[at];
                zt[g * kPackPitch + r + warp] = zeros[at];
            }
        __syncthreads();
        for (int g = warp; g < count; g += THREADS / 32)
            scales_out[(size_t)(g0 + g) * N + n] = __float2half_rn(st[g * kPackPitch + lane]);
        for (int g = threadIdx.x; g < count; g += THREADS) {
            uint32_t w[BITS];
#pragma unroll
            for (int i = 0; i < BITS; ++i) w[i] = 0u;
#pragma unroll
            for (int j = 0; j < 32; ++j)
                pack_insert<BITS>(w, j, (uint32_t)(long long)(zt[g * kPackPitch + j] - 1.f));
#pragma unroll
            for (int i = 0; i < BITS; ++i)
                qzeros[(size_t)(g0 + g) * (N / 32 * BITS) + strip * BITS + i] = (int32_t)w[i];
        }
        __syncthreads();
    }
}

template <int BITS, typename T>
__global__ void __launch_bounds__(kPackThreads, kPackCtas)
pack_linear_kernel(const T* __restrict__ weight, const float* __restrict__ scales, const float* __restrict__ zeros,
                   const int32_t* __restrict__ g_idx, int K, int N, int G, int chunks_per_cta, int use_table,
                   int32_t* __restrict__ qweight, int32_t* __restrict__ qzeros, __half* __restrict__ scales_out, int32_t* __restrict__ g_idx_out) {
    constexpr int VEC = 16 / (int)sizeof(T);                       // elements of one 16-byte read
    constexpr int PITCH = kPackChunk + VEC;                        // elements of a tile row: 16 bytes of padding
    constexpr int TILE = kPackCols * PITCH;
    extern __shared__ __align__(16) unsigned char pack_smem[];
    T* tiles = reinterpret_cast<T*>(pack_smem);                    // two of [32][PITCH]
    int* groups = reinterpret_cast<int*>(pack_smem + 2 * sizeof(T) * TILE);        // two of: groups of the chunk's rows
    float2* table = reinterpret_cast<float2*>(groups + 2 * kPackChunk);            // [G][33] (zero * scale, 1 / scale)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * kPackCols, n = n0 + lane;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int c_begin = blockIdx.y * chunks_per_cta, c_end = min((K + kPackChunk - 1) / kPackChunk, c_begin + chunks_per_cta);
    auto fetch = [&](int c, int buf) {
        const int k0 = c * kPackChunk;
#pragma unroll
        for (int i = threadIdx.x; i < kPackCols * kPackChunk / VEC; i += kPackThreads) {
            const int r = i / (kPackChunk / VEC), e = (i % (kPackChunk / VEC)) * VEC;
            if (k0 + e < K)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                             ::"r"((uint32_t)__cvta_generic_to_shared(tiles + buf * TILE + r * PITCH + e)), "l"(weight + (size_t)(n0 + r) * K + k0 + e)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto group_of = [&](int c) {
        const int k = c * kPackChunk + threadIdx.x;
        return k < K ? pack_group(g_idx, k, G, g_idx_out) : 0;
    };
    if (blockIdx.y == gridDim.y - 1) {
        pack_constants<BITS, kPackThreads>(scales, zeros, G, N, blockIdx.x, qzeros, scales_out, pack_smem);
        return;
    }
    fetch(c_begin, 0);
    int g_next = group_of(c_begin);
    auto entry = [&](size_t at) {                                  // at: [N, G]
        const float sf = scales[at];
        return make_float2(__fmul_rn(zeros[at], sf), __frcp_rn(__half2float(__float2half_rn(sf))));
    };
    if (use_table)
        for (int g = lane; g < G; g += 32)
#pragma unroll
            for (int r = 0; r < kPackCols; r += kPackThreads / 32)
                table[g * kPackPitch + r + warp] = entry((size_t)(n0 + r + warp) * G + g);
    for (int c = c_begin; c < c_end; ++c) {
        const int buf = (c - c_begin) & 1;
        groups[buf * kPackChunk + threadIdx.x] = g_next;
        if (c + 1 < c_end) {                                       // (the barrier that ended the last turn freed its buffers)
            fetch(c + 1, buf ^ 1);
            g_next = group_of(c + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const int rb = c * (kPackChunk / kRowsPerBlock) + warp;
        if (rb * kRowsPerBlock < K) {
            const T* row = tiles + buf * TILE + lane * PITCH + warp * kRowsPerBlock;
            const int* gr = groups + buf * kPackChunk + warp * kRowsPerBlock;
            uint32_t w[BITS];
            float far = 0.f;                                       // largest distance from an integer
            uint32_t any = 0u, all = ~0u;
            auto block = [&](auto look_up) {
#pragma unroll
                for (int i = 0; i < BITS; ++i) w[i] = 0u - pack_bias<BITS>(i);
#pragma unroll
                for (int j0 = 0; j0 < kRowsPerBlock; j0 += VEC) {
                    const uint4 raw = *reinterpret_cast<const uint4*>(row + j0);
                    const T* v = reinterpret_cast<const T*>(&raw);
#pragma unroll
                    for (int i = 0; i < VEC; i += 2) {
                        uint32_t ub[2];
                        float d[2];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float2 e = look_up(j0 + i + h);
                            const float a = __fadd_rn(PackIn<T>::get(v[i + h]), e.x), u = fmaf(a, e.y, kRound);
                            d[h] = fmaf(a, e.y, -__fadd_rn(u, -kRound));
                            ub[h] = __float_as_uint(u);
                            const int bit = BITS * (j0 + i + h), wi = bit >> 5, sh = bit & 31;
                            if (sh + BITS <= 32) {
                                w[wi] += ub[h] << sh;
                            } else {
                                w[wi] += (ub[h] - kRoundBits) << sh;
                                w[wi + 1] += (ub[h] - kRoundBits) >> (32 - sh);
                            }
                        }
                        far = fmaxf(far, fmaxf(fabsf(d[0]), fabsf(d[1])));
                        any |= ub[0] | ub[1];
                        all &= ub[0] & ub[1];
                    }
                }
            };
            const int g_lane = gr[lane], g_first = __shfl_sync(0xffffffffu, g_lane, 0);
            if (__all_sync(0xffffffffu, g_lane == g_first)) {      // rows in order, groups of whole blocks
                const float2 e = use_table ? table[g_first * kPackPitch + lane] : entry((size_t)n * G + g_first);
                block([&](int) { return e; });
            } else if (use_table) {
                block([&](int j) { return table[gr[j] * kPackPitch + lane]; });
            } else {
                block([&](int j) { return entry((size_t)n * G + gr[j]); });
            }
            const bool redo = far > 0.5f - (1 << BITS) * 4.76837158203125e-7f || (any >> BITS) != (kRoundBits >> BITS) ||
                              (all >> BITS) != (kRoundBits >> BITS);                     // (2^bits * 2^-21)
            int32_t* out = qweight + (size_t)rb * BITS * N + n;
            if (redo) {
                pack_divided<BITS, T>(row, gr, scales + (size_t)n * G, zeros + (size_t)n * G, out, N);
            } else {
#pragma unroll
                for (int i = 0; i < BITS; ++i) out[(size_t)i * N] = (int32_t)w[i];
            }
        }
        __syncthreads();
    }
}

// fp16 weights, 2 to 4 bits: two columns at a time in fp16.  t = w / s + z' with 1 / s and z' = zero * scale / s rounded to fp16, u = t + 1.5 *
// 2^10 the integer in the low bits of a half, d = t - (u - 1.5 * 2^10).  For an integer in the range of the fields and |z'| <= 32 (a table
// entry beyond that, or with 1 / s out of the normal numbers, is NaN) t is within 2^-11 (|w / s| + |z'|) + 2^-8 < 0.05 of the quotient,
// |w / s| being less than 16 + |z'|; so where |d| <= 0.4375 the quotient is within 0.49 of that integer, and fp32 rounds it to the same.
// Everything else (a half nearby, out of range, NaN, infinity) is redone with the division, and so is column c + 16 where column c is out of range.
//
// A thread takes columns c and c + 16 of a 32-row block, a half-warp a block: both columns' rows lie in one group, so that (1 / s, z') of
// both are one 8-byte look-up, and fields pile up in the two halves of a register.  (A column per thread, in fp32 17 instructions per
// element, in fp16 with two rows at a time 16.)  Two chunks are on their way from the start, while the table is made.  us, fp32 -> here:
// 4096 x 11008, 4 bits, groups of 128 in act-order 35.1 -> 26.0, in order 29.7 -> 24.7 (its bytes at the copy rate: 17.8, the start of the
// CTAs 4); 11008 x 4096, groups of 32 in act-order 106 -> 45.7 (344 groups: the table counts); 4096 x 4096, one group 13.8 -> 11.3; 2 bits, groups
// of 64 17.8 -> 13.1; 1024 x 1024 3.7 -> 2.8.  Chunks of 512 rows (1 KB of a row) instead of 256: 29.3; of 128: 37.9.
constexpr int kPairThreads = 128, kPairChunk = 2 * kPairThreads, kPairCtas = 6;
constexpr int kPairPitch = 17;                         // pairs of columns in a row of the table
constexpr uint32_t kHalfRound2 = 0x66006600u;          // 1.5 * 2^10 twice
constexpr uint32_t kHalfFar = 0x3700u;                 // 0.4375

template <int BITS>
__global__ void __launch_bounds__(kPairThreads, kPairCtas)
pack_pairs_kernel(const __half* __restrict__ weight, const float* __restrict__ scales, const float* __restrict__ zeros,
                  const int32_t* __restrict__ g_idx, int K, int N, int G, int chunks_per_cta, int32_t* __restrict__ qweight,
                  int32_t* __restrict__ qzeros, __half* __restrict__ scales_out, int32_t* __restrict__ g_idx_out) {
    constexpr int PITCH = kPairChunk + 8, TILE = kPackCols * PITCH;
    extern __shared__ __align__(16) unsigned char pack_smem[];
    __half* tiles = reinterpret_cast<__half*>(pack_smem);          // two of [32][PITCH]
    int* groups = reinterpret_cast<int*>(pack_smem + 2 * sizeof(__half) * TILE);   // two of: groups of the chunk's rows
    uint2* table = reinterpret_cast<uint2*>(groups + 2 * kPairChunk);              // [G][17]: 1 / s of both columns, z' of both
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n0 = blockIdx.x * kPackCols;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.y == gridDim.y - 1) {
        pack_constants<BITS, kPairThreads>(scales, zeros, G, N, blockIdx.x, qzeros, scales_out, pack_smem);
        return;
    }
    const int c_begin = blockIdx.y * chunks_per_cta, c_end = min((K + kPairChunk - 1) / kPairChunk, c_begin + chunks_per_cta);
    auto fetch = [&](int c, int buf) {
        // (whole rows of the tile by as many threads as they have pieces)
        constexpr int PIECES = kPairChunk / 8, STEP = kPairThreads / PIECES;
        const int k = c * kPairChunk + 8 * (threadIdx.x % PIECES), r0 = threadIdx.x / PIECES;
        if (k < K) {
            const __half* src = weight + (size_t)(n0 + r0) * K + k;
            uint32_t dst = (uint32_t)__cvta_generic_to_shared(tiles + buf * TILE + r0 * PITCH + 8 * (threadIdx.x % PIECES));
#pragma unroll
            for (int r = 0; r < kPackCols; r += STEP) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
                src += (size_t)STEP * K;
                dst += STEP * PITCH * 2;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto group_of = [&](int c, int i) {
        const int k = c * kPairChunk + threadIdx.x + i * kPairThreads;
        return k < K ? pack_group(g_idx, k, G, g_idx_out) : 0;
    };
    fetch(c_begin, 0);
    if (c_begin + 1 < c_end) fetch(c_begin + 1, 1);
    int g_next[2] = {group_of(c_begin, 0), group_of(c_begin, 1)};
    auto entry = [&](size_t at) -> uint32_t {                      // (1 / s, z')
        const float sf = scales[at];
        float r;
        asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(__half2float(__float2half_rn(sf))));
        const float z = zeros[at] * sf * r;
        if (!(fabsf(z) <= 32.f && fabsf(r) >= 0.0001220703125f && fabsf(r) <= 32768.f)) return 0x7fff7fffu;
        const __half2 h = __floats2half2_rn(r, z);
        return *reinterpret_cast<const uint32_t*>(&h);
    };
    for (int g = lane; g < G; g += 32)
#pragma unroll
        for (int r = 0; r < 16; r += kPairThreads / 32) {
            const uint32_t a = entry((size_t)(n0 + r + warp) * G + g), b = entry((size_t)(n0 + r + warp + 16) * G + g);
            table[g * kPairPitch + r + warp] = make_uint2(__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632));
        }
    auto as_h2 = [](uint32_t v) { return *reinterpret_cast<const __half2*>(&v); };
    auto as_u = [](__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); };
    const int col = lane & 15, block = 2 * warp + (lane >> 4);
    for (int c = c_begin; c < c_end; ++c) {
        const int buf = (c - c_begin) & 1;
#pragma unroll
        for (int i = 0; i < 2; ++i) groups[buf * kPairChunk + threadIdx.x + i * kPairThreads] = g_next[i];
        if (c + 1 < c_end) {
#pragma unroll
            for (int i = 0; i < 2; ++i) g_next[i] = group_of(c + 1, i);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const int rb = c * (kPairChunk / kRowsPerBlock) + block;
        const int* gr = groups + buf * kPairChunk + block * kRowsPerBlock;
        const int g_first = gr[0];
        const bool one_group = __all_sync(0xffffffffu, gr[col] == g_first && gr[col + 16] == g_first);   // rows in order, groups of whole blocks
        if (rb * kRowsPerBlock < K) {
            const __half* row = tiles + buf * TILE + col * PITCH + block * kRowsPerBlock;
            constexpr int PER = BITS == 4 ? 4 : (BITS == 2 ? 8 : 5), SUMS = (32 + PER - 1) / PER;        // fields of a half
            uint32_t sum[SUMS], any = 0u, far = 0u;                // all integers or'ed; largest distances from one
            const uint2* at = table + col;
            auto rows = [&](auto look_up) {
#pragma unroll
                for (int j0 = 0; j0 < kRowsPerBlock; j0 += 8) {
                    const uint4 a = *reinterpret_cast<const uint4*>(row + j0), b = *reinterpret_cast<const uint4*>(row + 16 * PITCH + j0);
                    const uint32_t pa[4] = {a.x, a.y, a.z, a.w}, pb[4] = {b.x, b.y, b.z, b.w};
                    uint2 e[8];
                    look_up(j0, e);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int j = j0 + i;
                        const __half2 x = as_h2(__byte_perm(pa[i >> 1], pb[i >> 1], i & 1 ? 0x7632 : 0x5410));
                        const __half2 t = __hfma2(x, as_h2(e[i].x), as_h2(e[i].y)), u = __hadd2(t, as_h2(kHalfRound2));
                        far = as_u(__hmax2(as_h2(far), __habs2(__hsub2(t, __hsub2(u, as_h2(kHalfRound2))))));
                        const uint32_t q = as_u(u) ^ kHalfRound2;
                        any |= q;
                        sum[j / PER] = j % PER == 0 ? q : sum[j / PER] + (q << (BITS * (j % PER)));
                    }
                }
            };
            if (one_group) {
                const uint2 one = at[g_first * kPairPitch];
                rows([&](int, uint2 (&e)[8]) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) e[i] = one;
                });
            } else {
                rows([&](int j0, uint2 (&e)[8]) {
                    const int4 lo = *reinterpret_cast<const int4*>(gr + j0), hi = *reinterpret_cast<const int4*>(gr + j0 + 4);
                    const int g[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) e[i] = at[g[i] * kPairPitch];
                });
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int n = n0 + col + 16 * h;
                int32_t* out = qweight + (size_t)rb * BITS * N + n;
                // (a field of the lower half that is out of range has been added to the upper half's sums as well)
                const uint32_t beyond = (h ? (any >> 16) | (any & 0xffffu) : any & 0xffffu) >> BITS, most = h ? far >> 16 : far & 0xffffu;
                if (beyond != 0u || most > kHalfFar) {
                    pack_divided<BITS, __half>(row + h * 16 * PITCH, gr, scales + (size_t)n * G, zeros + (size_t)n * G, out, N);
                } else if constexpr (BITS == 3) {                  // seven pieces of 15 bits
                    uint32_t v[SUMS];
#pragma unroll
                    for (int i = 0; i < SUMS; ++i) v[i] = h ? sum[i] >> 16 : sum[i] & 0xffffu;
                    out[0] = (int32_t)(v[0] | (v[1] << 15) | (v[2] << 30));
                    out[N] = (int32_t)((v[2] >> 2) | (v[3] << 13) | (v[4] << 28));
                    out[2 * (size_t)N] = (int32_t)((v[4] >> 4) | (v[5] << 11) | (v[6] << 26));
                } else {
#pragma unroll
                    for (int i = 0; i < BITS; ++i)
                        out[(size_t)i * N] = (int32_t)__byte_perm(sum[2 * i], sum[2 * i + 1], h ? 0x7632 : 0x5410);
                }
            }
        }
        __syncthreads();
        if (c + 2 < c_end) fetch(c + 2, buf);
    }
}

// Chunks of K per CTA, so that the waves of the grid are full and short: a CTA costs its chunks, the start of its pipeline and its table
// (an entry about as much as four elements).
int pack_split(int chunks, int strips, int resident, int G) {
    int per = chunks;
    long long best = -1;
    for (int p = 1; p <= chunks; ++p) {
        const int c = (chunks + p - 1) / p, ctas = strips * ((chunks + c - 1) / c);
        const long long cost = (long long)((ctas + resident - 1) / resident) * (64 * (c + 1) + G);
        if (best < 0 || cost < best) { best = cost; per = c; }
    }
    return per;
}

// Launched while the kernel in front ends (both kernels wait for it before they touch memory, and let none start before they have ended
// themselves): layers one behind the other 28.8 -> 26.3 us for 4096 x 11008, 16.6 -> 14.9 for 1664 x 10720 in groups of 32.
template <typename... P, typename... A>
int launch_pack_early(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    B200GPTQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
    return B200GPTQ_OK;
}

template <int BITS>
int launch_pack_pairs(const void* weight, const float* scales, const float* zeros, const int32_t* g_idx, int K, int N, int G,
                      int32_t* qweight, int32_t* qzeros, __half* scales_out, int32_t* g_idx_out, cudaStream_t stream) {
    const int chunks = (K + kPairChunk - 1) / kPairChunk, strips = N / kPackCols;
    const size_t used = 2 * (sizeof(__half) * kPackCols * (kPairChunk + 8) + kPairChunk * sizeof(int)) + (size_t)G * kPairPitch * sizeof(uint2);
    const size_t constants = 2 * 128 * kPackPitch * sizeof(float), smem = used > constants ? used : constants;
    static std::once_flag once[64];
    static int result[64];
    int dev = 0;
    B200GPTQ_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return B200GPTQ_ERR_TOO_LARGE;
    std::call_once(once[dev], [dev] {
        result[dev] = (int)cudaFuncSetAttribute(pack_pairs_kernel<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    });
    if (result[dev] != 0) { set_last_cuda_error(result[dev]); return B200GPTQ_ERR_CUDA; }
    const int fit = (int)(220 * 1024 / (smem + 1024));
    const int per = pack_split(chunks, strips, sm_count() * (fit < kPairCtas ? fit : kPairCtas), G);
    dim3 grid(strips, (chunks + per - 1) / per + 1);
    return launch_pack_early(pack_pairs_kernel<BITS>, grid, kPairThreads, smem, stream, static_cast<const __half*>(weight), scales, zeros,
                             g_idx, K, N, G, per, qweight, qzeros, scales_out, g_idx_out);
}

template <int BITS, typename T>
int launch_pack_linear(const void* weight, const float* scales, const float* zeros, const int32_t* g_idx, int K, int N,
                       int G, int32_t* qweight, int32_t* qzeros, __half* scales_out, int32_t* g_idx_out, cudaStream_t stream) {
    const int chunks = (K + kPackChunk - 1) / kPackChunk, strips = N / kPackCols;
    // fp16 weights of 2 to 4 bits whose table fits; 8 bits have no room for their integers in a half
    if constexpr (std::is_same<T, __half>::value && BITS != 8)
        if ((long long)G * kPairPitch * (int)sizeof(uint2) <= kPackTableMax)
            return launch_pack_pairs<BITS>(weight, scales, zeros, g_idx, K, N, G, qweight, qzeros, scales_out, g_idx_out, stream);
    const long long table = (long long)G * kPackPitch * sizeof(float2);
    const int use_table = table <= kPackTableMax;
    const size_t smem = 2 * (sizeof(T) * kPackCols * (kPackChunk + 16 / sizeof(T)) + kPackChunk * sizeof(int)) + (use_table ? table : 0);
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
    const int resident = sm_count() * (smem * kPackCtas <= 220 * 1024 ? kPackCtas : (int)(220 * 1024 / smem));
    const int per = pack_split(chunks, strips, resident, G);
    dim3 grid(strips, (chunks + per - 1) / per + 1);
    return launch_pack_early(pack_linear_kernel<BITS, T>, grid, kPackThreads, smem, stream, static_cast<const T*>(weight), scales, zeros,
                             g_idx, K, N, G, per, use_table, qweight, qzeros, scales_out, g_idx_out);
}

}  // namespace

int pack_linear_dispatch(const void* weight, int dtype, const float* scales, const float* zeros, const int32_t* g_idx,
                         int K, int N, int G, int bits, int32_t* qweight, int32_t* qzeros, __half* scales_out, int32_t* g_idx_out,
                         cudaStream_t stream) {
#define B200GPTQ_PACK(B)                                                                                                             \
    (dtype == B200GPTQ_F16    ? launch_pack_linear<B, __half>(weight, scales, zeros, g_idx, K, N, G, qweight, qzeros, scales_out,    \
                                                              g_idx_out, stream)                                                     \
     : dtype == B200GPTQ_BF16 ? launch_pack_linear<B, __nv_bfloat16>(weight, scales, zeros, g_idx, K, N, G, qweight, qzeros,         \
                                                                     scales_out, g_idx_out, stream)                                  \
                              : launch_pack_linear<B, float>(weight, scales, zeros, g_idx, K, N, G, qweight, qzeros, scales_out,     \
                                                             g_idx_out, stream))
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
