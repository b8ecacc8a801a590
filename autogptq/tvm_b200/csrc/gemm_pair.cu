// Prefill dequant-GEMM for more than 16 rows of x (2- and 8-bit layers: any number): pairs of CTAs on one tcgen05 tile.
//
//   y[M, N] = x[M, K] @ W[K, N] (+ bias),   W[k, n] = scales[g, n] * (q[k, n] - zero[g, n]),  rounded once to fp16
//
// Like gemm.cu the product is computed transposed, y^T = W^T x^T, with the dequantised weights as the A operand in tensor
// memory.  There one CTA took 128 columns x 256 rows and read all 256 rows of x itself: 1.6 GB of x through L2 for 2048 rows
// of 4096 x 12288, 36 KB per 64-row k-tile against the 550 clk its products take, which is what bounded it (182 us; with
// a quarter of the products 152, without the dequantisation 166).  Here two CTAs of a cluster share a 256-column tile
// (tcgen05 cta_group::2): each holds and dequantises its own 128 columns and HALF of the rows of x.
//
//   warps 0, 3  TMA: packed weights, scales and zero-points of 128 rows of K, into a ring of their own that runs ahead of
//               the products as far as shared memory allows (they come from DRAM, x from L2)
//   warp 1      TMA: this CTA's rows of x, into the stages; completion is counted in the first CTA of the pair
//   warp 2      first CTA: issues tcgen05.mma for both (M = 256 columns, N = TN rows of x, K = 16); allocates tensor memory
//   warps 4..11 epilogue: accumulators -> y
//   warps 12..27  four groups of four that take units of 128 rows in turn: a thread owns one column, dequantises it to the exact
//               fp16 values of the reference (auto_gptq/nn_modules/qlinear.py:242: one rounding) in the natural order of k and
//               stores them into the stage's A buffer in tensor memory.
//
// Up to about 180 rows per tile the weight warps are what bounds a launch.  Of a turn's 1800 clk per 64 rows 190 went to each of two
// barriers that were ready, 400 to the words and constants, 650 to the arithmetic (four warps share a scheduler), 250 to the rest of
// the loop, and the threads that issue copies and products spent about 200 clk per 64 rows on barriers too.  So everything moves in
// units of 128 rows, x and A (a stage) as well as the weights: half the hand-overs.  Clocks per 64 rows of K before and after:
// 3 bits, 32 rows of 9216 x 9216 505 and 335; 4 bits in groups of 64, 77 rows of 11008 x 4096 465 and 360; 8 bits, 512 rows of
// 4096 x 4096 550 and 480 (with a second warp for the weights 310, 340 and 430).  What is left is the arithmetic: without it 230,
// without the products 310.
//
// The pairs are persistent: the rings run on from one tile to the next, so only the drain of the accumulators stands
// between two tiles (nothing, where two sets of accumulators fit: up to 128 rows).  A stage is released in both CTAs by one
// multicast tcgen05.commit.  Every wait is bounded: on expiry the kernel raises a sticky status word, unwinds, frees its
// tensor memory and returns.
//
// Replaces the TVM-generated wmma kernels src/kernels/gemm_kernel.cu:25-142 of the reference.
#include <cuda.h>

#include <mutex>

#include "common.cuh"
#include "gemm_pair.h"
#include "ring_rules.h"

namespace b200gptq {

namespace {

constexpr int BN = kPairColumns;         // columns per CTA
constexpr int BK = kPairKTile;           // rows of K of a k-tile; a stage holds two
constexpr int kGroups = kPairGroups, kGroupWarps = 4;
constexpr int kFirstEpiWarp = 4, kEpiWarps = 8, kFirstWeightWarp = kFirstEpiWarp + kEpiWarps;
constexpr int kThreads = 32 * (kFirstWeightWarp + kGroups * kGroupWarps);
constexpr int kMaxStages = kPairMaxStages / 2, kMaxW = kPairMaxSlots;
constexpr int kTmemCols = kPairTmemCols; // accumulators in columns [0, TN) of a set, 64 columns of A per stage behind them
constexpr int kSmemMax = kPairSmem;
constexpr int kStatusWord = kMaxCounters - 1;
constexpr int kMaxSplits = 4;
constexpr int kSumWarps = kThreads / 32 - kFirstEpiWarp;     // warps that add the runs of a split K

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
    return ok != 0;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// On a barrier of the other CTA.  What it announces lies in tensor memory, ordered by the tcgen05 fences around it; no
// ordinary memory is handed over, so the default scope serves (with .cluster scope on arrive and wait: 244 us instead of
// 187 for 2048 rows of 4096 x 12288, a memory barrier and an L1 invalidation per hand-over).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity), "r"(4000u) : "memory");
    return ok != 0;
}
// Bounded wait: gives up after ~2e9 clocks or as soon as another warp of the CTA has.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        for (int i = 0; i < 8; ++i)
            if (mbar_try(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > 2000000000LL) { *abort_flag = 1; return false; }
    }
}
__device__ __forceinline__ uint32_t in_cta(uint32_t local, uint32_t rank) {   // the same shared-memory offset in CTA `rank`
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tma_1d(uint32_t dst, const CUtensorMap* map, int x, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.1d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2}], [%3];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// into this CTA's shared memory, counted on a barrier of the pair's first CTA
__device__ __forceinline__ void tma_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {   // arrives at this offset in both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((unsigned short)3) : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// (the registers pass through the wait, so that nothing reads them before it)
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :: "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
// K-major, 128-byte-swizzled operand tile: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);   // start address, 16-byte units
    d |= (uint64_t)1 << 16;                    // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset: next 8-row group
    d |= (uint64_t)1 << 46;                    // descriptor version of sm_100
    d |= (uint64_t)2 << 61;                    // SWIZZLE_128B
    return d;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t mask, uint32_t magic) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(magic));
    return r;
}
__device__ __forceinline__ __half2 as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
// fp16 exponent pattern that turns a field at bit p of a 16-bit half into 2^(10-p) + field
__host__ __device__ constexpr uint32_t magic_at(int p) { return (uint32_t)(25 - p) << 10; }
__host__ __device__ constexpr uint32_t magic2(int lo, int hi) { return magic_at(lo) | (magic_at(hi) << 16); }
// 2^(10-lo) + z, 2^(10-hi) + z
template <int LO, int HI>
__device__ __forceinline__ __half2 offsets(__half2 z2) { return __hadd2(as_h2(magic2(LO, HI)), z2); }
// (field + offset) pair -> scale * (field - zero): the subtraction is exact in fp16 and the product is rounded once
__device__ __forceinline__ uint32_t finish(uint32_t biased, __half2 offset_plus_zero, __half2 scale2) {
    const __half2 r = __hmul2(__hsub2(as_h2(biased), offset_plus_zero), scale2);
    return *reinterpret_cast<const uint32_t*>(&r);
}

// One 32-row block of one column -> 16 pairs in the natural order of k.
template <int BITS> struct Block;

// Byte b of a word replicated into all four lanes: low nibble in the low half, high nibble in the high half.
template <> struct Block<4> {
    __device__ static __forceinline__ void run(const uint32_t (&w)[4], __half2 s2, __half2 z2, uint32_t (&out)[16]) {
        const __half2 o = offsets<0, 4>(z2);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            out[i] = finish(lop3_and_or(__byte_perm(w[i >> 2], 0u, 0x1111u * (i & 3)), 0x00f0000fu, magic2(0, 4)), o, s2);
    }
};
template <> struct Block<8> {
    __device__ static __forceinline__ void run(const uint32_t (&w)[8], __half2 s2, __half2 z2, uint32_t (&out)[16]) {
        const __half2 o = offsets<0, 0>(z2);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            out[i] = finish(__byte_perm(w[i >> 1], 0x64646464u, (i & 1) ? 0x4342 : 0x4140), o, s2);
    }
};
template <> struct Block<2> {
    __device__ static __forceinline__ void run(const uint32_t (&w)[2], __half2 s2, __half2 z2, uint32_t (&out)[16]) {
        const __half2 o0 = offsets<0, 2>(z2), o1 = offsets<4, 6>(z2);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t rep = __byte_perm(w[i >> 2], 0u, 0x1111u * (i & 3));     // four fields
            out[2 * i] = finish(lop3_and_or(rep, 0x000c0003u, magic2(0, 2)), o0, s2);
            out[2 * i + 1] = finish(lop3_and_or(rep, 0x00c00030u, magic2(4, 6)), o1, s2);
        }
    }
};
// Pair i sits at bits 6 i .. 6 i + 5 of the 96-bit run.  The two bytes around it are copied into both halves; where the
// pair starts at bit 6 of a byte (every fourth) the run is shifted by 4 bits first.
template <> struct Block<3> {
    __device__ static __forceinline__ void run(const uint32_t (&w)[3], __half2 s2, __half2 z2, uint32_t (&out)[16]) {
        const __half2 o0 = offsets<0, 3>(z2), o2 = offsets<2, 5>(z2), o4 = offsets<4, 7>(z2);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int shift = (6 * i) % 8 == 6 ? 4 : 0, bit = 6 * i - shift, p = bit % 8;   // p = 0, 2 or 4
            const int wi = bit / 32, by = (bit % 32) / 8;
            const uint32_t lo = w[wi], hi = wi < 2 ? w[wi + 1] : 0u;
            const uint32_t a = shift ? (bit % 32 + shift + 6 <= 32 ? lo >> 4 : __funnelshift_r(lo, hi, 4)) : lo;
            // bytes by, by + 1 of (a, next word); pairs without a shift that cross into the next word start at byte 3
            const uint32_t rep = __byte_perm(a, shift ? 0u : hi, by * 0x0101u + 0x1010u * (by + 1));
            const uint32_t v = lop3_and_or(rep, (7u << p) | (7u << (p + 19)), p == 0 ? magic2(0, 3) : (p == 2 ? magic2(2, 5) : magic2(4, 7)));
            out[i] = finish(v, p == 0 ? o0 : (p == 2 ? o2 : o4), s2);
        }
    }
};

// Field of column `col` (0 .. 127) plus one, from words in shared memory.
template <int BITS>
__device__ __forceinline__ uint32_t zero_of(const uint8_t* row, int col) {
    const int bit = BITS * col;
    uint32_t v = row[bit >> 3];
    if (BITS == 8) return v + 1u;
    if (BITS == 3) v |= (uint32_t)row[(bit >> 3) + 1] << 8;
    return ((v >> (bit & 7)) & ((1u << BITS) - 1u)) + 1u;
}

struct PairArgs {
    int M, K, N, spg, groups_in_slot, TN, S, SW, acc_sets, splits;
    int pairs, row_tiles, tiles;         // 256-column tiles, TN-row tiles, all tiles (with the runs of K)
    unsigned int spg_inv;                // ceil(2^32 / spg), spg = 32-row blocks per group
};

template <int BITS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                 const __grid_constant__ CUtensorMap tmap_s, const __grid_constant__ CUtensorMap tmap_z,
                 const int32_t* __restrict__ g_idx, const int32_t* __restrict__ qzeros, const __half* __restrict__ scales,
                 const __half* __restrict__ bias, __half* __restrict__ y, const PairArgs p, unsigned int* __restrict__ status,
                 float* __restrict__ partial) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - raw);
    __shared__ __align__(8) uint64_t bars[2 * kMaxW + 2 * kMaxStages + 4];
    __shared__ uint32_t tmem_base_holder;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1;             // cluster rank; 0 issues the products
    const int K = p.K, N = p.N, TN = p.TN, S = p.S, SW = p.SW, TH = TN / 2;
    const int RB = K / 32, KT_all = (K + BK - 1) / BK, U_all = (K + 127) / 128;
    const int cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;
    const uint32_t x_bytes = (uint32_t)TH * BK * 2;      // of a k-tile; a stage holds two
    const int w_slot = pair_slot_bytes(BITS, p.groups_in_slot);
    const uint32_t w_off = S * 2 * x_bytes;

    const uint32_t bar_base = smem_u32(bars);
    auto w_full = [&](int s) { return bar_base + 8u * s; };
    auto w_empty = [&](int s) { return bar_base + 8u * (kMaxW + s); };
    auto full = [&](int s) { return bar_base + 8u * (2 * kMaxW + s); };             // x of both CTAs and A of both CTAs
    auto empty = [&](int s) { return bar_base + 8u * (2 * kMaxW + kMaxStages + s); };
    auto acc_full = [&](int a) { return bar_base + 8u * (2 * kMaxW + 2 * kMaxStages + a); };
    auto acc_empty = [&](int a) { return bar_base + 8u * (2 * kMaxW + 2 * kMaxStages + 2 + a); };

    // A tile: 256 columns x TN rows x a run of 128-row units.
    struct Tile { int n0, m0, z, u0, u1, kt0, KT; };
    auto tile_at = [&](int t) {
        Tile v;
        const int pr = t % p.pairs, r = t / p.pairs, row = r % p.row_tiles;
        v.z = r / p.row_tiles;
        v.n0 = (2 * pr + rank) * BN;
        v.m0 = row * TN;
        v.u0 = v.z * U_all / p.splits;
        v.u1 = (v.z + 1) * U_all / p.splits;
        v.kt0 = 2 * v.u0;
        v.KT = min(2 * v.u1, KT_all) - v.kt0;
        return v;
    };
    // group of a 32-row block without a division (140 clk each, in the one warp that feeds every k-tile)
    auto group_at = [&](int rb) { return p.spg == 1 ? rb : (int)__umulhi((unsigned int)rb, p.spg_inv); };
    const int zwords = N / 32 * BITS;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < SW; ++s) { mbar_init(w_full(s), 1); mbar_init(w_empty(s), kGroupWarps); }
        for (int s = 0; s < S; ++s) {
            mbar_init(full(s), 1 + 2 * kGroupWarps);     // the first CTA's expect_tx arrive, a group of weight warps in each
            mbar_init(empty(s), 1);                      // tcgen05.commit
        }
        for (int a = 0; a < 2; ++a) { mbar_init(acc_full(a), 1); mbar_init(acc_empty(a), 2 * kEpiWarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_holder)), "r"((uint32_t)kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();                                      // barriers of both CTAs exist, tensor memory is allocated
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_holder, tmem_a = tmem_base + (uint32_t)(p.acc_sets * TN);
    asm volatile("griddepcontrol.launch_dependents;");
    // What a preceding kernel may still be writing: x; what it may still be reading: y and the scratch.  The weights are unpacked
    // before the wait, as far as the stages go (77 rows of 11008 x 4096: the first product came 2.6 us after the wait, now 1.1).  From
    // there on what a warp waits for comes after the products, and these after x: it lets the preceding kernel end before
    // it starts the clock of a bounded wait (a sum over ranks may take its time).
    if (warp != 0 && warp != 3 && (warp < kFirstWeightWarp || g_idx)) asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---- epilogue: a warp reads the accumulators of 32 columns (tensor-memory lanes), 16 rows of x at a time ----
    const uint32_t lane_acc = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16);
    auto column_bias = [&](const Tile& v) -> float {
        const int n = v.n0 + 32 * (warp & 3) + lane;
        return bias && n < N ? __half2float(bias[n]) : 0.f;
    };
    // two lanes exchange values so that each stores a pair of columns of every other row (N is a multiple of 32: whole warps)
    auto store_rows = [&](const Tile& v, int m, float (&x)[16]) {
        const int n = v.n0 + 32 * (warp & 3) + lane, left = n < N ? p.M - m - (lane & 1) : 0;
        __half* dst = y + (size_t)(m + (lane & 1)) * N + (n & ~1);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float give = (lane & 1) ? x[2 * i] : x[2 * i + 1];
            const float got = __shfl_xor_sync(0xffffffffu, give, 1);
            const __half2 h = (lane & 1) ? __floats2half2_rn(got, x[2 * i + 1]) : __floats2half2_rn(x[2 * i], got);
            if (2 * i < left) *reinterpret_cast<__half2*>(dst) = h;
            dst += 2 * (size_t)N;
        }
    };

    if (warp == 0 || warp == 3) {
        // ===== packed weights, scales, zero-points.  (With a g_idx the number of groups is not known here, so boxes could not
        //       be clipped to the arrays: the weight warps read scales and zero-points themselves.  The first boxes sent off before the
        //       cluster has met: a launch 0.4 to 0.6 us longer, a box takes its thread 120 clk.) =====
        //       Two warps, every other unit each: one thread takes 600 clk for a unit's barrier and boxes, and the weight warps had to wait
        //       for it (8 bits, 128 rows per tile 480 clk per 64 rows of K, now 430; 3 bits, 32 rows 335, now 310).
        if (elect_one()) {
            const int rows_g = g_idx ? 0 : p.groups_in_slot;
            const uint32_t tx = pair_unit_bytes(BITS) + rows_g * (BN * 2 + pair_zero_words(BITS) * 4);
            int s = 0, round = 0, mine = warp == 0;
            bool ok = true;
            for (int t = cluster; t < p.tiles && ok; t += clusters) {
                const Tile v = tile_at(t);
                const int zn = v.n0 / 32 * BITS;
                for (int u = v.u0; u < v.u1; ++u, mine ^= 1) {
                    if (mine) {
                        const int g0 = group_at(4 * u);
                        if (round > 0 && !mbar_try(w_empty(s), (round - 1) & 1)) {
                            asm volatile("griddepcontrol.wait;" ::: "memory");
                            ok = mbar_wait(w_empty(s), (round - 1) & 1, &abort_flag);
                        }
                        if (!ok) break;
                        const uint32_t dst = base + w_off + s * w_slot, bar = w_full(s);
                        mbar_expect(bar, tx);
                        tma_2d(dst, &tmap_w, v.n0, u * 4 * BITS, bar);
                        if (rows_g) tma_2d(dst + pair_unit_bytes(BITS), &tmap_s, v.n0, g0, bar);
                        for (int r = 0; r < rows_g; ++r)
                            tma_1d(dst + pair_unit_bytes(BITS) + rows_g * BN * 2 + r * 128, &tmap_z, ((g0 + r) * zwords + zn) & ~3, bar);
                    }
                    if (++s == SW) { s = 0; ++round; }
                }
            }
        }
    } else if (warp == 1) {
        // ===== this CTA's rows of x =====
        if (elect_one()) {
            const uint32_t first_full = in_cta(full(0), 0);
            int s = 0, round = 0;
            bool ok = true;
            for (int t = cluster; t < p.tiles && ok; t += clusters) {
                const Tile v = tile_at(t);
                for (int kt = 0; kt < v.KT; kt += 2) {
                    if (round > 0) ok = mbar_wait(empty(s), (round - 1) & 1, &abort_flag);
                    if (!ok) break;
                    const uint32_t dst = base + s * 2 * x_bytes, bar = first_full + 8u * s;
                    const int k = (v.kt0 + kt) * BK, m = v.m0 + rank * TH;
                    const bool two = kt + 1 < v.KT;
                    if (rank == 0) mbar_expect(full(s), two ? 4 * x_bytes : 2 * x_bytes);
                    tma_2d_pair(dst, &tmap_x, k, m, bar);
                    if (two) tma_2d_pair(dst + x_bytes, &tmap_x, k + BK, m, bar);
                    if (++s == S) { s = 0; ++round; }
                }
            }
        }
    } else if (warp == 2) {
        // ===== products, for both CTAs =====
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = (1u << 4) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(2 * BN >> 4) << 24);
            bool ok = true;
            int s = 0, round = 0, set = 0, used = 0;     // used: times the sets have gone round
            for (int t = cluster; t < p.tiles && ok; t += clusters) {
                const Tile v = tile_at(t);
                if (used > 0) ok = mbar_wait(acc_empty(set), (used - 1) & 1, &abort_flag);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem_base + (uint32_t)(set * TN);
                for (int kt = 0; kt < v.KT; kt += 2) {
                    ok = mbar_wait(full(s), round & 1, &abort_flag);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t bdesc = make_smem_desc(base + s * 2 * x_bytes);
                    const uint32_t a_addr = tmem_a + 64u * s;
#pragma unroll
                    for (int k16 = 0; k16 < BK / 16; ++k16)
                        mma_pair(acc, a_addr + 8u * k16, bdesc + 2u * k16, idesc, (kt > 0 || k16 > 0) ? 1u : 0u);
                    if (kt + 1 < v.KT) {
                        const uint64_t second = bdesc + (x_bytes >> 4);
#pragma unroll
                        for (int k16 = 0; k16 < BK / 16; ++k16)
                            mma_pair(acc, a_addr + 32u + 8u * k16, second + 2u * k16, idesc, 1u);
                    }
                    mma_commit_pair(empty(s));
                    if (++s == S) { s = 0; ++round; }
                }
                if (ok) mma_commit_pair(acc_full(set));
                if (++set == p.acc_sets) { set = 0; ++used; }
            }
        }
    } else if (warp >= kFirstWeightWarp) {
        // ===== dequantisation =====
        const int quarter = warp & 3;                    // tensor-memory lanes 32 * quarter .. + 31
        const int wgroup = (warp - kFirstWeightWarp) / kGroupWarps, col = 32 * quarter + lane;
        const uint32_t lane_a = tmem_a + ((uint32_t)(32 * quarter) << 16);
        const uint32_t first_full = in_cta(full(0), 0);
        const bool early_words = BITS % 4 != 0 && (zwords & 3);       // zero-point boxes may start early
        bool ok = true;
        // Stage s and slot ws of the group's unit; from one turn to the next it moves on by kGroups units.
        int s = wgroup, round = 0, ws = wgroup, wround = 0, turn = wgroup;
        for (int t = cluster; t < p.tiles && ok; t += clusters) {
            const Tile v = tile_at(t);
            const int units = pair_turns(v.KT) / 2;
            for (; turn < units; turn += kGroups) {
                while (s >= S) { s -= S; ++round; }
                if (ws >= SW) { ws -= SW; ++wround; }
                const int u = v.u0 + turn, blocks = min(4, 2 * (v.KT - 2 * turn));
                // (an answer takes 190 clk: both questions are asked before the first answer is looked at)
                const bool there = mbar_try(w_full(ws), wround & 1), free = round == 0 || mbar_try(empty(s), (round - 1) & 1);
                if (!__all_sync(0xffffffffu, there && free)) {
                    if (round > 0 || wround > 0) asm volatile("griddepcontrol.wait;" ::: "memory");
                    ok = mbar_wait(w_full(ws), wround & 1, &abort_flag);
                    if (ok && round > 0) ok = mbar_wait(empty(s), (round - 1) & 1, &abort_flag);   // its products have retired
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint8_t* src = base_ptr + w_off + ws * w_slot;
                const uint32_t* pw = reinterpret_cast<const uint32_t*>(src) + col;
                const int g0 = group_at(4 * u);
                __half2 s2, z2;
                auto constants = [&](int b, int r) {      // of 32-row block b of the unit, group r of the slot
                    __half sc = __float2half(0.f);
                    uint32_t z = 1;
                    if (g_idx) {
                        const int grp = __ldg(g_idx + 32 * min(4 * u + b, RB - 1));
                        if (v.n0 + col < N) {
                            sc = __ldg(scales + (size_t)grp * N + v.n0 + col);
                            z = (uint32_t)zero_point<BITS>(qzeros + (size_t)grp * zwords, v.n0 + col);
                        }
                    } else {
                        const int early = early_words ? ((g0 + r) * zwords + v.n0 / 32 * BITS) & 3 : 0;
                        sc = reinterpret_cast<const __half*>(src + pair_unit_bytes(BITS) + r * BN * 2)[col];
                        z = zero_of<BITS>(src + pair_unit_bytes(BITS) + p.groups_in_slot * BN * 2 + r * 128 + 4 * early, col);
                    }
                    s2 = __half2half2(sc);
                    z2 = __half2half2(__ushort2half_rn((unsigned short)z));
                };
                uint32_t w[2][BITS];                      // this block's words and the next one's
#pragma unroll
                for (int r = 0; r < BITS; ++r) w[0][r] = pw[r * BN];
                int r_at = 0;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    if (b >= blocks) break;
                    if (b == 0 || g_idx) {
                        constants(b, 0);
                    } else if (p.groups_in_slot != 1) {
                        const int r = min(group_at(4 * u + b) - g0, p.groups_in_slot - 1);
                        if (r != r_at) constants(b, r);
                        r_at = r;
                    }
                    if (b + 1 < 4)
#pragma unroll
                        for (int r = 0; r < BITS; ++r) w[(b + 1) & 1][r] = pw[((b + 1) * BITS + r) * BN];
                    uint32_t out[16];
                    Block<BITS>::run(w[b & 1], s2, z2, out);
                    tmem_st16(lane_a + 64u * s + 16 * b, out);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(w_empty(ws));
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(first_full + 8u * s);
                s += kGroups;
                ws += kGroups;
            }
            turn -= units;                                // this group's first unit of the next tile
        }
    } else if (warp >= kFirstEpiWarp) {
        // ===== accumulators (lane = column, tensor-memory column = row of x) -> y =====
        const int half = (warp - kFirstEpiWarp) >> 2;
        const uint32_t first_empty = in_cta(acc_empty(0), 0);
        bool ok = true;
        int set = 0, used = 0;
        for (int t = cluster; t < p.tiles && p.splits == 1; t += clusters) {
            const Tile v = tile_at(t);
            const float b = column_bias(v);
            if (ok) ok = mbar_wait(acc_full(set), used & 1, &abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int chunks = min(TN, p.M - v.m0 + 15) / 16;        // 16 rows each; the next one is loaded meanwhile
            const uint32_t acc = lane_acc + (uint32_t)(set * TN);
            uint32_t r[16], next[16] = {};
            if (half < chunks) { tmem_ld16(acc + 16u * half, r); tmem_wait_ld(r); }
#pragma unroll 1
            for (int c = half; c < chunks; c += 2) {
                if (c + 2 < chunks) tmem_ld16(acc + 16u * (c + 2), next);
                float x[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(r[i]) + b;
                store_rows(v, v.m0 + 16 * c, x);
                tmem_wait_ld(next);
#pragma unroll
                for (int i = 0; i < 16; ++i) r[i] = next[i];
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(first_empty + 8u * set);
            if (++set == p.acc_sets) { set = 0; ++used; }
        }
    }

    if (p.splits > 1 && warp >= kFirstEpiWarp) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        // ===== split K (one tile per pair): a warp takes every sixth 16 rows of its 32 columns, all warps but the first four.  It puts its
        //       run's sums of them into the scratch and is counted in; the last of the runs' warps, of whichever CTA, adds the runs in
        //       order.  No warp waits for another.  The counting is done whatever happened before, so that every counter returns to
        //       zero.  (The last CTA of a tile to arrive adding all of it: 5000 clk for the sums in, 5000 for the sum, of the 40 000
        //       of 77 rows of 11008 x 4096.) =====
        const Tile v = tile_at(cluster);
        bool ok = mbar_wait(acc_full(0), 0, &abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int chunks = min(TN, p.M - v.m0 + 15) / 16, all_chunks = TN / 16, first = (warp - kFirstEpiWarp) >> 2;
        const int strips = N / 32, strip = v.n0 / 32 + (warp & 3), column = (v.m0 / TN) * strips + strip;
        if (strip < strips && first < chunks) {
            const size_t run = (size_t)p.row_tiles * strips * all_chunks * 512;          // floats of a run of K
            float* sums = partial + (size_t)column * all_chunks * 512 + 4 * lane;        // [16 rows][4 of them][column][row]
#pragma unroll 1
            for (int c = first; c < chunks; c += kSumWarps / 4) {
                uint32_t r[16] = {};
                if (ok) { tmem_ld16(lane_acc + 16u * c, r); tmem_wait_ld(r); }
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    *reinterpret_cast<uint4*>(sums + v.z * run + c * 512 + 128 * i) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
            }
            __syncwarp();
            unsigned int before = 0;                      // one lane's fences serve the warp, which it has just met and meets again
            if (lane == 0) {
                unsigned int* counter = status + column * (kSumWarps / 4) + first;
                asm volatile("fence.acq_rel.gpu;" ::: "memory");
                asm volatile("atom.relaxed.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(counter) : "memory");
                asm volatile("fence.acq_rel.gpu;" ::: "memory");
                if (before == (unsigned int)p.splits - 1u) *counter = 0u;
            }
            __syncwarp();
            if (__shfl_sync(0xffffffffu, before, 0) == (unsigned int)p.splits - 1u) {
                const float b = column_bias(v);
                // All runs' sums of 16 rows on their way at once, through the rings: nothing is in flight there any more, and 64 values
                // do not fit in registers (in two parts they took two round trips).  A lane reads what it has copied itself.
                float* copy = reinterpret_cast<float*>(base_ptr) + (warp - kFirstEpiWarp) * p.splits * 512 + 4 * lane;
#pragma unroll 1
                for (int c = first; c < chunks && ok; c += kSumWarps / 4) {
                    for (int z = 0; z < p.splits; ++z)
#pragma unroll
                        for (int i = 0; i < 4; ++i) cp_async16(smem_u32(copy + z * 512 + 128 * i), sums + z * run + c * 512 + 128 * i);
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    float x[16];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float4 sum = *reinterpret_cast<const float4*>(copy + 128 * i);
                        for (int z = 1; z < p.splits; ++z) {
                            const float4 f = *reinterpret_cast<const float4*>(copy + z * 512 + 128 * i);
                            sum.x += f.x; sum.y += f.y; sum.z += f.z; sum.w += f.w;
                        }
                        x[4 * i] = sum.x + b; x[4 * i + 1] = sum.y + b; x[4 * i + 2] = sum.z + b; x[4 * i + 3] = sum.w + b;
                    }
                    store_rows(v, v.m0 + 16 * c, x);
                }
            }
        }
    }

    // ===== teardown: every role arrives here, also after a timed-out wait; neither CTA leaves before the other has =====
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    __syncwarp();
    cluster_sync();
    if (threadIdx.x == 0 && abort_flag) atomicExch(status + kStatusWord, 1u);
    if (warp == 2)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kTmemCols) : "memory");
}

}  // namespace

// Rows of x per tile and runs of K.  In clocks, fitted to 4 bits, 100 to 1024 rows of 4096 x 4096, 4096 x 12288, 11008 x 4096,
// 2048 x 8192 and 8192 x 2048 (within 10 % of what was measured; 3 and 8 bits come within 5 % of 4): a k-tile takes what kPerTile
// says, the weight warps up to 128 rows and the products above; tiles of 160 rows, bound by the weight warps and with one set of
// accumulators, take 25 more where one follows another, their drain (2048 rows of 11008 x 4096 in groups of 32 139 us in such tiles,
// 129 in tiles of 256); start-up and drain take longer the more SMs work; the sum over runs
// grows with what goes through the scratch.  Several runs have a tile per pair of SMs, of eight units or more.  Up to 128 rows the
// caller says how many runs (`few`), in one tile of rows.  Against the best tile without runs: 256 rows of 11008 x 4096 32.1 -> 24.9 us,
// 256 rows of 8192 x 2048 23.3 -> 15.9, 512 rows 25.0 -> 21.2.  one_run: more than 128 rows without runs (no room for their sums).
GemmPairPlan gemm_pair_plan(int M, int N, int K, int few, bool one_run) {
    constexpr int kPerTile[8] = {300, 310, 325, 340, 390, 470, 540, 610};      // 32, 64, .. 256 rows
    const long long pairs = (N + 2 * BN - 1) / (2 * BN), slots = sm_count() / 2, units = (K + 127) / 128;
    const int least = M <= 128 ? few : 1, most = M <= 128 ? few : one_run ? 1 : kMaxSplits;
    long long best = -1;
    GemmPairPlan plan = {256, 1};
    for (int splits = least; splits <= most; ++splits)
        for (int t = 256; t >= 32; t -= 32) {
            const long long rows = (M + t - 1) / t, tiles = pairs * rows * splits, waves = (tiles + slots - 1) / slots;
            if (splits > 1 && (M <= 128 ? t < M : waves > 1 || units / splits < 8)) break;
            const long long kt = 2 * ((units + splits - 1) / splits), busy = tiles < slots ? tiles : slots;
            const long long cost = waves * kt * (kPerTile[t / 32 - 1] + (t == 160 && waves > 1 ? 25 : 0)) + 2850 + 8200 * busy / slots + (splits > 1 ? 6500 + 8 * t * splits : 0);
            if (best < 0 || cost < best) { best = cost; plan = {t, splits}; }
        }
    return plan;
}

namespace {

template <int BITS>
int launch(const __half* x, const int32_t* qweight, const int32_t* qzeros, const __half* scales, const int32_t* g_idx,
           const __half* bias, __half* y, int M, int K, int N, int group_size, GemmPairPlan plan, unsigned int* status,
           float* partial, cudaStream_t stream) {
    const EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) { set_last_cuda_error((int)cudaErrorNotSupported); return B200GPTQ_ERR_CUDA; }
    const int groups = (K + group_size - 1) / group_size;
    PairArgs a = {};
    const int splits = plan.splits, TN = plan.rows;
    a.M = M; a.K = K; a.N = N; a.splits = splits; a.TN = TN;
    a.spg = group_size >= K ? (K + 31) / 32 : (group_size >= 32 ? group_size / 32 : 1);
    a.spg_inv = (unsigned int)((0x100000000ULL + a.spg - 1) / a.spg);                 // (not used for 1)
    a.groups_in_slot = a.spg % 4 == 0 || groups == 1 ? 1 : (a.spg == 1 ? 4 : (a.spg == 2 ? 2 : 3));
    a.pairs = (N + 2 * BN - 1) / (2 * BN);
    a.row_tiles = (M + TN - 1) / TN;
    const long long tiles = (long long)a.pairs * a.row_tiles * splits;
    if (tiles > 0x7fffffff || (splits > 1 && (long long)(N / 32) * a.row_tiles * (kSumWarps / 4) >= kMaxCounters - 1)) return B200GPTQ_ERR_TOO_LARGE;
    a.tiles = (int)tiles;
    const int pairs_of_sms = sm_count() / 2;
    // (a second set of accumulators only serves a pair that has another tile to go on with)
    const PairRings rings = pair_rings(BITS, a.groups_in_slot, TN, a.tiles > pairs_of_sms);
    a.acc_sets = rings.acc_sets; a.S = rings.stages / 2; a.SW = rings.slots;
    const int x_stage = TN * BK * 2, w_slot = pair_slot_bytes(BITS, a.groups_in_slot);
    if (a.SW < 4 || rings.stages < kPairMinStages) return B200GPTQ_ERR_TOO_LARGE;
    // (the sums of a split K pass through the rings: 2 KB per run and warp)
    const int rings_bytes = a.S * x_stage + a.SW * w_slot, sum_bytes = splits > 1 ? kSumWarps * splits * 2048 : 0;
    const int smem = (rings_bytes > sum_bytes ? rings_bytes : sum_bytes) + 1024;
    auto map = [&](CUtensorMap* m, CUtensorMapDataType type, int rank, const void* ptr, const cuuint64_t* dims,
                   const cuuint64_t* strides, const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
        const cuuint32_t estr[2] = {1, 1};
        return encode(m, type, rank, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    CUtensorMap tx, tw, ts, tz;
    const cuuint64_t xd[2] = {(cuuint64_t)K, (cuuint64_t)M}, xs[1] = {(cuuint64_t)K * 2};
    const cuuint32_t xb[2] = {BK, (cuuint32_t)(TN / 2)};
    const cuuint64_t wd[2] = {(cuuint64_t)N, (cuuint64_t)(K / 32 * BITS)}, ws[1] = {(cuuint64_t)N * 4};
    const cuuint32_t wb[2] = {BN, 4 * BITS};
    const cuuint64_t sd[2] = {(cuuint64_t)N, (cuuint64_t)groups}, ss[1] = {(cuuint64_t)N * 2};
    const cuuint32_t sb[2] = {BN, (cuuint32_t)a.groups_in_slot};
    const cuuint64_t zd[1] = {(cuuint64_t)groups * (N / 32 * BITS)};
    const cuuint32_t zb[1] = {(cuuint32_t)pair_zero_words(BITS)};
    if (!map(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, xd, xs, xb, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !map(&tw, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, qweight, wd, ws, wb, CU_TENSOR_MAP_SWIZZLE_NONE) ||
        !map(&ts, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, scales, sd, ss, sb, CU_TENSOR_MAP_SWIZZLE_NONE) ||
        !map(&tz, CU_TENSOR_MAP_DATA_TYPE_INT32, 1, qzeros, zd, ws, zb, CU_TENSOR_MAP_SWIZZLE_NONE)) {
        set_last_cuda_error((int)cudaErrorInvalidValue);
        return B200GPTQ_ERR_CUDA;
    }
    static std::once_flag once[64];
    static int result[64];
    int dev = 0;
    B200GPTQ_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return B200GPTQ_ERR_TOO_LARGE;
    std::call_once(once[dev], [dev] {
        result[dev] = (int)cudaFuncSetAttribute(gemm_pair_kernel<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    });
    if (result[dev] != 0) { set_last_cuda_error(result[dev]); return B200GPTQ_ERR_CUDA; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (a.tiles < pairs_of_sms ? a.tiles : pairs_of_sms));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    B200GPTQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_pair_kernel<BITS>, tx, tw, ts, tz, g_idx, qzeros, scales, bias, y, a, status,
                                         partial));
    return B200GPTQ_OK;
}

}  // namespace

// fp32 partial sums of a launch whose k-tiles are cut into runs
size_t gemm_pair_partial_bytes(int M, int N, GemmPairPlan plan) {
    if (plan.splits == 1) return 0;
    return (size_t)plan.splits * ((M + plan.rows - 1) / plan.rows * plan.rows) * N * sizeof(float);
}

int gemm_pair_dispatch(const __half* x, const int32_t* qweight, const int32_t* qzeros, const __half* scales, const int32_t* g_idx,
                       const __half* bias, __half* y, int M, int K, int N, int bits, int group_size, GemmPairPlan plan,
                       unsigned int* status, float* partial, cudaStream_t stream) {
    switch (bits) {
        case 2: return launch<2>(x, qweight, qzeros, scales, g_idx, bias, y, M, K, N, group_size, plan, status, partial, stream);
        case 3: return launch<3>(x, qweight, qzeros, scales, g_idx, bias, y, M, K, N, group_size, plan, status, partial, stream);
        case 4: return launch<4>(x, qweight, qzeros, scales, g_idx, bias, y, M, K, N, group_size, plan, status, partial, stream);
        case 8: return launch<8>(x, qweight, qzeros, scales, g_idx, bias, y, M, K, N, group_size, plan, status, partial, stream);
    }
    return B200GPTQ_ERR_BITS;
}

}  // namespace b200gptq
