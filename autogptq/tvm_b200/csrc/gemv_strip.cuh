// Decode GEMV for groups of whole 32-row blocks (bits 2, 3, 4, 8; up to 16 rows of x; groups k / group_size).
//
//   y[m, n] = sum_k x[m, xk(k)] * scales[g, n] * (q[k, n] - zero[g, n]),   g = k / group_size
//
// One layer is 2..130 MB and lasts a few microseconds, so what counts is the chain of latencies of one launch as much as
// bandwidth: start-up, the wait for the previous kernel, x, the products, the sum over K.  The split below has no
// scratch and, from 75 strips of columns on, no cluster and no traffic between CTAs:
//
//  * The columns are cut into strips of 32; a CTA owns a run of strips over ALL of K, one CTA per SM.  Its warps split K
//    in units of 128 rows and are added up through shared memory at the end.  Where the strips would leave half the SMs
//    idle and K is long, clusters of two or four CTAs share one (the rule and its figures: gemv_strip.cu).
//  * Every warp streams its own units through its own ring: cp.async.bulk.tensor boxes of {32 columns, the unit's
//    word-rows, strips} (128-byte swizzle), of the unit's scales and of its zero-points, one mbarrier per slot, no barrier of
//    the CTA.  (16-byte cp.async by the lanes instead of the weight boxes: 13.0 against 7.0 us on 4096 x 12288, 4 bits;
//    scales and zero-points loaded one unit ahead: 38 against 32 us without them on 9216 x 36864, 3 bits.)  The ring is
//    filled before griddepcontrol.wait: under programmatic dependent launch while the kernel in front ends, where that leaves the SM room.
//  * One row of x: a warp puts its whole slice of x into shared memory in the order of the B registers, once.  Several
//    rows: copied with cp.async and permuted as they are read; all of x at once where it fits, else one to three units ahead
//    (one unit ahead is an L2 latency per unit: 16 rows, 9216 x 9216, 3 bits 29 us, two ahead 21).  Which k a lane multiplies
//    is free as long as x is read in the same order.
//  * One or two rows, 2 to 4 bits, whole units per group (4 bits: any groups): products on the integer tensor path.  A byte of weights
//    is q << p, one AND per four fields and no shift (4 bits, whole units: no AND in one of the two products); x is fixed point per unit, or per step where the groups of a unit are scaled apart
//    (4 bits |X| < 2^26, exact for every element within 2^-16 of the largest; 2 and 3 bits 2^22 and 2^-12), shifted by what
//    its weight byte lacks and split into four signed byte planes, which are columns of the B operand.  mma.sync m16n8k32
//    u8 x s8 costs what m16n8k16 f16 does and does twice the products; the fp16 form below needs 2.3 times the instructions.
//    One row with groups of 32, 64 or 96 rows: a product serves two groups, so that scaling their sums, four times a unit, is done by all
//    lanes (half of them had zeros: 4 bits, 8192 x 8192 9.9 -> 8.1 us, 11008 x 12288 23.6 -> 20.0).
//    Used where K is long enough for what the planes take to prepare (the plan in gemv_strip.cu has the measurements).
//  * Otherwise fp16.  4- and 8-bit fields are used as fp16 subnormals: a field masked in place at bit p of its half IS q * 2^(p - 24), so
//    unpacking is one AND (4 bits: and one shift per two words); the two positions of a nibble go to different
//    accumulators and the power of two is applied to the result.  2- and 3-bit fields are ORed into the mantissa of a
//    power of two.  What these powers contribute, and the sum of x that the zero-point multiplies (sum q x - zero * sum x),
//    come from one extra product per step whose A operand holds ones in its first eight rows and the powers in the
//    others; that leaves both in the lanes that need them.  Products are exact in the tensor core, accumulated in fp32
//    per group and scaled in fp32.
//
// Reference semantics: auto_gptq/nn_modules/qlinear.py:197-243; replaces src/kernels/gemv_kernel.cu:25-55.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "common.cuh"

namespace b200gptq {

namespace {

constexpr int kUnit = 128;                // rows of K per unit: four steps of 32
constexpr int kStripCols = 32;
constexpr int kMaxRing = 8;
constexpr int kStatusWord = kMaxCounters - 1;
constexpr int kXPitch = kUnit + 8;        // several rows: halves of a staged row of x (padded: conflict-free reads)

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// One lane of a converged warp (TMA instructions under `lane == 0` are wrapped in a loop over the active threads).
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
    return ok != 0;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
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
        : "=r"(ok) : "r"(bar), "r"(parity), "r"(2000u) : "memory");
    return ok != 0;
}
// Bounded wait: after ~1e9 clocks the kernel goes on with undefined results and a raised status word.
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity) {
    const long long t0 = clock64();
    while (clock64() - t0 < 1000000000LL)
        if (mbar_try(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, bool& ok) {
    if (mbar_try(bar, parity)) return;
    if (ok) ok = mbar_wait_slow(bar, parity);
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t mask, uint32_t magic) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(magic));
    return r;
}
// d += a * b (16 columns x 16 k x 8 rows of x).  Not volatile: the compiler may interleave independent tiles.
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// fp16 bits of 2^(10-p): the offset of a field masked at bit p of its half
__host__ __device__ constexpr uint32_t magic_at(int p) { return (uint32_t)(25 - p) << 10; }
__host__ __device__ constexpr uint32_t magic2(int lo, int hi) { return magic_at(lo) | (magic_at(hi) << 16); }

// The zero-point fields of columns c .. c + 3 (c % 4 == 0) of a strip whose fields start at `row`, in shared memory.
template <int BITS>
__device__ __forceinline__ uint32_t load_zeros(const uint8_t* row, int c) {
    const uint8_t* p = row + ((BITS * c) >> 3);
    if constexpr (BITS == 8) return *reinterpret_cast<const unsigned int*>(p);
    if constexpr (BITS == 4) return *reinterpret_cast<const unsigned short*>(p);
    if constexpr (BITS == 3) return ((uint32_t)p[0] | ((uint32_t)p[1] << 8)) >> (c & 4);   // 12 bits from bit 0 or 4
    return *p;
}

// ---------------------------------------------------------------------------------------------------------------
// Layouts of a unit (128 rows, four steps; in step s quad lane j = lane & 3 multiplies 8 rows).
//   load_row(i, j)   word-row of the lane's i-th 128-bit read (its four columns); step s needs reads s * kPer .. of kPer
//                    (kPer == 0: all kLoads reads serve every step)
//   a_regs           the A registers of one column for step s: {0, 1} of the first product, {2, 3} of the second
//   x_first(s, j)    first of the 8 rows of step s;  b_regs  their natural halves -> {b0, b1} of the two products
//   magic(s, i)      what the A registers hold on top of the fields
//   kMul1            weight of the second product's accumulator;  kScale  power of two of the result
// ---------------------------------------------------------------------------------------------------------------
// WHOLE: a unit lies in one group, so a step may take rows from anywhere in it; otherwise step s is rows 32 s .. 32 s + 31.
template <int BITS, bool WHOLE> struct Layout;

template <bool WHOLE> struct Layout<4, WHOLE> {
    static constexpr int kRows = 16, kLoads = 4, kPer = 1;
    static constexpr bool kMagic = false;
    static constexpr float kMul1 = 1.f / 16.f, kScale = 16777216.f;
    // (rows two apart are free of bank conflicts under the swizzle)
    __device__ static int load_row(int s, int j) { return WHOLE ? 2 * j + (s & 1) + 8 * (s >> 1) : 4 * s + j; }
    __device__ static int x_first(int s, int j) { return 8 * load_row(s, j); }
    // nibble pairs (0,4) (2,6) at bit 0 of their halves: first product; (1,5) (3,7) at bit 4: second
    __device__ static void a_regs(const uint32_t* w, int, int, uint32_t (&a)[4]) {
        const uint32_t lo = w[0], hi = lo >> 8;
        a[0] = lo & 0x000f000fu; a[1] = hi & 0x000f000fu; a[2] = lo & 0x00f000f0u; a[3] = hi & 0x00f000f0u;
    }
    __device__ static void b_regs(const uint4& x, uint32_t (&b)[4]) {
        b[0] = __byte_perm(x.x, x.z, 0x5410); b[1] = __byte_perm(x.y, x.w, 0x5410);
        b[2] = __byte_perm(x.x, x.z, 0x7632); b[3] = __byte_perm(x.y, x.w, 0x7632);
    }
    static constexpr uint32_t magic(int, int) { return 0; }
};

template <bool WHOLE> struct Layout<8, WHOLE> {
    static constexpr int kRows = 32, kLoads = 8, kPer = 2;
    static constexpr bool kMagic = false;
    static constexpr float kMul1 = 1.f, kScale = 16777216.f;
    // a word-row is four rows of K: reads 2s, 2s+1 are the two products of step s
    __device__ static int load_row(int i, int j) { return 2 * j + (i & 1) + 8 * (i >> 1); }
    __device__ static void a_regs(const uint32_t* w, int, int, uint32_t (&a)[4]) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            a[2 * i] = __byte_perm(w[i], 0u, 0x4140);
            a[2 * i + 1] = __byte_perm(w[i], 0u, 0x4342);
        }
    }
    static constexpr uint32_t magic(int, int) { return 0; }
};

template <bool WHOLE> struct Layout<2, WHOLE> {
    static constexpr int kRows = 8, kLoads = 4, kPer = 1;
    static constexpr bool kMagic = true;
    static constexpr float kMul1 = 1.f, kScale = 1.f;
    __device__ static int load_row(int s, int j) { return 2 * s + (j >> 1); }
    __device__ static int x_first(int s, int j) { return 32 * s + 8 * j; }
    // the lane's 8 fields are one half of its word: copied into both halves, pairs (0,1) (2,3) are masked in place, (4,5)
    // (6,7) after a shift by 8
    __device__ static void a_regs(const uint32_t* w, int, int j, uint32_t (&a)[4]) {
        const uint32_t r = __byte_perm(w[0], 0u, (j & 1) ? 0x3232 : 0x1010), h = r >> 8;
        a[0] = lop3_and_or(r, 0x000c0003u, magic2(0, 2)); a[1] = lop3_and_or(r, 0x00c00030u, magic2(4, 6));
        a[2] = lop3_and_or(h, 0x000c0003u, magic2(0, 2)); a[3] = lop3_and_or(h, 0x00c00030u, magic2(4, 6));
    }
    __device__ static void b_regs(const uint4& x, uint32_t (&b)[4]) { b[0] = x.x; b[1] = x.y; b[2] = x.z; b[3] = x.w; }
    static constexpr uint32_t magic(int, int i) { return i & 1 ? magic2(4, 6) : magic2(0, 2); }
};

// 3 bits, several groups in a unit: quad lane j takes fields 8j..8j+7 of each 32-row block, 24 bits at bit 24 j of the
// 96-bit run.
template <> struct Layout<3, false> {
    static constexpr int kRows = 12, kLoads = 12, kPer = 3;
    static constexpr bool kMagic = true;
    static constexpr float kMul1 = 1.f, kScale = 1.f;
    __device__ static int load_row(int i, int) { return i; }
    __device__ static int x_first(int s, int j) { return 32 * s + 8 * j; }
    __device__ static void a_regs(const uint32_t* w, int, int j, uint32_t (&a)[4]) {
        const uint32_t lo = j < 2 ? w[0] : (j == 2 ? w[1] : w[2]);
        const uint32_t hi = j == 1 ? w[1] : w[2];
        const uint32_t v = __funnelshift_r(lo, hi, (32 - 8 * j) & 31);            // field f at bit 3 f
        // fields 2, 3 from v >> 6 in the low half, 4, 5 from v << 4 in the high half
        const uint32_t m = __byte_perm(v >> 6, v << 4, 0x7610);
        a[0] = lop3_and_or(v, 0x001c0007u, magic2(0, 2)); a[1] = lop3_and_or(v, 0x00e00038u, magic2(3, 5));   // (0,6) (1,7)
        a[2] = lop3_and_or(m, 0x00070007u, magic2(0, 0)); a[3] = lop3_and_or(m, 0x00380038u, magic2(3, 3));   // (2,4) (3,5)
    }
    __device__ static void b_regs(const uint4& x, uint32_t (&b)[4]) {
        b[0] = __byte_perm(x.x, x.w, 0x5410); b[1] = __byte_perm(x.x, x.w, 0x7632);
        b[2] = __byte_perm(x.y, x.z, 0x5410); b[3] = __byte_perm(x.y, x.z, 0x7632);
    }
    static constexpr uint32_t magic(int, int i) {
        return i == 0 ? magic2(0, 2) : (i == 1 ? magic2(3, 5) : (i == 2 ? magic2(0, 0) : magic2(3, 3)));
    }
};

// 3 bits, one group per unit: quad lane j owns row block j (three word-rows); seven windows of its 96-bit run expose the
// 32 fields as 16 pairs (0,3) (1,7) (2,8) (4,9) (5,10) (6,11) (12,17) (13,18) (14,19) (15,20) (16,21) (22,27) (23,28)
// (24,29) (25,30) (26,31), four per step.
template <> struct Layout<3, true> {
    static constexpr int kRows = 12, kLoads = 3, kPer = 0;
    static constexpr bool kMagic = true;
    static constexpr float kMul1 = 1.f, kScale = 1.f;
    __device__ static int load_row(int i, int j) { return 3 * j + i; }
    template <int PLO, int PHI>
    __device__ static uint32_t pair(uint32_t v) {
        return lop3_and_or(v, (7u << PLO) | (7u << (PHI + 16)), magic2(PLO, PHI));
    }
    __device__ static void a_regs(const uint32_t* w, int s, int, uint32_t (&a)[4]) {
        if (s == 0) {
            const uint32_t v0 = w[0] << 7, v1 = w[0] >> 1, v2 = __funnelshift_r(w[0], w[1], 11);
            a[0] = pair<7, 0>(v0); a[1] = pair<2, 4>(v1); a[2] = pair<5, 7>(v1); a[3] = pair<1, 0>(v2);
        } else if (s == 1) {
            const uint32_t v2 = __funnelshift_r(w[0], w[1], 11), v3 = w[1];
            a[0] = pair<4, 3>(v2); a[1] = pair<7, 6>(v2); a[2] = pair<4, 3>(v3); a[3] = pair<7, 6>(v3);
        } else if (s == 2) {
            const uint32_t v4 = __funnelshift_r(w[1], w[2], 9), v5 = w[2] << 2;
            a[0] = pair<1, 0>(v4); a[1] = pair<4, 3>(v4); a[2] = pair<7, 6>(v4); a[3] = pair<4, 3>(v5);
        } else {
            const uint32_t v5 = w[2] << 2, v6 = w[2] >> 7;
            a[0] = pair<7, 6>(v5); a[1] = pair<1, 0>(v6); a[2] = pair<4, 3>(v6); a[3] = pair<7, 6>(v6);
        }
    }
    static constexpr uint32_t magic(int s, int i) {
        return s == 0 ? (i == 0 ? magic2(7, 0) : i == 1 ? magic2(2, 4) : i == 2 ? magic2(5, 7) : magic2(1, 0))
             : s == 1 ? ((i & 1) ? magic2(7, 6) : magic2(4, 3))
             : s == 2 ? (i == 0 ? magic2(1, 0) : i == 2 ? magic2(7, 6) : magic2(4, 3))
                      : (i == 1 ? magic2(1, 0) : i == 2 ? magic2(4, 3) : magic2(7, 6));
    }
    // the 32 natural halves of the row block (16 registers) -> the 16 pairs
    __device__ static void b_block(const uint32_t (&x)[16], uint32_t (&b)[16]) {
        constexpr int F[32] = {0, 3, 1, 7, 2, 8, 4, 9, 5, 10, 6, 11, 12, 17, 13, 18,
                               14, 19, 15, 20, 16, 21, 22, 27, 23, 28, 24, 29, 25, 30, 26, 31};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int lo = F[2 * i], hi = F[2 * i + 1];
            b[i] = __byte_perm(x[lo >> 1], x[hi >> 1], ((lo & 1) ? 0x32 : 0x10) | ((hi & 1) ? 0x7600 : 0x5400));
        }
    }
};

// ---------------------------------------------------------------------------------------------------------------
// Integer path.  kSteps tensor instructions (32 rows of K each) per unit and pair of columns; in step s a lane supplies
// two registers of four bytes per column.
//   load_row(i, j)  word-row of the lane's i-th 128-bit read;  regs(w, r)  one column's words -> 2 kSteps registers
//   kPre            log2 of (weight byte) * (pre-shifted X) over q * X
//   item(i, j, row, pre)  preparation of x: the 8 rows (relative to the unit) that item i = 0..3 of quad lane j handles
//                   and the left shift each X gets; items fill step i unless the layout says otherwise
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void imma(int (&d)[4], const int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                     uint32_t b0, uint32_t b1) {   // d = c + a (u8, 16 x 32) * b (s8, 32 x 8)
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}
// 4 x 4 byte transpose: plane p of the result holds byte p of a, b, c, d
__device__ __forceinline__ void planes_of(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&pl)[4]) {
    const uint32_t ab01 = __byte_perm(a, b, 0x5140), cd01 = __byte_perm(c, d, 0x5140);
    const uint32_t ab23 = __byte_perm(a, b, 0x7362), cd23 = __byte_perm(c, d, 0x7362);
    pl[0] = __byte_perm(ab01, cd01, 0x5410); pl[1] = __byte_perm(ab01, cd01, 0x7632);
    pl[2] = __byte_perm(ab23, cd23, 0x5410); pl[3] = __byte_perm(ab23, cd23, 0x7632);
}
struct Bytes8 { unsigned char v[8]; };
constexpr unsigned long long pack8(const Bytes8& t) {
    unsigned long long r = 0;
    for (int i = 0; i < 8; ++i) r |= (unsigned long long)t.v[i] << (8 * i);
    return r;
}

// WHOLE: a unit lies in one group; otherwise step s is rows 32 s .. 32 s + 31 (4 bits only).
template <int BITS, bool WHOLE> struct IntLayout;

// 4 bits: a word-row is a step, nibbles 0 2 4 6 (q) and 1 3 5 7 (q << 4).  Whole units: its bytes are used as they are (low + 16 * high nibble) and
// with the high nibble masked off; what the first product has too much of the low nibble is taken off the x of the second: (low + 16 high) X'
// + low (16 X - X') = 16 (low X + high X').  One AND per word instead of two: one and two rows, groups of 128, 1.00 to 1.04 times as fast
// (4096 x 4096 3.61 -> 3.57 us in each of eight processes, 5120 x 10240 7.63 -> 7.38); with groups scaled apart in a unit 0.99 to 1.00, so these keep both.
template <bool WHOLE> struct IntLayout<4, WHOLE> {
    static constexpr int kSteps = 4, kPre = 4, kLoads = 4;
    __device__ static int load_row(int i, int j) { return WHOLE ? 2 * j + (i & 1) + 8 * (i >> 1) : 4 * i + j; }
    __device__ static void regs(const uint32_t (&w)[kLoads], uint32_t (&r)[2 * kSteps]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { r[2 * i] = w[i] & 0x0f0f0f0fu; r[2 * i + 1] = WHOLE ? w[i] : w[i] & 0xf0f0f0f0u; }
    }
    __device__ static void item(int i, int j, int (&row)[8], int (&pre)[8]) {
#pragma unroll
        for (int e = 0; e < 8; ++e) { row[e] = 8 * load_row(i, j) + 2 * (e & 3) + (e >> 2); pre[e] = e < 4 ? 4 : 0; }
    }
};
template <bool WHOLE> struct IntLayout<8, WHOLE> : IntLayout<4, WHOLE> {};   // (not used: 8-bit fields need no unpacking in fp16 either)
template <> struct IntLayout<2, true> {                 // a word-row is two steps: fields f, f + 4, f + 8, f + 12 (q << 2 f), f = 0 .. 3
    static constexpr int kSteps = 4, kPre = 6, kLoads = 2;
    __device__ static int load_row(int i, int j) { return 2 * j + i; }
    __device__ static void regs(const uint32_t (&w)[kLoads], uint32_t (&r)[2 * kSteps]) {
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = w[i >> 2] & (0x03030303u << (2 * (i & 3)));
    }
    __device__ static void item(int i, int j, int (&row)[8], int (&pre)[8]) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int f = 2 * (i & 1) + (e >> 2);
            row[e] = 16 * load_row(i >> 1, j) + 4 * (e & 3) + f;
            pre[e] = 6 - 2 * f;
        }
    }
};
// 3 bits: quad lane j owns row block j of the unit (a 96-bit run per column, field f at bit 3 f).  Every byte of the
// three words holds two whole fields, which two ANDs per word expose as q << p; the eight fields that straddle
// bytes (2 5 10 13 18 21 26 29) sit at the start of a byte after a shift of the run by 6 bits.  Nine registers hold
// the 32 fields (and four empty bytes):
//   R0 = w0 & A: f0 p0, f3 p1, f6 p2, f8 p0      R1 = w0 & B: f1 p3, f4 p4, f7 p5, f9 p3
//   R2 = w1 & A': f11 p1, f14 p2, f16 p0, f19 p1  R3 = w1 & B': f12 p4, f15 p5, f17 p3, f20 p4
//   R4 = w2 & A": f22 p2, f24 p0, f27 p1, f30 p2  R5 = w2 & B": f23 p5, f25 p3, f28 p4, f31 p5
//   R6 = (run >> 6)  : f2 p0, f5 p1, -, f10 p0    R7 = (run >> 38): f13 p1, -, f18 p0, f21 p1
//   R8 = (run >> 70) : -, f26 p0, f29 p1, -
// Step s multiplies (R[2s], R[2s+1]); the fifth step has only R8.
template <> struct IntLayout<3, true> {
    static constexpr int kSteps = 5, kPre = 5, kLoads = 3;
    __device__ static int load_row(int i, int j) { return 3 * j + i; }
    static constexpr uint32_t m(int p0, int p1, int p2, int p3) {
        return (p0 < 0 ? 0u : 7u << p0) | (p1 < 0 ? 0u : 7u << (8 + p1)) | (p2 < 0 ? 0u : 7u << (16 + p2)) |
               (p3 < 0 ? 0u : 7u << (24 + p3));
    }
    __device__ static void regs(const uint32_t (&w)[kLoads], uint32_t (&r)[2 * kSteps]) {
        r[0] = w[0] & m(0, 1, 2, 0); r[1] = w[0] & m(3, 4, 5, 3);
        r[2] = w[1] & m(1, 2, 0, 1); r[3] = w[1] & m(4, 5, 3, 4);
        r[4] = w[2] & m(2, 0, 1, 2); r[5] = w[2] & m(5, 3, 4, 5);
        r[6] = __funnelshift_r(w[0], w[1], 6) & m(0, 1, -1, 0);
        r[7] = __funnelshift_r(w[1], w[2], 6) & m(1, -1, 0, 1);
        r[8] = (w[2] >> 6) & m(-1, 0, 1, -1);
        r[9] = 0u;
    }
    // items 0..2 fill their step; item 3 holds the eight straddling fields, which fill steps 3 and 4
    __device__ static void item(int i, int j, int (&row)[8], int (&pre)[8]) {
        constexpr unsigned long long F0 = pack8({{0, 3, 6, 8, 1, 4, 7, 9}}), P0 = pack8({{0, 1, 2, 0, 3, 4, 5, 3}});
        constexpr unsigned long long F1 = pack8({{11, 14, 16, 19, 12, 15, 17, 20}}), P1 = pack8({{1, 2, 0, 1, 4, 5, 3, 4}});
        constexpr unsigned long long F2 = pack8({{22, 24, 27, 30, 23, 25, 28, 31}}), P2 = pack8({{2, 0, 1, 2, 5, 3, 4, 5}});
        constexpr unsigned long long F3 = pack8({{2, 5, 10, 13, 18, 21, 26, 29}}), P3 = pack8({{0, 1, 0, 1, 0, 1, 0, 1}});
        const unsigned long long f = i == 0 ? F0 : (i == 1 ? F1 : (i == 2 ? F2 : F3));
        const unsigned long long p = i == 0 ? P0 : (i == 1 ? P1 : (i == 2 ? P2 : P3));
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            row[e] = 32 * j + (int)((f >> (8 * e)) & 0xffu);
            pre[e] = 5 - (int)((p >> (8 * e)) & 0xffu);
        }
    }
};
// Byte planes of M rows of x: a unit's B operands [step][quad lane][4 row + plane][b0, b1], and per unit and row its factors and the
// sums of x, of the unit or of each 32 rows where these are scaled apart (floats).
template <int BITS> __host__ __device__ constexpr int int_unit_bytes(int M) { return (BITS == 3 ? 5 : 4) * 128 * M; }
__host__ __device__ constexpr int int_factors(int sub) { return sub == 1 ? 2 : 8; }
// Bits of |X|.  Shifted by up to kPre, X has to fit in four signed bytes: 30 - kPre at most.  4 bits take all of them, their fp16 form
// being exact products summed in fp32.  2 and 3 bits keep 22: their fp16 form subtracts sums of up to 1024 times x and is off by more.
__host__ __device__ constexpr int int_x_bits(int bits) { return bits == 4 ? 26 : 22; }
__host__ __device__ constexpr bool int_takes(int bits, int sub) { return bits == 4 || (bits != 8 && sub == 1); }

// How x meets the weights: several rows in fp16, every unit's x kept or a few units at a time in turn; one row in fp16; one or two rows as
// byte planes, one row with groups scaled apart in a form of its own.  (The first two in one form, with a branch per unit, were 3 % slower for
// nine rows and more; the last two 6 % for two rows.)
enum { kSeveral = 0, kOne = 1, kInt = 2, kTurns = 3, kIntOne = 4 };

struct StripPlan {
    int units;        // units of 128 rows along K (the last one may be cut)
    int strips;       // strips of 32 columns of the layer
    int per_cta;      // strips of a CTA
    int passes;       // it works on T strips at a time
    int ring;         // slots of a warp's ring
    int spg;          // 32-row steps per group
    int groups;
    unsigned int spg_inv;   // ceil(2^32 / spg)
    int rows_g;       // groups whose constants a slot holds
    int x_bufs;       // several rows of which x is not kept: places of a warp, 2..4, used in turn
    int gather;       // x is picked through x_perm from a copy of it in shared memory
    int xact;         // activation applied to x as it is read: 0 none, 1 SwiGLU, 2 ReLU
    int split;        // CTAs (a cluster) that share a strip, a run of units each
    int cta_units;    // units of a CTA, at most
    int others;       // where the first of them keeps the others' sums (bytes behind the place of its own)
};

// A slot: weights (1024-byte aligned for the swizzle), and in a second ring the scales [group][32 T] and the zero-point
// words of each group.  Rows of qzeros of 4 and 8 bits are whole 16-byte pieces: one box holds every group's, unless `apart` asks for a
// box per group (the host says when).  Of 2 and 3 bits a group's words start anywhere, a box per group starts up to three words early.
__host__ __device__ constexpr int slot_bytes(int bits, int T) { return (4 * bits * 128 * T + 1023) & ~1023; }
__host__ __device__ constexpr int zero_words(int bits, int T) { return bits % 4 == 0 ? T * bits : (T * bits + 3 + 3) & ~3; }
__host__ __device__ constexpr int zero_pitch(int bits, int T, bool apart) { return bits % 4 == 0 && !apart ? T * bits * 4 : (zero_words(bits, T) * 4 + 127) & ~127; }
__host__ __device__ constexpr int scale_bytes(int T, int rows) { return (rows * T * 64 + 127) & ~127; }
__host__ __device__ constexpr int const_bytes(int bits, int T, int rows, bool apart) { return scale_bytes(T, rows) + ((rows * zero_pitch(bits, T, apart) + 127) & ~127); }

// The two activations folded into the read of x, rounded exactly like the stand-alone kernel (b200gptq_act).
__device__ __forceinline__ uint32_t act_relu2(uint32_t v) {
    const float2 f = __half22float2(*reinterpret_cast<__half2*>(&v));
    const __half2 r = __floats2half2_rn(fmaxf(f.x, 0.f), fmaxf(f.y, 0.f));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t act_swiglu2(uint32_t gv, uint32_t uv) {
    const float2 g = __half22float2(*reinterpret_cast<__half2*>(&gv)), u = __half22float2(*reinterpret_cast<__half2*>(&uv));
    const float s0 = __half2float(__float2half_rn(g.x / (1.f + __expf(-g.x))));
    const float s1 = __half2float(__float2half_rn(g.y / (1.f + __expf(-g.y))));
    const __half2 r = __floats2half2_rn(s0 * u.x, s1 * u.y);
    return *reinterpret_cast<const uint32_t*>(&r);
}

// SUB: groups of a unit that are scaled apart (1: a group is a whole number of units).  NT: rows of x / 8.
// MODE: kSeveral, kTurns, kOne, kInt.  T: strips of a pass.  W: warps of a CTA.
// Registers: a second CTA of eight warps would fit on an SM where K is short and two to eight rows of x leave registers (128 and less), and
// the next launch's weights would arrive beside the current one.  That serves such a layer alone (1024 x 7168, 3 bits, two rows 3.1 us for
// 3.5), but two CTAs share an SM while others idle (1024 x 3072, 2 bits, three rows 2.6 us for 2.4), and with a small kernel before each layer,
// as in a decode step, it loses: 1024 x 7424, 4 bits, 8 rows 4.8 us for 4.1; a step of a decoder with hidden size 1024, batches of 4 and 8,
// 253 and 241 us for 237 and 232.  So these launches carry warps that end at once, for the registers they hold.  Sixteen warps, or
// sixteen rows of x, leave 4096 or 8192 of an SM's for the kernel that comes next.  With all of them taken, the gather of x between
// two products of 8 rows, 9216 x 9216, 3 bits, only started when a CTA ended, and the next product's weights after that: 22 us
// against 16.6 (and 14.3 against 14.1 where nothing is gathered).
__host__ __device__ constexpr int idle_warps(int W, bool kept, int nt) { return W == 8 && kept && nt == 1 ? 3 : 0; }
// APART: a box for the zero-points of each group.
// SPLIT: the layer has fewer strips than half the SMs, so that clusters of plan.split CTAs share one, a run of K each; they push their sums
// into the first one's shared memory, which adds them in their order.
template <int BITS, int SUB, int NT, int MODE, int T, int W, bool APART, bool SPLIT = false>
__global__ void __maxnreg__(W == 16 ? 120 : NT == 1 ? 168 : 224)
gemv_strip_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_s,
                  const __grid_constant__ CUtensorMap tmap_z, const __half* __restrict__ x,
                  const int32_t* __restrict__ x_perm, const __half* __restrict__ bias, __half* __restrict__ y, int M_rows, int K, int N, const StripPlan plan,
                  unsigned int* __restrict__ status) {
    using L = Layout<BITS, SUB == 1>;
    using I = IntLayout<BITS, SUB == 1 || BITS != 4>;
    constexpr bool ONE = MODE == kOne, PAIRED = MODE == kIntOne, INT = MODE == kInt || PAIRED, KEPT = MODE == kSeveral, TURNS = MODE == kTurns, ROWS = KEPT || TURNS;
    static_assert(!INT || (NT == 1 && int_takes(BITS, SUB)), "not a case of the integer path");
    static_assert(!PAIRED || (BITS == 4 && SUB == 4), "not a case of paired groups");
    constexpr int STRIP_BYTES = L::kRows * 128, STEPS = 4 / SUB, SLOT = slot_bytes(BITS, T);
    constexpr int NC = ROWS ? 2 : 1;             // rows of x per lane and n-tile that exist
    constexpr int COLS = T * kStripCols;
    extern __shared__ __align__(1024) uint8_t dsm[];
    __shared__ __align__(8) uint64_t bars[W * kMaxRing];

    const int M = ONE || PAIRED ? 1 : M_rows;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, j = lane & 3;
    if (idle_warps(W, KEPT, NT) && warp >= W) return;     // (before any barrier)
    const int R = plan.ring;
    // The runs start evenly over the columns and all have per_cta strips: neighbours may share a strip, both then write
    // the same bits.  (A grid of fewer, disjoint runs left SMs idle, and the next launch, which becomes resident beside
    // this one, put two of its CTAs on each of those: up to twice the time.)
    uint32_t rank = 0;
    if constexpr (SPLIT) {
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");     // (waited for before the sums are pushed: all have started)
    }
    const int strip0 = SPLIT ? (int)blockIdx.x / plan.split : min((int)(((long long)blockIdx.x * plan.strips) / gridDim.x), plan.strips - plan.per_cta);
    const int last_window = plan.per_cta - T;     // (so is the last pass's window)
    const int u_cta = SPLIT ? (int)rank * plan.units / plan.split : 0, n_cta = SPLIT ? ((int)rank + 1) * plan.units / plan.split - u_cta : plan.units;
    const int u_begin = u_cta + (warp * n_cta) / W, nu = u_cta + ((warp + 1) * n_cta) / W - u_begin;
    const int total = plan.passes * nu;           // boxes of this warp

    // shared memory: rings | x | sums of the warps, and in the same bytes: x as it lies in memory
    uint8_t* aligned = dsm + ((1024u - (smem_u32(dsm) & 1023u)) & 1023u);
    const int cbytes = const_bytes(BITS, T, plan.rows_g, APART);
    uint8_t* p_ring = aligned + (size_t)warp * R * SLOT;
    uint8_t* p_const = aligned + (size_t)W * R * SLOT + (size_t)warp * R * cbytes;
    uint8_t* base_x = aligned + (size_t)W * R * (SLOT + cbytes);
    // one row: [unit][quad lane][16 registers]; planes: [unit][step]..., then (factor, sum) [unit][row]; several rows:
    // [unit][row][natural halves], or a few units in turn per warp
    const int unit_x = ONE ? kUnit * 2 : (INT ? int_unit_bytes<BITS>(M) : M * kXPitch * 2);
    const int cta_units = SPLIT ? plan.cta_units : plan.units;
    const int x_units = TURNS ? plan.x_bufs * W : cta_units;
    uint8_t* p_x = base_x + (size_t)(TURNS ? plan.x_bufs * warp : u_begin - u_cta) * unit_x;
    constexpr int FACTORS = int_factors(SUB);
    float* p_f = reinterpret_cast<float*>(base_x + (size_t)cta_units * unit_x) + (size_t)(u_begin - u_cta) * M * FACTORS;
    uint8_t* base_r = base_x + (size_t)x_units * unit_x + (INT ? (cta_units * M * FACTORS * 4 + 15) / 16 * 16 : 0);
    float* red = reinterpret_cast<float*>(base_r);                                 // [warp][m][column of the pass]
    unsigned short* raw = reinterpret_cast<unsigned short*>(base_r);               // [m][k]
    const uint32_t bar0 = smem_u32(bars) + 8u * (warp * kMaxRing);
    bool ok = true;

    // ---- weights, scales and zero-points of a unit and pass ----
    const int zwords = N / 32 * BITS;
    auto group_at = [&](int step) -> int {        // (steps past K: their x is zero, any group will do)
        const int grp = plan.spg == 1 ? step : (int)__umulhi((unsigned int)step, plan.spg_inv);
        return min(grp, plan.groups - 1);
    };
    const uint32_t tx_bytes = T * STRIP_BYTES + plan.rows_g * (T * 64 + zero_words(BITS, T) * 4);
    int q_w = 0, u_w = 0, win_w = 0, slot_w = 0;  // next to request: number, unit, first strip of the pass, slot
    auto request = [&]() {
        const int grp = group_at(4 * (u_begin + u_w)), strip = strip0 + win_w;
        if (elect_one()) {
            const uint32_t bar = bar0 + 8u * slot_w, cst = smem_u32(p_const) + slot_w * cbytes;
            mbar_expect(bar, tx_bytes);
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                ::"r"(smem_u32(p_ring) + slot_w * SLOT), "l"(&tmap_w), "r"(0), "r"((u_begin + u_w) * L::kRows),
                  "r"(strip), "r"(bar) : "memory");
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                ::"r"(cst), "l"(&tmap_s), "r"(strip * kStripCols), "r"(grp), "r"(bar) : "memory");
            if constexpr (!APART) {
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                    ::"r"(cst + scale_bytes(T, plan.rows_g)), "l"(&tmap_z), "r"(strip * BITS), "r"(grp), "r"(bar) : "memory");
            } else {
                for (int r = 0; r < plan.rows_g; ++r)
                    asm volatile(
                        "cp.async.bulk.tensor.1d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2}], [%3];"
                        ::"r"(cst + scale_bytes(T, plan.rows_g) + r * zero_pitch(BITS, T, APART)), "l"(&tmap_z),
                          "r"(((grp + r) * zwords + strip * BITS) & ~3), "r"(bar) : "memory");
            }
        }
        ++q_w;
        if (++u_w == nu) { u_w = 0; win_w = min(win_w + T, last_window); }
        if (++slot_w == R) slot_w = 0;
    };
    if (elect_one()) {
        for (int s = 0; s < R; ++s) mbar_init(bar0 + 8u * s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    for (int i = 0; i < R && i < total; ++i) request();

    const bool gather = plan.gather != 0;
    // What does not need x is done before the wait.  Byte planes: which rows of a 128-row unit a lane takes.  A gather: where these,
    // or the rows of an item of the other modes, lie in x, in the bytes that the item itself (planes: its unit) is written to.  Looked
    // up after the wait, two units at a time, they were a round trip to L2 each: 9 units per warp, 9216 x 36864, 3 bits, 34.2 us
    // against 29.7.  Planes: the first two units' in registers, the others' copied without waiting; a CTA that starts late is on its
    // way to x meanwhile (3 bits, 4096 x 11008, two units per warp, through shared memory 8.6 against 8.4).
    int row[8], pre[8], first[8];
    auto index_slot = [&](int i) { return reinterpret_cast<uint4*>(INT ? p_x + (i >> 4) * unit_x + (i & 15) * 32 : p_x + i * 16); };
    auto pack2 = [](int a, int b) { return (uint32_t)a | ((uint32_t)b << 16); };
    if constexpr (INT) {
        I::item((lane >> 2) & 3, lane & 3, row, pre);
#pragma unroll
        for (int e = 0; e < 8; ++e) asm volatile("" : "+r"(row[e]), "+r"(pre[e]));
        if (gather) {
#pragma unroll
            for (int e = 0; e < 8; ++e) first[e] = __ldg(x_perm + min((u_begin + (lane >> 4)) * kUnit + row[e], K - 1));
            for (int i = lane + 32; i < nu * 16; i += 32) {
                const int k0 = (u_begin + (i >> 4)) * kUnit;
                const uint32_t dst = smem_u32(index_slot(i));
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * e), "l"(x_perm + min(k0 + row[e], K - 1)) : "memory");
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) asm volatile("" : "+r"(first[e]));
        }
    }
    constexpr bool BLOCKS = ONE && BITS == 3 && SUB == 1;
    // the two runs of four rows of item i of one row in fp16
    auto item_rows = [&](int i, int& ka, int& kb) {
        const int k = (u_begin + (i >> 4)) * kUnit, jj = (i >> 2) & 3, st = i & 3;
        if constexpr (BITS == 8) {
            ka = k + 4 * L::load_row(2 * st, jj); kb = k + 4 * L::load_row(2 * st + 1, jj);
        } else if constexpr (BITS != 3 || SUB != 1) {
            ka = k + L::x_first(st, jj); kb = ka + 4;
        }
    };
    if constexpr (ONE && !BLOCKS)
        if (gather) {
#pragma unroll 2
            for (int i = lane; i < nu * 16; i += 32) {
                int ka = 0, kb = 0;
                item_rows(i, ka, kb);
                const int4 a = __ldg(reinterpret_cast<const int4*>(x_perm + min(ka, K - 4)));
                const int4 b = __ldg(reinterpret_cast<const int4*>(x_perm + min(kb, K - 4)));
                *index_slot(i) = make_uint4(pack2(a.x, a.y), pack2(a.z, a.w), pack2(b.x, b.y), pack2(b.z, b.w));
            }
        }
    if constexpr (KEPT)
        if (gather) {                              // of several rows: in the place of the first row's four values
#pragma unroll 2
            for (int i = lane; i < nu * 32; i += 32) {
                const int4 a = __ldg(reinterpret_cast<const int4*>(x_perm + min(u_begin * kUnit + 4 * i, K - 4)));
                *reinterpret_cast<uint2*>(p_x + (size_t)(i >> 5) * unit_x + 8 * lane) = make_uint2(pack2(a.x, a.y), pack2(a.z, a.w));
            }
        }
    constexpr int EARLY = 4;
    uint4 first4[EARLY];
    if (BLOCKS && gather) {
#pragma unroll
        for (int e = 0; e < EARLY; ++e) {
            first4[e] = __ldg(reinterpret_cast<const uint4*>(x_perm + min((u_begin + e) * kUnit + 4 * lane, K - 4)));
            asm volatile("" : "+r"(first4[e].x), "+r"(first4[e].y), "+r"(first4[e].z), "+r"(first4[e].w));
        }
    }
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (gather)                                   // all of x, by all warps
        for (int i = tid; i < M * K / 8; i += 32 * W)
            cp_async16(smem_u32(raw + 8 * (size_t)i), x + 8 * (size_t)i, true);
    // One row, and planes of 2 and 3 bits: the warp's slice of x is copied first (`raw`), so that its rows can be picked in any order
    // without 2-byte requests from every CTA to the same few L2 lines (they cost 7 us at 9216 rows).
    const bool staged = gather || (!ROWS && !(INT && BITS == 4) && plan.xact != 1);
    if (!ROWS && !gather && staged) {
        const int k0 = u_begin * kUnit, count = min(nu * kUnit, K - k0) / 8;
        for (int m = 0; m < M; ++m)
            for (int i = lane; i < count; i += 32)
                cp_async16(smem_u32(raw + (size_t)m * K + k0 + 8 * i), x + (size_t)m * K + k0 + 8 * i, true);
    }
    if (staged) asm volatile("cp.async.commit_group;" ::: "memory");
    // four halves of row m of the copy of x, those of rows k .. k + 3 of K (zeros past K)
    auto pick4 = [&](int m, int k, const uint4& idx) -> uint2 {
        const unsigned short* rm = raw + (size_t)m * K;
        uint2 v = make_uint2((uint32_t)rm[idx.x] | ((uint32_t)rm[idx.y] << 16), (uint32_t)rm[idx.z] | ((uint32_t)rm[idx.w] << 16));
        if (k >= K) v = make_uint2(0u, 0u);
        if (plan.xact == 2) v = make_uint2(act_relu2(v.x), act_relu2(v.y));
        return v;
    };
    // four consecutive halves of row m at row k of K (k % 4 == 0; zeros past K)
    auto load4 = [&](int m, int k) -> uint2 {
        uint2 v = make_uint2(0u, 0u);
        if (k < K) {
            const unsigned short* rm = raw + (size_t)m * K;
            if (gather) {
                const uint4 idx = __ldg(reinterpret_cast<const uint4*>(x_perm + k));
                v.x = (uint32_t)rm[idx.x] | ((uint32_t)rm[idx.y] << 16);
                v.y = (uint32_t)rm[idx.z] | ((uint32_t)rm[idx.w] << 16);
            } else if (staged) {
                v = *reinterpret_cast<const uint2*>(rm + k);
            } else {
                const __half* px = x + (size_t)m * (plan.xact == 1 ? 2 * K : K) + k;
                v = __ldcg(reinterpret_cast<const uint2*>(px));
                if (plan.xact == 1) {
                    const uint2 up = __ldcg(reinterpret_cast<const uint2*>(px + K));
                    v = make_uint2(act_swiglu2(v.x, up.x), act_swiglu2(v.y, up.y));
                }
            }
            if (plan.xact == 2) v = make_uint2(act_relu2(v.x), act_relu2(v.y));
        }
        return v;
    };
    auto load_swiglu = [&](int m, int k) -> uint32_t {
        const unsigned short* px = reinterpret_cast<const unsigned short*>(x) + (size_t)m * 2 * K + k;
        return act_swiglu2(__ldcg(px), __ldcg(px + K)) & 0xffffu;
    };
    const bool async_x = ROWS && !gather && plan.xact == 0;
    auto fetch_x = [&](int u, int buf) {          // several rows, as they lie in memory
        const uint32_t dst = smem_u32(p_x) + buf * M * kXPitch * 2;
        for (int i = lane; i < 16 * M; i += 32) {
            const int m = i >> 4, e = 8 * (i & 15), k = (u_begin + u) * kUnit + e;
            cp_async16(dst + (m * kXPitch + e) * 2, x + (size_t)m * K + (k < K ? k : 0), k < K);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (KEPT && async_x)                      // (waited for unit by unit, in the first pass)
        for (int u = 0; u < nu; ++u) fetch_x(u, u);
    if (gather || (!ROWS && staged)) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (gather) __syncthreads();
        else __syncwarp();
    }
    if (KEPT && !async_x) {
        for (int i = lane; i < nu * 32; i += 32) {
            uint2* to = reinterpret_cast<uint2*>(p_x + (size_t)(i >> 5) * unit_x + 8 * lane);
            const int k = u_begin * kUnit + 4 * i;
            const uint2 at = *to;                  // (where a gather finds them)
            for (int m = 0; m < M; ++m)
                to[m * kXPitch / 4] = gather ? pick4(m, k, make_uint4(at.x & 0xffffu, at.x >> 16, at.y & 0xffffu, at.y >> 16)) : load4(m, k);
        }
        __syncwarp();
    }
    if constexpr (ONE) {
        // the warp's slice of x in the order of the B registers: piece (unit, quad lane, step) is four registers
        if constexpr (BITS == 3 && SUB == 1) {
            // a 32-row block at a time: its pairs cross the 8-row pieces.  A gather picks its rows with all lanes first, into the
            // bytes that the block is written back to.
            if (gather) {
                auto put = [&](int u, uint2 v) { *reinterpret_cast<uint2*>(p_x + u * kUnit * 2 + 8 * lane) = v; };
#pragma unroll
                for (int u = 0; u < EARLY; ++u)
                    if (u < nu) put(u, pick4(0, (u_begin + u) * kUnit + 4 * lane, first4[u]));
                for (int u = EARLY; u < nu; ++u) put(u, load4(0, (u_begin + u) * kUnit + 4 * lane));
                __syncwarp();
            }
            for (int i = lane; i < nu * 4; i += 32) {
                uint32_t xr[16], b[16];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const uint2 v = gather ? *reinterpret_cast<const uint2*>(p_x + i * 64 + 8 * e)
                                           : load4(0, u_begin * kUnit + 32 * i + 4 * e);
                    xr[2 * e] = v.x; xr[2 * e + 1] = v.y;
                }
                L::b_block(xr, b);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    *reinterpret_cast<uint4*>(p_x + i * 64 + 16 * e) = make_uint4(b[4 * e], b[4 * e + 1], b[4 * e + 2], b[4 * e + 3]);
            }
        } else {
#pragma unroll 2
            for (int i = lane; i < nu * 16; i += 32) {
                int ka = 0, kb = 0;
                item_rows(i, ka, kb);
                uint2 v, w;
                if (gather) {
                    const uint4 at = *index_slot(i);
                    v = pick4(0, ka, make_uint4(at.x & 0xffffu, at.x >> 16, at.y & 0xffffu, at.y >> 16));
                    w = pick4(0, kb, make_uint4(at.z & 0xffffu, at.z >> 16, at.w & 0xffffu, at.w >> 16));
                } else {
                    v = load4(0, ka); w = load4(0, kb);
                }
                uint32_t b[4];
                if constexpr (BITS == 8) {
                    b[0] = v.x; b[1] = v.y; b[2] = w.x; b[3] = w.y;
                } else {
                    L::b_regs(make_uint4(v.x, v.y, w.x, w.y), b);
                }
                *reinterpret_cast<uint4*>(p_x + i * 16) = make_uint4(b[0], b[1], b[2], b[3]);
            }
        }
        __syncwarp();
    }
    if constexpr (INT) {
        // Fixed point per unit, four signed byte planes; the 16 items of a unit sit in 16 adjacent lanes.  V pairs of units at a time,
        // or each waits out the other's latencies.
        auto planes = [&](int q0, auto count) {
            constexpr int V = decltype(count)::value;
            const int jq = lane & 3, iq = (lane >> 2) & 3;
            uint4 at[V][2];
            bool active[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                active[v] = q0 + 32 * v + lane < nu * 16;
                at[v][0] = at[v][1] = make_uint4(0u, 0u, 0u, 0u);
                if (gather && v == 0 && q0 == 0) {
                    at[0][0] = make_uint4(first[0], first[1], first[2], first[3]); at[0][1] = make_uint4(first[4], first[5], first[6], first[7]);
                } else if (gather && active[v]) { at[v][0] = index_slot(q0 + 32 * v + lane)[0]; at[v][1] = index_slot(q0 + 32 * v + lane)[1]; }
            }
            __syncwarp();
            for (int m = 0; m < M; ++m) {
                uint32_t h[V][8], mx[V];
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    const int k0 = (u_begin + ((q0 + 32 * v + lane) >> 4)) * kUnit;
                    const uint32_t idx[8] = {at[v][0].x, at[v][0].y, at[v][0].z, at[v][0].w, at[v][1].x, at[v][1].y, at[v][1].z, at[v][1].w};
                    if (gather || (BITS != 4 && staged)) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const uint32_t from = gather ? idx[e] : k0 + row[e];
                            h[v][e] = active[v] && k0 + row[e] < K ? raw[(size_t)m * K + from] : 0u;
                            if (plan.xact) h[v][e] = act_relu2(h[v][e]) & 0xffffu;
                        }
                    } else if constexpr (BITS == 4) {          // a run of eight rows
                        uint2 a = make_uint2(0u, 0u), b = a;
                        if (active[v]) { a = load4(m, k0 + row[0]); b = load4(m, k0 + row[0] + 4); }
                        const uint32_t x4[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            h[v][e] = e < 4 ? x4[e & 3] & 0xffffu : x4[e & 3] >> 16;
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) h[v][e] = active[v] && k0 + row[e] < K ? load_swiglu(m, k0 + row[e]) : 0u;
                    }
                    mx[v] = 0u;
#pragma unroll
                    for (int e = 0; e < 8; ++e) mx[v] = max(mx[v], h[v][e] & 0x7fffu);    // the order of non-negative fp16 numbers
                }
                constexpr int XB = int_x_bits(BITS);
                float scale[V];
                int ex[V], sum[V];
                bool bad[V];
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    // 2^ex > max |x| of the rows that share a factor; X = x * 2^(126 + XB - ex) has |X| < 2^XB.  Rows of zeros take any
                    // scale; rows with an infinity or a NaN get a NaN factor, so that their columns come out as NaN.
                    if constexpr (SUB == 1) {
                        const uint32_t lo = __reduce_max_sync(0xffffffffu, lane < 16 ? mx[v] : 0u), hi = __reduce_max_sync(0xffffffffu, lane < 16 ? 0u : mx[v]);
                        mx[v] = lane < 16 ? lo : hi;
                    } else {
#pragma unroll
                        for (int o = 1; o < 4; o <<= 1) mx[v] = max(mx[v], __shfl_xor_sync(0xffffffffu, mx[v], o));
                    }
                    ex[v] = (int)(__float_as_uint(__half2float(__ushort_as_half((unsigned short)mx[v]))) >> 23);
                    bad[v] = mx[v] >= 0x7c00u;
                    if (mx[v] == 0u || bad[v]) ex[v] = 127;
                    scale[v] = __uint_as_float((uint32_t)(253 + XB - ex[v]) << 23);
                }
                uint32_t dg[V][8];
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    sum[v] = 0;
                    // round to nearest; up to 22 bits through the fp32 adder.  (26 bits through it, in two steps: more code, 0.1 to 0.5 us
                    // a launch longer)
                    auto fixed = [&](int e) {
                        const float xf = __half2float(__ushort_as_half((unsigned short)h[v][e]));
                        return XB > 22 ? __float2int_rn(xf * scale[v]) : __float_as_int(fmaf(xf, scale[v], 12582912.f)) - 0x4B400000;
                    };
                    auto digits = [](int X) { return (uint32_t)(X + 0x00808080) ^ 0x00808080u; };   // four signed base-256 digits
                    if constexpr (BITS == 4 && SUB == 1) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {              // (|16 X - X'| < 2^30 + 2^26, which four digits hold)
                            const int lo = fixed(e), hi = fixed(e + 4);
                            sum[v] += lo + hi;
                            dg[v][e] = digits(lo * 16 - hi);
                            dg[v][e + 4] = digits(hi);
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const int X = fixed(e);
                            sum[v] += X;
                            dg[v][e] = digits(X << pre[e]);
                        }
                    }
                }
                // (the X of 128 rows of 22 bits, or of 32 rows of 26, add up to less than 2^31)
                constexpr int WHOLE_SUM = SUB == 4 || XB > 22 ? 4 : 16;
#pragma unroll
                for (int o = 1; o < WHOLE_SUM; o <<= 1)
#pragma unroll
                    for (int v = 0; v < V; ++v) sum[v] += __shfl_xor_sync(0xffffffffu, sum[v], o);
                float sumf[V];
#pragma unroll
                for (int v = 0; v < V; ++v) sumf[v] = (float)sum[v];
#pragma unroll
                for (int o = WHOLE_SUM; o < (SUB == 1 ? 16 : 4); o <<= 1)
#pragma unroll
                    for (int v = 0; v < V; ++v) sumf[v] += __shfl_xor_sync(0xffffffffu, sumf[v], o);
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    if (!active[v]) continue;
                    const int u = (q0 + 32 * v + lane) >> 4;
                    const float delta = __uint_as_float((uint32_t)(ex[v] + 1 - XB) << 23);   // 2^(ex - 126 - XB)
                    const float factor = bad[v] ? __uint_as_float(0x7fc00000u) : __uint_as_float((uint32_t)(ex[v] + 1 - XB - I::kPre) << 23);
                    float* f = p_f + (u * M + m) * FACTORS;
                    if (SUB == 1 ? (lane & 15) == 0 : jq == 0) {       // factor of the planes and minus the sum of x, or four of each
                        f[SUB == 1 ? 0 : iq] = factor;
                        f[SUB == 1 ? 1 : 4 + iq] = -delta * sumf[v];
                    }
                    uint8_t* dst = p_x + (size_t)u * unit_x + jq * (32 * M) + m * 32;
                    auto store = [&](int step, const uint32_t (&lo)[4], const uint32_t (&hi)[4]) {
                        uint4* d = reinterpret_cast<uint4*>(dst + step * 4 * (32 * M));
                        d[0] = make_uint4(lo[0], hi[0], lo[1], hi[1]);
                        d[1] = make_uint4(lo[2], hi[2], lo[3], hi[3]);
                    };
                    uint32_t lo[4], hi[4];
                    if (BITS != 3 || iq < 3) {
                        planes_of(dg[v][0], dg[v][1], dg[v][2], dg[v][3], lo);
                        planes_of(dg[v][4], dg[v][5], dg[v][6], dg[v][7], hi);
                        store(iq, lo, hi);
                    } else {
                        planes_of(dg[v][0], dg[v][1], 0, dg[v][2], lo);
                        planes_of(dg[v][3], 0, dg[v][4], dg[v][5], hi);
                        store(3, lo, hi);
                        planes_of(0, dg[v][6], dg[v][7], 0, lo);
                        hi[0] = hi[1] = hi[2] = hi[3] = 0u;
                        store(4, lo, hi);
                    }
                }
            }
        };
        int q0 = 0;
        for (; q0 + 32 < nu * 16; q0 += 64) planes(q0, std::integral_constant<int, 2>{});
        if (q0 < nu * 16) planes(q0, std::integral_constant<int, 1>{});
        __syncwarp();
    }
    // planes: quad lane j holds planes 2j, 2j+1 of row j >> 1 ... of one row only j < 2; the zero-point term goes to one lane
    const float plane_weight = INT && (j >> 1) < M ? (j & 1 ? 65536.f : 1.f) : 0.f;
    const float sum_weight = INT && (j >> 1) < M && !(j & 1) ? 1.f : 0.f;

    float out[T][NT][4][NC];                      // columns 4g .. 4g+3 of a strip: rows 2j (, 2j+1) of x, or a pair of planes
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int r = 0; r < 4 * NC; ++r) out[t][nt][r / NC][r % NC] = 0.f;

    // byte offset of the lane's four columns of a word-row of strip t (swizzle: 16-byte piece p of line l sits at p ^ (l & 7))
    auto read_at = [&](int t, int row) {
        return (t * STRIP_BYTES + row * 128 + ((g ^ (row & 7)) << 4)) ^ (((t * L::kRows) & 7) << 4);
    };
    static_assert(L::kRows % 4 == 0, "strips start on lines 0 or 4 of the swizzle pattern");

    int slot = 0, parity = 0, buf = 0;
    if (TURNS && async_x && nu > 0)          // x that is not kept: x_bufs - 1 units (no more than nu) ahead
        for (int i = 0; i < plan.x_bufs - 1; ++i) fetch_x(i, i);
    for (int p = 0, win = 0; p < plan.passes; ++p, win = min(win + T, last_window)) {
#pragma unroll 1
        for (int u = 0; u < nu; ++u) {
            const uint8_t* src = p_ring + slot * SLOT;
            // this lane's scales and the strips' zero-points, of the unit's first group
            const int step0 = 4 * (u_begin + u), grp0 = group_at(step0);
            const uint8_t* csc = p_const + slot * cbytes + 8 * g;
            const uint8_t* cze = p_const + slot * cbytes + scale_bytes(T, plan.rows_g);
            auto zero_at = [&](int r, int t) {
                const int early = BITS % 4 == 0 ? 0 : ((grp0 + r) * zwords + (strip0 + win) * BITS) & 3;
                return cze + r * zero_pitch(BITS, T, APART) + 4 * early + t * BITS * 4;
            };
            if constexpr (PAIRED) {
                // One row, groups of 32 rows scaled apart: its planes are four of the eight columns of B.  Two groups share a product: the
                // first one's planes are columns 0..3 and lie along its first 16 rows of K, the second one's 4..7 and along the others,
                // zeros elsewhere; A has half of each group's rows.  As many products, and what follows them is done for two groups
                // at once, by lanes that had nothing to do: quad lanes 0, 1 hold the first group's planes, 2, 3 the second one's.
                uint2 bq[2];
                float cf[2], sx[2];
                int r[2];
                const float* f = p_f + u * FACTORS;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    bq[q] = *reinterpret_cast<const uint2*>(p_x + (size_t)u * unit_x + ((2 * q + (g >> 2)) * 4 + j) * 32 + (g & 3) * 8);
                    const int sub = 2 * q + (j >> 1);
                    cf[q] = j & 1 ? f[sub] * 65536.f : f[sub];
                    sx[q] = j & 1 ? 0.f : f[4 + sub];
                    r[q] = group_at(step0 + sub) - grp0;
                }
                mbar_wait(bar0 + 8u * slot, parity, ok);
#pragma unroll
                for (int t = 0; t < T; ++t) {
                    uint32_t w[4][I::kLoads];
#pragma unroll
                    for (int i = 0; i < I::kLoads; ++i) {
                        const uint4 v = *reinterpret_cast<const uint4*>(src + read_at(t, I::load_row(i, j)));
                        w[0][i] = v.x; w[1][i] = v.y; w[2][i] = v.z; w[3][i] = v.w;
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const uint2 sv = *reinterpret_cast<const uint2*>(csc + (r[q] * T + t) * 64);
                        const float2 s01 = __half22float2(*reinterpret_cast<const __half2*>(&sv.x));
                        const float2 s23 = __half22float2(*reinterpret_cast<const __half2*>(&sv.y));
                        const float sf[4] = {s01.x, s01.y, s23.x, s23.y};
                        const uint32_t zv = load_zeros<BITS>(zero_at(r[q], t), 4 * g);
                        const uint32_t lo0 = g < 4 ? bq[q].x : 0u, lo1 = g < 4 ? 0u : bq[q].x, hi0 = g < 4 ? bq[q].y : 0u, hi1 = g < 4 ? 0u : bq[q].y;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            constexpr int kBias = 0x4B400000;
                            int d[4] = {kBias, kBias, kBias, kBias};
                            const uint32_t a0 = w[2 * h][2 * q], a1 = w[2 * h + 1][2 * q], a2 = w[2 * h][2 * q + 1], a3 = w[2 * h + 1][2 * q + 1];
                            imma(d, d, a0 & 0x0f0f0f0fu, a1 & 0x0f0f0f0fu, a2 & 0x0f0f0f0fu, a3 & 0x0f0f0f0fu, lo0, lo1);
                            imma(d, d, a0 & 0xf0f0f0f0u, a1 & 0xf0f0f0f0u, a2 & 0xf0f0f0f0u, a3 & 0xf0f0f0f0u, hi0, hi1);
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                const float zf = __uint_as_float(0x4B000000u | ((zv >> (BITS * (2 * h + c))) & ((1u << BITS) - 1u))) - 8388607.f;
                                const float lo = __int_as_float(d[2 * c]) - 12582912.f, hi = __int_as_float(d[2 * c + 1]) - 12582912.f;
                                out[t][0][2 * h + c][0] = fmaf(sf[2 * h + c], fmaf(fmaf(256.f, hi, lo), cf[q], zf * sx[q]), out[t][0][2 * h + c][0]);
                            }
                        }
                    }
                }
            } else if constexpr (INT) {
                uint2 bx[I::kSteps];
#pragma unroll
                for (int s = 0; s < I::kSteps; ++s) {
                    bx[s] = make_uint2(0u, 0u);
                    if (g < 4 * M) bx[s] = *reinterpret_cast<const uint2*>(p_x + (size_t)u * unit_x + (s * 4 + j) * (32 * M) + g * 8);
                }
                const float* f = p_f + (u * M + (M == 2 ? j >> 1 : 0)) * FACTORS;
                float cf[SUB], sx[SUB];
                if constexpr (SUB == 1) {
                    const float2 v = *reinterpret_cast<const float2*>(f);
                    cf[0] = v.x * plane_weight; sx[0] = v.y * sum_weight;
                } else {
                    const float4 c = *reinterpret_cast<const float4*>(f), v = *reinterpret_cast<const float4*>(f + 4);
                    cf[0] = c.x * plane_weight; cf[1] = c.y * plane_weight; cf[2] = c.z * plane_weight; cf[3] = c.w * plane_weight;
                    sx[0] = v.x * sum_weight; sx[1] = v.y * sum_weight; sx[2] = v.z * sum_weight; sx[3] = v.w * sum_weight;
                }
                mbar_wait(bar0 + 8u * slot, parity, ok);
#pragma unroll
                for (int t = 0; t < T; ++t) {
                    uint32_t w[4][I::kLoads];
#pragma unroll
                    for (int i = 0; i < I::kLoads; ++i) {
                        const uint4 v = *reinterpret_cast<const uint4*>(src + read_at(t, I::load_row(i, j)));
                        w[0][i] = v.x; w[1][i] = v.y; w[2][i] = v.z; w[3][i] = v.w;
                    }
                    constexpr int SSTEPS = I::kSteps / SUB;
#pragma unroll
                    for (int sub = 0; sub < SUB; ++sub) {
                        const int r = SUB == 1 ? 0 : group_at(step0 + sub) - grp0;
                        const uint2 sv = *reinterpret_cast<const uint2*>(csc + (r * T + t) * 64);
                        const float2 s01 = __half22float2(*reinterpret_cast<const __half2*>(&sv.x));
                        const float2 s23 = __half22float2(*reinterpret_cast<const __half2*>(&sv.y));
                        const float sf[4] = {s01.x, s01.y, s23.x, s23.y};
                        const uint32_t zv = load_zeros<BITS>(zero_at(r, t), 4 * g);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t ra[2 * I::kSteps], rb[2 * I::kSteps];
                            I::regs(w[2 * h], ra);
                            I::regs(w[2 * h + 1], rb);
                            float zf[2];
#pragma unroll
                            for (int c = 0; c < 2; ++c)
                                zf[c] = __uint_as_float(0x4B000000u | ((zv >> (BITS * (2 * h + c))) & ((1u << BITS) - 1u))) - 8388607.f;
                            // the sums start at the bits of 1.5 * 2^23: |sum| < 2^22, so they end as floats with that offset
                            constexpr int kBias = 0x4B400000;
                            int d[4] = {kBias, kBias, kBias, kBias};
#pragma unroll
                            for (int s = sub * SSTEPS; s < (sub + 1) * SSTEPS; ++s)
                                imma(d, d, ra[2 * s], rb[2 * s], ra[2 * s + 1], rb[2 * s + 1], bx[s].x, bx[s].y);
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                const float lo = __int_as_float(d[2 * c]) - 12582912.f, hi = __int_as_float(d[2 * c + 1]) - 12582912.f;
                                out[t][0][2 * h + c][0] = fmaf(sf[2 * h + c], fmaf(fmaf(256.f, hi, lo), cf[sub], zf[c] * sx[sub]), out[t][0][2 * h + c][0]);
                            }
                        }
                    }
                }
            } else {
            // ---- B registers: 4 steps x 2 products x 2, per n-tile ----
            uint32_t b[NT][16];
            if constexpr (ONE) {
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    uint4 v = make_uint4(0u, 0u, 0u, 0u);
                    if (g == 0) v = *reinterpret_cast<const uint4*>(p_x + (u * 4 + j) * 64 + 16 * s);
                    b[0][4 * s] = v.x; b[0][4 * s + 1] = v.y; b[0][4 * s + 2] = v.z; b[0][4 * s + 3] = v.w;
                }
            } else {
                __half* xs = reinterpret_cast<__half*>(p_x + (size_t)(KEPT ? u : buf) * unit_x);
                if constexpr (KEPT) {
                    if (async_x && p == 0) {
                        // this unit's x; the copies of those behind it go on (8 rows of 4096 x 12288: all of x first 10.1 us, so 9.2)
                        const int behind = nu - 1 - u;
                        if (behind >= 4) asm volatile("cp.async.wait_group 4;" ::: "memory");
                        else if (behind == 3) asm volatile("cp.async.wait_group 3;" ::: "memory");
                        else if (behind == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
                        else if (behind == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
                        else asm volatile("cp.async.wait_group 0;" ::: "memory");
                        __syncwarp();
                    }
                } else {
                    if (async_x) {
                        if (plan.x_bufs == 4) asm volatile("cp.async.wait_group 2;" ::: "memory");
                        else if (plan.x_bufs == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
                        else asm volatile("cp.async.wait_group 0;" ::: "memory");
                        __syncwarp();
                        // into the place of the unit before this one; also for the next pass
                        const int ahead = u + plan.x_bufs - 1, to = buf == 0 ? plan.x_bufs - 1 : buf - 1;
                        if (ahead < nu || p + 1 < plan.passes) fetch_x(ahead < nu ? ahead : ahead - nu, to);
                        else asm volatile("cp.async.commit_group;" ::: "memory");    // keeps the count of groups
                    } else {
                        for (int m = 0; m < M; ++m)
                            *reinterpret_cast<uint2*>(xs + m * kXPitch + 4 * lane) = load4(m, (u_begin + u) * kUnit + 4 * lane);
                        __syncwarp();
                    }
                    if (++buf == plan.x_bufs) buf = 0;
                }
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const int m = 8 * nt + g;
                    const bool has = m < M;
                    const __half* xm = xs + m * kXPitch;
                    if constexpr (BITS == 8) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            uint2 v = make_uint2(0u, 0u);
                            if (has) v = *reinterpret_cast<const uint2*>(xm + 4 * L::load_row(i, j));
                            b[nt][2 * i] = v.x; b[nt][2 * i + 1] = v.y;
                        }
                    } else if constexpr (BITS == 3 && SUB == 1) {
                        uint32_t xr[16];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            uint4 v = make_uint4(0u, 0u, 0u, 0u);
                            if (has) v = *reinterpret_cast<const uint4*>(xm + 32 * j + 8 * i);
                            xr[4 * i] = v.x; xr[4 * i + 1] = v.y; xr[4 * i + 2] = v.z; xr[4 * i + 3] = v.w;
                        }
                        L::b_block(xr, b[nt]);
                    } else {
#pragma unroll
                        for (int s = 0; s < 4; ++s) {
                            uint4 v = make_uint4(0u, 0u, 0u, 0u);
                            if (has) v = *reinterpret_cast<const uint4*>(xm + L::x_first(s, j));
                            uint32_t bb[4];
                            L::b_regs(v, bb);
#pragma unroll
                            for (int i = 0; i < 4; ++i) b[nt][4 * s + i] = bb[i];
                        }
                    }
                }
            }
            // ---- per group: sum of x (rows 0..7 of the product) and what the powers of two contribute (rows 8..15) ----
            float sx[SUB][NT][NC], sm[SUB][NT][NC];
#pragma unroll
            for (int sub = 0; sub < SUB; ++sub)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    float d[2][4] = {};
                    constexpr uint32_t one = 0x3c003c00u;
#pragma unroll
                    for (int s = sub * STEPS; s < (sub + 1) * STEPS; ++s) {
                        mma(d[0], one, L::magic(s, 0), one, L::magic(s, 1), b[nt][4 * s], b[nt][4 * s + 1]);
                        mma(d[1], one, L::magic(s, 2), one, L::magic(s, 3), b[nt][4 * s + 2], b[nt][4 * s + 3]);
                    }
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        sx[sub][nt][c] = (d[0][c] + d[1][c]) * (-1.f / L::kScale);
                        sm[sub][nt][c] = d[0][2 + c] + d[1][2 + c];
                    }
                }
            mbar_wait(bar0 + 8u * slot, parity, ok);
#pragma unroll
            for (int t = 0; t < T; ++t) {
                uint4 wv[L::kLoads];
#pragma unroll
                for (int i = 0; i < L::kLoads; ++i) wv[i] = *reinterpret_cast<const uint4*>(src + read_at(t, L::load_row(i, j)));
#pragma unroll
                for (int sub = 0; sub < SUB; ++sub) {
                    float d[2][2][NT][4] = {};      // [pair of columns][product]
#pragma unroll
                    for (int s = sub * STEPS; s < (sub + 1) * STEPS; ++s) {
                        constexpr int PER = L::kPer == 0 ? L::kLoads : L::kPer;
                        uint32_t w[4][PER];
#pragma unroll
                        for (int i = 0; i < PER; ++i) {
                            const uint4& v = wv[L::kPer == 0 ? i : s * PER + i];
                            w[0][i] = v.x; w[1][i] = v.y; w[2][i] = v.z; w[3][i] = v.w;
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t a0[4], a1[4];
                            L::a_regs(w[2 * h], s, j, a0);
                            L::a_regs(w[2 * h + 1], s, j, a1);
#pragma unroll
                            for (int nt = 0; nt < NT; ++nt) {
                                mma(d[h][0][nt], a0[0], a1[0], a0[1], a1[1], b[nt][4 * s], b[nt][4 * s + 1]);
                                mma(d[h][1][nt], a0[2], a1[2], a0[3], a1[3], b[nt][4 * s + 2], b[nt][4 * s + 3]);
                            }
                        }
                    }
                    const int r = SUB == 1 ? 0 : group_at(step0 + sub * STEPS) - grp0;
                    const uint2 sv = *reinterpret_cast<const uint2*>(csc + (r * T + t) * 64);
                    const float2 s01 = __half22float2(*reinterpret_cast<const __half2*>(&sv.x));
                    const float2 s23 = __half22float2(*reinterpret_cast<const __half2*>(&sv.y));
                    const float sf[4] = {s01.x, s01.y, s23.x, s23.y};
                    const uint32_t zv = load_zeros<BITS>(zero_at(r, t), 4 * g);
                    float zf[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c)      // zero = field + 1
                        zf[c] = __uint_as_float(0x4B000000u | ((zv >> (BITS * c)) & ((1u << BITS) - 1u))) - 8388607.f;
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int c = 0; c < 4; ++c)
#pragma unroll
                            for (int r = 0; r < NC; ++r) {
                                const int e = 2 * (c & 1) + r;
                                const float v0 = d[c >> 1][0][nt][e], v1 = d[c >> 1][1][nt][e];
                                float v = L::kMul1 == 1.f ? v0 + v1 : fmaf(v1, L::kMul1, v0);
                                if (L::kMagic) v -= sm[sub][nt][r];
                                v = fmaf(zf[c], sx[sub][nt][r], v);
                                out[t][nt][c][r] = fmaf(sf[c], v, out[t][nt][c][r]);
                            }
                }
            }
            }
            __syncwarp();                          // the slot has been read by every lane
            if (q_w < total) request();
            if (++slot == R) { slot = 0; parity ^= 1; }
        }
        // ---- the warps' sums of this pass: four columns of every strip, rows 2j, 2j+1 of x ----
        __syncthreads();                           // the copy of x, or the previous pass's sums, have been read
        if constexpr (INT) {
#pragma unroll
            for (int t = 0; t < T; ++t) {
                float v[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    v[c] = out[t][0][c][0] + __shfl_xor_sync(0xffffffffu, out[t][0][c][0], 1);   // the row's other planes
                    if (PAIRED) v[c] += __shfl_xor_sync(0xffffffffu, v[c], 2);         // the other groups
                    out[t][0][c][0] = 0.f;
                }
                if (!(j & 1) && (j >> 1) < M)
                    *reinterpret_cast<float4*>(red + ((size_t)warp * M + (j >> 1)) * COLS + t * kStripCols + 4 * g) =
                        make_float4(v[0], v[1], v[2], v[3]);
            }
        } else
#pragma unroll
        for (int t = 0; t < T; ++t)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int r = 0; r < NC; ++r) {
                    const int m = 8 * nt + 2 * j + r;
                    if (m < M)
                        *reinterpret_cast<float4*>(red + ((size_t)warp * M + m) * COLS + t * kStripCols + 4 * g) =
                            make_float4(out[t][nt][0][r], out[t][nt][1][r], out[t][nt][2][r], out[t][nt][3][r]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) out[t][nt][c][r] = 0.f;
                }
        __syncthreads();
        const int n0 = (strip0 + win) * kStripCols;
        float2* others = nullptr;
        if constexpr (SPLIT) {
            // (one pass) the sums of the cluster's other CTAs, [CTA - 1][m][column]
            others = reinterpret_cast<float2*>(base_r + plan.others);
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            if (rank != 0)
                for (int i = tid; i < M * (COLS / 2); i += 32 * W) {
                    const int m = i / (COLS / 2), c = 2 * (i % (COLS / 2));
                    float2 v = make_float2(0.f, 0.f);
#pragma unroll
                    for (int w = 0; w < W; ++w) {
                        const float2 r = *reinterpret_cast<const float2*>(red + ((size_t)w * M + m) * COLS + c);
                        v.x += r.x; v.y += r.y;
                    }
                    uint32_t to;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(smem_u32(others + (rank - 1) * M * (COLS / 2) + i)), "r"(0));
                    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(to), "f"(v.x), "f"(v.y) : "memory");
                }
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            if (rank != 0) break;
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        for (int i = tid; i < M * (COLS / 2); i += 32 * W) {
            const int m = i / (COLS / 2), c = 2 * (i % (COLS / 2));
            float2 v = make_float2(0.f, 0.f);
#pragma unroll
            for (int w = 0; w < W; ++w) {
                const float2 r = *reinterpret_cast<const float2*>(red + ((size_t)w * M + m) * COLS + c);
                v.x += r.x; v.y += r.y;
            }
            if constexpr (SPLIT)
                for (int r = 0; r < plan.split - 1; ++r) {
                    const float2 o = others[r * M * (COLS / 2) + i];
                    v.x += o.x; v.y += o.y;
                }
            if (!INT) { v.x *= L::kScale; v.y *= L::kScale; }
            if (bias) {
                v.x += __half2float(bias[n0 + c]);
                v.y += __half2float(bias[n0 + c + 1]);
            }
            *reinterpret_cast<__half2*>(y + (size_t)m * N + n0 + c) = __floats2half2_rn(v.x, v.y);
        }
    }
    if (!ok) atomicExch(status + kStatusWord, 1u);
}

// The instantiation for (groups scaled apart in a unit, mode, rows of x / 8, strips of a pass, warps, zero-points in a box each, CTAs that share a
// strip), nullptr where there is none.
template <int BITS, int SUB, int NT, int MODE, int W>
const void* strip_kernel_t(int T, bool apart, bool split) {
    constexpr bool APART = BITS % 4 != 0;
    if constexpr (BITS == 4 && SUB == 4)
        if (T == 1 && apart && !split) return reinterpret_cast<const void*>(gemv_strip_kernel<BITS, SUB, NT, MODE, 1, W, true>);
    if (apart != APART) return nullptr;
    if (split) return T == 1 ? reinterpret_cast<const void*>(gemv_strip_kernel<BITS, SUB, NT, MODE, 1, W, APART, true>) : nullptr;
    if (T == 1) return reinterpret_cast<const void*>(gemv_strip_kernel<BITS, SUB, NT, MODE, 1, W, APART>);
    if (T == 2) return reinterpret_cast<const void*>(gemv_strip_kernel<BITS, SUB, NT, MODE, 2, W, APART>);
    if constexpr (NT == 1 && SUB == 1)
        if (T == 3) return reinterpret_cast<const void*>(gemv_strip_kernel<BITS, SUB, NT, MODE, 3, W, APART>);
    if constexpr (MODE == kInt && SUB == 1)
        if (T == 4) return reinterpret_cast<const void*>(gemv_strip_kernel<BITS, SUB, NT, MODE, 4, W, APART>);
    return nullptr;
}
template <int BITS, int SUB, int W>
const void* strip_kernel_m(int mode, int nt, int T, bool apart, bool split) {
    if constexpr (int_takes(BITS, SUB))
        if (mode == kInt) return strip_kernel_t<BITS, SUB, 1, kInt, W>(T, apart, split);
    if constexpr (BITS == 4 && SUB == 4)
        if (mode == kIntOne) return strip_kernel_t<BITS, SUB, 1, kIntOne, W>(T, apart, split);
    if (mode == kOne) return strip_kernel_t<BITS, SUB, 1, kOne, W>(T, apart, split);
    if (nt == 1)
        return mode == kTurns ? strip_kernel_t<BITS, SUB, 1, kTurns, W>(T, apart, split) : strip_kernel_t<BITS, SUB, 1, kSeveral, W>(T, apart, split);
    if constexpr (W == 8)
        return mode == kTurns ? strip_kernel_t<BITS, SUB, 2, kTurns, W>(T, apart, split) : strip_kernel_t<BITS, SUB, 2, kSeveral, W>(T, apart, split);
    return nullptr;
}
template <int BITS>
const void* strip_kernel_bits(int sub, int mode, int nt, int T, int warps, bool apart, bool split) {
    if (warps == 8) return sub == 1 ? strip_kernel_m<BITS, 1, 8>(mode, nt, T, apart, split) : strip_kernel_m<BITS, 4, 8>(mode, nt, T, apart, split);
    return sub == 1 ? strip_kernel_m<BITS, 1, 16>(mode, nt, T, apart, split) : strip_kernel_m<BITS, 4, 16>(mode, nt, T, apart, split);
}

}  // namespace

}  // namespace b200gptq
