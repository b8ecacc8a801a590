// The decoder layers of one decode step of one sequence in ONE launch.
//
// Launched one by one, a layer of such a step is eight kernels of 2.6 to 10 us (Llama-7B: 40 us a layer) whose weights need
// 16 us of HBM time: every launch waits for x, starts its weight rings, works through them and sums up, and while it does one of
// these the others rest.  Here one CTA per SM stays for the whole step:
//
//  * A producer warp streams this CTA's weights of ALL linears of ALL layers, in the order they will be needed, through one
//    ring of tensor boxes.  It depends on nothing but free slots, so the ring (170 KB per SM, 25 MB: the projection q|k|v of Llama-7B)
//    fills while the CTAs exchange x, normalise, attend and add up.  Tensor maps of the next linear are prefetched; a warp
//    of its own acquires them, layers ahead.  A slot is one strip of
//    32 columns times 16 units of 128 rows with the units' scales and zero-points: one box each, one barrier for the CTA (a ring per warp,
//    as in gemv_strip.cuh, needs 16 times the boxes).
//  * Eight warps multiply, two units of every slot each, as gemv_strip.cuh's byte planes do (x in fixed point per unit, exact integer
//    products, scaled in fp32), and are added up through shared memory.  Two slots at a time: one alone is a chain of latencies.
//  * What lies between the linears is done where the values are: residual sums and the activation by the warp that adds up a
//    strip; the norm, the act-order gather and the planes by every CTA as it reads x; attention by up to sixteen CTAs per head.
//  * Values travel between CTAs as words that carry the number of their phase (put_word), so there is no barrier of the grid and
//    no fence: a layer is five such exchanges.  All CTAs are resident (cooperative launch); every wait is bounded, and one
//    that expires raises the sticky status word and ends the launch with undefined results.
//
// us per layer with the kernels one by one -> here (a graph of the step; what 12 more layers take, / 12, so without the projection
// to the vocabulary), 4 bits unless said: Llama-7B, 512 positions 39.5 -> 35.4, 200 positions 38.5 -> 33.8, 3 bits 44.5 -> 39.9, act-order 41.3 -> 36.2;
// hidden 1024, inter 2816, 100 positions 21.0 -> 15.3; hidden 2048, inter 5504, 200 positions 24.0 -> 20.5; OPT, hidden 2048, inter 8192, 300 positions
// 23.8 -> 21.2, 3 bits act-order 27.8 -> 26.1 (16 layers of hidden 2048 and less lie in L2).  When a Llama-7B layer took 36.7, the weights
// alone streamed in 18.4 and the exchanges without the products took 30: what bounds it is their latency, five times read, norm,
// planes, sum and write.  Where the kernels one by one are faster: one_launch_pays (decoder.py).  Several sequences are left to these:
// in the fp16 form of the products a step of two took 58 us a layer for 52.
#include <cstring>
#include <new>

#include "gemv_strip.cuh"

namespace b200gptq {

namespace {

constexpr int kLayerWarps = 8, kLayerThreads = 32 * (kLayerWarps + 4);      // (registers are dealt to groups of four warps)
// Of the 65 536 registers 12 warps are launched with 168 each; the four of the producer give up what the others take.  A value in local
// memory costs an L2 round trip here, the shared memory leaves next to no cache.
constexpr int kLaunchRegs = 168, kMoreRegs = 232, kFewRegs = 24;
static_assert(kLayerWarps * 32 * kMoreRegs + 128 * kFewRegs <= kLayerThreads * kLaunchRegs, "the launch has these registers");
constexpr int kSlotUnits = 2 * kLayerWarps;         // units of 128 rows in a slot: two per warp
constexpr int kPasses = 3;                          // slots whose x is fetched at once; of a normalised x, all
constexpr int kMaxSlots = 8;
constexpr int kMaxSplit = 16, kPartsAtOnce = 3;     // CTAs that share a head; parts of it that are fetched at once
enum { kQkv = 0, kOut = 1, kUp = 2, kDown = 3 };

// Bytes of a slot's weights and constants.  Zero-points: rows of 4 bits are one 16-byte piece per strip; 3 (2) bits are three (two)
// words that start up to three (two) words behind a 16-byte boundary.
constexpr int slot_weights(int bits) { return kSlotUnits * 4 * bits * 128; }
constexpr int slot_zero_words(int bits) { return bits == 3 ? 8 : 4; }
constexpr int slot_scales() { return kSlotUnits * 64; }
constexpr int slot_consts(int bits) { return slot_scales() + kSlotUnits * slot_zero_words(bits) * 4; }

struct alignas(128) StepPointers {
    const __half* bias[4];
    const int32_t* perm[3];         // rows of x that q|k|v, o and up read in order (null: as they lie)
    const __half *norm_w[2], *norm_b[2];
    __half *k_cache, *v_cache;
};
static_assert(sizeof(StepPointers) == 128, "copied in 16-byte pieces");
struct alignas(128) StepLayer {
    CUtensorMap w[4], s[4], z[4];
    StepPointers at;
};

struct LinearShape {
    int K, units, slots;            // rows, units of 128, slots per strip
    int strips, pair;               // strips of the layer; > 0: strips come in pairs, this many apart (gate | up)
    int items;                      // strips or pairs: what is dealt to the CTAs
    int per_group;                  // units per group
    unsigned int per_group_inv;     // ceil(2^32 / per_group)
    int zero_words;                 // of a row of qzeros
};

struct StepParams {
    const StepLayer* layers;
    int n_layers, hidden, heads, inter, max_seq;
    int gated, rms, rope;
    float eps, scale, inv_hidden;
    const __half *cos_t, *sin_t;
    const long long* pos;
    __half* x;                             // residual
    uint32_t *xw, *qkv, *att, *act;        // words (below): x, and the outputs of the phases
    unsigned long long *part, *part_ml;    // attention, per head and CTA: sums of values; maximum and sum of weights: {float, tag}
    unsigned int* tag;                     // of the launch
    unsigned int* status;
    LinearShape lin[4];
    int slots;                             // of the ring
    int off_const, off_x, off_red;         // shared memory (from the aligned base)
    int sums_bytes;                        // of one of the two places at off_red; a power of two
    int warp_bytes;                        // what a warp keeps of x
    int off_factors, off_planes;           // within them: factors and sums per unit; planes
    int off_natural;                       // x in natural order, behind the planes of the normalised linears
};

// Values travel between CTAs as words {fp16 value, 16-bit tag}: a reader waits for the tag of the layer in the value itself, so there is
// no barrier, no fence and no second round trip (with a counter: release 1300 clk, its way to the waiting thread, a barrier of
// the CTA and the read of the values, 3000 clk more a phase).  Every word is written once per layer and every phase needs every value
// of the phase before, so a word is read by all before it is written again, and what is left in it carries another tag.
__device__ __forceinline__ void put_word(uint32_t* p, __half v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"((uint32_t)__half_as_ushort(v) | (tag << 16)) : "memory");
}
__device__ __forceinline__ uint4 get_words(const uint32_t* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t other_tag(const uint4& v, uint32_t tag) {      // not zero: a word is of another tag
    const uint32_t t = tag << 16;
    return ((v.x ^ t) | (v.y ^ t) | (v.z ^ t) | (v.w ^ t)) & 0xffff0000u;
}
__device__ __forceinline__ void put_float(unsigned long long* p, float v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((unsigned long long)__float_as_uint(v) | ((unsigned long long)tag << 32)) : "memory");
}
__device__ __forceinline__ unsigned long long get_float(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
constexpr long long kWaitClocks = 2000000000LL;      // about a second

__device__ __forceinline__ void consumers_meet() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kLayerWarps) : "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// The maps lie in the plan's memory, where other maps may have lain before: what wrote them has to be made visible to the copies, once per map, launch
// and CTA.
__device__ __forceinline__ void acquire_map(const CUtensorMap* m) {
    asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(m) : "memory");
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
// Bounded, without a call.
__device__ __forceinline__ void wait_for(uint32_t bar, uint32_t parity, bool& ok) {
    if (mbar_try(bar, parity) || !ok) return;
    const long long t0 = clock64();
    while (!mbar_try(bar, parity))
        if (clock64() - t0 > kWaitClocks) { ok = false; return; }
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int BITS, int HD>
__global__ void __launch_bounds__(kLayerThreads, 1)
decode_layers_kernel(const StepParams p) {
    using I = IntLayout<BITS, true>;
    constexpr int kWeights = slot_weights(BITS), kConsts = slot_consts(BITS), kScales = slot_scales(), kZeroPitch = slot_zero_words(BITS) * 4;
    constexpr int kUnitRows = 4 * BITS;                    // word-rows of a unit
    constexpr int kPlaneBytes = int_unit_bytes<BITS>(1);
    extern __shared__ __align__(1024) uint8_t dsm[];
    __shared__ __align__(8) uint64_t bars[2 * kMaxSlots];
    __shared__ __align__(16) float2 sm_sums[kLayerWarps];  // of x and x^2, per warp
    __shared__ __align__(16) StepPointers sm_layers[4];    // of the layers around the current one
    __shared__ int sm_items[4][2], sm_maps;
    __shared__ __align__(16) __half q_sm[HD], knew_sm[HD], vnew_sm[HD];
    __shared__ float sm_m[kLayerWarps], sm_l[kLayerWarps];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cta = blockIdx.x, ctas = gridDim.x;
    uint8_t* base = dsm + ((1024u - (smem_u32(dsm) & 1023u)) & 1023u);
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8u * kMaxSlots;
    bool ok = true;
    if (tid == 0) {
        sm_maps = 0;
        for (int s = 0; s < p.slots; ++s) {
            mbar_init(full0 + 8u * s, 1);
            mbar_init(empty0 + 8u * s, kLayerWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (tid < 16 && (tid >> 3) < p.n_layers)
        reinterpret_cast<uint4*>(sm_layers)[tid] = reinterpret_cast<const uint4*>(&p.layers[tid >> 3].at)[tid & 7];
    // items are dealt evenly, neighbours to the same CTA
    if (tid >= 32 && tid < 40) sm_items[(tid & 7) >> 1][tid & 1] = (int)(((long long)(cta + (tid & 1)) * p.lin[(tid & 7) >> 1].items) / ctas);
    __syncthreads();

    if (warp >= kLayerWarps) {
        // ---- the producer ----
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFewRegs));
        if (warp == kLayerWarps + 1) {
            // The maps of a layer, a lane each; how many layers of them, for the producer, which is a layer behind at least after the first.  (Acquired by
            // the producer itself, whose copies in flight each fence waits for, a layer took 4 us longer.)
#pragma unroll 1
            for (int l = 0; l < p.n_layers; ++l) {
                if (lane < 12) acquire_map(&p.layers[l].w[0] + lane);
                __syncwarp();
                if (lane == 0) asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(&sm_maps)), "r"(l + 1) : "memory");
            }
        }
        if (warp == kLayerWarps && elect_one()) {
            int have = 0;
            auto wait_for_maps = [&](int layers) {
                const long long t0 = clock64();
                while (have < layers && ok) {
                    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(have) : "r"(smem_u32(&sm_maps)) : "memory");
                    if (clock64() - t0 > kWaitClocks) ok = false;
                }
            };
            int slot = 0, parity = 1, issued = 0;          // (parity 1: the first round of slots is free)
            wait_for_maps(1);
            for (int i = 0; i < 3; ++i) prefetch_map(&p.layers[0].w[0] + 4 * i);
#pragma unroll 1
            for (int l = 0; l < p.n_layers && ok; ++l) {        // (none through a map that has not been acquired)
                const StepLayer& layer = p.layers[l];
#pragma unroll 1
                for (int ph = 0; ph < 4; ++ph) {
                    if (ph == 3) wait_for_maps(min(l + 2, p.n_layers));
                    const StepLayer& next = ph < 3 ? layer : p.layers[min(l + 1, p.n_layers - 1)];
                    for (int i = 0; i < 3; ++i) prefetch_map(&next.w[(ph + 1) & 3] + 4 * i);
                    const LinearShape& s = p.lin[ph];
                    const int end = sm_items[ph][1], pair = s.pair, n = s.slots, per_group = s.per_group;
                    const unsigned int inv = s.per_group_inv;
#pragma unroll 1
                    for (int it = sm_items[ph][0]; it < end && ok; ++it)
#pragma unroll 1
                        for (int i = 0; i < n && ok; ++i)
#pragma unroll 1
                            for (int strip = it; strip <= it + pair; strip += pair ? pair : 1) {
                                // (nothing more after a wait that has expired, and a slot is freed by warps that have seen its copy land only: two copies
                                // on one barrier, and the wait at the end would not be for all of them)
                                wait_for(empty0 + 8u * slot, parity, ok);
                                if (!ok) break;
                                const uint32_t bar = full0 + 8u * slot, cst = smem_u32(base) + p.off_const + slot * kConsts;
                                const int group = (int)(per_group == 1 ? i * kSlotUnits : __umulhi(i * kSlotUnits, inv));
                                mbar_expect(bar, kWeights + kConsts);
                                asm volatile(
                                    "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                    ::"r"(smem_u32(base) + slot * kWeights), "l"(&layer.w[ph]), "r"(strip * kStripCols),
                                      "r"(i * kSlotUnits * kUnitRows), "r"(bar) : "memory");
                                asm volatile(
                                    "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                    ::"r"(cst), "l"(&layer.s[ph]), "r"(strip * kStripCols), "r"(group), "r"(bar) : "memory");
                                asm volatile(
                                    "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                    ::"r"(cst + kScales), "l"(&layer.z[ph]), "r"((strip * BITS) & ~3), "r"(group), "r"(bar) : "memory");
                                ++issued;
                                if (++slot == p.slots) { slot = 0; parity ^= 1; }
                            }
                }
            }
            // the copies in flight have landed (always so unless a wait has expired)
            for (int i = 0; i < p.slots && i < issued; ++i) {
                if (--slot < 0) { slot = p.slots - 1; parity ^= 1; }
                bool landed = true;
                wait_for(full0 + 8u * slot, parity ^ 1, landed);
                ok = ok && landed;
            }
            if (!ok) atomicExch(p.status + kStatusWord, 1u);
        }
        return;
    }

    // ---- the warps that multiply ----
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kMoreRegs));
    const int H = p.hidden;
    const uint32_t tag0 = *p.tag + 1;                       // (not 0, which new memory holds)
    int slot = 0, parity = 0, sums_at = 0;
    const long long p64 = p.pos[0];
    const bool in_range = p64 >= 0 && p64 < p.max_seq;      // (a position outside the caches: no attention, as in b200gptq_attn_step)
    const int P = in_range ? (int)p64 : 0;
    // CTAs that share a head: as many as have a block of positions for each of their warps (a part per 192 positions, of four at most, made
    // steps at 300 positions 4 to 6 % and at 16 000 positions of 8 heads 70 % longer)
    constexpr int kRoundRows = kLayerWarps * 8 * (32 / (HD / 8));
    const int n_split = max(1, min(min(ctas / p.heads, kMaxSplit), (P + kRoundRows - 1) / kRoundRows));

    // A wait for words: until every lane of the warp has seen its tag, or time is up.
    long long t0 = 0;
    auto again = [&](bool missing) -> bool {
        if (!__any_sync(0xffffffffu, missing && ok)) return false;
        const long long t = clock64();
        if (t0 == 0) t0 = t;
        if (t - t0 > kWaitClocks) ok = false;
        return true;
    };
    // A linear: this CTA's strips (pairs of strips) one after the other.
    auto linear = [&](const StepPointers& layer, int ph, uint32_t tag, bool last) {
        const int g = lane >> 2, j = lane & 3;
        uint8_t* own = base + p.off_x + warp * p.warp_bytes;
        __half* own_x = reinterpret_cast<__half*>(own);                         // (of two units, as it lies in memory)
        float* own_f = reinterpret_cast<float*>(own + p.off_factors);
        uint8_t* own_planes = own + p.off_planes;
        auto pack8 = [](const uint4& a, const uint4& b) {
            return make_uint4(__byte_perm(a.x, a.y, 0x5410), __byte_perm(a.z, a.w, 0x5410), __byte_perm(b.x, b.y, 0x5410), __byte_perm(b.z, b.w, 0x5410));
        };
        // Eight values of each of kPasses units, `stride` words apart, once they are there (of those beyond `count`: zeros).
        auto read8 = [&](const uint32_t* src, int stride, uint32_t tag, int count, uint4 (&v)[kPasses]) {
            uint4 a[kPasses], b[kPasses];
            uint32_t missing;
            t0 = 0;
            do {
                missing = 0u;
#pragma unroll
                for (int r = 0; r < kPasses; ++r) {
                    a[r] = b[r] = make_uint4(tag << 16, tag << 16, tag << 16, tag << 16);
                    if (r < count) {
                        a[r] = get_words(src + (size_t)r * stride);
                        b[r] = get_words(src + (size_t)r * stride + 4);
                    }
                }
#pragma unroll
                for (int r = 0; r < kPasses; ++r) missing |= other_tag(a[r], tag) | other_tag(b[r], tag);
            } while (again(missing != 0u));
#pragma unroll
            for (int r = 0; r < kPasses; ++r) v[r] = pack8(a[r], b[r]);
        };

        // Planes of two of this warp's units (lanes 0..15 the first), from the eight values of the lane's item.
        const int jq = lane & 3, iq = (lane >> 2) & 3;
        auto make_planes = [&](int pass, const uint32_t (&h)[8], const int (&pre)[8]) {
            const int i = 2 * pass + (lane >> 4);
            uint32_t mx = 0u;
#pragma unroll
            for (int e = 0; e < 8; ++e) mx = max(mx, h[e] & 0x7fffu);
            // (2^ex > max |x| of the unit; zeros take any scale, an infinity or a NaN a NaN factor: gemv_strip.cuh)
            constexpr int XB = int_x_bits(BITS);
            const uint32_t lo16 = __reduce_max_sync(0xffffffffu, lane < 16 ? mx : 0u), hi16 = __reduce_max_sync(0xffffffffu, lane < 16 ? 0u : mx);
            mx = lane < 16 ? lo16 : hi16;
            int ex = (int)(__float_as_uint(__half2float(__ushort_as_half((unsigned short)mx))) >> 23);
            const bool bad = mx >= 0x7c00u;
            if (mx == 0u || bad) ex = 127;
            const float scale = __uint_as_float((uint32_t)(253 + XB - ex) << 23);
            int sum = 0, X[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float xf = __half2float(__ushort_as_half((unsigned short)h[e]));
                X[e] = XB > 22 ? __float2int_rn(xf * scale) : __float_as_int(fmaf(xf, scale, 12582912.f)) - 0x4B400000;
                sum += X[e];
            }
            uint32_t dg[8];                                // four signed base-256 digits each
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                // 4 bits: a byte of weights is used as it is, low + 16 * high, and once more with the high nibble masked off: what the first
                // product has too much of the low one is taken off the second one's x.  |16 X - X'| < 2^30 + 2^26 fits the digits.
                const int Y = BITS == 4 && e < 4 ? X[e] * 16 - X[(e + 4) & 7] : X[e] << (BITS == 4 ? 0 : pre[e]);
                dg[e] = (uint32_t)(Y + 0x00808080) ^ 0x00808080u;
            }
            constexpr int WHOLE_SUM = XB > 22 ? 4 : 16;    // (the X of 128 rows of 22 bits, or of 32 rows of 26, add up to less than 2^31)
#pragma unroll
            for (int o = 1; o < WHOLE_SUM; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            float sumf = (float)sum;
#pragma unroll
            for (int o = WHOLE_SUM; o < 16; o <<= 1) sumf += __shfl_xor_sync(0xffffffffu, sumf, o);
            const float delta = __uint_as_float((uint32_t)(ex + 1 - XB) << 23);
            const float factor = bad ? __uint_as_float(0x7fc00000u) : __uint_as_float((uint32_t)(ex + 1 - XB - I::kPre) << 23);
            if ((lane & 15) == 0) *reinterpret_cast<float2*>(own_f + 2 * i) = make_float2(factor, -delta * sumf);
            uint8_t* dst = own_planes + (size_t)i * kPlaneBytes + jq * 32;
            auto store = [&](int step, const uint32_t (&lo)[4], const uint32_t (&hi)[4]) {
                uint4* d = reinterpret_cast<uint4*>(dst + step * 4 * 32);
                d[0] = make_uint4(lo[0], hi[0], lo[1], hi[1]);
                d[1] = make_uint4(lo[2], hi[2], lo[3], hi[3]);
            };
            uint32_t lo[4], hi[4];
            if (BITS != 3 || iq < 3) {
                planes_of(dg[0], dg[1], dg[2], dg[3], lo);
                planes_of(dg[4], dg[5], dg[6], dg[7], hi);
                store(iq, lo, hi);
            } else {
                planes_of(dg[0], dg[1], 0, dg[2], lo);
                planes_of(dg[3], 0, dg[4], dg[5], hi);
                store(3, lo, hi);
                planes_of(0, dg[6], dg[7], 0, lo);
                hi[0] = hi[1] = hi[2] = hi[3] = 0u;
                store(4, lo, hi);
            }
        };

        // x of this warp's units, two units at a time (half a warp each, eight values per lane), ready to be multiplied.
        auto fetch_x = [&](const StepPointers& layer, int ph, uint32_t tag) {
            const LinearShape& s = p.lin[ph];
            const int units = s.units, passes = s.slots;
            const uint32_t* src = ph == kOut ? p.att : (ph == kDown ? p.act : p.xw);
            const bool normed = ph == kQkv || ph == kUp;
            const int which = ph == kQkv ? 0 : 1;
            const __half *nw = layer.norm_w[which], *nb = layer.norm_b[which];
            const int32_t* perm = ph == kDown ? nullptr : layer.perm[ph];
            auto norm_weights = [&](int k, uint4& w, uint4& b) {
                w = __ldg(reinterpret_cast<const uint4*>(nw + k));
                if (nb) b = __ldg(reinterpret_cast<const uint4*>(nb + k));
            };
            auto square = [&](const uint4& v, float& s1, float& s2) {
                const __half2* q = reinterpret_cast<const __half2*>(&v);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float2 f = __half22float2(q[c]);
                    s1 += f.x + f.y; s2 += f.x * f.x + f.y * f.y;
                }
            };
            auto leave_sums = [&](float s1, float s2) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
                    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
                }
                if (lane == 0) sm_sums[warp] = make_float2(s1, s2);
            };
            auto whole_sums = [&](float& mean, float& inv) {
                const float2 part = sm_sums[lane & (kLayerWarps - 1)];
                float a = part.x, a2 = part.y;
#pragma unroll
                for (int o = kLayerWarps / 2; o > 0; o >>= 1) {
                    a += __shfl_xor_sync(0xffffffffu, a, o);
                    a2 += __shfl_xor_sync(0xffffffffu, a2, o);
                }
                mean = p.rms ? 0.f : a * p.inv_hidden;
                inv = rsqrtf((p.rms ? a2 * p.inv_hidden : fmaxf(a2 * p.inv_hidden - mean * mean, 0.f)) + p.eps);
            };
            auto normalise = [&](uint4& v, const uint4& wv, const uint4& bv, float mean, float inv) {     // (the rounding of b200gptq_add_norm)
                __half2* q = reinterpret_cast<__half2*>(&v);
                const __half2 *pw = reinterpret_cast<const __half2*>(&wv), *pb = reinterpret_cast<const __half2*>(&bv);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float2 f = __half22float2(q[c]), fw = __half22float2(pw[c]), fb = __half22float2(pb[c]);
                    float a0 = (f.x - mean) * inv, a1 = (f.y - mean) * inv;
                    if (p.rms) { a0 = __half2float(__float2half_rn(a0)); a1 = __half2float(__float2half_rn(a1)); }
                    q[c] = __floats2half2_rn(a0 * fw.x + fb.x, a1 * fw.y + fb.y);
                }
            };
            const uint4 none = make_uint4(0u, 0u, 0u, 0u);
            // pass i, this half of the warp: unit first_unit + i kSlotUnits
            const int first_unit = 2 * warp + (lane >> 4), step = kSlotUnits * kUnit;
            const int mine = (units - first_unit + kSlotUnits - 1) / kSlotUnits;                // passes in which it exists
            {
                // The eight rows of the lane's item.  Of 4 bits they are adjacent and read as such; else, and where rows are picked through a
                // permutation, x is put down in natural order first.
                int row[8], pre[8];
                I::item(iq, jq, row, pre);
                const bool direct = BITS == 4 && !perm;
                const int at_row = direct ? row[0] : 8 * (lane & 15);
                const uint32_t* from = src + first_unit * kUnit + at_row;
                // (natural order: unit u lies behind the planes of its warp)
                uint8_t* natural = base + p.off_x + p.off_natural;
                auto natural_at = [&](int u) { return reinterpret_cast<__half*>(natural + ((u & (kSlotUnits - 1)) >> 1) * p.warp_bytes + (2 * (u / kSlotUnits) + (u & 1)) * (kUnit * 2)); };
                auto items = [&](const uint4& v, uint32_t (&h)[8]) {       // (evens, then odds)
                    h[0] = v.x & 0xffffu; h[4] = v.x >> 16; h[1] = v.y & 0xffffu; h[5] = v.y >> 16;
                    h[2] = v.z & 0xffffu; h[6] = v.z >> 16; h[3] = v.w & 0xffffu; h[7] = v.w >> 16;
                };
                if (ph != kDown) {                         // (all of x in registers: hidden <= kPasses * kSlotUnits * kUnit)
                    uint4 v[kPasses], w[kPasses], b[kPasses];
                    uint32_t picks[kPasses][8];
                    // (what does not need x is on its way while that is waited for)
#pragma unroll
                    for (int r = 0; r < kPasses; ++r) {
                        w[r] = b[r] = none;
                        const int k0 = first_unit * kUnit + r * step;
                        if (normed && r < mine) norm_weights(k0 + at_row, w[r], b[r]);
#pragma unroll
                        for (int e = 0; e < 8; ++e) picks[r][e] = perm && r < mine ? (uint32_t)__ldg(perm + k0 + row[e]) : 0u;
                    }
                    read8(from, step, tag, mine, v);
                    if (normed) {
                        float s1 = 0.f, s2 = 0.f, mean, inv;
#pragma unroll
                        for (int r = 0; r < kPasses; ++r)
                            if (r < passes) square(v[r], s1, s2);
                        leave_sums(s1, s2);
                        consumers_meet();
                        whole_sums(mean, inv);
#pragma unroll
                        for (int r = 0; r < kPasses; ++r)
                            if (r < mine) normalise(v[r], w[r], b[r], mean, inv);      // (a unit past the last: zeros)
                    }
                    if (!direct) {
#pragma unroll
                        for (int r = 0; r < kPasses; ++r)
                            if (r < passes) *reinterpret_cast<uint4*>(natural_at(first_unit + r * kSlotUnits) + at_row) = v[r];
                        if (perm) consumers_meet();
                        else __syncwarp();
                    }
#pragma unroll
                    for (int r = 0; r < kPasses; ++r)
                        if (r < passes) {
                            uint32_t h[8];
                            if (direct) {
                                items(v[r], h);
                            } else if (perm) {
#pragma unroll
                                for (int e = 0; e < 8; ++e)
                                    h[e] = r < mine ? __half_as_ushort(natural_at(picks[r][e] / kUnit)[picks[r][e] & (kUnit - 1)]) : 0u;
                            } else {
#pragma unroll
                                for (int e = 0; e < 8; ++e) h[e] = __half_as_ushort(natural_at(first_unit + r * kSlotUnits)[row[e]]);
                            }
                            make_planes(r, h, pre);
                        }
                } else {
#pragma unroll 1
                    for (int r0 = 0; r0 < passes; r0 += kPasses) {
                        uint4 v[kPasses];
                        read8(from + (size_t)r0 * step, step, tag, mine - r0, v);
#pragma unroll
                        for (int r = 0; r < kPasses; ++r)
                            if (r0 + r < passes) {
                                uint32_t h[8];
                                if (direct) {
                                    items(v[r], h);
                                } else {
                                    __half* stage = own_x + (lane >> 4) * kUnit;
                                    *reinterpret_cast<uint4*>(stage + at_row) = v[r];
                                    __syncwarp();
#pragma unroll
                                    for (int e = 0; e < 8; ++e) h[e] = __half_as_ushort(stage[row[e]]);
                                    __syncwarp();
                                }
                                make_planes(r0 + r, h, pre);
                            }
                    }
                }
            }
            __syncwarp();
        };

        // A slot's weights and constants of this lane.
        constexpr int kLoads = I::kLoads;
        struct Piece { uint4 w[2][kLoads]; uint2 scales[2]; uint32_t zeros[2]; };        // (of the warp's two units)
        uint32_t read_at[2][kLoads];               // four columns of some word-rows
#pragma unroll
        for (int v = 0; v < 2; ++v)
#pragma unroll
            for (int i = 0; i < kLoads; ++i) {
                const int r = (2 * warp + v) * kUnitRows + I::load_row(i, j);
                read_at[v][i] = r * 128 + ((g ^ (r & 7)) << 4);
            }
        // planes: quad lane j < 2 holds planes 2j, 2j + 1; the zero-point term goes to one lane
        const float plane_weight = j == 0 ? 1.f : (j == 1 ? 65536.f : 0.f), sum_weight = j == 0 ? 1.f : 0.f;
        auto load_slot = [&](Piece& to, const LinearShape& s, int i, int strip) {
            wait_for(full0 + 8u * slot, parity, ok);
            const uint8_t* src = base + slot * kWeights;
            const uint8_t* cst = base + p.off_const + slot * kConsts;
            // (rows past K, units past the last: zeros, whatever their constants)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int u = 2 * warp + v;
                const int r = s.per_group == 1 ? u : (int)(__umulhi(i * kSlotUnits + u, s.per_group_inv) - __umulhi(i * kSlotUnits, s.per_group_inv));
#pragma unroll
                for (int q = 0; q < kLoads; ++q) to.w[v][q] = *reinterpret_cast<const uint4*>(src + read_at[v][q]);
                to.scales[v] = *reinterpret_cast<const uint2*>(cst + r * 64 + 8 * g);
                to.zeros[v] = load_zeros<BITS>(cst + kScales + r * kZeroPitch + 4 * ((strip * BITS) & 3), 4 * g);
            }
            __syncwarp();                          // every lane has its part
            if (lane == 0 && ok) mbar_arrive(empty0 + 8u * slot);
            if (++slot == p.slots) { slot = 0; parity ^= 1; }
        };
        // (a slot of units past the last)
        auto pass_slot = [&]() {
            wait_for(full0 + 8u * slot, parity, ok);
            __syncwarp();
            if (lane == 0 && ok) mbar_arrive(empty0 + 8u * slot);
            if (++slot == p.slots) { slot = 0; parity ^= 1; }
        };
        auto column = [&](const uint4& v, int c) { return c == 0 ? v.x : (c == 1 ? v.y : (c == 2 ? v.z : v.w)); };
        auto scale_of = [&](const uint2& scales, int c) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(c < 2 ? &scales.x : &scales.y));
            return c & 1 ? f.y : f.x;
        };
        auto zero_of = [&](uint32_t zeros, int c) {        // field + 1
            return __uint_as_float(0x4B000000u | ((zeros >> (BITS * c)) & ((1u << BITS) - 1u))) - 8388607.f;
        };
        // Two slots at once (one alone is a chain of latencies): out[0] += slot 0 times the units of slot i0 of x, out[1] += slot 1
        // times those of i1.  `second`: there is another one.
        auto multiply = [&](bool second, int strip0, int strip1, const LinearShape& s, int i0, int i1, float (&out)[2][4]) {
            {
                uint2 bx[2][2][I::kSteps];
                float4 f[2];
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const int i = t ? i1 : i0;
#pragma unroll
                    for (int v = 0; v < 2; ++v)
#pragma unroll
                        for (int st = 0; st < I::kSteps; ++st) {
                            bx[t][v][st] = make_uint2(0u, 0u);
                            if (g < 4) bx[t][v][st] = *reinterpret_cast<const uint2*>(own_planes + (2 * i + v) * kPlaneBytes + (st * 4 + j) * 32 + g * 8);
                        }
                    f[t] = *reinterpret_cast<const float4*>(own_f + 4 * i);
                }
                Piece now[2];
                load_slot(now[0], s, i0, strip0);
                if (second) {
                    load_slot(now[1], s, i1, strip1);
                } else {                           // (zeros: it adds none)
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
#pragma unroll
                        for (int q = 0; q < kLoads; ++q) now[1].w[v][q] = make_uint4(0u, 0u, 0u, 0u);
                        now[1].scales[v] = make_uint2(0u, 0u);
                        now[1].zeros[v] = 0u;
                    }
                }
                // the sums start at the bits of 1.5 * 2^23: |sum| < 2^22, so they end as floats with that offset
                constexpr int kBias = 0x4B400000;
                int d[2][2][2][4];
#pragma unroll
                for (int e = 0; e < 32; ++e) d[e >> 4][(e >> 3) & 1][(e >> 2) & 1][e & 3] = kBias;
                if constexpr (BITS == 4) {
#pragma unroll
                    for (int st = 0; st < 4; ++st)
#pragma unroll
                        for (int t = 0; t < 2; ++t)
#pragma unroll
                            for (int v = 0; v < 2; ++v)
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    const uint32_t wa = column(now[t].w[v][st], 2 * h), wb = column(now[t].w[v][st], 2 * h + 1);
                                    imma(d[t][v][h], d[t][v][h], wa & 0x0f0f0f0fu, wb & 0x0f0f0f0fu, wa, wb, bx[t][v][st].x, bx[t][v][st].y);
                                }
                } else {
#pragma unroll
                    for (int t = 0; t < 2; ++t)
#pragma unroll
                        for (int v = 0; v < 2; ++v)
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                uint32_t ra[2 * I::kSteps], rb[2 * I::kSteps], wa[kLoads], wb[kLoads];
#pragma unroll
                                for (int q = 0; q < kLoads; ++q) { wa[q] = column(now[t].w[v][q], 2 * h); wb[q] = column(now[t].w[v][q], 2 * h + 1); }
                                I::regs(wa, ra);
                                I::regs(wb, rb);
#pragma unroll
                                for (int st = 0; st < I::kSteps; ++st)
                                    imma(d[t][v][h], d[t][v][h], ra[2 * st], rb[2 * st], ra[2 * st + 1], rb[2 * st + 1], bx[t][v][st].x, bx[t][v][st].y);
                            }
                }
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const float cf = (v ? f[t].z : f[t].x) * plane_weight, sx = (v ? f[t].w : f[t].y) * sum_weight;
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const float lo = __int_as_float(d[t][v][c >> 1][2 * (c & 1)]) - 12582912.f, hi = __int_as_float(d[t][v][c >> 1][2 * (c & 1) + 1]) - 12582912.f;
                            out[t][c] = fmaf(scale_of(now[t].scales[v], c), fmaf(fmaf(256.f, hi, lo), cf, zero_of(now[t].zeros[v], c) * sx), out[t][c]);
                        }
                    }
            }
        };
        const LinearShape& s = p.lin[ph];
        const int begin = sm_items[ph][0], end = sm_items[ph][1], pair = s.pair;
        if (begin == end) return;
        fetch_x(layer, ph, ph == kUp ? tag + 1 : tag);
        const __half* bias = layer.bias[ph];
        const int slots = s.slots, units = s.units;
#pragma unroll 1
        for (int it = begin; it < end; ++it) {
            // The item is written by one warp, a lane per column; what it needs beside the sums is on its way meanwhile.
            const int n = it * kStripCols + lane;
            const bool writes = warp == (it & (kLayerWarps - 1)), residual = ph == kOut || ph == kDown;
            __half b0 = __ushort_as_half(0), b1 = b0, xr = b0;
            if (writes) {
                if (bias) {
                    b0 = bias[n];
                    if (pair) b1 = bias[n + pair * kStripCols];
                }
                if (residual) xr = p.x[n];
            }
            float* red;                                          // [strip of the item][warp][32]
            {
                // a pair of strips: both strips' slot i, with the same x; else two slots of the strip
                float out[2][4] = {};
                const int step = pair ? 1 : 2;
#pragma unroll 1
                for (int i = 0; i < slots; i += step) {
                    const bool second = pair || i + 1 < slots;
                    const int i1 = pair || !second ? i : i + 1;
                    if (i * kSlotUnits + 2 * warp < units) {
                        multiply(second, it, it + pair, s, i, i1, out);
                    } else {
                        pass_slot();
                        if (second) pass_slot();
                    }
                }
                // Two places for the sums, in turn over all items of this CTA whatever linear they belong to: the warp that reads them joins
                // the next item's meeting after it has read, and no warp is past that meeting when it writes this place again.
                red = reinterpret_cast<float*>(base + p.off_red + sums_at);
                sums_at ^= p.sums_bytes;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (!pair) out[0][c] += out[1][c];
                    out[0][c] += __shfl_xor_sync(0xffffffffu, out[0][c], 1);                             // the other planes
                    if (pair) out[1][c] += __shfl_xor_sync(0xffffffffu, out[1][c], 1);
                }
                if (j == 0) {
                    *reinterpret_cast<float4*>(red + warp * 32 + 4 * g) = make_float4(out[0][0], out[0][1], out[0][2], out[0][3]);
                    if (pair) *reinterpret_cast<float4*>(red + (kLayerWarps + warp) * 32 + 4 * g) = make_float4(out[1][0], out[1][1], out[1][2], out[1][3]);
                }
            }
            consumers_meet();
            if (writes) {
                float v[2] = {0.f, 0.f};
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    if (t == 0 || pair)
#pragma unroll
                        for (int w = 0; w < kLayerWarps; ++w) v[t] += red[(t * kLayerWarps + w) * 32 + lane];
                const __half y = __float2half_rn(v[0] + __half2float(b0));
                if (ph == kQkv) {
                    put_word(p.qkv + n, y, tag);
                } else if (ph == kUp) {
                    __half a;
                    if (pair) {                          // (the rounding of b200gptq_act)
                        const float gf = __half2float(y), uf = __half2float(__float2half_rn(v[1] + __half2float(b1)));
                        a = __float2half_rn(__half2float(__float2half_rn(gf / (1.f + __expf(-gf)))) * uf);
                    } else {
                        a = __float2half_rn(fmaxf(__half2float(y), 0.f));
                    }
                    put_word(p.act + n, a, tag);
                } else {
                    const __half xn = __hadd(xr, y);
                    p.x[n] = xn;
                    if (!last) put_word(p.xw + n, xn, ph == kOut ? tag + 1 : tag + 2);
                }
            }
        }
    };

    // Single-query attention over positions 0 .. P: b200gptq_attn_step's arithmetic.  `split` CTAs share a head, their
    // warps take blocks of kRows positions in turn; the first of them adds the parts up.  us per layer, kernel by kernel / here: 32 heads of 128 (Llama-7B)
    // 1000 positions 40.4 / 36.9, 4000 47.1 / 46.4, 16 000 75 / 83 (the cache that the shared memory leaves is too small for more loads in flight);
    // 8 heads (hidden 1024) 1000 positions 22.3 / 17.3, 16 000 46.5 / 29.0; 4 heads (hidden 512) 32 000 positions 56.6 / 39.9.
    auto attention = [&](const StepPointers& layer, uint32_t tag) {
        constexpr int LP = HD / 8, GROUPS = 32 / LP, U = 8, kRows = U * GROUPS;    // lanes per position; positions per block
        constexpr int kWriters = HD / 32;                                          // warps that write, a lane per dim
        // (what depends on the item only is made anew in each layer: kept, it would be registers that the products need)
        int cta = blockIdx.x, d = threadIdx.x, split = n_split;
        const int items = p.heads * split;
        if (cta >= items) return;
        const int lane = d & 31, warp = d >> 5, grp = lane / LP, dim = (lane % LP) * 8, stride = kLayerWarps * split * kRows;
        float* own_acc = reinterpret_cast<float*>(base + p.off_x + warp * p.warp_bytes);                            // [HD] (x is not needed here)
#pragma unroll 1
        for (int item = cta; item < items; item += ctas) {
            const int head = item / split, sp = item - head * split;
            const size_t cache = (size_t)head * p.max_seq * HD;
            uint4 kv[U], vv[U];
            auto request = [&](const __half* from, int t0, uint4 (&to)[U]) {
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    const int t = min(t0 + i * GROUPS + grp, p.max_seq - 1);
                    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(to[i].x), "=r"(to[i].y), "=r"(to[i].z), "=r"(to[i].w)
                                 : "l"(from + cache + (size_t)t * HD + dim));
                }
            };
            int t_at = (warp * split + sp) * kRows;
            if (t_at < P) { request(layer.k_cache, t_at, kv); request(layer.v_cache, t_at, vv); }
            __half cs = __ushort_as_half(0), sn = cs;
            if (p.rope && d < HD / 2) { cs = p.cos_t[(size_t)P * (HD / 2) + d]; sn = p.sin_t[(size_t)P * (HD / 2) + d]; }
            if (warp < kWriters) {
                // q, k, v of the new token: two values of each per lane of the first warps
                const int i = d;                         // pair index
                const bool active = i < HD / 2;
                const uint32_t* src = p.qkv + (size_t)head * HD + 2 * (active ? i : 0);
                unsigned long long w[3];
                const uint32_t tg = tag << 16;
                uint32_t missing;
                t0 = 0;
                do {
                    missing = 0u;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        w[c] = get_float(reinterpret_cast<const unsigned long long*>(src + (size_t)c * H));
                        missing |= (((uint32_t)w[c] ^ tg) | ((uint32_t)(w[c] >> 32) ^ tg)) & 0xffff0000u;
                    }
                } while (again(missing != 0u));
                auto two = [&](unsigned long long v) {
                    const uint32_t r = __byte_perm((uint32_t)v, (uint32_t)(v >> 32), 0x5410);
                    return *reinterpret_cast<const __half2*>(&r);
                };
                __half2 q2 = two(w[0]), k2 = two(w[1]);
                const __half2 v2 = two(w[2]);
                if (active) {
                    if (p.rope) {
                        q2 = __halves2half2(__hsub(__hmul(q2.x, cs), __hmul(q2.y, sn)), __hadd(__hmul(q2.x, sn), __hmul(q2.y, cs)));
                        k2 = __halves2half2(__hsub(__hmul(k2.x, cs), __hmul(k2.y, sn)), __hadd(__hmul(k2.x, sn), __hmul(k2.y, cs)));
                    }
                    *reinterpret_cast<__half2*>(q_sm + 2 * i) = q2;
                    *reinterpret_cast<__half2*>(knew_sm + 2 * i) = k2;
                    *reinterpret_cast<__half2*>(vnew_sm + 2 * i) = v2;
                    if (sp == 0 && in_range) {
                        const size_t to = cache + (size_t)P * HD + 2 * i;
                        *reinterpret_cast<__half2*>(layer.k_cache + to) = k2;
                        *reinterpret_cast<__half2*>(layer.v_cache + to) = v2;
                    }
                }
            }
            consumers_meet();
            float qf[8], acc[8];
            auto widen = [&](const uint4& raw, float (&f)[8]) {
                const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 v = __half22float2(h[e]);
                    f[2 * e] = v.x; f[2 * e + 1] = v.y;
                }
            };
            widen(*reinterpret_cast<const uint4*>(q_sm + dim), qf);
            auto dot8 = [&](const uint4& raw) {          // over the lane's 8 dims, summed over the position's lanes
                float f[8], s = 0.f;
                widen(raw, f);
#pragma unroll
                for (int e = 0; e < 8; ++e) s = fmaf(f[e], qf[e], s);
#pragma unroll
                for (int o = 1; o < LP; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                return s * p.scale;
            };
            auto add8 = [&](const uint4& raw, float w) {
                float f[8];
                widen(raw, f);
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[e] = fmaf(w, f[e], acc[e]);
            };
            constexpr float kNone = -1e30f;              // below every score; finite, so that differences are
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] = 0.f;
            float mx = kNone, l = 0.f;
#pragma unroll 1
            while (t_at < P) {
                const int t = t_at + grp;
                float sc[U], m_new = mx;
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    sc[i] = dot8(kv[i]);
                    if (t + i * GROUPS < P) m_new = fmaxf(m_new, sc[i]);
                }
                // (the next block's keys are on their way while the values are worked on, its values while the keys are)
                t_at += stride;
                if (t_at < P) request(layer.k_cache, t_at, kv);
                const float corr = __expf(mx - m_new);
                l *= corr;
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[e] *= corr;
#pragma unroll
                for (int i = 0; i < U; ++i)
                    if (t + i * GROUPS < P) {
                        const float w = __expf(sc[i] - m_new);
                        l += w;
                        add8(vv[i], w);
                    }
                mx = m_new;
                if (t_at < P) request(layer.v_cache, t_at, vv);
            }
            if (sp == 0 && warp == kLayerWarps - 1) {
                // the new position: one more step of the online softmax for the first group
                const float s = dot8(*reinterpret_cast<const uint4*>(knew_sm + dim));
                if (grp == 0) {
                    const float m_new = fmaxf(mx, s), w = __expf(s - m_new), corr = __expf(mx - m_new);
                    l = l * corr + w;
                    mx = m_new;
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[e] *= corr;
                    add8(*reinterpret_cast<const uint4*>(vnew_sm + dim), w);
                }
            }
            // ---- the warp's groups ----
            float gm = mx;
#pragma unroll
            for (int o = LP; o < 32; o <<= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, o));
            const float wgt = __expf(mx - gm);
            l *= wgt;
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] *= wgt;
#pragma unroll
            for (int o = LP; o < 32; o <<= 1) {
                l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
            }
            if (lane == 0) { sm_m[warp] = gm; sm_l[warp] = l; }
            if (grp == 0) {
                *reinterpret_cast<float4*>(own_acc + dim) = make_float4(acc[0], acc[1], acc[2], acc[3]);
                *reinterpret_cast<float4*>(own_acc + dim + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
            }
            consumers_meet();
            // ---- the CTA's warps: one dim per lane of the first ones ----
            if (warp < kWriters) {
                float cm = kNone, cl = 0.f, ca = 0.f;
#pragma unroll
                for (int w = 0; w < kLayerWarps; ++w) cm = fmaxf(cm, sm_m[w]);
#pragma unroll
                for (int w = 0; w < kLayerWarps; ++w) {
                    const float e = __expf(sm_m[w] - cm);
                    cl += sm_l[w] * e;
                    ca += *reinterpret_cast<const float*>(base + p.off_x + w * p.warp_bytes + 4 * d) * e;
                }
                unsigned long long* part = p.part + (size_t)head * kMaxSplit * HD;
                unsigned long long* ml = p.part_ml + (size_t)(head * kWriters + warp) * kMaxSplit * 2;
                if (sp != 0) {
                    put_float(part + sp * HD + d, ca, tag);
                    if (lane < 2) put_float(ml + 2 * sp + lane, lane ? cl : cm, tag);
                } else {
                    if (split > 1) {
                        // maxima and sums of weights of all parts, a lane each; the first parts with them, more of them in turn
                        unsigned long long mlw = 0, a[kPartsAtOnce];
                        const bool has = lane >= 2 && lane < 2 * split;
                        float mine = 0.f, tm = cm;
#pragma unroll 1
                        for (int r0 = 1; r0 < split; r0 += kPartsAtOnce) {
                            bool missing;
                            t0 = 0;
                            do {
                                missing = false;
                                if (has && r0 == 1) mlw = get_float(ml + lane);
#pragma unroll
                                for (int r = 0; r < kPartsAtOnce; ++r)
                                    if (r0 + r < split) a[r] = get_float(part + (r0 + r) * HD + d);
                                missing = has && (uint32_t)(mlw >> 32) != tag;
#pragma unroll
                                for (int r = 0; r < kPartsAtOnce; ++r)
                                    if (r0 + r < split) missing = missing || (uint32_t)(a[r] >> 32) != tag;
                            } while (again(missing));
                            if (r0 == 1) {
                                mine = __uint_as_float((uint32_t)mlw);
                                if (has && !(lane & 1)) tm = fmaxf(cm, mine);
#pragma unroll
                                for (int o = 16; o > 0; o >>= 1) tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, o));
                                const float e0 = __expf(cm - tm);
                                cl *= e0; ca *= e0;
                            }
#pragma unroll
                            for (int r = 0; r < kPartsAtOnce; ++r)
                                if (r0 + r < split) {
                                    const float e = __expf(__shfl_sync(0xffffffffu, mine, 2 * (r0 + r)) - tm);
                                    cl += __shfl_sync(0xffffffffu, mine, 2 * (r0 + r) + 1) * e;
                                    ca += __uint_as_float((uint32_t)a[r]) * e;
                                }
                        }
                    }
                    put_word(p.att + head * HD + d, in_range ? __float2half_rn(ca / cl) : __ushort_as_half(0), tag);
                }
            }
            consumers_meet();                            // (the warps' sums have been read)
        }
    };

    // The step's input, where the first linear reads it.
    {
        const int begin = sm_items[kOut][0], end = sm_items[kOut][1];       // (its items are the strips of x)
        for (int i = begin * kStripCols + tid; i < end * kStripCols; i += 32 * kLayerWarps)
            put_word(p.xw + i, p.x[i], tag0);
    }
#pragma unroll 1
    for (int l = 0; l < p.n_layers; ++l) {
        const StepPointers& layer = sm_layers[l & 3];
        const uint32_t tag = tag0 + 2 * l;
        // Pointers of the layer after the next, into the place of the one before the last: a round trip to memory for every one of them
        // otherwise.  What was asked for a layer ago has landed, and this layer's meetings show it to the other warps.
        if (tid < 8) {
            cp_wait_all();
            if (l + 2 < p.n_layers)
                cp_async16(smem_u32(reinterpret_cast<uint4*>(&sm_layers[(l + 2) & 3]) + tid), reinterpret_cast<const uint4*>(&p.layers[l + 2].at) + tid, true);
        }
        __syncwarp();
        // (One copy of the code of each kind of phase: written out four times it was fetched anew for every phase.)
#pragma unroll 1
        for (int ph = 0; ph < 5; ++ph) {
            if (ph == 1) { attention(layer, tag); continue; }
            const int i = ph == 0 ? kQkv : ph - 1;
            const bool last = i == kDown && l + 1 == p.n_layers;
            linear(layer, i, tag, last);
        }
    }
    // (The last CTA has an item in every linear; every CTA that takes part has read the tag: what this one has just worked on came from
    // all of them.)
    if (cta == ctas - 1 && tid == 0) *p.tag = tag0 + 2 * p.n_layers;
    if (!ok) atomicExch(p.status + kStatusWord, 1u);
}

const void* layers_kernel(int bits, int hd) {
    if (hd == 128)
        return bits == 2 ? (const void*)decode_layers_kernel<2, 128> : bits == 3 ? (const void*)decode_layers_kernel<3, 128>
             : bits == 4 ? (const void*)decode_layers_kernel<4, 128> : nullptr;
    if (hd == 64)
        return bits == 2 ? (const void*)decode_layers_kernel<2, 64> : bits == 3 ? (const void*)decode_layers_kernel<3, 64>
             : bits == 4 ? (const void*)decode_layers_kernel<4, 64> : nullptr;
    return nullptr;
}

struct StepPlan {
    StepParams params;          // (pointers into the plan's memory are filled in by each run)
    const void* kernel;
    int smem;
    size_t off_xw, off_qkv, off_att, off_act, off_part, off_ml, off_tag, bytes;
};

constexpr int kLayersSmem = 227 * 1024 - 3072;      // dynamic, beside the kernel's static variables

// Geometry, shared memory and the plan's memory; false: not a shape of this kernel.
bool plan_step(const b200gptq_step_shape& q, StepPlan* plan) {
    StepParams& p = plan->params;
    if (q.layers < 1 || q.batch != 1 || q.heads < 1 || q.hidden < kUnit || q.hidden % q.heads) return false;
    const int hd = q.hidden / q.heads;
    plan->kernel = layers_kernel(q.bits, hd);
    if (!plan->kernel || q.hidden % kUnit || q.inter < kUnit || q.inter % kUnit || q.max_seq < 1) return false;
    if (q.group_size < 1 || (q.group_size % kUnit && q.group_size < (q.hidden > q.inter ? q.hidden : q.inter))) return false;
    p.n_layers = q.layers; p.hidden = q.hidden; p.heads = q.heads; p.inter = q.inter; p.max_seq = q.max_seq;
    p.gated = q.gated; p.rms = q.rms; p.rope = q.rope; p.eps = q.eps; p.scale = q.scale; p.inv_hidden = 1.f / q.hidden;
    const int K[4] = {q.hidden, q.hidden, q.hidden, q.inter}, N[4] = {3 * q.hidden, q.hidden, (q.gated ? 2 : 1) * q.inter, q.hidden};
    for (int i = 0; i < 4; ++i) {
        LinearShape& s = p.lin[i];
        s.K = K[i]; s.units = K[i] / kUnit; s.slots = (s.units + kSlotUnits - 1) / kSlotUnits;
        s.strips = N[i] / kStripCols;
        s.pair = i == kUp && q.gated ? s.strips / 2 : 0;
        s.items = s.pair ? s.pair : s.strips;
        s.per_group = q.group_size >= K[i] ? s.units : q.group_size / kUnit;
        s.per_group_inv = (unsigned int)((0x100000000ULL + s.per_group - 1) / s.per_group);
        s.zero_words = s.strips * q.bits;
        if (s.zero_words % 4) return false;              // (rows of qzeros are whole 16-byte pieces)
    }
    // shared memory: ring | per warp x, factors, planes | sums of the warps
    const int n_h = p.lin[kUp].slots, n_max = p.lin[kDown].slots > n_h ? p.lin[kDown].slots : n_h;
    const int plane_bytes = q.bits == 3 ? int_unit_bytes<3>(1) : int_unit_bytes<4>(1);
    if (n_h > kPasses) return false;
    p.off_factors = 2 * kUnit * 2;
    p.off_planes = p.off_factors + 2 * n_max * 8;
    p.off_natural = p.off_planes + 2 * n_h * plane_bytes;
    p.warp_bytes = p.off_natural + 2 * n_h * kUnit * 2;
    if (p.warp_bytes < p.off_planes + 2 * n_max * plane_bytes) p.warp_bytes = p.off_planes + 2 * n_max * plane_bytes;
    if (p.warp_bytes < hd * 4) p.warp_bytes = hd * 4;
    p.warp_bytes = (p.warp_bytes + 15) / 16 * 16;
    p.sums_bytes = (q.gated ? 2 : 1) * kLayerWarps * 32 * 4;
    const int fixed = 1024 + kLayerWarps * p.warp_bytes + 2 * p.sums_bytes, slot = slot_weights(q.bits) + slot_consts(q.bits);
    if (fixed > kLayersSmem) return false;
    int slots = (kLayersSmem - fixed) / slot;
    if (slots > kMaxSlots) slots = kMaxSlots;
    if (slots < 3) return false;
    p.slots = slots;
    p.off_const = slots * slot_weights(q.bits);
    p.off_x = p.off_const + slots * slot_consts(q.bits);
    p.off_red = p.off_x + kLayerWarps * p.warp_bytes;
    plan->smem = fixed + slots * slot;
    // the plan's memory
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t r = at; at += (bytes + 255) & ~(size_t)255; return r; };
    take(sizeof(StepLayer) * q.layers);
    plan->off_xw = take((size_t)q.hidden * 4);
    plan->off_qkv = take((size_t)3 * q.hidden * 4);
    plan->off_att = take((size_t)q.hidden * 4);
    plan->off_act = take((size_t)q.inter * 4);
    plan->off_part = take((size_t)q.heads * kMaxSplit * hd * 8);
    plan->off_ml = take((size_t)q.heads * kMaxSplit * (hd / 32) * 16);
    plan->off_tag = take(4);
    plan->bytes = at;
    return true;
}

bool aligned16(const void* q) { return ((uintptr_t)q & 15u) == 0; }

}  // namespace

}  // namespace b200gptq

using namespace b200gptq;

extern "C" {

B200GPTQ_API size_t b200gptq_step_plan_bytes(const b200gptq_step_shape* shape) {
    StepPlan plan = {};
    return shape && plan_step(*shape, &plan) ? plan.bytes : 0;
}
B200GPTQ_API size_t b200gptq_step_table_bytes(int layers) { return layers > 0 ? sizeof(StepLayer) * (size_t)layers : 0; }

B200GPTQ_API int b200gptq_step_plan_create(const b200gptq_step_shape* shape, const b200gptq_step_layer* layers, void* table,
                                           b200gptq_step_plan** out) {
    if (!shape || !layers || !table || !out || !shape->pos || (shape->rope && (!shape->cos_t || !shape->sin_t))) return B200GPTQ_ERR_NULL_POINTER;
    StepPlan plan = {};
    if (!plan_step(*shape, &plan)) return B200GPTQ_ERR_SHAPE;
    StepParams& p = plan.params;
    const EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) { set_last_cuda_error((int)cudaErrorNotSupported); return B200GPTQ_ERR_CUDA; }
    auto map = [&](CUtensorMap* m, CUtensorMapDataType type, const void* base, cuuint64_t cols, cuuint64_t rows, int size, cuuint32_t box_cols,
                   cuuint32_t box_rows, CUtensorMapSwizzle swizzle) {
        const cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * size};
        const cuuint32_t box[2] = {box_cols, box_rows}, one[2] = {1, 1};
        return encode(m, type, 2, const_cast<void*>(base), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    StepLayer* to = static_cast<StepLayer*>(table);
    for (int l = 0; l < shape->layers; ++l) {
        const b200gptq_step_layer& from = layers[l];
        StepLayer layer;
        memset(&layer, 0, sizeof(layer));
        for (int i = 0; i < 4; ++i) {
            const b200gptq_step_linear& w = from.linear[i];
            const LinearShape& s = p.lin[i];
            if (!w.qweight || !w.qzeros || !w.scales) return B200GPTQ_ERR_NULL_POINTER;
            if (!aligned16(w.qweight) || !aligned16(w.qzeros) || !aligned16(w.scales)) return B200GPTQ_ERR_ALIGNMENT;
            if (w.x_perm && i == kDown) return B200GPTQ_ERR_SHAPE;
            const cuuint64_t N = (cuuint64_t)s.strips * kStripCols, groups = (s.units + s.per_group - 1) / s.per_group;
            if (!map(&layer.w[i], CU_TENSOR_MAP_DATA_TYPE_INT32, w.qweight, N, (cuuint64_t)s.K / 32 * shape->bits, 4, kStripCols,
                     kSlotUnits * 4 * shape->bits, CU_TENSOR_MAP_SWIZZLE_128B) ||
                !map(&layer.s[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, w.scales, N, groups, 2, kStripCols, kSlotUnits, CU_TENSOR_MAP_SWIZZLE_NONE) ||
                !map(&layer.z[i], CU_TENSOR_MAP_DATA_TYPE_INT32, w.qzeros, s.zero_words, groups, 4, slot_zero_words(shape->bits), kSlotUnits,
                     CU_TENSOR_MAP_SWIZZLE_NONE)) {
                set_last_cuda_error((int)cudaErrorInvalidValue);
                return B200GPTQ_ERR_CUDA;
            }
            layer.at.bias[i] = static_cast<const __half*>(w.bias);
        }
        for (int i = 0; i < 3; ++i) layer.at.perm[i] = from.linear[i].x_perm;
        const void* norms[4] = {from.norm_w[0], from.norm_w[1], from.norm_b[0], from.norm_b[1]};
        for (int i = 0; i < 4; ++i)
            if (norms[i] ? !aligned16(norms[i]) : (i < 2 || !shape->rms)) return norms[i] ? B200GPTQ_ERR_ALIGNMENT : B200GPTQ_ERR_NULL_POINTER;
        for (int i = 0; i < 2; ++i) {
            layer.at.norm_w[i] = static_cast<const __half*>(norms[i]);
            layer.at.norm_b[i] = shape->rms ? nullptr : static_cast<const __half*>(norms[2 + i]);
        }
        if (!from.k_cache || !from.v_cache) return B200GPTQ_ERR_NULL_POINTER;
        if (!aligned16(from.k_cache) || !aligned16(from.v_cache)) return B200GPTQ_ERR_ALIGNMENT;
        layer.at.k_cache = static_cast<__half*>(from.k_cache);
        layer.at.v_cache = static_cast<__half*>(from.v_cache);
        memcpy(to + l, &layer, sizeof(layer));
    }
    p.cos_t = static_cast<const __half*>(shape->cos_t);
    p.sin_t = static_cast<const __half*>(shape->sin_t);
    p.pos = static_cast<const long long*>(shape->pos);
    // (the limit is the kernel's, not this plan's: the same for all, or a plan of less would refuse the launches of one of more)
    B200GPTQ_CUDA_TRY(cudaFuncSetAttribute(plan.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLayersSmem));
    int resident = 0;
    B200GPTQ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, plan.kernel, kLayerThreads, plan.smem));
    if (resident < 1) return B200GPTQ_ERR_TOO_LARGE;
    StepPlan* made = new (std::nothrow) StepPlan(plan);
    if (!made) return B200GPTQ_ERR_CUDA;
    *out = reinterpret_cast<b200gptq_step_plan*>(made);
    return B200GPTQ_OK;
}

B200GPTQ_API int b200gptq_step_plan_run(const b200gptq_step_plan* handle, void* memory, void* x, void* workspace, void* stream) {
    if (!handle || !memory || !x || !workspace) return B200GPTQ_ERR_NULL_POINTER;
    if (((uintptr_t)memory & 255u) || !aligned16(x)) return B200GPTQ_ERR_ALIGNMENT;
    const StepPlan* plan = reinterpret_cast<const StepPlan*>(handle);
    StepParams p = plan->params;
    unsigned char* m = static_cast<unsigned char*>(memory);
    p.layers = reinterpret_cast<const StepLayer*>(m);
    p.x = static_cast<__half*>(x);
    p.xw = reinterpret_cast<uint32_t*>(m + plan->off_xw);
    p.qkv = reinterpret_cast<uint32_t*>(m + plan->off_qkv);
    p.att = reinterpret_cast<uint32_t*>(m + plan->off_att);
    p.act = reinterpret_cast<uint32_t*>(m + plan->off_act);
    p.part = reinterpret_cast<unsigned long long*>(m + plan->off_part);
    p.part_ml = reinterpret_cast<unsigned long long*>(m + plan->off_ml);
    p.tag = reinterpret_cast<unsigned int*>(m + plan->off_tag);
    p.status = reinterpret_cast<unsigned int*>(workspace);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count());
    cfg.blockDim = dim3(kLayerThreads);
    cfg.dynamicSmemBytes = plan->smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;       // (every CTA is resident, or the launch is refused)
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {&p};
    const cudaError_t e = cudaLaunchKernelExC(&cfg, plan->kernel, args);
    if (e == cudaErrorCooperativeLaunchTooLarge) {       // (part of the device is withheld from this process)
        (void)cudaGetLastError();
        return B200GPTQ_ERR_TOO_LARGE;
    }
    B200GPTQ_CUDA_TRY(e);
    return B200GPTQ_OK;
}

B200GPTQ_API void b200gptq_step_plan_destroy(b200gptq_step_plan* handle) { delete reinterpret_cast<StepPlan*>(handle); }

}  // extern "C"
