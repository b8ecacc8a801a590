// Host side of the decode GEMV (gemv_strip.cuh): plan, tensor map, launch.
#include <mutex>
#include <new>

#include "gemv_strip.cuh"

namespace b200gptq {

const void* gemv_strip_kernel_b2(int sub, int mode, int nt, int T, int warps, bool apart, bool split);
const void* gemv_strip_kernel_b3(int sub, int mode, int nt, int T, int warps, bool apart, bool split);
const void* gemv_strip_kernel_b4(int sub, int mode, int nt, int T, int warps, bool apart, bool split);
const void* gemv_strip_kernel_b8(int sub, int mode, int nt, int T, int warps, bool apart, bool split);

struct GemvStripPlan {
    int M, K, N, smem, warps;          // of a CTA: shared memory, warps (with idle ones)
    StripPlan plan;
    CUtensorMap tmap_w, tmap_s, tmap_z;
    const void* kernel;
};

namespace {

constexpr int kSmemMax = 224 * 1024;      // dynamic shared memory of a CTA
constexpr int kRawMax = 48 * 1024;        // largest x (all rows) that a CTA copies whole to gather from

const void* strip_kernel(int bits, int sub, int mode, int nt, int T, int warps, bool apart, bool split) {
    switch (bits) {
        case 2: return gemv_strip_kernel_b2(sub, mode, nt, T, warps, apart, split);
        case 3: return gemv_strip_kernel_b3(sub, mode, nt, T, warps, apart, split);
        case 4: return gemv_strip_kernel_b4(sub, mode, nt, T, warps, apart, split);
        case 8: return gemv_strip_kernel_b8(sub, mode, nt, T, warps, apart, split);
    }
    return nullptr;
}

// Clusters of four (two) CTAs, one to an SM, that run at the same time: a cluster's SMs are neighbours, and what is left over of the
// groups of them that a device has is lost (33 clusters of four on 148 SMs).  Looked up once per device.
int clusters_at_once(int ctas) {
    static std::once_flag once[64];
    static int cached[64][2];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return sm_count() / ctas;
    std::call_once(once[dev], [dev] {
        for (int i = 0; i < 2; ++i) {
            const void* kernel = strip_kernel(4, 1, kOne, 1, 1, 8, false, true);
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 2 << i;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(sm_count() / (2 << i) * (2 << i));
            cfg.blockDim = dim3(32 * 8);
            cfg.dynamicSmemBytes = kSmemMax;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) != cudaSuccess ||
                cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                n = sm_count() / (2 << i);
            }
            cached[dev][i] = n;
        }
    });
    return cached[dev][ctas == 4];
}

}  // namespace

// Groups of whole 32-row blocks, up to 16 rows of x.
bool gemv_strip_supported(int M, int K, int N, int bits, int group_size) {
    (void)bits;
    return M >= 1 && M <= 16 && N % kStripCols == 0 && K % 32 == 0 && (group_size % 32 == 0 || group_size >= K);
}
// A gather from a copy of x in shared memory; larger x is gathered by a kernel of its own first.
bool gemv_strip_gathers(int M, int K) { return (size_t)M * K * 2 <= kRawMax; }

int gemv_strip_prepare(GemvStripPlan* p, const int32_t* qweight, const int32_t* qzeros,
                       const __half* scales, bool gather, bool permuted, int M, int K, int N, int bits, int group_size,
                       int ctas_per_sm, int xact) {
    p->M = M; p->K = K; p->N = N;
    StripPlan& s = p->plan;
    s.spg = group_size >= K ? K / 32 : group_size / 32;
    s.groups = (K / 32 + s.spg - 1) / s.spg;
    s.spg_inv = (unsigned int)((0x100000000ULL + s.spg - 1) / s.spg);     // (not used for 1)
    s.gather = gather ? 1 : 0;
    s.xact = xact;
    // a unit lies in one group when groups are whole units (or there is only one)
    const int sub = (s.spg % 4 == 0 || s.groups == 1) ? 1 : 4;
    s.units = (K + kUnit - 1) / kUnit;
    s.strips = N / kStripCols;
    // One CTA per SM: each takes the same whole number of strips.
    s.per_cta = (s.strips + sm_count() - 1) / sm_count();
    // Fewer strips than half the SMs: clusters of two or four CTAs share one, where the units of K that a CTA is spared take longer than
    // the cluster's sum.  Hundredths of a us, from layers of 1024 to 2304 columns one behind the other, 1 to 16 rows of 1024 to 11008 values
    // (600 of them): a unit takes 6 (one row), 7 or 14 (more than eight), the cluster 150 and more with the number of strips, with a gather (every CTA copies x)
    // and 8 bits.  us, unsplit -> split: 4 bits, 11008 x 1024, one row 6.6 -> 4.4, 8 rows 9.4 -> 4.9, 16 rows 17.2 -> 6.4; 11008 x 2304, one row
    // 6.9 -> 6.4, 8 rows 9.9 -> 7.5, 16 rows 17.1 -> 10.4; 8192 x 1536, 3 bits act-order, 4 rows 8.0 -> 6.3.  Below the line 4096 x 1536, one
    // row would be 3.1 -> 3.6 and 1024 x 1024 2.2 -> 2.8; rows in act-order gain less than they vary by from 57 strips on.  All clusters run at
    // once: 34 to 37 strips by four CTAs each were two waves (8192 x 1120, one row 4.8 unsplit, 6.7 by four, 3.7 by two).
    s.split = 1;
    if (ctas_per_sm == 0 && !(permuted && M <= 8 && s.strips > 56))
        for (int split = 4; split > 1 && s.split == 1; split /= 2) {
            const int unit = M == 1 ? 6 : (M <= 8 ? 7 : 14), many = s.strips > 48 ? s.strips - 48 : 0;
            const int cluster = 150 + many + (gather ? 60 + 2 * many : 0) + (bits == 8 ? 60 : 0);
            if (s.strips * split <= sm_count() && 10 * unit * (s.units - s.units / split) > 11 * cluster && s.strips <= clusters_at_once(split))
                s.split = split;
        }
    s.cta_units = (s.units + s.split - 1) / s.split;
    // One and two rows: planes of x where they pay and fit; one row: x kept whole.  Planes take a CTA longer to prepare than x in operand
    // order and save on every strip and unit, so they pay where a warp has several units, or several strips of one.  Times as fast as
    // fp16, in a chain of such layers and with a small kernel before each, as in a decode step:
    //   two strips   K from 3072 on 1.00 to 1.24, but two rows in groups of 32 without a gather 0.87 to 0.98 for 8192 and 9216 (planes leave
    //                room for eight warps, not sixteen); 2048 0.87 to 1.08, 1536 0.85 to 1.10, 1024 0.74 to 0.97; one row of 2 bits there
    //                0.95 to 0.99, 1.00 to 1.18, 0.86 to 1.11; 3 bits, which have more pieces, one row 1.00 to 1.24, with rows picked one
    //                by one (a gather) 0.99 to 1.04, two rows 0.92 to 1.08
    //   three, more  K from 2048 on one row 0.93 to 1.53, two rows of 2 and 4 bits 0.96 to 1.46; 1024 0.86 to 1.15.  Two rows of 3 bits 0.79 to
    //                0.97 up to K = 2048 and 1.02 to 1.16 above, but a step of a decoder (three layers, hidden size 4096, batch 2) takes 191 us with
    //                three strips on planes and 182 without, and 201 with seven on planes and 206 without
    //   one strip    4 bits, one row of 4096 1.02 and 1.03, of 11008 1.11, with a gather of 8192 1.07 and 4096 0.97 and 0.99; two rows with a
    //                gather 1.05 to 1.11, without 1.02 and 0.96
    const int plane_bytes = (s.cta_units * M * 4 * int_factors(sub) + 15) / 16 * 16 + s.cta_units * M * (bits == 3 ? 5 : 4) * 128;
    const bool one_strip = bits == 4 && (M == 1 ? s.cta_units >= (gather ? 64 : 32) : gather && s.cta_units >= 32);
    const bool two_strips = bits == 3 ? M == 1 && !gather
                          : (bits == 2 && M == 1) || (s.cta_units > 16 && !(sub == 4 && M == 2 && !gather && s.cta_units > 32));
    const bool more_strips = bits == 3 ? M == 1 || s.per_cta > 4 : (bits == 2 && M == 1) || s.cta_units >= 16;
    // One row in groups scaled apart, two groups to a product (gemv_strip.cuh): one strip, K from 3072 on 1.08 to 1.18 (11008 x 4096 9.05 -> 7.95 us),
    // 2048 0.96 to 1.02; more strips, K from 1536 on 1.10 to 1.33 (8192 x 8192 9.9 -> 8.1, 4096 x 12288 9.8 -> 8.5), 1024 1.07 to 1.19.
    const bool paired = bits == 4 && sub == 4 && M == 1;
    const bool planes_pay = paired ? s.cta_units > (s.per_cta == 1 ? 16 : 7) : s.per_cta == 1 ? one_strip : (s.per_cta == 2 ? two_strips : more_strips);
    int mode = M <= 2 && int_takes(bits, sub) && planes_pay && plane_bytes <= 96 * 1024 ? kInt : (M == 1 && K <= 65536 ? kOne : kSeveral);
    const int nt = M <= 8 ? 1 : 2;
    s.rows_g = sub == 1 ? 1 : (s.spg == 1 ? 4 : (s.spg == 2 ? 2 : 3));
    // Strips of a pass for W warps: a unit costs about half a strip's work on top of its strips, and the last pass is a whole
    // one.  The rings take at least two slots and what is left of the shared memory.
    // Zero-points of several groups: one box is 3 to 5 % faster (4 bits in groups of 32, 4096 x 4096 4.68 -> 4.46 us; 8 bits, 16 rows of 4096 x
    // 12288 27.5 -> 22.1).  4 bits in several passes of one strip, 16 bytes of a row at a time: a box each is faster up to K = 5120 (4096 x 12288, one
    // row 12.1 -> 10.5, three rows 15.0 -> 13.4; 5120 x 10240 15.2 -> 14.6), slower for 11008 x 12288 (23.6 -> 25.7).
    auto zeros_apart = [&](int t) { return bits % 4 != 0 || (bits == 4 && s.rows_g > 1 && t == 1 && s.per_cta > 1 && s.cta_units <= 64); };
    struct Choice { int W, T, ring, fixed, bufs, cost; };
    auto choose = [&](int W) {
        Choice c = {W, 0, 0, 0, 0, 1 << 30};
        const int tmax = sub == 1 && nt == 1 ? (mode == kInt ? 4 : 3) : 2;
        // (a gather works from a copy of x that the sums overwrite: it needs every unit's x kept)
        // x that is not kept: as many units ahead as leave the weights three slots, one ahead being the least.  Nine rows and
        // more are fetched again in every pass rather than kept where that saves a pass (9216 x 9216, 2 bits, 9 rows: 24 ->
        // 18.5 us).
        for (int bufs = 5; bufs >= (mode == kSeveral && !gather ? 2 : 5) && (nt == 2 || c.bufs != 5); --bufs)
            for (int t = 1; t <= tmax && t <= s.per_cta; ++t) {
                const int slot = slot_bytes(bits, t) + const_bytes(bits, t, s.rows_g, zeros_apart(t));
                const int others = (s.split - 1) * M * kStripCols * 4, sums = W * M * t * kStripCols * 4, copy = gather || mode == kOne || (mode == kInt && bits != 4) ? M * K * 2 : 0;
                const int x = mode == kInt ? plane_bytes
                            : (mode == kOne ? s.cta_units * kUnit * 2 : (bufs == 5 ? s.cta_units : bufs * W) * M * kXPitch * 2);
                const int f = x + (sums > copy ? sums : copy) + others + 1024, r = (kSmemMax - f) / (W * slot);
                const int cost = ((s.per_cta + t - 1) / t) * (2 * t + 1);
                const int least = bufs == 3 || bufs == 4 ? 3 : 2;
                if (bufs != 5 && bufs > 2 && s.cta_units / W < bufs - 1) continue;
                if (f < kSmemMax && r >= least && (cost < c.cost || (cost == c.cost && bufs == c.bufs))) c = {W, t, r, f, bufs, cost};
            }
        return c;
    };
    // Sixteen warps hide the latency of a unit better (4096 x 4096, 4 bits: 3.9 against 4.4 us, 11008 x 4096: 7.8 against
    // 9.8), but their rings may only hold narrow passes (4096 x 12288: 8.1 against 6.2, and 12 % of a Llama-7B step), short K
    // leaves some idle and a long row of x leaves their rings little room (36864 x 9216, 3 bits: 47 against 43).  Sixteen rows
    // of x take more than half of a thread's registers.
    Choice c = choose(8);
    if (mode == kOne && !gather) {
        // A long row in operand order and its copy, 4 bytes per value, leave the rings little room or none (8 bits from 39 000
        // values on, 3 and 4 bits from 46 000).  The form for several rows keeps x once, or a few units of it, and is taken where
        // that allows wider passes (4 bits, 40960 x 8192: 59 against 48 us; 8 bits, 32768 x 8192: 66 against 45).
        mode = kSeveral;
        const Choice several = choose(8);
        if (!c.T || several.cost < c.cost) c = several;
        else mode = kOne;
    }
    if (nt == 1 && ctas_per_sm <= 1) {
        const Choice w = choose(16);
        const bool pays = s.cta_units >= 16 && 10 * w.cost <= 11 * c.cost && (mode != kOne || K <= 16384);
        if (w.T && (ctas_per_sm == 1 || !c.T || pays)) c = w;
    }
    if (!c.T) return B200GPTQ_ERR_TOO_LARGE;
    const int W = c.W, T = c.T;
    s.passes = (s.per_cta + T - 1) / T;
    s.x_bufs = c.bufs == 5 ? 2 : c.bufs;
    if (c.bufs != 5) mode = kTurns;
    if (mode == kInt && paired) mode = kIntOne;
    const int longest = ((s.cta_units + W - 1) / W) * s.passes;
    const int sums = W * M * T * kStripCols * 4, copy = gather || mode == kOne || (mode == kInt && bits != 4) ? M * K * 2 : 0;
    s.others = sums > copy ? sums : copy;
    s.ring = c.ring < longest ? c.ring : longest;
    if (s.ring > kMaxRing) s.ring = kMaxRing;
    p->warps = W + idle_warps(W, mode == kSeveral, nt);
    const bool apart = zeros_apart(T);
    p->smem = W * s.ring * (slot_bytes(bits, T) + const_bytes(bits, T, s.rows_g, apart)) + c.fixed;
    p->kernel = strip_kernel(bits, sub, mode, nt, T, W, apart, s.split > 1);
    if (!p->kernel) return B200GPTQ_ERR_SHAPE;
    // (only the one that is used: raising the limit loads a kernel, and there are a hundred)
    B200GPTQ_CUDA_TRY(cudaFuncSetAttribute(p->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    const EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) { set_last_cuda_error((int)cudaErrorNotSupported); return B200GPTQ_ERR_CUDA; }
    auto map = [&](CUtensorMap* m, CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims,
                   const cuuint64_t* strides, const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
        const cuuint32_t estr[3] = {1, 1, 1};
        return encode(m, type, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    // qweight [K/32*bits, N] as {32 columns, word-rows, N/32 strips}; scales [G, N]; qzeros as one run of words.  What lies
    // past the end reads as zero.
    const cuuint64_t wd[3] = {kStripCols, (cuuint64_t)(K / 32 * bits), (cuuint64_t)s.strips}, ws[2] = {(cuuint64_t)N * 4, kStripCols * 4};
    const cuuint32_t wb[3] = {kStripCols, (cuuint32_t)(4 * bits), (cuuint32_t)T};
    const cuuint64_t sd[2] = {(cuuint64_t)N, (cuuint64_t)s.groups}, ss[1] = {(cuuint64_t)N * 2};
    const cuuint32_t sb[2] = {(cuuint32_t)(T * kStripCols), (cuuint32_t)s.rows_g};
    const bool rows_of_zeros = !apart;      // qzeros as [G, N/32*bits], or as one run of words
    const cuuint64_t zd[2] = {(cuuint64_t)(rows_of_zeros ? 1 : s.groups) * (N / 32 * bits), (cuuint64_t)s.groups};
    const cuuint64_t zs[1] = {(cuuint64_t)(N / 32 * bits) * 4};
    const cuuint32_t zb[2] = {(cuuint32_t)zero_words(bits, T), (cuuint32_t)s.rows_g};
    if (!map(&p->tmap_w, CU_TENSOR_MAP_DATA_TYPE_INT32, 3, qweight, wd, ws, wb, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !map(&p->tmap_s, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, scales, sd, ss, sb, CU_TENSOR_MAP_SWIZZLE_NONE) ||
        !map(&p->tmap_z, CU_TENSOR_MAP_DATA_TYPE_INT32, rows_of_zeros ? 2 : 1, qzeros, zd, zs, zb, CU_TENSOR_MAP_SWIZZLE_NONE)) {
        set_last_cuda_error((int)cudaErrorInvalidValue);
        return B200GPTQ_ERR_CUDA;
    }
    return B200GPTQ_OK;
}

int gemv_strip_run(const GemvStripPlan* p, const __half* x, const int32_t* x_perm,
                   const __half* bias, __half* y, void* workspace, cudaStream_t stream) {
    unsigned int* status = reinterpret_cast<unsigned int*>(workspace);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p->plan.split > 1 ? p->plan.strips * p->plan.split : (p->plan.strips < sm_count() ? p->plan.strips : sm_count()));
    cfg.blockDim = dim3(32 * p->warps);
    cfg.dynamicSmemBytes = p->smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = p->plan.split;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p->plan.split > 1 ? 2 : 1;
    int M = p->M, K = p->K, N = p->N;
    void* args[] = {const_cast<CUtensorMap*>(&p->tmap_w), const_cast<CUtensorMap*>(&p->tmap_s),
                    const_cast<CUtensorMap*>(&p->tmap_z), &x, &x_perm, &bias, &y, &M, &K, &N,
                    const_cast<StripPlan*>(&p->plan), &status};
    B200GPTQ_CUDA_TRY(cudaLaunchKernelExC(&cfg, p->kernel, args));
    return B200GPTQ_OK;
}

GemvStripPlan* gemv_strip_plan_create(const int32_t* qweight, const int32_t* qzeros, const __half* scales, bool gather, bool permuted, int M, int K, int N, int bits, int group_size,
                                      int ctas_per_sm, int xact, int* status_out) {
    GemvStripPlan* p = new (std::nothrow) GemvStripPlan;
    if (!p) { *status_out = B200GPTQ_ERR_CUDA; return nullptr; }
    *status_out = gemv_strip_prepare(p, qweight, qzeros, scales, gather, permuted, M, K, N, bits, group_size, ctas_per_sm, xact);
    if (*status_out != B200GPTQ_OK) { delete p; return nullptr; }
    return p;
}
void gemv_strip_plan_destroy(GemvStripPlan* p) { delete p; }

int gemv_strip_dispatch(const __half* x, const int32_t* qweight, const int32_t* qzeros, const __half* scales,
                        const int32_t* x_perm, bool permuted, const __half* bias, __half* y, int M, int K, int N, int bits, int group_size,
                        void* workspace, int ctas_per_sm, int xact, cudaStream_t stream) {
    GemvStripPlan p;
    if (int st = gemv_strip_prepare(&p, qweight, qzeros, scales, x_perm != nullptr, permuted, M, K, N, bits, group_size, ctas_per_sm, xact)) return st;
    return gemv_strip_run(&p, x, x_perm, bias, y, workspace, stream);
}

}  // namespace b200gptq
