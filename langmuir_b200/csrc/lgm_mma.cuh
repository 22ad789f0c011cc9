// lgm_mma.cuh -- the culled pair sum with r^2 from the tensor cores.
//
// u = r^2 - 1/2 of every (target, source) pair is one small matrix product:
// with the target row
//     A = (x, y, z, tt >> 10, tt & 1023, 1024, 1, 0),                 tt = |t|^2
// and the source column
//     B = (-2x', -2y', -2z', 1024, 1, D >> 10, (D & 1023) - 1/2, 0),  D = |s|^2
// A . B = tt + D - 2 t.s - 1/2.  Every entry is exact in FP16 (integers up to
// 2048 and half-integers below 1024: the lattice limit 6 L^2 < 2^22 gives
// coordinates up to 835 and squares below 2^21), and every product and partial
// sum is a multiple of 1/2 below 2^22 in magnitude, hence exact in the FP32
// accumulators in any order: u has the bits the FP32 tiles of lgm_pairs.cuh
// compute.
//
// Bound: the MUFU pipe, one reciprocal square root per pair examined, 16 per
// SM and clock.  The FP32 tiles spend 3 packed FMAs, the vote and the operand
// loads per 64 pairs beside it and kept it 45% busy; here one
// mma.sync.m16n8k8 gives 128 pairs, and a warp issues 4 instructions per 32
// pairs against 8 clocks of MUFU.  (mma.sync, not tcgen05: the accumulators
// are wanted in registers.  Reading them back from tensor memory takes about
// 7 clocks per 32 values and SM quadrant, as long as the MUFU itself: that
// form measured 86 us where the FP32 tiles take 94, 56 of them without any
// arithmetic.)
//
// Layout: column 2t + i of multiplication m (of 8) is source 2m + i of group
// t of four live groups, so that lane (g, t) = (lane / 4, lane % 4) gets, over
// the eight multiplications, all 16 sources of group t in order for the rows
// g, g + 8 of each row tile: a FP32 run stays in one thread and adds in source
// order, as in the FP32 tiles.  The four groups need not be neighbours: each
// warp packs the live ones of its own 32 targets.
//
// Work: a warp takes items {segment of 32 targets, range of source chunks}
// from a counter, with the live groups of the range in a bit mask from the
// cull; items hold about the same number of live groups, so no order and no
// barrier is needed.  Source fragments go straight from L2 to registers, one
// batch of four groups ahead of the arithmetic.
#pragma once

#include <cuda_fp16.h>

#include "lgm_cull.cuh"

namespace lgm {

constexpr int kSeg = 32;          // targets of a segment: a warp's
constexpr int kMmaWarps = 4;      // warps per CTA
constexpr int kMmaThreads = kMmaWarps * 32;
constexpr int kMmaCtas = 4;       // CTAs per SM (a register bound)
constexpr int kItemGroups = 24;   // live groups per item, about
constexpr int kMaxItemsPerSeg = 16;
constexpr int kCullSegs = kCullThreads / 32;  // segments per cull block

__device__ __forceinline__ uint32_t half2_bits(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 half2_floats(uint32_t b) {
    return __half22float2(*reinterpret_cast<const __half2*>(&b));
}

// A target's row.  pad: a slot past the last target (its mark meets a zero in
// the product; the cull reads it).
__device__ __forceinline__ uint4 target_row(int x, int y, int z, bool pad) {
    const int tt = x * x + y * y + z * z;
    return make_uint4(half2_bits((float)x, (float)y), half2_bits((float)z, (float)(tt >> 10)),
                      half2_bits((float)(tt & 1023), 1024.f), half2_bits(1.f, pad ? 1.f : 0.f));
}

// A source's column, four words.  Word w of source e of a group lies at word
// (4 (e & 1) + w) * 8 + e / 2 of the group's 64: a lane's eight fragments are
// then 32 consecutive bytes.
__device__ __forceinline__ void store_source(uint32_t* __restrict__ frag, float* __restrict__ q1,
                                             int dst, int x, int y, int z, float q) {
    const int d = x * x + y * y + z * z;
    const int e = dst % kGroup;
    uint32_t* g = frag + (size_t)(dst / kGroup) * 64 + (e & 1) * 32 + (e >> 1);
    g[0] = half2_bits(-2.f * x, -2.f * y);
    g[8] = half2_bits(-2.f * z, 1024.f);
    g[16] = half2_bits(1.f, (float)(d >> 10));
    g[24] = half2_bits((float)(d & 1023) - 0.5f, 0.f);
    q1[dst] = q;
}

// chunk_boxes_body over these records.
__device__ __forceinline__ void chunk_boxes_mma_body(const PairArgs& A, const CullArgs& C,
                                                     const int chunk) {
    const int n_chunks = A.dyn ? A.dyn[0] : A.n_chunks;
    chunk_boxes_reset(C, chunk);
    if (chunk >= n_chunks) return;
    const int j = chunk * CH + (int)threadIdx.x, e = j % kGroup;
    const uint32_t* g = A.frag + (size_t)(j / kGroup) * 64 + (e & 1) * 32 + (e >> 1);
    const float2 xy = half2_floats(g[0]), zw = half2_floats(g[8]);
    chunk_boxes_reduce(C, chunk, A.q1[j] != 0.f, (int)(-0.5f * xy.x), (int)(-0.5f * xy.y),
                       (int)(-0.5f * zw.x));
}

// The items of a segment from its mask bytes: an item begins at the first live
// chunk, and where the live groups ahead of a chunk pass a multiple of K (at
// least a chunk's groups, so that every cut is one item on).  begin[i]: the
// first chunk of item i, begin[items] the end of the last.  One warp; each
// lane reads the bytes that it wrote.
__device__ __forceinline__ int item_cuts(const uint8_t* mask, int n_chunks, int K, int* begin) {
    const int lane = (int)threadIdx.x & 31;
    int run = 0;       // live groups ahead of this round's chunks
    int last_ex = -1;  // those ahead of the last live chunk (-1: none yet)
    int last_c = -1;
    for (int c0 = 0; c0 < n_chunks; c0 += 32) {
        const int c = c0 + lane;
        const int cnt = c < n_chunks ? __popc((unsigned)mask[c]) : 0;
        const unsigned nz = __ballot_sync(0xffffffffu, cnt > 0);
        if (nz == 0u) continue;
        int inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        const int ex = run + inc - cnt;
        const unsigned below = nz & ((1u << lane) - 1u);
        const int pe = __shfl_sync(0xffffffffu, ex, below ? 31 - __clz(below) : 0);
        const int prev = below ? pe : last_ex;
        if (cnt > 0 && (prev < 0 || ex / K != prev / K)) begin[ex / K] = c;
        const int top = 31 - __clz(nz);
        last_ex = __shfl_sync(0xffffffffu, ex, top);
        last_c = c0 + top;
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
    const int nit = last_ex / K + 1;
    if (lane == 0) begin[nit] = last_c + 1;
    __syncwarp();
    return nit;
}

// One warp per segment: the byte of live groups of every chunk (bit g: group
// g's box comes within the cutoff of the segment's box) and the segment's
// items of per_item live groups (more where they would be over max_items).
__device__ __forceinline__ void cull_mma_body(const CullArgs& C, const int block, const int prob) {
    __shared__ int s_begin[kCullSegs][kMaxItemsPerSeg + 1];
    const int n_chunks = C.dyn ? C.dyn[0] : C.n_chunks;
    const int t_phys = C.dyn ? C.dyn[1] : C.t_phys;
    const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5;
    const int seg = block * kCullSegs + warp;
    if (seg >= C.max_tiles) return;
    if (seg * kSeg >= t_phys) {
        if (lane == 0) C.tile_items[seg] = 0;
        return;
    }
    Box sb;
    {
        int xl = 32767, yl = 32767, zl = 32767, xh = -32768, yh = -32768, zh = -32768;
        const int p = seg * kSeg + lane;
        if (p < t_phys) {
            const uint4 r = C.tgt16[p];
            const float2 xy = half2_floats(r.x), zt = half2_floats(r.y), ip = half2_floats(r.w);
            if (ip.y == 0.f) {
                xl = xh = (int)xy.x;
                yl = yh = (int)xy.y;
                zl = zh = (int)zt.x;
            }
        }
        warp_box(xl, yl, zl, xh, yh, zh);
        sb = make_box(xl, yl, zl, xh, yh, zh);
    }
    uint8_t* mask = C.gmask + (size_t)seg * C.mask_stride;
    int live = 0;  // this lane's
    for (int c0 = 0; c0 < n_chunks; c0 += 32) {
        const int c = c0 + lane;
        const unsigned near =
            __ballot_sync(0xffffffffu, c < n_chunks && box_gap2(sb, C.cbox[c]) < C.c2);
        unsigned byte = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            if (!((near >> (4 * w)) & 15u)) continue;  // warp-uniform
            const int g = (c0 + 4 * w) * kGroupsPerChunk + lane;
            const bool on = ((near >> (4 * w + (lane >> 3))) & 1u) && box_gap2(sb, C.gbox[g]) < C.c2;
            const unsigned b = __ballot_sync(0xffffffffu, on);
            if ((lane >> 2) == w) byte = (b >> (8 * (lane & 3))) & 0xffu;
        }
        if (c < n_chunks) mask[c] = (uint8_t)byte;
        live += __popc(byte);
    }
    const int total = __reduce_add_sync(0xffffffffu, live);
    const int K = max(C.per_item, (total + C.max_items - 1) / C.max_items);
    const int nit = total == 0 ? 0 : item_cuts(mask, n_chunks, K, s_begin[warp]);
    int base = 0, at = 0;
    if (lane == 0) {
        base = nit ? atomicAdd(C.item_count, nit) : 0;
        at = nit && C.list_count ? atomicAdd(C.list_count, nit) : base;
        C.tile_first[seg] = base;
        C.tile_items[seg] = nit;
    }
    base = __shfl_sync(0xffffffffu, base, 0);
    at = __shfl_sync(0xffffffffu, at, 0);
    for (int i = lane; i < nit; i += 32) {
        const int b = s_begin[warp][i], e = s_begin[warp][i + 1];
        C.items[at + i] = make_int4(seg, b, e, base + i);
        if (C.item_prob) C.item_prob[at + i] = prob;
    }
}

// D = A B, m16n8k8, FP16 in, FP32 out.
__device__ __forceinline__ void mma1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 "
        "{%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(b), "f"(0.f));
}

// A lane's eight B fragments of a batch (columns of group gb) and the 16
// charges of group gq.
__device__ __forceinline__ void load_frag(uint4 (&f)[2], const PairArgs& A, int gb, int lane) {
    const uint4* p = reinterpret_cast<const uint4*>(A.frag) + (size_t)gb * 16 +
                     (((lane >> 2) & 1) * 4 + (lane & 3)) * 2;
    f[0] = p[0];
    f[1] = p[1];
}
__device__ __forceinline__ void load_charges(float4 (&q)[4], const PairArgs& A, int gq) {
    const float4* c = reinterpret_cast<const float4*>(A.q1) + (size_t)gq * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = c[i];
}

// Two sources (u, q: r^2 - 1/2 and charges) of one target, in order.
//
// TAB: w(r^2) from the shared-memory table, entry k = r^2 at tab + k * 4 (8 for
// PATH 2), by the lanes inside the cutoff; the float r^2 + 2^21 (2^20) holds
// 4 r^2 (8 r^2) in its low mantissa bits, and tab carries minus its exponent.
// Else 1/r by MUFU, with the correction table s_tab for Gaussian charges (the
// clamped entry tab_k is NaN: past it fminf gives 1/r).
template <int KIND, int PATH, bool TAB>
__device__ __forceinline__ void two_pairs(float u0, float u1, float q0, float q1, unsigned ulim,
                                          uint32_t tab, int tab_k, const float* s_tab, float& acc,
                                          double& acc64) {
    const unsigned k0 = __float_as_uint(u0), k1 = __float_as_uint(u1);
    if constexpr (TAB) {
        constexpr float kBias = PATH == 2 ? 1048576.5f : 2097152.5f;
        const float2 ix = __fadd2_rn(f2(u0, u1), f2(kBias, kBias));
        const uint32_t a0 = __float_as_uint(ix.x) + tab, a1 = __float_as_uint(ix.y) + tab;
        if constexpr (PATH == 2) {
            fma_tab64_if_below(acc64, (double)q0, a0, k0, ulim);
            fma_tab64_if_below(acc64, (double)q1, a1, k1, ulim);
        } else {
            fma_tab_if_below(acc, q0, a0, k0, ulim);
            fma_tab_if_below(acc, q1, a1, k1, ulim);
        }
    } else {
        const float2 r2 = __fadd2_rn(f2(u0, u1), f2(0.5f, 0.5f));
        float wx = rsqrt_mufu(r2.x), wy = rsqrt_mufu(r2.y);
        if constexpr (KIND == 1) {
            wx = fminf(s_tab[min(__float_as_int(r2.x + 8388608.f) & 0x7fffff, tab_k)], wx);
            wy = fminf(s_tab[min(__float_as_int(r2.y + 8388608.f) & 0x7fffff, tab_k)], wy);
        }
        fma_if_below(acc, q0, wx, k0, ulim);
        fma_if_below(acc, q1, wy, k1, ulim);
    }
}

// The pair sum over the items (see the file comment).  Rows g + 8k, k = 0..3,
// are a lane's targets; its sums run over the groups its quad position took,
// and the four lanes of a quad are added at the item's end.
//
// LM of a batch's eight multiplications take w(r^2) from a table in shared
// memory, the others from the MUFU (PATH 0): the two pipes then share the
// work.  For PATH 0 the table is built here, by the same MUFU instruction (and
// Gaussian correction) on every integer below c^2, so both ways give the same
// bits.  PATH 1 and 2 take all from their tables.
template <int KIND, int PATH, int LM, bool NORM, class PS>
__device__ __forceinline__ void pair_items_mma(const PS& P) {
    static_assert(PATH != 2 || !NORM, "the FP64-table path carries no FP32 run norms");
    static_assert(PATH == 0 || LM == 8, "the table paths read their tables");
    const int nit = P.count();
    const PairArgs& A0 = P.first();
    extern __shared__ __align__(128) unsigned char smem[];
    float* s_tab = reinterpret_cast<float*>(smem);
    __shared__ int s_list[kMmaWarps][256 + 4];  // live groups: 32 chunks' and those left over
    if constexpr (PATH == 2) {
        double* s_tab64 = reinterpret_cast<double*>(smem);
        for (int k = threadIdx.x; k <= A0.tab_k; k += kMmaThreads) s_tab64[k] = A0.tab64[k];
    } else if constexpr (PATH == 0 && LM > 0) {
        const int n = P.table_entries();
        for (int k = threadIdx.x; k < n; k += kMmaThreads) {
            float w = rsqrt_mufu((float)k);
            if (KIND == 1) w = fminf(A0.tab[min(k, A0.tab_k)], w);
            s_tab[k] = w;
        }
    } else if constexpr (KIND == 1 || PATH == 1) {
        for (int k = threadIdx.x; k <= A0.tab_k; k += kMmaThreads) s_tab[k] = A0.tab[k];
    }
    if constexpr (KIND == 1 || LM > 0) __syncthreads();
    const uint32_t tab = smem_addr(smem) - (PATH == 2 ? 0x49800000u : 0x4a000000u);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & 3, g8 = lane >> 2;
    int* list = s_list[warp];

    // Every warp starts with an item of its own and claims the next one while
    // it works (the claim's round trip overlaps the item); the claims begin
    // past the first items.
    const int warps = (int)gridDim.x * kMmaWarps;
    int it = (int)blockIdx.x + warp * (int)gridDim.x;
    while (it < nit) {
        int prob;
        const int4 r = P.mma_item(it, prob);
        int next = 0;
        if (lane == 0) next = warps + atomicAdd(P.work(), 1);
        const PairArgs& A = P.A(prob);
        const CullArgs& C = P.C(prob);
        const int seg = r.x, t_phys = A.dyn ? A.dyn[1] : A.t_phys, tab_k = A.tab_k;
        const unsigned ulim = __float_as_uint(A.c2 - 0.5f);
        uint32_t a[4];  // rows g8 + 8k, halves 2t and 2t + 1
        {
            const uint32_t* row =
                reinterpret_cast<const uint32_t*>(A.tgt16 + (size_t)seg * kSeg) + t;
#pragma unroll
            for (int k = 0; k < 4; ++k) a[k] = row[(g8 + 8 * k) * 4];
        }
        double acc64[4] = {0.0, 0.0, 0.0, 0.0};
        float nrm[4] = {0.f, 0.f, 0.f, 0.f};
        const uint8_t* mask = C.gmask + (size_t)seg * C.mask_stride;
        int left = 0, examined = 0;
        for (int c0 = r.y; c0 < r.z; c0 += 32) {
            // the live groups of the next 32 chunks, behind those left over
            const int c = c0 + lane;
            unsigned byte = c < r.z ? mask[c] : 0u;
            const int cnt = __popc(byte);
            int inc = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            int at = left + inc - cnt;
            while (byte) {
                list[at++] = c * kGroupsPerChunk + __ffs((int)byte) - 1;
                byte &= byte - 1;
            }
            int total = left + __shfl_sync(0xffffffffu, inc, 31);
            examined += total - left;
            const bool last = c0 + 32 >= r.z;
            if (last && lane < ((4 - total) & 3)) list[total + lane] = A.pad_group;
            if (last) total = (total + 3) & ~3;
            __syncwarp();
            const int nb = total / 4;
            // the next batch's fragments are in flight over this one's
            // arithmetic; its charges are not (16 more registers cost a CTA)
            uint4 fcur[2], fnext[2];
            if (nb > 0) load_frag(fcur, A, list[lane >> 3], lane);
#pragma unroll 1
            for (int b = 0; b < nb; ++b) {
                float4 q[4];
                load_charges(q, A, list[4 * b + t]);
                if (b + 1 < nb) load_frag(fnext, A, list[4 * b + 4 + (lane >> 3)], lane);
                const uint32_t bf[8] = {fcur[0].x, fcur[0].y, fcur[0].z, fcur[0].w,
                                        fcur[1].x, fcur[1].y, fcur[1].z, fcur[1].w};
                const float qs[16] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w,
                                      q[2].x, q[2].y, q[2].z, q[2].w, q[3].x, q[3].y, q[3].z, q[3].w};
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int m = 0; m < 8; ++m)
#pragma unroll
                    for (int rt = 0; rt < 2; ++rt) {
                        float d[4];
                        mma1688(d, a[2 * rt], a[2 * rt + 1], bf[m]);
                        // spread over the batch: m * LM / 8 steps LM times
                        constexpr int lm = LM;
                        if ((m + 1) * lm / 8 != m * lm / 8) {
                            two_pairs<KIND, PATH, true>(d[0], d[1], qs[2 * m], qs[2 * m + 1], ulim,
                                                        tab, tab_k, s_tab, acc[2 * rt],
                                                        acc64[2 * rt]);
                            two_pairs<KIND, PATH, true>(d[2], d[3], qs[2 * m], qs[2 * m + 1], ulim,
                                                        tab, tab_k, s_tab, acc[2 * rt + 1],
                                                        acc64[2 * rt + 1]);
                        } else {
                            two_pairs<KIND, 0, false>(d[0], d[1], qs[2 * m], qs[2 * m + 1], ulim,
                                                      tab, tab_k, s_tab, acc[2 * rt],
                                                      acc64[2 * rt]);
                            two_pairs<KIND, 0, false>(d[2], d[3], qs[2 * m], qs[2 * m + 1], ulim,
                                                      tab, tab_k, s_tab, acc[2 * rt + 1],
                                                      acc64[2 * rt + 1]);
                        }
                    }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (PATH != 2) acc64[k] += (double)acc[k];
                    if (NORM) nrm[k] += fabsf(acc[k]);
                }
                fcur[0] = fnext[0];
                fcur[1] = fnext[1];
            }
            left = total - 4 * nb;
            int keep = 0;
            if (lane < left) keep = list[4 * nb + lane];
            __syncwarp();
            if (lane < left) list[lane] = keep;
        }
        // the quad's sums, then lane t keeps row g8 + 8t
        double out = 0.0;
        float on = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            double s = acc64[k];
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (t == k) out = s;
            if (NORM) {
                float n = nrm[k];
                n += __shfl_xor_sync(0xffffffffu, n, 1);
                n += __shfl_xor_sync(0xffffffffu, n, 2);
                if (t == k) on = n;
            }
        }
        const int loc = g8 + 8 * t;
        if (seg * kSeg + loc < t_phys) {
            A.part[(size_t)r.w * kSeg + loc] = out;
            if (NORM) A.part_norm[(size_t)r.w * kSeg + loc] = on;
        }
        if (C.examined && lane == 0)
            atomicAdd(C.examined, (unsigned long long)examined * kGroup * kSeg);
        it = __shfl_sync(0xffffffffu, next, 0);
    }
}

// Dynamic shared memory: the table alone, `entries` of `elem` bytes.
inline size_t mma_smem_bytes(int entries, int elem) { return (size_t)entries * elem + 16; }
// PATH 0: cutoffs whose table of w(r^2) leaves the SM's CTAs their shared
// memory; past it every term is taken from the MUFU.
constexpr int kMmaTabEntries = 11000;
// LM of the MUFU path with a table (of 0 .. 8).  Point charges, 20,970 on
// 256x256x16 with images, pair kernel: 0 66 us, 2 59, 3 57, 4 61, 5 68.
// Gaussian charges, 128x128x64: 3 86 us, 4 80, 5 80, 8 103 (their MUFU terms
// read the correction table as well).
constexpr int kMmaTabPoint = 3, kMmaTabGauss = 4;

// Live groups per item and items per segment, at most, for `segs` segments
// against `groups` source groups.  Items of kItemGroups end the kernel within
// a few microseconds of one another; with many targets there are items enough
// for that anyway, and larger ones write fewer partials; with few, smaller
// ones occupy the GPU (not in a batch: its other replicas do).  max_items
// bounds the partials' memory; a segment with more live groups than that many
// items hold gets larger ones.
inline void mma_items(long long segs, int groups, bool batch, int* per_item, int* max_items) {
    const long long few = segs * groups / 16384;  // about two items a warp, a quarter live
    int per = segs > 8192 ? 3 * kItemGroups : kItemGroups;
    if (!batch && few < per) per = few < kGroupsPerChunk ? kGroupsPerChunk : (int)few;
    *per_item = per;
    *max_items = std::min(groups / per + 1, segs > 8192 ? kMaxItemsPerSeg / 2 : kMaxItemsPerSeg);
}

// Items that a call of at most so many segments and groups writes, at most (not in
// a batch).  Fewer segments may mean more items: room by this bound serves every
// smaller call too, such as one captured after a larger one has run.
inline size_t mma_item_room(long long segs, int groups) {
    const long long most = groups / kGroupsPerChunk + 1;  // items are never smaller
    const long long few = std::min<long long>(segs, 8192) * std::min<long long>(kMaxItemsPerSeg, most);
    const long long many = segs > 8192 ? segs * std::min<long long>(kMaxItemsPerSeg / 2, most) : 0;
    return (size_t)std::max(few, many);
}

template <int KIND, int PATH, int LM, bool NORM = false>
__global__ void __launch_bounds__(kMmaThreads, PATH == 2 ? kMmaCtas - 1 : kMmaCtas) pair_kernel_mma(PairArgs A, CullArgs C) {
    pdl_wait();
    pdl_trigger();
    pair_items_mma<KIND, PATH, LM, NORM, OneProblem>(OneProblem{A, C});
}

// The culled replicas of a batch (point charges): the items of all of them in
// one list, item g of problem prob[g].
struct MmaList {
    const PairArgs* pa;
    const CullArgs* ca;
    const int4* items;
    const int* prob;
    int* counts;   // [2]: items in the list, items claimed
    int any;       // a problem of the list
    int tab;       // entries of the w(r^2) table: the largest cutoff^2
    __device__ __forceinline__ int count() const { return counts[0]; }
    __device__ __forceinline__ int* work() const { return counts + 1; }
    __device__ __forceinline__ int4 mma_item(int g, int& p) const {
        p = prob[g];
        return items[g];
    }
    __device__ __forceinline__ const PairArgs& A(int p) const { return pa[p]; }
    __device__ __forceinline__ const CullArgs& C(int p) const { return ca[p]; }
    __device__ __forceinline__ const PairArgs& first() const { return pa[any]; }
    __device__ __forceinline__ int table_entries() const { return tab; }
};
template <int LM, bool NORM>
__global__ void __launch_bounds__(kMmaThreads, kMmaCtas) pair_kernel_mma_list(MmaList L) {
    pair_items_mma<0, 0, LM, NORM, MmaList>(L);
}

static __global__ void __launch_bounds__(CH) chunk_boxes_mma_kernel(PairArgs A, CullArgs C) {
    pdl_wait();
    pdl_trigger();
    chunk_boxes_mma_body(A, C, (int)blockIdx.x);
}

static __global__ void __launch_bounds__(kCullThreads) cull_mma_kernel(CullArgs C) {
    pdl_wait();
    pdl_trigger();
    cull_mma_body(C, (int)blockIdx.x, 0);
}

}  // namespace lgm
