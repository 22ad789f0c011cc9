// lgm_small.cuh -- a whole call of few sources in one kernel.
//
// The general chain (sort, records, boxes, cull, pair sum, finalize) is seven
// launches, 35-40 us however small the call.  With few sources every CTA can
// sort all of them in shared memory, write their fragments there and sum its
// own segments of 32 targets against them: one launch, no scratch in global
// memory, and the potentials go straight to the caller's buffer (for the
// host-buffer call pinned host memory, with the call's number behind them for
// the host to see).
//
// The source order is the chain's, (cell rank, site, index), so the FP32 runs
// of 16 are too, and with them the potentials up to the FP64 order of the runs.
// Targets keep the caller's order: a segment's box is large and culls little,
// but few sources need no culling; an image term's box still drops the sources
// far from the electrode.
#pragma once

#include "lgm_mma.cuh"

namespace lgm {

constexpr int kSmallThreads = 256, kSmallWarps = kSmallThreads / 32;
constexpr size_t kSmallSmem = 96 * 1024;  // dynamic shared memory, at most
// Sources of a call in this form, at most: its sort's places in s_list and the index
// in its keys hold 2048.
constexpr int kSmallSources = 2048;
// The calls this form is the faster one for.  fp64: terms from FP64 tables; mufu: point
// charges' from the MUFU.
inline bool small_size(int n, long long t, int nterms, bool fp64, bool mufu, bool all_sites) {
    // The chain sorts the targets too, and culls; this form sorts the sources again in
    // every CTA, by counting up to 512 of them, in some microseconds more beyond that.
    // us a device call, this form and the chain, 256x256x16, cutoff 50:
    //   128 sources, 2^27 pairs 63 and 298; 512, 2^26 58 and 56, 2^27 72 and 85
    //   1024 sources, 2^24 pairs 28 and 31, 2^25 33 and 34, 2^27 77 and 61
    //   1500 sources, 2^23 pairs 43 and 30; 2048, 2^25 52 and 33
    // Past 1024 sources the sort sets the time, and the line is one CTA an SM (148 segments
    // of 32): 2000 sources, 4000 targets 32 and 30 (host call 59 and 60), 42 and 39 when
    // each call is waited for, 18 and 19 a call with three streams at work (1260 sources,
    // 2520 targets, three terms: 15 and 19), since one launch leaves room for the others'.
    // FP64 terms: 512 sources, 2^25 pairs 46 and 46; 800, 2^23 36 and 33, 2^24 44 and 34;
    //   1024, 2^22 25 and 32, 2^24 47 and 35.
    // Every site: a segment is a run along x and culls well.  MUFU: 1024 sources on 2^20
    //   sites 137 and 245, 2048 230 and 285 (cutoff 10 141 and 169), on 2^18 199 and 219
    //   (108 and 100), on 2^14 51 and 36.  FP64 terms, 2^20 sites: 100 sources 110 and
    //   197, 400 184 and 235 (the tile 187), 700 247 and 274 (the tile 229).
    const long long pairs = n * t * nterms;
    if (all_sites ? n <= (fp64 ? 400 : 1024) : n <= 512 && !fp64) return true;
    if (all_sites && mufu && t >= 1ll << 19) return true;
    if (n <= 512 || (n <= 1024 && !(fp64 && !all_sites))) return pairs <= 1ll << 25;
    return n <= 1024 ? pairs <= 1ll << 23 : t <= 148 * kSeg;
}

struct SmallArgs {
    const int32_t *src, *q;   // n sources
    int n;
    const int32_t* tgt;       // t targets (null: target g is site g)
    int t;
    int X, Y, XY, volume, drains;
    int shift, cells_x, cells_y, ncells;
    const int32_t* cell_rank;
    unsigned terms;
    float c2;
    const float* tab;         // as PairArgs
    const double* tab64;
    int tab_k;
    double prefactor;
    double* out;
    unsigned* err;
    int split;                // warps per segment: 1, 2, 4 or 8
    unsigned* done;           // CTAs done (zero between calls)
    unsigned long long* flag; // null, or where the last CTA writes {call, error word}
    unsigned call;
};

// Bytes of shared memory ahead of the table: the source fragments and charges
// of `groups` groups (and a group of padding), the group boxes.
__host__ __device__ inline size_t small_records(int groups) {
    return (size_t)(groups + 1) * (256 + 64 + sizeof(Box));
}
inline int small_keys(int n) {  // the sort's keys, a power of two
    int k = 64;
    while (k < n) k *= 2;
    return k;
}
inline size_t small_smem(int n, int tab_entries, int elem) {
    const int groups = (n + kGroup - 1) / kGroup;
    return small_records(groups) + std::max((size_t)small_keys(n) * 12, (size_t)tab_entries * elem) + 16;
}

// a[0 .. N), N a power of two from 64 on, ascending.  A warp's pairs of a step
// of stride up to 32 lie in its own 64 entries: those steps need no block barrier.
__device__ __forceinline__ void sort_keys(unsigned long long* a, int N) {
    const int tid = threadIdx.x;
    for (int k = 2; k <= N; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int p = tid; p < N / 2; p += kSmallThreads) {
                const int i = 2 * p - (p & (j - 1));
                const unsigned long long x = a[i], y = a[i + j];
                if ((x > y) == ((i & k) == 0)) {
                    a[i] = y;
                    a[i + j] = x;
                }
            }
            // the next step's stride: j / 2, or k at the end of a merge
            if ((j > 1 ? j >> 1 : k) >= 64 || j >= 64) __syncthreads();
            else __syncwarp();
        }
}

template <int KIND, int PATH>
__global__ void __launch_bounds__(kSmallThreads, 2) small_sums(SmallArgs S) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int groups = (S.n + kGroup - 1) / kGroup;
    uint32_t* s_frag = reinterpret_cast<uint32_t*>(smem);                      // [groups + 1][64]
    float* s_q = reinterpret_cast<float*>(s_frag + (size_t)(groups + 1) * 64);  // [groups + 1][16]
    Box* s_box = reinterpret_cast<Box*>(s_q + (groups + 1) * kGroup);           // [groups + 1]
    unsigned char* s_tail = smem + small_records(groups);  // the sort's keys, then the table
    unsigned long long* s_key = reinterpret_cast<unsigned long long*>(s_tail);
    __shared__ double s_part[kSmallWarps][kSeg];
    __shared__ int s_list[kSmallWarps][kSmallSources / kGroup + 4];
    __shared__ unsigned s_err;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, t4 = lane & 3, g8 = lane >> 2;
    pdl_wait();
    pdl_trigger();

    // What comes from outside is asked for at once: the first segment's target,
    // earlier calls' errors, the sources.  (From pinned host memory each round
    // trip is about 2 us.)
    const int segs = (S.t + kSeg - 1) / kSeg, per = kSmallWarps / S.split;
    const int part = warp % S.split, mine = warp / S.split;
    auto target_of = [&](int seg) {
        const int p = seg * kSeg + lane;
        return seg < segs && p < S.t ? (S.tgt ? S.tgt[p] : p) : -1;
    };
    int next_target = target_of((int)blockIdx.x * per + mine);
    const unsigned old_err = S.flag ? *S.err : 0u;
    if (tid == 0) s_err = 0u;
    int N = 64;
    while (N < S.n) N *= 2;
    int* s_q0 = reinterpret_cast<int*>(s_key + N);  // the charges as given
    for (int j = tid; j < N; j += kSmallThreads) {
        unsigned long long key = ~0ull;
        if (j < S.n) {
            const int s = S.src[j];
            s_q0[j] = S.q[j];
            unsigned rank = (unsigned)S.ncells;
            if (s >= 0 && s < S.volume) {
                const int z = s / S.XY, y = s / S.X - z * S.Y, x = s % S.X;
                rank = (unsigned)S.cell_rank[(x >> S.shift) +
                                             S.cells_x * ((y >> S.shift) + S.cells_y * (z >> S.shift))];
            }
            // rank: at most 65536; the site's 31 bits; the index
            key = ((unsigned long long)rank << 43) | ((unsigned long long)(unsigned)(s & 0x7fffffff) << 11) |
                  (unsigned long long)j;
        }
        s_key[j] = key;
    }
    __syncthreads();

    // ---- the sources in the chain's order
    auto record = [&](int slot, unsigned long long key) {
        const int s = (int)((key >> 11) & 0x7fffffffu);
        int x = 0, y = 0, z = 0;
        float q = 0.f;
        if ((int)(key >> 43) < S.ncells) {
            z = s / S.XY;
            y = s / S.X - z * S.Y;
            x = s % S.X;
            q = (float)s_q0[key & 2047u];
        } else {
            atomicOr(&s_err, DEVERR_SOURCE_RANGE);
        }
        store_source(s_frag, s_q, slot, x, y, z, q);
    };
    if (S.n <= 2 * kSmallThreads) {
        // every key's place by counting the smaller ones (fewer barriers)
        const int n2 = (S.n + 1) & ~1;  // key N is ~0
        for (int j = tid; j < S.n; j += kSmallThreads) {
            const unsigned long long key = s_key[j];
            int r = 0;
#pragma unroll 4
            for (int i = 0; i < n2; i += 2) {
                const ulonglong2 o = *reinterpret_cast<const ulonglong2*>(s_key + i);
                r += (o.x < key) + (o.y < key);
            }
            record(r, key);
        }
    } else {
        sort_keys(s_key, N);
        for (int j = tid; j < S.n; j += kSmallThreads) record(j, s_key[j]);
    }
    for (int j = S.n + tid; j < (groups + 1) * kGroup; j += kSmallThreads)
        store_source(s_frag, s_q, j, 0, 0, 0, 0.f);
    __syncthreads();
    for (int j = tid; j < (groups + 1) * kGroup; j += kSmallThreads) {
        // the group's box: the 16 lanes of its sources
        const uint32_t* g = s_frag + (j / kGroup) * 64 + (j & 1) * 32 + ((j % kGroup) >> 1);
        const float2 xy = half2_floats(g[0]), zw = half2_floats(g[8]);
        const int x = (int)(-0.5f * xy.x), y = (int)(-0.5f * xy.y), z = (int)(-0.5f * zw.x);
        const bool on = s_q[j] != 0.f;
        int xl = on ? x : 32767, yl = on ? y : 32767, zl = on ? z : 32767;
        int xh = on ? x : -32768, yh = on ? y : -32768, zh = on ? z : -32768;
        const unsigned half = (j & 16) ? 0xffff0000u : 0x0000ffffu;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            xl = min(xl, __shfl_xor_sync(half, xl, o));
            yl = min(yl, __shfl_xor_sync(half, yl, o));
            zl = min(zl, __shfl_xor_sync(half, zl, o));
            xh = max(xh, __shfl_xor_sync(half, xh, o));
            yh = max(yh, __shfl_xor_sync(half, yh, o));
            zh = max(zh, __shfl_xor_sync(half, zh, o));
        }
        if (j % kGroup == 0) s_box[j / kGroup] = make_box(xl, yl, zl, xh, yh, zh);
    }
    __syncthreads();  // the keys are read: the table takes their place
    float* s_tab = reinterpret_cast<float*>(s_tail);
    if constexpr (PATH == 2) {
        double* tab = reinterpret_cast<double*>(s_tail);
        for (int k = tid; k <= S.tab_k; k += kSmallThreads) tab[k] = S.tab64[k];
    } else if constexpr (KIND == 1 || PATH == 1) {
        for (int k = tid; k <= S.tab_k; k += kSmallThreads) s_tab[k] = S.tab[k];
    }
    if constexpr (KIND == 1 || PATH > 0) __syncthreads();
    const uint32_t tab = smem_addr(s_tail) - (PATH == 2 ? 0x49800000u : 0x4a000000u);

    // ---- segments, `split` warps each
    const int c2 = (int)S.c2;
    const unsigned ulim = __float_as_uint(S.c2 - 0.5f);
    const int lo = part * groups / S.split, hi = (part + 1) * groups / S.split;
    int* list = s_list[warp];
    for (int s0 = (int)blockIdx.x * per; s0 < segs; s0 += (int)gridDim.x * per) {
        const int seg = s0 + mine;
        double out = 0.0;  // of target seg * 32 + g8 + 8 t4
        const int s = next_target;
        next_target = target_of(seg + (int)gridDim.x * per);
        if (seg < segs) {
            // lane l holds target l's site; the rows of this lane's fragments come by shuffle
            const int p = seg * kSeg + lane;
            int x = 0, y = 0, z = 0;
            const bool valid = p < S.t;
            if (valid) {
                if (s < 0 || s >= S.volume + S.drains) {
                    atomicOr(&s_err, DEVERR_TARGET_RANGE);
                } else {
                    z = s / S.XY;
                    y = s / S.X - z * S.Y;
                    x = s % S.X;
                }
            }
#pragma unroll 1
            for (int term = 0; term < 3; ++term) {
                if (!(S.terms & (1u << term))) continue;
                const int xp = term == 0 ? x : term == 1 ? -1 - x : 2 * S.X - 1 - x;
                const uint4 row = target_row(xp, y, z, !valid);
                int xl = valid ? xp : 32767, yl = valid ? y : 32767, zl = valid ? z : 32767;
                int xh = valid ? xp : -32768, yh = valid ? y : -32768, zh = valid ? z : -32768;
                warp_box(xl, yl, zl, xh, yh, zh);
                const Box sb = make_box(xl, yl, zl, xh, yh, zh);
                uint32_t a[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int l = g8 + 8 * k;
                    const uint32_t w0 = __shfl_sync(0xffffffffu, row.x, l);
                    const uint32_t w1 = __shfl_sync(0xffffffffu, row.y, l);
                    const uint32_t w2 = __shfl_sync(0xffffffffu, row.z, l);
                    const uint32_t w3 = __shfl_sync(0xffffffffu, row.w, l);
                    a[k] = t4 == 0 ? w0 : t4 == 1 ? w1 : t4 == 2 ? w2 : w3;
                }
                // this warp's groups within the cutoff
                int total = 0;
                for (int g0 = lo; g0 < hi; g0 += 32) {
                    const int g = g0 + lane;
                    const bool on = g < hi && box_gap2(sb, s_box[g]) < c2;
                    const unsigned m = __ballot_sync(0xffffffffu, on);
                    if (on) list[total + __popc(m & ((1u << lane) - 1u))] = g;
                    total += __popc(m);
                }
                if (lane < ((4 - total) & 3)) list[total + lane] = groups;  // zero charges
                total = (total + 3) & ~3;
                __syncwarp();
                double acc64[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
                for (int b = 0; b < total; b += 4) {
                    const uint4* f = reinterpret_cast<const uint4*>(s_frag) + list[b + (lane >> 3)] * 16 +
                                     (((lane >> 2) & 1) * 4 + t4) * 2;
                    const uint4 f0 = f[0], f1 = f[1];
                    const uint32_t bfr[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
                    const float2* q = reinterpret_cast<const float2*>(s_q + list[b + t4] * kGroup);
                    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        const float2 qs = q[m];
#pragma unroll
                        for (int rt = 0; rt < 2; ++rt) {
                            float d[4];
                            mma1688(d, a[2 * rt], a[2 * rt + 1], bfr[m]);
                            two_pairs<KIND, PATH, PATH != 0>(d[0], d[1], qs.x, qs.y, ulim, tab, S.tab_k,
                                                             s_tab, acc[2 * rt], acc64[2 * rt]);
                            two_pairs<KIND, PATH, PATH != 0>(d[2], d[3], qs.x, qs.y, ulim, tab, S.tab_k,
                                                             s_tab, acc[2 * rt + 1], acc64[2 * rt + 1]);
                        }
                    }
                    if (PATH != 2)
#pragma unroll
                        for (int k = 0; k < 4; ++k) acc64[k] += (double)acc[k];
                }
                __syncwarp();  // the list is read before the next term writes it
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    double s = acc64[k];
                    s += __shfl_xor_sync(0xffffffffu, s, 1);
                    s += __shfl_xor_sync(0xffffffffu, s, 2);
                    if (t4 == k) out = term == 0 ? s : out - s;
                }
            }
        }
        const int loc = g8 + 8 * t4;
        if (S.split > 1) {
            s_part[warp][loc] = out;
            __syncthreads();
            if (part == 0)
                for (int w = 1; w < S.split; ++w) out += s_part[warp + w][loc];
        }
        if (part == 0 && seg < segs && seg * kSeg + loc < S.t)
            S.out[seg * kSeg + loc] = S.prefactor * out;
        if (S.split > 1) __syncthreads();  // the partials are read before the next segments'
    }
    __syncthreads();  // the CTA's results are written
    if (tid != 0) return;
    const unsigned mine_err = s_err;
    if (mine_err) atomicOr(S.err, mine_err);
    if (!S.flag) return;
    // The last CTA tells the host; the counter carries whether any CTA met a
    // site out of range.
    __threadfence_system();
    unsigned before = 0u;
    if (gridDim.x > 1) before = atomicAdd(S.done, mine_err ? 0x10001u : 1u);
    if ((before & 0xffffu) != gridDim.x - 1) return;
    unsigned e = old_err | mine_err;
    if (gridDim.x > 1) {
        *S.done = 0u;
        __threadfence_system();
        if (before >> 16) e |= *reinterpret_cast<volatile unsigned*>(S.err);
    }
    *reinterpret_cast<volatile unsigned long long*>(S.flag) = ((unsigned long long)S.call << 32) | e;
}

}  // namespace lgm
