// lgm_api.cu -- C ABI of the Coulomb path: context, buffers, launches.
//
// Host side of the drop-in for OpenClHelper (src/langmuirCore/openclhelper.cpp):
// validation with status codes instead of qFatal, device buffers that stay
// resident, and the prep -> pair -> finalize launch sequence on one stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "langmuir_b200.h"
#include "lgm_context.hpp"
#include "lgm_cull.cuh"
#include "lgm_mma.cuh"
#include "lgm_small.cuh"

using namespace lgm;

namespace {

thread_local std::string g_create_error;

constexpr int kMaxSplits = 64;
// The host-buffer call of few sources: bytes its CTAs may read over the bus (a
// copy to the device costs about 5 us), and polls of the kernel's word before
// the stream is waited for (a few milliseconds).
constexpr size_t kZeroCopyBytes = 96 * 1024;
constexpr int kFlagPolls = 1 << 20;
constexpr int kDrainIds = 35;       // Grid::m_specialAgentReserve (cubicgrid.cpp:22)

lgm_status fail(lgm_ctx* c, lgm_status st, const std::string& msg) {
    if (c) c->err = msg;
    return st;
}

lgm_status cuda_fail(lgm_ctx* c, cudaError_t e, const char* what) {
    std::string m = std::string(what) + ": " + cudaGetErrorString(e);
    return fail(c, LGM_ERR_CUDA, m);
}

#define LGM_CUDA(c, call)                                    \
    do {                                                     \
        cudaError_t e_ = (call);                             \
        if (e_ != cudaSuccess) return cuda_fail((c), e_, #call); \
    } while (0)

template <class T>
lgm_status grow_device(lgm_ctx* c, T** p, size_t* cap, size_t need) {
    if (need <= *cap && *p) return LGM_OK;
    size_t n = std::max(need, (size_t)(*cap * 3 / 2));
    n = std::max<size_t>(n, 256);
    if (*p) LGM_CUDA(c, cudaFree(*p));
    *p = nullptr;
    *cap = 0;
    LGM_CUDA(c, cudaMalloc(reinterpret_cast<void**>(p), n * sizeof(T)));
    *cap = n;
    return LGM_OK;
}

template <class T>
lgm_status grow_host(lgm_ctx* c, T** p, size_t* cap, size_t need) {
    if (need <= *cap && *p) return LGM_OK;
    size_t n = std::max(need, (size_t)(*cap * 3 / 2));
    n = std::max<size_t>(n, 256);
    if (*p) LGM_CUDA(c, cudaFreeHost(*p));
    *p = nullptr;
    *cap = 0;
    LGM_CUDA(c, cudaMallocHost(reinterpret_cast<void**>(p), n * sizeof(T)));
    *cap = n;
    return LGM_OK;
}

// ---- prep kernels ---------------------------------------------------------

// Source records (see lgm_pairs.cuh) in spatial order (prep_records).  The sources were
// counted into bins by lattice cell (bins_both) and scattered by bin
// (scatter_both, in no particular order inside a bin); slot j of that scatter
// takes its final place here: the bin's start plus its rank inside the bin by
// (site, index), so the order depends on the sources alone and the sums are
// deterministic.  bins_end[b] is the end of bin b after the scatter.  Entries
// n .. n_pad-1 are zero-charge padding at the origin; their weight is
// (q*m) * y = 0 * finite = 0.
//
// fmt selects the records a call's pair kernel reads: kFmtFloat (the FP32 and
// FP64 tiles), kFmtHalf (the tensor-core sums), or both (the autotuner).
constexpr int kFmtFloat = 1, kFmtHalf = 2;
struct Records {
    int fmt;
    float4* geo;
    float2* qq;
    float4* tgt;
    uint32_t* frag;
    float* q1;
    uint4* tgt16;
};

// The record of one source at slot dst; empty: a zero-charge record at the origin.
__device__ __forceinline__ void write_source(const Records& R, int dst, int x, int y, int z,
                                             float q) {
    if (R.fmt & kFmtFloat) {
        const float a = -2.f * x, b = -2.f * y, c = -2.f * z;
        const float d = (float)(x * x + y * y + z * z) - 0.5f;
        R.geo[2 * dst] = make_float4(a, a, b, b);
        R.geo[2 * dst + 1] = make_float4(c, c, d, d);
        R.qq[dst] = make_float2(q, q);
    }
    if (R.fmt & kFmtHalf) store_source(R.frag, R.q1, dst, x, y, z, q);
}

__device__ __forceinline__ void prep_source(const int j, const int32_t* __restrict__ s,
                                            const int32_t* __restrict__ q, int n, int n_pad,
                                            const int32_t* __restrict__ key,
                                            const int32_t* __restrict__ tmp,
                                            const int32_t* __restrict__ bins_end, int X, int Y,
                                            int XY, int volume, const Records& R, unsigned* err) {
    // (one more group of padding, behind the last chunk: lgm_mma.cuh's pad_group)
    if (j >= n_pad + kGroup || (j >= n_pad && !(R.fmt & kFmtHalf))) return;
    if (j >= n) {
        if (j < n_pad) write_source(R, j, 0, 0, 0, 0.f);
        else store_source(R.frag, R.q1, j, 0, 0, 0, 0.f);
        return;
    }
    const int i = tmp[j];
    const int b = key[i];
    const int lo = b > 0 ? bins_end[b - 1] : 0, hi = bins_end[b];
    const int si = s[i];
    int rank = 0;
    for (int k = lo; k < hi; ++k) {
        const int o = tmp[k];
        const int so = s[o];
        rank += (so < si) | ((so == si) & (o < i));
    }
    if (si < 0 || si >= volume) {
        atomicOr(err, DEVERR_SOURCE_RANGE);
        write_source(R, lo + rank, 0, 0, 0, 0.f);
    } else {
        // Grid::getIndexX/Y/Z (cubicgrid.cpp:132-145), as kernel.cl:266-268.
        const int z = si / XY, y = si / X - z * Y, x = si % X;
        write_source(R, lo + rank, x, y, z, (float)q[i]);
    }
}

// Physical targets: for each requested term the (possibly mirrored) target
// position.  Term order in `tgt`: direct, left image, right image (present
// ones only), each block t_pad long.  A left image is the direct sum at
// x' = -1 - x (distance x_i + x_j + 1, cubicgrid.cpp:117-120); a right image
// at x' = 2X - 1 - x.  all_sites != 0: target g is lattice site g (kernel 1).
__device__ __forceinline__ void prep_target(const int j, const int32_t* __restrict__ ts, int t,
                                            int t_pad, int all_sites, unsigned terms, int X,
                                            int Y, int XY, int volume, int shift,
                                            const int32_t* __restrict__ tkey,
                                            const int32_t* __restrict__ ttmp,
                                            const int32_t* __restrict__ bins_end,
                                            int32_t* __restrict__ perm, const Records& R,
                                            unsigned* err) {
    if (j >= t_pad) return;  // j: the scatter slot
    // The target scattered to slot j goes to physical slot g: its bin's start
    // plus its rank inside the bin by index (perm[g] = target).  A target's
    // sum is split into the work items of its tile (the culled tiles), so its
    // tile, and with it the rounding of the item partials' sum, must not
    // depend on the scatter's order: with this rank the sums are a function
    // of the target list and the source set.  bins_end[b] is the end of bin b
    // after the scatter.
    // Every site (kernel 1): a cell's bin holds all its sites, and the rank
    // by index is the site's raster position inside the (edge-clipped) cell.
    int g = j, x = 0, y = 0, z = 0;
    if (j < t) {
        const int i = ttmp[j];
        const int b = tkey[i];
        const int lo = b > 0 ? bins_end[b - 1] : 0;
        const int sg = all_sites ? i : ts[i];
        if (sg < 0 || sg >= volume + kDrainIds) {
            atomicOr(err, DEVERR_TARGET_RANGE);
        } else {
            z = sg / XY; y = sg / X - z * Y; x = sg % X;
        }
        int rank = 0;
        if (all_sites) {
            const int c = 1 << shift;
            const int x0 = (x >> shift) << shift, y0 = (y >> shift) << shift;
            const int z0 = (z >> shift) << shift;
            const int cw = min(c, X - x0), ch = min(c, Y - y0);
            rank = ((z - z0) * ch + (y - y0)) * cw + (x - x0);
        } else {
            const int hi = bins_end[b];
            for (int k = lo; k < hi; ++k) rank += ttmp[k] < i;
        }
        g = lo + rank;
        perm[g] = i;
    }
    int slot = 0;
    for (int term = 0; term < 3; ++term) {
        if (!(terms & (1u << term))) continue;
        int xp = x;
        if (term == 1) xp = -1 - x;
        if (term == 2) xp = 2 * X - 1 - x;
        // padding slots (g >= t) carry a mark (w = -1): the cull leaves them
        // out of the tiles' boxes, and their sums are never read
        if (R.fmt & kFmtFloat)
            R.tgt[(size_t)slot * t_pad + g] =
                make_float4((float)xp, (float)y, (float)z,
                            g < t ? (float)(xp * xp + y * y + z * z) : -1.f);
        if (R.fmt & kFmtHalf) R.tgt16[(size_t)slot * t_pad + g] = target_row(xp, y, z, g >= t);
        ++slot;
    }
}

// The target records (blocks [0, tb)) and the source records (the blocks
// after), one launch.
__global__ void prep_records(int tb, const int32_t* __restrict__ ts, int t, int t_pad,
                             int all_sites, unsigned terms, int X, int Y, int XY, int volume,
                             int shift, const int32_t* __restrict__ tkey,
                             const int32_t* __restrict__ ttmp,
                             const int32_t* __restrict__ tbins_end, int32_t* __restrict__ perm,
                             const Records R, const int32_t* __restrict__ s,
                             const int32_t* __restrict__ q, int n, int n_pad,
                             const int32_t* __restrict__ skey, const int32_t* __restrict__ stmp,
                             const int32_t* __restrict__ sbins_end, unsigned* err) {
    pdl_wait();
    pdl_trigger();
    const int b = (int)blockIdx.x;
    if (b < tb)
        prep_target(b * (int)blockDim.x + (int)threadIdx.x, ts, t, t_pad, all_sites, terms, X, Y,
                    XY, volume, shift, tkey, ttmp, tbins_end, perm, R, err);
    else
        prep_source((b - tb) * (int)blockDim.x + (int)threadIdx.x, s, q, n, n_pad, skey, stmp,
                    sbins_end, X, Y, XY, volume, R, err);
}

// The last kernel of a call clears both bin arrays (their last reader,
// prep_records, has completed), so the next call's bins_both counts into
// zeros without a memset of its own.  Thread i of the grid (one row of the
// block) clears entries i, i + stride, ...
__device__ __forceinline__ void zero_bins(int32_t* __restrict__ bins, int nbins) {
    const int stride = (int)(gridDim.x * blockDim.x);
    for (int i = (int)(blockIdx.x * blockDim.x + threadIdx.x); i < nbins; i += stride) bins[i] = 0;
}

// out[perm[g]] = prefactor * (sum over splits of the direct block - image
// blocks) of physical slot g.
__global__ void finalize(const double* __restrict__ part, int splits, int t_phys, int t,
                         int t_pad, int nterms, double prefactor,
                         const int32_t* __restrict__ perm, double* __restrict__ out,
                         int32_t* __restrict__ bins, int nbins, const unsigned* err,
                         unsigned* err_out) {
    pdl_wait();
    pdl_trigger();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    zero_bins(bins, nbins);
    if (err_out && g == 0) *err_out = *err;
    if (g >= t) return;
    double total = 0.0;
    for (int slot = 0; slot < nterms; ++slot) {
        double s = 0.0;
        const double* p = part + (size_t)slot * t_pad + g;
        // eight loads in flight, then the adds in split order (same bits)
        int sp = 0;
        for (; sp + 8 <= splits; sp += 8) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = p[(size_t)(sp + u) * t_phys];
#pragma unroll
            for (int u = 0; u < 8; ++u) s += v[u];
        }
        for (; sp < splits; ++sp) s += p[(size_t)sp * t_phys];
        total = (slot == 0) ? s : total - s;
    }
    out[perm[g]] = prefactor * total;
}

// Counting sort of the targets and of the sources by lattice cell (the
// spatial order the SKIP and culled pair tiles run in).  bins_both: the bin of
// every target and every source -- the Morton rank of its cell, sites beyond
// the lattice (drains, or ids the prep flags as out of range) in the last bin
// -- and the bin counts (target bins tbins, source bins sbins).
__device__ __forceinline__ int cell_bin(int sg, int X, int Y, int XY, int volume, int shift,
                                        int cells_x, int cells_y,
                                        const int32_t* __restrict__ cell_rank, int ncells) {
    if (sg < 0 || sg >= volume) return ncells;
    const int z = sg / XY, y = sg / X - z * Y, x = sg % X;
    return cell_rank[(x >> shift) + cells_x * ((y >> shift) + cells_y * (z >> shift))];
}

__global__ void bins_both(const int32_t* __restrict__ ts, int t, int all_sites,
                          const int32_t* __restrict__ ss, int n, int X, int Y, int XY, int volume,
                          int shift, int cells_x, int cells_y,
                          const int32_t* __restrict__ cell_rank, int ncells,
                          int32_t* __restrict__ tkey, int32_t* __restrict__ tbins,
                          int32_t* __restrict__ skey, int32_t* __restrict__ sbins,
                          int32_t* __restrict__ done) {
    __shared__ int s_last;
    pdl_wait();
    pdl_trigger();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < t) {
        const int b = cell_bin(all_sites ? g : ts[g], X, Y, XY, volume, shift, cells_x, cells_y,
                               cell_rank, ncells);
        tkey[g] = b;
        atomicAdd(&tbins[b], 1);
    }
    if (g < n) {
        const int b =
            cell_bin(ss[g], X, Y, XY, volume, shift, cells_x, cells_y, cell_rank, ncells);
        skey[g] = b;
        atomicAdd(&sbins[b], 1);
    }
    // The last block to finish turns both counts into exclusive scans in
    // place (the counts were added by atomics in L2; this block read none of
    // them before, and fences after seeing the others done).
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(done, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    block_exclusive_scan(tbins, ncells + 1);
    block_exclusive_scan(sbins, ncells + 1);
    if (threadIdx.x == 0) *done = 0;  // every block has counted itself: ready for the next call
}


// ttmp[slot] = target and stmp[slot] = source: each takes the next slot of
// its bin, in no particular order inside the bin; prep_target and
// prep_source (prep_records) fix the final order.
__global__ void scatter_both(const int32_t* __restrict__ tkey, int t, int32_t* __restrict__ tbins,
                             int32_t* __restrict__ ttmp, const int32_t* __restrict__ skey, int n,
                             int32_t* __restrict__ sbins, int32_t* __restrict__ stmp) {
    pdl_wait();
    pdl_trigger();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < t) ttmp[atomicAdd(&tbins[tkey[g]], 1)] = g;
    if (g < n) stmp[atomicAdd(&sbins[skey[g]], 1)] = g;
}

// out[perm[g]] = prefactor * (sum of the item partials of the direct slot -
// those of the image slots) of target g, for the culled pair sums.  A block
// of 32 x 3 threads takes 32 targets: warp y sums term slot y's partials of
// each target in item order, sixteen items in flight; warp 0 then combines the
// slots through shared memory.
__global__ void __launch_bounds__(96) finalize_items(const double* __restrict__ part,
                                                     const int* __restrict__ tile_first,
                                                     const int* __restrict__ tile_items,
                                                     int tile_size, int t, int t_pad, int nterms,
                                                     double prefactor,
                                                     const int32_t* __restrict__ perm,
                                                     double* __restrict__ out,
                                                     int32_t* __restrict__ bins, int nbins,
                                                     const unsigned* err, unsigned* err_out) {
    constexpr int kRows = 16;  // loads in flight (a tile has at most 32 items)
    __shared__ double s_sum[3][32];
    pdl_wait();
    pdl_trigger();
    const int g = blockIdx.x * 32 + (int)threadIdx.x, slot = (int)threadIdx.y;
    const int dst = slot == 0 && g < t ? perm[g] : 0;  // loaded ahead of the sums
    if (slot == 0) zero_bins(bins, nbins);
    if (err_out && g == 0 && slot == 0) *err_out = *err;
    double sum = 0.0;
    if (g < t && slot < nterms) {
        const int p = slot * t_pad + g;
        const int tile = p / tile_size, loc = p - tile * tile_size;
        const int n = tile_items[tile];
        const double* q = part + (size_t)tile_first[tile] * tile_size + loc;
        for (int i = 0; i < n; i += kRows) {
            double v[kRows];
#pragma unroll
            for (int u = 0; u < kRows; ++u)
                v[u] = i + u < n ? q[(size_t)(i + u) * tile_size] : 0.0;
#pragma unroll
            for (int u = 0; u < kRows; ++u)
                if (i + u < n) sum += v[u];
        }
    }
    s_sum[slot][threadIdx.x] = sum;
    __syncthreads();
    if (slot == 0 && g < t) {
        const int x = (int)threadIdx.x;
        out[dst] = prefactor * (s_sum[0][x] - s_sum[1][x] - s_sum[2][x]);
    }
}

__global__ void fill_zero(double* out, int t, const unsigned* err, unsigned* err_out) {
    pdl_wait();
    pdl_trigger();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (err_out && g == 0) *err_out = *err;
    if (g < t) out[g] = 0.0;
}

// The FP64 precision's tables are laid out up to this much shared memory of the
// culled kernel (cutoff 159; its one CTA an SM is still the faster there).  128x128x8,
// 2622 charges, host call with both images, tables and every term computed: cutoff
// 50 65 us and 132, 90 85 and 134, 150 96 and 136; 400 charges at cutoff 158 62 and
// 133.  The error against extended
// precision halves (1.0e-15 to 5e-16 of the largest sum).
constexpr size_t kF64TableSmem = 200 * 1024;

// FP64 path: every term in double, 1/sqrt and erf of the CUDA runtime.
// Sources staged in shared memory by plain loads; one thread per physical
// target and split.
constexpr int kF64Threads = 256;
constexpr int kF64Tile = 512;

__global__ void __launch_bounds__(kF64Threads)
pair_kernel_f64(const float4* __restrict__ geo, const float2* __restrict__ qq, int n_pad,
                int splits, const float4* __restrict__ tgt, int t_phys, double* __restrict__ part,
                int c2, int kind, double erffactor) {
    __shared__ int4 s_g[kF64Tile];  // x, y, z, q
    pdl_wait();
    pdl_trigger();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int split = blockIdx.y;
    const int j_begin = (int)((long long)split * n_pad / splits);
    const int j_end = (int)((long long)(split + 1) * n_pad / splits);
    float4 tp = p < t_phys ? tgt[p] : make_float4(0.f, 0.f, 0.f, 0.f);
    // target coordinates are exact small integers
    const int tx = (int)tp.x, ty = (int)tp.y, tz = (int)tp.z;
    double acc = 0.0;
    for (int j0 = j_begin; j0 < j_end; j0 += kF64Tile) {
        const int m = min(kF64Tile, j_end - j0);
        __syncthreads();
        for (int k = threadIdx.x; k < m; k += blockDim.x) {
            const float4 g0 = geo[2 * (j0 + k)], g1 = geo[2 * (j0 + k) + 1];
            s_g[k] = make_int4((int)(-0.5f * g0.x), (int)(-0.5f * g0.z), (int)(-0.5f * g1.x),
                               (int)qq[j0 + k].x);
        }
        __syncthreads();
        for (int k = 0; k < m; ++k) {
            const int4 sk = s_g[k];
            const int dx = tx - sk.x, dy = ty - sk.y, dz = tz - sk.z;
            const int r2 = dx * dx + dy * dy + dz * dz;
            if (r2 > 0 && r2 < c2) {
                const double r = (double)r2;
                if (kind == 0) {
                    acc += (double)sk.w * (1.0 / sqrt(r));
                } else {
                    const double rr = sqrt(r);
                    acc += (double)sk.w * erf(erffactor * rr) / rr;
                }
            }
        }
    }
    if (p < t_phys) part[(size_t)split * t_phys + p] = acc;
}

// ---- launch plumbing --------------------------------------------------------

// Launches a kernel of a call's chain.  With overlap on it carries the
// programmatic stream serialization attribute: the kernel may be scheduled
// while the one ahead of it in the stream is still running, and waits for it
// in pdl_wait() (lgm_device.cuh) before touching memory, so the launch
// latency between the chain's kernels overlaps the kernel ahead.
template <typename... P, typename... A>
cudaError_t launch_chain(bool overlap, void (*k)(P...), dim3 grid, dim3 block, size_t smem,
                         cudaStream_t st, A... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

using PairFn = void (*)(PairArgs);
using CulledFn = void (*)(PairArgs, CullArgs);

// Compiled tile variants of the pair kernel: threads per CTA, target pairs per
// thread, FP32 run length.  fn[0] point/rsqrt, fn[1] gauss/rsqrt, fn[2] table.
// skip: warp-owned spatially sorted targets with the per-source warp vote
// (the rsqrt paths; the table path runs the plain tile).  cull: the work-list
// kernel of lgm_cull.cuh over the live source chunks of each tile, per_item
// chunks per work item (cfn[] instead of fn[]).
struct Variant {
    int nt, rp, sub, skip, cull, per_item;
    PairFn fn[4];
    CulledFn cfn[4];  // [3]: the FP64-table path (culled variants only)
    int ws = 0;       // warp-specialised culled kernel: its stages (0: not)
    int tc = 0;       // r^2 on the tensor cores (lgm_mma.cuh): FP16 records
};
#define LGM_VARIANT_S(NT, RP, SUB, SK)                                                    \
    Variant {                                                                             \
        NT, RP, SUB, SK, 0, 0,                                                            \
            {&pair_kernel<0, 0, NT, RP, SUB, false, SK>,                                  \
             &pair_kernel<1, 0, NT, RP, SUB, false, SK>, &pair_kernel<0, 1, NT, RP, SUB>,  \
             nullptr},                                                                    \
        {                                                                                 \
            nullptr, nullptr, nullptr, nullptr                                            \
        }                                                                                 \
    }
#define LGM_VARIANT(NT, RP, SUB) LGM_VARIANT_S(NT, RP, SUB, false)
#define LGM_VARIANT_SKIP(NT, RP, SUB) LGM_VARIANT_S(NT, RP, SUB, true)
#define LGM_VARIANT_CULL(NT, RP, SUB, K)                                                      \
    Variant {                                                                                 \
        NT, RP, SUB, 1, 1, K, {nullptr, nullptr, nullptr, nullptr}, {                         \
            &pair_kernel_culled<0, 0, NT, RP, SUB>, &pair_kernel_culled<1, 0, NT, RP, SUB>,   \
                &pair_kernel_culled<0, 1, NT, RP, SUB>, &pair_kernel_culled<0, 2, NT, RP, SUB> \
        }                                                                                     \
    }
#define LGM_VARIANT_CULL_WS(NW, RP, SUB, K, S, MINB, PIPE)                                  \
    Variant {                                                                                 \
        NW * 32, RP, SUB, 1, 1, K, {nullptr, nullptr, nullptr, nullptr},                      \
            {&pair_kernel_culled_ws<0, 0, NW, RP, SUB, S, MINB, false, PIPE>,                 \
             &pair_kernel_culled_ws<1, 0, NW, RP, SUB, S, MINB, false, PIPE>,                 \
             &pair_kernel_culled_ws<0, 1, NW, RP, SUB, S, MINB>,                              \
             &pair_kernel_culled_ws<0, 2, NW, RP, SUB, S, MINB>},                             \
            S                                                                                 \
    }
// VOTE: sources per warp vote of the MUFU path (0: none; lgm_cull.cuh)
#define LGM_VARIANT_CULL_WSV(NW, RP, SUB, K, S, MINB, VOTE)                                  \
    Variant {                                                                                 \
        NW * 32, RP, SUB, 1, 1, K, {nullptr, nullptr, nullptr, nullptr},                      \
            {&pair_kernel_culled_ws<0, 0, NW, RP, SUB, S, MINB, false, false, VOTE>,          \
             &pair_kernel_culled_ws<1, 0, NW, RP, SUB, S, MINB, false, false, VOTE>,          \
             &pair_kernel_culled_ws<0, 1, NW, RP, SUB, S, MINB>,                              \
             &pair_kernel_culled_ws<0, 2, NW, RP, SUB, S, MINB>},                             \
            S                                                                                 \
    }
// r^2 on the tensor cores: warps of 32 targets, items by the call's size (mma_items)
#define LGM_VARIANT_MMA                                                                      \
    Variant {                                                                                 \
        kMmaThreads, 1, kGroup, 1, 1, 0,                                                      \
            {nullptr, nullptr, nullptr, nullptr},                                             \
            {&pair_kernel_mma<0, 0, kMmaTabPoint>, &pair_kernel_mma<1, 0, kMmaTabGauss>,      \
             &pair_kernel_mma<0, 1, 8>, &pair_kernel_mma<0, 2, 8>},                           \
            0, 1                                                                              \
    }
const Variant kVariants[] = {
    LGM_VARIANT(128, 4, 16),       LGM_VARIANT(128, 4, 8),        LGM_VARIANT(128, 2, 16),
    LGM_VARIANT(128, 8, 16),       LGM_VARIANT(256, 4, 16),       LGM_VARIANT(64, 4, 16),
    LGM_VARIANT(128, 4, 32),       LGM_VARIANT(256, 2, 16),       LGM_VARIANT_SKIP(128, 4, 32),
    LGM_VARIANT_SKIP(128, 4, 16),  LGM_VARIANT_SKIP(128, 2, 32),  LGM_VARIANT_SKIP(64, 4, 32),
    LGM_VARIANT_SKIP(64, 3, 32),   LGM_VARIANT_SKIP(128, 3, 32),
    LGM_VARIANT_CULL(128, 4, 16, 2), LGM_VARIANT_CULL(128, 4, 16, 1),
    LGM_VARIANT_CULL(128, 4, 16, 4), LGM_VARIANT_CULL(128, 2, 16, 2),
    LGM_VARIANT_CULL(64, 4, 16, 2),  LGM_VARIANT_CULL(128, 4, 8, 2),
    LGM_VARIANT_CULL(64, 2, 16, 2),
    // warp-specialised: (target warps, target pairs, run, chunks per item,
    // stages, CTAs per SM); the register bound counts the producer warp
    LGM_VARIANT_CULL_WS(4, 4, 16, 2, 4, 4, false), LGM_VARIANT_CULL_WS(8, 2, 16, 2, 4, 3, false),
    LGM_VARIANT_CULL_WS(4, 2, 16, 2, 4, 5, false), LGM_VARIANT_CULL_WS(7, 2, 16, 2, 4, 3, false),
    LGM_VARIANT_CULL_WS(4, 4, 16, 4, 4, 4, false),
    // 4 CTAs of 4 target warps and 2 target pairs per thread measured best on
    // the 256x256x16 and 128x128x64 workloads (96 registers; the 5-CTA bound
    // of 72 registers was 36% slower); the next source's r^2 ahead of each
    // vote (PIPE) measured the same
    LGM_VARIANT_CULL_WS(4, 2, 16, 2, 4, 4, true), LGM_VARIANT_CULL_WS(4, 2, 16, 2, 4, 4, false),
    LGM_VARIANT_CULL_WS(2, 2, 16, 2, 4, 6, true), LGM_VARIANT_CULL_WS(4, 2, 16, 3, 4, 4, false),
    LGM_VARIANT_CULL_WS(4, 2, 16, 1, 4, 4, true), LGM_VARIANT_CULL_WS(4, 2, 16, 4, 4, 4, false),
    // one vote per 2 or 4 sources, or none
    LGM_VARIANT_CULL_WSV(4, 2, 16, 2, 4, 4, 2), LGM_VARIANT_CULL_WSV(4, 2, 16, 2, 4, 4, 0),
    LGM_VARIANT_CULL_WSV(4, 2, 16, 2, 4, 4, 4),
    LGM_VARIANT_MMA,
};
constexpr int kNumVariants = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
static_assert(kNumVariants <= (int)(sizeof(lgm_ctx::bps) / sizeof(lgm_ctx::bps[0])),
              "lgm_ctx::bps holds every variant");
// The defaults (choose_variant): r^2 on the tensor cores; for large calls with
// tables the warp-specialised culled tile with 4 target warps, 2 target pairs, runs
// of 16, 2 chunks per item and one vote per 2 sources (2% faster than a vote per
// source on the 256x256x16 and 128x128x64 workloads, the same bits).
constexpr int kDefaultVariant = kNumVariants - 1, kTileVariant = 32;

// The culled kernel of variant V for path index fi and cutoff^2 c2.
CulledFn culled_fn(const Variant& V, int fi, int c2) {
    if (V.tc && fi < 2 && c2 > kMmaTabEntries)
        return fi == 0 ? &pair_kernel_mma<0, 0, 0> : &pair_kernel_mma<1, 0, 0>;
    return V.cfn[fi];
}
const void* kernel_of(const Variant& V, int fi, int c2) {
    return V.cull ? reinterpret_cast<const void*>(culled_fn(V, fi, c2))
                  : reinterpret_cast<const void*>(V.fn[fi]);
}

// Threads of a CTA (a warp-specialised variant adds its producer warp) and
// dynamic shared memory for path index fi with table entries 0 .. tab_k.
int variant_threads(const Variant& V) { return V.nt + (V.ws ? 32 : 0); }
size_t variant_smem(const Variant& V, int fi, int tab_k, int c2) {
    if (V.tc) return mma_smem_bytes(fi < 2 && c2 <= kMmaTabEntries ? c2 : tab_k + 1, fi == 3 ? 8 : 4);
    if (V.ws) return ws_smem_bytes(V.ws, tab_k, fi == 3 ? 8 : 4);
    return fi == 3 ? pair_smem_bytes64(tab_k) : pair_smem_bytes(tab_k);
}

// Targets of a tile.  (The tensor-core variant's is a warp's 32 targets; its
// target_pairs reads 1.)
int variant_tile(const Variant& V) { return V.tc ? kSeg : V.nt * 2 * V.rp; }
int variant_targets_per_thread(const Variant& V) { return V.tc ? 1 : 2 * V.rp; }

int fn_index(int kind, int path) {
    if (path == LGM_PATH_TABLE64) return 3;  // one kernel: the table holds w for the kind
    if (path == LGM_PATH_TABLE) return 2;
    return kind == LGM_GAUSS ? 1 : 0;
}

// Size bucket of a pair launch: half-octaves of physical targets and chunks.
uint64_t tune_key(int kind, int path, int t_phys, int n_chunks) {
    auto hb = [](int x) { return (uint64_t)std::lround(2.0 * std::log2((double)std::max(x, 1))); };
    return ((uint64_t)kind << 60) | ((uint64_t)path << 56) | (hb(t_phys) << 28) | hb(n_chunks);
}

int popcount3(unsigned terms) {
    return ((terms & 1u) ? 1 : 0) + ((terms & 2u) ? 1 : 0) + ((terms & 4u) ? 1 : 0);
}

// Source and target records for a call (see lgm_pairs.cuh).
struct Shape {
    int nterms, n_pad, n_chunks, t_pad, t_phys;
};

Shape shape_of(int n, int t, unsigned terms) {
    Shape sh;
    sh.nterms = popcount3(terms);
    sh.n_pad = (n + CH - 1) / CH * CH;
    sh.n_chunks = sh.n_pad / CH;
    sh.t_pad = (t + 63) / 64 * 64;
    sh.t_phys = sh.nterms * sh.t_pad;
    return sh;
}

// Slices one after another of a block, 256-byte aligned; without a block, their bytes.
struct Cut {
    char* base;
    size_t at;
    template <class T>
    void operator()(T** p, size_t n) {
        if (base) *p = reinterpret_cast<T*>(base + at);
        at += (n * sizeof(T) + 255) / 256 * 256;
    }
};

// The sort of n sources and t targets, and their records.
void cut_records(lgm_ctx* c, Cut& cut, const Shape& sh, int n, int t, int fmt) {
    const size_t ns = (size_t)sh.n_pad + kGroup;
    if (fmt & kFmtFloat) {
        cut(&c->d_geo, (size_t)sh.n_pad * 2);
        cut(&c->d_qq, (size_t)sh.n_pad);
        cut(&c->d_tgt, (size_t)sh.t_phys + 4096);  // room for any variant's widest tile
    }
    if (fmt & kFmtHalf) {
        cut(&c->d_frag, ns * 4);
        cut(&c->d_q1, ns);
        cut(&c->d_tgt16, (size_t)sh.t_phys);  // whole segments: t_pad is a multiple of 64
    }
    cut(&c->d_key, (size_t)t);
    cut(&c->d_perm, (size_t)t);
    cut(&c->d_ttmp, (size_t)t);
    cut(&c->d_skey, (size_t)n);
    cut(&c->d_stmp, (size_t)n);
}

// Sizes of a culled variant's work lists.
struct CulledPlan {
    int tile, tiles, per_item, max_items, mask_stride;
    size_t item_cap;  // room for items: never less than a smaller call's
};
CulledPlan culled_plan(const Variant& V, const Shape& sh) {
    CulledPlan p;
    p.tile = variant_tile(V);
    p.tiles = (sh.t_phys + p.tile - 1) / p.tile;
    p.per_item = V.per_item;
    if (V.tc)
        mma_items(p.tiles, sh.n_chunks * kGroupsPerChunk, false, &p.per_item, &p.max_items);
    else
        p.max_items =
            std::max(1, std::min(kMaxItemsPerTile, (sh.n_chunks + p.per_item - 1) / p.per_item));
    p.mask_stride = (sh.n_chunks + 31) / 32 * 32;
    p.item_cap = V.tc ? mma_item_room(p.tiles, sh.n_chunks * kGroupsPerChunk)
                      : (size_t)p.tiles * p.max_items;
    return p;
}

int splits_for(const lgm_ctx* c, int v, int fi, const Shape& sh, int* tiles_out);
int direct_splits(const lgm_ctx* c, const Shape& sh);
constexpr int kDirect = -1;  // in place of a variant: pair_kernel_f64

// The pair sum of variant v (or kDirect): boxes, live lists, items, partial sums.
void cut_sums(lgm_ctx* c, Cut& cut, const Shape& sh, int v, int fi) {
    if (v == kDirect || !kVariants[v].cull) {
        int tiles;
        const int splits = v == kDirect ? direct_splits(c, sh) : splits_for(c, v, fi, sh, &tiles);
        cut(&c->d_part, (size_t)splits * sh.t_phys);
        return;
    }
    const Variant& V = kVariants[v];
    const CulledPlan p = culled_plan(V, sh);
    cut(&c->d_cbox, (size_t)sh.n_chunks);
    cut(&c->d_gbox, (size_t)sh.n_chunks * kGroupsPerChunk);
    if (V.tc) {
        cut(&c->d_gmask, (size_t)p.tiles * p.mask_stride);
    } else {
        cut(&c->d_live, (size_t)p.tiles * sh.n_chunks);
        cut(&c->d_order, p.item_cap);
        cut(&c->d_oitems, p.item_cap);
    }
    cut(&c->d_items, p.item_cap);
    cut(&c->d_tile_first, (size_t)p.tiles);
    cut(&c->d_tile_items, (size_t)p.tiles);
    cut(&c->d_part, p.item_cap * p.tile);
}

// The scratch of a call, records in format fmt and any of the variants vs; the
// slices of the sums are cut again for each variant.  A new context's first call
// pays for the allocations: the driver serves up to 1 MB in 2 us from pieces of
// 2 MB that it holds, and maps anything larger in 330.  So a call of at most 2 MB
// takes two blocks, a larger one takes one.
constexpr size_t kTwoBlocks = 2 << 20;
lgm_status lay_out(lgm_ctx* c, const Shape& sh, int n, int t, int fmt, int fi,
                   const std::vector<int>& vs) {
    Cut dry{nullptr, 0};
    cut_records(c, dry, sh, n, t, fmt);
    const size_t records = dry.at;
    size_t need = records;
    for (int v : vs) {
        dry.at = records;
        cut_sums(c, dry, sh, v, fi);
        need = std::max(need, dry.at);
    }
    const bool one = need <= c->scratch_cap || need > kTwoBlocks;
    lgm_status s = grow_device(c, &c->d_scratch, &c->scratch_cap, one ? need : records);
    if (s == LGM_OK && !one) s = grow_device(c, &c->d_sums, &c->sums_cap, need - records);
    if (s != LGM_OK) return s;
    c->sums = one ? c->d_scratch + records : c->d_sums;
    Cut cut{c->d_scratch, 0};
    cut_records(c, cut, sh, n, t, fmt);
    return LGM_OK;
}

// Sorts and writes the records of a call that lay_out made room for.
lgm_status prep(lgm_ctx* c, unsigned terms, const int32_t* d_src, const int32_t* d_q, int n,
                const int32_t* d_tgt_site, int t, int all_sites, const Shape& sh, int fmt,
                cudaStream_t st) {
    const lgm_config& cf = c->cfg;
    const Records R{fmt, c->d_geo, c->d_qq, c->d_tgt, c->d_frag, c->d_q1, c->d_tgt16};
    // targets and sources in spatial order: bins, scans, scatters.  Both bin
    // arrays and the bins_both block counter behind them start at zero: the
    // last kernel of the previous call cleared them (bins_both's last block
    // clears the counter), else one memset does.
    if (!c->bins_clean)
        LGM_CUDA(c, cudaMemsetAsync(c->d_bins, 0, sizeof(int32_t) * (2 * c->bins_stride + 4), st));
    c->bins_clean = false;
    const bool ov = c->overlap;
    const int tb = (std::max(t, n) + 255) / 256;
    LGM_CUDA(c, launch_chain(ov, bins_both, tb, 256, 0, st, d_tgt_site, t, all_sites, d_src, n,
                             cf.grid_x, cf.grid_y, c->xy, c->volume, c->cell_shift, c->cells_x,
                             c->cells_y, c->d_cell_rank, c->ncells, c->d_key, c->d_bins,
                             c->d_skey, c->d_sbins, c->d_bins + 2 * c->bins_stride));
    LGM_CUDA(c, launch_chain(ov, scatter_both, tb, 256, 0, st, c->d_key, t, c->d_bins, c->d_ttmp,
                             c->d_skey, n, c->d_sbins, c->d_stmp));
    const int ptb = (sh.t_pad + 255) / 256, psb = (sh.n_pad + kGroup + 255) / 256;
    LGM_CUDA(c, launch_chain(ov, prep_records, ptb + psb, 256, 0, st, ptb, d_tgt_site, t, sh.t_pad,
                             all_sites, terms, cf.grid_x, cf.grid_y, c->xy, c->volume,
                             c->cell_shift, c->d_key, c->d_ttmp, c->d_bins, c->d_perm, R, d_src,
                             d_q, n, sh.n_pad, c->d_skey, c->d_stmp, c->d_sbins, c->d_err));
    return LGM_OK;
}

// Splits of the source range for variant v: as many as fill kSplitWaves
// waves of resident CTAs, never more than the chunks.  With the warp skip the
// CTAs of one launch do uneven work (tiles near few charges, image tiles far
// from the electrode skip most sources), and three waves of smaller CTAs let
// the block scheduler even it out; more waves cost more in the FP64 partials
// that finalize sums than they save (256x256x16 lattice, 20,970 charges,
// images at both electrodes: 1 wave 0.647 ms, 3 waves 0.607 ms, 8 waves
// 0.614 ms per call).
constexpr int kSplitWaves = 3;
int splits_for(const lgm_ctx* c, int v, int fi, const Shape& sh, int* tiles_out) {
    const Variant& V = kVariants[v];
    const int tiles = (sh.t_phys + V.nt * 2 * V.rp - 1) / (V.nt * 2 * V.rp);
    const int capacity = c->sm_count * std::max(1, c->bps[v][fi]);
    *tiles_out = tiles;
    return std::max(1, std::min({kMaxSplits, kSplitWaves * capacity / tiles, sh.n_chunks}));
}

// Splits of the source range for pair_kernel_f64.
int direct_splits(const lgm_ctx* c, const Shape& sh) {
    const int ctas = (sh.t_phys + kF64Threads - 1) / kF64Threads;
    return std::max(1, std::min({kMaxSplits, (c->sm_count * 8) / std::max(1, ctas),
                                 (sh.n_pad + kF64Tile - 1) / kF64Tile}));
}

// Culled variant v: chunk boxes, the cull, the persistent pair kernel (one
// wave of resident CTAs).  *splits_out = 0 tells the caller to finalize from
// the item partials.
lgm_status launch_culled(lgm_ctx* c, int fi, int v, const Shape& sh, const PairArgs& A,
                         cudaStream_t st, int* splits_out) {
    const Variant& V = kVariants[v];
    const CulledPlan p = culled_plan(V, sh);
    const int tiles = p.tiles, grid = c->sm_count * std::max(1, c->bps[v][fi]);
    if (V.nt / 32 > kMaxSegments) return fail(c, LGM_ERR_STATE, "culled variant wider than the cull");
    Cut cut{c->sums, 0};
    cut_sums(c, cut, sh, v, fi);
    PairArgs P = A;
    P.part = c->d_part;
    CullArgs C;
    C.n_chunks = sh.n_chunks;
    C.cbox = reinterpret_cast<Box*>(c->d_cbox);
    C.gbox = reinterpret_cast<Box*>(c->d_gbox);
    C.tgt = c->d_tgt;
    C.t_phys = sh.t_phys;
    C.c2 = c->cfg.electrostatic_cutoff * c->cfg.electrostatic_cutoff;
    C.tile_size = p.tile;
    C.per_item = p.per_item;
    C.max_items = p.max_items;
    C.live = c->d_live;
    C.tgt16 = c->d_tgt16;
    C.gmask = c->d_gmask;
    C.mask_stride = p.mask_stride;
    C.max_tiles = tiles;
    C.live_stride = sh.n_chunks;
    C.items = c->d_items;
    C.item_count = c->d_item_count;
    C.work = c->d_item_count + 1;
    C.tile_first = c->d_tile_first;
    C.tile_items = c->d_tile_items;
    // the items largest first (costs from the pair kernel's warp segments)
    C.warp_targets = 64 * V.rp;
    C.hist = c->d_cost_hist;
    C.order = c->d_order;
    C.oitems = c->d_oitems;
    C.done = c->d_item_count + 2;
    if (c->counting) {
        LGM_CUDA(c, cudaMemsetAsync(c->d_examined, 0, sizeof(unsigned long long), st));
        C.examined = c->d_examined;
        c->count_pending = true;
    }
    const bool ov = c->overlap;
    if (V.tc) {
        LGM_CUDA(c, launch_chain(ov, chunk_boxes_mma_kernel, sh.n_chunks, CH, 0, st, P, C));
        LGM_CUDA(c, launch_chain(ov, cull_mma_kernel, (tiles + kCullSegs - 1) / kCullSegs,
                                 kCullThreads, 0, st, C));
    } else {
        LGM_CUDA(c, launch_chain(ov, chunk_boxes_kernel, sh.n_chunks, CH, 0, st, P, C));
        // its last block orders the items
        LGM_CUDA(c, launch_chain(ov, cull_kernel, tiles, kCullThreads, 0, st, C));
    }
    // timing on: the events bracket the pair kernel alone (recorded again here)
    if (c->timing) LGM_CUDA(c, cudaEventRecord(c->ev_pair0, st));
    LGM_CUDA(c, launch_chain(ov, culled_fn(V, fi, C.c2), grid, variant_threads(V),
                             variant_smem(V, fi, P.tab_k, C.c2), st, P, C));
    c->last.ctas = grid;
    c->last.threads = variant_threads(V);
    c->last.targets_per_thread = variant_targets_per_thread(V);
    c->last.variant = v;
    c->last.splits = 0;
    *splits_out = 0;
    return LGM_OK;
}

lgm_status launch_pair(lgm_ctx* c, int kind, int path, int v, const Shape& sh, cudaStream_t st,
                       int* splits_out) {
    const lgm_config& cf = c->cfg;
    const int fi = fn_index(kind, path);
    if (kVariants[v].cull) {
        PairArgs A;
        A.geo = c->d_geo; A.qq = c->d_qq; A.n_chunks = sh.n_chunks; A.splits = 1;
        A.tgt = c->d_tgt; A.t_phys = sh.t_phys;
        A.frag = c->d_frag; A.q1 = c->d_q1; A.tgt16 = c->d_tgt16;
        A.pad_group = sh.n_chunks * kGroupsPerChunk;
        A.c2 = (float)(cf.electrostatic_cutoff * cf.electrostatic_cutoff);
        A.err = c->d_err;
        if (path == LGM_PATH_TABLE64) {
            A.tab64 = kind == LGM_GAUSS ? c->d_gtab64 : c->d_rtab64;
            A.tab_k = c->rtab_k;  // both hold every r^2 <= c^2 (entries 0 and c^2 are 0)
        } else if (path == LGM_PATH_TABLE) {
            A.tab = kind == LGM_GAUSS ? c->d_gtab : c->d_rtab;
            A.tab_k = kind == LGM_GAUSS ? c->gtab_k : c->rtab_k;
        } else {
            A.tab = c->d_gtab;
            A.tab_k = kind == LGM_GAUSS ? c->gtab_k : 0;
        }
        return launch_culled(c, fi, v, sh, A, st, splits_out);
    }
    int tiles;
    const int splits = splits_for(c, v, fi, sh, &tiles);
    Cut cut{c->sums, 0};
    cut_sums(c, cut, sh, v, fi);
    PairArgs A;
    A.geo = c->d_geo; A.qq = c->d_qq; A.n_chunks = sh.n_chunks; A.splits = splits;
    A.tgt = c->d_tgt; A.t_phys = sh.t_phys; A.part = c->d_part;
    A.c2 = (float)(cf.electrostatic_cutoff * cf.electrostatic_cutoff);
    A.err = c->d_err;
    if (path == LGM_PATH_TABLE) {
        A.tab = kind == LGM_GAUSS ? c->d_gtab : c->d_rtab;  // both hold every r^2 < c^2
        A.tab_k = kind == LGM_GAUSS ? c->gtab_k : c->rtab_k;
    } else {
        A.tab = c->d_gtab;
        A.tab_k = kind == LGM_GAUSS ? c->gtab_k : 0;
    }
    const Variant& V = kVariants[v];
    dim3 grid(tiles, splits);
    LGM_CUDA(c, launch_chain(c->overlap, V.fn[fi], grid, V.nt, pair_smem_bytes(A.tab_k), st, A));
    c->last.ctas = grid.x * grid.y;
    c->last.threads = V.nt;
    c->last.targets_per_thread = 2 * V.rp;
    c->last.variant = v;
    *splits_out = splits;
    return LGM_OK;
}

// Untuned calls with terms from tables that the FP32 tile (kTileVariant) sums
// faster than the tensor-core kernel: its vote skips a table read that no lane of
// the warp needs, where the other's conflicting reads bound it.  `inside` is about
// the pairs within the cutoff.  us a device call, tile and tensor-core kernel:
//   table64, cutoff 50: 2000 sources, 16,000 targets of 256x256x16 54 and 43; 6000,
//   12,000 of 64x64x64 (inside 2^26) 103 and 104; 20,000, 40,000 (2^29) 605 and 667;
//   every site of 64x64x64, 2000 sources 460 and 504, of 256x256x16, 600: 217 and 264
//   table64, cutoff 100: 2000 and 4000 of 128x128x32 (2^22) 56 and 45; 2000 and
//   16,000 (2^24) 70 and 76
//   table, cutoff 150: 2000 and 4000 of 128x128x32 1.14 to 1.18 times faster by the
//   latter; 2000 and 16,000 (2^24) 59 and 64
//   table, every site, 6000 sources: 64x64x64, cutoff 30 417 and 376, 50 743 and 769, 100
//   840 and 990; 92x166x64, 30 747 and 600, 50 1407 and 1309, 70 2070 and 2056, 100 2659
//   and 2888; 256x256x16, 70 938 and 916, 100 1452 and 1491: the cutoff against the
//   lattice's mean side decides (a short one leaves few reads that only the vote skips)
// With terms from the MUFU the tensor-core kernel is never more than 4% behind; but
// its masks grow as targets x sources, twice as fast as the tile's lists, and are
// left alone past 64 GB.
bool tile_faster(const lgm_ctx* c, const Shape& sh, int n) {
    const lgm_config& cf = c->cfg;
    if ((long long)(sh.t_phys / kSeg) * sh.n_chunks > 1ll << 36) return true;
    if (cf.path == LGM_PATH_RSQRT) return false;
    double inside = (double)sh.t_phys * n;
    for (int side : {cf.grid_x, cf.grid_y, cf.grid_z})
        inside *= std::min(1.0, 2.0 * cf.electrostatic_cutoff / side);
    if (cf.path == LGM_PATH_TABLE64)
        return sh.t_phys > 65536 || inside > (cf.electrostatic_cutoff > 60 ? 0x1p24 : 0x1p27);
    const double side = std::cbrt((double)c->volume);
    return (cf.electrostatic_cutoff >= 0.78 * side && sh.t_phys > 200000) ||
           (cf.electrostatic_cutoff > 110 && inside > 0x1p24);
}

int choose_variant(const lgm_ctx* c, int kind, const Shape& sh, int n) {
    int v = tile_faster(c, sh, n) ? kTileVariant : kDefaultVariant;
    if (c->forced_variant >= 0) {
        v = c->forced_variant;
    } else {
        auto it = c->tune_cache.find(tune_key(kind, c->cfg.path, sh.t_phys, sh.n_chunks));
        if (it != c->tune_cache.end()) v = it->second;
    }
    // the FP64-table path is served by the culled variants only
    if (c->cfg.path == LGM_PATH_TABLE64 && !kVariants[v].cull) v = kDefaultVariant;
    return v;
}

// The FP64 precision's sums: with their terms from the FP64 tables (d_rtab64,
// laid out when the culled kernel's shared memory holds them) the TABLE64 path
// does the same arithmetic in FP64, culled, and the terms are rounded once.
// Every term computed in the kernel instead (pair_kernel_f64) stays for larger
// cutoffs and for counting calls, which report no culled pairs.
bool f64_table(const lgm_ctx* c) {
    return c->cfg.precision == LGM_PREC_FP64 && c->d_rtab64 && !c->counting;
}
int sum_path(const lgm_ctx* c) { return f64_table(c) ? LGM_PATH_TABLE64 : c->cfg.path; }

// Entries of the table a one-kernel call holds in shared memory.
int small_table(const lgm_ctx* c, int kind) {
    const int path = sum_path(c);
    if (path == LGM_PATH_TABLE64) return c->rtab_k + 1;
    if (path == LGM_PATH_TABLE) return (kind == LGM_GAUSS ? c->gtab_k : c->rtab_k) + 1;
    return kind == LGM_GAUSS ? c->gtab_k + 1 : 0;
}

using SmallFn = void (*)(SmallArgs);
SmallFn small_fn(int kind, int path) {
    if (path == LGM_PATH_TABLE64) return &small_sums<0, 2>;
    if (path == LGM_PATH_TABLE) return &small_sums<0, 1>;
    return kind == LGM_GAUSS ? &small_sums<1, 0> : &small_sums<0, 0>;
}

// A call of few sources takes the one-kernel form (lgm_small.cuh): up to
// kSmallSources of them and small_pairs unculled pairs, where the chain's
// launches cost more than the pairs it culls, and a table that leaves two CTAs
// their shared memory.
bool small_fits(const lgm_ctx* c, int kind, const Shape& sh, int n, int t, bool all_sites) {
    const bool fp64_terms = sum_path(c) == LGM_PATH_TABLE64;
    const bool mufu = kind == LGM_POINT && sum_path(c) == LGM_PATH_RSQRT;
    return n >= 1 && n <= kSmallSources &&
           small_size(n, t, sh.nterms, fp64_terms, mufu, all_sites) &&
           small_smem(n, small_table(c, kind), fp64_terms ? 8 : 4) <= kSmallSmem;
}

// It does so with no variant forced, no pair counting, and none tuned for the size
// (the FP64 precision has none).  The tuner tries the form where it would serve a
// call with given targets: there its choice stands.
bool small_call(const lgm_ctx* c, int kind, const Shape& sh, int n, int t, bool all_sites) {
    const bool f64 = c->cfg.precision == LGM_PREC_FP64;
    if (f64 ? !f64_table(c) : c->forced_variant >= 0 || c->counting) return false;
    if (!small_fits(c, kind, sh, n, t, all_sites)) return false;
    return f64 || !c->tune_cache.count(tune_key(kind, c->cfg.path, sh.t_phys, sh.n_chunks)) ||
           !small_fits(c, kind, sh, n, t, false);
}

// flag: null, or the host-visible word the last CTA writes {call, error} to.
lgm_status launch_small(lgm_ctx* c, int kind, unsigned terms, const int32_t* src, const int32_t* q,
                        int n, const int32_t* tgt, int t, int all_sites, double* out,
                        cudaStream_t st, unsigned long long* flag, unsigned call) {
    const lgm_config& cf = c->cfg;
    const int path = sum_path(c);
    SmallArgs S{};
    S.src = src; S.q = q; S.n = n;
    S.tgt = all_sites ? nullptr : tgt; S.t = t;
    S.X = cf.grid_x; S.Y = cf.grid_y; S.XY = c->xy; S.volume = c->volume; S.drains = kDrainIds;
    S.shift = c->cell_shift; S.cells_x = c->cells_x; S.cells_y = c->cells_y; S.ncells = c->ncells;
    S.cell_rank = c->d_cell_rank;
    S.terms = terms;
    S.c2 = (float)(cf.electrostatic_cutoff * cf.electrostatic_cutoff);
    if (path == LGM_PATH_TABLE64) S.tab64 = kind == LGM_GAUSS ? c->d_gtab64 : c->d_rtab64;
    else if (path == LGM_PATH_TABLE) S.tab = kind == LGM_GAUSS ? c->d_gtab : c->d_rtab;
    else S.tab = c->d_gtab;
    S.tab_k = small_table(c, kind) - 1;
    S.prefactor = cf.electrostatic_prefactor;
    S.out = out;
    S.err = c->d_err;
    S.done = reinterpret_cast<unsigned*>(c->d_item_count + 3);
    S.flag = flag;
    S.call = call;
    // few segments: a CTA's warps share one, each with a slice of the groups
    const int segs = (t + kSeg - 1) / kSeg, batches = (n + 4 * kGroup - 1) / (4 * kGroup);
    S.split = kSmallWarps;
    while (S.split > 1 && (S.split > batches || segs * S.split > 2 * kSmallWarps * c->sm_count))
        S.split /= 2;
    const int per = kSmallWarps / S.split;
    const int grid = std::min((segs + per - 1) / per, 4 * c->sm_count);
    if (c->timing) LGM_CUDA(c, cudaEventRecord(c->ev_pair0, st));
    LGM_CUDA(c, launch_chain(c->overlap, small_fn(kind, path), grid, kSmallThreads,
                             small_smem(n, S.tab_k + 1, path == LGM_PATH_TABLE64 ? 8 : 4), st, S));
    if (c->timing) {
        LGM_CUDA(c, cudaEventRecord(c->ev_pair1, st));
        c->timed_pending = true;
    }
    c->last.ctas = grid;
    c->last.threads = kSmallThreads;
    c->last.targets_per_thread = 1;
    c->last.variant = cf.precision == LGM_PREC_FP64 ? -1 : kDefaultVariant;
    c->last.kernel_launches = 1;
    c->last.pairs_tested = (int64_t)popcount3(terms) * t * (int64_t)n;
    c->last.splits = 0;
    return LGM_OK;
}

void reset_last(lgm_ctx* c) {
    c->last = lgm_launch_info{};
    c->last.pair_kernel_ms = -1.f;
    c->last.variant = -1;
    c->last.pairs_examined = -1;
    c->timed_pending = false;
    c->count_pending = false;
}

// Shared launch sequence.  d_src/d_q: n sources; d_tgt_site: t targets (or
// all lattice sites when all_sites).  Everything on `st`.
lgm_status launch_potentials(lgm_ctx* c, int kind, unsigned terms, const int32_t* d_src,
                             const int32_t* d_q, int n, const int32_t* d_tgt_site, int t,
                             int all_sites, double* d_out, cudaStream_t st,
                             unsigned* err_out = nullptr) {
    const lgm_config& cf = c->cfg;
    reset_last(c);
    if (t == 0) return LGM_OK;
    if (n == 0) {
        LGM_CUDA(c, launch_chain(c->overlap, fill_zero, (t + 255) / 256, 256, 0, st, d_out, t,
                                 c->d_err, err_out));
        c->last.kernel_launches = 1;
        return LGM_OK;
    }
    const Shape sh = shape_of(n, t, terms);
    // (err_out: the host-buffer call, which takes the small form itself)
    if (!err_out && small_call(c, kind, sh, n, t, all_sites))
        return launch_small(c, kind, terms, d_src, d_q, n, d_tgt_site, t, all_sites, d_out, st, nullptr,
                            0);
    const bool f64 = cf.precision == LGM_PREC_FP64, direct = f64 && !f64_table(c);
    const int v = f64 ? kDefaultVariant : choose_variant(c, kind, sh, n);
    const int fmt = direct || !kVariants[v].tc ? kFmtFloat : kFmtHalf;
    lgm_status s;
    // room for every variant that a smaller call may take: with tables both
    // defaults, and those that were tuned
    std::vector<int> vs = {direct ? kDirect : v};
    int room = fmt;
    if (!f64 && c->forced_variant < 0 && (cf.path != LGM_PATH_RSQRT || !c->tune_cache.empty())) {
        room = kFmtFloat | kFmtHalf;
        vs.push_back(kDefaultVariant);
        if (cf.path != LGM_PATH_RSQRT) vs.push_back(kTileVariant);
        for (const auto& tuned : c->tune_cache) vs.push_back(tuned.second);
    }
    if ((s = lay_out(c, sh, n, t, room, fn_index(kind, sum_path(c)), vs)) != LGM_OK) return s;
    if ((s = prep(c, terms, d_src, d_q, n, d_tgt_site, t, all_sites, sh, fmt, st)) != LGM_OK)
        return s;
    int splits = 1;
    if (c->timing) LGM_CUDA(c, cudaEventRecord(c->ev_pair0, st));
    if (direct) {
        const double erffactor =
            cf.coulomb_gaussian_sigma > 0 ? 1.0 / (std::sqrt(2.0) * cf.coulomb_gaussian_sigma) : 0.0;
        splits = direct_splits(c, sh);
        Cut cut{c->sums, 0};
        cut_sums(c, cut, sh, kDirect, 0);
        dim3 grid((sh.t_phys + kF64Threads - 1) / kF64Threads, splits);
        LGM_CUDA(c, launch_chain(c->overlap, pair_kernel_f64, grid, kF64Threads, 0, st, c->d_geo,
                                 c->d_qq, sh.n_pad, splits, c->d_tgt, sh.t_phys, c->d_part,
                                 cf.electrostatic_cutoff * cf.electrostatic_cutoff, kind,
                                 erffactor));
        c->last.ctas = grid.x * grid.y;
        c->last.threads = kF64Threads;
        c->last.targets_per_thread = 1;
    } else {
        if ((s = launch_pair(c, kind, sum_path(c), v, sh, st, &splits)) != LGM_OK) return s;
    }
    if (c->timing) {
        LGM_CUDA(c, cudaEventRecord(c->ev_pair1, st));
        c->timed_pending = true;
    }
    // the last kernel also clears both bin arrays for the next call
    const int nbins = 2 * c->bins_stride;
    if (splits > 0) {
        LGM_CUDA(c, launch_chain(c->overlap, finalize, (t + 255) / 256, 256, 0, st, c->d_part,
                                 splits, sh.t_phys, t, sh.t_pad, sh.nterms,
                                 cf.electrostatic_prefactor, c->d_perm, d_out, c->d_bins, nbins,
                                 c->d_err, err_out));
        c->last.kernel_launches = 5;  // bins (+ scan), scatter, records, pair, finalize
    } else {
        const Variant& V = kVariants[v];
        LGM_CUDA(c, launch_chain(c->overlap, finalize_items, (t + 31) / 32, dim3(32, 3), 0, st,
                                 c->d_part, c->d_tile_first, c->d_tile_items, variant_tile(V), t,
                                 sh.t_pad, sh.nterms, cf.electrostatic_prefactor, c->d_perm, d_out,
                                 c->d_bins, nbins, c->d_err, err_out));
        c->last.kernel_launches = 7;  // bins (+ scan), scatter, records, boxes, cull, pair, finalize
    }
    c->bins_clean = true;
    if (f64) c->last.variant = -1;
    c->last.pairs_tested = (int64_t)sh.nterms * t * (int64_t)n;
    c->last.splits = splits;
    return LGM_OK;
}

// The status of device error word e (read back into c->h_err); a nonzero word
// is cleared on the device for the next call.
lgm_status device_error_status(lgm_ctx* c, cudaStream_t st, unsigned e) {
    if (e == 0) return LGM_OK;
    LGM_CUDA(c, cudaMemsetAsync(c->d_err, 0, sizeof(unsigned), st));
    LGM_CUDA(c, cudaStreamSynchronize(st));
    if (e & DEVERR_TIMEOUT) return fail(c, LGM_ERR_TIMEOUT, "a bounded device wait ran out");
    if (e & DEVERR_SOURCE_RANGE)
        return fail(c, LGM_ERR_OUT_OF_RANGE, "a source site lies outside [0, volume)");
    if (e & DEVERR_TARGET_RANGE)
        return fail(c, LGM_ERR_OUT_OF_RANGE, "a target site lies outside [0, volume + 35)");
    return fail(c, LGM_ERR_STATE, "device reported an inconsistent state");
}

lgm_status check_device_error(lgm_ctx* c, cudaStream_t st) {
    LGM_CUDA(c, cudaMemcpyAsync(c->h_err, c->d_err, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    LGM_CUDA(c, cudaStreamSynchronize(st));
    return device_error_status(c, st, *c->h_err);
}

lgm_status check_common(lgm_ctx* c, int kind, unsigned terms, int n, int t) {
    if (!c) return LGM_ERR_INVALID_ARGUMENT;
    c->err.clear();
    if (kind != LGM_POINT && kind != LGM_GAUSS)
        return fail(c, LGM_ERR_INVALID_ARGUMENT, "kind must be LGM_POINT or LGM_GAUSS");
    if (kind == LGM_GAUSS && !(c->cfg.coulomb_gaussian_sigma > 0))
        return fail(c, LGM_ERR_INVALID_ARGUMENT, "LGM_GAUSS needs coulomb.gaussian.sigma > 0");
    if (terms == 0 || (terms & ~7u) || !(terms & LGM_TERM_DIRECT))
        return fail(c, LGM_ERR_INVALID_ARGUMENT,
                    "terms must include LGM_TERM_DIRECT and only the three term bits");
    if (n < 0 || t < 0) return fail(c, LGM_ERR_INVALID_ARGUMENT, "negative size");
    if (c->cfg.max_charges > 0 && n > c->cfg.max_charges)
        return fail(c, LGM_ERR_CAPACITY, "more sources than max_charges");
    if (c->cfg.max_targets > 0 && t > c->cfg.max_targets)
        return fail(c, LGM_ERR_CAPACITY, "more targets than max_targets");
    return LGM_OK;
}


lgm_status check_sites(lgm_ctx* c, const int32_t* src, int n, const int32_t* tgt, int t) {
    for (int j = 0; j < n; ++j)
        if (src[j] < 0 || src[j] >= c->volume) {
            char b[128];
            std::snprintf(b, sizeof b, "source %d: site %d outside [0, %d)", j, src[j], c->volume);
            return fail(c, LGM_ERR_OUT_OF_RANGE, b);
        }
    for (int g = 0; g < t; ++g)
        if (tgt[g] < 0 || tgt[g] >= c->volume + kDrainIds) {
            char b[128];
            std::snprintf(b, sizeof b, "target %d: site %d outside [0, %d)", g, tgt[g],
                          c->volume + kDrainIds);
            return fail(c, LGM_ERR_OUT_OF_RANGE, b);
        }
    return LGM_OK;
}

}  // namespace

// ---- ABI ----------------------------------------------------------------------

extern "C" {

int32_t lgm_abi_version(void) { return LGM_ABI_VERSION; }

const char* lgm_status_string(lgm_status s) {
    switch (s) {
    case LGM_OK: return "ok";
    case LGM_ERR_INVALID_ARGUMENT: return "invalid argument";
    case LGM_ERR_OUT_OF_RANGE: return "site out of range";
    case LGM_ERR_CUDA: return "CUDA error";
    case LGM_ERR_NO_DEVICE: return "no usable sm_100 device";
    case LGM_ERR_CAPACITY: return "capacity exceeded";
    case LGM_ERR_TIMEOUT: return "device wait timed out";
    case LGM_ERR_PARSE: return "parse error";
    case LGM_ERR_UNSUPPORTED: return "unsupported";
    case LGM_ERR_STATE: return "invalid state";
    default: return "unknown status";
    }
}

void lgm_config_default(lgm_config* cfg) {
    if (!cfg) return;
    std::memset(cfg, 0, sizeof *cfg);
    // SimulationParameters() defaults (parameters.h:285-378)
    cfg->grid_x = 128; cfg->grid_y = 128; cfg->grid_z = 1;
    cfg->electrostatic_cutoff = 50;
    // setCalculatedValues (parameters.h:384-390) with the constants of
    // parameters.h:358-362 and dielectric.constant 3.5.
    const double e = 1.60217646e-19, eps0 = 8.854187817e-12, a = 1e-9, epsr = 3.5;
    cfg->electrostatic_prefactor = e / (4.0 * M_PI * epsr * eps0 * a);
    cfg->coulomb_gaussian_sigma = 0.0;
    cfg->work_x = cfg->work_y = cfg->work_z = 4;
    cfg->work_size = 256;
    cfg->opencl_threshold = 256;
    cfg->max_charges = 0;
    cfg->max_targets = 0;
    cfg->precision = LGM_PREC_FP32C;
    cfg->path = LGM_PATH_RSQRT;
}

lgm_status lgm_create(const lgm_config* cfg, int32_t device, lgm_ctx** out) {
    g_create_error.clear();
    if (!cfg || !out) {
        g_create_error = "null argument";
        return LGM_ERR_INVALID_ARGUMENT;
    }
    *out = nullptr;
    const lgm_config& cf = *cfg;
    if (cf.grid_x < 1 || cf.grid_y < 1 || cf.grid_z < 1) {
        g_create_error = "grid.x, grid.y and grid.z must be >= 1 (parameters.h:403-414)";
        return LGM_ERR_INVALID_ARGUMENT;
    }
    if (cf.electrostatic_cutoff < 1 || cf.electrostatic_cutoff > 1000) {
        g_create_error = "electrostatic.cutoff must be in [1, 1000]";
        return LGM_ERR_INVALID_ARGUMENT;
    }
    if (!(cf.coulomb_gaussian_sigma >= 0) || !std::isfinite(cf.electrostatic_prefactor)) {
        g_create_error = "coulomb.gaussian.sigma must be >= 0 and the prefactor finite";
        return LGM_ERR_INVALID_ARGUMENT;
    }
    if (cf.precision != LGM_PREC_FP32C && cf.precision != LGM_PREC_FP64) {
        g_create_error = "unknown precision";
        return LGM_ERR_INVALID_ARGUMENT;
    }
    if (cf.path != LGM_PATH_RSQRT && cf.path != LGM_PATH_TABLE && cf.path != LGM_PATH_TABLE64) {
        g_create_error = "unknown path";
        return LGM_ERR_INVALID_ARGUMENT;
    }
    // FP32 exactness of r^2 - 1/2 in expanded form: every intermediate a
    // half-integer below 2^22 with the right-image targets at x' < 2X
    // (6 L^2 < 2^22).
    const long long L = std::max<long long>({2LL * cf.grid_x, cf.grid_y, cf.grid_z + 1});
    if (6 * L * L >= (1LL << 22) ||
        (long long)cf.grid_x * cf.grid_y * cf.grid_z + kDrainIds > INT32_MAX) {
        g_create_error = "lattice too large for exact FP32 r^2 (need 6*max(2X,Y,Z+1)^2 < 2^22)";
        return LGM_ERR_UNSUPPORTED;
    }
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) {
        g_create_error = std::string("no CUDA device: ") + cudaGetErrorString(e);
        return LGM_ERR_NO_DEVICE;
    }
    const int dev = device < 0 ? 0 : device;
    if (dev >= ndev) {
        g_create_error = "device id out of range";
        return LGM_ERR_NO_DEVICE;
    }
    // attribute reads: cudaGetDeviceProperties takes 2.5 ms and more
    int cc_major = 0, n_sms = 0;
    if ((e = cudaDeviceGetAttribute(&cc_major, cudaDevAttrComputeCapabilityMajor, dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) {
        g_create_error = std::string("cudaDeviceGetAttribute: ") + cudaGetErrorString(e);
        return LGM_ERR_NO_DEVICE;
    }
    if (cc_major != 10) {
        g_create_error = "device is not sm_100 (B200); this library is built for sm_100a only";
        return LGM_ERR_NO_DEVICE;
    }
    lgm_ctx* c = new (std::nothrow) lgm_ctx();
    if (!c) {
        g_create_error = "out of host memory";
        return LGM_ERR_INVALID_ARGUMENT;
    }
    c->cfg = cf;
    c->device = dev;
    c->sm_count = n_sms;
    c->xy = cf.grid_x * cf.grid_y;
    c->volume = c->xy * cf.grid_z;
    auto bail = [&](const char* what, cudaError_t err) {
        g_create_error = std::string(what) + ": " + cudaGetErrorString(err);
        lgm_destroy(c);
        return LGM_ERR_CUDA;
    };
    if ((e = cudaSetDevice(dev)) != cudaSuccess) return bail("cudaSetDevice", e);
    if ((e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)) != cudaSuccess)
        return bail("cudaStreamCreate", e);
    if ((e = cudaMalloc(&c->d_err, sizeof(unsigned))) != cudaSuccess) return bail("cudaMalloc", e);
    if ((e = cudaMemset(c->d_err, 0, sizeof(unsigned))) != cudaSuccess) return bail("cudaMemset", e);
    if ((e = cudaMallocHost(&c->h_err, sizeof(unsigned))) != cudaSuccess)
        return bail("cudaMallocHost", e);

    // Tables indexed by the integer r^2 (potential.cpp:268-308 restated per r^2):
    //   rtab[k] = 1/sqrt(k) for 0 < k < c^2, 0 at k = 0 and k = c^2 (point, table path);
    //   gauss: gtab[k] = erf(f sqrt(k))/sqrt(k); with the rsqrt path only the
    //   k where it differs from 1/sqrt(k) in FP32 are kept and entry gtab_k
    //   is NaN (the kernel then falls back to 1/r).
    const int c2 = cf.electrostatic_cutoff * cf.electrostatic_cutoff;
    {
        std::vector<float> rt(c2 + 1, 0.f);
        for (int k = 1; k < c2; ++k) rt[k] = (float)(1.0 / std::sqrt((double)k));
        c->rtab_k = c2;
        if ((e = cudaMalloc(&c->d_rtab, rt.size() * sizeof(float))) != cudaSuccess)
            return bail("cudaMalloc", e);
        if ((e = cudaMemcpy(c->d_rtab, rt.data(), rt.size() * sizeof(float),
                            cudaMemcpyHostToDevice)) != cudaSuccess)
            return bail("cudaMemcpy", e);
    }
    {
        const double sig = cf.coulomb_gaussian_sigma;
        std::vector<float> gt;
        if (sig > 0) {
            const double f = 1.0 / (std::sqrt(2.0) * sig);
            int kmax = c2;
            if (cf.path == LGM_PATH_RSQRT) {
                // erfc(f sqrt(k)) < 2^-30 beyond kmax: erf rounds to 1 in FP32
                kmax = 1;
                while (kmax < c2 && std::erfc(f * std::sqrt((double)kmax)) >= 0x1p-30) ++kmax;
            }
            gt.assign(kmax + 1, 0.f);
            for (int k = 1; k < kmax; ++k) {
                const double r = std::sqrt((double)k);
                gt[k] = (float)(std::erf(f * r) / r);
            }
            gt[kmax] = cf.path == LGM_PATH_RSQRT ? std::nanf("") : 0.f;
            c->gtab_k = kmax;
        } else {
            gt.assign(2, 0.f);
            c->gtab_k = 0;
        }
        if ((e = cudaMalloc(&c->d_gtab, gt.size() * sizeof(float))) != cudaSuccess)
            return bail("cudaMalloc", e);
        if ((e = cudaMemcpy(c->d_gtab, gt.data(), gt.size() * sizeof(float),
                            cudaMemcpyHostToDevice)) != cudaSuccess)
            return bail("cudaMemcpy", e);
    }
    // FP64 tables of the TABLE64 path and of the FP64 precision: w(k) for every
    // integer r^2 = k <= c^2, correctly rounded in IEEE double, 0 at k = 0 and
    // k = c^2.
    const bool tab64 = cf.path == LGM_PATH_TABLE64 ||
                       (cf.precision == LGM_PREC_FP64 &&
                        mma_smem_bytes(c2 + 1, 8) <= kF64TableSmem);
    if (tab64) {
        std::vector<double> rt(c2 + 1, 0.0), gt(c2 + 1, 0.0);
        const double sig = cf.coulomb_gaussian_sigma;
        const double f = sig > 0 ? 1.0 / (std::sqrt(2.0) * sig) : 0.0;
        for (int k = 1; k < c2; ++k) {
            const double r = std::sqrt((double)k);
            rt[k] = 1.0 / r;
            gt[k] = sig > 0 ? std::erf(f * r) / r : rt[k];
        }
        if ((e = cudaMalloc(&c->d_rtab64, rt.size() * sizeof(double))) != cudaSuccess ||
            (e = cudaMalloc(&c->d_gtab64, gt.size() * sizeof(double))) != cudaSuccess)
            return bail("cudaMalloc", e);
        if ((e = cudaMemcpy(c->d_rtab64, rt.data(), rt.size() * sizeof(double),
                            cudaMemcpyHostToDevice)) != cudaSuccess ||
            (e = cudaMemcpy(c->d_gtab64, gt.data(), gt.size() * sizeof(double),
                            cudaMemcpyHostToDevice)) != cudaSuccess)
            return bail("cudaMemcpy", e);
    }
    // Lattice cells for the spatial target order (Morton rank per cell).
    {
        const std::vector<int32_t> rank =
            cell_ranks(cf.grid_x, cf.grid_y, cf.grid_z, &c->cell_shift, &c->cells_x, &c->cells_y);
        c->ncells = (int)rank.size();
        c->bins_stride = (c->ncells + 2 + 3) / 4 * 4;
        if ((e = cudaMalloc(&c->d_cell_rank, sizeof(int32_t) * rank.size())) != cudaSuccess ||
            (e = cudaMalloc(&c->d_bins, sizeof(int32_t) * (2 * c->bins_stride + 4))) !=
                cudaSuccess ||
            (e = cudaMalloc(&c->d_item_count, 4 * sizeof(int32_t))) != cudaSuccess ||
            (e = cudaMalloc(&c->d_cost_hist, kCostBuckets * sizeof(int32_t))) != cudaSuccess)
            return bail("cudaMalloc", e);
        if ((e = cudaMemset(c->d_item_count, 0, 4 * sizeof(int32_t))) != cudaSuccess)
            return bail("cudaMemset", e);
        // the source bins follow the target bins, 16-byte aligned (the scan reads int4)
        c->d_sbins = c->d_bins + c->bins_stride;
        if ((e = cudaMemcpy(c->d_cell_rank, rank.data(), sizeof(int32_t) * rank.size(),
                            cudaMemcpyHostToDevice)) != cudaSuccess)
            return bail("cudaMemcpy", e);
    }
    // Shared memory above the 48 KB default for large cutoffs, and the
    // resident CTAs per SM of every variant (the split count fills
    // kSplitWaves waves of them).
    {
        const int tab_of[4] = {0, c->gtab_k, std::max(c->rtab_k, c->gtab_k), c->rtab_k};
        for (int v = 0; v < kNumVariants; ++v)
            for (int fi = 0; fi < 4; ++fi) {
                if (!kernel_of(kVariants[v], fi, c2)) continue;
                // the table kernels serve only their own path
                if (fi == 2 && cf.path != LGM_PATH_TABLE) continue;
                if (fi == 3 && cf.path != LGM_PATH_TABLE64 && !(tab64 && v == kDefaultVariant))
                    continue;
                const size_t smem = variant_smem(kVariants[v], fi, tab_of[fi], c2);
                bool fits = false;
                if ((e = allow_smem(kernel_of(kVariants[v], fi, c2), smem, &fits)) != cudaSuccess)
                    return bail("shared-memory limit", e);
                if (!fits) {
                    g_create_error = "cutoff too large for the shared-memory tables";
                    lgm_destroy(c);
                    return LGM_ERR_UNSUPPORTED;
                }
                int bps = 0;
                if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                         &bps, kernel_of(kVariants[v], fi, c2), variant_threads(kVariants[v]),
                         smem)) != cudaSuccess)
                    return bail("cudaOccupancyMaxActiveBlocksPerMultiprocessor", e);
                c->bps[v][fi] = bps;
            }
    }
    for (int k : {LGM_POINT, LGM_GAUSS})
        if ((e = cudaFuncSetAttribute(small_fn(k, tab64 ? (int)LGM_PATH_TABLE64 : cf.path), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kSmallSmem)) != cudaSuccess)
            return bail("cudaFuncSetAttribute", e);
    *out = c;
    return LGM_OK;
}

lgm_status lgm_destroy(lgm_ctx* c) {
    if (!c) return LGM_OK;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    void* dev_ptrs[] = {c->d_scratch, c->d_sums, c->d_s,        c->d_q,      c->d_t,         c->d_o,
                        c->d_gtab,    c->d_rtab,     c->d_rtab64, c->d_gtab64,    c->d_err,
                        c->d_cell_rank, c->d_bins,   c->d_item_count, c->d_examined, c->d_cost_hist};
    for (void* p : dev_ptrs)
        if (p) cudaFree(p);
    void* host_ptrs[] = {c->h_s, c->h_q, c->h_t, c->h_o, c->h_err};
    for (void* p : host_ptrs)
        if (p) cudaFreeHost(p);
    if (c->ev_pair0) cudaEventDestroy(c->ev_pair0);
    if (c->ev_pair1) cudaEventDestroy(c->ev_pair1);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
    return LGM_OK;
}

const char* lgm_last_error(const lgm_ctx* c) {
    if (!c) return g_create_error.c_str();
    return c->err.c_str();
}

lgm_status lgm_last_launch(lgm_ctx* c, lgm_launch_info* info) {
    if (!c || !info) return LGM_ERR_INVALID_ARGUMENT;
    if (c->timed_pending) {
        LGM_CUDA(c, cudaEventSynchronize(c->ev_pair1));
        float ms = -1.f;
        LGM_CUDA(c, cudaEventElapsedTime(&ms, c->ev_pair0, c->ev_pair1));
        c->last.pair_kernel_ms = ms;
        c->timed_pending = false;
    }
    if (c->count_pending) {
        unsigned long long n = 0;
        LGM_CUDA(c, cudaMemcpy(&n, c->d_examined, sizeof n, cudaMemcpyDeviceToHost));
        c->last.pairs_examined = (int64_t)n;
        c->count_pending = false;
    }
    *info = c->last;
    return LGM_OK;
}

lgm_status lgm_set_counting(lgm_ctx* c, int32_t enable) {
    if (!c) return LGM_ERR_INVALID_ARGUMENT;
    LGM_CUDA(c, cudaSetDevice(c->device));
    if (enable && !c->d_examined)
        LGM_CUDA(c, cudaMalloc(&c->d_examined, sizeof(unsigned long long)));
    c->counting = enable != 0;
    c->count_pending = false;
    return LGM_OK;
}

lgm_status lgm_set_launch_overlap(lgm_ctx* c, int32_t enable) {
    if (!c) return LGM_ERR_INVALID_ARGUMENT;
    c->overlap = enable != 0;
    return LGM_OK;
}

lgm_status lgm_set_timing(lgm_ctx* c, int32_t enable) {
    if (!c) return LGM_ERR_INVALID_ARGUMENT;
    LGM_CUDA(c, cudaSetDevice(c->device));
    if (enable && !c->ev_pair0) {
        LGM_CUDA(c, cudaEventCreate(&c->ev_pair0));
        LGM_CUDA(c, cudaEventCreate(&c->ev_pair1));
    }
    c->timing = enable != 0;
    c->timed_pending = false;
    return LGM_OK;
}

int32_t lgm_variant_count(void) { return kNumVariants; }

lgm_status lgm_variant_info(int32_t v, int32_t* threads, int32_t* target_pairs, int32_t* run) {
    if (v < 0 || v >= kNumVariants) return LGM_ERR_INVALID_ARGUMENT;
    if (threads) *threads = kVariants[v].nt;
    if (target_pairs) *target_pairs = kVariants[v].rp;
    if (run) *run = kVariants[v].sub;
    return LGM_OK;
}

lgm_status lgm_variant_flags(int32_t v, int32_t* flags) {
    if (v < 0 || v >= kNumVariants || !flags) return LGM_ERR_INVALID_ARGUMENT;
    *flags = (kVariants[v].skip ? LGM_VARIANT_WARP_SKIP : 0) |
             (kVariants[v].cull ? LGM_VARIANT_CULLED : 0) |
             (kVariants[v].ws ? LGM_VARIANT_WARP_SPECIALISED : 0);
    return LGM_OK;
}

lgm_status lgm_variant_items(int32_t v, int32_t* chunks_per_item, int32_t* stages) {
    if (v < 0 || v >= kNumVariants) return LGM_ERR_INVALID_ARGUMENT;
    if (chunks_per_item) *chunks_per_item = kVariants[v].cull ? kVariants[v].per_item : 0;
    if (stages) *stages = kVariants[v].ws;
    return LGM_OK;
}

lgm_status lgm_set_variant(lgm_ctx* c, int32_t v) {
    if (!c) return LGM_ERR_INVALID_ARGUMENT;
    if (v < -1 || v >= kNumVariants) return fail(c, LGM_ERR_INVALID_ARGUMENT, "no such variant");
    c->forced_variant = v;
    return LGM_OK;
}

lgm_status lgm_autotune(lgm_ctx* c, lgm_kind kind, uint32_t terms, int32_t n, int32_t t,
                        int32_t* chosen) {
    lgm_status s = check_common(c, kind, terms, n, t);
    if (s != LGM_OK) return s;
    if (n < 1 || t < 1) return fail(c, LGM_ERR_INVALID_ARGUMENT, "autotune needs n, t >= 1");
    LGM_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t st = c->stream;
    // Synthetic charges of this size: sites spread over the lattice, q = +-1.
    std::vector<int32_t> hs(n), hq(n), ht(t);
    uint64_t x = 0x9E3779B97F4A7C15ull;
    auto next = [&]() { x ^= x << 13; x ^= x >> 7; x ^= x << 17; return x; };
    for (int j = 0; j < n; ++j) { hs[j] = (int32_t)(next() % c->volume); hq[j] = (next() & 1) ? 1 : -1; }
    for (int g = 0; g < t; ++g) ht[g] = (int32_t)(next() % c->volume);
    if ((s = grow_device(c, &c->d_s, &c->s_cap, (size_t)n)) != LGM_OK) return s;
    if ((s = grow_device(c, &c->d_q, &c->q_cap, (size_t)n)) != LGM_OK) return s;
    if ((s = grow_device(c, &c->d_t, &c->t_cap, (size_t)t)) != LGM_OK) return s;
    LGM_CUDA(c, cudaMemcpyAsync(c->d_s, hs.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
    LGM_CUDA(c, cudaMemcpyAsync(c->d_q, hq.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
    LGM_CUDA(c, cudaMemcpyAsync(c->d_t, ht.data(), sizeof(int32_t) * t, cudaMemcpyHostToDevice, st));
    const Shape sh = shape_of(n, t, terms);
    std::vector<int> vs;
    for (int v = 0; v < kNumVariants; ++v)
        if (c->cfg.path != LGM_PATH_TABLE64 || kVariants[v].cull) vs.push_back(v);
    if ((s = lay_out(c, sh, n, t, kFmtFloat | kFmtHalf, fn_index(kind, c->cfg.path), vs)) != LGM_OK ||
        (s = prep(c, terms, c->d_s, c->d_q, n, c->d_t, t, 0, sh, kFmtFloat | kFmtHalf, st)) !=
            LGM_OK)
        return s;
    cudaEvent_t e0, e1;
    LGM_CUDA(c, cudaEventCreate(&e0));
    LGM_CUDA(c, cudaEventCreate(&e1));
    int best = kDefaultVariant;
    float best_ms = 1e30f;
    for (int v : vs) {
        int splits;
        if ((s = launch_pair(c, kind, c->cfg.path, v, sh, st, &splits)) != LGM_OK) break;  // warm
        float ms[3];
        for (int r = 0; r < 3; ++r) {
            cudaEventRecord(e0, st);
            if ((s = launch_pair(c, kind, c->cfg.path, v, sh, st, &splits)) != LGM_OK) break;
            cudaEventRecord(e1, st);
            cudaEventSynchronize(e1);
            cudaEventElapsedTime(&ms[r], e0, e1);
        }
        if (s != LGM_OK) break;
        std::sort(ms, ms + 3);
        if (ms[1] < best_ms) { best_ms = ms[1]; best = v; }
    }
    // Where the one-kernel form would serve the call, it is timed against the whole
    // chain of the fastest variant; if it wins, no variant is remembered.
    bool one_kernel = false;
    const uint64_t key = tune_key(kind, c->cfg.path, sh.t_phys, sh.n_chunks);
    if (s == LGM_OK && c->cfg.precision != LGM_PREC_FP64 && small_fits(c, kind, sh, n, t, false) &&
        (s = grow_device(c, &c->d_o, &c->o_cap, (size_t)t)) == LGM_OK) {
        const int forced = c->forced_variant;
        const bool counting = c->counting, timing = c->timing;
        c->counting = c->timing = false;
        c->tune_cache.erase(key);
        float form_ms[2] = {0.f, 0.f};
        for (int form = 0; form < 2 && s == LGM_OK; ++form) {
            c->forced_variant = form == 0 ? best : -1;
            float ms[3];
            for (int r = -1; r < 3 && s == LGM_OK; ++r) {  // the first to warm up
                cudaEventRecord(e0, st);
                s = launch_potentials(c, kind, terms, c->d_s, c->d_q, n, c->d_t, t, 0, c->d_o, st);
                cudaEventRecord(e1, st);
                cudaEventSynchronize(e1);
                if (r >= 0) cudaEventElapsedTime(&ms[r], e0, e1);
            }
            if (s != LGM_OK) break;
            std::sort(ms, ms + 3);
            form_ms[form] = ms[1];
        }
        c->forced_variant = forced;
        c->counting = counting;
        c->timing = timing;
        one_kernel = form_ms[1] <= form_ms[0];
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (s != LGM_OK) return s;
    if ((s = check_device_error(c, st)) != LGM_OK) return s;
    if (one_kernel) best = kDefaultVariant;
    else c->tune_cache[key] = best;
    if (chosen) *chosen = best;
    return LGM_OK;
}

lgm_status lgm_potentials_async(lgm_ctx* c, lgm_kind kind, uint32_t terms,
                                const int32_t* d_src_site, const int32_t* d_src_q, int32_t n,
                                const int32_t* d_tgt_site, int32_t t, double* d_out,
                                void* stream) {
    lgm_status s = check_common(c, kind, terms, n, t);
    if (s != LGM_OK) return s;
    if ((n > 0 && (!d_src_site || !d_src_q)) || (t > 0 && (!d_tgt_site || !d_out)))
        return fail(c, LGM_ERR_INVALID_ARGUMENT, "null buffer");
    LGM_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
    return launch_potentials(c, kind, terms, d_src_site, d_src_q, n, d_tgt_site, t, 0, d_out, st);
}

lgm_status lgm_sync(lgm_ctx* c, void* stream) {
    if (!c) return LGM_ERR_INVALID_ARGUMENT;
    LGM_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
    return check_device_error(c, st);
}

lgm_status lgm_potentials(lgm_ctx* c, lgm_kind kind, uint32_t terms, const int32_t* src_site,
                          const int32_t* src_q, int32_t n, const int32_t* tgt_site, int32_t t,
                          double* out) {
    lgm_status s = check_common(c, kind, terms, n, t);
    if (s != LGM_OK) return s;
    if ((n > 0 && (!src_site || !src_q)) || (t > 0 && (!tgt_site || !out)))
        return fail(c, LGM_ERR_INVALID_ARGUMENT, "null buffer");
    LGM_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t st = c->stream;
    if (t == 0) return check_sites(c, src_site, n, nullptr, 0);
    // One pinned staging buffer and one device buffer, laid out [targets t]
    // [charges n][sources n, unless they are the first n targets], cross in
    // one copy; the results come back in one copy with the device error word
    // behind them (written by the call's last kernel).
    const bool alias = tgt_site == src_site && n <= t;
    const size_t words = (size_t)t + n + (alias ? 0 : n);
    if ((s = grow_host(c, &c->h_t, &c->ht_cap, words)) != LGM_OK) return s;
    if ((s = grow_host(c, &c->h_o, &c->ho_cap, (size_t)t + 1)) != LGM_OK) return s;
    if ((s = grow_device(c, &c->d_t, &c->t_cap, words)) != LGM_OK) return s;
    if ((s = grow_device(c, &c->d_o, &c->o_cap, (size_t)t + 1)) != LGM_OK) return s;
    const Shape sh = shape_of(n, t, terms);
    const bool small = n > 0 && small_call(c, kind, sh, n, t, false);
    // The sites are checked on the device (prep_records), which gives each an
    // empty record and raises an error bit; only then are they checked here,
    // for the first bad one (sources first, then targets, as check_sites
    // reports them).  When the sources are the first n targets (kernel 2: w
    // aliases s, openclhelper.cpp:154) they cross once, as targets.
    std::memcpy(c->h_t, tgt_site, sizeof(int32_t) * t);
    if (n > 0) std::memcpy(c->h_t + t, src_q, sizeof(int32_t) * n);
    if (!alias && n > 0) std::memcpy(c->h_t + t + n, src_site, sizeof(int32_t) * n);
    unsigned e = 0;
    if (small) {
        // One kernel, results straight into the pinned buffer.  Every CTA reads
        // the sources: from the pinned staging while that is little, else from
        // the device after one copy.
        const size_t reads = sizeof(int32_t) * ((size_t)2 * n * std::min((t + kSeg - 1) / kSeg,
                                                                         4 * c->sm_count) + t);
        const int32_t* in = c->h_t;
        if (reads > kZeroCopyBytes) {
            LGM_CUDA(c, cudaMemcpyAsync(c->d_t, c->h_t, sizeof(int32_t) * words,
                                        cudaMemcpyHostToDevice, st));
            in = c->d_t;
        }
        reset_last(c);
        volatile unsigned long long* flag = reinterpret_cast<volatile unsigned long long*>(c->h_o + t);
        const unsigned call = ++c->call_number;
        *flag = (unsigned long long)(call - 1) << 32;
        if ((s = launch_small(c, kind, terms, alias ? in : in + t + n, in + t, n, in, t, 0, c->h_o, st,
                              const_cast<unsigned long long*>(flag), call)) != LGM_OK)
            return s;
        // the kernel's own word comes sooner than the stream's; if it does not
        // come soon, wait for the stream (and learn of an error)
        bool seen = false;
        for (int i = 0; i < kFlagPolls && !seen; ++i) seen = (unsigned)(*flag >> 32) == call;
        if (!seen) LGM_CUDA(c, cudaStreamSynchronize(st));
        std::atomic_thread_fence(std::memory_order_acquire);
        e = (unsigned)*flag;
    } else {
        LGM_CUDA(c, cudaMemcpyAsync(c->d_t, c->h_t, sizeof(int32_t) * words, cudaMemcpyHostToDevice,
                                    st));
        const int32_t* d_src = alias ? c->d_t : c->d_t + t + n;
        unsigned* d_err_out = reinterpret_cast<unsigned*>(c->d_o + t);
        if ((s = launch_potentials(c, kind, terms, d_src, c->d_t + t, n, c->d_t, t, 0, c->d_o, st,
                                   d_err_out)) != LGM_OK)
            return s;
        LGM_CUDA(c, cudaMemcpyAsync(c->h_o, c->d_o, sizeof(double) * ((size_t)t + 1),
                                    cudaMemcpyDeviceToHost, st));
        LGM_CUDA(c, cudaStreamSynchronize(st));
        e = *reinterpret_cast<const unsigned*>(c->h_o + t);
    }
    if (e != 0) {
        const lgm_status ds = device_error_status(c, st, e);  // clears the device word
        if (e & (DEVERR_SOURCE_RANGE | DEVERR_TARGET_RANGE)) {
            const lgm_status hs = check_sites(c, src_site, n, tgt_site, t);
            if (hs != LGM_OK) return hs;
        }
        return ds;
    }
    std::memcpy(out, c->h_o, sizeof(double) * t);
    return LGM_OK;
}

lgm_status lgm_coulomb_kernel2(lgm_ctx* c, lgm_kind kind, const int32_t* s, const int32_t* q,
                               int32_t n, int32_t total, double* o) {
    if (c && (n < 0 || n > total)) return fail(c, LGM_ERR_INVALID_ARGUMENT, "need 0 <= n <= total");
    // kernel 2: w aliases s (openclhelper.cpp:154), the first n entries are
    // the sources, every entry is a target.
    return lgm_potentials(c, kind, LGM_TERM_DIRECT, s, q, n, s, total, o);
}

lgm_status lgm_coulomb_kernel1_async(lgm_ctx* c, lgm_kind kind, const int32_t* d_s,
                                     const int32_t* d_q, int32_t n, double* d_o, void* stream) {
    if (!c) return LGM_ERR_INVALID_ARGUMENT;
    lgm_status st = check_common(c, kind, LGM_TERM_DIRECT, n, 0);
    if (st != LGM_OK) return st;
    if ((n > 0 && (!d_s || !d_q)) || !d_o) return fail(c, LGM_ERR_INVALID_ARGUMENT, "null buffer");
    LGM_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t s = stream ? (cudaStream_t)stream : c->stream;
    return launch_potentials(c, kind, LGM_TERM_DIRECT, d_s, d_q, n, nullptr, c->volume, 1, d_o, s);
}

lgm_status lgm_coulomb_kernel1(lgm_ctx* c, lgm_kind kind, const int32_t* s, const int32_t* q,
                               int32_t n, double* o) {
    if (!c) return LGM_ERR_INVALID_ARGUMENT;
    lgm_status st = check_common(c, kind, LGM_TERM_DIRECT, n, 0);
    if (st != LGM_OK) return st;
    if ((n > 0 && (!s || !q)) || !o) return fail(c, LGM_ERR_INVALID_ARGUMENT, "null buffer");
    if ((st = check_sites(c, s, n, nullptr, 0)) != LGM_OK) return st;
    LGM_CUDA(c, cudaSetDevice(c->device));
    cudaStream_t str = c->stream;
    const size_t nn = std::max(n, 1);
    const size_t vv = (size_t)c->volume;
    if ((st = grow_host(c, &c->h_s, &c->hs_cap, nn)) != LGM_OK) return st;
    if ((st = grow_host(c, &c->h_q, &c->hq_cap, nn)) != LGM_OK) return st;
    if ((st = grow_host(c, &c->h_o, &c->ho_cap, vv)) != LGM_OK) return st;
    if ((st = grow_device(c, &c->d_s, &c->s_cap, nn)) != LGM_OK) return st;
    if ((st = grow_device(c, &c->d_q, &c->q_cap, nn)) != LGM_OK) return st;
    if ((st = grow_device(c, &c->d_o, &c->o_cap, vv)) != LGM_OK) return st;
    std::memcpy(c->h_s, s, sizeof(int32_t) * n);
    std::memcpy(c->h_q, q, sizeof(int32_t) * n);
    LGM_CUDA(c, cudaMemcpyAsync(c->d_s, c->h_s, sizeof(int32_t) * n, cudaMemcpyHostToDevice, str));
    LGM_CUDA(c, cudaMemcpyAsync(c->d_q, c->h_q, sizeof(int32_t) * n, cudaMemcpyHostToDevice, str));
    if ((st = launch_potentials(c, kind, LGM_TERM_DIRECT, c->d_s, c->d_q, n, nullptr, c->volume, 1,
                                c->d_o, str)) != LGM_OK)
        return st;
    LGM_CUDA(c, cudaMemcpyAsync(c->h_o, c->d_o, sizeof(double) * vv, cudaMemcpyDeviceToHost, str));
    if ((st = check_device_error(c, str)) != LGM_OK) return st;
    std::memcpy(o, c->h_o, sizeof(double) * vv);
    return LGM_OK;
}

}  // extern "C"
