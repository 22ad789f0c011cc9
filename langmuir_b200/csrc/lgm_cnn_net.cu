// lgm_cnn_net.cu -- the surrogate network, forward and backward, as two native
// calls over kernels that share one activation layout.
//
// Activations of 32 channels lie in four planes of eight channels,
//     act[image][c8][y][x][8]  (BF16),
// so that a pixel's eight channels are one 16-byte row of an operand without
// swizzle: a patch of pixels staged once serves all nine taps of a 3x3
// convolution as plain offsets (16 bytes a column, one patch row a row), where
// the NHWC kernel (lgm_cnn_tc.cu) stages it three times, shifted.  The TMA box
// is rows of (x, 8 channels), 160 bytes long.
//
// What the backward pass needs of a ReLU is a bit per value.  The first three
// layers keep those bits and their pooled outputs, not their full-resolution
// activations, and the gradient of a pooled ReLU is formed where it is used:
// in the epilogue of the convolution that yields the pooled gradient (layers
// 3 and 2), or in the first layer's weight gradient.
//
// Rounding points are those of the layer-by-layer kernels: BF16 weights,
// pooled activations, activations of layer 4, pooled mean, hidden layer,
// gradients between layers; FP32 sums.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "langmuir_b200_cnn.h"
#include "lgm_tcgen05.cuh"

namespace {

using bf16 = __nv_bfloat16;
using lgm::smem_addr;

constexpr int CH = LGM_CNN_CHANNELS;  // 32
constexpr int PL = CH / 8;            // planes
constexpr int HID = 64, OUT = 2;      // fully connected layers

__device__ unsigned g_net_error = 0;  // DEVERR_* bits

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float bf(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }
__device__ __forceinline__ uint16_t to_bf(float v) {
    return __bfloat16_as_ushort(__float2bfloat16(v));
}
// D = A (16x16 bf16, row) B (16x8 bf16, col) + D.
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// D = A B + C.
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1, float c0, float c1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void ldsm4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
// 0xffff in each half whose bit of m (bit 0, bit 16) is set.
__device__ __forceinline__ uint32_t half_mask(uint32_t m) { return (m & 0x10001u) * 0xffffu; }

// ---- layer 1 ------------------------------------------------------------------------------
// x [B,H,W] -> pooled p1 planes [B][4][H/2][W/2][8] and (optional) the ReLU bits
// mask1 [B][H/2][W/2][4]: word c8, bit 8 s + j for sub-pixel s = 2 dy + dx and
// channel 8 c8 + j.
//
// A warp takes one pooled row, eight pooled pixels at a time.  GEMM rows g and
// g + 8 are the upper and lower image row of pooled pixel g, K = 12 slots (3
// rows x 4 columns around the pixel pair; 16 with zeros), and the weights come
// in two column sets, for the left and the right pixel of the pair, over the
// same A fragments but for the column that is no neighbour.  So the four values of a pooling window meet in one thread,
// without shuffles; with the columns permuted a thread holds channels 8t ..
// 8t+7 and stores one 16-byte vector.  The input comes straight from L1, two
// words and a funnel shift per fragment.
// A row is a few steps long, so the first words of the warp's next row are
// loaded over the last step of this one, and the row index is stepped without a
// division.  Two blocks an SM hold that without spills (128 registers): 4096
// images of 128x128, four networks, 4.92 ms plain with three blocks, 4.79 so.
// (At 80 registers for three blocks it spilled and lost 2%; with 8 pixels in
// flight instead of 16 half the gain was left.)
// Bound: the ReLU/pool arithmetic, about 100 instructions per 1024 values (ALU
// pipe 60% busy, issue slots 63%), then HBM (the pooled output of 1024 images, 41 us).
// 1024 images: the shared-memory tile of conv1_fwd 234 us, the plain loop 120, now 106.
constexpr int C1_WARPS = 8;
constexpr int C1_CTAS = 2;  // an SM
template <bool MASK>
__global__ void __launch_bounds__(C1_WARPS * 32, C1_CTAS)
conv1_planes(const uint32_t* __restrict__ x, const float* __restrict__ w,
             const float* __restrict__ bias, uint4* __restrict__ pooled,
             uint32_t* __restrict__ mask, int B, int H, int W) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // weight of channel ch at slot k = 4 row + j for the left (0) or right (1) pixel
    auto slot = [&](int ch, int k, int right) {
        const int row = k >> 2, kx = (k & 3) - right;
        return (k < 12 && kx >= 0 && kx < 3) ? w[ch * 9 + row * 3 + kx] : 0.f;
    };
    uint32_t bw[2][4][2];
    float bv[4][2];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        const int ch = 8 * (g >> 1) + 2 * n + (g & 1);
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                bw[r][n][h] = pack2(slot(ch, 2 * t + 8 * h, r), slot(ch, 2 * t + 8 * h + 1, r));
        bv[n][0] = bias[8 * t + 2 * n];
        bv[n][1] = bias[8 * t + 2 * n + 1];
    }
    const int H2 = H / 2, W2 = W / 2;  // W2 is also the words of an input row
    const int i0 = g - 1 + (t & 1);    // this thread's first word
    // The fourth column is no neighbour of the left pixel, nor the first of the
    // right one: out of the A fragments too, since zero weights do not stop an
    // infinity or NaN (8 more ALU operations a step: 4096 images, four networks,
    // 4.92 -> 5.00 ms).
    const uint32_t in_left = t & 1 ? 0x0000ffffu : ~0u, in_right = t & 1 ? ~0u : 0xffff0000u;
    // pooled rows of the batch (a row's output is 1 KB or more, so 31 bits hold them)
    const int rows = B * H2, stride = (int)gridDim.x * C1_WARPS;
    const int sb = stride / H2, sy = stride - sb * H2;  // a stride in images and rows
    int r = (int)blockIdx.x * C1_WARPS + (threadIdx.x >> 5);
    if (r >= rows) return;
    int b = r / H2, py = r - b * H2;
    // The rows of this thread's four fragments, from its first word on.  Outside
    // the image, and in the zero slots, a row inside is read and masked out.
    const uint32_t* rp[4];
    uint32_t keep[4];
    auto set_row = [&] {
        const uint32_t* img = x + (size_t)b * H * W2 + i0;
        const int ya = 2 * py - 1 + (t >> 1), yd = 2 * py + 2;
        keep[0] = ya >= 0 ? ~0u : 0u;
        keep[1] = ~0u;
        keep[2] = t < 2 ? ~0u : 0u;
        keep[3] = t < 2 && yd < H ? ~0u : 0u;
        rp[0] = img + max(ya, 0) * W2;
        rp[1] = img + (ya + 1) * W2;
        rp[2] = img + (2 * py + 1) * W2;
        rp[3] = img + min(yd, H - 1) * W2;
    };
    // words i, i+1 hold pixels 2i+1, 2i+2; a row's ends have none outside
    uint32_t lo[2][4], hi[2][4];
    auto load = [&](int p0) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                lo[j][k] = j == 0 && p0 == 0 && i0 < 0 ? 0u : rp[k][p0 + 8 * j];
                hi[j][k] = j == 1 && p0 + 16 == W2 && i0 == 7 ? 0u : rp[k][p0 + 8 * j + 1];
            }
    };
    set_row();
    load(0);
    for (;;) {
        uint4* prow = pooled + (((size_t)b * PL + t) * H2 + py) * W2 + g;
        uint32_t* mrow = MASK ? mask + (((size_t)b * H2 + py) * W2 + g) * 4 + t : nullptr;
        for (int p0 = 0; p0 < W2; p0 += 16) {
            uint32_t a[2][2][4];  // of the left and right pixels
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t f = __funnelshift_r(lo[j][k], hi[j][k], 16);
                    a[j][0][k] = f & keep[k] & in_left;
                    a[j][1][k] = f & keep[k] & in_right;
                }
            // the next words are in flight over this step's arithmetic, past the
            // row's end those of the warp's next row
            if (p0 + 16 < W2) {
                load(p0 + 16);
            } else if ((r += stride) < rows) {
                b += sb;
                py += sy;
                if (py >= H2) { py -= H2; ++b; }
                set_row();
                load(0);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                uint32_t out[4], sub[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    float d[2][4];
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        mma16816(d[s], a[j][s], bw[s][n][0], bw[s][n][1], 0.f, 0.f);
#pragma unroll
                        for (int v = 0; v < 4; v += 2) {  // the bias in FP32, after the sum
                            const float2 e = __fadd2_rn(make_float2(d[s][v], d[s][v + 1]),
                                                        make_float2(bv[n][0], bv[n][1]));
                            d[s][v] = e.x;
                            d[s][v + 1] = e.y;
                        }
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            d[s][v] = fmaxf(d[s][v], 0.f);
                            // sign bit of bits + 0x7fffffff: the value is above zero
                            if (MASK)
                                sub[2 * (v >> 1) + s] =
                                    __funnelshift_l(__float_as_uint(d[s][v]) + 0x7fffffffu,
                                                    sub[2 * (v >> 1) + s], 1);
                        }
                    }
                    const float2 l = __fadd2_rn(make_float2(d[0][0], d[0][1]),
                                                make_float2(d[0][2], d[0][3]));
                    const float2 q = __fadd2_rn(make_float2(d[1][0], d[1][1]),
                                                make_float2(d[1][2], d[1][3]));
                    const float2 s = __fmul2_rn(__fadd2_rn(l, q), make_float2(0.25f, 0.25f));
                    out[n] = pack2(s.x, s.y);
                }
                if (MASK)  // the bits came in from channel 0 on: reversed in each byte
                    mrow[(size_t)(p0 + 8 * j) * 4] =
                        __byte_perm(__brev(sub[0] | (sub[1] << 8) | (sub[2] << 16) | (sub[3] << 24)), 0,
                                    0x0123);
                prow[p0 + 8 * j] = make_uint4(out[0], out[1], out[2], out[3]);
            }
        }
        if (r >= rows) return;
    }
}

// dW1[o][tap] += sum over pixels of dA[px][o] x[px + tap], db1[o] += sum dA, with
// dA = (bit ? dP / 4 : 0) formed here.  A warp takes a pooled row, four windows
// (16 pixels, K) at a time: thread t has window t's pixels, rows are output
// channels g + 8 i, columns the nine taps and a column of ones (db).
__global__ void __launch_bounds__(256)
wgrad1_planes(const uint32_t* __restrict__ x, const uint16_t* __restrict__ dp,
              const uint4* __restrict__ mask, float* __restrict__ dW, float* __restrict__ db, int B,
              int H, int W) {
    __shared__ float s_w[CH][10];
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    for (int i = tid; i < CH * 10; i += 256) (&s_w[0][0])[i] = 0.f;
    __syncthreads();
    lgm::pdl_wait();
    lgm::pdl_trigger();
    const int H2 = H / 2, W2 = W / 2;
    const size_t plane = (size_t)H2 * W2 * 8;
    float acc[2][2][4];
#pragma unroll
    for (int i = 0; i < 16; ++i) (&acc[0][0][0])[i] = 0.f;
    const int ky = g / 3, kx = g % 3;  // column g: tap g
    const long long rows = (long long)B * H2;
    for (long long r = (long long)blockIdx.x * 8 + (tid >> 5); r < rows;
         r += (long long)gridDim.x * 8) {
        const int b = (int)(r / H2), py = (int)(r - (long long)b * H2);
        const uint32_t* img = x + (size_t)b * H * W2;
        const uint16_t* d0 = dp + (size_t)b * PL * plane + (size_t)py * W2 * 8 + g;
        const uint4* m0 = mask + ((size_t)b * H2 + py) * W2;
        // the two image rows of column g's tap, and of tap 8 (2, 2), in words of
        // two pixels; a row outside reads one inside and is masked out
        const int y0 = 2 * py + ky - 1, z0 = 2 * py + 1;
        const uint32_t k0 = y0 >= 0 && ky < 3 ? ~0u : 0u;
        const uint32_t k1 = y0 + 1 < H ? ~0u : 0u, kz = z0 + 1 < H ? ~0u : 0u;
        const uint32_t* r0 = img + (size_t)max(y0, 0) * W2;
        const uint32_t* r1 = img + (size_t)min(y0 + 1, H - 1) * W2;
        const uint32_t* s0 = img + (size_t)z0 * W2;
        const uint32_t* s1 = img + (size_t)min(z0 + 1, H - 1) * W2;
#pragma unroll 4
        for (int p0 = 0; p0 < W2; p0 += 4) {
            const int px = p0 + t;
            const uint4 m = m0[px];
            const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
            // pixels 2px + kx - 1 and the next: halves of two words
            const int il = kx == 0 ? px - 1 : px, ih = kx == 0 ? px : px + 1;
            const int jl = max(il, 0), jh = min(ih, W2 - 1);
            const uint32_t kl = il >= 0 ? ~0u : 0u, kh = ih < W2 ? ~0u : 0u;
            const uint32_t w0l = r0[jl] & kl, w0h = r0[jh] & kh, w1l = r1[jl] & kl, w1h = r1[jh] & kh;
            const uint32_t z = min(px + 1, W2 - 1), kn = px + 1 < W2 ? ~0u : 0u;
            const uint32_t v0l = s0[px], v0h = s0[z] & kn, v1l = s1[px], v1h = s1[z] & kn;
            uint32_t a[2][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint16_t v = to_bf(0.25f * bf(d0[i * plane + (size_t)px * 8]));
                const uint32_t vv = (uint32_t)v | ((uint32_t)v << 16);
                const uint32_t k = mw[i] >> g;  // bits 0, 8, 16, 24: the four sub-pixels
                a[i >> 1][i & 1] = vv & half_mask((k & 1u) | ((k << 8) & 0x10000u));
                a[i >> 1][2 + (i & 1)] = vv & half_mask(((k >> 16) & 1u) | ((k >> 8) & 0x10000u));
            }
            const int sh = kx == 1 ? 0 : 16;
            const uint32_t b0 = __funnelshift_r(w0l, w0h, sh) & k0, b1 = __funnelshift_r(w1l, w1h, sh) & k1;
            const uint32_t ones = g == 1 ? 0x3f803f80u : 0u;
            const uint32_t c0 = g == 0 ? __funnelshift_r(v0l, v0h, 16) : ones;
            const uint32_t c1 = g == 0 ? __funnelshift_r(v1l, v1h, 16) & kz : ones;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                mma16816(acc[i][0], a[i], b0, b1);
                mma16816(acc[i][1], a[i], c0, c1);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int o = 16 * i + 8 * h + g;
                atomicAdd(&s_w[o][2 * t + j], acc[i][0][2 * h + j]);
                if (t == 0) atomicAdd(&s_w[o][8 + j], acc[i][1][2 * h + j]);
            }
    __syncthreads();
    for (int i = tid; i < CH * 10; i += 256) {
        const int o = i / 10, k = i % 10;
        atomicAdd(k < 9 ? &dW[o * 9 + k] : &db[o], s_w[o][k]);
    }
}

// ---- 32 -> 32 channels ---------------------------------------------------------------------
// A tile is 8 columns x 16 rows: GEMM row 8 r + c is pixel (r, c), so that an
// eight-row core matrix is one run of pixels and the next one the row below.
constexpr int TX = 8, TY = 16;
constexpr int PX = TX + 2, PY = TY + 2;                    // the patch
constexpr uint32_t ROW_B = PX * 16, PLANE_B = PY * ROW_B;  // 160, 2880
constexpr uint32_t PATCH_B = PL * PLANE_B;                 // 11520
constexpr int NST = 4;                                     // stages (patch and 32 TMEM columns)
constexpr uint32_t WTS_B = 9u * PL * CH * 16u;             // 18432
constexpr uint32_t CONV_SMEM = NST * PATCH_B + WTS_B + CH * 4 + 3 * NST * 8 + 16;
constexpr uint32_t TMEM_COLS = NST * 32;
constexpr int EPI_WARPS = 8, CONV_THREADS = EPI_WARPS * 32 + 64;
constexpr uint32_t kIdesc = lgm::umma_idesc_bf16(128, CH);

enum { EP_POOL, EP_ACT, EP_PLAIN, EP_EXPAND };

__device__ __forceinline__ bool net_wait(uint64_t* bar, int use) {
    return lgm::mbar_wait_bounded(bar, (uint32_t)(use & 1), &g_net_error);
}

// Implicit GEMM, M = 128 pixels, N = 32, K = 9 taps x 32 channels as 18
// tcgen05.mma of K 16.  One thread of warp 8 copies patches (one TMA box each),
// one of warp 9 multiplies; two groups of four warps take alternate tiles'
// epilogues.
//   EP_POOL    bias, ReLU, 2x2 mean -> out planes [H/2][W/2]; bits (optional) a
//              word per pixel [B][H][W]
//   EP_ACT     bias, ReLU -> out planes [H][W]
//   EP_PLAIN   out planes [H][W]
//   EP_EXPAND  the gradient behind a pooled ReLU: value / 4 at the four pixels
//              whose bit is set in bits [B][2H][2W] -> out planes [2H][2W]
// w: FP32 masters [32][288], or with FLIP the same masters of the layer whose
// input gradient this is (taps reversed, channels transposed).
// Bound: the tensor core's reads of the A operand, 4 KB per multiplication of only 32
// columns.  Layer 2, 1024 images: 121 us, 868 clocks a tile and SM, the tcgen05 pipe
// busy in 89% of them (43 clocks a multiplication).
template <int EP, bool FLIP>
__global__ void __launch_bounds__(CONV_THREADS, 3)
conv_planes(const __grid_constant__ CUtensorMap xmap, const float* __restrict__ w,
            const float* __restrict__ bias, uint4* __restrict__ out, uint32_t* __restrict__ bits,
            int B, int H, int W) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* ws = smem + NST * PATCH_B;  // [9][PL][CH][16 B]
    float* s_bias = reinterpret_cast<float*>(ws + WTS_B);
    uint64_t* full = reinterpret_cast<uint64_t*>(ws + WTS_B + CH * 4);
    uint64_t* done = full + NST;
    uint64_t* empty = full + 2 * NST;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(full + 3 * NST);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles_x = W / TX, tiles_y = (H + TY - 1) / TY;
    const int ntiles = B * tiles_x * tiles_y;
    const int n = ((int)blockIdx.x < ntiles) ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

    if (warp == 0) lgm::tmem_alloc(tslot, TMEM_COLS);
    if (tid == 0) {
        for (int i = 0; i < 2 * NST; ++i) lgm::mbar_init(&full[i], 1);        // full, done
        for (int i = 2 * NST; i < 3 * NST; ++i) lgm::mbar_init(&full[i], 4);  // empty
        lgm::fence_mbar_init();
    }
    if (tid < CH) s_bias[tid] = (EP == EP_POOL || EP == EP_ACT) ? bias[tid] : 0.f;
    // ws[t][c8][o] = the eight input channels 8 c8 .. of tap t, output channel
    // o; neighbouring threads read neighbouring masters
    for (int i = tid; i < 9 * PL * CH; i += CONV_THREADS) {
        const int o = FLIP ? i % CH : i / (9 * PL), q = FLIP ? i / CH : i % (9 * PL);
        const int t = q / PL, c8 = q % PL;
        float v[8];
        if constexpr (FLIP) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = w[(8 * c8 + j) * 9 * CH + (8 - t) * CH + o];
        } else {
            const float4* p = reinterpret_cast<const float4*>(w + o * 9 * CH + q * 8);
            const float4 a = p[0], c = p[1];
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
            v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
        }
        *reinterpret_cast<uint4*>(ws + (size_t)(q * CH + o) * 16) =
            make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
    }
    lgm::fence_proxy_async_smem();
    lgm::tc_fence_before();
    __syncthreads();
    lgm::tc_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t xs_a = smem_addr(smem), ws_a = smem_addr(ws);

    lgm::pdl_wait();  // what follows reads and writes the pass's activations
    lgm::pdl_trigger();

    auto origin = [&](int k, int& b, int& y0, int& x0) {
        const int tile = (int)blockIdx.x + k * (int)gridDim.x;
        b = tile / (tiles_x * tiles_y);
        const int rem = tile - b * (tiles_x * tiles_y);
        y0 = (rem / tiles_x) * TY;
        x0 = (rem % tiles_x) * TX;
    };

    if (warp == EPI_WARPS) {  // ---- copies
        if (lane == 0) {
            int k = 0;
            for (; k < n; ++k) {
                const int st = k % NST;
                // the tile before in this buffer is multiplied
                if (k >= NST && !net_wait(&done[st], k / NST - 1)) break;
                int b, y0, x0;
                origin(k, b, y0, x0);
                lgm::mbar_arrive_expect_tx(&full[st], PATCH_B);
                lgm::tma_box_4d(xs_a + st * PATCH_B, &xmap, (x0 - 1) * 8, y0 - 1, 0, b, &full[st]);
            }
            // after a timeout: the copies in flight land before the CTA leaves (bounded)
            if (k < n) lgm::mbar_drain_ring(full, NST, (uint32_t)std::max(0, k - NST), (uint32_t)k);
        }
        __syncwarp();
    } else if (warp == EPI_WARPS + 1) {  // ---- multiplications
        if (lane == 0 && n > 0) {
            const uint64_t a0 = lgm::umma_desc(xs_a, PLANE_B, ROW_B);
            const uint64_t b0 = lgm::umma_desc(ws_a, CH * 16, 128);
            int k = 0;
            for (; k < n; ++k) {
                const int st = k % NST;
                if (!net_wait(&full[st], k / NST) || (k >= NST && !net_wait(&empty[st], k / NST - 1)))
                    break;
                lgm::tc_fence_after();
                // a descriptor's address field counts 16 bytes
                const uint64_t a = a0 + (uint64_t)(st * (PATCH_B / 16));
                const uint32_t d = tmem + (uint32_t)(st * 32);
#pragma unroll
                for (int t = 0; t < 9; ++t)
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        lgm::umma_f16(d,
                                      a + (uint64_t)(((t / 3) * ROW_B + (t % 3) * 16 + 2 * j * PLANE_B) / 16),
                                      b0 + (uint64_t)((t * PL + 2 * j) * CH), kIdesc, (t | j) ? 1u : 0u);
                lgm::umma_commit_to(&done[st]);
            }
            // the last multiplications end before the tensor memory is freed (bounded)
            for (int i = std::max(0, k - NST); i < k; ++i)
                for (int it = 0; it < lgm::kWaitLimit; ++it)
                    if (lgm::mbar_try_wait(&done[i % NST], (uint32_t)((i / NST) & 1))) break;
        }
        __syncwarp();
    } else {
        const int grp = warp >> 2, wq = warp & 3;
        const int c = lane & 7, rr = 4 * wq + (lane >> 3);  // this thread's pixel of the tile
        for (int k = grp; k < n; k += 2) {
            const int st = k % NST;
            if (!__all_sync(0xffffffffu, net_wait(&done[st], k / NST))) break;
            lgm::tc_fence_after();
            float v[32];
            lgm::tmem_ld32x(tmem + (uint32_t)(st * 32) + ((uint32_t)(wq * 32) << 16), v);
            lgm::tc_fence_before();
            __syncwarp();
            if (lane == 0) lgm::mbar_arrive(&empty[st]);
            int b, y0, x0;
            origin(k, b, y0, x0);
            const int y = y0 + rr, xx = x0 + c;
            if (EP == EP_POOL || EP == EP_ACT) {
#pragma unroll
                for (int ch = 0; ch < 32; ch += 4) {
                    const float4 bb = *reinterpret_cast<const float4*>(s_bias + ch);
                    v[ch] = fmaxf(v[ch] + bb.x, 0.f);
                    v[ch + 1] = fmaxf(v[ch + 1] + bb.y, 0.f);
                    v[ch + 2] = fmaxf(v[ch + 2] + bb.z, 0.f);
                    v[ch + 3] = fmaxf(v[ch + 3] + bb.w, 0.f);
                }
            }
            if constexpr (EP == EP_POOL) {
                if (bits && y < H) {
                    uint32_t m = 0;
#pragma unroll
                    for (int ch = 31; ch >= 0; --ch)
                        m = __funnelshift_l(__float_as_uint(v[ch]) + 0x7fffffffu, m, 1);
                    bits[((size_t)b * H + y) * W + xx] = m;
                }
                // Rows first, then columns; each exchange halves a lane's
                // channels, so the window's four lanes end with a plane each.
                const bool lower = (lane >> 3) & 1, right = lane & 1;
                float s[16], p[8];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float keep = lower ? v[16 + i] : v[i], send = lower ? v[i] : v[16 + i];
                    s[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float keep = right ? s[8 + i] : s[i], send = right ? s[i] : s[8 + i];
                    p[i] = 0.25f * (keep + __shfl_xor_sync(0xffffffffu, send, 1));
                }
                const int H2 = H / 2, W2 = W / 2, pl = (lower ? 2 : 0) + (right ? 1 : 0);
                if (y < H)
                    out[(((size_t)b * PL + pl) * H2 + y / 2) * W2 + xx / 2] =
                        make_uint4(pack2(p[0], p[1]), pack2(p[2], p[3]), pack2(p[4], p[5]),
                                   pack2(p[6], p[7]));
            } else if constexpr (EP == EP_EXPAND) {
                if (y < H) {
                    uint32_t pk[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) pk[i] = pack2(0.25f * v[2 * i], 0.25f * v[2 * i + 1]);
                    const int H2 = 2 * H, W2 = 2 * W;
#pragma unroll
                    for (int dy = 0; dy < 2; ++dy) {
                        const uint2 mm = *reinterpret_cast<const uint2*>(
                            bits + ((size_t)b * H2 + 2 * y + dy) * W2 + 2 * xx);
#pragma unroll
                        for (int dx = 0; dx < 2; ++dx) {
                            const uint32_t m = dx ? mm.y : mm.x;
#pragma unroll
                            for (int pl = 0; pl < PL; ++pl) {
                                uint32_t q[4];
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const uint32_t tb = m >> (8 * pl + 2 * i);
                                    q[i] = pk[4 * pl + i] & half_mask((tb & 1u) | ((tb << 15) & 0x10000u));
                                }
                                out[(((size_t)b * PL + pl) * H2 + 2 * y + dy) * W2 + 2 * xx + dx] =
                                    make_uint4(q[0], q[1], q[2], q[3]);
                            }
                        }
                    }
                }
            } else {
                if (y < H) {
#pragma unroll
                    for (int pl = 0; pl < PL; ++pl)
                        out[(((size_t)b * PL + pl) * H + y) * W + xx] =
                            make_uint4(pack2(v[8 * pl], v[8 * pl + 1]), pack2(v[8 * pl + 2], v[8 * pl + 3]),
                                       pack2(v[8 * pl + 4], v[8 * pl + 5]),
                                       pack2(v[8 * pl + 6], v[8 * pl + 7]));
                }
            }
        }
    }
    lgm::tc_fence_before();
    __syncthreads();
    lgm::tc_fence_after();
    if (warp == 0) lgm::tmem_free(tmem, TMEM_COLS);
}

// dW[o][tap 32 + c] += sum over pixels of dA[px][o] x[px + tap][c], db[o] += sum dA.
// A CTA walks tiles of 8 x 16 pixels; warp (ky, q) has tap row ky (96 columns)
// and the tile's rows 4q .. 4q+3, 16 pixels (two rows) per step: fragments of
// both operands by transposing ldmatrix, 24 multiplications per 8 of them.  The
// four row quarters are added in shared memory at the end, and the CTA's sums
// to global memory.  Bound: shared-memory reads and the mma.sync rate.
constexpr int WG_WARPS = 12, WG_ST = 4;
constexpr uint32_t DTILE_B = PL * TY * TX * 16;  // 8192
constexpr uint32_t WG_STAGE = PATCH_B + DTILE_B;
constexpr uint32_t WG_SMEM = WG_ST * WG_STAGE + 2 * WG_ST * 8;

__global__ void __launch_bounds__(WG_WARPS * 32, 1)
wgrad_planes(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap dmap,
             float* __restrict__ dW, float* __restrict__ db, int B, int H, int W) {
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + WG_ST * WG_STAGE);
    uint64_t* empty = full + WG_ST;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int ky = warp % 3, q = warp / 3;
    const int tiles_x = W / TX, tiles_y = (H + TY - 1) / TY;
    const int ntiles = B * tiles_x * tiles_y;
    const int n = ((int)blockIdx.x < ntiles) ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (tid == 0) {
        for (int i = 0; i < WG_ST; ++i) {
            lgm::mbar_init(&full[i], 1);
            lgm::mbar_init(&empty[i], WG_WARPS);
        }
        lgm::fence_mbar_init();
    }
    __syncthreads();
    lgm::pdl_wait();
    lgm::pdl_trigger();
    auto copy = [&](int k) {
        const int tile = (int)blockIdx.x + k * (int)gridDim.x, st = k % WG_ST;
        const int b = tile / (tiles_x * tiles_y), rem = tile - b * (tiles_x * tiles_y);
        const int y0 = (rem / tiles_x) * TY, x0 = (rem % tiles_x) * TX;
        const uint32_t s = smem_addr(smem) + st * WG_STAGE;
        lgm::mbar_arrive_expect_tx(&full[st], WG_STAGE);
        lgm::tma_box_4d(s, &xmap, (x0 - 1) * 8, y0 - 1, 0, b, &full[st]);
        // rows past the image read zeros and are left out
        lgm::tma_box_4d(s + PATCH_B, &dmap, x0 * 8, y0, 0, b, &full[st]);
    };
    int copied = 0;
    if (tid == 0)
        for (; copied < WG_ST && copied < n; ++copied) copy(copied);
    float acc[3][4][2][4];
    float accb[2][4];
#pragma unroll
    for (int i = 0; i < 96; ++i) (&acc[0][0][0][0])[i] = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) (&accb[0][0])[i] = 0.f;
    // ldmatrix row of this lane: matrices (pixels 0-7 | 8-15) x (plane | next plane)
    const int mi = lane >> 3, ri = lane & 7;
    bool ok = true;
    for (int k = 0; k < n; ++k) {
        const int st = k % WG_ST;
        ok = __all_sync(0xffffffffu, net_wait(&full[st], k / WG_ST));
        if (!ok) break;
        const uint32_t xs = smem_addr(smem) + st * WG_STAGE, ds = xs + PATCH_B;
        const int tile = (int)blockIdx.x + k * (int)gridDim.x;
        const int rows = H - tile / tiles_x % tiles_y * TY;  // of the image from the tile's first on
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = 4 * q + 2 * h;  // tile rows row, row + 1 (H is even)
            // Past the image dA is zero, but the row above is not: no gradient there
            // does not stop an infinity.
            if (row >= rows) continue;
            uint32_t a[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i)  // a0, a1: planes 2i, 2i+1, pixels 0-7; a2, a3: 8-15
                ldsm4_trans(a[i], ds + (uint32_t)(((2 * i + (mi & 1)) * TY + row + (mi >> 1)) * TX + ri) * 16);
            if (ky == 1) {
                mma16816(accb[0], a[0], 0x3f803f80u, 0x3f803f80u);
                mma16816(accb[1], a[1], 0x3f803f80u, 0x3f803f80u);
            }
#pragma unroll
            for (int kx = 0; kx < 3; ++kx)
#pragma unroll
                for (int cp = 0; cp < 2; ++cp) {  // b: plane 2cp pixels 0-7, 8-15, then plane 2cp+1
                    uint32_t bb[4];
                    ldsm4_trans(bb, xs + (uint32_t)(2 * cp + (mi >> 1)) * PLANE_B +
                                        (uint32_t)(row + (mi & 1) + ky) * ROW_B + (uint32_t)(ri + kx) * 16);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        mma16816(acc[kx][2 * cp][i], a[i], bb[0], bb[1]);
                        mma16816(acc[kx][2 * cp + 1][i], a[i], bb[2], bb[3]);
                    }
                }
        }
        __syncwarp();
        if (lane == 0) lgm::mbar_arrive(&empty[st]);
        if (tid == 0 && copied < n && copied < k + WG_ST + 1) {
            ok = net_wait(&empty[st], k / WG_ST);
            if (ok) {
                lgm::fence_proxy_async_smem();
                copy(copied++);
            }
        }
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (!ok) break;
    }
    if (tid == 0)  // after a timeout: the copies in flight land first (bounded)
        for (int k = std::max(0, copied - WG_ST); k < copied; ++k)
            for (int it = 0; it < lgm::kWaitLimit; ++it)
                if (lgm::mbar_try_wait(&full[k % WG_ST], (uint32_t)((k / WG_ST) & 1))) break;
    __syncthreads();
    if (n == 0) return;
    constexpr int WSUM = 9 * CH + 8;              // row stride (bank skew)
    float* sum = reinterpret_cast<float*>(smem);  // [CH][WSUM] and [CH]
    for (int r = 0; r < 4; ++r) {
        if (q == r) {
#pragma unroll
            for (int kx = 0; kx < 3; ++kx)
#pragma unroll
                for (int cn = 0; cn < 4; ++cn)
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int o = 16 * i + g + 8 * h;
                            const int col = (ky * 3 + kx) * CH + 8 * cn + 2 * t;
                            float2* p = reinterpret_cast<float2*>(sum + o * WSUM + col);
                            float2 v = make_float2(acc[kx][cn][i][2 * h], acc[kx][cn][i][2 * h + 1]);
                            if (r > 0) v = __fadd2_rn(*p, v);
                            *p = v;
                        }
            if (ky == 1 && t == 0)
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float* p = sum + CH * WSUM + 16 * i + 8 * h + g;
                        *p = r == 0 ? accb[i][2 * h] : *p + accb[i][2 * h];
                    }
        }
        __syncthreads();
    }
    for (int i = tid; i < CH * 9 * CH / 4; i += WG_WARPS * 32) {
        const float4 v = *reinterpret_cast<const float4*>(sum + (i / (9 * CH / 4)) * WSUM +
                                                          (i % (9 * CH / 4)) * 4);
        asm volatile("red.global.add.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(dW + 4 * i), "f"(v.x),
                     "f"(v.y), "f"(v.z), "f"(v.w)
                     : "memory");
    }
    if (tid < CH) atomicAdd(&db[tid], sum[CH * WSUM + tid]);
}

// ---- the head --------------------------------------------------------------------------------
// One block per image: the mean over the pixels of a4 (planes, pixel by pixel
// in FP32), then the two fully connected layers.  Keeps the BF16 mean and
// hidden layer for the backward pass.
constexpr int GAP_CHUNK = 256;                    // pixels staged at a time
constexpr int GAP_STRIDE = GAP_CHUNK * 16 + 16;   // bytes of a staged plane (bank skew)
__global__ void __launch_bounds__(256)
head_fwd(const uint4* __restrict__ a4, int HW, const float* __restrict__ w1,
         const float* __restrict__ b1, const float* __restrict__ w2, const float* __restrict__ b2,
         uint16_t* __restrict__ g16, uint16_t* __restrict__ h16, float* __restrict__ y) {
    __shared__ __align__(16) unsigned char s_a[PL * GAP_STRIDE];
    __shared__ __align__(4) uint16_t s_g[CH], s_h[HID];
    const int b = blockIdx.x, tid = threadIdx.x;
    // The products on the tensor cores, K in steps of 16, the image in row 0 of
    // 16; a warp takes eight hidden units.
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    uint32_t f1[CH / 16][2], f2[HID / 16][2];
#pragma unroll
    for (int k = 0; k < CH / 16; ++k)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float* p = w1 + (8 * warp + g) * CH + 16 * k + 8 * h + 2 * t;
            f1[k][h] = pack2(p[0], p[1]);
        }
#pragma unroll
    for (int k = 0; k < HID / 16; ++k)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float* p = w2 + g * HID + 16 * k + 8 * h + 2 * t;
            f2[k][h] = warp == 0 && g < OUT ? pack2(p[0], p[1]) : 0u;
        }
    lgm::pdl_wait();
    lgm::pdl_trigger();
    const uint4* img = a4 + (size_t)b * PL * HW;
    float s = 0.f;
    for (int p0 = 0; p0 < HW; p0 += GAP_CHUNK) {
        const int m = min(GAP_CHUNK, HW - p0);
        for (int i = tid; i < PL * m; i += 256)
            *reinterpret_cast<uint4*>(s_a + (i / m) * GAP_STRIDE + (i % m) * 16) =
                img[(size_t)(i / m) * HW + p0 + i % m];
        __syncthreads();
        if (tid < CH) {
            const uint16_t* a = reinterpret_cast<const uint16_t*>(s_a + (tid >> 3) * GAP_STRIDE) + (tid & 7);
#pragma unroll 8
            for (int p = 0; p < m; ++p) s += bf(a[p * 8]);
        }
        __syncthreads();
    }
    if (tid < CH) {
        const uint16_t v = to_bf(s / (float)HW);
        s_g[tid] = v;
        g16[(size_t)b * CH + tid] = v;
    }
    __syncthreads();
    // row 0 of A: thread t of the first four holds k = 2t, 2t+1, 2t+8, 2t+9
    auto row0 = [&](const uint16_t* src, int k, uint32_t (&a)[4]) {
        a[0] = g == 0 ? *reinterpret_cast<const uint32_t*>(src + 16 * k + 2 * t) : 0u;
        a[2] = g == 0 ? *reinterpret_cast<const uint32_t*>(src + 16 * k + 8 + 2 * t) : 0u;
        a[1] = a[3] = 0u;
    };
    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < CH / 16; ++k) {
        uint32_t a[4];
        row0(s_g, k, a);
        mma16816(c, a, f1[k][0], f1[k][1]);
    }
    if (g == 0)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int n = 8 * warp + 2 * t + i;
            const uint16_t v = to_bf(fmaxf(c[i] + b1[n], 0.f));
            s_h[n] = v;
            h16[(size_t)b * HID + n] = v;
        }
    __syncthreads();
    if (warp != 0) return;
    c[0] = c[1] = c[2] = c[3] = 0.f;
#pragma unroll
    for (int k = 0; k < HID / 16; ++k) {
        uint32_t a[4];
        row0(s_h, k, a);
        mma16816(c, a, f2[k][0], f2[k][1]);
    }
    if (lane == 0)
        for (int i = 0; i < OUT; ++i) y[(size_t)b * OUT + i] = c[i] + b2[i];
}

// One block per image: the gradient through the head down to a4's ReLU,
// dA4 planes = (a4 > 0) ? dg / HW : 0; keeps dh (BF16) for the weight gradients.
__global__ void __launch_bounds__(256)
head_bwd(const float* __restrict__ dy, const uint16_t* __restrict__ h16,
         const uint4* __restrict__ a4, int HW, const float* __restrict__ w1,
         const float* __restrict__ w2, uint16_t* __restrict__ dh16, uint4* __restrict__ dA4) {
    __shared__ float s_dh[HID];
    __shared__ __align__(16) uint16_t s_g[CH];
    const int b = blockIdx.x, tid = threadIdx.x;
    lgm::pdl_wait();
    lgm::pdl_trigger();
    if (tid < HID) {
        float d = 0.f;
#pragma unroll
        for (int k = 0; k < OUT; ++k)
            d = fmaf(bf(to_bf(dy[(size_t)b * OUT + k])), bf(to_bf(w2[k * HID + tid])), d);
        const uint16_t v = h16[(size_t)b * HID + tid] ? to_bf(d) : (uint16_t)0;  // h >= 0
        s_dh[tid] = bf(v);
        dh16[(size_t)b * HID + tid] = v;
    }
    __syncthreads();
    if (tid < CH) {
        float d = 0.f;
#pragma unroll 8
        for (int j = 0; j < HID; ++j) d = fmaf(s_dh[j], bf(to_bf(w1[j * CH + tid])), d);
        s_g[tid] = to_bf(d / (float)HW);
    }
    __syncthreads();
    for (int i = tid; i < PL * HW; i += 256) {
        const uint4 a = a4[(size_t)b * PL * HW + i];
        const uint4 d = *reinterpret_cast<const uint4*>(s_g + 8 * (i / HW));
        const uint32_t av[4] = {a.x, a.y, a.z, a.w}, dv[4] = {d.x, d.y, d.z, d.w};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)  // a4 >= 0: positive unless its bits are zero
            o[j] = dv[j] & (((av[j] & 0xffffu) ? 0xffffu : 0u) | ((av[j] >> 16) ? 0xffff0000u : 0u));
        dA4[(size_t)b * PL * HW + i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// The head's weight and bias gradients, one output per thread, images in order:
// dW1 [64][32], db1 [64], dW2 [2][64], db2 [2].
constexpr int HEAD_OUTS = HID * CH + HID + OUT * HID + OUT;
__global__ void __launch_bounds__(128)
head_wgrad(const float* __restrict__ dy, const uint16_t* __restrict__ dh16,
           const uint16_t* __restrict__ h16, const uint16_t* __restrict__ g16, int B,
           float* __restrict__ dw1, float* __restrict__ db1, float* __restrict__ dw2,
           float* __restrict__ db2) {
    lgm::pdl_wait();
    lgm::pdl_trigger();
    int i = blockIdx.x * 128 + threadIdx.x;
    if (i >= HEAD_OUTS) return;
    float s = 0.f;
    if (i < HID * CH) {
        const int j = i / CH, c = i % CH;
#pragma unroll 16
        for (int b = 0; b < B; ++b) s = fmaf(bf(dh16[(size_t)b * HID + j]), bf(g16[(size_t)b * CH + c]), s);
        dw1[i] = s;
    } else if ((i -= HID * CH) < HID) {
#pragma unroll 16
        for (int b = 0; b < B; ++b) s += bf(dh16[(size_t)b * HID + i]);
        db1[i] = s;
    } else if ((i -= HID) < OUT * HID) {
        const int k = i / HID, j = i % HID;
#pragma unroll 16
        for (int b = 0; b < B; ++b)
            s = fmaf(bf(to_bf(dy[(size_t)b * OUT + k])), bf(h16[(size_t)b * HID + j]), s);
        dw2[i] = s;
    } else {
        i -= OUT * HID;
#pragma unroll 16
        for (int b = 0; b < B; ++b) s += bf(to_bf(dy[(size_t)b * OUT + i]));
        db2[i] = s;
    }
}

// The gradients that are added to, cleared: weights and biases of the convolutions.
struct ConvGrads {
    float* w[4];
    float* b[4];
};
__global__ void __launch_bounds__(256) zero_grads(ConvGrads G) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < CH * 9) G.w[0][i] = 0.f;
    if (i < CH * 9 * CH) G.w[1][i] = G.w[2][i] = G.w[3][i] = 0.f;
    if (i < CH) G.b[0][i] = G.b[1][i] = G.b[2][i] = G.b[3][i] = 0.f;
}

// The weights the backward pass reads, as they are now: a program may change
// its masters in between.
constexpr int W3 = CH * 9 * CH, KEPT_FLOATS = 3 * W3 + HID * CH + OUT * HID;
struct KeptWeights {
    const float* p[5];  // c2w, c3w, c4w, f1w, f2w
};
__global__ void __launch_bounds__(256) keep_weights(KeptWeights K, float* __restrict__ dst) {
    lgm::pdl_wait();
    lgm::pdl_trigger();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < 3 * W3) dst[i] = K.p[i / W3][i % W3];
    else if (i < 3 * W3 + HID * CH) dst[i] = K.p[3][i - 3 * W3];
    else if (i < KEPT_FLOATS) dst[i] = K.p[4][i - 3 * W3 - HID * CH];
}

// ---- host side ---------------------------------------------------------------------------------

// What the two calls share of a pass, in one allocation (256-byte aligned slices).
struct Saved {
    size_t p1, p2, p3, a4, m1, m2, m3, g16, h16, w, total;
};
Saved saved_layout(int B, int H, int W, bool keep) {
    Saved s{};
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) / 256 * 256;
        return o;
    };
    const size_t px = (size_t)B * H * W;
    s.p1 = take(px / 4 * 64);
    s.p2 = take(px / 16 * 64);
    s.p3 = take(px / 64 * 64);
    s.a4 = take(px / 64 * 64);
    s.g16 = take((size_t)B * CH * 2);
    s.h16 = take((size_t)B * HID * 2);
    if (keep) {
        s.m1 = take(px / 4 * 16);
        s.m2 = take(px / 4 * 4);
        s.m3 = take(px / 16 * 4);
        s.w = take(KEPT_FLOATS * sizeof(float));
    }
    s.total = at;
    return s;
}
struct Grad {
    size_t dp1, dA2, dA3, dA4, dh16, total;
};
Grad grad_layout(int B, int H, int W) {
    Grad g{};
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) / 256 * 256;
        return o;
    };
    const size_t px = (size_t)B * H * W;
    g.dp1 = take(px / 4 * 64);
    g.dA2 = take(px / 4 * 64);
    g.dA3 = take(px / 16 * 64);
    g.dA4 = take(px / 64 * 64);
    g.dh16 = take((size_t)B * HID * 2);
    g.total = at;
    return g;
}

struct Device {
    int sms = 0, conv_ctas = 0;
    PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
};

// A kernel of the pass after the first: it may start while the one ahead of it
// runs, and waits for it (pdl_wait) before it touches the pass's data.
template <typename... P, typename... A>
void launch(void (*k)(P...), int grid, int block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

template <int EP, bool FLIP>
cudaError_t conv_attributes() {
    cudaError_t e = cudaFuncSetAttribute(conv_planes<EP, FLIP>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CONV_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(conv_planes<EP, FLIP>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    return e;
}

// Attributes and limits of the current device, looked up once per device.
lgm_status device_of(Device* out) {
    constexpr int kDevices = 64;
    static std::mutex lock;
    static Device known[kDevices];
    int dev = 0, smem_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return LGM_ERR_CUDA;
    std::lock_guard<std::mutex> hold(lock);
    Device* d = &known[dev];
    if (d->encode) {
        *out = *d;
        return LGM_OK;
    }
    if (cudaDeviceGetAttribute(&d->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) !=
            cudaSuccess ||
        conv_attributes<EP_POOL, false>() != cudaSuccess ||
        conv_attributes<EP_ACT, false>() != cudaSuccess ||
        conv_attributes<EP_PLAIN, true>() != cudaSuccess ||
        conv_attributes<EP_EXPAND, true>() != cudaSuccess ||
        cudaFuncSetAttribute(wgrad_planes, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)WG_SMEM) != cudaSuccess)
        return LGM_ERR_CUDA;
    // CTAs per SM from the shared memory (1 KB reserved per CTA) and the tensor
    // memory: the occupancy query answers one for a kernel that allocates it
    d->conv_ctas = d->sms * std::max(1, std::min({3, smem_sm / (int)(CONV_SMEM + 1024),
                                                  512 / (int)TMEM_COLS}));
    cudaDriverEntryPointQueryResult q;
    void* fn = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
        return LGM_ERR_CUDA;
    d->encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    *out = *d;
    return LGM_OK;
}

// Planes [B][4][H][W][8] with a box of bx pixels x by rows of all planes.
bool plane_map(const Device& d, CUtensorMap* map, const void* p, int B, int H, int W, int bx, int by) {
    const cuuint64_t dims[4] = {(cuuint64_t)W * 8, (cuuint64_t)H, (cuuint64_t)PL, (cuuint64_t)B};
    const cuuint64_t strides[3] = {(cuuint64_t)W * 16, (cuuint64_t)H * W * 16,
                                   (cuuint64_t)PL * H * W * 16};
    const cuuint32_t box[4] = {(cuuint32_t)bx * 8, (cuuint32_t)by, (cuuint32_t)PL, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return d.encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p), dims, strides, box,
                    estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
}

int tiles_of(int B, int H, int W) { return B * (W / TX) * ((H + TY - 1) / TY); }

template <int EP, bool FLIP>
bool conv(const Device& d, const void* in, const float* w, const float* bias, void* out, void* bits,
          int B, int H, int W, cudaStream_t st) {
    CUtensorMap map;
    if (!plane_map(d, &map, in, B, H, W, PX, PY)) return false;
    launch(conv_planes<EP, FLIP>, std::min(tiles_of(B, H, W), d.conv_ctas), CONV_THREADS, CONV_SMEM, st,
           map, w, bias, (uint4*)out, (uint32_t*)bits, B, H, W);
    return true;
}
bool wgrad(const Device& d, const void* x, const void* dA, float* dW, float* db, int B, int H, int W,
           cudaStream_t st) {
    CUtensorMap xm, dm;
    if (!plane_map(d, &xm, x, B, H, W, PX, PY) || !plane_map(d, &dm, dA, B, H, W, TX, TY)) return false;
    launch(wgrad_planes, std::min(tiles_of(B, H, W), d.sms), WG_WARPS * 32, WG_SMEM, st, xm, dm, dW, db,
           B, H, W);
    return true;
}

bool shape_ok(int B, int H, int W) {
    // layer 4 works on H/8 x W/8 in tiles of 8 columns
    return B >= 1 && H >= 16 && W >= 64 && H % 16 == 0 && W % 64 == 0 &&
           (long long)B * H * W < (1ll << 40);
}

}  // namespace

unsigned lgm_cnn_net_error_take() {
    unsigned v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_net_error, sizeof v) != cudaSuccess ||
        cudaMemcpyToSymbol(g_net_error, &zero, sizeof zero) != cudaSuccess)
        return ~0u;
    return v;
}

extern "C" {

size_t lgm_cnn_net_bytes(int32_t B, int32_t H, int32_t W, int32_t which) {
    if (!shape_ok(B, H, W)) return 0;
    return which == 2 ? grad_layout(B, H, W).total : saved_layout(B, H, W, which == 1).total;
}

lgm_status lgm_cnn_net_forward(const void* x, const float* const* params, void* saved, float* y,
                               int32_t B, int32_t H, int32_t W, int32_t keep, void* stream) {
    if (!x || !params || !saved || !y || !shape_ok(B, H, W)) return LGM_ERR_INVALID_ARGUMENT;
    if (((uintptr_t)x & 3u) || ((uintptr_t)saved & 255u)) return LGM_ERR_INVALID_ARGUMENT;
    for (int i = 0; i < 12; ++i)  // conv_planes reads the masters of layers 2 to 4 as float4
        if (!params[i] || ((uintptr_t)params[i] & (i == 2 || i == 4 || i == 6 ? 15u : 3u)))
            return LGM_ERR_INVALID_ARGUMENT;
    Device d;
    lgm_status s = device_of(&d);
    if (s != LGM_OK) return s;
    cudaStream_t st = (cudaStream_t)stream;
    const Saved L = saved_layout(B, H, W, keep != 0);
    char* w = (char*)saved;
    const int grid1 = (int)std::min<long long>(((long long)B * (H / 2) + C1_WARPS - 1) / C1_WARPS,
                                               (long long)d.sms * C1_CTAS);
    if (keep)
        conv1_planes<true><<<grid1, C1_WARPS * 32, 0, st>>>((const uint32_t*)x, params[0], params[1],
                                                            (uint4*)(w + L.p1), (uint32_t*)(w + L.m1),
                                                            B, H, W);
    else
        conv1_planes<false><<<grid1, C1_WARPS * 32, 0, st>>>((const uint32_t*)x, params[0], params[1],
                                                             (uint4*)(w + L.p1), nullptr, B, H, W);
    if (keep)
        launch(keep_weights, (KEPT_FLOATS + 255) / 256, 256, 0, st,
               KeptWeights{{params[2], params[4], params[6], params[8], params[10]}}, (float*)(w + L.w));
    if (!conv<EP_POOL, false>(d, w + L.p1, params[2], params[3], w + L.p2, keep ? w + L.m2 : nullptr, B,
                              H / 2, W / 2, st) ||
        !conv<EP_POOL, false>(d, w + L.p2, params[4], params[5], w + L.p3, keep ? w + L.m3 : nullptr, B,
                              H / 4, W / 4, st) ||
        !conv<EP_ACT, false>(d, w + L.p3, params[6], params[7], w + L.a4, nullptr, B, H / 8, W / 8, st))
        return LGM_ERR_CUDA;
    launch(head_fwd, B, 256, 0, st, (const uint4*)(w + L.a4), (H / 8) * (W / 8), params[8], params[9],
           params[10], params[11], (uint16_t*)(w + L.g16), (uint16_t*)(w + L.h16), y);
    return cudaGetLastError() == cudaSuccess ? LGM_OK : LGM_ERR_CUDA;
}

lgm_status lgm_cnn_net_backward(const void* x, const void* saved, const float* dy,
                                void* work, float* const* grads, int32_t B, int32_t H,
                                int32_t W, void* stream) {
    if (!x || !saved || !dy || !work || !grads || !shape_ok(B, H, W))
        return LGM_ERR_INVALID_ARGUMENT;
    if (((uintptr_t)x & 3u) || ((uintptr_t)saved & 255u) || ((uintptr_t)work & 255u))
        return LGM_ERR_INVALID_ARGUMENT;
    for (int i = 0; i < 12; ++i)
        if (!grads[i] || ((uintptr_t)grads[i] & 15u)) return LGM_ERR_INVALID_ARGUMENT;
    Device d;
    lgm_status s = device_of(&d);
    if (s != LGM_OK) return s;
    cudaStream_t st = (cudaStream_t)stream;
    const Saved L = saved_layout(B, H, W, true);
    const Grad G = grad_layout(B, H, W);
    char* w = (char*)saved;
    char* k = (char*)work;
    const float* c2w = (const float*)(w + L.w);
    const float *c3w = c2w + W3, *c4w = c3w + W3, *f1w = c4w + W3, *f2w = f1w + HID * CH;
    const int HW = (H / 8) * (W / 8);
    zero_grads<<<(CH * 9 * CH + 255) / 256, 256, 0, st>>>(
        ConvGrads{{grads[0], grads[2], grads[4], grads[6]}, {grads[1], grads[3], grads[5], grads[7]}});
    launch(head_bwd, B, 256, 0, st, dy, (const uint16_t*)(w + L.h16), (const uint4*)(w + L.a4), HW,
                                f1w, f2w, (uint16_t*)(k + G.dh16), (uint4*)(k + G.dA4));
    launch(head_wgrad, (HEAD_OUTS + 127) / 128, 128, 0, st, dy, (const uint16_t*)(k + G.dh16),
                                                        (const uint16_t*)(w + L.h16),
                                                        (const uint16_t*)(w + L.g16), B, grads[8],
                                                        grads[9], grads[10], grads[11]);
    if (!wgrad(d, w + L.p3, k + G.dA4, grads[6], grads[7], B, H / 8, W / 8, st) ||
        !conv<EP_EXPAND, true>(d, k + G.dA4, c4w, nullptr, k + G.dA3, w + L.m3, B, H / 8, W / 8, st) ||
        !wgrad(d, w + L.p2, k + G.dA3, grads[4], grads[5], B, H / 4, W / 4, st) ||
        !conv<EP_EXPAND, true>(d, k + G.dA3, c3w, nullptr, k + G.dA2, w + L.m2, B, H / 4, W / 4, st) ||
        !wgrad(d, w + L.p1, k + G.dA2, grads[2], grads[3], B, H / 2, W / 2, st) ||
        !conv<EP_PLAIN, true>(d, k + G.dA2, c2w, nullptr, k + G.dp1, nullptr, B, H / 2, W / 2, st))
        return LGM_ERR_CUDA;
    const int grid1 = (int)std::min<long long>(((long long)B * (H / 2) + 7) / 8, d.sms * 4ll);
    launch(wgrad1_planes, grid1, 256, 0, st, (const uint32_t*)x, (const uint16_t*)(k + G.dp1),
                                         (const uint4*)(w + L.m1), grads[0], grads[1], B, H, W);
    return cudaGetLastError() == cudaSuccess ? LGM_OK : LGM_ERR_CUDA;
}

}  // extern "C"
