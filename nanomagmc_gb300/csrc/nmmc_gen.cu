// Learned warm start: a conditional convolutional generator for 2-D Heisenberg lattices.
//
// No reference counterpart. The plain sampler produces equilibrium snapshots x at points
// c = (T, B, D); the network learns to denoise y = normalise(sqrt(1-s^2) x + s g) (g standard
// normal per site and component, s the noise level; at s = 1, y is a uniform random start)
// back to x. A warm start runs a few denoising steps from a random start and hands the
// result to the Metropolis chain, which does all sampling.
//
// Network: 8 periodic 3x3 convolutions, 48 channels, ReLU between layers. Input channels:
// y (3), T/1.5, B, D/0.8, s, 0. Output: 3 channels v, spin = v/|v|. Loss: mean over sites of
// |v/|v| - x|^2. Weights and activations are stored in BF16, every product is accumulated in
// FP32; gradients, biases, master weights and the Adam moments are FP32.
//
// Layouts: activations NHWC [image][y][x][channel]; weights [tap = 3*(dy+1)+(dx+1)][cin][cout].
#include <cuda_bf16.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <vector>

#include "nmmc_kernels.cuh"

namespace nmmc {

constexpr int kGenC = 48;        // hidden channels
constexpr int kGenLayers = 8;
constexpr int kGenCin0 = 8;      // 3 spin + 4 condition + 1 zero
constexpr int kGenCout = 4;      // 3 spin components + 1 zero (vector loads)
constexpr int kWimgBytes = 9 * (kGenC / 8) * (kGenC / 8) * 128;   // largest layer weight image (48 -> 48)
constexpr int kTile = 16;        // pixel tile edge of the convolution kernels

__device__ __forceinline__ __nv_bfloat16 ld_seq(const __nv_bfloat16* p) {
    unsigned short v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return __ushort_as_bfloat16(v);
}

// Activations and gradients are stored chunk-planar: C channels of element type T as
// [image][C / epc][L*L pixels][epc], epc = 16 / sizeof(T) (8 BF16 or 4 FP32 channels per
// 16-byte chunk), so that a chunk of consecutive pixels of a row is contiguous: one bulk copy
// per (row, chunk) of a convolution window and coalesced stores. A tensor of a single chunk
// (the 8-channel input, the 4-channel output and its gradient) is plain [pixel][C].
template <typename T>
__host__ __device__ constexpr int epc() { return 16 / (int)sizeof(T); }
// element offset of channel c of pixel pp (y*L + x) of image img
template <typename T>
__host__ __device__ __forceinline__ size_t pl_off(int C, size_t LL, size_t img, size_t pp, int c) {
    return ((img * (size_t)(C / epc<T>()) + (size_t)(c / epc<T>())) * LL + pp) * (size_t)epc<T>() + (size_t)(c % epc<T>());
}

struct GenLayer {
    int cin = 0, cout = 0;           // cout padded to kGenCout for the last layer
    float* w = nullptr;              // FP32 master [9][cin][cout]
    float* b = nullptr;              // [cout]
    __nv_bfloat16* wb = nullptr;     // BF16 compute copy [9][cin][cout]
    __nv_bfloat16* wt = nullptr;     // BF16 flipped transpose [9][cout][cin] (data gradient)
    uint8_t* wimg = nullptr;         // BF16 weights in the tensor-core B layout (tc::place)
                                     // (kWimgBytes), staged by one bulk copy per CTA
    uint8_t* wtimg = nullptr;        // hidden layers: wt as TF32 in that layout (2 kWimgBytes)
    int kch = 0;                     // 16-byte chunks of K per tap in wimg
    float* gw = nullptr;
    float* gb = nullptr;
    float* mw = nullptr;
    float* vw = nullptr;
    float* mb = nullptr;
    float* vb = nullptr;
    size_t nw() const { return (size_t)9 * cin * cout; }
};

}  // namespace nmmc

struct nmmc_gen {
    int L = 0;
    uint64_t seed = 0;
    cudaStream_t stream = nullptr;
    nmmc::GenLayer layer[nmmc::kGenLayers];
    // dataset
    int cap = 0, count = 0;
    __nv_bfloat16* snaps = nullptr;  // [cap][L][L][3]
    float* cond = nullptr;           // [cap][3]
    // batch workspace
    int bcap = 0;
    __nv_bfloat16* act[nmmc::kGenLayers] = {};   // act[0] input (8 ch); act[l] output of layer l-1,
                                                 // [b][6][L][L][8] (chunk-planar)
    float* vout = nullptr;           // [b][L][L][4] linear output of the last layer
    float* target = nullptr;         // [b][L][L][4]
    float* g0 = nullptr;             // gradient ping-pong [b][12][L][L][4] (chunk-planar)
    float* g1 = nullptr;
    float* gv = nullptr;             // [b][L][L][4]
    float* grads = nullptr;          // every layer's gw and gb, in parameter order
    float* wpart = nullptr;          // weight-gradient partials
    size_t wpart_cap = 0;
    int* d_idx = nullptr;            // snapshot index per batch item
    float* d_sig = nullptr;          // noise level per batch item
    float* d_cnd = nullptr;          // condition per batch item (3)
    double* d_loss = nullptr;
    int* d_flag = nullptr;           // device error word (4: a tensor-core wait gave up)
    int use_tc = 1;                  // hidden layers on tcgen05 (NMMC_GEN_OPT_TENSOR_CORES)
    int use_ws = 0;                  // warp-specialised tcgen05 kernel for the BF16 modes (opt-in)
    int use_rows = 1;                // L = 128: the row-ring kernels (0: cp.async staging)
    int schedule = 0;                // warm-start noise levels: 0 linear, 1 quadratic, 2 cosine
    int use_wimg = 1;                // the tensor-core kernels stage the weights by one bulk copy of
                                     // their image (0: the threads rearrange the BF16 weights)
    int sm_count = 0;
    int smem_per_sm = 0;             // shared memory per SM of the generator's device
    std::map<const void*, int> attr_smem;   // dynamic shared memory set per kernel on that device
    long long adam_t = 0;
    unsigned long long draws = 0;    // Philox counter for noise
};

namespace nmmc {

// ------------------------------------------------------------------------------------------
// Convolution (forward and data gradient share it): out[p, co] = sum_{tap, ci} in[p + tap, ci] *
// W[tap][ci][co] (+ bias), periodic in x and y. One CTA = one 16x16 pixel tile of one image;
// 256 threads = 128 pixel pairs (rows y and y+8) x 2 halves of the output channels.
// EPI 0: ReLU, BF16 out.  EPI 1: linear, FP32 out.  EPI 2: times (mask > 0), FP32 out.
// ------------------------------------------------------------------------------------------
template <int CIN, int COUT, typename TIN, int EPI>
__global__ void __launch_bounds__(256)
k_gen_conv(const TIN* in, const __nv_bfloat16* w, const float* bias,
           const __nv_bfloat16* mask, int mask_c, void* out, int L) {
    seq_begin();
    extern __shared__ __align__(16) float gsm[];
    constexpr int HALF = (COUT + 1) / 2;          // output channels per thread
    constexpr int T2 = kTile + 2;
    float* wsm = gsm;                              // [9][CIN][COUT]
    float* tsm = gsm + 9 * CIN * COUT;             // [CIN][T2][T2]
    const int img = blockIdx.z;
    const int ty0 = blockIdx.y * kTile, tx0 = blockIdx.x * kTile;
    // weights and the wrapped input tile through 16-byte loads, several in flight per thread
    // (weight arrays and pixel rows are 16-byte multiples and the buffers 16-byte aligned)
    static_assert((9 * CIN * COUT) % 8 == 0 && (CIN * sizeof(TIN)) % 16 == 0, "16-byte staging");
#pragma unroll 4
    for (int i = threadIdx.x; i < 9 * CIN * COUT / 8; i += blockDim.x) {
        const uint4 q = ld_seq(reinterpret_cast<const uint4*>(w) + i);
        const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&q);
        float4* d = reinterpret_cast<float4*>(wsm + 8 * i);
        d[0] = make_float4(__bfloat162float(e[0]), __bfloat162float(e[1]), __bfloat162float(e[2]), __bfloat162float(e[3]));
        d[1] = make_float4(__bfloat162float(e[4]), __bfloat162float(e[5]), __bfloat162float(e[6]), __bfloat162float(e[7]));
    }
    const size_t LL = (size_t)L * L, ibase = (size_t)img * LL;
    constexpr int EPV = epc<TIN>(), V = CIN / EPV;   // elements per load, chunks per pixel
    const uint4* src = reinterpret_cast<const uint4*>(in + ibase * CIN);   // this image's chunk planes
#pragma unroll 4
    for (int i = threadIdx.x; i < T2 * T2 * V; i += blockDim.x) {   // x fastest: coalesced rows
        const int v = i / (T2 * T2), r = i - v * T2 * T2, yy = r / T2, xx = r - yy * T2;
        int gy = ty0 + yy - 1, gx = tx0 + xx - 1;   // in [-1, L]: one wrap
        gy += (gy < 0) ? L : ((gy >= L) ? -L : 0);
        gx += (gx < 0) ? L : ((gx >= L) ? -L : 0);
        const uint4 q = ld_seq(src + (size_t)v * LL + (size_t)gy * L + gx);
        const TIN* e = reinterpret_cast<const TIN*>(&q);
#pragma unroll
        for (int k = 0; k < EPV; ++k) tsm[((v * EPV + k) * T2 + yy) * T2 + xx] = (float)e[k];
    }
    __syncthreads();
    const int pair = threadIdx.x & 127, half = threadIdx.x >> 7;
    const int px = pair & 15, py = pair >> 4;      // rows py and py + 8
    const int co0 = half * HALF;
    static_assert(HALF % 2 == 0 && COUT == 2 * HALF, "channel pairs");
    // the mask of both pixels arrives during the sums
    constexpr bool kWide = EPI == 2 && HALF % 8 == 0;   // whole 16-byte chunks
    uint4 m4[kWide ? 2 : 1][kWide ? HALF / 8 : 1];
    if constexpr (kWide)
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int c = 0; c < HALF / 8; ++c)
                m4[r][c] = ld_seq(reinterpret_cast<const uint4*>(
                    mask + pl_off<__nv_bfloat16>(mask_c, LL, img, (size_t)(ty0 + py + 8 * r) * L + tx0 + px, co0 + 8 * c)));
    f2 a0[HALF / 2], a1[HALF / 2];   // channel pairs: packed multiply-adds
#pragma unroll
    for (int k = 0; k < HALF / 2; ++k) {
        a0[k] = bias ? pk(ld_seq(bias + co0 + 2 * k), ld_seq(bias + co0 + 2 * k + 1)) : f2{0ull};
        a1[k] = a0[k];
    }
#pragma unroll 1
    for (int tap = 0; tap < 9; ++tap) {
        const int dy = tap / 3, dx = tap - 3 * (tap / 3);
#pragma unroll 4
        for (int ci = 0; ci < CIN; ++ci) {
            const float x0 = tsm[(ci * T2 + py + dy) * T2 + px + dx];
            const float x1 = tsm[(ci * T2 + py + 8 + dy) * T2 + px + dx];
            const f2 p0 = pk(x0, x0), p1 = pk(x1, x1);
            const float* wr = wsm + (tap * CIN + ci) * COUT + co0;
            if constexpr (HALF % 4 == 0) {   // two channel pairs per load
#pragma unroll
                for (int k = 0; k < HALF / 2; k += 2) {
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(wr + 2 * k);
                    a0[k] = fma2(p0, f2{q.x}, a0[k]);
                    a1[k] = fma2(p1, f2{q.x}, a1[k]);
                    a0[k + 1] = fma2(p0, f2{q.y}, a0[k + 1]);
                    a1[k + 1] = fma2(p1, f2{q.y}, a1[k + 1]);
                }
            } else {
#pragma unroll
                for (int k = 0; k < HALF / 2; ++k) {
                    const f2 wv{*reinterpret_cast<const unsigned long long*>(wr + 2 * k)};
                    a0[k] = fma2(p0, wv, a0[k]);
                    a1[k] = fma2(p1, wv, a1[k]);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int y = ty0 + py + 8 * r, x = tx0 + px;
        const size_t pp = (size_t)y * L + x;
        float v[HALF];
#pragma unroll
        for (int k = 0; k < HALF / 2; ++k) {
            v[2 * k] = lo(r ? a1[k] : a0[k]);
            v[2 * k + 1] = hi(r ? a1[k] : a0[k]);
        }
        if constexpr (EPI == 0 && HALF % 8 == 0) {   // whole 16-byte chunks
#pragma unroll
            for (int c = 0; c < HALF / 8; ++c) {
                uint32_t q[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const __nv_bfloat162 h = __floats2bfloat162_rn(fmaxf(v[8 * c + 2 * k], 0.0f), fmaxf(v[8 * c + 2 * k + 1], 0.0f));
                    q[k] = *reinterpret_cast<const uint32_t*>(&h);
                }
                *reinterpret_cast<uint4*>((__nv_bfloat16*)out + pl_off<__nv_bfloat16>(COUT, LL, img, pp, co0 + 8 * c)) =
                    make_uint4(q[0], q[1], q[2], q[3]);
            }
            continue;
        }
        if constexpr (kWide) {
#pragma unroll
            for (int c = 0; c < HALF / 8; ++c) {
                const __nv_bfloat16* mh = reinterpret_cast<const __nv_bfloat16*>(&m4[r][c]);
                float o[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) o[k] = __bfloat162float(mh[k]) > 0.0f ? v[8 * c + k] : 0.0f;
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    *reinterpret_cast<float4*>((float*)out + pl_off<float>(COUT, LL, img, pp, co0 + 8 * c + 4 * q)) =
                        make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
            }
            continue;
        }
#pragma unroll
        for (int k = 0; k < HALF; ++k) {
            const int co = co0 + k;
            if (EPI == 0) {
                ((__nv_bfloat16*)out)[pl_off<__nv_bfloat16>(COUT, LL, img, pp, co)] = __float2bfloat16(fmaxf(v[k], 0.0f));
            } else if (EPI == 1) {
                ((float*)out)[pl_off<float>(COUT, LL, img, pp, co)] = v[k];
            } else {
                const float mk = __bfloat162float(mask[pl_off<__nv_bfloat16>(mask_c, LL, img, pp, co)]);
                ((float*)out)[pl_off<float>(COUT, LL, img, pp, co)] = mk > 0.0f ? v[k] : 0.0f;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// Hidden-layer convolutions (48 -> 48 channels) on the 5th-generation tensor cores, as an
// implicit GEMM over the periodically padded image: with rows of pitch L+2 (one wrapped
// column each side), output position P of the padded grid is sum_tap in[P + off_tap] W_tap,
// off_tap = (dy-1)(L+2) + (dx-1), so every tap is one shifted window of the same staged
// data. A tile is 128 consecutive padded positions of rows 1..L (one TMEM lane each; halo
// positions are computed and dropped), N = 48 output channels (FP32 TMEM columns), K = 9 taps
// x 48 input channels, 32 bytes of K per MMA.
//
//   MODE 0 (forward):  BF16 activations, tcgen05.mma kind::f16; bias + ReLU, BF16 out.
//   MODE 1 (probe):    as 0 with bias only and FP32 out.
//   MODE 2 (data gradient): FP32 gradients as TF32 operands (kind::tf32) with the flipped,
//                      transposed weights; out = result x (activation > 0), FP32.
//
// Shared-memory operands use the K-major layout without swizzling, 8-row x 16-byte core
// matrices. The staged input window (W = 128 + 2(L+3) padded positions, wrapped while
// loading) is stored chunk-major: the 16-byte atom of chunk c (8 BF16 or 4 FP32 channels) of
// window position w at (c*W + w)*16, so a core matrix is 8 consecutive positions (stride byte
// offset 128 B), the next chunk is W*16 B further (leading byte offset), and a tap's window
// starts 16 B per position of its offset later. The layer's weights are staged once per CTA
// (persistent CTAs). One thread issues the MMAs of a tile and commits them to an mbarrier;
// after a bounded wait, each warp reads its 32 TMEM lanes (tcgen05.ld) for the epilogue.
// ------------------------------------------------------------------------------------------
namespace tc {
constexpr int kM = 128;                         // padded positions per tile = TMEM lanes
constexpr int kC = 48;                          // channels in and out
constexpr int kCore = 128;                      // bytes per core matrix
constexpr int kTmemCols = 64;                   // power of two >= 48
constexpr unsigned kWaitLimit = 1u << 26;

template <int MODE>
struct Traits {
    using TA = __nv_bfloat16;                   // operand element type
    static constexpr int kEpc = 8;              // elements per 16-byte chunk
    static constexpr uint32_t kFmt = 1;         // BF16
};
template <>
struct Traits<2> {
    using TA = float;
    static constexpr int kEpc = 4;
    static constexpr uint32_t kFmt = 2;         // TF32
};
// place of tap 3 (dy + 1) + dx + 1 among the weights: by dx, then dy descending, so that the three
// taps of a dx are, in the row-ring kernel, the columns of the output rows r-1, r, r+1
__host__ __device__ constexpr int place(int tap) { return tap % 3 * 3 + 2 - tap / 3; }
template <int MODE>
__host__ __device__ constexpr int chunks() { return kC / Traits<MODE>::kEpc; }        // 6 (BF16) or 12 (TF32)
template <int MODE>
__host__ __device__ constexpr int btap() { return (kC / 8) * chunks<MODE>() * kCore; } // weight bytes per tap
// instruction descriptor: D F32 (bits 4-5 = 1), A and B format (bits 7-9, 10-12), both
// K-major (bits 15, 16 = 0), N >> 3 at bits 17-22, M >> 4 at bits 24-28
template <int MODE, int N = kC, int M = kM>
__host__ __device__ constexpr uint32_t idesc() {
    return (1u << 4) | (Traits<MODE>::kFmt << 7) | (Traits<MODE>::kFmt << 10) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}
// the same for a number of columns n known at run time
template <int MODE>
__device__ __forceinline__ uint32_t idesc_n(uint32_t n) {
    return (1u << 4) | (Traits<MODE>::kFmt << 7) | (Traits<MODE>::kFmt << 10) | ((n >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
}
__host__ __device__ constexpr int window(int L) { return kM + 2 * (L + 3); }
template <int MODE>
__host__ __device__ constexpr int smem_bytes(int L) { return 9 * btap<MODE>() + chunks<MODE>() * window(L) * 16 + 1024; }
constexpr int kSmemMax = 232448;                // dynamic shared memory per block (227 KB)
}  // namespace tc

__device__ __forceinline__ uint32_t gen_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: start address, leading and stride byte offsets (all >> 4),
// descriptor version 1 (bit 46), no swizzle (bits 61-63 = 0).
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ bool gen_mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait for phase `parity` of `bar`; gives up (abort word and error flag `code` set) after
// the limit or as soon as another role has given up.
__device__ __forceinline__ bool gen_wait(uint32_t bar, uint32_t parity, volatile int* abort, int* flag, int code) {
    for (unsigned it = 0; it < tc::kWaitLimit; ++it) {
        if (gen_mbar_try_wait(bar, parity)) return true;
        if (*abort) return false;
    }
    *abort = 1;
    atomicExch(flag, code);
    return false;
}

// The same for two barriers, polled together (one after the other, a wait for a phase that is already
// complete takes 100 cycles each).
__device__ __forceinline__ bool gen_wait2(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1, volatile int* abort,
                                          int* flag, int code) {
    for (unsigned it = 0; it < tc::kWaitLimit; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4;\n\t"
            "and.pred p, p, q;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar0), "r"(parity0), "r"(bar1), "r"(parity1)
            : "memory");
        if (ok) return true;
        if (*abort) return false;
    }
    *abort = 1;
    atomicExch(flag, code);
    return false;
}

__device__ __forceinline__ void gen_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void gen_mbar_init(void* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(gen_smem_u32(bar)), "r"(count) : "memory");
}
// barrier 1 for `threads` of the block's threads
__device__ __forceinline__ void gen_bar_sync(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

// an arrival on `bar` when the MMAs issued so far by this thread have completed
__device__ __forceinline__ void gen_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 consecutive FP32 columns of this thread's TMEM lane <- 0 (before a wait::st)
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(
            taddr),
        "r"(0)
        : "memory");
}

// Weights w[tap][k][n] (BF16, 16-byte aligned) -> B_tap[n][k] as K-major core matrices in
// shared memory. One 16-byte load brings 8 consecutive n (48 is a multiple of 8) and the loop
// is unrolled so that several loads are in flight per thread; element by element, the loads
// would each wait for the previous store.
template <int MODE, bool ROWS = false>
__device__ __forceinline__ void stage_weights(uint8_t* sB, const __nv_bfloat16* __restrict__ w, int tid, int nthr) {
    using TA = typename tc::Traits<MODE>::TA;
    constexpr int kEpc = tc::Traits<MODE>::kEpc, kCh = tc::chunks<MODE>(), kBT = tc::btap<MODE>();
    constexpr int kC = tc::kC, kG = 9 * kC * kC / 8;
#pragma unroll 7
    for (int g8 = tid; g8 < kG; g8 += nthr) {
        const uint4 v = ld_seq(reinterpret_cast<const uint4*>(w) + g8);
        const int i = g8 * 8;
        const int tap = i / (kC * kC), r = i - tap * kC * kC, k = r / kC, n = r - k * kC;
        uint8_t* base = sB + (ROWS ? tc::place(tap) : tap) * kBT + ((n >> 3) * kCh + k / kEpc) * tc::kCore + (k % kEpc) * (int)sizeof(TA);
        const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&v);
#pragma unroll
        for (int q = 0; q < 8; ++q) *(TA*)(base + q * 16) = (TA)e[q];
    }
}

// The mask of one output position (MODE 2): all loads before the first store, which they could
// not pass (one by one a data gradient of 16 x 128^2 took 85 us instead of 55).
template <int MODE>
__device__ __forceinline__ void load_mask(uint4* m4, const __nv_bfloat16* __restrict__ mask, size_t img, size_t pp, size_t LL) {
    if (MODE == 2) {
        const uint4* mk = reinterpret_cast<const uint4*>(mask + img * LL * tc::kC) + pp;
#pragma unroll
        for (int c = 0; c < tc::kC / 8; ++c) m4[c] = ld_seq(mk + (size_t)c * LL);
    }
}

// Epilogue of one output position of a tensor-core convolution: v[48] FP32 accumulators of
// pixel pp (y*L + x) of image img, written chunk-planar (16 bytes per chunk, consecutive
// pixels of a warp contiguous). MODE 0: bias + ReLU, BF16. MODE 1: bias, FP32. MODE 2:
// times (mask > 0) with the mask the layer's BF16 activation (m4, load_mask), FP32.
template <int MODE>
__device__ __forceinline__ void conv_store(const float* v, const float* sbias, void* out_v,
                                           const uint4* m4, size_t img, size_t pp, size_t LL) {
    constexpr int kC = tc::kC;
    if (MODE == 0) {
        uint4* dst = reinterpret_cast<uint4*>((__nv_bfloat16*)out_v + img * LL * kC) + pp;
#pragma unroll
        for (int c = 0; c < kC / 8; ++c) {
            uint32_t h[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const __nv_bfloat162 b2 = __floats2bfloat162_rn(fmaxf(v[8 * c + 2 * q] + sbias[8 * c + 2 * q], 0.0f),
                                                                fmaxf(v[8 * c + 2 * q + 1] + sbias[8 * c + 2 * q + 1], 0.0f));
                h[q] = *(const uint32_t*)&b2;
            }
            dst[(size_t)c * LL] = make_uint4(h[0], h[1], h[2], h[3]);
        }
    } else if (MODE == 1) {
        float4* dst = reinterpret_cast<float4*>((float*)out_v + img * LL * kC) + pp;
#pragma unroll
        for (int c = 0; c < kC / 4; ++c)
            dst[(size_t)c * LL] = make_float4(v[4 * c] + sbias[4 * c], v[4 * c + 1] + sbias[4 * c + 1],
                                              v[4 * c + 2] + sbias[4 * c + 2], v[4 * c + 3] + sbias[4 * c + 3]);
    } else {
        float4* dst = reinterpret_cast<float4*>((float*)out_v + img * LL * kC) + pp;
#pragma unroll
        for (int c = 0; c < kC / 8; ++c) {
            const __nv_bfloat16* mh = reinterpret_cast<const __nv_bfloat16*>(&m4[c]);
            float o[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) o[k] = (__bfloat162float(mh[k]) > 0.0f) ? v[8 * c + k] : 0.0f;
            dst[(size_t)(2 * c) * LL] = make_float4(o[0], o[1], o[2], o[3]);
            dst[(size_t)(2 * c + 1) * LL] = make_float4(o[4], o[5], o[6], o[7]);
        }
    }
}

template <int MODE, int N = tc::kC>
__device__ __forceinline__ void tc_mma(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t acc) {
    if (MODE == 2)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(tc::idesc<MODE, N>()), "r"(acc)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(tc::idesc<MODE, N>()), "r"(acc)
            : "memory");
}

// The same, always accumulating, with the instruction descriptor as a value and the operand
// descriptors in halves (only the low one, with the start address, changes), so that little but the
// MMA itself is issued: one of N = 144 takes 74 cycles, and with the descriptors computed per MMA
// in one lane's branch the issue took 130.
template <int MODE>
__device__ __forceinline__ void tc_mma_n(uint32_t tmem, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi, uint32_t idesc) {
    if (MODE == 2)
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, 1, 0;\n\t"
            "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], a, b, %5, p;\n\t}" ::"r"(tmem),
            "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, 1, 0;\n\t"
            "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}" ::"r"(tmem),
            "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc)
            : "memory");
}

// one lane of a warp that is together, known as such to the compiler (unlike lane == 0)
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}

// Per tile: stage the window, issue the MMAs, wait for their commit, run the epilogue; two
// CTAs per SM overlap one another's phases. (Measured on GB300: a double-buffered variant with
// two accumulators, which fits one CTA per SM, and issuing the next tile's loads before the
// epilogue were both slower.) With the weights rearranged by the threads of every CTA a hidden layer
// of 16 x 64^2 took 18.8 us, with their image 10.8 (a warm start of 8 passes there 1369 and 921 us).
template <int MODE>
__global__ void __launch_bounds__(128, 2)
k_gen_conv_tc(const typename tc::Traits<MODE>::TA* in, const __nv_bfloat16* w, const uint8_t* wimg,
              const float* bias, const __nv_bfloat16* mask, void* out_v,
              int L, int tiles_per_img, int ntiles, int* flag) {
    seq_begin();
    using namespace tc;
    using TA = typename Traits<MODE>::TA;
    constexpr int kCh = chunks<MODE>();
    constexpr int kBT = btap<MODE>();
    constexpr int kRound = 96 / kCh;            // window positions per loader round (96 threads)
    extern __shared__ uint8_t tsm_raw[];
    __shared__ __align__(8) unsigned long long mbar, wbar;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) float sbias[kC];
    uint8_t* sB = (uint8_t*)(((uintptr_t)tsm_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sA = sB + 9 * kBT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int P = L + 2;                      // padded row pitch
    const int W = window(L);                  // staged window positions
    const int npad = P * P;

    // weights w[tap][k][n] (k: input channel of this convolution) -> B_tap[n][k], K-major: their image by
    // one bulk copy, which lands while the first window does, or rearranged by the threads
    if (!wimg) stage_weights<MODE, true>(sB, w, tid, blockDim.x);
    if (tid < kC) sbias[tid] = (MODE == 2) ? 0.0f : ld_seq(bias + tid);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gen_smem_u32(&tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        gen_mbar_init(&mbar, 1);
        gen_mbar_init(&wbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (wimg) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(gen_smem_u32(&wbar)), "r"(9u * kBT)
                         : "memory");
            gen_bulk(gen_smem_u32(sB), wimg, 9u * kBT, gen_smem_u32(&wbar));
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const uint32_t aBase = gen_smem_u32(sA), bBase = gen_smem_u32(sB);

    // staged window of tile t into buffer buf: padded position w0 + j, wrapped onto the image;
    // outside the padded grid (only read by dropped halo outputs) zero. cp.async: every copy
    // of a thread is in flight at once. Threads 0..95 = kRound positions x kCh chunks per
    // round; a thread's padded row and column advance by kRound per round (P >= kRound).
    auto load_window = [&](int t) {
        const int img = t / tiles_per_img;
        const int w0 = (t - img * tiles_per_img) * kM - 1;        // q0 - (P + 1), q0 = P + tile*kM
        const TA* src_img = in + (size_t)img * L * L * kC;
        if (tid < kRound * kCh) {
            const int c = tid % kCh;
            int j = tid / kCh, pos = w0 + j;
            int py = (pos >= 0) ? pos / P : -1;
            int px = pos - py * P;
            const uint32_t dst0 = aBase + (uint32_t)(c * W * 16);
            for (; j < W; j += kRound, pos += kRound) {
                const bool inside = pos >= 0 && pos < npad;
                const uint4* src = (const uint4*)src_img;
                if (inside) {
                    int y = py - 1, x = px - 1;
                    y += (y < 0) ? L : ((y >= L) ? -L : 0);
                    x += (x < 0) ? L : ((x >= L) ? -L : 0);
                    src = (const uint4*)src_img + ((size_t)c * L * L + (size_t)y * L + x);   // chunk plane c
                }
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst0 + (uint32_t)(j * 16)), "l"(src),
                             "r"(inside ? 16 : 0)
                             : "memory");
                px += kRound;
                if (px >= P) {
                    px -= P;
                    ++py;
                }
            }
        }
    };
    // the 9 x kCh/2 MMAs of a tile (thread 0), committed to the mbarrier
    auto issue_mmas = [&]() {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a0 = aBase, d = tmem;
#pragma unroll 1
        for (int tap = 0; tap < 9; ++tap) {
            const int shift = (P + 1) + (tap / 3 - 1) * P + (tap % 3 - 1);   // window slot of output 0
#pragma unroll
            for (int ks = 0; ks < kCh / 2; ++ks) {
                const uint64_t ad = umma_desc(a0 + (uint32_t)((2 * ks * W + shift) * 16), (uint32_t)(W * 16), 128);
                const uint64_t bd = umma_desc(bBase + place(tap) * kBT + 2 * ks * kCore, kCore, kCh * kCore);
                tc_mma<MODE>(d, ad, bd, (tap | ks) ? 1u : 0u);
            }
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         gen_smem_u32(&mbar))
                     : "memory");
    };
    // epilogue of tile t: warp w holds positions q0 + 32w .. in TMEM lanes 32w ..
    auto epilogue = [&](int t) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int img = t / tiles_per_img;
        const int q0 = P + (t - img * tiles_per_img) * kM;
        float v[kC];
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
        tmem_ld16(taddr + 0, v);
        tmem_ld16(taddr + 16, v + 16);
        tmem_ld16(taddr + 32, v + 32);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const int pos = q0 + warp * 32 + lane, py = pos / P, px = pos - py * P;
        if (py >= 1 && py <= L && px >= 1 && px <= L) {
            uint4 m4[kC / 8];
            load_mask<MODE>(m4, mask, (size_t)img, (size_t)(py - 1) * L + (px - 1), (size_t)L * L);
            conv_store<MODE>(v, sbias, out_v, m4, (size_t)img, (size_t)(py - 1) * L + (px - 1), (size_t)L * L);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    };
    // bounded wait for the commit; false (and the error word set) on timeout
    uint32_t phase = 0;
    const uint32_t bar = gen_smem_u32(&mbar);
    auto wait_mmas = [&]() -> bool {
        bool done = false;
        for (unsigned it = 0; it < kWaitLimit && !done; ++it) done = gen_mbar_try_wait(bar, phase);
        if (__syncthreads_or(!done)) {
            if (tid == 0) atomicExch(flag, 4);
            return false;
        }
        phase ^= 1u;
        return true;
    };

    auto weights_in = [&]() -> bool {   // bounded wait for the weight image
        bool done = !wimg;
        for (unsigned it = 0; it < kWaitLimit && !done; ++it) done = gen_mbar_try_wait(gen_smem_u32(&wbar), 0);
        return done;
    };

    const int first = blockIdx.x, stride = gridDim.x;
    const int n = (ntiles > first) ? (ntiles - first + stride - 1) / stride : 0;   // tiles of this CTA
    bool failed = false;
    for (int k = 0; k < n; ++k) {
        load_window(first + k * stride);
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0 && (k > 0 || weights_in())) issue_mmas();
        if (!wait_mmas()) {
            failed = true;
            break;
        }
        epilogue(first + k * stride);
        __syncthreads();
    }
    if (failed) {   // give in-flight MMAs a bounded chance to land before the TMEM is freed
        bool done = false;
        for (unsigned it = 0; it < kWaitLimit && !done; ++it) done = gen_mbar_try_wait(bar, phase);
        if (tid == 0) weights_in();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

// Every convolution of the generator at L = 128 (the configured size), warp-specialised, one CTA
// per SM. The CTAs take equal runs of consecutive rows of the batch; an input row (128 positions =
// the 128 TMEM lanes) is copied once and used once: for each x shift one MMA multiplies it by the
// weights of the three vertical taps side by side, N = 3 x 48 columns, into the accumulators of
// the output rows r-1, r, r+1, which are neighbours in a ring of kAcc accumulators in tensor
// memory (two MMAs where the three wrap around the ring's end). An output row is finished when the
// row below it has been multiplied. The order of the taps in a sum is that of the other forms.
// A row buffer holds KCH blocks (one per 16-byte channel chunk) of 130 slots (x = -1 .. 128); a
// row of a chunk plane is 2048 contiguous bytes, one cp.async.bulk. (A bulk copy takes about 100
// cycles to issue, whatever its size, so the periodic neighbours x = 127 and x = 0 are copied
// within shared memory: as two more bulk copies per chunk they bounded the kernel.)
//   warps 0-7: epilogue, two groups of four: group g takes the tiles k = g mod 2, its warp w the
//              TMEM lanes 32 (w & 3) ..; the data gradient's mask is loaded before the wait for
//              the accumulator, so it arrives during the MMAs;
//   warp 8:    producer: after empty[slot], the byte count of raw[slot] and the row's copies;
//   warp 10:   after raw[slot], slots 0 and 129 of the blocks, then full[slot];
//   warp 9:    after full of the next row and tempty of the accumulator it begins, 3 x KCH/2
//              MMAs, committed to empty of the row and tfull of the finished accumulator. The
//              warp stays together (uniform descriptors), lane 0 issues.
// Every MMA accumulates: the epilogue clears an accumulator that it has read.
// Every wait is bounded and ends when another role gave up (a shared abort word); before the
// tensor memory is freed the last copies have landed and a last commit has been waited for.
// What bounds it: an MMA of M = 128 and K = 32 bytes reads A and B from shared memory, 45 cycles for
// N = 48 and 74 for N = 144, so one per tap (27 in BF16, 54 in TF32 per row) costs nearly twice
// what 9 or 18 wide ones do; beside that the start of a CTA (about 5 us) and, for the data
// gradient, memory. 16 x 128^2: hidden forward layer 14.2 us, data gradient 21.0 us, first layer
// 10.2 us, last 12.7 us; single-role CTAs with windows of four rows and one MMA per tap took
// 18.5, 55, 12 and 17 us. 50 MB and 126 MB at the copy rate are 7.4 and 18.5 us.
//   MODE 0: bias + ReLU, BF16 out (48 channels);  MODE 1: bias, FP32 out (48 channels);
//   MODE 2: TF32 data gradient, times (activation > 0), FP32 out;
//   MODE 3: bias, FP32 out of CO = 4 channels [pixel][4] (the generator's last layer).
// ICH input chunks (16 bytes of channels each) come in by bulk copies; the K of one tap is KCH
// chunks (KCH - ICH zero blocks when a layer's inputs do not fill an MMA's K: the first layer's
// 8 BF16 channels are one chunk of the two of K = 16); N = CO output channels rounded up to 16.
// With wimg the weights arrive by one bulk copy of their tensor-core image (k_gen_update) instead
// of being rearranged by the threads.
namespace row {
constexpr int kSlots = 130;                   // x = -1 .. 128
constexpr int kBlk = 2176;                    // bytes per (row, chunk) block: 130 x 16 B, 128-B aligned
constexpr int kAcc = 10;                      // accumulators: 480 of 512 TMEM columns
static_assert(kAcc < 15, "one lane per barrier");
constexpr int kEpi = 8;                       // epilogue warps
constexpr int kThreads = (kEpi + 3) * 32;
// MMA N for co output channels: M = 128 takes N in multiples of 16
__host__ __device__ constexpr int nmma(int co) { return (co + 15) / 16 * 16; }
template <int CO>
__host__ __device__ constexpr int cols() { return kAcc * nmma(CO) <= 256 ? 256 : 512; }   // TMEM columns allocated
template <int KCH, int CO>
__host__ __device__ constexpr int btap() { return (nmma(CO) / 8) * KCH * tc::kCore; }   // B bytes per tap
// row buffers: what fits beside the weights, eight at most (the data gradient: five)
template <int KCH, int CO>
__host__ __device__ constexpr int ring() {
    const int fit = (tc::kSmemMax - 1024 - 9 * btap<KCH, CO>()) / (KCH * kBlk);
    return fit < 8 ? fit : 8;
}
template <int KCH, int CO>
__host__ __device__ constexpr int smem_bytes() { return 9 * btap<KCH, CO>() + ring<KCH, CO>() * KCH * kBlk + 1024; }
}  // namespace row

template <int MODE, int ICH, int KCH, int CO>
__global__ void __launch_bounds__(row::kThreads, 1)
k_gen_conv_row(const typename tc::Traits<MODE>::TA* in, const __nv_bfloat16* w,
               const uint8_t* wimg, const float* bias,
               const __nv_bfloat16* mask, void* out_v, int nrows, int* flag) {
    seq_begin();
    using namespace tc;
    using TA = typename Traits<MODE>::TA;
    constexpr int kEpc = Traits<MODE>::kEpc;
    constexpr int NN = row::nmma(CO);
    constexpr int CI = ICH * kEpc;                           // real input channels
    constexpr int kBT = row::btap<KCH, CO>();
    constexpr int kS = row::ring<KCH, CO>();
    constexpr int kL = kM;                                   // lattice edge of this kernel
    constexpr uint32_t kRowB = kL * 16u;                     // bytes per row of a chunk plane
    constexpr uint32_t kTx = ICH * kRowB;                    // bytes copied per row buffer
    constexpr uint32_t kBuf = (uint32_t)KCH * row::kBlk;     // row buffer stride
    static_assert(KCH % 2 == 0 && KCH >= ICH && ICH <= 16 && row::kAcc * NN <= 512 && (MODE != 3 || CO == 4) &&
                  (MODE == 3 || CO == kC) && kS >= 4, "convolution shape");
    extern __shared__ uint8_t tsm_raw[];
    __shared__ __align__(8) unsigned long long raw[kS], full[kS], empty[kS], tfull[row::kAcc], tempty[row::kAcc], wbar, done;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_word;
    __shared__ __align__(16) float sbias[NN];
    uint8_t* sB = (uint8_t*)(((uintptr_t)tsm_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sA = sB + 9 * kBT;                              // 1024-aligned + 9 kBT (multiple of 128)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t aBase = gen_smem_u32(sA), bBase = gen_smem_u32(sB);
    const bool use_img = wimg != nullptr;
    // rows [r0, r1) of the batch, in segments of one image each
    const int r0 = (int)((long long)nrows * blockIdx.x / gridDim.x);
    const int r1 = (int)((long long)nrows * (blockIdx.x + 1) / gridDim.x);

    // the block comes together once, after the barriers; the producer then begins, while the others
    // clear the accumulators
    if (warp == row::kEpi) {
        if (lane < kS) {
            gen_mbar_init(&raw[lane], 1);
            gen_mbar_init(&full[lane], 1);
            gen_mbar_init(&empty[lane], 1);
        }
        if (lane >= 16 && lane < 16 + row::kAcc) {
            gen_mbar_init(&tfull[lane - 16], 1);
            gen_mbar_init(&tempty[lane - 16], 4);
        }
        if (lane == 31) {
            gen_mbar_init(&wbar, 1);
            gen_mbar_init(&done, 1);
            abort_word = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
        if (lane == 31 && use_img) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(gen_smem_u32(&wbar)), "r"(9u * kBT)
                         : "memory");
            gen_bulk(bBase, wimg, 9u * kBT, gen_smem_u32(&wbar));
        }
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gen_smem_u32(&tmem_slot)),
                     "r"(row::cols<CO>())
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if constexpr (KCH > ICH) {   // K-padding blocks: zero once, never copied over
        constexpr int kZ = KCH - ICH, kU = row::kBlk / 16;
        for (int i = tid; i < kS * kZ * kU; i += row::kThreads) {
            const int zb = i / kU, s = zb / kZ, c = ICH + (zb - s * kZ);
            *(uint4*)(sA + s * kBuf + c * row::kBlk + (i - zb * kU) * 16) = make_uint4(0, 0, 0, 0);
        }
    }
    if (!use_img) {
        if constexpr (ICH == KCH && CI == kC && CO == kC) {
            stage_weights<MODE, true>(sB, w, tid, row::kThreads);   // 48 -> 48: 16-byte loads
        } else {
            // w[tap][k][n] (CI x CO) -> B_tap[n][k] over the padded NN x KCH*epc, zeros outside
            constexpr int KK = KCH * kEpc;
#pragma unroll 4
            for (int i = tid; i < 9 * NN * KK; i += row::kThreads) {
                const int tap = i / (NN * KK), r = i - tap * NN * KK, nn = r / KK, k = r - nn * KK;
                const float v = (nn < CO && k < CI) ? __bfloat162float(ld_seq(w + (tap * CI + k) * CO + nn)) : 0.0f;
                *(TA*)(sB + tc::place(tap) * kBT + ((nn >> 3) * KCH + k / kEpc) * kCore + (nn & 7) * 16 +
                       (k % kEpc) * (int)sizeof(TA)) = (TA)v;
            }
        }
    }
    if (tid < NN) sbias[tid] = (MODE == 2 || tid >= CO) ? 0.0f : ld_seq(bias + tid);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    if (warp != row::kEpi) {
        if (warp < 8) {   // every accumulator starts at zero
            for (int c = warp >> 2; c < row::kAcc * NN / 16; c += 2)
                tmem_zero16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(16 * c));
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        gen_bar_sync(row::kThreads - 32);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }

    if (warp < row::kEpi) {
        const int grp = warp >> 2;
        for (int r = r0 + grp; r < r1; r += 2) {
            const int k = r - r0, acc = k % row::kAcc;
            const int img = r / kL;
            const size_t LL = (size_t)kL * kL, pp = (size_t)(r - img * kL) * kL + (size_t)((warp & 3) * 32 + lane);
            uint4 m4[kC / 8];
            load_mask<MODE>(m4, mask, (size_t)img, pp, LL);
            const bool ok = gen_wait(gen_smem_u32(&tfull[acc]), (uint32_t)(k / row::kAcc) & 1u, &abort_word, flag, 4);
            if (!__all_sync(0xFFFFFFFFu, ok)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float v[NN];
            const uint32_t taddr = tmem + (uint32_t)(acc * NN) + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
            for (int j = 0; j < NN / 16; ++j) tmem_ld16(taddr + 16 * j, v + 16 * j);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < NN / 16; ++j) tmem_zero16(taddr + 16 * j);   // the next tile is added to zero
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)   // the accumulator may be used again
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gen_smem_u32(&tempty[acc])) : "memory");
            if constexpr (MODE == 3) {
                float4* dst = reinterpret_cast<float4*>(out_v) + (size_t)img * LL + pp;
                *dst = make_float4(v[0] + sbias[0], v[1] + sbias[1], v[2] + sbias[2], v[3] + sbias[3]);
            } else {
                conv_store<MODE>(v, sbias, out_v, m4, (size_t)img, pp, LL);
            }
        }
    } else if (warp == row::kEpi) {
        int q = 0;   // rows copied
        bool ok = true;
        for (int r = r0; r < r1 && ok;) {
            const int img = r / kL, y0 = r - img * kL, len = min(r1 - r, kL - y0);
            const char* src = reinterpret_cast<const char*>(in) + (size_t)img * ICH * kL * kRowB;
            for (int i = 0; i < len + 2; ++i, ++q) {
                const int s = q % kS;
                if (q >= kS) {
                    ok = gen_wait(gen_smem_u32(&empty[s]), (uint32_t)(q / kS - 1) & 1u, &abort_word, flag, 5);
                    if (!(ok = __all_sync(0xFFFFFFFFu, ok))) break;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                }
                const int yy = (y0 + i - 1) & (kL - 1);
                const uint32_t bar = gen_smem_u32(&raw[s]), buf = aBase + (uint32_t)s * kBuf;
                if (lane == 0)
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kTx) : "memory");
                __syncwarp();
                for (int c = lane; c < ICH; c += 32)
                    gen_bulk(buf + (uint32_t)(c * row::kBlk + 16), src + ((size_t)c * kL + yy) * kRowB, kRowB, bar);
            }
            r += len;
        }
        // the last fill of every slot lands before the CTA's shared memory can be released
        if (lane == 0)
            for (int j = max(0, q - kS); j < q; ++j)
                for (unsigned it = 0; it < (kWaitLimit >> 4); ++it)
                    if (gen_mbar_try_wait(gen_smem_u32(&raw[j % kS]), (uint32_t)(j / kS) & 1u)) break;
    } else if (warp == row::kEpi + 1) {
        const bool lead = elect_one();
        const uint64_t a00 = umma_desc(aBase, (uint32_t)row::kBlk, 128), b00 = umma_desc(bBase, kCore, KCH * kCore);
        const uint32_t alo = (uint32_t)a00, ahi = (uint32_t)(a00 >> 32), blo = (uint32_t)b00, bhi = (uint32_t)(b00 >> 32);
        int q = 0, k0 = 0;   // input rows used; tiles of the segments before
        bool ok = !use_img || gen_wait(gen_smem_u32(&wbar), 0, &abort_word, flag, 6);
        for (int r = r0; r < r1 && ok;) {
            const int len = min(r1 - r, kL - r % kL);
            for (int i = 0; i < len + 2; ++i, ++q) {
                const int s = q % kS;
                // output rows j0 .. j1 of the segment take this input row
                const int j0 = max(0, i - 2), j1 = min(len - 1, i), k = k0 + i;
                // the row's copy and the accumulator that it begins
                const bool fresh = i < len && k >= row::kAcc;
                const uint32_t fb = gen_smem_u32(&full[s]), fp = (uint32_t)(q / kS) & 1u;
                ok = gen_wait2(fb, fp, fresh ? gen_smem_u32(&tempty[k % row::kAcc]) : fb,
                               fresh ? (uint32_t)(k / row::kAcc - 1) & 1u : fp, &abort_word, flag, 5);
                if (!(ok = __all_sync(0xFFFFFFFFu, ok))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int c = j1 - j0 + 1, c0 = (k0 + j0) % row::kAcc, n1 = min(c, row::kAcc - c0), n2 = c - n1;
                // the first row's place among the three taps, and that of the first after the ring's end
                const uint32_t as = alo + (((uint32_t)s * kBuf) >> 4), bs = blo + (uint32_t)(((2 - i + j0) * kBT) >> 4);
                const uint32_t bs2 = bs + (uint32_t)((n1 * kBT) >> 4), d = tmem + (uint32_t)(c0 * NN);
                const uint32_t i1 = idesc_n<MODE>((uint32_t)(n1 * NN)), i2 = idesc_n<MODE>((uint32_t)(n2 * NN));
                if (lead) {
#pragma unroll
                    for (int m = 0; m < 3 * (KCH / 2); ++m) {
                        const uint32_t ao = (uint32_t)((2 * (m % (KCH / 2)) * row::kBlk + m / (KCH / 2) * 16) >> 4);
                        const uint32_t bo = (uint32_t)((3 * (m / (KCH / 2)) * kBT + 2 * (m % (KCH / 2)) * kCore) >> 4);
                        tc_mma_n<MODE>(d, as + ao, ahi, bs + bo, bhi, i1);
                    }
                    if (n2) {   // the rest, at the ring's start
#pragma unroll
                        for (int m = 0; m < 3 * (KCH / 2); ++m) {
                            const uint32_t ao = (uint32_t)((2 * (m % (KCH / 2)) * row::kBlk + m / (KCH / 2) * 16) >> 4);
                            const uint32_t bo = (uint32_t)((3 * (m / (KCH / 2)) * kBT + 2 * (m % (KCH / 2)) * kCore) >> 4);
                            tc_mma_n<MODE>(tmem, as + ao, ahi, bs2 + bo, bhi, i2);
                        }
                    }
                    gen_commit(gen_smem_u32(&empty[s]));
                    if (i >= 2) gen_commit(gen_smem_u32(&tfull[(k0 + i - 2) % row::kAcc]));
                }
                __syncwarp();
            }
            k0 += len;
            r += len;
        }
        // every MMA has completed before the tensor memory is freed (all waits above are bounded)
        if (lead) {
            gen_commit(gen_smem_u32(&done));
            bool drained = false;
            for (unsigned it = 0; it < kWaitLimit && !drained; ++it) drained = gen_mbar_try_wait(gen_smem_u32(&done), 0);
            if (!drained) atomicExch(flag, 4);
            if (use_img)   // the weight copy too, should the wait for it have given up
                for (unsigned it = 0; it < (kWaitLimit >> 4); ++it)
                    if (gen_mbar_try_wait(gen_smem_u32(&wbar), 0)) break;
        }
        __syncwarp();
    } else {   // the periodic neighbours of the copied rows
        int n = 0;   // rows of this CTA, with the two beside each segment
        for (int r = r0; r < r1; n += 2) {
            const int len = min(r1 - r, kL - r % kL);
            n += len;
            r += len;
        }
        for (int q = 0; q < n; ++q) {
            const int s = q % kS;
            const bool ok = gen_wait(gen_smem_u32(&raw[s]), (uint32_t)(q / kS) & 1u, &abort_word, flag, 5);
            if (!__all_sync(0xFFFFFFFFu, ok)) break;
            if (lane < 2 * ICH) {   // slot 0 <- x = 127 (slot 128), slot 129 <- x = 0 (slot 1)
                uint8_t* blk = sA + (uint32_t)s * kBuf + (lane >> 1) * row::kBlk;
                const int to = (lane & 1) ? (row::kSlots - 1) : 0, from = (lane & 1) ? 1 : kL;
                *(uint4*)(blk + to * 16) = *(const uint4*)(blk + from * 16);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gen_smem_u32(&full[s])) : "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(row::cols<CO>())
                     : "memory");
}

// Warp-specialised variant of the BF16 modes (forward and probe), opt-in: one CTA per SM with a
// two-stage window ring and two TMEM accumulators, so the loads of tile k+1, the MMAs of tile k
// and the epilogue of tile k-1 run at once. Measured on GB300 at 16 x 128^2 it is slower than
// two single-role CTAs per SM (75.7 vs 61.6 us per layer): the two producer warps and their
// cp.async completion waits (long-scoreboard stalls) bound the tile rate, not the MMAs.
//   warps 0-3: epilogue (warp w drains TMEM lanes 32w ..), then arrive on tempty[acc];
//   warps 4-5: producers: cp.async of tile k into ring slot k&1 (after empty[slot]), one
//              commit group per tile; once the previous tile's group has landed, fence it to
//              the async proxy and arrive on full[slot];
//   warp 6:    MMA issue (lane 0): wait full[slot] and tempty[acc], 27 MMAs, commit to
//              empty[slot] and tfull[acc]; the warp owns the TMEM allocation.
// Every wait is bounded; a role that gives up sets the error word and stops, and the others
// then time out on the barriers it no longer signals.
constexpr int kWsThreads = 224;

template <int MODE>
__host__ __device__ constexpr int ws_smem_bytes(int L) {
    return 9 * tc::btap<MODE>() + 2 * tc::chunks<MODE>() * tc::window(L) * 16 + 1024;
}

template <int MODE>
__global__ void __launch_bounds__(kWsThreads, 1)
k_gen_conv_ws(const __nv_bfloat16* __restrict__ in, const __nv_bfloat16* __restrict__ w,
              const float* __restrict__ bias, void* __restrict__ out_v, int L, int tiles_per_img, int ntiles,
              int* __restrict__ flag) {
    static_assert(MODE == 0 || MODE == 1, "BF16 modes only");
    using namespace tc;
    constexpr int kCh = chunks<MODE>();        // 6
    constexpr int kBT = btap<MODE>();
    constexpr int kProd = 64;                  // producer threads
    constexpr int kRound = 10;                 // window positions per producer round (60 threads)
    extern __shared__ uint8_t tsm_raw[];
    __shared__ __align__(8) unsigned long long bars[8];   // full[2], empty[2], tfull[2], tempty[2]
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) float sbias[kC];
    uint8_t* sB = (uint8_t*)(((uintptr_t)tsm_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sA = sB + 9 * kBT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int P = L + 2, W = window(L), npad = P * P;
    const uint32_t winBytes = (uint32_t)(kCh * W * 16);

    stage_weights<MODE>(sB, w, tid, blockDim.x);
    if (tid < kC) sbias[tid] = bias[tid];
    if (warp == 6) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gen_smem_u32(&tmem_slot)),
                     "r"(2 * kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        const unsigned counts[8] = {kProd, kProd, 1, 1, 1, 1, 128, 128};
        for (int b = 0; b < 8; ++b)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(gen_smem_u32(&bars[b])), "r"(counts[b]) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const uint32_t aBase = gen_smem_u32(sA), bBase = gen_smem_u32(sB);
    const uint32_t full0 = gen_smem_u32(&bars[0]), empty0 = gen_smem_u32(&bars[2]);
    const uint32_t tfull0 = gen_smem_u32(&bars[4]), tempty0 = gen_smem_u32(&bars[6]);
    const int first = blockIdx.x, stride = gridDim.x;
    const int n = (ntiles > first) ? (ntiles - first + stride - 1) / stride : 0;
    auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
        for (unsigned it = 0; it < (1u << 24); ++it)   // bounded polls
            if (gen_mbar_try_wait(bar, parity)) return true;
        atomicExch(flag, 4);
        return false;
    };
    auto arrive = [&](uint32_t bar) {
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
    };

    if (warp >= 4 && warp < 6) {
        // ---- producers ----
        const int pt = tid - 128;
        auto issue = [&](int k) {
            const int t = first + k * stride, img = t / tiles_per_img;
            const int w0 = (t - img * tiles_per_img) * kM - 1;
            const __nv_bfloat16* src_img = in + (size_t)img * L * L * kC;
            if (pt < kRound * kCh) {
                const int c = pt % kCh;
                int j = pt / kCh, pos = w0 + j;
                int py = (pos >= 0) ? pos / P : -1;
                int px = pos - py * P;
                const uint32_t dst0 = aBase + (uint32_t)(k & 1) * winBytes + (uint32_t)(c * W * 16);
                for (; j < W; j += kRound, pos += kRound) {
                    const bool inside = pos >= 0 && pos < npad;
                    const uint4* src = (const uint4*)src_img;
                    if (inside) {
                        int y = py - 1, x = px - 1;
                        y += (y < 0) ? L : ((y >= L) ? -L : 0);
                        x += (x < 0) ? L : ((x >= L) ? -L : 0);
                        src = (const uint4*)src_img + ((size_t)c * L * L + (size_t)y * L + x);   // chunk plane c
                    }
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst0 + (uint32_t)(j * 16)),
                                 "l"(src), "r"(inside ? 16 : 0)
                                 : "memory");
                    px += kRound;
                    if (px >= P) {
                        px -= P;
                        ++py;
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        bool ok = true;
        for (int k = 0; k < n && ok; ++k) {
            if (k >= 2) ok = wait(empty0 + 8 * (k & 1), ((k >> 1) - 1) & 1);   // MMAs of tile k-2 done
            if (!ok) break;
            issue(k);
            if (k >= 1) {   // tile k-1 landed: publish it
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                arrive(full0 + 8 * ((k - 1) & 1));
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (ok && n > 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            arrive(full0 + 8 * ((n - 1) & 1));
        }
    } else if (warp == 6) {
        // ---- MMA issue ----
        if (lane == 0) {
            for (int k = 0; k < n; ++k) {
                const int sl = k & 1;
                if (!wait(full0 + 8 * sl, (k >> 1) & 1)) break;
                if (k >= 2 && !wait(tempty0 + 8 * sl, ((k >> 1) - 1) & 1)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a0 = aBase + (uint32_t)sl * winBytes, d = tmem + (uint32_t)(sl * kTmemCols);
#pragma unroll 1
                for (int tap = 0; tap < 9; ++tap) {
                    const int shift = (P + 1) + (tap / 3 - 1) * P + (tap % 3 - 1);
#pragma unroll
                    for (int ks = 0; ks < kCh / 2; ++ks) {
                        const uint64_t ad =
                            umma_desc(a0 + (uint32_t)((2 * ks * W + shift) * 16), (uint32_t)(W * 16), 128);
                        const uint64_t bd = umma_desc(bBase + tap * kBT + 2 * ks * kCore, kCore, kCh * kCore);
                        tc_mma<MODE>(d, ad, bd, (tap | ks) ? 1u : 0u);
                    }
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 empty0 + 8 * sl)
                             : "memory");
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 tfull0 + 8 * sl)
                             : "memory");
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue (warps 0-3) ----
        for (int k = 0; k < n; ++k) {
            const int ac = k & 1;
            if (!wait(tfull0 + 8 * ac, (k >> 1) & 1)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int t = first + k * stride, img = t / tiles_per_img;
            const int q0 = P + (t - img * tiles_per_img) * kM;
            float v[kC];
            const uint32_t taddr = tmem + (uint32_t)(ac * kTmemCols) + ((uint32_t)(warp * 32) << 16);
            tmem_ld16(taddr + 0, v);
            tmem_ld16(taddr + 16, v + 16);
            tmem_ld16(taddr + 32, v + 32);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            arrive(tempty0 + 8 * ac);   // the accumulator may be overwritten now
            const int pos = q0 + warp * 32 + lane, py = pos / P, px = pos - py * P;
            if (py >= 1 && py <= L && px >= 1 && px <= L) {
                conv_store<MODE>(v, sbias, out_v, nullptr, (size_t)img, (size_t)(py - 1) * L + (px - 1), (size_t)L * L);
            }
        }
    }
    // every committed MMA has been drained by the epilogue (or timed out); free the TMEM
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 6)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kTmemCols) : "memory");
}

// ------------------------------------------------------------------------------------------
// Weight gradient of a hidden layer on the tensor cores: dW[tap][ci][co] = sum_p
// in[p + tap, ci] * dout[p, co], the positions p as the contraction (kind::f16, FP32
// accumulators in tensor memory). The layer input is BF16 already; the FP32 output gradient
// is split into BF16 hi + lo (lo = the remainder rounded again, 16 significant bits in all)
// and both halves are multiplied into the same accumulator, which is more accurate than TF32.
// The order of the additions is part of the result (an Adam step divides the gradient by its own
// size and the weights are rounded to BF16, so that a last bit here is 1e-4 of the gradients a few
// steps on) and does not depend on how the work is laid out: a K-block is W = min(L, 64)
// consecutive positions of one image row, partial p takes the blocks p, p + nparts, ..., each in
// steps of 16 positions, hi before lo; k_gen_sum_parts adds the partials from the first to the last.
// Both operands are MN-major: a slot holds 8 channels (16 bytes) per position, the positions 16
// bytes apart, so the window of a tap shifted by dx positions is the same slot started dx * 16
// bytes later. A is the output gradient, hi or lo, 48 of M = 64 rows (the others read what follows
// in the stage and are not looked at). B is the input: 6 slots of each of the rows y-1, y, y+1 are
// N = 144 columns (row, input channel). Three accumulators, one per dx, by one CTA per partial or,
// where there are few partials, by three.
// Roles, over a ring of kStages stages (ready / gfull / free per stage):
//   warps 1-3:   after `free`, copy the input rows with their periodic neighbours (cp.async, two
//                blocks in flight), then `ready`;
//   warps 4-15:  read the raw gradient, a block ahead, from global memory into registers, write its
//                hi / lo operands and arrive on gfull;
//   warp 0:      after `ready` and gfull, 2 W/16 MMAs per dx, committed to `free`. The warp stays
//                together, one lane issues;
//   warps 16-19: the bias gradient's first stage (bias_block), beside the MMAs; CTAs past the last
//                partial do nothing else.
// Every wait is bounded and also ends when another role gave up (a shared abort word); a last
// commit is waited for before the tensor memory is read or freed.
// What bounds it: the MMAs (tensor pipe 59 % active, 72 cycles each for N = 144 whatever the rows of
// A hold), what a CTA takes to start and to store its partials, and the reads from L2 beside them
// (16 x 128^2: 78 MB of input, every row for three blocks, and the gradient's 50 MB twice; without the
// input's copies 34 us, without the bias 37). 39 us with the bias gradient; with 30 bulk copies per
// block and the bias in launches of its own it was 62 + 31 us. Whole rows in order with hi and lo in
// separate accumulators took 28.5 us, but that is another sum.
// ------------------------------------------------------------------------------------------
namespace wg {
constexpr int kStages = 6;
constexpr int kThreads = 640;
constexpr int kLoad = 96;                                 // loading threads, warps 1-3
constexpr int kConv = 384;                                // converting threads, warps 4-15
constexpr int kBias = 128;                                // bias threads, warps 16-19
constexpr int kN = 3 * tc::kC;                            // 144 columns: (row, input channel)
constexpr int kM = 64;                                    // rows of A: 48 output channels, the rest not looked at
constexpr int kAccCols = 160;                             // step of the accumulators
constexpr int kCols = 512;                                // columns allocated (a power of two)
constexpr int kPart = 9 * tc::kC * tc::kC;                // floats per partial
__host__ __device__ constexpr int slot(int W) { return W * 16; }          // bytes per gradient slot
__host__ __device__ constexpr int slot_in(int W) { return (W + 2) * 16; }   // bytes per input slot
// a stage: hi and lo (6 slots each), then the input rows (18 slots)
__host__ __device__ constexpr int stage(int W) { return (12 * slot(W) + 18 * slot_in(W) + 127) / 128 * 128; }
constexpr size_t smem(int W) { return (size_t)kStages * stage(W) + 1024; }
static_assert(14 * slot(64) <= stage(64) && 14 * slot(16) <= stage(16), "A of lo ends inside the stage");
// BF16 A and B, both MN-major (instruction-descriptor bits 15 and 16), N = 144, M = 64
constexpr uint32_t kIdesc = tc::idesc<0, kN, kM>() | (1u << 15) | (1u << 16);
// K-block length for an L x L image (0: the tensor-core form does not apply)
__host__ __device__ constexpr int block_len(int L) { return L % 16 != 0 ? 0 : (L <= 64 ? L : (L % 64 == 0 ? 64 : 0)); }
__device__ __forceinline__ void mma(uint32_t tmem, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %6, 0;\n\t"
        "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}" ::"r"(tmem),
        "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(kIdesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
}  // namespace wg

// Bias gradient, first stage: block b sums pixels [b * chunk, (b + 1) * chunk) of the planar FP32
// gradient (G groups of 4 channels) into part[b][4 G], by `lanes` = 256 / G lanes a group: lane l
// takes every lanes-th pixel from l on, then the lanes are added in order. bias_lane is one lane's
// sum, bias_channel one channel's over the lanes.
struct BiasArgs {
    float* part;
    int npix, chunk, nblk;
};
__device__ __forceinline__ float4 bias_lane(const float* dout, int G, int LL, int lanes, int g, int p, int p1) {
    constexpr int kBatch = 8;   // loads in flight
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    const int img = p / LL;
    int pp = p - img * LL;
    const float4* src = reinterpret_cast<const float4*>(dout) + ((size_t)img * G + g) * LL + pp;
    for (; p < p1; p += kBatch * lanes) {
        float4 v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            v[k] = p + k * lanes < p1 ? ld_seq(src) : make_float4(0.f, 0.f, 0.f, 0.f);   // s + 0 is s
            src += lanes;
            pp += lanes;
            if (pp >= LL) {   // the next image (an image holds at least as many pixels as there are lanes)
                pp -= LL;
                src += (size_t)(G - 1) * LL;
            }
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            s.x += v[k].x;
            s.y += v[k].y;
            s.z += v[k].z;
            s.w += v[k].w;
        }
    }
    return s;
}
__device__ __forceinline__ float bias_channel(const float4* red, int lanes, int c) {
    const float* r = reinterpret_cast<const float*>(red + (c >> 2) * lanes) + (c & 3);
    float v = 0.0f;
    for (int k = 0; k < lanes; ++k) v += r[4 * k];
    return v;
}

template <int KS>   // MMA K-steps (16 positions) per K-block: W = 16 KS
__global__ void __launch_bounds__(wg::kThreads, 1)
k_gen_wgrad_tc(const __nv_bfloat16* in, const float* dout, float* part, int L, int nkb, int nparts, int split, BiasArgs bias,
               int* flag) {
    seq_begin();
    using namespace wg;
    constexpr int kC = tc::kC, W = 16 * KS, kSlot = slot(W), kSlotIn = slot_in(W), kStage = stage(W);
    constexpr int kIn = 12 * kSlot;                         // the input rows' place in a stage
    constexpr int kJobs = kC / 8 * W;                       // (channel group, position) of a K-block, one per thread
    static_assert(kJobs <= kConv && kJobs % 32 == 0, "whole converting warps");
    extern __shared__ uint8_t wsm_raw[];
    __shared__ __align__(8) unsigned long long ready[kStages], gfull[kStages], sfree[kStages], done;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_word;
    __shared__ float4 red[252];                             // 12 groups x 21 lanes
    uint8_t* smem = (uint8_t*)(((uintptr_t)wsm_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const size_t LL = (size_t)L * L;
    const int bpr = L / W;                                  // K-blocks per image row
    const uint32_t sbase = gen_smem_u32(smem);
    // this CTA's partial and accumulators dx0 .. dx0 + ndx - 1; its K-blocks first, first + nparts, ...
    const int first = blockIdx.x / split, ndx = 3 / split, dx0 = (blockIdx.x - first * split) * ndx;
    const bool mine = first < nparts;
    const int n = mine ? (nkb - first + nparts - 1) / nparts : 0;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gen_smem_u32(&tmem_slot)),
                     "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp == 1) {
        if (lane < kStages) {
            gen_mbar_init(&ready[lane], kLoad / 32);
            gen_mbar_init(&gfull[lane], kJobs / 32);
            gen_mbar_init(&sfree[lane], 1);
        }
        if (lane == 31) {
            gen_mbar_init(&done, 1);
            abort_word = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    auto place = [&](int j, int& img, int& y, int& x0) {   // of this CTA's K-block j
        const int kb = first + j * nparts, row = kb / bpr;
        img = row / L;
        y = row - img * L;
        x0 = (kb - row * bpr) * W;
    };
    auto fresh = [&](int j) {   // stage of K-block j: its previous MMAs have completed
        return j < kStages || gen_wait(gen_smem_u32(&sfree[j % kStages]), (uint32_t)(j / kStages - 1) & 1u, &abort_word, flag, 4);
    };
    bool ok = true;
    if (warp == 0) {
        const bool lead = elect_one();
        // MN-major, no swizzle: LBO = 128 (8-position K groups), SBO = one slot (8-channel MN
        // groups); the start address field (bits 0-13, address >> 4) is offset per MMA
        const uint64_t a00 = umma_desc(sbase, 128, kSlot), b00 = umma_desc(sbase + (uint32_t)kIn, 128, kSlotIn);
        const uint32_t alo = (uint32_t)a00, ahi = (uint32_t)(a00 >> 32), blo = (uint32_t)b00, bhi = (uint32_t)(b00 >> 32);
        for (int k = 0; k < n; ++k) {
            const int s = k % kStages;
            const uint32_t par = (uint32_t)(k / kStages) & 1u;
            ok = gen_wait2(gen_smem_u32(&ready[s]), par, gen_smem_u32(&gfull[s]), par, &abort_word, flag, 4);
            if (!(ok = __all_sync(0xFFFFFFFFu, ok))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t at = (uint32_t)(s * kStage) >> 4;
            if (lead) {
                for (int d = 0; d < ndx; ++d) {
                    const uint32_t acc = tmem + (uint32_t)(d * kAccCols);
#pragma unroll
                    for (int ks = 0; ks < KS; ++ks) {
                        const uint32_t a = alo + at + (uint32_t)(16 * ks), b = blo + at + (uint32_t)(dx0 + d + 16 * ks);
                        mma(acc, a, ahi, b, bhi, (k | ks) ? 1u : 0u);
                        mma(acc, a + (uint32_t)((6 * kSlot) >> 4), ahi, b, bhi, 1u);
                    }
                }
                gen_commit(gen_smem_u32(&sfree[s]));
            }
            __syncwarp();
        }
        // every MMA has completed before the accumulators are read or freed
        if (lead && n > 0) {
            gen_commit(gen_smem_u32(&done));
            bool drained = false;
            for (unsigned it = 0; it < tc::kWaitLimit && !drained; ++it) drained = gen_mbar_try_wait(gen_smem_u32(&done), 0);
            if (!drained) {
                atomicExch(flag, 4);
                ok = false;
            }
        }
        __syncwarp();
    } else if (warp <= kLoad / 32) {
        const int lt = tid - 32;
        auto landed = [&](int j) {   // K-block j's copies of this warp are in shared memory
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gen_smem_u32(&ready[j % kStages])) : "memory");
        };
        constexpr int kDepth = 2;   // blocks in flight
        int j = 0;
        for (; j < n; ++j) {
            ok = fresh(j);
            if (!(ok = __all_sync(0xFFFFFFFFu, ok))) break;
            int img, y, x0;
            place(j, img, y, x0);
            const uint4* src = reinterpret_cast<const uint4*>(in) + (size_t)img * (kC / 8) * LL;
            const uint32_t dst = sbase + (uint32_t)((j % kStages) * kStage + kIn);
            for (int i = lt; i < 18 * (W + 2); i += kLoad) {   // slot (row, channel group), column x0 - 1 + c
                const int sl = i / (W + 2), c = i - sl * (W + 2), R = sl / 6, h = sl - 6 * R;
                int yy = y + R - 1, x = x0 - 1 + c;
                yy += yy < 0 ? L : (yy >= L ? -L : 0);
                x += x < 0 ? L : (x >= L ? -L : 0);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)(i * 16)),
                             "l"(src + (size_t)h * LL + (size_t)yy * L + x)
                             : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (j >= kDepth) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kDepth) : "memory");
                landed(j - kDepth);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (ok)
            for (int q = max(0, n - kDepth); q < n; ++q) landed(q);
    } else if (warp < 16) {
        const int ct = tid - 128;
        if (ct < kJobs) {   // channel group h at position c of every K-block
            const int h = ct / W, c = ct - h * W;
            float4 a, b;   // the next K-block's gradient
            auto fetch = [&](int j) {
                int img, y, x0;
                place(j, img, y, x0);
                const float4* p = reinterpret_cast<const float4*>(dout) + ((size_t)img * (kC / 4) + 2 * h) * LL + (size_t)y * L + x0 + c;
                a = ld_seq(p);
                b = ld_seq(p + LL);
            };
            if (n > 0) fetch(0);
            for (int j = 0; j < n; ++j) {
                const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                if (j + 1 < n) fetch(j + 1);
                ok = fresh(j);
                if (!(ok = __all_sync(0xFFFFFFFFu, ok))) break;
                uint8_t* sG = smem + (j % kStages) * kStage + h * kSlot + c * 16;
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    hi[e] = pack_bf16(f[2 * e], f[2 * e + 1]);
                    lo[e] = pack_bf16(f[2 * e] - __uint_as_float(hi[e] << 16), f[2 * e + 1] - __uint_as_float(hi[e] & 0xFFFF0000u));
                }
                *reinterpret_cast<uint4*>(sG) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(sG + 6 * kSlot) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gen_smem_u32(&gfull[j % kStages])) : "memory");
            }
        }
    } else if (bias.part) {
        const int bt = tid - (kThreads - kBias);
        for (int b = blockIdx.x; b < bias.nblk; b += gridDim.x) {
            const int p0 = b * bias.chunk, p1 = min(p0 + bias.chunk, bias.npix);
            for (int t = bt; t < 252; t += kBias) {
                const int g = t / 21, pl = t - 21 * g;
                red[t] = bias_lane(dout, kC / 4, (int)LL, 21, g, p0 + pl, p1);
            }
            gen_bar_sync(kBias);
            if (bt < kC) bias.part[(size_t)b * kC + bt] = bias_channel(red, 21, bt);
            gen_bar_sync(kBias);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (__syncthreads_or(!ok)) {
        if (tid == 0) atomicExch(flag, 4);
    } else if (mine) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // a warp reads its own lane quarter q = warp % 4 in chunks of 16 columns: the rows 16 q .. 16 q
        // + 15 of M = 64 are the quarter's first 16 lanes
        const int q = warp & 3, co = lane < 16 ? q * 16 + lane : kC;
        float* dst = part + (size_t)first * kPart;
        if (q < 3)
            for (int c = warp >> 2; c < 9 * ndx; c += kThreads / 128) {
                const int d = c / 9, R = c % 9 / 3, ci0 = c % 3 * 16;
                float v[16];
                tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(d * kAccCols + c % 9 * 16), v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (co < kC)
#pragma unroll
                    for (int e = 0; e < 16; ++e) dst[((R * 3 + dx0 + d) * kC + ci0 + e) * kC + co] = v[e];
            }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
}

// Weight gradient: dW[tap][ci][co] = sum_p in[p + tap, ci] * dout[p, co], over the images and
// tiles given to one CTA; per-CTA partials go to `part` and are summed by k_gen_sum_parts.
// Thread layout: 9 taps x (CIN/6) ci groups x (COUT/8) co groups (6 x 8 accumulators each).
template <int CIN, int COUT>
__global__ void __launch_bounds__(432)
k_gen_wgrad(const __nv_bfloat16* in, const float* dout, float* part,
            int L, int images_per_cta, int nimg) {
    seq_begin();
    extern __shared__ float gsm[];
    constexpr int T2 = kTile + 2;
    constexpr int CG = (CIN + 5) / 6, OG = (COUT + 7) / 8;
    float* tin = gsm;                       // [T2*T2][CIN]
    float* tdo = gsm + T2 * T2 * CIN;       // [kTile*kTile][COUT]
    const int tiles_x = L / kTile;
    const int tile = blockIdx.x % (tiles_x * tiles_x);
    const int igrp = blockIdx.x / (tiles_x * tiles_x);
    const int ty0 = (tile / tiles_x) * kTile, tx0 = (tile % tiles_x) * kTile;
    const int t = threadIdx.x;
    const bool active = t < 9 * CG * OG;
    const int tap = t / (CG * OG), rr = t % (CG * OG), cg = rr / OG, og = rr % OG;
    const int dy = tap / 3, dx = tap % 3;
    float acc[6][8];
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    for (int im = 0; im < images_per_cta; ++im) {
        const int img = igrp * images_per_cta + im;
        if (img >= nimg) break;
        const size_t ibase = (size_t)img * L * L;
        __syncthreads();
        // 16-byte loads (8 BF16 inputs, 4 FP32 gradients), several in flight per thread
        static_assert(CIN % 8 == 0 && COUT % 4 == 0, "16-byte staging");
        // chunk planes of this image; pixel index fastest, so consecutive threads read consecutive pixels
        const size_t LL = (size_t)L * L;
        const uint4* isrc = reinterpret_cast<const uint4*>(in + ibase * CIN);
        const float4* gsrc = reinterpret_cast<const float4*>(dout + ibase * COUT);
#pragma unroll 4
        for (int i = threadIdx.x; i < T2 * T2 * (CIN / 8); i += blockDim.x) {
            const int c8 = i / (T2 * T2), pix = i - c8 * T2 * T2, yy = pix / T2, xx = pix - yy * T2;
            int gy = ty0 + yy - 1, gx = tx0 + xx - 1;   // in [-1, L]: one wrap
            gy += (gy < 0) ? L : ((gy >= L) ? -L : 0);
            gx += (gx < 0) ? L : ((gx >= L) ? -L : 0);
            const uint4 q = ld_seq(isrc + (size_t)c8 * LL + (size_t)gy * L + gx);
            const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&q);
            float* d = tin + pix * CIN + c8 * 8;
#pragma unroll
            for (int k = 0; k < 8; ++k) d[k] = __bfloat162float(e[k]);
        }
#pragma unroll 4
        for (int i = threadIdx.x; i < kTile * kTile * (COUT / 4); i += blockDim.x) {
            const int c4 = i / (kTile * kTile), pix = i - c4 * kTile * kTile, yy = pix / kTile, xx = pix - yy * kTile;
            reinterpret_cast<float4*>(tdo + pix * COUT)[c4] =
                ld_seq(gsrc + (size_t)c4 * LL + (size_t)(ty0 + yy) * L + tx0 + xx);
        }
        __syncthreads();
        if (active) {
            for (int py = 0; py < kTile; ++py)
                for (int px = 0; px < kTile; ++px) {
                    const float* xi = tin + ((py + dy) * T2 + px + dx) * CIN + cg * 6;
                    const float* go = tdo + (py * kTile + px) * COUT + og * 8;
                    float xv[6], gv[8];
#pragma unroll
                    for (int i = 0; i < 6; ++i) xv[i] = (cg * 6 + i < CIN) ? xi[i] : 0.0f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) gv[j] = (og * 8 + j < COUT) ? go[j] : 0.0f;
#pragma unroll
                    for (int i = 0; i < 6; ++i)
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(xv[i], gv[j], acc[i][j]);
                }
        }
    }
    if (!active) return;
    float* dst = part + (size_t)blockIdx.x * 9 * CIN * COUT;
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int ci = cg * 6 + i, co = og * 8 + j;
            if (ci < CIN && co < COUT) dst[(tap * CIN + ci) * COUT + co] = acc[i][j];
        }
}

// The same for the two edge layers (8 -> 48 and 48 -> 4), whose few channels leave most threads of
// that layout without work and one scalar load per multiply-add: 108 threads take one tap x TI
// input x TO output channels each, with 16-byte loads and packed multiply-adds (two input channels
// to an instruction), while the other 128 bring the next half tile into the second buffer. A sum
// runs over the CTA's pixels in their order, as in k_gen_wgrad: the order is part of the result.
// Rows of a pixel are padded by 4 floats so that the staging's stores spread over the banks.
// What bounds it: 256 CTAs on 152 SMs leave two of them on most SMs, seven computing warps in all,
// whose multiply-adds take 28 us. 16 x 128^2: 51 us (8 -> 48) and 36 us (48 -> 4) against 136 and
// 54 in k_gen_wgrad's form; with 8 x 8 outputs to a thread 106 us.
template <int CIN, int COUT, int TI, int TO>
struct EdgeGrad {
    static constexpr int CG = CIN / TI, OG = COUT / TO, kThr = 9 * CG * OG;
    static constexpr int kCompute = 128, kThreads = 256, kHalf = kTile / 2;
    static constexpr int SI = CIN + (CIN > 8 ? 4 : 0), SO = COUT + (COUT > 8 ? 4 : 0);   // floats per pixel
    static constexpr int kTin = (kHalf + 2) * (kTile + 2) * SI, kTdo = kHalf * kTile * SO;
    static constexpr size_t smem = (size_t)2 * (kTin + kTdo) * sizeof(float);
    static_assert(CIN % 8 == 0 && COUT % 4 == 0 && TI % 4 == 0 && TO % 4 == 0 && kThr <= kCompute, "16-byte accesses");
};

template <int CIN, int COUT, int TI, int TO>
__global__ void __launch_bounds__(256, 2)
k_gen_wgrad_edge(const __nv_bfloat16* in, const float* dout, float* part, int L, int images_per_cta, int nimg) {
    seq_begin();
    using E = EdgeGrad<CIN, COUT, TI, TO>;
    extern __shared__ __align__(16) float gsm[];
    constexpr int T2 = kTile + 2, kRowsIn = E::kHalf + 2;
    const int tiles_x = L / kTile;
    const int tile = blockIdx.x % (tiles_x * tiles_x);
    const int img0 = blockIdx.x / (tiles_x * tiles_x) * images_per_cta;
    const int ty0 = (tile / tiles_x) * kTile, tx0 = (tile % tiles_x) * kTile;
    const int steps = 2 * min(images_per_cta, nimg - img0);   // half tiles
    const size_t LL = (size_t)L * L;
    // half tile `s` into its buffer, by threads t0, t0 + 1, ... (nthr of them)
    auto stage = [&](int s, int t0, int nthr) {
        const size_t ibase = (size_t)(img0 + (s >> 1)) * LL;
        const int y0 = ty0 + (s & 1) * E::kHalf;
        float* const tin = gsm + (s & 1) * (E::kTin + E::kTdo);   // [kRowsIn * T2][SI], then [kHalf * kTile][SO]
        float* const tdo = tin + E::kTin;
        const uint4* isrc = reinterpret_cast<const uint4*>(in + ibase * CIN);
        const float4* gsrc = reinterpret_cast<const float4*>(dout + ibase * COUT);
        // chunk planes of the image; pixel index fastest, so consecutive threads read consecutive pixels
#pragma unroll 6
        for (int i = t0; i < E::kHalf * kTile * (COUT / 4); i += nthr) {
            const int c4 = i / (E::kHalf * kTile), pix = i - c4 * E::kHalf * kTile, yy = pix / kTile, xx = pix - yy * kTile;
            *reinterpret_cast<float4*>(tdo + pix * E::SO + c4 * 4) = ld_seq(gsrc + (size_t)c4 * LL + (size_t)(y0 + yy) * L + tx0 + xx);
        }
#pragma unroll 4
        for (int i = t0; i < kRowsIn * T2 * (CIN / 8); i += nthr) {
            const int c8 = i / (kRowsIn * T2), pix = i - c8 * kRowsIn * T2, yy = pix / T2, xx = pix - yy * T2;
            int gy = y0 + yy - 1, gx = tx0 + xx - 1;   // in [-1, L]: one wrap
            gy += (gy < 0) ? L : ((gy >= L) ? -L : 0);
            gx += (gx < 0) ? L : ((gx >= L) ? -L : 0);
            const uint4 q = ld_seq(isrc + (size_t)c8 * LL + (size_t)gy * L + gx);
            float4* d = reinterpret_cast<float4*>(tin + pix * E::SI + c8 * 8);   // a BF16 is an FP32's top half
            d[0] = make_float4(__uint_as_float(q.x << 16), __uint_as_float(q.x & 0xFFFF0000u),
                               __uint_as_float(q.y << 16), __uint_as_float(q.y & 0xFFFF0000u));
            d[1] = make_float4(__uint_as_float(q.z << 16), __uint_as_float(q.z & 0xFFFF0000u),
                               __uint_as_float(q.w << 16), __uint_as_float(q.w & 0xFFFF0000u));
        }
    };
    const int t = threadIdx.x;
    const int tap = t / (E::CG * E::OG), rr = t % (E::CG * E::OG), cg = rr / E::OG, og = rr % E::OG;
    const int dy = tap / 3, dx = tap % 3;
    f2 acc[TI / 2][TO];
#pragma unroll
    for (int i = 0; i < TI / 2; ++i)
#pragma unroll
        for (int j = 0; j < TO; ++j) acc[i][j] = f2{0ull};
    stage(0, t, E::kThreads);
    __syncthreads();
    for (int s = 0; s < steps; ++s) {
        if (t >= E::kCompute) {
            if (s + 1 < steps) stage(s + 1, t - E::kCompute, E::kThreads - E::kCompute);
        } else if (t < E::kThr) {
            const float* const tin = gsm + (s & 1) * (E::kTin + E::kTdo);
            const float* const tdo = tin + E::kTin;
            for (int py = 0; py < E::kHalf; ++py) {
                const float* xi = tin + ((py + dy) * T2 + dx) * E::SI + cg * TI;
                const float* go = tdo + py * kTile * E::SO + og * TO;
#pragma unroll 8
                for (int px = 0; px < kTile; ++px, xi += E::SI, go += E::SO) {
                    f2 xv[TI / 2];
#pragma unroll
                    for (int i = 0; i < TI / 4; ++i) {
                        const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(xi + 4 * i);
                        xv[2 * i].v = q.x;
                        xv[2 * i + 1].v = q.y;
                    }
#pragma unroll
                    for (int j = 0; j < TO / 4; ++j) {
                        const float4 q = *reinterpret_cast<const float4*>(go + 4 * j);
                        const f2 gv[4] = {pk(q.x, q.x), pk(q.y, q.y), pk(q.z, q.z), pk(q.w, q.w)};
#pragma unroll
                        for (int i = 0; i < TI / 2; ++i)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[i][4 * j + e] = fma2(xv[i], gv[e], acc[i][4 * j + e]);
                    }
                }
            }
        }
        __syncthreads();
    }
    if (t >= E::kThr) return;
    float* dst = part + (size_t)blockIdx.x * 9 * CIN * COUT;
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TO; j += 4) {
            float o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = (i & 1) ? hi(acc[i >> 1][j + e]) : lo(acc[i >> 1][j + e]);
            *reinterpret_cast<float4*>(dst + (tap * CIN + cg * TI + i) * COUT + og * TO + j) = make_float4(o[0], o[1], o[2], o[3]);
        }
}

// Sums of partials, one job per blockIdx.y, a backward pass's in one launch. Weights: a thread per
// output adds the nparts partials from the first to the last. Biases (wide): a block per output,
// thread t adds the partials t, t + 128, ..., then a tree. Both orders are part of the result.
// What bounds it: the loads in flight, one chain of additions per output. The eight layers of 16 x
// 128^2 (82 MB of partials) take 24 us with eight loads in flight per thread; in one comparison 8 27.5,
// 4 29.7, 16 and 32 in predicated batches 51 and 90, two or four outputs per thread 34 and 45.
struct SumJob {
    const float* part;
    float* out;
    int nparts, n;   // partials of n floats
    int wide;
};
constexpr int kSumJobs = 2 * kGenLayers;
struct SumArgs {
    SumJob job[kSumJobs];
    int n = 0;         // jobs
    size_t used = 0;   // floats of the scratch that they hold
};
__global__ void __launch_bounds__(128) k_gen_sum_parts(const __grid_constant__ SumArgs a) {
    seq_begin();
    const SumJob& j = a.job[blockIdx.y];
    const int t = threadIdx.x, n = j.n, nparts = j.nparts;
    if (!j.wide) {
        const int i = blockIdx.x * 128 + t;
        if (i >= n) return;
        constexpr int kBatch = 8;
        const float* p = j.part + i;
        float s = 0.0f;
        int k0 = 0;
        for (; k0 + kBatch <= nparts; k0 += kBatch, p += (size_t)kBatch * n) {
            float v[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; ++k) v[k] = ld_seq(p + (size_t)k * n);
#pragma unroll
            for (int k = 0; k < kBatch; ++k) s += v[k];
        }
        for (; k0 < nparts; ++k0, p += n) s += ld_seq(p);
        j.out[i] = s;
        return;
    }
    __shared__ float red[128];
    if ((int)blockIdx.x >= n) return;
    float s = 0.0f;
    for (int k = t; k < nparts; k += 128) s += ld_seq(j.part + (size_t)k * n + blockIdx.x);
    red[t] = s;
    __syncthreads();
    for (int h = 64; h > 0; h >>= 1) {
        if (t < h) red[t] += red[t + h];
        __syncthreads();
    }
    if (t == 0) j.out[blockIdx.x] = red[0];
}

// First stage of a layer's bias gradient (the hidden layers' on the tensor cores: k_gen_wgrad_tc).
__global__ void __launch_bounds__(256) k_gen_bgrad_part(const float* dout, int LL, int cout, BiasArgs b) {
    seq_begin();
    __shared__ float4 red[256];
    const int G = cout / 4, lanes = 256 / G, t = threadIdx.x, g = t / lanes;
    const int p0 = blockIdx.x * b.chunk, p1 = min(p0 + b.chunk, b.npix);
    if (g < G) red[t] = bias_lane(dout, G, LL, lanes, g, p0 + t - g * lanes, p1);
    __syncthreads();
    if (t < cout) b.part[(size_t)blockIdx.x * cout + t] = bias_channel(red, lanes, t);
}

// Weight update and every form of the weights that a pass reads, one launch for all layers (the
// Adam steps, BF16 copies and operand images were 46 launches of about 3 us): thread i of layer
// blockIdx.y steps weight i, then the biases (adam != 0), and writes wb[tap][ci][co], the flipped
// transpose wt[8-tap][co][ci], and where the layer has them its images in the B-operand layout
// k_gen_conv_row uses in shared memory: per tap, NN/8 x KCH core matrices of 8 rows (n) x 16 bytes
// (8 BF16 or 4 TF32 consecutive k); entries past cin and cout stay zero from the allocation.
struct UpdateArgs {
    GenLayer layer[kGenLayers];
    float lr, b1, b2, c1, c2, eps;
    int adam;
};

__device__ __forceinline__ float adam_step(const UpdateArgs& u, float* p, const float* g, float* m, float* v, int i) {
    const float gi = g[i];
    // fused as written: left to the compiler, the fused product depends on the code around it, and a
    // weight's last bit decides now and then how its BF16 copy is rounded
    const float mi = __fmaf_rn(1.0f - u.b1, gi, __fmul_rn(u.b1, m[i]));
    const float vi = __fmaf_rn(__fmul_rn(1.0f - u.b2, gi), gi, __fmul_rn(u.b2, v[i]));
    m[i] = mi;
    v[i] = vi;
    p[i] -= u.lr * (mi / u.c1) / (sqrtf(vi / u.c2) + u.eps);
    return p[i];
}

__global__ void __launch_bounds__(128) k_gen_update(const __grid_constant__ UpdateArgs u) {
    seq_begin();
    const GenLayer& y = u.layer[blockIdx.y];
    const int cin = y.cin, cout = y.cout, n = 9 * cin * cout;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) {
        if (u.adam && i < n + cout) adam_step(u, y.b, y.gb, y.mb, y.vb, i - n);
        return;
    }
    const float w = u.adam ? adam_step(u, y.w, y.gw, y.mw, y.vw, i) : y.w[i];
    const int tap = i / (cin * cout), r = i - tap * cin * cout, ci = r / cout, co = r - ci * cout;
    const __nv_bfloat16 v = __float2bfloat16(w);
    y.wb[i] = v;
    y.wt[((8 - tap) * cout + co) * cin + ci] = v;
    const int kch = y.kch, nn = (cout + 15) / 16 * 16;
    *reinterpret_cast<__nv_bfloat16*>(y.wimg + tc::place(tap) * (nn / 8) * kch * 128 + ((co >> 3) * kch + ci / 8) * 128 + (co & 7) * 16 +
                                      (ci % 8) * 2) = v;
    if (y.wtimg)   // hidden layers: wt's k is co, its n is ci
        *reinterpret_cast<float*>(y.wtimg + tc::place(8 - tap) * (kGenC / 8) * (kGenC / 4) * 128 +
                                  ((ci >> 3) * (kGenC / 4) + co / 4) * 128 + (ci & 7) * 16 + (co % 4) * 4) =
            __bfloat162float(v);
}

// Network input for a batch: y = normalise(sqrt(1 - s^2) x + s g) and the condition channels.
// mode 0: x from the dataset (index per item), target = x.  mode 1: x = current estimate `cur`
// (sampling), g fresh noise from Philox (stream NOISE, counter = draws + item).  mode 2: as 1,
// but g is the noise predicted from the previous input y' at level s_prev,
// g = (y' - sqrt(1 - s_prev^2) x) / s_prev (deterministic DDIM-style update).  mode 3: the
// variance-preserving posterior step from y' at s_prev to level s (DDPM-style): with
// a' = 1 - s_prev^2, a = 1 - s^2, alpha = a'/a, y = sqrt(a)(1-alpha)/(1-a') x
// + sqrt(alpha)(1-a)/(1-a') y' + sqrt((1-a)(1-alpha)/(1-a')) g, then normalised.
__global__ void k_gen_input(int mode, const __nv_bfloat16* __restrict__ snaps, const int* __restrict__ idx,
                            const float* cur, const float* __restrict__ sig,
                            const float* __restrict__ cnd, int L, uint32_t k0, uint32_t k1,
                            unsigned long long draw0, __nv_bfloat16* act0,
                            float* target, float s_prev) {
    seq_begin();
    const int item = blockIdx.y;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= L * L) return;
    float x[3];
    if (mode == 0) {
        const __nv_bfloat16* s = snaps + ((size_t)idx[item] * L * L + p) * 3;
        for (int c = 0; c < 3; ++c) x[c] = __bfloat162float(s[c]);
    } else {
        const float4 e = ld_seq(reinterpret_cast<const float4*>(cur) + (size_t)item * L * L + p);
        x[0] = e.x;
        x[1] = e.y;
        x[2] = e.z;
    }
    const float s = sig[item];
    const unsigned long long d = draw0 + (unsigned long long)item;
    nmmc_u4 r = nmmc_philox((uint32_t)p, (uint32_t)d, (uint32_t)(d >> 32) | (NMMC_STREAM_NOISE << 28), 0u, k0, k1);
    // Box-Muller: three normals from four uniforms
    const float u1 = nmmc_u01f(r.x), u2 = nmmc_u01f(r.y), u3 = nmmc_u01f(r.z), u4 = nmmc_u01f(r.w);
    const float rA = sqrtf(-2.0f * logf(u1)), rB = sqrtf(-2.0f * logf(u3));
    float sa, ca, sb, cb;
    sincospif(2.0f * u2, &sa, &ca);
    sincospif(2.0f * u4, &sb, &cb);
    float g[3] = {rA * ca, rA * sa, rB * cb};
    // the 8 input channels of a pixel are one 16-byte access (element by element, 9 us for 16 x 128^2,
    // now 7 us)
    uint4* const ap = reinterpret_cast<uint4*>(act0) + (size_t)item * L * L + p;
    uint4 prev = make_uint4(0u, 0u, 0u, 0u);
    if (mode >= 2) prev = *ap;
    const __nv_bfloat16* yp = reinterpret_cast<const __nv_bfloat16*>(&prev);
    if (mode == 2 && s_prev < 1.0f) {
        const float kp = sqrtf(fmaxf(0.0f, 1.0f - s_prev * s_prev));
        for (int c = 0; c < 3; ++c) g[c] = (__bfloat162float(yp[c]) - kp * x[c]) / s_prev;
    }
    const float keep = sqrtf(fmaxf(0.0f, 1.0f - s * s));
    float y[3], n2 = 0.0f;
    if (mode == 3 && s_prev < 1.0f && s_prev > s) {
        const float ap = 1.0f - s_prev * s_prev, a = 1.0f - s * s, alpha = ap / a;
        const float cx = sqrtf(a) * (1.0f - alpha) / (1.0f - ap);
        const float cy = sqrtf(alpha) * (1.0f - a) / (1.0f - ap);
        const float cg = sqrtf(fmaxf(0.0f, (1.0f - a) * (1.0f - alpha) / (1.0f - ap)));
        for (int c = 0; c < 3; ++c) {
            y[c] = cx * x[c] + cy * __bfloat162float(yp[c]) + cg * g[c];
            n2 += y[c] * y[c];
        }
    } else {
        for (int c = 0; c < 3; ++c) {
            y[c] = keep * x[c] + s * g[c];
            n2 += y[c] * y[c];
        }
    }
    const float inv = n2 > 0.0f ? rsqrtf(n2) : 0.0f;
    __align__(16) __nv_bfloat16 a[8];
    for (int c = 0; c < 3; ++c) a[c] = __float2bfloat16(y[c] * inv);
    const float* cd = cnd + 3 * (size_t)(mode == 0 ? idx[item] : item);   // mode 0: the snapshot's own
    a[3] = __float2bfloat16(cd[0] / 1.5f);
    a[4] = __float2bfloat16(cd[1]);
    a[5] = __float2bfloat16(cd[2] / 0.8f);
    a[6] = __float2bfloat16(s);
    a[7] = __float2bfloat16(0.0f);
    *ap = *reinterpret_cast<const uint4*>(a);
    if (mode == 0 && target) {
        reinterpret_cast<float4*>(target)[(size_t)item * L * L + p] = make_float4(x[0], x[1], x[2], 0.0f);
    }
}

// Loss and its gradient through spin = v/|v|: loss += |s - x|^2 / npix_total;
// dL/dv = (g - s (s.g)) / |v| with g = 2 (s - x) / npix_total.
__global__ void __launch_bounds__(256)
k_gen_head(const float* v, const float* target, int npix, float scale,
           float* gv, double* loss) {
    seq_begin();
    __shared__ float red[8];
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.0f;
    if (p < npix) {
        const float4 a4 = ld_seq(reinterpret_cast<const float4*>(v) + p), x4 = ld_seq(reinterpret_cast<const float4*>(target) + p);
        const float a[3] = {a4.x, a4.y, a4.z}, x[3] = {x4.x, x4.y, x4.z};
        const float n2 = a[0] * a[0] + a[1] * a[1] + a[2] * a[2] + 1e-12f;
        const float inv = rsqrtf(n2);
        float s[3], g[3], sg = 0.0f;
        for (int c = 0; c < 3; ++c) {
            s[c] = a[c] * inv;
            const float d = s[c] - x[c];
            l += d * d;
            g[c] = 2.0f * d * scale;
            sg += s[c] * g[c];
        }
        reinterpret_cast<float4*>(gv)[p] =
            make_float4((g[0] - s[0] * sg) * inv, (g[1] - s[1] * sg) * inv, (g[2] - s[2] * sg) * inv, 0.0f);
    }
    // one FP64 addition per block of 256 pixels (one per warp took 15 us for 16 x 128^2)
    for (int off = 16; off > 0; off >>= 1) l += __shfl_down_sync(0xffffffffu, l, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += (double)(red[w] * scale);
        atomicAdd(loss, t);
    }
}

// Sampling: cur <- normalise(v) (the denoised estimate)
__global__ void k_gen_normalise(const float* v, int npix, float* cur) {
    seq_begin();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    const float4 a = ld_seq(reinterpret_cast<const float4*>(v) + p);
    const float n2 = a.x * a.x + a.y * a.y + a.z * a.z;
    const float inv = n2 > 0.0f ? rsqrtf(n2) : 0.0f;
    reinterpret_cast<float4*>(cur)[p] = make_float4(a.x * inv, a.y * inv, a.z * inv, 0.0f);
}

// Sampler chain (split-colour FP32 planes, 2-D) <-> NHWC
__global__ void k_gen_from_chain(const DevModel m, const float* __restrict__ spins, const int* __restrict__ chains,
                                 __nv_bfloat16* __restrict__ snaps, int slot0) {
    const int item = blockIdx.y, chain = chains[item];
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int L = m.edge;
    if (p >= L * L) return;
    const int y = p / L, x = p - y * L, colour = (x + y) & 1;
    const size_t P = (size_t)m.nhalf_pad, i = (size_t)y * m.hx + (x >> 1);
    const float* pl = spins + ((size_t)chain * 2 + colour) * 3 * P;
    __nv_bfloat16* o = snaps + ((size_t)(slot0 + item) * L * L + p) * 3;
    o[0] = __float2bfloat16(pl[i]);
    o[1] = __float2bfloat16(pl[P + i]);
    o[2] = __float2bfloat16(pl[2 * P + i]);
}

__global__ void k_gen_to_chain(const DevModel m, float* __restrict__ spins, const int* __restrict__ chains,
                               const float* __restrict__ cur) {
    const int item = blockIdx.y, chain = chains[item];
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int L = m.edge;
    if (p >= L * L) return;
    const int y = p / L, x = p - y * L, colour = (x + y) & 1;
    const size_t P = (size_t)m.nhalf_pad, i = (size_t)y * m.hx + (x >> 1);
    float* pl = spins + ((size_t)chain * 2 + colour) * 3 * P;
    const float* a = cur + ((size_t)item * L * L + p) * kGenCout;
    pl[i] = a[0];
    pl[P + i] = a[1];
    pl[2 * P + i] = a[2];
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
namespace {

// Raises a kernel's dynamic shared-memory limit on the generator's device (once per kernel and generator);
// max_shared also asks for the whole L1/shared array as shared memory.
int ensure_smem(nmmc_gen* g, const void* fn, int bytes, bool max_shared) {
    if (bytes <= g->attr_smem[fn]) return NMMC_OK;
    // The limit belongs to the kernel, not to the generator: every generator sets the device's, so that one of
    // a smaller edge does not lower it for the others.
    cudaFuncAttributes at{};
    int dev = 0, most = 0;
    cudaError_t e = cudaFuncGetAttributes(&at, fn);
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    most -= (int)at.sharedSizeBytes;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, std::max(most, bytes));
    if (e == cudaSuccess && max_shared)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return cuda_check(e, "cudaFuncSetAttribute(generator kernel)");
    g->attr_smem[fn] = most;
    return NMMC_OK;
}

template <int CIN, int COUT, typename TIN, int EPI>
int conv_launch(nmmc_gen* g, const TIN* in, const __nv_bfloat16* w, const float* bias,
                const __nv_bfloat16* mask, int mask_c, void* out, int nimg) {
    const size_t smem = (size_t)(9 * CIN * COUT + CIN * (kTile + 2) * (kTile + 2)) * sizeof(float);
    if (int rc = ensure_smem(g, (const void*)k_gen_conv<CIN, COUT, TIN, EPI>, (int)smem, false)) return rc;
    dim3 grid(g->L / kTile, g->L / kTile, nimg);
    launch_seq(g->stream, k_gen_conv<CIN, COUT, TIN, EPI>, dim3(grid), 256, smem, in, w, bias, mask, mask_c, out, g->L);
    return cuda_check(cudaGetLastError(), "k_gen_conv");
}

// L = 128: the row-ring kernel (every mode and layer shape), one CTA per SM. wimg: the layer's
// weight image (nullptr: the threads rearrange w).
template <int MODE, int ICH = tc::chunks<MODE>(), int KCH = ICH, int CO = tc::kC>
int conv_row_launch(nmmc_gen* g, const typename tc::Traits<MODE>::TA* in, const __nv_bfloat16* w, const float* bias,
                    const __nv_bfloat16* mask, void* out, int nimg, const uint8_t* wimg = nullptr) {
    constexpr int smem = row::smem_bytes<KCH, CO>();
    if (int rc = ensure_smem(g, (const void*)k_gen_conv_row<MODE, ICH, KCH, CO>, smem, true)) return rc;
    const int nrows = nimg * g->L;
    launch_seq(g->stream, k_gen_conv_row<MODE, ICH, KCH, CO>, dim3(std::min(nrows, g->sm_count)), row::kThreads, smem, in, w,
               g->use_wimg ? wimg : nullptr, bias, mask, out, nrows, g->d_flag);
    return cuda_check(cudaGetLastError(), "k_gen_conv_row");
}

// The first (8 -> 48, ReLU) and last (48 -> 4, linear) layers on the tensor cores when L = 128
// and the row-ring kernels are on; false when they run on the FMA pipes.
bool edge_layers_on_tc(const nmmc_gen* g) { return g->use_tc && g->use_rows && g->L == tc::kM; }

// Hidden-layer convolution on the tensor cores: the row-ring kernel at L = 128, else persistent CTAs,
// as many per SM as the shared memory allows (at most two).
template <int MODE>
int conv_tc_launch(nmmc_gen* g, const typename tc::Traits<MODE>::TA* in, const __nv_bfloat16* w, const float* bias,
                   const __nv_bfloat16* mask, void* out, int nimg, const uint8_t* wimg = nullptr) {
    if (g->use_rows && g->L == tc::kM && !(MODE != 2 && g->use_ws))
        return conv_row_launch<MODE>(g, in, w, bias, mask, out, nimg, wimg);
    if constexpr (MODE != 2) {   // BF16 modes: the warp-specialised kernel when two windows fit
        const int ws = ws_smem_bytes<MODE>(g->L);
        if (g->use_ws && ws <= tc::kSmemMax) {
            if (int rc = ensure_smem(g, (const void*)k_gen_conv_ws<MODE>, ws, true)) return rc;
            const int tiles_per_img = (g->L * (g->L + 2) + tc::kM - 1) / tc::kM;
            const int ntiles = nimg * tiles_per_img;
            const int grid = std::min(ntiles, g->sm_count);
            k_gen_conv_ws<MODE><<<grid, kWsThreads, ws, g->stream>>>(in, w, bias, out, g->L, tiles_per_img, ntiles,
                                                                      g->d_flag);
            return cuda_check(cudaGetLastError(), "k_gen_conv_ws");
        }
    }
    const int smem = tc::smem_bytes<MODE>(g->L);
    if (smem > tc::kSmemMax)
        return set_error(NMMC_ERR_UNSUPPORTED, "lattice edge %d too large for the tensor-core convolution", g->L);
    // the whole unified L1/shared array as shared memory, so two BF16 CTAs fit per SM
    if (int rc = ensure_smem(g, (const void*)k_gen_conv_tc<MODE>, smem, true)) return rc;
    // CTAs per SM from the shared memory (+ static and the 1 KB the driver reserves), at most two
    // (64 TMEM columns and 128 threads each). The runtime's occupancy query answers 1 for this
    // kernel on GB300 although two CTAs are co-resident when launched.
    const int per_sm = std::max(1, std::min(2, g->smem_per_sm / (smem + 2048)));
    const int tiles_per_img = (g->L * (g->L + 2) + tc::kM - 1) / tc::kM;   // padded rows 1..L
    const int ntiles = nimg * tiles_per_img;
    const int grid = std::min(ntiles, per_sm * g->sm_count);
    launch_seq(g->stream, k_gen_conv_tc<MODE>, dim3(grid), 128, smem, in, w, g->use_wimg ? wimg : nullptr, bias, mask, out, g->L, tiles_per_img, ntiles, g->d_flag);
    return cuda_check(cudaGetLastError(), "k_gen_conv_tc");
}

// Reads and clears the device error word after the stream has drained.
int check_flag(nmmc_gen* g) {
    int f = 0;
    NMMC_CUDA(cudaMemcpy(&f, g->d_flag, sizeof(int), cudaMemcpyDeviceToHost));
    if (!f) return NMMC_OK;
    cudaMemset(g->d_flag, 0, sizeof(int));
    return set_error(NMMC_ERR_TIMEOUT, "a tensor-core convolution gave up waiting for its MMAs (code %d)", f);
}

// The sums asked for so far, one launch.
int launch_sums(nmmc_gen* g, SumArgs& a) {
    int most = 0;
    for (int k = 0; k < a.n; ++k) most = std::max(most, a.job[k].wide ? a.job[k].n : (a.job[k].n + 127) / 128);
    if (a.n) launch_seq(g->stream, k_gen_sum_parts, dim3(most, a.n), 128, 0, a);
    a.n = 0;
    a.used = 0;
    return cuda_check(cudaGetLastError(), "k_gen_sum_parts");
}

// `floats` of the scratch for the partials of the next `jobs` sums; sums that hold too much of it are
// launched first. nullptr: too small.
float* sum_room(nmmc_gen* g, SumArgs& a, size_t floats, int jobs) {
    const size_t need = (floats + 3) / 4 * 4;
    if (a.n + jobs > kSumJobs || a.used + need > g->wpart_cap)
        if (launch_sums(g, a)) return nullptr;
    if (need > g->wpart_cap) return nullptr;
    a.used += need;
    return g->wpart + a.used - need;
}
void sum_add(SumArgs& a, const float* part, int nparts, int n, float* out, int wide) {
    a.job[a.n++] = SumJob{part, out, nparts, n, wide};
}

// Blocks of a bias gradient's first stage: about two per SM, chunks of a multiple of 64 pixels.
BiasArgs bias_shape(const nmmc_gen* g, int nimg) {
    const int npix = nimg * g->L * g->L, want = 2 * std::max(1, g->sm_count);
    BiasArgs b{nullptr, npix, 0, 0};
    b.chunk = std::max(64, ((npix + want - 1) / want + 63) / 64 * 64);
    b.nblk = (npix + b.chunk - 1) / b.chunk;
    return b;
}

// Bias gradient gb[co] = sum over the batch's pixels of dout[p, co].
int bgrad_launch(nmmc_gen* g, const float* dout, int nimg, int cout, float* gb, SumArgs& sums) {
    BiasArgs b = bias_shape(g, nimg);
    if (cout % 4 != 0 || cout > 256) return set_error(NMMC_ERR_ARG, "bias gradient: channels not a multiple of 4");
    b.part = sum_room(g, sums, (size_t)b.nblk * cout, 1);
    if (!b.part) return set_error(NMMC_ERR_ARG, "bias-gradient scratch too small");
    launch_seq(g->stream, k_gen_bgrad_part, dim3(b.nblk), 256, 0, dout, g->L * g->L, cout, b);
    sum_add(sums, b.part, b.nblk, cout, gb, 1);
    return cuda_check(cudaGetLastError(), "k_gen_bgrad_part");
}

// Partials of a weight gradient on the FMA pipes: one per pixel tile and kPartImages images.
constexpr int kPartImages = 4;
size_t tile_parts(int L, int nimg) { return (size_t)(L / kTile) * (L / kTile) * ((nimg + kPartImages - 1) / kPartImages); }

// Hidden-layer weight and bias gradient on the tensor cores (k_gen_wgrad_tc). The number of partials,
// and with it the order of the sums, is that of SMs, K-blocks or the largest batch's pixel tiles,
// whichever is the smallest; few partials are shared by three CTAs each.
int wgrad_tc_launch(nmmc_gen* g, const __nv_bfloat16* in, const float* dout, float* gw, float* gb, int nimg, SumArgs& sums) {
    const int W = wg::block_len(g->L), sms = std::max(1, g->sm_count);
    const int nkb = (int)((size_t)nimg * g->L * (g->L / W));
    const int nparts = (int)std::min<size_t>({(size_t)nkb, (size_t)sms, tile_parts(g->L, g->bcap)});
    if (nparts < 1) return set_error(NMMC_ERR_ARG, "weight-gradient scratch too small");
    BiasArgs bias = gb ? bias_shape(g, nimg) : BiasArgs{nullptr, 0, 0, 0};
    const size_t nw = (size_t)nparts * wg::kPart;
    float* part = sum_room(g, sums, nw + (size_t)bias.nblk * tc::kC, gb ? 2 : 1);
    if (!part) return set_error(NMMC_ERR_ARG, "weight-gradient scratch too small");
    if (gb) bias.part = part + nw;
    const int split = 3 * nparts <= sms ? 3 : 1;
    const int grid = std::max(nparts * split, std::min(sms, bias.nblk));
    auto fn = W == 64 ? k_gen_wgrad_tc<4> : W == 48 ? k_gen_wgrad_tc<3> : W == 32 ? k_gen_wgrad_tc<2> : k_gen_wgrad_tc<1>;
    const int smem = (int)wg::smem(W);
    if (int rc = ensure_smem(g, (const void*)fn, smem, true)) return rc;
    launch_seq(g->stream, fn, dim3(grid), wg::kThreads, smem, in, dout, part, g->L, nkb, nparts, split, bias, g->d_flag);
    sum_add(sums, part, nparts, wg::kPart, gw, 0);
    if (gb) sum_add(sums, bias.part, bias.nblk, tc::kC, gb, 1);
    return cuda_check(cudaGetLastError(), "k_gen_wgrad_tc");
}

// Weight gradient of a layer, and its bias gradient where gb is not null.
template <int CIN, int COUT>
int wgrad_launch(nmmc_gen* g, const __nv_bfloat16* in, const float* dout, float* gw, float* gb, int nimg,
                 SumArgs& sums) {
    if (CIN == tc::kC && COUT == tc::kC && g->use_tc && wg::block_len(g->L) > 0)
        return wgrad_tc_launch(g, in, dout, gw, gb, nimg, sums);
    const int nparts = (int)tile_parts(g->L, nimg), n = 9 * CIN * COUT;
    float* part = sum_room(g, sums, (size_t)nparts * n, 1);
    if (!part) return set_error(NMMC_ERR_ARG, "weight-gradient scratch too small");
    if constexpr (CIN == kGenC && COUT == kGenC) {
        const size_t smem = (size_t)((kTile + 2) * (kTile + 2) * CIN + kTile * kTile * COUT) * sizeof(float);
        if (int rc = ensure_smem(g, (const void*)k_gen_wgrad<CIN, COUT>, (int)smem, false)) return rc;
        launch_seq(g->stream, k_gen_wgrad<CIN, COUT>, dim3(nparts), 432, smem, in, dout, part, g->L, kPartImages, nimg);
    } else {
        constexpr int TI = COUT < 8 ? 4 : 8, TO = 4;   // 108 threads
        using E = EdgeGrad<CIN, COUT, TI, TO>;
        auto fn = k_gen_wgrad_edge<CIN, COUT, TI, TO>;
        if (int rc = ensure_smem(g, (const void*)fn, (int)E::smem, false)) return rc;
        launch_seq(g->stream, fn, dim3(nparts), E::kThreads, E::smem, in, dout, part, g->L, kPartImages, nimg);
    }
    sum_add(sums, part, nparts, n, gw, 0);
    if (int rc = cuda_check(cudaGetLastError(), "k_gen_wgrad")) return rc;
    return gb ? bgrad_launch(g, dout, nimg, COUT, gb, sums) : NMMC_OK;
}

// The weights' compute forms, after one Adam step where `step` says so.
int update_weights(nmmc_gen* g, const UpdateArgs* step) {
    UpdateArgs u{};
    if (step) u = *step;
    u.adam = step != nullptr;
    int most = 0;
    for (int l = 0; l < kGenLayers; ++l) {
        u.layer[l] = g->layer[l];
        most = std::max(most, (int)g->layer[l].nw() + g->layer[l].cout);
    }
    launch_seq(g->stream, k_gen_update, dim3((most + 127) / 128, kGenLayers), 128, 0, u);
    return cuda_check(cudaGetLastError(), "k_gen_update");
}

int ensure_batch(nmmc_gen* g, int b) {
    if (b <= g->bcap) return NMMC_OK;
    for (int l = 0; l < kGenLayers; ++l) cudaFree(g->act[l]);
    cudaFree(g->vout);
    cudaFree(g->target);
    cudaFree(g->g0);
    cudaFree(g->g1);
    cudaFree(g->gv);
    cudaFree(g->wpart);
    cudaFree(g->d_idx);
    cudaFree(g->d_sig);
    cudaFree(g->d_cnd);
    const size_t np = (size_t)b * g->L * g->L;
    NMMC_CUDA(cudaMalloc(&g->act[0], np * kGenCin0 * sizeof(__nv_bfloat16)));
    for (int l = 1; l < kGenLayers; ++l) NMMC_CUDA(cudaMalloc(&g->act[l], np * kGenC * sizeof(__nv_bfloat16)));
    NMMC_CUDA(cudaMalloc(&g->vout, np * kGenCout * sizeof(float)));
    NMMC_CUDA(cudaMalloc(&g->target, np * kGenCout * sizeof(float)));
    NMMC_CUDA(cudaMalloc(&g->g0, np * kGenC * sizeof(float)));
    NMMC_CUDA(cudaMalloc(&g->g1, np * kGenC * sizeof(float)));
    NMMC_CUDA(cudaMalloc(&g->gv, np * kGenCout * sizeof(float)));
    // the partials of one hidden layer on the FMA pipes, or of all on the tensor cores; beside them those
    // of the edge layers and of the biases
    const size_t parts = tile_parts(g->L, b), tc_parts = std::min<size_t>(parts, std::max(1, g->sm_count));
    g->wpart_cap = std::max(parts, (kGenLayers - 2) * tc_parts) * wg::kPart + parts * 9 * kGenC * (kGenCin0 + kGenCout) +
                   (size_t)bias_shape(g, b).nblk * kGenLayers * kGenC;
    NMMC_CUDA(cudaMalloc(&g->wpart, g->wpart_cap * sizeof(float)));
    NMMC_CUDA(cudaMalloc(&g->d_idx, sizeof(int) * b));
    NMMC_CUDA(cudaMalloc(&g->d_sig, sizeof(float) * b));
    NMMC_CUDA(cudaMalloc(&g->d_cnd, sizeof(float) * 3 * b));
    g->bcap = b;
    return NMMC_OK;
}

// forward pass of nb images from act[0]; leaves act[1..7] and vout
int forward(nmmc_gen* g, int nb) {
    int rc;
    GenLayer* y = g->layer;
    rc = edge_layers_on_tc(g)
             ? conv_row_launch<0, 1, 2, kGenC>(g, g->act[0], y[0].wb, y[0].b, nullptr, g->act[1], nb, y[0].wimg)
             : conv_launch<kGenCin0, kGenC, __nv_bfloat16, 0>(g, g->act[0], y[0].wb, y[0].b, nullptr, 0, g->act[1], nb);
    if (rc) return rc;
    for (int l = 1; l < kGenLayers - 1; ++l) {
        rc = g->use_tc ? conv_tc_launch<0>(g, g->act[l], y[l].wb, y[l].b, nullptr, g->act[l + 1], nb, y[l].wimg)
                       : conv_launch<kGenC, kGenC, __nv_bfloat16, 0>(g, g->act[l], y[l].wb, y[l].b, nullptr, 0,
                                                                    g->act[l + 1], nb);
        if (rc) return rc;
    }
    const GenLayer& yl = y[kGenLayers - 1];
    if (edge_layers_on_tc(g))
        return conv_row_launch<3, 6, 6, kGenCout>(g, g->act[kGenLayers - 1], yl.wb, yl.b, nullptr, g->vout, nb,
                                                  yl.wimg);
    return conv_launch<kGenC, kGenCout, __nv_bfloat16, 1>(g, g->act[kGenLayers - 1], yl.wb, yl.b, nullptr, 0, g->vout, nb);
}

// backward from gv (dL/dv): fills gw/gb of every layer
int backward(nmmc_gen* g, int nb) {
    int rc;
    GenLayer* y = g->layer;
    const int last = kGenLayers - 1;
    SumArgs sums;
    // last layer: weights and bias, then data gradient into g0 (masked by act[last] > 0)
    if ((rc = wgrad_launch<kGenC, kGenCout>(g, g->act[last], g->gv, y[last].gw, y[last].gb, nb, sums))) return rc;
    if ((rc = conv_launch<kGenCout, kGenC, float, 2>(g, g->gv, y[last].wt, nullptr, g->act[last], kGenC, g->g0, nb)))
        return rc;
    float* cur = g->g0;
    float* nxt = g->g1;
    for (int l = last - 1; l >= 1; --l) {
        if ((rc = wgrad_launch<kGenC, kGenC>(g, g->act[l], cur, y[l].gw, y[l].gb, nb, sums))) return rc;
        rc = g->use_tc ? conv_tc_launch<2>(g, cur, y[l].wt, nullptr, g->act[l], nxt, nb, y[l].wtimg)
                       : conv_launch<kGenC, kGenC, float, 2>(g, cur, y[l].wt, nullptr, g->act[l], kGenC, nxt, nb);
        if (rc) return rc;
        float* t = cur;
        cur = nxt;
        nxt = t;
    }
    if ((rc = wgrad_launch<kGenCin0, kGenC>(g, g->act[0], cur, y[0].gw, y[0].gb, nb, sums))) return rc;
    return launch_sums(g, sums);
}

void free_gen(nmmc_gen* g) {
    if (!g) return;
    for (int l = 0; l < kGenLayers; ++l) {
        GenLayer& y = g->layer[l];
        cudaFree(y.w);
        cudaFree(y.b);
        cudaFree(y.wb);
        cudaFree(y.wt);
        cudaFree(y.wimg);
        cudaFree(y.wtimg);
        cudaFree(y.mw);
        cudaFree(y.vw);
        cudaFree(y.mb);
        cudaFree(y.vb);
        cudaFree(g->act[l]);
    }
    cudaFree(g->grads);
    cudaFree(g->snaps);
    cudaFree(g->cond);
    cudaFree(g->vout);
    cudaFree(g->target);
    cudaFree(g->g0);
    cudaFree(g->g1);
    cudaFree(g->gv);
    cudaFree(g->wpart);
    cudaFree(g->d_idx);
    cudaFree(g->d_sig);
    cudaFree(g->d_cnd);
    cudaFree(g->d_loss);
    cudaFree(g->d_flag);
    if (g->stream) cudaStreamDestroy(g->stream);
    delete g;
}

}  // namespace
}  // namespace nmmc

using namespace nmmc;
struct nmmc_ctx : public nmmc::Ctx {};

extern "C" {

int nmmc_gen_create(int L, int capacity, uint64_t seed, nmmc_gen** out) {
    if (!out || L < kTile || L % kTile || capacity < 0) return set_error(NMMC_ERR_ARG, "L must be a multiple of 16");
    *out = nullptr;
    nmmc_gen* g = new nmmc_gen();
    g->L = L;
    g->seed = seed;
    g->cap = capacity;
#define NMMC_GTRY(call)                                  \
    do {                                                 \
        cudaError_t _e = (call);                         \
        if (_e != cudaSuccess) {                         \
            int _rc = cuda_check(_e, #call);             \
            free_gen(g);                                 \
            return _rc;                                  \
        }                                                \
    } while (0)
    NMMC_GTRY(cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
    for (int l = 0; l < kGenLayers; ++l) {
        g->layer[l].cin = (l == 0) ? kGenCin0 : kGenC;
        g->layer[l].cout = (l == kGenLayers - 1) ? kGenCout : kGenC;
    }
    NMMC_GTRY(cudaMalloc(&g->grads, (size_t)nmmc_gen_param_count(g) * sizeof(float)));
    size_t goff = 0;
    // He-style initialisation from Philox (host)
    for (int l = 0; l < kGenLayers; ++l) {
        GenLayer& y = g->layer[l];
        y.cin = (l == 0) ? kGenCin0 : kGenC;
        y.cout = (l == kGenLayers - 1) ? kGenCout : kGenC;
        const size_t n = y.nw();
        std::vector<float> w(n), b(y.cout, 0.0f);
        const float sd = sqrtf(2.0f / (9.0f * y.cin)) * (l == kGenLayers - 1 ? 0.5f : 1.0f);
        for (size_t i = 0; i < n; ++i) {
            nmmc_u4 r = nmmc_philox((uint32_t)i, (uint32_t)l, NMMC_STREAM_NOISE << 28, 7u, (uint32_t)seed,
                                    (uint32_t)(seed >> 32));
            const double u1 = ((double)r.x + 0.5) / 4294967296.0, u2 = ((double)r.y + 0.5) / 4294967296.0;
            w[i] = (float)(sd * sqrt(-2.0 * log(u1)) * cos(2.0 * M_PI * u2));
            const int co = (int)(i % y.cout);
            if (l == kGenLayers - 1 && co == 3) w[i] = 0.0f;   // padding channel
        }
        NMMC_GTRY(cudaMalloc(&y.w, n * sizeof(float)));
        NMMC_GTRY(cudaMalloc(&y.b, y.cout * sizeof(float)));
        NMMC_GTRY(cudaMalloc(&y.wb, n * sizeof(__nv_bfloat16)));
        NMMC_GTRY(cudaMalloc(&y.wt, n * sizeof(__nv_bfloat16)));
        y.kch = l == 0 ? 2 : kGenC / 8;   // the first layer's 8 channels are one chunk of the two of K = 16
        NMMC_GTRY(cudaMalloc(&y.wimg, kWimgBytes));
        NMMC_GTRY(cudaMemset(y.wimg, 0, kWimgBytes));
        if (l > 0 && l < kGenLayers - 1) NMMC_GTRY(cudaMalloc(&y.wtimg, 2 * kWimgBytes));
        y.gw = g->grads + goff;
        y.gb = y.gw + n;
        goff += n + y.cout;
        NMMC_GTRY(cudaMalloc(&y.mw, n * sizeof(float)));
        NMMC_GTRY(cudaMalloc(&y.vw, n * sizeof(float)));
        NMMC_GTRY(cudaMalloc(&y.mb, y.cout * sizeof(float)));
        NMMC_GTRY(cudaMalloc(&y.vb, y.cout * sizeof(float)));
        NMMC_GTRY(cudaMemcpy(y.w, w.data(), n * sizeof(float), cudaMemcpyHostToDevice));
        NMMC_GTRY(cudaMemcpy(y.b, b.data(), y.cout * sizeof(float), cudaMemcpyHostToDevice));
        NMMC_GTRY(cudaMemset(y.mw, 0, n * sizeof(float)));
        NMMC_GTRY(cudaMemset(y.vw, 0, n * sizeof(float)));
        NMMC_GTRY(cudaMemset(y.mb, 0, y.cout * sizeof(float)));
        NMMC_GTRY(cudaMemset(y.vb, 0, y.cout * sizeof(float)));
    }
    if (capacity > 0) {
        NMMC_GTRY(cudaMalloc(&g->snaps, (size_t)capacity * L * L * 3 * sizeof(__nv_bfloat16)));
        NMMC_GTRY(cudaMalloc(&g->cond, (size_t)capacity * 3 * sizeof(float)));
    }
    NMMC_GTRY(cudaMalloc(&g->d_loss, sizeof(double)));
    NMMC_GTRY(cudaMalloc(&g->d_flag, sizeof(int)));
    NMMC_GTRY(cudaMemset(g->d_flag, 0, sizeof(int)));
    {
        int dev = 0;
        NMMC_GTRY(cudaGetDevice(&dev));
        NMMC_GTRY(cudaDeviceGetAttribute(&g->sm_count, cudaDevAttrMultiProcessorCount, dev));
        NMMC_GTRY(cudaDeviceGetAttribute(&g->smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    }
#undef NMMC_GTRY
    int rc = update_weights(g, nullptr);
    if (!rc) rc = cuda_check(cudaStreamSynchronize(g->stream), "nmmc_gen_create");
    if (rc) {
        free_gen(g);
        return rc;
    }
    *out = g;
    return NMMC_OK;
}

void nmmc_gen_destroy(nmmc_gen* g) {
    if (g) cudaStreamSynchronize(g->stream);
    free_gen(g);
}

int nmmc_gen_param_count(const nmmc_gen* g) {
    if (!g) return 0;
    size_t n = 0;
    for (int l = 0; l < kGenLayers; ++l) n += g->layer[l].nw() + g->layer[l].cout;
    return (int)n;
}

// parameters in layer order: W [9][cin][cout] then b [cout]
int nmmc_gen_get_params(nmmc_gen* g, float* out, int n) {
    if (!g || !out || n != nmmc_gen_param_count(g)) return set_error(NMMC_ERR_ARG, "bad parameter buffer");
    NMMC_CUDA(cudaStreamSynchronize(g->stream));
    size_t o = 0;
    for (int l = 0; l < kGenLayers; ++l) {
        GenLayer& y = g->layer[l];
        NMMC_CUDA(cudaMemcpy(out + o, y.w, y.nw() * sizeof(float), cudaMemcpyDeviceToHost));
        o += y.nw();
        NMMC_CUDA(cudaMemcpy(out + o, y.b, y.cout * sizeof(float), cudaMemcpyDeviceToHost));
        o += y.cout;
    }
    return NMMC_OK;
}

int nmmc_gen_set_params(nmmc_gen* g, const float* in, int n) {
    if (!g || !in || n != nmmc_gen_param_count(g)) return set_error(NMMC_ERR_ARG, "bad parameter buffer");
    NMMC_CUDA(cudaStreamSynchronize(g->stream));
    size_t o = 0;
    for (int l = 0; l < kGenLayers; ++l) {
        GenLayer& y = g->layer[l];
        NMMC_CUDA(cudaMemcpy(y.w, in + o, y.nw() * sizeof(float), cudaMemcpyHostToDevice));
        o += y.nw();
        NMMC_CUDA(cudaMemcpy(y.b, in + o, y.cout * sizeof(float), cudaMemcpyHostToDevice));
        o += y.cout;
    }
    return update_weights(g, nullptr);
}

// Snapshots of 2-D Heisenberg chains of `ctx` (edge == generator L) with their (T, B, D).
int nmmc_gen_add_snapshots(nmmc_gen* g, nmmc_ctx* c, const int* chains, int n, const double* cond) {
    if (!g || !c || !chains || !cond || n <= 0) return set_error(NMMC_ERR_ARG, "bad argument");
    if (c->dim != 2 || c->ising || c->edge != g->L || c->masked)
        return set_error(NMMC_ERR_UNSUPPORTED, "snapshots must come from unmasked 2-D Heisenberg lattices of edge %d", g->L);
    if (g->count + n > g->cap) return set_error(NMMC_ERR_ARG, "dataset capacity %d exceeded", g->cap);
    for (int i = 0; i < n; ++i)
        if (chains[i] < 0 || chains[i] >= c->nchains) return set_error(NMMC_ERR_ARG, "chain index out of range");
    DeviceScratch ds;
    int* d_ch = nullptr;
    NMMC_CUDA(ds.alloc(&d_ch, sizeof(int) * n));
    std::vector<float> cf(3 * (size_t)n);
    for (size_t i = 0; i < cf.size(); ++i) cf[i] = (float)cond[i];
    NMMC_CUDA(cudaStreamSynchronize(c->stream));
    NMMC_CUDA(cudaMemcpy(d_ch, chains, sizeof(int) * n, cudaMemcpyHostToDevice));
    NMMC_CUDA(cudaMemcpy(g->cond + 3 * (size_t)g->count, cf.data(), cf.size() * sizeof(float), cudaMemcpyHostToDevice));
    dim3 grid((g->L * g->L + 255) / 256, n);
    k_gen_from_chain<<<grid, 256, 0, g->stream>>>(c->m, (const float*)c->d_spins, d_ch, g->snaps, g->count);
    int rc = cuda_check(cudaStreamSynchronize(g->stream), "k_gen_from_chain");
    if (rc) return rc;
    g->count += n;
    return NMMC_OK;
}

int nmmc_gen_dataset_size(const nmmc_gen* g) { return g ? g->count : 0; }

// One optimisation step per batch: idx[b] snapshot indices, sig[b] noise levels. Returns the
// batch loss. lr <= 0 computes loss and gradients without updating (gradient checks).
int nmmc_gen_train_step(nmmc_gen* g, const int* idx, const float* sig, int nb, float lr, double* loss) {
    if (!g || !idx || !sig || nb <= 0) return set_error(NMMC_ERR_ARG, "bad argument");
    for (int i = 0; i < nb; ++i)
        if (idx[i] < 0 || idx[i] >= g->count) return set_error(NMMC_ERR_ARG, "snapshot index %d out of range", idx[i]);
    int rc = ensure_batch(g, nb);
    if (rc) return rc;
    NMMC_CUDA(cudaMemcpyAsync(g->d_idx, idx, sizeof(int) * nb, cudaMemcpyHostToDevice, g->stream));
    NMMC_CUDA(cudaMemcpyAsync(g->d_sig, sig, sizeof(float) * nb, cudaMemcpyHostToDevice, g->stream));
    const int npix = g->L * g->L;
    dim3 gi((npix + 255) / 256, nb);
    launch_seq(g->stream, k_gen_input, dim3(gi), 256, 0, 0, g->snaps, g->d_idx, nullptr, g->d_sig, g->cond, g->L, (uint32_t)g->seed,
                                           (uint32_t)(g->seed >> 32), g->draws, g->act[0], g->target, 1.0f);
    g->draws += (unsigned long long)nb;
    if ((rc = forward(g, nb))) return rc;
    NMMC_CUDA(cudaMemsetAsync(g->d_loss, 0, sizeof(double), g->stream));
    const int np = nb * npix;
    launch_seq(g->stream, k_gen_head, dim3((np + 255) / 256), 256, 0, g->vout, g->target, np, 1.0f / (float)np, g->gv, g->d_loss);
    if ((rc = backward(g, nb))) return rc;
    if (lr > 0) {
        g->adam_t++;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.0f - powf(b1, (float)g->adam_t), c2 = 1.0f - powf(b2, (float)g->adam_t);
        UpdateArgs u{};
        u.lr = lr;
        u.b1 = b1;
        u.b2 = b2;
        u.c1 = c1;
        u.c2 = c2;
        u.eps = 1e-8f;
        if ((rc = update_weights(g, &u))) return rc;
    }
    double l = 0;
    NMMC_CUDA(cudaMemcpyAsync(&l, g->d_loss, sizeof(double), cudaMemcpyDeviceToHost, g->stream));
    NMMC_CUDA(cudaStreamSynchronize(g->stream));
    if ((rc = check_flag(g))) return rc;
    if (loss) *loss = l;
    return NMMC_OK;
}

// Gradients of the last train step (lr <= 0 keeps them for inspection), parameter order.
int nmmc_gen_get_grads(nmmc_gen* g, float* out, int n) {
    if (!g || !out || n != nmmc_gen_param_count(g)) return set_error(NMMC_ERR_ARG, "bad parameter buffer");
    NMMC_CUDA(cudaStreamSynchronize(g->stream));
    NMMC_CUDA(cudaMemcpy(out, g->grads, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost));
    return NMMC_OK;
}

// Network input of the last step (BF16 values as float), [nb][L][L][8], for checks.
int nmmc_gen_get_input(nmmc_gen* g, int nb, float* out) {
    if (!g || !out || nb <= 0 || nb > g->bcap) return set_error(NMMC_ERR_ARG, "bad argument");
    const size_t n = (size_t)nb * g->L * g->L * kGenCin0;
    std::vector<__nv_bfloat16> h(n);
    NMMC_CUDA(cudaStreamSynchronize(g->stream));
    NMMC_CUDA(cudaMemcpy(h.data(), g->act[0], n * sizeof(__nv_bfloat16), cudaMemcpyDeviceToHost));
    for (size_t i = 0; i < n; ++i) out[i] = __bfloat162float(h[i]);
    return NMMC_OK;
}

// Warm start: for each listed chain of `ctx` (2-D Heisenberg, edge L), start from uniform
// random spins and run `steps` denoising passes at noise levels s_k = 1 - k/steps (k = 0 ..
// steps-1), re-noising the estimate to s_{k+1} between passes; the final estimate replaces
// the chain's spins. cond: (T, B, D) per chain.
int nmmc_gen_warm_start(nmmc_gen* g, nmmc_ctx* c, const int* chains, int n, const double* cond, int steps,
                        int reuse_noise) {
    if (!g || !c || !chains || !cond || n <= 0 || steps <= 0) return set_error(NMMC_ERR_ARG, "bad argument");
    if (c->dim != 2 || c->ising || c->edge != g->L || c->masked)
        return set_error(NMMC_ERR_UNSUPPORTED, "warm starts need unmasked 2-D Heisenberg lattices of edge %d", g->L);
    for (int i = 0; i < n; ++i)
        if (chains[i] < 0 || chains[i] >= c->nchains) return set_error(NMMC_ERR_ARG, "chain index out of range");
    int rc = ensure_batch(g, n);
    if (rc) return rc;
    const int npix = g->L * g->L;
    float* cur = g->target;   // the current estimate lives in the target buffer
    NMMC_CUDA(cudaMemsetAsync(cur, 0, (size_t)n * npix * kGenCout * sizeof(float), g->stream));
    std::vector<float> cf(3 * (size_t)n);
    for (size_t i = 0; i < cf.size(); ++i) cf[i] = (float)cond[i];
    NMMC_CUDA(cudaMemcpyAsync(g->d_cnd, cf.data(), cf.size() * sizeof(float), cudaMemcpyHostToDevice, g->stream));
    dim3 gi((npix + 255) / 256, n);
    // every pass's noise level goes up in one copy, so the passes run back to back with no
    // host synchronisation between them
    DeviceScratch ds;
    float* d_sigs = nullptr;
    NMMC_CUDA(ds.alloc(&d_sigs, sizeof(float) * (size_t)steps * n));
    std::vector<float> sall((size_t)steps * n);
    // noise level of pass k: linear 1 - k/steps, quadratic (1 - k/steps)^2 (more passes at low
    // noise, where the fine structure forms), or cos(pi/2 k/steps)
    const int sch = g->schedule;
    auto sched = [&](int k) -> float {
        const float f = (float)k / (float)steps;
        if (sch == 1) return (1.0f - f) * (1.0f - f);
        if (sch == 2) return cosf(1.57079632679f * f);
        return 1.0f - f;
    };
    for (int k = 0; k < steps; ++k)
        for (int i = 0; i < n; ++i) sall[(size_t)k * n + i] = sched(k);
    NMMC_CUDA(cudaMemcpyAsync(d_sigs, sall.data(), sizeof(float) * sall.size(), cudaMemcpyHostToDevice, g->stream));
    float s_prev = 1.0f;
    for (int k = 0; k < steps; ++k) {
        const float s = sched(k);
        launch_seq(g->stream, k_gen_input, dim3(gi), 256, 0, reuse_noise == 2 ? 3 : (reuse_noise ? 2 : 1), nullptr, nullptr, cur,
                                               d_sigs + (size_t)k * n, g->d_cnd, g->L,
                                               (uint32_t)g->seed, (uint32_t)(g->seed >> 32), g->draws, g->act[0],
                                               nullptr, k == 0 ? 1.0f : s_prev);
        s_prev = s;
        g->draws += (unsigned long long)n;
        if ((rc = forward(g, n))) return rc;
        launch_seq(g->stream, k_gen_normalise, dim3((n * npix + 255) / 256), 256, 0, g->vout, n * npix, cur);
    }
    int* d_ch = nullptr;
    NMMC_CUDA(ds.alloc(&d_ch, sizeof(int) * n));
    NMMC_CUDA(cudaMemcpy(d_ch, chains, sizeof(int) * n, cudaMemcpyHostToDevice));
    NMMC_CUDA(cudaStreamSynchronize(c->stream));
    k_gen_to_chain<<<gi, 256, 0, g->stream>>>(c->m, (float*)c->d_spins, d_ch, cur);
    rc = cuda_check(cudaStreamSynchronize(g->stream), "k_gen_to_chain");
    return rc ? rc : check_flag(g);
}

// One layer's convolution of caller data, for checks: layer 0 (8 -> 48 channels), 1..6
// (48 -> 48) or 7 (48 -> 4); in [nimg][L][L][cin] (rounded to BF16 here), out
// [nimg][L][L][cout] FP32 = conv + bias, no activation; tensor != 0 runs the layer as the
// generator does on the tensor cores (the first and last layers only at L = 128, the FMA
// pipes otherwise), 0 on the FP32 FMA pipes.
int nmmc_gen_probe_conv(nmmc_gen* g, int layer, int nimg, const float* in, float* out, int tensor) {
    if (!g || !in || !out || layer < 0 || layer > kGenLayers - 1 || nimg <= 0) return set_error(NMMC_ERR_ARG, "bad argument");
    const int cin = layer == 0 ? kGenCin0 : kGenC, cout = layer == kGenLayers - 1 ? kGenCout : kGenC;
    const size_t LL = (size_t)g->L * g->L, ni = (size_t)nimg * LL * cin, no = (size_t)nimg * LL * cout;
    std::vector<__nv_bfloat16> h(ni);   // [img][pixel][cin] -> chunk-planar
    for (size_t i = 0; i < ni; ++i) {
        const size_t img = i / (LL * cin), r = i - img * LL * cin, pp = r / cin;
        h[pl_off<__nv_bfloat16>(cin, LL, img, pp, (int)(r - pp * cin))] = __float2bfloat16(in[i]);
    }
    DeviceScratch ds;
    __nv_bfloat16* d_in = nullptr;
    float* d_out = nullptr;
    NMMC_CUDA(cudaStreamSynchronize(g->stream));
    NMMC_CUDA(ds.alloc(&d_in, ni * sizeof(__nv_bfloat16)));
    NMMC_CUDA(ds.alloc(&d_out, no * sizeof(float)));
    int rc = cuda_check(cudaMemcpy(d_in, h.data(), ni * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice), "probe H2D");
    const GenLayer& y = g->layer[layer];
    const bool tc_edge = tensor && edge_layers_on_tc(g);
    if (rc) {
    } else if (layer == 0) {
        rc = tc_edge ? conv_row_launch<1, 1, 2, kGenC>(g, d_in, y.wb, y.b, nullptr, d_out, nimg, y.wimg)
                     : conv_launch<kGenCin0, kGenC, __nv_bfloat16, 1>(g, d_in, y.wb, y.b, nullptr, 0, d_out, nimg);
    } else if (layer == kGenLayers - 1) {
        rc = tc_edge ? conv_row_launch<3, 6, 6, kGenCout>(g, d_in, y.wb, y.b, nullptr, d_out, nimg, y.wimg)
                     : conv_launch<kGenC, kGenCout, __nv_bfloat16, 1>(g, d_in, y.wb, y.b, nullptr, 0, d_out, nimg);
    } else {
        rc = tensor ? conv_tc_launch<1>(g, d_in, y.wb, y.b, nullptr, d_out, nimg, y.wimg)
                    : conv_launch<kGenC, kGenC, __nv_bfloat16, 1>(g, d_in, y.wb, y.b, nullptr, 0, d_out, nimg);
    }
    if (!rc) rc = cuda_check(cudaStreamSynchronize(g->stream), "probe conv");
    if (!rc) rc = check_flag(g);
    std::vector<float> ho(rc ? 0 : no);
    if (!rc) rc = cuda_check(cudaMemcpy(ho.data(), d_out, no * sizeof(float), cudaMemcpyDeviceToHost), "probe D2H");
    if (!rc)
        for (size_t i = 0; i < no; ++i) {   // chunk-planar -> [img][pixel][cout]
            const size_t img = i / (LL * cout), r = i - img * LL * cout, pp = r / cout;
            out[i] = ho[pl_off<float>(cout, LL, img, pp, (int)(r - pp * cout))];
        }
    return rc;
}

int nmmc_gen_probe_wgrad(nmmc_gen* g, int nimg, const float* in, const float* dout, float* gw, int tensor) {
    if (!g || !in || !dout || !gw || nimg <= 0) return set_error(NMMC_ERR_ARG, "bad argument");
    if (nimg > g->bcap) {
        if (int rc = ensure_batch(g, nimg)) return rc;
    }
    const int C = kGenC;
    const size_t LL = (size_t)g->L * g->L, ne = (size_t)nimg * LL * C;
    std::vector<__nv_bfloat16> hi(ne);
    std::vector<float> hg(ne);
    for (size_t i = 0; i < ne; ++i) {   // [img][pixel][c] -> chunk-planar
        const size_t img = i / (LL * C), r = i - img * LL * C, pp = r / C;
        hi[pl_off<__nv_bfloat16>(C, LL, img, pp, (int)(r - pp * C))] = __float2bfloat16(in[i]);
        hg[pl_off<float>(C, LL, img, pp, (int)(r - pp * C))] = dout[i];
    }
    DeviceScratch ds;
    __nv_bfloat16* d_in = nullptr;
    float *d_g = nullptr, *d_w = nullptr;
    NMMC_CUDA(cudaStreamSynchronize(g->stream));
    NMMC_CUDA(ds.alloc(&d_in, ne * sizeof(__nv_bfloat16)));
    NMMC_CUDA(ds.alloc(&d_g, ne * sizeof(float)));
    NMMC_CUDA(ds.alloc(&d_w, (size_t)9 * C * C * sizeof(float)));
    int rc = cuda_check(cudaMemcpy(d_in, hi.data(), ne * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice), "probe H2D");
    if (!rc) rc = cuda_check(cudaMemcpy(d_g, hg.data(), ne * sizeof(float), cudaMemcpyHostToDevice), "probe H2D");
    const int keep = g->use_tc;
    g->use_tc = tensor ? 1 : 0;
    SumArgs sums;
    if (!rc) rc = wgrad_launch<kGenC, kGenC>(g, d_in, d_g, d_w, nullptr, nimg, sums);
    if (!rc) rc = launch_sums(g, sums);
    g->use_tc = keep;
    if (!rc) rc = cuda_check(cudaStreamSynchronize(g->stream), "probe wgrad");
    if (!rc) rc = check_flag(g);
    if (!rc) rc = cuda_check(cudaMemcpy(gw, d_w, (size_t)9 * C * C * sizeof(float), cudaMemcpyDeviceToHost), "probe D2H");
    return rc;
}

int nmmc_gen_set_option(nmmc_gen* g, int key, int64_t v) {
    if (!g) return set_error(NMMC_ERR_ARG, "null generator");
    if (key == NMMC_GEN_OPT_TENSOR_CORES) {
        if (v < 0 || v > 4) return set_error(NMMC_ERR_ARG, "tensor-core option must be 0 .. 4");
        NMMC_CUDA(cudaStreamSynchronize(g->stream));
        g->use_tc = v ? 1 : 0;
        g->use_ws = (v == 2) ? 1 : 0;
        g->use_rows = v != 3;   // 4: the same kernels as 1
        return NMMC_OK;
    }
    if (key == NMMC_GEN_OPT_SCHEDULE) {
        if (v < 0 || v > 2) return set_error(NMMC_ERR_ARG, "schedule must be 0, 1 or 2");
        g->schedule = (int)v;
        return NMMC_OK;
    }
    if (key == NMMC_GEN_OPT_WEIGHT_IMAGE) {
        if (v != 0 && v != 1) return set_error(NMMC_ERR_ARG, "weight image must be 0 or 1");
        NMMC_CUDA(cudaStreamSynchronize(g->stream));
        g->use_wimg = (int)v;
        return NMMC_OK;
    }
    if (key == NMMC_GEN_OPT_TILE_ROWS) {
        if (v != 1 && v != 2) return set_error(NMMC_ERR_ARG, "tile rows must be 1 or 2");
        return NMMC_OK;   // the L = 128 kernels take one row per tile in either case
    }
    return set_error(NMMC_ERR_ARG, "unknown generator option %d", key);
}

int nmmc_gen_save(nmmc_gen* g, const char* path) {
    if (!g || !path) return set_error(NMMC_ERR_ARG, "bad argument");
    const int n = nmmc_gen_param_count(g);
    std::vector<float> p(n);
    int rc = nmmc_gen_get_params(g, p.data(), n);
    if (rc) return rc;
    FILE* f = fopen(path, "wb");
    if (!f) return set_error(NMMC_ERR_IO, "cannot write %s", path);
    const int hdr[4] = {0x4e4d4d47, g->L, kGenLayers, n};
    bool ok = fwrite(hdr, sizeof hdr, 1, f) == 1 && fwrite(p.data(), sizeof(float), n, f) == (size_t)n;
    ok = (fclose(f) == 0) && ok;
    return ok ? NMMC_OK : set_error(NMMC_ERR_IO, "short write to %s", path);
}

int nmmc_gen_load(nmmc_gen* g, const char* path) {
    if (!g || !path) return set_error(NMMC_ERR_ARG, "bad argument");
    FILE* f = fopen(path, "rb");
    if (!f) return set_error(NMMC_ERR_IO, "cannot read %s", path);
    int hdr[4];
    const int n = nmmc_gen_param_count(g);
    std::vector<float> p(n);
    bool ok = fread(hdr, sizeof hdr, 1, f) == 1 && hdr[0] == 0x4e4d4d47 && hdr[2] == kGenLayers && hdr[3] == n &&
              fread(p.data(), sizeof(float), n, f) == (size_t)n;
    fclose(f);
    if (!ok) return set_error(NMMC_ERR_IO, "%s is not a generator of this shape", path);
    return nmmc_gen_set_params(g, p.data(), n);
}

}  // extern "C"
