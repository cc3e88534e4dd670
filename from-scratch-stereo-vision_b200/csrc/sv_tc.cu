// sv_tc.cu -- BF16 implicit-GEMM convolutions on the sm_100a tensor cores
// (tcgen05.mma, FP32 accumulator in tensor memory) for the network's BF16
// path: the feature tower's 2-D convolutions (FeatureNet, stereonet.py:
// 1022-1070) and the cost filter's first two 3-D convolutions (CostFilter,
// 1071-1109), the first one fused with the cost volume (CostVolume,
// 740-842).
//
// GEMM view: M = output positions (a CTA tile of 128), N = output channels
// padded to 16, K = input channels x taps padded to a multiple of 16.
//  * B (weights) is packed once at checkpoint upload into the canonical
//    K-major, no-swizzle UMMA layout (8 x 16-byte core matrices, 128
//    contiguous bytes each) and copied to shared memory once per CTA;
//  * A (the im2col tile) is gathered from an input patch in shared memory
//    straight into that layout -- one output row per thread, in 16-byte
//    chunks of 8 consecutive k -- and fenced into the async proxy;
//  * one thread issues Kpad/16 tcgen05.mma (M=128, N=16, K=16) into a
//    32-column tensor-memory accumulator and commits them to an mbarrier;
//  * each warp reads its 32 accumulator rows back with tcgen05.ld
//    (32x32b.x16) and applies bias + activation.
// CTAs are persistent over tiles.  Every mbarrier wait is bounded: on
// timeout the kernel records SV_ERR_CUDA, stops and still frees its tensor
// memory.

#include <cuda_bf16.h>

#include <mutex>
#include <type_traits>

#include "sv_common.cuh"
#include "sv_tc.cuh"

namespace sv {

namespace {

constexpr int kTcM = 128, kTcN = 16, kTmemCols = 32;
constexpr int kTcMaxK = 432;                  // 16 channels x 27 taps
constexpr unsigned kWaitLimit = 1u << 24;     // polls before a wait is declared failed

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// UMMA shared-memory descriptor, K-major without swizzle: start address,
// leading byte offset (between the two 8-element K halves of one MMA),
// stride byte offset (between 8-row groups), all >> 4; version 1 (sm_100).
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// kind::f16 instruction descriptor: D F32 (bits 4-5 = 1), A and B BF16
// (bits 7-9 = 1, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
constexpr uint32_t kIdescBf16 = (1u << 4) | (1u << 7) | (1u << 10) |
                                ((uint32_t)(kTcN >> 3) << 17) | ((uint32_t)(kTcM >> 4) << 24);

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

// Bounded wait for phase `parity` of the barrier; true when it completed.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity,
                                          unsigned limit = kWaitLimit) {
    const uint32_t a = smem_u32(bar);
    for (unsigned it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

}  // namespace

// 3x3x3 convolutions, stride 1, same padding: of a tensor (mode 0) or of the cost
// volume of two feature maps, made here (mode 1).  A tile is one disparity of
// 4 rows x 32 columns, and a CTA walks the disparities of one place in order: a
// ring of three planes (every channel, 6 x 34 values with the halo) in shared
// memory as BF16, the plane after next read from memory while the operand of this
// one is built.  Operand A is the im2col tile, two threads per row, K halves
// apart: element k is the ring's at a distance that k and the row's place give,
// known at compile time for the shipped channel counts.  k stays channel-major, 16
// to an MMA, so every output is the same sum as with any other tiling.
// What bounds it is the copy into A, some 600 warp instructions a step and warp.
// At 160 x 120 x 12, fetching each element of A from memory with its own bounds
// tests took 381 us for 12 -> 6 channels and 113 for 6 -> 6; from the ring 41 and 26
// (45 with two-byte reads, 58 when a plane was made as it was read).
constexpr int kC3Threads = 256, kC3Pitch = 36, kC3Rows = 6, kC3W = 32, kC3H = 4;
constexpr int kC3Pairs = 17;            // column pairs of a plane row

// Chunks [G0, G1) of 8 elements of one row of A; b0, b1, b2 are the row's place
// in the ring's planes of taps kd = 0, 1, 2, rounded down to a word.  Six elements
// (two rows of taps, three words of A) come from four words of the ring; odd
// columns pick the other halves (s0, s1, s2).
template <int IC, int G0, int G1>
__device__ __forceinline__ void c3_gather(const unsigned char *b0, const unsigned char *b1,
                                          const unsigned char *b2, unsigned s0, unsigned s1,
                                          unsigned s2, unsigned char *row) {
    static_assert(G0 % 3 == 0, "whole row pairs");
    constexpr int NW = (G1 - G0) * 4;                      // words of A
    uint32_t w[4];
#pragma unroll
    for (int p = 0; p < (NW + 2) / 3; ++p) {
        uint32_t q[2][2] = {};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int t = G0 * 8 / 3 + 2 * p + u;          // row of taps (c, kd, ky)
            if (t >= IC * 9) continue;
            const int c = t / 9, kd = t % 9 / 3, ky = t % 3;
            const unsigned char *b = kd == 0 ? b0 : kd == 1 ? b1 : b2;
            const uint32_t *r = reinterpret_cast<const uint32_t *>(
                b + (c * kC3Rows + ky) * kC3Pitch * 2);
            q[u][0] = r[0];
            q[u][1] = r[1];
        }
        const uint32_t o[3] = {__byte_perm(q[0][0], q[0][1], s0), __byte_perm(q[0][1], q[1][0], s1),
                               __byte_perm(q[1][0], q[1][1], s2)};
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const int n = 3 * p + e;
            if (n >= NW) continue;
            w[n % 4] = o[e];
            if (n % 4 == 3)
                *reinterpret_cast<uint4 *>(row + (size_t)(G0 + n / 4) * (kTcM / 8) * 128) =
                    make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// ICT: the channel count, 0 to read it from the arguments; MODE: a.mode
template <int ICT, int MODE>
__global__ void __launch_bounds__(kC3Threads) k_conv3d_tc(TcConv a, int per_cta) {
    pdl_sync();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    __shared__ int ktab[ICT > 0 ? 1 : kTcMaxK];    // ring offset of k without its plane, and kd
    const int IC = ICT > 0 ? ICT : a.IC;
    const int Kpad = ICT > 0 ? (ICT * 27 + 15) / 16 * 16 : a.Kpad;
    unsigned char *sA = smem;                                   // 128 x Kpad BF16
    unsigned char *sB = smem + (size_t)Kpad * kTcM * 2;          // 16 x Kpad BF16
    __nv_bfloat16 *ring = reinterpret_cast<__nv_bfloat16 *>(sB + (size_t)Kpad * kTcN * 2);
    const int psize = IC * kC3Rows * kC3Pitch;                  // one plane
    const int tid = threadIdx.x, warp = tid >> 5;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    const uint4 *wsrc = reinterpret_cast<const uint4 *>(a.wB);
    uint4 *wdst = reinterpret_cast<uint4 *>(sB);
    for (int i = tid; i < Kpad * kTcN * 2 / 16; i += kC3Threads) wdst[i] = __ldg(wsrc + i);
    if constexpr (ICT == 0)
        for (int k = tid; k < Kpad; k += kC3Threads) {
            const int c = k / 27, t = k - c * 27, kd = t / 9, ky = t % 9 / 3, kx = t % 3;
            ktab[k] = k < a.K ? ((c * kC3Rows + ky) * kC3Pitch + kx) * 4 + kd : -1;
        }
    if (tid == 0) {
        mbar_init(&mbar, 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_slot;

    const int D = a.D, H = a.H, W = a.W;
    const int tx_n = (W + kC3W - 1) / kC3W, ty_n = (H + kC3H - 1) / kC3H;
    const int places = tx_n * ty_n, nb = a.nb > 0 ? a.nb : 1;
    const long steps = (long)places * (MODE == 0 ? a.nimg : 1) * nb * D;
    const long hw = (long)H * W, M = hw * D;
    const int m = tid & 127, my = m >> 5, mx = m & 31;

    // A plane's column pairs, up to kU per thread, their places fixed while the CTA
    // stays at one place: off the pair's offset, at = its column (+ 1) and whether
    // either column is inside.  A plane is read into registers, without a branch or
    // a use before the operand is built, and rounded into the ring after.
    constexpr int kU = ((ICT > 0 ? ICT : 16) * kC3Rows * kC3Pairs + kC3Threads - 1) / kC3Threads;
    const int npairs = IC * kC3Rows * kC3Pairs;
    float2 v[kU], left[MODE == 1 ? kU : 1];
    std::conditional_t<MODE == 0, long, int> off[kU];     // a volume may pass 2^31 values
    int at[kU];
    const float *x0 = nullptr, *x1 = nullptr;
    int ty0 = 0, tx0 = 0;
    auto places_of = [&]() {
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = tid + u * kC3Threads;
            const int r = i / kC3Pairs, xx = tx0 - 1 + 2 * (i - r * kC3Pairs);
            const int c = r / kC3Rows, yy = ty0 - 1 + r - c * kC3Rows;
            const bool row = i < npairs && yy >= 0 && yy < H;
            off[u] = c * (MODE == 0 ? D * hw : hw) + (long)yy * W + xx;
            at[u] = (xx + 1) * 4 + (row && xx >= 0 && xx < W ? 1 : 0) + (row && xx + 1 < W ? 2 : 0);
            if constexpr (MODE == 1) {
                left[u].x = at[u] & 1 ? __ldg(x0 + off[u]) : 0.f;
                left[u].y = at[u] & 2 ? __ldg(x0 + off[u] + 1) : 0.f;
            }
        }
    };
    auto fetch = [&](int z) {
        const bool in = z >= 0 && z < D;
        const float *p = MODE == 0 ? x0 + (in ? z * hw : 0) : x1 - z;
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int xx = (at[u] >> 2) - 1;
            const bool on0 = in && (at[u] & 1) && (MODE == 0 || xx >= z);
            const bool on1 = in && (at[u] & 2) && (MODE == 0 || xx + 1 >= z);
            v[u].x = on0 ? __ldg(p + off[u]) : 0.f;
            v[u].y = on1 ? __ldg(p + off[u] + 1) : 0.f;
        }
    };
    auto put = [&](int z) {
        const bool in = z >= 0 && z < D;
        __nv_bfloat16 *dst = ring + (z + 3) % 3 * psize;
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = tid + u * kC3Threads;
            if (i >= npairs) break;
            const int r = i / kC3Pairs, j = i - r * kC3Pairs;
            float2 f = v[u];
            if constexpr (MODE == 1) {
                const int xx = (at[u] >> 2) - 1;
                f.x = !in || !(at[u] & 1) ? 0.f : xx < z ? 2.0f : fabsf(left[u].x - f.x);
                f.y = !in || !(at[u] & 2) ? 0.f : xx + 1 < z ? 2.0f : fabsf(left[u].y - f.y);
            }
            *reinterpret_cast<__nv_bfloat162 *>(dst + r * kC3Pitch + 2 * j) =
                __floats2bfloat162_rn(f.x, f.y);
        }
    };

    unsigned phase = 0;
    const long s0 = (long)blockIdx.x * per_cta, s1 = min(s0 + per_cta, steps);
    int item = -1, img = 0, bi = 0;
    for (long s = s0; s < s1; ++s) {
        const long place = s / D;
        const int d = (int)(s - place * D);
        if (s == s0 || d == 0) {                           // a new place: its first planes
            item = (int)(place / places);
            const int pl = (int)(place - (long)item * places);
            img = item / nb;
            bi = item - img * nb;
            ty0 = pl / tx_n * kC3H;
            tx0 = pl % tx_n * kC3W;
            x0 = (img ? a.x[1] : a.x[0]) + bi * a.xs;
            x1 = a.x[1] + bi * a.xs;
            places_of();
            for (int z = d - 1; z <= d + 1; ++z) {
                fetch(z);
                put(z);
            }
            __syncthreads();
        }
        const bool more = s + 1 < s1 && d + 1 < D;
        if (more) fetch(d + 2);
        {
            const __nv_bfloat16 *b = ring + my * kC3Pitch + mx;
            const __nv_bfloat16 *b0 = b + (d + 2) % 3 * psize, *b1 = b + d % 3 * psize,
                                *b2 = b + (d + 1) % 3 * psize;
            unsigned char *row = sA + (m >> 3) * 128 + (m & 7) * 16;
            if constexpr (ICT > 0) {
                constexpr int G = (ICT * 27 + 15) / 16 * 2, G2 = (G / 2 + 1) / 3 * 3;
                const unsigned odd = mx & 1;
                const unsigned e0 = odd ? 0x5432 : 0x3210, e1 = odd ? 0x7632 : 0x5410,
                               e2 = odd ? 0x7654 : 0x5432;
                const unsigned char *c0 = reinterpret_cast<const unsigned char *>(b0 - odd),
                                    *c1 = reinterpret_cast<const unsigned char *>(b1 - odd),
                                    *c2 = reinterpret_cast<const unsigned char *>(b2 - odd);
                if (tid < kTcM) c3_gather<ICT, 0, G2>(c0, c1, c2, e0, e1, e2, row);
                else c3_gather<ICT, G2, G>(c0, c1, c2, e0, e1, e2, row);
            } else {
                for (int g = tid >> 7; g < Kpad / 8; g += 2) {
                    __align__(16) __nv_bfloat16 e[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int t = ktab[g * 8 + j], kd = t & 3;
                        const __nv_bfloat16 *p = kd == 0 ? b0 : kd == 1 ? b1 : b2;
                        e[j] = t >= 0 ? p[t >> 2] : __float2bfloat16_rn(0.f);
                    }
                    *reinterpret_cast<uint4 *>(row + (size_t)g * (kTcM / 8) * 128) =
                        *reinterpret_cast<const uint4 *>(e);
                }
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (tid == 0 && !failed) {
            const uint32_t a0 = smem_u32(sA), w0 = smem_u32(sB);
            for (int ks = 0; ks < Kpad / 16; ++ks) {
                const uint64_t da = umma_desc(a0 + ks * 2 * (kTcM / 8) * 128, (kTcM / 8) * 128, 128);
                const uint64_t db = umma_desc(w0 + ks * 2 * (kTcN / 8) * 128, (kTcN / 8) * 128, 128);
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    ::"r"(tmem), "l"(da), "l"(db), "r"(kIdescBf16), "r"(ks));
            }
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                ::"r"(smem_u32(&mbar))
                : "memory");
        }
        if (more) put(d + 2);                              // over plane d - 1, read by all
        // ---- wait for the accumulator (bounded), then the epilogue
        if (!failed && !mbar_wait(&mbar, phase)) {
            failed = 1;
            flag_error(a.err, SV_ERR_TIMEOUT);
        }
        phase ^= 1u;
        __syncthreads();
        if (failed) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (warp < 4) {
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                  "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                  "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(tmem + ((uint32_t)(warp * 32) << 16)));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int oy = ty0 + my, ox = tx0 + mx;
            if (oy < H && ox < W) {
                const long mi = (long)d * hw + (long)oy * W + ox;
                float *y = (img ? a.y[1] : a.y[0]) + bi * a.ys;
                const float *aux = a.aux ? a.aux + bi * a.ys : nullptr;
#pragma unroll
                for (int n = 0; n < kTcN; ++n) {
                    if (n < a.OC) {
                        float f = __uint_as_float(r[n]);
                        if (a.bias) f += __ldg(a.bias + n);
                        if (a.act == 1) f = f > 0.f ? f : f * 0.2f;
                        if (a.act == 2) f = __ldg(aux + (long)n * M + mi) > 0.f ? f : f * 0.2f;
                        y[(long)n * M + mi] = f;
                    }
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem), "r"(kTmemCols));
}

// Element (n, k) of the 16 x Kpad operand B sits in core matrix
// (k / 8, n / 8) -- core matrices ordered k-group-major, 2 per k group --
// at row n % 8 (16 bytes per row), column k % 8.
void tc_pack_weights(const double *w, int OC, int K, uint16_t *out) {
    const int Kpad = tc_kpad(K);
    for (int n = 0; n < kTcN; ++n)
        for (int k = 0; k < Kpad; ++k) {
            const float v = (n < OC && k < K) ? (float)w[(long)n * K + k] : 0.f;
            const __nv_bfloat16 b = __float2bfloat16_rn(v);
            const size_t byte = (size_t)((k / 8) * 2 + n / 8) * 128 + (n % 8) * 16 + (k % 8) * 2;
            out[byte / 2] = *reinterpret_cast<const uint16_t *>(&b);
        }
}

// 2-D convolutions (mode 0, nd 2).  A CTA tile is 32 x 4 output pixels.
// The input patch the tile reads -- every channel, the tile's rows and
// columns scaled by the stride plus the dilated halo -- is first staged in
// shared memory as BF16 by whole warps reading rows (coalesced, all loads
// independent), and the im2col operand A is then built from shared memory:
// element (m, k) is patch[ktab[k] + base(m)].  The MMA issue, the bounded
// wait and the epilogue are those of k_conv3d_tc.
constexpr int kT2W = 32, kT2H = 4;
constexpr int kT2Cols = 3;              // patch columns per lane: PW <= 96

__global__ void __launch_bounds__(kTcM) k_conv2d_tc(TcConv a, int PH, int PW) {
    pdl_sync();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    __shared__ int ktab[kTcMaxK];                  // patch offset of k, -1 for K padding
    unsigned char *sA = smem;                                   // 128 x Kpad BF16
    unsigned char *sB = smem + (size_t)a.Kpad * kTcM * 2;        // 16 x Kpad BF16
    __nv_bfloat16 *patch = reinterpret_cast<__nv_bfloat16 *>(sB + (size_t)a.Kpad * kTcN * 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    const uint4 *wsrc = reinterpret_cast<const uint4 *>(a.wB);
    uint4 *wdst = reinterpret_cast<uint4 *>(sB);
    for (int i = tid; i < a.Kpad * kTcN * 2 / 16; i += kTcM) wdst[i] = __ldg(wsrc + i);
    const int pplane = PH * PW;
    for (int k = tid; k < a.Kpad; k += kTcM) {
        int e = -1;
        if (k < a.K) {
            const int c = k / 9, t = k - (k / 9) * 9;
            const int ky = t / 3, kx = t - (t / 3) * 3;
            e = c * pplane + ky * a.dil * PW + kx * a.dil;
        }
        ktab[k] = e;
    }
    if (tid == 0) {
        mbar_init(&mbar, 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_slot;

    const int tiles_x = (a.OW + kT2W - 1) / kT2W, tiles_y = (a.OH + kT2H - 1) / kT2H;
    const long tiles_img = (long)tiles_x * tiles_y;
    const int nb = a.nb > 0 ? a.nb : 1;
    const long tiles = tiles_img * a.nimg * nb;
    const long plane = (long)a.H * a.W, M = (long)a.OH * a.OW;
    const int my = tid / kT2W, mx = tid - (tid / kT2W) * kT2W;
    const int base = my * a.stride * PW + mx * a.stride;
    unsigned phase = 0;
    for (long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int item = (int)(tile / tiles_img);
        const int img = item / nb, bi = item - img * nb;
        const int t2 = (int)(tile - item * tiles_img);
        const int ty0 = (t2 / tiles_x) * kT2H, tx0 = (t2 - (t2 / tiles_x) * tiles_x) * kT2W;
        const float *x0 = (img ? a.x[1] : a.x[0]) + bi * a.xs;
        const int iy0 = ty0 * a.stride - a.pad, ix0 = tx0 * a.stride - a.pad;
        // ---- stage the patch: each warp takes 8 patch rows at a time, every
        // lane up to kT2Cols columns of each, all loads issued before the stores
        const int nrows = a.IC * PH;
        for (int r0 = warp; r0 < nrows; r0 += (kTcM / 32) * 8) {
            float v[8][kT2Cols];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int r = r0 + u * (kTcM / 32);
                const int c = r / PH, py = r - (r / PH) * PH;
                const int gy = iy0 + py;
                const bool rok = r < nrows && gy >= 0 && gy < a.H;
                const float *src = x0 + c * plane + (long)gy * a.W;
#pragma unroll
                for (int q = 0; q < kT2Cols; ++q) {
                    const int px = lane + 32 * q, gx = ix0 + px;
                    v[u][q] = rok && px < PW && gx >= 0 && gx < a.W ? __ldg(src + gx) : 0.f;
                }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int r = r0 + u * (kTcM / 32);
                if (r >= nrows) break;
#pragma unroll
                for (int q = 0; q < kT2Cols; ++q) {
                    const int px = lane + 32 * q;
                    if (px < PW) patch[(long)r * PW + px] = __float2bfloat16_rn(v[u][q]);
                }
            }
        }
        __syncthreads();
        const int oy = ty0 + my, ox = tx0 + mx;
        const bool row_ok = oy < a.OH && ox < a.OW;
        for (int kg = 0; kg < a.Kpad / 8; ++kg) {
            __align__(16) __nv_bfloat16 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int e = ktab[kg * 8 + j];
                v[j] = row_ok && e >= 0 ? patch[e + base] : __float2bfloat16_rn(0.f);
            }
            *reinterpret_cast<uint4 *>(sA + (size_t)(kg * (kTcM / 8) + (tid >> 3)) * 128 +
                                       (tid & 7) * 16) = *reinterpret_cast<const uint4 *>(v);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (tid == 0 && !failed) {
            const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
            for (int ks = 0; ks < a.Kpad / 16; ++ks) {
                const uint64_t da = umma_desc(a0 + ks * 2 * (kTcM / 8) * 128, (kTcM / 8) * 128, 128);
                const uint64_t db = umma_desc(b0 + ks * 2 * (kTcN / 8) * 128, (kTcN / 8) * 128, 128);
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    ::"r"(tmem), "l"(da), "l"(db), "r"(kIdescBf16), "r"(ks));
            }
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                ::"r"(smem_u32(&mbar))
                : "memory");
        }
        if (!failed && !mbar_wait(&mbar, phase)) {
            failed = 1;
            flag_error(a.err, SV_ERR_TIMEOUT);
        }
        phase ^= 1u;
        __syncthreads();
        if (failed) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        uint32_t r[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
              "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
              "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(tmem + ((uint32_t)(warp * 32) << 16)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (row_ok) {
            const long mi = (long)oy * a.OW + ox;
            float *y = (img ? a.y[1] : a.y[0]) + bi * a.ys;
            const float *aux = a.aux ? a.aux + bi * a.ys : nullptr;
#pragma unroll
            for (int n = 0; n < kTcN; ++n) {
                if (n < a.OC) {
                    float v = __uint_as_float(r[n]);
                    if (a.bias) v += __ldg(a.bias + n);
                    if (a.act == 1) v = v > 0.f ? v : v * 0.2f;
                    if (a.act == 2) v = __ldg(aux + (long)n * M + mi) > 0.f ? v : v * 0.2f;
                    y[(long)n * M + mi] = v;
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem), "r"(kTmemCols));
}

// Stride-1 2-D convolutions with at most 16 input channels, without an
// im2col operand.  A tile is 128 consecutive output pixels of one row; the
// three input rows its taps read (rows oy - pad + ky * dil) are staged in
// shared memory as BF16 in the UMMA K-major layout directly: two planes of 8
// channels each, every pixel 16 bytes, so 8 consecutive pixels form one
// 128-byte core matrix.  The A operand of tap (ky, kx) is then the same
// patch read from pixel ky * PWp + kx * dil on (start address shifted by a
// multiple of 16 bytes; LBO = one channel plane, SBO = 128 bytes), and a
// tile is 9 MMAs of K = 16 -- one per tap -- accumulating in tensor memory.
// Operand B is re-ordered on the way into shared memory from the packed
// channel-major K (k = c * 9 + t) to one 16-channel block per tap
// (k = t * 16 + c, zero for c >= IC).  The bounded wait and the epilogue
// are those of k_conv2d_tc.
constexpr int kTapW = 128;              // output pixels per tile
constexpr int kTapMaxDil = 8;

__device__ __forceinline__ int tc_b_off(int n, int k) {    // BF16 index in a packed operand B
    return (((k >> 3) * 2 + (n >> 3)) * 128 + (n & 7) * 16 + (k & 7) * 2) >> 1;
}

constexpr int kTapCtas = 5;             // resident CTAs per SM (registers)
// ICT, OCT, ACT: the channel counts and the activation fixed at compile time (0,
// 0, -1: read from the arguments).  What bounds a tile is instruction issue
// around 9 small MMAs: dividing an element index into (row, pixel) and testing
// every channel cost 2,570 warp instructions per tile and layer (16 -> 16
// channels at 640x480: 36 us); a fixed pixel per thread, all loads of a tile
// before the first packing and the counts known take 21 us.
template <int ICT, int OCT, int ACT>
__global__ void __launch_bounds__(kTcM, kTapCtas) k_conv2d_tc_tap(TcConv a, int PWp) {
    pdl_sync();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    unsigned char *sB = smem;                                    // 9 taps x 16 x 16 BF16
    unsigned char *patch = smem + 9 * 512;                       // [2][3][PWp] x 16 bytes
    const int tid = threadIdx.x, warp = tid >> 5;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    {
        uint16_t *wd = reinterpret_cast<uint16_t *>(sB);
        uint16_t v[9 * 256 / kTcM];
#pragma unroll
        for (int u = 0; u < 9 * 256 / kTcM; ++u) {
            const int i = tid + u * kTcM, t = i >> 8, n = (i >> 4) & 15, c = i & 15;
            v[u] = c < a.IC ? a.wB[tc_b_off(n, c * 9 + t)] : (uint16_t)0;
        }
#pragma unroll
        for (int u = 0; u < 9 * 256 / kTcM; ++u) {
            const int i = tid + u * kTcM, t = i >> 8, n = (i >> 4) & 15, c = i & 15;
            wd[tc_b_off(n, t * 16 + c)] = v[u];
        }
    }
    if (tid == 0) {
        mbar_init(&mbar, 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_slot;

    const int tiles_x = (a.OW + kTapW - 1) / kTapW;
    const long tiles_img = (long)tiles_x * a.OH;
    const int nb = a.nb > 0 ? a.nb : 1;
    const long tiles = tiles_img * a.nimg * nb;
    const long plane = (long)a.H * a.W, M = (long)a.OH * a.OW;
    const uint32_t lbo = 3u * (uint32_t)PWp * 16u;               // one 8-channel plane
    // this thread's pixel of the rows' tails (6 rows of 2 dil pixels <= 96)
    const int tail = 2 * a.dil, hr = tid / tail, hpx = tid - hr * tail;
    const int IC = ICT > 0 ? ICT : a.IC, OC = OCT > 0 ? OCT : a.OC, act = ACT >= 0 ? ACT : a.act;
    const bool halo = hr < 6, two = IC > 8;
    unsigned phase = 0;
    for (long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int item = (int)(tile / tiles_img);
        const int img = item / nb, bi = item - img * nb;
        const int t2 = (int)(tile - item * tiles_img);
        const int oy = t2 / tiles_x, ox0 = (t2 - oy * tiles_x) * kTapW;
        const float *x0 = (img ? a.x[1] : a.x[0]) + bi * a.xs;
        // ---- stage rows oy - pad + ky * dil: thread t packs 8 channels of
        // pixel t of each row (and one pixel of the rows' 2 dil tail) into one
        // 16-byte store.  All loads of a tile are issued before the first is
        // packed: one memory latency per tile.
        float f[7][8];
        auto load8 = [&](int ch, int ky, int px, bool on, float (&v)[8]) {
            const int iy = oy - a.pad + ky * a.dil, ix = ox0 - a.pad + px;
            const bool ok = on && (unsigned)iy < (unsigned)a.H && (unsigned)ix < (unsigned)a.W;
            // a channel plane's base is the same for the whole CTA
            const unsigned off = ok ? (unsigned)(iy * a.W + ix) : 0u;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                v[j] = ok && ch * 8 + j < IC ? __ldg(x0 + (ch * 8 + j) * plane + off) : 0.f;
        };
        auto put8 = [&](int r, int px, const float (&v)[8]) {
            uint32_t q[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __nv_bfloat162 h2 = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                q[j] = *reinterpret_cast<const uint32_t *>(&h2);
            }
            *reinterpret_cast<uint4 *>(patch + (size_t)(r * PWp + px) * 16) =
                make_uint4(q[0], q[1], q[2], q[3]);
        };
#pragma unroll
        for (int r = 0; r < 6; ++r) load8(r / 3, r % 3, tid, r < 3 || two, f[r]);
        load8(hr / 3, hr % 3, kTapW + hpx, halo && (hr < 3 || two), f[6]);
#pragma unroll
        for (int r = 0; r < 6; ++r) put8(r, tid, f[r]);
        if (halo) put8(hr, kTapW + hpx, f[6]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (tid == 0 && !failed) {
            const uint32_t p0 = smem_u32(patch), b0 = smem_u32(sB);
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                const int ky = t / 3, kx = t - (t / 3) * 3;
                const uint64_t da =
                    umma_desc(p0 + (uint32_t)(ky * PWp + kx * a.dil) * 16u, lbo, 128);
                const uint64_t db = umma_desc(b0 + t * 512, (kTcN / 8) * 128, 128);
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    ::"r"(tmem), "l"(da), "l"(db), "r"(kIdescBf16), "r"(t));
            }
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                ::"r"(smem_u32(&mbar))
                : "memory");
        }
        if (!failed && !mbar_wait(&mbar, phase)) {
            failed = 1;
            flag_error(a.err, SV_ERR_TIMEOUT);
        }
        phase ^= 1u;
        __syncthreads();
        if (failed) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        uint32_t r[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
              "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
              "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(tmem + ((uint32_t)(warp * 32) << 16)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const int ox = ox0 + tid;
        if (ox < a.OW) {
            const long mi = (long)oy * a.OW + ox;
            float *y = (img ? a.y[1] : a.y[0]) + bi * a.ys;
            const float *aux = a.aux ? a.aux + bi * a.ys : nullptr;
#pragma unroll
            for (int n = 0; n < kTcN; ++n) {
                if (n < OC) {
                    float v = __uint_as_float(r[n]);
                    if (a.bias) v += __ldg(a.bias + n);
                    if (act == 1) v = v > 0.f ? v : v * 0.2f;
                    if (act == 2) v = __ldg(aux + (long)n * M + mi) > 0.f ? v : v * 0.2f;
                    y[(long)n * M + mi] = v;
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem), "r"(kTmemCols));
}

// Per-device launch set-up, done once: the SM count and each kernel's
// dynamic shared-memory limit (raised to kTcSmemMax; every launch checks
// its own size against it).  Launches stay free of attribute calls.
constexpr size_t kTcSmemMax = 200 * 1024;
enum { kKConv3d, kKConv3dV, kKConv3d12, kKConv3d6, kKConv2d, kKWgrad, kKConv2dTap, kKCount };

static int tc_setup(int which, const void *fn, int *sms) {
    static std::mutex mu;
    static int cached_sms[64];
    static bool attr_done[64][kKCount];
    int dev = 0;
    SV_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_error("device ordinal %d out of range", dev);
        return SV_ERR_CUDA;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (!cached_sms[dev])
        SV_CUDA_TRY(cudaDeviceGetAttribute(&cached_sms[dev], cudaDevAttrMultiProcessorCount, dev));
    if (!attr_done[dev][which]) {
        SV_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kTcSmemMax));
        attr_done[dev][which] = true;
    }
    *sms = cached_sms[dev];
    return SV_OK;
}

// CTAs per SM for a kernel using `smem` bytes of dynamic shared memory.
static long tc_ctas_per_sm(size_t smem) {
    const long per = (long)((220 * 1024) / (smem + 8 * 1024));
    return per < 1 ? 1 : (per > 4 ? 4 : per);
}

static int launch_conv2d_tc(const TcConv &a, cudaStream_t st) {
    if (a.stride == 1 && a.IC <= 16 && a.dil <= kTapMaxDil && a.pad >= 0 &&
        a.K == a.IC * 9) {
        const int PWp = kTapW + 2 * a.dil;
        const size_t smem = 9 * 512 + (size_t)2 * 3 * PWp * 16;
        const long tiles = (long)((a.OW + kTapW - 1) / kTapW) * a.OH * a.nimg *
                           (a.nb > 0 ? a.nb : 1);
        if (tiles == 0) return SV_OK;
        int sms = 148;
        const int rc = tc_setup(kKConv2dTap, (const void *)k_conv2d_tc_tap<0, 0, -1>, &sms);
        if (rc) return rc;
        // up to kTapCtas CTAs (32 TMEM columns each) per SM, as many as give every
        // CTA the same number of tiles (2,400 tiles at 640x480 over 8 x 148 CTAs
        // were a third round for the last 32)
        const long cap = (long)sms * kTapCtas, rounds = (tiles + cap - 1) / cap;
        const unsigned blocks = (unsigned)((tiles + rounds - 1) / rounds);
        count_launch();
        // FeatureNet c3 / c4 of the shipped checkpoint and the band net's layers
        if (a.IC == 12 && a.OC == 12 && a.act == 1)
            pdl(k_conv2d_tc_tap<12, 12, 1>, blocks, kTcM, smem, st)(a, PWp);
        else if (a.IC == 12 && a.OC == 12 && a.act == 0)
            pdl(k_conv2d_tc_tap<12, 12, 0>, blocks, kTcM, smem, st)(a, PWp);
        else if (a.IC == 8 && a.OC == 16 && a.act == 1)
            pdl(k_conv2d_tc_tap<8, 16, 1>, blocks, kTcM, smem, st)(a, PWp);
        else if (a.IC == 16 && a.OC == 16 && a.act == 1)
            pdl(k_conv2d_tc_tap<16, 16, 1>, blocks, kTcM, smem, st)(a, PWp);
        else if (a.IC == 16 && a.OC == 2 && a.act == 0)
            pdl(k_conv2d_tc_tap<16, 2, 0>, blocks, kTcM, smem, st)(a, PWp);
        else
            pdl(k_conv2d_tc_tap<0, 0, -1>, blocks, kTcM, smem, st)(a, PWp);
        SV_LAUNCH_CHECK();
        return SV_OK;
    }
    const int PH = (kT2H - 1) * a.stride + 2 * a.dil + 1;
    const int PW = (kT2W - 1) * a.stride + 2 * a.dil + 1;
    const size_t patch = ((size_t)a.IC * PH * PW * 2 + 15) / 16 * 16;
    const size_t smem = (size_t)a.Kpad * (kTcM + kTcN) * 2 + patch;
    if (smem > kTcSmemMax || PW > 32 * kT2Cols) {
        set_error("tensor-core conv: IC=%d dil=%d stride=%d patch too large", a.IC, a.dil,
                  a.stride);
        return SV_ERR_PARAM;
    }
    const long tiles = (long)((a.OW + kT2W - 1) / kT2W) * ((a.OH + kT2H - 1) / kT2H) * a.nimg *
                       (a.nb > 0 ? a.nb : 1);
    if (tiles == 0) return SV_OK;
    int sms = 148;
    const int rc = tc_setup(kKConv2d, (const void *)k_conv2d_tc, &sms);
    if (rc) return rc;
    const long cap = (long)sms * tc_ctas_per_sm(smem);
    const unsigned blocks = (unsigned)(tiles < cap ? tiles : cap);
    count_launch();
    pdl(k_conv2d_tc, blocks, kTcM, smem, st)(a, PH, PW);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

// Self-test of the failure path every tensor-core kernel here shares: a CTA
// allocates its tensor memory, arms an mbarrier that nothing will arrive at
// (no MMA is issued), and waits with a bounded poll count.  The wait must
// give up, record SV_ERR_TIMEOUT in the flag, free the tensor memory and
// return, leaving the context usable.  done receives 1 once the CTA has
// passed its dealloc.
__global__ void __launch_bounds__(kTcM) k_selftest_wait(unsigned limit, int *flag, int *done) {
    pdl_sync();
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    const int warp = threadIdx.x >> 5;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        mbar_init(&mbar, 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_slot;
    if (threadIdx.x == 0 && !mbar_wait(&mbar, 0, limit)) {
        failed = 1;
        flag_error(flag, SV_ERR_TIMEOUT);
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem), "r"(kTmemCols));
    __syncthreads();
    if (threadIdx.x == 0) *done = failed ? 1 : 2;
}

int launch_selftest_wait(unsigned limit, int *flag, int *done, cudaStream_t st) {
    count_launch();
    pdl(k_selftest_wait, 1, kTcM, 0, st)(limit, flag, done);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

int launch_conv_tc(const TcConv &a, cudaStream_t st) {
    if (a.OC < 1 || a.OC > kTcN || a.K < 1 || a.K > kTcMaxK || a.Kpad != tc_kpad(a.K) ||
        (a.mode == 0 && (a.nimg < 1 || a.nimg > 2)) || (a.mode == 1 && a.nd != 3) ||
        !a.wB || !a.err || (a.act == 2 && !a.aux) || a.nb < 0) {
        set_error("tensor-core conv: IC=%d OC=%d K=%d outside the kernel's shapes", a.IC, a.OC,
                  a.K);
        return SV_ERR_PARAM;
    }
    if (a.mode == 0 && a.nd == 2) {
        if (a.K != a.IC * 9 || a.D != 1 || a.OD != 1 || a.stride < 1 || a.dil < 1) {
            set_error("tensor-core conv2d: inconsistent shape");
            return SV_ERR_PARAM;
        }
        return launch_conv2d_tc(a, st);
    }
    if (a.nd != 3 || a.K != a.IC * 27 || a.stride != 1 || a.pad != 1 || a.dil != 1 ||
        a.OD != a.D || a.OH != a.H || a.OW != a.W) {
        set_error("tensor-core conv3d: inconsistent shape");
        return SV_ERR_PARAM;
    }
    const size_t smem = (size_t)a.Kpad * (kTcM + kTcN) * 2 +
                        (size_t)3 * a.IC * kC3Rows * kC3Pitch * 2;
    const long steps = (long)((a.W + kC3W - 1) / kC3W) * ((a.H + kC3H - 1) / kC3H) * a.D *
                       (a.mode == 0 ? a.nimg : 1) * (a.nb > 0 ? a.nb : 1);
    if (steps == 0) return SV_OK;
    int sms = 148;
    // the shipped checkpoint's cost filter (12, then 6 channels), and any other
    void (*f)(TcConv, int) = a.mode == 1 ? k_conv3d_tc<0, 1> : k_conv3d_tc<0, 0>;
    int which = a.mode == 1 ? kKConv3dV : kKConv3d;
    if (a.mode == 1 && a.IC == 12) f = k_conv3d_tc<12, 1>, which = kKConv3d12;
    if (a.mode == 0 && a.IC == 6) f = k_conv3d_tc<6, 0>, which = kKConv3d6;
    const int rc = tc_setup(which, (const void *)f, &sms);
    if (rc) return rc;
    // consecutive steps (disparities of a place) to a CTA, the same number to each
    // (two CTAs of 12 channels fill the SM's 228 KB)
    const long cap = (long)sms * (smem + 2 * 1024 <= 114 * 1024 ? 2 : 1);
    const int per = (int)((steps + cap - 1) / cap);
    const unsigned blocks = (unsigned)((steps + per - 1) / per);
    count_launch();
    pdl(f, blocks, kC3Threads, smem, st)(a, per);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

// ------------------------------------------------------- weight gradient
// D[m][n] = sum over pixels p of A[m][p] * B[n][p] with A[m = c*9 + t][p] =
// x[c][p + tap t] (row IC*9 is all ones, giving the bias gradient) and
// B[n = o][p] = g[o][p].  M is 1 or 2 tiles of 128 rows (IC*9 + 1 <= 256),
// N = 16, K = the pixels, 64 per chunk.  CTAs stride over chunks with two
// shared-memory stages: the gather of chunk i overlaps the MMAs of chunk
// i-1, and stage reuse waits for the commit of chunk i-2.  At the end every
// CTA adds its FP32 partial sums into gw / gb.
constexpr int kWgK = 64;

__global__ void __launch_bounds__(kTcM) k_wgrad_tc(TcWgrad a, int mtiles) {
    pdl_sync();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    __shared__ int4 pix[2][kWgK];                    // (item, y, x, valid)
    const size_t a_tile = (size_t)kTcM * kWgK * 2;
    const size_t stage = (size_t)mtiles * a_tile + (size_t)kTcN * kWgK * 2;
    const int tid = threadIdx.x, warp = tid >> 5;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        mbar_init(&mbar[0], 1);
        mbar_init(&mbar[1], 1);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_slot;
    const long HW = (long)a.H * a.W;
    const long P = HW * a.nb;
    const long chunks = (P + kWgK - 1) / kWgK;
    const int KR = a.IC * 9;
    // this thread's A rows, one per M tile
    int rc[2], rdy[2], rdx[2], rkind[2];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
        const int m = mt * kTcM + tid;
        rc[mt] = 0; rdy[mt] = 0; rdx[mt] = 0;
        rkind[mt] = m < KR ? 0 : (m == KR ? 1 : 2);
        if (m < KR) {
            const int c = m / 9, t = m - (m / 9) * 9;
            rc[mt] = c;
            rdy[mt] = (t / 3 - 1) * a.dil;
            rdx[mt] = (t - (t / 3) * 3 - 1) * a.dil;
        }
    }
    int it = 0;
    for (long ch = blockIdx.x; ch < chunks; ch += gridDim.x, ++it) {
        const int s = it & 1;
        unsigned char *sA = smem + s * stage;
        unsigned char *sB = sA + (size_t)mtiles * a_tile;
        if (it >= 2 && !failed && !mbar_wait(&mbar[s], ((it - 2) >> 1) & 1)) {
            failed = 1;
            flag_error(a.err, SV_ERR_TIMEOUT);
        }
        __syncthreads();
        if (failed) break;
        if (tid < kWgK) {
            const long p = ch * kWgK + tid;
            int4 e = make_int4(0, 0, 0, 0);
            if (p < P) {
                const int item = (int)(p / HW);
                const int r = (int)(p - item * HW);
                e = make_int4(item, r / a.W, r - (r / a.W) * a.W, 1);
            }
            pix[s][tid] = e;
        }
        __syncthreads();
        {   // B: thread (n, 8 pixels)
            const int n = tid >> 3, kg = tid & 7;
            __align__(16) __nv_bfloat16 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int4 e = pix[s][kg * 8 + j];
                float f = 0.f;
                if (e.w && n < a.OC)
                    f = __ldg(a.g + e.x * a.gs + n * HW + (long)e.y * a.W + e.z);
                v[j] = __float2bfloat16_rn(f);
            }
            *reinterpret_cast<uint4 *>(sB + (size_t)(kg * 2 + (n >> 3)) * 128 + (n & 7) * 16) =
                *reinterpret_cast<const uint4 *>(v);
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {        // A: this thread's row of each M tile
            if (mt >= mtiles) break;
            unsigned char *tA = sA + (size_t)mt * a_tile;
            const float *xc = a.x + (long)rc[mt] * HW;
            for (int kg = 0; kg < kWgK / 8; ++kg) {
                __align__(16) __nv_bfloat16 v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int4 e = pix[s][kg * 8 + j];
                    float f = 0.f;
                    if (e.w) {
                        if (rkind[mt] == 0) {
                            const int yy = e.y + rdy[mt], xx = e.z + rdx[mt];
                            if (yy >= 0 && yy < a.H && xx >= 0 && xx < a.W)
                                f = __ldg(xc + e.x * a.xs + (long)yy * a.W + xx);
                        } else if (rkind[mt] == 1) {
                            f = 1.f;
                        }
                    }
                    v[j] = __float2bfloat16_rn(f);
                }
                *reinterpret_cast<uint4 *>(tA + (size_t)(kg * (kTcM / 8) + (tid >> 3)) * 128 +
                                           (tid & 7) * 16) = *reinterpret_cast<const uint4 *>(v);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (tid == 0) {
            const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
            for (int mt = 0; mt < mtiles; ++mt) {
                for (int ks = 0; ks < kWgK / 16; ++ks) {
                    const uint64_t da = umma_desc(a0 + mt * (uint32_t)a_tile +
                                                      ks * 2 * (kTcM / 8) * 128,
                                                  (kTcM / 8) * 128, 128);
                    const uint64_t db =
                        umma_desc(b0 + ks * 2 * (kTcN / 8) * 128, (kTcN / 8) * 128, 128);
                    const uint32_t acc = (it > 0 || ks > 0) ? 1u : 0u;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                        ::"r"(tmem + mt * kTcN), "l"(da), "l"(db), "r"(kIdescBf16), "r"(acc));
                }
            }
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                ::"r"(smem_u32(&mbar[s]))
                : "memory");
        }
    }
    // the last commit covers every MMA this CTA issued
    if (it > 0 && !failed && !mbar_wait(&mbar[(it - 1) & 1], ((it - 1) >> 1) & 1)) {
        failed = 1;
        flag_error(a.err, SV_ERR_TIMEOUT);
    }
    __syncthreads();
    if (it > 0 && !failed) {
        asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            if (mt >= mtiles) break;
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                  "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                  "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(tmem + ((uint32_t)(warp * 32) << 16) + mt * kTcN));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int m = mt * kTcM + tid;
#pragma unroll
            for (int n = 0; n < kTcN; ++n) {
                if (n >= a.OC) break;
                const float v = __uint_as_float(r[n]);
                if (m < KR) atomicAdd(a.gw + (long)n * KR + m, v);
                else if (m == KR) atomicAdd(a.gb + n, v);
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem), "r"(kTmemCols));
}

int launch_wgrad_tc(const TcWgrad &a, cudaStream_t st) {
    if (a.IC < 1 || a.OC < 1 || a.OC > kTcN || a.IC * 9 + 1 > 2 * kTcM || a.dil < 1 ||
        a.H < 1 || a.W < 1 || a.nb < 1 || !a.x || !a.g || !a.gw || !a.gb || !a.err) {
        set_error("tensor-core weight gradient: IC=%d OC=%d outside the kernel's shapes", a.IC,
                  a.OC);
        return SV_ERR_PARAM;
    }
    const int mtiles = (a.IC * 9 + 1 + kTcM - 1) / kTcM;
    const size_t smem = 2 * ((size_t)mtiles * kTcM * kWgK * 2 + (size_t)kTcN * kWgK * 2);
    const long chunks = ((long)a.H * a.W * a.nb + kWgK - 1) / kWgK;
    int sms = 148;
    const int rc = tc_setup(kKWgrad, (const void *)k_wgrad_tc, &sms);
    if (rc) return rc;
    const long cap = (long)sms * 2;
    const unsigned blocks = (unsigned)(chunks < cap ? chunks : cap);
    count_launch();
    pdl(k_wgrad_tc, blocks, kTcM, smem, st)(a, mtiles);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

__global__ void k_pack_weights(const float *__restrict__ w, int OC, int IC, int transpose,
                               int K, int Kpad, uint16_t *__restrict__ out) {
    pdl_sync();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kTcN * Kpad) return;
    const int n = i / Kpad, k = i - (i / Kpad) * Kpad;
    float v = 0.f;
    if (!transpose) {
        if (n < OC && k < K) v = w[n * K + k];
    } else if (n < IC && k < K) {
        const int o = k / 9, t = k - (k / 9) * 9;
        v = w[(o * IC + n) * 9 + (8 - t)];
    }
    const __nv_bfloat16 b = __float2bfloat16_rn(v);
    out[((size_t)((k >> 3) * 2 + (n >> 3)) * 128 + (n & 7) * 16 + (k & 7) * 2) / 2] =
        *reinterpret_cast<const uint16_t *>(&b);
}

int launch_pack_weights(const float *w, int OC, int IC, int transpose, uint16_t *out,
                        cudaStream_t st) {
    const int K = (transpose ? OC : IC) * 9;
    if ((transpose ? IC : OC) > kTcN) {
        set_error("packed operand has more than 16 rows");
        return SV_ERR_PARAM;
    }
    const int Kpad = tc_kpad(K);
    count_launch();
    pdl(k_pack_weights, (kTcN * Kpad + 255) / 256, 256, 0, st)(w, OC, IC, transpose, K, Kpad,
                                                              out);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

}  // namespace sv
