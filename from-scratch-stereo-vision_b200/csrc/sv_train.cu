// sv_train.cu -- StereoNet training on the GPU: train_grads
// (stereonet.py:1619-1653) over a batch of crops and Adam.step (1368-1387),
// the batch gradient being the mean of the per-sample gradients, which is
// what the reference's data-parallel harness computes with one process per
// sample (train_parallel.py:144-156).
//
// FP32 activations and gradients, FP64 parameters, Adam state and weight
// gradient sums.  The forward keeps every activation it needs (after the
// leaky ReLU only: with slope 0.2 or 0, a post-activation value is positive
// exactly when its input is, so it also gives the ReLU derivative).
// Every reduction has a fixed order, so a step is deterministic:
//   * input gradients are gathers (a thread sums the taps of its own input
//     elements), never atomics;
//   * a weight gradient is a sum over (image, pixel) of x * gy: each CTA
//     walks tiles of outputs, stages the input patch and the output
//     gradients in shared memory, and writes its partial sums for every
//     (out channel, in channel, tap) and the bias; one kernel at the end adds
//     the partials of all layers in order in FP64.
// The convolutions run on the FP32 pipe, since nothing here is held in fewer
// than 32 bits, and what bounds them is the shared-memory reads that feed it.
// So each keeps a block of results in registers (4 columns x all channels, or a
// row of taps x all channels), and one read feeds 4 to 12 FMAs instead of one.
// Every sum keeps the order it would have with one result per thread, so the split
// into threads shows in no bit of the gradients.  A step of 64 crops of 96x64 went
// from 2855 to 1172 us, 1037 with launches set up ahead (a pass among others).
// Layouts are the reference's planar ones with a leading image index; the
// siamese towers run as one batch of 2B images (the B left views, then the
// B right views).

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "sv_common.cuh"
#include "sv_network.cuh"

namespace sv {
namespace {

constexpr int kMaxB = 4096;

// n elements staged by nt threads, kStage loads in flight per thread: a loop that
// loads and stores one element at a time waits a memory latency for each (the
// tiles below are 10 to 60 elements per thread).
constexpr int kStage = 8;
template <typename L, typename S>
__device__ __forceinline__ void stage(int n, int tid, int nt, L load, S store) {
    for (int i0 = tid; i0 < n; i0 += nt * kStage) {
        float v[kStage];
#pragma unroll
        for (int u = 0; u < kStage; ++u) {
            const int i = i0 + u * nt;
            v[u] = i < n ? load(i) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kStage; ++u) {
            const int i = i0 + u * nt;
            if (i < n) store(i, v[u]);
        }
    }
}

// nrows rows of NCOLS elements, a warp per row (the row's own arithmetic is
// then shared by its elements), kRows rows in flight per warp.  src(r) gives the
// row's pointer or NULL (zeros); element j is column xb + j, zero outside [0, W).
constexpr int kRows = 6;
template <int NCOLS, typename R, typename D>
__device__ __forceinline__ void stage_rows(int nrows, int warp, int nwarps, int lane, int xb, int W,
                                           R src, D dst) {
    constexpr int NB = (NCOLS + 31) / 32;
    bool in[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) in[b] = xb + lane + 32 * b >= 0 && xb + lane + 32 * b < W;
    for (int r0 = warp; r0 < nrows; r0 += nwarps * kRows) {
        float v[kRows][NB];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const int r = r0 + u * nwarps;
            const float *p = r < nrows ? src(r) : nullptr;
#pragma unroll
            for (int b = 0; b < NB; ++b)
                v[u][b] = p && in[b] && lane + 32 * b < NCOLS ? __ldg(p + xb + lane + 32 * b) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const int r = r0 + u * nwarps;
            if (r >= nrows) break;
            float *q = dst(r);
#pragma unroll
            for (int b = 0; b < NB; ++b)
                if (lane + 32 * b < NCOLS) q[lane + 32 * b] = v[u][b];
        }
    }
}

// ------------------------------------------------------------- forward
// Both directions of a 3x3 convolution: the forward one, and the input gradient
// of a stride-1 one, which is a convolution of gy with the flipped taps (FLIP:
// IC counts gy's channels, OC the input channels computed, WC the input channels
// of the weights w[IC][WC][9]).  A CTA computes 32 columns x TR rows of one
// image, a thread 4 columns of every output channel: a row of the staged tile is
// read once, 16 bytes at a time, and feeds 3 taps x 4 columns x OC outputs, and a
// tap's weights are read as 16-byte broadcasts, so about 12 FMAs follow each
// shared-memory read (one output column and 4 channels per thread read a weight
// per FMA: 8 -> 8 channels, 64 crops of 96x64, 61 to 87 us forward and 75 to 100
// backward, now 25 for either).  Each output
// is one chain of FMAs over (channel, ky, kx), from the bias (forward) or 0.
// MODE: 0 none, 1 leaky 0.2, 2 residual + relu0, 3 times leaky'(xin).
// DIL: the dilation, 0 to read it from dil.
template <int IC, int OC, int WC, int S, int DIL, int MODE, bool FLIP, int TR>
__global__ void __launch_bounds__(8 * TR, OC <= 8 ? 6 : 1)
    k_tconv2d(const float *__restrict__ x, int H, int W, int OH, int OW, int dil_,
              const float *__restrict__ w, const float *__restrict__ b, float *__restrict__ y,
              const float *__restrict__ aux, long aux_stride) {
    pdl_sync();
    constexpr int OCP = OC >= 4 ? (OC + 3) / 4 * 4 : OC, NT = 8 * TR;
    static_assert(!FLIP || S == 1, "flipped taps: stride 1");
    extern __shared__ __align__(16) float tile[];
    __shared__ __align__(16) float sw[IC * 9 * OCP];
    __shared__ float sb[OC];
    const int dil = DIL > 0 ? DIL : dil_;
    const int img = blockIdx.z, tid = threadIdx.x;
    for (int i = tid; i < IC * 9 * OCP; i += NT) {
        const int o = i % OCP, ct = i / OCP, c = ct / 9, t = ct - c * 9;
        sw[i] = o >= OC ? 0.f : FLIP ? w[(c * WC + o) * 9 + 8 - t] : w[(o * IC + c) * 9 + t];
    }
    if (tid < OC) sb[tid] = FLIP ? 0.f : b[tid];
    const long HW = (long)H * W;
    const float *xi = x + (long)img * IC * HW;
    const int ox0 = blockIdx.x * 32, oy0 = blockIdx.y * TR;
    const int ix0 = ox0 * S - dil, iy0 = oy0 * S - dil;
    const int th = (TR - 1) * S + 2 * dil + 1, tw = 31 * S + 2 * dil + 1;
    const int tp = (tw + 3) / 4 * 4 + 4;               // row stride: 16-byte rows, spread banks
    auto row_of = [&](int r) -> const float * {
        const int c = r / th, gy = iy0 + r - c * th;
        return gy >= 0 && gy < H ? xi + c * HW + (long)gy * W : nullptr;
    };
    auto tile_row = [&](int r) { return tile + r * tp; };
    if constexpr (DIL > 0) {
        stage_rows<(31 * S + 2 * DIL + 1 + 3) / 4 * 4 + 4>(IC * th, tid >> 5, NT >> 5, tid & 31, ix0, W,
                                                       row_of, tile_row);
    } else {
        stage(IC * th * tp, tid, NT,
              [&](int i) {
                  const int r = i / tp, gx = ix0 + i - r * tp;
                  const float *p = row_of(r);
                  return p && gx >= 0 && gx < W ? __ldg(p + gx) : 0.f;
              },
              [&](int i, float v) { tile[i] = v; });
    }
    __syncthreads();
    const int lx = (tid & 7) * 4, ly = tid >> 3;
    const int ox = ox0 + lx, oy = oy0 + ly;
    if (ox >= OW || oy >= OH) return;
    float acc[4][OC];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int o = 0; o < OC; ++o) acc[q][o] = sb[o];
    for (int c = 0; c < IC; ++c) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int ky = FLIP ? 2 - k : k;
            const float *row = tile + (c * th + ly * S + ky * dil) * tp + lx * S;
            constexpr int SPAN = DIL > 0 ? 3 * S + 2 * DIL + 1 : 4, NV = (SPAN + 3) / 4;
            float v[4 * NV];
            if constexpr (DIL > 0) {
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    const float4 f = *reinterpret_cast<const float4 *>(row + 4 * i);
                    v[4 * i] = f.x;
                    v[4 * i + 1] = f.y;
                    v[4 * i + 2] = f.z;
                    v[4 * i + 3] = f.w;
                }
            }
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int kx = FLIP ? 2 - j : j;
                const float *wt = sw + (c * 9 + ky * 3 + kx) * OCP;
                float u[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if constexpr (DIL > 0) u[q] = v[q * S + kx * DIL];
                    else u[q] = row[q * S + kx * dil];
                }
                if constexpr (OC >= 4) {
#pragma unroll
                    for (int o4 = 0; o4 < OCP; o4 += 4) {
                        const float4 f = *reinterpret_cast<const float4 *>(wt + o4);
                        const float wv[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (o4 + e < OC)
#pragma unroll
                                for (int q = 0; q < 4; ++q)
                                    acc[q][o4 + e] = fmaf(u[q], wv[e], acc[q][o4 + e]);
                    }
                } else {
#pragma unroll
                    for (int o = 0; o < OC; ++o)
#pragma unroll
                        for (int q = 0; q < 4; ++q) acc[q][o] = fmaf(u[q], wt[o], acc[q][o]);
                }
            }
        }
    }
    const long OHW = (long)OH * OW, oi = (long)oy * OW + ox;
    const bool vec = (OW & 3) == 0 && OHW % 4 == 0;    // whole 16-byte stores
#pragma unroll
    for (int o = 0; o < OC; ++o) {
        float r[4];
        float *yo = y + ((long)img * OC + o) * OHW + oi;
        const float *ax = MODE == 2 ? aux + img * aux_stride + oi
                                    : aux + ((long)img * WC + o) * OHW + oi;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float f = acc[q][o];
            const bool in = vec || ox + q < OW;
            if (MODE == 1) f = f > 0.f ? f : f * 0.2f;
            if (MODE == 2 && in) {                     // Refinement: relu0(disp + residual)
                f = ax[q] + f;
                f = f > 0.f ? f : f * 0.f;
            }
            if (MODE == 3 && in) f = ax[q] > 0.f ? f : f * 0.2f;
            r[q] = f;
        }
        if (vec) {
            *reinterpret_cast<float4 *>(yo) = make_float4(r[0], r[1], r[2], r[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (ox + q < OW) yo[q] = r[q];
        }
    }
}

size_t tconv2d_smem(int IC, int s, int dil, int TR) {
    const int tw = 31 * s + 2 * dil + 1;
    return sizeof(float) * IC * ((TR - 1) * s + 2 * dil + 1) * ((tw + 3) / 4 * 4 + 4);
}

// The same for 3x3x3 convolutions, stride 1, same padding: a CTA computes one
// row (b, y) for every disparity and up to 32 columns, a thread 4 columns of
// every output channel of one disparity; channels are staged CCH at a time.
// MODE 0 none, 1 leaky, 3 times leaky'(xin).  12 -> 6 channels over 64 volumes of
// 12 x 16 x 24: 250 us with 2 channels of one voxel per thread, 76 with all 6 of
// four; its input gradient 205 us with one value per thread, now 65.
template <int IC, int OC, int WC, int CCH, int MODE, bool FLIP, int nxg>
__global__ void __launch_bounds__(128)
    k_tconv3d(const float *__restrict__ x, int D, int h, int w,
              const float *__restrict__ wt, const float *__restrict__ b, float *__restrict__ y,
              const float *__restrict__ xin) {
    pdl_sync();
    constexpr int OCP = OC >= 2 ? (OC + 1) / 2 * 2 : OC;
    static_assert(IC % CCH == 0, "channel chunks");
    extern __shared__ __align__(16) float tile[];      // [CCH][D + 2][3][rs]
    __shared__ __align__(16) float sw[IC * 27 * OCP];
    __shared__ float sb[OC];
    __shared__ int off[54];                            // (disparity, row) -> offset in a channel
    constexpr int rs = 4 * nxg + 4;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int bi = blockIdx.z, oy = blockIdx.y, x0 = blockIdx.x * 4 * nxg;
    for (int i = tid; i < IC * 27 * OCP; i += nt) {
        const int o = i % OCP, ct = i / OCP, c = ct / 27, t = ct - c * 27;
        sw[i] = o >= OC ? 0.f : FLIP ? wt[(c * WC + o) * 27 + 26 - t] : wt[(o * IC + c) * 27 + t];
    }
    if (tid < OC) sb[tid] = FLIP ? 0.f : b[tid];
    const long hw = (long)h * w, total = (long)D * hw;
    const float *xb = x + (long)bi * IC * total;
    for (int r = tid; r < (D + 2) * 3; r += nt) {
        const int dz = r / 3, dd = dz - 1, yy = oy - 1 + r - dz * 3;
        off[r] = dd >= 0 && dd < D && yy >= 0 && yy < h ? (int)(dd * hw) + yy * w : -1;
    }
    const int xg = tid % nxg, od = tid / nxg;
    const bool on = od < D;
    float acc[4][OC];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int o = 0; o < OC; ++o) acc[q][o] = sb[o];
    for (int c0 = 0; c0 < IC; c0 += CCH) {
        if (c0) __syncthreads();
        for (int c = 0; c < CCH; ++c) {
            const float *xc = xb + (c0 + c) * total;
            float *tc = tile + c * (D + 2) * 3 * rs;
            stage_rows<rs>((D + 2) * 3, tid >> 5, nt >> 5, tid & 31, x0 - 1, w,
                           [&](int r) { return off[r] < 0 ? nullptr : xc + off[r]; },
                           [&](int r) { return tc + r * rs; });
        }
        __syncthreads();
        if (!on) continue;
        auto row_of = [&](int c, int kd, int ky, float (&v)[6]) {
            const float *row = tile + ((c * (D + 2) + od + kd) * 3 + ky) * rs + 4 * xg;
            const float4 f = *reinterpret_cast<const float4 *>(row);
            const float2 f2 = *reinterpret_cast<const float2 *>(row + 4);
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; v[4] = f2.x; v[5] = f2.y;
        };
        auto tap = [&](const float (&v)[6], const float *wr, int kx) {
            if constexpr (OC >= 2) {
#pragma unroll
                for (int o = 0; o < OCP; o += 2) {
                    const float2 g = *reinterpret_cast<const float2 *>(wr + o);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        acc[q][o] = fmaf(v[q + kx], g.x, acc[q][o]);
                        if (o + 1 < OC)
                            acc[q][o + 1 < OC ? o + 1 : o] =
                                fmaf(v[q + kx], g.y, acc[q][o + 1 < OC ? o + 1 : o]);
                    }
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[q][0] = fmaf(v[q + kx], wr[0], acc[q][0]);
            }
        };
        if constexpr (FLIP) {
            // taps from the last to the first, a tap's channels inner
            static_assert(CCH == IC, "all channels staged");
#pragma unroll 1
            for (int kd = 2; kd >= 0; --kd)
#pragma unroll 1                        // (9 x the code leaves the instruction cache)
                for (int ky = 2; ky >= 0; --ky) {
                    float v[IC][6];
#pragma unroll
                    for (int c = 0; c < IC; ++c) row_of(c, kd, ky, v[c]);
#pragma unroll
                    for (int kx = 2; kx >= 0; --kx)
#pragma unroll
                        for (int c = 0; c < IC; ++c)
                            tap(v[c], sw + (c * 27 + kd * 9 + ky * 3 + kx) * OCP, kx);
                }
        } else {
            for (int c = 0; c < CCH; ++c)
#pragma unroll
                for (int kd = 0; kd < 3; ++kd)
#pragma unroll
                    for (int ky = 0; ky < 3; ++ky) {
                        float v[6];
                        row_of(c, kd, ky, v);
#pragma unroll
                        for (int kx = 0; kx < 3; ++kx)
                            tap(v, sw + ((c0 + c) * 27 + kd * 9 + ky * 3 + kx) * OCP, kx);
                    }
        }
    }
    if (!on) return;
    const int ox = x0 + 4 * xg;
    const long idx = (long)od * hw + (long)oy * w + ox;
    const bool vec = (w & 3) == 0;
#pragma unroll
    for (int o = 0; o < OC; ++o) {
        const long at = ((long)bi * OC + o) * total + idx;
        float r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float f = acc[q][o];
            if (MODE == 1) f = f > 0.f ? f : f * 0.2f;
            if (MODE == 3 && ox + q < w) f = xin[at + q] > 0.f ? f : f * 0.2f;
            r[q] = f;
        }
        if (vec && ox < w) {
            *reinterpret_cast<float4 *>(y + at) = make_float4(r[0], r[1], r[2], r[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (ox + q < w) y[at + q] = r[q];
        }
    }
}

// CostVolume.forward (771-799): vol[b][c][d][y][x] = |fl - fr(x - d)|, 2.0
// where x - d < 0; fl is image b of f, fr image B + b.
__global__ void __launch_bounds__(256)
    k_tcostvol(const float *__restrict__ f, int B, int C, int D, int h, int w,
               float *__restrict__ vol) {
    pdl_sync();
    // one (sample, channel) per CTA; a warp takes whole rows of one disparity
    const int hw = h * w, bc = blockIdx.x, b = bc / C, c = bc - b * C;
    const float *l = f + ((long)b * C + c) * hw, *r = f + ((long)(B + b) * C + c) * hw;
    float *v = vol + (long)bc * D * hw;
    for (int row = blockIdx.y * 8 + (threadIdx.x >> 5); row < D * h; row += gridDim.y * 8) {
        const int d = row / h, y = row - d * h;
        for (int x = threadIdx.x & 31; x < w; x += 32)
            v[(long)row * w + x] = x - d < 0 ? 2.0f : fabsf(l[y * w + x] - r[y * w + x - d]);
    }
}

// SoftArgmin.forward with CostVolume.invalid_mask (858-885, 827-840): probs
// and disparity, FP32 with max-subtraction.
__global__ void k_tsoftargmin(const float *__restrict__ cost, int B, int D, int h, int w,
                              float *__restrict__ probs, float *__restrict__ d0) {
    pdl_sync();
    const long hw = (long)h * w;
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= B * hw) return;
    const int b = (int)(i / hw);
    const long p = i - b * hw;
    const int x = (int)(p % w);
    const float *cb = cost + (long)b * D * hw + p;
    float *pb = probs + (long)b * D * hw + p;
    float c[16];
    float best = -INFINITY;
    for (int d = 0; d < D; ++d) {
        c[d] = cb[d * hw] + ((d >= 1 && x < d) ? 8.0f : 0.0f);
        best = fmaxf(best, -c[d]);
    }
    float total = 0.f;
    for (int d = 0; d < D; ++d) {
        c[d] = expf(-c[d] - best);
        total += c[d];
    }
    const float inv = 1.0f / total;
    float acc = 0.f;
    for (int d = 0; d < D; ++d) {
        const float pr = c[d] * inv;
        pb[d * hw] = pr;
        acc += (float)d * pr;
    }
    d0[i] = acc;
}

// A refinement level's input [b][2][H2][W2]: 2 * bilinear(prev), guide.
__global__ void k_tupcat(const float *__restrict__ prev, int B, int h, int w, int H2, int W2,
                         const float *__restrict__ guide, float *__restrict__ rin) {
    pdl_sync();
    const long n2 = (long)H2 * W2;
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= B * n2) return;
    const int b = (int)(i / n2);
    const long p = i - b * n2;
    const int oy = (int)(p / W2), ox = (int)(p - (long)oy * W2);
    const Taps t = bilinear_taps(oy, ox, h, w, H2, W2);
    const float *s = prev + (long)b * h * w;
    const float v = s[t.i00] * (float)t.w00 + s[t.i01] * (float)t.w01 + s[t.i10] * (float)t.w10 +
                    s[t.i11] * (float)t.w11;
    rin[(long)b * 2 * n2 + p] = v * 2.0f;
    rin[(long)b * 2 * n2 + n2 + p] = guide[(long)b * n2 + p];
}

// build_targets (1572-1611) one level down: disparity 0.25 * sum * 0.5,
// valid = all four, guide (optional) 0.25 * sum.
__global__ void k_tpool(const float *__restrict__ d, const uint8_t *__restrict__ v,
                        const float *__restrict__ g, int B, int H, int W, float *__restrict__ dd,
                        uint8_t *__restrict__ vv, float *__restrict__ gg) {
    pdl_sync();
    const int H2 = H / 2, W2 = W / 2;
    const long n2 = (long)H2 * W2;
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= B * n2) return;
    const int b = (int)(i / n2);
    const long p = i - b * n2;
    const int y = (int)(p / W2), x = (int)(p - (long)y * W2);
    const long r0 = (long)b * H * W + (long)(2 * y) * W + 2 * x, r1 = r0 + W;
    dd[i] = 0.25f * (d[r0] + d[r0 + 1] + d[r1] + d[r1 + 1]) * 0.5f;
    vv[i] = (v[r0] && v[r0 + 1] && v[r1] && v[r1 + 1]) ? 1 : 0;
    if (g) gg[i] = 0.25f * (g[r0] + g[r0 + 1] + g[r1] + g[r1 + 1]);
}

// disparity_ce's target (1274-1323): fexp(-e^2 / (2 sigma^2)) is exactly 0
// below -700, so a pixel whose every e^2 / (2 sigma^2) exceeds 700 has
// qsum == 0 and is skipped.  Decided in FP64 as the reference does.
__device__ __forceinline__ bool ce_counted(float dg, int D) {
    const double inv2s2 = 1.0 / (2.0 * 0.8 * 0.8);
    for (int d = 0; d < D; ++d) {
        const double e = (double)d - (double)dg;
        if (!(e * e * inv2s2 > 700.0)) return true;
    }
    return false;
}

// Per-sample counts: valid pixels at 1/4, 1/2, 1/1 and the CE count.
__global__ void __launch_bounds__(256)
    k_tcounts(const uint8_t *__restrict__ vq, const uint8_t *__restrict__ vh,
              const uint8_t *__restrict__ vf, const float *__restrict__ dq, long n4, long n2,
              long n1, int D, int *__restrict__ counts) {
    pdl_sync();
    __shared__ int s[4][256];
    const int b = blockIdx.x, t = threadIdx.x;
    int c0 = 0, c1 = 0, c2 = 0, c3 = 0;
    for (long i = t; i < n4; i += 256) {
        if (vq[b * n4 + i]) {
            ++c0;
            if (ce_counted(dq[b * n4 + i], D)) ++c3;
        }
    }
    for (long i = t; i < n2; i += 256) c1 += vh[b * n2 + i] != 0;
    for (long i = t; i < n1; i += 256) c2 += vf[b * n1 + i] != 0;
    s[0][t] = c0; s[1][t] = c1; s[2][t] = c2; s[3][t] = c3;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (t < k)
            for (int j = 0; j < 4; ++j) s[j][t] += s[j][t + k];
        __syncthreads();
    }
    if (t < 4) counts[b * 4 + t] = s[t][0];
}

// pseudo_huber (1326-1351) of one level, weighted and averaged over the
// batch: g = wgt * (x / r) / count / B; term = r - 1 for the loss.
__global__ void k_thuber(const float *__restrict__ pred, const float *__restrict__ tgt,
                         const uint8_t *__restrict__ valid, int B, long n,
                         const int *__restrict__ counts, int lv, float wgt, float invB,
                         float *__restrict__ g, float *__restrict__ term) {
    pdl_sync();
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= B * n) return;
    const int b = (int)(i / n);
    const int cnt = counts[b * 4 + lv];
    if (!valid[i] || cnt == 0) {
        g[i] = 0.f;
        term[i] = 0.f;
        return;
    }
    const float x = pred[i] - tgt[i];
    const float r = sqrtf(x * x + 1.0f);
    g[i] = (x / r) * (1.0f / (float)cnt) * wgt * invB;
    term[i] = r - 1.0f;
}

// SoftArgmin.backward (887-901) plus the distribution cross-entropy
// gradient (q - p) / count, weighted: gcost[b][d][p].
__global__ void k_tsoft_bwd(const float *__restrict__ probs, const float *__restrict__ d0,
                            const float *__restrict__ gd0, const float *__restrict__ dq,
                            const uint8_t *__restrict__ vq, const int *__restrict__ counts,
                            int B, int D, long hw, float ce_w, float invB,
                            float *__restrict__ gcost, float *__restrict__ term) {
    pdl_sync();
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= B * hw) return;
    const int b = (int)(i / hw);
    const long p = i - b * hw;
    const float *pb = probs + (long)b * D * hw + p;
    float *gb = gcost + (long)b * D * hw + p;
    const float g = gd0[i], di = d0[i];
    const int cnt = counts[b * 4 + 3];
    const bool ce = vq[i] && cnt > 0 && ce_counted(dq[i], D);
    float q[16];
    if (ce) {
        const float inv2s2 = 1.0f / (2.0f * 0.8f * 0.8f);
        const float dg = dq[i];
        float xm = -INFINITY;
        for (int d = 0; d < D; ++d) {
            const float e = (float)d - dg;
            q[d] = -e * e * inv2s2;
            xm = fmaxf(xm, q[d]);
        }
        float qs = 0.f;
        for (int d = 0; d < D; ++d) {
            q[d] = q[d] < -700.f ? 0.f : expf(q[d] - xm);
            qs += q[d];
        }
        for (int d = 0; d < D; ++d) q[d] /= qs;
    }
    const float sc = ce ? ce_w / (float)cnt * invB : 0.f;
    float ce_term = 0.f;
    for (int d = 0; d < D; ++d) {
        const float pr = pb[d * hw];
        float v = g != 0.f ? g * pr * (di - (float)d) : 0.f;
        if (ce) {
            v += (q[d] - pr) * sc;
            if (pr > 1.0e-12f) ce_term -= q[d] * logf(pr);
        }
        gb[d * hw] = v;
    }
    term[i] = ce_term;
}

// Per-sample loss: 0.5 L0 + 0.7 L1 + 1.0 L2 + 2.0 CE (train_grads 1628-1649).
__global__ void __launch_bounds__(256)
    k_tloss(const float *__restrict__ t0, const float *__restrict__ t1,
            const float *__restrict__ t2, const float *__restrict__ tce, long n4, long n2,
            long n1, const int *__restrict__ counts, double *__restrict__ loss) {
    pdl_sync();
    __shared__ double s[4][256];
    const int b = blockIdx.x, t = threadIdx.x;
    double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    for (long i = t; i < n4; i += 256) { a0 += t0[b * n4 + i]; a3 += tce[b * n4 + i]; }
    for (long i = t; i < n2; i += 256) a1 += t1[b * n2 + i];
    for (long i = t; i < n1; i += 256) a2 += t2[b * n1 + i];
    s[0][t] = a0; s[1][t] = a1; s[2][t] = a2; s[3][t] = a3;
    __syncthreads();
    for (int k = 128; k > 0; k >>= 1) {
        if (t < k)
            for (int j = 0; j < 4; ++j) s[j][t] += s[j][t + k];
        __syncthreads();
    }
    if (t == 0) {
        const int *c = counts + b * 4;
        double l = 0.0;
        if (c[0]) l += 0.5 * (s[0][0] / c[0]);
        if (c[1]) l += 0.7 * (s[1][0] / c[1]);
        if (c[2]) l += 1.0 * (s[2][0] / c[2]);
        if (c[3]) l += 2.0 * (s[3][0] / c[3]);
        loss[b] = l;
    }
}

// ------------------------------------------------------------ backward
// Refinement output ReLU (slope 0): g where the output is positive.
__global__ void k_tmask0(const float *__restrict__ g, const float *__restrict__ out, long n,
                         float *__restrict__ gs) {
    pdl_sync();
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i < n) gs[i] = out[i] > 0.f ? g[i] : 0.f;
}

// Input gradient of a stride-2 3x3 convolution (528-570) with the leaky-ReLU
// derivative of the input: a thread computes the 2x2 inputs around an output
// pixel of every channel.  Input row 2a takes tap ky = 1 of output row a, row
// 2a + 1 taps ky = 2 of row a and ky = 0 of row a + 1; columns alike.
template <int IC, int OC>
__global__ void __launch_bounds__(128)
    k_tdgrad2d_s2(const float *__restrict__ gy, int nimg, int H, int W, int OH, int OW,
                  const float *__restrict__ w, const float *__restrict__ xin,
                  float *__restrict__ gx) {
    pdl_sync();
    constexpr int ICP = (IC + 3) / 4 * 4;
    __shared__ __align__(16) float sw[OC * 9 * ICP];       // [o][tap][c]
    for (int i = threadIdx.x; i < OC * 9 * ICP; i += blockDim.x) {
        const int c = i % ICP, ot = i / ICP, o = ot / 9, t = ot - o * 9;
        sw[i] = c < IC ? w[(o * IC + c) * 9 + t] : 0.f;
    }
    __syncthreads();
    const int qw = (W + 1) / 2, qh = (H + 1) / 2;
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= (long)nimg * qh * qw) return;
    const int img = (int)(i / (qh * qw)), r = (int)(i - (long)img * qh * qw);
    const int a = r / qw, b = r - a * qw;
    const long OHW = (long)OH * OW, HW = (long)H * W;
    const float *g = gy + (long)img * OC * OHW + (long)a * OW + b;
    const bool ya = a < OH, yb = a + 1 < OH, xa = b < OW, xb = b + 1 < OW;
    // one of the four inputs at a time, its taps in order, a tap's channels inner
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            float acc[IC];
#pragma unroll
            for (int c = 0; c < IC; ++c) acc[c] = 0.f;
#pragma unroll
            for (int ky = 1 - u; ky < 3; ky += 1 + u)
#pragma unroll
                for (int kx = 1 - v; kx < 3; kx += 1 + v) {
                    if ((u == 0 && ky != 1) || (v == 0 && kx != 1)) continue;
                    const bool on = (ky == 0 ? yb : ya) && (kx == 0 ? xb : xa);
                    const float *gt = g + (ky == 0 ? OW : 0) + (kx == 0 ? 1 : 0);
                    float e[OC];
#pragma unroll
                    for (int o = 0; o < OC; ++o) e[o] = on ? gt[o * OHW] : 0.f;
#pragma unroll
                    for (int o = 0; o < OC; ++o) {
                        const float *wt = sw + (o * 9 + ky * 3 + kx) * ICP;
#pragma unroll
                        for (int c4 = 0; c4 < ICP; c4 += 4) {
                            const float4 f = *reinterpret_cast<const float4 *>(wt + c4);
                            const float wv[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                if (c4 + k < IC) acc[c4 + k] = fmaf(wv[k], e[o], acc[c4 + k]);
                        }
                    }
                }
            const int iy = 2 * a + u, ix = 2 * b + v;
            if (iy >= H || ix >= W) continue;
#pragma unroll
            for (int c = 0; c < IC; ++c) {
                const long p = ((long)img * IC + c) * HW + (long)iy * W + ix;
                gx[p] = xin[p] > 0.f ? acc[c] : acc[c] * 0.2f;
            }
        }
}

// Weight gradients, per-CTA partial sums.  A CTA walks tiles t = blockIdx.x,
// blockIdx.x + gridDim.x, ... of 4 x 32 outputs (a fixed assignment, so the sums
// are deterministic): the input patch and the output gradients come to shared memory by asynchronous copies, in 2-D a tile ahead.
// A thread owns a row of taps -- (c, ky), or (c, kd, ky) in 3-D -- for OG output
// channels: 3 x OG sums, each one chain of FMAs over the CTA's pixels in order, so
// a sum does not depend on how the rows are dealt to threads.  Four columns take
// one 16-byte read of the patch and one per channel of gradients (a broadcast) for
// 12 x OG FMAs (one tap per thread and a gradient read per FMA: 8 x 8 channels 114
// us, 12 x 6 in 3-D 170 us for 64 crops of 96x64; now 30 and 59).  One more row per channel group sums the gradients themselves
// (the bias).  partial[cta][o][k], k < K - 1 the taps, k == K - 1 the bias.
constexpr int kWgCtas = 4 * 148;
constexpr int kWgThreads = 128;

template <int OC, int ROWS>             // ROWS: rows of taps, the bias one included
struct WgSplit {
    // as many threads at work as there are: 8 x 8 channels took 71 us on one warp (OG
    // 8, every gradient read once), 47 on two (4)
    static constexpr int groups() {
        int n = 1;
        for (int g = 2; g <= OC; ++g)
            if (OC % g == 0 && ROWS * g <= kWgThreads) n = g;
        return n;
    }
    static constexpr int NOG = groups(), OG = OC / NOG, N = ROWS * NOG;
    static constexpr int GSZ = OC * 128 + 4 * NOG;         // groups 4 floats apart: other banks
    static_assert(OC % OG == 0 && N <= kWgThreads, "a row of taps per thread");
};

// The staged width of a patch row and where column ox0 * S lies in it: rows start
// 4 columns early (8 when the dilation is read at run time), 16-byte aligned.
template <int S, int DIL>
struct WgRow {
    static constexpr int PAD = DIL > 0 ? 4 : 8;
    static constexpr int NCH = S == 2 ? 17 : DIL > 0 ? 10 : 12;     // 16-byte chunks
    static constexpr int RW = NCH % 2 ? 4 * NCH : 4 * NCH + 4;      // odd number: spreads banks
};

__device__ __forceinline__ void cp16(float *dst, const float *src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(on ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp4(float *dst, const float *src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(on ? 4 : 0)
                 : "memory");
}

// nrows patch rows to rows of RW floats, zeros outside [0, W); src(r) is the row's
// pointer or NULL.  16-byte copies where W and the base allow them: a chunk is
// then inside the row or outside.
template <typename Rw, typename R>
__device__ __forceinline__ void patch_rows(float *dst, int nrows, int tid, int xs, int W, bool vec,
                                           const float *base, R src) {
    if (vec) {
        for (int i = tid; i < nrows * Rw::NCH; i += kWgThreads) {
            const int r = i / Rw::NCH, ch = i - r * Rw::NCH, xx = xs + 4 * ch;
            const float *p = src(r);
            const bool on = p && xx >= 0 && xx < W;
            cp16(dst + r * Rw::RW + 4 * ch, on ? p + xx : base, on);
        }
    } else {
        for (int i = tid; i < nrows * Rw::NCH * 4; i += kWgThreads) {
            const int r = i / (Rw::NCH * 4), j = i - r * (Rw::NCH * 4), xx = xs + j;
            const float *p = src(r);
            const bool on = p && xx >= 0 && xx < W;
            cp4(dst + r * Rw::RW + j, on ? p + xx : base, on);
        }
    }
}

// a tile's gradients to [OC][4][32], a group of channels 4 floats after the last;
// src(o, r) is row r's pointer, of which n columns exist, or NULL
template <int OC, int OG, typename R>
__device__ __forceinline__ void tile_grads(float *dst, int tid, int n, bool vec, const float *base,
                                           R src) {
    if (vec) {
        for (int i = tid; i < OC * 32; i += kWgThreads) {
            const int o = i >> 5, r = (i >> 3) & 3, j = 4 * (i & 7);
            const float *p = src(o, r);
            const bool on = p && j < n;
            cp16(dst + o * 128 + 4 * (o / OG) + r * 32 + j, on ? p + j : base, on);
        }
    } else {
        for (int i = tid; i < OC * 128; i += kWgThreads) {
            const int o = i >> 7, r = (i >> 5) & 3, j = i & 31;
            const float *p = src(o, r);
            const bool on = p && j < n;
            cp4(dst + o * 128 + 4 * (o / OG) + r * 32 + j, on ? p + j : base, on);
        }
    }
}

// n4 groups of four columns of one row: xr the patch row (of the taps' first
// column when DIL is 0), gr the row's gradients of this thread's channels
template <int S, int DIL, int OG>
__device__ __forceinline__ void row_taps(const float *xr, const float *gr, int n4, int dil, bool bias,
                                         float (&acc)[3][OG]) {
    constexpr int B0 = DIL > 0 ? 4 - DIL : 0, STEP = 4 * S, KEEP = 12 - STEP;
    static_assert(DIL == 0 || B0 + 3 * S + 2 * DIL < 12, "a window of 12 columns");
    float v[12];
    if constexpr (DIL > 0) {
#pragma unroll
        for (int j = 0; j < KEEP; j += 4) {
            const float4 f = *reinterpret_cast<const float4 *>(xr + j);
            v[j] = f.x; v[j + 1] = f.y; v[j + 2] = f.z; v[j + 3] = f.w;
        }
    }
#pragma unroll 4
    for (int n = 0; n < n4; ++n) {
        float g[OG][4];
#pragma unroll
        for (int o = 0; o < OG; ++o) {
            const float4 f = *reinterpret_cast<const float4 *>(gr + o * 128 + 4 * n);
            g[o][0] = f.x; g[o][1] = f.y; g[o][2] = f.z; g[o][3] = f.w;
        }
        if constexpr (DIL > 0) {
#pragma unroll
            for (int j = KEEP; j < 12; j += 4) {
                const float4 f = *reinterpret_cast<const float4 *>(xr + n * STEP + j);
                v[j] = f.x; v[j + 1] = f.y; v[j + 2] = f.z; v[j + 3] = f.w;
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                float xv;
                if constexpr (DIL > 0) xv = v[B0 + q * S + j * DIL];
                else xv = xr[(4 * n + q) * S + j * dil];
                if (bias) xv = 1.f;
#pragma unroll
                for (int o = 0; o < OG; ++o) acc[j][o] = fmaf(xv, g[o][q], acc[j][o]);
            }
        if constexpr (DIL > 0) {
#pragma unroll
            for (int j = 0; j < KEEP; ++j) v[j] = v[j + STEP];
        }
    }
}

// A thread's place in the CTA's work.  Warp w of a CTA runs on scheduler w % 4, and
// most layers keep one or two of the four warps busy, so they are turned by the
// CTA's place on its SM.  Who computes a sum does not change it.
__device__ __forceinline__ int wg_item(int tid) {
    __shared__ int slot;
    if (tid == 0) {
        unsigned id;
        asm volatile("mov.u32 %0, %%warpid;" : "=r"(id));
        slot = (int)(id >> 2);
    }
    __syncthreads();
    return (((tid >> 5) + slot) & 3) * 32 + (tid & 31);
}

template <int IC, int OC, int S, int DIL>
__global__ void __launch_bounds__(kWgThreads)
    k_twgrad2d(const float *__restrict__ x, const float *__restrict__ gy, int nimg, int H, int W,
               int OH, int OW, int dil_, float *__restrict__ partial) {
    pdl_sync();
    using G = WgSplit<OC, IC * 3 + 1>;
    using Rw = WgRow<S, DIL>;
    constexpr int K = IC * 9 + 1;
    const int dil = DIL > 0 ? DIL : dil_;
    extern __shared__ __align__(16) float sm[];
    const int th = 3 * S + 2 * dil + 1;
    const int bufsz = G::GSZ + IC * th * Rw::RW;           // gradients, then [IC][th][RW]
    const int tid = threadIdx.x, item = wg_item(tid);
    const bool on = item < G::N;
    const int row = on ? item / G::NOG : 0, og = on ? item - row * G::NOG : 0;
    const bool bias = row == IC * 3;
    const int c = bias ? 0 : row / 3, ky = bias ? 0 : row - c * 3;
    const long HW = (long)H * W, OHW = (long)OH * OW;
    const int tx_n = (OW + 31) / 32, ty_n = (OH + 3) / 4;
    const long ntiles = (long)nimg * tx_n * ty_n;
    const bool vec = (W & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    const bool gvec = (OW & 3) == 0 && (reinterpret_cast<uintptr_t>(gy) & 15) == 0;
    auto fetch = [&](long tile, float *buf) {
        const int img = (int)(tile / (tx_n * ty_n));
        const int rem = (int)(tile - (long)img * tx_n * ty_n);
        const int oy0 = rem / tx_n * 4, ox0 = rem % tx_n * 32;
        const float *gi = gy + (long)img * OC * OHW, *xi = x + (long)img * IC * HW;
        const int iy0 = oy0 * S - dil;
        tile_grads<OC, G::OG>(buf, tid, OW - ox0, gvec, gy, [&](int o, int r) -> const float * {
            return oy0 + r < OH ? gi + o * OHW + (long)(oy0 + r) * OW + ox0 : nullptr;
        });
        patch_rows<Rw>(buf + G::GSZ, IC * th, tid, ox0 * S - Rw::PAD, W, vec, x,
                       [&](int r) -> const float * {
                           const int cc = r / th, yy = iy0 + r - cc * th;
                           return yy >= 0 && yy < H ? xi + cc * HW + (long)yy * W : nullptr;
                       });
    };
    float acc[3][G::OG];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int o = 0; o < G::OG; ++o) acc[j][o] = 0.f;
    fetch(blockIdx.x, sm);
    asm volatile("cp.async.commit_group;" ::: "memory");
    int cur = 0;
    for (long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, cur ^= 1) {
        if (tile + gridDim.x < ntiles) fetch(tile + gridDim.x, sm + (cur ^ 1) * bufsz);
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        if (on) {
            const int rem = (int)(tile % (tx_n * ty_n));
            const int oy0 = rem / tx_n * 4, ox0 = rem % tx_n * 32;
            const int n4 = (min(32, OW - ox0) + 3) / 4, ny = min(4, OH - oy0);
            const float *gt = sm + cur * bufsz + og * (G::OG * 128 + 4), *xt = sm + cur * bufsz + G::GSZ;
            const float *xr = xt + (c * th + ky * dil) * Rw::RW + (DIL > 0 ? 0 : Rw::PAD - dil);
            for (int r = 0; r < ny; ++r)
                row_taps<S, DIL, G::OG>(xr + r * S * Rw::RW, gt + r * 32, n4, dil, bias, acc);
        }
        __syncthreads();                                   // before the next fetch into this buffer
    }
    if (!on) return;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int o = 0; o < G::OG; ++o)
            if (!bias || j == 0)
                partial[((long)blockIdx.x * OC + og * G::OG + o) * K + row * 3 + j] = acc[j][o];
}

template <int IC, int OC, int S, int DIL>
size_t twgrad2d_smem(int dil) {
    return 2 * sizeof(float) * (WgSplit<OC, IC * 3 + 1>::GSZ +
                                (size_t)IC * (3 * S + 2 * dil + 1) * WgRow<S, DIL>::RW);
}

// 3-D: a tile is one sample's 4 disparities x 1 row x 32 columns.  One buffer: two
// would leave room for half the CTAs, and these cover each other's copies.
template <int IC, int OC>
struct Wg3 {
    using G = WgSplit<OC, IC * 9 + 1>;
    using Rw = WgRow<1, 1>;
    static constexpr int K = IC * 27 + 1;
    static constexpr size_t SMEM = sizeof(float) * (G::GSZ + IC * 18 * Rw::RW);
};

template <int IC, int OC>
__global__ void __launch_bounds__(kWgThreads)
    k_twgrad3d(const float *__restrict__ x, const float *__restrict__ gy, int B, int D, int h,
               int w, float *__restrict__ partial) {
    pdl_sync();
    using G = typename Wg3<IC, OC>::G;
    using Rw = typename Wg3<IC, OC>::Rw;
    constexpr int K = Wg3<IC, OC>::K;
    extern __shared__ __align__(16) float sm[];
    float *gt = sm, *xt = sm + G::GSZ;                     // gradients; [IC][6][3][RW]
    const int tid = threadIdx.x, item = wg_item(tid);
    const bool on = item < G::N;
    const int row = on ? item / G::NOG : 0, og = on ? item - row * G::NOG : 0;
    const bool bias = row == IC * 9;
    const int c = bias ? 0 : row / 9, kd = bias ? 0 : row % 9 / 3, ky = bias ? 0 : row % 3;
    const int nd = (D + 3) / 4, nxt = (w + 31) / 32;
    const long ntiles = (long)B * h * nd * nxt;
    const long hw = (long)h * w, total = (long)D * hw;
    const bool vec = (w & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    const bool gvec = (w & 3) == 0 && (reinterpret_cast<uintptr_t>(gy) & 15) == 0;
    float acc[3][G::OG];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int o = 0; o < G::OG; ++o) acc[j][o] = 0.f;
    for (long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int b = (int)(tile / ((long)h * nd * nxt));
        const int rem = (int)(tile - (long)b * h * nd * nxt);
        const int oy = rem / (nd * nxt), r2 = rem - oy * nd * nxt;
        const int d0 = (r2 / nxt) * 4, x0 = (r2 % nxt) * 32;
        const float *gi = gy + (long)b * OC * total, *xi = x + (long)b * IC * total;
        __syncthreads();                                   // the previous tile's reads are done
        tile_grads<OC, G::OG>(gt, tid, w - x0, gvec, gy, [&](int o, int r) -> const float * {
            return d0 + r < D ? gi + o * total + (d0 + r) * hw + (long)oy * w + x0 : nullptr;
        });
        patch_rows<Rw>(xt, IC * 18, tid, x0 - Rw::PAD, w, vec, x, [&](int r) -> const float * {
            const int cc = r / 18, rr = r - cc * 18, dz = rr / 3;
            const int dd = d0 - 1 + dz, yy = oy - 1 + rr - dz * 3;
            return dd >= 0 && dd < D && yy >= 0 && yy < h
                       ? xi + cc * total + dd * hw + (long)yy * w
                       : nullptr;
        });
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (on) {
            const int n4 = (min(32, w - x0) + 3) / 4, nz = min(4, D - d0);
            const float *xr = xt + (c * 18 + kd * 3 + ky) * Rw::RW;
            for (int r = 0; r < nz; ++r)
                row_taps<1, 1, G::OG>(xr + r * 3 * Rw::RW, gt + og * (G::OG * 128 + 4) + r * 32, n4, 1,
                                      bias, acc);
        }
    }
    if (!on) return;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int o = 0; o < G::OG; ++o)
            if (!bias || j == 0)
                partial[((long)blockIdx.x * OC + og * G::OG + o) * K + row * 3 + j] = acc[j][o];
}

// CTA partials -> every layer's weight and bias gradient in FP64, one launch (a
// launch per layer took 12 us each, 15 of them).  A block takes 32 weights of one
// layer (threadIdx.x); its 32 rows (threadIdx.y) add the partials t = y, y + 32,
// ... in order, and row sums are then added in row order, so the result does not
// depend on scheduling.  Parameter layout: weights [o][taps], then bias [o].
constexpr int kMaxLayers = 25;          // 4 + 3 + 2 * (8 + 1)
struct ReduceJobs {
    int n;
    int block[kMaxLayers + 1];          // first block of each layer
    int nblk[kMaxLayers], OC[kMaxLayers], K[kMaxLayers];
    long partial[kMaxLayers], gw[kMaxLayers], gb[kMaxLayers];      // offsets
};

__global__ void __launch_bounds__(1024)
    k_treduce(const float *__restrict__ partials, ReduceJobs jobs, double *__restrict__ grads) {
    pdl_sync();
    __shared__ double rs[32][33];
    int l = 0;
    while ((int)blockIdx.x >= jobs.block[l + 1]) ++l;
    const int j = (blockIdx.x - jobs.block[l]) * 32 + threadIdx.x, OC = jobs.OC[l], K = jobs.K[l];
    const long stride = (long)OC * K;
    const float *partial = partials + jobs.partial[l];
    double s = 0.0;
    if (j < OC * K)
        for (int t = threadIdx.y; t < jobs.nblk[l]; t += 32) s += (double)partial[t * stride + j];
    rs[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y != 0 || j >= OC * K) return;
    double tot = 0.0;
    for (int y = 0; y < 32; ++y) tot += rs[y][threadIdx.x];
    const int o = j / K, k = j - o * K;
    if (k < K - 1) grads[jobs.gw[l] + o * (K - 1) + k] = tot;
    else grads[jobs.gb[l] + o] = tot;
}

// CostVolume.backward (801-824) as a gather: gfl[c][y][x] sums over d the
// gradient times sign(fl - fr(x - d)); gfr[c][y][x] subtracts it at x + d.
__global__ void k_tcostvol_bwd(const float *__restrict__ gvol, const float *__restrict__ f,
                               int B, int C, int D, int h, int w, float *__restrict__ gf) {
    pdl_sync();
    const long hw = (long)h * w, n = (long)B * C * hw;
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = (int)(i / (C * hw));
    const long r = i - (long)b * C * hw;
    const int c = (int)(r / hw);
    const long p = r - (long)c * hw;
    const int y = (int)(p / w), x = (int)(p - (long)y * w);
    const float *fl = f + ((long)b * C + c) * hw + (long)y * w;
    const float *fr = f + ((long)(B + b) * C + c) * hw + (long)y * w;
    const float *g = gvol + ((long)b * C + c) * D * hw + (long)y * w;
    float al = 0.f, ar = 0.f;
    for (int d = 0; d < D; ++d) {
        if (x - d >= 0) {
            const float v = fl[x] - fr[x - d];
            const float gg = g[d * hw + x];
            al += v < 0.f ? -gg : gg;
        }
        if (x + d < w) {
            const float v = fl[x + d] - fr[x];
            const float gg = g[d * hw + x + d];
            ar -= v < 0.f ? -gg : gg;
        }
    }
    gf[((long)b * C + c) * hw + p] = al;
    gf[((long)(B + b) * C + c) * hw + p] = ar;
}

// BilinearUpsample.backward (958-974) of `2 * (grin0 + gs)` from the
// (H2, W2) level to the (h, w) level, as a gather over the destination
// pixels whose taps touch (ys, xs); plus `add`; times (mask > 0) when a mask
// is given (the previous level's output ReLU).
__global__ void k_tup_bwd(const float *__restrict__ grin, long grin_stride,
                          const float *__restrict__ gs, int B, int H2, int W2, int h, int w,
                          int ry, int rx, const float *__restrict__ add,
                          const float *__restrict__ mask, float *__restrict__ out) {
    pdl_sync();
    const long hw = (long)h * w, n2 = (long)H2 * W2;
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= B * hw) return;
    const int b = (int)(i / hw);
    const long p = i - b * hw;
    const int ys = (int)(p / w), xs = (int)(p - (long)ys * w);
    const float *g1 = grin + b * grin_stride;
    const float *g2 = gs + (long)b * n2;
    // destination rows / columns whose source taps can reach (ys, xs): of a
    // window that surely holds them, the ones whose two taps do (BilinearUpsample's
    // positions, as bilinear_taps computes them)
    const int cy = (int)(((double)ys + 0.5) * H2 / h), cx = (int)(((double)xs + 0.5) * W2 / w);
    const double sy = __ddiv_rn((double)h, (double)H2), sx = __ddiv_rn((double)w, (double)W2);
    auto tap = [](int o, double sc, int n, int &i0, int &i1, double &wt) {
        double f = __dsub_rn(__dmul_rn(__dadd_rn((double)o, 0.5), sc), 0.5);
        if (f < 0.0) f = 0.0;
        i0 = (int)f;
        if (i0 > n - 1) i0 = n - 1;
        i1 = i0 + 1 < n ? i0 + 1 : i0;
        wt = __dsub_rn(f, (double)i0);
    };
    int lo = W2, hi = -1;
    for (int ox = max(0, cx - rx); ox <= min(W2 - 1, cx + rx); ++ox) {
        int a0, a1;
        double wt;
        tap(ox, sx, w, a0, a1, wt);
        if (a0 == xs || a1 == xs) {
            lo = min(lo, ox);
            hi = ox;
        }
    }
    float acc = 0.f;
    for (int oy = max(0, cy - ry); oy <= min(H2 - 1, cy + ry); ++oy) {
        int y0, y1;
        double wy;
        tap(oy, sy, h, y0, y1, wy);
        if (y0 != ys && y1 != ys) continue;
        for (int ox = lo; ox <= hi; ++ox) {
            int x0, x1;
            double wx;
            tap(ox, sx, w, x0, x1, wx);
            float wgt = 0.f;
            if (y0 == ys && x0 == xs) wgt += (float)__dmul_rn(__dsub_rn(1.0, wy), __dsub_rn(1.0, wx));
            if (y0 == ys && x1 == xs) wgt += (float)__dmul_rn(__dsub_rn(1.0, wy), wx);
            if (y1 == ys && x0 == xs) wgt += (float)__dmul_rn(wy, __dsub_rn(1.0, wx));
            if (y1 == ys && x1 == xs) wgt += (float)__dmul_rn(wy, wx);
            if (wgt != 0.f) {
                const long q = (long)oy * W2 + ox;
                acc = fmaf((g1[q] + g2[q]) * 2.0f, wgt, acc);
            }
        }
    }
    float v = acc + add[i];
    if (mask) v = mask[i] > 0.f ? v : 0.f;
    out[i] = v;
}

// Adam.step (1368-1387) in FP64 on the master parameters; refreshes the
// FP32 copy the kernels read.
__global__ void k_tadam(double *__restrict__ p, const double *__restrict__ g,
                        double *__restrict__ m, double *__restrict__ v, long n, double lr,
                        double c1, double c2, double clip, float *__restrict__ p32) {
    pdl_sync();
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double b1 = 0.9, b2 = 0.999, eps = 1.0e-8;
    double gi = g[i];
    if (gi > clip) gi = clip;
    else if (gi < -clip) gi = -clip;
    const double mi = b1 * m[i] + (1.0 - b1) * gi;
    const double vi = b2 * v[i] + (1.0 - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const double pi = p[i] - lr * (mi * c1) / (sqrt(vi * c2) + eps);
    p[i] = pi;
    p32[i] = (float)pi;
}

__global__ void k_f64_to_f32(const double *__restrict__ a, long n, float *__restrict__ b) {
    pdl_sync();
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i < n) b[i] = (float)a[i];
}

unsigned nblocks(long n, int t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace
}  // namespace sv

using namespace sv;

// --------------------------------------------------------------- trainer
struct sv_trainer {
    int arch[13];
    int C, Cm, D, Rc, nd, dil[8];
    long np;
    long off_fw[4], off_fb[4], off_cw[3], off_cb[3], off_rw[2][9], off_rb[2][9];
    double *p64 = nullptr, *g64 = nullptr, *m = nullptr, *v = nullptr;
    float *p32 = nullptr;
    double b1t = 1.0, b2t = 1.0;
};

namespace {

long layout(sv_trainer *t) {
    long p = 0;
    const int fic[4] = {1, t->C, t->C, t->C};
    for (int i = 0; i < 4; ++i) {
        t->off_fw[i] = p; p += (long)t->C * fic[i] * 9;
        t->off_fb[i] = p; p += t->C;
    }
    const int cic[3] = {t->C, t->Cm, t->Cm}, coc[3] = {t->Cm, t->Cm, 1};
    for (int i = 0; i < 3; ++i) {
        t->off_cw[i] = p; p += (long)coc[i] * cic[i] * 27;
        t->off_cb[i] = p; p += coc[i];
    }
    for (int lv = 0; lv < 2; ++lv) {
        int prev = 2;
        for (int i = 0; i < t->nd; ++i) {
            t->off_rw[lv][i] = p; p += (long)t->Rc * prev * 9;
            t->off_rb[lv][i] = p; p += t->Rc;
            prev = t->Rc;
        }
        t->off_rw[lv][t->nd] = p; p += (long)prev * 9;
        t->off_rb[lv][t->nd] = p; p += 1;
    }
    return p;
}

struct TrainBufs {
    float *img, *a1, *a2, *a3, *f4, *vol, *b1, *b2, *cost, *probs, *d0;
    float *rin[2], *r[2][8], *out[2];
    float *dh, *gh, *dq;
    uint8_t *vh, *vq;
    int *counts;
    float *t0, *t1, *t2, *tce, *gl0, *gl1, *gl2;
    float *gs, *gs0, *gA, *gB, *grin, *gd0, *gcost, *gq2, *gq1, *gvol, *gf, *gF3, *gF4;
    float *partial;
    long partial_n;
    double *loss;
};

struct Dims {
    int B, H, W, h1, w1, h, w, H2, W2;
    long HW, HW2, hw, h1w1;
};

Dims dims(int B, int W, int H) {
    Dims d;
    d.B = B; d.H = H; d.W = W;
    d.h1 = (H - 1) / 2 + 1; d.w1 = (W - 1) / 2 + 1;
    d.h = (d.h1 - 1) / 2 + 1; d.w = (d.w1 - 1) / 2 + 1;
    d.H2 = H / 2; d.W2 = W / 2;
    d.HW = (long)H * W; d.HW2 = (long)d.H2 * d.W2; d.hw = (long)d.h * d.w;
    d.h1w1 = (long)d.h1 * d.w1;
    return d;
}

long tiles2d(int nimg, int OH, int OW) {
    return (long)nimg * ((OH + 3) / 4) * ((OW + 31) / 32);
}

// Partial sums, at most kWgCtas CTAs a layer: of every layer, so that one launch adds
// them all up, or (all false) of the widest one, the least a step can do with.
long partial_floats(const sv_trainer *t, bool all) {
    const int C = t->C, Cm = t->Cm, Rc = t->Rc;
    if (!all) {
        const long layers[3] = {(long)C * (C * 9 + 1), (long)Cm * (C * 27 + 1),
                                (long)Rc * (Rc * 9 + 1)};
        return *std::max_element(layers, layers + 3) * kWgCtas;
    }
    long n = (long)C * (9 + 1) + 3L * C * (C * 9 + 1);
    n += (long)Cm * (C * 27 + 1) + (long)Cm * (Cm * 27 + 1) + (Cm * 27 + 1);
    n += 2L * (Rc * (2 * 9 + 1) + (long)(t->nd - 1) * Rc * (Rc * 9 + 1) + (Rc * 9 + 1));
    return n * kWgCtas;
}

void carve(const sv_trainer *t, const Dims &d, Carver &cv, TrainBufs &b, bool all) {
    const int B = d.B, C = t->C, Cm = t->Cm, D = t->D, Rc = t->Rc;
    const long DHW = (long)D * d.hw;
    b.img = cv.take<float>(2 * B * d.HW);
    b.a1 = cv.take<float>(2L * B * C * d.h1w1);
    b.a2 = cv.take<float>(2L * B * C * d.hw);
    b.a3 = cv.take<float>(2L * B * C * d.hw);
    b.f4 = cv.take<float>(2L * B * C * d.hw);
    b.vol = cv.take<float>((long)B * C * DHW);
    b.b1 = cv.take<float>((long)B * Cm * DHW);
    b.b2 = cv.take<float>((long)B * Cm * DHW);
    b.cost = cv.take<float>((long)B * DHW);
    b.probs = cv.take<float>((long)B * DHW);
    b.d0 = cv.take<float>((long)B * d.hw);
    const long HWl[2] = {d.HW2, d.HW};
    for (int lv = 0; lv < 2; ++lv) {
        b.rin[lv] = cv.take<float>(2L * B * HWl[lv]);
        for (int i = 0; i < t->nd; ++i) b.r[lv][i] = cv.take<float>((long)B * Rc * HWl[lv]);
        b.out[lv] = cv.take<float>((long)B * HWl[lv]);
    }
    b.dh = cv.take<float>((long)B * d.HW2);
    b.gh = cv.take<float>((long)B * d.HW2);
    b.dq = cv.take<float>((long)B * d.hw);
    b.vh = cv.take<uint8_t>((long)B * d.HW2);
    b.vq = cv.take<uint8_t>((long)B * d.hw);
    b.counts = cv.take<int>(4L * B);
    b.t0 = cv.take<float>((long)B * d.hw);
    b.t1 = cv.take<float>((long)B * d.HW2);
    b.t2 = cv.take<float>((long)B * d.HW);
    b.tce = cv.take<float>((long)B * d.hw);
    b.gl0 = cv.take<float>((long)B * d.hw);
    b.gl1 = cv.take<float>((long)B * d.HW2);
    b.gl2 = cv.take<float>((long)B * d.HW);
    b.gs = cv.take<float>((long)B * d.HW);
    b.gs0 = cv.take<float>((long)B * d.HW2);
    b.gA = cv.take<float>((long)B * Rc * d.HW);
    b.gB = cv.take<float>((long)B * Rc * d.HW);
    b.grin = cv.take<float>((long)B * d.HW);
    b.gd0 = cv.take<float>((long)B * d.hw);
    b.gcost = cv.take<float>((long)B * DHW);
    b.gq2 = cv.take<float>((long)B * Cm * DHW);
    b.gq1 = cv.take<float>((long)B * Cm * DHW);
    b.gvol = cv.take<float>((long)B * C * DHW);
    b.gf = cv.take<float>(2L * B * C * d.hw);
    b.gF3 = cv.take<float>(2L * B * C * d.h1w1);
    b.gF4 = cv.take<float>(2L * B * C * d.hw);
    b.partial_n = partial_floats(t, all);
    b.partial = cv.take<float>(b.partial_n);
    b.loss = cv.take<double>(B);
}

constexpr int kMaxDil = 8, kMaxD = 16;     // of a trainable architecture

// Raised limit of a kernel that stages more than the default 48 KB; most: the largest
// that any architecture asks of it.
template <typename F>
int big_smem(F *f, size_t sm, size_t most, const char *what) {
    if (sm > 200 * 1024) {
        set_error("%s needs %zu bytes of shared memory", what, sm);
        return SV_ERR_SHAPE;
    }
    return allow_smem(f, sm, most);
}

template <int IC, int OC, int WC, int S, int DIL, int MODE, bool FLIP, int TR>
int conv2d_go(const float *x, int nimg, int H, int W, int OH, int OW, int dil, const float *w,
              const float *b, float *y, const float *aux, long stride, cudaStream_t st) {
    const size_t sm = tconv2d_smem(IC, S, dil, TR);
    const int rc = big_smem(k_tconv2d<IC, OC, WC, S, DIL, MODE, FLIP, TR>, sm,
                            tconv2d_smem(IC, S, DIL > 0 ? DIL : kMaxDil, TR), "convolution tile");
    if (rc) return rc;
    const dim3 g((OW + 31) / 32, (OH + TR - 1) / TR, nimg);
    count_launch();
    pdl(k_tconv2d<IC, OC, WC, S, DIL, MODE, FLIP, TR>, g, 8 * TR, sm, st)(x, H, W, OH, OW, dil, w, b,
                                                                         y, aux, stride);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

// stride 1: the dilations of the shipped nets fixed, others at run time
template <int IC, int OC, int WC, int MODE, bool FLIP>
int conv2d_s1(const float *x, int nimg, int H, int W, int dil, const float *w, const float *b,
              float *y, const float *aux, long stride, cudaStream_t st) {
#define SV_C2(DIL) \
    return conv2d_go<IC, OC, WC, 1, DIL, MODE, FLIP, 16>(x, nimg, H, W, H, W, dil, w, b, y, aux, stride, st)
    switch (dil) {
    case 1: SV_C2(1);
    case 2: SV_C2(2);
    case 4: SV_C2(4);
    default: SV_C2(0);
    }
#undef SV_C2
}

template <int IC, int OC, int WC, int CCH, int MODE, bool FLIP, int nxg = 8>
int conv3d_go(const float *x, int B, int D, int h, int w, const float *wt, const float *b, float *y,
              const float *xin, cudaStream_t st) {
    if (nxg == 8 && w <= 24)                               // groups of 4 columns
        return conv3d_go<IC, OC, WC, CCH, MODE, FLIP, 6>(x, B, D, h, w, wt, b, y, xin, st);
    auto tile = [](int d) { return sizeof(float) * CCH * (d + 2) * 3 * (4 * nxg + 4); };
    const size_t sm = tile(D);
    const int rc = big_smem(k_tconv3d<IC, OC, WC, CCH, MODE, FLIP, nxg>, sm, tile(kMaxD),
                            "3-D convolution tile");
    if (rc) return rc;
    const dim3 g((w + 4 * nxg - 1) / (4 * nxg), h, B);
    count_launch();
    pdl(k_tconv3d<IC, OC, WC, CCH, MODE, FLIP, nxg>, g, (nxg * D + 31) / 32 * 32, sm, st)(
        x, D, h, w, wt, b, y, xin);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

// The weight gradients leave their partial sums in b.partial and a job each; reduce
// adds up the ones there: at the end, or before a layer whose sums no longer fit.
struct WGrads {
    float *partial;
    long cap;
    double *grads;
    cudaStream_t st;
    long used = 0;
    ReduceJobs jobs{};
    void reduce() {
        count_launch();
        pdl(k_treduce, jobs.block[jobs.n], dim3(32, 32), 0, st)(partial, jobs, grads);
        jobs = ReduceJobs{};
        used = 0;
    }
    int add(int nblk, int OC, int K, long gw, long gb) {
        if (used + (long)nblk * OC * K > cap) reduce();
        const int l = jobs.n++;
        jobs.nblk[l] = nblk;
        jobs.OC[l] = OC;
        jobs.K[l] = K;
        jobs.partial[l] = used;
        jobs.gw[l] = gw;
        jobs.gb[l] = gb;
        jobs.block[l + 1] = jobs.block[l] + (OC * K + 31) / 32;
        used += (long)nblk * OC * K;
        return l;
    }
};

template <int IC, int OC, int S, int DIL>
int wgrad2d_go(const float *x, const float *gy, int nimg, int H, int W, int OH, int OW, int dil,
               WGrads &g, long gw, long gb, cudaStream_t st) {
    const size_t sm = twgrad2d_smem<IC, OC, S, DIL>(dil);
    const int rc = big_smem(k_twgrad2d<IC, OC, S, DIL>, sm,
                            twgrad2d_smem<IC, OC, S, DIL>(DIL > 0 ? DIL : kMaxDil),
                            "weight-gradient tile");
    if (rc) return rc;
    const long ntiles = tiles2d(nimg, OH, OW);
    const int nblk = (int)(ntiles < kWgCtas ? ntiles : kWgCtas);
    const int l = g.add(nblk, OC, IC * 9 + 1, gw, gb);
    count_launch();
    pdl(k_twgrad2d<IC, OC, S, DIL>, nblk, kWgThreads, sm, st)(x, gy, nimg, H, W, OH, OW, dil,
                                                             g.partial + g.jobs.partial[l]);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

template <int IC, int OC, int S>
int wgrad2d(const float *x, const float *gy, int nimg, int H, int W, int OH, int OW, int dil,
            WGrads &g, long gw, long gb, cudaStream_t st) {
#define SV_W2(DIL) return wgrad2d_go<IC, OC, S, DIL>(x, gy, nimg, H, W, OH, OW, dil, g, gw, gb, st)
    if constexpr (S == 2) {                                // the feature net's: dilation 1
        SV_W2(1);
    } else {
        if (dil == 1) SV_W2(1);
        if (dil == 2) SV_W2(2);
        if (dil == 4) SV_W2(4);
        SV_W2(0);
    }
#undef SV_W2
}

template <int IC, int OC>
int wgrad3d(const float *x, const float *gy, int B, int D, int h, int w, WGrads &g, long gw, long gb,
            cudaStream_t st) {
    using Gm = Wg3<IC, OC>;
    const int rc = big_smem(k_twgrad3d<IC, OC>, Gm::SMEM, Gm::SMEM, "weight-gradient tile");
    if (rc) return rc;
    const long ntiles = (long)B * h * ((D + 3) / 4) * ((w + 31) / 32);
    const int nblk = (int)(ntiles < kWgCtas ? ntiles : kWgCtas);
    const int l = g.add(nblk, OC, Gm::K, gw, gb);
    count_launch();
    pdl(k_twgrad3d<IC, OC>, nblk, kWgThreads, Gm::SMEM, st)(x, gy, B, D, h, w,
                                                       g.partial + g.jobs.partial[l]);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

template <int C, int CM, int RC>
int train_impl(sv_trainer *t, const float *left, const float *right, const float *disp,
               const uint8_t *valid, const Dims &d, const TrainBufs &b, float *pred,
               double *loss, cudaStream_t st) {
    const int B = d.B, D = t->D, nd = t->nd;
    const float *P = t->p32;
    const float invB = 1.0f / (float)B;
    constexpr int CH = C % 4 == 0 ? 4 : C, CMH = CM % 3 == 0 ? 3 : 2;   // staged channels in 3-D
    WGrads wg{b.partial, b.partial_n, t->g64, st};
    int rc;
    // inputs: the B left views, then the B right views
    if (cudaMemcpyAsync(b.img, left, sizeof(float) * B * d.HW, cudaMemcpyDeviceToDevice, st) !=
            cudaSuccess ||
        cudaMemcpyAsync(b.img + (long)B * d.HW, right, sizeof(float) * B * d.HW,
                        cudaMemcpyDeviceToDevice, st) != cudaSuccess) {
        set_error("input copy failed");
        return SV_ERR_CUDA;
    }
    // ---- targets (build_targets) and counts
    count_launch();
    pdl(k_tpool, nblocks(B * d.HW2), 256, 0, st)(disp, valid, left, B, d.H, d.W, b.dh, b.vh, b.gh);
    count_launch();
    pdl(k_tpool, nblocks(B * d.hw), 256, 0, st)(b.dh, b.vh, nullptr, B, d.H2, d.W2, b.dq, b.vq,
                                               nullptr);
    count_launch();
    pdl(k_tcounts, B, 256, 0, st)(b.vq, b.vh, valid, b.dq, d.hw, d.HW2, d.HW, D, b.counts);
    SV_LAUNCH_CHECK();
    // ---- forward: FeatureNet on 2B images
    if ((rc = conv2d_go<1, C, C, 2, 1, 1, false, 16>(b.img, 2 * B, d.H, d.W, d.h1, d.w1, 1,
                                                     P + t->off_fw[0], P + t->off_fb[0], b.a1,
                                                     nullptr, 0, st)))
        return rc;
    if ((rc = conv2d_go<C, C, C, 2, 1, 1, false, 8>(b.a1, 2 * B, d.h1, d.w1, d.h, d.w, 1,
                                                    P + t->off_fw[1], P + t->off_fb[1], b.a2,
                                                    nullptr, 0, st)))
        return rc;
    if ((rc = conv2d_s1<C, C, C, 1, false>(b.a2, 2 * B, d.h, d.w, 1, P + t->off_fw[2],
                                           P + t->off_fb[2], b.a3, nullptr, 0, st)))
        return rc;
    if ((rc = conv2d_s1<C, C, C, 0, false>(b.a3, 2 * B, d.h, d.w, 1, P + t->off_fw[3],
                                           P + t->off_fb[3], b.f4, nullptr, 0, st)))
        return rc;
    count_launch();
    pdl(k_tcostvol, dim3(B * C, (D * d.h + 63) / 64), 256, 0, st)(b.f4, B, C, D, d.h, d.w, b.vol);
    SV_LAUNCH_CHECK();
    if ((rc = conv3d_go<C, CM, CM, CH, 1, false>(b.vol, B, D, d.h, d.w, P + t->off_cw[0],
                                                 P + t->off_cb[0], b.b1, nullptr, st)))
        return rc;
    if ((rc = conv3d_go<CM, CM, CM, CMH, 1, false>(b.b1, B, D, d.h, d.w, P + t->off_cw[1],
                                                   P + t->off_cb[1], b.b2, nullptr, st)))
        return rc;
    if ((rc = conv3d_go<CM, 1, 1, CMH, 0, false>(b.b2, B, D, d.h, d.w, P + t->off_cw[2],
                                                 P + t->off_cb[2], b.cost, nullptr, st)))
        return rc;
    count_launch();
    pdl(k_tsoftargmin, nblocks(B * d.hw), 256, 0, st)(b.cost, B, D, d.h, d.w, b.probs, b.d0);
    SV_LAUNCH_CHECK();
    // ---- refinement levels
    const int Hs[2] = {d.H2, d.H}, Ws[2] = {d.W2, d.W};
    const long HWl[2] = {d.HW2, d.HW};
    const float *guides[2] = {b.gh, b.img};
    const float *prev = b.d0;
    int ph = d.h, pw = d.w;
    for (int lv = 0; lv < 2; ++lv) {
        const int Hl = Hs[lv], Wl = Ws[lv];
        count_launch();
        pdl(k_tupcat, nblocks(B * HWl[lv]), 256, 0, st)(prev, B, ph, pw, Hl, Wl, guides[lv],
                                                       b.rin[lv]);
        const float *cur = b.rin[lv];
        for (int i = 0; i < nd; ++i) {
            const int dl = t->dil[i];
            rc = i == 0 ? conv2d_s1<2, RC, RC, 1, false>(cur, B, Hl, Wl, dl, P + t->off_rw[lv][i],
                                                         P + t->off_rb[lv][i], b.r[lv][i], nullptr,
                                                         0, st)
                        : conv2d_s1<RC, RC, RC, 1, false>(cur, B, Hl, Wl, dl, P + t->off_rw[lv][i],
                                                          P + t->off_rb[lv][i], b.r[lv][i], nullptr,
                                                          0, st);
            if (rc) return rc;
            cur = b.r[lv][i];
        }
        if ((rc = conv2d_s1<RC, 1, 1, 2, false>(cur, B, Hl, Wl, 1, P + t->off_rw[lv][nd],
                                                P + t->off_rb[lv][nd], b.out[lv], b.rin[lv],
                                                2 * HWl[lv], st)))
            return rc;
        prev = b.out[lv];
        ph = Hl;
        pw = Wl;
    }
    // ---- losses
    count_launch();
    pdl(k_thuber, nblocks(B * d.hw), 256, 0, st)(b.d0, b.dq, b.vq, B, d.hw, b.counts, 0, 0.5f,
                                                invB, b.gl0, b.t0);
    count_launch();
    pdl(k_thuber, nblocks(B * d.HW2), 256, 0, st)(b.out[0], b.dh, b.vh, B, d.HW2, b.counts, 1,
                                                 0.7f, invB, b.gl1, b.t1);
    count_launch();
    pdl(k_thuber, nblocks(B * d.HW), 256, 0, st)(b.out[1], disp, valid, B, d.HW, b.counts, 2,
                                                1.0f, invB, b.gl2, b.t2);
    SV_LAUNCH_CHECK();
    // ---- backward: refinement levels, fine to coarse.  gsl[lv] is the
    // gradient on level lv's output after its ReLU (Refinement.backward's g).
    float *gsl[2] = {b.gs0, b.gs};
    count_launch();
    pdl(k_tmask0, nblocks(B * d.HW), 256, 0, st)(b.gl2, b.out[1], B * d.HW, gsl[1]);
    for (int lv = 1; lv >= 0; --lv) {
        const int Hl = Hs[lv], Wl = Ws[lv];
        const float *gs = gsl[lv];
        // final conv (x = r[nd-1], gy = gs)
        if ((rc = wgrad2d<RC, 1, 1>(b.r[lv][nd - 1], gs, B, Hl, Wl, Hl, Wl, 1, wg, t->off_rw[lv][nd],
                                    t->off_rb[lv][nd], st)))
            return rc;
        if ((rc = conv2d_s1<1, RC, RC, 3, true>(gs, B, Hl, Wl, 1, P + t->off_rw[lv][nd], nullptr, b.gA,
                                                b.r[lv][nd - 1], 0, st)))
            return rc;
        float *gcur = b.gA, *gnext = b.gB;
        for (int i = nd - 1; i >= 1; --i) {
            const int dl = t->dil[i];
            if ((rc = wgrad2d<RC, RC, 1>(b.r[lv][i - 1], gcur, B, Hl, Wl, Hl, Wl, dl, wg,
                                         t->off_rw[lv][i], t->off_rb[lv][i], st)))
                return rc;
            if ((rc = conv2d_s1<RC, RC, RC, 3, true>(gcur, B, Hl, Wl, dl, P + t->off_rw[lv][i],
                                                     nullptr, gnext, b.r[lv][i - 1], 0, st)))
                return rc;
            float *tmp = gcur;
            gcur = gnext;
            gnext = tmp;
        }
        if ((rc = wgrad2d<2, RC, 1>(b.rin[lv], gcur, B, Hl, Wl, Hl, Wl, t->dil[0], wg,
                                    t->off_rw[lv][0], t->off_rb[lv][0], st)))
            return rc;
        // only the disparity channel of the input gradient is needed
        if ((rc = conv2d_s1<RC, 1, 2, 0, true>(gcur, B, Hl, Wl, t->dil[0], P + t->off_rw[lv][0],
                                               nullptr, b.grin, nullptr, 0, st)))
            return rc;
        // up-sample backward of 2 * (input gradient + skip) to the previous
        // level, plus that level's loss gradient, through its output ReLU
        const int sh = lv ? d.H2 : d.h, sw = lv ? d.W2 : d.w;
        const int ry = (int)ceil(2.0 * Hl / sh) + 2, rx = (int)ceil(2.0 * Wl / sw) + 2;
        count_launch();
        pdl(k_tup_bwd, nblocks((long)B * sh * sw), 256, 0, st)(
            b.grin, HWl[lv], gs, B, Hl, Wl, sh, sw, ry, rx, lv ? b.gl1 : b.gl0,
            lv ? b.out[0] : nullptr, lv ? gsl[0] : b.gd0);
        SV_LAUNCH_CHECK();
    }
    // ---- soft-argmin + cross-entropy, cost filter, cost volume
    count_launch();
    pdl(k_tsoft_bwd, nblocks(B * d.hw), 256, 0, st)(b.probs, b.d0, b.gd0, b.dq, b.vq, b.counts, B,
                                                   D, d.hw, 2.0f, invB, b.gcost, b.tce);
    if ((rc = wgrad3d<CM, 1>(b.b2, b.gcost, B, D, d.h, d.w, wg, t->off_cw[2], t->off_cb[2], st)))
        return rc;
    if ((rc = conv3d_go<1, CM, CM, 1, 3, true>(b.gcost, B, D, d.h, d.w, P + t->off_cw[2], nullptr,
                                               b.gq2, b.b2, st)))
        return rc;
    if ((rc = wgrad3d<CM, CM>(b.b1, b.gq2, B, D, d.h, d.w, wg, t->off_cw[1], t->off_cb[1], st)))
        return rc;
    if ((rc = conv3d_go<CM, CM, CM, CM, 3, true>(b.gq2, B, D, d.h, d.w, P + t->off_cw[1], nullptr,
                                                  b.gq1, b.b1, st)))
        return rc;
    if ((rc = wgrad3d<C, CM>(b.vol, b.gq1, B, D, d.h, d.w, wg, t->off_cw[0], t->off_cb[0], st)))
        return rc;
    if ((rc = conv3d_go<CM, C, C, CM, 0, true>(b.gq1, B, D, d.h, d.w, P + t->off_cw[0], nullptr,
                                                b.gvol, nullptr, st)))
        return rc;
    count_launch();
    pdl(k_tcostvol_bwd, nblocks((long)B * C * d.hw), 256, 0, st)(b.gvol, b.f4, B, C, D, d.h, d.w,
                                                                b.gf);
    SV_LAUNCH_CHECK();
    // ---- FeatureNet, both towers as one batch of 2B images
    if ((rc = wgrad2d<C, C, 1>(b.a3, b.gf, 2 * B, d.h, d.w, d.h, d.w, 1, wg, t->off_fw[3],
                               t->off_fb[3], st)))
        return rc;
    if ((rc = conv2d_s1<C, C, C, 3, true>(b.gf, 2 * B, d.h, d.w, 1, P + t->off_fw[3], nullptr, b.gF4,
                                          b.a3, 0, st)))
        return rc;
    if ((rc = wgrad2d<C, C, 1>(b.a2, b.gF4, 2 * B, d.h, d.w, d.h, d.w, 1, wg, t->off_fw[2],
                               t->off_fb[2], st)))
        return rc;
    if ((rc = conv2d_s1<C, C, C, 3, true>(b.gF4, 2 * B, d.h, d.w, 1, P + t->off_fw[2], nullptr, b.gf,
                                          b.a2, 0, st)))
        return rc;
    if ((rc = wgrad2d<C, C, 2>(b.a1, b.gf, 2 * B, d.h1, d.w1, d.h, d.w, 1, wg, t->off_fw[1],
                               t->off_fb[1], st)))
        return rc;
    count_launch();
    pdl(k_tdgrad2d_s2<C, C>, nblocks(2L * B * ((d.h1 + 1) / 2) * ((d.w1 + 1) / 2), 128), 128, 0, st)(
        b.gf, 2 * B, d.h1, d.w1, d.h, d.w, P + t->off_fw[1], b.a1, b.gF3);
    SV_LAUNCH_CHECK();
    if ((rc = wgrad2d<1, C, 2>(b.img, b.gF3, 2 * B, d.H, d.W, d.h1, d.w1, 1, wg, t->off_fw[0],
                               t->off_fb[0], st)))
        return rc;
    wg.reduce();
    SV_LAUNCH_CHECK();
    // ---- per-sample loss and the prediction
    count_launch();
    pdl(k_tloss, B, 256, 0, st)(b.t0, b.t1, b.t2, b.tce, d.hw, d.HW2, d.HW, b.counts,
                               loss ? loss : b.loss);
    SV_LAUNCH_CHECK();
    if (pred && cudaMemcpyAsync(pred, b.out[1], sizeof(float) * B * d.HW,
                                cudaMemcpyDeviceToDevice, st) != cudaSuccess) {
        set_error("prediction copy failed");
        return SV_ERR_CUDA;
    }
    return SV_OK;
}

int check_dims(const sv_trainer *t, int B, int W, int H) {
    if (B < 1 || B > kMaxB) {
        set_error("batch %d outside 1..%d", B, kMaxB);
        return SV_ERR_SHAPE;
    }
    if (W % 4 || H % 4 || W < 8 || H < 8 || (long)W * H > (1l << 24)) {
        set_error("crop %dx%d: W and H must be multiples of 4 (the pyramid targets of "
                  "build_targets line up with the network's outputs only then), 8..", W, H);
        return SV_ERR_SHAPE;
    }
    if (W / 4 <= t->D - 2) {
        set_error("quarter width %d <= D-2 (the reference's invalid_mask raises there)", W / 4);
        return SV_ERR_SHAPE;
    }
    for (int i = 0; i < t->nd; ++i)
        if (t->dil[i] < 1 || t->dil[i] > kMaxDil) {
            set_error("dilation %d outside 1..%d", t->dil[i], kMaxDil);
            return SV_ERR_NET;
        }
    return SV_OK;
}

}  // namespace

extern "C" {

int sv_trainer_create(const int *arch, int n_arch, const double *params, long n_params,
                      sv_trainer **out) {
    if (!arch || !params || !out) { set_error("NULL argument"); return SV_ERR_NULL; }
    if (n_arch < 6 || n_arch > 13 || arch[4] < 1 || arch[4] > 8 || n_arch != 5 + arch[4]) {
        set_error("arch vector must be {feat_C, cost_C, D, refine_C, ndil, dil...}");
        return SV_ERR_NET;
    }
    const bool ok_arch = (arch[0] == 12 && arch[1] == 6 && arch[3] == 8) ||
                         (arch[0] == 8 && arch[1] == 4 && arch[3] == 8);
    if (!ok_arch || arch[2] < 2 || arch[2] > kMaxD) {
        set_error("trainable architectures: feat_C/cost_C/refine_C 12/6/8 or 8/4/8, D 2..16");
        return SV_ERR_NET;
    }
    sv_trainer *t = new sv_trainer();
    memcpy(t->arch, arch, sizeof(int) * n_arch);
    t->C = arch[0]; t->Cm = arch[1]; t->D = arch[2]; t->Rc = arch[3]; t->nd = arch[4];
    for (int i = 0; i < t->nd; ++i) t->dil[i] = arch[5 + i];
    t->np = layout(t);
    if (t->np != n_params) {
        set_error("checkpoint has %ld parameters, the architecture needs %ld", n_params, t->np);
        delete t;
        return SV_ERR_NET;
    }
    const size_t nb = sizeof(double) * t->np;
    cudaError_t e = cudaMalloc(&t->p64, nb);
    if (e == cudaSuccess) e = cudaMalloc(&t->g64, nb);
    if (e == cudaSuccess) e = cudaMalloc(&t->m, nb);
    if (e == cudaSuccess) e = cudaMalloc(&t->v, nb);
    if (e == cudaSuccess) e = cudaMalloc(&t->p32, sizeof(float) * t->np);
    if (e == cudaSuccess) e = cudaMemcpy(t->p64, params, nb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(t->g64, 0, nb);
    if (e == cudaSuccess) e = cudaMemset(t->m, 0, nb);
    if (e == cudaSuccess) e = cudaMemset(t->v, 0, nb);
    if (e == cudaSuccess) {
        k_f64_to_f32<<<nblocks(t->np), 256>>>(t->p64, t->np, t->p32);
        e = cudaDeviceSynchronize();
    }
    if (e != cudaSuccess) {
        set_error("trainer allocation failed: %s", cudaGetErrorString(e));
        sv_trainer_destroy(t);
        return SV_ERR_CUDA;
    }
    *out = t;
    return SV_OK;
}

void sv_trainer_destroy(sv_trainer *t) {
    if (!t) return;
    cudaFree(t->p64);
    cudaFree(t->g64);
    cudaFree(t->m);
    cudaFree(t->v);
    cudaFree(t->p32);
    delete t;
}

long sv_trainer_param_count(const sv_trainer *t) { return t ? t->np : 0; }

static int copy_out(const double *src, double *dst, long n, long np) {
    if (!dst) { set_error("NULL argument"); return SV_ERR_NULL; }
    if (n != np) { set_error("expected %ld values, got %ld", np, n); return SV_ERR_PARAM; }
    if (cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(dst, src, sizeof(double) * n, cudaMemcpyDeviceToHost) != cudaSuccess) {
        set_error("device copy failed");
        return SV_ERR_CUDA;
    }
    return SV_OK;
}

int sv_trainer_get_params(const sv_trainer *t, double *out, long n) {
    if (!t) { set_error("NULL trainer"); return SV_ERR_NULL; }
    return copy_out(t->p64, out, n, t->np);
}

int sv_trainer_get_grads(const sv_trainer *t, double *out, long n) {
    if (!t) { set_error("NULL trainer"); return SV_ERR_NULL; }
    return copy_out(t->g64, out, n, t->np);
}

int sv_trainer_set_params(sv_trainer *t, const double *p, long n) {
    if (!t || !p) { set_error("NULL argument"); return SV_ERR_NULL; }
    if (n != t->np) { set_error("expected %ld values, got %ld", t->np, n); return SV_ERR_PARAM; }
    if (cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(t->p64, p, sizeof(double) * n, cudaMemcpyHostToDevice) != cudaSuccess) {
        set_error("device copy failed");
        return SV_ERR_CUDA;
    }
    k_f64_to_f32<<<nblocks(t->np), 256>>>(t->p64, t->np, t->p32);
    if (cudaDeviceSynchronize() != cudaSuccess) { set_error("conversion failed"); return SV_ERR_CUDA; }
    return SV_OK;
}

int sv_trainer_set_grads(sv_trainer *t, const double *g, long n) {
    if (!t || !g) { set_error("NULL argument"); return SV_ERR_NULL; }
    if (n != t->np) { set_error("expected %ld values, got %ld", t->np, n); return SV_ERR_PARAM; }
    if (cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(t->g64, g, sizeof(double) * n, cudaMemcpyHostToDevice) != cudaSuccess) {
        set_error("device copy failed");
        return SV_ERR_CUDA;
    }
    return SV_OK;
}

size_t sv_train_workspace_size(const sv_trainer *t, int B, int W, int H) {
    if (!t) { set_error("NULL trainer"); return 0; }
    if (check_dims(t, B, W, H) != SV_OK) return 0;
    Carver cv(nullptr);
    TrainBufs b;
    carve(t, dims(B, W, H), cv, b, true);
    return cv.off + 256;
}

int sv_train_grads(sv_trainer *t, const float *left, const float *right, const float *disp,
                   const uint8_t *valid, int B, int W, int H, double *loss, float *pred,
                   void *workspace, size_t workspace_bytes, void *stream) {
    if (!t || !left || !right || !disp || !valid) { set_error("NULL argument"); return SV_ERR_NULL; }
    int rc = check_dims(t, B, W, H);
    if (rc) return rc;
    // a smaller workspace does too: the partial sums are then added up more often
    const size_t need = sv_train_workspace_size(t, B, W, H);
    const bool all = workspace_bytes >= need;
    const Dims d = dims(B, W, H);
    TrainBufs b;
    Carver least(nullptr);
    carve(t, d, least, b, false);
    if (!workspace || workspace_bytes < least.off + 256 || ((uintptr_t)workspace & 255)) {
        set_error("workspace must be 256-byte aligned and hold %zu bytes (%zu for the fewest "
                  "launches)", least.off + 256, need);
        return SV_ERR_WORKSPACE;
    }
    Carver cv(workspace);
    carve(t, d, cv, b, all);
    cudaStream_t st = (cudaStream_t)stream;
    if (t->C == 12)
        return train_impl<12, 6, 8>(t, left, right, disp, valid, d, b, pred, loss, st);
    return train_impl<8, 4, 8>(t, left, right, disp, valid, d, b, pred, loss, st);
}

int sv_train_adam(sv_trainer *t, double lr, double clip, void *stream) {
    if (!t) { set_error("NULL trainer"); return SV_ERR_NULL; }
    if (!(lr >= 0.0) || !(clip > 0.0)) { set_error("lr must be >= 0 and clip > 0"); return SV_ERR_PARAM; }
    t->b1t *= 0.9;
    t->b2t *= 0.999;
    const double c1 = 1.0 / (1.0 - t->b1t), c2 = 1.0 / (1.0 - t->b2t);
    count_launch();
    pdl(k_tadam, nblocks(t->np), 256, 0, (cudaStream_t)stream)(t->p64, t->g64, t->m, t->v, t->np,
                                                                lr, c1, c2, clip, t->p32);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

int sv_trainer_reset_adam(sv_trainer *t) {
    if (!t) { set_error("NULL trainer"); return SV_ERR_NULL; }
    t->b1t = 1.0;
    t->b2t = 1.0;
    if (cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemset(t->m, 0, sizeof(double) * t->np) != cudaSuccess ||
        cudaMemset(t->v, 0, sizeof(double) * t->np) != cudaSuccess) {
        set_error("reset failed");
        return SV_ERR_CUDA;
    }
    return SV_OK;
}

}  // extern "C"
