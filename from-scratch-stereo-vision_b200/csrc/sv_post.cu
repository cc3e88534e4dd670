// sv_post.cu -- the rest of refine_disparity (stereonet.py:5865-5883):
// median_filter (2231-2259), SLIC superpixels (5394-5455) and plane_snap
// (5458-5563), all bit-identical to the reference.
//
// * median: one thread per pixel; the window is clipped at the borders, the
//   result is element n//2 of the stably sorted window (an O(n^2) rank
//   selection that also reproduces the order of equal values, signed zeros
//   included).
// * SLIC assignment: every cluster visits its window twice -- first an
//   atomicMin of the distance's bits per pixel (distances are non-negative
//   doubles, so their bits order like their values), then an atomicMin of the
//   cluster index among the clusters that reached that minimum: the first
//   strict minimum in cluster order, as the reference's loop finds it.
//   Pixels no window covers keep their label, as in the reference.
// * SLIC update: the reference sums each cluster's colours and coordinates
//   over the pixels in index order, in FP64.  A cluster's pixels lie in its
//   window, which grows to hold the ones that no window covered and that keep
//   its label, and row order of a window is index order: a warp per cluster
//   gathers them in that order, and five lanes add one sum each.
// * plane_snap: one CTA per segment gathers its valid points from the window, in
//   index order, for RANSAC (a thread per trial makes the plane in the
//   reference's order, a warp counts a trial's inliers), least squares over
//   the inliers in order (a lane per sum), and the snap.  The reference draws
//   from one xorshift32 stream that runs through the segments; xorshift32 is
//   linear over GF(2), so each segment's starting state is computed from the
//   number of earlier segments that drew (3 * trials draws each) by 32x32
//   bit-matrix powers, and each trial jumps to its own three draws.

#include <climits>
#include <cmath>

#include "sv_common.cuh"
#include "sv_post.cuh"

namespace sv {

// ================================================================= median
constexpr int kMedMaxR = 3;

__global__ void k_median(const double *__restrict__ in, int W, int H, int r,
                         double *__restrict__ out) {
    pdl_sync();
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const int y0 = y - r > 0 ? y - r : 0, y1 = y + r < H - 1 ? y + r : H - 1;
    const int x0 = x - r > 0 ? x - r : 0, x1 = x + r < W - 1 ? x + r : W - 1;
    double v[(2 * kMedMaxR + 1) * (2 * kMedMaxR + 1)];
    int n = 0;
    for (int yy = y0; yy <= y1; ++yy)
        for (int xx = x0; xx <= x1; ++xx) v[n++] = in[(long)yy * W + xx];
    const int k = n / 2;
    double res = v[0];
    for (int i = 0; i < n; ++i) {
        int pos = 0;
        for (int j = 0; j < n; ++j) pos += (v[j] < v[i]) || (j < i && v[j] == v[i]);
        if (pos == k) {
            res = v[i];
            break;
        }
    }
    out[(long)y * W + x] = res;
}

int launch_median(const double *in, int W, int H, int radius, int passes, double *out,
                  double *tmp, cudaStream_t st) {
    if (radius < 0 || radius > kMedMaxR || passes < 0) {
        set_error("median_filter: radius %d (0..%d), passes %d", radius, kMedMaxR, passes);
        return SV_ERR_PARAM;
    }
    const long N = (long)W * H;
    if (passes == 0) {
        SV_CUDA_TRY(cudaMemcpyAsync(out, in, sizeof(double) * N, cudaMemcpyDeviceToDevice, st));
        return SV_OK;
    }
    const dim3 blk(32, 8), grd((W + 31) / 32, (H + 7) / 8);
    // passes alternate between tmp and out so the last one lands in out
    const double *src = in;
    for (int p = 0; p < passes; ++p) {
        double *dst = ((passes - 1 - p) & 1) ? tmp : out;
        count_launch();
        pdl(k_median, grd, blk, 0, st)(src, W, H, radius, dst);
        src = dst;
    }
    SV_LAUNCH_CHECK();
    return SV_OK;
}

// =================================================================== SLIC
struct SlicCenter {
    double r, g, b, x, y;
};

__device__ __forceinline__ int4 slic_window(const SlicCenter &c, int step, int W, int H) {
    int x0 = __double2int_rz(c.x) - step, x1 = __double2int_rz(c.x) + step;
    int y0 = __double2int_rz(c.y) - step, y1 = __double2int_rz(c.y) + step;
    if (x0 < 0) x0 = 0;
    if (y0 < 0) y0 = 0;
    if (x1 >= W) x1 = W - 1;
    if (y1 >= H) y1 = H - 1;
    return make_int4(x0, x1, y0, y1);
}

__device__ __forceinline__ double slic_dd(const double *__restrict__ rgb, long i, int xx, int yy,
                                          const SlicCenter &c, double m2) {
    const double a = __dsub_rn(__dmul_rn(rgb[3 * i], 255.0), c.r);
    const double b = __dsub_rn(__dmul_rn(rgb[3 * i + 1], 255.0), c.g);
    const double cc = __dsub_rn(__dmul_rn(rgb[3 * i + 2], 255.0), c.b);
    const double dx = __dsub_rn((double)xx, c.x), dy = __dsub_rn((double)yy, c.y);
    const double col = __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(cc, cc));
    return __dadd_rn(col, __dmul_rn(m2, __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy))));
}

__global__ void k_slic_init(const double *__restrict__ rgb, int W, int step, int ncx, int nc,
                            SlicCenter *__restrict__ cs) {
    pdl_sync();
    const int ci = blockIdx.x * blockDim.x + threadIdx.x;
    if (ci >= nc) return;
    const int cx = step / 2 + (ci % ncx) * step, cy = step / 2 + (ci / ncx) * step;
    const long i = (long)cy * W + cx;
    cs[ci] = {__dmul_rn(rgb[3 * i], 255.0), __dmul_rn(rgb[3 * i + 1], 255.0),
              __dmul_rn(rgb[3 * i + 2], 255.0), (double)cx, (double)cy};
}

__global__ void k_slic_reset(long N, unsigned long long *__restrict__ dist,
                             int *__restrict__ labtmp) {
    pdl_sync();
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= N) return;
    dist[i] = (unsigned long long)__double_as_longlong(1.0e30);
    labtmp[i] = INT_MAX;
}

// pass 0: atomicMin of the distance bits, and the cluster's window; pass 1: cluster
// index at the minimum
__global__ void __launch_bounds__(256)
    k_slic_assign(const double *__restrict__ rgb, int W, int H, int step, double m2,
                  const SlicCenter *__restrict__ cs, int pass, unsigned long long *__restrict__ dist,
                  int *__restrict__ labtmp, int4 *__restrict__ win) {
    pdl_sync();
    const int ci = blockIdx.x;
    const SlicCenter c = cs[ci];
    const int4 w = slic_window(c, step, W, H);
    const int ww = w.y - w.x + 1, n = ww * (w.w - w.z + 1);
    if (pass == 0 && threadIdx.x == 0) win[ci] = w;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        const int yy = w.z + t / ww, xx = w.x + t % ww;
        const long i = (long)yy * W + xx;
        const unsigned long long dd =
            (unsigned long long)__double_as_longlong(slic_dd(rgb, i, xx, yy, c, m2));
        if (pass == 0) atomicMin(dist + i, dd);
        else if (dd == dist[i]) atomicMin(labtmp + i, ci);
    }
}

// Labels of the iteration.  A pixel that no window covers keeps its label, and its
// cluster's window grows to hold it: then the cluster's pixels in index order are
// again those with its label in row order of the window.  Resets the scratch for the
// next iteration.
__global__ void k_slic_commit(long N, int W, int *__restrict__ labtmp, int *__restrict__ lab,
                              unsigned long long *__restrict__ dist, int4 *__restrict__ win) {
    pdl_sync();
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= N) return;
    int l = labtmp[i];
    labtmp[i] = INT_MAX;
    dist[i] = (unsigned long long)__double_as_longlong(1.0e30);
    if (l != INT_MAX) {
        lab[i] = l;
        return;
    }
    l = lab[i];
    if (l < 0) return;
    const int x = (int)(i % W), y = (int)(i / W);
    atomicMin(&win[l].x, x);
    atomicMax(&win[l].y, x);
    atomicMin(&win[l].z, y);
    atomicMax(&win[l].w, y);
}

// One warp per cluster (window order == index order).  The lanes gather the cluster's
// pixels, in order, as five rows of doubles in shared memory; five lanes then add a
// row each, in order (the sums' order is part of the result).  A full buffer is added
// up before the gathering goes on, so any window fits.  What bounds it is the chain of
// additions and the two dependent reads per pixel (label, colour), 8 at a time.  450 x
// 375, step 12: 21 us with all five sums in one lane, now 12; with a pixel that no
// window covered, 29 ms an iteration in one thread.
// The last iteration's counts (and valid counts) are the segments'.
constexpr int kUpdWarps = 2, kUpdCap = 512, kUpdLoads = 8;

__global__ void __launch_bounds__(32 * kUpdWarps)
    k_slic_update(const double *__restrict__ rgb, int W, int nc, SlicCenter *__restrict__ cs,
                  const int *__restrict__ lab, const int4 *__restrict__ win,
                  const uint8_t *__restrict__ valid, int *__restrict__ count,
                  int *__restrict__ nvalid) {
    pdl_sync();
    __shared__ double sv[kUpdWarps][5][kUpdCap + 2];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const int ci = blockIdx.x * kUpdWarps + wi;
    if (ci >= nc) return;                              // whole warps leave together
    const int4 w = win[ci];
    const int ww = w.y - w.x + 1, wn = ww * (w.w - w.z + 1);
    double sum = 0.0;                                  // lanes 0..4: r, g, b, x, y
    int base = 0, cnt = 0, nv = 0;
    const int comp = lane < 5 ? lane : 4;
    auto add_up = [&]() {
        __syncwarp();
        const double *v = sv[wi][comp];
        int k = 0;
        for (; k + 8 <= base; k += 8) {
            double e[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) e[u] = v[k + u];
#pragma unroll
            for (int u = 0; u < 8; ++u) sum = __dadd_rn(sum, e[u]);
        }
        for (; k < base; ++k) sum = __dadd_rn(sum, v[k]);
        __syncwarp();
        cnt += base;
        base = 0;
    };
    // the window 32 pixels at a time, without a branch around a read
    const int sx = 32 % ww, sy = 32 / ww;
    int xx = w.x + lane % ww, yy = w.z + lane / ww;
    for (int t0 = 0; t0 < wn; t0 += 32 * kUpdLoads) {
        if (base + 32 * kUpdLoads > kUpdCap) add_up();
        int px[kUpdLoads], py[kUpdLoads], lb[kUpdLoads];
#pragma unroll
        for (int u = 0; u < kUpdLoads; ++u) {
            px[u] = xx;
            py[u] = yy;
            lb[u] = lab[(long)min(yy, w.w) * W + xx];
            xx += sx;
            yy += sy;
            const bool over = xx > w.y;
            xx -= over ? ww : 0;
            yy += over;
        }
        double c[kUpdLoads][3];
#pragma unroll
        for (int u = 0; u < kUpdLoads; ++u) {
            if (py[u] > w.w) lb[u] = -1;
            const bool ok = lb[u] == ci;
            const long i = ok ? (long)py[u] * W + px[u] : 0;
#pragma unroll
            for (int q = 0; q < 3; ++q) c[u][q] = ok ? rgb[3 * i + q] : 0.0;
            if (valid) nv += ok && valid[i];
        }
#pragma unroll
        for (int u = 0; u < kUpdLoads; ++u) {
            const bool ok = lb[u] == ci;
            const unsigned m = __ballot_sync(kFull, ok);
            if (ok) {
                const int pos = base + __popc(m & ((1u << lane) - 1u));
                sv[wi][0][pos] = c[u][0];
                sv[wi][1][pos] = c[u][1];
                sv[wi][2][pos] = c[u][2];
                sv[wi][3][pos] = (double)px[u];
                sv[wi][4][pos] = (double)py[u];
            }
            base += __popc(m);
        }
    }
    add_up();
    if (count) {
        for (int m = 16; m > 0; m >>= 1) nv += __shfl_xor_sync(kFull, nv, m);
        if (lane == 0) {
            count[ci] = cnt;
            nvalid[ci] = valid ? nv : cnt;
        }
    }
    if (lane < 5 && cnt) {
        const double q = __ddiv_rn(sum, (double)cnt);
        reinterpret_cast<double *>(cs + ci)[lane] = lane < 3 ? __dmul_rn(q, 255.0) : q;
    }
}

// ============================================================= plane_snap
// Block-wide exclusive prefix sum of v (blockDim <= 1024); *total gets the sum.
__device__ __forceinline__ int block_excl_sum(int v, int *total, int *sbuf) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sbuf[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int s = lane < nw ? sbuf[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, s, o);
            if (lane >= o) s += y;
        }
        sbuf[lane] = s;
    }
    __syncthreads();
    const int pre = wid ? sbuf[wid - 1] : 0;
    *total = sbuf[nw - 1];
    __syncthreads();
    return pre + x - v;
}

__device__ __forceinline__ uint32_t xorshift32(uint32_t s) {
    s ^= s << 13;
    s ^= s >> 17;
    s ^= s << 5;
    return s;
}

// y = A x over GF(2); A as 32 columns (column b = image of bit b)
__device__ __forceinline__ uint32_t gf2_apply(const uint32_t *A, uint32_t x) {
    uint32_t y = 0;
#pragma unroll
    for (int b = 0; b < 32; ++b)
        if ((x >> b) & 1u) y ^= A[b];
    return y;
}

// The same from a table per 4 bits of x: tab[16 * i + e] = A (e << 4 i).
constexpr int kGfTab = 8 * 16;
__device__ __forceinline__ uint32_t gf2_entry(const uint32_t *A, int k) {
    const uint32_t *c = A + 4 * (k >> 4);
    return (k & 1 ? c[0] : 0u) ^ (k & 2 ? c[1] : 0u) ^ (k & 4 ? c[2] : 0u) ^ (k & 8 ? c[3] : 0u);
}
__device__ __forceinline__ uint32_t gf2_lookup(const uint32_t *tab, uint32_t x) {
    uint32_t y = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) y ^= tab[16 * i + ((x >> (4 * i)) & 15u)];
    return y;
}

constexpr int kJumpBits = 24;                // up to 2^24 segments
constexpr int kDrawBits = 7;                 // up to 64 trials

// Offsets of the segments' pixels, and the starting xorshift32 state of every
// segment: seed advanced by 3*trials draws for each earlier segment with at
// least 12 valid pixels.  One CTA: the jump matrices J_j = M^(3*trials*2^j) by
// squaring (as many as nseg has bits), their tables, then a scan of the
// eligibility and one table look-up per set bit of each segment's count (by
// columns, four times the instructions: 16 us for 1,147 segments, now 13).
// draw[j] is M^(3*2^j): the segments jump to their trials' draws.
__global__ void __launch_bounds__(1024)
    k_seg_rng(int nseg, const int *__restrict__ count, const int *__restrict__ nvalid, int trials,
              uint32_t seed, int *__restrict__ start, uint32_t *__restrict__ state,
              uint32_t *__restrict__ draw) {
    pdl_sync();
    __shared__ uint32_t J[kJumpBits][32], JT[kJumpBits][kGfTab];
    __shared__ uint32_t T[2][32], DJ[kDrawBits][32];
    __shared__ int sbuf[32];
    const int t = threadIdx.x;
    // M^(3*trials): square-and-multiply on columns (warp 0)
    if (t < 32) {
        T[0][t] = xorshift32(xorshift32(xorshift32(1u << t)));     // M^3
        T[1][t] = 1u << t;                             // identity (accumulator)
        __syncwarp();
        for (int j = 0; j < kDrawBits; ++j) {
            const uint32_t acc = (trials >> j) & 1 ? gf2_apply(T[0], T[1][t]) : T[1][t];
            const uint32_t sq = gf2_apply(T[0], T[0][t]);
            DJ[j][t] = T[0][t];
            __syncwarp();
            T[1][t] = acc;
            T[0][t] = sq;
            __syncwarp();
        }
        J[0][t] = T[1][t];
        __syncwarp();
        for (int j = 1; j < kJumpBits && (nseg >> j); ++j) {
            J[j][t] = gf2_apply(J[j - 1], J[j - 1][t]);
            __syncwarp();
        }
    }
    __syncthreads();
    if (t < kDrawBits * 32) draw[t] = DJ[t / 32][t % 32];
    for (int k = t; k < kJumpBits * kGfTab && (nseg >> (k / kGfTab)); k += blockDim.x)
        JT[k / kGfTab][k % kGfTab] = gf2_entry(J[k / kGfTab], k % kGfTab);
    __syncthreads();
    int base = 0, first = 0;
    for (int g0 = 0; g0 < nseg; g0 += blockDim.x) {
        const int g = g0 + t;
        const int nv = g < nseg ? nvalid[g] : 0;
        int tot;
        const int c = base + block_excl_sum(g < nseg && nv >= 12, &tot, sbuf);
        if (g < nseg) {
            uint32_t s = seed;
            for (int j = 0; j < kJumpBits && (c >> j); ++j)
                if ((c >> j) & 1) s = gf2_lookup(JT[j], s);
            state[g] = s;
        }
        base += tot;
        const int pos = first + block_excl_sum(g < nseg ? count[g] : 0, &tot, sbuf);
        if (g < nseg) start[g] = pos;
        first += tot;
    }
}

// _solve3, stereonet.py:5458-5469 (0 when |det| < 1e-9)
__device__ int solve3_dev(const double A[3][3], const double bv[3], double out[3]) {
    const double a = A[0][0], bb = A[0][1], c = A[0][2];
    const double d = A[1][0], e = A[1][1], f = A[1][2];
    const double g = A[2][0], h = A[2][1], k = A[2][2];
#define M_ __dmul_rn
#define S_ __dsub_rn
#define A_ __dadd_rn
    const double m1 = S_(M_(e, k), M_(f, h)), m2 = S_(M_(d, k), M_(f, g)), m3 = S_(M_(d, h), M_(e, g));
    const double det = A_(S_(M_(a, m1), M_(bb, m2)), M_(c, m3));
    if (fabs(det) < 1.0e-9) return 0;
    const double x = A_(S_(M_(bv[0], m1), M_(bb, S_(M_(bv[1], k), M_(f, bv[2])))),
                        M_(c, S_(M_(bv[1], h), M_(e, bv[2]))));
    const double y = A_(S_(M_(a, S_(M_(bv[1], k), M_(f, bv[2]))), M_(bv[0], m2)),
                        M_(c, S_(M_(d, bv[2]), M_(bv[1], g))));
    const double z = A_(S_(M_(a, S_(M_(e, bv[2]), M_(bv[1], h))),
                           M_(bb, S_(M_(d, bv[2]), M_(bv[1], g)))),
                        M_(bv[0], m3));
    out[0] = __ddiv_rn(x, det);
    out[1] = __ddiv_rn(y, det);
    out[2] = __ddiv_rn(z, det);
    return 1;
}

__device__ __forceinline__ double plane_at(const double *pl, int i, int W) {
    return __dadd_rn(__dadd_rn(__dmul_rn(pl[0], (double)(i % W)), __dmul_rn(pl[1], (double)(i / W))),
                     pl[2]);
}

constexpr int kMaxTrials = 64;
constexpr int kSnapCap = 2048;          // most points of a segment in shared memory
constexpr int kSnapThreads = 128, kSnapScan = 5;

// The points of a segment: rows of x, y and d in shared memory, or pixel indices.
struct SnapRows {
    const double *rows;
    int cap;
    __device__ __forceinline__ double operator()(int c, int j) const { return rows[c * cap + j]; }
};
struct SnapList {
    const int *list;
    const double *disp;
    int W;
    __device__ __forceinline__ double operator()(int c, int j) const {
        const int i = list[j];
        return c == 0 ? (double)(i % W) : c == 1 ? (double)(i / W) : disp[i];
    }
};

template <typename P>
__device__ __forceinline__ int snap_ok(const P &p, const double *pl, double thr, int j) {
    const double v = __dadd_rn(__dadd_rn(__dmul_rn(pl[0], p(0, j)), __dmul_rn(pl[1], p(1, j))), pl[2]);
    return fabs(__dsub_rn(v, p(2, j))) <= thr;
}

// the points within thr of a plane, counted by a warp
template <typename P>
__device__ __forceinline__ int snap_count(const P &p, const double *pl, double thr, int n, int lane) {
    int c = 0, j = lane;
    for (; j + 96 < n; j += 128) {
        int e[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) e[u] = snap_ok(p, pl, thr, j + 32 * u);
        c += (e[0] + e[1]) + (e[2] + e[3]);
    }
    for (; j < n; j += 32) c += snap_ok(p, pl, thr, j);
    for (int m = 16; m > 0; m >>= 1) c += __shfl_xor_sync(kFull, c, m);
    return c;
}

// s plus f(0), f(1), ..., f(n - 1) in order, the terms 8 at a time ahead of the chain
template <typename F>
__device__ __forceinline__ double chain_sum(double s, int n, F f) {
    int k = 0;
    for (; k + 8 <= n; k += 8) {
        double e[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) e[u] = f(k + u);
#pragma unroll
        for (int u = 0; u < 8; ++u) s = __dadd_rn(s, e[u]);
    }
    for (; k < n; ++k) s = __dadd_rn(s, f(k));
    return s;
}

// _lsq_plane, stereonet.py:5472-5502, by one warp: sums in the points' order
template <typename P>
__device__ __forceinline__ void snap_fit(const P &p, int n, int lane, double *fit) {
    const int c3 = lane < 3 ? lane : 2;                    // lanes 0..2: x, y, d
    const double mean = __ddiv_rn(chain_sum(0.0, n, [&](int k) { return p(c3, k); }), (double)n);
    const double mx = __shfl_sync(kFull, mean, 0), my = __shfl_sync(kFull, mean, 1),
                 md = __shfl_sync(kFull, mean, 2);
    // lanes 0..4: xx, xy, yy, xd, yd
    const int ca = lane == 2 || lane == 4 ? 1 : 0;
    const int cb = lane == 0 ? 0 : lane <= 2 ? 1 : 2;
    const double ma = ca ? my : mx, mb = cb == 0 ? mx : cb == 1 ? my : md;
    const double s = chain_sum(0.0, n, [&](int k) {
        return __dmul_rn(__dsub_rn(p(ca, k), ma), __dsub_rn(p(cb, k), mb));
    });
    const double sxx = __shfl_sync(kFull, s, 0), sxy = __shfl_sync(kFull, s, 1),
                 syy = __shfl_sync(kFull, s, 2), sxd = __shfl_sync(kFull, s, 3),
                 syd = __shfl_sync(kFull, s, 4);
    if (lane != 0) return;
    const double det = __dsub_rn(__dmul_rn(sxx, syy), __dmul_rn(sxy, sxy));
    if (fabs(det) < 1.0e-9) {
        fit[0] = 0.0;
        fit[1] = 0.0;
        fit[2] = md;
    } else {
        const double a = __ddiv_rn(__dsub_rn(__dmul_rn(sxd, syy), __dmul_rn(syd, sxy)), det);
        const double b = __ddiv_rn(__dsub_rn(__dmul_rn(syd, sxx), __dmul_rn(sxd, sxy)), det);
        fit[0] = a;
        fit[1] = b;
        fit[2] = __dsub_rn(__dsub_rn(md, __dmul_rn(a, mx)), __dmul_rn(b, my));
    }
}

// One CTA per segment: RANSAC, least squares over the inliers, snap.  The segment's
// valid points are gathered from its window, in index order, as rows of x, y and d in
// shared memory (cap of them; a larger segment keeps their indices in pts and inl:
// same values, same order).  The draws are one stream, so a trial's thread jumps to
// its own three; a warp counts a trial's inliers; the least-squares sums, whose order
// is part of the result, are one chain each, so a lane each adds them up.  What bounds
// it is those chains and the scan of the window.  450 x 375, step 12, 40 trials: 125
// us with draws and sums in one thread and a list made by kernels ahead (18 us), now
// 33.
__global__ void __launch_bounds__(kSnapThreads)
    k_seg_snap(const double *__restrict__ disp, int W, const uint8_t *__restrict__ valid,
               const int *__restrict__ lab, const int4 *__restrict__ win,
               const int *__restrict__ start, const int *__restrict__ nvalid,
               const uint32_t *__restrict__ state, const uint32_t *__restrict__ draw, int trials,
               double thr, double min_inl, int cap, int *__restrict__ pts, int *__restrict__ inl,
               double *__restrict__ out) {
    pdl_sync();
    __shared__ double planes[kMaxTrials][3];
    __shared__ int ok[kMaxTrials], cnt[kMaxTrials];
    __shared__ int sbuf[32], wcnt[kSnapScan][kSnapThreads / 32];
    __shared__ double fit[3];
    __shared__ uint32_t jump[kDrawBits * kGfTab];      // tables of the jumps over draws
    extern __shared__ __align__(16) double rows[];     // [3][cap]
    const int g = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int n = nvalid[g];
    if (n < 12) return;
    const int4 w = win[g];
    const int ww = w.y - w.x + 1, wn = ww * (w.w - w.z + 1);
    const bool staged = n <= cap;
    int *const gp = pts + start[g], *const gi = inl + start[g];
    for (int k = t; k < kDrawBits * kGfTab; k += kSnapThreads)
        jump[k] = gf2_entry(draw + k / kGfTab * 32, k % kGfTab);
    // valid pixels in index order, kSnapScan x kSnapThreads of the window at a time
    int base = 0;
    for (int k0 = 0; k0 < wn; k0 += kSnapScan * kSnapThreads) {
        long i[kSnapScan];
        unsigned m[kSnapScan];
        double d[kSnapScan];
        bool take[kSnapScan];
#pragma unroll
        for (int u = 0; u < kSnapScan; ++u) {
            const int k = k0 + u * kSnapThreads + t;
            i[u] = (long)(w.z + k / ww) * W + w.x + k % ww;
            take[u] = k < wn && lab[i[u]] == g;
        }
#pragma unroll
        for (int u = 0; u < kSnapScan; ++u) {
            take[u] = take[u] && (!valid || valid[i[u]]);
            d[u] = take[u] ? disp[i[u]] : 0.0;
            m[u] = __ballot_sync(kFull, take[u]);
            if (lane == 0) wcnt[u][warp] = __popc(m[u]);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kSnapScan; ++u) {
            int pos = base + __popc(m[u] & ((1u << lane) - 1u));
#pragma unroll
            for (int q = 0; q < kSnapThreads / 32; ++q) {
                if (q < warp) pos += wcnt[u][q];
                base += wcnt[u][q];
            }
            if (!take[u]) continue;
            if (staged) {
                const int y = (int)(i[u] / W);
                rows[pos] = (double)((int)i[u] - y * W);
                rows[cap + pos] = (double)y;
                rows[2 * cap + pos] = d[u];
            } else {
                gp[pos] = (int)i[u];
            }
        }
        __syncthreads();
    }
    const SnapRows pr{rows, cap};
    const SnapList pp{gp, disp, W}, pi{gi, disp, W};
    auto at = [&](int c, int j) { return staged ? pr(c, j) : pp(c, j); };
    if (t < trials) {
        uint32_t s = state[g];
        for (int j = 0; j < kDrawBits; ++j)
            if ((t >> j) & 1) s = gf2_lookup(jump + kGfTab * j, s);
        double A[3][3], bv[3];
        for (int u = 0; u < 3; ++u) {
            s = xorshift32(s);
            const int j = (int)(s % (uint32_t)n);
            A[u][0] = at(0, j);
            A[u][1] = at(1, j);
            A[u][2] = 1.0;
            bv[u] = at(2, j);
        }
        ok[t] = solve3_dev(A, bv, planes[t]);
    }
    __syncthreads();
    for (int tr = warp; tr < trials; tr += kSnapThreads / 32) {
        if (!ok[tr]) continue;
        const double pl[3] = {planes[tr][0], planes[tr][1], planes[tr][2]};
        const int c = staged ? snap_count(pr, pl, thr, n, lane) : snap_count(pp, pl, thr, n, lane);
        if (lane == 0) cnt[tr] = c;
    }
    __syncthreads();
    int best = -1, bestc = -1;
    for (int tr = 0; tr < trials; ++tr)
        if (ok[tr] && cnt[tr] > bestc) {
            bestc = cnt[tr];
            best = tr;
        }
    if (best < 0 || (double)bestc < __dmul_rn(min_inl, (double)n)) return;
    // the inliers, in order, over the points (an inlier moves down or stays)
    const double pl[3] = {planes[best][0], planes[best][1], planes[best][2]};
    base = 0;
    for (int k0 = 0; k0 < n; k0 += kSnapThreads) {
        const int k = k0 + t;
        const int take = k < n && (staged ? snap_ok(pr, pl, thr, k) : snap_ok(pp, pl, thr, k));
        double x = 0.0, y = 0.0, d = 0.0;
        if (take && staged) {
            x = rows[k];
            y = rows[cap + k];
            d = rows[2 * cap + k];
        }
        int tot;
        const int pos = base + block_excl_sum(take, &tot, sbuf);
        if (take) {
            if (staged) {
                rows[pos] = x;
                rows[cap + pos] = y;
                rows[2 * cap + pos] = d;
            } else {
                gi[pos] = gp[k];
            }
        }
        base += tot;
    }
    __syncthreads();
    if (warp == 0) {
        if (staged) snap_fit(pr, base, lane, fit);
        else snap_fit(pi, base, lane, fit);
    }
    __syncthreads();
    for (int k = t; k < wn; k += kSnapThreads) {
        const long i = (long)(w.z + k / ww) * W + w.x + k % ww;
        if (lab[i] != g) continue;
        const double v = plane_at(fit, (int)i, W);
        if (fabs(__dsub_rn(v, disp[i])) <= thr || (valid && !valid[i])) out[i] = v > 0.0 ? v : 0.0;
    }
#undef M_
#undef S_
#undef A_
}

__global__ void k_status_valid(long N, const uint8_t *__restrict__ status,
                               uint8_t *__restrict__ valid) {
    pdl_sync();
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i < N) valid[i] = status[i] == 0;
}

// ------------------------------------------------------------ host side
int slic_grid(int W, int H, int step, int *ncx, int *ncy) {
    int a = 0, b = 0;
    for (int x = step / 2; x < W; x += step) ++a;
    for (int y = step / 2; y < H; y += step) ++b;
    *ncx = a;
    *ncy = b;
    return a * b;
}

double slic_m2(double compactness, int step) {
    // the reference's (compactness / step) ** 2 is CPython's float power,
    // i.e. the C library's pow(); a volatile exponent keeps the compiler
    // from replacing the call by a multiplication
    volatile double two = 2.0;
    return std::pow(compactness / step, (double)two);
}

size_t carve_post(void *ws, int W, int H, int step, PostWs *o) {
    Carver cv(ws);
    PostWs p{};
    const long N = (long)W * H;
    int ncx, ncy;
    const int nc = slic_grid(W, H, step, &ncx, &ncy);
    const int nca = nc > 0 ? nc : 1;
    p.flags = cv.take<DevFlags>(1);
    p.cs = cv.take<unsigned char>(sizeof(SlicCenter) * nca);
    p.win = cv.take<int4>(nca);
    // the jump matrices lie where SLIC's distances were
    const size_t words = (size_t)kDrawBits * 32 * sizeof(uint32_t);
    p.dist = cv.take<unsigned long long>(N * sizeof(unsigned long long) > words ? N
                                             : words / sizeof(unsigned long long));
    p.draw = reinterpret_cast<uint32_t *>(p.dist);
    p.labtmp = cv.take<int>(N);
    p.lab = cv.take<int>(N);
    p.count = cv.take<int>(nca);
    p.start = cv.take<int>(nca);
    p.pts = cv.take<int>(N);
    p.inl = cv.take<int>(N);
    p.nvalid = cv.take<int>(nca);
    p.state = cv.take<uint32_t>(nca);
    p.valid = cv.take<uint8_t>(N);
    p.tmp = cv.take<double>(N);
    if (o) *o = p;
    return cv.off;
}

int launch_slic(const double *rgb, int W, int H, int step, double compactness, int iters,
                const PostWs &w, cudaStream_t st, const uint8_t *valid) {
    if (W < 1 || H < 1 || step < 1 || iters < 0) {
        set_error("slic: bad shape or step");
        return SV_ERR_PARAM;
    }
    int ncx, ncy;
    const int nc = slic_grid(W, H, step, &ncx, &ncy);
    const long N = (long)W * H;
    const double m2 = slic_m2(compactness, step);
    SlicCenter *cs = reinterpret_cast<SlicCenter *>(w.cs);
    SV_CUDA_TRY(cudaMemsetAsync(w.lab, 0xFF, sizeof(int) * N, st));       // -1
    if (nc == 0) return SV_OK;
    count_launch();
    pdl(k_slic_init, (nc + 127) / 128, 128, 0, st)(rgb, W, step, ncx, nc, cs);
    const int nb = grid_for(N, 256, 1 << 30);
    if (iters > 0) {
        count_launch();
        pdl(k_slic_reset, nb, 256, 0, st)(N, w.dist, w.labtmp);
    }
    for (int it = 0; it < iters; ++it) {
        const bool last = it + 1 == iters;
        count_launch();
        pdl(k_slic_assign, nc, 256, 0, st)(rgb, W, H, step, m2, cs, 0, w.dist, w.labtmp, w.win);
        count_launch();
        pdl(k_slic_assign, nc, 256, 0, st)(rgb, W, H, step, m2, cs, 1, w.dist, w.labtmp, w.win);
        count_launch();
        pdl(k_slic_commit, nb, 256, 0, st)(N, W, w.labtmp, w.lab, w.dist, w.win);
        count_launch();
        pdl(k_slic_update, (nc + kUpdWarps - 1) / kUpdWarps, 32 * kUpdWarps, 0, st)(
            rgb, W, nc, cs, w.lab, w.win, valid, last ? w.count : nullptr,
            last ? w.nvalid : nullptr);
    }
    SV_LAUNCH_CHECK();
    return SV_OK;
}

int launch_plane_snap(const double *disp, const double *rgb, int W, int H, const uint8_t *valid,
                      int step, double thr, double min_inl, int trials, uint32_t seed,
                      double *out, const PostWs &w, cudaStream_t st) {
    if (trials < 0 || trials > kMaxTrials) {
        set_error("plane_snap: trials %d outside 0..%d", trials, kMaxTrials);
        return SV_ERR_PARAM;
    }
    const long N = (long)W * H;
    SV_CUDA_TRY(cudaMemcpyAsync(out, disp, sizeof(double) * N, cudaMemcpyDeviceToDevice, st));
    int ncx, ncy;
    const int nc = slic_grid(W, H, step, &ncx, &ncy);
    SV_TRY_POST(launch_slic(rgb, W, H, step, 10.0, 5, w, st, valid));
    if (nc == 0 || trials == 0) return SV_OK;
    count_launch();
    pdl(k_seg_rng, 1, 1024, 0, st)(nc, w.count, w.nvalid, trials, seed, w.start, w.state, w.draw);
    // shared memory for a whole window's points, at most kSnapCap
    const long wmax = (long)(2 * step + 1) * (2 * step + 1);
    const int cap = wmax < kSnapCap ? (int)wmax : kSnapCap;
    const size_t smem = (size_t)cap * 3 * sizeof(double);
    SV_TRY_POST(allow_smem(k_seg_snap, smem, (size_t)kSnapCap * 3 * sizeof(double)));
    count_launch();
    pdl(k_seg_snap, nc, kSnapThreads, smem, st)(disp, W, valid, w.lab, w.win, w.start, w.nvalid,
                                               w.state, w.draw, trials, thr, min_inl, cap, w.pts,
                                               w.inl, out);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

int launch_status_valid(const uint8_t *status, long N, uint8_t *valid, cudaStream_t st) {
    count_launch();
    pdl(k_status_valid, grid_for(N, 256, 1 << 30), 256, 0, st)(N, status, valid);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

}  // namespace sv

namespace sv {

// ====================================== network-level LR consistency
// mirror_h (stereonet.py:4974-4983) of one [H][W] plane of esize-byte values
__global__ void k_mirror(const unsigned char *__restrict__ in, int esize, int W, int H,
                         unsigned char *__restrict__ out) {
    pdl_sync();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W || y >= H) return;
    const long src = ((long)y * W + (W - 1 - x)) * esize, dst = ((long)y * W + x) * esize;
    for (int b = 0; b < esize; ++b) out[dst + b] = in[src + b];
}

// lr_consistency, stereonet.py:4986-5009 (FP64, the reference's order)
__global__ void k_lr_consistency(const double *__restrict__ dl, const double *__restrict__ dr,
                                 int W, int H, double tol, uint8_t *__restrict__ valid,
                                 unsigned long long *__restrict__ kept) {
    pdl_sync();
    const long N = (long)W * H;
    const long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
    int ok = 0;
    if (p < N) {
        const int x = (int)(p % W);
        const long row = p - x;
        const double d = dl[p];
        const double xr = __dsub_rn((double)x, d);
        ok = 1;
        if (xr < 0.0 || xr > (double)(W - 1)) {
            ok = 0;
        } else {
            const int x0 = __double2int_rz(xr);
            const int x1 = x0 + 1 < W ? x0 + 1 : x0;
            const double f = __dsub_rn(xr, (double)x0);
            const double e = __dadd_rn(__dmul_rn(dr[row + x0], __dsub_rn(1.0, f)),
                                       __dmul_rn(dr[row + x1], f));
            double diff = __dsub_rn(d, e);
            if (diff < 0.0) diff = -diff;
            if (diff > tol) ok = 0;
        }
        valid[p] = (uint8_t)ok;
    }
    unsigned c = __popc(__ballot_sync(kFull, ok));
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(kept, (unsigned long long)c);
}

// fill_invalid, stereonet.py:5012-5045: one CTA per row.  Pass 1 records the
// nearest valid column to the left of each pixel (chunked block scans),
// pass 2 walks from the right with the nearest valid column to the right
// and fills.
__global__ void __launch_bounds__(1024)
    k_fill_invalid(const double *__restrict__ disp, const uint8_t *__restrict__ valid, int W,
                   int H, int *__restrict__ left_idx, double *__restrict__ out) {
    pdl_sync();
    __shared__ int sbuf[32];
    __shared__ int carry;
    const int y = blockIdx.x, t = threadIdx.x, bd = blockDim.x;
    const long row = (long)y * W;
    if (t == 0) carry = -1;
    __syncthreads();
    for (int c0 = 0; c0 < W; c0 += bd) {
        const int x = c0 + t;
        const int v = x < W && valid[row + x] ? x : -1;
        const int ex = block_excl_max(v, -1, sbuf);
        const int c = carry;
        if (x < W) left_idx[row + x] = max(c, ex);
        __syncthreads();
        if (t == bd - 1) carry = max(c, max(ex, v));
        __syncthreads();
    }
    if (t == 0) carry = W;
    __syncthreads();
    const int nch = (W + bd - 1) / bd;
    for (int ci = nch - 1; ci >= 0; --ci) {
        const int x = ci * bd + t;
        const int v = x < W && valid[row + x] ? x : W;
        const int ex = block_excl_min_suffix(v, W, sbuf);
        const int c = carry;
        if (x < W) {
            double r = disp[row + x];
            if (!valid[row + x]) {
                const int lf = left_idx[row + x], rt = min(c, ex);
                const bool hl = lf >= 0, hr = rt < W;
                if (hl && hr) {
                    const double lv = disp[row + lf], rv = disp[row + rt];
                    r = lv < rv ? lv : rv;
                } else if (hl) {
                    r = disp[row + lf];
                } else if (hr) {
                    r = disp[row + rt];
                }
            }
            out[row + x] = r;
        }
        __syncthreads();
        if (t == 0) carry = min(c, min(ex, v));
        __syncthreads();
    }
}

int launch_mirror(const void *in, int esize, int W, int H, void *out, cudaStream_t st) {
    count_launch();
    pdl(k_mirror, dim3((W + 255) / 256, H), 256, 0, st)((const unsigned char *)in, esize, W, H,
                                                       (unsigned char *)out);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

int launch_lr_consistency(const double *dl, const double *dr, int W, int H, double tol,
                          uint8_t *valid, unsigned long long *kept, cudaStream_t st) {
    SV_CUDA_TRY(cudaMemsetAsync(kept, 0, sizeof(unsigned long long), st));
    const long N = (long)W * H;
    count_launch();
    pdl(k_lr_consistency, (unsigned)((N + 255) / 256), 256, 0, st)(dl, dr, W, H, tol, valid, kept);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

int launch_fill_invalid(const double *disp, const uint8_t *valid, int W, int H, int *scratch,
                        double *out, cudaStream_t st) {
    count_launch();
    const int bd = W >= 1024 ? 1024 : (W + 31) / 32 * 32;
    pdl(k_fill_invalid, H, bd, 0, st)(disp, valid, W, H, scratch, out);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

}  // namespace sv
