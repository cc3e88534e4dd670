// sv_sgm.cu -- the band costs, 8-path SGM and winner-take-all of the fused
// refinement (refine_fullres / lr_refine), on a circular slot layout built
// for packed 16-bit SIMD.
//
// Slot layout.  Each pixel owns Kp slots (K + 2 rounded up to a table size,
// a multiple of 8); candidate disparity d = base - R + k of the band lives in
// slot d mod Kp, whatever the pixel's band centre, and the Kp - K other slots
// hold "no candidate" (cost byte 0xFF, path-cost byte 0xFF).  Two neighbours
// whose bands are shifted against each other (stereonet.py:5218) therefore
// keep a disparity in the same slot: the SGM recurrence needs no re-centring
// as long as the shift is at most Kp - K - 1, because the slots that enter
// the band were "no candidate" before.  A row's bytes pair slot R with slot
// R + Kp/2: byte 2R is slot R, byte 2R + 1 slot R + Kp/2, so that a register
// of two 16-bit values holds slots R and R + Kp/2, the neighbours of both are
// the neighbouring registers, and only the ends of the row (which meet with
// the halves swapped) take a byte_perm.
//
// SGM (stereonet.py:5192-5241).  GL lanes sweep one scanline of one direction
// of one view, each holding NR = Kp / (2 GL) registers.  Per pixel:
//   t(k) = min(Lq(k), Lq(k-1) + P1, Lq(k+1) + P1)
//   L(k) = min(t(k) + C(k) - mq, C(k) + P2),  mq = min_k Lq(k)
// which is C(k) + min(t(k), mq + P2) - mq, the reference's value, with the
// path minimum mq entering as late as possible (it is the longest chain).
//
// WTA (stereonet.py:5271-5303).  S = sum of the path costs; the first minimum
// is the smallest key S * 32 + k (K <= 30) or S * 256 + k; the neighbours of
// the winner are re-read for the FP64 parabola.

#include "sv_common.cuh"
#include "sv_refine.cuh"

namespace sv {

__device__ __forceinline__ void dir_of(int d, int &dx, int &dy) {
    // order of refine_fullres's dirs list (stereonet.py:5266-5268)
    dx = (d == 0 || d == 4 || d == 6) ? 1 : (d == 2 || d == 3) ? 0 : -1;
    dy = (d == 0 || d == 1) ? 0 : (d == 2 || d == 4 || d == 5) ? 1 : -1;
}

// Row formats.  A row is GL lane chunks of 2 NR slot bytes, in the order above.
// Kp = 24 (K = 15..22, refine_disparity's R = 10 among them): 2 lanes of 12
// slots; in a cost row each lane's 12 bytes are followed by the pixel's 32-bit
// band centre, so a step loads one 16-byte word per lane and nothing else; in
// a padded path-cost row by 4 unused bytes, so a step stores one aligned
// 16-byte word per lane.  Other widths: Kp bytes, the band centre from its own
// array.
__host__ __device__ constexpr int cost_row(int Kp) { return Kp == 24 ? 32 : Kp; }
__host__ __device__ constexpr int path_row(int Kp, bool pad) { return Kp == 24 && pad ? 32 : Kp; }

// Slot of byte p of the Kp slot bytes of a row.
__host__ __device__ constexpr int slot_of_byte(int p, int Kp) { return (p >> 1) + (p & 1) * (Kp / 2); }
// Element of slot j in a path-cost row.
__device__ __forceinline__ int elem_of_slot(int j, int Kp, bool pad) {
    const int b = j < Kp / 2 ? 2 * j : 2 * (j - Kp / 2) + 1;
    return Kp == 24 && pad && b >= 12 ? b + 4 : b;
}

// Slot of a band's first candidate a = base - R (>= -R > -Kp).
__device__ __forceinline__ int first_slot(int a, int Kp) {
    return (int)((unsigned)(a + Kp) % (unsigned)Kp);
}

// ----------------------------------------------------------- band costs
// The 24-slot row of one pixel by one thread.  The K costs are computed in
// band order from one run of the other view's descriptors (no per-candidate
// tests where the whole band is inside the image, KC = K fixed), packed, and
// rotated into their slots as bytes: 3 selects of words and a byte_perm.  POPC
// (16 lanes a clock per SM, two per candidate) bounds it.
template <int KC>
__device__ __forceinline__ void cost_pixel_slot(const uint64_t *__restrict__ ref,
                                                const uint64_t *__restrict__ oth,
                                                const int32_t *__restrict__ base, int W, int x,
                                                long p, int R, int K, int invalid, int view,
                                                uint8_t *__restrict__ C, int rk) {
    const int bc = base[p], a = bc - R;
    const uint64_t c = ref[p];
    const int kk = KC > 0 ? KC : K;
    unsigned w[6] = {0u, 0u, 0u, 0u, 0u, 0u};          // byte k: band index k
    const int room = view == 0 ? x : W - 1 - x;        // largest disparity with a match
    if (KC > 0 && a >= 0 && a + KC - 1 <= room && rk >= R) {
        const uint64_t *q = view == 0 ? oth + p - a : oth + p + a;
        if (view == 0) {
#pragma unroll
            for (int k = 0; k < KC; ++k) w[k >> 2] += (unsigned)__popcll(c ^ __ldg(q - k)) << (8 * (k & 3));
        } else {
#pragma unroll
            for (int k = 0; k < KC; ++k) w[k >> 2] += (unsigned)__popcll(c ^ __ldg(q + k)) << (8 * (k & 3));
        }
#pragma unroll
        for (int k = KC; k < 24; ++k) w[k >> 2] |= 0xFFu << (8 * (k & 3));
    } else {
#pragma unroll
        for (int k = 0; k < 24; ++k) {
            const int d = a + k;
            unsigned v = 0xFFu;
            if (k < kk) {
                v = (unsigned)invalid;
                if (abs(k - R) <= rk && d >= 0 && d <= room)
                    v = (unsigned)__popcll(c ^ __ldg(view == 0 ? oth + p - d : oth + p + d));
            }
            w[k >> 2] |= v << (8 * (k & 3));
        }
    }
    // byte k to slot (am + k) mod 24: rotate up by am bytes
    const int am = first_slot(a, 24), wq = am >> 2;
    unsigned t[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) t[i] = wq & 4 ? w[(i + 2) % 6] : w[i];
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = wq & 2 ? t[(i + 4) % 6] : t[i];
#pragma unroll
    for (int i = 0; i < 6; ++i) t[i] = wq & 1 ? w[(i + 5) % 6] : w[i];
    const unsigned sel = 0x7654u - 0x1111u * (unsigned)(am & 3);
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = __byte_perm(t[(i + 5) % 6], t[i], sel);
    // slots 4i..4i+3 and 4i+12..4i+15 interleaved
    unsigned o[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        o[2 * i] = __byte_perm(w[i], w[i + 3], 0x5140);
        o[2 * i + 1] = __byte_perm(w[i], w[i + 3], 0x7362);
    }
    uint4 *dst = reinterpret_cast<uint4 *>(C + p * cost_row(24));
    dst[0] = make_uint4(o[0], o[1], o[2], (unsigned)bc);
    dst[1] = make_uint4(o[3], o[4], o[5], (unsigned)bc);
}

// 8 slots (a chunk of a row) of one pixel, for the other widths: neighbouring
// threads take neighbouring chunks (a thread that wrote a whole wide row
// stored 8 bytes every Kp: 182 us for K = 155 at 640x480).
__device__ __forceinline__ void cost_chunk_slot(const uint64_t *__restrict__ ref,
                                                const uint64_t *__restrict__ oth,
                                                const int32_t *__restrict__ base, int W, int x,
                                                long p, int chunk, int R, int K, int Kp,
                                                int invalid, int view, uint8_t *__restrict__ C,
                                                int rk) {
    const uint64_t c = ref[p];
    const int a = base[p] - R, am = first_slot(a, Kp);
    const int room = view == 0 ? x : W - 1 - x;
    const uint64_t *q = oth + p;
    unsigned w[2] = {0u, 0u};
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        int k = 4 * chunk + (u >> 1) + (u & 1) * (Kp / 2) - am;
        k += k < 0 ? Kp : 0;
        const int d = a + k;
        unsigned v = k < K ? (unsigned)invalid : 0xFFu;
        if (k < K && d >= 0 && d <= room && abs(k - R) <= rk)
            v = (unsigned)__popcll(c ^ __ldg(view == 0 ? q - d : q + d));
        w[u >> 2] |= v << (8 * (u & 3));
    }
    reinterpret_cast<uint2 *>(C + p * Kp)[chunk] = make_uint2(w[0], w[1]);
}

// Pixels [p0, p1) of a view, by a CTA.
template <bool KP24, int KC>
__device__ __forceinline__ void cost_pixels(const uint64_t *__restrict__ ref,
                                            const uint64_t *__restrict__ oth,
                                            const int32_t *__restrict__ base, int W, long p0,
                                            long p1, int R, int K, int Kp, int invalid, int view,
                                            uint8_t *__restrict__ C,
                                            const uint8_t *__restrict__ rad) {
    if constexpr (KP24) {
        long p = p0 + threadIdx.x;
        int x = (int)(p % W);
        for (; p < p1; p += blockDim.x) {
            cost_pixel_slot<KC>(ref, oth, base, W, x, p, R, K, invalid, view, C,
                                rad ? (int)rad[p] : R);
            x += blockDim.x;
            while (x >= W) x -= W;
        }
    } else {
        const int chunks = Kp / 8, per = blockDim.x / chunks;    // pixels per round
        const int chunk = threadIdx.x % chunks, i = threadIdx.x / chunks;
        if (i >= per) return;
        long p = p0 + i;
        int x = (int)(p % W);
        for (; p < p1; p += per) {
            cost_chunk_slot(ref, oth, base, W, x, p, chunk, R, K, Kp, invalid, view, C,
                            rad ? (int)rad[p] : R);
            x += per;
            while (x >= W) x -= W;
        }
    }
}

// KC: K fixed at compile time; KP24: the 24-slot rows.
template <bool KP24, int KC>
__global__ void __launch_bounds__(256)
    k_band_costs_slot(const uint64_t *__restrict__ cl, const uint64_t *__restrict__ cr,
                      const int32_t *__restrict__ base0, const int32_t *__restrict__ base1, int W,
                      long N, int R, int K, int Kp, int invalid, uint8_t *__restrict__ C0,
                      uint8_t *__restrict__ C1, const uint8_t *__restrict__ rad0) {
    pdl_sync();
    const int view = blockIdx.y;
    const uint64_t *ref = view ? cr : cl;
    const uint64_t *oth = view ? cl : cr;
    const int32_t *base = view ? base1 : base0;
    uint8_t *C = view ? C1 : C0;
    const long per = (N + gridDim.x - 1) / gridDim.x, p0 = blockIdx.x * per;
    cost_pixels<KP24, KC>(ref, oth, base, W, p0, min(N, p0 + per), R, K, Kp, invalid, view, C,
                          view == 0 ? rad0 : nullptr);
}

// ------------------------------------------------------------------ SGM
// Start pixel and length of scanline q of direction (dx, dy) in a W x H image,
// the longest first: a diagonal direction's full-length lines, then the lines
// towards the two corners in turn, each one pixel shorter.
__device__ __forceinline__ void scanline_of(int W, int H, int dx, int dy, int q, int &x0,
                                            int &y0, int &n) {
    if (dy == 0) {
        y0 = q; x0 = 0; n = W;
    } else if (dx == 0) {
        x0 = q; y0 = 0; n = H;
    } else {
        const int full = abs(W - H) + 1, m = min(W, H);
        const int r = q - full, e = r < 0 ? 0 : (r >> 1) + 1;
        // along the row edge (x0 = c) or the column edge (y0 = c)
        const bool col = r < 0 ? H > W : (r & 1) != 0;
        const int c = r < 0 ? q : (col == (H > W) ? full - 1 : 0) + e;
        x0 = col ? 0 : c;
        y0 = col ? c : 0;
        n = m - e;
    }
    if (dx < 0) x0 = W - 1 - x0;
    if (dy < 0) y0 = H - 1 - y0;
}

// Packed arithmetic of the recurrence on two 16-bit values.  With 8-bit path
// costs (LT = uint8_t) every finite value is an integer below 2048 and its
// bit pattern, read as binary16, is that integer times 2^-24 (0..1023 are
// subnormals, 1024..2047 the next binade with the same spacing): half-precision
// adds of such patterns are exact integer adds, and "no candidate" is a NaN,
// which every add keeps (0x7FFF) and every unsigned minimum loses to.  The
// adds then run on the FMA pipe beside the minima and byte_perms of the
// integer pipe, which bounds the step.  Wider path costs use integer adds and
// put "no candidate" (>= 0x7F00) back by an OR.
template <typename LT>
struct SgmMath;
__device__ __forceinline__ unsigned h2_add(unsigned a, unsigned b) {
    unsigned d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ unsigned h2_sub(unsigned a, unsigned b) {
    unsigned d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// byte_perm with the selector's top bits: a nibble 8 + i replicates the sign
// of byte i.
template <unsigned SEL>
__device__ __forceinline__ unsigned prmt(unsigned a) {
    unsigned d;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(d) : "r"(a), "n"(SEL));
    return d;
}
template <>
struct SgmMath<uint8_t> {
    static __device__ __forceinline__ unsigned add(unsigned a, unsigned b) { return h2_add(a, b); }
    // min(t + c - m, c + p2): c's "no candidate" makes both NaN
    static __device__ __forceinline__ unsigned step(unsigned t, unsigned c, unsigned m,
                                                    unsigned p2) {
        return __vminu2(h2_sub(h2_add(t, c), m), h2_add(c, p2));
    }
};
template <>
struct SgmMath<uint16_t> {
    static __device__ __forceinline__ unsigned add(unsigned a, unsigned b) { return a + b; }
    static __device__ __forceinline__ unsigned step(unsigned t, unsigned c, unsigned m,
                                                    unsigned p2) {
        const unsigned v = c & 0x00FF00FFu;
        return (v + __vminu2(t - m, p2)) | (c & 0x7F007F00u);
    }
};

// One scanline (one path of one view, start to end) swept by GL lanes, each
// holding NR = Kp / (2 GL) registers.  All 32 lanes of a warp call it together
// with 32 / GL scanlines; a lane without one passes n = 0.  C, Lo: the view's
// costs and the path's path costs; bimg: the band centres (unused at Kp = 24,
// whose cost rows carry them).
//
// A jump of the band centre by more than Kp - K - 1 (a depth edge) in any lane
// of the warp (a warp-uniform branch) first sets the slots whose disparity is
// not the predecessor's to "no candidate".  A scanline's first pixel needs no
// case of its own: from L = 0 and m = 0 the recurrence gives L = C.
//
// A pixel's costs and band centre arrive through cp.async in a per-lane shared
// ring of PF pixels ([pixel][word][lane], no bank conflicts), copied
// PF - 1 steps ahead and read one step ahead.  Async copies are tracked by
// groups, not by the few scoreboards of a warp, which made a use of a register
// prefetch wait for the youngest load in flight.

template <int BYTES>
__device__ __forceinline__ void cp_async(unsigned smem_dst, const void *gsrc) {
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(gsrc) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_dst), "l"(gsrc), "n"(BYTES)
                     : "memory");
}
__device__ __forceinline__ uint4 lds128(unsigned a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint2 lds64(unsigned a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ int lds32(unsigned a) {
    int v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

template <int NR, int GL>
struct SgmRing {
    static constexpr int Kp = 2 * NR * GL, NW = NR / 2;
    static constexpr bool INROW = Kp == 24;         // the band centre is in the cost row
    static constexpr int LB = INROW ? 16 : 2 * NR;  // cost bytes a lane copies per pixel
    // the widest copy that every lane's share of a row is aligned to
    static constexpr int PB = LB % 16 == 0 ? 16 : LB % 8 == 0 ? 8 : 4, NP = LB / PB;
    static_assert(LB % PB == 0, "a lane's share in whole copies");
    static constexpr int SLOT = 32 * (LB + (INROW ? 0 : 4));     // bytes per pixel of a warp
    static constexpr int PF = NR > 8 ? 8 : 16;      // pixels
    static constexpr int WARP = PF * SLOT;
};

template <int NR, int GL, typename LT, bool PAD>
__device__ __forceinline__ void sgm_scan(const uint8_t *__restrict__ C,
                                         const int32_t *__restrict__ bimg,
                                         LT *__restrict__ Lo, long p0, long step, int n, int R,
                                         int K, int P1, int P2, int lane,
                                         unsigned char *__restrict__ ring) {
    using M = SgmMath<LT>;
    using Rg = SgmRing<NR, GL>;
    constexpr int Kp = Rg::Kp, HK = Kp / 2, NW = Rg::NW, PF = Rg::PF, U = 4;
    constexpr bool INROW = Rg::INROW;
    constexpr int CROW = cost_row(Kp), LROW = path_row(Kp, PAD);
    static_assert(NR % 2 == 0 && (GL & (GL - 1)) == 0 && GL <= 32 && (!INROW || NR == 6) &&
                      PF % U == 0, "slot split");
    const int h = lane & (GL - 1);                  // lane within the scanline
    const uint8_t *cp = C + p0 * CROW + CROW / GL * h;
    const int32_t *bp = bimg + p0;
    LT *lp = Lo + p0 * LROW + LROW / GL * h;
    const long cstep = step * CROW, lstep = step * LROW;
    const unsigned free_shift = (unsigned)(Kp - K - 1);
    // P1 above P2 never wins against the cap: P1 = P2 gives the same minima
    const unsigned P1P1 = (unsigned)min(P1, P2) * 0x10001u, P2P2 = (unsigned)P2 * 0x10001u;
    // the row's ends meet with their halves swapped
    const unsigned sel_l = h == 0 ? 0x1032u : 0x3210u, sel_r = h == GL - 1 ? 0x1032u : 0x3210u;
    const int nmax = (int)__reduce_max_sync(kFull, (unsigned)n);

    const unsigned r0 = (unsigned)__cvta_generic_to_shared(ring);
    const unsigned mine = r0 + Rg::PB * lane, mineb = r0 + 32 * Rg::LB + 4 * lane;
    auto copy = [&](int t, int off) {               // pixel t into the ring slot at byte off
        if (t < n) {
#pragma unroll
            for (int i = 0; i < Rg::NP; ++i)
                cp_async<Rg::PB>(mine + off + 32 * Rg::PB * i, cp + Rg::PB * i);
            if (!INROW) cp_async<4>(mineb + off, bp);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        cp += cstep;
        if (!INROW) bp += step;
    };
    auto read = [&](int off, unsigned (&c)[NW], int &b) {
        if constexpr (INROW) {
            const uint4 v = lds128(mine + off);
            c[0] = v.x;
            c[1] = v.y;
            c[2] = v.z;
            b = (int)v.w;
        } else {
#pragma unroll
            for (int i = 0; i < Rg::NP; ++i) {
                const unsigned q = mine + off + 32 * Rg::PB * i;
                if constexpr (Rg::PB == 16) {
                    const uint4 v = lds128(q);
                    c[4 * i] = v.x;
                    c[4 * i + 1] = v.y;
                    c[4 * i + 2] = v.z;
                    c[4 * i + 3] = v.w;
                } else if constexpr (Rg::PB == 8) {
                    const uint2 v = lds64(q);
                    c[2 * i] = v.x;
                    c[2 * i + 1] = v.y;
                } else {
                    c[i] = (unsigned)lds32(q);
                }
            }
            b = lds32(mineb + off);
        }
    };

    unsigned L[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) L[r] = 0u;
    unsigned mm = 0u;                               // path minimum in both halves
    // the slots of pixel 0 .. PF - 2, then pixel 0's values
#pragma unroll
    for (int t = 0; t < PF - 1; ++t) copy(t, t * Rg::SLOT);
    asm volatile("cp.async.wait_group %0;" ::"n"(PF - 2) : "memory");
    unsigned cn[NW];                                // the next pixel's costs and band centre
    int bn;
    read(0, cn, bn);
    int bq = bn;                                    // the predecessor's band centre
    bool far = false;
    for (int t0 = 0; t0 < nmax; t0 += U) {
        const int o0 = t0 % PF * Rg::SLOT;          // ring slot of pixel t0
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = t0 + u;
            unsigned cw[NW];
#pragma unroll
            for (int i = 0; i < NW; ++i) cw[i] = cn[i];
            const int bw = bn;
            const bool jump = far;
            copy(t + PF - 1, (o0 + (u + PF - 1) * Rg::SLOT) % (PF * Rg::SLOT));
            asm volatile("cp.async.wait_group %0;" ::"n"(PF - 2) : "memory");
            read(u + 1 < U ? o0 + (u + 1) * Rg::SLOT : (o0 + U * Rg::SLOT) % (PF * Rg::SLOT), cn, bn);
            if (jump) {                             // warp-uniform
                // candidates the predecessor has, of this band and one beside
                const int an = bw - R, aq = bq - R;
                const int lo = max(aq, an - 1), len = min(aq + K - 1, an + K) - lo + 1;
                const int lom = (int)((unsigned)(lo + 2 * Kp) % (unsigned)Kp);
                if constexpr (Kp <= 32) {
                    // bit j: slot j holds none of them; its two halves 16 bits apart
                    const unsigned m = len > 0 ? (1u << len) - 1u : 0u;
                    const unsigned long long rot = (unsigned long long)m << lom;
                    const unsigned none = ~((unsigned)rot | (unsigned)(rot >> Kp));
                    const unsigned both = (none & ((1u << HK) - 1u)) | (none >> HK) << 16;
                    const unsigned mine = both >> (NR * h);
#pragma unroll
                    for (int r = 0; r < NR; ++r)
                        L[r] |= prmt<0xBB99>(mine << (15 - r)) & 0x7FFF7FFFu;
                } else {
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        int k0 = h * NR + r - lom, k1 = k0 + HK;
                        k0 += k0 < 0 ? Kp : 0;
                        k1 += k1 < 0 ? Kp : 0;
                        L[r] |= (k0 < len ? 0u : 0x7FFFu) | (k1 < len ? 0u : 0x7FFF0000u);
                    }
                }
            }
            bq = bw;
            far = __any_sync(kFull, (unsigned)(bn - bw) + free_shift > 2u * free_shift);
            unsigned left, right;
            if (GL == 1) {
                left = __byte_perm(L[NR - 1], 0, 0x1032);
                right = __byte_perm(L[0], 0, 0x1032);
            } else if (GL == 2) {
                left = __byte_perm(__shfl_xor_sync(kFull, L[NR - 1], 1), 0, sel_l);
                right = __byte_perm(__shfl_xor_sync(kFull, L[0], 1), 0, sel_r);
            } else {
                const int g0 = lane & ~(GL - 1);
                left = __byte_perm(__shfl_sync(kFull, L[NR - 1], g0 | ((h - 1) & (GL - 1))), 0, sel_l);
                right = __byte_perm(__shfl_sync(kFull, L[0], g0 | ((h + 1) & (GL - 1))), 0, sel_r);
            }
            unsigned Lp[NR + 2];
            Lp[0] = M::add(left, P1P1);
            Lp[NR + 1] = M::add(right, P1P1);
#pragma unroll
            for (int r = 0; r < NR; ++r) Lp[r + 1] = M::add(L[r], P1P1);
            unsigned none[NR];                      // uint16 only: the slots without a candidate
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const unsigned c = r & 1 ? prmt<0xB3A2>(cw[r >> 1]) : prmt<0x9180>(cw[r >> 1]);
                none[r] = c;
                L[r] = M::step(__vimin3_u16x2(L[r], Lp[r], Lp[r + 2]), c, mm, P2P2);
            }
            // path minimum over the scanline's slots, in both halves of mm
            unsigned m[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) m[r] = L[r];
#pragma unroll
            for (int k = NR; k > 1; k = (k + 2) / 3) {
#pragma unroll
                for (int r = 0; r < (k + 2) / 3; ++r) {
                    if (3 * r + 2 < k) m[r] = __vimin3_u16x2(m[3 * r], m[3 * r + 1], m[3 * r + 2]);
                    else if (3 * r + 1 < k) m[r] = __vminu2(m[3 * r], m[3 * r + 1]);
                    else m[r] = m[3 * r];
                }
            }
            mm = __vminu2(m[0], __byte_perm(m[0], 0, 0x1032));
#pragma unroll
            for (int o = 1; o < GL; o <<= 1) mm = __vminu2(mm, __shfl_xor_sync(kFull, mm, o));
            // the pixel's path costs: "no candidate" is byte 0xFF (the low byte
            // of 0x7FFF), or 0 in 16 bits
            if (t < n) {
                if constexpr (sizeof(LT) == 1) {
                    unsigned o[NW + 1];
#pragma unroll
                    for (int i = 0; i < NW; ++i) o[i] = __byte_perm(L[2 * i], L[2 * i + 1], 0x6420);
                    if constexpr (INROW && PAD) {
                        *reinterpret_cast<uint4 *>(lp) = make_uint4(o[0], o[1], o[2], 0u);
                    } else if constexpr (NW % 4 == 0) {
#pragma unroll
                        for (int i = 0; i < NW; i += 4)
                            reinterpret_cast<uint4 *>(lp)[i / 4] =
                                make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
                    } else if constexpr (NW % 2 == 0) {
#pragma unroll
                        for (int i = 0; i < NW; i += 2)
                            reinterpret_cast<uint2 *>(lp)[i / 2] = make_uint2(o[i], o[i + 1]);
                    } else {
#pragma unroll
                        for (int i = 0; i < NW; ++i) reinterpret_cast<unsigned *>(lp)[i] = o[i];
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < NR; r += 2)
                        reinterpret_cast<uint2 *>(lp)[r / 2] = make_uint2(
                            L[r] & ~prmt<0xBB99>(none[r]), L[r + 1] & ~prmt<0xBB99>(none[r + 1]));
                }
            }
            lp += lstep;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The scanlines of a pair by chunks of 32 / GL (one warp each), longest first:
// the two directions along the longer side, the two along the shorter one,
// then the diagonals of every direction and view in turn.
struct SgmPlan {
    int W, H, nviews, npaths, spw;
    int ca, cb, cd;              // chunks per (direction, view) of each kind
    int total;
};
static SgmPlan sgm_plan(int W, int H, int nviews, int npaths, int spw) {
    SgmPlan p{W, H, nviews, npaths, spw, 0, 0, 0, 0};
    const int lines_x = H, lines_y = W;              // scanlines along x, along y
    p.ca = ((W >= H ? lines_x : lines_y) + spw - 1) / spw;
    p.cb = ((W >= H ? lines_y : lines_x) + spw - 1) / spw;
    p.cd = npaths == 8 ? (W + H - 1 + spw - 1) / spw : 0;
    p.total = nviews * (2 * p.ca + 2 * p.cb + 4 * p.cd);
    return p;
}
// Chunk c's direction, view and first scanline.
__device__ __forceinline__ void sgm_chunk(const SgmPlan &p, int c, int &dir, int &view, int &q0) {
    const int na = 2 * p.nviews * p.ca, nb = 2 * p.nviews * p.cb;
    int d0, nd = 2;                                  // first direction, directions of this kind
    if (c < na) {
        d0 = p.W >= p.H ? 0 : 2;
    } else if (c < na + nb) {
        c -= na;
        d0 = p.W >= p.H ? 2 : 0;
    } else {
        c -= na + nb;
        d0 = 4;
        nd = 4;
    }
    const int s = c % (nd * p.nviews);
    dir = d0 + s / p.nviews;
    view = s % p.nviews;
    q0 = c / (nd * p.nviews) * p.spw;
}

// The warps of the launch (one CTA per SM) take the chunks in rounds, every
// second row of CTAs and every second round in reverse order, so that each SM
// and each warp gets its share of the long scanlines.  At most SGM_WARPS warps
// per SM: more of them only thrash the caches that merge the path-cost rows
// (32 uneven pairs, 8 to 28 warps per SM: 1.8 to 2.7 ms).
constexpr int SGM_SMS = 148, SGM_WARPS = 8;

template <int NR, int GL, typename LT, bool PAD>
__global__ void __launch_bounds__(SGM_WARPS * 32)
    k_sgm_scan(const uint8_t *__restrict__ C0, const uint8_t *__restrict__ C1,
               const int32_t *__restrict__ base0, const int32_t *__restrict__ base1, SgmPlan plan,
               int R, int K, int P1, int P2, LT *__restrict__ Lout) {
    pdl_sync();
    constexpr int Kp = 2 * NR * GL;
    extern __shared__ __align__(16) unsigned char sgm_ring[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = (int)(gridDim.x * (blockDim.x >> 5));
    const int me = warp * (int)gridDim.x +
                   (warp & 1 ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x);
    const int W = plan.W, H = plan.H;
    for (int c0 = 0, odd = 0; c0 < plan.total; c0 += warps, odd ^= 1) {
        const int c = c0 + (odd ? warps - 1 - me : me);
        if (c >= plan.total) continue;                     // warp-uniform
        int dir, view, q0, dx, dy, x0, y0, n;
        sgm_chunk(plan, c, dir, view, q0);
        const int lines = dir < 2 ? H : dir < 4 ? W : W + H - 1;
        const int q = q0 + lane / GL;
        dir_of(dir, dx, dy);
        scanline_of(W, H, dx, dy, min(q, lines - 1), x0, y0, n);
        sgm_scan<NR, GL, LT, PAD>(
            view ? C1 : C0, view ? base1 : base0,
            Lout + (long)(view * plan.npaths + dir) * W * H * path_row(Kp, PAD),
            (long)y0 * W + x0, (long)dy * W + dx, q < lines ? n : 0, R, K, P1, P2, lane,
            sgm_ring + warp * SgmRing<NR, GL>::WARP);
    }
}

// ------------------------------------------------------------------ WTA
// Sum over the paths of band index k's path cost (L: the pixel's row in path
// array 0).
template <typename LT>
__device__ __forceinline__ int path_sum(const LT *__restrict__ L, long stride, int npaths, int am,
                                        int Kp, bool pad, int k) {
    int j = am + k;
    j -= j >= Kp ? Kp : 0;
    const int e = elem_of_slot(j, Kp, pad);
    int acc = 0;
    for (int d = 0; d < npaths; ++d) acc += (int)L[d * stride + e];
    return acc;
}

// 8 slots of one path as four registers of two 16-bit values.
template <typename LT>
__device__ __forceinline__ void add_slots(const LT *__restrict__ row, unsigned (&acc)[4]) {
    if constexpr (sizeof(LT) == 1) {
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(row));
        acc[0] += __byte_perm(v.x, 0, 0x4140);
        acc[1] += __byte_perm(v.x, 0, 0x4342);
        acc[2] += __byte_perm(v.y, 0, 0x4140);
        acc[3] += __byte_perm(v.y, 0, 0x4342);
    } else {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(row));
        acc[0] += v.x;
        acc[1] += v.y;
        acc[2] += v.z;
        acc[3] += v.w;
    }
}

// The refined disparity of a pixel from its winner bk (value bv), the sums
// beside it and the best sum away from it (stereonet.py:5280-5303).
__device__ __forceinline__ double wta_value(int bk, int bv, int va, int vb, int base_p, int R) {
    const double a = (double)va, b = (double)vb, dbv = (double)bv;
    const double den = __dadd_rn(__dsub_rn(a, __dmul_rn(2.0, dbv)), b);
    double off = 0.0;
    if (den > 1.0e-9) off = __ddiv_rn(__dmul_rn(0.5, __dsub_rn(a, b)), den);
    return __dadd_rn((double)(base_p - R + bk), off);
}
__device__ __forceinline__ double wta_conf(int sv, int bv) {
    if (sv == 0x7FFFFFFF) return 1.0;
    const double dsv = (double)sv, dbv = (double)bv;
    return __ddiv_rn(__dsub_rn(dsv, dbv), __dadd_rn(dbv, 1.0e-6));
}

// One pixel by one thread, 8-bit path costs, K <= 30.  S <= 8 * 255 < 2048
// and k < 32, so S * 32 + k is a 16-bit key and the first minimum is the
// smaller of packed keys; the slots without a candidate sum to npaths * 255,
// at least any candidate's sum, with k >= K: no mask is needed.
template <int KP, bool PAD, int NPC>
__device__ __forceinline__ void wta_pixel(const uint8_t *__restrict__ Lp, long stride, int npaths,
                                          int K, int R, int32_t base_p,
                                          const double *__restrict__ d0p, double uniq,
                                          bool want_conf, double *__restrict__ outp,
                                          double *__restrict__ confp) {
    const int np = NPC > 0 ? NPC : npaths;
    const int am = first_slot(base_p - R, KP);
    const unsigned am2 = (unsigned)am * 0x10001u;
    unsigned best = 0xFFFFFFFFu;
    // register r: slots r and r + KP / 2
    auto take = [&](int r, unsigned acc) {
        // k = (slot - am) mod KP of both, from slot + KP - am < 2 KP
        const unsigned t = (unsigned)((r + KP) | (r + KP + KP / 2) << 16) - am2;
        const unsigned k = __viaddmin_u16x2(t, (0x10000u - KP) * 0x10001u, t);
        best = __vminu2(best, acc * 32u + k);
    };
    if constexpr (KP == 24 && PAD) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            unsigned acc[6] = {0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
            for (int d = 0; d < np; ++d) {
                const uint4 v = __ldg(reinterpret_cast<const uint4 *>(Lp + d * stride) + c);
                acc[0] += __byte_perm(v.x, 0, 0x4140);
                acc[1] += __byte_perm(v.x, 0, 0x4342);
                acc[2] += __byte_perm(v.y, 0, 0x4140);
                acc[3] += __byte_perm(v.y, 0, 0x4342);
                acc[4] += __byte_perm(v.z, 0, 0x4140);
                acc[5] += __byte_perm(v.z, 0, 0x4342);
            }
#pragma unroll
            for (int i = 0; i < 6; ++i) take(6 * c + i, acc[i]);
        }
    } else {
#pragma unroll
        for (int c = 0; c < KP; c += 8) {
            unsigned acc[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int d = 0; d < np; ++d) add_slots<uint8_t>(Lp + d * stride + c, acc);
#pragma unroll
            for (int i = 0; i < 4; ++i) take(c / 2 + i, acc[i]);
        }
    }
    const unsigned key = min(best & 0xFFFFu, best >> 16);
    const int bk = (int)(key & 31u), bv = (int)(key >> 5);
    if (bk == 0 || bk == K - 1) {
        *outp = *d0p;
        if (want_conf) *confp = 0.0;
        return;
    }
    const int va = path_sum(Lp, stride, np, am, KP, PAD, bk - 1);
    const int vb = path_sum(Lp, stride, np, am, KP, PAD, bk + 1);
    if (uniq > 0.0 || want_conf) {
        // second best away from the winner's neighbours (stereonet.py:5286-5290)
        int sv = 0x7FFFFFFF;
        for (int k = 0; k < K; ++k)
            if (k < bk - 1 || k > bk + 1) sv = min(sv, path_sum(Lp, stride, np, am, KP, PAD, k));
        const double conf = wta_conf(sv, bv);
        if (want_conf) *confp = conf;
        if (conf < uniq) {
            *outp = *d0p;
            return;
        }
    }
    *outp = wta_value(bk, bv, va, vb, base_p, R);
}

// One pixel by LPP neighbouring lanes (any band, any path-cost width): lane l
// takes the 8-slot chunks l, l + LPP, ... of every path's row, so a warp reads
// whole rows (one thread per pixel read 8 bytes every Kp: 1,940 us at 640x480
// with K = 155, against 0.94 GB of path costs).  All LPP lanes call it.
template <typename LT, int LPP>
__device__ __forceinline__ void wta_pixel_wide(const LT *__restrict__ Lp, long stride, int npaths,
                                               int K, int Kp, int R, int32_t base_p,
                                               const double *__restrict__ d0p, double uniq,
                                               bool want_conf, double *__restrict__ outp,
                                               double *__restrict__ confp) {
    const int lane = threadIdx.x & 31, l = lane & (LPP - 1);
    const unsigned mask = ((1u << LPP) - 1u) << (lane & ~(LPP - 1));
    const int am = first_slot(base_p - R, Kp);
    // smallest S * 256 + k over the band indices outside [x0, x1]
    auto scan = [&](int x0, int x1) {
        unsigned best = 0xFFFFFFFFu;
        for (int c = 8 * l; c < Kp; c += 8 * LPP) {
            unsigned acc[4] = {0u, 0u, 0u, 0u};
            if (npaths == 8) {
#pragma unroll
                for (int d = 0; d < 8; ++d) add_slots<LT>(Lp + d * stride + c, acc);
            } else {
#pragma unroll 4
                for (int d = 0; d < npaths; ++d) add_slots<LT>(Lp + d * stride + c, acc);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                int k0 = c / 2 + i - am, k1 = k0 + Kp / 2;
                k0 += k0 < 0 ? Kp : 0;
                k1 += k1 < 0 ? Kp : 0;
                if (k0 < K && (k0 < x0 || k0 > x1)) best = min(best, (acc[i] & 0xFFFFu) * 256u + k0);
                if (k1 < K && (k1 < x0 || k1 > x1)) best = min(best, (acc[i] >> 16) * 256u + k1);
            }
        }
#pragma unroll
        for (int o = 1; o < LPP; o <<= 1) best = min(best, __shfl_xor_sync(mask, best, o));
        return best;
    };
    const unsigned key = scan(1, 0);
    const int bk = (int)(key & 255u), bv = (int)(key >> 8);
    if (bk == 0 || bk == K - 1) {                          // the same for the LPP lanes
        if (l == 0) {
            *outp = *d0p;
            if (want_conf) *confp = 0.0;
        }
        return;
    }
    // the sums beside the winner, the paths dealt to the lanes (both fit 16 bits)
    unsigned ab = 0u;
    {
        int ja = am + bk - 1, jb = am + bk + 1;
        ja -= ja >= Kp ? Kp : 0;
        jb -= jb >= Kp ? Kp : 0;
        const int ea = elem_of_slot(ja, Kp, false), eb = elem_of_slot(jb, Kp, false);
#pragma unroll
        for (int d = 0; d < 8; d += LPP)
            if (d + l < npaths) {
                const LT *row = Lp + (d + l) * stride;
                ab += (unsigned)row[ea] | (unsigned)row[eb] << 16;
            }
    }
#pragma unroll
    for (int o = 1; o < LPP; o <<= 1) ab += __shfl_xor_sync(mask, ab, o);
    bool use_d0 = false;
    double conf = 0.0;
    if (uniq > 0.0 || want_conf) {
        const unsigned second = scan(bk - 1, bk + 1);
        conf = wta_conf(second == 0xFFFFFFFFu ? 0x7FFFFFFF : (int)(second >> 8), bv);
        use_d0 = conf < uniq;
    }
    if (l) return;
    if (want_conf) *confp = conf;
    *outp = use_d0 ? *d0p : wta_value(bk, bv, (int)(ab & 0xFFFFu), (int)(ab >> 16), base_p, R);
}

// nviews <= 2; KP > 0: one thread per pixel with Kp fixed, else LPP lanes.
template <typename LT, int KP, bool PAD, int NPC, int LPP>
__global__ void __launch_bounds__(256)
    k_wta_slot(const LT *__restrict__ Lall, int npaths, int nviews, long N, int K, int Kp, int R,
               const int32_t *__restrict__ base0, const int32_t *__restrict__ base1,
               const double *__restrict__ d00, const double *__restrict__ d01, double uniq,
               int want_conf, double *__restrict__ out0, double *__restrict__ out1,
               double *__restrict__ conf0) {
    pdl_sync();
    const int row = path_row(KP > 0 ? KP : Kp, PAD);
    const long stride = N * row;                           // between path arrays
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < nviews * N * LPP;
         i += (long)gridDim.x * blockDim.x) {
        const long w = i / LPP;
        const int view = w >= N ? 1 : 0;
        const long p = w - view * N;
        const LT *Lp = Lall + (long)view * npaths * stride + p * row;
        const int b = (view ? base1 : base0)[p];
        const double *d0 = (view ? d01 : d00) + p;
        double *out = (view ? out1 : out0) + p, *conf = conf0 ? conf0 + p : nullptr;
        if constexpr (KP > 0)
            wta_pixel<KP, PAD, NPC>(Lp, stride, npaths, K, R, b, d0, uniq, want_conf && view == 0,
                                    out, conf);
        else
            wta_pixel_wide<LT, LPP>(Lp, stride, npaths, K, Kp, R, b, d0, uniq,
                                    want_conf && view == 0, out, conf);
    }
}

// ====================================================================
// Host
// ====================================================================

// Slots of a pixel.  Without padding (the static scratch and the smaller workspaces)
// also 48: a lane's share of such a row is no 16-byte copy, and 64 slots are faster on
// small images although they are more (500 x 150, K = 31: 271 us a pass, 328 with 48; 310
// before this layout).  Images whose path costs leave the L2 are the other way round
// (1397 x 1101: 1481 us with 64, 1410 with 48, 2370 before), by 5 %.
int slot_width(int K, bool pad) {
    static const int widths[] = {8, 16, 24, 32, 48, 64, 96, 128, 160, 192, 256};
    for (int w : widths)
        if (w >= K + 2 && (w != 48 || !pad)) return w;
    return 256;
}

size_t cost_row_bytes(int K, bool pad) { return cost_row(slot_width(K, pad)); }
size_t path_row_bytes(int K, bool l16, bool pad) {
    return l16 ? 2 * slot_width(K, pad) : path_row(slot_width(K, pad), pad);
}

int launch_band_costs_slot(const uint64_t *cl, const uint64_t *cr, const int32_t *base0,
                           const int32_t *base1, int W, int H, int R, int invalid, uint8_t *C0,
                           uint8_t *C1, int nviews, cudaStream_t st, const uint8_t *rad0, bool pad) {
    const long N = (long)W * H;
    const int K = 2 * R + 1, Kp = slot_width(K, pad);
    const dim3 px(grid_for(N, Kp == 24 ? 256 : 256 / (Kp / 8), 148 * 8), nviews);
    count_launch();
    if (K == 21)    // R = 10, the refine_disparity default
        pdl(k_band_costs_slot<true, 21>, px, 256, 0, st)(cl, cr, base0, base1, W, N, R, K, Kp,
                                                        invalid, C0, C1, rad0);
    else if (Kp == 24)
        pdl(k_band_costs_slot<true, 0>, px, 256, 0, st)(cl, cr, base0, base1, W, N, R, K, Kp,
                                                       invalid, C0, C1, rad0);
    else
        pdl(k_band_costs_slot<false, 0>, px, 256, 0, st)(cl, cr, base0, base1, W, N, R, K, Kp,
                                                        invalid, C0, C1, rad0);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

template <int NR, int GL, typename LT, bool PAD>
static int sgm_go(const uint8_t *C0, const uint8_t *C1, const int32_t *b0, const int32_t *b1,
                  int W, int H, int K, int P1, int P2, void *Lout, int nviews, int npaths,
                  cudaStream_t st) {
    const SgmPlan plan = sgm_plan(W, H, nviews, npaths, 32 / GL);
    const int blocks = plan.total < SGM_SMS ? plan.total : SGM_SMS;
    constexpr int FIT = 227 * 1024 / SgmRing<NR, GL>::WARP, MAXW = FIT < SGM_WARPS ? FIT : SGM_WARPS;
    int warps = (plan.total + blocks - 1) / blocks;
    if (warps > MAXW) warps = MAXW;
    const size_t smem = (size_t)warps * SgmRing<NR, GL>::WARP;
    const int rc = allow_smem(k_sgm_scan<NR, GL, LT, PAD>, smem, MAXW * SgmRing<NR, GL>::WARP);
    if (rc) return rc;
    count_launch();
    pdl(k_sgm_scan<NR, GL, LT, PAD>, blocks, warps * 32, smem, st)(
        C0, C1, b0, b1, plan, (K - 1) / 2, K, P1, P2, (LT *)Lout);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

template <typename LT, bool PAD>
static int sgm_dispatch(const uint8_t *C0, const uint8_t *C1, const int32_t *b0,
                        const int32_t *b1, int W, int H, int K, int Kp, int P1, int P2, void *Lout,
                        int nviews, int npaths, cudaStream_t st) {
    // More lanes shorten a step, whose latency a warp alone on its scheduler pays; the
    // fewest registers per lane that leave 16-byte copies (640 x 480, a pass: K = 49 2
    // lanes 460 us, 4 414; K = 101 4 lanes 660, 8 634; K = 25 2 lanes 311, 4 and 8-byte
    // copies 326).  From 160 slots on at most 12 registers whatever the copies: steps of
    // 20 and more cost more than in proportion.  The SGM launch, 8- / 16-bit path costs:
    // 640 x 480, K = 155: 4 lanes of 20 375 / 903 us, 8 of 10 364 / 547; K = 159: 4 of 24
    // 963 / 1600, 8 of 12 344 / 672; K = 253: 4 of 32 1567 / 2695, 8 of 16 561 / 1509, 16
    // of 8 520 / 774; 160 x 120, K = 253: 229 / 301, 59 / 100 and 43 / 59.  K = 191 to 222
    // take 256 slots too (640 x 480: 224 slots in 8 lanes of 14 551 / 991).
    // K <= 6: one lane; lr_refine, 8- / 16-bit path costs, one lane and two: 450 x 375
    // 85 / 102 and 89 / 92 us, 1397 x 1101 443 / 554 and 390 / 424, 16 uneven pairs 782 /
    // 1023 and 631 / 642 (with the earlier kernels 800 for the pairs): two lanes are the
    // better choice for all but small 8-bit images.
#define SV_SGM(NR, GL) \
    return sgm_go<NR, GL, LT, PAD>(C0, C1, b0, b1, W, H, K, P1, P2, Lout, nviews, npaths, st)
    switch (Kp) {
    case 8: SV_SGM(4, 1);
    case 16: SV_SGM(4, 2);
    case 24: SV_SGM(6, 2);
    case 32: SV_SGM(8, 2);
    case 48:                                       // slot_width: only without padding
        if constexpr (!PAD) SV_SGM(6, 4);
        break;
    case 64: SV_SGM(8, 4);
    case 96: SV_SGM(12, 4);
    case 128: SV_SGM(8, 8);
    case 160: SV_SGM(10, 8);
    case 192: SV_SGM(12, 8);
    case 256: SV_SGM(8, 16);
    default: break;
    }
#undef SV_SGM
    set_error("no SGM geometry for K=%d", K);
    return SV_ERR_SHAPE;
}

int launch_sgm_packed(const uint8_t *C0, const uint8_t *C1, const int32_t *b0,
                      const int32_t *b1, int W, int H, int K, int P1, int P2, void *Lout,
                      bool l16, bool pad, int nviews, int npaths, cudaStream_t st) {
    const int Kp = slot_width(K, pad);
    if (l16)
        return sgm_dispatch<uint16_t, false>(C0, C1, b0, b1, W, H, K, Kp, P1, P2, Lout, nviews, npaths, st);
    if (pad)
        return sgm_dispatch<uint8_t, true>(C0, C1, b0, b1, W, H, K, Kp, P1, P2, Lout, nviews, npaths, st);
    return sgm_dispatch<uint8_t, false>(C0, C1, b0, b1, W, H, K, Kp, P1, P2, Lout, nviews, npaths, st);
}

int launch_wta_slot(const void *L, bool l16, bool pad, int npaths, int nviews, int W, int H, int R,
                    const int32_t *b0, const int32_t *b1, const double *d00, const double *d01,
                    double uniq, double *out0, double *out1, double *conf0, cudaStream_t st) {
    const long N = (long)W * H;
    const int K = 2 * R + 1;
    const int Kp = slot_width(K, pad);
    count_launch();
    if (nviews < 1 || nviews > 2) {
        set_error("wta: nviews=%d", nviews);
        return SV_ERR_PARAM;
    }
#define SV_WTA(LT, KP, PAD, NP, LPP, BLOCKS)                                                \
    pdl(k_wta_slot<LT, KP, PAD, NP, LPP>, BLOCKS, 256, 0, st)(                               \
        (const LT *)L, npaths, nviews, N, K, Kp, R, b0, b1, d00, d01, uniq, conf0 != nullptr, \
        out0, out1, conf0)
    const int blocks = grid_for(nviews * N, 256, 148 * 16);
    const int wide = grid_for(nviews * N * 8, 256, 148 * 64);
    // 16-bit path costs of a narrow band: as many lanes as leave each a chunk or two, or
    // most of them idle (1397 x 1101, both views, lanes 1 / 2 / 4 / 8: K = 11 160 / 175 /
    // 299 / 516 us, K = 21 234 / 231 / 312 / 527, K = 25 321 / 280 / 336 / 547; with 64
    // slots or more 8 lanes are the fastest, K = 95 at 160 x 120 45 / 24 / 20 / 18).
    if (l16 && Kp <= 16) SV_WTA(uint16_t, 0, false, 0, 1, blocks);
    else if (l16 && Kp <= 32) SV_WTA(uint16_t, 0, false, 0, 2, grid_for(nviews * N * 2, 256, 148 * 64));
    else if (l16) SV_WTA(uint16_t, 0, false, 0, 8, wide);
    else if (Kp == 24 && pad && npaths == 8) SV_WTA(uint8_t, 24, true, 8, 1, blocks);
    else if (Kp == 24 && pad) SV_WTA(uint8_t, 24, true, 0, 1, blocks);
    else if (Kp == 24) SV_WTA(uint8_t, 24, false, 0, 1, blocks);
    else if (Kp == 8) SV_WTA(uint8_t, 8, false, 0, 1, blocks);
    else if (Kp == 16) SV_WTA(uint8_t, 16, false, 0, 1, blocks);
    else if (Kp == 32) SV_WTA(uint8_t, 32, false, 0, 1, blocks);
    else SV_WTA(uint8_t, 0, false, 0, 8, wide);
#undef SV_WTA
    SV_LAUNCH_CHECK();
    return SV_OK;
}

// ====================================================================
// Batched lr_refine, middle stages.  Costs and WTA run one block per
// px_per_block pixels of a pair (blockIdx.y = view).  The SGM is a
// persistent kernel over a device-side queue: every warp takes sgm_fetch / GL
// scanlines (sgm_fetch 32 by default) at a time from one atomic counter.  The
// host orders them pair by pair, the largest pair first, and within a pair by
// length (segments of (view, direction)), so all pairs share one launch, a
// pair's directions find its costs in L2, and the small pairs come last.
// ====================================================================

// KC > 0: K fixed at compile time, as in the single-pair kernel (the whole batch
// shares K).
template <bool KP24, int KC>
__global__ void __launch_bounds__(256) k_b_costs(BatchTables t) {
    pdl_sync();
    const int i = batch_find(t.px_blk, t.n, blockIdx.x);
    const BatchPair &P = t.pairs[i];
    const int view = blockIdx.y;
    const long N = (long)P.W * P.H;
    const long p0 = (long)(blockIdx.x - t.px_blk[i]) * t.px_per_block;
    const long p1 = min(N, p0 + (long)t.px_per_block);
    const uint64_t *ref = view ? P.cen1 : P.cen0;
    const uint64_t *oth = view ? P.cen0 : P.cen1;
    const int32_t *base = view ? P.base1 : P.base0;
    uint8_t *C = view ? P.C1 : P.C0;
    cost_pixels<KP24, KC>(ref, oth, base, P.W, p0, p1, t.R, t.K, t.Kp, t.invalid, view, C, nullptr);
}

template <int NR, int GL, typename LT, bool PAD>
__global__ void __launch_bounds__(256) k_b_sgm(BatchTables t, long long total) {
    pdl_sync();
    constexpr int SPW = 32 / GL;
    extern __shared__ __align__(16) unsigned char sgm_ring[];
    const int lane = threadIdx.x & 31;
    unsigned char *ring = sgm_ring + (threadIdx.x >> 5) * SgmRing<NR, GL>::WARP;
    const int fetch = t.sgm_fetch / GL;                    // a multiple of 32 / GL
    for (;;) {
        long long first = 0;
        if (lane == 0) first = atomicAdd(t.queue, fetch);
        first = __shfl_sync(kFull, first, 0);
        if (first >= total) return;                        // warp-uniform
        for (int j = 0; j < fetch; j += SPW) {
            if (first + j >= total) break;                 // warp-uniform
            const bool on = first + j + lane / GL < total;
            const long long task = on ? first + j + lane / GL : total - 1;
            const int s = batch_find(t.seg_start, t.nseg, task);
            const BatchPair &P = t.pairs[t.seg_pair[s]];
            const int view = t.seg_vd[s] >> 3, dir = t.seg_vd[s] & 7;
            int dx, dy, x0, y0, n;
            dir_of(dir, dx, dy);
            scanline_of(P.W, P.H, dx, dy, (int)(task - t.seg_start[s]), x0, y0, n);
            const long N = (long)P.W * P.H;
            sgm_scan<NR, GL, LT, PAD>(view ? P.C1 : P.C0, view ? P.base1 : P.base0,
                                      reinterpret_cast<LT *>(P.L) +
                                          (long)(view * t.npaths + dir) * N *
                                              path_row(2 * NR * GL, PAD),
                                      (long)y0 * P.W + x0, (long)dy * P.W + dx, on ? n : 0, t.R,
                                      t.K, t.P1, t.P2, lane, ring);
        }
    }
}

template <typename LT, int KP, bool PAD, int NPC, int LPP>
__global__ void __launch_bounds__(256) k_b_wta(BatchTables t) {
    pdl_sync();
    const int i = batch_find(t.px_blk, t.n, blockIdx.x);
    const BatchPair &P = t.pairs[i];
    const int view = blockIdx.y;
    const long N = (long)P.W * P.H;
    const int row = path_row(KP > 0 ? KP : t.Kp, PAD);
    const long stride = N * row;
    const long p0 = (long)(blockIdx.x - t.px_blk[i]) * t.px_per_block;
    const long p1 = min(N, p0 + (long)t.px_per_block);
    const LT *Lv = reinterpret_cast<const LT *>(P.L) + (long)view * t.npaths * stride;
    for (long j = p0 * LPP + threadIdx.x; j < p1 * LPP; j += blockDim.x) {
        const long p = j / LPP;
        const int b = (view ? P.base1 : P.base0)[p];
        const double *d0 = (view ? P.d0r : P.disp0) + p;
        double *out = (view ? P.dr : P.dl) + p;
        if constexpr (KP > 0)
            wta_pixel<KP, PAD, NPC>(Lv + p * row, stride, t.npaths, t.K, t.R, b, d0, t.uniq, false,
                                    out, nullptr);
        else
            wta_pixel_wide<LT, LPP>(Lv + p * row, stride, t.npaths, t.K, t.Kp, t.R, b, d0,
                                    t.uniq, false, out, nullptr);
    }
}

int launch_batch_front(const BatchTables &t, long long px_blocks, long long rows,
                       long long tiles, cudaStream_t st);
int launch_batch_back(const BatchTables &t, long long rows, cudaStream_t st);

template <int NR, int GL, typename LT, bool PAD>
static int batch_sgm_go(const BatchTables &t, long long tasks, int threads, int ctas_per_sm,
                        cudaStream_t st) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long want = (tasks * GL + threads - 1) / threads;
    // persistent: ctas_per_sm CTAs on each SM, but no more than SGM_WARPS warps
    // (128 scanlines at 2 lanes each).  More of them read and write more rows at
    // once than the caches hold: 20 uneven pairs took 1.8 ms with 8 warps per SM,
    // 2.0 with 12, 2.7 with 28, and 2.3 with 4.
    const int most = threads / 32 < SGM_WARPS ? SGM_WARPS / (threads / 32) : 1;
    const long long cap = (long long)sms * (ctas_per_sm < most ? ctas_per_sm : most);
    const unsigned blocks = (unsigned)(want < cap ? (want < 1 ? 1 : want) : cap);
    const size_t smem = (size_t)(threads / 32) * SgmRing<NR, GL>::WARP;
    const int rc = allow_smem(k_b_sgm<NR, GL, LT, PAD>, smem, SGM_WARPS * SgmRing<NR, GL>::WARP);
    if (rc) return rc;
    count_launch();
    pdl(k_b_sgm<NR, GL, LT, PAD>, blocks, threads, smem, st)(t, tasks);
    SV_LAUNCH_CHECK();
    return SV_OK;
}

int launch_batch_refine(const BatchTables &t, long long px_blocks, long long rows,
                        long long tiles, long long tasks, bool l16, int sgm_threads,
                        int sgm_ctas_per_sm, cudaStream_t st) {
    int rc = launch_batch_front(t, px_blocks, rows, tiles, st);
    if (rc) return rc;
    const dim3 px((unsigned)px_blocks, 2);
    count_launch();
    if (t.K == 21) pdl(k_b_costs<true, 21>, px, 256, 0, st)(t);    // R = 10
    else if (t.Kp == 24) pdl(k_b_costs<true, 0>, px, 256, 0, st)(t);
    else pdl(k_b_costs<false, 0>, px, 256, 0, st)(t);
    SV_LAUNCH_CHECK();
#define SV_BGO(KP, NR, GL)                                                                   \
    case KP:                                                                                 \
        rc = l16 ? batch_sgm_go<NR, GL, uint16_t, false>(t, tasks, sgm_threads,              \
                                                         sgm_ctas_per_sm, st)                \
                 : batch_sgm_go<NR, GL, uint8_t, true>(t, tasks, sgm_threads,                \
                                                       sgm_ctas_per_sm, st);                 \
        break;
    switch (t.Kp) {
        SV_BGO(8, 4, 1)
        SV_BGO(16, 4, 2)
    case 24:
        rc = l16 ? batch_sgm_go<6, 2, uint16_t, false>(t, tasks, sgm_threads, sgm_ctas_per_sm, st)
             : t.pad ? batch_sgm_go<6, 2, uint8_t, true>(t, tasks, sgm_threads, sgm_ctas_per_sm, st)
                     : batch_sgm_go<6, 2, uint8_t, false>(t, tasks, sgm_threads, sgm_ctas_per_sm, st);
        break;
        SV_BGO(32, 8, 2)
    default:
        set_error("batched refinement supports bands up to K = 30 (got K = %d)", t.K);
        return SV_ERR_SHAPE;
    }
#undef SV_BGO
    if (rc) return rc;
    count_launch();
    if (l16 && t.Kp <= 16) pdl(k_b_wta<uint16_t, 0, false, 0, 1>, px, 256, 0, st)(t);
    else if (l16) pdl(k_b_wta<uint16_t, 0, false, 0, 2>, px, 256, 0, st)(t);
    else if (t.Kp == 24 && !t.pad) pdl(k_b_wta<uint8_t, 24, false, 0, 1>, px, 256, 0, st)(t);
    else if (t.Kp == 24 && t.npaths == 8) pdl(k_b_wta<uint8_t, 24, true, 8, 1>, px, 256, 0, st)(t);
    else if (t.Kp == 24) pdl(k_b_wta<uint8_t, 24, true, 0, 1>, px, 256, 0, st)(t);
    else if (t.Kp == 8) pdl(k_b_wta<uint8_t, 8, true, 0, 1>, px, 256, 0, st)(t);
    else if (t.Kp == 16) pdl(k_b_wta<uint8_t, 16, true, 0, 1>, px, 256, 0, st)(t);
    else pdl(k_b_wta<uint8_t, 32, true, 0, 1>, px, 256, 0, st)(t);
    SV_LAUNCH_CHECK();
    return launch_batch_back(t, rows, st);
}

}  // namespace sv
