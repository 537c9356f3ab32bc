// blind_rotate_warp.cu -- the blind rotation with one warp per bootstrap and every FFT exchange in
// tensor memory (tfhe_blindRotate_FFT, lwe-bootstrapping-functions-fft.cpp:88-112, with the external
// product tGswFFTExternMulToTLwe, tgsw-fft-operations.cpp:89-114); N = 1024.
//
// The same arithmetic in the same order per accumulator and per transform as blind_rotate_kernel, so
// the same bits.  What differs is where the points sit and how they move.  A warp holds a whole
// transform, 16 points per lane: the two radix-8 butterflies that TeamFft gives to the threads lane and
// lane + 32 of a team.  Between stages the points change lanes through tensor memory instead of shared
// memory: a store in the 32x32b shape puts a lane's words into the columns of its own row, and a load in
// the 16x256b shape gives lane 4a + b the words of columns 8j + 2b, 8j + 2b + 1 of the rows a, a + 8,
// a + 16 and a + 24.  One such pass swaps the lane index's two high bits with two register bits (the
// other three lane bits move up), so the 8 x 8 x 8 plan takes one pass to its first exchange (two bits
// of n1 are in the lane, the third in the register index) and two to its second (all three bits of n2);
// see WarpExch.  The inverse transform runs the passes backwards.
//
// Why: with the exchanges in shared memory that pipe was 80 % busy (43 % of it the exchanges) and set the pace.
// TMEM has its own path per warp quadrant; a pass measured 211 cycles alone and 164 cycles of the
// quadrant when its two warps run at once.  No barrier is left in the step but __syncwarp.  What is left
// issues the instructions of the transforms and little else: 5.5k warp-instructions per split bootstrap
// step (7.05k in the paired kernel), of which 3.3k are packed FP32.
// What bounds it: register read ports and issue.  A scheduler reads two 32-bit registers per lane and cycle, so a
// packed multiply-add of three register pairs takes three cycles, and one with a single word for both
// halves of an operand 2.5; hence single-word twiddle factors, and spectra that multiply the key's
// {hi, lo} limb pairs one word at a time.
// Measured, one wave of 1184 bootstraps (eight per SM): split 6.89 ms against 7.71 ms per 1036 for the paired
// kernel (1.37 against 1.75 us per bootstrap step and SM), FP64 10.1 ms against 12.4 ms for two waves of 592 on
// blind_rotate_kernel.  One warp per bootstrap leaves a scheduler one warp at four per SM, and its latencies
// show (split 4.97 ms per 592, FP64 6.6 ms); with two warps per bootstrap (DUO) that wave takes 3.91 and 5.24 ms,
// against 4.95 and 6.22 ms for the paired and the team kernel.
// N = 2048: two warps per bootstrap, each with half of every transform's points (big below): one wave of 592 takes 10.6 ms
// split and 14.9 ms FP64, against 10.2 ms per 444 for the paired kernel and 10.35 ms per 296 for the team kernel.
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "async_copy.cuh"
#include "br_common.cuh"
#include "fft.cuh"
#include "internal.h"
#include "tmem.cuh"

namespace tfheb {

namespace {

constexpr int kWarpTeams = 8;  // most bootstraps per CTA
enum class WarpMode {
    solo,  // N = 1024, one warp per bootstrap
    duo,   // N = 1024, two warps per bootstrap, each with half of the transforms
    big    // N = 2048, two warps per bootstrap, each with half of every transform's points
};

// ---- the exchange passes -----------------------------------------------------------------------
// v[64]: the warp's 16 points per lane, 4 words each (two components ri = re, im of two words e: the
// two packed floats, or the low and high word of a double).  `col` is a 64-column region of the warp's
// quadrant.  forward(): the registers become v[32 hh + 4 j + 2 q + e] = word 8 j + 2 (lane & 3) + e of
// lane 16 hh + 8 q + (lane >> 2).  backward() is its inverse.
// S16: 16 words per store instruction instead of 32.  The doubles' results reach the registers of a store with
// fewer moves that way (8.0k instructions per bootstrap step against 8.7k, 10.1 ms per 1184 bootstraps
// against 10.5); packed floats need next to none either way.
// swap() (BIG): the two warps of a team, `half` 0 and 1, trade the group bit of the registers (v[0..31], v[32..63])
// for their own: warp w gets group w of warp 0, then group w of warp 1.  Every lane keeps its place.
template <bool S16>
struct WarpExch {
    uint32_t col;
    int bar;  // BIG: named barrier of the team's two warps
    __device__ __forceinline__ void team() const {
        tmem_fence_before_sync();
        team_sync(bar, 64);
        tmem_fence_after_sync();
    }
    __device__ __forceinline__ void swap(uint32_t (&v)[64], int half) const {
        if constexpr (S16) {
#pragma unroll
            for (int c = 0; c < 64; c += 16) tmem_st16(col + (uint32_t)c, v + c);
        } else {
            tmem_st32p(col, v);
            tmem_st32p(col + 32u, v + 32);
        }
        tmem_wait_st();
        team();
        const uint32_t first = col - (uint32_t)(256 * half) + (uint32_t)(32 * half);
        tmem_ld32(first, v);
        tmem_ld32(first + 256u, v + 32);
        tmem_wait_ld64(v);
        team();  // the regions are free again
    }
    __device__ __forceinline__ void forward(uint32_t (&v)[64]) const {
        if constexpr (S16) {
#pragma unroll
            for (int c = 0; c < 64; c += 16) tmem_st16(col + (uint32_t)c, v + c);
        } else {
            tmem_st32p(col, v);
            tmem_st32p(col + 32u, v + 32);
        }
        tmem_wait_st();
        tmem_ld_16x256x8(col, v);
        tmem_ld_16x256x8(col + (16u << 16), v + 32);
        tmem_wait_ld64(v);
    }
    __device__ __forceinline__ void backward(uint32_t (&v)[64]) const {
        if constexpr (S16) {
#pragma unroll
            for (int c = 0; c < 64; c += 16)
                tmem_st_16x256x4(col + (c < 32 ? 0u : 16u << 16) + 2u * (uint32_t)(c & 16), v + c);
        } else {
            tmem_st_16x256x8(col, v);
            tmem_st_16x256x8(col + (16u << 16), v + 32);
        }
        tmem_wait_st();
        tmem_ld32(col, v);
        tmem_ld32(col + 32u, v + 32);
        tmem_wait_ld64(v);
    }
};

// Word positions of the three passes.  Stage 0's butterfly h of lane l is t = l + 32 h = 8 n1 + n2 with
// outputs k0; stage 1 runs over n1 for (k0, n2) with outputs k1; stage 2 over n2 for (k0, k1).
//   pass 1  in:  butterfly h, k0 = 2 b + kl           out (lane = n2, b):  kl, n1
//   pass 2  in:  kl, k1                               out (lane = n2 & 1, b, kl, k1 >> 2):  n2 >> 1, q = k1 & 3
//   pass 3  in:  i (forward: k2 & 3; inverse: n2 >> 1), q   out (lane = b & 1, kl, k1):  h = b >> 1, n2 & 1, i
// so that stage 2's butterfly h of lane l is again the virtual thread l + 32 h = 8 k0 + k1.  Registers leave
// a load in another order than the next store wants them, so there is arithmetic between any two passes to
// write its results in that order (64 register moves per transform otherwise): in the forward transform stage 2's
// radix-4 half, which needs n2 >> 1 only, runs between passes 2 and 3; in the inverse stage 1's twiddle
// factors are applied between passes 3 and 2.
__device__ __forceinline__ constexpr int p1_in(int h, int k0, int ri, int e) {
    return 32 * h + 16 * (k0 & 1) + 8 * ri + 2 * (k0 >> 1) + e;
}
__device__ __forceinline__ constexpr int p1_out(int kl, int n1, int ri, int e) {
    return 32 * ((n1 >> 1) & 1) + 4 * (4 * (n1 >> 2) + 2 * kl + ri) + 2 * (n1 & 1) + e;
}
__device__ __forceinline__ constexpr int p2_in(int kl, int k1, int ri, int e) {
    return 16 * (k1 & 3) + 8 * ri + 4 * kl + 2 * (k1 >> 2) + e;
}
__device__ __forceinline__ constexpr int p2_out(int n2h, int q, int ri, int e) {
    return 32 * (n2h >> 1) + 4 * (2 * q + ri) + 2 * (n2h & 1) + e;
}
__device__ __forceinline__ constexpr int p3_in(int i, int q, int ri, int e) { return 8 * (2 * i + ri) + 2 * q + e; }
__device__ __forceinline__ constexpr int p3_out(int h, int odd, int i, int ri, int e) {
    return 32 * odd + 8 * i + 4 * ri + 2 * h + e;
}

// the two words of a component of one point
__device__ __forceinline__ uint32_t word_of(float2 c, int e) { return __float_as_uint(e ? c.y : c.x); }
__device__ __forceinline__ uint32_t word_of(double c, int e) {
    return (uint32_t)(e ? __double2hiint(c) : __double2loint(c));
}
__device__ __forceinline__ void from_words(float2 &c, uint32_t w0, uint32_t w1) {
    c = make_float2(__uint_as_float(w0), __uint_as_float(w1));
}
__device__ __forceinline__ void from_words(double &c, uint32_t w0, uint32_t w1) { c = __hiloint2double((int)w1, (int)w0); }

// Arithmetic of one transform of packed FP32 pairs (TeamFft2's) or of doubles (TeamFft<double>'s).  A packed
// instruction takes one word for both halves of an operand, or its negation, at no cost, so the factors are
// single words: TeamFft<float>'s table, two factors per 16-byte load.
template <int M>
struct PairOps {
    static constexpr int NT = M / kR, st1 = M / (kR * kR);  // virtual team threads, stage 1's stride
    using point = cpair;
    using factor = float2;
    using Exch = WarpExch<false>;
    template <bool INV>
    __device__ static __forceinline__ void dft8(point *x) { pdft8<INV>(x); }
    template <bool INV>
    __device__ static __forceinline__ void dft4(point &a, point &b, point &c, point &d) { pdft4<INV>(a, b, c, d); }
    // the last step of pdft8: x[k], x[k + 4] from the radix-4 results of the even and odd points
    __device__ static __forceinline__ void combine(point *x, const point (&e)[4], const point (&o)[4]) {
        const float2 h = bc2(rsqrt2<float>()), nh = bc2(-rsqrt2<float>());
        x[0] = padd(e[0], o[0]);
        x[4] = psub(e[0], o[0]);
        const float2 u1 = add2(o[1].re, o[1].im), v1 = sub2(o[1].im, o[1].re);
        const float2 u3 = sub2(o[3].im, o[3].re), p3 = add2(o[3].re, o[3].im);
        x[1] = {fma2(u1, h, e[1].re), fma2(v1, h, e[1].im)};
        x[5] = {fma2(u1, nh, e[1].re), fma2(v1, nh, e[1].im)};
        x[3] = {fma2(u3, h, e[3].re), fma2(p3, nh, e[3].im)};
        x[7] = {fma2(u3, nh, e[3].re), fma2(p3, h, e[3].im)};
        x[2] = {add2(e[2].re, o[2].im), sub2(e[2].im, o[2].re)};
        x[6] = {sub2(e[2].re, o[2].im), add2(e[2].im, o[2].re)};
    }
    template <bool INV>
    __device__ static __forceinline__ void mul(point &a, factor w) {
        const float2 wr = bc2(w.x), wi = bc2(w.y), nwi = bc2(-w.y);
        a = INV ? pmulconj(a, wr, wi, nwi) : pmul(a, wr, wi, nwi);
    }
    template <bool INV>
    __device__ static __forceinline__ void fold(point *x) { TeamFft2<M>::fold_consts<INV>(x); }
    // tables: stage 0 factors 2 q, 2 q + 1 at t (see WarpFft); stages 1 and 2 factors 2 q + 1, 2 q + 2 at n;
    // mid-table factors 2 i, 2 i + 1 of a row
    static constexpr size_t table_bytes = tw_table_bytes<float, M>(), row_bytes = 9 * 16;
    __device__ static __forceinline__ void two(const void *tab, int at, factor &a, factor &b) {
        const float4 w = reinterpret_cast<const float4 *>(tab)[at];
        a = make_float2(w.x, w.y);
        b = make_float2(w.z, w.w);
    }
    __device__ static __forceinline__ void stage0(const void *tab, int q, int t, factor &a, factor &b) {
        two(tab, q * NT + t, a, b);
    }
    template <int S>
    __device__ static __forceinline__ void stage(const void *tab, int q, int n, factor &a, factor &b) {
        two(tab, tw4_offset<M>(S) + q * (S == 1 ? st1 : st1 / kR) + n, a, b);
    }
    __device__ static __forceinline__ void mid(const void *tab, int i, int row, factor &a, factor &b) {
        two(tab, row * 9 + i, a, b);
    }
    // entry f of a mid-table row = stage 1's factor of (k1, n), 1 where k1 = 0
    __device__ static __forceinline__ void put_mid(void *mid_tab, const void *tab, int row, int f, int k1, int n) {
        const factor *w = static_cast<const factor *>(tab) + 2 * (tw4_offset<M>(1) + n);
        static_cast<factor *>(mid_tab)[row * 18 + f] =
            k1 ? w[2 * st1 * ((k1 - 1) / 2) + (k1 - 1) % 2] : make_float2(1.0f, 0.0f);
    }
};
template <int M>
struct DoubleOps {
    static constexpr int NT = M / kR, st1 = M / (kR * kR);
    using point = cplx<double>;
    using factor = cplx<double>;
    using Exch = WarpExch<true>;
    template <bool INV>
    __device__ static __forceinline__ void dft8(point *x) { tfheb::dft8<double, INV>(x); }
    template <bool INV>
    __device__ static __forceinline__ void dft4(point &a, point &b, point &c, point &d) {
        tfheb::dft4<double, INV>(a, b, c, d);
    }
    __device__ static __forceinline__ void combine(point *x, const point (&e)[4], const point (&o)[4]) {
        const double h = rsqrt2<double>();
        x[0] = cadd(e[0], o[0]);
        x[4] = csub(e[0], o[0]);
        const double u1 = o[1].re + o[1].im, v1 = o[1].im - o[1].re;
        const double u3 = o[3].im - o[3].re, v3 = -(o[3].re + o[3].im);
        x[1] = {fma(u1, h, e[1].re), fma(v1, h, e[1].im)};
        x[5] = {fma(-u1, h, e[1].re), fma(-v1, h, e[1].im)};
        x[3] = {fma(u3, h, e[3].re), fma(v3, h, e[3].im)};
        x[7] = {fma(-u3, h, e[3].re), fma(-v3, h, e[3].im)};
        const point w2 = rot_quarter<double, false>(o[2]);
        x[2] = cadd(e[2], w2);
        x[6] = csub(e[2], w2);
    }
    template <bool INV>
    __device__ static __forceinline__ void mul(point &a, factor w) { a = INV ? cmulconj(a, w) : cmul(a, w); }
    template <bool INV>
    __device__ static __forceinline__ void fold(point *x) { TeamFft<double, M, kR>::template fold_consts<INV>(x); }
    static constexpr size_t table_bytes = tw_table_bytes<double, M>(), row_bytes = 17 * 16;
    __device__ static __forceinline__ void stage0(const void *tab, int q, int t, factor &a, factor &b) {
        const factor *w = static_cast<const factor *>(tab) + 2 * q * NT + t;
        a = w[0];
        b = w[NT];
    }
    template <int S>
    __device__ static __forceinline__ void stage(const void *tab, int q, int n, factor &a, factor &b) {
        constexpr int st = S == 1 ? st1 : st1 / kR;
        const factor *w = static_cast<const factor *>(tab) + tw_offset<M>(S) + 2 * q * st + n;
        a = w[0];
        if (2 * q + 2 < kR) b = w[st];
    }
    __device__ static __forceinline__ void mid(const void *tab, int i, int row, factor &a, factor &b) {
        const factor *w = static_cast<const factor *>(tab) + row * 17 + 2 * i;
        a = w[0];
        b = w[1];
    }
    __device__ static __forceinline__ void put_mid(void *mid_tab, const void *tab, int row, int f, int k1, int n) {
        const factor *w = static_cast<const factor *>(tab) + tw_offset<M>(1) + n;
        static_cast<factor *>(mid_tab)[row * 17 + f] = k1 ? w[(k1 - 1) * st1] : factor{1.0, 0.0};
    }
};

__device__ __forceinline__ cpair point_add(const cpair &a, const cpair &b) { return padd(a, b); }
__device__ __forceinline__ cpair point_sub(const cpair &a, const cpair &b) { return psub(a, b); }
__device__ __forceinline__ cplx<double> point_add(const cplx<double> &a, const cplx<double> &b) { return cadd(a, b); }
__device__ __forceinline__ cplx<double> point_sub(const cplx<double> &a, const cplx<double> &b) { return csub(a, b); }

// BIG (N = 2048): the plan 8 x 8 x 8 x 2 over two warps, half = 0 or 1.  Stage 0's butterfly is t = 16 n1 + 2 n2 + n3; a
// warp starts with n3 = half, so that up to stage 2 both do what one does at N = 1024 (t >> 1 in the place of t, and
// the factors of their n3: stage 2's are 1 for n3 = 0).  Then WarpExch::swap trades n3 for h, the high bit of k0:
// stage 3's radix-2 butterfly has its two points in one warp.  Slot (k3, k2) of lane l in warp `half` is position
// p = 2 (t' + 128 c) + k3 with t' = 64 (l >> 3 & 1) + 8 (l & 7) + k2 and c = 2 half + (l >> 4).
template <class Ops, bool BIG>
struct WarpFft {
    using point = typename Ops::point;
    using factor = typename Ops::factor;

    __device__ static __forceinline__ void get(point &p, const uint32_t *v, int re, int im) {
        from_words(p.re, v[re], v[re + 1]);
        from_words(p.im, v[im], v[im + 1]);
    }
    __device__ static __forceinline__ void put(uint32_t *v, int re, int im, const point &p) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            v[re + e] = word_of(p.re, e);
            v[im + e] = word_of(p.im, e);
        }
    }

    // In: z[h][r] = a_j - i a_{j+M}, j = lane + 32 h + 64 r (BIG: 2 (lane + 32 h) + half + 128 r).  Out: slot r of
    // virtual thread lane + 32 h (BIG: slot (h, r) as above).
    __device__ static __forceinline__ void forward(point (&z)[2][kR], const typename Ops::Exch &x, const void *tab, int lane,
                                                   int half) {
        const int t0 = lane + (BIG ? 64 * half : 0), n = BIG ? 2 * (lane >> 2) + half : lane >> 2;
        uint32_t v[64], w[64];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            Ops::template fold<false>(z[h]);
            Ops::template dft8<false>(z[h]);
#pragma unroll
            for (int q = 0; q < kR / 2; q++) {
                factor a, b;
                Ops::stage0(tab, q, t0 + 32 * h, a, b);
                Ops::template mul<false>(z[h][2 * q], a);
                Ops::template mul<false>(z[h][2 * q + 1], b);
            }
#pragma unroll
            for (int k = 0; k < kR; k++) put(v, p1_in(h, k, 0, 0), p1_in(h, k, 1, 0), z[h][k]);
        }
        x.forward(v);
        point y[2][kR];
#pragma unroll
        for (int kl = 0; kl < 2; kl++) {
#pragma unroll
            for (int n = 0; n < kR; n++) get(y[kl][n], v, p1_out(kl, n, 0, 0), p1_out(kl, n, 1, 0));
            Ops::template dft8<false>(y[kl]);
        }
#pragma unroll
        for (int q = 0; q < kR / 2; q++) {
            factor a, b;
            Ops::template stage<1>(tab, q, n, a, b);
#pragma unroll
            for (int kl = 0; kl < 2; kl++) {
                Ops::template mul<false>(y[kl][2 * q + 1], a);
                if (2 * q + 2 < kR) Ops::template mul<false>(y[kl][2 * q + 2], b);
            }
        }
#pragma unroll
        for (int kl = 0; kl < 2; kl++)
#pragma unroll
            for (int k = 0; k < kR; k++) put(w, p2_in(kl, k, 0, 0), p2_in(kl, k, 1, 0), y[kl][k]);
        x.forward(w);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            point g[4];
#pragma unroll
            for (int i = 0; i < 4; i++) get(g[i], w, p2_out(i, q, 0, 0), p2_out(i, q, 1, 0));
            Ops::template dft4<false>(g[0], g[1], g[2], g[3]);
#pragma unroll
            for (int i = 0; i < 4; i++) put(v, p3_in(i, q, 0, 0), p3_in(i, q, 1, 0), g[i]);
        }
        x.forward(v);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            point e[4], o[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                get(e[i], v, p3_out(h, 0, i, 0, 0), p3_out(h, 0, i, 1, 0));
                get(o[i], v, p3_out(h, 1, i, 0, 0), p3_out(h, 1, i, 1, 0));
            }
            Ops::combine(z[h], e, o);
        }
        if constexpr (BIG) {
            stage2_factors<false>(z, tab, half);
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int k = 0; k < kR; k++) put(v, 32 * h + 4 * k, 32 * h + 4 * k + 2, z[h][k]);
            x.swap(v, half);
            butterflies(z, v);
        }
    }
    // stage 2's factors, 1 in the warp with n3 = 0
    template <bool INV>
    __device__ static __forceinline__ void stage2_factors(point (&z)[2][kR], const void *tab, int half) {
        if (half == 0) return;
#pragma unroll
        for (int q = 0; q < kR / 2; q++) {
            factor a, b;
            Ops::template stage<2>(tab, q, 1, a, b);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                Ops::template mul<INV>(z[h][2 * q + 1], a);
                if (2 * q + 2 < kR) Ops::template mul<INV>(z[h][2 * q + 2], b);
            }
        }
    }
    // radix 2 over the two groups of v
    __device__ static __forceinline__ void butterflies(point (&z)[2][kR], const uint32_t *v) {
#pragma unroll
        for (int k = 0; k < kR; k++) {
            point a, b;
            get(a, v, 4 * k, 4 * k + 2);
            get(b, v, 32 + 4 * k, 32 + 4 * k + 2);
            z[0][k] = point_add(a, b);
            z[1][k] = point_sub(a, b);
        }
    }

    // Slot r of virtual thread lane + 32 h in, z[h][r] = M (c_j - i c_{j+M}) out (the adjoint stages).
    __device__ static __forceinline__ void inverse(point (&z)[2][kR], const typename Ops::Exch &x, const void *tab,
                                                   const void *mid_tab, int lane, int half) {
        const int t0 = lane + (BIG ? 64 * half : 0);
        uint32_t v[64], w[64];
        if constexpr (BIG) {
#pragma unroll
            for (int k = 0; k < kR; k++) {
                put(v, 4 * k, 4 * k + 2, point_add(z[0][k], z[1][k]));
                put(v, 32 + 4 * k, 32 + 4 * k + 2, point_sub(z[0][k], z[1][k]));
            }
            x.swap(v, half);
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int k = 0; k < kR; k++) get(z[h][k], v, 32 * h + 4 * k, 32 * h + 4 * k + 2);
            stage2_factors<true>(z, tab, half);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            Ops::template dft8<true>(z[h]);
#pragma unroll
            for (int n = 0; n < kR; n++)
                put(v, p3_out(h, n & 1, n >> 1, 0, 0), p3_out(h, n & 1, n >> 1, 1, 0), z[h][n]);
        }
        x.backward(v);
        const int row = (BIG ? 4 * half : 0) + 2 * (lane >> 4) + (lane & 1);  // (n3,) n2 & 1, k1 >> 2
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int qq = 0; qq < 2; qq++) {
                factor f[2];
                Ops::mid(mid_tab, 2 * i + qq, row, f[0], f[1]);
#pragma unroll
                for (int s = 0; s < 2; s++) {
                    const int q = 2 * qq + s;
                    point p;
                    get(p, v, p3_in(i, q, 0, 0), p3_in(i, q, 1, 0));
                    Ops::template mul<true>(p, f[s]);
                    put(w, p2_out(i, q, 0, 0), p2_out(i, q, 1, 0), p);
                }
            }
        x.backward(w);
        point y[2][kR];
#pragma unroll
        for (int kl = 0; kl < 2; kl++) {
#pragma unroll
            for (int k = 0; k < kR; k++) get(y[kl][k], w, p2_in(kl, k, 0, 0), p2_in(kl, k, 1, 0));
            Ops::template dft8<true>(y[kl]);
#pragma unroll
            for (int n = 0; n < kR; n++) put(v, p1_out(kl, n, 0, 0), p1_out(kl, n, 1, 0), y[kl][n]);
        }
        x.backward(v);
#pragma unroll
        for (int h = 0; h < 2; h++) {
#pragma unroll
            for (int q = 0; q < kR / 2; q++) {
                factor a, b;
                Ops::stage0(tab, q, t0 + 32 * h, a, b);
#pragma unroll
                for (int s = 0; s < 2; s++) {
                    get(z[h][2 * q + s], v, p1_in(h, 2 * q + s, 0, 0), p1_in(h, 2 * q + s, 1, 0));
                    Ops::template mul<true>(z[h][2 * q + s], s ? b : a);
                }
            }
            Ops::template dft8<true>(z[h]);
            Ops::template fold<true>(z[h]);
        }
    }
};

// ---- shared memory and TMEM ---------------------------------------------------------------------
// Per warp 256 TMEM columns (two warps of a quadrant side by side).  Split: the KPL spectra, 64 words per
// lane and digit pair, from column 0, the step's rotated words (64 per lane) from 128 on -- the last pair's
// spectra overwrite them once they have been read.  FP64: the two outputs' accumulators, 64 words per lane
// each, then the rotated words.  Both: the exchange region from 192 on.  The key ring's unit is 16 KB: one
// output's slots of a digit pair (split), or one digit's row (FP64); the ring holds whole steps.
// DUO: a quadrant's two warps share one bootstrap and its 512 columns: spectra or (FP64) two outputs'
// accumulators per warp, rotated words, an exchange region per warp.
// big: as solo, with every column count per warp, and the ring holds half a step.
template <bool SPLIT, int L, int D, WarpMode MODE>
struct WarpLayout {
    static constexpr bool duo = MODE == WarpMode::duo, big = MODE == WarpMode::big;
    static constexpr int N = big ? 2048 : 1024, M = N / 2, NT = M / kR;
    using Ops = std::conditional_t<SPLIT, PairOps<M>, DoubleOps<M>>;
    static constexpr int KP1 = 2, KPL = KP1 * L;
    static constexpr int teams = MODE == WarpMode::solo ? kWarpTeams : kWarpTeams / 2;  // most bootstraps per CTA
    static constexpr uint32_t half = (uint32_t)M * 16;  // one output's slots of one key row
    static constexpr uint32_t unit = 2 * half;          // KPL units per step
    static constexpr size_t bars = 0;                   // full[D], empty[D], abort flag, TMEM address
    static constexpr size_t ring = (2 * D * 8 + 8 + 127) / 128 * 128;
    static constexpr size_t tables = ring + (size_t)D * unit;
    static constexpr size_t mid = tables + Ops::table_bytes;
    static constexpr int mid_rows = big ? 8 : 4;
    static constexpr size_t accs = (mid + mid_rows * Ops::row_bytes + 127) / 128 * 128;
    static constexpr size_t acc_bytes = 4 * (size_t)KP1 * N;
    static constexpr size_t bytes(int G) { return accs + (size_t)G * acc_bytes; }
    static constexpr uint32_t col_xr = !duo ? 128 : SPLIT ? 192 : 256, col_exch = !duo ? 192 : SPLIT ? 256 : 320;
    // ring slot and mbarrier phase of unit i of a step: fixed within a step, or within half of one
    static_assert(D % KPL == 0 || (D == L && KPL == 2 * D), "whole steps, or half a step");
    __device__ static __forceinline__ int slot(int step, int i) {
        return D % KPL == 0 ? (step % (D / KPL)) * KPL + i : i % D;
    }
    __device__ static __forceinline__ uint32_t phase(int step, int i) {
        return D % KPL == 0 ? (uint32_t)(step / (D / KPL)) & 1u : (uint32_t)(i / D);  // two turns a step
    }
    static_assert(KPL * 32 <= 192 && KPL % 2 == 0, "spectra columns");
    static_assert(bytes(teams) <= 227 * 1024, "shared memory of the variant");
};

// the digits' top bits of a rotated word are kept in its low 23 bits (split form, N = 1024): no parameter set with
// wider digits may come here
constexpr int kDigitBits = 23, kDigitShift = 32 - kDigitBits;

__device__ __forceinline__ float2 digit_pair(uint32_t a, uint32_t b) {
    return make_float2(__int_as_float(0x4B000000u | a), __int_as_float(0x4B000000u | b));
}

}  // namespace

// Three warpgroups: eight warps of which the first args.teams run a bootstrap each, with 232 registers, and one
// whose first thread streams the key in the order of the multiply-accumulates (the other three warps
// only take part in the register split: a ninth warp alone would cap all of them at 168).
// DUO, for at most four bootstraps per CTA: warps w and w + 4, which share a scheduler and a TMEM quadrant, run one
// bootstrap together, so that each scheduler still has two warps to choose from.  Warp (role) u keeps
// polynomial u of the accumulator and computes output u.  Split: the digit pairs go to the two in turn, and both
// read all spectra from TMEM.  FP64: each transforms its polynomial's digits and multiplies them with the key of
// both outputs; the two partial sums of an output meet at the end (FP64 sums round to the exact integers in
// any order, as long as digits are narrow enough: kReorderBits in blind_rotate.cu).
//
// big: warps w and w + 4 hold the two halves of every transform (WarpFft), and of the slots, key rows and accumulator
// words; the accumulator keeps even and odd coefficients apart, so that a warp's are consecutive.
template <bool SPLIT, int L, int D, WarpMode MODE>
__global__ void __launch_bounds__((kWarpTeams + 4) * 32, 1) blind_rotate_warp_kernel(const BrArgs args) {
    using Lay = WarpLayout<SPLIT, L, D, MODE>;
    using Ops = typename Lay::Ops;
    constexpr bool DUO = Lay::duo, BIG = Lay::big;
    constexpr int N = Lay::N, NT = Lay::NT, KP1 = 2, KPL = KP1 * L;
    constexpr bool SHIFTED = SPLIT && !BIG;  // digits from words shifted into a float's mantissa
    using F = WarpFft<Ops, BIG>;
    extern __shared__ __align__(128) unsigned char smem[];

    // the same in every lane, in a way the compiler can see (uniform registers for the TMEM addresses)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int G = args.teams;
    const int active = min(G, args.boots - (int)blockIdx.x * G);
    const uint32_t bar0 = smem_addr(smem + Lay::bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (D + s); };
    volatile int32_t *abort_flag = reinterpret_cast<volatile int32_t *>(smem + Lay::bars + 16 * D);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + Lay::bars + 16 * D + 4);
    const uint32_t ring = smem_addr(smem + Lay::ring);

    if (threadIdx.x == 0) {
        for (int s = 0; s < D; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), (uint32_t)(BIG ? 2 * active : active));
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(smem_addr(tmem_slot), 512);
    {
        const int4 *g_tab = reinterpret_cast<const int4 *>(args.tables);
        int4 *s_tab4 = reinterpret_cast<int4 *>(smem + Lay::tables);
        constexpr int stage0 = (SPLIT ? kR / 2 : kR) * NT;
        for (int i = threadIdx.x; i < (int)(Ops::table_bytes / 16); i += blockDim.x) {
            int at = i;  // big: stage 0's factors of even t, then of odd t
            if (BIG && i < stage0) at = (i & ~(NT - 1)) + (i & 1) * (NT / 2) + ((i & (NT - 1)) >> 1);
            s_tab4[at] = g_tab[i];
        }
        // mid-table row (n3, n2 & 1, k1 >> 2), entry 4 (n2 >> 1) + (k1 & 3)
        if (threadIdx.x < 16 * Lay::mid_rows) {
            const int row = threadIdx.x >> 4, f = threadIdx.x & 15, n2 = 2 * (f >> 2) + (row >> 1 & 1);
            Ops::put_mid(smem + Lay::mid, args.tables, row, f, 4 * (row & 1) + (f & 3), BIG ? 2 * n2 + (row >> 2) : n2);
        }
    }
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp >= kWarpTeams) {  // ---- producer ----
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (threadIdx.x == kWarpTeams * 32) {
            const uint8_t *bsk = SPLIT || BIG ? args.bsk2 : args.bsk;
            const int total = args.nsteps * KPL;
            int sent = 0;
            if (!args.stall_producer) {
                for (int c = 0; c < total; c++) {
                    const int s = c % D;
                    if (c >= D && !wait_bounded(empty_bar(s), ((c / D) - 1) & 1, abort_flag, args.timeout_ns, args.err))
                        break;
                    const uint32_t dst = ring + (uint32_t)s * Lay::unit;
                    mbar_arrive_expect_tx(full_bar(s), Lay::unit);
                    if constexpr (SPLIT) {
                        const int step = c / KPL, rem = c - step * KPL;
                        const int v = rem / L, d = 2 * (rem - v * L);
                        const uint8_t *src = bsk + ((size_t)(step * KPL + d) * KP1 + v) * Lay::half;
                        bulk_copy_g2s(dst, src, Lay::half, full_bar(s));
                        bulk_copy_g2s(dst + Lay::half, src + (size_t)KP1 * Lay::half, Lay::half, full_bar(s));
                    } else {
                        bulk_copy_g2s(dst, bsk + (size_t)c * Lay::unit, Lay::unit, full_bar(s));
                    }
                    sent = c + 1;
                }
            }
            volatile int32_t no_abort = 0;
            for (int c = (sent > D ? sent - D : 0); c < sent; c++)
                wait_bounded(full_bar(c % D), (c / D) & 1, &no_abort, args.timeout_ns, args.err);
        }
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    const int team = DUO || BIG ? warp & 3 : warp, role = DUO ? warp >> 2 : 0, half = BIG ? warp >> 2 : 0;
    if (team >= active) return;  // no TMEM use, not counted in any barrier below

    // ---- consumer warps ----
    const int boot = blockIdx.x * G + team;
    uint32_t *s_acc = reinterpret_cast<uint32_t *>(smem + Lay::accs + (size_t)team * Lay::acc_bytes);
    const void *s_tab = smem + Lay::tables, *s_mid = smem + Lay::mid;
    const uint32_t tmem = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (DUO ? 0u : (uint32_t)((warp >> 2) * 256));
    const typename Ops::Exch exch{tmem + Lay::col_exch + (uint32_t)(64 * role), 2 + team};
    // DUO: both warps of the bootstrap, their TMEM accesses before it ordered before those after it
    auto duo_sync = [&] {
        if constexpr (DUO) exch.team();
    };
    const int first = lane + 32 * (role + half), stride = DUO || BIG ? 64 : 32;
    // place of coefficient j of a polynomial (i over both)
    auto place = [](int i) { return BIG ? (i & ~(N - 1)) + ((i & 1) << 10) + ((i & (N - 1)) >> 1) : i; };

    const int32_t *my_bara = args.bara + (size_t)boot * args.bara_stride;
    if (args.acc_in) {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(args.acc_in) + (size_t)boot * KP1 * N;
        for (int i = first; i < KP1 * N; i += stride) s_acc[place(i)] = src[i];
    } else {
        // acc = (0, X^{2N-barb} * [mu,...,mu])  (lwe-bootstrapping-functions-fft.cpp:142-145)
        const int e = 2 * N - my_bara[args.nsteps];
        for (int i = first; i < N; i += stride) s_acc[i] = 0u;
        for (int j = first; j < N; j += stride) {
            int src = j - e;
            uint32_t neg = 0;
            while (src < 0) {
                src += N;
                neg ^= 1u;
            }
            s_acc[N + place(j)] = neg ? 0u - (uint32_t)args.mu : (uint32_t)args.mu;
        }
    }
    __syncwarp();
    if constexpr (DUO || BIG) team_sync(2 + team, 64);

    // gadget constants (tgsw.cpp:7-29)
    const int Bgbit = args.Bgbit;
    uint32_t offset = 0;
#pragma unroll
    for (int q = 0; q < L; q++) offset += 1u << (32 - (q + 1) * Bgbit);
    offset *= 1u << (Bgbit - 1);
    const uint32_t maskBg = (1u << Bgbit) - 1u;

    const int split_shift = args.split_shift;
    int a_next = args.nsteps > 0 ? my_bara[0] : 0;
    for (int step = 0; step < args.nsteps; step++) {
        const int ai = a_next & (2 * N - 1);
        if (step + 1 < args.nsteps) a_next = my_bara[step + 1];

        // 1. (X^a - 1) * poly + offset of both polynomials (rot_minus_one); word i of a lane is j = lane + 32 i.
        //    Coefficient e = j - a mod 2N is e mod N, negated when e has the N bit; both polynomials share
        //    the index and the sign.  Split: only the l Bgbit <= 23 top bits are digits, and they are shifted
        //    down into a float's mantissa here, so that a digit is one mask away from being a float below.
        //    A loop of two halves: the whole step unrolled misses the instruction cache (one warp per
        //    scheduler ran 14.9k cycles a step with this loop, 16.0k without).
        {
            // byte index of e; big: of e's place among the even or odd coefficients, the same for all of the warp's j
            const uint32_t rot = 4u * (uint32_t)(BIG ? (2 * lane + half - ai) >> 1 : lane - ai);
            const uint32_t *polys = s_acc + role * N;  // DUO: the warp's own polynomial only
            const uint32_t *from = BIG ? polys + (((half - ai) & 1) << 10) : polys;
#pragma unroll 1
            for (int i0 = 0; i0 < 32; i0 += 16) {
                uint32_t x0[16], x1[16];
                const uint32_t *own = polys + 1024 * half + lane + 32 * i0;
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const uint32_t e = rot + 128u * (uint32_t)(i0 + i);
                    const uint32_t neg = (uint32_t)((int32_t)(e << 19) >> 31);
                    const uint32_t on = offset - neg;
                    const uint32_t *src =
                        reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(from) + (e & 4095u));
                    x0[i] = ((src[0] ^ neg) + (on - own[32 * i])) >> (SHIFTED ? kDigitShift : 0);
                    if constexpr (!DUO) x1[i] = ((src[N] ^ neg) + (on - own[32 * i + N])) >> (SHIFTED ? kDigitShift : 0);
                }
                tmem_st16(tmem + Lay::col_xr + (uint32_t)(32 * role + i0), x0);
                if constexpr (!DUO) tmem_st16(tmem + Lay::col_xr + 32u + (uint32_t)i0, x1);
            }
        }
        tmem_wait_st();

        if constexpr (SPLIT) {
            // 2. digits two at a time, forward transforms, spectra to TMEM (DUO: which the other warp has read
            //    when it gets here)
            duo_sync();
#pragma unroll 1
            for (int d0 = 2 * role; d0 < KPL; d0 += DUO ? 4 : 2) {
                const int u0 = d0 / L, u1 = (d0 + 1) / L;
                // digit q of a word: its bits under the exponent of 2^23 are the float 2^23 + d 2^sh; times
                // 2^-sh, minus (2^23 2^-sh + Bg/2): exact, one operation for the pair
                const int sh0 = 32 - (d0 - u0 * L + 1) * Bgbit - (SHIFTED ? kDigitShift : 0);
                const int sh1 = 32 - (d0 + 1 - u1 * L + 1) * Bgbit - (SHIFTED ? kDigitShift : 0);
                const uint32_t m0 = SHIFTED ? maskBg << sh0 : maskBg, m1 = SHIFTED ? maskBg << sh1 : maskBg;
                const float2 sc = SHIFTED ? make_float2(__int_as_float((127 - sh0) << 23), __int_as_float((127 - sh1) << 23))
                                          : make_float2(1.0f, 1.0f);
                const float half_bg = float(1 << (Bgbit - 1));
                const float2 bias = make_float2(8388608.0f * sc.x + half_bg, 8388608.0f * sc.y + half_bg);
                uint32_t xa[32], xb[32];
                tmem_ld32(tmem + Lay::col_xr + (uint32_t)(32 * u0), xa);
                tmem_ld32(tmem + Lay::col_xr + (uint32_t)(32 * u1), xb);
                tmem_wait_ld32(xa);
                tmem_tie32(xb);
                cpair z[2][kR];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int r = 0; r < kR; r++) {  // j = lane + 32 (h + 2 r); j + M is word 16 on
                        const int i = h + 2 * r;
                        const int s0 = SHIFTED ? 0 : sh0, s1 = SHIFTED ? 0 : sh1;
                        const float2 lo = digit_pair((xa[i] >> s0) & m0, (xb[i] >> s1) & m1);
                        const float2 hi = digit_pair((xa[i + 16] >> s0) & m0, (xb[i + 16] >> s1) & m1);
                        if constexpr (SHIFTED) z[h][r] = {fma2(lo, sc, neg2(bias)), fma2(neg2(hi), sc, bias)};
                        else z[h][r] = {sub2(lo, bias), sub2(bias, hi)};
                    }
                F::forward(z, exch, s_tab, lane, half);
                // per butterfly h and slot r: re of both digits, im of both
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint32_t w[32];
#pragma unroll
                    for (int r = 0; r < kR; r++) F::put(w, 4 * r, 4 * r + 2, z[h][r]);
                    tmem_st32p(tmem + (uint32_t)(32 * d0 + 32 * h), w);
                }
            }
            tmem_wait_st();
            duo_sync();

            // 3. per output polynomial: multiply-accumulate over the digits against the key, each accumulator the
            //    pair of the key's limbs (hi, lo), then both limbs' inverse transforms as one pair, exact
            //    rounding, accumulate
#pragma unroll 1
            for (int v = role; v < (DUO ? role + 1 : KP1); v++) {
                cpair acc[2][kR];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int r = 0; r < kR; r++) acc[h][r] = {{0.f, 0.f}, {0.f, 0.f}};
                // keys of butterfly h and digit dd of the ring unit at `at`: {hi.re, lo.re, hi.im, lo.im} per slot.  Each
                // quarter of a unit is loaded while the one before is multiplied.
                auto load = [&](float4(&k)[kR], const unsigned char *at, int h, int dd) {
                    const float4 *kp = reinterpret_cast<const float4 *>(at + dd * Lay::half) + lane +
                                       (BIG ? 512 * half + 256 * h : 32 * h);
#pragma unroll
                    for (int r = 0; r < kR; r++) k[r] = kp[r * (BIG ? 32 : NT)];
                };
                auto mac = [&](cpair(&a)[kR], const uint32_t(&f)[32], int dd, const float4(&k)[kR]) {
#pragma unroll
                    for (int r = 0; r < kR; r++) {
                        const float zr = __uint_as_float(f[4 * r + dd]), zi = __uint_as_float(f[4 * r + 2 + dd]);
                        const float2 kr = make_float2(k[r].x, k[r].y), ki = make_float2(k[r].z, k[r].w);
                        a[r].re = fma2(bc2(zr), kr, a[r].re);
                        a[r].im = fma2(bc2(zr), ki, a[r].im);
                        a[r].re = fma2(bc2(-zi), ki, a[r].re);
                        a[r].im = fma2(bc2(zi), kr, a[r].im);
                    }
                };
                auto ring_at = [&](int s) { return smem + Lay::ring + (size_t)s * Lay::unit; };
                uint32_t f0[32], f1[32];
                float4 ka[kR], kb[kR];
                int slot = Lay::slot(step, v * L);
                const uint32_t phase = Lay::phase(step, v * L);
                tmem_ld32(tmem, f0);
                tmem_ld32(tmem + 32u, f1);
                wait_bounded(full_bar(slot), phase, abort_flag, args.timeout_ns, args.err);
                __syncwarp();
                load(ka, ring_at(slot), 0, 0);
                tmem_wait_ld32(f0);
                tmem_tie32(f1);
#pragma unroll 1
                for (int d = 0; d < KPL; d += 2) {
                    const bool more = d + 2 < KPL;
                    const unsigned char *at = ring_at(slot);
                    load(kb, at, 0, 1);
                    mac(acc[0], f0, 0, ka);
                    load(ka, at, 1, 0);
                    const bool ready = more && mbar_test_wait(full_bar(slot + 1), phase);
                    mac(acc[0], f0, 1, kb);
                    load(kb, at, 1, 1);
                    if (more) tmem_ld32(tmem + (uint32_t)(32 * d + 64), f0);
                    mac(acc[1], f1, 0, ka);
                    if (more) {
                        if (!ready) wait_bounded(full_bar(slot + 1), phase, abort_flag, args.timeout_ns, args.err);
                        __syncwarp();
                        load(ka, at + Lay::unit, 0, 0);
                    }
                    mac(acc[1], f1, 1, kb);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(empty_bar(slot));
                    slot++;
                    if (more) {
                        tmem_ld32(tmem + (uint32_t)(32 * d + 96), f1);
                        tmem_wait_ld32(f0);
                        tmem_tie32(f1);
                    }
                }
                F::inverse(acc, exch, s_tab, s_mid, lane, half);
                uint32_t *poly = s_acc + v * N + 1024 * half + lane;
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int r = 0; r < kR; r++) {  // (c_j - i c_{j+M}) of each limb, the high limb weighted 2^S
                        const int j = 32 * h + 64 * r;
                        poly[j] += ((uint32_t)__float2ll_rn(acc[h][r].re.x) << split_shift) + (uint32_t)__float2ll_rn(acc[h][r].re.y);
                        poly[j + 512] +=
                            ((uint32_t)__float2ll_rn(-acc[h][r].im.x) << split_shift) + (uint32_t)__float2ll_rn(-acc[h][r].im.y);
                    }
            }
        } else {
            // 2. per digit: forward transform, then its products with the key row, added to both outputs'
            //    accumulators in TMEM (with the 64 registers of a transform, 128 more for accumulators
            //    would not fit); they start at zero
            const uint32_t sums = tmem + (uint32_t)(128 * role);
            {
                const uint32_t zero[32] = {};
#pragma unroll
                for (int q = 0; q < 4; q++) tmem_st32p(sums + (uint32_t)(32 * q), zero);
            }
#pragma unroll 1
            for (int d = role * L; d < (DUO ? (role + 1) * L : KPL); d++) {
                const int u = d / L, sh = 32 - (d - u * L + 1) * Bgbit;
                // the masked word under the exponent of 2^52 is 1.5 * 2^52 + digit * 2^sh, as in the split form
                const uint32_t mask = maskBg << sh;
                const double scale = __hiloint2double((1023 - sh) << 20, 0);
                const double bias = 6755399441055744.0 * scale + double(1 << (Bgbit - 1));
                uint32_t x[32];
                tmem_ld32(tmem + Lay::col_xr + (uint32_t)(32 * u), x);
                tmem_wait_ld32(x);
                cplx<double> z[2][kR];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int r = 0; r < kR; r++) {  // j = lane + 32 (h + 2 r); j + M is word 16 on
                        const double lo = __hiloint2double(0x43380000, (int)(x[h + 2 * r] & mask));
                        const double hi = __hiloint2double(0x43380000, (int)(x[h + 2 * r + 16] & mask));
                        z[h][r] = {fma(lo, scale, -bias), fma(-hi, scale, bias)};
                    }
                F::forward(z, exch, s_tab, lane, half);
                const int slot = Lay::slot(step, d);
                wait_bounded(full_bar(slot), Lay::phase(step, d), abort_flag, args.timeout_ns, args.err);
                __syncwarp();
                const double2 *kp = reinterpret_cast<const double2 *>(smem + Lay::ring + (size_t)slot * Lay::unit) + lane + 512 * half;
                // quarters (output v, butterfly h), the next one's accumulators loading meanwhile, and its keys (9.93
                // against 10.15 ms per 1184 bootstraps; at l = 2, one warp per bootstrap, 5.86 against 5.83)
                constexpr bool AHEAD = L == 3 || DUO;
                auto key = [&](int q, int r) {
                    return BIG ? kp[1024 * (q >> 1) + 256 * (q & 1) + 32 * r] : kp[((q >> 1) * kR + r) * NT + 32 * (q & 1)];
                };
                uint32_t a[2][32];
                double2 kk[2][kR];
                tmem_ld32(sums, a[0]);
                if (AHEAD)
#pragma unroll
                    for (int r = 0; r < kR; r++) kk[0][r] = key(0, r);
                tmem_wait_ld32(a[0]);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    uint32_t *acc = a[q & 1];
                    if (q < 3) tmem_ld32(sums + (uint32_t)(32 * q + 32), a[(q + 1) & 1]);
                    if (AHEAD && q < 3)
#pragma unroll
                        for (int r = 0; r < kR; r++) kk[(q + 1) & 1][r] = key(q + 1, r);
                    uint32_t w[32];
#pragma unroll
                    for (int r = 0; r < kR; r++) {
                        const double2 k = AHEAD ? kk[q & 1][r] : key(q, r);
                        cplx<double> p;
                        F::get(p, acc, 4 * r, 4 * r + 2);
                        cmac(p, z[q & 1][r], cplx<double>{k.x, k.y});
                        F::put(w, 4 * r, 4 * r + 2, p);
                    }
                    tmem_st32p(sums + (uint32_t)(32 * q), w);
                    if (q < 3) tmem_wait_ld32(a[(q + 1) & 1]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty_bar(slot));
                tmem_wait_st();
            }
            // 3. per output polynomial: inverse transform, exact rounding, accumulate
            duo_sync();
#pragma unroll 1
            for (int v = role; v < (DUO ? role + 1 : KP1); v++) {
                uint32_t a[64];
                tmem_ld32(sums + (uint32_t)(64 * v), a);
                tmem_ld32(sums + (uint32_t)(64 * v + 32), a + 32);
                tmem_wait_ld64(a);
                cplx<double> z[2][kR];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int r = 0; r < kR; r++) F::get(z[h][r], a, 32 * h + 4 * r, 32 * h + 4 * r + 2);
                if constexpr (DUO) {  // the other warp's part; its next step's zeros wait for these loads
                    uint32_t b[64];
                    tmem_ld32(tmem + (uint32_t)(128 * (role ^ 1) + 64 * v), b);
                    tmem_ld32(tmem + (uint32_t)(128 * (role ^ 1) + 64 * v + 32), b + 32);
                    tmem_wait_ld64(b);
                    duo_sync();
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int r = 0; r < kR; r++) {
                            cplx<double> p;
                            F::get(p, b, 32 * h + 4 * r, 32 * h + 4 * r + 2);
                            z[h][r] = cadd(z[h][r], p);
                        }
                }
                F::inverse(z, exch, s_tab, s_mid, lane, half);
                uint32_t *poly = s_acc + v * N + 1024 * half + lane;
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int r = 0; r < kR; r++) {  // (c_j - i c_{j+M})
                        const int j = 32 * h + 64 * r;
                        poly[j] += round_f64_mod32(z[h][r].re);
                        poly[j + 512] += round_f64_mod32(-z[h][r].im);
                    }
            }
        }
        if constexpr (BIG) team_sync(2 + team, 64);  // the other warp rotates these words too
        else __syncwarp();
    }

    uint32_t *dst = reinterpret_cast<uint32_t *>(args.acc_out) + (size_t)boot * KP1 * N;
    if constexpr (BIG) {
        for (int i = first; i < KP1 * N; i += stride) dst[i] = s_acc[place(i)];
    } else {
        for (int i = lane + role * N; i < (DUO ? (role + 1) * N : KP1 * N); i += 32) dst[i] = s_acc[i];
    }

    // every consumer's TMEM accesses are complete; warp 0 frees the columns
    tmem_fence_before_sync();
    team_sync(1, active * (DUO || BIG ? 64 : 32));
    tmem_fence_after_sync();
    __syncwarp();
    if (warp == 0) tmem_free(tmem_base, 512);
}

template <bool SPLIT, int L, int G, int D, WarpMode MODE>
static cudaError_t launch_warp_impl(const BrArgs &args, cudaStream_t s) {
    using Lay = WarpLayout<SPLIT, L, D, MODE>;
    static_assert(G <= Lay::teams, "one warp per bootstrap, or two");
    if ((SPLIT || Lay::big) && !args.bsk2) return cudaErrorInvalidValue;
    if (SPLIT && !Lay::big && L * args.Bgbit > kDigitBits) return cudaErrorInvalidValue;
    auto kern = blind_rotate_warp_kernel<SPLIT, L, D, MODE>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Lay::bytes(Lay::teams));
    if (e != cudaSuccess) return e;
    BrArgs a = args;
    a.teams = G;
    kern<<<(a.boots + G - 1) / G, 32 * (kWarpTeams + 4), Lay::bytes(G), s>>>(a);
    return cudaGetLastError();
}
template <bool SPLIT, int L, int G, int D>
cudaError_t launch_warp(const BrArgs &a, cudaStream_t s) {
    return launch_warp_impl<SPLIT, L, G, D, WarpMode::solo>(a, s);
}
template <bool SPLIT, int L, int G, int D>
cudaError_t launch_warp_duo(const BrArgs &a, cudaStream_t s) {
    return launch_warp_impl<SPLIT, L, G, D, WarpMode::duo>(a, s);
}
template <bool SPLIT, int L, int G>
cudaError_t launch_warp_big(const BrArgs &a, cudaStream_t s) {
    return launch_warp_impl<SPLIT, L, G, L, WarpMode::big>(a, s);
}

template cudaError_t launch_warp<true, 3, 8, 6>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp<false, 3, 8, 6>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp<true, 2, 8, 8>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp<false, 2, 8, 8>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp_duo<true, 3, 4, 6>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp_duo<true, 3, 3, 6>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp_duo<false, 3, 4, 6>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp_duo<false, 3, 3, 6>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp_duo<true, 2, 4, 8>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp_duo<false, 2, 4, 8>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp_big<true, 3, 4>(const BrArgs &, cudaStream_t);
template cudaError_t launch_warp_big<false, 3, 4>(const BrArgs &, cudaStream_t);

}  // namespace tfheb
