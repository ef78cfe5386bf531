// fft_fx.cuh -- the FP64 form's transforms, in 64-bit block floating point on the integer units.
//
// One FP64 instruction holds its SMSP's FP64 pipe for 64 cycles a warp on this chip (measured: DADD,
// DFMA and the double <-> integer conversions alike), a 64-bit integer addition 2.2 and a
// 32 x 32 -> 64 multiply-add about 4-5.  A radix-8 butterfly with its twiddles is some 84 FP64
// instructions (5400 cycles) or about 650 cycles of integer instructions, so the transforms take
// each row's values as 64-bit integers q on one exponent, value = q 2^e:
//   * the exponent comes from the row's largest component (a maximum over the row's threads), so
//     that it fills 59 bits; a double's 53 bits are kept whole down to 2^-5 of the row's largest
//     value, and below that to 2^-59 of it;
//   * a twiddle is a 62-bit fraction in two balanced 32-bit halves; a complex product is twelve
//     32 x 32 -> 64 multiply-adds (the low x low parts, below the last bit, are left out) and is
//     rounded once;
//   * every intermediate value of a transform is a sum of rotated inputs, so its modulus is at most
//     the smaller of (inputs combined so far) x (largest) and the row's sum of moduli.  Before a
//     stage the row is shifted down by what that bound needs to stay below 2^62 -- three bits a
//     radix-8 stage for a flat row, none for a row with one large value -- with rounding.
// The error relative to the row's result is that of the FP64 stages or less: a flat row keeps some
// 60 significant bits of its largest result, FP64 53 (measured against 64-bit transforms in
// extended precision over the row shapes of the solver: tests/test_fx_algorithm.py).
// Measured (GB300, 1024^2, ns = 256, the coupled FP64 step): k_nl_y 325 -> 181 us, k_press_x 334 -> 153,
// k_press_y 145 -> 70, k_nl_x's advection part 148 -> 62, the step 1142 -> 601; at 256^2 the step
// 323 -> 256 us.
// A row whose largest value is not finite or above 2^1006 comes out as NaN; values below 2^-980
// lose digits and those below 2^-989 count as zero.
#pragma once
#include "common.cuh"

namespace fsibe {

struct __align__(16) q2 { long long x, y; };
static_assert(sizeof(q2) == sizeof(double2), "a fixed-point value takes its double's place in the row buffers");

// bits of the largest input component of a transform (FX_BITS) and of a half spectrum before its merge
// (FX_BITS_C; the merge adds two bits of modulus, and the sums are known before the first stage)
constexpr int FX_BITS = 59, FX_BITS_C = 60;
constexpr int FX_LIM = 62;    // the moduli stay below 2^62.5, so that sums of two components fit
constexpr unsigned FX_EMIN = 96, FX_EMAX = 1023 + 1006;

__device__ __forceinline__ long long fx_wide(int a, int b, long long c) {
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
__device__ __forceinline__ int fx_lo(long long a) { return (int)a; }
__device__ __forceinline__ int fx_hi(long long a) { return (int)(a >> 32) + (int)((unsigned)(int)a >> 31); }  // balanced
// (hi 2^64 + cross 2^32) / 2^62, the cross products already carrying the rounding constant 2^29
__device__ __forceinline__ long long fx_fold(long long hi, long long cross) {
    const unsigned c = (unsigned)cross, l = (unsigned)hi, h = (unsigned)(hi >> 32);
    return (long long)(((unsigned long long)__funnelshift_l(l, h, 2) << 32) | __funnelshift_l(c, l, 2));
}
constexpr long long FX_HALF = 1LL << 29;

// a (c + i s), the halves of c and s in w = (c hi, c lo, s hi, s lo)
__device__ __forceinline__ q2 fx_cmul(q2 a, int4 w) {
    const int xl = fx_lo(a.x), xh = fx_hi(a.x), yl = fx_lo(a.y), yh = fx_hi(a.y);
    const int nh = -w.z, nl = -w.w;
    const long long cr = fx_wide(xh, w.y, fx_wide(xl, w.x, fx_wide(yh, nl, fx_wide(yl, nh, FX_HALF))));
    const long long ci = fx_wide(xh, w.w, fx_wide(xl, w.z, fx_wide(yh, w.y, fx_wide(yl, w.x, FX_HALF))));
    const long long hr = fx_wide(xh, w.x, fx_wide(yh, nh, (long long)(int)(cr >> 32)));
    const long long hi = fx_wide(xh, w.z, fx_wide(yh, w.x, (long long)(int)(ci >> 32)));
    q2 r;
    r.x = fx_fold(hr, cr);
    r.y = fx_fold(hi, ci);
    return r;
}
// a / sqrt 2
__device__ __forceinline__ long long fx_mulh(long long a) {
    // round(2^62 / sqrt 2) in balanced halves
    constexpr int HH = 759250125, HL = -25716447;
    const int l = fx_lo(a), h = fx_hi(a);
    const long long c = fx_wide(h, HL, fx_wide(l, HH, FX_HALF));
    return fx_fold(fx_wide(h, HH, (long long)(int)(c >> 32)), c);
}
__device__ __forceinline__ q2 fx_add(q2 a, q2 b) { q2 r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
__device__ __forceinline__ q2 fx_sub(q2 a, q2 b) { q2 r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
// i a (INV) or -i a
template <bool INV> __device__ __forceinline__ q2 fx_rot(q2 a) {
    q2 r;
    r.x = INV ? -a.y : a.y;
    r.y = INV ? a.x : -a.x;
    return r;
}
// a / 2^s to nearest (s > 0, half = 2^(s-1)), a tie away from zero: an odd function, so that a field
// with a mirror symmetry keeps it in every bit (a pressure difference across a symmetric body is
// then as exact as in FP64, where it is what is left of values 10^7 times as large)
__device__ __forceinline__ long long fx_shr(long long a, int s, int half) {
    return (a + (unsigned)(half + (int)(a >> 63))) >> s;
}

template <bool INV> __device__ __forceinline__ void fx_dft2(q2* v) {
    const q2 a = v[0];
    v[0] = fx_add(a, v[1]);
    v[1] = fx_sub(a, v[1]);
}
template <bool INV> __device__ __forceinline__ void fx_dft4(q2* v) {
    const q2 a = fx_add(v[0], v[2]), b = fx_sub(v[0], v[2]);
    const q2 c = fx_add(v[1], v[3]), d = fx_rot<INV>(fx_sub(v[1], v[3]));
    v[0] = fx_add(a, c);
    v[2] = fx_sub(a, c);
    v[1] = fx_add(b, d);
    v[3] = fx_sub(b, d);
}
template <bool INV> __device__ __forceinline__ void fx_dft8(q2* v) {
    q2 e[4], o[4];
    e[0] = fx_add(v[0], v[4]); o[0] = fx_sub(v[0], v[4]);
    e[1] = fx_add(v[1], v[5]); const q2 t1 = fx_sub(v[1], v[5]);
    e[2] = fx_add(v[2], v[6]); o[2] = fx_rot<INV>(fx_sub(v[2], v[6]));
    e[3] = fx_add(v[3], v[7]); const q2 t3 = fx_sub(v[3], v[7]);
    if (!INV) {  // (1 - i)/sqrt 2, (-1 - i)/sqrt 2
        o[1].x = fx_mulh(t1.x + t1.y); o[1].y = fx_mulh(t1.y - t1.x);
        o[3].x = fx_mulh(t3.y - t3.x); o[3].y = -fx_mulh(t3.x + t3.y);
    } else {     // (1 + i)/sqrt 2, (-1 + i)/sqrt 2
        o[1].x = fx_mulh(t1.x - t1.y); o[1].y = fx_mulh(t1.x + t1.y);
        o[3].x = -fx_mulh(t3.x + t3.y); o[3].y = fx_mulh(t3.x - t3.y);
    }
    fx_dft4<INV>(e);
    fx_dft4<INV>(o);
    v[0] = e[0]; v[2] = e[1]; v[4] = e[2]; v[6] = e[3];
    v[1] = o[0]; v[3] = o[1]; v[5] = o[2]; v[7] = o[3];
}
template <int P, bool INV> __device__ __forceinline__ void fx_dftp(q2* v) {
    if constexpr (P == 8) fx_dft8<INV>(v);
    else if constexpr (P == 4) fx_dft4<INV>(v);
    else fx_dft2<INV>(v);
}

// ---- doubles to and from a row's scale ----------------------------------------------------
// the high word without the sign: monotonic in the magnitude, its exponent field in bits 20..30
__device__ __forceinline__ unsigned fx_mag(double d) { return (unsigned)__double2hiint(d) & 0x7fffffffu; }
// d on the scale where the exponent field em fills BITS bits, rounded to nearest
template <int BITS> __device__ __forceinline__ long long fx_from(double d, unsigned em) {
    const int hi = __double2hiint(d);
    const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
    const unsigned s = min(em - e, 63u);
    const unsigned long long m = (((unsigned long long)(((unsigned)hi & 0xfffffu) | 0x100000u)) << 32) | (unsigned)__double2loint(d);
    const long long v = (long long)((((m << (BITS - 53 + 1)) >> s) + 1) >> 1);
    const long long g = (long long)(hi >> 31);
    return (v ^ g) - g;
}
// q 2^e as a double (rounded to nearest), eb = e + 63 + 1022 (above zero for every scale); a row
// that was not finite has nan = the exponent and quiet bits
__device__ __forceinline__ double fx_to(long long q, int eb, unsigned nan) {
    const long long g = q >> 63;
    const unsigned long long m = (unsigned long long)((q ^ g) - g);
    const int lz = __clzll((long long)m);
    const unsigned long long n = m << (lz & 63);
    // the mantissa with its leading bit, which adds one to the exponent field
    const unsigned long long b = (n >> 11) + ((n >> 10) & 1ull) + ((unsigned long long)(unsigned)(eb - lz) << 52);
    const unsigned hi = (m == 0 ? 0u : (unsigned)(b >> 32)) | nan | ((unsigned)(g >> 32) & 0x80000000u);
    return __hiloint2double((int)hi, m == 0 ? 0 : (int)(unsigned)b);
}

// ---- reductions over the threads of a row ----------------------------------------------------
// A row's G threads are part of one warp (G <= 32; the rows of a warp then share one scale) or
// whole warps.  The lanes' maxima (sums) of NB values, over the row's warps; with G > 32 the
// partials go through slots (the caller synchronises before fx_row_read).
template <int G> __device__ __forceinline__ unsigned fx_lanes() {
    return blockDim.x >= 32 ? 0xffffffffu : (1u << blockDim.x) - 1u;
}
template <int G, int NB, bool SUM>
__device__ __forceinline__ void fx_row_reduce(unsigned (&m)[NB], unsigned (*slot)[32]) {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        m[b] = SUM ? __reduce_add_sync(fx_lanes<G>(), m[b]) : __reduce_max_sync(fx_lanes<G>(), m[b]);
        if (G > 32 && (threadIdx.x & 31) == 0) slot[b][threadIdx.x >> 5] = m[b];
    }
}
template <int G, int NB, bool SUM>
__device__ __forceinline__ void fx_row_read(unsigned (&m)[NB], const unsigned (*slot)[32]) {
    if constexpr (G > 32) {
        constexpr int NW = G / 32;
        const int w0 = (threadIdx.x >> 5) & ~(NW - 1);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            unsigned r = slot[b][w0];
#pragma unroll
            for (int w = 1; w < NW; ++w) r = SUM ? r + slot[b][w0 + w] : max(r, slot[b][w0 + w]);
            m[b] = r;
        }
    }
}
// The scale of a row from its largest high word: the exponent field that fills its bits, and
// the NaN bits of a row out of range.
__device__ __forceinline__ unsigned fx_scale(unsigned hi, unsigned& nan) {
    const unsigned e = hi >> 20;
    nan = e > FX_EMAX ? 0x7ff80000u : 0u;
    return min(max(e, FX_EMIN), 2046u);
}
// |a| in units of 2^44, rounded up
__device__ __forceinline__ unsigned fx_l1(long long a) { return (unsigned)abs((int)(a >> 44)) + 1u; }
__device__ __forceinline__ int fx_bitlen(unsigned a) { return 32 - __clz((int)a); }
// bits a row is shifted down by before the stage after which 2^g inputs are combined
__device__ __forceinline__ int fx_down(int b0, int g, int lb) { return max(min(b0 + g, lb) - FX_LIM, 0); }

// ---- the stages ------------------------------------------------------------------------------
__device__ __forceinline__ q2 fx_ldrow(const double2* b) { return *reinterpret_cast<const q2*>(b); }
__device__ __forceinline__ void fx_strow(double2* b, q2 v) { *reinterpret_cast<q2*>(b) = v; }

// shift, twiddle and butterflies of one stage (radix P, 2^lg = the product of the radices already
// applied) on v[b][q P + r] (input r of butterfly q)
template <int N, int P, bool INV, bool TWID, int NB>
__device__ __forceinline__ void fx_compute(q2 (&v)[NB][8], const int4* __restrict__ tw, int t, int lg, const int (&sh)[NB]) {
    constexpr int G = N / 8, PER = 8 / P;
#pragma unroll
    for (int b = 0; b < NB; ++b)
        if (sh[b] > 0) {  // the same for the whole warp
            const int half = (1 << sh[b]) >> 1;
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                v[b][m].x = fx_shr(v[b][m].x, sh[b], half);
                v[b][m].y = fx_shr(v[b][m].y, sh[b], half);
            }
        }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int k = (t + q * G) & ((1 << lg) - 1);
#pragma unroll
        for (int r = 1; r < P; ++r) {
            if (!TWID) continue;
            int4 w = __ldg(&tw[(r * k * (N / P)) >> lg]);
            if (INV) { w.z = -w.z; w.w = -w.w; }
#pragma unroll
            for (int b = 0; b < NB; ++b) v[b][q * P + r] = fx_cmul(v[b][q * P + r], w);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) fx_dftp<P, INV>(v[b] + q * P);
    }
}

// NB transforms of q values in registers, v[b][m] = element t + m G with moduli below 2^(B0 + 1/2)
// (a component of B0 bits) and the
// row's sum of moduli in lsum (fx_l1's units); LATE: the sums of a row of several warps are still
// in their slots and are read after the first exchange's synchronisation.  Leaves the transformed
// elements in place and adds the shifts to e[b].
template <int N, bool INV, int NB, int B0, bool LATE>
__device__ __forceinline__ void fx_stages(q2 (&v)[NB][8], double2* buf, int bstride, const int4* __restrict__ tw, int t,
                                          unsigned (&lsum)[NB], const unsigned (*lslot)[32], int (&e)[NB]) {
    constexpr int G = N / 8;
    constexpr int LOGN = N == 16 ? 4 : N == 32 ? 5 : N == 64 ? 6 : N == 128 ? 7 : N == 256 ? 8 : N == 512 ? 9 : N == 1024 ? 10 : N == 2048 ? 11 : 12;
    static_assert((1 << LOGN) == N, "length");
    constexpr int LAST = LOGN % 3 == 0 ? 8 : (LOGN % 3 == 1 ? 2 : 4);
    int lb[NB], sh[NB], down[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        if (LATE) sh[b] = 0;  // the first stage fits (B0 + 3 <= FX_LIM)
        else { lb[b] = 44 + fx_bitlen(lsum[b]); sh[b] = fx_down(B0, 3, lb[b]); }
        down[b] = sh[b];
    }
    static_assert(!LATE || B0 + 3 <= FX_LIM, "first stage without the sums");
    fx_compute<N, 8, INV, false, NB>(v, tw, t, 0, sh);
    // the exchange after a radix-8 stage: outputs to their autosorted positions, then the next
    // stage's inputs (radix P2)
    auto exchange = [&](int ns, auto p2) {
        constexpr int P2 = decltype(p2)::value, PER2 = 8 / P2, B2 = N / P2;
        const int k = t & (ns - 1), base = (t - k) * 8 + k;
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int r = 0; r < 8; ++r) fx_strow(&buf[b * bstride + pad8(base + r * ns)], v[b][r]);
        __syncthreads();
        if (LATE && ns == 1) {
            fx_row_read<G, NB, true>(lsum, lslot);
#pragma unroll
            for (int b = 0; b < NB; ++b) lb[b] = 44 + fx_bitlen(lsum[b]);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int q = 0; q < PER2; ++q)
#pragma unroll
                for (int r = 0; r < P2; ++r) v[b][q * P2 + r] = fx_ldrow(&buf[b * bstride + pad8(t + q * G + r * B2)]);
        __syncthreads();  // every thread has its inputs before the buffer is written again
    };
    auto shifts = [&](int g) {
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const int d = fx_down(B0, g, lb[b]);
            sh[b] = d - down[b];
            down[b] = d;
        }
    };
    int ns = 1, g = 3;
    if constexpr (N >= 64) {
        // the further radix-8 stages share one body (the code is long: one copy stays in the
        // instruction cache)
#pragma unroll 1
        for (; ns * 64 <= N; ns *= 8) {
            exchange(ns, std::integral_constant<int, 8>{});
            shifts(g + 3);
            fx_compute<N, 8, INV, true, NB>(v, tw, t, g, sh);
            g += 3;
        }
    }
    if constexpr (LAST != 8) {
        exchange(ns, std::integral_constant<int, LAST>{});
        shifts(LOGN);
        fx_compute<N, LAST, INV, true, NB>(v, tw, t, g, sh);
        // the last stage's butterfly q, output r is element t + (q + PER r) G: element order
        constexpr int PER = 8 / LAST;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            q2 o[8];
#pragma unroll
            for (int q = 0; q < PER; ++q)
#pragma unroll
                for (int r = 0; r < LAST; ++r) o[q + PER * r] = v[b][q * LAST + r];
#pragma unroll
            for (int m = 0; m < 8; ++m) v[b][m] = o[m];
        }
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) e[b] += down[b];
}

// doubles in registers to fixed point: the row's scale (one synchronisation when a row spans
// warps) and the partial sums of moduli
template <int G, int BITS, int NB>
__device__ __forceinline__ void fx_enter(const double2 (&v)[NB][8], q2 (&z)[NB][8], unsigned (*mslot)[32], unsigned (*lslot)[32],
                                         unsigned (&lsum)[NB], unsigned (&nan)[NB], int (&e)[NB]) {
    unsigned mx[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        mx[b] = 0;
#pragma unroll
        for (int m = 0; m < 8; ++m) mx[b] = max(mx[b], max(fx_mag(v[b][m].x), fx_mag(v[b][m].y)));
    }
    fx_row_reduce<G, NB, false>(mx, mslot);
    if (G > 32) __syncthreads();
    fx_row_read<G, NB, false>(mx, mslot);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const unsigned em = fx_scale(mx[b], nan[b]);
        e[b] = (int)em - 1022 - BITS;
        lsum[b] = 0;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            z[b][m].x = fx_from<BITS>(v[b][m].x, em);
            z[b][m].y = fx_from<BITS>(v[b][m].y, em);
            lsum[b] += fx_l1(z[b][m].x) + fx_l1(z[b][m].y);
        }
    }
    fx_row_reduce<G, NB, true>(lsum, lslot);
}

// NB transforms of doubles in registers (block_fft_reg_m's contract; all threads of the block
// call it): v[b][m] = element t + m (N/8), the rows of buf free when called and on return.  The
// result is scaled by 2^ex (the normalisation 1/(nx ny), a power of two, costs nothing here).
template <int N, bool INV, int NB, int NBA>
__device__ __forceinline__ void fx_fft_reg(double2 (&v)[NBA][8], double2* buf, int bstride, const int4* __restrict__ tw, int t,
                                           int ex) {
    constexpr int G = N / 8;
    __shared__ unsigned mslot[NB][32], lslot[NB][32];
    q2 z[NB][8];
    unsigned lsum[NB], nan[NB];
    int e[NB];
    {
        double2 w[NB][8];
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int m = 0; m < 8; ++m) w[b][m] = v[b][m];
        fx_enter<G, FX_BITS>(w, z, mslot, lslot, lsum, nan, e);
    }
    fx_stages<N, INV, NB, FX_BITS, true>(z, buf, bstride, tw, t, lsum, lslot, e);
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            v[b][m].x = fx_to(z[b][m].x, e[b] + ex + 63 + 1022, nan[b]);
            v[b][m].y = fx_to(z[b][m].y, e[b] + ex + 63 + 1022, nan[b]);
        }
}

// ---- real rows of 2H values as H complex ones (see r2c_split_m and c2r_merge_m) ---------------
// The pairs (k, H - k) of a thread: k = 1 + t + i G, i < 4; the last thread's last pair is
// (H/2, H/2), which it takes as the pair (0, H/2) of the two special elements.

// Half spectra of doubles in the row buffers to real rows in registers: v[b][m] = element
// t + m (H/8) (its x and y two neighbouring real values).  The rows are free on return.
template <int H, int NB, int NBA>
__device__ __forceinline__ void fx_c2r_reg(double2* rb, int bstride, const int4* __restrict__ twR, const int4* __restrict__ twX,
                                           int t, double2 (&v)[NBA][8]) {
    constexpr int G = H / 8;
    __shared__ unsigned mslot[NB][32], lslot[NB][32];
    q2 z[NB][8];
    unsigned lsum[NB], nan[NB];
    int e[NB];
    {
        double2 x[NB][8];
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int k = 1 + t + i * G;
                const bool sp = k == H / 2;
                x[b][2 * i] = rb[b * bstride + pad8(sp ? 0 : k)];
                x[b][2 * i + 1] = rb[b * bstride + pad8(H - k)];
                if (i == 3 && sp) x[b][2 * i].y = 0.0;  // the imaginary part of X[0] is ignored
            }
        fx_enter<G, FX_BITS_C>(x, z, mslot, lslot, lsum, nan, e);
    }
    // Z[k] = (X[k] + conj X[H-k]) + i (X[k] - conj X[H-k]) conj(w^k), and Z[H-k] likewise
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k = 1 + t + i * G;
        const bool sp = i == 3 && k == H / 2;
        const int4 wk = __ldg(&twR[k]);
        const int4 wm = make_int4(wk.x, wk.y, -wk.z, -wk.w);  // conj
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const q2 a = z[b][2 * i], c = z[b][2 * i + 1];
            q2 s, d;
            s.x = a.x + c.x; s.y = a.y - c.y;
            d.x = a.x - c.x; d.y = a.y + c.y;
            const q2 o = fx_cmul(d, wm);
            // w^(H-k) = -conj(w^k): Z[H-k] = conj(s - i o)
            q2 zk, zm;
            zk.x = s.x - o.y; zk.y = s.y + o.x;
            zm.x = s.x + o.y; zm.y = o.x - s.y;
            if (sp) {
                zk.x = a.x; zk.y = a.x;             // Z[0] = X[0] (1 + i)
                zm.x = 2 * c.x; zm.y = -2 * c.y;    // Z[H/2] = 2 conj X[H/2]
            }
            fx_strow(&rb[b * bstride + pad8(sp ? 0 : k)], zk);
            fx_strow(&rb[b * bstride + pad8(H - k)], zm);
        }
    }
    // |Z[k]|^2 + |Z[H-k]|^2 = 4 (|X[k]|^2 + |X[H-k]|^2), so the sum of the moduli grows by at most
    // 2 sqrt 2
    __syncthreads();
    fx_row_read<G, NB, true>(lsum, lslot);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        lsum[b] *= 3;
#pragma unroll
        for (int m = 0; m < 8; ++m) z[b][m] = fx_ldrow(&rb[b * bstride + pad8(t + m * G)]);
    }
    __syncthreads();
    fx_stages<H, true, NB, FX_BITS_C + 2, false>(z, rb, bstride, twX, t, lsum, lslot, e);
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            v[b][m].x = fx_to(z[b][m].x, e[b] + 63 + 1022, nan[b]);
            v[b][m].y = fx_to(z[b][m].y, e[b] + 63 + 1022, nan[b]);
        }
}

// Real rows in registers to half spectra of doubles in the row buffers (free when called; the
// caller reads them after this returns, synchronised).
template <int H, int NB, int NBA>
__device__ __forceinline__ void fx_r2c_reg(double2 (&v)[NBA][8], double2* rb, int bstride, const int4* __restrict__ twR,
                                           const int4* __restrict__ twX, int t) {
    constexpr int G = H / 8;
    __shared__ unsigned mslot[NB][32], lslot[NB][32];
    q2 z[NB][8];
    unsigned lsum[NB], nan[NB];
    int e[NB];
    {
        double2 w[NB][8];
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int m = 0; m < 8; ++m) w[b][m] = v[b][m];
        fx_enter<G, FX_BITS>(w, z, mslot, lslot, lsum, nan, e);
    }
    fx_stages<H, false, NB, FX_BITS, true>(z, rb, bstride, twX, t, lsum, lslot, e);
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            // halves, for the split's sums
            q2 h;
            h.x = fx_shr(z[b][m].x, 1, 1);
            h.y = fx_shr(z[b][m].y, 1, 1);
            fx_strow(&rb[b * bstride + pad8(t + m * G)], h);
        }
    __syncthreads();
    // X[k] = (z[k] + conj z[H-k])/2 + w^k (z[k] - conj z[H-k])/(2i), and X[H-k] likewise
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k = 1 + t + i * G;
        const bool sp = i == 3 && k == H / 2;
        const int4 wk = __ldg(&twR[k]);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            double2* pk = &rb[b * bstride + pad8(sp ? 0 : k)];
            double2* pm = &rb[b * bstride + pad8(H - k)];
            const q2 a = fx_ldrow(pk), c = fx_ldrow(pm);
            q2 s, d;
            s.x = a.x + c.x; s.y = a.y - c.y;
            d.x = a.y + c.y; d.y = c.x - a.x;       // (z[k] - conj z[H-k]) / i
            const q2 o = fx_cmul(d, wk);
            q2 xk = fx_add(s, o), xm;
            xm.x = s.x - o.x; xm.y = o.y - s.y;     // conj(s - o): w^(H-k) = -conj(w^k)
            if (sp) {
                xk.x = 2 * (a.x + a.y); xk.y = 0;   // X[0] = Re z[0] + Im z[0]
                xm.x = 2 * c.x; xm.y = -2 * c.y;    // X[H/2] = conj z[H/2]
            }
            const int eb = e[b] + 63 + 1022;
            *pk = make_double2(fx_to(xk.x, eb, nan[b]), sp ? 0.0 : fx_to(xk.y, eb, nan[b]));
            *pm = make_double2(fx_to(xm.x, eb, nan[b]), fx_to(xm.y, eb, nan[b]));
        }
    }
    __syncthreads();
}

}  // namespace fsibe
