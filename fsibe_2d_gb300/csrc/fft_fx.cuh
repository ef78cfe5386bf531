// fft_fx.cuh -- the FP64 form's transforms, in 64-bit block floating point on the integer units.
//
// One FP64 instruction holds its SMSP's FP64 pipe for 64 cycles a warp on this chip (measured: DADD,
// DFMA and the double <-> integer conversions alike), a 64-bit integer addition 2.2 and a
// 32 x 32 -> 64 multiply-add about 4-5.  A radix-8 butterfly with its twiddles is some 84 FP64
// instructions (5400 cycles) or about 650 cycles of integer instructions, so the transforms take
// each row's values as 64-bit integers q on one exponent, value = q 2^e:
//   * the exponent comes from the row's largest component (a maximum over the row's threads), so
//     that it fills 59 bits; a double's 53 bits are kept whole down to 2^-6 of the row's largest
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
// It holds relative to the row, not element by element: where a row's large part cancels exactly (equal
// values at every second place, say) and its small part does not, FP64 gives the small part's
// modes to 53 bits of their own and this to some 2^-59 of the large part's (256 values, ones and 10^-12
// noise in turn: 2^-59.2 at most).
// Measured (GB300, 1024^2, ns = 256, the coupled FP64 step; the transforms alone): k_nl_y 325 -> 181 us,
// k_press_x 334 -> 153, k_press_y 145 -> 70, k_nl_x's advection part 148 -> 62, the step 1142 -> 601, at 256^2
// 323 -> 256; with the pointwise work off the FP64 pipe as well (over_k2) 533 and 232 us a step, and
// with a group of threads a transform (fluid_fx.cuh) 447 and 165.  What bounds the kernels then
// (1024^2): k_nl_y's ALU pipe is busy 44% of the time, the FP64 pipe 29%, with 28 warps an SM that wait
// at their barriers and on those two; k_press_x 35% and 34%.
// Range.  The transforms that take or give a caller's arrays (WIDE) take every finite row: one whose largest
// value is below 2^-927 is scaled up by a power of two as it enters, and results near the ends of the
// exponent range are scaled as they leave (to zero, a denormal or infinity, rounded as any FP64 result).
// The time step's and the adjoint's kernels leave both out (with them the 256^2 step took 1% longer, the
// 512^2 gradient 2%): of a row below 2^-927 they hold no digits below 2^-985, and one above
// 2^1006, whose square no double holds, comes out as NaN, as does any row with a value that is not
// finite.
#pragma once
#include "common.cuh"

namespace fsibe {

struct __align__(16) q2 { long long x, y; };
static_assert(sizeof(q2) == sizeof(double2), "a fixed-point value takes its double's place in the row buffers");

// bits of the largest input component of a transform (FX_BITS) and of a half spectrum before its merge
// (FX_BITS_C; the merge adds two bits of modulus, and the sums are known before the first stage)
constexpr int FX_BITS = 59, FX_BITS_C = 60;
constexpr int FX_LIM = 62;    // the moduli stay below 2^62.5, so that sums of two components fit
// Exponent fields: the scales of a row whose elements and results are formed without the powers of two of
// WIDE, and the range in which fx_to forms every result itself.
constexpr unsigned FX_EMIN = 96, FX_EMAX = 1023 + 1006;
constexpr int FX_EB_MIN = 64, FX_EB_MAX = 2045;

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
// q 2^e as a double (rounded to nearest), eb = e + 63 + 1022 in [FX_EB_MIN, FX_EB_MAX]; a row that was
// not finite has nan = the exponent and quiet bits
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

// ---- the threads of one transform -----------------------------------------------------------
// A transform of N points is the work of G = N/8 threads: part of a warp, or whole warps with a
// named barrier of their own (id, from 1 on), so that the transforms of a block do not wait on one
// another.  slot: G/32 words of shared memory of the group's own, twice (largest values, sums).
struct FxGroup {
    int t, id;        // thread of the group; its barrier
    unsigned* slot;
};
// the group of the calling thread in a block whose groups are one row each (t: thread of the row)
template <int G> __device__ __forceinline__ FxGroup fx_block_group(int t) {
    __shared__ unsigned slots[64];  // 1024 threads' warps, twice
    const int g = threadIdx.x / G;
    return FxGroup{t, g + 1, slots + g * 2 * (G / 32)};
}
template <int G> __device__ __forceinline__ unsigned fx_mask() {
    return G >= 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) & ~(G - 1));
}
template <int G> __device__ __forceinline__ void fx_sync(const FxGroup& g) {
    if constexpr (G > 32) asm volatile("bar.sync %0, %1;" ::"r"(g.id), "n"(G) : "memory");
    else __syncwarp(fx_mask<G>());
}
// the group's largest value (sum) of m; with G > 32 the warps' go to slots, read after a fx_sync
template <int G, bool SUM> __device__ __forceinline__ unsigned fx_reduce(unsigned m, unsigned* slot) {
    if constexpr (G >= 32) {
        m = SUM ? __reduce_add_sync(0xffffffffu, m) : __reduce_max_sync(0xffffffffu, m);
        if (G > 32 && (threadIdx.x & 31) == 0) slot[(threadIdx.x >> 5) & (G / 32 - 1)] = m;
    } else {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            const unsigned x = __shfl_xor_sync(fx_mask<G>(), m, o);
            m = SUM ? m + x : max(m, x);
        }
    }
    return m;
}
template <int G, bool SUM> __device__ __forceinline__ unsigned fx_read(unsigned m, const unsigned* slot) {
    if constexpr (G > 32) {
        m = slot[0];
#pragma unroll
        for (int w = 1; w < G / 32; ++w) m = SUM ? m + slot[w] : max(m, slot[w]);
    }
    return m;
}
// The scale of a row from its largest high word: the exponent field that fills its bits, and
// the NaN bits of a row out of range.
template <bool WIDE> __device__ __forceinline__ unsigned fx_scale(unsigned hi, unsigned& nan) {
    const unsigned e = hi >> 20;
    nan = e > (WIDE ? 2046u : FX_EMAX) ? 0x7ff80000u : 0u;
    return min(max(e, WIDE ? 1u : FX_EMIN), 2046u);
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
// applied) on v[q P + r] (input r of butterfly q)
template <int N, int P, bool INV, bool TWID>
__device__ __forceinline__ void fx_compute(q2 (&v)[8], const int4* __restrict__ tw, int t, int lg, int sh) {
    constexpr int G = N / 8, PER = 8 / P;
    if (sh > 0) {  // the same for the whole group
        const int half = (1 << sh) >> 1;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            v[m].x = fx_shr(v[m].x, sh, half);
            v[m].y = fx_shr(v[m].y, sh, half);
        }
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        if constexpr (TWID) {
            const int k = (t + q * G) & ((1 << lg) - 1);
#pragma unroll
            for (int r = 1; r < P; ++r) {
                int4 w = __ldg(&tw[(r * k * (N / P)) >> lg]);
                if (INV) { w.z = -w.z; w.w = -w.w; }
                v[q * P + r] = fx_cmul(v[q * P + r], w);
            }
        }
        fx_dftp<P, INV>(v + q * P);
    }
}

// The transform of q values in registers, v[m] = element t + m G with components of B0 bits (moduli
// below 2^(B0 + 1/2)) and the group's sum of moduli in lsum (fx_l1's units); LATE: the sum of a group
// of several warps is still in its slots and is read after the first exchange's synchronisation.
// Leaves the transformed elements in place and returns the bits shifted down.
template <int N, bool INV, int B0, bool LATE>
__device__ __forceinline__ int fx_stages(q2 (&v)[8], double2* buf, const int4* __restrict__ tw, const FxGroup& gr,
                                         unsigned lsum) {
    constexpr int G = N / 8;
    constexpr int LOGN = N == 16 ? 4 : N == 32 ? 5 : N == 64 ? 6 : N == 128 ? 7 : N == 256 ? 8 : N == 512 ? 9 : N == 1024 ? 10 : N == 2048 ? 11 : 12;
    static_assert((1 << LOGN) == N, "length");
    static_assert(!LATE || B0 + 3 <= FX_LIM, "first stage without the sum");
    constexpr int LAST = LOGN % 3 == 0 ? 8 : (LOGN % 3 == 1 ? 2 : 4);
    const int t = gr.t;
    int lb = 44 + fx_bitlen(lsum), down = LATE ? 0 : fx_down(B0, 3, lb);
    fx_compute<N, 8, INV, false>(v, tw, t, 0, down);
    // the exchange after a radix-8 stage: outputs to their autosorted positions, then the next
    // stage's inputs (radix P2)
    auto exchange = [&](int ns, auto p2) {
        constexpr int P2 = decltype(p2)::value, PER2 = 8 / P2, B2 = N / P2;
        const int k = t & (ns - 1), base = (t - k) * 8 + k;
#pragma unroll
        for (int r = 0; r < 8; ++r) fx_strow(&buf[pad8(base + r * ns)], v[r]);
        fx_sync<G>(gr);
        if (LATE && ns == 1) lb = 44 + fx_bitlen(fx_read<G, true>(lsum, gr.slot + G / 32));
#pragma unroll
        for (int q = 0; q < PER2; ++q)
#pragma unroll
            for (int r = 0; r < P2; ++r) v[q * P2 + r] = fx_ldrow(&buf[pad8(t + q * G + r * B2)]);
        fx_sync<G>(gr);  // every thread has its inputs before the row is written again
    };
    auto shift = [&](int g) {
        const int d = fx_down(B0, g, lb), sh = d - down;
        down = d;
        return sh;
    };
    int ns = 1, g = 3;
    if constexpr (N >= 64) {
        // the further radix-8 stages share one body (the code is long: one copy stays in the
        // instruction cache)
#pragma unroll 1
        for (; ns * 64 <= N; ns *= 8) {
            exchange(ns, std::integral_constant<int, 8>{});
            fx_compute<N, 8, INV, true>(v, tw, t, g, shift(g + 3));
            g += 3;
        }
    }
    if constexpr (LAST != 8) {
        exchange(ns, std::integral_constant<int, LAST>{});
        fx_compute<N, LAST, INV, true>(v, tw, t, g, shift(LOGN));
        // the last stage's butterfly q, output r is element t + (q + PER r) G: element order
        constexpr int PER = 8 / LAST;
        q2 o[8];
#pragma unroll
        for (int q = 0; q < PER; ++q)
#pragma unroll
            for (int r = 0; r < LAST; ++r) o[q + PER * r] = v[q * LAST + r];
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = o[m];
    }
    return down;
}

// doubles in registers to fixed point: the group's scale (one synchronisation when it spans
// warps), the exponent and the partial sum of moduli (complete for a group within a warp)
template <int G, int BITS, bool WIDE>
__device__ __forceinline__ int fx_enter(const double2 (&v)[8], q2 (&z)[8], const FxGroup& gr, unsigned& lsum, unsigned& nan) {
    unsigned mx = 0;
#pragma unroll
    for (int m = 0; m < 8; ++m) mx = max(mx, max(fx_mag(v[m].x), fx_mag(v[m].y)));
    mx = fx_reduce<G, false>(mx, gr.slot);
    if (G > 32) fx_sync<G>(gr);
    mx = fx_read<G, false>(mx, gr.slot);
    const unsigned em = fx_scale<WIDE>(mx, nan);
    if (!WIDE || em >= FX_EMIN) {  // the same for the whole group
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            z[m].x = fx_from<BITS>(v[m].x, em);
            z[m].y = fx_from<BITS>(v[m].y, em);
        }
    } else {
        // a row of zeros, or of the smallest scales
        unsigned any = 0;
#pragma unroll
        for (int m = 0; m < 8; ++m)
            any |= fx_mag(v[m].x) | fx_mag(v[m].y) | (unsigned)__double2loint(v[m].x) | (unsigned)__double2loint(v[m].y);
#pragma unroll
        for (int m = 0; m < 8; ++m) z[m].x = z[m].y = 0;
        if (any != 0) {
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                z[m].x = fx_from<BITS>(v[m].x * 0x1p128, em + 128);
                z[m].y = fx_from<BITS>(v[m].y * 0x1p128, em + 128);
            }
        }
    }
    lsum = 0;
#pragma unroll
    for (int m = 0; m < 8; ++m) lsum += fx_l1(z[m].x) + fx_l1(z[m].y);
    lsum = fx_reduce<G, true>(lsum, gr.slot + G / 32);
    return (int)em - 1022 - BITS;
}
// fixed point to doubles on the exponent e: fx_to's on one in its range, and with WIDE the power of two
// between (scale: 0 for none)
template <bool WIDE>
struct FxOut {
    int eb, scale = 0;
    unsigned nan;
    __device__ __forceinline__ FxOut(int e, unsigned nan_) : eb(e + 63 + 1022), nan(nan_) {
        if (WIDE) {
            const int b = eb;
            eb = min(max(b, FX_EB_MIN), FX_EB_MAX);
            scale = b - eb;
        }
    }
    __device__ __forceinline__ double2 operator()(q2 z) const { return make_double2(fx_to(z.x, eb, nan), fx_to(z.y, eb, nan)); }
    __device__ __forceinline__ double2 scaled(double2 v) const {  // (zeros stay out of the FP64 pipe)
        const double s = __hiloint2double((1023 + scale) << 20, 0);
        if (fx_mag(v.x) | fx_mag(v.y)) { v.x *= s; v.y *= s; }
        return v;
    }
};
template <bool WIDE>
__device__ __forceinline__ void fx_leave(const q2 (&z)[8], int e, unsigned nan, double2 (&v)[8]) {
    const FxOut<WIDE> out(e, nan);
#pragma unroll
    for (int m = 0; m < 8; ++m) v[m] = out(z[m]);
    if (WIDE && out.scale != 0) {
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = out.scaled(v[m]);
    }
}

// The transform of doubles in registers by one group: v[m] = element t + m (N/8); buf is the group's
// row, free when called and on return.  The result is scaled by 2^ex (the normalisation 1/(nx ny),
// a power of two, costs nothing here).
template <int N, bool INV, bool WIDE = false>
__device__ __forceinline__ void fx_fft(double2 (&v)[8], double2* buf, const int4* __restrict__ tw, const FxGroup& gr, int ex = 0) {
    q2 z[8];
    unsigned lsum, nan;
    int e = fx_enter<N / 8, FX_BITS, WIDE>(v, z, gr, lsum, nan);
    e += ex + fx_stages<N, INV, FX_BITS, true>(z, buf, tw, gr, lsum);
    fx_leave<WIDE>(z, e, nan, v);
}

// ---- real rows of 2H values as H complex ones (see r2c_split_m and c2r_merge_m) ---------------
// The pairs (k, H - k) of a thread: k = 1 + t + i G, i < 4; the last thread's last pair is
// (H/2, H/2), which it takes as the pair (0, H/2) of the two special elements.

// A half spectrum of doubles in the group's row (the group synchronised after it was written) to a
// real row in registers: v[m] = element t + m (H/8), its x and y two neighbouring real values.
// The row is free on return.
template <int H, bool WIDE = false>
__device__ __forceinline__ void fx_c2r(double2* rb, const int4* __restrict__ twR, const int4* __restrict__ twX,
                                       const FxGroup& gr, double2 (&v)[8]) {
    constexpr int G = H / 8;
    const int t = gr.t;
    q2 z[8];
    unsigned lsum, nan;
    int e;
    {
        double2 x[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = 1 + t + i * G;
            const bool sp = k == H / 2;
            x[2 * i] = rb[pad8(sp ? 0 : k)];
            x[2 * i + 1] = rb[pad8(H - k)];
            if (i == 3 && sp) x[2 * i].y = 0.0;  // the imaginary part of X[0] is ignored
        }
        e = fx_enter<G, FX_BITS_C, WIDE>(x, z, gr, lsum, nan);
    }
    // Z[k] = (X[k] + conj X[H-k]) + i (X[k] - conj X[H-k]) conj(w^k), and Z[H-k] likewise
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k = 1 + t + i * G;
        const bool sp = i == 3 && k == H / 2;
        const int4 wk = __ldg(&twR[k]);
        const q2 a = z[2 * i], c = z[2 * i + 1];
        q2 s, d;
        s.x = a.x + c.x; s.y = a.y - c.y;
        d.x = a.x - c.x; d.y = a.y + c.y;
        const q2 o = fx_cmul(d, make_int4(wk.x, wk.y, -wk.z, -wk.w));
        // w^(H-k) = -conj(w^k): Z[H-k] = conj(s - i o)
        q2 zk, zm;
        zk.x = s.x - o.y; zk.y = s.y + o.x;
        zm.x = s.x + o.y; zm.y = o.x - s.y;
        if (sp) {
            zk.x = a.x; zk.y = a.x;             // Z[0] = X[0] (1 + i)
            zm.x = 2 * c.x; zm.y = -2 * c.y;    // Z[H/2] = 2 conj X[H/2]
        }
        fx_strow(&rb[pad8(sp ? 0 : k)], zk);
        fx_strow(&rb[pad8(H - k)], zm);
    }
    fx_sync<G>(gr);
    // |Z[k]|^2 + |Z[H-k]|^2 = 4 (|X[k]|^2 + |X[H-k]|^2), so the sum of the moduli grows by at most
    // 2 sqrt 2
    lsum = 3 * fx_read<G, true>(lsum, gr.slot + G / 32);
#pragma unroll
    for (int m = 0; m < 8; ++m) z[m] = fx_ldrow(&rb[pad8(t + m * G)]);
    fx_sync<G>(gr);
    e += fx_stages<H, true, FX_BITS_C + 2, false>(z, rb, twX, gr, lsum);
    fx_leave<WIDE>(z, e, nan, v);
}

// A real row in registers to the half spectrum of doubles in the group's row (free when called;
// readers outside the group synchronise first).
template <int H, bool WIDE = false>
__device__ __forceinline__ void fx_r2c(const double2 (&v)[8], double2* rb, const int4* __restrict__ twR,
                                       const int4* __restrict__ twX, const FxGroup& gr) {
    constexpr int G = H / 8;
    const int t = gr.t;
    q2 z[8];
    unsigned lsum, nan;
    int e = fx_enter<G, FX_BITS, WIDE>(v, z, gr, lsum, nan);
    e += fx_stages<H, false, FX_BITS, true>(z, rb, twX, gr, lsum);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        q2 h;  // halves, for the split's sums
        h.x = fx_shr(z[m].x, 1, 1);
        h.y = fx_shr(z[m].y, 1, 1);
        fx_strow(&rb[pad8(t + m * G)], h);
    }
    fx_sync<G>(gr);
    const FxOut<WIDE> out(e, nan);
    // X[k] = (z[k] + conj z[H-k])/2 + w^k (z[k] - conj z[H-k])/(2i), and X[H-k] likewise
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k = 1 + t + i * G;
        const bool sp = i == 3 && k == H / 2;
        double2 *pk = &rb[pad8(sp ? 0 : k)], *pm = &rb[pad8(H - k)];
        const q2 a = fx_ldrow(pk), c = fx_ldrow(pm);
        q2 s, d;
        s.x = a.x + c.x; s.y = a.y - c.y;
        d.x = a.y + c.y; d.y = c.x - a.x;       // (z[k] - conj z[H-k]) / i
        const q2 o = fx_cmul(d, __ldg(&twR[k]));
        q2 xk = fx_add(s, o), xm;
        xm.x = s.x - o.x; xm.y = o.y - s.y;     // conj(s - o): w^(H-k) = -conj(w^k)
        if (sp) {
            xk.x = 2 * (a.x + a.y); xk.y = 0;   // X[0] = Re z[0] + Im z[0]
            xm.x = 2 * c.x; xm.y = -2 * c.y;    // X[H/2] = conj z[H/2]
        }
        *pk = out(xk);
        if (sp) pk->y = 0.0;
        *pm = out(xm);
    }
    if (WIDE && out.scale != 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // the thread's own elements
            const int k = 1 + t + i * G;
            double2 *pk = &rb[pad8(i == 3 && k == H / 2 ? 0 : k)], *pm = &rb[pad8(H - k)];
            *pk = out.scaled(*pk);
            *pm = out.scaled(*pm);
        }
    }
}

}  // namespace fsibe
