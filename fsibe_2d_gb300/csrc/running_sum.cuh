// The four running sums of integrate_position (integrate_position.f90:14-44), bit for bit the
// sequential FP64 loop s_0 = +0, s_(k+1) = s_k + a_k (round to nearest even).
//
// A dependent FP64 addition costs about 75 cycles on this chip.  While s_k and s_(k+1) stay in
// one binade [2^e, 2^(e+1)), the FP64 sum is an integer sum on that binade's grid 2^g
// (g = e - 52): with s_k = m 2^g,
//     s_(k+1) = (m + RN(a_k / 2^g)) 2^g,
// where RN rounds to the nearest integer; only a tie depends on m.  So a warp a sum
//   * sums the terms approximately in fixed point (each lane a run of consecutive terms, one scan),
//     which tells every s_k's binade where the error bound leaves no doubt;
//   * rounds the terms of steps within a binade to its grid in parallel: their increments and those
//     increments' prefix sums do not depend on the running value.  What is left are the events:
//     steps into another binade, ties, zeros, values near a power of two;
//   * walks the events in order: the value before an event is the value after the last one plus a
//     prefix difference (integers), the event itself an FP64 addition;
//   * fills in every s_k in parallel.
// Afterwards every step is checked in parallel by the FP64 addition, bits(s_k + a_k) ==
// bits(s_(k+1)), and a sum with any mismatch is formed again by the serial loop: the result is that
// loop's in every case.  A beam of 1024 nodes has 11 to 81 events a sum.  Up to rs_serial terms the
// serial loop itself is the shortest (78 cycles a step from shared memory): this code runs once a
// launch, on one warp, and its integer chains are long.  Sums with many events, non-finite or very
// small terms take the serial loop too.
// Measured (GB300, k cycles of the phase in k_beam_cl, serial / by events; a straight beam and, after
// the semicolon, a heaving one, which has fewer events): ns = 256 22 / 27, 384 33 / 38; 34 / 28, 512 43 / 58-70; 43 / 59,
// 576 52 / 57; 52 / 46, 768 67 / 63; 67 / 51, 1024 87 / 73; 87 / 60.  The kernel, us: 512 103 / 120; 110 / 120,
// 576 147 / 151; 154 / 151, 640 152 / 154; 157 / 155, 832 173 / 171; 180 / 171 (one process to another differs by 3).
#pragma once
#include "common.cuh"

namespace fsibe {

// a / 2^g rounded to the nearest integer, for a term that allows an integer step (ok): zero, or
// finite and below the grid's unit.  A tie (tie) returns its lower candidate; its rounding
// depends on the running value's parity.
__device__ __forceinline__ long long term_inc(double a, int g, bool& ok, bool& tie) {
    const unsigned long long TWO52 = 1ull << 52, FRAC = TWO52 - 1ull;
    const unsigned long long ab = (unsigned long long)__double_as_longlong(a);
    const int ex = (int)((ab >> 52) & 0x7FF);
    const unsigned long long ma = (ab & FRAC) | (ex ? TWO52 : 0ull);
    const int sh = g - (ex ? ex - 1075 : -1074);      // a = ma 2^(g - sh)
    const int shc = sh < 1 ? 1 : (sh > 63 ? 63 : sh);  // for sh >= 63 the quotient rounds to 0 all the same
    const unsigned long long q = ma >> shc, rem = ma & ((1ull << shc) - 1ull), half = 1ull << (shc - 1);
    const bool neg = (ab >> 63) != 0;
    const long long r = (long long)(q + (rem > half ? 1ull : 0ull));
    ok = ma == 0ull || (sh > 0 && ex != 0x7FF);
    tie = ma != 0ull && rem == half;
    if (ma == 0ull) return 0;
    if (tie) return neg ? -(long long)q - 1 : (long long)q;
    return neg ? -r : r;
}

constexpr int RS_MAX = 2016, RS_EVENTS = 96;  // RS_MAX: 63 terms a lane
// Terms up to which the serial loop is taken: its step is 78 cycles from shared memory (SH), 112 else.
template <bool SH> constexpr int rs_serial() { return SH ? 544 : 320; }

// The serial loop, by lane 0 of a warp: 78 cycles a step with the rows in shared memory (SH), 112
// through generic addresses.
template <bool SH>
__device__ __forceinline__ void running_sum_serial(const double* __restrict__ src, double* __restrict__ dst, int n) {
    if ((threadIdx.x & 31) != 0) return;
    if (SH) { __builtin_assume(__isShared(src)); __builtin_assume(__isShared(dst)); }
    double v = 0.0;
    int k = 0;
    for (; k + 8 <= n; k += 8) {
        double t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = src[k + i];
#pragma unroll
        for (int i = 0; i < 8; ++i) { dst[k + i] = v; v = v + t[i]; }
    }
    for (; k < n; ++k) { dst[k] = v; v = v + src[k]; }
}

template <typename T> __device__ __forceinline__ T rs_scan(T v) {  // exclusive sum over the lanes
    const int lane = threadIdx.x & 31;
    T p = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T x = __shfl_up_sync(0xffffffffu, p, o);
        if (lane >= o) p += x;
    }
    return p - v;
}
// the value d steps of cur's grid further, in its binade
__device__ __forceinline__ double rs_advance(double cur, long long d) {
    const unsigned long long TWO52 = 1ull << 52, FRAC = TWO52 - 1ull;
    const unsigned long long b = (unsigned long long)__double_as_longlong(cur);
    const long long mc = (long long)((b & FRAC) | TWO52), m = ((long long)b < 0 ? -mc : mc) + d;
    return d == 0 ? cur : __longlong_as_double((long long)((b & ~FRAC) | ((unsigned long long)(m < 0 ? -m : m) & FRAC)));
}

// One sum on one warp (all 32 lanes, the same arguments): dst[k] = s_k for k < n <= RS_MAX; start
// and base have RS_EVENTS entries of shared memory.  False when the sum is left to the serial loop.
template <bool SH>
__device__ __noinline__ bool running_sum_warp(const double* __restrict__ src, double* __restrict__ dst, int n, double* start, long long* base) {
    if (SH) { __builtin_assume(__isShared(src)); __builtin_assume(__isShared(dst)); }
    // an odd run of terms a lane: the lanes' accesses fall in different banks
    const int lane = threadIdx.x & 31, c = ((n + 31) / 32) | 1;
    const int k0 = min(lane * c, n), k1 = min(k0 + c, n);
    long long* pre = reinterpret_cast<long long*>(dst);  // prefix sums until the sums replace them
    unsigned mx = 0;
#pragma unroll 4
    for (int k = k0; k < k1; ++k) mx = max(mx, (unsigned)__double2hiint(src[k]) & 0x7fffffffu);
    const int em = (int)(__reduce_max_sync(0xffffffffu, mx) >> 20);
    if (em == 0x7FF || em < 64) return false;
    // a term in units of 2^(em - 1073), towards zero (below 2^51; n of them below 2^62)
    auto fix = [&](double a) {
        const int hi = __double2hiint(a), e = (hi >> 20) & 0x7FF;
        const unsigned long long m = (((unsigned long long)(((unsigned)hi & 0xfffffu) | 0x100000u)) << 32) | (unsigned)__double2loint(a);
        const long long v = (long long)(m >> min(em - e + 2, 63));
        return hi < 0 ? -v : v;
    };
    long long tot = 0, mag = 0;
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
        const long long q = fix(src[k]);
        tot += q;
        mag += q < 0 ? -q : q;
    }
    long long s = rs_scan(tot);
    mag = rs_scan(mag) + mag;
    mag = __shfl_sync(0xffffffffu, mag, 31);
    // error of s against the sequential sum: the truncations, and the n rounding errors, each at most
    // 2^-53 of the sum of magnitudes
    const long long err = 2 * n + (mag >> 41);
    // s_k's binade: 1 + its exponent above the unit, with the sign; 0 in doubt
    auto binade = [&](long long v) {
        const long long a = v < 0 ? -v : v, lo = a - err, hi = a + err;
        if (lo <= 0) return 0;
        const int bl = 64 - __clzll(lo), bh = 64 - __clzll(hi);
        return bl != bh ? 0 : (v < 0 ? -bl : bl);
    };
    unsigned long long events = 0;  // of the lane's steps
    long long p = 0;                // prefix sum of its increments
    int bin = lane == 0 ? 0 : binade(s);
#pragma unroll 2
    for (int k = k0; k < k1; ++k) {
        const double a = src[k];
        s += fix(a);
        const int next = binade(s);
        bool ok = false, tie = false;
        long long inc = 0;
        if (bin != 0 && bin == next) inc = term_inc(a, (bin < 0 ? -bin : bin) - 53 + (em - 1073), ok, tie);
        pre[k] = p;
        if (ok && !tie) p += inc;
        else events |= 1ull << (k - k0);
        bin = next;
    }
    const long long off = rs_scan(p);
    const int nev = __popcll(events), ord = rs_scan(nev);
    if (__shfl_sync(0xffffffffu, ord + nev, 31) > RS_EVENTS) return false;
    __syncwarp();
    // the events in order, every lane alike: step 0 is one (s_0 = 0)
    double cur = 0.0;
    long long at = 0;
    int ne = 0;
    for (int l = 0; l < 32; ++l) {
        unsigned long long m = __shfl_sync(0xffffffffu, events, l);
        const long long o = __shfl_sync(0xffffffffu, off, l);
        while (m) {
            const int k = l * c + __ffsll((long long)m) - 1;
            m &= m - 1ull;
            const long long pk = o + pre[k];
            cur = rs_advance(cur, pk - at) + src[k];
            at = pk;
            if (lane == 0) { start[ne] = cur; base[ne] = pk; }
            ++ne;
        }
    }
    __syncwarp();
    int j = ord;  // events before step k
    for (int k = k0; k < k1; ++k) {
        dst[k] = k == 0 ? 0.0 : rs_advance(start[j - 1], off + pre[k] - base[j - 1]);
        if ((events >> (k - k0)) & 1ull) ++j;
    }
    return true;
}

// The four sums of rows src + q sld into dst + q dld (q < 4), each by warp q, then checked by
// all threads of the (256-thread) block.  idle(i, m) runs on
// warps 4..7 (i < m) meanwhile.  flags: 4 ints of shared memory.  Returns the number of sums the
// check sent to the plain serial loop.  Ends with a barrier.
// SH: src and dst are shared memory.
template <bool SH, typename Idle>
__device__ int running_sums4(const double* src, int sld, double* dst, int dld, int n, int* flags, Idle idle) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    __shared__ double start[4][RS_EVENTS];
    __shared__ long long base[4][RS_EVENTS];
    if (warp < 4) {
        const double* s = src + (size_t)warp * sld;
        double* d = dst + (size_t)warp * dld;
        if (lane == 0) flags[warp] = 0;
        if (n <= rs_serial<SH>() || n > RS_MAX || !running_sum_warp<SH>(s, d, n, start[warp], base[warp])) {
            __syncwarp();
            running_sum_serial<SH>(s, d, n);
        }
    } else {
        idle(tid - 128, blockDim.x - 128);
    }
    __syncthreads();
    if (n <= rs_serial<SH>()) return 0;
    for (int j = tid; j < 4 * n; j += blockDim.x) {
        const int q = j / n, k = j - q * n;
        if (k + 1 < n) {
            const double* s = src + (size_t)q * sld;
            const double* d = dst + (size_t)q * dld;
            // (a NaN's bits differ from one operation to another: two NaNs agree)
            const double v = d[k] + s[k], x = d[k + 1];
            if (__double_as_longlong(v) != __double_as_longlong(x) && (v == v || x == x)) flags[q] = 1;
        }
    }
    __syncthreads();
    const int bad = (flags[0] != 0) + (flags[1] != 0) + (flags[2] != 0) + (flags[3] != 0);
    if (warp < 4 && flags[warp]) running_sum_serial<SH>(src + (size_t)warp * sld, dst + (size_t)warp * dld, n);
    __syncthreads();
    return bad;
}

struct NoIdle {
    __device__ void operator()(int, int) const {}
};

}  // namespace fsibe
