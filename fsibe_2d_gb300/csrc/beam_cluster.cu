// beam_cluster.cu -- the Newton step of the beam (the work of k_beam: IBES_solver after the
// step's loads are known, SolidSolver.f90:197-414, with integrate_position and SolidEnergies)
// on one thread-block cluster of R CTAs (16, 8 or 4: beam_cluster_setup).
//
// Why a cluster: FP64 issue limits the beam (one FP64 warp instruction per SMSP every ~64
// cycles on this chip) and one CTA has four SMSPs.  Spreading F, the Jacobian rows and the
// residuals over R SMs divides that work by R; the cluster's hardware barrier and distributed
// shared memory (DSMEM) keep every exchange between the SMs on chip.
//
// Layout: CTA r owns a run of the interleaved rows (cl_rows) of the Newton system
// (n = 2 ns + 4): their F values, their FP64 Jacobian band rows, and the same rows of M^-1,
// the inverse of the row-scaled FP32 LU factor that preconditions the FP64 iterative
// refinement.  Every CTA keeps a full copy of the iterate x and of the refinement solution.
// One refinement pass:
//   FP64 residual of the own rows -> all-gather of the FP32 right-hand side -> barrier ->
//   own rows of M^-1 y (FP32) -> FP64 update of the own solution rows -> all-gather of those
//   rows and of the pass's maxima -> barrier -> the same convergence decision in every CTA.
// A new factor: each CTA scales its band rows and all-gathers them; every CTA runs the same
// FP32 band LU (the routine of the single-CTA kernel, so every copy is bitwise identical) and
// computes its own rows of M^-1 by transposed solves.  M^-1 persists between steps in global
// memory (kept while it contracts: newton_pass).
// The iterate update, the norms and the stopping test run redundantly in every CTA on
// identical data, so they need no exchange.
// What bounds it: chains of dependent FP64 (an addition is some 70 cycles) and the barriers, two a
// pass.  A warp evaluates one of the two node equations (they alternate by row, and a warp of both ran
// the two codes one after the other), and the passes end when their corrections no longer change the
// iterate (newton_pass).  Measured (us, before -> after both, and rows of the band on different banks):
// ns = 64 55 -> 46, 128 (heaving) 74 -> 59, 256 84 -> 62, 1024 333 -> 250 (and 212 with more loads in
// flight in the product).
// Large beams (ns >= 512: M^-1's rows and the factor exceed a CTA's shared memory) run the
// same algorithm with both in global memory, where they stay L2-resident: each CTA reads its
// rows of M^-1 from its slice of the persistent copy, and factors its own copy of the band
// (the all-gather of the scaled rows writes every CTA's copy directly; the cluster barrier's
// release/acquire orders those global stores as it orders the DSMEM ones).
#include <math.h>

#include <mutex>

#include "beam_impl.cuh"
#include "running_sum.cuh"

namespace fsibe {
namespace {

// ---- cluster primitives (PTX) --------------------------------------------------------
__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cl_nrank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// Cluster-wide barrier of all threads; release/acquire orders the DSMEM writes before it
// against the reads after it.
__device__ __forceinline__ void cl_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The generic address of the same shared-memory location in CTA `rank` of the cluster.
template <typename T>
__device__ __forceinline__ T* cl_map(T* p, unsigned rank) {
    unsigned long long out;
    asm volatile("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<unsigned long long>(p)), "r"(rank));
    return reinterpret_cast<T*>(out);
}
__device__ __forceinline__ void cp_async16(void* s, const void* g) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// ---- shared-memory layout (the same function sizes the launch on the host) ------------
// Row stride of M^-1: >= n, 16-byte rows, = 4 (mod 32) words.
__host__ __device__ inline int cl_mld(int n) { return ((n + 27) / 32) * 32 + 4; }
__host__ __device__ inline size_t al16(size_t v) { return (v + 15) & ~(size_t)15; }
// doubles a band row: one more than its 16 entries, so that the rows of a warp's lanes fall in different
// banks (at 16 every access of a Jacobian warp was a 32-way conflict)
constexpr int CL_BAND = 17;
constexpr int CL_NODE = 9;  // per-node FP64 arrays: tdn, bo3, bo4, bo5, bo6, oo5, oo6, old_rhs, taun_s

struct ClLayout {
    int n, L, R, rmax, mld;
    size_t x, xdi, node, bvec, band, part, slots, yf, fact, minv, total;  // byte offsets
};

// The rows [lo, hi) of CTA r: quads of rows, so that every CTA's slice of the FP32 right-hand side (and
// of the FP64 solution) starts on a 16-byte boundary.  With R >= 8 and n <= 600 the first and the last
// CTA hold the four boundary equations alone (and one node, when ns is odd) and the others share the
// rest evenly: a warp of generic rows takes its time whether one row or 32, and the boundary
// equations' beside it on the same SMSPs made those two CTAs the slowest (F and J of an iteration
// 4.6k cycles with them, 3.1k without).  The others' slices of M^-1 are larger for it: from ns = 302 on they
// no longer fit 16 CTAs' shared memory, where an even split does up to 318.  The kernel in us, alone / even,
// both in shared memory: ns = 144 55 / 57, 256 65 / 67.5, 296 70 / 73; alone in global memory: 312 78-82 /
// 72-74, 318 77-84 / 74-75 (one process to another differs by up to 3).  Above, all share evenly.
__host__ __device__ inline bool cl_ends_alone(int n, int R) {
    const int nq = (n + 3) / 4, last = nq - (n - 4) / 4;
    return R >= 8 && n <= 600 && nq - 1 - last >= R - 2;
}
__host__ __device__ inline void cl_rows(int n, int R, int r, int& lo, int& hi) {
    const int nq = (n + 3) / 4;
    if (cl_ends_alone(n, R)) {
        const int mid = (n - 4) / 4 - 1;  // quads of the CTAs between
        lo = (r == 0) ? 0 : 1 + (r - 1) * mid / (R - 2);
        hi = (r == R - 1) ? nq : 1 + r * mid / (R - 2);
        lo *= 4;
        hi *= 4;
    } else {
        lo = 4 * (int)(((long long)r * nq) / R);
        hi = 4 * (int)(((long long)(r + 1) * nq) / R);
    }
    lo = lo < n ? lo : n;
    hi = hi < n ? hi : n;
}
__host__ __device__ inline int cl_rmax(int n, int R) {
    const int nq = (n + 3) / 4;
    if (!cl_ends_alone(n, R)) return 4 * ((nq + R - 1) / R);
    const int mid = ((n - 4) / 4 - 1 + R - 3) / (R - 2), last = nq - (n - 4) / 4;
    return 4 * (mid > last ? mid : last);
}

// Floats of one CTA's global copy of the factor area in the large-beam form (the factor, or
// after the Newton loop the position sums, as in shared memory), a multiple of 4.
__host__ __device__ inline size_t cl_fact_floats(int ns) {
    const int n = 2 * ns + 4, L = ns + 8;
    const size_t fact = 25 * (size_t)(n + 16), post = 20 * (size_t)L;
    return ((fact > post ? fact : post) + 3) & ~(size_t)3;
}

// big: the factor area and M^-1 live in global memory (not in the shared-memory layout)
__host__ __device__ inline void cl_layout(int ns, int R, ClLayout& Y, bool big = false) {
    Y.n = 2 * ns + 4;
    Y.L = ns + 8;
    Y.R = R;
    Y.rmax = cl_rmax(Y.n, R);
    Y.mld = cl_mld(Y.n);
    size_t o = 0;
    Y.x = o;     o = al16(o + 8 * (size_t)(Y.n + 8));
    Y.xdi = o;   o = al16(o + 8 * (size_t)(Y.n + 8));
    Y.node = o;  o = al16(o + 8 * (size_t)CL_NODE * Y.L);
    Y.bvec = o;  o = al16(o + 8 * (size_t)Y.rmax);
    Y.band = o;  o = al16(o + 8 * CL_BAND * (size_t)Y.rmax);
    Y.part = o;  o = al16(o + 8 * 4 * (size_t)Y.rmax);
    Y.slots = o; o = al16(o + 8 * 3 * (size_t)R);
    Y.yf = o;    o = al16(o + 4 * (size_t)(Y.mld + 16));
    if (big) { Y.fact = Y.minv = Y.total = o; return; }
    Y.fact = o;
    // the factor (U 16, L 8 floats and a row-scale exponent per row); after the Newton loop
    // CTA 0 reuses it for the position sums (cs, pre: 4 L each) and th, thd (L each)
    const size_t fact = 4 * 25 * (size_t)(Y.n + 16), post = 8 * 10 * (size_t)Y.L;
    o = al16(o + (fact > post ? fact : post));
    Y.minv = o;  o = al16(o + 4 * (size_t)Y.rmax * Y.mld);
    Y.total = o;
}

// Fortran equation (1-based) of interleaved row r: the inverse of row_of.
__device__ __forceinline__ int k_of_row(int ns, int r) {
    if (r <= 3) return (r == 3) ? 7 : r + 1;
    if (r >= 2 * ns) { const int q = r - 2 * ns; return (q == 0) ? 8 : 7 - q; }
    if ((r & 1) == 0) return 8 + (r / 2 - 1);
    return 8 + (ns - 2) + ((r - 1) / 2 - 1);
}

// Row i of M^-1 = (P L U)^-1 of the FP32 factor (band_factor_f32's U and L rows):
// z = U^-T e_i by forward substitution, then the transposed elimination steps in reverse
// order -- step k: v_k -= sum_r l_(k,r) v_(k+r), then the interchange of v_k and v_(k+p_k).
// Written to out[0 .. mld) (zeros from n on).
__device__ void inv_row(const float* __restrict__ U, const float* __restrict__ Lm, int n, int mld, int i,
                        float* __restrict__ out) {
    for (int k = 0; k < i; ++k) out[k] = 0.f;
    float zw[15];
#pragma unroll
    for (int j = 0; j < 15; ++j) zw[j] = 0.f;
    for (int k = i; k < n; ++k) {
        float acc = (k == i) ? 1.f : 0.f;
#pragma unroll
        for (int j = 14; j >= 2; --j) {
            const int m = (k - j) > 0 ? (k - j) : 0;  // rows before 0 meet zw[j] == 0
            acc = __fmaf_rn(-U[(size_t)m * 16 + j], zw[j], acc);
        }
        acc = __fmaf_rn(-U[(size_t)((k - 1) > 0 ? (k - 1) : 0) * 16 + 1], zw[1], acc);
        const float zk = __fmul_rn(acc, U[(size_t)k * 16]);
        out[k] = zk;
#pragma unroll
        for (int j = 14; j >= 2; --j) zw[j] = zw[j - 1];
        zw[1] = zk;
    }
    float wv[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) wv[r] = 0.f;
    for (int k = n - 1; k >= 0; --k) {
        if (k + 8 < n) out[k + 8] = wv[7];  // v_(k+8) is final: later steps reach k+6 at most
#pragma unroll
        for (int r = 7; r >= 1; --r) wv[r] = wv[r - 1];
        const float4 la = *reinterpret_cast<const float4*>(Lm + (size_t)k * 8);
        const float4 lb = *reinterpret_cast<const float4*>(Lm + (size_t)k * 8 + 4);
        float t = out[k];
        t = __fmaf_rn(-la.y, wv[1], t);
        t = __fmaf_rn(-la.z, wv[2], t);
        t = __fmaf_rn(-la.w, wv[3], t);
        t = __fmaf_rn(-lb.x, wv[4], t);
        t = __fmaf_rn(-lb.y, wv[5], t);
        t = __fmaf_rn(-lb.z, wv[6], t);
        t = __fmaf_rn(-lb.w, wv[7], t);
        wv[0] = t;
        const int p = __float_as_int(la.x);
        if (p != 0) {
#pragma unroll
            for (int r = 1; r <= 7; ++r)
                if (r == p) { wv[0] = wv[r]; wv[r] = t; }
        }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r)
        if (r < n) out[r] = wv[r];
    for (int k = n; k < mld; ++k) out[k] = 0.f;
}

// The value of a double whose high word (sign cleared) is h, rounded down to its 20 bits, in FP32 (zero
// and infinity outside FP32's normal range).
__device__ __forceinline__ float hi_to_float(unsigned h) {
    const int e = (int)(h >> 20) - 1023;
    if (e < -126) return 0.f;
    if (e > 127) return __int_as_float(0x7f800000);
    return __uint_as_float((unsigned)(e + 127) << 23 | (h & 0xfffffu) << 3);
}

// The decision after a pass of the iterative refinement of Newton's linear system: 1 done, 0 another
// pass, -1 a new factor.  Of [0] the angles and [1] the tensions, cm is the pass's largest correction,
// cp the previous pass's (at pass 0 the last one of the iteration before), c0 the first pass's, i.e. the
// size of dx, and xmax the iterate's largest entry.
//
// The first two iterations are always followed by another, whose residual sees what they leave:
//   iter 0  dx to 2^-30, by the size of the last correction, or of the one that would follow it;
//   iter 1  the correction that would follow small beside the stopping tolerance (by sqrt(n) 16), so
//           that the stopping test at iter 2 sees what it would after an exact solve;
//   iter 2 on  either unknown to 2^-30 of its dx or 2^-58 of its iterate, whichever is larger, judged
//           by the correction that would follow; at pass 0 the contraction is that since the
//           iteration before.  The norms of the angles and of the tensions are kept apart: the
//           tensions' rounding is often larger than every angle.  Both are taken to contract as
//           the slower does.
// An FP64 solve's error is at 2^-53 of the iterate at best.  2^-30 of every dx, in every iteration, took
// 7 to 10 passes a step, the last three or four of them on corrections below the iterate's last place;
// this takes 5 or 6.  The positions' and the loads' errors against the oracle are the same.
// A first contraction above 2^-6 asks for a new factor in the next iteration (slow).  Corrections that
// stop shrinking end the passes: with a good first contraction they are at the residual's rounding and
// dx stands if it is known to 2^-30, else a factor kept from an earlier step is replaced.
__device__ __forceinline__ int newton_pass(int iter, int pass, const float* cm, const float* cp, const float* c0,
                                           const float* xmax, float rn, float tol, bool is_new, bool& slow) {
    const float cn = fmaxf(cm[0], cm[1]), c0n = fmaxf(c0[0], c0[1]), xn = fmaxf(xmax[0], xmax[1]);
    const bool exact = !(cn > 0x1p-30f * c0n);  // also NaN, which the update flags
    const float most = is_new ? 0.5f : 0.125f;
    bool conv, stall = false;
    const float q0 = cm[0] > 0.f ? cm[0] / cp[0] : 0.f, q1 = cm[1] > 0.f ? cm[1] / cp[1] : 0.f;
    const float ratio = fmaxf(q0, q1);
    if (iter < 2) {
        const float cpn = fmaxf(cp[0], cp[1]);
        const bool next = (iter == 0) ? cn * (cn / cpn) <= 0x1p-30f * c0n : 16.f * rn * (cn * ratio) <= tol * fmaxf(1.f, xn);
        conv = exact || (pass >= 1 && next);
        stall = pass >= 2 && cn > most * cpn;
        slow |= pass == 1 && !conv && cn > 0x1p-6f * cpn;
    } else {
        conv = true;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float t = fmaxf(fmaxf(0x1p-30f * c0[q], 0x1p-58f * xmax[q]), 0x1p-86f * xn);
            const bool cv = !(cm[q] > t) || cm[q] * ratio <= t;
            conv = conv && cv;
            stall |= pass >= 2 && !cv && cm[q] > most * cp[q];
            slow |= pass == 1 && !cv && cm[q] > 0x1p-6f * cp[q];
        }
    }
    if (conv) return 1;
    if (!stall && pass < 9) return 0;
    return (exact && (is_new || !slow)) ? 1 : -1;
}

}  // namespace

#define PH(k) do { const long long t_ = clock64(); ph[k] += t_ - ph_t; ph_t = t_; } while (0)

// The cluster form of k_beam (one cluster of R CTAs of 256 threads; R from the launch).
// k_beam_pre of the same step ran before it and left the step's constants in b.pred.
// k_forces lets it start early (pdl_trigger): the set-up that reads only what earlier kernels
// wrote (the beam state, the predictor's output, the stored inverse rows) runs before its
// pdl_wait, which precedes every read of the forces' loads and of the status.
__device__ __forceinline__ void beam_cl_run(const BeamArgs& b) {
    extern __shared__ __align__(16) unsigned char cl_smem[];
    DevScalars* S = b.S;
    const unsigned rank = cl_rank(), R = cl_nrank();
    const int ns = b.ns, n = 2 * ns + 4;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x, nwarp = nthr >> 5;
    const bool big = b.cl_big != 0;
    const size_t fstride = cl_fact_floats(ns);
    ClLayout Y;
    cl_layout(ns, (int)R, Y, big);
    const int L = Y.L, mld = Y.mld, rmax = Y.rmax;
    int lo, hi;
    cl_rows(n, (int)R, (int)rank, lo, hi);
    const int nr = hi - lo;
    double* x = reinterpret_cast<double*>(cl_smem + Y.x);
    double* xdi = reinterpret_cast<double*>(cl_smem + Y.xdi);
    double* nd = reinterpret_cast<double*>(cl_smem + Y.node);
    double *tdn = nd, *bo3 = nd + L, *bo4 = nd + 2 * L, *bo5 = nd + 3 * L, *bo6 = nd + 4 * L, *oo5 = nd + 5 * L,
           *oo6 = nd + 6 * L, *old_rhs = nd + 7 * L, *taun_s = nd + 8 * L;
    double* bvec = reinterpret_cast<double*>(cl_smem + Y.bvec);
    double* band = reinterpret_cast<double*>(cl_smem + Y.band);
    double* part = reinterpret_cast<double*>(cl_smem + Y.part);
    // exchange words, written by every CTA into every CTA: [0, R) the passes' max |c| of the angles
    // and, in the high word, of the tensions (FP32 bits), [R, 2R) the flags sent with the right-hand
    // side, [2R, 3R) the flags sent with the factor rows
    unsigned long long* slots = reinterpret_cast<unsigned long long*>(cl_smem + Y.slots);
    float* yf = reinterpret_cast<float*>(cl_smem + Y.yf);
    float* Uf = big ? b.clws + (size_t)rank * fstride : reinterpret_cast<float*>(cl_smem + Y.fact);
    float* Lf = Uf + (size_t)16 * (n + 16);
    int* rse = reinterpret_cast<int*>(Lf + (size_t)8 * (n + 16));
    float* minv = big ? b.minv + (size_t)rank * rmax * mld : reinterpret_cast<float*>(cl_smem + Y.minv);
    __shared__ D1DTab dtab;
    __shared__ NewtonCtx cs;
    __shared__ double red[2][8];
    __shared__ unsigned redu[2][8];
    __shared__ __align__(16) unsigned xhi[2][8];
    __shared__ int flag_s, stop_s, info_s;

    BeamWS w;
    memset(&w, 0, sizeof(w));
    w.x = x; w.tdn = tdn; w.bo5 = bo5; w.bo6 = bo6; w.oo5 = oo5; w.oo6 = oo6;
    w.old_rhs = old_rhs; w.taun_s = taun_s; w.dtab = &dtab; w.Uf = Uf; w.Lf = Lf; w.rse = rse;

    long long ph_t = clock64(), ph[28] = {};
    // the cluster barrier that guarantees every CTA runs before the first DSMEM access comes
    // just before that access (cl_up), so the set-up overlaps the CTAs' start
    bool cl_up = false;
    d1d_load(&dtab, b.d1d);
    const double time = S->time, dt = S->dt1, grav = S->grav;
    const double ds = b.ds, mue = b.mue, eta = b.eta;
    for (int i = tid; i < ns; i += nthr) {
        bo3[i] = b.vx[i]; bo4[i] = b.vy[i]; bo5[i] = b.th[i]; bo6[i] = b.thd[i];
        oo5[i] = b.oo[4 * ns + i]; oo6[i] = b.oo[5 * ns + i];
    }
    for (int i = n + tid; i < mld + 16; i += nthr) yf[i] = 0.f;
    if (tid == 0) flag_s = 0;
    __syncthreads();

    const bool released = time > b.t_release;
    const Motion mo = motion_at(b.mo, time + dt);  // mouvement(time + dt) of the new level
    int iter = 0;
    const bool have_inv = released && S->beam_fact != 0;
    if (released) {
        if (have_inv) {
            // this CTA's rows of M^-1 and their row-scale exponents, kept from an earlier step
            const float* g = b.minv + (size_t)rank * rmax * mld;
            const int nv = nr * mld / 4;
            if (!big)  // the large-beam form reads its rows where they are
                for (int q = tid; q < nv; q += nthr) cp_async16(minv + 4 * q, g + 4 * q);
            for (int k = lo + tid; k < hi; k += nthr) rse[k] = b.minv_rse[k];
        }
        for (int i = tid; i < n; i += nthr)
            if (i != xi_th(-1) && i != xi_T(ns, -1)) x[i] = b.pred[i];
        for (int i = tid; i < ns; i += nthr) old_rhs[i] = b.pred[n + i];
        // the Newton constants (divisions done by the predictor)
        if (tid == 32) {
            cs.time = time; cs.dt = dt; cs.dt_old = S->dt_old; cs.alpha_t = mo.alpha_t; cs.alpha_tt = mo.alpha_tt; cs.grav = grav;
            newton_consts_pre(cs, b, b.pred + pred_consts(ns));
        }
        __syncthreads();
        for (int i = tid; i < ns; i += nthr) tdn[i] = cs.D * (x[xi_th(i)] - cs.C3 * bo5[i] - cs.C4 * oo5[i]) - cs.C2 * bo6[i];
    }
    // the loads' share of the initial ghost values (SolidSolver.f90:175-187, 197-202) is added below
    const double* K = b.pred + pred_consts(ns);
    const double* g5 = b.pred + n + ns;
    const double* T = g5 + ns;
    double gh0 = 0.0, gh1 = 0.0, gh2 = 0.0, gh3 = 0.0;
    if (released && tid == 0) {
        gh0 = mue * (mo.le[5] * mo.ca - mo.le[4] * mo.sa + grav * mo.ca);
        gh1 = T[0] * g5[1];
        gh2 = (eta / (ds * ds)) * (10.0 * g5[0] - 12.0 * g5[1] + 6.0 * g5[2] - g5[3]);
    }
    if (released && tid == 64) {
        gh0 = mue * (mo.le[4] * mo.ca + mo.le[5] * mo.sa + grav * mo.sa);
        const double th_ss0 = (2.0 * g5[0] - 5.0 * g5[1] + 4.0 * g5[2] - 1.0 * g5[3]) * b.k.ids2;
        const double th_s0 = (-1.5 * g5[0] + 2.0 * g5[1] - 0.5 * g5[2]) * b.k.ids;
        gh1 = -eta * th_ss0;
        gh2 = th_s0;
        gh3 = T[1];
    }
    pdl_wait();     // k_forces has completed: its loads and any status it raised are visible
    if (S->status != 0) {  // the same value in every CTA: they all return here
        cp_async_wait_all();
        return;
    }
    if (released) {
        for (int i = tid; i < ns; i += nthr) taun_s[i] = d1d(&dtab, b.tau_new, ns, 1, i);
        // initial guess ghost values from the new loads (SolidSolver.f90:175-187, 197-202), on two warps
        if (tid == 0) {
            const double K2 = b.p_new[0] + gh0;
            cs.K2 = K2;
            const double C2v = 2.0 * ds * K2 - gh1 + gh2;
            x[xi_th(-1)] = div_cr(C2v, K[8], K[9]);  // C2v / (3 eta/ds^2 - T_0), correctly rounded
        }
        if (tid == 64) {
            const double K1 = gh0 - b.tau_new[0];
            cs.K1 = K1;
            const double T_s0 = gh1 * gh2 + K1;
            x[xi_T(ns, -1)] = gh3 - 2.0 * ds * T_s0;
        }
        __syncthreads();
        const NewtonCtx& c = cs;
        bool inv_pending = have_inv && !big;  // the stored inverse rows are still arriving (cp.async)
        bool need_factor = !have_inv, factored = false;
        // own rows: generic ones [glo, ghi); the boundary equations (rows 0..3: k = 1, 2, 3, 7;
        // rows 2ns..2ns+3: k = 8, 6, 5, 4) sit in the first and last CTA and take warps 4..7, so that
        // their separate code paths do not serialise a warp of generic rows
        const int glo = lo > 4 ? lo : 4, ghi = hi < 2 * ns ? hi : 2 * ns;
        const int ngen = ghi > glo ? ghi - glo : 0;
        const bool has_sp = (lo < 4) || (hi > 2 * ns);
        // generic rows alternate between the two node equations, whose code differs: a warp takes one
        // of them, for F or for J (warp & 3: the four SMSPs), 32 rows at a time
        const int neq = ngen / 2, nseg = has_sp ? 1 : 2;
        const int ja = lo / 2 - 1 > 0 ? lo / 2 - 1 : 0, jb = hi / 2 < ns ? hi / 2 : ns;  // nodes of the own rows
        // the refinement's state, the same in every thread: the first, the previous and the last
        // correction's maxima of the angles and of the tensions, and the iterate's
        float c0[2] = {0.f, 0.f}, cp[2] = {0.f, 0.f}, xmax[2] = {0.f, 0.f};
        const float rn = sqrtf((float)n), tolf = (float)b.tol;
        PH(22);
        for (;;) {
            if ((warp >> 2) < nseg) {
                const int odd = (warp >> 1) & 1;
                for (int g = warp >> 2; g * 32 < neq; g += nseg) {
                    const int q = g * 32 + lane;
                    if (q < neq) {
                        const int r = glo + 2 * q + odd;
                        const int k = odd ? 8 + (ns - 2) + ((r - 1) / 2 - 1) : 8 + (r / 2 - 1);
                        if ((warp & 1) == 0) {
                            const double f = f_eq(b, w, c, k);
                            if (isnan(f)) flag_s = FSIBE_ERR_NAN;
                            bvec[r - lo] = -1.0 * f;
                        } else if (jac_row(b, w, c, k, band + (size_t)(r - lo) * CL_BAND)) {
                            flag_s = FSIBE_ERR_NAN;
                        }
                    }
                }
            } else if (has_sp && warp >= 4) {
                // the boundary equations: the long one's (k = 7 or 8) F and J on warps 4 and 5, one a lane
                // of the other three on warps 6 and 7
                const int base = (lo < 4) ? 0 : 2 * ns, heavy = (lo < 4) ? 3 : 0;
                const int s = (warp < 6) ? heavy : (lane < heavy ? lane : lane + 1);
                const int r = base + s;
                if (lane < (warp < 6 ? 1 : 3) && r >= lo && r < hi) {
                    const int k = k_of_row(ns, r);
                    if ((warp & 1) == 0) {
                        const double f = f_eq(b, w, c, k);
                        if (isnan(f)) flag_s = FSIBE_ERR_NAN;
                        bvec[r - lo] = -1.0 * f;
                    } else if (jac_row(b, w, c, k, band + (size_t)(r - lo) * CL_BAND)) {
                        flag_s = FSIBE_ERR_NAN;
                    }
                }
            }
            __syncthreads();
            PH(4);
            if (inv_pending) {
                cp_async_wait_all();
                inv_pending = false;
            }
            if (!cl_up) { cl_sync(); cl_up = true; }
            int solves = 0;
            bool slow = false;  // a contraction of more than 2^-6
            float dxb = 0.f;    // the corrections' maxima summed: no entry of dx is larger
            for (int attempt = 0; attempt < 2; ++attempt) {
                const bool fresh = need_factor;
                if (need_factor) {
                    // the scaled FP32 rows: own copy first, then every other CTA's
                    for (int r = lo + tid; r < hi; r += nthr)
                        scale_band_row(band + (size_t)(r - lo) * CL_BAND, Uf + (size_t)r * 16, rse + r);
                    __syncthreads();
                    for (int e = tid; e < nr * 5 * ((int)R - 1); e += nthr) {
                        const unsigned dst = (rank + 1 + (unsigned)(e / (nr * 5))) % R;
                        const int q = e % (nr * 5), r = lo + q / 5, part5 = q % 5;
                        float* Ud = big ? b.clws + (size_t)dst * fstride : nullptr;  // dst's global copy
                        if (part5 < 4) {
                            float4* s4 = reinterpret_cast<float4*>(Uf + (size_t)r * 16) + part5;
                            if (big) reinterpret_cast<float4*>(Ud + (size_t)r * 16)[part5] = *s4;
                            else *cl_map(s4, dst) = *s4;
                        } else {
                            if (big) reinterpret_cast<int*>(Ud + (size_t)24 * (n + 16))[r] = rse[r];
                            else *cl_map(rse + r, dst) = rse[r];
                        }
                    }
                    if (tid < (int)R) *cl_map(slots + 2 * R + rank, (unsigned)tid) = (unsigned long long)flag_s;
                    cl_sync();
                    int fl = 0;
                    for (unsigned q = 0; q < R; ++q) fl = fl ? fl : (int)slots[2 * R + q];
                    if (fl) { if (rank == 0 && tid == 0) set_status(S, fl); return; }
                    if (warp == 0) {
                        const int info = band_factor_f32(w, n);
                        if (tid == 0) info_s = info;
                    }
                    __syncthreads();
                    if (info_s) { if (rank == 0 && tid == 0) set_status(S, FSIBE_ERR_SINGULAR); return; }
                    for (int t = tid; t < nr; t += nthr) inv_row(Uf, Lf, n, mld, lo + t, minv + (size_t)t * mld);
                    __syncthreads();
                    need_factor = false;
                    factored = true;
                }
                PH(5);
                bool ok = false;
                for (int pass = 0;; ++pass) {
                    // FP32 right-hand side of the own rows: -F, or the FP64 residual, its 15
                    // band products split in four column chunks over four warps (SMSPs)
                    if (pass > 0) {
                        const int ch = warp & 3;
                        for (int g = warp >> 2; g * 32 < nr; g += nwarp >> 2) {
                            const int t = g * 32 + lane;
                            if (t < nr) {
                                const int k = lo + t;
                                const double* Bk = band + (size_t)t * CL_BAND;
                                double acc = 0.0;
#pragma unroll
                                for (int u = 0; u < 4; ++u) {
                                    const int ci = 4 * ch + u, j = k - KL + ci;
                                    if (ci < BW && j >= 0 && j < n) acc = fma(Bk[ci], xdi[j], acc);
                                }
                                part[ch * rmax + t] = acc;
                            }
                        }
                        __syncthreads();
                    }
                    for (int t = tid; t < nr; t += nthr) {
                        const int k = lo + t;
                        double acc = bvec[t];
                        if (pass > 0) acc = acc - ((part[t] + part[rmax + t]) + (part[2 * rmax + t] + part[3 * rmax + t]));
                        yf[k] = __double2float_rn(acc * row_scale(rse[k]));
                    }
                    __syncthreads();
                    PH(19);
                    // the own rows to every other CTA, 16 bytes a store (slices start on quads)
                    {
                        const int nq4 = (nr + 3) / 4;
                        for (int e = tid; e < nq4 * ((int)R - 1); e += nthr) {
                            const unsigned dst = (rank + 1 + (unsigned)(e / nq4)) % R;
                            float4* p4 = reinterpret_cast<float4*>(yf + lo + 4 * (e % nq4));
                            *cl_map(p4, dst) = *p4;
                        }
                    }
                    if (tid < (int)R) *cl_map(slots + R + rank, (unsigned)tid) = (unsigned long long)flag_s;
                    PH(20);
                    cl_sync();
                    PH(16);
                    {
                        int fl = 0;
#pragma unroll
                        for (int q = 0; q < 16; ++q)
                            if (q < (int)R) fl = fl ? fl : (int)slots[R + q];
                        if (fl) { if (rank == 0 && tid == 0) set_status(S, fl); return; }
                    }
                    // own rows of M^-1 y, eight rows per warp: lanes split the columns (float4),
                    // a transposing butterfly leaves the sum of row
                    // 4 ((l >> 4) & 1) + 2 ((l >> 3) & 1) + ((l >> 2) & 1) in lanes l = 0 (mod 4);
                    // those lanes update the FP64 solution rows
                    unsigned cmt = 0, cmT = 0;  // max |c| of the angles and of the tensions (FP32 bits)
                    const float4* y4 = reinterpret_cast<const float4*>(yf);
                    for (int g = warp; g * 8 < nr; g += nwarp) {
                        const int t0 = g * 8;
                        const float4* mr[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const int t = (t0 + j < nr) ? t0 + j : nr - 1;  // rows past nr: repeat the last
                            mr[j] = reinterpret_cast<const float4*>(minv + (size_t)t * mld);
                        }
                        float acc[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
                        auto add = [&](const float4& v, const float4 (&m)[8]) {
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                acc[j] = __fmaf_rn(m[j].x, v.x, acc[j]);
                                acc[j] = __fmaf_rn(m[j].y, v.y, acc[j]);
                                acc[j] = __fmaf_rn(m[j].z, v.z, acc[j]);
                                acc[j] = __fmaf_rn(m[j].w, v.w, acc[j]);
                            }
                        };
                        const int nq = mld >> 2;
                        int q = lane;
                        if (big) {
                            // rows in L2: what bounds the product is how many loads are in flight, so
                            // twice eight a lane (ns = 1024: 30k cycles a pass with eight, 20k with sixteen)
                            for (; q + 32 < nq; q += 64) {
                                float4 m0[8], m1[8];
#pragma unroll
                                for (int j = 0; j < 8; ++j) { m0[j] = __ldcg(mr[j] + q); m1[j] = __ldcg(mr[j] + q + 32); }
                                add(y4[q], m0);
                                add(y4[q + 32], m1);
                            }
                        }
                        for (; q < nq; q += 32) {
                            float4 m0[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j) m0[j] = mr[j][q];
                            add(y4[q], m0);
                        }
                        {
                            const bool up = (lane & 16) != 0;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float send = up ? acc[j] : acc[j + 4], keep = up ? acc[j + 4] : acc[j];
                                acc[j] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, 16));
                            }
                            const bool b8 = (lane & 8) != 0;
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                const float send = b8 ? acc[j] : acc[j + 2], keep = b8 ? acc[j + 2] : acc[j];
                                acc[j] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, 8));
                            }
                            const bool b4 = (lane & 4) != 0;
                            const float send = b4 ? acc[0] : acc[1], keep = b4 ? acc[1] : acc[0];
                            acc[0] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, 4));
                            acc[0] = __fadd_rn(acc[0], __shfl_xor_sync(0xffffffffu, acc[0], 2));
                            acc[0] = __fadd_rn(acc[0], __shfl_xor_sync(0xffffffffu, acc[0], 1));
                        }
                        const int t = t0 + 4 * ((lane >> 4) & 1) + 2 * ((lane >> 3) & 1) + ((lane >> 2) & 1);
                        if ((lane & 3) == 0 && t < nr) {
                            const float s = acc[0];
                            const int k = lo + t;
                            const double xn = (pass == 0) ? (double)s : xdi[k] + (double)s;
                            xdi[k] = xn;
                            const unsigned a = __float_as_uint(s) & 0x7fffffffu;
                            if ((k & 1) && k < 2 * ns + 2) cmT = (a > cmT) ? a : cmT;
                            else cmt = (a > cmt) ? a : cmt;
                        }
                    }
                    cmt = __reduce_max_sync(0xffffffffu, cmt);
                    cmT = __reduce_max_sync(0xffffffffu, cmT);
                    if (lane == 0) { redu[0][warp] = cmt; redu[1][warp] = cmT; }
                    __syncthreads();
                    PH(17);
                    if (warp == 0) {
                        const unsigned mt = __reduce_max_sync(0xffffffffu, lane < nwarp ? redu[0][lane] : 0u);
                        const unsigned mT = __reduce_max_sync(0xffffffffu, lane < nwarp ? redu[1][lane] : 0u);
                        if (lane < (int)R) *cl_map(slots + rank, (unsigned)lane) = ((unsigned long long)mT << 32) | mt;
                    }
                    // the own solution rows to every other CTA, 16 bytes a store
                    {
                        const int nq2 = (nr + 1) / 2;
                        for (int e = tid; e < nq2 * ((int)R - 1); e += nthr) {
                            const unsigned dst = (rank + 1 + (unsigned)(e / nq2)) % R;
                            double2* p2 = reinterpret_cast<double2*>(xdi + lo + 2 * (e % nq2));
                            *cl_map(p2, dst) = *p2;
                        }
                    }
                    PH(21);
                    cl_sync();
                    PH(18);
                    ++solves;
                    // the decision, from the cluster's maxima, by every warp (newton_pass)
                    const unsigned long long sl = (lane < (int)R) ? slots[lane] : 0ull;
                    const float cm[2] = {__uint_as_float(__reduce_max_sync(0xffffffffu, (unsigned)sl)),
                                         __uint_as_float(__reduce_max_sync(0xffffffffu, (unsigned)(sl >> 32)))};
                    if (pass == 0) { c0[0] = cm[0]; c0[1] = cm[1]; dxb = 0.f; }
                    dxb += fmaxf(cm[0], cm[1]);
                    const int dec = newton_pass(iter, pass, cm, cp, c0, xmax, rn, tolf, fresh || factored, slow);
                    cp[0] = cm[0];
                    cp[1] = cm[1];
                    if (dec > 0) { ok = true; break; }
                    if (dec < 0) break;
                }
                if (ok || fresh) break;
                need_factor = true;
            }
            if (solves > 5 || (slow && !factored)) need_factor = true;
            if (tid == 0) ph[10] += solves;
            PH(6);
            // x += dx in Fortran order, the norms and the stopping test: the same data in every
            // CTA, so the same decisions without an exchange
            // the stopping test needs iter > 2: before that the norms are not formed, nor where the bound
            // sqrt(n) max |dx| on the update's norm (and max |x| below the iterate's) decides: its
            // margin of 2^-6 covers the FP32 arithmetic
            const bool test = iter + 1 > 2;
            const float xlow = fmaxf(xmax[0], xmax[1]) - dxb;
            const bool below = test && 1.015625f * rn * dxb < tolf * fmaxf(1.f, xlow);
            const bool norms = test && !below;
            double sd = 0.0, sx = 0.0;
            unsigned xt = 0, xT = 0;
            for (int l = tid; l < n; l += nthr) {
                const double d = xdi[col_of(ns, l + 1)];
                if ((__double2hiint(d) & 0x7ff00000) == 0x7ff00000 && isnan(d)) flag_s = FSIBE_ERR_NAN;
                const double xn = x[l] + d;
                x[l] = xn;
                const unsigned h = (unsigned)__double2hiint(xn) & 0x7fffffffu;
                if (l < ns + 3) xt = h > xt ? h : xt;
                else xT = h > xT ? h : xT;
                if (l > ja && l <= jb) tdn[l - 1] = c.D * (xn - c.C3 * bo5[l - 1] - c.C4 * oo5[l - 1]) - c.C2 * bo6[l - 1];
                if (norms) {
                    sd += d * d;
                    sx += xn * xn;
                }
            }
            xt = __reduce_max_sync(0xffffffffu, xt);
            xT = __reduce_max_sync(0xffffffffu, xT);
            if (lane == 0) { xhi[0][warp] = xt; xhi[1][warp] = xT; }
            if (norms) {
                for (int o = 16; o > 0; o >>= 1) {
                    sd += __shfl_xor_sync(0xffffffffu, sd, o);
                    sx += __shfl_xor_sync(0xffffffffu, sx, o);
                }
                if (lane == 0) { red[0][warp] = sd; red[1][warp] = sx; }
            }
            __syncthreads();
            if (flag_s) { if (rank == 0 && tid == 0) set_status(S, flag_s); return; }
            iter = iter + 1;
            if (norms) {
                if (tid < 32) {
                    double tsd = (lane < nwarp) ? red[0][lane] : 0.0, tsx = (lane < nwarp) ? red[1][lane] : 0.0;
                    for (int o = 4; o > 0; o >>= 1) {
                        tsd += __shfl_xor_sync(0xffffffffu, tsd, o);
                        tsx += __shfl_xor_sync(0xffffffffu, tsx, o);
                    }
                    if (lane == 0) stop_s = newton_stop(tsd, tsx, b.tol);
                }
                __syncthreads();
            }
            // the iterate's maxima, rounded down to 20 bits
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const unsigned m = __reduce_max_sync(0xffffffffu, xhi[q][lane & 7]);
                xmax[q] = hi_to_float(m);
            }
            PH(23);
            const bool stop = below || (norms && stop_s != 0);
            if (iter > b.maxit - 1) {
                if (rank == 0 && tid == 0) set_status(S, FSIBE_ERR_NEWTON_MAXIT);
                return;
            }
            if (stop) break;
            __syncthreads();
        }
        if (factored) {
            float* g = b.minv + (size_t)rank * rmax * mld;
            const int nv = nr * mld / 4;
            if (!big)  // the large-beam form formed its rows in place
                for (int q = tid; q < nv; q += nthr)
                    reinterpret_cast<float4*>(g)[q] = reinterpret_cast<const float4*>(minv)[q];
            for (int k = lo + tid; k < hi; k += nthr) b.minv_rse[k] = rse[k];
            if (rank == 0 && tid == 0) S->beam_fact = 1;
        }
    }
    PH(7);
    // integrate_position (integrate_position.f90:14-44): each CTA evaluates theta, theta_dot
    // and the four position increments of its nodes into CTA 0; CTA 0 runs the sums in order.
    // They go to the start of CTA 0's factor area (cs[4][L], pre[4][L], th[L], thd[L]: 80 L
    // bytes), which its factor no longer needs; its row exponents, which it may still be
    // saving, start 96 (n + 16) > 80 L bytes in.  The third sum subtracts: its terms are
    // stored negated and added (s - a and s + (-a) round the same).
    double* pcs = big ? reinterpret_cast<double*>(b.clws) : reinterpret_cast<double*>(cl_smem + Y.fact);
    if (!cl_up) { cl_sync(); cl_up = true; }
    {
        const int q0 = (int)(((long long)rank * ns) / R), q1 = (int)(((long long)(rank + 1) * ns) / R);
        double* dst = big ? pcs : cl_map(pcs, 0u);  // CTA 0's area (its global copy when big)
        for (int i = q0 + tid; i < q1; i += nthr) {
            double th, td;
            if (released) {
                th = x[xi_th(i)];
                td = cs.D * (th - cs.C3 * bo5[i] - cs.C4 * oo5[i]) - cs.C2 * bo6[i];
            } else {
                th = b.th[i];
                td = b.thd[i];
            }
            double sn, cn;
            sincos(th, &sn, &cn);
            dst[i] = cn * ds;
            dst[L + i] = sn * ds;
            dst[2 * L + i] = -(td * sn * ds);
            dst[3 * L + i] = td * cn * ds;
            dst[8 * L + i] = th;
            dst[9 * L + i] = td;
        }
    }
    PH(24);
    cl_sync();  // the last DSMEM traffic; CTAs other than 0 are done
    if (rank != 0) return;
    PH(25);
    const double* thv = pcs + 8 * L;
    const double* tdv = pcs + 9 * L;
    // the new angles and rates, and beam_oldold = beam_old (the state at entry); done by the
    // threads that the running sums leave idle
    auto copies = [&](int i0, int stride) {
        if (!released) return;
        for (int i = i0; i < ns; i += stride) { b.th[i] = thv[i]; b.thd[i] = tdv[i]; }
        for (int i = i0; i < ns; i += stride) {
            b.oo[0 * ns + i] = b.x[i]; b.oo[1 * ns + i] = b.y[i]; b.oo[2 * ns + i] = bo3[i];
            b.oo[3 * ns + i] = bo4[i]; b.oo[4 * ns + i] = bo5[i]; b.oo[5 * ns + i] = bo6[i];
        }
    };
    if (released && tid == 0) {
        S->newton_iters = iter;
        if (S->actually_bdf2) { S->method = FSIBE_BDF2; S->actually_bdf2 = 0; }
        S->dt_old = dt;
    }
    // the four running sums in the reference's order (the positions decide grid-aligned boxes
    // of the mask and the drag window, so their roundings must be the reference's;
    // running_sum.cuh), a warp a sum, while the other warps copy.  The large-beam form first
    // stages the terms into the shared memory of the solution vectors x and xdi (32 ns + 192
    // bytes, at least the 32 ns needed), and the sums go to the node arrays oo5 .. taun_s: the
    // Newton loop is done with both.
    const double* src0 = pcs;
    double* pre = pcs + 4 * L;
    if (big) {
        double* st = x;  // x, then xdi: contiguous
        for (int i = tid; i < ns; i += nthr) {
            st[i] = pcs[i]; st[ns + i] = pcs[L + i]; st[2 * ns + i] = pcs[2 * L + i]; st[3 * ns + i] = pcs[3 * L + i];
        }
        src0 = st;
        pre = oo5;
        __syncthreads();
    }
    {
        __shared__ int rs_flags[4];
        const int nser = running_sums4<true>(src0, big ? ns : L, pre, L, ns, rs_flags, copies);
        if (tid == 0 && nser) S->phase[30] += nser;
    }
    PH(8);
    // positions and velocities, and in the same pass each thread's terms of the emergency brake
    // (SolidSolver.f90:370-380) and of SolidEnergies (SolidSolver.f90:76-92); the block then
    // reduces the six columns in FP64, one warp a column
    {
        __shared__ double ecol[6][256];
        static_assert(256 >= 32 * 6, "one warp a column");
        const double ca = mo.ca, sa = mo.sa, alpha_t = mo.alpha_t, idt = 1.0 / dt;
        double sk = 0, sp = 0, se = 0, sax = 0, say = 0, mx = 0;
        for (int i = tid; i < ns; i += nthr) {
            const double xrel = pre[i], yrel = pre[L + i];
            const double vxrel = pre[2 * L + i], vyrel = pre[3 * L + i];
            const double yi = mo.le[1] + yrel * ca + xrel * sa;
            b.x[i] = mo.le[0] + xrel * ca - yrel * sa;
            b.y[i] = yi;
            const double vx = mo.le[2] + ca * (vxrel - alpha_t * yrel) - sa * (vyrel + alpha_t * xrel);
            const double vy = mo.le[3] + ca * (vyrel + alpha_t * xrel) + sa * (vxrel - alpha_t * yrel);
            b.vx[i] = vx;
            b.vy[i] = vy;
            double ax, ay;
            if (released) {
                ax = (vx - bo3[i]) * idt;
                ay = (vy - bo4[i]) * idt;
                b.ax[i] = ax;
                b.ay[i] = ay;
                mx = fmax(mx, fabs(tdv[i] - bo6[i]));
            } else {
                ax = b.ax[i];
                ay = b.ay[i];
            }
            const double th_s = d1d(&dtab, thv, ns, 1, i);
            sk += vx * vx + vy * vy;
            sp += yi - b.y0;
            se += th_s * th_s;
            sax += ax;
            say += ay;
        }
        ecol[0][tid] = sk; ecol[1][tid] = sp; ecol[2][tid] = se;
        ecol[3][tid] = sax; ecol[4][tid] = say; ecol[5][tid] = mx;
        __syncthreads();
        PH(26);
        if (warp < 6) {
            double v = 0.0;
            for (int k = lane; k < nthr; k += 32) v = (warp == 5) ? fmax(v, ecol[5][k]) : v + ecol[warp][k];
            for (int o = 16; o > 0; o >>= 1) {
                const double u = __shfl_xor_sync(0xffffffffu, v, o);
                v = (warp == 5) ? fmax(v, u) : v + u;
            }
            if (lane == 0) {
                if (warp == 0) S->e_kinetic = mue * 0.5 * ds * v;
                else if (warp == 1) S->e_pot = mue * grav * ds * v;
                else if (warp == 2) S->e_elastic = eta * 0.5 * ds * v;
                else if (warp == 3) S->inertial_force[0] = mue * ds * v;
                else if (warp == 4) S->inertial_force[1] = mue * ds * v;
                else if (released && v > 100.0) set_status(S, FSIBE_ERR_BRAKE);
            }
        }
    }
    PH(9);
    if (b.fuse_adv) {
        // the end of the time step, which the host would otherwise launch next (k_advance)
        __syncthreads();
        advance_state(b.adv);
    }
    PH(27);
    if (tid == 0)
        for (int k = 4; k < 28; ++k) S->phase[k] += ph[k];
}
__global__ void __launch_bounds__(256, 1) k_beam_cl(const __grid_constant__ BeamArgs b) { beam_cl_run(b); }
__global__ void __launch_bounds__(256, 1) k_beam_cl_b(const __grid_constant__ Batch<BeamArgs> b) { beam_cl_run(b.a[blockIdx.z]); }

// ---- host side ------------------------------------------------------------------------
// Floats of the global copy of M^-1 (R slices of rmax rows) and ints of its row exponents.
size_t beam_cluster_minv_floats(int ns, int R) {
    ClLayout Y;
    cl_layout(ns, R, Y);
    return (size_t)R * Y.rmax * Y.mld;
}

// The cluster size for a beam of ns nodes: 16 CTAs above 144 nodes, 8 up to there, 4 where 8 would
// leave a CTA without a quad of rows (ns < 14); the next smaller where the device does not place one
// with this kernel's shared memory, and 0 (the single-CTA kernel) where none fits.  A wider cluster
// divides the rows' FP64 and the inverse products, a narrower one has the cheaper barriers (two a
// pass).  Measured (GB300, 16 / 8 / 4 CTAs, the beam kernel in us): ns = 16 - / 47 / 47 (single CTA
// 100), 64 - / 49 / 51, 101 - / 52 / 53, 127 - / 59 / 63, 256 66 / 83 / 93; 16 / 8 with the sums by events, some
// 4 us, 144 61.3 / 60.4, 160 61.3 / 61.3, 192 64.1 / 63.0, 224 64.2 / 76.6: from 145 nodes on the two are within 2%
// until, from 215, the rows of M^-1 of 8 CTAs do not fit shared memory.  want caps it.
// *big_out = 1 when only the large-beam form (factor and M^-1 in global memory) fits.
int beam_cluster_setup(int ns, int want, size_t* smem_out, int* big_out) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, (const void*)k_beam_cl) != cudaSuccess) return 0;
    static size_t cur = 0;
    for (int R = ns > 144 ? 16 : 8; R >= 4; R /= 2) {
        if (R > want || 2 * ns + 4 < 4 * R) continue;  // at least one quad of rows per CTA
        for (int big = 0; big <= 1; ++big) {
            ClLayout Y;
            cl_layout(ns, R, Y, big != 0);
            if (Y.total + fa.sharedSizeBytes > (size_t)optin) continue;
            if (Y.total > cur) {
                if (cudaFuncSetAttribute((const void*)k_beam_cl, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Y.total) != cudaSuccess ||
                    cudaFuncSetAttribute((const void*)k_beam_cl_b, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Y.total) != cudaSuccess) continue;
                cur = Y.total;
            }
            if (R > 8 && (cudaFuncSetAttribute((const void*)k_beam_cl, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
                          cudaFuncSetAttribute((const void*)k_beam_cl_b, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) continue;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(R);
            cfg.blockDim = dim3(256);
            cfg.dynamicSmemBytes = Y.total;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = R;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int nclusters = 0;
            if (cudaOccupancyMaxActiveClusters(&nclusters, (const void*)k_beam_cl, &cfg) != cudaSuccess || nclusters < 1) {
                cudaGetLastError();
                continue;
            }
            *smem_out = Y.total;
            *big_out = big;
            return R;
        }
    }
    cudaGetLastError();
    return 0;
}

// Floats of the large-beam form's global factor copies (one a CTA).
size_t beam_cluster_fact_floats(int ns, int R) { return (size_t)R * cl_fact_floats(ns); }

// The running sums on arbitrary terms (a diagnostic of their exactness): one 256-thread block,
// the terms and sums in global memory.
__global__ void __launch_bounds__(256, 1) k_running_sums(const double* src, double* dst, int n, int* nserial) {
    __shared__ int flags[4];
    const int r = running_sums4<false>(src, n, dst, n, n, flags, NoIdle());
    if (threadIdx.x == 0) *nserial = r;
}
cudaError_t launch_running_sums(const double* src, double* dst, int n, int* nserial, cudaStream_t st) {
    k_running_sums<<<1, 256, 0, st>>>(src, dst, n, nserial);
    return cudaGetLastError();
}

void launch_beam_cluster(const BeamArgs& b, int R, size_t smem, cudaStream_t st, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(R);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = R;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 2 : 1;
    if (!g_batch) { cudaLaunchKernelEx(&cfg, k_beam_cl, b); return; }
    launch_batched<BeamArgs>((const void*)k_beam_cl, k_beam_cl_b, dim3(R), dim3(256), smem, pdl, b, [&](dim3 gz, const Batch<BeamArgs>& ba) {
        cfg.gridDim = gz;
        return cudaLaunchKernelEx(&cfg, k_beam_cl_b, ba);
    });
}

}  // namespace fsibe
