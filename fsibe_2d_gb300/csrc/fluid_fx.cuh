// fluid_fx.cuh -- the FP64 form's fused kernels (the map onto the reference is fluid.cuh's).
//
// Each transform of a block belongs to its own group of threads (fft_fx.cuh), with a row of shared
// memory for its exchanges; the pointwise work between transforms goes over all threads of the
// block, its operands and results in those rows.  A thread then holds one transform's eight values
// (some 80 registers where two or three transforms at once took 250), so an SM keeps three times
// the warps that wait on the integer chains, and a small grid, where the length of one thread's
// program is the time, runs a row's transforms side by side instead of one after another.
// Measured (GB300; both forms fixed point, three and two transforms a thread before): 256^2 k_nl_y 53 ->
// 17 us, k_press_x 47 -> 24, the step 232 -> 165; 64^2 k_nl_y 46 -> 16, the step 245 -> 193; 1024^2
// k_nl_y 160 -> 97, the step 533 -> 447 us.
// Included by fluid.cuh.
#pragma once

namespace fsibe {

template <int G> constexpr int fx_slots() { return 2 * (G >= 32 ? G / 32 : 1); }  // words a group

// ---- y pass --------------------------------------------------------------------------------
// Groups of k_nl_y_d.  The seven inverse transforms side by side and the pointwise work one or two
// elements a thread, as far as 1024 threads (and their registers) go.
template <int NY> constexpr int nl_y_groups() { return NY <= 512 ? 8 : (NY == 1024 ? 7 : (NY == 2048 ? 2 : 1)); }
template <int NY> constexpr int press_y_groups() { return NY <= 2048 ? 2 : 1; }
template <int NY, int NG> constexpr int nl_y_smem_d() {
    return (2 + NG) * padded_len(NY) * 16;
}
template <int NY, int NG> constexpr int press_y_smem_d() { return 2 * padded_len(NY) * 16; }

// k_nl_y: forward y of A and B, the AB2 / Euler update, the inverse-y outputs
template <int NY, int NG>
__global__ void __launch_bounds__(NG * NY / 8) k_nl_y_d(KArgs<double> a) {
    pdl_wait();     // the previous kernel of the stream has completed
    constexpr int G = NY / 8, T = NG * G, PLY = padded_len(NY), EPT = (NY + T - 1) / T;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned slots[NG * fx_slots<G>()];
    double2* rows = reinterpret_cast<double2*>(smem_raw);
    double2 *wn = rows, *ps = rows + PLY;  // omega and psi, element by element in A's and B's places
    const int kx = blockIdx.x, gi = threadIdx.x / G;
    const FxGroup gr{(int)threadIdx.x % G, gi + 1, slots + gi * fx_slots<G>()};
    const Geometry& g = a.g;
    const size_t row = (size_t)kx * NY;
    if (kx >= a.kcut) {
        // every mode of this row is removed by the 2/3 rule (see k_nl_y)
        for (int e = threadIdx.x; e < NY; e += T) a.W[row + e] = a.M[row + e] = make_double2(0.0, 0.0);
        return;
    }
    double2 v[8];
    for (int s = gi; s < 2; s += NG) {
        const double2* in = (s == 0 ? a.A : a.B) + row;
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = in[gr.t + m * G];
        fx_fft<NY, false>(v, rows + s * PLY, a.twY, gr, a.enorm);
#pragma unroll
        for (int m = 0; m < 8; ++m) rows[s * PLY + pad8(gr.t + m * G)] = v[m];
    }
    // the state, on its way while the forward transforms run in the first two groups
    double2 wo[EPT], mo[EPT];
#pragma unroll
    for (int q = 0; q < EPT; ++q) {
        const int ky = threadIdx.x + q * T;
        if (ky < NY) { wo[q] = a.W[row + ky]; mo[q] = a.M[row + ky]; }
    }
    const DevScalars* S = a.S;
    const double dt1 = S->dt1, b10 = S->b10, b11 = S->b11, etx = a.etab[kx], kx2 = __dmul_rn((double)(kx * kx), g.scalex);
    const bool expl = S->explicit_step != 0;
    const int cut = a.dcut[kx];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < EPT; ++q) {
        const int ky = threadIdx.x + q * T;
        if (ky >= NY) break;
        const int ks = signed_k(ky, NY), ka = ks < 0 ? -ks : ks;
        const bool nyq = (ky == NY / 2), keep = (g.idealis != 1) || (ka < cut);
        const double kys = __ldg(&a.kyd[ky]), E1 = etx * __ldg(&a.etab[g.hx + ka]);
        double2 N = csub<double>(rows[pad8(ky)], cimul<double>(rows[PLY + pad8(ky)], kys));
        if (nyq) N = make_double2(0.0, 0.0);
        const double2 Wo = wo[q], Mo = mo[q];
        double2 Wn;
        if (expl) Wn = make_double2((Wo.x + dt1 * N.x) * E1, (Wo.y + dt1 * N.y) * E1);
        else Wn = make_double2(((Wo.x + b10 * N.x) + b11 * Mo.x) * E1, ((Wo.y + b10 * N.y) + b11 * Mo.y) * E1);
        if (!keep || nyq) Wn = make_double2(0.0, 0.0);
        a.W[row + ky] = Wn;
        a.M[row + ky] = cscale<double>(N, E1);
        wn[pad8(ky)] = Wn;
        ps[pad8(ky)] = (kx == 0 && ky == 0) ? make_double2(0.0, 0.0) : over_k2(a, Wn, kx2, kx, ka);
    }
    __syncthreads();
    // spectra: 0 cofdy psi, 1 cofdx psi, 2 omega, 3 cofdy omega, 4 (kx^2 - ky^2) psi, 5 cofdx omega,
    // 6 d2psi/dxdy; without the stresses 0..3 and 5
    const double kxs = __ldg(&a.kxd[kx]);
    const int ntr = a.viscous ? 7 : 5;
    for (int s = gi; s < ntr; s += NG) {
        const int sp = (!a.viscous && s == 4) ? 5 : s;
        const double2* src = (sp == 2 || sp == 3 || sp == 5) ? wn : ps;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int ky = gr.t + m * G;
            const double2 x = src[pad8(ky)];
            const double kys = __ldg(&a.kyd[ky]);
            double2 val;
            if (sp == 2) val = x;
            else if (sp == 0 || sp == 3) val = cimul<double>(x, kys);
            else if (sp == 1 || sp == 5) val = cimul<double>(x, kxs);
            else val = cscale<double>(x, sp == 4 ? kxs * kxs - kys * kys : -(kxs * kys));
            v[m] = (ky == NY / 2) ? make_double2(0.0, 0.0) : val;
        }
        fx_fft<NY, true>(v, rows + (2 + gi) * PLY, a.twY, gr);
        double2* dst = (sp == 0 ? a.Tu : sp == 1 ? a.Tv : sp == 2 ? a.Tw : sp == 3 ? a.Tdy : sp == 4 ? a.Tsb : sp == 5 ? a.Tdx : a.Tsa) + row;
#pragma unroll
        for (int m = 0; m < 8; ++m) dst[gr.t + m * G] = v[m];
    }
}

// k_press_y: forward y of P1 and P2, divergence, Poisson divide, inverse y
template <int NY, int NG>
__global__ void __launch_bounds__(NG * NY / 8) k_press_y_d(KArgs<double> a) {
    pdl_wait();     // the previous kernel of the stream has completed
    constexpr int G = NY / 8, T = NG * G, PLY = padded_len(NY);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned slots[NG * fx_slots<G>()];
    double2* rows = reinterpret_cast<double2*>(smem_raw);
    const int kx = blockIdx.x, gi = threadIdx.x / G;
    const FxGroup gr{(int)threadIdx.x % G, gi + 1, slots + gi * fx_slots<G>()};
    const size_t row = (size_t)kx * NY;
    double2 v[8];
    for (int s = gi; s < 2; s += NG) {
        const double2* in = (s == 0 ? a.P1 : a.P2) + row;
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = in[gr.t + m * G];
        fx_fft<NY, false>(v, rows + s * PLY, a.twY, gr, a.enorm);
#pragma unroll
        for (int m = 0; m < 8; ++m) rows[s * PLY + pad8(gr.t + m * G)] = v[m];
    }
    const double kx2 = __dmul_rn((double)(kx * kx), a.g.scalex);
    __syncthreads();
    for (int ky = threadIdx.x; ky < NY; ky += T) {
        const int ks = signed_k(ky, NY);
        const double2 Q = cadd<double>(rows[pad8(ky)], cimul<double>(rows[PLY + pad8(ky)], __ldg(&a.kyd[ky])));
        const bool zero = (kx == 0 && ky == 0) || ky == NY / 2;
        rows[pad8(ky)] = zero ? make_double2(0.0, 0.0) : over_k2(a, Q, kx2, kx, ks < 0 ? -ks : ks);
    }
    __syncthreads();
    if (gi > 0) return;
#pragma unroll
    for (int m = 0; m < 8; ++m) v[m] = rows[pad8(gr.t + m * G)];
    fx_fft<NY, true>(v, rows + PLY, a.twY, gr);
#pragma unroll
    for (int m = 0; m < 8; ++m) a.Tq[row + gr.t + m * G] = v[m];
}

// ---- x pass ----------------------------------------------------------------------------------
// A block of TR rows and NF fields: group f TR + r transforms row r of field f.
template <int H, int TR, int NF>
struct XGroups {
    static constexpr int G = H / 8, PL = padded_len(H) + 1, BS = TR * PL, THREADS = NF * TR * G;
    static constexpr int SMEM = NF * BS * 16;
};
// fields of k_nl_x's parts: the derivatives (and, with the vorticity sponge, the vorticity), and
// what is transformed forward
template <int PART, int SPG> constexpr int nl_x_fields() { return (PART == NL_WHOLE || SPG == 1) ? 3 : 2; }
// A tile height for the FP64 kernels: tr when its block of three fields has a full warp and at most
// 1024 threads (with G > 32, then, at most 15 groups: the named barriers), else the default.
template <int H>
constexpr int xgroups_valid(int tr, int def) {
    return (tr >= 1 && (H / 8) * tr >= 32 && 3 * (H / 8) * tr <= 1024 && 3 * tr * (padded_len(H) + 1) * 16 <= 128 * 1024) ? tr : def;
}

template <int H, int TR, int NF>
struct XBlock {
    using X = XGroups<H, TR, NF>;
    double2* rows;
    FxGroup gr;
    int f, r;      // the group's field and row
    __device__ __forceinline__ XBlock(unsigned char* smem, unsigned* slots) {
        const int gi = threadIdx.x / X::G;
        rows = reinterpret_cast<double2*>(smem);
        gr = FxGroup{(int)threadIdx.x % X::G, gi + 1, slots + gi * fx_slots<X::G>()};
        f = gi / TR;
        r = gi % TR;
    }
    __device__ __forceinline__ double2* own() const { return rows + f * X::BS + r * X::PL; }
    // the group's half spectrum to a real row of pairs, in place
    __device__ __forceinline__ void to_real(const KArgs<double>& a) const {
        double2 v[8];
        fx_c2r<H>(own(), a.twR, a.twX, gr, v);
#pragma unroll
        for (int m = 0; m < 8; ++m) own()[pad8(gr.t + m * X::G)] = v[m];
    }
    __device__ __forceinline__ void to_half(const KArgs<double>& a) const {
        double2 v[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = own()[pad8(gr.t + m * X::G)];
        fx_sync<X::G>(gr);
        fx_r2c<H>(v, own(), a.twR, a.twX, gr);
    }
};

// cal_nlk's physical-space part (nl_x_tile)
template <int H, int TR, int PART, int SPG>
__device__ __forceinline__ void nl_x_tile_d(const KArgs<double>& a, const int iy0, unsigned* slots) {
    constexpr int NF = nl_x_fields<PART, SPG>();
    using X = XGroups<H, TR, NF>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int ny = a.g.ny;
    if (PART == NL_PENAL && (iy0 + TR - 1 < a.rect[2] || iy0 > a.rect[3])) return;
    const XBlock<H, TR, NF> B(smem_raw, slots);
    double2 *bufA = B.rows, *bufB = bufA + X::BS, *bufC = bufB + X::BS;
    // the penalization part adds to the advection part's A, loaded first
    constexpr int NLA = H * TR / X::THREADS;
    const int nout = a.kcut * TR;
    double2 av[NLA];
    if (PART == NL_PENAL) {
#pragma unroll
        for (int u = 0; u < NLA; ++u) {
            const int i = threadIdx.x + u * X::THREADS;
            if (i < nout) av[u] = a.A[(size_t)(i / TR) * ny + iy0 + i % TR];
        }
    } else {
        const int kin = a.explicit_step ? H : a.kcut;
        load_tileT<double, H, TR, X::PL>(bufA, a.Tdx, ny, iy0, kin);
        load_tileT<double, H, TR, X::PL>(bufB, a.Tdy, ny, iy0, kin);
        if (SPG == 1) load_tileT<double, H, TR, X::PL>(bufC, a.Tw, ny, iy0, kin);
        cp_async_wait_f();
        __syncthreads();
        if (B.f < (SPG == 1 ? 3 : 2)) B.to_real(a);
        __syncthreads();
    }
    const size_t roff = (size_t)iy0 * H;
    const double2 *u2 = reinterpret_cast<const double2*>(a.u) + roff, *v2 = reinterpret_cast<const double2*>(a.v) + roff;
    const double2 *k2 = reinterpret_cast<const double2*>(a.mask) + roff;
    const double2 *x2 = reinterpret_cast<const double2*>(a.mvx) + roff, *y2 = reinterpret_cast<const double2*>(a.mvy) + roff;
    const bool pen = PART != NL_ADVECT && a.penalize;
    for (int i = threadIdx.x; i < TR * H; i += X::THREADS) {
        const int o = (i / H) * X::PL + pad8(i % H);
        const double2 uu = u2[i], vv = v2[i];
        double2 px = make_double2(0.0, 0.0), py = px;
        if (pen) {
            const double2 kk = k2[i];
            if (!(is_zero(kk.x) && is_zero(kk.y))) {
                const double2 mx = x2[i], my = y2[i];
                px = make_double2(-kk.x * (uu.x - mx.x), -kk.y * (uu.y - mx.y));
                py = make_double2(-kk.x * (vv.x - my.x), -kk.y * (vv.y - my.y));
            }
            if (SPG == 2) {
                const double2 si = reinterpret_cast<const double2*>(a.s10)[roff + i];
                px = make_double2(px.x + si.x, px.y + si.y);
            }
        }
        if (PART == NL_PENAL) {
            bufA[o] = py;
            bufB[o] = px;
        } else {
            const double2 dx = bufA[o], dy = bufB[o];
            double2 w = make_double2(-uu.x * dx.x - vv.x * dy.x, -uu.y * dx.y - vv.y * dy.y);
            if (SPG == 1) {
                const double2 sg = reinterpret_cast<const double2*>(a.spg)[roff + i], om = bufC[o];
                w = make_double2(w.x - sg.x * om.x, w.y - sg.y * om.y);
            }
            bufA[o] = w;
            if (PART == NL_WHOLE) { bufB[o] = py; bufC[o] = px; }
        }
    }
    __syncthreads();
    if (B.f < (PART == NL_WHOLE ? 3 : (PART == NL_PENAL ? 2 : 1))) B.to_half(a);
    __syncthreads();
    // A = X(w) + i kx X(pen_y), B = X(pen_x) on the modes the update keeps (see nl_x_tile)
    if constexpr (PART == NL_PENAL) {
#pragma unroll
        for (int u = 0; u < NLA; ++u) {
            const int i = threadIdx.x + u * X::THREADS;
            if (i >= nout) break;
            const int s = (i % TR) * X::PL + pad8(i / TR);
            const size_t o = (size_t)(i / TR) * ny + iy0 + i % TR;
            a.A[o] = cadd<double>(av[u], cimul<double>(bufA[s], __ldg(&a.kxd[i / TR])));
            a.B[o] = bufB[s];
        }
    } else {
        for (int i = threadIdx.x; i < nout; i += X::THREADS) {
            const int s = (i % TR) * X::PL + pad8(i / TR);
            const size_t o = (size_t)(i / TR) * ny + iy0 + i % TR;
            if (PART == NL_WHOLE) {
                a.A[o] = cadd<double>(bufA[s], cimul<double>(bufB[s], __ldg(&a.kxd[i / TR])));
                a.B[o] = bufC[s];
            } else {
                a.A[o] = bufA[s];
                a.B[o] = make_double2(0.0, 0.0);
            }
        }
    }
}

template <int H, int TR, int PART, int SPG>
__global__ void __launch_bounds__(XGroups<H, TR, nl_x_fields<PART, SPG>()>::THREADS) k_nl_x_d(KArgs<double> a) {
    pdl_wait();     // the previous kernel of the stream has completed
    constexpr int NF = nl_x_fields<PART, SPG>();
    __shared__ unsigned slots[NF * TR * fx_slots<H / 8>()];
    if constexpr (PART == NL_ADVECT) {
        for (int tile = blockIdx.x; tile < a.g.ny / TR; tile += gridDim.x) {  // (see k_nl_x)
            nl_x_tile_d<H, TR, PART, SPG>(a, tile * TR, slots);
            __syncthreads();  // the next tile reuses the rows
        }
    } else {
        nl_x_tile_d<H, TR, PART, SPG>(a, blockIdx.x * TR, slots);
    }
}

// the viscous stresses (k_stress_x)
template <int H, int TR>
__device__ __forceinline__ void stress_tile_d(const KArgs<double>& a, const int iy0, unsigned* slots) {
    using X = XGroups<H, TR, 2>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const XBlock<H, TR, 2> B(smem_raw, slots);
    load_tileT<double, H, TR, X::PL>(B.rows, a.Tsa, a.g.ny, iy0, a.kcut);
    load_tileT<double, H, TR, X::PL>(B.rows + X::BS, a.Tsb, a.g.ny, iy0, a.kcut);
    cp_async_wait_f();
    __syncthreads();
    if (B.f > 1) return;
    double2 v[8];
    fx_c2r<H>(B.own(), a.twR, a.twX, B.gr, v);
    double2* out = reinterpret_cast<double2*>(B.f == 0 ? a.sa : a.sb) + (size_t)(iy0 + B.r) * H;
    const double c = B.f == 0 ? 2.0 * a.nu : a.nu;
#pragma unroll
    for (int m = 0; m < 8; ++m) out[B.gr.t + m * X::G] = make_double2(c * v[m].x, c * v[m].y);
}
template <int H, int TR>
__global__ void __launch_bounds__(XGroups<H, TR, 2>::THREADS) k_stress_x_d(KArgs<double> a) {
    __shared__ unsigned slots[2 * TR * fx_slots<H / 8>()];
    const int iy0 = blockIdx.x * TR;
    if (a.srows) {
        const int j0 = a.S->srow[0], j1 = a.S->srow[1];
        if (iy0 + TR - 1 < j0 || iy0 > j1) return;
    }
    stress_tile_d<H, TR>(a, iy0, slots);
}

// shared memory of k_press_x_d: the rows of three fields and the reduction's columns
template <int H, int TR> constexpr int press_x_smem_d() { return XGroups<H, TR, 3>::SMEM + RED_NSLOTS * XGroups<H, TR, 3>::THREADS * 8; }

// k_press_x: u, v and omega, the penalization, the sums, vor_mean, the pressure's right-hand side
template <int H, int TR>
__global__ void __launch_bounds__(XGroups<H, TR, 3>::THREADS) k_press_x_d(KArgs<double> a) {
    pdl_wait();     // the previous kernel of the stream has completed
    using X = XGroups<H, TR, 3>;
    constexpr int T = X::THREADS, NW = TR * X::G / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned slots[3 * TR * fx_slots<X::G>()];
    __shared__ double vm_w[2];
    const XBlock<H, TR, 3> B(smem_raw, slots);
    double2 *bufU = B.rows, *bufV = bufU + X::BS, *bufW = bufV + X::BS;
    double* cols = reinterpret_cast<double*>(smem_raw + X::SMEM);
    const int iy0 = blockIdx.x * TR, ny = a.g.ny;
    const DevScalars* S = a.S;
    if (threadIdx.x == 0) {  // time_avg_vort's weights
        const double time = S->time, dt1 = S->dt1;
        vm_w[0] = time / (time + dt1);
        vm_w[1] = dt1 / (time + dt1);
    }
    load_tileT<double, H, TR, X::PL>(bufU, a.Tu, ny, iy0, a.kcut);
    load_tileT<double, H, TR, X::PL>(bufV, a.Tv, ny, iy0, a.kcut);
    load_tileT<double, H, TR, X::PL>(bufW, a.Tw, ny, iy0, a.kcut);
    cp_async_wait_f();
    __syncthreads();
    B.to_real(a);
    __syncthreads();
    const size_t roff = (size_t)iy0 * H;
    double2 *u2 = reinterpret_cast<double2*>(a.u) + roff, *v2 = reinterpret_cast<double2*>(a.v) + roff;
    double2* vm2 = reinterpret_cast<double2*>(a.vor_mean) + roff;
    const double2 *k2 = reinterpret_cast<const double2*>(a.mask) + roff;
    const double2 *x2 = reinterpret_cast<const double2*>(a.mvx) + roff, *y2 = reinterpret_cast<const double2*>(a.mvy) + roff;
    const double U = S->mean_u_next, V = S->mean_v_next, ca = vm_w[0], cb = vm_w[1];
    const int ixmin = S->win[0], ixmax = S->win[1], iymin = S->win[2], iymax = S->win[3];
    double acc[RED_NSLOTS];
#pragma unroll
    for (int s = 0; s < RED_NSLOTS; ++s) acc[s] = 0.0;
    long long um = 0;  // bits of the largest |u|^2; NaN is passed over, as fmax does
    bool masked = false;
    // thirteen FP64 instructions a cell outside the mask, where the penalization and its sums add
    // nothing and are left out (a comparison or a conversion would take the FP64 pipe as long as an
    // addition: the mask's test and the maximum are on the bits)
    for (int i = threadIdx.x; i < TR * H; i += T) {
        const int rr = i / H, m = i % H, o = rr * X::PL + pad8(m), iy = iy0 + rr;
        const double2 kk = k2[i], vmo = vm2[i];
        const double2 ur = bufU[o], vr = bufV[o], w = bufW[o];
        const double2 uu = make_double2(ur.x + U, ur.y + U), vv = make_double2(-vr.x + V, -vr.y + V);
        u2[i] = uu;
        v2[i] = vv;
        const double uc[2] = {uu.x, uu.y}, vc[2] = {vv.x, vv.y}, wc[2] = {w.x, w.y};
        const double upc[2] = {ur.x, ur.y}, vpc[2] = {vr.x, vr.y};
        double px[2] = {0.0, 0.0}, py[2] = {0.0, 0.0};
        if (!(is_zero(kk.x) && is_zero(kk.y))) {
            masked = true;
            const double2 mx = x2[i], my = y2[i];
            const double kc[2] = {kk.x, kk.y}, xc[2] = {mx.x, mx.y}, yc[2] = {my.x, my.y};
            const bool in_rows = (iy >= iymin && iy <= iymax);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int ix = 2 * m + e;
                const double rx = uc[e] - xc[e], ry = vc[e] - yc[e];
                const double penx = kc[e] * rx, peny = kc[e] * ry;
                acc[RED_POROUS] += kc[e] * (rx * rx + ry * ry);
                acc[RED_INFLOW_SOLID] += kc[e] * (xc[e] * rx + yc[e] * ry);
                acc[RED_INFLOW_MEAN] += U * penx + V * peny;
                if (in_rows && ix >= ixmin && ix <= ixmax) {
                    acc[RED_DRAG_X] += penx;
                    acc[RED_DRAG_Y] += peny;
                    acc[RED_UNST_X] += xc[e] * kc[e];
                    acc[RED_UNST_Y] += yc[e] * kc[e];
                }
                px[e] = penx;
                py[e] = peny;
            }
        }
        const double vmc[2] = {vmo.x, vmo.y};
        double vmn[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            acc[RED_OMEGA2] += wc[e] * wc[e];
            acc[RED_KIN] += upc[e] * upc[e] + vpc[e] * vpc[e];
            acc[RED_SUM_U] += uc[e];
            acc[RED_SUM_V] += vc[e];
            const long long ub = __double_as_longlong(uc[e] * uc[e] + vc[e] * vc[e]);
            if (ub > um && ub <= 0x7ff0000000000000LL) um = ub;
            vmn[e] = vmc[e] * ca + wc[e] * cb;
            px[e] = px[e] - wc[e] * vc[e];
            py[e] = py[e] + wc[e] * uc[e];
        }
        vm2[i] = make_double2(vmn[0], vmn[1]);
        bufU[o] = make_double2(px[0], px[1]);
        bufV[o] = make_double2(py[0], py[1]);
    }
    acc[RED_UMAX2] = __longlong_as_double(um);
#pragma unroll
    for (int s = 0; s < RED_NSLOTS; ++s) cols[s * T + threadIdx.x] = acc[s];
    // a block without mask has zeros in the penalization's columns: they are not summed
    const bool any = __syncthreads_or(masked) != 0;
    if (B.f < 2) {
        if (a.pressure_on) B.to_half(a);  // the right-hand side's x and y parts
    } else {
        // the block's sums in a fixed order, one warp of the third field's groups a column
        const int w = (threadIdx.x - 2 * TR * X::G) >> 5, l = threadIdx.x & 31;
        for (int s = w; s < RED_NSLOTS; s += NW) {
            double v = 0.0;
            if (s == RED_UMAX2) {
                long long b = 0;
                for (int i = l; i < T; i += 32) b = max(b, __double_as_longlong(cols[s * T + i]));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
                v = __longlong_as_double(b);
            } else if (any || s == RED_OMEGA2 || s == RED_KIN || s == RED_SUM_U || s == RED_SUM_V) {
                for (int i = l; i < T; i += 32) v += cols[s * T + i];
                v = warp_sum<double>(v);
            }
            if (l == 0) a.red[(size_t)blockIdx.x * RED_NSLOTS + s] = v;
        }
        if (blockIdx.x == 0 && w == 0 && l == 0) a.S->nred = (int)gridDim.x;
    }
    __syncthreads();
    if (a.pressure_on) {
        for (int i = threadIdx.x; i < H * TR; i += T) {
            const int kx = i / TR, s = (i % TR) * X::PL + pad8(kx);
            const size_t o = (size_t)kx * ny + iy0 + i % TR;
            a.P1[o] = cimul<double>(bufU[s], __ldg(&a.kxd[kx]));
            a.P2[o] = bufV[s];
        }
    }
    if (a.viscous && !a.stress_split) {
        __syncthreads();
        stress_tile_d<H, TR>(a, iy0, slots);
    }
}

}  // namespace fsibe
