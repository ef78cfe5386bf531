// fluid_fx.cuh -- fused kernels with a group of threads a transform (the map onto the reference is
// fluid.cuh's): the FP64 form's y and x passes, and the FP32 form's x pass.
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
__device__ __forceinline__ void nl_y_d_run(const KArgs<double>& a) {
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
template <int NY, int NG>
__global__ void __launch_bounds__(NG * NY / 8) k_nl_y_d(const __grid_constant__ KArgs<double> a) { nl_y_d_run<NY, NG>(a); }
template <int NY, int NG>
__global__ void __launch_bounds__(NG * NY / 8) k_nl_y_d_b(const __grid_constant__ Batch<KArgs<double>> a) { nl_y_d_run<NY, NG>(a.a[blockIdx.z]); }

// k_press_y: forward y of P1 and P2, divergence, Poisson divide, inverse y
template <int NY, int NG>
__device__ __forceinline__ void press_y_d_run(const KArgs<double>& a) {
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
template <int NY, int NG>
__global__ void __launch_bounds__(NG * NY / 8) k_press_y_d(const __grid_constant__ KArgs<double> a) { press_y_d_run<NY, NG>(a); }
template <int NY, int NG>
__global__ void __launch_bounds__(NG * NY / 8) k_press_y_d_b(const __grid_constant__ Batch<KArgs<double>> a) { press_y_d_run<NY, NG>(a.a[blockIdx.z]); }

// ---- x pass (both forms) -----------------------------------------------------------------------
// A block of TR rows and NF fields, RG rows of every field at a time: group f RG + q transforms the
// rows q, q + RG, ... of field f.
template <typename R, int H, int TR, int RG, int NF>
struct XGroups {
    static constexpr int G = H / 8, PL = row_stride<R>(H, TR), BS = TR * PL, THREADS = NF * RG * G;
    static constexpr int SMEM = NF * BS * (int)sizeof(C2<R>);
    static_assert(TR % RG == 0, "whole rounds of rows");
};
// fields of k_nl_x's parts: the derivatives (and, with the vorticity sponge, the vorticity), and
// what is transformed forward
template <int PART, int SPG> constexpr int nl_x_fields() { return (PART == NL_WHOLE || SPG == 1) ? 3 : 2; }
// Rows at a time for a tile of tr: as many as give three fields at most 768 threads (with G > 32,
// then, at most 15 groups: the named barriers).
template <int H> constexpr int xgroups_rg(int tr) {
    int rg = tr;
    while (rg > 1 && 3 * (H / 8) * rg > 768) rg /= 2;
    return rg;
}
// A tile height of the group kernels: tr when its block has whole warps and three fields' rows fit
// shared memory, else the default.
template <typename R, int H>
constexpr int xgroups_valid(int tr, int def) {
    return (tr >= 1 && (H / 8) * xgroups_rg<H>(tr) >= 32 &&
            3 * tr * row_stride<R>(H, tr) * (int)sizeof(C2<R>) <= 128 * 1024) ? tr : def;
}

template <typename R, int H, int TR, int RG, int NF>
struct XBlock {
    using X = XGroups<R, H, TR, RG, NF>;
    C2<R>* rows;
    FxGroup gr;
    int f, r0;      // the group's field and first row
    __device__ __forceinline__ XBlock(unsigned char* smem, unsigned* slots) {
        const int gi = threadIdx.x / X::G;
        rows = reinterpret_cast<C2<R>*>(smem);
        gr = FxGroup{(int)threadIdx.x % X::G, gi + 1, slots + gi * fx_slots<X::G>()};
        f = gi / RG;
        r0 = gi % RG;
    }
    __device__ __forceinline__ C2<R>* row(int r) const { return rows + f * X::BS + r * X::PL; }
    // a half spectrum of the group's to its real row of pairs in registers (DX: FP32, of i kx times it)
    template <bool DX = false>
    __device__ __forceinline__ void c2r(const KArgs<R>& a, int r, C2<R> (&v)[8]) const {
        if constexpr (kIsF32<R>) f32_c2r<H, DX>(row(r), a.twR, a.twX, gr, v, (float)a.g.kxs);
        else fx_c2r<H>(row(r), a.twR, a.twX, gr, v);
    }
    template <bool DX = false>
    __device__ __forceinline__ void to_real(const KArgs<R>& a) const {  // in place, every row
        C2<R> v[8];
        for (int r = r0; r < TR; r += RG) {
            c2r<DX>(a, r, v);
#pragma unroll
            for (int m = 0; m < 8; ++m) row(r)[pad<R>(gr.t + m * X::G)] = v[m];
        }
    }
    __device__ __forceinline__ void to_half(const KArgs<R>& a) const {
        C2<R> v[8];
        for (int r = r0; r < TR; r += RG) {
#pragma unroll
            for (int m = 0; m < 8; ++m) v[m] = row(r)[pad<R>(gr.t + m * X::G)];
            fx_sync<X::G>(gr);
            if constexpr (kIsF32<R>) f32_r2c<H>(v, row(r), a.twR, a.twX, gr);
            else fx_r2c<H>(v, row(r), a.twR, a.twX, gr);
        }
    }
};

// cal_nlk's physical-space part (nl_x_tile)
template <typename R, int H, int TR, int RG, int PART, int SPG>
__device__ __forceinline__ void nl_x_tile_g(const KArgs<R>& a, const int iy0, unsigned* slots) {
    constexpr int NF = nl_x_fields<PART, SPG>();
    using X = XGroups<R, H, TR, RG, NF>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int ny = a.g.ny;
    if (PART == NL_PENAL && (iy0 + TR - 1 < a.rect[2] || iy0 > a.rect[3])) return;
    const XBlock<R, H, TR, RG, NF> B(smem_raw, slots);
    C2<R> *bufA = B.rows, *bufB = bufA + X::BS, *bufC = bufB + X::BS;
    // the penalization part adds to the advection part's A, loaded first
    constexpr int NLA = (H * TR + X::THREADS - 1) / X::THREADS;
    const int nout = a.kcut * TR;
    C2<R> av[NLA];
    if (PART == NL_PENAL) {
#pragma unroll
        for (int u = 0; u < NLA; ++u) {
            const int i = threadIdx.x + u * X::THREADS;
            if (i < nout) av[u] = a.A[(size_t)(i / TR) * ny + iy0 + i % TR];
        }
    } else {
        const int kin = a.explicit_step ? H : a.kcut;
        load_tileT<R, H, TR, X::PL>(bufA, kIsF32<R> ? a.Tw : a.Tdx, ny, iy0, kin);
        load_tileT<R, H, TR, X::PL>(bufB, a.Tdy, ny, iy0, kin);
        if (SPG == 1) load_tileT<R, H, TR, X::PL>(bufC, a.Tw, ny, iy0, kin);
        cp_async_wait_f();
        __syncthreads();
        if (kIsF32<R> && B.f == 0) B.template to_real<kIsF32<R>>(a);
        else if (B.f < (SPG == 1 ? 3 : 2)) B.to_real(a);
        __syncthreads();
    }
    const size_t roff = (size_t)iy0 * H;
    const C2<R> *u2 = reinterpret_cast<const C2<R>*>(a.u) + roff, *v2 = reinterpret_cast<const C2<R>*>(a.v) + roff;
    const C2<R> *k2 = reinterpret_cast<const C2<R>*>(a.mask) + roff;
    const C2<R> *x2 = reinterpret_cast<const C2<R>*>(a.mvx) + roff, *y2 = reinterpret_cast<const C2<R>*>(a.mvy) + roff;
    const bool pen = PART != NL_ADVECT && a.penalize;
    const R Uc = kIsF32<R> ? (R)a.S->mean_u_cur : (R)0, Vc = kIsF32<R> ? (R)a.S->mean_v_cur : (R)0;
    for (int i = threadIdx.x; i < TR * H; i += X::THREADS) {
        const int o = (i / H) * X::PL + pad<R>(i % H);
        C2<R> uu = u2[i], vv = v2[i];
        if (kIsF32<R>) {  // the stored velocity is the perturbation
            uu = mk<R>(uu.x + Uc, uu.y + Uc);
            vv = mk<R>(vv.x + Vc, vv.y + Vc);
        }
        C2<R> px = mk<R>(0, 0), py = px;
        if (pen) {
            const C2<R> kk = k2[i];
            if (!(is_zero(kk.x) && is_zero(kk.y))) {
                const C2<R> mx = x2[i], my = y2[i];
                px = mk<R>(-kk.x * (uu.x - mx.x), -kk.y * (uu.y - mx.y));
                py = mk<R>(-kk.x * (vv.x - my.x), -kk.y * (vv.y - my.y));
            }
            if (SPG == 2) {
                const C2<R> si = reinterpret_cast<const C2<R>*>(a.s10)[roff + i];
                px = mk<R>(px.x + si.x, px.y + si.y);
            }
        }
        if (PART == NL_PENAL) {
            bufA[o] = py;
            bufB[o] = px;
        } else {
            const C2<R> dx = bufA[o], dy = bufB[o];
            C2<R> w = mk<R>(-uu.x * dx.x - vv.x * dy.x, -uu.y * dx.y - vv.y * dy.y);
            if (SPG == 1) {
                const C2<R> sg = reinterpret_cast<const C2<R>*>(a.spg)[roff + i], om = bufC[o];
                w = mk<R>(w.x - sg.x * om.x, w.y - sg.y * om.y);
            }
            bufA[o] = w;
            if (PART == NL_WHOLE) { bufB[o] = py; bufC[o] = px; }
        }
    }
    __syncthreads();
    if (B.f < (PART == NL_WHOLE ? 3 : (PART == NL_PENAL ? 2 : 1))) B.to_half(a);
    __syncthreads();
    // the right-hand side only matters where the update keeps modes (kx < kcut): A = X(w) +
    // i kx X(pen_y), B = X(pen_x); the advection part writes X(w) and a zero B, the penalization part
    // adds its terms to that
    if constexpr (PART == NL_PENAL) {
#pragma unroll
        for (int u = 0; u < NLA; ++u) {
            const int i = threadIdx.x + u * X::THREADS;
            if (i >= nout) break;
            const int s = (i % TR) * X::PL + pad<R>(i / TR);
            const size_t o = (size_t)(i / TR) * ny + iy0 + i % TR;
            a.A[o] = cadd<R>(av[u], cimul<R>(bufA[s], kx_wave<R>(a, i / TR)));
            a.B[o] = bufB[s];
        }
    } else {
        for (int i = threadIdx.x; i < nout; i += X::THREADS) {
            const int s = (i % TR) * X::PL + pad<R>(i / TR);
            const size_t o = (size_t)(i / TR) * ny + iy0 + i % TR;
            if (PART == NL_WHOLE) {
                a.A[o] = cadd<R>(bufA[s], cimul<R>(bufB[s], kx_wave<R>(a, i / TR)));
                a.B[o] = bufC[s];
            } else {
                a.A[o] = bufA[s];
                a.B[o] = mk<R>(0, 0);
            }
        }
    }
}

template <typename R, int H, int TR, int PART, int SPG>
__device__ __forceinline__ void nl_x_g_run(const KArgs<R>& a) {
    pdl_wait();     // the previous kernel of the stream has completed
    constexpr int NF = nl_x_fields<PART, SPG>(), RG = xgroups_rg<H>(TR);
    __shared__ unsigned slots[NF * RG * fx_slots<H / 8>()];
    if constexpr (PART == NL_ADVECT) {
        // the advection part runs beside the mask kernels on fewer blocks than tiles (the
        // launch gives one a SM), each taking tiles in turn, so that the raster launched after
        // it still finds room on every SM
        for (int tile = blockIdx.x; tile < a.g.ny / TR; tile += gridDim.x) {
            nl_x_tile_g<R, H, TR, RG, PART, SPG>(a, tile * TR, slots);
            __syncthreads();  // the next tile reuses the rows
        }
    } else {
        nl_x_tile_g<R, H, TR, RG, PART, SPG>(a, blockIdx.x * TR, slots);
    }
}
template <typename R, int H, int TR, int PART, int SPG>
__global__ void __launch_bounds__(XGroups<R, H, TR, xgroups_rg<H>(TR), nl_x_fields<PART, SPG>()>::THREADS) k_nl_x_g(const __grid_constant__ KArgs<R> a) { nl_x_g_run<R, H, TR, PART, SPG>(a); }
template <typename R, int H, int TR, int PART, int SPG>
__global__ void __launch_bounds__(XGroups<R, H, TR, xgroups_rg<H>(TR), nl_x_fields<PART, SPG>()>::THREADS) k_nl_x_g_b(const __grid_constant__ Batch<KArgs<R>> a) { nl_x_g_run<R, H, TR, PART, SPG>(a.a[blockIdx.z]); }

// The viscous stresses (NavierStokes.f90:354-370: 2 nu d2psi/dxdy, nu (d2psi/dy2 - d2psi/dx2))
// to physical space, beside k_press_x on another stream: only GetForces reads them.  With
// a.srows set, a block whose rows no stencil of the forces reaches (rows j - 4 .. j + 4 of the
// stress points' cells j, BeamForces.f90:105-124, which lie within the stress points' offset
// of the beam's y range; k_step_begin forms the range into S->srow) leaves them.
template <typename R, int H, int TR, int RG>
__device__ __forceinline__ void stress_tile_g(const KArgs<R>& a, const int iy0, unsigned* slots) {
    using X = XGroups<R, H, TR, RG, 2>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const XBlock<R, H, TR, RG, 2> B(smem_raw, slots);
    load_tileT<R, H, TR, X::PL>(B.rows, kIsF32<R> ? a.Tu : a.Tsa, a.g.ny, iy0, a.kcut);  // FP32: du/dx = i kx Tu
    load_tileT<R, H, TR, X::PL>(B.rows + X::BS, a.Tsb, a.g.ny, iy0, a.kcut);
    cp_async_wait_f();
    __syncthreads();
    if (B.f > 1) return;
    const R c = B.f == 0 ? (R)(2.0 * a.nu) : (R)a.nu;
    C2<R> v[8];
    for (int r = B.r0; r < TR; r += RG) {
        if (kIsF32<R> && B.f == 0) B.template c2r<kIsF32<R>>(a, r, v);
        else B.c2r(a, r, v);
        C2<R>* out = reinterpret_cast<C2<R>*>(B.f == 0 ? a.sa : a.sb) + (size_t)(iy0 + r) * H;
#pragma unroll
        for (int m = 0; m < 8; ++m) out[B.gr.t + m * X::G] = mk<R>(c * v[m].x, c * v[m].y);
    }
}
template <typename R, int H, int TR>
__global__ void __launch_bounds__(XGroups<R, H, TR, xgroups_rg<H>(TR), 2>::THREADS) k_stress_x_g(KArgs<R> a) {
    constexpr int RG = xgroups_rg<H>(TR);
    __shared__ unsigned slots[2 * RG * fx_slots<H / 8>()];
    const int iy0 = blockIdx.x * TR;
    if (a.srows) {
        const int j0 = a.S->srow[0], j1 = a.S->srow[1];
        if (iy0 + TR - 1 < j0 || iy0 > j1) return;
    }
    stress_tile_g<R, H, TR, RG>(a, iy0, slots);
}

// k_press_x_g's sums: the columns every cell adds to, and those of the penalization (INFLOW_MEAN as
// the sums of chi (u - u_s) and chi (v - v_s) in the FP32 form)
constexpr int PXC_ALL = 5, PXC_PEN = 8;
enum { PX_OMEGA2 = 0, PX_KIN, PX_SUM_U, PX_SUM_V, PX_UMAX2, PX_POROUS, PX_INFLOW, PX_PENX, PX_PENY, PX_DRAGX, PX_DRAGY, PX_UNSTX, PX_UNSTY };
// shared memory: the rows of three fields, and the threads' columns (one thread's are never
// reduced before another's are written: they have their own place)
template <typename R, int H, int TR> constexpr int press_x_smem_g() {
    using X = XGroups<R, H, TR, xgroups_rg<H>(TR), 3>;
    return X::SMEM + (PXC_ALL + PXC_PEN) * X::THREADS * (int)sizeof(R);
}

// k_press_x: u, v and omega, the penalization, the sums, vor_mean, the pressure's right-hand side
template <typename R, int H, int TR>
__device__ __forceinline__ void press_x_g_run(const KArgs<R>& a) {
    pdl_wait();     // the previous kernel of the stream has completed
    constexpr int RG = xgroups_rg<H>(TR);
    using X = XGroups<R, H, TR, RG, 3>;
    constexpr int T = X::THREADS, NW = RG * X::G / 32;
    constexpr bool F32 = kIsF32<R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned slots[3 * RG * fx_slots<X::G>()];
    __shared__ R vm_w[2];
    __shared__ double red_s[PXC_ALL + PXC_PEN];
    const XBlock<R, H, TR, RG, 3> B(smem_raw, slots);
    C2<R> *bufU = B.rows, *bufV = bufU + X::BS, *bufW = bufV + X::BS;
    R* cols = reinterpret_cast<R*>(smem_raw + X::SMEM);
    const int iy0 = blockIdx.x * TR, ny = a.g.ny;
    const DevScalars* S = a.S;
    if (threadIdx.x == 0) {  // time_avg_vort's weights
        const double time = S->time, dt1 = S->dt1;
        vm_w[0] = (R)(time / (time + dt1));
        vm_w[1] = (R)(dt1 / (time + dt1));
    }
    load_tileT<R, H, TR, X::PL>(bufU, a.Tu, ny, iy0, a.kcut);
    load_tileT<R, H, TR, X::PL>(bufV, a.Tv, ny, iy0, a.kcut);
    load_tileT<R, H, TR, X::PL>(bufW, a.Tw, ny, iy0, a.kcut);
    cp_async_wait_f();
    __syncthreads();
    B.to_real(a);
    __syncthreads();
    const size_t roff = (size_t)iy0 * H;
    C2<R> *u2 = reinterpret_cast<C2<R>*>(a.u) + roff, *v2 = reinterpret_cast<C2<R>*>(a.v) + roff;
    C2<R>* vm2 = reinterpret_cast<C2<R>*>(a.vor_mean) + roff;
    const C2<R> *k2 = reinterpret_cast<const C2<R>*>(a.mask) + roff;
    const C2<R> *x2 = reinterpret_cast<const C2<R>*>(a.mvx) + roff, *y2 = reinterpret_cast<const C2<R>*>(a.mvy) + roff;
    const double Ud = S->mean_u_next, Vd = S->mean_v_next;
    const R U = (R)Ud, V = (R)Vd, ca = vm_w[0], cb = vm_w[1];
    const int ixmin = S->win[0], ixmax = S->win[1], iymin = S->win[2], iymax = S->win[3];
    R acc[PXC_ALL + PXC_PEN];
#pragma unroll
    for (int s = 0; s < PXC_ALL + PXC_PEN; ++s) acc[s] = (R)0;
    long long um = 0;  // FP64: bits of the largest |u|^2; NaN is passed over, as fmax does
    bool masked = false;
    // Outside the mask the penalization and its sums add nothing and are left out.  In FP64 that leaves
    // thirteen FP64 instructions a cell (a comparison or a conversion would take the FP64 pipe as long
    // as an addition: the mask's test and the maximum are on the bits).
    for (int i = threadIdx.x; i < TR * H; i += T) {
        const int rr = i / H, m = i % H, o = rr * X::PL + pad<R>(m), iy = iy0 + rr;
        const C2<R> kk = k2[i], vmo = vm2[i];
        const C2<R> ur = bufU[o], vr = bufV[o], w = bufW[o];
        const C2<R> uu = mk<R>(ur.x + U, ur.y + U), vv = mk<R>(-vr.x + V, -vr.y + V);
        // the FP32 form stores the perturbation (the mean flow stays in FP64 scalars)
        u2[i] = F32 ? ur : uu;
        v2[i] = F32 ? mk<R>(-vr.x, -vr.y) : vv;
        const R uc[2] = {uu.x, uu.y}, vc[2] = {vv.x, vv.y}, wc[2] = {w.x, w.y};
        const R upc[2] = {ur.x, ur.y}, vpc[2] = {vr.x, vr.y};
        R px[2] = {0, 0}, py[2] = {0, 0};
        if (!(is_zero(kk.x) && is_zero(kk.y))) {
            masked = true;
            const C2<R> mx = x2[i], my = y2[i];
            const R kc[2] = {kk.x, kk.y}, xc[2] = {mx.x, mx.y}, yc[2] = {my.x, my.y};
            const bool in_rows = (iy >= iymin && iy <= iymax);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int ix = 2 * m + e;
                const R rx = uc[e] - xc[e], ry = vc[e] - yc[e];
                const R penx = kc[e] * rx, peny = kc[e] * ry;
                acc[PX_POROUS] += kc[e] * (rx * rx + ry * ry);
                acc[PX_INFLOW] += kc[e] * (xc[e] * rx + yc[e] * ry);
                acc[PX_PENX] += penx;
                acc[PX_PENY] += peny;
                if (in_rows && ix >= ixmin && ix <= ixmax) {
                    acc[PX_DRAGX] += penx;
                    acc[PX_DRAGY] += peny;
                    acc[PX_UNSTX] += xc[e] * kc[e];
                    acc[PX_UNSTY] += yc[e] * kc[e];
                }
                px[e] = penx;
                py[e] = peny;
            }
        }
        const R vmc[2] = {vmo.x, vmo.y};
        R vmn[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            acc[PX_OMEGA2] += wc[e] * wc[e];
            acc[PX_KIN] += upc[e] * upc[e] + vpc[e] * vpc[e];
            acc[PX_SUM_U] += uc[e];
            acc[PX_SUM_V] += vc[e];
            const R q2 = uc[e] * uc[e] + vc[e] * vc[e];
            if constexpr (F32) {
                acc[PX_UMAX2] = fmaxf(acc[PX_UMAX2], q2);
            } else {
                const long long ub = __double_as_longlong(q2);
                if (ub > um && ub <= 0x7ff0000000000000LL) um = ub;
            }
            vmn[e] = vmc[e] * ca + wc[e] * cb;
            px[e] = px[e] - wc[e] * vc[e];
            py[e] = py[e] + wc[e] * uc[e];
        }
        vm2[i] = mk<R>(vmn[0], vmn[1]);
        bufU[o] = mk<R>(px[0], px[1]);
        bufV[o] = mk<R>(py[0], py[1]);
    }
    if constexpr (!F32) acc[PX_UMAX2] = __longlong_as_double(um);
    // a block without mask has zeros in the penalization's columns: they are not summed
    const bool any = __syncthreads_or(masked) != 0;
    const int ncol = any ? PXC_ALL + PXC_PEN : PXC_ALL;
#pragma unroll
    for (int s = 0; s < PXC_ALL + PXC_PEN; ++s)
        if (s < ncol) cols[s * T + threadIdx.x] = acc[s];
    __syncthreads();
    if (B.f < 2) {
        if (a.pressure_on) B.to_half(a);  // the right-hand side's x and y parts
    } else {
        // the block's sums in a fixed order, one warp of the third field's groups a column
        const int w = (threadIdx.x - 2 * RG * X::G) >> 5, l = threadIdx.x & 31;
        for (int s = w; s < PXC_ALL + PXC_PEN; s += NW) {
            double v = 0.0;
            if (s < ncol) {
                if constexpr (F32) {
                    v = col_reduce_ff(cols + s * T, T, s == PX_UMAX2);
                } else if (s == PX_UMAX2) {
                    long long b = 0;
                    for (int i = l; i < T; i += 32) b = max(b, __double_as_longlong(cols[s * T + i]));
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
                    v = __longlong_as_double(b);
                } else {
                    for (int i = l; i < T; i += 32) v += cols[s * T + i];
                    v = warp_sum<double>(v);
                }
            }
            if (l == 0) red_s[s] = v;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double* out = a.red + (size_t)blockIdx.x * RED_NSLOTS;
        out[RED_OMEGA2] = red_s[PX_OMEGA2]; out[RED_KIN] = red_s[PX_KIN];
        out[RED_POROUS] = red_s[PX_POROUS]; out[RED_INFLOW_SOLID] = red_s[PX_INFLOW];
        out[RED_INFLOW_MEAN] = any ? Ud * red_s[PX_PENX] + Vd * red_s[PX_PENY] : 0.0;
        out[RED_SUM_U] = red_s[PX_SUM_U]; out[RED_SUM_V] = red_s[PX_SUM_V];
        out[RED_DRAG_X] = red_s[PX_DRAGX]; out[RED_DRAG_Y] = red_s[PX_DRAGY];
        out[RED_UNST_X] = red_s[PX_UNSTX]; out[RED_UNST_Y] = red_s[PX_UNSTY];
        out[RED_UMAX2] = red_s[PX_UMAX2];
        if (blockIdx.x == 0) a.S->nred = (int)gridDim.x;
    }
    if (a.pressure_on) {
        for (int i = threadIdx.x; i < H * TR; i += T) {
            const int kx = i / TR, s = (i % TR) * X::PL + pad<R>(kx);
            const size_t o = (size_t)kx * ny + iy0 + i % TR;
            a.P1[o] = cimul<R>(bufU[s], kx_wave<R>(a, kx));
            a.P2[o] = bufV[s];
        }
    }
    if (a.viscous && !a.stress_split) {
        __syncthreads();
        stress_tile_g<R, H, TR, RG>(a, iy0, slots);
    }
}
template <typename R, int H, int TR>
__global__ void __launch_bounds__(XGroups<R, H, TR, xgroups_rg<H>(TR), 3>::THREADS) k_press_x_g(const __grid_constant__ KArgs<R> a) { press_x_g_run<R, H, TR>(a); }
template <typename R, int H, int TR>
__global__ void __launch_bounds__(XGroups<R, H, TR, xgroups_rg<H>(TR), 3>::THREADS) k_press_x_g_b(const __grid_constant__ Batch<KArgs<R>> a) { press_x_g_run<R, H, TR>(a.a[blockIdx.z]); }

}  // namespace fsibe
