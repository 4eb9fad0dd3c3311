// ins and cd element residual, straight triangles, sum-factorised with one lane per triangle.
//
// tri_hp::rsdl's element loop (tri_hp/nstage.cpp:52-73: ugtouht, element_rsdl, lftog) with
// tri_hp_ins::element_rsdl's straight-element branch (tri_hp/ins/rsdl.cpp:259-433) or
// tri_hp_cd::element_rsdl (tri_hp/cd/rsdl.cpp:14-154, CONST_A) and the tri_basis operators they
// call (proj.cpp:22-119, intgrt.cpp:81-158, derivr / derivs proj.cpp:339-402), FP64 or FP32, plain
// or correction form.
//
// A CTA takes batches of 32 triangles, lane = triangle, and has one warp per eta point j: a
// thread owns the line (triangle, j) of the tensor-product points. Everything that is not per
// triangle -- mode, point, table entry -- is then uniform across a warp, so the basis tables are
// constant-bank operands of the FMAs, shared-memory rows of 32 lanes have no bank conflicts, and
// no index is computed per lane; the point data of a line stay in its thread's registers.
//   gather   modes -> U[var][mode][lane] (cp.async, one batch ahead; the connectivity two ahead)
//   proj     the thread's column sums over the modes (value, d/deta), then its G points
//   strong   x-direction part of the strong residual in registers; the s fluxes are exchanged
//            through shared memory for the eta-direction part (warp = x point i there)
//   SUPG     point by point
//   intgrtrs per part: x-direction sums of the thread's line -> A, B [var][column][j], exchange,
//            then every warp sums its share of the modes over j
//   lftog    results staged [mode][var][lane], written with consecutive threads on
//            consecutive addresses of the assembly slots (or atomics)
// Why vector FMAs: on B200 the FP64 tensor instruction runs on the FP64 pipe at its rate (measured
// 37.0 TFLOP/s against 34.5 for DFMA, and 31 in sum when mixed), so the dense per-point operators
// that a fragment needs (98k flops per triangle at p = 6 with the padding) lose to the
// sum-factorised form (43.6k as the reference's loops are counted). Measured, FP64, 131k triangles,
// full residual, against two triangles per warp on mma.m8n8k4.f64: p = 3 157 -> 91 us, p = 4
// 308 -> 168, p = 5 503 -> 249, p = 6 719 -> 409, p = 8 1884 -> 1236; p = 2 against the scalar warp
// kernel 197 -> 50 (the boundary fluxes, a kernel of their own before, included). Bound by latency
// (fixed-length instructions, shared memory) at the 7 to 16 warps an SM that fit: at p = 6 the FP64
// pipe is 36 % busy and the schedulers issue in 33 % of the cycles, at p = 3 the pipe is 41 % busy.
// FP32: the same form beats TF32 fragments (mma.m16n8k8, operands rounded to 10 bits), and in
// full FP32: an update of the FP32 smoother, 131k triangles, p = 3 728 -> 464 us, p = 4 1202 ->
// 796, p = 6 2625 -> 1901, p = 8 7305 -> 3835, p = 2 against the scalar warp kernel 670 -> 236; in
// plain form against the scalar warp kernel p = 6 4475 -> 1741. Half of the instructions are FMAs.
// cd against the scalar warp kernel, an FP64 update of 80k triangles: p = 1 126 -> 68 us (with
// k_vert_p1), p = 2 282 -> 118, p = 4 739 -> 308; p = 6 of 20k 626 -> 320. (The pairs at the choices
// below were measured together, when each choice was made.)
#pragma once
#include <utility>
#include "hp_line.h"

namespace hpb {

template <typename R, int P, int PHYS, bool DIFF, bool RE>
struct LineCfg {
    static constexpr int G = P + 1, GG = G * G, X = P + 2, T = (P + 1) * (P + 2) / 2, SM = P - 1,
                         IM = (P - 1) * (P - 2) / 2, BM = 3 * P, NV = PHYS == 1 ? 3 : 1;
    static constexpr int NTHR = 32 * G;
    // FP64, p = 6, a stage without the real part: the modes are gathered into the exchange area, once
    // that has been read, instead of into an area of their own, so that a second CTA fits an SM (its
    // 128 registers a thread hold what such a stage keeps; 131k triangles: 246 -> 160 us). With the
    // real part the point data do not fit: 404 us with two CTAs against 413, 30 against 22 us on 2k
    // triangles. p = 7, 8 need more than half of the shared memory, p <= 5 have two CTAs as it is.
    static constexpr bool TIGHT = PHYS == 1 && G == 7 && sizeof(R) == 8 && !RE;
    static constexpr int OUT = 0;                           // results [NV T][33]
    static constexpr int U = NV * T * 33;                   // gathered modes [NV T][33]
    static constexpr int EX = TIGHT ? U : 2 * NV * T * 33;  // s fluxes [NV][G][G][32], then A, B [NV][2][X][G][32]
    static constexpr int LEN = EX + 2 * NV * X * G * 32;
    static constexpr int IDX = 16 * 32;  // connectivity of a batch: pnt, seg, sgn, vpos, spos [32][3], tri_cv [32]
    static constexpr int LPS = SM > 0 ? SM * NV : 1, LPI = IM > 0 ? IM * NV : 1;  // values of a side, of an interior
    static constexpr int XH = NV == 1 ? X : (X + 1) / 2;  // columns whose x sums share the registers
    static constexpr int SMEM = LEN * (int)sizeof(R) + 3 * IDX * 4;
    static constexpr int by_smem = 227 * 1024 / (SMEM + 1024);
    // CTAs an SM, as many as leave the point data in registers (ins, 131k triangles, FP64: p = 4 with
    // 1, 2, 3 CTAs 269, 198, 171 us, although 3 spill a little; p = 5 with 1, 2: 347, 246).
    // FP32, an update at 131k triangles: p = 2 with 4, 6, 8 CTAs 292, 279, 265 us; p = 8 with 1, 2:
    // 4932, 4052
    static constexpr int by_cd = G <= 2 ? 8 : G <= 4 ? 6 : G == 5 ? 5 : G == 6 ? 4 : G == 7 ? 3 : 2;
    static constexpr int by_regs = PHYS == 0 ? (sizeof(R) == 8 ? by_cd : 2 * by_cd)
                                 : sizeof(R) == 8
                                     ? (G == 2 ? 8 : G == 3 ? 5 : G == 4 ? 4 : G == 5 ? 3 : G == 6 || TIGHT ? 2 : 1)
                                     : (G == 2 ? 12 : G == 3 ? 8 : G <= 5 ? 5 : G == 6 ? 4 : G == 7 ? 3 : 2);
    static constexpr int MINB = by_smem < by_regs ? (by_smem < 1 ? 1 : by_smem) : by_regs;
};

template <typename R>
struct alignas(2 * sizeof(R)) R2 {
    R x, y;
};

// Tables of one (precision, p), a kernel parameter. The first index of g and w is the warp's (its
// eta point; the mode it sums), the others are compile-time. Every entry is used for the three
// variables at once: an FP64 FMA whose constant is loaded for it alone runs at under half rate
// (measured: 15 TFLOP/s with one use of each constant, 30 with three).
template <typename R, int P>
struct LineTab {
    static constexpr int G = P + 1, X = P + 2, T = (P + 1) * (P + 2) / 2;
    R2<R> g[G][T];                     // proj, mode sums: gn, dgn
    R2<R> w[T][G];                     // intgrtrs, eta-direction: gnwtnn0, dgnwtn, with its minus sign
    R gx[G][X], dgx[G][X];             // proj, column sums to point i
    R ar[G][G], as1[G][G], as2[G][G];  // derivr / derivs: 1D derivative operators
    R dgxw[X][G], gxw[X][G];           // intgrtrs, x-direction
    R x0[G], n0[G], src[T];            // src: intgrt of 1 against the modes
    // intgrtrs, eta-direction: warp w sums items iptr[w] .. iptr[w + 1] - 1; an item is the column
    // icol and its modes mode[ifst[item] .. ifst[item + 1] - 1]
    unsigned char iptr[G + 1], icol[G + X], ifst[G + X + 1], mode[T];
    unsigned char odd[T];  // the side of an odd side mode, 3 for the other modes
};

// What the kernel takes of Phys. ins: rho, mu, nu2 = 2 mu / rho, adis, gfloor (mu + bd0 == 0); cd:
// rhocv, kcond, the velocity, the source.
struct LinePar {
    double beta, omb, rho, mu, nu2, adis, rhocv, kcond, ax, ay, src;
    int gfloor;
};

// c / sqrt(gam). FP64 by rsqrt: over gam from 1e-8 to 1e12 its error is 0.425 ulp rms, 1.48 at most,
// that of the quotient 0.426 and 1.46, and the full residual takes 446 us instead of 459 at p = 6, 193
// instead of 197 at p = 4 (131k triangles), though 367 instead of 343 at p = 8 (33k).
template <typename R>
__device__ __forceinline__ R line_tau0(R c, R gam);
template <>
__device__ __forceinline__ double line_tau0<double>(double c, double gam) { return c * rsqrt(gam); }
template <>
__device__ __forceinline__ float line_tau0<float>(float c, float gam) { return c / sqrtf(gam); }

// f(0), ..., f(N - 1) with compile-time arguments: the column of a mode is then a constant, so the
// column sums stay in registers (a loop does not fold ModeCols::col beyond p = 4)
template <typename F, int... M>
__device__ __forceinline__ void each_mode(F &&f, std::integer_sequence<int, M...>) {
    (f(std::integral_constant<int, M>{}), ...);
}

// An optimisation barrier on a register: what depends on it is computed again.
__device__ __forceinline__ void opaque(double &x) { asm volatile("" : "+d"(x)); }
__device__ __forceinline__ void opaque(float &x) { asm volatile("" : "+f"(x)); }

// x with its sign changed where bit (0 or the sign bit) is set
__device__ __forceinline__ void flip_if(double &x, int bit) {
    x = __hiloint2double(__double2hiint(x) ^ bit, __double2loint(x));
}
__device__ __forceinline__ void flip_if(float &x, int bit) { x = __int_as_float(__float_as_int(x) ^ bit); }

template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(BYTES));
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Point values (u, v) of the base state of the correction form, State::bpt, in batches of 32
// triangles [ceil(ntri / 32)][2][G^2][32] (lanes past the last triangle repeat it): the projection
// (proj.cpp:121-186 as dense sums) of the gathered base modes, one thread per (triangle, variable).
template <int P>
__global__ void k_base_points(const DevTables<float, P> *__restrict__ tb, Mesh mesh, const float *__restrict__ ubv,
                              const float *__restrict__ ubs, const float *__restrict__ ubi, float *bpt) {
    constexpr int G = P + 1, GG = G * G, T = (P + 1) * (P + 2) / 2, SM = (P > 1 ? P - 1 : 1),
                  IM = (P - 1) * (P - 2) / 2, BM = 3 * P, NV = 3;
    const long item = (long)blockIdx.x * blockDim.x + threadIdx.x;  // (batch, variable, lane)
    const int b = (int)(item >> 6), n = (int)(item >> 5) & 1, lane = (int)item & 31;
    if (b >= (mesh.ntri + 31) / 32) return;
    const int t = min(b * 32 + lane, mesh.ntri - 1);
    float lin[T];
#pragma unroll
    for (int m = 0; m < T; ++m) {
        float val;
        if (m < 3) {
            val = ubv[mesh.tri_pnt[3 * t + m] * NV + n];
        } else if (m < BM) {
            const int i = (m - 3) / SM, k = (m - 3) - i * SM;
            val = ubs[(mesh.tri_seg[3 * t + i] * SM + k) * NV + n];
            if ((k & 1) && mesh.tri_sgn[3 * t + i] < 0) val = -val;
        } else {
            val = ubi[((size_t)t * IM + (m - BM)) * NV + n];
        }
        lin[m] = val;
    }
    float *out = bpt + ((size_t)b * 2 + n) * GG * 32 + lane;
    for (int q = 0; q < GG; ++q) {
        const int i = q / G, j = q - i * G;
        float acc = 0.f;
#pragma unroll
        for (int m = 0; m < T; ++m) acc += lin[m] * tb->gn[j][m] * tb->gx[i][ModeCols<P>::col(m)];
        out[q * 32] = acc;
    }
}

// Boundary fluxes of bdry_ins::generic (hp_boundary.cpp:973-1049, ins/bdry_ins.h:35-50) of the
// kernel's share of the boundary edges, 16 lanes an edge: lane k < G evaluates the flux at Gauss
// point k, lane m < SM + 2 integrates it against the side's function m (end 0, end 1, side modes).
// It runs in the element kernel before its first batch, whose copies are in flight meanwhile: as a
// kernel of its own, one thread an edge, it was 7 to 14 us of every stage.
template <typename R, int P, bool DIFF>
__device__ __forceinline__ void line_bdry_flux(const DevTables<R, P> *__restrict__ tb, const Mesh &mesh,
                                               const State<R> &st, R rho) {
    constexpr int G = P + 1, SM = P - 1, NM = SM + 2;
    const int l = threadIdx.x & 15, per = blockDim.x >> 4, lg = l < G ? l : 0, lm = l < NM ? l : 0;
    const unsigned mask = 0xffffu << (threadIdx.x & 16);
    // from the last CTA on: those have a batch less when the batches do not come out even
    for (int e = (gridDim.x - 1 - blockIdx.x) * per + (threadIdx.x >> 4); e < mesh.nbseg; e += gridDim.x * per) {
        if ((mesh.bkind[e] & (0xF << 8)) != (1 << 8)) continue;
        const int sd = mesh.bseg[e], v0 = mesh.seg_pnt[2 * sd], v1 = mesh.seg_pnt[2 * sd + 1];
        // normal at the lane's point (straight side, or its position modes: crdtocht1d)
        R dx = (R)mesh.pnts[2 * v0] * tb->dgx[lg][1] + (R)mesh.pnts[2 * v1] * tb->dgx[lg][2];
        R dy = (R)mesh.pnts[2 * v0 + 1] * tb->dgx[lg][1] + (R)mesh.pnts[2 * v1 + 1] * tb->dgx[lg][2];
        if (mesh.bcrd)
            for (int m = 0; m < SM; ++m) {
                dx += (R)mesh.bcrd[((size_t)e * SM + m) * 2] * tb->dgx[lg][m + 3];
                dy += (R)mesh.bcrd[((size_t)e * SM + m) * 2 + 1] * tb->dgx[lg][m + 3];
            }
        auto value = [&](const R *uv, const R *us, int n) {
            R a = uv[(size_t)v0 * 3 + n] * tb->gx[lg][1] + uv[(size_t)v1 * 3 + n] * tb->gx[lg][2];
#pragma unroll
            for (int m = 0; m < SM; ++m) a += us[((size_t)sd * SM + m) * 3 + n] * tb->gx[lg][m + 3];
            return a;
        };
        const R u0 = value(st.ugv, st.ugs, 0), u1 = value(st.ugv, st.ugs, 1);
        const R fm = rho * (u0 * dy - u1 * dx);
        R f[3] = {(R)0, (R)0, fm};
        if constexpr (DIFF) {  // F(b + d) - F(b); the boundary pressure cancels
            const R b0 = value(st.ubv, st.ubs, 0), b1 = value(st.ubv, st.ubs, 1), mb = rho * (b0 * dy - b1 * dx);
            f[0] = fm * (b0 + u0) + mb * u0;
            f[1] = fm * (b1 + u1) + mb * u1;
        } else {
            const R pb = (R)mesh.bpibc[e * G + lg];
            f[0] = fm * u0 + pb * dy;
            f[1] = fm * u1 - pb * dx;
        }
        R acc[3] = {(R)0, (R)0, (R)0};
#pragma unroll
        for (int k = 0; k < G; ++k) {
            const R w = tb->gxwtx[lm + 1][k];
#pragma unroll
            for (int n = 0; n < 3; ++n) acc[n] += w * __shfl_sync(mask, f[n], k, 16);
        }
        if (l < NM)
            for (int n = 0; n < 3; ++n) {
                if (st.bres) st.bres[((size_t)e * NM + l) * 3 + n] = acc[n];
                else if (l < 2) atomic_add(st.resv + (size_t)(l ? v1 : v0) * 3 + n, acc[n]);
                else atomic_add(st.ress + ((size_t)sd * SM + l - 2) * 3 + n, acc[n]);
            }
    }
}

template <typename R, int P, int PHYS, bool DIFF, bool RE>
__global__ void __launch_bounds__(LineCfg<R, P, PHYS, DIFF, RE>::NTHR, LineCfg<R, P, PHYS, DIFF, RE>::MINB)
    k_rsdl_line(const __grid_constant__ LineTab<R, P> tab, const DevTables<R, P> *__restrict__ gtab, Mesh mesh,
                State<R> st, LinePar par) {
    using C = LineCfg<R, P, PHYS, DIFF, RE>;
    constexpr int G = C::G, X = C::X, T = C::T, SM = C::SM, IM = C::IM, BM = C::BM, NV = C::NV, NTHR = C::NTHR;
    constexpr bool INS = PHYS == 1;
    const R beta = (R)par.beta, omb = (R)par.omb, rho = (R)par.rho;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R *sm = reinterpret_cast<R *>(smem_raw);
    R *out = sm + C::OUT;
    int *ring = reinterpret_cast<int *>(sm + C::LEN);
    const int tid = threadIdx.x, lane = tid & 31;
    const int j = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // the thread index anew: the indices of the copy loops are computed in each batch and not kept
    // in registers across the loop over batches
    auto fresh_tid = [&]() {
        int t = tid;
        asm volatile("" : "+r"(t));
        return t;
    };
    const int nbatch = (mesh.ntri + 31) / 32, last = mesh.ntri - 1;
    // connectivity of batch b into ring slot s (lanes past the last triangle repeat it)
    auto fetch_idx = [&](int b, int s) {
        if (b >= nbatch) return;
        const int tid = fresh_tid();
        int *d = ring + s * C::IDX;
        for (int w = tid; w < C::IDX; w += NTHR) {
            const int a = w / 96, r = w - a * 96;
            if (a == 5) {
                if (mesh.tri_cv) cp_async<4>(d + w, mesh.tri_cv + min(b * 32 + r, last));
                continue;
            }
            const int *src = a == 0   ? mesh.tri_pnt
                             : a == 1 ? mesh.tri_seg
                             : a == 2 ? mesh.tri_sgn
                             : a == 3 ? mesh.vpos
                                      : mesh.spos;
            cp_async<4>(d + w, src + min(b * 96 + r, 3 * last + r % 3));
        }
    };
    // modes of batch b (ugtouht, gtol.cpp:14-55; the signs of the side modes are applied when
    // they are read): a thread keeps to one value of the 3 T of a triangle, so its place and its
    // source are worked out once, and goes through the triangles; consecutive threads are on
    // consecutive values of a vertex, a side, an interior
    auto fetch_u = [&](int b, int s) {
        if (b >= nbatch) return;
        constexpr int TPP = NTHR / (NV * T);  // triangles a pass
        const int tid = fresh_tid(), sub = tid / (NV * T), rr = tid - sub * (NV * T);
        if (sub >= TPP) return;
        const int *d = ring + s * C::IDX;
        const R *base;
        int stride, row;
        bool inner = false;
        if (rr < 3 * NV) {
            const int m = rr / NV, n = rr - m * NV;
            base = st.ugv + n;
            stride = NV;
            d += m;
            row = n * T + m;
        } else if (rr < NV * BM) {
            const int i = (rr - 3 * NV) / C::LPS, r = rr - 3 * NV - i * C::LPS, k = r / NV, n = r - k * NV;
            base = st.ugs + r;
            stride = C::LPS;
            d += 96 + i;
            row = n * T + 3 + i * SM + k;
        } else {
            const int r = rr - NV * BM, k = r / NV, n = r - k * NV;
            base = st.ugi + r;
            stride = C::LPI;
            inner = true;
            row = n * T + BM + k;
        }
        R *dst = sm + C::U + row * 33;
#pragma unroll
        for (int it = 0; it < (32 + TPP - 1) / TPP; ++it) {
            const int e = sub + it * TPP;
            if (e >= 32) break;
            int v = d[3 * e];
            if (inner) v = min(b * 32 + e, last);
            cp_async<sizeof(R)>(dst + e, base + (size_t)v * stride);
        }
    };
    const int step = gridDim.x;
    int b = blockIdx.x, slot = 0;
    chain_next();
    fetch_idx(b, 0);
    fetch_idx(b + step, 1);
    cp_async_wait();
    __syncthreads();
    fetch_u(b, 0);
    if constexpr (INS && P > 1) line_bdry_flux<R, P, DIFF>(gtab, mesh, st, rho);
    for (; b < nbatch; b += step, slot = slot == 2 ? 0 : slot + 1) {
        const int *idx = ring + slot * C::IDX;
        const int t0 = b * 32;
        // per-triangle constants (Mesh::lgeo): ldcrd, 1 / |J|, tau length scale h, 1 / h
        const double *lg = mesh.lgeo + (size_t)b * (kLineGeo * 32) + lane;
        const R d00 = (R)lg[0], d01 = (R)lg[32], d10 = (R)lg[64], d11 = (R)lg[96];
        // ins: -mu / |J|, 2 nu / h, adis h / |J|
        const R cm = INS && RE ? (R)(-par.mu * lg[128]) : (R)0;
        const R c5 = INS && RE ? (R)(par.nu2 * lg[192]) : (R)0;
        const R c6 = INS && RE ? (R)(par.adis * lg[160] * lg[128]) : (R)0;
        // cd: the velocity's r and s components, the diffusion tensor, -|J| src, tau
        const R sr = INS ? (R)0 : d11 * (R)par.ax - d01 * (R)par.ay;
        const R ss = INS ? (R)0 : d00 * (R)par.ay - d10 * (R)par.ax;
        R k00 = (R)0, k01 = (R)0, k11 = (R)0, msrc = (R)0, taue = (R)0;
        if constexpr (!INS && RE) {
            const R kc = (R)(par.kcond * lg[128]);
            k00 = -kc * (d11 * d11 + d01 * d01);
            k11 = -kc * (d10 * d10 + d00 * d00);
            k01 = kc * (d11 * d10 + d01 * d00);
            msrc = -(d00 * d11 - d10 * d01) * (R)par.src;
            taue = st.tau[min(t0 + lane, last)];
        }
        R bu[DIFF ? G : 1], bv[DIFF ? G : 1];
        if constexpr (DIFF) {
            const R *bp = st.bpt + (size_t)b * (2 * G * G * 32) + lane;
#pragma unroll
            for (int i = 0; i < G; ++i) {
                bu[i] = bp[(i * G + j) * 32];
                bv[i] = bp[(G * G + i * G + j) * 32];
            }
        }
        cp_async_wait();
        __syncthreads();
        // sign bits of the triangle's sides (tri_sgn < 0): odd side modes change sign
        const int sbit[3] = {idx[192 + 3 * lane] & (int)0x80000000, idx[192 + 3 * lane + 1] & (int)0x80000000,
                             idx[192 + 3 * lane + 2] & (int)0x80000000};
        // ---- proj (proj.cpp:22-119): column sums of the thread's line, then its points: u, v, p and
        //      the viscous stress -mu (2 u_x, u_y + v_x, 2 v_y); cd: u and the diffusive r, s fluxes
        constexpr int GV = INS ? G : 1;
        R uq[G], vq[GV], pq[GV], xx[RE ? G : 1], xy[RE ? G : 1], yy[RE && INS ? G : 1];
        if constexpr (!INS) vq[0] = pq[0] = (R)0;
        {
            constexpr int XV = INS ? X : 1;
            R wu[X], wv[XV], wp[XV], wu1[X], wv1[XV];
#pragma unroll
            for (int c = 0; c < X; ++c) wu[c] = wu1[c] = (R)0;
#pragma unroll
            for (int c = 0; c < XV; ++c) wv[c] = wp[c] = wv1[c] = (R)0;
            const R *um = sm + C::U + lane;
            int jl = j;  // anew in each batch: the line's table entries are not kept across the loop
            asm volatile("" : "+r"(jl));
            each_mode([&](auto mm) {
                constexpr int m = decltype(mm)::value, c = ModeCols<P>::col(m);
                constexpr bool odd = m >= 3 && m < BM && (((m - 3) % (SM > 0 ? SM : 1)) & 1);
                const int bit = odd ? sbit[odd ? (m - 3) / (SM > 0 ? SM : 1) : 0] : 0;
                const R2<R> g = tab.g[jl][m];
                R x = um[m * 33];
                if constexpr (odd) flip_if(x, bit);
                wu[c] += x * g.x;
                if constexpr (RE) wu1[c] += x * g.y;
                if constexpr (INS) {
                    R y = um[(T + m) * 33], z = um[(2 * T + m) * 33];
                    if constexpr (odd) {
                        flip_if(y, bit);
                        flip_if(z, bit);
                    }
                    wv[c] += y * g.x;
                    wp[c] += z * g.x;
                    if constexpr (RE) wv1[c] += y * g.y;
                }
            }, std::make_integer_sequence<int, T>{});
            const R n0 = tab.n0[j];
#pragma unroll
            for (int i = 0; i < G; ++i) {
                R u = (R)0, v = (R)0, p = (R)0;
#pragma unroll
                for (int c = 0; c < X; ++c) {
                    u += wu[c] * tab.gx[i][c];
                    if constexpr (INS) {
                        v += wv[c] * tab.gx[i][c];
                        p += wp[c] * tab.gx[i][c];
                    }
                }
                uq[i] = u;
                if constexpr (INS) {
                    vq[i] = v;
                    pq[i] = p;
                }
                if constexpr (RE) {
                    R ur = (R)0, vr = (R)0, us = (R)0, vs = (R)0;
#pragma unroll
                    for (int c = 0; c < X; ++c) {
                        ur += wu[c] * tab.dgx[i][c];
                        us += wu1[c] * tab.gx[i][c];
                        if constexpr (INS) {
                            vr += wv[c] * tab.dgx[i][c];
                            vs += wv1[c] * tab.gx[i][c];
                        }
                    }
                    ur *= n0;
                    us += tab.x0[i] * ur;
                    if constexpr (INS) {
                        vr *= n0;
                        vs += tab.x0[i] * vr;
                        xx[i] = (cm + cm) * (d11 * ur - d10 * us);
                        xy[i] = cm * ((d00 * us - d01 * ur) + (d11 * vr - d10 * vs));
                        yy[i] = (cm + cm) * (d00 * vs - d01 * vr);
                    } else {
                        xx[i] = k00 * ur + k01 * us;
                        xy[i] = k01 * ur + k11 * us;
                    }
                }
            }
        }
        const R cr = (R)par.rhocv * sr, cs = (R)par.rhocv * ss;  // cd: convective flux = (cr, cs) u
        // convective flux (r, s components) of u and v at point i without the pressure, and the
        // mass flux; correction form: F(b + d) - F(b) with the products expanded
        auto conv = [&](int i, R &m0, R &m1, R &r0, R &s0, R &r1, R &s1) {
            const R u = uq[i], v = vq[INS ? i : 0];
            m0 = rho * (d11 * u - d01 * v);
            m1 = rho * (d00 * v - d10 * u);
            if constexpr (DIFF) {
                const R e0 = rho * (d11 * bu[i] - d01 * bv[i]), e1 = rho * (d00 * bv[i] - d10 * bu[i]);
                const R f0 = bu[i] + u, f1 = bv[i] + v;
                r0 = f0 * m0 + u * e0;
                s0 = f0 * m1 + u * e1;
                r1 = f1 * m0 + v * e0;
                s1 = f1 * m1 + v * e1;
            } else {
                r0 = u * m0;
                s0 = u * m1;
                r1 = v * m0;
                s1 = v * m1;
            }
        };
        R pr[RE ? NV : 1][RE ? G : 1], ps[RE ? NV : 1][RE ? G : 1];  // real flux pairs of the line: fr + x0 fs, fs
        if constexpr (RE) {
            // ---- strong residual (derivr + derivs of the full fluxes, proj.cpp:339-402):
            //      res(i, j) = n0(j) (sum_q Ar(i, q) fr(q, j) + As1(i, q) fs(q, j)) + sum_l As2(j, l) fs(i, l)
            R res[NV][G];
            R *ex = sm + C::EX + j * 32 + lane;  // s flux n at point i: ex[(n G + i) G 32]
#pragma unroll
            for (int n = 0; n < NV; ++n)
#pragma unroll
                for (int i = 0; i < G; ++i) res[n][i] = (R)0;
#pragma unroll
            for (int q = 0; q < G; ++q) {
                R r[NV], f[NV];
                if constexpr (INS) {
                    conv(q, r[2], f[2], r[0], f[0], r[1], f[1]);
                    const R px = xx[q] + pq[q], py = yy[q] + pq[q];
                    r[0] += d11 * px - d01 * xy[q];
                    f[0] += d00 * xy[q] - d10 * px;
                    r[1] += d11 * xy[q] - d01 * py;
                    f[1] += d00 * py - d10 * xy[q];
                } else {
                    r[0] = cr * uq[q] + xx[q];
                    f[0] = cs * uq[q] + xy[q];
                }
#pragma unroll
                for (int n = 0; n < NV; ++n) ex[((n * G + q) * G) * 32] = f[n];
#pragma unroll
                for (int i = 0; i < G; ++i)
#pragma unroll
                    for (int n = 0; n < NV; ++n) res[n][i] += tab.ar[i][q] * r[n] + tab.as1[i][q] * f[n];
            }
            __syncthreads();  // (the gathered modes are dead, too)
            fetch_u(b + step, slot == 2 ? 0 : slot + 1);
            fetch_idx(b + 2 * step, slot == 0 ? 2 : slot - 1);
            // eta-direction part, warp = x point: in place on the exchanged rows
            {
                R *f = sm + C::EX + (j * G) * 32 + lane;
                R s[NV][G];
#pragma unroll
                for (int n = 0; n < NV; ++n)
#pragma unroll
                    for (int l = 0; l < G; ++l) s[n][l] = f[(n * G * G + l) * 32];
#pragma unroll
                for (int k = 0; k < G; ++k) {
                    R a[NV];
#pragma unroll
                    for (int n = 0; n < NV; ++n) a[n] = (R)0;
#pragma unroll
                    for (int l = 0; l < G; ++l)
#pragma unroll
                        for (int n = 0; n < NV; ++n) a[n] += tab.as2[k][l] * s[n][l];
#pragma unroll
                    for (int n = 0; n < NV; ++n) f[(n * G * G + k) * 32] = a[n];
                }
            }
            __syncthreads();
            // ---- SUPG (ins/rsdl.cpp:341-431, CALC_TAU2; tau of the base in correction form): real
            //      pairs, viscous minus SUPG for u, v and the continuity term for p
            const R n0 = tab.n0[j];
#pragma unroll
            for (int i = 0; i < G; ++i) {
                if constexpr (!INS) {
                    const R tres = taue * (msrc + n0 * res[0][i] + ex[(i * G) * 32]);
                    const R fs = xy[i] - ss * tres;
                    pr[0][i] = xx[i] - sr * tres + tab.x0[i] * fs;
                    ps[0][i] = fs;
                } else {
                    R u = uq[i], v = vq[i], qv;
                    if constexpr (DIFF) {
                        qv = bu[i] * bu[i] + bv[i] * bv[i];
                        u += bu[i];
                        v += bv[i];
                    } else {
                        qv = u * u + v * v;
                    }
                    R gam = (R)3 * qv + c5 * c5;
                    if (par.gfloor) gam = gam > (R)0.1 ? gam : (R)0.1;
                    const R tau0 = line_tau0<R>(c6, gam), tau2 = sqrt(qv) * tau0;
                    const R a0 = tau0 * (n0 * res[0][i] + ex[(i * G) * 32]);
                    const R a1 = tau0 * (n0 * res[1][i] + ex[((G + i) * G) * 32]);
                    const R a2 = tau2 * (n0 * res[2][i] + ex[((2 * G + i) * G) * 32]);
                    // physical SUPG fluxes: x-momentum (2 u a0 + a2, v a0 + u a1), y-momentum
                    // (v a0 + u a1, 2 v a1 + a2), continuity (a0, a1)
                    const R sxx = xx[i] - ((u + u) * a0 + a2), sxy = xy[i] - (v * a0 + u * a1),
                            syy = yy[i] - ((v + v) * a1 + a2);
                    pr[0][i] = d11 * sxx - d01 * sxy;
                    ps[0][i] = d00 * sxy - d10 * sxx;
                    pr[1][i] = d11 * sxy - d01 * syy;
                    ps[1][i] = d00 * syy - d10 * sxy;
                    pr[2][i] = d01 * a1 - d11 * a0;
                    ps[2][i] = d10 * a0 - d00 * a1;
#pragma unroll
                    for (int n = 0; n < 3; ++n) pr[n][i] += tab.x0[i] * ps[n][i];
                }
            }
            __syncthreads();  // A, B take the place of the exchanged rows
        }
        // ---- intgrtrs (intgrt.cpp:81-158): x-direction sums of the flux pairs, given by
        //      pair(i, fr + x0 fs, fs), XH columns at a time (their sums share the registers)
        auto xsums = [&](auto &&pair) {
            constexpr int XH = C::XH;
            R *ab = sm + C::EX + j * 32 + lane;  // A of (n, c): row (2 n X + c) G, B X rows further
#pragma unroll
            for (int h = 0; h < (X + XH - 1) / XH; ++h) {
                R a[NV][XH], bb[NV][XH];
#pragma unroll
                for (int n = 0; n < NV; ++n)
#pragma unroll
                    for (int c = 0; c < XH; ++c) a[n][c] = bb[n][c] = (R)0;
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    R fr[NV], fs[NV];
                    pair(i, fr, fs);
#pragma unroll
                    for (int c = 0; c < XH; ++c)
                        if (h * XH + c < X)
#pragma unroll
                            for (int n = 0; n < NV; ++n) {
                                a[n][c] += tab.dgxw[h * XH + c][i] * fr[n];
                                bb[n][c] += tab.gxw[h * XH + c][i] * fs[n];
                            }
                }
#pragma unroll
                for (int n = 0; n < NV; ++n)
#pragma unroll
                    for (int c = 0; c < XH; ++c)
                        if (h * XH + c < X) {
                            ab[((n * 2 * X + h * XH + c) * G) * 32] = a[n][c];
                            ab[((n * 2 * X + X + h * XH + c) * G) * 32] = bb[n][c];
                        }
            }
        };
        // eta-direction sums of the warp's modes into the staging rows; src0: integral of a constant
        auto esums = [&](R scale, R src0) {
#pragma unroll 1
            for (int it = tab.iptr[j]; it < tab.iptr[j + 1]; ++it) {
                const R *pa = sm + C::EX + (tab.icol[it] * G) * 32 + lane;
                R a[NV][G], bb[NV][G];
#pragma unroll
                for (int n = 0; n < NV; ++n)
#pragma unroll
                    for (int k = 0; k < G; ++k) {
                        a[n][k] = pa[(n * 2 * X * G + k) * 32];
                        bb[n][k] = pa[((n * 2 * X + X) * G + k) * 32];
                    }
#pragma unroll 1
                for (int q = tab.ifst[it]; q < tab.ifst[it + 1]; ++q) {
                    const int m = tab.mode[q];
                    R s0[NV], s1[NV];
#pragma unroll
                    for (int n = 0; n < NV; ++n) s0[n] = s1[n] = (R)0;
                    if constexpr (!INS) s0[0] = src0 * tab.src[m];
#pragma unroll
                    for (int k = 0; k < G; ++k) {
                        const R2<R> w = tab.w[m][k];
#pragma unroll
                        for (int n = 0; n < NV; ++n) {
                            s0[n] += w.x * a[n][k];
                            s1[n] += w.y * bb[n][k];
                        }
                    }
                    R sc = scale;  // odd side modes in the side's own direction
                    const int sd = tab.odd[m];
                    flip_if(sc, sd == 0 ? sbit[0] : sd == 1 ? sbit[1] : sd == 2 ? sbit[2] : 0);
#pragma unroll
                    for (int n = 0; n < NV; ++n) out[(m * NV + n) * 33 + lane] = sc * (s0[n] + s1[n]);
                }
            }
        };
        if constexpr (C::TIGHT) __syncthreads();  // the gathered modes have been read
        xsums([&](int i, R (&fr)[NV], R (&fs)[NV]) {
            if constexpr (INS) {
                conv(i, fr[2], fs[2], fr[0], fs[0], fr[1], fs[1]);
                fr[0] += d11 * pq[i];
                fs[0] -= d10 * pq[i];
                fr[1] -= d01 * pq[i];
                fs[1] += d00 * pq[i];
#pragma unroll
                for (int n = 0; n < NV; ++n) fr[n] += tab.x0[i] * fs[n];
                // the second half of the columns forms the fluxes again instead of keeping them
                opaque(uq[i]);
                opaque(vq[i]);
            } else {
                fs[0] = cs * uq[i];
                fr[0] = cr * uq[i] + tab.x0[i] * fs[0];
            }
        });
        // lftog (gtol.cpp:364-402), threads as in fetch_u; curved triangles are done by the curved
        // launch. The interior values of the imaginary part wait in registers for the real part.
        constexpr int TPS = NTHR / (NV * BM), TPI = NTHR / (IM > 0 ? C::LPI : NTHR);
        constexpr int NKEEP = IM > 0 ? (32 + TPI - 1) / TPI : 1;
        R keep[NKEEP];
        auto act = [&](int e) { return t0 + e <= last && (!mesh.tri_cv || idx[480 + e] < 0); };
        // res_r of the interior values, in a stage without the real part: read ahead of the sums
        // (FP64: p = 6 165 -> 159 us; FP32 has no registers to hold them, an update 2018 -> 2060 us)
        constexpr bool RRI = sizeof(R) == 8 && !RE;
        auto load_rr = [&]() {
            const int sub = tid / C::LPI, r = tid - sub * C::LPI;
            if constexpr (RRI && IM > 0) {
#pragma unroll
                for (int it = 0; it < NKEEP; ++it) {
                    const int e = sub + it * TPI;
                    keep[it] = (R)0;
                    if (omb != (R)0 && sub < TPI && e < 32 && t0 + e <= last)
                        keep[it] = st.rri[(size_t)(t0 + e) * C::LPI + r] * omb;
                }
            }
        };
        auto scatter = [&](int part) {
            const int tid = fresh_tid();
            {
                const int sub = tid / (NV * BM), rr = tid - sub * (NV * BM);
                if (sub < TPS) {
                    R *el = part ? st.elre : st.elim, *base;
                    const int *d = idx;
                    int stride = NV;
                    if (rr < 3 * NV) {
                        const int m = rr / NV, n = rr - m * NV;
                        base = (el ? el : part ? st.rrv : st.resv) + n;
                        d += (el ? 288 : 0) + m;
                    } else {
                        const int i = (rr - 3 * NV) / C::LPS, r = rr - 3 * NV - i * C::LPS;
                        base = (el ? el + (size_t)3 * mesh.ntri * NV : part ? st.rrs : st.ress) + r;
                        d += (el ? 384 : 96) + i;
                        stride = C::LPS;
                    }
                    const R *src = out + rr * 33;
#pragma unroll
                    for (int it = 0; it < (32 + TPS - 1) / TPS; ++it) {
                        const int e = sub + it * TPS;
                        if (e >= 32) break;
                        if (!act(e)) continue;
                        R *p = base + (size_t)d[3 * e] * stride;
                        if (el) *p = src[e];
                        else atomic_add(p, src[e]);
                    }
                }
            }
            if constexpr (IM > 0) {
                const int sub = tid / C::LPI, r = tid - sub * C::LPI;
                if (sub < TPI) {
#pragma unroll
                    for (int it = 0; it < NKEEP; ++it) {
                        const int e = sub + it * TPI;
                        if (e >= 32) break;
                        if (!act(e)) continue;
                        const R val = out[(NV * BM + r) * 33 + e];
                        const size_t gi = (size_t)(t0 + e) * C::LPI + r;
                        const R rr = RRI ? keep[it] : omb != (R)0 && (part || !RE) ? st.rri[gi] * omb : (R)0;
                        if (part) {
                            st.rri[gi] = rr + val;
                            st.resi[gi] = keep[it] + (rr + val);
                        } else {
                            keep[it] = st.dresi ? val + st.dresi[gi] : val;
                            if constexpr (!RE) st.resi[gi] = keep[it] + rr;  // res_r unchanged when beta = 0
                        }
                    }
                }
            }
        };
        __syncthreads();
        auto fetch = [&]() {
            fetch_u(b + step, slot == 2 ? 0 : slot + 1);
            fetch_idx(b + 2 * step, slot == 0 ? 2 : slot - 1);
        };
        if constexpr (!RE && !C::TIGHT) fetch();
        load_rr();
        esums((R)1, (R)0);
        __syncthreads();
        if constexpr (C::TIGHT) fetch();
        scatter(0);
        if constexpr (RE) {
            xsums([&](int i, R (&fr)[NV], R (&fs)[NV]) {
#pragma unroll
                for (int n = 0; n < NV; ++n) {
                    fr[n] = pr[n][i];
                    fs[n] = ps[n][i];
                }
            });
            __syncthreads();
            esums(beta, msrc);
            __syncthreads();
            scatter(1);
        }
    }
}

}  // namespace hpb
