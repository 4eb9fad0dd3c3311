// One stage of tri_hp::update at p = 1 in one kernel, vertex by vertex (straight elements).
//
// At p = 1 every unknown is a vertex value, so tri_hp::rsdl(stage) (tri_hp/nstage.cpp:12-110), the
// boundary fluxes (hp_edge_bdry::rsdl, hp_boundary.cpp:973-1049), tri_hp::minvrt
// (setup_preconditioner.cpp:102-373) and the stage update (nstage.cpp:387-409) of a vertex need
// only the triangles around it. A warp takes a vertex: lane 4 e + q evaluates Gauss point
// q = 2 i + j of the vertex's triangle e (eight at a time) with the dense per-point operators, and
// keeps its share of the one test function that belongs to the vertex; the shares are summed by
// shuffles in a fixed order and lane n finishes variable n. A triangle is evaluated three times,
// once for each of its vertices, and nothing goes through memory between the element loop and the
// update: the separate kernels (element, boundary flux, assembly, vertex phase) were a chain of four
// launches of 5 to 10 us each, latency and not work. The state is read from one buffer and written
// to another (neighbours are read), see enqueue_p1_update.
// For small levels (p1_small); larger ones take the element kernel and k_vert_p1, since the
// threefold evaluation then costs more than the launch it saves.
// Measured per FP64 update (five stages): 512 triangles 86 -> 29 us, 8192 triangles 89 -> 49 us,
// 131k triangles 212 -> 390 us, where the element kernel and k_vert_p1 take 143 (hence the rule).
// Bound by latency (vertex -> incidence -> state loads, then the FP64 chain of a point).
#pragma once
#include "hp_chain.cuh"
#include "hp_p1.h"

namespace hpb {

template <typename R>
__device__ __forceinline__ R warp_sum(R v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Variable n of the generic boundary flux (bdry_ins::generic, ins/bdry_ins.h:35-50) at Gauss point k
// of boundary edge b / 2, times the end function b % 2 there.
template <typename R, bool DIFF>
__device__ __forceinline__ R p1_bflux(const P1Ops<R> *ops, const Mesh &mesh, const R *u, const R *ub, R rho, int b,
                                      int k, int n) {
    const int e = b >> 1, sg = mesh.bseg[e], a = mesh.seg_pnt[2 * sg], z = mesh.seg_pnt[2 * sg + 1];
    const R g0 = ops->BG[k][0], g1 = ops->BG[k][1];
    const R dx = (R)mesh.pnts[2 * a] * ops->BD[k][0] + (R)mesh.pnts[2 * z] * ops->BD[k][1];
    const R dy = (R)mesh.pnts[2 * a + 1] * ops->BD[k][0] + (R)mesh.pnts[2 * z + 1] * ops->BD[k][1];
    R ue[2];
#pragma unroll
    for (int m = 0; m < 2; ++m) ue[m] = g0 * u[(size_t)a * 3 + m] + g1 * u[(size_t)z * 3 + m];
    const R fm = rho * (ue[0] * dy - ue[1] * dx);
    R f = fm;
    if (n < 2) {
        const R un = n == 0 ? ue[0] : ue[1];
        if constexpr (DIFF) {  // F(b + d) - F(b); the boundary pressure cancels
            const R c0 = g0 * ub[(size_t)a * 3] + g1 * ub[(size_t)z * 3];
            const R c1 = g0 * ub[(size_t)a * 3 + 1] + g1 * ub[(size_t)z * 3 + 1];
            f = fm * ((n == 0 ? c0 : c1) + un) + rho * (c0 * dy - c1 * dx) * un;
        } else {
            const R pb = (R)mesh.bpibc[2 * e + k];
            f = fm * un + (n == 0 ? pb * dy : -pb * dx);
        }
    }
    return ops->BW[k][b & 1] * f;
}

template <typename R, int PHYS, bool DIFF>
__global__ void __launch_bounds__(128, sizeof(R) == 8 ? 5 : 6)
    k_stage_p1(const P1Ops<R> *__restrict__ ops, Mesh mesh, P1Stage<R> s, Phys ph) {
    constexpr int NV = PHYS == 1 ? 3 : 1;
    const int lane = threadIdx.x & 31, q = lane & 3, i = q >> 1, j = q & 1;
    const R rho = (R)ph.rho;
    // this lane's rows of the operators
    R V[3], DR[3], DS[3], WR[3], WS[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        V[m] = ops->V[q][m]; DR[m] = ops->DR[q][m]; DS[m] = ops->DS[q][m];
        WR[m] = ops->WR[q][m]; WS[m] = ops->WS[q][m];
    }
    const R ar_ii = ops->AR[i][i], ar_io = ops->AR[i][1 - i], as1_ii = ops->AS1[i][i], as1_io = ops->AS1[i][1 - i];
    const R as2_jj = ops->AS2[j][j], as2_jo = ops->AS2[j][1 - j], n0j = ops->N0[j];
    R rmax = (R)0;
    const int nwarp = (gridDim.x * blockDim.x) >> 5;
    // The next stage may start its CTAs; this one, while the stage before it ends, brings in what no
    // stage writes: the operators and the incidences and geometry of its first vertices.
    chain_next();
    {
        const int v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        if (v < mesh.npnt) {
            const int v0 = mesh.vt_ptr[v], nt = mesh.vt_ptr[v + 1] - v0, k = lane >> 2, kk = v0 + (k < nt ? k : 0);
            if (nt > 0) {  // a last vertex without triangles has v0 past the end of the incidences
                const double *tg = mesh.tgeo + (size_t)8 * (mesh.vt_idx[kk] >> 2);
                asm volatile("prefetch.global.L1 [%0];" ::"l"(tg));
                asm volatile("prefetch.global.L1 [%0];" ::"l"(mesh.vt_pnt + 3 * kk));
            }
            if (PHYS == 1 && mesh.nbseg > 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(mesh.vb_idx + 2 * v));
        }
    }
    chain_wait();
    for (int v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < mesh.npnt; v += nwarp) {
        const int v0 = mesh.vt_ptr[v], nt = mesh.vt_ptr[v + 1] - v0;
        R im[NV], re[NV];
#pragma unroll
        for (int n = 0; n < NV; ++n) im[n] = re[n] = (R)0;
        for (int b0 = 0; b0 < nt; b0 += 8) {
            const int k = b0 + (lane >> 2);
            const bool act = k < nt;
            const int kk = v0 + (act ? k : 0), code = mesh.vt_idx[kk], t = code >> 2, c = code & 3;
            const int pv[3] = {mesh.vt_pnt[3 * kk], mesh.vt_pnt[3 * kk + 1], mesh.vt_pnt[3 * kk + 2]};
            R u[NV][3];
#pragma unroll
            for (int m = 0; m < 3; ++m)
#pragma unroll
                for (int n = 0; n < NV; ++n) u[n][m] = s.u_in[(size_t)pv[m] * NV + n];
            const double *tg = mesh.tgeo + (size_t)8 * t;  // per-triangle constants (Mesh::tgeo)
            const R d00 = (R)tg[0], d01 = (R)tg[1], d10 = (R)tg[2], d11 = (R)tg[3];
            const R wr = act ? (c == 0 ? WR[0] : c == 1 ? WR[1] : WR[2]) : (R)0;
            const R ws = act ? (c == 0 ? WS[0] : c == 1 ? WS[1] : WS[2]) : (R)0;
            R uq[NV];
#pragma unroll
            for (int n = 0; n < NV; ++n) uq[n] = V[0] * u[n][0] + V[1] * u[n][1] + V[2] * u[n][2];
            if constexpr (PHYS == 1) {
                R b0v = (R)0, b1v = (R)0;
                if constexpr (DIFF) {
#pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        b0v += V[m] * s.ub[(size_t)pv[m] * NV];
                        b1v += V[m] * s.ub[(size_t)pv[m] * NV + 1];
                    }
                }
                // pointwise fluxes (ins/rsdl.cpp:259-340); correction form: F(b + d) - F(b)
                const R m0 = +d11 * (rho * uq[0]) - d01 * (rho * uq[1]);
                const R m1 = -d10 * (rho * uq[0]) + d00 * (rho * uq[1]);
                R c00, c01, c10, c11;
                if constexpr (DIFF) {
                    const R mb0 = +d11 * (rho * b0v) - d01 * (rho * b1v);
                    const R mb1 = -d10 * (rho * b0v) + d00 * (rho * b1v);
                    const R uf0 = b0v + uq[0], uf1 = b1v + uq[1];
                    c00 = uf0 * m0 + uq[0] * mb0;
                    c01 = uf0 * m1 + uq[0] * mb1;
                    c10 = uf1 * m0 + uq[1] * mb0;
                    c11 = uf1 * m1 + uq[1] * mb1;
                } else {
                    c00 = uq[0] * m0; c01 = uq[0] * m1; c10 = uq[1] * m0; c11 = uq[1] * m1;
                }
                const R fir[3] = {c00 + d11 * uq[2], c10 - d01 * uq[2], m0};
                const R fis[3] = {c01 - d10 * uq[2], c11 + d00 * uq[2], m1};
#pragma unroll
                for (int n = 0; n < 3; ++n) im[n] += wr * fir[n] + ws * fis[n];
                if (s.re) {
                    R dr[2], ds[2];
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        dr[n] = DR[0] * u[n][0] + DR[1] * u[n][1] + DR[2] * u[n][2];
                        ds[n] = DS[0] * u[n][0] + DS[1] * u[n][1] + DS[2] * u[n][2];
                    }
                    // viscous stress -mu (2 u_x, u_y + v_x, 2 v_y) and its r, s fluxes
                    const R cm = (R)(-ph.mu * tg[4]);
                    const R xx = (cm + cm) * (d11 * dr[0] - d10 * ds[0]);
                    const R xy = cm * ((d00 * ds[0] - d01 * dr[0]) + (d11 * dr[1] - d10 * ds[1]));
                    const R yy = (cm + cm) * (d00 * ds[1] - d01 * dr[1]);
                    R fxr[3] = {d11 * xx - d01 * xy, d11 * xy - d01 * yy, (R)0};
                    R fxs[3] = {d00 * xy - d10 * xx, d00 * yy - d10 * xy, (R)0};
                    // strong residual at this point (derivr + derivs of the full fluxes)
                    R res[3];
#pragma unroll
                    for (int n = 0; n < 3; ++n) {
                        const R fr = fir[n] + fxr[n], fs = fis[n] + fxs[n];
                        const R fr_oi = __shfl_xor_sync(0xffffffffu, fr, 2);
                        const R fs_oi = __shfl_xor_sync(0xffffffffu, fs, 2);
                        const R fs_oj = __shfl_xor_sync(0xffffffffu, fs, 1);
                        res[n] = n0j * (ar_ii * fr + ar_io * fr_oi + as1_ii * fs + as1_io * fs_oi) +
                                 (as2_jj * fs + as2_jo * fs_oj);
                    }
                    // SUPG (ins/rsdl.cpp:341-431, CALC_TAU2), tau of the base in correction form
                    const R a0 = uq[0] + b0v, a1 = uq[1] + b1v;
                    const R qv = DIFF ? b0v * b0v + b1v * b1v : uq[0] * uq[0] + uq[1] * uq[1];
                    const R t2 = (R)(2. * (ph.mu / ph.rho) * tg[6]);
                    R gam = (R)3 * qv + t2 * t2;
                    if (ph.mu + ph.bd0 == 0.0) gam = (gam > (R)0.1 ? gam : (R)0.1);
                    const R tau0 = (R)(ph.adis * tg[5] * tg[4]) / sqrt(gam);
                    const R tau2 = sqrt(qv) * tau0;
                    const R tr0 = tau0 * res[0], tr1 = tau0 * res[1], tr2 = tau2 * res[2];
                    const R sx = (a0 + a0) * tr0 + tr2, sxy = a1 * tr0 + a0 * tr1, sy = (a1 + a1) * tr1 + tr2;
                    fxr[0] -= d11 * sx - d01 * sxy;
                    fxs[0] -= d00 * sxy - d10 * sx;
                    fxr[1] -= d11 * sxy - d01 * sy;
                    fxs[1] -= d00 * sy - d10 * sxy;
                    fxr[2] = -(d11 * tr0 - d01 * tr1);
                    fxs[2] = -(d00 * tr1 - d10 * tr0);
#pragma unroll
                    for (int n = 0; n < 3; ++n) re[n] += wr * fxr[n] + ws * fxs[n];
                }
            } else {
                // cd (cd/rsdl.cpp:14-154, CONST_A)
                const R ax = (R)ph.ax, ay = (R)ph.ay;
                const R fx = (R)ph.rhocv * ax * uq[0], fy = (R)ph.rhocv * ay * uq[0];
                const R c0 = +d11 * fx - d01 * fy, c1 = -d10 * fx + d00 * fy;
                im[0] += wr * c0 + ws * c1;
                if (s.re) {
                    const R dr = DR[0] * u[0][0] + DR[1] * u[0][1] + DR[2] * u[0][2];
                    const R ds = DS[0] * u[0][0] + DS[1] * u[0][1] + DS[2] * u[0][2];
                    const R cj = d00 * d11 - d10 * d01, kc = (R)ph.kcond / cj;
                    const R v00 = -kc * (d11 * d11 + d01 * d01), v11 = -kc * (d10 * d10 + d00 * d00);
                    const R v01 = kc * (d11 * d10 + d01 * d00);
                    R e0 = v00 * dr + v01 * ds, e1 = v01 * dr + v11 * ds;
                    const R fr = c0 + e0, fs = c1 + e1, src = -cj * (R)ph.src;
                    const R fr_oi = __shfl_xor_sync(0xffffffffu, fr, 2), fs_oi = __shfl_xor_sync(0xffffffffu, fs, 2);
                    const R fs_oj = __shfl_xor_sync(0xffffffffu, fs, 1);
                    const R tres = s.tau[t] * (src + n0j * (ar_ii * fr + ar_io * fr_oi + as1_ii * fs + as1_io * fs_oi) +
                                               (as2_jj * fs + as2_jo * fs_oj));
                    e0 -= (d11 * ax - d01 * ay) * tres;
                    e1 -= (-d10 * ax + d00 * ay) * tres;
                    re[0] += wr * e0 + ws * e1;
                    if (act && src != (R)0) re[0] += src * ops->W0[q][c];
                }
            }
        }
        if constexpr (PHYS == 1) {
            // the (at most two) boundary edges of the vertex, lane = 2 edge + Gauss point
            if (lane < 4 && mesh.nbseg > 0) {
                const int b = mesh.vb_idx[2 * v + i];
                if (b >= 0 && (mesh.bkind[b >> 1] & (0xF << 8)) == (1 << 8)) {
#pragma unroll
                    for (int n = 0; n < 3; ++n) im[n] += p1_bflux<R, DIFF>(ops, mesh, s.u_in, s.ub, rho, b, j, n);
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            im[n] = warp_sum(im[n]);
            if (s.re) re[n] = warp_sum(re[n]);
        }
        if (lane < NV) {
            const size_t g = (size_t)v * NV + lane;
            const R sim = NV == 1 || lane == 0 ? im[0] : lane == 1 ? im[NV > 1 ? 1 : 0] : im[NV > 1 ? 2 : 0];
            const R sre = NV == 1 || lane == 0 ? re[0] : lane == 1 ? re[NV > 1 ? 1 : 0] : re[NV > 1 ? 2 : 0];
            // res_r = (1 - beta) res_r + beta re (nstage.cpp:21-49), res = im + res_r + dres
            R rr = s.omb != (R)0 ? s.rr[g] * s.omb : (R)0;
            if (s.re) rr += s.beta * sre;
            s.rr[g] = rr;
            R r = sim + rr + (s.dres ? s.dres[g] : (R)0);
            if (s.u_out) {
                r *= s.vprcn[g];
                if (mesh.vess[v] & (1 << lane)) r = (R)0;
                s.u_out[g] = s.u0[g] - s.cfla * r;
                if (nt > 0) rmax = max_nan(rmax, (R)fabs(r));
            }
            if (s.res) s.res[g] = r;
        }
    }
    if (s.slot) {  // tri_hp::maxres of the last stage, per variable
        __shared__ R sm[4][3];
        if (lane < NV) sm[threadIdx.x >> 5][lane] = rmax;
        __syncthreads();
        if (threadIdx.x < NV) {
            R a = sm[0][threadIdx.x];
            for (int w = 1; w < 4; ++w) a = max_nan(a, sm[w][threadIdx.x]);
            atomicMax(&s.slot[threadIdx.x], ord_key(a));
        }
    }
}

// The vertex half of a stage when the element kernel has written the element slots (State::elim,
// elre): k_assemble, the boundary fluxes and the vertex phase of minvrt with the update in one pass,
// one thread per (vertex, variable). The state goes from one buffer to another as in k_stage_p1 (the
// boundary fluxes read neighbours). Bound by memory: the slots are read once.
template <typename R, int PHYS, bool DIFF>
__global__ void __launch_bounds__(128)
    k_vert_p1(const P1Ops<R> *__restrict__ ops, Mesh mesh, const R *__restrict__ elim, const R *__restrict__ elre,
              P1Stage<R> s, Phys ph) {
    constexpr int NV = PHYS == 1 ? 3 : 1;
    const int g = blockIdx.x * blockDim.x + threadIdx.x, v = g / NV, n = g - v * NV;
    R ar = (R)0;
    if (v < mesh.npnt) {
        R sim = (R)0, sre = (R)0;
        const int j1 = mesh.vt_ptr[v + 1];
        for (int j = mesh.vt_ptr[v]; j < j1; ++j) {
            sim += elim[(size_t)j * NV + n];
            if (s.re) sre += elre[(size_t)j * NV + n];
        }
        if constexpr (PHYS == 1) {
            if (mesh.nbseg > 0)
                for (int q = 0; q < 2; ++q) {
                    const int b = mesh.vb_idx[2 * v + q];
                    if (b < 0 || (mesh.bkind[b >> 1] & (0xF << 8)) != (1 << 8)) continue;
                    for (int k = 0; k < 2; ++k) sim += p1_bflux<R, DIFF>(ops, mesh, s.u_in, s.ub, (R)ph.rho, b, k, n);
                }
        }
        R rr = s.omb != (R)0 ? s.rr[g] * s.omb : (R)0;
        if (s.re) rr += sre;
        s.rr[g] = rr;
        R r = sim + rr + (s.dres ? s.dres[g] : (R)0);
        if (s.u_out) {
            r *= s.vprcn[g];
            if (mesh.vess[v] & (1 << n)) r = (R)0;
            s.u_out[g] = s.u0[g] - s.cfla * r;
            if (j1 > mesh.vt_ptr[v]) ar = fabs(r);
        }
        if (s.res) s.res[g] = r;
    }
    if (s.slot) {
        __shared__ unsigned long long mx[3];
        if (threadIdx.x < 3) mx[threadIdx.x] = 0;
        __syncthreads();
        if (v < mesh.npnt) atomicMax(&mx[n], ord_key(ar));
        __syncthreads();
        if (threadIdx.x < NV) atomicMax(&s.slot[threadIdx.x], mx[threadIdx.x]);
    }
}

}  // namespace hpb
