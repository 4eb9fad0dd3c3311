// Host side of the fused p = 1 stage kernel (hp_stage_p1.cuh), compiled in hp_p1.cu.
#pragma once
#include <vector>

#include "hp_gpu.h"
#include "hp_kernels.cuh"

namespace hpb {

// The operators at p = 1 (G = 2, T = 3) as dense arrays over the points q = 2 i + j: values V and
// derivatives DR, DS of the modes, weights of the r and s fluxes WR, WS, those of intgrt W0; the 1D
// derivative operators AR, AS1, AS2 and factors N0 of the strong residual; the boundary side's
// tables at its Gauss points: values and derivatives of the two end functions BG, BD [k][end],
// integration weights BW [k][end].
template <typename R>
struct P1Ops {
    R V[4][3], DR[4][3], DS[4][3], WR[4][3], WS[4][3], W0[4][3];
    R AR[2][2], AS1[2][2], AS2[2][2], N0[2];
    R BG[2][2], BD[2][2], BW[2][2];
};

// One stage: the state in, the state at the start of the update, the state out (NULL: residual
// only, folded into res), residual out (or NULL), res_r, preconditioner, source, base state
// (correction form), cd tau; re: beta > 0; slot: maxres (last stage) or NULL.
template <typename R>
struct P1Stage {
    const R *u_in, *u0;
    R *u_out, *res, *rr;
    const R *vprcn, *dres, *ub, *tau;
    R beta, omb, cfla;
    int re;
    unsigned long long *slot;
};

template <typename R>
void p1_ops(const hp_basis_tables &, P1Ops<R> &);

// Whether a level's stage runs vertex by vertex (k_stage_p1): its vertices, one warp each, are two
// waves of the resident warps at most. Measured per update (five stages), vertex by vertex / element
// kernel and k_vert_p1: FP64 4225 vertices 49 / 55 us, 66k vertices 390 / 143; FP32 4225 vertices
// 38 / 57, 66k vertices 252 / 116.
template <typename R>
bool p1_small(const Mesh &m, int nsm) {
    return m.npnt <= 2 * nsm * (sizeof(R) == 8 ? 20 : 24);
}

// chained (hp_chain.cuh): the kernel before it on the stream is the same update's previous stage. An
// update of 512 triangles 30.9 -> 28.8 us, cd 20.6 -> 16.5, 11k triangles 53.3 -> 50.1.
template <typename R>
void p1_stage(const P1Ops<R> *dev_ops, const Mesh &, const P1Stage<R> &, const Phys &, int diff, int nsm, int chained,
              cudaStream_t);

// k_vert_p1 after the element kernel.
template <typename R>
void p1_vert(const P1Ops<R> *dev_ops, const Mesh &, const R *elim, const R *elre, const P1Stage<R> &, const Phys &,
             int diff, cudaStream_t);

}  // namespace hpb
