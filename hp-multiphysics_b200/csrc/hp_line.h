// Host side of the line kernel (hp_elem_line.cuh): per (precision, p) table builder and
// launcher, compiled in hp_line.cu.
#pragma once
#include <vector>

#include "hp_gpu.h"
#include "hp_kernels.cuh"

namespace hpb {

// The 1D derivative operators of derivr / derivs (proj.cpp:339-402) as matrices, so that
// the strong residual at point (i, j) is
//   res(i, j) = n0(j) (sum_q Ar(i, q) flux_r(q, j) + sum_q As1(i, q) flux_s(q, j))
//             + sum_l As2(j, l) flux_s(i, l), with (which = 0: Ar, 1: As1, 2: As2)
//   Ar(i, q)  = q == i ? dltx(i) sum_{q' != i} dltx1(i, q') : dltx(q) dltx1(i, q)
//   As1(i, q) = q == i ? dltx(i) sum_{q' != i} dltn1(i, q') : dltx(q) dltn1(i, q)
//   As2(j, l) = l == j ? dltn(j) sum_{l' != j} dltn2(j, l') : dltn(l) dltn2(j, l).
inline double deriv_op(const hp_basis_tables &b, int G, int which, int r, int k) {
    if (r >= G || k >= G) return 0.0;
    auto tab = [&](int a, int c) {
        return which == 0 ? b.dltx1[a][c] : (which == 1 ? b.dltn1[a][c] : b.dltn2[a][c]);
    };
    const double *dl = which == 2 ? b.dltn : b.dltx;
    if (k != r) return dl[k] * tab(r, k);
    double sum = 0.0;
    for (int c = 0; c < G; ++c)
        if (c != r) sum += tab(r, c);
    return dl[r] * sum;
}

// Rows of Mesh::lgeo.
constexpr int kLineGeo = 7;

template <typename R>
struct LineLaunch {
    // tables as the launcher's kernel parameter; shared-memory attributes; k_rsdl_line, with the
    // level's DevTables on the device (ins at p > 1: the boundary fluxes, too)
    void (*build)(const hp_basis_tables &, std::vector<unsigned char> &tab) = nullptr;
    cudaError_t (*set_smem)() = nullptr;
    void (*launch)(const void *tab, const void *dev_tables, const Mesh &, const State<R> &, const Phys &, int stage,
                   int zero_rr, int diff, int nsm, cudaStream_t) = nullptr;
    // FP32: the base state's point values of the correction form (State::bpt), their number
    void (*base_pts)(const void *dev_tables, const Mesh &, const State<R> &, R *bpt, cudaStream_t) = nullptr;
    size_t (*bpt_len)(int ntri) = nullptr;
};

// The line kernel of p and physics, 1 <= p <= HP_MAXP.
template <typename R>
LineLaunch<R> line_launch(int p, int physics);
template <>
LineLaunch<double> line_launch<double>(int p, int physics);
template <>
LineLaunch<float> line_launch<float>(int p, int physics);

}  // namespace hpb
