// Table builder and launchers of the line kernel (hp_elem_line.cuh), compiled once for each
// precision (LINE_R double or float).
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "hp_line.h"
#include "hp_elem_line.cuh"

namespace hpb {

namespace {

// proj and intgrtrs sum-factorised, the derivr / derivs matrices, and each warp's modes of
// intgrtrs' eta-direction: an equal share of the modes in column order, so that a warp reads few
// columns (one read of a column's sums costs about as much as one mode).
template <typename R, int P>
void build_tab(const hp_basis_tables &b, LineTab<R, P> &t) {
    constexpr int G = P + 1, X = P + 2, T = (P + 1) * (P + 2) / 2, SD = P > 1 ? P - 1 : 1;
    std::memset(&t, 0, sizeof(t));
    for (int i = 0; i < G; ++i) {
        for (int m = 0; m < T; ++m) {
            t.g[i][m] = {(R)b.gn[i][m], (R)b.dgn[i][m]};
            t.w[m][i] = {(R)-b.gnwtnn0[m][i], (R)-b.dgnwtn[m][i]};
        }
        for (int c = 0; c < X; ++c) {
            t.gx[i][c] = (R)b.gx[i][c]; t.dgx[i][c] = (R)b.dgx[i][c];
            t.gxw[c][i] = (R)b.gxwtx[c][i]; t.dgxw[c][i] = (R)b.dgxwtx[c][i];
        }
        for (int q = 0; q < G; ++q) {
            t.ar[i][q] = (R)deriv_op(b, G, 0, i, q);
            t.as1[i][q] = (R)deriv_op(b, G, 1, i, q);
            t.as2[i][q] = (R)deriv_op(b, G, 2, i, q);
        }
        t.x0[i] = (R)b.x0[i]; t.n0[i] = (R)b.n0[i];
    }
    for (int m = 0; m < T; ++m) {
        double s = 0.0;
        for (int j = 0; j < G; ++j)
            for (int i = 0; i < G; ++i) s += b.gnwtn[m][j] * b.gxwtx[ModeCols<P>::col(m)][i];
        t.src[m] = (R)s;
    }
    for (int m = 0; m < T; ++m)
        t.odd[m] = (unsigned char)(m >= 3 && m < 3 * P && ((m - 3) % SD) % 2 ? (m - 3) / SD : 3);
    int n = 0, it = 0, col[T];
    for (int c = 0; c < X; ++c)
        for (int m = 0; m < T; ++m)
            if (ModeCols<P>::col(m) == c) {
                t.mode[n] = (unsigned char)m;
                col[n++] = c;
            }
    for (int w = 0; w < G; ++w) {
        t.iptr[w] = (unsigned char)it;
        for (int q = T * w / G; q < T * (w + 1) / G; ++q)
            if (q == T * w / G || col[q] != col[q - 1]) {
                t.icol[it] = (unsigned char)col[q];
                t.ifst[it++] = (unsigned char)q;
            }
    }
    t.iptr[G] = (unsigned char)it;
    t.ifst[it] = (unsigned char)T;
}

template <typename R, int P, int PHYS>
struct Impl {
    static constexpr bool F32 = std::is_same<R, float>::value, HAS_DIFF = F32 && PHYS == 1;
    static void build(const hp_basis_tables &b, std::vector<unsigned char> &out) {
        out.resize(sizeof(LineTab<R, P>));
        build_tab<R, P>(b, *reinterpret_cast<LineTab<R, P> *>(out.data()));
    }
    template <bool DIFF>
    static cudaError_t smem_attr() {
        const cudaError_t e = cudaFuncSetAttribute(k_rsdl_line<R, P, PHYS, DIFF, true>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   LineCfg<R, P, PHYS, DIFF, true>::SMEM);
        if (e != cudaSuccess) return e;
        return cudaFuncSetAttribute(k_rsdl_line<R, P, PHYS, DIFF, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    LineCfg<R, P, PHYS, DIFF, false>::SMEM);
    }
    static cudaError_t set_smem() {
        const cudaError_t e = smem_attr<false>();
        if constexpr (HAS_DIFF)
            if (e == cudaSuccess) return smem_attr<true>();
        return e;
    }
    template <bool DIFF, bool RE>
    static void go(const void *tab, const void *gtab, const Mesh &m, const State<R> &s, const LinePar &par, int nsm,
                   cudaStream_t st) {
        using C = LineCfg<R, P, PHYS, DIFF, RE>;
        const int nb = (m.ntri + 31) / 32;
        k_rsdl_line<R, P, PHYS, DIFF, RE><<<std::min(nb, nsm * C::MINB), C::NTHR, C::SMEM, st>>>(
            *static_cast<const LineTab<R, P> *>(tab), static_cast<const DevTables<R, P> *>(gtab), m, s, par);
    }
    static void launch(const void *tab, const void *gtab, const Mesh &m, const State<R> &s, const Phys &ph, int stage,
                       int zero_rr, int diff, int nsm, cudaStream_t st) {
        LinePar par;
        par.beta = ph.beta[stage];
        par.omb = zero_rr ? 0.0 : (double)((R)1 - (R)ph.beta[stage]);
        par.rho = ph.rho; par.mu = ph.mu; par.nu2 = 2. * (ph.mu / ph.rho); par.adis = ph.adis;
        par.rhocv = ph.rhocv; par.kcond = ph.kcond; par.ax = ph.ax; par.ay = ph.ay; par.src = ph.src;
        par.gfloor = ph.mu + ph.bd0 == 0.0 ? 1 : 0;
        const bool re = ph.beta[stage] > 0.0;
        if constexpr (HAS_DIFF) {
            if (diff) {
                if (re) go<true, true>(tab, gtab, m, s, par, nsm, st);
                else go<true, false>(tab, gtab, m, s, par, nsm, st);
                return;
            }
        }
        if (re) go<false, true>(tab, gtab, m, s, par, nsm, st);
        else go<false, false>(tab, gtab, m, s, par, nsm, st);
    }
    static void base_pts(const void *tab, const Mesh &m, const State<R> &s, R *bpt, cudaStream_t st) {
        if constexpr (HAS_DIFF)
            k_base_points<P><<<(m.ntri + 31) / 32, 64, 0, st>>>(static_cast<const DevTables<float, P> *>(tab), m, s.ubv,
                                                               s.ubs, s.ubi, bpt);
    }
    static size_t bpt_len(int ntri) {
        return (size_t)((ntri + 31) / 32) * 2 * (P + 1) * (P + 1) * 32;
    }
    static LineLaunch<R> get() {
        LineLaunch<R> l;
        l.build = &build;
        l.set_smem = &set_smem;
        l.launch = &launch;
        if (HAS_DIFF) {
            l.base_pts = &base_pts;
            l.bpt_len = &bpt_len;
        }
        return l;
    }
};

template <typename R, int PHYS>
LineLaunch<R> pick(int p) {
    switch (p) {
        case 1: return Impl<R, 1, PHYS>::get();
        case 2: return Impl<R, 2, PHYS>::get();
        case 3: return Impl<R, 3, PHYS>::get();
        case 4: return Impl<R, 4, PHYS>::get();
        case 5: return Impl<R, 5, PHYS>::get();
        case 6: return Impl<R, 6, PHYS>::get();
        case 7: return Impl<R, 7, PHYS>::get();
        case 8: return Impl<R, 8, PHYS>::get();
    }
    return LineLaunch<R>();
}

}  // namespace

template <>
LineLaunch<LINE_R> line_launch<LINE_R>(int p, int physics) {
    return physics == HP_PHYS_INS ? pick<LINE_R, 1>(p) : pick<LINE_R, 0>(p);
}

}  // namespace hpb
