// Table builder and launchers of the ins line kernel (hp_elem_line.cuh).
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
    constexpr int G = P + 1, X = P + 2, T = (P + 1) * (P + 2) / 2;
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
    for (int m = 0; m < T; ++m)
        t.odd[m] = (unsigned char)(m >= 3 && m < 3 * P && ((m - 3) % (P - 1)) % 2 ? (m - 3) / (P - 1) : 3);
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

template <typename R, int P>
struct Impl {
    static constexpr bool F32 = std::is_same<R, float>::value;
    static void build(const hp_basis_tables &b, std::vector<unsigned char> &out) {
        out.resize(sizeof(LineTab<R, P>));
        build_tab<R, P>(b, *reinterpret_cast<LineTab<R, P> *>(out.data()));
    }
    template <bool DIFF>
    static cudaError_t smem_attr() {
        using C = LineCfg<R, P, DIFF>;
        cudaError_t e = cudaFuncSetAttribute(k_rsdl_ins_line<R, P, DIFF, true>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        if (e != cudaSuccess) return e;
        return cudaFuncSetAttribute(k_rsdl_ins_line<R, P, DIFF, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    C::SMEM);
    }
    static cudaError_t set_smem() {
        const cudaError_t e = smem_attr<false>();
        if constexpr (F32)
            if (e == cudaSuccess) return smem_attr<true>();
        return e;
    }
    template <bool DIFF, bool RE>
    static void go(const void *tab, const Mesh &m, const State<R> &s, const Phys &ph, int stage, int zero_rr, int nsm,
                   cudaStream_t st) {
        using C = LineCfg<R, P, DIFF>;
        const int nb = (m.ntri + 31) / 32;
        k_rsdl_ins_line<R, P, DIFF, RE><<<std::min(nb, nsm * C::MINB), C::NTHR, C::SMEM, st>>>(
            *static_cast<const LineTab<R, P> *>(tab), m, s, (R)ph.beta[stage],
            zero_rr ? (R)0 : (R)1 - (R)ph.beta[stage], (R)ph.rho, (R)ph.mu, 2. * (ph.mu / ph.rho), ph.adis,
            ph.mu + ph.bd0 == 0.0 ? 1 : 0);
    }
    static void launch(const void *tab, const Mesh &m, const State<R> &s, const Phys &ph, int stage, int zero_rr,
                       int diff, int nsm, cudaStream_t st) {
        const bool re = ph.beta[stage] > 0.0;
        if constexpr (F32) {
            if (diff) {
                if (re) go<true, true>(tab, m, s, ph, stage, zero_rr, nsm, st);
                else go<true, false>(tab, m, s, ph, stage, zero_rr, nsm, st);
                return;
            }
        }
        if (re) go<false, true>(tab, m, s, ph, stage, zero_rr, nsm, st);
        else go<false, false>(tab, m, s, ph, stage, zero_rr, nsm, st);
    }
    static void base_pts(const void *tab, const Mesh &m, const State<R> &s, R *bpt, cudaStream_t st) {
        if constexpr (F32)
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
        if (F32) {
            l.base_pts = &base_pts;
            l.bpt_len = &bpt_len;
        }
        return l;
    }
};

}  // namespace

template <typename R>
LineLaunch<R> line_launch(int p) {
    switch (p) {
        case 2: return Impl<R, 2>::get();
        case 3: return Impl<R, 3>::get();
        case 4: return Impl<R, 4>::get();
        case 5: return Impl<R, 5>::get();
        case 6: return Impl<R, 6>::get();
        case 7: return Impl<R, 7>::get();
        case 8: return Impl<R, 8>::get();
    }
    return LineLaunch<R>();
}
template LineLaunch<double> line_launch<double>(int);
template LineLaunch<float> line_launch<float>(int);

}  // namespace hpb
