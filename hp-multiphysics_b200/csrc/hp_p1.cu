// Operators and launcher of the fused p = 1 stage kernel (hp_stage_p1.cuh).
#include <algorithm>

#include "hp_chain.cuh"
#include "hp_line.h"
#include "hp_stage_p1.cuh"

namespace hpb {

template <typename R>
void p1_ops(const hp_basis_tables &b, P1Ops<R> &o) {
    constexpr int G = 2;
    for (int q = 0; q < 4; ++q)
        for (int m = 0; m < 3; ++m) {
            const int i = q / G, j = q - i * G, c = ModeCols<1>::col(m);
            const double dr = b.n0[j] * b.gn[j][m] * b.dgx[i][c];
            o.V[q][m] = (R)(b.gn[j][m] * b.gx[i][c]);
            o.DR[q][m] = (R)dr;
            o.DS[q][m] = (R)(b.dgn[j][m] * b.gx[i][c] + b.x0[i] * dr);
            o.WR[q][m] = (R)(-b.dgxwtx[c][i] * b.gnwtnn0[m][j]);
            o.WS[q][m] = (R)(-(b.x0[i] * b.dgxwtx[c][i] * b.gnwtnn0[m][j] + b.gxwtx[c][i] * b.dgnwtn[m][j]));
            o.W0[q][m] = (R)(b.gnwtn[m][j] * b.gxwtx[c][i]);
        }
    for (int r = 0; r < G; ++r) {
        for (int k = 0; k < G; ++k) {
            o.AR[r][k] = (R)deriv_op(b, G, 0, r, k);
            o.AS1[r][k] = (R)deriv_op(b, G, 1, r, k);
            o.AS2[r][k] = (R)deriv_op(b, G, 2, r, k);
            o.BG[r][k] = (R)b.gx[r][1 + k];
            o.BD[r][k] = (R)b.dgx[r][1 + k];
            o.BW[r][k] = (R)b.gxwtx[1 + k][r];
        }
        o.N0[r] = (R)b.n0[r];
    }
}
template void p1_ops<double>(const hp_basis_tables &, P1Ops<double> &);
template void p1_ops<float>(const hp_basis_tables &, P1Ops<float> &);

template <typename R>
void p1_stage(const P1Ops<R> *ops, const Mesh &m, const P1Stage<R> &s, const Phys &ph, int diff, int nsm, int chained,
              cudaStream_t st) {
    const unsigned blocks = std::min((m.npnt + 3) / 4, nsm * (sizeof(R) == 8 ? 5 : 6));
    if (ph.physics == HP_PHYS_CD) launch_chained(chained, k_stage_p1<R, 0, false>, blocks, 128, 0, st, ops, m, s, ph);
    else if (diff) launch_chained(chained, k_stage_p1<R, 1, true>, blocks, 128, 0, st, ops, m, s, ph);
    else launch_chained(chained, k_stage_p1<R, 1, false>, blocks, 128, 0, st, ops, m, s, ph);
}
template void p1_stage<double>(const P1Ops<double> *, const Mesh &, const P1Stage<double> &, const Phys &, int, int,
                               int, cudaStream_t);
template void p1_stage<float>(const P1Ops<float> *, const Mesh &, const P1Stage<float> &, const Phys &, int, int, int,
                              cudaStream_t);

template <typename R>
void p1_vert(const P1Ops<R> *ops, const Mesh &m, const R *elim, const R *elre, const P1Stage<R> &s, const Phys &ph,
             int diff, cudaStream_t str) {
    const int n = m.npnt * (ph.physics == HP_PHYS_INS ? 3 : 1), blocks = (n + 127) / 128;
    if (ph.physics == HP_PHYS_CD) k_vert_p1<R, 0, false><<<blocks, 128, 0, str>>>(ops, m, elim, elre, s, ph);
    else if (diff) k_vert_p1<R, 1, true><<<blocks, 128, 0, str>>>(ops, m, elim, elre, s, ph);
    else k_vert_p1<R, 1, false><<<blocks, 128, 0, str>>>(ops, m, elim, elre, s, ph);
}
template void p1_vert<double>(const P1Ops<double> *, const Mesh &, const double *, const double *,
                              const P1Stage<double> &, const Phys &, int, cudaStream_t);
template void p1_vert<float>(const P1Ops<float> *, const Mesh &, const float *, const float *, const P1Stage<float> &,
                             const Phys &, int, cudaStream_t);

}  // namespace hpb
