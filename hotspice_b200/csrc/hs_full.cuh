// One cell of the direct full sum (hotspice/energies.py:290-308), shared by the direct kernel and
// by the fast convolution's fallback for non-finite inputs.
#pragma once

#include "hs_common.cuh"

// sum_j K_{s}(j - i) mm_j and, with use_perp, the perp-self sum, of target cell (y, x) on
// sublattice s >= 0, over every cell (FULLWIN) or over the window.
template <typename Acc, bool FULLWIN>
HS_DEV void dip_full_cell(const HsLattice &L, int s, int y, int x, Acc &acc, Acc &accp) {
    acc = 0;
    accp = 0;
    if (FULLWIN) {
        for (int jy = 0; jy < L.ny; ++jy) {
            const int dy = jy - y;
            const int64_t jrow = (int64_t)jy * L.nx;
            for (int jx = 0; jx < L.nx; ++jx) {
                const Acc mj = (Acc)L.mm[jrow + jx];
                if (mj == (Acc)0) continue;
                acc += (Acc)hs_kval(L, L.K, s, dy, jx - x) * mj;
                if (L.use_perp) accp += (Acc)hs_kval(L, L.Kps, s, dy, jx - x) * mj;
            }
        }
    } else {
        for (int dy = -L.dip_wy; dy <= L.dip_wy; ++dy) {
            int jy = y + dy;
            if (L.dip_wrap) jy = hs_wrap(jy, L.ny);
            else if (jy < 0 || jy >= L.ny) continue;
            const int64_t jrow = (int64_t)jy * L.nx;
            for (int dx = -L.dip_wx; dx <= L.dip_wx; ++dx) {
                int jx = x + dx;
                if (L.dip_wrap) jx = hs_wrap(jx, L.nx);
                else if (jx < 0 || jx >= L.nx) continue;
                const Acc mj = (Acc)L.mm[jrow + jx];
                if (mj == (Acc)0) continue;
                const int64_t k = (int64_t)s * (2 * L.dip_wy + 1) * (2 * L.dip_wx + 1) +
                                  (int64_t)(dy + L.dip_wy) * (2 * L.dip_wx + 1) + (dx + L.dip_wx);
                acc += (Acc)__ldg(L.K + k) * mj;
                if (L.use_perp) accp += (Acc)__ldg(L.Kps + k) * mj;
            }
        }
    }
}
