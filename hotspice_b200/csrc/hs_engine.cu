// Persistent cluster engine: many update steps of many lattice instances in one launch.
//
// Each thread-block cluster (CS CTAs, CS in {1, 2, 4, 8, 16}) repeatedly claims an instance
// from a work counter and advances it by its step budget (or until the progress() stop
// rule of hotspice/core.py:753-760 holds), with cluster barriers between the phases of a
// step instead of kernel boundaries:
//   Metropolis: [CTA 0] selection + acceptance + flips (metro_step_cta)  | barrier |
//               [all]   dipolar update of the touched strips              | barrier |
//   Néel:       on owned cells for a uniform temperature (neel_run_owned); else
//               [all]   barrier/log-time keys of a slice of the cells, CTA argmin -> CTA 0
//                       through distributed shared memory                 | barrier |
//               [CTA 0] final argmin, switching time, flip                | barrier |
//               [all]   dipolar update                                    | barrier |
//   Wolff:      [CTA 0] sparse cluster growth (wolff_step_cta)            | barrier |
// Every branch that decides how many barriers are executed is taken on values every CTA of
// the cluster reads after a barrier, so all CTAs always execute the same barrier sequence.
//
// The dipolar update of up to FEW_MAX switches distributes pieces of their windows (few_items); a
// longer list's distributes work items (switch k, window row, 128-column segment) over
// all warps of the cluster. A strip (row, segment) is processed by the item of the first
// switch whose window covers it, which accumulates the contributions of every covering
// switch in list order: each strip is written once, deterministically, and the work is
// proportional to the area the windows touch.
#include <cooperative_groups.h>

#include "hs_steps.cuh"
#include "hs_internal.h"

namespace cg = cooperative_groups;

namespace {

#ifndef HS_ENGINE_THREADS
#define HS_ENGINE_THREADS 512
#endif
#ifndef HS_ENGINE_REGS
#define HS_ENGINE_REGS 128
#endif
#ifndef HS_NEEL_WIN_UNROLL
#define HS_NEEL_WIN_UNROLL 4
#endif
constexpr int ENG_NT = HS_ENGINE_THREADS;   // threads per CTA
constexpr int ENG_MIN_CTAS = 65536 / (ENG_NT * HS_ENGINE_REGS);  // resident CTAs per SM at that register budget
constexpr int ENG_FEW_R = 4;    // rows per item of a short list: 128 registers hold four rows' cells
constexpr int ENG_SWCAP = 512;  // switches staged per CTA in shared memory
constexpr int ENG_WS_MAX = HS_ENGINE_WS_MAX;  // largest dynamic shared workspace a launch may ask for

struct SwX {                    // staged switch with its window footprint
    int y, x, mode, sub;
    float mm;
    int ylo, nrows;             // window rows: (ylo + i) mod ny, i < nrows
    int sa0, sa1, sb0, sb1;     // covered 32-column segments: [sa0, sa1) and [sb0, sb1)
};

HS_DEV void footprint(const HsLattice &L, SwX &w) {
    int hy, wy, hx, wx;
    hs_window(L, w.mode, true, hy, wy);
    hs_window(L, w.mode, false, hx, wx);
    const int nseg = (L.nx + 31) >> 5;
    if (wy) {
        if (2 * hy + 1 >= L.ny) { w.ylo = 0; w.nrows = L.ny; }
        else { w.ylo = hs_wrap(w.y - hy, L.ny); w.nrows = 2 * hy + 1; }
    } else {
        const int lo = max(0, w.y - hy), hi = min(L.ny - 1, w.y + hy);
        w.ylo = lo; w.nrows = hi - lo + 1;
    }
    w.sb0 = w.sb1 = 0;
    if (wx && 2 * hx + 1 >= L.nx) { w.sa0 = 0; w.sa1 = nseg; }
    else if (wx) {
        const int lo = w.x - hx, hi = w.x + hx;
        if (lo >= 0 && hi < L.nx) { w.sa0 = lo >> 5; w.sa1 = (hi >> 5) + 1; }
        else if (lo < 0) { w.sa0 = 0; w.sa1 = (hi >> 5) + 1; w.sb0 = (lo + L.nx) >> 5; w.sb1 = nseg; }
        else { w.sa0 = lo >> 5; w.sa1 = nseg; w.sb0 = 0; w.sb1 = ((hi - L.nx) >> 5) + 1; }
        if (w.sb1 > w.sb0 && w.sb0 < w.sa1 && w.sa0 < w.sb1) {  // ranges touch: merge
            w.sa0 = min(w.sa0, w.sb0); w.sa1 = max(w.sa1, w.sb1); w.sb0 = w.sb1 = 0;
        }
    } else {
        const int lo = max(0, w.x - hx), hi = min(L.nx - 1, w.x + hx);
        w.sa0 = lo >> 5; w.sa1 = (hi >> 5) + 1;
    }
}

// Stage the switch list into shared memory with footprints.
HS_DEV int stage_switches(const HsLattice &L, const HsSwitchList &sw, int nsw, SwX *s_sw) {
    const int n = min(nsw, ENG_SWCAP);
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        SwX w;
        w.y = __ldcg(sw.y + k); w.x = __ldcg(sw.x + k); w.mode = sw.mode ? __ldcg(sw.mode + k) : 0;
        w.sub = hs_sub(L, w.y, w.x);
        w.mm = __ldcg(L.mm + (int64_t)w.y * L.nx + w.x);
        footprint(L, w);
        s_sw[k] = w;
    }
    __syncthreads();
    return n;
}

// Contributions of staged switch w to the 4 cells x0..x0+3 of `row`; tch[v] is set for every
// cell inside the switch's window.
HS_DEV void contrib4(const HsLattice &L, const SwX &w, int row, int x0, float acc[4], float accp[4], bool neg[4],
                     bool tch[4]) {
    if (!w.mode && !L.dip_wrap) {
        // exact window without wrapping: one kernel row, consecutive columns
        const int dy = row - w.y;
        if (dy < -L.dip_wy || dy > L.dip_wy) return;
        const int64_t W = 2 * L.dip_wx + 1, H = 2 * L.dip_wy + 1;
        const int64_t base = (int64_t)w.sub * H * W + (int64_t)(dy + L.dip_wy) * W + (L.dip_wx - w.x);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int x = x0 + v, dx = x - w.x;
            if (x < L.nx && dx >= -L.dip_wx && dx <= L.dip_wx) {
                tch[v] = true;
                acc[v] += w.mm * __ldg(L.K + base + x);
                if (L.use_perp) accp[v] += w.mm * __ldg(L.Kpo + base + x);
            }
            if (dy == 0 && dx == 0) neg[v] = true;
        }
        return;
    }
    SwInfo wi{w.y, w.x, w.mode, w.sub, w.mm};
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const int x = x0 + v;
        if (x >= L.nx) continue;
        tch[v] = true;
        hs_contrib(L, wi, row, x, acc[v], accp[v]);
        if (w.y == row && w.x == x) neg[v] = true;
    }
}

HS_DEV bool covers_seg(const HsLattice &L, const SwX &w, int row, int seg128) {
    int d = row - w.ylo;
    if (d < 0) d += L.ny;
    if (d >= w.nrows) return false;
    // 128-column segment seg128 spans 32-column segments [4 seg128, 4 seg128 + 4)
    const int a0 = 4 * seg128, a1 = a0 + 4;
    return (a0 < w.sa1 && w.sa0 < a1) || (a0 < w.sb1 && w.sb0 < a1);
}

// Dipolar update of the strips covered by the staged switches. Work item = (switch k, one
// row of its window); warps gw = 0..nw-1 of the whole cluster take items gw, gw + nw, ...
// Along the row the warp walks 128-column segments (4 cells per lane). A segment is written
// by the item of the first switch covering it, which accumulates every covering switch in
// list order.
HS_DEV void update_items(const HsLattice &L, const SwX *s_sw, int n, int semantics, int gw, int nw,
                         const HsSwitchList &sw, int nsw_total) {
    if (n == 0) return;
    const int lane = threadIdx.x & 31;
    const float pref2 = (float)(2.0 * L.dip_pref);
    const bool vec = (L.nx & 3) == 0;
    const bool flip_perp = !(L.dip_keep_perp_sign && nsw_total > 1);  // one switch: update_single
    int it0 = 0;
    for (int k = 0; k < n; ++k) {
        const SwX &wk = s_sw[k];
        if (wk.sub < 0) continue;
        const int nr = wk.nrows;
        // first item index of this switch assigned to this warp
        int r = gw - it0;
        r %= nw; if (r < 0) r += nw;
        for (; r < nr; r += nw) {
            int row = wk.ylo + r;
            if (row >= L.ny) row -= L.ny;
            // 128-column segments this switch covers in this row
            const int ranges[2][2] = {{wk.sa0 >> 2, (wk.sa1 + 3) >> 2}, {wk.sb0 >> 2, (wk.sb1 + 3) >> 2}};
            for (int g = 0; g < 2; ++g) {
                for (int seg = ranges[g][0]; seg < ranges[g][1]; ++seg) {
                    if (g == 1 && seg >= ranges[0][0] && seg < ranges[0][1]) continue;  // already done in range 0
                    bool owned = true;
                    for (int q = 0; q < k; ++q)
                        if (s_sw[q].sub >= 0 && covers_seg(L, s_sw[q], row, seg)) { owned = false; break; }
                    if (!owned) continue;  // warp-uniform
                    const int x0 = seg * 128 + lane * 4;
                    float acc[4] = {0.f, 0.f, 0.f, 0.f}, accp[4] = {0.f, 0.f, 0.f, 0.f};
                    bool neg[4] = {false, false, false, false}, tch[4] = {false, false, false, false};
                    for (int q = k; q < n; ++q) {
                        const SwX &w = s_sw[q];
                        if (w.sub < 0 || !covers_seg(L, w, row, seg)) continue;
                        contrib4(L, w, row, x0, acc, accp, neg, tch);
                    }
                    for (int q = n; q < nsw_total; ++q) {  // beyond the staged ones: from global memory
                        SwX w;
                        w.y = __ldcg(sw.y + q); w.x = __ldcg(sw.x + q); w.mode = sw.mode ? __ldcg(sw.mode + q) : 0;
                        w.sub = hs_sub(L, w.y, w.x);
                        if (w.sub < 0) continue;
                        w.mm = __ldcg(L.mm + (int64_t)w.y * L.nx + w.x);
                        footprint(L, w);
                        if (!covers_seg(L, w, row, seg)) continue;
                        contrib4(L, w, row, x0, acc, accp, neg, tch);
                    }
                    // cells that no window reaches keep their energies (E + 0 = E): skip the
                    // read-modify-write of lanes whose 4 cells are all outside the windows
                    if (x0 >= L.nx || !(tch[0] || tch[1] || tch[2] || tch[3])) continue;
                    const int64_t i = (int64_t)row * L.nx + x0;
                    float mv[4];
                    double ev[4], pv[4];
                    if (vec) {
                        const float4 a = __ldcg(reinterpret_cast<const float4 *>(L.mm + i));
                        const double2 e0 = __ldcg(reinterpret_cast<const double2 *>(L.E_dip + i));
                        const double2 e1 = __ldcg(reinterpret_cast<const double2 *>(L.E_dip + i + 2));
                        mv[0] = a.x; mv[1] = a.y; mv[2] = a.z; mv[3] = a.w;
                        ev[0] = e0.x; ev[1] = e0.y; ev[2] = e1.x; ev[3] = e1.y;
                        if (L.use_perp) {
                            const double2 p0 = __ldcg(reinterpret_cast<const double2 *>(L.E_dip_perp + i));
                            const double2 p1 = __ldcg(reinterpret_cast<const double2 *>(L.E_dip_perp + i + 2));
                            pv[0] = p0.x; pv[1] = p0.y; pv[2] = p1.x; pv[3] = p1.y;
                        }
                    } else {
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            const bool in = x0 + v < L.nx;
                            mv[v] = in ? __ldcg(L.mm + i + v) : 0.f;
                            ev[v] = in ? __ldcg(L.E_dip + i + v) : 0.0;
                            pv[v] = (in && L.use_perp) ? __ldcg(L.E_dip_perp + i + v) : 0.0;
                        }
                    }
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        if (semantics == HS_UPDATE_MULTIPLE) {
                            if (neg[v]) { ev[v] = -ev[v]; if (flip_perp) pv[v] = -pv[v]; }
                            ev[v] += (double)(pref2 * (mv[v] * acc[v]));
                            pv[v] += (double)(pref2 * (mv[v] * accp[v]));
                        } else {
                            ev[v] += (double)(pref2 * (mv[v] * acc[v]));
                            pv[v] += (double)(pref2 * (mv[v] * accp[v]));
                            if (neg[v]) { ev[v] = -ev[v]; pv[v] = -pv[v]; }
                        }
                    }
                    if (vec) {
                        *reinterpret_cast<double2 *>(L.E_dip + i) = make_double2(ev[0], ev[1]);
                        *reinterpret_cast<double2 *>(L.E_dip + i + 2) = make_double2(ev[2], ev[3]);
                        if (L.use_perp) {
                            *reinterpret_cast<double2 *>(L.E_dip_perp + i) = make_double2(pv[0], pv[1]);
                            *reinterpret_cast<double2 *>(L.E_dip_perp + i + 2) = make_double2(pv[2], pv[3]);
                        }
                    } else {
                        for (int v = 0; v < 4 && x0 + v < L.nx; ++v) {
                            L.E_dip[i + v] = ev[v];
                            if (L.use_perp) L.E_dip_perp[i + v] = pv[v];
                        }
                    }
                }
            }
        }
        it0 += nr;
    }
}

// Window update of a single switch (the Néel step without the owner path): every thread of the
// cluster takes window cells directly (row-major over the window, consecutive threads on
// consecutive columns) and issues the loads of its cells together. Per cell the arithmetic is that
// of update_items for one switch (acc = mm_s K, E += 2 pref mm_j acc in the same float order, then
// E_s negated), so the energies are the same bit for bit; cells outside the window receive nothing
// there either.
HS_DEV void update_one(const HsLattice &L, int sy, int sx, float smm, int t0, int nt) {
    const int sub = hs_sub(L, sy, sx);
    if (sub < 0) return;
    int hy, wy, hx, wx;
    hs_window(L, 0, true, hy, wy);
    hs_window(L, 0, false, hx, wx);
    int ylo, nrows, xlo, ncols;
    if (wy) {
        if (2 * hy + 1 >= L.ny) { ylo = 0; nrows = L.ny; } else { ylo = hs_wrap(sy - hy, L.ny); nrows = 2 * hy + 1; }
    } else { ylo = max(0, sy - hy); nrows = min(L.ny - 1, sy + hy) - ylo + 1; }
    if (wx) {
        if (2 * hx + 1 >= L.nx) { xlo = 0; ncols = L.nx; } else { xlo = hs_wrap(sx - hx, L.nx); ncols = 2 * hx + 1; }
    } else { xlo = max(0, sx - hx); ncols = min(L.nx - 1, sx + hx) - xlo + 1; }
    const int total = nrows * ncols;
    const float pref2 = (float)(2.0 * L.dip_pref);
    const bool two = L.use_perp != 0;
    constexpr int U = HS_NEEL_WIN_UNROLL;   // window cells per thread per pass
    // window cell c = r ncols + q of this thread, advanced by nt cells per slot without divisions
    const int dr = nt / ncols, dq = nt - dr * ncols;
    int r0 = t0 / ncols, q0 = t0 - r0 * ncols;
    for (int base = t0; base < total; base += nt * U) {
        int idx[U], rw[U], cl[U];
        float kv[U], kp[U], mv[U];
        double ev[U], pv[U];
        bool live[U];   // in the window and on a unit-cell site that holds magnets
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int c = base + k * nt;
            const int r = r0, q = q0;
            r0 += dr; q0 += dq;
            if (q0 >= ncols) { q0 -= ncols; ++r0; }
            int row = ylo + r, col = xlo + q;
            if (row >= L.ny) row -= L.ny;
            if (col >= L.nx) col -= L.nx;
            rw[k] = row; cl[k] = col;
            idx[k] = row * L.nx + col;
            // a site without a kernel never holds a magnet: its energy stays 0 (the reference adds
            // m * ... = 0 there)
            live[k] = c < total && hs_sub(L, row, col) >= 0;
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const bool v = live[k];
            const int i = idx[k];
            kv[k] = v ? hs_kval(L, L.K, sub, rw[k] - sy, cl[k] - sx) : 0.f;
            kp[k] = (v && two) ? hs_kval(L, L.Kpo, sub, rw[k] - sy, cl[k] - sx) : 0.f;
            // the switched cell's new moment comes from the handover (smm): its global write may
            // still be in flight
            mv[k] = v ? (rw[k] == sy && cl[k] == sx ? smm : __ldcg(L.mm + i)) : 0.f;
            ev[k] = v ? __ldcg(L.E_dip + i) : 0.0;
            pv[k] = (v && two) ? __ldcg(L.E_dip_perp + i) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            if (!live[k]) continue;
            const int i = idx[k];
            float acc = 0.f, accp = 0.f;
            acc += smm * kv[k];
            if (two) accp += smm * kp[k];
            double e = ev[k] + (double)(pref2 * (mv[k] * acc));
            double p = pv[k] + (double)(pref2 * (mv[k] * accp));
            if (rw[k] == sy && cl[k] == sx) { e = -e; p = -p; }
            L.E_dip[i] = e;
            if (two) L.E_dip_perp[i] = p;
        }
    }
}

template <int CS>
struct Sync {
    HS_DEV static void all() {
        if constexpr (CS == 1) __syncthreads();
        else cg::this_cluster().sync();
    }
    // all(), with f() run by the threads for which `run` holds between their arrival and their
    // wait (cluster barrier: its release covers only what came before the arrival)
    template <typename F>
    HS_DEV static void all_then(bool run, F f) {
        if constexpr (CS == 1) {
            if (run) f();
            __syncthreads();
        } else {
            asm volatile("barrier.cluster.arrive;" ::: "memory");
            if (run) f();
            asm volatile("barrier.cluster.wait;" ::: "memory");
        }
    }
    HS_DEV static int rank() {
        if constexpr (CS == 1) return 0;
        else return (int)cg::this_cluster().block_rank();
    }
    template <typename T>
    HS_DEV static void publish(T *local, T v) {  // rank 0 thread writes v into every CTA's copy
        if constexpr (CS == 1) *local = v;
        else {
            cg::cluster_group c = cg::this_cluster();
            for (int r = 0; r < CS; ++r) *c.map_shared_rank(local, r) = v;
        }
    }
};

// Block minimum of (key, index).
HS_DEV HsKeyIdx eng_block_kmin(HsKeyIdx v, HsKeyIdx *sm) {
    v = hs_warp_kmin(v);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = (lane < (int)(blockDim.x >> 5)) ? sm[lane] : HsKeyIdx{0.0, -1};
        v = hs_warp_kmin(v);
    }
    __syncthreads();
    return v;
}

HS_DEV double eng_block_dmin(double v, double *sm) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = (lane < (int)(blockDim.x >> 5)) ? sm[lane] : INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    }
    __syncthreads();
    return v;
}

HS_DEV MetroScratch metro_scratch_of(const HsLattice &L, const HsGridPlan &P, void *base) {
    int cap, gsz;
    hs_metro_sizes(L, P, cap, gsz);
    char *p = reinterpret_cast<char *>(base);
    MetroScratch S;
    S.cap = cap; S.gsz = gsz;
    S.py = reinterpret_cast<int32_t *>(p); S.px = S.py + cap; p += hs_align_up_d(8LL * cap, 256);
    S.grid = reinterpret_cast<int32_t *>(p); p += hs_align_up_d(4LL * gsz, 256);
    S.ptx = reinterpret_cast<double *>(p); p += hs_align_up_d(8LL * gsz, 256);
    S.pty = reinterpret_cast<double *>(p); p += hs_align_up_d(8LL * gsz, 256);
    S.queue = reinterpret_cast<int32_t *>(p);
    return S;
}

HS_DEV WolffScratch wolff_scratch_of(const HsLattice &L, void *base) {
    const int64_t N = (int64_t)L.nx * L.ny;
    char *p = reinterpret_cast<char *>(base);
    WolffScratch S;
    S.chk_ep = reinterpret_cast<int32_t *>(p); p += hs_align_up_d(4 * N, 256);
    S.cl_ep = reinterpret_cast<int32_t *>(p); p += hs_align_up_d(4 * N, 256);
    S.list = reinterpret_cast<int32_t *>(p); p += hs_align_up_d(4 * N, 256);
    S.cand = reinterpret_cast<int32_t *>(p); p += hs_align_up_d(4 * N, 256);
    S.epoch = reinterpret_cast<int32_t *>(p);
    return S;
}

constexpr int NEEL_OWN_UY = 64;     // rows of a period that the owner path's table holds

// Shared state of one CTA while it runs an instance.
struct __align__(16) EngShared {
    HsInstance I;                       // the instance descriptor, staged (read through references)
    HsCounters C;                       // rank 0: the instance's counters for the whole run
    unsigned long long call[2];         // Philox call of step st in call[st & 1]
    HsKeyIdx part[2][16];               // owner path: the CTAs' minima of step st in part[st & 1]
    HsKeyIdx red[32];
    double dred[32];
    int inst, n1, y1, x1, nsw;
    int go[2];                          // step st runs while go[st & 1] (double-buffered)
    float mm1;
    double thr[2];                      // owner path: a key below thr[st & 1] switches for certain
    int few_w[FEW_MAX / 32];
    float tw[32];                       // owner path: the warps' bounds
    int rowpre[NEEL_OWN_UY + 1];        // owner path: occupied cells before row y of a period of uy rows
    union {
        struct { int q[ENG_NT / 32][NEEL_QCAP]; float lb[ENG_NT / 32][NEEL_QCAP]; } nq;   // owner path: candidates
        SwX sw[ENG_SWCAP];
        FewSw few[FEW_MAX];
        WolffFast wolff;
    };
};
static_assert(sizeof(HsInstance) % 8 == 0, "HsInstance is copied in 8-byte words");
static_assert(sizeof(HsCounters) % 8 == 0, "HsCounters is copied in 8-byte words");

// Barriers and publication over the CTAs that run the current instance: the whole cluster, or
// this CTA alone (CTA mode). One copy of the step code serves both (a uniform branch per
// barrier), which keeps the kernel's register allocation that of the cluster path.
template <int CS>
struct RunSync {
    bool alone;
    HS_DEV void all() const {
        if (CS == 1 || alone) __syncthreads();
        else Sync<CS>::all();
    }
    template <typename F>
    HS_DEV void all_then(bool run, F f) const {
        if (CS == 1 || alone) { if (run) f(); __syncthreads(); }
        else Sync<CS>::all_then(run, f);
    }
    template <typename T>
    HS_DEV void publish(T *local, T v) const {
        if (CS == 1 || alone) *local = v;
        else Sync<CS>::publish(local, v);
    }
    // v into every CTA's copy of *local, one CTA per lane of the calling warp
    template <typename T>
    HS_DEV void publish_warp(T *local, T v, int n_cta) const {
        const int lane = threadIdx.x & 31;
        if (CS == 1 || alone) { if (lane == 0) *local = v; }
        else if (lane < n_cta) *cg::this_cluster().map_shared_rank(local, lane) = v;
    }
    // *from (in this CTA) into every CTA's copy of *local, 8 bytes per lane of the calling warp
    template <typename T>
    HS_DEV void copy_to_all(T *local, const T *from, int n_cta) const {
        constexpr int NW = sizeof(T) / 8;
        static_assert(sizeof(T) % 8 == 0, "copied in 8-byte words");
        const unsigned long long *src = reinterpret_cast<const unsigned long long *>(from);
        for (int k = threadIdx.x & 31; k < n_cta * NW; k += 32)
            reinterpret_cast<unsigned long long *>(cg::this_cluster().map_shared_rank(local, k / NW))[k % NW] = src[k % NW];
    }
    // rank 0's slot r of a per-CTA array receives v (r = this CTA's rank)
    template <typename T>
    HS_DEV void to_rank0(T *arr, int r, T v) const {
        if constexpr (CS == 1) arr[0] = v;
        else if (alone) arr[0] = v;
        else *cg::this_cluster().map_shared_rank(&arr[r], 0) = v;
    }
};

// ---- Néel steps with owned cells ---------------------------------------------------------
// The Néel path for a uniform temperature without exchange (bounds per cell that only a switch in
// reach changes). A step is one scan, one exchange of minima and one window update. The magnets are
// numbered in cell order ("slots"; the cell itself when every cell holds one), and chunk c of 32
// slots belongs to warp c mod W of the instance's W owner warps: the same lane scans a slot,
// updates its energies and refreshes its bound for the whole run. So what a warp reads it wrote
// itself, the energies stay in its SM's L1, and no barrier separates an update from the next scan.
// Per step: two block barriers and, on a cluster, one cluster barrier.
//   scan      per slot the bound log u + s from the first Philox word (s = b_low beta rounded down,
//             kept per slot); a warp queues the slots whose bound does not rule them out
//   barrier   the block's smallest upper bound; what it rules out leaves the queues, the exact keys
//             of the rest (a few in the block) are computed
//   exchange  the CTA's winner goes to every CTA of the cluster; each warp takes the minimum itself
//   update    the owners of the window's slots; meanwhile one helper warp of rank 0, which owns no
//             slots, computes the switching time, the counters and the stop rule (neel_finalize),
//             which the next step needs only at its exchange.
// A switch whose key is clearly below the limit thr (log of the time left, 1e-3 off) happens for
// certain and its update does not wait for the time; otherwise the helper decides first.
// Results are those of the step kernels bit for bit (same keys, same updates).
// Measured (B200), us per step, cutoff 16a, before (all threads scan and update any cell, the record
// decided by one thread between two cluster barriers) and now: 64 x 64 uncut on one CTA 15.5 -> 9.6,
// on 16 CTAs 12.2 -> 4.7; 200 x 111 kagome on two CTAs 20.2 -> 11.9, on 16 13.6 -> 6.1. Bound on one
// CTA: instructions (IPC 2.3, L1 hit rate 99.6%); on 16: the latency of the chain scan 1,800 cycles,
// exact key 800, exchange 2,100, update 3,100.
HS_DEV unsigned ordered_f32(float f) {
    const unsigned b = __float_as_uint(f);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}
HS_DEV float unordered_f32(unsigned b) { return __uint_as_float(b & 0x80000000u ? b & 0x7fffffffu : ~b); }
HS_DEV float warp_min_f32(float f) { return unordered_f32(__reduce_min_sync(0xffffffffu, ordered_f32(f))); }

// Lane holding the smallest (key, idx) of the warp (idx < 0: no candidate), or -1.
HS_DEV int warp_kmin_lane(double key, int idx) {
    uint64_t k = (uint64_t)__double_as_longlong(key + 0.0);
    k = k >> 63 ? ~k : k | (1ULL << 63);
    // every lane takes part in every reduction
    bool c = idx >= 0;
    const unsigned hi = c ? (unsigned)(k >> 32) : 0xffffffffu;
    const unsigned mhi = __reduce_min_sync(0xffffffffu, hi);
    c = c && hi == mhi;
    const unsigned lo = c ? (unsigned)k : 0xffffffffu;
    const unsigned mlo = __reduce_min_sync(0xffffffffu, lo);
    c = c && lo == mlo;
    const unsigned id = c ? (unsigned)idx : 0xffffffffu;
    const unsigned mid = __reduce_min_sync(0xffffffffu, id);
    c = c && id == mid;
    return __ffs(__ballot_sync(0xffffffffu, c)) - 1;
}

// What the owner path reads of the lattice, in registers: through the descriptor in shared memory
// every field would be loaded again after each store to an array (which might alias it): 64 x 64
// uncut on one CTA 11.0 -> 9.2 us per step.
struct NeelOwn {
    int W, w;            // owner warps of the instance, and this one
    int M, nch;          // slots, chunks
    float *s;            // bound per slot
    const int32_t *list; // occupied cells, or null when the slots are the cells
    double *E, *Ep;      // null without a dipolar energy (a second channel)
    int8_t *m;
    float *mm;
    const float *zee, *zeep, *EB, *K, *Kpo;
    double beta, m_perp_factor;
    int nx, ny, wy, wx, dip_wrap, use_perp, barrier_method;
    float pref2, inv_W, inv_nx;
};

HS_DEV int own_cell(const NeelOwn &O, int j) { return O.list ? __ldg(O.list + j) : j; }

// First slot at or after row y.
HS_DEV int own_row(const HsLattice &L, const NeelOwn &O, const int *rowpre, int y) {
    if (!O.list) return y * L.nx;
    if (L.uy <= NEEL_OWN_UY) {
        const int p = y / L.uy;
        return p * rowpre[L.uy] + rowpre[y - p * L.uy];
    }
    int lo = 0, hi = O.M;                 // a period longer than the table: search the sorted list
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(L.nonzero + mid) < y * L.nx) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// What a cell's bound needs besides its energies and spin.
struct OwnStatic { float zee, zeep, EB; };
HS_DEV OwnStatic own_static(const NeelOwn &O, int i, bool v) {
    return OwnStatic{(v && O.zee) ? __ldg(O.zee + i) : 0.f, (v && O.zee && O.use_perp) ? __ldg(O.zeep + i) : 0.f,
                     v ? __ldg(O.EB + i) : 0.f};
}
// Bound of a cell with energies E, Ep and spin m, rounded down.
HS_DEV float own_bound(const NeelOwn &O, const OwnStatic &c, double E, double Ep, int m) {
    if (O.zee) {
        E += (double)m * (double)c.zee;
        if (O.use_perp) Ep += (double)m * (double)c.zeep;
    }
    double b1, b2;
    hs_barriers_from(O, E, Ep, (double)c.EB, b1, b2);
    return __double2float_rd(fmin(b1, b2) * O.beta);
}

// Exact log-domain key of occupied cell i from its (owned) energies: the operations of
// neel_scan_range with b_min = 0, so both give the same key bit for bit.
HS_DEV HsKeyIdx own_key(const NeelOwn &O, int i, uint32_t call_lo, uint32_t call_hi, const HsRoundKeys &RK) {
    double E = O.E ? O.E[i] : 0.0, Ep = O.Ep ? O.Ep[i] : 0.0;
    const int mv = O.m[i];
    const float mm = O.mm[i];
    const double uk = hs_u53_of(hs_philox_rk((uint32_t)i, call_lo, call_hi, 0u, RK));
    if (O.zee) { E += (double)mv * (double)__ldg(O.zee + i); if (O.use_perp) Ep += (double)mv * (double)__ldg(O.zeep + i); }
    double b1, b2;
    hs_barriers_from(O, E, Ep, (double)__ldg(O.EB + i), b1, b2);
    const double le1 = (double)hs_log_exp1_f32(uk);
    double key;
    if (!O.use_perp) key = le1 + b1 * O.beta;
    else {
        const double bm = fmin(b1, b2), dd = fabs(b1 - b2);
        key = le1 + bm * O.beta - (double)log1pf(expf((float)(-dd * O.beta)));
    }
    return HsKeyIdx{key, i, b1, b2, mm, mv};
}

// The warp's part of a scan: queues the slots that may hold the smallest key and returns an upper
// bound T of the smallest key among its slots. `best` collects exact keys when the queue fills up.
template <int OWN_UNR>       // chunks in flight
HS_DEV float own_scan_u(const NeelOwn &O, uint64_t call, const HsRoundKeys &RK, int *q, float *ql,
                      int &qn, HsKeyIdx &best) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t call_lo = (uint32_t)call, call_hi = (uint32_t)(call >> 32);
    const float slack = O.use_perp ? 0.69314722f + 1e-4f : 1e-4f;   // two channels lower a key by at most ln 2
    float T = INFINITY;   // warp-uniform, as qn
    qn = 0;
    auto load = [&](int c, int (&ci)[OWN_UNR], float (&sc)[OWN_UNR]) {
#pragma unroll
        for (int k = 0; k < OWN_UNR; ++k) {
            const int cc = c + k * O.W, j = 32 * cc + lane;
            const bool v = cc < O.nch && j < O.M;
            ci[k] = v ? own_cell(O, j) : 0;
            sc[k] = v ? O.s[j] : INFINITY;
        }
    };
    int ci[OWN_UNR];
    float sc[OWN_UNR];
    load(O.w, ci, sc);
    for (int c = O.w; c < O.nch; c += OWN_UNR * O.W) {
        int cn[OWN_UNR];
        float sn[OWN_UNR];
        load(c + OWN_UNR * O.W, cn, sn);
        uint32_t x[OWN_UNR];
#pragma unroll
        for (int k = 0; k < OWN_UNR; ++k) x[k] = hs_philox_rk((uint32_t)ci[k], call_lo, call_hi, 0u, RK).x;
        // lower bounds, rounded down; the slot of the lane's smallest gives an upper bound
        float lb[OWN_UNR], lmin = INFINITY, smin = INFINITY;
        uint32_t xmin = 0u;
#pragma unroll
        for (int k = 0; k < OWN_UNR; ++k) {
            const float u = (float)(x[k] >> 8) * 5.9604644775390625e-08f;
            lb[k] = __fadd_rd(__fadd_rd(__logf(u), sc[k]), -slack);
            if (sc[k] == INFINITY) lb[k] = INFINITY;     // log 0 + inf is not a number
            if (lb[k] < lmin) { lmin = lb[k]; xmin = x[k]; smin = sc[k]; }
        }
        if (__any_sync(0xffffffffu, lmin <= T && lmin < INFINITY)) {
            // An upper bound of the exact key (own_key): u53 < u24 + 2^-24 and E1 = -log1p(-u) grows
            // with u, the two-channel term only lowers the key, s is below the next float up;
            // 1e-4 covers the float logarithms (absolute errors below 1e-5), the sums round up.
            const float uh = (float)(xmin >> 8) * 5.9604644775390625e-08f + 5.9604644775390625e-08f;
            const float le = __logf(-log1pf(-uh));
            const float sh = __fadd_ru(smin, __fmaf_ru(fabsf(smin), 2.4e-7f, 1e-30f));
            const float ub = lmin < INFINITY ? __fadd_ru(__fadd_ru(le, sh), 1e-4f) : INFINITY;
            T = fminf(T, warp_min_f32(ub));
        }
#pragma unroll
        for (int k = 0; k < OWN_UNR; ++k) {
            const bool adm = lb[k] <= T && lb[k] < INFINITY;
            const unsigned m = __ballot_sync(0xffffffffu, adm);
            if (!m) continue;
            const int pos = qn + __popc(m & below);
            if (adm) { q[pos] = ci[k]; ql[pos] = lb[k]; }
            qn += __popc(m);
            if (qn > NEEL_QCAP - 32) {       // full: drop what T rules out by now, else evaluate
                __syncwarp();
                int n = 0;
                for (int b = 0; b < qn; b += 32) {
                    const bool v = b + lane < qn;
                    const int i = v ? q[b + lane] : 0;
                    const float l = v ? ql[b + lane] : INFINITY;
                    const unsigned keep = __ballot_sync(0xffffffffu, v && l <= T);
                    __syncwarp();
                    if (v && l <= T) { q[n + __popc(keep & below)] = i; ql[n + __popc(keep & below)] = l; }
                    n += __popc(keep);
                    __syncwarp();
                }
                qn = n;
                if (qn > NEEL_QCAP - 32) {
                    for (int b = 0; b < qn; b += 32)
                        if (b + lane < qn) best = hs_kmin(best, own_key(O, q[b + lane], call_lo, call_hi, RK));
                    T = fminf(T, warp_min_f32(best.idx >= 0 ? __double2float_ru(best.key) : INFINITY));
                    qn = 0;
                    __syncwarp();
                }
            }
        }
#pragma unroll
        for (int k = 0; k < OWN_UNR; ++k) { ci[k] = cn[k]; sc[k] = sn[k]; }
    }
    __syncwarp();
    return T;
}

HS_DEV float own_scan(const NeelOwn &O, uint64_t call, const HsRoundKeys &RK, int *q, float *ql, int &qn,
                      HsKeyIdx &best) {
    // a warp with a single chunk does not pay for empty ones
    return O.w + O.W >= O.nch ? own_scan_u<1>(O, call, RK, q, ql, qn, best) : own_scan_u<3>(O, call, RK, q, ql, qn, best);
}

// A switch: its cell, new spin and new moment, its kernels at offset 0.
struct OwnSwitch { int i0, sy, sx, sm; float smm; const float *K0, *Kp0; };

// Chunks c, c + W, ... < c1 of a window update, slots [j0, j1), U chunks in flight. The arithmetic
// per cell is that of update_one.
template <int U>
HS_DEV void own_update_chunks(const NeelOwn &O, const OwnSwitch &w, int c, int c1, int j0, int j1) {
    const int lane = threadIdx.x & 31;
    const int nx = O.nx, ny = O.ny, wy = O.wy, wx = O.wx, KW = 2 * wx + 1;
    const bool wrap = O.dip_wrap != 0;
    for (; c < c1; c += U * O.W) {
        int ci[U], j[U], ko[U];
        bool in[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            j[k] = 32 * (c + k * O.W) + lane;
            in[k] = j[k] >= j0 && j[k] < j1;
            ci[k] = in[k] ? own_cell(O, j[k]) : 0;
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            int row = ci[k] < (1 << 24) ? (int)((float)ci[k] * O.inv_nx) : ci[k] / nx;
            int col = ci[k] - row * nx;
            if (col < 0) { --row; col += nx; }
            else if (col >= nx) { ++row; col -= nx; }
            int dy = row - w.sy, dx = col - w.sx;
            if (wrap) {
                dy = dy < 0 ? dy + ny : dy; dy = 2 * dy >= ny ? dy - ny : dy;
                dx = dx < 0 ? dx + nx : dx; dx = 2 * dx >= nx ? dx - nx : dx;
            }
            in[k] = in[k] && dy >= -wy && dy <= wy && dx >= -wx && dx <= wx;
            ko[k] = dy * KW + dx;
        }
        float kv[U], kp[U], mv[U];
        double ev[U], pv[U];
        int ms[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int i = ci[k];
            const bool src = i == w.i0;
            kv[k] = (in[k] && w.K0) ? __ldg(w.K0 + ko[k]) : 0.f;
            kp[k] = (in[k] && w.Kp0) ? __ldg(w.Kp0 + ko[k]) : 0.f;
            mv[k] = in[k] ? (src ? w.smm : O.mm[i]) : 0.f;
            ms[k] = in[k] ? (src ? w.sm : (int)O.m[i]) : 0;
            ev[k] = (in[k] && O.E) ? O.E[i] : 0.0;
            pv[k] = (in[k] && O.Ep) ? O.Ep[i] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            if (!in[k]) continue;
            const int i = ci[k];
            const float acc = w.smm * kv[k], accp = w.smm * kp[k];
            double e = ev[k] + (double)(O.pref2 * (mv[k] * acc));
            double p = pv[k] + (double)(O.pref2 * (mv[k] * accp));
            if (i == w.i0) {
                e = -e; p = -p;
                O.m[i] = (int8_t)w.sm;
                O.mm[i] = w.smm;
            }
            if (O.E) O.E[i] = e;
            if (O.Ep) O.Ep[i] = p;
            O.s[j[k]] = own_bound(O, own_static(O, i, true), e, O.use_perp ? p : 0.0, ms[k]);
        }
    }
}

// Window update of the switch of cell i0 (new moment smm, new spin sm) for the slots this warp owns, with
// their bounds.
HS_DEV void own_update(const HsLattice &L, const NeelOwn &O, const int *rowpre, int i0, float smm, int sm) {
    const int lane = threadIdx.x & 31;
    const int nx = O.nx, ny = O.ny, wy = O.wy, wx = O.wx;
    const int sy = i0 / nx, sx = i0 - sy * nx;
    const bool wrap = O.dip_wrap != 0;
    const int sub = O.E ? hs_sub(L, sy, sx) : -1;
    const int64_t k0 = ((int64_t)max(sub, 0) * (2 * wy + 1) + wy) * (2 * wx + 1) + wx;      // offset 0 of the kernel
    const OwnSwitch w{i0, sy, sx, sm, smm, sub >= 0 ? O.K + k0 : nullptr, (sub >= 0 && O.Ep) ? O.Kpo + k0 : nullptr};
    // rows [r0, r1) and, wrapped, [q0, q1)
    int r0 = max(0, sy - wy), r1 = min(ny, sy + wy + 1), q0 = 0, q1 = 0;
    if (wrap) {
        if (2 * wy + 1 >= ny) { r0 = 0; r1 = ny; }
        else if (sy - wy < 0) { q0 = sy - wy + ny; q1 = ny; }
        else if (sy + wy >= ny) { q0 = 0; q1 = sy + wy + 1 - ny; }
    }
    for (int part = 0; part < 2; ++part) {
        const int y0 = part ? q0 : r0, y1 = part ? q1 : r1;
        if (y0 >= y1) continue;
        const int j0 = y0 == 0 ? 0 : own_row(L, O, rowpre, y0), j1 = y1 == ny ? O.M : own_row(L, O, rowpre, y1);
        const int c0 = j0 >> 5, c1 = (j1 + 31) >> 5;
        // the warp's first chunk at or after c0
        int c = (int)((float)c0 * O.inv_W) * O.W + O.w;
        while (c < c0) c += O.W;
        while (c - O.W >= c0) c -= O.W;
        // a warp with a single chunk does not pay for an empty one
        if (c + O.W >= c1) { if (c < c1) own_update_chunks<1>(O, w, c, c1, j0, j1); }
        else own_update_chunks<2>(O, w, c, c1, j0, j1);
    }
}

// Can the instance's Néel steps run on owned cells?
HS_DEV bool neel_owned(const HsInstance &I) {
    return I.L.beta_uniform > 0.0 && !I.L.has_exchange &&
           I.scratch_bytes >= HS_NEEL_CACHE_OFFSET + 4 * (int64_t)I.L.nx * I.L.ny;
}

// All Néel steps of an instance on owned cells. `go_next(next)`, on rank 0's helper lane, is whether
// step `next` runs.
template <int CS, typename Go>
HS_DEV void neel_run_owned(EngShared &sh, const RunSync<CS> &S, int rank, int SCS, int64_t budget, Go go_next) {
    const HsInstance &I = sh.I;
    const HsLattice &L = sh.I.L;
    HsCounters *const C = &sh.C;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const bool helper = rank == 0 && warp == nwarps - 1;
    NeelOwn O;
    O.W = SCS * nwarps - 1;
    O.w = rank * nwarps + warp - (rank ? 1 : 0);
    O.list = (int64_t)L.n_occ < (int64_t)L.nx * L.ny ? L.nonzero : nullptr;
    O.M = O.list ? L.n_occ : L.nx * L.ny;
    O.nch = (O.M + 31) >> 5;
    O.s = reinterpret_cast<float *>(reinterpret_cast<char *>(I.scratch) + HS_NEEL_CACHE_OFFSET);
    const bool dip = L.has_dipolar != 0, two = L.use_perp != 0;
    O.E = dip ? L.E_dip : nullptr;
    O.Ep = dip && two ? L.E_dip_perp : nullptr;
    O.m = L.m; O.mm = L.mm;
    O.zee = L.zee; O.zeep = L.zee_perp; O.EB = L.E_B; O.K = L.K; O.Kpo = L.Kpo;
    O.beta = L.beta_uniform; O.m_perp_factor = L.m_perp_factor;
    O.nx = L.nx; O.ny = L.ny;
    O.wy = dip ? L.dip_wy : 0; O.wx = dip ? L.dip_wx : 0; O.dip_wrap = dip ? L.dip_wrap : 0;
    O.use_perp = L.use_perp; O.barrier_method = L.barrier_method;
    O.pref2 = (float)(2.0 * L.dip_pref);
    O.inv_W = 1.0f / (float)O.W;
    O.inv_nx = 1.0f / (float)O.nx;
    // occupied cells of a period of uy rows (the first ones of the list)
    const bool table = O.list && L.uy <= NEEL_OWN_UY;
    if (table)
        for (int k = threadIdx.x; k <= L.uy; k += blockDim.x) sh.rowpre[k] = 0;
    __syncthreads();
    if (table)
        for (int k = threadIdx.x; k < min(O.M, L.uy * L.nx); k += blockDim.x) {
            const int y = __ldg(L.nonzero + k) / L.nx;
            if (y < L.uy) atomicAdd(&sh.rowpre[y + 1], 1);
        }
    __syncthreads();
    if (table && threadIdx.x == 0)
        for (int k = 0; k < L.uy; ++k) sh.rowpre[k + 1] += sh.rowpre[k];
    if (!helper)
        for (int c = O.w; c < O.nch; c += O.W) {
            const int j = 32 * c + lane;
            if (j >= O.M) break;
            const int i = own_cell(O, j);
            O.s[j] = own_bound(O, own_static(O, i, true), O.E ? __ldcg(O.E + i) : 0.0, O.Ep ? __ldcg(O.Ep + i) : 0.0, (int)__ldcg(O.m + i));
        }
    // helper: whether step `next` runs, and below which key its switch happens for certain
    const double af = two ? I.attempt_freq / 2.0 : I.attempt_freq;
    auto publish_next = [&](int64_t next) {
        int go = 0;
        double thr = -INFINITY;
        if (lane == 0) {
            go = go_next(next);
            const double left = C->progress ? (C->t_max - (C->t - C->t0)) : C->t_max;
            if (af > 0.0 && af < INFINITY && left > 0.0) {
                const double l = log(left) + log(af);
                thr = left == INFINITY ? INFINITY : l - 1e-3 - 1e-6 * fabs(l);
            }
        }
        go = __shfl_sync(0xffffffffu, go, 0);
        thr = __shfl_sync(0xffffffffu, thr, 0);
        S.publish_warp(&sh.go[next & 1], go, SCS);
        S.publish_warp(&sh.thr[next & 1], thr, SCS);
    };
    if (helper) {
        publish_next(0);
        S.publish_warp(&sh.call[0], (unsigned long long)C->rng_call, SCS);
        S.publish_warp(&sh.nsw, C->progress, SCS);
    }
    S.all();
    const uint64_t call0 = sh.call[0];
    const bool fixed = sh.nsw == 0;          // run(steps): no stop rule but the budget
    const HsRoundKeys RK = hs_round_keys(L.seed);
    for (int64_t st = 0;; ++st) {
        if (fixed && st >= budget) break;
        const uint64_t call = call0 + (uint64_t)st;
        const uint32_t call_lo = (uint32_t)call, call_hi = (uint32_t)(call >> 32);
        HsKeyIdx best{0.0, -1};
        int qn = 0;
        float T = INFINITY;
        if (!helper) T = own_scan(O, call, RK, sh.nq.q[warp], sh.nq.lb[warp], qn, best);
        if (lane == 0) sh.tw[warp] = T;
        __syncthreads();
        T = warp_min_f32(lane < nwarps ? sh.tw[lane] : INFINITY);
        for (int b = 0; b < qn; b += 32) {
            const bool v = b + lane < qn && sh.nq.lb[warp][b + lane] <= T;
            if (__any_sync(0xffffffffu, v) && v) best = hs_kmin(best, own_key(O, sh.nq.q[warp][b + lane], call_lo, call_hi, RK));
        }
        {
            const int wl = __any_sync(0xffffffffu, best.idx >= 0) ? warp_kmin_lane(best.key, best.idx) : -1;
            if (lane == max(wl, 0)) sh.red[warp] = best;      // idx < 0 when there is none
        }
        __syncthreads();
        const HsKeyIdx *rec = sh.red;
        int nrec = nwarps;
        if (CS > 1 && SCS > 1) {
            if (warp == 0) {
                const HsKeyIdx r = lane < nwarps ? sh.red[lane] : HsKeyIdx{0.0, -1};
                const int wl = max(warp_kmin_lane(r.key, r.idx), 0);
                S.copy_to_all(&sh.part[st & 1][rank], &sh.red[wl], SCS);
            }
            S.all();
            rec = sh.part[st & 1];
            nrec = SCS;
        }
        if (!sh.go[st & 1]) break;
        const double key = lane < nrec ? rec[lane].key : 0.0;
        const int wl = warp_kmin_lane(key, lane < nrec ? rec[lane].idx : -1);
        const HsKeyIdx w = wl >= 0 ? rec[wl] : HsKeyIdx{0.0, -1};
        const bool certain = wl >= 0 && isfinite(w.key) && w.key < sh.thr[st & 1];
        bool flip = certain;
        NeelFlip f{};
        if (helper && lane == 0) neel_finalize(L, C, sh.I.sw, w, call, 0.0, true, two, I.attempt_freq, &f);
        if (!certain) {          // uniform over the instance's threads
            if (helper) S.publish_warp(&sh.n1, (int)__shfl_sync(0xffffffffu, (int)f.flip, 0), SCS);
            S.all();
            flip = sh.n1 != 0;
        }
        if (helper) {
            if (lane == 0 && f.flip) {
                sh.I.sw.y[0] = f.y;
                sh.I.sw.x[0] = f.x;
                if (sh.I.sw.mode) sh.I.sw.mode[0] = 0;
            }
            publish_next(st + 1);
        } else if (flip) own_update(L, O, sh.rowpre, w.idx, -w.mm, -w.m);
    }
}

// Run instance ii to the end of its step budget (or its stop rule) on the whole cluster
// (`rank` = this CTA's rank) or, in CTA mode, on this CTA alone (rank 0).
template <int CS>
HS_DEV void run_instance(EngShared &sh, const HsInstance *insts, int ii, int rank, bool alone, unsigned char *s_ws,
                         int ws_bytes, long long *elapsed_ns) {
    const RunSync<CS> S{alone};
    const int SCS = (CS == 1 || alone) ? 1 : CS;   // CTAs running the instance
    const int warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    const unsigned long long t_claim = hs_globaltimer_ns();   // used by rank 0, thread 0
    {   // stage the instance descriptor in shared memory
        const unsigned long long *src = reinterpret_cast<const unsigned long long *>(insts + ii);
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(&sh.I);
        for (int k = threadIdx.x; k < (int)(sizeof(HsInstance) / 8); k += blockDim.x) dst[k] = __ldg(src + k);
        __syncthreads();
    }
    const HsInstance &I = sh.I;
    const HsLattice &L = sh.I.L;
    const HsSwitchList &sw = sh.I.sw;
    const HsGridPlan &P = sh.I.P;
    // The counters live in rank 0's shared memory while the instance runs (every step reads
    // and updates them) and go back to global memory when it stops; other CTAs receive the
    // values they need (Philox call, switch count) through distributed shared memory.
    HsCounters *const Cg = sh.I.C;
    HsCounters *const C = &sh.C;
    if (rank == 0) {
        const unsigned long long *src = reinterpret_cast<const unsigned long long *>(Cg);
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(&sh.C);
        for (int k = threadIdx.x; k < (int)(sizeof(HsCounters) / 8); k += blockDim.x) dst[k] = __ldcg(src + k);
    }
    __syncthreads();
    const int scheme = sh.I.scheme;
    // progress() runs: at most `budget` steps in this launch; an unfinished run keeps done = 0
    // and the next launch continues it, so every launch ends
    const int64_t budget = I.steps > 0 ? I.steps : (int64_t)HS_PROGRESS_STEPS_MAX;
    // Whether step st runs, and its Philox call, are decided by rank 0's thread 0 as soon as
    // the counters of step st - 1 are final (right after its decision phase) and published
    // to every CTA in slot st & 1; the barriers that end step st - 1 make them visible, so a
    // step needs no barrier of its own for this. Slot st & 1 was last read at the start of
    // step st - 2, before that step's barriers, so the write cannot overtake a read.
    auto go_next = [&](int64_t next) {
        int go;
        if (C->done) go = 0;
        else if (C->progress) {
            if (C->status || next >= budget) go = 0;   // a failed step, or the budget: not done
            else { go = hs_progress_continue(C, L.n_occ); if (!go) { C->done = 1; C->n_sw = 0; } }
        }
        else go = next < I.steps;
        return go;
    };
    auto decide_next = [&](int64_t next) {
        S.publish(&sh.go[next & 1], go_next(next));
        S.publish(&sh.call[next & 1], (unsigned long long)C->rng_call);
    };
    const bool owned = scheme == HS_SCHEME_NEEL && neel_owned(I);
    if (owned) neel_run_owned(sh, S, rank, SCS, I.steps, go_next);
    else {
        if (rank == 0 && threadIdx.x == 0) decide_next(0);
        S.all();
    }
    for (int64_t st = 0; !owned; ++st) {
        if (!sh.go[st & 1]) break;
        if (scheme == HS_SCHEME_METROPOLIS) {
            if (rank == 0) {
                metro_step_cta<true>(L, C, sw, P, metro_scratch_of(L, P, I.scratch), ws_bytes > 0 ? s_ws : nullptr,
                               ws_bytes);
                __syncthreads();
                if (threadIdx.x == 0) { S.publish(&sh.nsw, C->n_sw); decide_next(st + 1); }
            }
            S.all();
            if (L.has_dipolar) {
                const int nsw = sh.nsw;
                // Short lists go by their windows, whatever their size. Us per step on 1 / 16 CTAs, beside
                // the longer lists' code: 512 x 512, cutoff 20a, 5 switches 13.7 / 8.2 (32.5 / 10.7);
                // 256 x 256 uncut, 21 switches 103 / 18.6 (299 / 51.8); 1024 x 1024 uncut, 22 switches
                // 1472 / 123 (2050 / 174).
                if (nsw > 0 && nsw <= FEW_MAX) {       // uniform over the instance's threads
                    FewSw w{};
                    if ((int)threadIdx.x < nsw) {
                        w.y = __ldcg(sw.y + threadIdx.x);
                        w.x = __ldcg(sw.x + threadIdx.x);
                        w.mode = sw.mode ? __ldcg(sw.mode + threadIdx.x) : 0;
                    }
                    const int items = few_stage<ENG_FEW_R>(L, w, nsw, HS_UPDATE_MULTIPLE, sh.few, sh.few_w);
                    few_items<ENG_FEW_R>(L, sh.few, nsw, items, HS_UPDATE_MULTIPLE, rank * nwarps + warp, SCS * nwarps);
                } else if (nsw > 0) {
                    const int n = stage_switches(L, sw, nsw, sh.sw);
                    update_items(L, sh.sw, n, HS_UPDATE_MULTIPLE, rank * nwarps + warp, SCS * nwarps, sw, nsw);
                }
            }
            S.all();
        } else if (scheme == HS_SCHEME_NEEL) {
            const uint64_t call = sh.call[st & 1];
            const int64_t N = (int64_t)L.nx * L.ny;
            const int64_t gt = (int64_t)rank * blockDim.x + threadIdx.x, gs = (int64_t)SCS * blockDim.x;
            const bool unif = L.beta_uniform > 0.0;
            double bmin = 0.0;
            if (!unif) {  // b_min pass (hotspice/core.py:688, 696)
                double v = INFINITY;
                for (int64_t i = gt; i < N; i += gs) {
                    if (!L.occ[i]) continue;
                    double b1, b2;
                    hs_barriers(L, (int)(i / L.nx), (int)(i % L.nx), b1, b2);
                    v = fmin(v, fmin(b1, b2));
                }
                v = eng_block_dmin(v, sh.dred);
                if (threadIdx.x == 0) S.to_rank0(sh.part[0], rank, HsKeyIdx{v, rank});
                S.all();
                if (rank == 0 && threadIdx.x == 0) {
                    double b = INFINITY;
                    for (int r = 0; r < SCS; ++r) b = fmin(b, sh.part[0][r].key);
                    C->bmin = b;
                    S.publish(&sh.dred[0], b);
                }
                S.all();
                bmin = sh.dred[0];
                S.all();
            }
            const bool two = L.use_perp != 0;
            HsKeyIdx best = neel_scan_range(L, gt, gs, N, call, bmin, HsKeyIdx{0.0, -1});
            best = eng_block_kmin(best, sh.red);
            if (threadIdx.x == 0) S.to_rank0(sh.part[0], rank, best);
            S.all();
            NeelFlip flip{};   // thread 0 of rank 0: the step's flip, written after the handover
            if (rank == 0 && threadIdx.x == 0) {
                HsKeyIdx w{0.0, -1};
                for (int r = 0; r < SCS; ++r) w = hs_kmin(w, sh.part[0][r]);
                neel_finalize(L, C, sw, w, call, bmin, unif, two, I.attempt_freq, &flip);
                const int n1 = C->n_sw;
                // hand the switch to every CTA through shared memory (no global round trip)
                S.publish(&sh.n1, n1);
                if (n1 > 0) {
                    S.publish(&sh.y1, flip.y);
                    S.publish(&sh.x1, flip.x);
                    S.publish(&sh.mm1, flip.mm_new);
                }
                decide_next(st + 1);
            }
            // The flip's global writes (spin, moment, switch list) are issued after this
            // thread's arrival at the barrier, so the barrier does not wait for them: the
            // window update takes the switched cell's new moment from the handover, and the
            // writes are ordered before the next step by the barrier that ends this one.
            S.all_then(rank == 0 && threadIdx.x == 0 && flip.flip, [&] { neel_apply(L, sw, flip); });
            if (L.has_dipolar && sh.n1 > 0)
                update_one(L, sh.y1, sh.x1, sh.mm1, rank * blockDim.x + threadIdx.x, SCS * blockDim.x);
            S.all();
        } else {  // Wolff
            if (rank == 0) {
                wolff_step_cta(L, C, sw, wolff_scratch_of(L, I.scratch), sh.wolff);
                __syncthreads();
                if (threadIdx.x == 0) decide_next(st + 1);
            }
            S.all();
        }
    }
    S.all();
    if (rank == 0) {  // counters back to global memory
        const unsigned long long *src = reinterpret_cast<const unsigned long long *>(&sh.C);
        unsigned long long *dst = reinterpret_cast<unsigned long long *>(Cg);
        for (int k = threadIdx.x; k < (int)(sizeof(HsCounters) / 8); k += blockDim.x) dst[k] = src[k];
        // the device time spent on this instance in this launch
        if (elapsed_ns && threadIdx.x == 0) elapsed_ns[ii] = (long long)(hs_globaltimer_ns() - t_claim);
    }
    __syncthreads();
}

// Clusters claim instances from the work counter (rank 0 claims for the cluster). An instance
// flagged HS_INST_ONE_CTA switches the cluster to CTA mode for the rest of the launch: rank 0
// runs that instance alone, every other CTA claims one of its own, and from then on each CTA
// claims and runs instances by itself, with block barriers only. The switch is decided on the
// same flag by every CTA of the cluster, right after the barrier that follows the claim, and
// no cluster barrier or distributed shared memory access follows it, so a CTA may leave the
// launch while the others of its cluster still run. The host lists the flagged instances
// after all others (a flagged instance is never followed by one that needs the cluster; one
// that is still runs correctly, on one CTA).
template <int CS>
__global__ void __launch_bounds__(ENG_NT, ENG_MIN_CTAS) engine_kernel(const HsInstance *insts, int n_inst, int *work,
                                                                      int ws_bytes, long long *elapsed_ns) {
    // dynamic shared workspace (the Poisson-disc sampler's arrays), given only to launches that
    // hold Poisson-disc instances: it takes L1 capacity from the other phases
    extern __shared__ __align__(16) unsigned char s_ws[];
    __shared__ EngShared sh;
    const int rank = Sync<CS>::rank();
    bool alone = false;
    for (;;) {
        int ii;
        if (!alone) {
            if (rank == 0 && threadIdx.x == 0) Sync<CS>::publish(&sh.inst, atomicAdd(work, 1));
            Sync<CS>::all();
            ii = sh.inst;
            if (ii >= n_inst) break;
            if constexpr (CS > 1) {
                if (__ldg(&insts[ii].flags) & HS_INST_ONE_CTA) {
                    alone = true;
                    if (rank != 0) {
                        __syncthreads();   // every thread has read the cluster's claim
                        if (threadIdx.x == 0) sh.inst = atomicAdd(work, 1);
                        __syncthreads();
                        ii = sh.inst;
                        if (ii >= n_inst) break;
                    }
                }
            }
        } else {
            if (threadIdx.x == 0) sh.inst = atomicAdd(work, 1);
            __syncthreads();
            ii = sh.inst;
            if (ii >= n_inst) break;
        }
        run_instance<CS>(sh, insts, ii, alone ? 0 : rank, alone, s_ws, ws_bytes, elapsed_ns);
    }
}

// Run controls of every instance of a launch: one kernel in place of a small copy per field and
// instance (256 instances: 4.6 ms of host time per run_from_host()).
__global__ void engine_controls_kernel(const HsInstance *insts, int n, double t_max) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    HsCounters *C = insts[i].C;
    C->progress = 0;
    C->done = 0;
    C->t_max = t_max;
}

template <int CS>
cudaError_t engine_allow_ws(int bytes) {
    // opt in to the dynamic workspace: static (about 30 KB) plus dynamic shared memory above
    // 48 KB needs it; the largest size granted so far covers every smaller one
    static int granted = 0;
    if (bytes <= granted) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(engine_kernel<CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) granted = bytes;
    return e;
}

template <int CS>
int launch_engine(const HsInstance *insts, int n_inst, int *work, int n_clusters, int ws_bytes, long long *elapsed_ns,
                  cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_clusters * CS, 1, 1);
    cfg.blockDim = dim3(ENG_NT, 1, 1);
    cfg.dynamicSmemBytes = (size_t)ws_bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (CS > 8) {
        cudaError_t e = cudaFuncSetAttribute(engine_kernel<CS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) { hs_set_error("engine: cluster size %d not allowed: %s", CS, cudaGetErrorString(e)); return HS_ECUDA; }
    }
    {
        cudaError_t e = engine_allow_ws<CS>(ws_bytes);
        if (e != cudaSuccess) { hs_set_error("engine: shared workspace: %s", cudaGetErrorString(e)); return HS_ECUDA; }
    }
    cudaError_t e = cudaLaunchKernelEx(&cfg, engine_kernel<CS>, insts, n_inst, work, ws_bytes, elapsed_ns);
    if (e != cudaSuccess) { hs_set_error("engine launch (cluster %d x %d): %s", CS, n_clusters, cudaGetErrorString(e)); return HS_ECUDA; }
    return hs_check_launch("engine_kernel");
}

}  // namespace

int hs_launch_engine(const HsInstance *insts, int n_inst, int cluster_size, int n_clusters, int *work, int ws_bytes,
                     long long *elapsed_ns, cudaStream_t st) {
    if (ws_bytes < 0 || ws_bytes > ENG_WS_MAX) {
        hs_set_error("engine: shared workspace of %d bytes outside [0, %d]", ws_bytes, ENG_WS_MAX);
        return HS_EINVAL;
    }
    cudaError_t e = cudaMemsetAsync(work, 0, sizeof(int), st);
    if (e != cudaSuccess) { hs_set_error("engine: work counter reset: %s", cudaGetErrorString(e)); return HS_ECUDA; }
    switch (cluster_size) {
        case 1: return launch_engine<1>(insts, n_inst, work, n_clusters, ws_bytes, elapsed_ns, st);
        case 2: return launch_engine<2>(insts, n_inst, work, n_clusters, ws_bytes, elapsed_ns, st);
        case 4: return launch_engine<4>(insts, n_inst, work, n_clusters, ws_bytes, elapsed_ns, st);
        case 8: return launch_engine<8>(insts, n_inst, work, n_clusters, ws_bytes, elapsed_ns, st);
        case 16: return launch_engine<16>(insts, n_inst, work, n_clusters, ws_bytes, elapsed_ns, st);
        default: hs_set_error("engine: cluster size must be 1, 2, 4, 8 or 16"); return HS_EINVAL;
    }
}

int hs_engine_controls_impl(const HsInstance *insts, int n_inst, double t_max, cudaStream_t st) {
    engine_controls_kernel<<<(n_inst + 127) / 128, 128, 0, st>>>(insts, n_inst, t_max);
    return hs_check_launch("engine_controls_kernel");
}

int hs_engine_max_clusters_impl(int cluster_size) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster_size, 1, 1);
    cfg.blockDim = dim3(ENG_NT, 1, 1);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster_size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    cudaError_t e;
    switch (cluster_size) {
        case 1: e = cudaOccupancyMaxActiveClusters(&n, engine_kernel<1>, &cfg); break;
        case 2: e = cudaOccupancyMaxActiveClusters(&n, engine_kernel<2>, &cfg); break;
        case 4: e = cudaOccupancyMaxActiveClusters(&n, engine_kernel<4>, &cfg); break;
        case 8: e = cudaOccupancyMaxActiveClusters(&n, engine_kernel<8>, &cfg); break;
        case 16:
            cudaFuncSetAttribute(engine_kernel<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            e = cudaOccupancyMaxActiveClusters(&n, engine_kernel<16>, &cfg); break;
        default: hs_set_error("engine: bad cluster size"); return HS_EINVAL;
    }
    if (e != cudaSuccess) { hs_set_error("cudaOccupancyMaxActiveClusters: %s", cudaGetErrorString(e)); return HS_ECUDA; }
    return n;
}
