// Step bodies shared by the standalone step kernels and the persistent cluster engine.
#pragma once

#include "hs_common.cuh"

// ---- dipolar window helpers ----------------------------------------------------------


struct SwInfo { int y, x, mode, sub; float mm; };

// Does the window of switch (ys, mode) reach rows [t0, t0 + tn) (1-D test, axis length n)?
HS_DEV bool hs_axis_overlap(int s, int half, int wrap, int n, int t0, int tn) {
    if (wrap) {
        if (2 * half + 1 >= n) return true;
        const int ws = s - half;
        return hs_wrap(t0 - ws, n) <= 2 * half || hs_wrap(ws - t0, n) < tn;
    }
    return !(s + half < t0 || s - half >= t0 + tn);
}

// Window half-width and wrap flag of a switch along one axis.
HS_DEV void hs_window(const HsLattice &L, int mode, bool yaxis, int &half, int &wrap) {
    const int n = yaxis ? L.ny : L.nx;
    if (mode) {
        half = L.trunc_size ? min(L.trunc_size, n - 1) : n - 1;
        wrap = L.pbc;
    } else {
        half = yaxis ? L.dip_wy : L.dip_wx;
        wrap = L.dip_wrap;
    }
}

// Sum of kernel values that switch `w` contributes to target (y, x).
HS_DEV void hs_contrib(const HsLattice &L, const SwInfo &w, int y, int x, float &acc, float &accp) {
    if (!w.mode) {
        const int dy = y - w.y, dx = x - w.x;
        acc += w.mm * hs_kval(L, L.K, w.sub, dy, dx);
        if (L.use_perp) accp += w.mm * hs_kval(L, L.Kpo, w.sub, dy, dx);
        return;
    }
    const int ky = L.trunc_size ? min(L.trunc_size, L.ny - 1) : L.ny - 1;
    const int kx = L.trunc_size ? min(L.trunc_size, L.nx - 1) : L.nx - 1;
    int dys[2], dxs[2], ny_ = 0, nx_ = 0;
    if (L.pbc) {
        const int d0y = hs_wrap(y - w.y, L.ny), d0x = hs_wrap(x - w.x, L.nx);
        if (d0y <= ky) dys[ny_++] = d0y;
        if (d0y - L.ny >= -ky) dys[ny_++] = d0y - L.ny;
        if (d0x <= kx) dxs[nx_++] = d0x;
        if (d0x - L.nx >= -kx) dxs[nx_++] = d0x - L.nx;
    } else {
        const int dy = y - w.y, dx = x - w.x;
        if (dy >= -ky && dy <= ky) dys[ny_++] = dy;
        if (dx >= -kx && dx <= kx) dxs[nx_++] = dx;
    }
    for (int a = 0; a < ny_; ++a)
        for (int b = 0; b < nx_; ++b) {
            acc += w.mm * hs_kval(L, L.K, w.sub, dys[a], dxs[b]);
            if (L.use_perp) accp += w.mm * hs_kval(L, L.Kpo, w.sub, dys[a], dxs[b]);
        }
}


// ---- dipolar update of a short switch list ------------------------------------------------
// Update of a short list (up to FEW_MAX switches): work follows the switches instead of the lattice.
// An item is 32 columns x R rows of one switch's window, one warp's work (a lane has a column, so a
// kernel row is read by consecutive lanes); the items of all switches are numbered through and
// dealt to the warps. A cell in several windows belongs to the first of them in list order; its
// item adds the later ones' contributions in order, so the sums are those of dip_update_kernel bit
// for bit. The common item meets no other window and reads nothing but its own cells and kernel rows.
// Measured on B200 (cutoff 20a, 79 x 79 windows): us per step of two kernels, 512 x 512
// 7.7 -> 6.7 and 1500 x 1201 with about 20 switches 18.6 -> 10.8; bound by the latencies of list,
// moments, cells and the two launches. Where the windows add up to more than the lattice
// (few_crowded), one inside an earlier one gets no items: with uncut windows a cell is visited once,
// not once per switch.
constexpr int FEW_MAX = 64, FEW_ITEMS = 128;

struct FewSw {
    int y, x, mode, sub;
    float mm;
    int hy, hx, kind;        // kind 0: plain window, 1: minimum image, 2: truncated and periodic (hs_contrib)
    int ylo, nr, xlo, nc;    // window rows and columns (ylo, xlo may be negative where they wrap)
    int end;                 // items of the switches up to this one
};

// hs_minimage of the difference of two coordinates, without the remainder.
HS_DEV int few_minimage(int d, int n) {
    d = d < 0 ? d + n : d;
    return 2 * d >= n ? d - n : d;
}

HS_DEV bool few_covers(const HsLattice &L, const FewSw &w, int y, int x) {
    int dy = y - w.y, dx = x - w.x;
    if (w.kind) { dy = few_minimage(dy, L.ny); dx = few_minimage(dx, L.nx); }
    return abs(dy) <= w.hy && abs(dx) <= w.hx;
}

// Are all of coordinates t0 .. t0 + tn - 1 (not reduced to 0 .. n - 1 where windows wrap) within `half` of s?
HS_DEV bool few_axis_inside(int s, int half, bool wrap, int n, int t0, int tn) {
    if (!wrap) return t0 >= s - half && t0 + tn - 1 <= s + half;
    return 2 * half + 1 >= n || hs_wrap(t0 - (s - half), n) + tn <= 2 * half + 1;
}

// Does the window of w, which comes earlier in the list, hold all of the rectangle (`wraps`: it may
// reach beyond the lattice)? Its cells are w's then, or an even earlier window's.
HS_DEV bool few_holds(const HsLattice &L, const FewSw &w, int semantics, bool wraps, int y0, int nr, int x0, int nc) {
    if ((w.sub < 0 && semantics != HS_UPDATE_MULTIPLE) || (wraps && w.kind == 0)) return false;
    return few_axis_inside(w.y, w.hy, w.kind != 0, L.ny, y0, nr) && few_axis_inside(w.x, w.hx, w.kind != 0, L.nx, x0, nc);
}

// Do the windows add up to more than the lattice, so that many of them lie in earlier ones?
template <int R>
HS_DEV bool few_crowded(const HsLattice &L, int nsw, int n_items) {
    return nsw > 1 && (int64_t)n_items * (32 * R) > (int64_t)L.nx * L.ny;
}

// Stage switch k (w.y, w.x, w.mode loaded by thread k < nsw) and number the items through; returns
// their total. The whole block calls it.
template <int R>
HS_DEV int few_stage(const HsLattice &L, FewSw w, int nsw, int semantics, FewSw *s_sw, int *s_w) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = threadIdx.x;
    const int nx = L.nx, ny = L.ny;
    int items = 0;
    if (k < nsw) {
        w.sub = hs_sub(L, w.y, w.x);
        w.mm = __ldcg(L.mm + (int64_t)w.y * nx + w.x);
        int wy, wx;
        hs_window(L, w.mode, true, w.hy, wy);
        hs_window(L, w.mode, false, w.hx, wx);
        w.kind = wy ? (w.mode ? 2 : 1) : 0;
        if (w.sub < 0) { w.hy = w.hx = 0; w.kind = 0; }      // no kernel: only the sign flip of E applies
        if (w.kind == 0) {
            // a truncated plain window ends where the kernel does
            if (w.sub >= 0) { w.hy = min(w.hy, L.dip_wy); w.hx = min(w.hx, L.dip_wx); }
            w.ylo = max(0, w.y - w.hy); w.nr = min(ny - 1, w.y + w.hy) - w.ylo + 1;
            w.xlo = max(0, w.x - w.hx); w.nc = min(nx - 1, w.x + w.hx) - w.xlo + 1;
        } else {
            if (2 * w.hy + 1 >= ny) { w.ylo = 0; w.nr = ny; } else { w.ylo = w.y - w.hy; w.nr = 2 * w.hy + 1; }
            if (2 * w.hx + 1 >= nx) { w.xlo = 0; w.nc = nx; } else { w.xlo = w.x - w.hx; w.nc = 2 * w.hx + 1; }
        }
        if (w.sub >= 0 || semantics == HS_UPDATE_MULTIPLE)
            items = ((w.nr + R - 1) / R) * ((w.nc + 31) / 32);
    }
    auto number = [&]() {
        int incl = items, before = 0, total = 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += t; }
        if (lane == 31 && warp < FEW_MAX / 32) s_w[warp] = incl;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < FEW_MAX / 32; ++q) { if (q < warp) before += s_w[q]; total += s_w[q]; }
        if (k < nsw) { w.end = before + incl; s_sw[k] = w; }
        __syncthreads();
        return total;
    };
    int n_items = number();
    if (few_crowded<R>(L, nsw, n_items)) {       // uniform; windows inside an earlier one need no items
        if (k < nsw)
            for (int q = 0; q < k && items; ++q)
                if (few_holds(L, s_sw[q], semantics, w.kind != 0, w.ylo, w.nr, w.xlo, w.nc)) items = 0;
        __syncthreads();
        n_items = number();
    }
    return n_items;
}

// The items gw, gw + nw, ... of a staged list; a warp calls it. CROWDED: an item inside an earlier
// window leaves before it loads anything, and one whose cells all belong to earlier windows before it
// adds the later ones. Without overlaps these tests cost 5%, so they are compiled apart.
template <int R, bool CROWDED>
HS_DEV void few_items_of(const HsLattice &L, const FewSw *s_sw, int nsw, int n_items, int semantics, int gw, int nw) {
    const int lane = threadIdx.x & 31, nx = L.nx, ny = L.ny;
    const bool two = L.use_perp != 0, flip_perp = !(L.dip_keep_perp_sign && nsw > 1);
    const float pref2 = (float)(2.0 * L.dip_pref);
    const int KW = 2 * L.dip_wx + 1, KH = 2 * L.dip_wy + 1;
    const float *const Kg = L.K, *const Kpg = L.Kpo, *const mmg = L.mm;
    double *const Eg = L.E_dip, *const Epg = L.E_dip_perp;
    for (int item = gw; item < n_items; item += nw) {
        int k = 0;                         // the switch: how many end at or before the item
        for (int b = 0; b < nsw; b += 32)
            k += __popc(__ballot_sync(0xffffffffu, b + lane < nsw && s_sw[b + lane].end <= item));
        const FewSw own = s_sw[k];
        const int tc_n = (own.nc + 31) / 32, tile = item - (k ? s_sw[k - 1].end : 0);
        const int tr = tile / tc_n, tc = tile - tr * tc_n;
        const int y0 = own.ylo + R * tr, x0 = own.xlo + 32 * tc, nr = min(R, own.nr - R * tr);
        const int ncol = min(32, own.nc - 32 * tc);
        const bool wraps = y0 < 0 || y0 + nr > ny || x0 < 0 || x0 + ncol > nx;
        if constexpr (CROWDED) {           // leave before any load when an earlier window holds the item
            bool held = false;
            for (int b = lane; b < k; b += 32) held |= few_holds(L, s_sw[b], semantics, wraps, y0, nr, x0, ncol);
            if (__any_sync(0xffffffffu, held)) continue;
        }
        int x = x0 + lane;
        const bool inx = lane < ncol;
        x = x < 0 ? x + nx : (x >= nx ? x - nx : x);
        // the cells' energies and moments first: their loads complete while the sums are formed
        float mv[R];
        double ev[R], pv[R];
        int row[R];
#pragma unroll
        for (int v = 0; v < R; ++v) {
            int y = y0 + v;
            y = y < 0 ? y + ny : (y >= ny ? y - ny : y);
            row[v] = y;
            const bool in = inx && v < nr;
            const int64_t i = (int64_t)y * nx + x;
            mv[v] = in ? __ldcg(mmg + i) : 0.f;
            ev[v] = in ? __ldcg(Eg + i) : 0.0;
            pv[v] = in && two ? __ldcg(Epg + i) : 0.0;
        }
        float acc[R] = {}, accp[R] = {};
        unsigned mine = inx ? (1u << nr) - 1u : 0u, neg = 0u;
        auto apply = [&](const FewSw &w, bool item_own) {
            int dx = x - w.x;
            const bool own_col = dx == 0;
            if (w.kind == 0 && item_own) {   // the item's own plain window: every cell lies in it
                const float *K = Kg + ((int64_t)max(w.sub, 0) * KH + (row[0] - w.y + L.dip_wy)) * KW + (dx + L.dip_wx);
                const float *Kp = two ? Kpg + (K - Kg) : nullptr;
                float kv[R], kp[R];
#pragma unroll
                for (int v = 0; v < R; ++v) {
                    const bool in = inx && v < nr && w.sub >= 0;
                    kv[v] = in ? __ldg(K + v * KW) : 0.f;
                    kp[v] = in && two ? __ldg(Kp + v * KW) : 0.f;
                    if (own_col && row[v] == w.y) neg |= 1u << v;
                }
#pragma unroll
                for (int v = 0; v < R; ++v) { acc[v] += w.mm * kv[v]; accp[v] += w.mm * kp[v]; }
                return;
            }
            if (w.kind == 2) {
#pragma unroll
                for (int v = 0; v < R; ++v) {
                    if (!inx || v >= nr || !(item_own || few_covers(L, w, row[v], x))) continue;
                    if (own_col && row[v] == w.y) neg |= 1u << v;
                    if (w.sub >= 0) hs_contrib(L, SwInfo{w.y, w.x, w.mode, w.sub, w.mm}, row[v], x, acc[v], accp[v]);
                }
                return;
            }
            // no branch per cell, so that the loads of all rows are in flight together
            if (w.kind) dx = few_minimage(dx, nx);
            const float *K = Kg + ((int64_t)max(w.sub, 0) * KH + L.dip_wy) * KW + (L.dip_wx + dx);
            const float *Kp = two ? Kpg + (K - Kg) : nullptr;
            float kv[R], kp[R];
            bool in[R];
            const bool in_col = inx && abs(dx) <= w.hx;
#pragma unroll
            for (int v = 0; v < R; ++v) {
                int dy = row[v] - w.y;
                if (w.kind) dy = few_minimage(dy, ny);
                in[v] = in_col && v < nr && abs(dy) <= w.hy;
                if (in[v] && own_col && row[v] == w.y) neg |= 1u << v;
                in[v] = in[v] && w.sub >= 0;
                kv[v] = in[v] ? __ldg(K + dy * KW) : 0.f;
                kp[v] = in[v] && two ? __ldg(Kp + dy * KW) : 0.f;
            }
#pragma unroll
            for (int v = 0; v < R; ++v) if (in[v]) { acc[v] += w.mm * kv[v]; accp[v] += w.mm * kp[v]; }
        };
        // windows that may meet the item, in list order
        bool live = true;                  // warp-uniform: some cell is not an earlier window's (CROWDED)
        for (int b = 0; b < nsw && live; b += 32) {
            bool meets = false;
            if (b + lane < nsw) {
                const FewSw &w = s_sw[b + lane];
                meets = b + lane == k || wraps ||
                        (hs_axis_overlap(w.y, w.hy, w.kind != 0, ny, y0, nr) && hs_axis_overlap(w.x, w.hx, w.kind != 0, nx, x0, ncol));
            }
            for (unsigned m = __ballot_sync(0xffffffffu, meets); m && live; m &= m - 1u) {
                const int q = b + __ffs(m) - 1;
                if (q == k) { apply(own, true); continue; }
                const FewSw w = s_sw[q];
                if (w.sub < 0 && semantics != HS_UPDATE_MULTIPLE) continue;
                if (q > k) { apply(w, false); continue; }
#pragma unroll
                for (int v = 0; v < R; ++v)
                    if (((mine >> v) & 1u) && few_covers(L, w, row[v], x)) mine &= ~(1u << v);   // an earlier window's cell
                if constexpr (CROWDED) live = __any_sync(0xffffffffu, mine != 0u);
            }
        }
#pragma unroll
        for (int v = 0; v < R; ++v) {
            if (!((mine >> v) & 1u)) continue;
            const bool ng = (neg >> v) & 1u;
            const double de = (double)(pref2 * (mv[v] * acc[v])), dp = (double)(pref2 * (mv[v] * accp[v]));
            double e = ev[v], p = pv[v];
            if (semantics == HS_UPDATE_MULTIPLE) {
                if (ng) { e = -e; if (flip_perp) p = -p; }
                e += de; p += dp;
            } else {
                e += de; p += dp;
                if (ng) { e = -e; p = -p; }
            }
            const int64_t i = (int64_t)row[v] * nx + x;
            Eg[i] = e;
            if (two) Epg[i] = p;
        }
    }
}

template <int R>
HS_DEV void few_items(const HsLattice &L, const FewSw *s_sw, int nsw, int n_items, int semantics, int gw, int nw) {
    if (few_crowded<R>(L, nsw, n_items)) few_items_of<R, true>(L, s_sw, nsw, n_items, semantics, gw, nw);
    else few_items_of<R, false>(L, s_sw, nsw, n_items, semantics, gw, nw);
}

// ---- Metropolis ------------------------------------------------------------------------

constexpr int MT = 1024;              // threads of the step CTA
constexpr int MAX_RETRY = 1 << 14;    // bound on select() retries before reporting

struct MetroScratch {
    int32_t *py, *px;                  // candidate positions (capacity cap)
    int32_t *grid;                     // Poisson background grid (gsz)
    double  *ptx, *pty;                // Poisson points (gsz)
    int32_t *queue;                    // Poisson active list (gsz)
    int32_t cap, gsz;
};

HS_DEV int block_excl_scan(int flag, int *warp_tot, int &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(0xffffffffu, flag);
    if (lane == 0) warp_tot[warp] = __popc(bal);
    __syncthreads();
    if (warp == 0) {
        int v = lane < (int)(blockDim.x >> 5) ? warp_tot[lane] : 0;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { int t = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += t; }
        if (lane < (int)(blockDim.x >> 5)) warp_tot[lane] = incl - v;
        if (lane == 31) warp_tot[32] = incl;
    }
    __syncthreads();
    const int pre = warp_tot[warp] + __popc(bal & ((1u << lane) - 1u));
    total = warp_tot[32];
    __syncthreads();
    return pre;
}

// Stable in-place compaction of (py, px)[0..n) keeping entries for which keep(y, x) holds.
template <typename F>
HS_DEV int block_compact(int32_t *py, int32_t *px, int n, F keep, int *warp_tot) {
    int out = 0;
    for (int base = 0; base < n; base += blockDim.x) {
        const int i = base + threadIdx.x;
        int y = 0, x = 0, f = 0;
        if (i < n) { y = py[i]; x = px[i]; f = keep(y, x) ? 1 : 0; }
        int tot;
        const int pre = block_excl_scan(f, warp_tot, tot);
        if (f) { py[out + pre] = y; px[out + pre] = x; }
        out += tot;
        __syncthreads();
    }
    return out;
}

HS_DEV int pymod(int a, int n) { int r = a % n; return r < 0 ? r + n : r; }

// Work arrays of the Poisson-disc sampler: shared memory when they fit, else the step's scratch.
struct PoissonMem {
    int32_t *grid;     // background grid: point index per cell, or -1
    double *ptx, *pty; // points
    int32_t *queue;    // active list
};

// Bytes of the work arrays for a grid of gsz cells (one point per cell at most).
HS_HD inline int64_t hs_poisson_mem_bytes(int64_t gsz) { return 24 * gsz + 64; }

HS_DEV PoissonMem poisson_mem_in(void *base, int gsz) {
    char *p = reinterpret_cast<char *>(base);
    PoissonMem M;
    M.ptx = reinterpret_cast<double *>(p);
    M.pty = M.ptx + gsz;
    M.grid = reinterpret_cast<int32_t *>(M.pty + gsz);
    M.queue = M.grid + gsz;
    return M;
}

// Poisson-disc dart throwing in cell units (hotspice/poisson.py:72-128 restated in cells),
// executed by one warp, for any number of tries K; poisson_block is the form for the usual one.
// Returns the number of points, and advances `call` by the variates consumed.
// Bridson's loop is sequential over active points, but the k tries of one active point always
// consume 1 + 2k variates (queue pick, then angle and distance of each try), so the warp
// evaluates the k candidates at once (lane t: try t) and their 5x5-cell conflict checks against
// the existing points in parallel, then resolves them in try order: try t is accepted if it is
// in bounds, conflicts with no existing point, and with no earlier accepted try whose cell is
// among the 25 it checks. Two points in one cell always conflict (the cell diagonal is r), so an
// accepted try never hides an existing point from a later try: the accepted set is the one the
// sequential loop would build, in the same order, with the same variates.
HS_DEV int poisson_warp(const HsLattice &L, const HsGridPlan &P, const MetroScratch &S, const PoissonMem &M,
                        uint64_t &call, int *status) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const double width = L.nx, height = L.ny;
    const double r = P.r_cells + 1.0;
    const double cs = r / sqrt(2.0);
    const double rSq = r * r;
    const int gw = (int)ceil(width / cs), gh = (int)ceil(height / cs);
    const int gsz = gw * gh;
    const int K = P.poisson_k;
    for (int g = lane; g < gsz; g += 32) M.grid[g] = -1;
    __syncwarp();
    auto rnd_at = [&](uint64_t c) { return hs_u53(L.seed, c, 0u); };
    const double p0x = (double)(int)(width * rnd_at(call));
    const double p0y = (double)(int)(height * rnd_at(call + 1));
    call += 2;
    int npts = 1, nq = 1;
    if (lane == 0) { M.ptx[0] = p0x; M.pty[0] = p0y; M.queue[0] = 0; M.grid[(int)(p0x / cs) + (int)(p0y / cs) * gw] = 0; }
    __syncwarp();
    auto conflicts = [&](double px, double py, int g) {   // the distance rule of the grid check
        double dx = fabs(px - M.ptx[g]), dy = fabs(py - M.pty[g]);
        if (dx > width * 0.5) dx -= width;
        if (dy > height * 0.5) dy -= height;
        return (dx * dx + dy * dy) <= rSq;
    };
    bool overflow = false;
    while (nq > 0 && !overflow) {
        const int qi = (int)(rnd_at(call) * nq);
        const uint64_t cbase = call + 1;
        call += 1 + 2 * (uint64_t)K;
        const int q = M.queue[qi];
        // list.pop(qi): shift the tail left, preserving order
        for (int j = qi + lane; j < nq - 1; j += 32) {
            const int v = M.queue[j + 1];
            __syncwarp(__activemask());
            M.queue[j] = v;
        }
        __syncwarp();
        nq -= 1;
        const double qx = M.ptx[q], qy = M.pty[q];
        // candidates of the k tries, one per lane
        double px = 0.0, py = 0.0;
        int gx = 0, gy = 0, inb = 0;
        if (lane < K) {
            const double alpha = 6.283185307179586 * rnd_at(cbase + 2 * lane);
            const double d = r * sqrt(3.0 * rnd_at(cbase + 2 * lane + 1) + 1.0);
            px = qx + d * cos(alpha);
            py = qy + d * sin(alpha);
            inb = 0.0 <= px && px < width && 0.0 <= py && py < height;
            if (inb) { gx = (int)(px / cs); gy = (int)(py / cs); }
        }
        // conflicts with existing points: task id = 25 t + c (cell c of try t's 5x5 neighbourhood)
        unsigned cmask = 0u;
        for (int base = 0; base < 25 * K; base += 32) {
            const int id = base + lane;
            const int t = id < 25 * K ? id / 25 : 0, c = id - 25 * t;
            const double tx = __shfl_sync(0xffffffffu, px, t), ty = __shfl_sync(0xffffffffu, py, t);
            const int tgx = __shfl_sync(0xffffffffu, gx, t), tgy = __shfl_sync(0xffffffffu, gy, t);
            const int tin = __shfl_sync(0xffffffffu, inb, t);
            if (id < 25 * K && tin) {
                const int xx = tgx - 2 + c / 5, yy = tgy - 2 + c % 5;
                const int g = M.grid[pymod(xx + yy * gw, gsz)];
                if (g >= 0 && conflicts(tx, ty, g)) cmask |= 1u << t;
            }
        }
        cmask = __reduce_or_sync(0xffffffffu, cmask);
        // resolve in try order (every lane the same decisions)
        unsigned amask = 0u;
        int nacc = 0;
        for (int t = 0; t < K; ++t) {
            const double tx = __shfl_sync(0xffffffffu, px, t), ty = __shfl_sync(0xffffffffu, py, t);
            const int tgx = __shfl_sync(0xffffffffu, gx, t), tgy = __shfl_sync(0xffffffffu, gy, t);
            const int tin = __shfl_sync(0xffffffffu, inb, t);
            bool ok = tin && !((cmask >> t) & 1u);
            for (int u = 0; u < t; ++u) {
                const double ux = __shfl_sync(0xffffffffu, px, u), uy = __shfl_sync(0xffffffffu, py, u);
                const int ucell = __shfl_sync(0xffffffffu, gx, u) + __shfl_sync(0xffffffffu, gy, u) * gw;
                if (!ok || !((amask >> u) & 1u)) continue;
                // is u's cell among the 25 that try t checks (flat indices (xx + yy gw) mod gsz,
                // xx in [tgx-2, tgx+2])? per row yy: (ucell - yy gw - (tgx-2)) mod gsz <= 4
                bool seen = false;
                for (int b = 0; b < 5 && !seen; ++b) seen = pymod(ucell - (tgy - 2 + b) * gw - (tgx - 2), gsz) <= 4;
                if (seen) {
                    double dx = fabs(tx - ux), dy = fabs(ty - uy);
                    if (dx > width * 0.5) dx -= width;
                    if (dy > height * 0.5) dy -= height;
                    if ((dx * dx + dy * dy) <= rSq) ok = false;
                }
            }
            if (!ok) continue;
            if (npts + nacc >= S.gsz) { overflow = true; break; }
            amask |= 1u << t;
            ++nacc;
        }
        if (lane < K && ((amask >> lane) & 1u)) {
            const int rank = __popc(amask & below);
            const int id = npts + rank;
            M.ptx[id] = px; M.pty[id] = py;
            M.queue[nq + rank] = id;
            M.grid[gx + gy * gw] = id;
        }
        __syncwarp();
        npts += nacc;
        nq += nacc;
    }
    if (overflow && lane == 0) *status |= HS_ST_POISSON_OVERFLOW;
    __syncwarp();
    return npts;
}

constexpr int POISSON_K = 4;                        // tries per active point of the block form
constexpr int POISSON_BATCH = 32;                   // active points whose variates are made together
constexpr int POISSON_PROD = POISSON_K * POISSON_BATCH;   // producer threads

// Work arrays of poisson_block in the same shared memory (24 bytes per background cell): the point
// in each cell, or POISSON_EMPTY; the cell of each point number; the active numbers as a bitmap.
constexpr double POISSON_EMPTY = 1e300;             // farther than any radius
struct PoissonCells {
    double2 *pos;
    int32_t *cell_of;
    unsigned *words;
};
HS_DEV PoissonCells poisson_cells_in(unsigned char *base, int gsz) {
    PoissonCells M;
    M.pos = reinterpret_cast<double2 *>(base);
    M.cell_of = reinterpret_cast<int32_t *>(M.pos + gsz);
    M.words = reinterpret_cast<unsigned *>(M.cell_of + gsz);
    return M;
}

// The loop of poisson_warp for K = POISSON_K on the dynamic shared memory of a CTA of at least
// 32 + POISSON_PROD threads: the points, their order and the variates are the same. An active
// point's variates depend only on how many points came before it, so warps 1-4 make the next 32
// points' variates, sines and distances while warp 0 runs the sequential part, which has no
// transcendental left. The queue is the set of active point numbers in order (appended in order,
// popped anywhere), so it is a bitmap and the pick the qi-th set bit; eight lanes per try check
// its 25 cells, and the tries' mutual conflicts are tested in parallel. The chain of one point is
// bound by its instructions' latencies (loads, shuffles and ballots of 30 cycles each, one warp):
// about 1,600 cycles against 3,000 for poisson_warp on one warp. The selection kernel at 1024^2,
// r = 84 cells, about 65 points a step: 203 -> 61 us.
HS_DEV int poisson_block(const HsLattice &L, const HsGridPlan &P, int cap, uint64_t call0, int *n_iter, int *status) {
    extern __shared__ __align__(16) unsigned char s_ws[];
    __shared__ double s_u[2][POISSON_BATCH], s_d[2][POISSON_PROD], s_c[2][POISSON_PROD], s_s[2][POISSON_PROD];
    __shared__ int s_np, s_it, s_more[2];   // s_more: by batch parity, so a late reader never sees the next one
    constexpr int K = POISSON_K;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const double width = L.nx, height = L.ny;
    const double r = P.r_cells + 1.0;
    const double cs = r / sqrt(2.0), inv = 1.0 / cs;
    const double rSq = r * r;
    const int gw = (int)ceil(width / cs), gh = (int)ceil(height / cs);
    const int gsz = gw * gh;
    const int nw = (gsz + 31) >> 5, cw = (nw + 31) >> 5;   // bitmap words, and words per lane
    const PoissonCells M = poisson_cells_in(s_ws, gsz);
    for (int g = threadIdx.x; g < gsz; g += blockDim.x) M.pos[g] = make_double2(POISSON_EMPTY, POISSON_EMPTY);
    for (int g = threadIdx.x; g < nw; g += blockDim.x) M.words[g] = g == 0 ? 1u : 0u;
    // (int)(v / cs); the division itself only next to a cell border
    auto cell = [&](double v) {
        const double q = v * inv;
        const int i = (int)q;
        const double f = q - (double)i;
        return (f < 1e-6 || f > 1.0 - 1e-6) ? (int)(v / cs) : i;
    };
    const bool small = gsz < 4 * gw + 16;       // flat cell numbers may wrap more than once
    const double hw = width * 0.5, hh = height * 0.5;
    auto near = [&](double dx, double dy) {     // the distance rule of the grid check
        dx = fabs(dx);
        dy = fabs(dy);
        dx = dx > hw ? dx - width : dx;
        dy = dy > hh ? dy - height : dy;
        return dx * dx + dy * dy <= rSq;
    };
    auto produce = [&](int batch) {   // threads 32 .. 32 + POISSON_PROD - 1
        const int e = threadIdx.x - 32, it = e / K, t = e - it * K, b = batch & 1;
        const uint64_t c = call0 + 2 + (uint64_t)(batch * POISSON_BATCH + it) * (1 + 2 * K);
        if (t == 0) s_u[b][it] = hs_u53(L.seed, c, 0u);
        const double alpha = 6.283185307179586 * hs_u53(L.seed, c + 1 + 2 * t, 0u);
        s_d[b][e] = r * sqrt(3.0 * hs_u53(L.seed, c + 2 + 2 * t, 0u) + 1.0);
        s_c[b][e] = cos(alpha);
        s_s[b][e] = sin(alpha);
    };
    __syncthreads();
    if (warp >= 1 && warp <= POISSON_PROD / 32) produce(0);
    else if (warp == 0 && lane == 0) {
        const double p0x = (double)(int)(width * hs_u53(L.seed, call0, 0u));
        const double p0y = (double)(int)(height * hs_u53(L.seed, call0 + 1, 0u));
        const int c = (int)(p0x / cs) + (int)(p0y / cs) * gw;
        M.pos[c] = make_double2(p0x, p0y);
        M.cell_of[0] = c;
    }
    __syncthreads();
    if (warp == 0) {
        int npts = 1, nq = 1, it = 0;
        // bitmap: lane l counts the set bits of words [l cw, (l + 1) cw) and those before them
        int cnt = lane == 0 ? 1 : 0, pre = lane == 0 ? 0 : 1;
        unsigned mine = lane == 0 ? 1u : 0u;               // the lane's word when cw == 1
        const int own = 32 * cw * lane;                    // the lane's first point number
        const int t = lane >> 3, sub = lane & 7;
        int off[4];                                        // the lane's cells of a try's 5 x 5 (the last one again)
#pragma unroll
        for (int j = 0; j < 4; ++j) { const int c = min(sub + 8 * j, 24); off[j] = (c / 5 - 2) + (c % 5 - 2) * gw; }
        // pairs of tries u < v, on lanes 0-5: (0,1) (0,2) (1,2) (0,3) (1,3) (2,3)
        const int lv = lane == 0 ? 8 : (lane < 3 ? 16 : 24), lu = 8 * (lane < 3 ? (lane == 2 ? 1 : 0) : (lane - 3) & 3);
        bool overflow = false;
        for (int batch = 0;; ++batch) {
            const int b = batch & 1;
            for (int k = 0; k < POISSON_BATCH && nq > 0 && !overflow; ++k, ++it) {
                const int qi = (int)(s_u[b][k] * nq);
                const int e = k * K + t;
                const double d = s_d[b][e], ca = s_c[b][e], sa = s_s[b][e];
                // the qi-th active point
                const int src = __ffs(__ballot_sync(0xffffffffu, pre <= qi && qi < pre + cnt)) - 1;
                int rank = qi - __shfl_sync(0xffffffffu, pre, src);
                int wi = src;
                unsigned word;
                if (cw == 1) word = __shfl_sync(0xffffffffu, mine, src);
                else {                              // cw < 32: the arrays fit shared memory
                    const unsigned w = (lane < cw && src * cw + lane < nw) ? M.words[src * cw + lane] : 0u;
                    const int c = __popc(w);
                    int inc = c;
#pragma unroll
                    for (int s = 1; s < 32; s <<= 1) { const int v = __shfl_up_sync(0xffffffffu, inc, s); if (lane >= s) inc += v; }
                    const int sl = __ffs(__ballot_sync(0xffffffffu, inc > rank)) - 1;
                    rank -= __shfl_sync(0xffffffffu, inc - c, sl);
                    word = __shfl_sync(0xffffffffu, w, sl);
                    wi = src * cw + sl;
                }
                const int bit = __ffs(__ballot_sync(0xffffffffu, ((word >> lane) & 1u) && __popc(word & below) == rank)) - 1;
                // try t of this point (the same on its eight lanes) and its cell
                const double2 q = M.pos[M.cell_of[32 * wi + bit]];
                word &= ~(1u << bit);
                if (lane == src) { --cnt; mine = word; }
                if (lane > src) --pre;
                if (cw > 1 && lane == 0) M.words[wi] = word;
                nq -= 1;
                const double px = q.x + d * ca, py = q.y + d * sa;
                const bool inb = 0.0 <= px && px < width && 0.0 <= py && py < height;
                const int flat = inb ? cell(px) + cell(py) * gw : 0;
                // existing points in the cells around it (branch-free, so that the loads overlap)
                int g[4];
                if (small) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) g[j] = pymod(flat + off[j], gsz);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) { const int c = flat + off[j]; g[j] = c < 0 ? c + gsz : (c >= gsz ? c - gsz : c); }
                }
                double2 h[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) h[j] = M.pos[g[j]];
                // tries u < v in conflict, u's cell being among those v checks
                const double ux = __shfl_sync(0xffffffffu, px, lu), uy = __shfl_sync(0xffffffffu, py, lu);
                const double vx = __shfl_sync(0xffffffffu, px, lv), vy = __shfl_sync(0xffffffffu, py, lv);
                const int df = __shfl_sync(0xffffffffu, flat, lu) - __shfl_sync(0xffffffffu, flat, lv) + 2;
                bool hit = !inb;
#pragma unroll
                for (int j = 0; j < 4; ++j) hit |= near(px - h[j].x, py - h[j].y);
                bool pair = near(vx - ux, vy - uy) && lane < 6;
                if (pair) {                         // (uf - vf - a gw + 2) mod gsz <= 4 for a row a = -2..2
                    bool seen = false;
                    for (int a = -2; a <= 2; ++a) seen |= pymod(df - a * gw, gsz) <= 4;
                    pair = seen;
                }
                const unsigned hits = __ballot_sync(0xffffffffu, hit);
                const unsigned pairs = __ballot_sync(0xffffffffu, pair);
                unsigned amask = 0u;
                if (!(hits & 0xffu)) amask = 1u;
                if (!(hits & 0xff00u) && !(amask & (pairs & 1u))) amask |= 2u;
                if (!(hits & 0xff0000u) && !(amask & ((pairs >> 1) & 3u))) amask |= 4u;
                if (!(hits & 0xff000000u) && !(amask & ((pairs >> 3) & 7u))) amask |= 8u;
                if (amask) {                        // warp-uniform
                    while (npts + __popc(amask) > cap) { amask &= ~(0x80000000u >> __clz(amask)); overflow = true; }
                    const int nacc = __popc(amask);
                    if (sub == 0 && ((amask >> t) & 1u)) {
                        M.pos[flat] = make_double2(px, py);
                        M.cell_of[npts + __popc(amask & ((1u << t) - 1u))] = flat;
                    }
                    // the new numbers [npts, npts + nacc) are active
                    const int lo = min(max(npts - own, 0), 32 * cw), hi = min(max(npts + nacc - own, 0), 32 * cw);
                    cnt += hi - lo;
                    pre += min(max(own - npts, 0), nacc);
                    if (cw == 1) mine |= hi > lo ? (0xffffffffu >> (32 - (hi - lo))) << lo : 0u;
                    else if (lane == 0)
                        for (int id = npts; id < npts + nacc; ++id) M.words[id >> 5] |= 1u << (id & 31);
                    npts += nacc;
                    nq += nacc;
                }
                __syncwarp();
            }
            const bool more = nq > 0 && !overflow;
            if (lane == 0) s_more[b] = more;
            asm volatile("bar.sync 1, %0;" ::"n"(32 + POISSON_PROD) : "memory");   // the next batch is ready
            if (!more) break;
        }
        if (lane == 0) {
            s_np = npts;
            s_it = it;
            if (overflow) *status |= HS_ST_POISSON_OVERFLOW;
        }
    } else if (warp <= POISSON_PROD / 32) {
        for (int batch = 1;; ++batch) {
            produce(batch);
            asm volatile("bar.sync 1, %0;" ::"n"(32 + POISSON_PROD) : "memory");
            if (!s_more[(batch & 1) ^ 1]) break;
        }
    }
    __syncthreads();
    *n_iter = s_it;
    return s_np;
}

// Select from the sampled points, by the whole CTA: those with x < max(r, w - r), y < max(r, h - r)
// (PBC=True default), offset by the next two variates, in grid-cell order. point(g, x, y) gives the
// point of background cell g, if there is one. Returns how many nearest cell indices were written to
// (S.py, S.px).
template <typename Point>
HS_DEV int poisson_select(const HsLattice &L, const HsGridPlan &P, const MetroScratch &S, Point point, uint64_t &call,
                          int *warp_tot, int *status) {
    const double width = L.nx, height = L.ny;
    const double r = P.r_cells + 1.0;
    const double cs = r / sqrt(2.0);
    const int gsz = (int)ceil(width / cs) * (int)ceil(height / cs);
    const double lx = fmax(r, width - r), ly = fmax(r, height - r);
    const double ox = (double)(int)(hs_u53(L.seed, call, 0u) * width), oy = (double)(int)(hs_u53(L.seed, call + 1, 0u) * height);
    call += 2;
    int k = 0;
    for (int g0 = 0; g0 < gsz; g0 += blockDim.x) {
        const int g = g0 + (int)threadIdx.x;
        double x = 0.0, y = 0.0;
        bool keep = g < gsz && point(g, x, y);
        int ix = 0, iy = 0;
        keep = keep && x >= 0.0 && y >= 0.0 && x < lx && y < ly;
        if (keep) {
            const double fx = fmod(x + ox, width), fy = fmod(y + oy, height);
            // nearest cell index, ties to the lower index
            ix = (int)floor(fx); if (fx - ix > 0.5) ix += 1; ix = min(max(ix, 0), L.nx - 1);
            iy = (int)floor(fy); if (fy - iy > 0.5) iy += 1; iy = min(max(iy, 0), L.ny - 1);
        }
        int tot;
        const int pos = k + block_excl_scan(keep, warp_tot, tot);
        if (keep && pos < S.cap) { S.py[pos] = iy; S.px[pos] = ix; }
        k += tot;
    }
    if (k > S.cap) { if (threadIdx.x == 0) *status |= HS_ST_POISSON_OVERFLOW; k = S.cap; }
    return k;
}

// Block-wide exclusive scans of two flags at once (3 barriers in total).
HS_DEV void block_excl_scan2(int f0, int f1, int *wt, int &pre0, int &pre1, int &tot0, int &tot1) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned b0 = __ballot_sync(0xffffffffu, f0), b1 = __ballot_sync(0xffffffffu, f1);
    if (lane == 0) { wt[warp] = __popc(b0); wt[33 + warp] = __popc(b1); }
    __syncthreads();
    if (warp == 0) {
        int v0 = lane < nw ? wt[lane] : 0, v1 = lane < nw ? wt[33 + lane] : 0;
        int i0 = v0, i1 = v1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, i0, o), b = __shfl_up_sync(0xffffffffu, i1, o);
            if (lane >= o) { i0 += a; i1 += b; }
        }
        if (lane < nw) { wt[lane] = i0 - v0; wt[33 + lane] = i1 - v1; }
        if (lane == 31) { wt[32] = i0; wt[65] = i1; }
    }
    __syncthreads();
    const unsigned below = (1u << lane) - 1u;
    pre0 = wt[warp] + __popc(b0 & below);
    pre1 = wt[33 + warp] + __popc(b1 & below);
    tot0 = wt[32]; tot1 = wt[65];
    __syncthreads();
}

// Grid-selection Metropolis step with one candidate per thread (n_sc <= blockDim.x), kept in
// registers: the supercell filter, the offset and the occupation filter of
// hotspice/core.py:534-553 and 484-487 become one pair of fused ballot scans. Returns false,
// without side effects, when the step needs the rare branches (no candidate survives the
// supercell filter -> _select_single, or none is occupied -> select() retries); the general
// path then runs the step from the same RNG call.
HS_DEV bool metro_grid_fast(const HsLattice &L, HsCounters *C, const HsSwitchList &sw, const HsGridPlan &P,
                            uint64_t call) {
    __shared__ int wt[66];
    __shared__ int s_bins[256];
    __shared__ double s_tsum[32];
    const int t = threadIdx.x;
    int ox, oy;
    if (L.pbc) {
        ox = (int)floor(hs_u53(L.seed, call, 0u) * L.nx);
        oy = (int)floor(hs_u53(L.seed, call + 1, 0u) * L.ny);
    } else {
        ox = -P.Rx + (int)floor(hs_u53(L.seed, call, 0u) * (2.0 * P.Rx));
        oy = -P.Ry + (int)floor(hs_u53(L.seed, call + 1, 0u) * (2.0 * P.Ry));
    }
    if (P.Rx == L.nx) ox = 0;
    if (P.Ry == L.ny) oy = 0;
    const int phase = pymod(oy, L.uy) * L.ux + pymod(ox, L.ux);
    const int off = P.phase_off[phase], len = P.phase_off[phase + 1] - off;
    if (len <= 0) return false;
    const int nscx = (min(P.snx, L.nx) + 1) / 2;
    int ok = 0, valid = 0, x = 0, y = 0;
    if (t < P.n_sc) {
        const int pick = (int)floor(hs_u53(L.seed, call + 2, (uint32_t)t) * len);
        const int yx = __ldg(P.phase_yx + off + pick);
        x = 2 * (t % nscx) * P.Rx + (yx & 0xffff);
        y = 2 * (t / nscx) * P.Ry + (yx >> 16);
        if (L.pbc) {
            ok = x < max(P.Rx, L.nx - P.Rx) && y < max(P.Ry, L.ny - P.Ry);
            x = (x + ox) % L.nx; y = (y + oy) % L.ny;
        } else {
            x += ox; y += oy;
            ok = x >= 0 && x < L.nx && y >= 0 && y < L.ny;
        }
    }
    // occupation, spin, moment and energies in one round trip
    int8_t m_old = 0;
    float mm_old = 0.f;
    double E = 0.0, Ep;
    if (ok) {
        const int64_t i = (int64_t)y * L.nx + x;
        const int8_t oc = __ldg(L.occ + i);
        m_old = __ldcg(L.m + i);
        mm_old = __ldcg(L.mm + i);
        hs_energy_at(L, y, x, E, Ep);
        valid = oc != 0;
    }
    int pre_ok, r, n_ok, k;
    block_excl_scan2(ok, valid, wt, pre_ok, r, n_ok, k);
    if (n_ok == 0 || k == 0) return false;  // block-uniform
    const bool mtime = P.metropolis_time != 0;
    const uint64_t call_time = call + 3;
    const uint64_t call_acc = mtime ? call + 4 : call + 3;
    for (int b = t; b < 256; b += blockDim.x) s_bins[b] = 0;
    int acc = 0;
    double tpart = 0.0;
    long long near = 0;
    if (valid) {
        const int64_t i = (int64_t)y * L.nx + x;
        const double beta = hs_beta(L, i);
        const double p = fmin(fmax(exp(2.0 * E * beta), 1e-10), 1e10);
        if (mtime) {
            double b1, b2;
            hs_barriers(L, y, x, b1, b2);
            const double u = hs_u53(L.seed, call_time, (uint32_t)r);
            tpart = -log(u) / P.attempt_freq / (double)L.n_occ * exp(fmin(b1, b2) * beta);
        }
        const double u = hs_u53(L.seed, call_acc, (uint32_t)r);
        acc = u < p;
        if (fabs(u - p) <= p * beta * 2e-6 * fabs(E) && p < 1e10 && p > 1e-10) near = 1;
    }
    int pa, dummy, nacc, dtot;
    block_excl_scan2(acc, 0, wt, pa, dummy, nacc, dtot);
    const int bin = acc ? (x % L.ux) + (y % L.uy) * L.ux : 0;
    if (acc) {
        const int64_t i = (int64_t)y * L.nx + x;
        L.m[i] = (int8_t)(-m_old);
        L.mm[i] = -mm_old;
        if (pa < sw.cap) { sw.y[pa] = y; sw.x[pa] = x; }
        atomicAdd(&s_bins[bin], 1);
    }
    if (mtime) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tpart += __shfl_xor_sync(0xffffffffu, tpart, o);
        if ((t & 31) == 0) s_tsum[t >> 5] = tpart;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) near += __shfl_xor_sync(0xffffffffu, near, o);
    if ((t & 31) == 0 && near) atomicAdd((unsigned long long *)&C->near_threshold, (unsigned long long)near);
    __syncthreads();
    if (acc && sw.mode && pa < sw.cap) sw.mode[pa] = s_bins[bin] > L.trunc_cutoff ? 1 : 0;
    if (t == 0) {
        if (mtime) {
            double ts = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) ts += s_tsum[w];
            C->t += ts;
        }
        const int ncap = min(nacc, sw.cap);
        C->attempted += k;
        C->switches += ncap;
        C->rng_call = call_acc + 1;
        C->n_sw = ncap;
        C->steps += 1;
        if (nacc > sw.cap) C->status |= HS_ST_SWITCH_OVERFLOW;
    }
    __syncthreads();
    return true;
}

// The same step as metro_grid_fast when every supercell fits one warp (n_sc <= 32), executed
// by a single warp with ballots instead of block scans: candidates, acceptances and switch
// list in the same order, the per-sublattice switch counts by __match_any_sync, the
// METROPOLIS_TIME sum by the same xor-shuffle tree (the other warps held only zeros), so the
// results are identical. Returns false, without side effects, when the step needs the rare
// branches (the general path then runs it from the same call).
HS_DEV bool metro_grid_warp(const HsLattice &L, HsCounters *C, const HsSwitchList &sw, const HsGridPlan &P,
                            uint64_t call) {
    const int lane = threadIdx.x & 31;
    // the lane's pick variate does not depend on the offsets: drawn alongside them
    const double upick = lane < P.n_sc ? hs_u53(L.seed, call + 2, (uint32_t)lane) : 0.0;
    int ox, oy;
    if (L.pbc) {
        ox = (int)floor(hs_u53(L.seed, call, 0u) * L.nx);
        oy = (int)floor(hs_u53(L.seed, call + 1, 0u) * L.ny);
    } else {
        ox = -P.Rx + (int)floor(hs_u53(L.seed, call, 0u) * (2.0 * P.Rx));
        oy = -P.Ry + (int)floor(hs_u53(L.seed, call + 1, 0u) * (2.0 * P.Ry));
    }
    if (P.Rx == L.nx) ox = 0;
    if (P.Ry == L.ny) oy = 0;
    const int phase = pymod(oy, L.uy) * L.ux + pymod(ox, L.ux);
    const int off = P.phase_off[phase], len = P.phase_off[phase + 1] - off;
    if (len <= 0) return false;
    const int nscx = (min(P.snx, L.nx) + 1) / 2;
    int ok = 0, valid = 0, x = 0, y = 0;
    if (lane < P.n_sc) {
        const int pick = (int)floor(upick * len);
        const int yx = __ldg(P.phase_yx + off + pick);
        x = 2 * (lane % nscx) * P.Rx + (yx & 0xffff);
        y = 2 * (lane / nscx) * P.Ry + (yx >> 16);
        if (L.pbc) {
            ok = x < max(P.Rx, L.nx - P.Rx) && y < max(P.Ry, L.ny - P.Ry);
            x = (x + ox) % L.nx; y = (y + oy) % L.ny;
        } else {
            x += ox; y += oy;
            ok = x >= 0 && x < L.nx && y >= 0 && y < L.ny;
        }
    }
    // occupation, spin, moment and energies in one round trip
    int8_t m_old = 0;
    float mm_old = 0.f;
    double E = 0.0, Ep;
    if (ok) {
        const int64_t i = (int64_t)y * L.nx + x;
        const int8_t oc = __ldg(L.occ + i);
        m_old = __ldcg(L.m + i);
        mm_old = __ldcg(L.mm + i);
        hs_energy_at(L, y, x, E, Ep);
        valid = oc != 0;
    }
    const unsigned below = (1u << lane) - 1u;
    const unsigned okb = __ballot_sync(0xffffffffu, ok), vb = __ballot_sync(0xffffffffu, valid);
    const int k = __popc(vb);
    if (okb == 0u || k == 0) return false;   // warp-uniform
    const int r = __popc(vb & below);
    const bool mtime = P.metropolis_time != 0;
    const uint64_t call_time = call + 3;
    const uint64_t call_acc = mtime ? call + 4 : call + 3;
    int acc = 0;
    double tpart = 0.0;
    int near = 0;
    if (valid) {
        const int64_t i = (int64_t)y * L.nx + x;
        const double beta = hs_beta(L, i);
        const double p = fmin(fmax(exp(2.0 * E * beta), 1e-10), 1e10);
        if (mtime) {
            double b1, b2;
            hs_barriers(L, y, x, b1, b2);
            const double u = hs_u53(L.seed, call_time, (uint32_t)r);
            tpart = -log(u) / P.attempt_freq / (double)L.n_occ * exp(fmin(b1, b2) * beta);
        }
        const double u = hs_u53(L.seed, call_acc, (uint32_t)r);
        acc = u < p;
        if (fabs(u - p) <= p * beta * 2e-6 * fabs(E) && p < 1e10 && p > 1e-10) near = 1;
    }
    const unsigned accb = __ballot_sync(0xffffffffu, acc);
    const int nacc = __popc(accb), pa = __popc(accb & below);
    const int bin = (x % L.ux) + (y % L.uy) * L.ux;
    const unsigned same = __match_any_sync(0xffffffffu, acc ? bin : -1);
    if (acc) {
        const int64_t i = (int64_t)y * L.nx + x;
        L.m[i] = (int8_t)(-m_old);
        L.mm[i] = -mm_old;
        if (pa < sw.cap) {
            sw.y[pa] = y; sw.x[pa] = x;
            if (sw.mode) sw.mode[pa] = __popc(same & accb) > L.trunc_cutoff ? 1 : 0;
        }
    }
    if (mtime) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tpart += __shfl_xor_sync(0xffffffffu, tpart, o);
    }
    const int nnear = __popc(__ballot_sync(0xffffffffu, near));
    if (lane == 0) {
        if (nnear) C->near_threshold += nnear;
        if (mtime) C->t += tpart;
        const int ncap = min(nacc, sw.cap);
        C->attempted += k;
        C->switches += ncap;
        C->rng_call = call_acc + 1;
        C->n_sw = ncap;
        C->steps += 1;
        if (nacc > sw.cap) C->status |= HS_ST_SWITCH_OVERFLOW;
    }
    return true;
}

// One Metropolis step executed by one CTA (selection, acceptance, flips, switch list). POISSON: the
// plan may be a Poisson-disc one (a kernel that never sees one leaves the sampler's code out).
template <bool POISSON>
HS_DEV void metro_step_cta(const HsLattice &L, HsCounters *C, const HsSwitchList &sw, const HsGridPlan &P,
                           const MetroScratch &S, void *ws = nullptr, int ws_bytes = 0) {
    __shared__ int warp_tot[33];
    __shared__ uint64_t s_call;
    __shared__ int s_status;
    __shared__ int s_bins[256];
    __shared__ double s_tsum[32];
    if (C->done) return;
    if (!hs_progress_continue(C, L.n_occ)) {
        if (threadIdx.x == 0) { C->done = 1; C->n_sw = 0; }
        return;
    }
    uint64_t call = C->rng_call;
    if (P.sample_scheme == HS_SAMPLE_GRID && P.n_sc <= 32) {
        __shared__ int s_done;
        __syncthreads();   // every warp has tested the stop rule before warp 0 writes what it reads
        if (threadIdx.x < 32) {
            const bool d = metro_grid_warp(L, C, sw, P, call);
            if (threadIdx.x == 0) s_done = d;
        }
        __syncthreads();
        const int d = s_done;
        __syncthreads();   // s_done is rewritten by the next step
        if (d) return;
    } else if (P.sample_scheme == HS_SAMPLE_GRID && P.n_sc <= (int)blockDim.x && L.ux * L.uy <= 256 &&
               metro_grid_fast(L, C, sw, P, call))
        return;
    if (threadIdx.x == 0) s_status = 0;
    int k = 0;
    int retry = 0;
    for (; retry < MAX_RETRY; ++retry) {
        // ---- selection -------------------------------------------------------------------
        if (P.sample_scheme == HS_SAMPLE_GRID) {
            int ox, oy;
            if (L.pbc) {
                ox = (int)floor(hs_u53(L.seed, call, 0u) * L.nx);
                oy = (int)floor(hs_u53(L.seed, call + 1, 0u) * L.ny);
            } else {
                ox = -P.Rx + (int)floor(hs_u53(L.seed, call, 0u) * (2.0 * P.Rx));
                oy = -P.Ry + (int)floor(hs_u53(L.seed, call + 1, 0u) * (2.0 * P.Ry));
            }
            if (P.Rx == L.nx) ox = 0;
            if (P.Ry == L.ny) oy = 0;
            const int phase = pymod(oy, L.uy) * L.ux + pymod(ox, L.ux);
            const int off = P.phase_off[phase], len = P.phase_off[phase + 1] - off;
            const int nscx = (min(P.snx, L.nx) + 1) / 2;
            const int limx = max(P.Rx, L.nx - P.Rx), limy = max(P.Ry, L.ny - P.Ry);
            // candidates, in the row-major supercell order of ixx[:sny:2, :snx:2].ravel()
            for (int t = threadIdx.x; t < P.n_sc; t += blockDim.x) {
                int ix = -1, iy = -1;
                if (len > 0) {
                    const int pick = (int)floor(hs_u53(L.seed, call + 2, (uint32_t)t) * len);
                    const int yx = P.phase_yx[off + pick];
                    ix = 2 * (t % nscx) * P.Rx + (yx & 0xffff);
                    iy = 2 * (t / nscx) * P.Ry + (yx >> 16);
                }
                S.py[t] = iy; S.px[t] = ix;
            }
            if (len <= 0 && threadIdx.x == 0) s_status |= HS_ST_SELECT_RETRY;
            __syncthreads();
            const int nx = L.nx, ny = L.ny, pbc = L.pbc;
            k = block_compact(S.py, S.px, P.n_sc, [&](int y, int x) {
                if (x < 0) return false;
                if (pbc) return x < limx && y < limy;
                x += ox; y += oy;
                return x >= 0 && x < nx && y >= 0 && y < ny;
            }, warp_tot);
            for (int t = threadIdx.x; t < k; t += blockDim.x) {
                if (pbc) { S.px[t] = (S.px[t] + ox) % L.nx; S.py[t] = (S.py[t] + oy) % L.ny; }
                else { S.px[t] += ox; S.py[t] += oy; }
            }
            call += 3;
            __syncthreads();
            if (k == 0) {  // no sample survived: _select_single (core.py:558)
                const int i = (int)floor(hs_u53(L.seed, call, 0u) * L.n_occ);
                if (threadIdx.x == 0) { const int f = L.nonzero[i]; S.py[0] = f / L.nx; S.px[0] = f % L.nx; }
                call += 1;
                k = 1;
            }
        } else if (P.sample_scheme == HS_SAMPLE_SINGLE) {
            const int i = (int)floor(hs_u53(L.seed, call, 0u) * L.n_occ);
            if (threadIdx.x == 0) { const int f = L.nonzero[i]; S.py[0] = f / L.nx; S.px[0] = f % L.nx; }
            call += 1;
            k = 1;
        } else if constexpr (POISSON) {
            // the sampler's arrays in the shared workspace when they fit, else in the scratch
            const int64_t g = (int64_t)hs_poisson_grid_cells(L, P);
            if (g > S.gsz || P.poisson_k < 1 || 25 * P.poisson_k > 32 * 32) {   // no samples: retry, then report
                if (threadIdx.x == 0) s_status |= HS_ST_POISSON_OVERFLOW;
                k = 0;
                continue;
            }
            const bool fits = ws && hs_poisson_mem_bytes(g) <= ws_bytes;
            int st = 0;
            if (fits && P.poisson_k == POISSON_K && blockDim.x >= 32 + POISSON_PROD) {
                int iters;
                poisson_block(L, P, S.gsz, call, &iters, &st);
                call += 2 + (uint64_t)iters * (1 + 2 * POISSON_K);
                const PoissonCells M = poisson_cells_in(reinterpret_cast<unsigned char *>(ws), (int)g);
                k = poisson_select(L, P, S, [&](int c, double &x, double &y) {
                    const double2 p = M.pos[c];
                    x = p.x; y = p.y;
                    return p.x < POISSON_EMPTY;
                }, call, warp_tot, &st);
            } else {
                PoissonMem M;
                if (fits) M = poisson_mem_in(ws, (int)g);
                else { M.grid = S.grid; M.ptx = S.ptx; M.pty = S.pty; M.queue = S.queue; }
                if (threadIdx.x < 32) {
                    uint64_t c = call;
                    poisson_warp(L, P, S, M, c, &st);
                    if (threadIdx.x == 0) s_call = c;
                }
                __syncthreads();
                call = s_call;
                k = poisson_select(L, P, S, [&](int c, double &x, double &y) {
                    const int p = M.grid[c];
                    if (p < 0) return false;
                    x = M.ptx[p]; y = M.pty[p];
                    return true;
                }, call, warp_tot, &st);
            }
            if (threadIdx.x == 0) s_status |= st;
        }
        __syncthreads();
        // ---- select(): drop unoccupied picks, retry if none is left (core.py:484-487) -------
        const int8_t *occ = L.occ;
        const int nx = L.nx;
        k = block_compact(S.py, S.px, k, [&](int y, int x) { return occ[(int64_t)y * nx + x] != 0; }, warp_tot);
        if (k > 0) break;
    }
    if (retry == MAX_RETRY) {
        if (threadIdx.x == 0) { C->status |= HS_ST_SELECT_RETRY; C->rng_call = call; C->n_sw = 0; }
        return;
    }
    // ---- acceptance --------------------------------------------------------------------------
    const bool mtime = P.metropolis_time != 0;
    const uint64_t call_time = call;
    const uint64_t call_acc = mtime ? call + 1 : call;
    for (int b = threadIdx.x; b < 256; b += blockDim.x) s_bins[b] = 0;
    double tpart = 0.0;
    long long near = 0;
    int acc_base = 0;
    __syncthreads();
    for (int base = 0; base < k; base += blockDim.x) {
        const int t = base + threadIdx.x;
        int acc = 0, y = 0, x = 0;
        if (t < k) {
            y = S.py[t]; x = S.px[t];
            const int64_t i = (int64_t)y * L.nx + x;
            double E, Ep;
            hs_energy_at(L, y, x, E, Ep);
            const double dE = -2.0 * E;
            const double beta = hs_beta(L, i);
            const double p = fmin(fmax(exp(-dE * beta), 1e-10), 1e10);
            if (mtime) {
                double b1, b2;
                hs_barriers(L, y, x, b1, b2);
                const double u = hs_u53(L.seed, call_time, (uint32_t)t);
                tpart += -log(u) / P.attempt_freq / (double)L.n_occ * exp(fmin(b1, b2) * beta);
            }
            const double u = hs_u53(L.seed, call_acc, (uint32_t)t);
            acc = u < p;
            // decision margin below a 1e-6 relative energy perturbation
            if (fabs(u - p) <= p * beta * 2e-6 * fabs(E) && p < 1e10 && p > 1e-10) near += 1;
        }
        int tot;
        const int pre = block_excl_scan(acc, warp_tot, tot);
        if (acc) {
            const int out = acc_base + pre;
            if (out < sw.cap) { sw.y[out] = y; sw.x[out] = x; }
        }
        acc_base += tot;
    }
    const int nacc = acc_base;
    // time sum (METROPOLIS_TIME)
    if (mtime) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tpart += __shfl_xor_sync(0xffffffffu, tpart, o);
        if ((threadIdx.x & 31) == 0) s_tsum[threadIdx.x >> 5] = tpart;
    }
    // near-threshold count
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) near += __shfl_xor_sync(0xffffffffu, near, o);
    if ((threadIdx.x & 31) == 0 && near) atomicAdd((unsigned long long *)&C->near_threshold, (unsigned long long)near);
    __syncthreads();
    const int ncap = min(nacc, sw.cap);
    // flips and per-sublattice counts
    for (int t = threadIdx.x; t < ncap; t += blockDim.x) {
        const int y = sw.y[t], x = sw.x[t];
        const int64_t i = (int64_t)y * L.nx + x;
        L.m[i] = (int8_t)(-L.m[i]);
        L.mm[i] = -L.mm[i];
        const int bin = (x % L.ux) + (y % L.uy) * L.ux;
        if (bin < 256) atomicAdd(&s_bins[bin], 1);
    }
    __syncthreads();
    if (sw.mode)
        for (int t = threadIdx.x; t < ncap; t += blockDim.x) {
            const int y = sw.y[t], x = sw.x[t];
            const int bin = (x % L.ux) + (y % L.uy) * L.ux;
            sw.mode[t] = (bin < 256 && s_bins[bin] > L.trunc_cutoff) ? 1 : 0;
        }
    if (threadIdx.x == 0) {
        if (mtime) {
            double ts = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) ts += s_tsum[w];
            C->t += ts;
        }
        C->attempted += k;
        C->switches += ncap;
        C->rng_call = call_acc + 1;
        C->n_sw = ncap;
        C->steps += 1;
        C->status |= s_status;
        if (nacc > sw.cap) C->status |= HS_ST_SWITCH_OVERFLOW;
    }
}

// ---- Wolff -------------------------------------------------------------------------------

constexpr int WT = 1024;

struct WolffScratch {
    int32_t *chk_ep;   // epoch in which the cell was checked (seed or frontier)
    int32_t *cl_ep;    // epoch in which the cell joined the cluster, written when its layer is complete
    int32_t *list;     // cluster cells in BFS order (capacity N)
    int32_t *cand;     // frontier of the current layer (capacity N)
    int32_t *epoch;    // last epoch used with these stamps; kept here, not in the counters, so that
                       // restoring an earlier counter state never makes an old stamp current again
};

// A cluster that fits these lists grows on one warp in shared memory.
constexpr int WF_HASH = 512;        // slots: cells checked, with the layer in which they joined
constexpr int WF_CHECKED = 320;     // cells checked at most (load factor 5/8)
constexpr int WF_CELLS = 160;       // cells of the cluster at most
constexpr int WF_MASK = sizeof(HsLattice::nn);   // entries of a neighbour mask at most
static_assert(WF_MASK <= 32, "a lane per entry");
struct __align__(16) WolffFast {       // key is cleared in 16-byte words
    int key[WF_HASH];               // flat cell index, -1 empty
    int layer[WF_HASH];             // -1: checked, not a member
    int cell[WF_CELLS], yx[WF_CELLS];
    int cand[WF_CHECKED], cand_yx[WF_CHECKED], cand_slot[WF_CHECKED];
    int off[WF_MASK], w[WF_MASK];   // the neighbour mask's entries: (dy << 16) + dx + 32768, weight
    int nb;                         // of them
    int lstart, lend, layers, grown; // where a larger cluster goes on; grown: the step is complete
    unsigned long long call;
};

HS_DEV int wolff_slot(const WolffFast &F, int cell) {
    unsigned h = ((unsigned)cell * 2654435761u) >> 23;     // 9 bits: WF_HASH
    while (F.key[h] != cell && F.key[h] != -1) h = (h + 1) & (WF_HASH - 1);   // never full
    return (int)h;
}

// Bond probability 1 - exp(-2 J / kBT count), kBT = 1/beta (hotspice/core.py:599).
HS_DEV double wolff_bond_of(const HsLattice &L, int j, int count) {
    if (L.wolff_bond && count <= 24) return L.wolff_bond[count];
    const double kBT = 1.0 / hs_beta(L, j);
    return 1.0 - exp(-2.0 * L.J / kBT * (double)count);
}

// Growth of one cluster by the calling warp: the layers, frontiers and variates of wolff_step_cta's
// loop. Stops before a layer that might not fit (F.grown = 0; nothing outside F has been touched).
HS_DEV void wolff_grow_warp(const HsLattice &L, WolffFast &F, int seed, uint64_t call) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int nx = L.nx, ny = L.ny, ch = L.nn_h / 2, cw = L.nn_w / 2;
    for (int k = lane; k < WF_HASH / 4; k += 32) reinterpret_cast<int4 *>(F.key)[k] = make_int4(-1, -1, -1, -1);
    const int n_mask = L.nn_h * L.nn_w;           // at most WF_MASK
    const int wt = lane < n_mask ? L.nn[lane] : 0;
    const unsigned nz = __ballot_sync(0xffffffffu, wt != 0);
    if (wt) {
        const int k = __popc(nz & below);
        F.off[k] = (lane / L.nn_w - ch) * 65536 + (lane % L.nn_w - cw) + 32768;
        F.w[k] = wt;
    }
    const int nb = __popc(nz);
    const int sy = seed / nx, sx = seed - sy * nx;
    const int8_t ms = L.m[seed];
    __syncwarp();
    if (lane == 0) {
        const int h = wolff_slot(F, seed);
        F.key[h] = seed;
        F.layer[h] = 0;
        F.cell[0] = seed;
        F.yx[0] = sy * 65536 + sx;
        F.nb = nb;
    }
    __syncwarp();
    auto coord = [](int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); };    // one period off at most
    // a neighbour wraps twice, or a coordinate is beyond the packing
    const bool odd_size = nx < max(3, cw) || ny < max(3, ch) || nx > 65535 || ny > 32767;
    int lstart = 0, lend = 1, checked = 1, layer = 1;
    bool grown = false;
    for (;; ++layer) {
        const int pairs = (lend - lstart) * nb;
        if (checked + pairs > WF_CHECKED || lend + pairs > WF_CELLS || odd_size) break;
        // frontier: unchecked cells of the seed's spin next to the new cells
        int ncand = 0;
        for (int p0 = 0; p0 < pairs; p0 += 32) {
            const int p = p0 + lane;
            bool fresh = false;
            int j = 0, yx = 0, slot = 0;
            if (p < pairs) {
                const int q = p / nb, o = F.off[p - q * nb], c = F.yx[lstart + q];
                int y = (c >> 16) + (o >> 16), x = (c & 65535) + (o & 65535) - 32768;
                bool in = true;
                if (L.pbc) { y = coord(y, ny); x = coord(x, nx); }
                else in = y >= 0 && y < ny && x >= 0 && x < nx;
                j = y * nx + x;
                yx = y * 65536 + x;
                if (in && L.m[j] == ms) {
                    unsigned h = ((unsigned)j * 2654435761u) >> 23;
                    for (;; h = (h + 1) & (WF_HASH - 1)) {
                        const int was = atomicCAS(&F.key[h], -1, j);
                        if (was == -1) { fresh = true; slot = (int)h; F.layer[h] = -1; break; }
                        if (was == j) break;
                    }
                }
            }
            const unsigned b = __ballot_sync(0xffffffffu, fresh);
            if (fresh) {
                const int k = ncand + __popc(b & below);
                F.cand[k] = j; F.cand_yx[k] = yx; F.cand_slot[k] = slot;
            }
            ncand += __popc(b);
        }
        __syncwarp();
        if (ncand == 0) { grown = true; break; }     // empty frontier: no draw
        checked += ncand;
        int nacc = 0;
        for (int t0 = 0; t0 < ncand; t0 += 32) {
            const int t = t0 + lane;
            bool acc = false;
            int j = 0, yx = 0;
            if (t < ncand) {
                j = F.cand[t];
                yx = F.cand_yx[t];
                const double u = hs_u53(L.seed, call, (uint32_t)j);
                int count = 0;
                for (int k = 0; k < nb; ++k) {       // cluster neighbours of earlier layers
                    const int o = F.off[k];
                    int y = (yx >> 16) - (o >> 16), x = (yx & 65535) - ((o & 65535) - 32768);
                    if (L.pbc) { y = coord(y, ny); x = coord(x, nx); }
                    else if (y < 0 || y >= ny || x < 0 || x >= nx) continue;
                    const int n = y * nx + x, h = wolff_slot(F, n);
                    if (F.key[h] == n && F.layer[h] >= 0 && F.layer[h] < layer) count += F.w[k];
                }
                acc = !(u > wolff_bond_of(L, j, count));
            }
            const unsigned b = __ballot_sync(0xffffffffu, acc);
            if (acc) {
                const int k = lend + nacc + __popc(b & below);
                F.cell[k] = j;
                F.yx[k] = yx;
                F.layer[F.cand_slot[t]] = layer;
            }
            nacc += __popc(b);
        }
        call += 1;
        __syncwarp();
        lstart = lend;
        lend += nacc;
    }
    if (lane == 0) { F.lstart = lstart; F.lend = lend; F.layers = layer; F.grown = grown; F.call = call; }
    __syncwarp();
}

// One Wolff cluster step executed by one CTA. Small clusters (the rule above the critical
// temperature: two to three cells on a 300 x 300 lattice at J / kT = 0.24) grow on one warp in shared
// memory, where a layer costs no barrier and no global atomic; a larger one goes on from there with
// the whole CTA and the stamps in the scratch. Engine, 300 x 300 periodic: 15.2 -> 5.8 us per step,
// bound by the latencies of the chain (two Philox calls, two spin loads, the hash, per layer).
HS_DEV void wolff_step_cta(const HsLattice &L, HsCounters *C, const HsSwitchList &sw, const WolffScratch &S, WolffFast &F) {
    __shared__ int s_ncand, s_nacc[2], s_epoch;   // s_nacc: by layer parity, so a late reader never meets the next layer's reset
    if (C->done) return;
    if (!hs_progress_continue(C, L.n_occ)) {
        if (threadIdx.x == 0) { C->done = 1; C->n_sw = 0; }
        return;
    }
    const int nx = L.nx, ny = L.ny;
    const int64_t N = (int64_t)nx * ny;
    __syncthreads();   // every warp has tested the stop rule before warp 0 writes what it reads
    if (threadIdx.x < 32) {
        // seed: _select_single (np.random.randint(n) -> nonzero index)
        const uint64_t c = C->rng_call;
        const int seed = L.nonzero[(int)floor(hs_u53(L.seed, c, 0u) * L.n_occ)];
        wolff_grow_warp(L, F, seed, c + 1);
        if (F.grown) {
            // flip the cluster; counters as in core.py:714-716
            const int n = F.lend;
            for (int t = threadIdx.x; t < n; t += 32) {
                const int j = F.cell[t];
                L.m[j] = (int8_t)(-L.m[j]);
                L.mm[j] = -L.mm[j];
                if (t < sw.cap) { sw.y[t] = F.yx[t] >> 16; sw.x[t] = F.yx[t] & 65535; if (sw.mode) sw.mode[t] = 0; }
            }
            __syncwarp();
            if (threadIdx.x == 0) {
                C->attempted += n;
                C->switches += n;
                C->rng_call = F.call;
                C->n_sw = min(n, sw.cap);
                C->steps += 1;
                if (n > sw.cap) C->status |= HS_ST_SWITCH_OVERFLOW;
            }
        }
    }
    __syncthreads();
    if (F.grown) return;
    // larger: the state so far into the stamps
    if (threadIdx.x == 0) { s_epoch = *S.epoch + 1; *S.epoch = s_epoch; C->epoch = s_epoch; }
    __syncthreads();
    const int epoch = s_epoch;
    for (int h = threadIdx.x; h < WF_HASH; h += blockDim.x) {
        const int j = F.key[h];
        if (j < 0) continue;
        S.chk_ep[j] = epoch;
    }
    for (int t = threadIdx.x; t < F.lend; t += blockDim.x) { S.list[t] = F.cell[t]; S.cl_ep[F.cell[t]] = epoch; }
    const int8_t ms = L.m[F.cell[0]];
    uint64_t call = F.call;
    int lstart = F.lstart, lend = F.lend, layer = F.layers;
    const int ch = L.nn_h / 2, cw = L.nn_w / 2;
    __syncthreads();
    for (; layer <= (int)N + 1; ++layer) {
        if (threadIdx.x == 0) { s_ncand = 0; s_nacc[layer & 1] = 0; }
        __syncthreads();
        // frontier: unchecked same-spin cells j with q = j + c - b for a new cell q, mask[b] != 0; the
        // new cells are stamped here, so that no stamp changes while the bonds below read them
        for (int t = lstart + threadIdx.x; t < lend; t += blockDim.x) {
            const int q = S.list[t];
            S.cl_ep[q] = epoch;
            const int qy = q / nx, qx = q % nx;
            for (int a = 0; a < L.nn_h; ++a)
                for (int b = 0; b < L.nn_w; ++b) {
                    if (!L.nn[a * L.nn_w + b]) continue;
                    int jy = qy - ch + a, jx = qx - cw + b;
                    if (L.pbc) { jy = hs_wrap(jy, ny); jx = hs_wrap(jx, nx); }
                    else if (jy < 0 || jy >= ny || jx < 0 || jx >= nx) continue;
                    const int j = jy * nx + jx;
                    if (L.m[j] != ms) continue;
                    if (atomicExch(&S.chk_ep[j], epoch) == epoch) continue;
                    S.cand[atomicAdd(&s_ncand, 1)] = j;
                }
        }
        __syncthreads();
        const int ncand = s_ncand;
        if (ncand == 0) break;  // empty frontier: the reference's while-loop ends, no draw
        for (int t = threadIdx.x; t < ncand; t += blockDim.x) {
            const int j = S.cand[t];
            const int jy = j / nx, jx = j % nx;
            int count = 0;
            for (int a = 0; a < L.nn_h; ++a)
                for (int b = 0; b < L.nn_w; ++b) {
                    const int w = L.nn[a * L.nn_w + b];
                    if (!w) continue;
                    int yy = jy + ch - a, xx = jx + cw - b;
                    if (L.pbc) { yy = hs_wrap(yy, ny); xx = hs_wrap(xx, nx); }
                    else if (yy < 0 || yy >= ny || xx < 0 || xx >= nx) continue;
                    const int k = yy * nx + xx;
                    if (S.cl_ep[k] == epoch) count += w;
                }
            const double bond = wolff_bond_of(L, j, count);
            const double u = hs_u53(L.seed, call, (uint32_t)j);
            if (!(u > bond)) {
                S.list[lend + atomicAdd(&s_nacc[layer & 1], 1)] = j;
            }
        }
        call += 1;
        __syncthreads();
        lstart = lend;
        lend += s_nacc[layer & 1];
    }
    if (layer > (int)N + 1 && threadIdx.x == 0) C->status |= HS_ST_WOLFF_OVERFLOW;
    // flip the cluster; counters as in core.py:714-716
    for (int t = threadIdx.x; t < lend; t += blockDim.x) {
        const int j = S.list[t];
        L.m[j] = (int8_t)(-L.m[j]);
        L.mm[j] = -L.mm[j];
        if (t < sw.cap) { sw.y[t] = j / nx; sw.x[t] = j % nx; if (sw.mode) sw.mode[t] = 0; }
    }
    if (threadIdx.x == 0) {
        C->attempted += lend;
        C->switches += lend;
        C->rng_call = call;
        C->n_sw = min(lend, sw.cap);
        C->steps += 1;
        if (lend > sw.cap) C->status |= HS_ST_SWITCH_OVERFLOW;
    }
}

// ---- Néel -------------------------------------------------------------------------------
// Final stage of a Néel step once the global argmin `w` of the log-domain keys is known:
// switching time in FP64, flip, counters and the one-entry switch list
// (hotspice/core.py:699-709). Executed by a single thread.
// The flip a Néel decision made, for a caller that writes it itself (neel_finalize's `defer`).
struct NeelFlip { int64_t i; int y, x; int8_t m_new; float mm_new; bool flip; };
HS_DEV void neel_apply(const HsLattice &L, const HsSwitchList &sw, const NeelFlip &f) {
    L.m[f.i] = f.m_new;
    L.mm[f.i] = f.mm_new;
    sw.y[0] = f.y;
    sw.x[0] = f.x;
    if (sw.mode) sw.mode[0] = 0;
}

// `defer`: the flip (spin, moment, switch list) is returned there instead of being written.
HS_DEV void neel_finalize(const HsLattice &L, HsCounters *C, const HsSwitchList &sw, HsKeyIdx w, uint64_t call,
                          double bmin, bool unif, bool two, double attempt_freq, NeelFlip *defer = nullptr) {
    if (defer) defer->flip = false;
    C->rng_call = call + 1;
    C->attempted += 1;
    C->steps += 1;
    const double t_eff = C->progress ? (C->t_max - (C->t - C->t0)) : C->t_max;
    if (w.idx < 0) {  // no occupied cell: nanargmin would raise; record and stop
        C->status |= HS_ST_SELECT_RETRY;
        C->n_sw = 0;
        C->t += t_eff;
        return;
    }
    const int64_t i = w.idx;
    // the cell's spin and moment: carried by the scan's record, else loaded first, so that
    // their round trips overlap the switching-time arithmetic below
    const int8_t m_old = w.m ? (int8_t)w.m : L.m[i];
    const float mm_old = w.m ? w.mm : L.mm[i];
    const int y = (int)(i / L.nx), x = (int)(i % L.nx);
    // the barriers the scan computed for this cell (the same operations as hs_barriers)
    const double b1 = w.b1, b2 = w.b2;
    const double beta = hs_beta(L, i);
    const double e1 = hs_exp1_f64(hs_u53(L.seed, call, (uint32_t)i));
    double time;
    if (!two) {
        // time = E1 * exp((b - bmin) beta) * exp(bmin beta) / nu   (hotspice/core.py:698-700)
        time = unif ? e1 * exp(b1 * beta) / attempt_freq
                    : e1 * exp((b1 - bmin) * beta) * exp(bmin * beta) / attempt_freq;
    } else {
        const double bm = fmin(b1, b2), dd = fabs(b1 - b2);
        // tau = E1 / (exp(-(b1-bmin) beta) + exp(-(b2-bmin) beta)); nu halves (core.py:691-693)
        const double scale = exp((bm - bmin) * beta) / (1.0 + exp(-dd * beta));
        time = e1 * scale * exp(bmin * beta) / (attempt_freq / 2.0);
    }
    C->last_time = time;
    if (time > t_eff || isnan(time)) {
        C->t += t_eff;
        C->n_sw = 0;
        return;
    }
    const NeelFlip f{i, y, x, (int8_t)(-m_old), -mm_old, true};
    if (defer) *defer = f;
    else neel_apply(L, sw, f);
    C->switches += 1;
    C->t += time;
    C->n_sw = 1;
}

// Scratch layout of the Metropolis step (shared by the host launcher and the engine).
HS_HD inline int64_t hs_align_up_d(int64_t v, int64_t a) { return (v + a - 1) / a * a; }
HS_HD inline void hs_metro_sizes(const HsLattice &L, const HsGridPlan &P, int &cap, int &gsz) {
    cap = P.n_sc > 1 ? P.n_sc : 1;
    gsz = 0;
    if (P.sample_scheme == HS_SAMPLE_POISSON) {
        const double g = hs_poisson_grid_cells(L, P);
        gsz = g <= (double)HS_POISSON_GRID_MAX ? (int)g : HS_POISSON_GRID_MAX;   // validated by the entry points
        cap = cap > gsz ? cap : gsz;
    }
}

// Barriers of hotspice/core.py:625-656 from an already-loaded total energy E, perpendicular
// energy Ep (before m_perp_factor) and E_B.
// (V: HsLattice, or a copy of its fields use_perp, barrier_method and m_perp_factor.)
template <typename V>
HS_DEV void hs_barriers_from(const V &L, double E, double Ep, double EB, double &b1, double &b2) {
    const double dE = -2.0 * E;
    const double Ecur = E;             // -dE / 2, exactly
    if (!L.use_perp) {
        double b;
        if (L.barrier_method == HS_BARRIER_SIMPLE) {
            b = fmax(dE, EB - Ecur);
        } else {
            const double inv4 = 0.25 / EB;
            const double q = dE * inv4 + 1.0;
            b = (dE > 4.0 * EB) ? dE : fmin(EB * q * q, dE + 4.0 * EB);
        }
        b1 = b2 = b;
    } else {
        const double Ept = L.m_perp_factor * Ep;
        b1 = fmax(dE, (EB + Ept) - Ecur);
        b2 = fmax(dE, (EB - Ept) - Ecur);
    }
}

// Néel log-domain keys (see hs_neel.cu) of the occupied cells, folded into `best`. The work
// is the occupied cells start, start + stride, ... : taken from the occupied-cell list when the
// lattice is sparse (fewer than 3/4 of its cells hold a magnet), else all cells with an
// occupation test. The loads of NEEL_UNR cells are issued before any of them is used, so that
// one thread keeps several L2 round trips in flight. A cell whose key cannot beat the thread's
// best so far is skipped before the accurate logarithms: log E1 >= log u (E1 = -log(1 - u) >= u)
// and the two-channel term is >= -ln 2, so log u + (b_low - b_min) beta - ln 2 (less a margin
// for the fast logarithm) is a lower bound of the key. The (key, index) minimum does not depend
// on the visiting order or on the skipping (ties go to the smaller index; only cells whose key
// is strictly larger than a key already seen are skipped).
// Bounds of the engine's Néel path: per magnet s = b_low * beta (uniform beta), rounded down to
// float. They live in the Néel scratch at this offset and are valid only inside one engine launch
// (built at an instance's start, refreshed by the window update).
constexpr int64_t HS_NEEL_CACHE_OFFSET = 65536;
#ifndef HS_NEEL_UNROLL
#define HS_NEEL_UNROLL 3
#endif
constexpr int NEEL_UNR = HS_NEEL_UNROLL;
HS_DEV HsKeyIdx neel_scan_range(const HsLattice &L, int64_t start64, int64_t stride64, int64_t N64, uint64_t call,
                                double bmin, HsKeyIdx best) {
    const bool two = L.use_perp != 0;
    const bool sparse = 4 * (int64_t)L.n_occ < 3 * N64;
    const int M = sparse ? L.n_occ : (int)N64;     // cell indices fit in int (HsKeyIdx.idx)
    const int start = (int)start64, stride = (int)stride64;
    const double slack = (two ? 0.6931471805599453 : 0.0) + 1e-4;
    for (int base = start; base < M; base += stride * NEEL_UNR) {
        int ci[NEEL_UNR];
        int8_t oc[NEEL_UNR], mv[NEEL_UNR];
        double ed[NEEL_UNR], edp[NEEL_UNR];
        float zf[NEEL_UNR], zfp[NEEL_UNR], eb[NEEL_UNR], bt[NEEL_UNR];
#pragma unroll
        for (int k = 0; k < NEEL_UNR; ++k) {
            const int j = base + k * stride;
            const bool v = j < M;
            ci[k] = v ? (sparse ? __ldg(L.nonzero + j) : j) : 0;
        }
#pragma unroll
        for (int k = 0; k < NEEL_UNR; ++k) {
            const bool v = base + k * stride < M;
            const int i = ci[k];
            oc[k] = v ? (sparse ? (int8_t)1 : L.occ[i]) : (int8_t)0;
            mv[k] = v ? __ldcg(L.m + i) : (int8_t)0;
            ed[k] = (v && L.has_dipolar) ? __ldcg(L.E_dip + i) : 0.0;
            edp[k] = (v && L.has_dipolar && two) ? __ldcg(L.E_dip_perp + i) : 0.0;
            zf[k] = (v && L.zee) ? __ldg(L.zee + i) : 0.f;
            zfp[k] = (v && L.zee && two) ? __ldg(L.zee_perp + i) : 0.f;
            eb[k] = v ? __ldg(L.E_B + i) : 0.f;
            bt[k] = (v && L.beta_uniform <= 0.0) ? __ldg(L.beta + i) : 0.f;
        }
        // branch-free phases, so the NEEL_UNR Philox chains and barrier evaluations interleave
        double u[NEEL_UNR], lb[NEEL_UNR], b1v[NEEL_UNR], b2v[NEEL_UNR], btv[NEEL_UNR];
#pragma unroll
        for (int k = 0; k < NEEL_UNR; ++k) u[k] = hs_u53(L.seed, call, (uint32_t)ci[k]);
#pragma unroll
        for (int k = 0; k < NEEL_UNR; ++k) {
            double E = ed[k], Ep = edp[k];
            if (L.zee) { E += (double)mv[k] * (double)zf[k]; if (two) Ep += (double)mv[k] * (double)zfp[k]; }
            if (L.has_exchange) {
                double e, ep;
                hs_exchange_at(L, ci[k] / L.nx, ci[k] % L.nx, e, ep);
                E += e;
                if (two) Ep += ep;
            }
            hs_barriers_from(L, E, Ep, (double)eb[k], b1v[k], b2v[k]);
            btv[k] = L.beta_uniform > 0.0 ? L.beta_uniform : (double)bt[k];
            const double bm = two ? fmin(b1v[k], b2v[k]) : b1v[k];
            lb[k] = (double)__logf((float)u[k]) + (bm - bmin) * btv[k] - slack;
        }
#pragma unroll
        for (int k = 0; k < NEEL_UNR; ++k) {
            if (!oc[k]) continue;
            if (best.idx >= 0 && lb[k] > best.key) continue;
            const double b1 = b1v[k], b2 = b2v[k], beta = btv[k];
            const double le1 = (double)hs_log_exp1_f32(u[k]);
            double key;
            if (!two) key = le1 + (b1 - bmin) * beta;
            else {
                const double bm = fmin(b1, b2), dd = fabs(b1 - b2);
                key = le1 + (bm - bmin) * beta - (double)log1pf(expf((float)(-dd * beta)));
            }
            best = hs_kmin(best, HsKeyIdx{key, ci[k], b1, b2});
        }
    }
    return best;
}

// Per-warp queue of the engine's scan (shared memory): slots whose lower bound does not rule them out.
constexpr int NEEL_QCAP = 64;
