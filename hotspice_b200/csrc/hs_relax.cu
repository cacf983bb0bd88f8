// Relaxation to a (meta)stable state: Magnets._minimize_all / relax / minimize
// (hotspice/core.py:763-861).
//
// _minimize_all (one "sweep"): the lattice is cut into (2 ux) x (2 uy) interleaved subgrids
// (one subgrid when simultaneous), visited in a random order. In each subgrid every magnet
// whose switch lowers the energy (switch_energy < 0; or switch_energy / 2 + E_B < 0 when the
// barrier is not ignored) switches at once, and the energies are updated before the next
// subgrid is decided. On the device a sweep is:
//   relax_perm_kernel      the subgrid order: stable argsort of one Philox call of P variates
//   per subgrid i:
//     relax_decide_kernel  switch decisions (from E before any flip of this subgrid), a flag
//                          per candidate and a count per block
//     relax_apply_kernel   order-preserving compaction into the switch list, the flips, the
//                          counters; the list's truncated-window flag follows
//                          DipolarEnergy.update_multiple's per-sublattice rule
//     dip_update_kernel    (hs_dipolar.cu) consumes the list
// relax() adds, after every sweep, its stop rule: nothing switched, the state equals the one
// two sweeps before, or int(sqrt(nx^2 + ny^2)) sweeps (relax_compare_kernel, relax_end_kernel).
// Every kernel reads the control state from device memory and returns at once when the stop
// rule has fired, so the host can enqueue (or replay as a CUDA graph) several sweeps and look
// at the state once. relax() itself runs its sweeps in one cooperative launch instead
// (relax_grid_kernel): most subgrids of most sweeps switch a handful of magnets, and three
// launches each were almost all of their time.
//
// minimize() (sequential): per iteration the switch energy of every cell, the number n of
// magnets gaining more than kBT and the first argmin. If n > 0, ceil(0.3 n) of those n switch:
// the ones with the smallest Philox keys of one call over n elements (the stream's
// choice(n, k, replace=False)), found exactly by a 5-pass radix select on the 53-bit keys;
// else the argmin switches if it lowers the energy and was not picked three times.
#include "hs_common.cuh"
#include "hs_internal.h"
#include "hs_steps.cuh"

namespace {

constexpr int RX_T = 256;               // threads per block of the grid kernels
constexpr int RX_PER = 4;               // candidates per thread
constexpr int RX_CH = RX_T * RX_PER;    // candidates per block
constexpr int RX_MAX_P = 1024;          // subgrids per sweep (4 * 256 unit-cell sites)
constexpr int RX_MAX_U = 256;           // unit-cell sites
constexpr int RX_GAVE_UP = 2;           // RelaxState::done after a grid barrier that ran out of time
constexpr int MN_PASSES = 5;            // radix-select passes over the 53-bit keys
constexpr int MN_BINS = 2048;           // largest digit (11 bits)
__constant__ int c_mn_lo[MN_PASSES] = {42, 31, 20, 10, 0};
__constant__ int c_mn_bits[MN_PASSES] = {11, 11, 11, 10, 10};

struct RelaxState {
    int32_t done;       // stop rule fired (or RX_GAVE_UP): the remaining kernels of the sweep do nothing
    int32_t sweep;      // sweeps completed (relax)
    int32_t differs;    // the state after this sweep differs from the one two sweeps before
    int32_t pad0;
    int64_t sw_start;   // C->switches when the sweep began
    // minimize()
    int32_t mode;       // 0: stop, 1: the argmin switches, 2: ceil(frac n) of n switch
    int32_t count;      // n
    int32_t k;          // ceil(frac n)
    int32_t k_rem;      // radix select: how many keys equal to the threshold are taken
    int32_t eq_total;   // keys equal to the threshold
    int32_t imin;
    uint64_t prefix;    // radix select: threshold key bits found so far
    uint64_t call;      // Philox call of the choice
    double vmin;
};

struct RelaxBufs {
    RelaxState *st;
    int32_t *order;      // RX_MAX_P
    int32_t *blk;        // per-block counts
    int32_t *blk2;       // second per-block array (minimize: equal-key counts)
    double *blk_v;       // minimize: per-block minimum
    int32_t *blk_i;      //           and its index
    int32_t *sub_counts; // RX_MAX_U
    uint8_t *flags;      // N
    int8_t *snap;        // 2 N (relax) / visited N (minimize)
    int32_t *cells;      // N (minimize)
    int32_t *hist;       // MN_PASSES * MN_BINS (minimize)
};

HS_DEV uint64_t u53_bits(uint64_t seed, uint64_t call, uint32_t e) {
    HsU4 w = hs_philox(e, (uint32_t)call, (uint32_t)(call >> 32), 0u, (uint32_t)seed, (uint32_t)(seed >> 32));
    return ((uint64_t)(w.x >> 5) << 26) | (uint64_t)(w.y >> 6);
}

// Exclusive prefix of v over the block (RX_T threads) and the block total.
HS_DEV int block_scan(int v, int &total, int *s_w) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < RX_T / 32 ? s_w[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < RX_T / 32) s_w[lane] = w;   // inclusive warp prefix
    }
    __syncthreads();
    total = s_w[RX_T / 32 - 1];
    const int before = warp ? s_w[warp - 1] : 0;
    __syncthreads();
    return before + x - v;
}

HS_DEV int block_sum(int v, int *s_w) {
    int t;
    block_scan(v, t, s_w);
    return t;
}

HS_DEV double kbt_at(const HsLattice &L, int64_t i) {
    const double b = hs_beta(L, i);
    return 1.0 / b;     // beta = inf (T = 0) gives kBT = 0
}

// ---------------------------------------------------------------------------------------
// _minimize_all / relax
// ---------------------------------------------------------------------------------------
struct Subgrid {
    int y0, x0, nys, nxs, M;
    bool active;
};

HS_DEV Subgrid subgrid(const HsLattice &L, const RelaxBufs &B, int i, int sx, int sy) {
    Subgrid g;
    const int o = B.order[i];
    if (o < 0 || o >= sx * sy) {   // no order drawn for this layout: an empty subgrid
        g.y0 = g.x0 = g.nys = g.nxs = g.M = 0;
        g.active = false;
        return g;
    }
    g.y0 = o / sx;
    g.x0 = o % sx;
    g.active = L.occ[(int64_t)g.y0 * L.nx + g.x0] != 0;
    g.nys = (L.ny - g.y0 + sy - 1) / sy;
    g.nxs = (L.nx - g.x0 + sx - 1) / sx;
    g.M = g.nys * g.nxs;
    return g;
}

__global__ void __launch_bounds__(1024) relax_perm_kernel(HsLattice L, HsCounters *C, RelaxBufs B, int P) {
    __shared__ uint64_t s_key[RX_MAX_P];
    if (B.st->done) return;
    const uint64_t call = C->rng_call;
    for (int e = threadIdx.x; e < P; e += blockDim.x) s_key[e] = u53_bits(L.seed, call, (uint32_t)e);
    __syncthreads();
    for (int e = threadIdx.x; e < P; e += blockDim.x) {
        const uint64_t k = s_key[e];
        int rank = 0;
        for (int j = 0; j < P; ++j) rank += (s_key[j] < k) || (s_key[j] == k && j < e);
        B.order[rank] = e;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        C->rng_call = call + 1;
        B.st->sw_start = C->switches;
    }
}

__global__ void __launch_bounds__(RX_T) relax_decide_kernel(HsLattice L, RelaxBufs B, int i, int sx, int sy,
                                                            int ignore_barrier, int simultaneous) {
    __shared__ int s_w[RX_T / 32];
    if (B.st->done) return;
    const Subgrid g = subgrid(L, B, i, sx, sy);
    int cnt = 0;
#pragma unroll
    for (int k = 0; k < RX_PER; ++k) {
        const int t = blockIdx.x * RX_CH + k * RX_T + threadIdx.x;
        if (t >= g.M) continue;
        uint8_t f = 0;
        if (g.active) {
            const int y = g.y0 + (t / g.nxs) * sy, x = g.x0 + (t % g.nxs) * sx;
            double E, Ep;
            hs_energy_at(L, y, x, E, Ep);
            const double dE = -2.0 * E;
            f = ignore_barrier ? (dE < 0.0) : (dE / 2.0 + (double)L.E_B[(int64_t)y * L.nx + x] < 0.0);
            if (f && simultaneous) atomicAdd(&B.sub_counts[(y % L.uy) * L.ux + (x % L.ux)], 1);
        }
        B.flags[t] = f;
        cnt += f;
    }
    cnt = block_sum(cnt, s_w);
    if (threadIdx.x == 0) B.blk[blockIdx.x] = cnt;
}

__global__ void __launch_bounds__(RX_T) relax_apply_kernel(HsLattice L, HsCounters *C, RelaxBufs B, HsSwitchList sw,
                                                           int i, int sx, int sy, int simultaneous, int nblk) {
    __shared__ int s_w[RX_T / 32];
    if (B.st->done) {
        if (blockIdx.x == 0 && threadIdx.x == 0) C->n_sw = 0;
        return;
    }
    const Subgrid g = subgrid(L, B, i, sx, sy);
    // offset of this block and the subgrid total
    int before = 0, all = 0;
    for (int j = threadIdx.x; j < nblk; j += RX_T) {
        const int c = B.blk[j];
        all += c;
        if (j < (int)blockIdx.x) before += c;
    }
    before = block_sum(before, s_w);
    all = block_sum(all, s_w);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        C->n_sw = all;
        C->switches += all;
        C->attempted += all;
    }
    int pos = before;
#pragma unroll 1
    for (int k = 0; k < RX_PER; ++k) {
        const int t = blockIdx.x * RX_CH + k * RX_T + threadIdx.x;
        const int f = (t < g.M) ? B.flags[t] : 0;
        int tot;
        const int p = pos + block_scan(f, tot, s_w);
        if (f) {
            const int y = g.y0 + (t / g.nxs) * sy, x = g.x0 + (t % g.nxs) * sx;
            const int64_t c = (int64_t)y * L.nx + x;
            const int cnt = simultaneous ? B.sub_counts[(y % L.uy) * L.ux + (x % L.ux)] : all;
            sw.y[p] = y;
            sw.x[p] = x;
            if (sw.mode) sw.mode[p] = cnt > L.trunc_cutoff ? 1 : 0;
            L.m[c] = (int8_t)(-L.m[c]);
            L.mm[c] = -L.mm[c];
        }
        pos += tot;
    }
}

__global__ void __launch_bounds__(RX_T) relax_compare_kernel(HsLattice L, const HsCounters *C, RelaxBufs B) {
    __shared__ int s_w[RX_T / 32];
    if (B.st->done || C->switches == B.st->sw_start) return;
    const int64_t N = (int64_t)L.nx * L.ny;
    int8_t *snap = B.snap + ((B.st->sweep + 1) & 1) * N;
    int d = 0;
    for (int64_t c = (int64_t)blockIdx.x * RX_T + threadIdx.x; c < N; c += (int64_t)gridDim.x * RX_T) {
        const int8_t a = L.m[c];
        d |= a != snap[c];
        snap[c] = a;
    }
    d = block_sum(d, s_w);
    if (threadIdx.x == 0 && d) atomicOr(&B.st->differs, 1);
}

__global__ void relax_end_kernel(const HsCounters *C, RelaxBufs B, int n_max) {
    RelaxState *s = B.st;
    if (s->done) return;
    const int n = ++s->sweep;
    if (C->switches == s->sw_start) s->done = 1;       // nothing changed
    else if (!s->differs) s->done = 1;                 // 2-cycle
    else if (n >= n_max) s->done = 1;
    s->differs = 0;
}

// ---------------------------------------------------------------------------------------
// relax(): sweeps and stop rule in one cooperative launch
// ---------------------------------------------------------------------------------------
// The lattice is cut into tiles of TY rows x 32 sx columns, so that a row of a tile holds one
// 32-bit word of candidates of any subgrid; CTA b owns tiles b, b + grid, ... for the whole launch.
// Per subgrid:
//   decide   the owners' candidates, a ballot per word into the subgrid's bitmap, and the flips
//   barrier  with the number of switches (one grid barrier; with an exchange energy another one between decisions and flips,
//            since a decision may read a neighbour in another tile)
//   update   every cell of a tile with a switch in reach gathers their contributions straight
//            from the bitmap, rows and columns ascending: the order of the switch list, hence the
//            sums of dip_update_kernel bit for bit
// A subgrid without a switch costs one barrier, and bitmaps alternate, so no barrier separates a
// subgrid's update from the next one's decisions.
// Measured on B200: 512 x 512 pinwheel, cutoff 8.3a, about 190 sweeps: 59 ms (launched kernel by
// kernel) -> 14.5 ms. Bound: three quarters of the subgrids switch at most 20 magnets and take 11 K
// cycles, decisions 2.1 K, barrier 6 K (half of it waiting for the tile that holds a switch),
// update 2.5 K.
struct RelaxGrid {          // zeroed before every launch
    // grid barriers alternate between two words: arrivals in the low half, the sum of what the CTAs
    // brought along in the high half
    unsigned long long bar[2];
    int abort;              // a barrier gave up
};

struct RelaxPlan {
    int sx, sy, TX, TY, tiles_x, tiles, words, rows;   // words per bitmap row, rows of the largest subgrid
    int ignore_barrier, n_max, max_sweeps;
    unsigned poll_mask;                 // a waiting CTA looks at the time and at `abort` every poll_mask + 1 polls
    unsigned long long wait_ns;         // limit of one barrier
    unsigned *bits;         // [2][rows][words]
    RelaxGrid *g;
};

// Limit of a grid barrier: hs_set_wait_limit's when one is set, else 4 s more than the longest time
// between two barriers of one CTA. That time is bounded by the switches in reach of a warp's cells
// times the warp's parts; a switch takes a warp 0.3 us (512 x 512 pinwheel, 160 in reach: 96 K cycles
// for the update of a crowded subgrid), several times that with truncated periodic windows.
constexpr unsigned long long RX_WAIT_NS = 4000000000ULL;
constexpr double RX_SWITCH_NS = 4000.0;

// Grid barrier number `k` (0, 1, ...) of this launch, adding up every CTA's `v`: the sum of this
// barrier's, or -1 when it gave up (then on every CTA, sooner or later). `seen` keeps the two words'
// earlier sums. A CTA still polling a word never meets later arrivals: those of barrier k + 1 go to
// the other word, and those of k + 2 wait for it at k + 1.
HS_DEV int grid_barrier(const RelaxPlan &P, unsigned k, unsigned v, unsigned (&seen)[2]) {
    __shared__ int s_sum;
    RelaxGrid *const g = P.g;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long *word = &g->bar[k & 1];
        // release: the CTA's writes before the __syncthreads above come before the arrival
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(((unsigned long long)v << 32) | 1ull) : "memory");
        const unsigned want = ((k >> 1) + 1) * gridDim.x;
        const unsigned long long t0 = hs_globaltimer_ns();
        int sum = -1;
        for (unsigned it = 0;; ++it) {
            unsigned long long w;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(word) : "memory");
            if ((unsigned)w >= want) { sum = (int)((unsigned)(w >> 32) - seen[k & 1]); break; }
            if ((it & P.poll_mask) == P.poll_mask) {
                if (*(volatile int *)&g->abort) break;
                if (hs_globaltimer_ns() - t0 > P.wait_ns) { atomicExch(&g->abort, 1); break; }
            }
        }
        s_sum = sum;
    }
    __syncthreads();
    const int sum = s_sum;
    seen[k & 1] += (unsigned)sum;
    return sum;
}

// Cells a..b (inclusive) of an axis within `h` of coordinate v, ascending: one range, or two where
// they wrap.
struct Reach { int a[2], b[2], n; };
HS_DEV Reach reach_of(int v0, int v1, int h, bool wrap, int n) {
    Reach r;
    r.n = 1;
    if (!wrap) { r.a[0] = max(0, v0 - h); r.b[0] = min(n - 1, v1 + h); }
    else if (v1 - v0 + 2 * h + 1 >= n) { r.a[0] = 0; r.b[0] = n - 1; }
    else if (v0 - h < 0) { r.a[0] = 0; r.b[0] = v1 + h; r.a[1] = v0 - h + n; r.b[1] = n - 1; r.n = 2; }
    else if (v1 + h >= n) { r.a[0] = 0; r.b[0] = v1 + h - n; r.a[1] = v0 - h; r.b[1] = n - 1; r.n = 2; }
    else { r.a[0] = v0 - h; r.b[0] = v1 + h; }
    return r;
}
// Subgrid indices k (coordinate o + k s) in [a, b]: first and one past the last.
HS_DEV int first_at(int a, int o, int s) { return a <= o ? 0 : (a - o + s - 1) / s; }
HS_DEV int past_at(int b, int o, int s) { return b < o ? 0 : (b - o) / s + 1; }

struct SubUpdate {
    int y0, x0, sub, hy, hx, kind;      // kind 0: plain window, 1: minimum image, 2: hs_contrib (truncated, periodic)
    bool wrap, flip_perp;
    int mode;
    const unsigned *bits;
};

// The candidates in reach of a tile, staged row by row: rows [r0[p], r0[p] + nr[p]) of the subgrid,
// words [w0[q], w0[q] + nw[q]) of each, in ascending order.
constexpr int RX_WORDS = 512;            // staged bitmap words (and 32 times as many moments)
struct RelaxTile {
    Reach ry, rx;
    int r0[2], nr[2], w0[2], nw[2], rows, words;
    HS_DEV int row(int p, int r) const { return (p ? nr[0] : 0) + r - r0[p]; }
    HS_DEV int word(int q, int w) const { return (q ? nw[0] : 0) + w - w0[q]; }
};
constexpr int RX_LIST = 64;              // up to so many switches in reach of a tile go through a list
struct RelaxHit { int y, x; float mm; };
struct RelaxShared {
    unsigned bits[RX_WORDS];
    float mm[32 * RX_WORDS];             // moments of the staged candidates that switched
    RelaxHit hit[RX_LIST];
    int n;                               // switches in reach of the tile
};

// A warp's 32 columns x RX_V rows of a tile: their energies with the contributions of the switches in
// reach, in list order. The warp takes one switch at a time, so that a kernel row is read by
// consecutive lanes (with each lane on its own switches a crowded subgrid's update took 128 K
// cycles, now 96 K).
constexpr int RX_V = 8;
template <bool PERIODIC_CROP>      // kind 2
HS_DEV void relax_update_warp(const HsLattice &L, const RelaxPlan &P, const SubUpdate &u, const RelaxTile &T,
                              const RelaxShared &S, bool staged, int y, int x_base, int y_end, int x_end) {
    const int x = x_base + (threadIdx.x & 31);
    const int nyv = min(RX_V, y_end - y), nxw = min(32, x_end - x_base);
    const bool inx = x < x_end;
    float acc[RX_V] = {}, accp[RX_V] = {};
    unsigned touched = 0u, neg = 0u;     // bit v: row y + v
    const int KW = 2 * L.dip_wx + 1;
    const int64_t k0 = ((int64_t)max(u.sub, 0) * (2 * L.dip_wy + 1) + L.dip_wy) * KW + L.dip_wx;
    const float *K = L.K + k0, *Kp = L.use_perp ? L.Kpo + k0 : nullptr;
    const int kind = u.kind, hy = u.hy, hx = u.hx, nx = L.nx, ny = L.ny;
    const bool has = u.sub >= 0, two = has && Kp;
    auto apply = [&](int ys, int xs, float ms) {     // warp-uniform arguments
        if constexpr (PERIODIC_CROP) {
            if (!inx || !hs_axis_overlap(xs, hx, u.wrap, nx, x, 1)) return;
#pragma unroll
            for (int v = 0; v < RX_V; ++v) {
                if (v >= nyv || !hs_axis_overlap(ys, hy, u.wrap, ny, y + v, 1)) continue;
                touched |= 1u << v;
                if (ys == y + v && xs == x) neg |= 1u << v;
                if (has) hs_contrib(L, SwInfo{ys, xs, u.mode, u.sub, ms}, y + v, x, acc[v], accp[v]);
            }
            return;
        }
        else {
        int dx = x - xs;
        const bool own = dx == 0;
        if (kind == 1) dx = hs_minimage(dx, nx);
        const bool in = inx && dx >= -hx && dx <= hx;
        const float *Kx = K + dx, *Kpx = Kp + dx;
        float kv[RX_V], kp[RX_V];
#pragma unroll
        for (int v = 0; v < RX_V; ++v) {
            int dy = y + v - ys;
            if (own && dy == 0) neg |= 1u << v;
            if (kind == 1) dy = hs_minimage(dy, ny);
            const bool t = in && v < nyv && dy >= -hy && dy <= hy;
            if (t) touched |= 1u << v;
            kv[v] = t && has ? __ldg(Kx + dy * KW) : 0.f;
            kp[v] = t && two ? __ldg(Kpx + dy * KW) : 0.f;
        }
#pragma unroll
        for (int v = 0; v < RX_V; ++v) { acc[v] += ms * kv[v]; accp[v] += ms * kp[v]; }
        }
    };
    if (staged && S.n <= RX_LIST) {
        for (int h = 0; h < S.n; ++h) {
            const RelaxHit hit = S.hit[h];
            // does its window meet the warp's cells at all?
            if (!hs_axis_overlap(hit.y, hy, u.wrap, ny, y, nyv) || !hs_axis_overlap(hit.x, hx, u.wrap, nx, x_base, nxw)) continue;
            apply(hit.y, hit.x, hit.mm);
        }
    } else {
        const Reach ry = reach_of(y, y + nyv - 1, hy, u.wrap, ny), rx = reach_of(x_base, x_base + nxw - 1, hx, u.wrap, nx);
        int ca[2], cb[2];
        for (int q = 0; q < rx.n; ++q) { ca[q] = first_at(rx.a[q], u.x0, P.sx); cb[q] = past_at(rx.b[q], u.x0, P.sx); }
        for (int p = 0; p < ry.n; ++p) {
            const int r1 = past_at(ry.b[p], u.y0, P.sy);
            for (int r = first_at(ry.a[p], u.y0, P.sy); r < r1; ++r) {
                const int ys = u.y0 + r * P.sy;
                // the row's place in the tile's staging (a warp's range may lie in the tile's other one)
                const int tp = T.ry.n == 2 && r >= T.r0[1] ? 1 : 0;
                for (int q = 0; q < rx.n; ++q)
                    for (int w = ca[q] >> 5; 32 * w < cb[q]; ++w) {
                        const int tq = T.rx.n == 2 && w >= T.w0[1] ? 1 : 0;
                        const int at = staged ? T.row(tp, r) * T.words + T.word(tq, w) : 0;
                        unsigned b = staged ? S.bits[at] : __ldcg(u.bits + (int64_t)r * P.words + w);
                        if (32 * w < ca[q]) b &= 0xffffffffu << (ca[q] - 32 * w);
                        if (cb[q] - 32 * w < 32) b &= (1u << (cb[q] - 32 * w)) - 1u;
                        for (; b; b &= b - 1u) {
                            const int bit = __ffs(b) - 1, xs = u.x0 + (32 * w + bit) * P.sx;
                            apply(ys, xs, staged ? S.mm[32 * at + bit] : __ldcg(L.mm + (int64_t)ys * L.nx + xs));
                        }
                    }
            }
        }
    }
    if (!touched) return;
    const float pref2 = (float)(2.0 * L.dip_pref);
    const int64_t i0 = (int64_t)y * L.nx + x;
    float mv[RX_V];
    double ev[RX_V], pv[RX_V];
#pragma unroll
    for (int v = 0; v < RX_V; ++v) {
        const bool t = (touched >> v) & 1u;
        const int64_t i = i0 + (int64_t)v * nx;
        mv[v] = t ? L.mm[i] : 0.f;
        ev[v] = t ? L.E_dip[i] : 0.0;
        pv[v] = t && Kp ? L.E_dip_perp[i] : 0.0;
    }
#pragma unroll
    for (int v = 0; v < RX_V; ++v) {
        if (mv[v] == 0.f) continue;                  // not touched, or nothing is added to an empty cell
        const int64_t i = i0 + (int64_t)v * nx;
        if ((neg >> v) & 1u) { ev[v] = -ev[v]; if (u.flip_perp) pv[v] = -pv[v]; }
        L.E_dip[i] = ev[v] + (double)(pref2 * (mv[v] * acc[v]));
        if (Kp) L.E_dip_perp[i] = pv[v] + (double)(pref2 * (mv[v] * accp[v]));
    }
}

// Update of the tile of rows [ty0, ty1) and columns [tx0, tx1), by the whole CTA.
HS_DEV void relax_update_tile(const HsLattice &L, const RelaxPlan &P, const SubUpdate &u, RelaxShared &S, int ty0, int ty1,
                              int tx0, int tx1) {
    RelaxTile T;
    T.ry = reach_of(ty0, ty1 - 1, u.hy, u.wrap, L.ny);
    T.rx = reach_of(tx0, tx1 - 1, u.hx, u.wrap, L.nx);
    T.nr[1] = T.nw[1] = T.r0[1] = T.w0[1] = 0;
    for (int p = 0; p < T.ry.n; ++p) { T.r0[p] = first_at(T.ry.a[p], u.y0, P.sy); T.nr[p] = past_at(T.ry.b[p], u.y0, P.sy) - T.r0[p]; }
    for (int q = 0; q < T.rx.n; ++q) {
        T.w0[q] = first_at(T.rx.a[q], u.x0, P.sx) >> 5;
        T.nw[q] = ((past_at(T.rx.b[q], u.x0, P.sx) + 31) >> 5) - T.w0[q];
    }
    // wrapped ranges may share the word between them
    if (T.rx.n == 2 && T.w0[1] < T.w0[0] + T.nw[0]) { T.nw[1] -= T.w0[0] + T.nw[0] - T.w0[1]; T.w0[1] = T.w0[0] + T.nw[0]; }
    if (T.nw[1] < 0) T.nw[1] = 0;
    T.rows = T.nr[0] + T.nr[1];
    T.words = T.nw[0] + T.nw[1];
    const int n = T.rows * T.words;
    const bool staged = n <= RX_WORDS;
    unsigned any = 0u;
    for (int k = threadIdx.x; k < n; k += RX_T) {
        const int tr = k / T.words, tw = k - tr * T.words;
        const int r = tr < T.nr[0] ? T.r0[0] + tr : T.r0[1] + tr - T.nr[0];
        const int w = tw < T.nw[0] ? T.w0[0] + tw : T.w0[1] + tw - T.nw[0];
        const unsigned b = __ldcg(u.bits + (int64_t)r * P.words + w);
        any |= b;
        if (staged) S.bits[k] = b;
    }
    if (!__syncthreads_or(any != 0u)) return;      // no switch in reach
    if (staged) {
        auto place = [&](int k, int &r, int &w) {      // subgrid row and word of staged word k
            const int tr = k / T.words, tw = k - tr * T.words;
            r = tr < T.nr[0] ? T.r0[0] + tr : T.r0[1] + tr - T.nr[0];
            w = tw < T.nw[0] ? T.w0[0] + tw : T.w0[1] + tw - T.nw[0];
        };
        auto moment = [&](int r, int w, int bit) {
            return __ldcg(L.mm + (int64_t)(u.y0 + r * P.sy) * L.nx + u.x0 + (32 * w + bit) * P.sx);
        };
        if (threadIdx.x < 32) {       // the list, 32 words at a time, in order
            int at = 0;
            for (int k0 = 0; k0 < n; k0 += 32) {
                const int k = k0 + (int)threadIdx.x;
                unsigned b = k < n ? S.bits[k] : 0u;
                int incl = __popc(b);
                const int own = incl;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, incl, o); if ((int)threadIdx.x >= o) incl += t; }
                int pos = at + incl - own, r = 0, w = 0;
                if (b) place(k, r, w);
                for (; b && pos < RX_LIST; b &= b - 1u, ++pos) {
                    const int bit = __ffs(b) - 1;
                    S.hit[pos] = RelaxHit{u.y0 + r * P.sy, u.x0 + (32 * w + bit) * P.sx, moment(r, w, bit)};
                }
                at += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (threadIdx.x == 0) S.n = at;
        }
        __syncthreads();
        if (S.n > RX_LIST) {
            for (int k = threadIdx.x; k < 32 * n; k += RX_T) {     // moments of the switches
                if (!((S.bits[k >> 5] >> (k & 31)) & 1u)) continue;
                int r, w;
                place(k >> 5, r, w);
                S.mm[k] = moment(r, w, k & 31);
            }
            __syncthreads();
        }
    }
    const int gx = (tx1 - tx0 + 31) / 32, parts = gx * ((ty1 - ty0 + RX_V - 1) / RX_V);
    for (int e = threadIdx.x >> 5; e < parts; e += RX_T / 32) {
        const int y = ty0 + RX_V * (e / gx), x = tx0 + 32 * (e % gx);
        if (u.kind == 2) relax_update_warp<true>(L, P, u, T, S, staged, y, x, ty1, tx1);
        else relax_update_warp<false>(L, P, u, T, S, staged, y, x, ty1, tx1);
    }
    __syncthreads();       // the staging is free again; the next decisions read this CTA's energies
}

__global__ void __launch_bounds__(RX_T, 1) relax_grid_kernel(HsLattice L, HsCounters *C, RelaxBufs B, RelaxPlan P) {
    extern __shared__ __align__(16) unsigned char s_rx_raw[];
    RelaxShared &s_rx = *reinterpret_cast<RelaxShared *>(s_rx_raw);
    __shared__ uint64_t s_key[RX_MAX_P];
    __shared__ int s_order[RX_MAX_P];
    __shared__ unsigned char s_active[RX_MAX_P];
    __shared__ int s_w[RX_T / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_sub = P.sx * P.sy;
    for (int o = threadIdx.x; o < n_sub; o += RX_T) s_active[o] = L.occ[(int64_t)(o / P.sx) * L.nx + o % P.sx] != 0;
    const int64_t N = (int64_t)L.nx * L.ny;
    if (B.st->done) return;
    int sweep = B.st->sweep, done = 0;
    const uint64_t call0 = C->rng_call;
    long long switched = 0, sweep_total = 0;   // by this launch and by the sweep (every CTA counts)
    unsigned nbar = 0, slot = 0;         // barriers passed, subgrids so far
    unsigned seen[2] = {0u, 0u};
    int made = 0;
    bool ok = true;
    for (; made < P.max_sweeps && !done && ok; ++made) {
        // the subgrid order: a stable argsort of the sweep's variates
        for (int e = threadIdx.x; e < n_sub; e += RX_T) s_key[e] = u53_bits(L.seed, call0 + made, (uint32_t)e);
        __syncthreads();
        for (int e = threadIdx.x; e < n_sub; e += RX_T) {
            const uint64_t k = s_key[e];
            int rank = 0;
            for (int j = 0; j < n_sub; ++j) rank += (s_key[j] < k) || (s_key[j] == k && j < e);
            s_order[rank] = e;
        }
        __syncthreads();
        sweep_total = 0;
        for (int i = 0; i < n_sub && ok; ++i) {
            const int o = s_order[i];
            const int y0 = o / P.sx, x0 = o % P.sx;
            if (!s_active[o]) continue;
            unsigned *bits = P.bits + (int64_t)(slot & 1) * P.rows * P.words;
            // decisions: one word (32 candidates of a row) per warp
            int mine = 0;
            for (int t = blockIdx.x; t < P.tiles; t += gridDim.x) {
                const int ty0 = (t / P.tiles_x) * P.TY, w = t % P.tiles_x;
                const int r0 = first_at(ty0, y0, P.sy), r1 = past_at(min(ty0 + P.TY, L.ny) - 1, y0, P.sy);
                const int x = x0 + (32 * w + lane) * P.sx;
                if (w >= P.words) continue;
                for (int r = r0 + warp; r < r1; r += RX_T / 32) {
                    const int y = y0 + r * P.sy;
                    bool f = false;
                    if (x < L.nx) {
                        double E = 0.0, Ep;
                        if (L.has_exchange) hs_energy_at(L, y, x, E, Ep);
                        else {          // the operations of hs_energy_at on this CTA's own cells (through L1)
                            const int64_t c = (int64_t)y * L.nx + x;
                            if (L.has_dipolar) E += L.E_dip[c];
                            if (L.zee) E += (double)L.m[c] * (double)__ldg(L.zee + c);
                        }
                        const double dE = -2.0 * E;
                        f = P.ignore_barrier ? dE < 0.0 : dE / 2.0 + (double)L.E_B[(int64_t)y * L.nx + x] < 0.0;
                    }
                    const unsigned b = __ballot_sync(0xffffffffu, f);
                    if (lane == 0) bits[(int64_t)r * P.words + w] = b;
                    mine += __popc(b);
                    if (f && !L.has_exchange) {
                        const int64_t c = (int64_t)y * L.nx + x;
                        L.m[c] = (int8_t)(-L.m[c]);
                        L.mm[c] = -L.mm[c];
                    }
                }
            }
            mine = block_sum(lane == 0 ? mine : 0, s_w);
            const int all = grid_barrier(P, nbar++, (unsigned)mine, seen);
            ok = all >= 0;
            if (L.has_exchange && ok) {
                for (int t = blockIdx.x; t < P.tiles; t += gridDim.x) {
                    const int ty0 = (t / P.tiles_x) * P.TY, w = t % P.tiles_x;
                    const int r0 = first_at(ty0, y0, P.sy), r1 = past_at(min(ty0 + P.TY, L.ny) - 1, y0, P.sy);
                    if (w >= P.words) continue;
                    for (int r = r0 + warp; r < r1; r += RX_T / 32)
                        if ((bits[(int64_t)r * P.words + w] >> lane) & 1u) {
                            const int64_t c = (int64_t)(y0 + r * P.sy) * L.nx + x0 + (32 * w + lane) * P.sx;
                            L.m[c] = (int8_t)(-L.m[c]);
                            L.mm[c] = -L.mm[c];
                        }
                }
                ok = grid_barrier(P, nbar++, 0u, seen) >= 0;
            }
            if (!ok) break;
            sweep_total += all;
            if (all && L.has_dipolar) {
                SubUpdate u;
                u.y0 = y0; u.x0 = x0;
                u.sub = hs_sub(L, y0, x0);
                u.mode = all > L.trunc_cutoff ? 1 : 0;
                u.flip_perp = !(L.dip_keep_perp_sign && all > 1);
                u.bits = bits;
                int wy, wx;
                hs_window(L, u.mode, true, u.hy, wy);
                hs_window(L, u.mode, false, u.hx, wx);
                u.wrap = wy != 0;
                u.kind = u.wrap ? (u.mode ? 2 : 1) : 0;
                if (!u.wrap) { u.hy = min(u.hy, L.dip_wy); u.hx = min(u.hx, L.dip_wx); }   // the kernel ends there
                for (int t = blockIdx.x; t < P.tiles; t += gridDim.x) {
                    const int ty0 = (t / P.tiles_x) * P.TY, tx0 = (t % P.tiles_x) * P.TX;
                    const int ty1 = min(ty0 + P.TY, L.ny), tx1 = min(tx0 + P.TX, L.nx);
                    relax_update_tile(L, P, u, s_rx, ty0, ty1, tx0, tx1);
                }
            }
            ++slot;
        }
        switched += sweep_total;
        if (!ok) break;
        // the stop rule (relax_compare_kernel, relax_end_kernel)
        if (sweep_total == 0) { done = 1; ++sweep; continue; }
        int8_t *snap = B.snap + ((sweep + 1) & 1) * N;
        int d = 0;
        for (int t = blockIdx.x; t < P.tiles; t += gridDim.x) {
            const int ty0 = (t / P.tiles_x) * P.TY, tx0 = (t % P.tiles_x) * P.TX;
            const int ty1 = min(ty0 + P.TY, L.ny), tw = min(tx0 + P.TX, L.nx) - tx0, n = (ty1 - ty0) * tw;
            for (int e = threadIdx.x; e < n; e += RX_T) {
                const int64_t c = (int64_t)(ty0 + e / tw) * L.nx + tx0 + e % tw;
                const int8_t a = L.m[c];
                d |= a != snap[c];
                snap[c] = a;
            }
        }
        d = block_sum(d, s_w);
        const int differs = grid_barrier(P, nbar++, d ? 1u : 0u, seen);
        ok = differs >= 0;
        if (!ok) break;
        ++sweep;
        if (!differs || sweep >= P.n_max) done = 1;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        B.st->sweep = sweep;
        B.st->done = done;
        C->rng_call = call0 + made + (ok ? 0 : 1);
        C->switches += switched;
        C->attempted += switched;
        C->n_sw = 0;
        if (!ok) { C->status |= HS_ST_TIMEOUT; B.st->done = RX_GAVE_UP; }
    }
}

// ---------------------------------------------------------------------------------------
// minimize
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(RX_T) mn_scan_kernel(HsLattice L, RelaxBufs B) {
    __shared__ int s_w[RX_T / 32];
    __shared__ double s_v[RX_T];
    __shared__ int s_i[RX_T];
    if (B.st->done) return;
    const int64_t N = (int64_t)L.nx * L.ny;
    int cnt = 0;
    double vmin = INFINITY;
    int imin = INT32_MAX;
#pragma unroll
    for (int k = 0; k < RX_PER; ++k) {
        const int64_t c = (int64_t)blockIdx.x * RX_CH + k * RX_T + threadIdx.x;
        if (c >= N) continue;
        const int y = (int)(c / L.nx), x = (int)(c % L.nx);
        double E, Ep;
        hs_energy_at(L, y, x, E, Ep);
        const double dE = -2.0 * E;
        const uint8_t f = dE < -kbt_at(L, c);
        B.flags[c] = f;
        cnt += f;
        if (dE < vmin) { vmin = dE; imin = (int)c; }   // increasing c: first occurrence kept
    }
    cnt = block_sum(cnt, s_w);
    s_v[threadIdx.x] = vmin;
    s_i[threadIdx.x] = imin;
    __syncthreads();
    for (int o = RX_T / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            const double v2 = s_v[threadIdx.x + o];
            const int i2 = s_i[threadIdx.x + o];
            if (v2 < s_v[threadIdx.x] || (v2 == s_v[threadIdx.x] && i2 < s_i[threadIdx.x])) {
                s_v[threadIdx.x] = v2;
                s_i[threadIdx.x] = i2;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        B.blk[blockIdx.x] = cnt;
        B.blk_v[blockIdx.x] = s_v[0];
        B.blk_i[blockIdx.x] = s_i[0];
    }
}

__global__ void __launch_bounds__(1024) mn_decide_kernel(HsLattice L, HsCounters *C, RelaxBufs B, HsSwitchList sw,
                                                         int nblk, double frac) {
    __shared__ long long s_cnt[32];
    __shared__ double s_v[1024];
    __shared__ int s_i[1024];
    RelaxState *s = B.st;
    if (s->done) {   // the update that follows must see an empty list
        if (threadIdx.x == 0) C->n_sw = 0;
        return;
    }
    long long cnt = 0;
    double vmin = INFINITY;
    int imin = INT32_MAX;
    for (int j = threadIdx.x; j < nblk; j += blockDim.x) {
        cnt += B.blk[j];
        const double v = B.blk_v[j];
        const int ii = B.blk_i[j];
        if (v < vmin || (v == vmin && ii < imin)) { vmin = v; imin = ii; }
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) s_cnt[threadIdx.x >> 5] = cnt;
    s_v[threadIdx.x] = vmin;
    s_i[threadIdx.x] = imin;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            const double v2 = s_v[threadIdx.x + o];
            const int i2 = s_i[threadIdx.x + o];
            if (v2 < s_v[threadIdx.x] || (v2 == s_v[threadIdx.x] && i2 < s_i[threadIdx.x])) {
                s_v[threadIdx.x] = v2;
                s_i[threadIdx.x] = i2;
            }
        }
        __syncthreads();
    }
    // zero the radix-select histograms and the sublattice counts for this iteration
    for (int j = threadIdx.x; j < MN_PASSES * MN_BINS; j += blockDim.x) B.hist[j] = 0;
    for (int j = threadIdx.x; j < RX_MAX_U; j += blockDim.x) B.sub_counts[j] = 0;
    if (threadIdx.x != 0) return;
    long long total = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) total += s_cnt[w];
    s->vmin = s_v[0];
    s->imin = s_i[0];
    if (total > 0) {
        s->mode = 2;
        s->count = (int)total;
        s->k = (int)ceil((double)total * frac);
        s->k_rem = s->k;
        s->prefix = 0;
        s->call = C->rng_call;
        C->rng_call += 1;
        return;
    }
    s->mode = 0;
    C->n_sw = 0;
    const int c = s->imin;
    if (!(s->vmin < 0.0) || c == INT32_MAX) { s->done = 1; return; }   // no switch lowers the energy
    const int vis = ++B.snap[c];
    if (vis >= 3) { s->done = 1; return; }
    s->mode = 1;
    const int y = c / L.nx, x = c % L.nx;
    sw.y[0] = y;
    sw.x[0] = x;
    if (sw.mode) sw.mode[0] = 0;
    L.m[c] = (int8_t)(-L.m[c]);
    L.mm[c] = -L.mm[c];
    C->n_sw = 1;
    C->switches += 1;
    C->attempted += 1;
}

// Ordered list of the cells that gain more than kBT (row-major, as numpy.where gives them).
__global__ void __launch_bounds__(RX_T) mn_compact_kernel(HsLattice L, RelaxBufs B, int nblk) {
    __shared__ int s_w[RX_T / 32];
    if (B.st->done || B.st->mode != 2) return;
    const int64_t N = (int64_t)L.nx * L.ny;
    int before = 0;
    for (int j = threadIdx.x; j < (int)blockIdx.x; j += RX_T) before += B.blk[j];
    int pos = block_sum(before, s_w);
#pragma unroll 1
    for (int k = 0; k < RX_PER; ++k) {
        const int64_t c = (int64_t)blockIdx.x * RX_CH + k * RX_T + threadIdx.x;
        const int f = c < N ? B.flags[c] : 0;
        int tot;
        const int p = pos + block_scan(f, tot, s_w);
        if (f) B.cells[p] = (int)c;
        pos += tot;
    }
}

__global__ void __launch_bounds__(RX_T) mn_hist_kernel(HsLattice L, RelaxBufs B, int pass) {
    __shared__ int s_h[MN_BINS];
    const RelaxState *s = B.st;
    if (s->done || s->mode != 2) return;
    const int lo = c_mn_lo[pass], bits = c_mn_bits[pass];
    const int hi = lo + bits;
    for (int j = threadIdx.x; j < MN_BINS; j += RX_T) s_h[j] = 0;
    __syncthreads();
    const uint64_t prefix = s->prefix, call = s->call;
    const int n = s->count;
    for (int e = blockIdx.x * RX_T + threadIdx.x; e < n; e += gridDim.x * RX_T) {
        const uint64_t key = u53_bits(L.seed, call, (uint32_t)e);
        if ((key >> hi) == prefix) atomicAdd(&s_h[(key >> lo) & ((1u << bits) - 1u)], 1);
    }
    __syncthreads();
    int *g = B.hist + pass * MN_BINS;
    for (int j = threadIdx.x; j < (1 << bits); j += RX_T)
        if (s_h[j]) atomicAdd(&g[j], s_h[j]);
}

__global__ void __launch_bounds__(1024) mn_pick_kernel(RelaxBufs B, int pass) {
    __shared__ int s_c[1024];
    RelaxState *s = B.st;
    if (s->done || s->mode != 2) return;
    const int bits = c_mn_bits[pass];
    const int nb = 1 << bits;
    const int *h = B.hist + pass * MN_BINS;
    const int per = (nb + 1023) / 1024;
    int loc = 0;
    for (int j = 0; j < per; ++j) {
        const int b = threadIdx.x * per + j;
        if (b < nb) loc += h[b];
    }
    s_c[threadIdx.x] = loc;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {      // inclusive scan (Hillis-Steele)
        const int v = (int)threadIdx.x >= o ? s_c[threadIdx.x - o] : 0;
        __syncthreads();
        s_c[threadIdx.x] += v;
        __syncthreads();
    }
    const int k = s->k_rem;
    int cum = threadIdx.x ? s_c[threadIdx.x - 1] : 0;
    if (cum < k && k <= s_c[threadIdx.x]) {   // exactly one thread holds the crossing bin
        for (int j = 0; j < per; ++j) {
            const int b = threadIdx.x * per + j;
            if (b >= nb) break;
            if (cum + h[b] >= k) {
                s->prefix = (s->prefix << bits) | (uint64_t)b;
                s->k_rem = k - cum;
                s->eq_total = h[b];
                break;
            }
            cum += h[b];
        }
    }
}

// Per block: keys below the threshold and keys equal to it.
__global__ void __launch_bounds__(RX_T) mn_select_count_kernel(HsLattice L, RelaxBufs B) {
    __shared__ int s_w[RX_T / 32];
    const RelaxState *s = B.st;
    if (s->done || s->mode != 2) return;
    const uint64_t T = s->prefix, call = s->call;
    const int n = s->count;
    int lt = 0, eq = 0;
#pragma unroll
    for (int k = 0; k < RX_PER; ++k) {
        const int e = blockIdx.x * RX_CH + k * RX_T + threadIdx.x;
        if (e >= n) continue;
        const uint64_t key = u53_bits(L.seed, call, (uint32_t)e);
        lt += key < T;
        eq += key == T;
    }
    lt = block_sum(lt, s_w);
    eq = block_sum(eq, s_w);
    if (threadIdx.x == 0) { B.blk[blockIdx.x] = lt; B.blk2[blockIdx.x] = eq; }
}

// The k chosen cells in list order: every key below the threshold and the first k_rem keys
// equal to it; flips, counters, sublattice counts.
__global__ void __launch_bounds__(RX_T) mn_select_write_kernel(HsLattice L, HsCounters *C, RelaxBufs B,
                                                               HsSwitchList sw) {
    __shared__ int s_w[RX_T / 32];
    __shared__ int s_base[2];
    const RelaxState *s = B.st;
    if (s->done || s->mode != 2) return;
    const uint64_t T = s->prefix, call = s->call;
    const int n = s->count, k_rem = s->k_rem;
    // taken / equal keys in the blocks before this one (a scan over the block counts)
    int taken = 0, eq_run = 0;
    for (int j0 = 0; j0 < (int)blockIdx.x; j0 += RX_T) {
        const int j = j0 + threadIdx.x;
        const int e_here = j < (int)blockIdx.x ? B.blk2[j] : 0;
        int e_tot;
        const int eq_before = eq_run + block_scan(e_here, e_tot, s_w);
        const int t_here = j < (int)blockIdx.x ? B.blk[j] + max(0, min(e_here, k_rem - eq_before)) : 0;
        taken += block_sum(t_here, s_w);
        eq_run += e_tot;
    }
    if (threadIdx.x == 0) {
        s_base[0] = taken;
        s_base[1] = eq_run;
        if (blockIdx.x == 0) {
            C->n_sw = s->k;
            C->switches += s->k;
            C->attempted += s->k;
        }
    }
    __syncthreads();
    int pos = s_base[0], eqb = s_base[1];
#pragma unroll 1
    for (int k = 0; k < RX_PER; ++k) {
        const int e = blockIdx.x * RX_CH + k * RX_T + threadIdx.x;
        uint64_t key = ~0ull;
        if (e < n) key = u53_bits(L.seed, call, (uint32_t)e);
        const int is_eq = e < n && key == T;
        int eq_tot;
        const int eq_rank = eqb + block_scan(is_eq, eq_tot, s_w);
        const int take = e < n && (key < T || (is_eq && eq_rank < k_rem));
        int tot;
        const int p = pos + block_scan(take, tot, s_w);
        if (take) {
            const int c = B.cells[e];
            const int y = c / L.nx, x = c % L.nx;
            sw.y[p] = y;
            sw.x[p] = x;
            L.m[c] = (int8_t)(-L.m[c]);
            L.mm[c] = -L.mm[c];
            atomicAdd(&B.sub_counts[(y % L.uy) * L.ux + (x % L.ux)], 1);
        }
        pos += tot;
        eqb += eq_tot;
    }
}

__global__ void __launch_bounds__(RX_T) mn_mode_kernel(HsLattice L, const HsCounters *C, RelaxBufs B, HsSwitchList sw) {
    const RelaxState *s = B.st;
    if (s->done || s->mode != 2 || !sw.mode) return;
    const int n = C->n_sw;
    for (int j = blockIdx.x * RX_T + threadIdx.x; j < n; j += gridDim.x * RX_T) {
        const int y = sw.y[j], x = sw.x[j];
        sw.mode[j] = B.sub_counts[(y % L.uy) * L.ux + (x % L.ux)] > L.trunc_cutoff ? 1 : 0;
    }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
int64_t n_cells(const HsLattice &L) { return (int64_t)L.nx * L.ny; }
int grid_blocks(const HsLattice &L) { return (int)((n_cells(L) + RX_CH - 1) / RX_CH); }

// One layout serves relax and minimize.
int64_t layout(const HsLattice &L, char *base, RelaxBufs *B) {
    const int64_t N = n_cells(L), nb = grid_blocks(L);
    int64_t off = 0;
    auto take = [&](int64_t bytes) { char *p = base ? base + off : nullptr; off += hs_align_up(bytes, 256); return p; };
    RelaxBufs b;
    b.st = reinterpret_cast<RelaxState *>(take(sizeof(RelaxState)));
    b.order = reinterpret_cast<int32_t *>(take(4LL * RX_MAX_P));
    b.blk = reinterpret_cast<int32_t *>(take(4 * nb));
    b.blk2 = reinterpret_cast<int32_t *>(take(4 * nb));
    b.blk_v = reinterpret_cast<double *>(take(8 * nb));
    b.blk_i = reinterpret_cast<int32_t *>(take(4 * nb));
    b.sub_counts = reinterpret_cast<int32_t *>(take(4LL * RX_MAX_U));
    b.flags = reinterpret_cast<uint8_t *>(take(N));
    b.snap = reinterpret_cast<int8_t *>(take(2 * N));
    b.cells = reinterpret_cast<int32_t *>(take(4 * N));
    b.hist = reinterpret_cast<int32_t *>(take(4LL * MN_PASSES * MN_BINS));
    if (B) *B = b;
    return off;
}

int check_common(const HsLattice &L, const char *who, int64_t bytes) {
    if (L.nx <= 0 || L.ny <= 0 || !L.m || !L.mm || !L.occ) { hs_set_error("%s: empty lattice", who); return HS_EINVAL; }
    if (L.ux * L.uy > RX_MAX_U) { hs_set_error("%s: unit cell larger than %d sites", who, RX_MAX_U); return HS_ERANGE; }
    if (n_cells(L) > (int64_t)INT32_MAX / 2) { hs_set_error("%s: lattice too large", who); return HS_ERANGE; }
    if (bytes < layout(L, nullptr, nullptr)) {
        hs_set_error("%s: scratch %lld < %lld bytes", who, (long long)bytes, (long long)layout(L, nullptr, nullptr));
        return HS_ENOMEM;
    }
    return HS_OK;
}

void steps_of(const HsLattice &L, int simultaneous, int &sx, int &sy) {
    sx = simultaneous ? 1 : 2 * L.ux;
    sy = simultaneous ? 1 : 2 * L.uy;
}

}  // namespace

int64_t hs_relax_scratch(const HsLattice &L) { return layout(L, nullptr, nullptr); }

int hs_relax_begin_impl(const HsLattice &L, void *scratch, int64_t bytes, cudaStream_t st) {
    int rc = check_common(L, "hs_relax_begin", bytes);
    if (rc) return rc;
    RelaxBufs B;
    layout(L, reinterpret_cast<char *>(scratch), &B);
    const int64_t N = n_cells(L);
    if (cudaMemsetAsync(B.st, 0, sizeof(RelaxState), st) != cudaSuccess ||
        cudaMemsetAsync(B.order, 0xff, 4 * RX_MAX_P, st) != cudaSuccess ||                // no order yet
        cudaMemcpyAsync(B.snap, L.m, N, cudaMemcpyDeviceToDevice, st) != cudaSuccess ||   // two sweeps back: m0
        cudaMemsetAsync(B.snap + N, 0, N, st) != cudaSuccess) {                            // before it: zeros
        hs_set_error("hs_relax_begin: %s", cudaGetErrorString(cudaGetLastError()));
        return HS_ECUDA;
    }
    return HS_OK;
}

int hs_relax_permute_impl(const HsLattice &L, HsCounters *C, int simultaneous, void *scratch, int64_t bytes,
                          cudaStream_t st) {
    int rc = check_common(L, "hs_relax_permute", bytes);
    if (rc) return rc;
    RelaxBufs B;
    layout(L, reinterpret_cast<char *>(scratch), &B);
    int sx, sy;
    steps_of(L, simultaneous, sx, sy);
    if (sx > L.nx || sy > L.ny) { hs_set_error("hs_relax_permute: lattice smaller than two unit cells"); return HS_EINVAL; }
    relax_perm_kernel<<<1, 1024, 0, st>>>(L, C, B, sx * sy);
    return hs_check_launch("relax_perm_kernel");
}

int hs_relax_subset_impl(const HsLattice &L, HsCounters *C, const HsSwitchList &sw, int i, int ignore_barrier,
                         int simultaneous, void *scratch, int64_t bytes, cudaStream_t st) {
    int rc = check_common(L, "hs_relax_subset", bytes);
    if (rc) return rc;
    RelaxBufs B;
    layout(L, reinterpret_cast<char *>(scratch), &B);
    int sx, sy;
    steps_of(L, simultaneous, sx, sy);
    if (sx > L.nx || sy > L.ny) { hs_set_error("hs_relax_subset: lattice smaller than two unit cells"); return HS_EINVAL; }
    if (i < 0 || i >= sx * sy) { hs_set_error("hs_relax_subset: subgrid %d of %d", i, sx * sy); return HS_EINVAL; }
    const int64_t Mmax = (int64_t)((L.ny + sy - 1) / sy) * ((L.nx + sx - 1) / sx);
    if (sw.cap < Mmax) { hs_set_error("hs_relax_subset: switch list capacity %d < %lld", sw.cap, (long long)Mmax); return HS_EINVAL; }
    const int nblk = (int)((Mmax + RX_CH - 1) / RX_CH);
    if (simultaneous && cudaMemsetAsync(B.sub_counts, 0, 4 * RX_MAX_U, st) != cudaSuccess) {
        hs_set_error("hs_relax_subset: memset failed");
        return HS_ECUDA;
    }
    relax_decide_kernel<<<nblk, RX_T, 0, st>>>(L, B, i, sx, sy, ignore_barrier, simultaneous);
    if ((rc = hs_check_launch("relax_decide_kernel"))) return rc;
    relax_apply_kernel<<<nblk, RX_T, 0, st>>>(L, C, B, sw, i, sx, sy, simultaneous, nblk);
    if ((rc = hs_check_launch("relax_apply_kernel"))) return rc;
    if (L.has_dipolar) return hs_launch_dipolar_update(L, sw, &C->n_sw, 0, HS_UPDATE_MULTIPLE, C, st);
    return HS_OK;
}

int hs_relax_check_impl(const HsLattice &L, HsCounters *C, int n_max, void *scratch, int64_t bytes, cudaStream_t st) {
    int rc = check_common(L, "hs_relax_check", bytes);
    if (rc) return rc;
    RelaxBufs B;
    layout(L, reinterpret_cast<char *>(scratch), &B);
    const int nb = std::min(grid_blocks(L) * RX_PER, 148 * 8);
    relax_compare_kernel<<<nb, RX_T, 0, st>>>(L, C, B);
    if ((rc = hs_check_launch("relax_compare_kernel"))) return rc;
    relax_end_kernel<<<1, 1, 0, st>>>(C, B, n_max);
    return hs_check_launch("relax_end_kernel");
}

int hs_relax_run_impl(const HsLattice &L, HsCounters *C, int ignore_barrier, int n_max, int max_sweeps, void *scratch,
                      int64_t bytes, cudaStream_t st) {
    int rc = check_common(L, "hs_relax_run", bytes);
    if (rc) return rc;
    RelaxBufs B;
    layout(L, reinterpret_cast<char *>(scratch), &B);
    RelaxPlan P{};
    steps_of(L, 0, P.sx, P.sy);
    if (P.sx > L.nx || P.sy > L.ny) { hs_set_error("hs_relax_run: lattice smaller than two unit cells"); return HS_EINVAL; }
    int dev = 0, sms = 148, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = cudaFuncSetAttribute(relax_grid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RelaxShared));
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, relax_grid_kernel, RX_T, sizeof(RelaxShared));
    if (e != cudaSuccess) { hs_set_error("hs_relax_run: %s", cudaGetErrorString(e)); return HS_ECUDA; }
    P.TX = 32 * P.sx;
    P.tiles_x = (L.nx + P.TX - 1) / P.TX;
    // the shortest tiles that still give every SM at most one: a barrier costs less with fewer CTAs
    P.TY = P.sy;
    while ((int64_t)P.tiles_x * ((L.ny + P.TY - 1) / P.TY) > sms && P.TY < 64) P.TY += P.sy;
    P.tiles = P.tiles_x * ((L.ny + P.TY - 1) / P.TY);
    P.rows = (L.ny + P.sy - 1) / P.sy;
    P.words = ((L.nx + P.sx - 1) / P.sx + 31) / 32;
    P.ignore_barrier = ignore_barrier;
    P.n_max = n_max;
    P.max_sweeps = max_sweeps;
    const unsigned long long limit = hs_wait_limit_impl();
    P.wait_ns = limit;
    P.poll_mask = limit && limit < 1000000ULL ? 0u : 255u;
    P.bits = reinterpret_cast<unsigned *>(B.cells);       // at most 4 N bytes: minimize()'s list
    P.g = reinterpret_cast<RelaxGrid *>(B.hist);
    static_assert(sizeof(RelaxGrid) <= 4 * MN_PASSES * MN_BINS, "the grid state lives in minimize()'s histograms");
    if (8LL * P.rows * P.words > 4 * n_cells(L)) { hs_set_error("hs_relax_run: bitmap larger than its buffer"); return HS_ERANGE; }
    e = cudaMemsetAsync(P.g, 0, sizeof(RelaxGrid), st);
    if (e != cudaSuccess) { hs_set_error("hs_relax_run: %s", cudaGetErrorString(e)); return HS_ECUDA; }
    HsLattice Lv = L;
    void *args[] = {&Lv, &C, &B, &P};
    const int grid = std::max(1, std::min(P.tiles, sms * std::max(per, 1)));
    if (!limit) {
        const int hy = L.trunc_size ? std::max(L.dip_wy, std::min(L.trunc_size, L.ny - 1)) : L.ny - 1;
        const int hx = L.trunc_size ? std::max(L.dip_wx, std::min(L.trunc_size, L.nx - 1)) : L.nx - 1;
        const double reach = (std::min(L.ny, 2 * hy + RX_V) / P.sy + 1.0) * (std::min(L.nx, 2 * hx + 32) / P.sx + 1.0);
        const double parts = std::ceil(P.sx * std::ceil((double)P.TY / RX_V) / (RX_T / 32)) * ((P.tiles + grid - 1) / grid);
        P.wait_ns = RX_WAIT_NS + (unsigned long long)(reach * parts * RX_SWITCH_NS);
    }
    e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(relax_grid_kernel), dim3(grid), dim3(RX_T), args,
                                    sizeof(RelaxShared), st);
    if (e != cudaSuccess) { hs_set_error("relax_grid_kernel: %s", cudaGetErrorString(e)); return HS_ECUDA; }
    return hs_check_launch("relax_grid_kernel");
}

int hs_minimize_begin_impl(const HsLattice &L, void *scratch, int64_t bytes, cudaStream_t st) {
    int rc = check_common(L, "hs_minimize_begin", bytes);
    if (rc) return rc;
    RelaxBufs B;
    layout(L, reinterpret_cast<char *>(scratch), &B);
    if (cudaMemsetAsync(B.st, 0, sizeof(RelaxState), st) != cudaSuccess ||
        cudaMemsetAsync(B.snap, 0, n_cells(L), st) != cudaSuccess) {   // visited counts
        hs_set_error("hs_minimize_begin: memset failed");
        return HS_ECUDA;
    }
    return HS_OK;
}

int hs_minimize_step_impl(const HsLattice &L, HsCounters *C, const HsSwitchList &sw, double frac, void *scratch,
                          int64_t bytes, cudaStream_t st) {
    int rc = check_common(L, "hs_minimize_step", bytes);
    if (rc) return rc;
    if (!(frac > 0.0 && frac <= 1.0)) { hs_set_error("hs_minimize_step: frac must lie in (0, 1]"); return HS_EINVAL; }
    if (sw.cap < n_cells(L)) { hs_set_error("hs_minimize_step: switch list capacity %d < nx*ny", sw.cap); return HS_EINVAL; }
    RelaxBufs B;
    layout(L, reinterpret_cast<char *>(scratch), &B);
    const int nblk = grid_blocks(L);
    const int nh = std::min(nblk * RX_PER, 148 * 8);
    mn_scan_kernel<<<nblk, RX_T, 0, st>>>(L, B);
    if ((rc = hs_check_launch("mn_scan_kernel"))) return rc;
    mn_decide_kernel<<<1, 1024, 0, st>>>(L, C, B, sw, nblk, frac);
    if ((rc = hs_check_launch("mn_decide_kernel"))) return rc;
    mn_compact_kernel<<<nblk, RX_T, 0, st>>>(L, B, nblk);
    if ((rc = hs_check_launch("mn_compact_kernel"))) return rc;
    for (int p = 0; p < MN_PASSES; ++p) {
        mn_hist_kernel<<<nh, RX_T, 0, st>>>(L, B, p);
        if ((rc = hs_check_launch("mn_hist_kernel"))) return rc;
        mn_pick_kernel<<<1, 1024, 0, st>>>(B, p);
        if ((rc = hs_check_launch("mn_pick_kernel"))) return rc;
    }
    mn_select_count_kernel<<<nblk, RX_T, 0, st>>>(L, B);
    if ((rc = hs_check_launch("mn_select_count_kernel"))) return rc;
    mn_select_write_kernel<<<nblk, RX_T, 0, st>>>(L, C, B, sw);
    if ((rc = hs_check_launch("mn_select_write_kernel"))) return rc;
    mn_mode_kernel<<<std::min(nblk, 148), RX_T, 0, st>>>(L, C, B, sw);
    if ((rc = hs_check_launch("mn_mode_kernel"))) return rc;
    if (L.has_dipolar) return hs_launch_dipolar_update(L, sw, &C->n_sw, 0, HS_UPDATE_MULTIPLE, C, st);
    return HS_OK;
}
