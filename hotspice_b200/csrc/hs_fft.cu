// (b) Full dipolar recompute as a fast convolution in FP64 (hotspice/energies.py:290-308).
//
//   out_s[y, x] = sum_{dy, dx} K_s[dy, dx] mm[y + dy, x + dx]
//
// is a correlation of the source field with each sublattice's window, so it costs three passes of
// short transforms instead of one product per pair. All of it is FP64 from the FP32 kernels and
// source field, as in the direct sum; the result differs from the direct sum's by FP64 rounding of the
// largest sum the sources could give, about 2^-52 max|K| max|m mu| sqrt(magnets), where the direct
// sum rounds relative to each cell's own terms. For two lone magnets 720 cells apart that is 1.5e-9 of
// their energy, 2047 cells apart (2048 x 2 cells) 8e-7; the FP32 kernel values are off by 6e-8.
//   fft_rows_kernel   transforms along x of the source rows and of every kernel row (reversed, so
//                     that the correlation becomes a convolution)
//   fft_cols_kernel   per column of the spectrum: transforms along y of the source and of each
//                     kernel, their product, and the transform back
//   fft_cells_kernel  per lattice row: the transform back along x, the cells' energies
// Both energy channels of a kernel share one complex transform (K + i K_perp-self: the source is
// real); with one channel two sublattices share it.
//
// Lengths: M = 2^a times 1, 3, 5 or 9, at least n + w (outputs 0..n-1 only see offsets up to
// w, so the zeros of [n, M) serve both ends), or n + 2w with minimum-image wrapping, where the
// source is extended by its periodic images instead. Transforms run in shared memory, in place:
// the forward ones from natural to digit-reversed order (decimation in frequency), the backward
// ones from digit-reversed to natural (decimation in time), so nothing is ever reordered: every
// spectrum has the same order. A backward transform is the forward arithmetic on numbers with
// their parts swapped.
//
// Measured on B200: 96 x 96 square lattice, uncut, 1453 (direct sum) -> 25 us; 640 x 571 pinwheel,
// two channels, 210 ms -> 151 us (rows 41, columns 87, cells 23). Bound: latency and shared memory
// (a first form that took every stage from shared memory to shared memory with computed twiddle
// indices needed 303 us, at 8% of the FP64 pipe and an IPC of 1.1 to 1.4). 128 registers hold a
// radix-16 butterfly, so an SM has 16 warps.
#include "hs_common.cuh"
#include "hs_full.cuh"
#include "hs_internal.h"

namespace {

constexpr int FFT_T = 256;            // threads per CTA
constexpr int FFT_MIN_CTAS = 2;       // per SM: 128 registers a thread hold a radix-16 butterfly
constexpr int FFT_MAX_STAGES = 8;
constexpr int FFT_MAX_M = 4096;       // two lines and a twiddle table in shared memory
constexpr int FFT_HAS = 1024;         // (slot, row phase) flags kept in shared memory
constexpr int FFT_ROW_CTAS = 148 * FFT_MIN_CTAS;   // of the row pass: each builds the twiddle table once

struct FftAxis {                      // one transform length
    int M, n_stages;
    int radix[FFT_MAX_STAGES];        // in decimation-in-frequency order, odd radices first
    int toff[FFT_MAX_STAGES];         // each stage's twiddles in the table
    int tlen;                         // entries of the table
    int lg;                           // log2 of the last radix: one element of padding per 2^lg
    int Mp;                           // line pitch in shared memory
};

struct FftStat { unsigned kmax, mmax; int count, pad; };   // bits of max |K|, of max |mm|; non-zero sources

struct FftParams {
    FftAxis X, Y;
    int nys, nxs;                     // source rows and columns, halo included
    int oy, ox;                       // halo: outputs start at (oy, ox)
    int KH, KW;                       // window
    int n_slots, slot_rows;           // complex kernels; rows of scratch per slot
    int two;                          // both channels
    int n_lines;                      // lines of the row pass
    int stat_blocks;
    double2 *spec;                    // [nys + n_slots slot_rows][X.M]
    double2 *twx, *twy;               // twiddle tables (fft_twiddles)
    FftStat *stat;
    double *E, *Ep;
};

HS_DEV double2 cmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
HS_DEV double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
HS_DEV double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
HS_DEV double2 cswap(double2 a) { return make_double2(a.y, a.x); }
HS_DEV double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }     // -i a

// Forward transforms of R values, natural order in and out.
template <int R> struct Dft;
template <> struct Dft<3> {
    HS_DEV static void run(double2 *v) {
        const double s = 0.86602540378443864676;   // sin(2 pi / 3)
        const double2 t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
        const double2 m = make_double2(v[0].x - 0.5 * t.x, v[0].y - 0.5 * t.y);
        v[0] = cadd(v[0], t);
        v[1] = make_double2(m.x + s * d.y, m.y - s * d.x);
        v[2] = make_double2(m.x - s * d.y, m.y + s * d.x);
    }
};
template <> struct Dft<4> {
    HS_DEV static void run(double2 *v) {
        const double2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = mul_mi(csub(v[1], v[3]));
        v[0] = cadd(a, c); v[1] = cadd(b, d); v[2] = csub(a, c); v[3] = csub(b, d);
    }
};
template <> struct Dft<5> {
    HS_DEV static void run(double2 *v) {
        const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;   // cos(2 pi / 5), cos(4 pi / 5)
        const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;    // sin(2 pi / 5), sin(4 pi / 5)
        const double2 a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]), a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
        const double2 p = make_double2(v[0].x + c1 * a1.x + c2 * a2.x, v[0].y + c1 * a1.y + c2 * a2.y);
        const double2 q = make_double2(v[0].x + c2 * a1.x + c1 * a2.x, v[0].y + c2 * a1.y + c1 * a2.y);
        const double2 f = make_double2(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y);
        const double2 g = make_double2(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y);
        v[0] = cadd(v[0], cadd(a1, a2));
        v[1] = make_double2(p.x + f.y, p.y - f.x);
        v[4] = make_double2(p.x - f.y, p.y + f.x);
        v[2] = make_double2(q.x + g.y, q.y - g.x);
        v[3] = make_double2(q.x - g.y, q.y + g.x);
    }
};
template <> struct Dft<8> {
    HS_DEV static void run(double2 *v) {
        const double h = 0.70710678118654752440;
        double2 e[4], o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) { e[k] = cadd(v[k], v[k + 4]); o[k] = csub(v[k], v[k + 4]); }
        o[1] = make_double2(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x));        // exp(-i pi / 4)
        o[2] = mul_mi(o[2]);
        o[3] = make_double2(h * (o[3].y - o[3].x), -h * (o[3].x + o[3].y));       // exp(-3 i pi / 4)
        Dft<4>::run(e);
        Dft<4>::run(o);
#pragma unroll
        for (int k = 0; k < 4; ++k) { v[2 * k] = e[k]; v[2 * k + 1] = o[k]; }
    }
};
template <> struct Dft<9> {
    HS_DEV static void run(double2 *v) {
        const double2 w1 = make_double2(0.76604444311897803520, -0.64278760968653932632);    // exp(-2 pi i / 9)
        const double2 w2 = make_double2(0.17364817766693034885, -0.98480775301220805937);
        const double2 w4 = make_double2(-0.93969262078590838405, -0.34202014332566873304);
        double2 u[3][3];                     // u[n2][k1]
#pragma unroll
        for (int n2 = 0; n2 < 3; ++n2) {
            double2 t[3] = {v[n2], v[n2 + 3], v[n2 + 6]};
            Dft<3>::run(t);
#pragma unroll
            for (int k1 = 0; k1 < 3; ++k1) u[n2][k1] = t[k1];
        }
        u[1][1] = cmul(u[1][1], w1);
        u[1][2] = cmul(u[1][2], w2);
        u[2][1] = cmul(u[2][1], w2);
        u[2][2] = cmul(u[2][2], w4);
#pragma unroll
        for (int k1 = 0; k1 < 3; ++k1) {
            double2 t[3] = {u[0][k1], u[1][k1], u[2][k1]};
            Dft<3>::run(t);
#pragma unroll
            for (int k2 = 0; k2 < 3; ++k2) v[k1 + 3 * k2] = t[k2];
        }
    }
};
template <> struct Dft<16> {
    HS_DEV static void run(double2 *v) {
        const double c = 0.92387953251128675613, s = 0.38268343236508977173, h = 0.70710678118654752440;   // pi / 8
        const double2 w1 = make_double2(c, -s), w3 = make_double2(s, -c);
        double2 u[4][4];                     // u[n2][k1]
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) {
            double2 t[4] = {v[n2], v[n2 + 4], v[n2 + 8], v[n2 + 12]};
            Dft<4>::run(t);
#pragma unroll
            for (int k1 = 0; k1 < 4; ++k1) u[n2][k1] = t[k1];
        }
        u[1][1] = cmul(u[1][1], w1);
        u[1][2] = make_double2(h * (u[1][2].x + u[1][2].y), h * (u[1][2].y - u[1][2].x));
        u[1][3] = cmul(u[1][3], w3);
        u[2][1] = make_double2(h * (u[2][1].x + u[2][1].y), h * (u[2][1].y - u[2][1].x));
        u[2][2] = mul_mi(u[2][2]);
        u[2][3] = make_double2(h * (u[2][3].y - u[2][3].x), -h * (u[2][3].x + u[2][3].y));
        u[3][1] = cmul(u[3][1], w3);
        u[3][2] = make_double2(h * (u[3][2].y - u[3][2].x), -h * (u[3][2].x + u[3][2].y));
        u[3][3] = cmul(u[3][3], make_double2(-c, s));      // exp(-9 i pi / 8)
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            double2 t[4] = {u[0][k1], u[1][k1], u[2][k1], u[3][k1]};
            Dft<4>::run(t);
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = t[k2];
        }
    }
};

// Position of element i of a line in shared memory. The stride of every stage but the last is a
// multiple of 2^lg, so the padded positions of a butterfly's elements are equally spaced too, and
// the last stage's blocks of 2^lg elements start in different banks.
HS_HD inline int fft_pad(int i, int lg) { return i + (i >> lg); }

// Lines in shared memory.
struct FftLines {
    double2 *s;
    int pitch, lg;
    // elements i0 + q sub of a line, q < R
    template <int R>
    HS_DEV void get(int line, int i0, int sub, double2 (&v)[R]) const {
        const double2 *p = s + line * pitch + fft_pad(i0, lg);
        const int d = sub == 1 ? 1 : fft_pad(sub, lg);
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = p[q * d];
    }
    template <int R>
    HS_DEV void put(int line, int i0, int sub, const double2 (&v)[R]) const {
        double2 *p = s + line * pitch + fft_pad(i0, lg);
        const int d = sub == 1 ? 1 : fft_pad(sub, lg);
#pragma unroll
        for (int q = 0; q < R; ++q) p[q * d] = v[q];
    }
};

// Stage st of `lines` transforms: blocks of Lb elements, R values sub = Lb / R apart each. Forward:
// transform, then the twiddles exp(-2 pi i j q / Lb); backward (DIT): the twiddles first. Butterfly
// k of a line has the elements i0 + q sub: load(line, k, i0, sub, v) fills them and
// store(line, k, i0, sub, v) takes the results, so that the first and the last stage of a
// transform work on global memory (or on the energies) directly and only the exchanges between
// stages go through shared memory. COLS: consecutive threads take the lines of one butterfly
// (columns of a row-major array), otherwise the butterflies of one line.
template <int R, bool DIT, bool COLS, typename Load, typename Store>
HS_DEV void fft_stage(int lines, const FftAxis &A, int st, int Lb, const double2 *table, Load load, Store store) {
    const int nb = A.M / R, sub = Lb / R;
    const int lg = 31 - __clz(sub);          // sub is a power of two whenever Lb < M
    const float inv = 1.0f / (float)nb;
    for (int b = threadIdx.x; b < lines * nb; b += blockDim.x) {
        int line, k;
        if (COLS) { line = lines == 2 ? b & 1 : 0; k = lines == 2 ? b >> 1 : b; }
        else { line = (int)(((float)b + 0.5f) * inv); k = b - line * nb; }   // exact: b < 2^20
        const int j = Lb == A.M ? k : k & (sub - 1);
        const int i0 = Lb == A.M ? k : (k >> lg) * Lb + j;
        const double2 *tw = table + A.toff[st] + j;
        double2 v[R];
        load(line, k, i0, sub, v);
        if (DIT && sub > 1) {
#pragma unroll
            for (int q = 1; q < R; ++q) v[q] = cmul(v[q], tw[q * sub]);
        }
        Dft<R>::run(v);
        if (!DIT && sub > 1) {
#pragma unroll
            for (int q = 1; q < R; ++q) v[q] = cmul(v[q], tw[q * sub]);
        }
        store(line, k, i0, sub, v);
    }
}

template <bool DIT, bool COLS, typename Load, typename Store>
HS_DEV void fft_stage_of(int lines, const FftAxis &A, int st, int Lb, const double2 *tw, Load load, Store store) {
    switch (A.radix[st]) {
        case 16: fft_stage<16, DIT, COLS>(lines, A, st, Lb, tw, load, store); break;
        case 9: fft_stage<9, DIT, COLS>(lines, A, st, Lb, tw, load, store); break;
        case 8: fft_stage<8, DIT, COLS>(lines, A, st, Lb, tw, load, store); break;
        case 5: fft_stage<5, DIT, COLS>(lines, A, st, Lb, tw, load, store); break;
        case 4: fft_stage<4, DIT, COLS>(lines, A, st, Lb, tw, load, store); break;
        default: fft_stage<3, DIT, COLS>(lines, A, st, Lb, tw, load, store); break;
    }
}

// A stage between the first and the last, in shared memory: radix 4, 8 or 16.
template <bool DIT>
HS_DEV void fft_inner_stage(const FftLines &B, int lines, const FftAxis &A, int st, int Lb, const double2 *tw) {
    auto load = [&](int l, int, int i0, int sub, auto &v) { B.get(l, i0, sub, v); };
    auto store = [&](int l, int, int i0, int sub, const auto &v) { B.put(l, i0, sub, v); };
    switch (A.radix[st]) {
        case 16: fft_stage<16, DIT, false>(lines, A, st, Lb, tw, load, store); break;
        case 8: fft_stage<8, DIT, false>(lines, A, st, Lb, tw, load, store); break;
        default: fft_stage<4, DIT, false>(lines, A, st, Lb, tw, load, store); break;
    }
    __syncthreads();
}

// The stages of a forward (backward) transform between its first and its last. Every transform has
// at least two stages; the caller runs the first and the last.
HS_DEV void fft_inner_forward(const FftLines &B, int lines, const FftAxis &A, const double2 *tw) {
    int Lb = A.M / A.radix[0];
    for (int k = 1; k + 1 < A.n_stages; ++k) {
        fft_inner_stage<false>(B, lines, A, k, Lb, tw);
        Lb /= A.radix[k];
    }
}
HS_DEV void fft_inner_backward(const FftLines &B, int lines, const FftAxis &A, const double2 *tw) {
    int Lb = A.radix[A.n_stages - 1];
    for (int k = A.n_stages - 2; k >= 1; --k) {
        Lb *= A.radix[k];
        fft_inner_stage<true>(B, lines, A, k, Lb, tw);
    }
}

// Last forward stage, product with the other spectrum and first backward stage of a convolution:
// blocks of R contiguous elements (no twiddles), all in registers.
template <int R>
HS_DEV void fft_product(const FftLines &B, const FftLines &S, int lines, int M) {
    const int nb = M / R;
    const float inv = 1.0f / (float)nb;
    for (int b = threadIdx.x; b < lines * nb; b += blockDim.x) {
        const int line = (int)(((float)b + 0.5f) * inv), i0 = (b - line * nb) * R;
        double2 v[R], w[R];
        B.get(line, i0, 1, v);
        Dft<R>::run(v);
        S.get(line, i0, 1, w);
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = cswap(cmul(v[q], w[q]));
        Dft<R>::run(v);
        B.put(line, i0, 1, v);
    }
}

// Stage st's twiddles exp(-2 pi i j q / Lb), q < R, j < sub, at toff[st] + q sub + j: consecutive
// threads (j) read consecutive entries. The last stage has none.
HS_DEV void fft_twiddles(double2 *tw, const FftAxis &A) {
    int Lb = A.M;
    for (int st = 0; st + 1 < A.n_stages; ++st) {
        const int R = A.radix[st], sub = Lb / R;
        const float inv = 1.0f / (float)sub;
        for (int e = threadIdx.x; e < Lb; e += blockDim.x) {
            const int q = (int)(((float)e + 0.5f) * inv), j = e - q * sub;
            double sn, cs;
            sincospi(-2.0 * (j * q) / Lb, &sn, &cs);
            tw[A.toff[st] + e] = make_double2(cs, sn);
        }
        Lb = sub;
    }
}

// The kernels of a slot: real part K[re], imaginary part Kps[re] (two channels) or K[im].
HS_DEV void slot_kernels(const HsLattice &L, const FftParams &P, int slot, const float *&re, const float *&im) {
    const int64_t W = (int64_t)P.KH * P.KW;
    if (P.two) { re = L.K + slot * W; im = L.Kps + slot * W; return; }
    re = L.K + 2 * slot * W;
    im = 2 * slot + 1 < L.n_sub ? re + W : nullptr;
}

__global__ void __launch_bounds__(FFT_T, FFT_MIN_CTAS) fft_rows_kernel(HsLattice L, FftParams P, int lines) {
    extern __shared__ __align__(16) double2 s_fft[];
    double2 *tw = s_fft;
    const FftLines B{s_fft + P.X.tlen, P.X.Mp, P.X.lg};
    __shared__ FftStat s_stat[FFT_T / 32];
    fft_twiddles(tw, P.X);
    unsigned kmax = 0u, mmax = 0u;
    int count = 0;
    const int M = P.X.M, w = P.KW / 2, last = P.X.n_stages - 1;
    for (int l0 = blockIdx.x * lines; l0 < P.n_lines; l0 += gridDim.x * lines) {
        const int n = min(lines, P.n_lines - l0);
        __syncthreads();   // tw is filled, the buffer is free
        fft_stage_of<false, false>(n, P.X, 0, M, tw, [&](int line, int, int i0, int sub, auto &v) {
            constexpr int R = sizeof(v) / sizeof(double2);
            const int l = l0 + line;
            if (l < P.nys) {
                const bool wrap = P.oy || P.ox;
                const float *row = L.mm + (int64_t)(wrap ? hs_wrap(l - P.oy, L.ny) : l) * L.nx;
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    const int p = i0 + q * sub;
                    const float f = p < P.nxs ? __ldg(row + (wrap ? hs_wrap(p - P.ox, L.nx) : p)) : 0.f;
                    v[q] = make_double2((double)f, 0.0);
                    mmax = max(mmax, __float_as_uint(f) & 0x7fffffffu);
                    count += f != 0.f;
                }
                return;
            }
            const int r = l - P.nys, slot = r / P.KH;
            const float *re, *im;
            slot_kernels(L, P, slot, re, im);
            const int64_t at = (int64_t)(r - slot * P.KH) * P.KW + w;      // offset 0 of the kernel row
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int p = i0 + q * sub, e = p <= w ? p : p - M;         // reversed: position e holds offset -e
                const bool in = e >= -w && e <= w;
                const float a = in ? __ldg(re + at - e) : 0.f, b = (in && im) ? __ldg(im + at - e) : 0.f;
                v[q] = make_double2((double)a, (double)b);
                kmax = max(kmax, max(__float_as_uint(a) & 0x7fffffffu, __float_as_uint(b) & 0x7fffffffu));
            }
        }, [&](int line, int, int i0, int sub, const auto &v) { B.put(line, i0, sub, v); });
        __syncthreads();
        fft_inner_forward(B, n, P.X, tw);
        // The order of a line's spectrum in global memory: element q of butterfly k of the last
        // stage at q (M / R) + k, so that consecutive threads write (and later read) consecutive
        // elements. Every line has the same order, and no pass needs another one.
        fft_stage_of<false, false>(n, P.X, last, P.X.radix[last], tw,
                                   [&](int line, int, int i0, int sub, auto &v) { B.get(line, i0, sub, v); },
                                   [&](int line, int k, int, int, const auto &v) {
            constexpr int R = sizeof(v) / sizeof(double2);
            const int l = l0 + line, r = l - P.nys, slot = r / P.KH;
            double2 *out = P.spec + (l < P.nys ? l : P.nys + (int64_t)slot * P.slot_rows + (r - slot * P.KH)) * M + k;
            const int nb = M / R;
#pragma unroll
            for (int q = 0; q < R; ++q) out[q * nb] = v[q];
        });
    }
    // this block's largest |K| and |mm| (as ordered bits: infinities and NaN come out largest)
    for (int o = 16; o; o >>= 1) {
        kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
        mmax = max(mmax, __shfl_xor_sync(0xffffffffu, mmax, o));
        count += __shfl_xor_sync(0xffffffffu, count, o);
    }
    if ((threadIdx.x & 31) == 0) s_stat[threadIdx.x >> 5] = FftStat{kmax, mmax, count, 0};
    __syncthreads();
    if (threadIdx.x == 0) {
        FftStat t = s_stat[0];
        for (int k = 1; k < FFT_T / 32; ++k) {
            t.kmax = max(t.kmax, s_stat[k].kmax);
            t.mmax = max(t.mmax, s_stat[k].mmax);
            t.count += s_stat[k].count;
        }
        P.stat[blockIdx.x] = t;
    }
    // the tables of the other passes
    if (blockIdx.x == 0)
        for (int k = threadIdx.x; k < P.X.tlen; k += blockDim.x) P.twx[k] = tw[k];
    if (blockIdx.x == gridDim.x - 1) fft_twiddles(P.twy, P.Y);
}

// Does a cell of the rows with phase `ry` belong to slot `slot`?
HS_DEV bool slot_in_row(const HsLattice &L, const FftParams &P, int slot, int ry) {
    for (int rx = 0; rx < L.ux; ++rx) {
        const int s = L.sub_of[ry * L.ux + rx];
        if (s >= 0 && (P.two ? s : s >> 1) == slot) return true;
    }
    return false;
}

__global__ void __launch_bounds__(FFT_T, FFT_MIN_CTAS) fft_cols_kernel(HsLattice L, FftParams P, int cols) {
    extern __shared__ __align__(16) double2 s_fft[];
    __shared__ unsigned char s_has[FFT_HAS];
    double2 *tw = s_fft;
    const int M = P.Y.M, MX = P.X.M, w = P.KH / 2;
    const FftLines S{s_fft + P.Y.tlen, P.Y.Mp, P.Y.lg}, B{S.s + cols * P.Y.Mp, P.Y.Mp, P.Y.lg};
    const int c0 = blockIdx.x * cols, nc = min(cols, MX - c0);
    const bool masked = P.n_slots * L.uy <= FFT_HAS;
    if (masked)
        for (int k = threadIdx.x; k < P.n_slots * L.uy; k += blockDim.x) s_has[k] = slot_in_row(L, P, k / L.uy, k % L.uy);
    for (int k = threadIdx.x; k < P.Y.tlen; k += blockDim.x) tw[k] = P.twy[k];
    __syncthreads();
    const int last = P.Y.n_stages - 1, rlast = P.Y.radix[last];
    auto to_lines = [](const FftLines &T) {
        return [&T](int c, int, int i0, int sub, const auto &v) { T.put(c, i0, sub, v); };
    };
    auto of_lines = [](const FftLines &T) {
        return [&T](int c, int, int i0, int sub, auto &v) { T.get(c, i0, sub, v); };
    };
    fft_stage_of<false, true>(cols, P.Y, 0, M, tw, [&](int c, int, int i0, int sub, auto &v) {
        constexpr int R = sizeof(v) / sizeof(double2);
        const double2 *in = P.spec + c0 + c;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int p = i0 + q * sub;
            v[q] = (c < nc && p < P.nys) ? in[(int64_t)p * MX] : make_double2(0.0, 0.0);
        }
    }, to_lines(S));
    __syncthreads();
    fft_inner_forward(S, cols, P.Y, tw);
    fft_stage_of<false, false>(cols, P.Y, last, rlast, tw, of_lines(S), to_lines(S));
    for (int slot = 0; slot < P.n_slots; ++slot) {
        double2 *rows = P.spec + (P.nys + (int64_t)slot * P.slot_rows) * MX + c0;
        __syncthreads();
        fft_stage_of<false, true>(cols, P.Y, 0, M, tw, [&](int c, int, int i0, int sub, auto &v) {
            constexpr int R = sizeof(v) / sizeof(double2);
            const double2 *in = rows + (int64_t)w * MX + c;      // offset 0 of the kernel
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int p = i0 + q * sub, e = p <= w ? p : p - M;
                v[q] = (c < nc && e >= -w && e <= w) ? in[-(int64_t)e * MX] : make_double2(0.0, 0.0);
            }
        }, to_lines(B));
        __syncthreads();
        fft_inner_forward(B, cols, P.Y, tw);
        switch (rlast) {
            case 16: fft_product<16>(B, S, cols, M); break;
            case 8: fft_product<8>(B, S, cols, M); break;
            default: fft_product<4>(B, S, cols, M); break;
        }
        __syncthreads();
        fft_inner_backward(B, cols, P.Y, tw);
        fft_stage_of<true, true>(cols, P.Y, 0, M, tw, of_lines(B),
                                 [&](int c, int, int i0, int sub, const auto &v) {      // parts still swapped
            constexpr int R = sizeof(v) / sizeof(double2);
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int y = i0 + q * sub - P.oy;
                if (c < nc && y >= 0 && y < L.ny && (!masked || s_has[slot * L.uy + y % L.uy])) rows[(int64_t)y * MX + c] = v[q];
            }
        });
    }
}

// The direct sum of one cell, for inputs that hold infinities or NaN (which a transform would
// spread over the whole lattice).
__device__ __noinline__ double2 direct_cell(const HsLattice &L, int s, int y, int x) {
    double a, ap;
    if (!L.dip_wrap && L.dip_wy == L.ny - 1 && L.dip_wx == L.nx - 1) dip_full_cell<double, true>(L, s, y, x, a, ap);
    else dip_full_cell<double, false>(L, s, y, x, a, ap);
    return make_double2(a, ap);
}

__global__ void __launch_bounds__(FFT_T, FFT_MIN_CTAS) fft_cells_kernel(HsLattice L, FftParams P) {
    extern __shared__ __align__(16) double2 s_fft[];
    __shared__ FftStat s_stat[FFT_T / 32];
    double2 *tw = s_fft;
    const FftLines B{s_fft + P.X.tlen, P.X.Mp, P.X.lg};
    const int M = P.X.M, y = blockIdx.x, ry = y % L.uy, last = P.X.n_stages - 1;
    for (int k = threadIdx.x; k < P.X.tlen; k += blockDim.x) tw[k] = P.twx[k];
    FftStat t{0u, 0u, 0, 0};
    for (int k = threadIdx.x; k < P.stat_blocks; k += blockDim.x) {
        const FftStat q = P.stat[k];
        t.kmax = max(t.kmax, q.kmax); t.mmax = max(t.mmax, q.mmax); t.count += q.count;
    }
    for (int o = 16; o; o >>= 1) {
        t.kmax = max(t.kmax, __shfl_xor_sync(0xffffffffu, t.kmax, o));
        t.mmax = max(t.mmax, __shfl_xor_sync(0xffffffffu, t.mmax, o));
        t.count += __shfl_xor_sync(0xffffffffu, t.count, o);
    }
    if ((threadIdx.x & 31) == 0) s_stat[threadIdx.x >> 5] = t;
    __syncthreads();
    t = s_stat[0];
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
        t.kmax = max(t.kmax, s_stat[k].kmax); t.mmax = max(t.mmax, s_stat[k].mmax); t.count += s_stat[k].count;
    }
    const bool finite = t.kmax < 0x7f800000u && t.mmax < 0x7f800000u;
    // Sums that vanish (no partner in reach, exact cancellation) come out of the transforms as
    // rounding noise, whose sign relax() would act on; the direct sum gives 0 there. Values below
    // the rounding of the largest possible terms are therefore 0: 2^-52 max|K| max|mm| sqrt(#sources).
    const double floor_ = 2.220446049250313e-16 * (double)__uint_as_float(t.kmax) * (double)__uint_as_float(t.mmax) *
                          sqrt((double)t.count);
    const double norm = 1.0 / ((double)P.X.M * (double)P.Y.M);
    const int64_t row = (int64_t)y * L.nx;
    for (int x = threadIdx.x; x < L.nx; x += blockDim.x) {   // sites without a kernel
        if (hs_sub(L, y, x) >= 0) continue;
        const double none = L.dip_pref * (double)L.moment[row + x] * (double)L.m[row + x] * 0.0;
        P.E[row + x] = none;
        if (P.Ep) P.Ep[row + x] = none;
    }
    for (int slot = 0; slot < P.n_slots; ++slot) {
        if (!slot_in_row(L, P, slot, ry)) continue;     // block-uniform
        const double2 *in = P.spec + (P.nys + (int64_t)slot * P.slot_rows + y) * M;
        __syncthreads();                                // tw is filled, buf is free again
        fft_stage_of<true, false>(1, P.X, last, P.X.radix[last], tw, [&](int, int k, int, int, auto &v) {
            constexpr int R = sizeof(v) / sizeof(double2);
            const int nb = M / R;
#pragma unroll
            for (int q = 0; q < R; ++q) v[q] = in[q * nb + k];
        }, [&](int l, int, int i0, int sub, const auto &v) { B.put(l, i0, sub, v); });
        __syncthreads();
        fft_inner_backward(B, 1, P.X, tw);
        fft_stage_of<true, false>(1, P.X, 0, M, tw, [&](int l, int, int i0, int sub, auto &v) { B.get(l, i0, sub, v); },
                                  [&](int, int, int i0, int sub, const auto &v) {
            constexpr int R = sizeof(v) / sizeof(double2);
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int x = i0 + q * sub - P.ox;
                if (x < 0 || x >= L.nx) continue;
                const int s = hs_sub(L, y, x);
                if (s < 0 || (P.two ? s : s >> 1) != slot) continue;
                const double2 z = cswap(v[q]);
                double a = ((P.two || !(s & 1)) ? z.x : z.y) * norm, ap = z.y * norm;
                if (fabs(a) < floor_) a = 0.0;
                if (fabs(ap) < floor_) ap = 0.0;
                const int mi = L.m[row + x];
                if (!finite && mi) {
                    const double2 d = direct_cell(L, s, y, x);
                    a = d.x;
                    ap = d.y;
                }
                const double scale = L.dip_pref * (double)L.moment[row + x] * (double)mi;
                P.E[row + x] = scale * (mi ? a : 0.0);
                if (P.Ep) P.Ep[row + x] = scale * (mi ? ap : 0.0);
            }
        });
    }
}

// Smallest length of the supported form that is at least n; 0 when that exceeds FFT_MAX_M.
int fft_length(int n) {
    int best = 0;
    for (int odd : {1, 3, 5, 9}) {
        int m = odd == 1 ? 32 : 16 * odd;      // two stages at least
        while (m < n) m *= 2;
        if (m <= FFT_MAX_M && (!best || m < best)) best = m;
    }
    return best;
}

FftAxis fft_axis(int M) {
    FftAxis A{};
    A.M = M;
    int m = M;
    for (int odd : {9, 5, 3})
        if (m % odd == 0) { A.radix[A.n_stages++] = odd; m /= odd; }
    int a = 0;
    while ((1 << a) < m) ++a;
    const int stages = (a + 3) / 4;           // the factors of two, spread evenly over radices 4 to 16
    for (int k = 0; k < stages; ++k) {
        A.lg = a / stages + (k < a % stages ? 1 : 0);
        A.radix[A.n_stages++] = 1 << A.lg;
    }
    for (int st = 0, Lb = M; st + 1 < A.n_stages; Lb /= A.radix[st++]) { A.toff[st] = A.tlen; A.tlen += Lb; }
    A.Mp = fft_pad(M, A.lg);
    A.Mp += (12 - (A.Mp & 7)) & 7;            // 4 mod 8: the two columns of a tile fall into different banks
    return A;
}

struct FftLayout {
    FftParams P;
    int64_t twx_off, twy_off, stat_off, total;
    int row_lines, cols;
    size_t row_smem, col_smem, cell_smem;
};

// False when the lattice is beyond the transform lengths.
bool fft_layout(const HsLattice &L, FftLayout &o) {
    FftParams &P = o.P;
    P = FftParams{};
    P.oy = L.dip_wrap ? L.dip_wy : 0;
    P.ox = L.dip_wrap ? L.dip_wx : 0;
    const int64_t needy = (int64_t)L.ny + (L.dip_wrap ? 2 : 1) * (int64_t)L.dip_wy;
    const int64_t needx = (int64_t)L.nx + (L.dip_wrap ? 2 : 1) * (int64_t)L.dip_wx;
    if (needy > FFT_MAX_M || needx > FFT_MAX_M) return false;
    P.X = fft_axis(fft_length((int)needx));
    P.Y = fft_axis(fft_length((int)needy));
    P.nys = L.ny + 2 * P.oy;
    P.nxs = L.nx + 2 * P.ox;
    P.KH = 2 * L.dip_wy + 1;
    P.KW = 2 * L.dip_wx + 1;
    P.two = L.use_perp ? 1 : 0;
    P.n_slots = P.two ? L.n_sub : (L.n_sub + 1) / 2;
    P.slot_rows = std::max(P.KH, L.ny);
    const int64_t lines = P.nys + (int64_t)P.n_slots * P.KH;
    if (lines > (1 << 24)) return false;
    P.n_lines = (int)lines;
    // Rows: as many lines per CTA as its threads have radix-16 butterflies for, while the 148 SMs
    // still get two CTAs each. Columns: two per CTA (a whole 32-byte sector of every row) unless
    // that leaves SMs without one.
    o.row_lines = 1;
    while (o.row_lines < 4 && (o.row_lines + 1) * (P.X.M / 16) <= FFT_T && P.n_lines / (o.row_lines + 1) >= 296)
        ++o.row_lines;
    o.cols = (P.X.M >= 2 * 148 && P.Y.M <= 2048) ? 2 : 1;
    o.row_smem = (size_t)(P.X.tlen + o.row_lines * P.X.Mp) * sizeof(double2);
    o.col_smem = (size_t)(P.Y.tlen + 2 * o.cols * P.Y.Mp) * sizeof(double2);
    o.cell_smem = (size_t)(P.X.tlen + P.X.Mp) * sizeof(double2);
    const int64_t rows = P.nys + (int64_t)P.n_slots * P.slot_rows;
    o.twx_off = hs_align_up(rows * P.X.M * (int64_t)sizeof(double2), 256);
    o.twy_off = o.twx_off + hs_align_up(P.X.tlen * (int64_t)sizeof(double2), 256);
    o.stat_off = o.twy_off + hs_align_up(P.Y.tlen * (int64_t)sizeof(double2), 256);
    o.total = o.stat_off + hs_align_up(FFT_ROW_CTAS * (int64_t)sizeof(FftStat), 256);
    return true;
}

template <typename F>
int fft_allow(F *kernel, size_t smem, const char *name) {
    if (smem <= 40 * 1024) return HS_OK;      // dynamic plus static shared memory below the default limit
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { hs_set_error("%s: %s", name, cudaGetErrorString(e)); return HS_ECUDA; }
    return HS_OK;
}

}  // namespace

int64_t hs_fft_scratch(const HsLattice &L) {
    FftLayout o;
    return fft_layout(L, o) ? o.total : 0;
}

int hs_launch_dipolar_full_fft(const HsLattice &L, void *scratch, int64_t scratch_bytes, double *E64, double *Ep64,
                               cudaStream_t st) {
    FftLayout o;
    if (!fft_layout(L, o)) {
        hs_set_error("hs_dipolar_full_fft: lattice plus window longer than %d cells", FFT_MAX_M);
        return HS_ERANGE;
    }
    if (scratch_bytes < o.total) {
        hs_set_error("hs_dipolar_full_fft: scratch %lld < %lld bytes", (long long)scratch_bytes, (long long)o.total);
        return HS_ENOMEM;
    }
    char *base = reinterpret_cast<char *>(scratch);
    FftParams &P = o.P;
    P.spec = reinterpret_cast<double2 *>(base);
    P.twx = reinterpret_cast<double2 *>(base + o.twx_off);
    P.twy = reinterpret_cast<double2 *>(base + o.twy_off);
    P.stat = reinterpret_cast<FftStat *>(base + o.stat_off);
    P.E = E64;
    P.Ep = L.use_perp ? Ep64 : nullptr;
    int rc;
    if ((rc = fft_allow(fft_rows_kernel, o.row_smem, "fft_rows_kernel"))) return rc;
    if ((rc = fft_allow(fft_cols_kernel, o.col_smem, "fft_cols_kernel"))) return rc;
    if ((rc = fft_allow(fft_cells_kernel, o.cell_smem, "fft_cells_kernel"))) return rc;
    P.stat_blocks = std::min((P.n_lines + o.row_lines - 1) / o.row_lines, FFT_ROW_CTAS);
    fft_rows_kernel<<<P.stat_blocks, FFT_T, o.row_smem, st>>>(L, P, o.row_lines);
    if ((rc = hs_check_launch("fft_rows_kernel"))) return rc;
    fft_cols_kernel<<<(P.X.M + o.cols - 1) / o.cols, FFT_T, o.col_smem, st>>>(L, P, o.cols);
    if ((rc = hs_check_launch("fft_cols_kernel"))) return rc;
    // one radix-16 butterfly per thread
    const int cell_threads = std::min(FFT_T, (int)hs_align_up(std::max(P.X.M / 16, 64), 32));
    fft_cells_kernel<<<L.ny, cell_threads, o.cell_smem, st>>>(L, P);
    return hs_check_launch("fft_cells_kernel");
}
