// qg_wilson.cuh -- all planar Wilson loops R x T of a field in one gauge.
// Part of qg_fields.cu: a program that measures has that module loaded, and
// another one would be loaded by the first call (0.4 ms).
//
// W(R,T) = sum over x and i in {x,y,z} of Re Tr(L_t^T(x) L_i^R(x+T t)
// L_t^T(x+R i)^+ L_i^R(x)^+) (lattice_measurement_wilson, wilson_loop.cl:
// 55-454, for every R <= Rmax, T <= Tmax).  With V_x(t) the ordered product of
// the time links of column x from 0 to t (periodic beyond N4) the time lines
// are V_x(t0)^-1 V_x(t0+T), so
//
//   W = Re Tr( D_R(x,t0+T) E_R(x,t0)^+ ),
//   D_R(x,t) = V_x S_R V_(x+Ri)^+,   E_R(x,t) = V_x^-+ S_R V_(x+Ri)^-1
//
// with S_R(x,t) the spatial line of R links: no time line is multiplied up
// for any (t0, T), and a loop is a real inner product of 18 (SU(2): 8)
// numbers.  D and E grow by one product per R,
//
//   D_0 = V_x V_x^+,     D_R = D_(R-1) K(x+(R-1)i),  K = V_x^-+ U_i V_(x+i)^+
//   E_0 = (V_x V_x^+)^-1, E_R = E_(R-1) F(x+(R-1)i),  F = V_x U_i V_(x+i)^-1.
//
// The identities hold for any invertible links (no unitarity is used), but
// the rounding of a loop grows with the condition of V squared: a time line
// that is far from a multiple of a unitary matrix, or whose determinant could
// carry D and E out of range, raises *flag and the caller takes the column
// kernel (k_line_links).
//
// Cost per (x, i, t) at Rmax = Tmax = 8: 16 products and 64 inner products
// in FP64 (2900 multiply-adds) and 6 products and 2 inverses of
// preparation, against 128 products, 64 traces and 28 line products of the
// column kernel (k_wilson_cols).  All 8 x 8 loops of SU(3) 64^4 FP32: 47 ms
// against 90 ms (the column kernel's FP32 products) and 205 ms (its FP64
// ones); 6 x 6 loops of 20 x 18 x 22 x 14: 0.38 against 0.71 ms.
#pragma once
#include <algorithm>

#include "qg_internal.h"
#include "qg_observe.cuh"

namespace qg {

namespace {

constexpr int kSlots = 148 * 3;                         // blocks of k_loops: those resident at once
// their sums, at the start of the scratch (256-byte multiples)
size_t slots_doubles(int Rmax, int Tmax) { return ((size_t)kSlots * Rmax * Tmax + 31) / 32 * 32; }

template <int NC> struct CM { CX<double> m[NC][NC]; };

template <int NC, bool AH, bool BH>
__device__ __forceinline__ CM<NC> cmul(const CM<NC> &a, const CM<NC> &b)      // op(a) op(b), op = ^+ where AH / BH
{
    CM<NC> r;
#pragma unroll
    for (int i = 0; i < NC; i++)
#pragma unroll
        for (int j = 0; j < NC; j++) {
            double re = 0.0, im = 0.0;
#pragma unroll
            for (int k = 0; k < NC; k++) {
                const double ar = AH ? a.m[k][i].re : a.m[i][k].re, ai = AH ? -a.m[k][i].im : a.m[i][k].im;
                const double br = BH ? b.m[j][k].re : b.m[k][j].re, bi = BH ? -b.m[j][k].im : b.m[k][j].im;
                re = fma(ar, br, re);
                re = fma(-ai, bi, re);
                im = fma(ar, bi, im);
                im = fma(ai, br, im);
            }
            r.m[i][j] = { re, im };
        }
    return r;
}

__device__ __forceinline__ CX<double> cx_mul(const CX<double> &a, const CX<double> &b)
{
    return { fma(-a.im, b.im, a.re * b.re), fma(a.im, b.re, a.re * b.im) };
}
__device__ __forceinline__ CX<double> cx_sub(const CX<double> &a, const CX<double> &b)
{
    return { a.re - b.re, a.im - b.im };
}

// the inverse by the adjugate; det2 = |det|^2
template <int NC>
__device__ __forceinline__ CM<NC> cinv(const CM<NC> &a, double &det2)
{
    CM<NC> r;
    CX<double> d;
    if constexpr (NC == 2) {
        d = cx_sub(cx_mul(a.m[0][0], a.m[1][1]), cx_mul(a.m[0][1], a.m[1][0]));
        r.m[0][0] = a.m[1][1];
        r.m[1][1] = a.m[0][0];
        r.m[0][1] = { -a.m[0][1].re, -a.m[0][1].im };
        r.m[1][0] = { -a.m[1][0].re, -a.m[1][0].im };
    } else {
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const int p = (i + 1) % 3, q = (i + 2) % 3, u = (j + 1) % 3, v = (j + 2) % 3;
                r.m[j][i] = cx_sub(cx_mul(a.m[p][u], a.m[q][v]), cx_mul(a.m[p][v], a.m[q][u]));
            }
        d = cx_mul(a.m[0][0], r.m[0][0]);
        const CX<double> d1 = cx_mul(a.m[0][1], r.m[1][0]), d2 = cx_mul(a.m[0][2], r.m[2][0]);
        d = { d.re + d1.re + d2.re, d.im + d1.im + d2.im };
    }
    det2 = d.re * d.re + d.im * d.im;
    const double s = 1.0 / det2;
    const CX<double> id = { d.re * s, -d.im * s };
#pragma unroll
    for (int i = 0; i < NC; i++)
#pragma unroll
        for (int j = 0; j < NC; j++) r.m[i][j] = cx_mul(r.m[i][j], id);
    return r;
}

// Columns of a chunk: column g of 3 Vs (direction i = g / Vs; then line by
// line along i), columns [g0, g0 + ncol) in the scratch arrays
// [column][t / 8][component][t % 8]: a component is a fixed distance from
// the first (no address arithmetic per component) and eight lanes share two
// sectors.  NT1 >= N4 + Tmax, a multiple of 8.  Columns from `cut` on lie in
// the second part of the scratch (`jump` further); a line lies in one part.
struct Lines {
    Geom G;
    uint32_t Vs, g0, ncol, cut;
    int NT1, Rmax, Tmax;
    ptrdiff_t jump;
    double *V, *K, *F;
};
template <int NC>
__device__ __forceinline__ ptrdiff_t at_index(const Lines &L, uint32_t col, int t)
{
    return ((ptrdiff_t)col * (L.NT1 / 8) + t / 8) * (2 * NC * NC * 8) + t % 8 + (col < L.cut ? 0 : L.jump);
}

__device__ __forceinline__ Crd column(const Lines &L, uint32_t g, int &i, int &x)
{
    i = (int)(g / L.Vs);
    const uint32_t r = g - (uint32_t)i * L.Vs;
    const uint32_t ni = (uint32_t)(i == 0 ? L.G.n[0] : i == 1 ? L.G.n[1] : L.G.n[2]);
    const uint32_t line = r / ni;
    x = (int)(r - line * ni);
    const uint32_t n1 = (uint32_t)(i == 1 ? L.G.n[2] : L.G.n[1]);       // the faster transverse extent
    const int a = (int)(line % n1), b = (int)(line / n1);
    Crd c;
    c.t = 0;
    if (i == 0) { c.x = x; c.y = a; c.z = b; }
    else if (i == 1) { c.x = b; c.y = x; c.z = a; }
    else { c.x = b; c.y = a; c.z = x; }
    return c;
}

template <int NC, typename Real>
__device__ __forceinline__ CM<NC> link_cm(const Field<Real> &U, const Geom &G, const Crd &c, int mu,
                                          const double *params, int twist)
{
    const M3<double> d = load_d<NC, Real>(U, G, c, mu, params, twist);
    CM<NC> r;
#pragma unroll
    for (int i = 0; i < NC; i++)
#pragma unroll
        for (int j = 0; j < NC; j++) r.m[i][j] = d.m[i][j];
    return r;
}

// V of 8 columns a block.  The time links of a window of t are brought to
// shared memory first (all loads of the block in flight at once).  A thread
// per (row of V, segment of kSeg links, column) -- rows grow independently
// (V(t+1) row = V(t) row times the link): each multiplies its segment up from
// the unit row, one thread per (row, column) multiplies the segments'
// totals up, and each runs over its segment again from there and stores.
// Bound by latency and the FP64 pipe's chain (21 us for 3872 columns of
// N4 = 32; one serial chain of N4 steps, a load each, 24 us, and 39 against
// 25 us for 2112 columns of N4 = 64).
constexpr int kSeg = 8, kTLCols = 8;
template <int NC, typename Real> constexpr int kTLSegs = NC * sizeof(Real) == 24 ? 4 : 8;   // of a window (48 KB of links at most)

template <int NC, typename Real>
__global__ void __launch_bounds__(kTLCols * NC * kTLSegs<NC, Real>) k_time_lines(Field<Real> U, Lines L)
{
    constexpr int kSegs = kTLSegs<NC, Real>;
    using Vec = typename V4<Real>::T;
    constexpr int PL = NC == 3 ? 3 : 1;                 // planes of a link
    __shared__ Vec raw[kSeg * kSegs][PL][kTLCols];
    __shared__ double tot[kSegs][kTLCols][NC * 2 * NC + 1];    // [row][2 NC], padded: columns in other banks
    const int col0 = threadIdx.x % kTLCols, rs = threadIdx.x / kTLCols, row = rs % NC, worker = rs / NC;
    const uint32_t col = blockIdx.x * kTLCols + col0;
    const bool on = col < L.ncol;
    int i = 0, x = 0;
    Crd c0 = { 0, 0, 0, 0 };
    if (on) c0 = column(L, L.g0 + col, i, x);
    const int nt = L.G.n[3];
    double *out = L.V + at_index<NC>(L, on ? col : 0, 0) + (size_t)row * 2 * NC * 8;
    auto run = [&](int s0, CX<double> (&v)[NC], bool store) {    // segment worker of the window at s0 kSeg
        double keep[2 * NC][4];
#pragma unroll
        for (int k = 0; k < kSeg; k++) {
#pragma unroll
            for (int j = 0; j < NC; j++) { keep[2 * j][k % 4] = v[j].re; keep[2 * j + 1][k % 4] = v[j].im; }
            if (store && k % 4 == 3) {
                double *o = out + (size_t)(s0 + worker) * (2 * NC * NC * 8) + (k / 4) * 4;
#pragma unroll
                for (int j = 0; j < 2 * NC; j++) {
                    double2 *q = reinterpret_cast<double2 *>(o + j * 8);
                    q[0] = make_double2(keep[j][0], keep[j][1]);
                    q[1] = make_double2(keep[j][2], keep[j][3]);
                }
            }
            const Vec *r = &raw[worker * kSeg + k][0][col0];
            M3<double> u;
            if constexpr (NC == 3) {
                const Vec a = r[0], b = r[kTLCols], d = r[2 * kTLCols];
                u.m[0][0] = { (double)a.x, (double)b.x };
                u.m[0][1] = { (double)a.y, (double)b.y };
                u.m[0][2] = { (double)a.z, (double)b.z };
                u.m[1][0] = { (double)d.x, (double)d.z };
                u.m[1][1] = { (double)d.y, (double)d.w };
                u.m[1][2] = { (double)a.w, (double)b.w };
                fill_row3(u);
            } else {
                const Vec a = r[0];
                u.m[0][0] = { (double)a.x, (double)a.z };
                u.m[0][1] = { (double)a.y, (double)a.w };
                u.m[1][0] = { -(double)a.y, (double)a.w };
                u.m[1][1] = { (double)a.x, -(double)a.z };
            }
            CX<double> n[NC];
#pragma unroll
            for (int j = 0; j < NC; j++) {
                double re = 0.0, im = 0.0;
#pragma unroll
                for (int q = 0; q < NC; q++) {
                    re = fma(v[q].re, u.m[q][j].re, re);
                    re = fma(-v[q].im, u.m[q][j].im, re);
                    im = fma(v[q].re, u.m[q][j].im, im);
                    im = fma(v[q].im, u.m[q][j].re, im);
                }
                n[j] = { re, im };
            }
#pragma unroll
            for (int j = 0; j < NC; j++) v[j] = n[j];
        }
    };
    constexpr unsigned kRows = (1u << (kTLCols * NC)) - 1u;      // worker 0: the first lanes of warp 0
    CX<double> V[NC];                                   // worker 0: row of V at the next segment's start
#pragma unroll
    for (int j = 0; j < NC; j++) V[j] = { j == row ? 1.0 : 0.0, 0.0 };
    const int nseg = L.NT1 / kSeg;
    for (int s0 = 0; s0 < nseg; s0 += kSegs) {
        const int ns = min(kSegs, nseg - s0);
        if (on)
            for (int k = rs; k < ns * kSeg; k += blockDim.x / kTLCols) {
                Crd c = c0;
                c.t = (s0 * kSeg + k) % nt;
                const uint32_t e = cb_index(L.G, c, parity_of(c));
#pragma unroll
                for (int p = 0; p < PL; p++) raw[k][p][col0] = U.p[(size_t)(3 + 4 * p) * U.pstride + e];
            }
        __syncthreads();
        if (on && worker < ns) {
            CX<double> v[NC];
#pragma unroll
            for (int j = 0; j < NC; j++) v[j] = { j == row ? 1.0 : 0.0, 0.0 };
            run(s0, v, false);
            double *q = &tot[worker][col0][row * 2 * NC];
#pragma unroll
            for (int j = 0; j < NC; j++) { q[2 * j] = v[j].re; q[2 * j + 1] = v[j].im; }
        }
        __syncthreads();
        // tot[k] becomes V at the segment's start; a row of the product needs
        // all rows of the segment's total, so the rows go in step
        if (worker == 0) {
            for (int k = 0; k < ns; k++) {
                double *q = tot[k][col0];
                CX<double> n[NC];
#pragma unroll
                for (int j = 0; j < NC; j++) n[j] = { 0.0, 0.0 };
                if (on) {
#pragma unroll
                    for (int a = 0; a < NC; a++)
#pragma unroll
                        for (int j = 0; j < NC; j++) {
                            const double br = q[(a * NC + j) * 2], bi = q[(a * NC + j) * 2 + 1];
                            n[j].re = fma(V[a].re, br, n[j].re);
                            n[j].re = fma(-V[a].im, bi, n[j].re);
                            n[j].im = fma(V[a].re, bi, n[j].im);
                            n[j].im = fma(V[a].im, br, n[j].im);
                        }
                }
                __syncwarp(kRows);
                if (on) {
#pragma unroll
                    for (int j = 0; j < NC; j++) { q[(row * NC + j) * 2] = V[j].re; q[(row * NC + j) * 2 + 1] = V[j].im; }
                }
#pragma unroll
                for (int j = 0; j < NC; j++) V[j] = n[j];
            }
        }
        __syncthreads();
        if (on && worker < ns) {
            const double *q = &tot[worker][col0][row * 2 * NC];
            CX<double> v[NC];
#pragma unroll
            for (int j = 0; j < NC; j++) v[j] = { q[2 * j], q[2 * j + 1] };
            run(s0, v, true);
        }
        __syncthreads();
    }
}

template <int NC>
__device__ __forceinline__ CM<NC> load_soa(const double *p)
{
    CM<NC> r;
#pragma unroll
    for (int i = 0; i < NC; i++)
#pragma unroll
        for (int j = 0; j < NC; j++) {
            r.m[i][j].re = p[2 * (i * NC + j) * 8];
            r.m[i][j].im = p[(2 * (i * NC + j) + 1) * 8];
        }
    return r;
}
template <int NC>
__device__ __forceinline__ void store_soa(double *p, const CM<NC> &a)
{
#pragma unroll
    for (int i = 0; i < NC; i++)
#pragma unroll
        for (int j = 0; j < NC; j++) {
            p[2 * (i * NC + j) * 8] = a.m[i][j].re;
            p[(2 * (i * NC + j) + 1) * 8] = a.m[i][j].im;
        }
}

// K (t < N4 + Tmax) and F (t < N4) of every column and t of the chunk.
// *flag unless |V|^2 |V^-1|^2 (Frobenius norms; NC^2 for a unitary V) is below
// twice its least, so that no loop loses more than a few roundings, and
// |det V|^2 lies in (1/4, 4).  The determinant alone says nothing of the
// condition: rows scaled by s and 1/s leave it at 1.  Links rounded to FP32
// stay within 1e-9 of the least over 72 factors, links with 1 % of noise in
// every number within 3 %.
template <int NC, typename Real, bool TW>
__global__ void __launch_bounds__(128) k_line_links(Field<Real> U, Lines L, const double *params, int twist,
                                                     double *flag)
{
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t col = idx / (uint32_t)L.NT1;
    const int t = (int)(idx - col * (uint32_t)L.NT1), nt = L.G.n[3];
    if (col >= L.ncol || t >= nt + L.Tmax) return;
    int i, x;
    Crd c = column(L, L.g0 + col, i, x);
    const int ni = i == 0 ? L.G.n[0] : i == 1 ? L.G.n[1] : L.G.n[2];
    const ptrdiff_t at = at_index<NC>(L, col, t);
    const ptrdiff_t nx = at_index<NC>(L, x + 1 == ni ? col - (uint32_t)x : col + 1, t);     // column x + i of the line
    c.t = t % nt;
    const CM<NC> u = link_cm<NC, Real>(U, L.G, c, i, params, TW ? twist : 0);
    const CM<NC> v = load_soa<NC>(L.V + at), w = load_soa<NC>(L.V + nx);
    double det2;
    const CM<NC> vi = cinv(v, det2);
    double vv = 0.0, ww = 0.0;
#pragma unroll
    for (int a = 0; a < NC; a++)
#pragma unroll
        for (int b = 0; b < NC; b++) {
            vv = fma(v.m[a][b].re, v.m[a][b].re, fma(v.m[a][b].im, v.m[a][b].im, vv));
            ww = fma(vi.m[a][b].re, vi.m[a][b].re, fma(vi.m[a][b].im, vi.m[a][b].im, ww));
        }
    if (!(det2 > 0.25 && det2 < 4.0 && vv * ww < 2.0 * NC * NC)) *flag = 1.0;
    store_soa(L.K + at, cmul<NC, false, true>(cmul<NC, true, false>(vi, u), w));
    if (t < nt) {
        const CM<NC> wi = cinv(w, det2);
        store_soa(L.F + at, cmul<NC, false, false>(cmul<NC, false, false>(v, u), wi));
    }
}

constexpr int kLoopThreads = 160;                       // of k_loops at most: three blocks per SM
constexpr int kTB = 8;                                  // t0 of one inner-product item

// A block takes `cols` columns and a window of TW values of t0: a thread per
// (column, t) of D (TW + Tmax of them) and of E (TW), each growing its matrix
// in registers; per R the matrices go to shared memory and the inner products
// of all T are taken there, a thread per component, column and eight t0
// for all T at once (8 + 8 + Tmax - 1 shared reads for 8 Tmax multiply-adds;
// a read per operand would be bound by shared memory, four to one).  The next
// link matrix is loaded under the inner products.  TM: the T's computed (4, 8
// or 16 >= Tmax).  Measured on 3872 columns of N4 = 32, all 8 x 8 loops: 91 us,
// the L1 data path 71 % busy (shared reads and writes and the link loads),
// the FP64 pipe 39 %; with one buffer, skewed rows and more threads a block
// 109 us.
template <int NC, int TM>
__global__ void __launch_bounds__(kLoopThreads, 3) k_loops(Lines L, int cols, int TW, int nwin, double *slots)
{
    constexpr int NR = 2 * NC * NC;
    extern __shared__ double sm[];
    const int TWp = (TW + kTB - 1) / kTB * kTB;
    // lengths of a column's D and E: odd, so that the rows the lanes of a warp
    // read lie in different banks
    const int dl = (TWp + TM) | 1, el = TWp | 1, buf = NR * cols * (dl + el);
    double *sacc = sm + 2 * buf;
    const int nl = L.Rmax * L.Tmax, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    for (int k = tid; k < 2 * buf + nw * nl; k += blockDim.x) sm[k] = 0.0;
    const int nt = L.G.n[3], nD = TW + L.Tmax;
    const bool isD = tid < cols * nD;
    const int q0 = isD ? tid : tid - cols * nD, per = isD ? nD : TW;
    const int ci = q0 / per, tl = q0 - ci * per;
    const bool mine = ci < cols;
    // D [component][column][dl], then E [component][column][el], in two buffers
    const int s = (isD ? ci * dl : NR * cols * dl + ci * el) + tl, ss = cols * (isD ? dl : el);
    const size_t step = (size_t)(L.NT1 / 8) * (NR * 8);          // one column on
    const double *link = isD ? L.K : L.F;
    // this thread's inner products
    const int nblk = TWp / kTB, items = NR * cols * nblk;
    const bool item = tid < items;
    const int blk = item ? tid / (NR * cols) : 0, row = item ? tid - blk * (NR * cols) : 0;   // row: component, column
    const int pd = row * dl + blk * kTB, pe = NR * cols * dl + row * el + blk * kTB;
    double *sa = sacc + wid * nl + lane / (32 / TM);
    const bool adds = lane % (32 / TM) == 0 && lane / (32 / TM) < L.Tmax;
    const uint32_t groups = (L.ncol + cols - 1) / cols, units = groups * (uint32_t)nwin;
    __syncthreads();
    int par = 0;
    for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
        const uint32_t grp = u / (uint32_t)nwin;
        const uint32_t col = grp * cols + ci;
        const int t = (int)(u - grp * nwin) * TW + tl;
        const bool on = mine && col < L.ncol && t < (isD ? nt + L.Tmax : nt);
        int x = 0, ni = 1;
        CM<NC> m, k;
#pragma unroll
        for (int a = 0; a < NC; a++)
#pragma unroll
            for (int b = 0; b < NC; b++) m.m[a][b] = { 0.0, 0.0 };
        const double *at = link;
        if (on) {
            int i;
            column(L, L.g0 + col, i, x);
            ni = i == 0 ? L.G.n[0] : i == 1 ? L.G.n[1] : L.G.n[2];
            const ptrdiff_t o = at_index<NC>(L, col, t);
            at = link + o;
            CM<NC> v = load_soa<NC>(L.V + o);
            k = load_soa<NC>(at);
            if (isD) {
                m = cmul<NC, false, true>(v, v);
            } else {
                double det2;
                v = cinv(v, det2);
                m = cmul<NC, true, false>(v, v);
            }
        }
        for (int R = 1; R <= L.Rmax; R++) {
            // the buffer that the inner products of two steps ago were taken
            // from: the barrier of the last step has seen them done
            double *b0 = sm + par * buf;
            par ^= 1;
            if (on) {
#pragma unroll
                for (int a = 0; a < NC; a++) {
                    CX<double> n[NC];
#pragma unroll
                    for (int b = 0; b < NC; b++) {
                        double re = 0.0, im = 0.0;
#pragma unroll
                        for (int q = 0; q < NC; q++) {
                            re = fma(m.m[a][q].re, k.m[q][b].re, re);
                            re = fma(-m.m[a][q].im, k.m[q][b].im, re);
                            im = fma(m.m[a][q].re, k.m[q][b].im, im);
                            im = fma(m.m[a][q].im, k.m[q][b].re, im);
                        }
                        n[b] = { re, im };
                    }
#pragma unroll
                    for (int b = 0; b < NC; b++) m.m[a][b] = n[b];
                }
                if (R < L.Rmax) {
                    if (++x == ni) { x = 0; at -= (size_t)(ni - 1) * step; } else at += step;
                    k = load_soa<NC>(at);
                }
            }
            if (mine) {
#pragma unroll
                for (int a = 0; a < NC; a++)
#pragma unroll
                    for (int b = 0; b < NC; b++) {
                        b0[s + (2 * (a * NC + b)) * ss] = m.m[a][b].re;
                        b0[s + (2 * (a * NC + b) + 1) * ss] = m.m[a][b].im;
                    }
            }
            __syncthreads();
            double acc[TM];
#pragma unroll
            for (int T = 0; T < TM; T++) acc[T] = 0.0;
            if (item) {
                double e[kTB];
#pragma unroll
                for (int j = 0; j < kTB; j++) e[j] = b0[pe + j];
#pragma unroll
                for (int o = 1; o < kTB + TM; o++) {
                    const double d = b0[pd + o];
#pragma unroll
                    for (int T = 1; T <= TM; T++)
                        if (o - T >= 0 && o - T < kTB) acc[T - 1] = fma(e[o - T], d, acc[T - 1]);
                }
            }
            // sums over the warp, scattered: lane l ends with T = l / (32 / TM) + 1
            int off = 16;
#pragma unroll
            for (int n = TM; n > 1; n >>= 1, off >>= 1) {
                const bool up = lane & off;
#pragma unroll
                for (int j = 0; j < n / 2; j++) {
                    const double send = up ? acc[j] : acc[j + n / 2], keep = up ? acc[j + n / 2] : acc[j];
                    acc[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
            }
#pragma unroll
            for (int o = 16 / TM; o > 0; o >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
            if (adds) sa[(R - 1) * L.Tmax] += acc[0];
        }
    }
    __syncthreads();
    for (int k = tid; k < nl; k += blockDim.x) {
        double a = slots[(size_t)blockIdx.x * nl + k];
        for (int w = 0; w < nw; w++) a += sacc[w * nl + k];
        slots[(size_t)blockIdx.x * nl + k] = a;
    }
}

// out[loop] = the blocks' sums in a fixed order, one warp per loop
__global__ void __launch_bounds__(128) k_loops_sum(const double *slots, int nslots, int nl, double *out)
{
    const int q = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (q >= nl) return;
    double a = 0.0;
    for (int b = lane; b < nslots; b += 32) a += slots[(size_t)b * nl + q];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) out[q] = a;
}


int padded_nt(const Geom &G, int Tmax) { return (G.n[3] + Tmax + 7) / 8 * 8; }
size_t column_bytes(const Geom &G, int group, int Tmax)
{
    return (size_t)3 * 2 * group * group * sizeof(double) * padded_nt(G, Tmax);
}

template <int NC, int TM>
cudaError_t loops(const Lines &L, double *slots, cudaStream_t s)
{
    // windows of t0 and columns such that both the matrices (2 TW + Tmax a
    // column) and the inner products (NR TWp / 8) have a thread each
    constexpr int NR = 2 * NC * NC;
    const int nt = L.G.n[3], TW = nt <= 64 ? nt : 48, nwin = (nt + TW - 1) / TW;
    const int per = std::max(2 * TW + L.Tmax, NR * ((TW + kTB - 1) / kTB));
    const int cols = kLoopThreads / per;
    const int threads = (cols * per + 31) / 32 * 32;
    const int TWp = (TW + kTB - 1) / kTB * kTB;
    const size_t smem = sizeof(double) * ((size_t)2 * NR * cols * (((TWp + TM) | 1) + (TWp | 1)) +
                                          (size_t)(threads / 32) * L.Rmax * L.Tmax);
    cudaError_t e = cudaFuncSetAttribute(k_loops<NC, TM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const uint32_t units = (L.ncol + cols - 1) / cols * (uint32_t)nwin;
    const int grid = (int)(units < (uint32_t)kSlots ? units : (uint32_t)kSlots);
    k_loops<NC, TM><<<grid, threads, smem, s>>>(L, cols, TW, nwin, slots);
    return cudaGetLastError();
}

template <int NC, typename Real>
cudaError_t wilson_lines(const Field<Real> &U, const Geom &G, int Rmax, int Tmax, const double *params, int twist,
                         double *const parts[2], size_t part_bytes, double *out, cudaStream_t s)
{
    const size_t head = slots_doubles(Rmax, Tmax);      // left free in the second part
    double *slots = parts[0];
    Lines L;
    L.G = G;
    L.Vs = (uint32_t)G.n[0] * G.n[1] * G.n[2];
    L.Rmax = Rmax;
    L.Tmax = Tmax;
    L.NT1 = padded_nt(G, Tmax);
    const uint32_t total = 3 * L.Vs;
    const size_t column = (size_t)2 * NC * NC * L.NT1;
    const uint32_t maxcol = (uint32_t)std::min<size_t>((part_bytes / sizeof(double) - head) / (3 * column), total);
    L.V = parts[0] + head;
    L.K = L.V + maxcol * column;
    L.F = L.K + maxcol * column;
    double *flag = out + Rmax * Tmax;
    cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(double), s);
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(slots, 0, slots_doubles(Rmax, Tmax) * sizeof(double), s)) != cudaSuccess) return e;
    // whole lines from column g on, as many as a part holds (they may run on
    // from one direction's lines to the next one's)
    auto part_end = [&](uint32_t g) {
        const uint32_t g0 = g;
        while (g < total) {
            const int i = (int)(g / L.Vs);
            const uint32_t ni = (uint32_t)G.n[i], room = maxcol - (g - g0), left = (uint32_t)(i + 1) * L.Vs - g;
            const uint32_t take = std::min(room / ni * ni, left);
            g += take;
            if (take < left) break;
        }
        return g;
    };
    for (uint32_t g0 = 0; g0 < total;) {
        const uint32_t gc = part_end(g0), g1 = parts[1] ? part_end(gc) : gc;
        L.g0 = g0;
        L.ncol = g1 - g0;
        L.cut = gc - g0;
        L.jump = parts[1] ? parts[1] - parts[0] - (ptrdiff_t)(L.cut * column) : 0;
        const int nwork = std::min(L.NT1 / kSeg, kTLSegs<NC, Real>);
        k_time_lines<NC, Real><<<(L.ncol + kTLCols - 1) / kTLCols, kTLCols * NC * nwork, 0, s>>>(U, L);
        const unsigned nb = (unsigned)(((size_t)L.ncol * L.NT1 + 127) / 128);
        if (twist) k_line_links<NC, Real, true><<<nb, 128, 0, s>>>(U, L, params, twist, flag);
        else k_line_links<NC, Real, false><<<nb, 128, 0, s>>>(U, L, params, twist, flag);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if (Tmax <= 4) e = loops<NC, 4>(L, slots, s);
        else if (Tmax <= 8) e = loops<NC, 8>(L, slots, s);
        else e = loops<NC, 16>(L, slots, s);
        if (e != cudaSuccess) return e;
        g0 = g1;
    }
    k_loops_sum<<<(Rmax * Tmax + 3) / 4, 128, 0, s>>>(slots, kSlots, Rmax * Tmax, out);
    return cudaGetLastError();
}

}  // namespace

// the sums of the blocks and the arrays of a chunk (read from L2 then), in one
// part where the lattice needs no more, else in two: 0 when one line does
// not fit a part
size_t wilson_lines_scratch(const Geom &G, int group, int Rmax, int Tmax, int &parts)
{
    const size_t col = column_bytes(G, group, Tmax), slots = slots_doubles(Rmax, Tmax) * sizeof(double);
    const size_t line = col * std::max(G.n[0], std::max(G.n[1], G.n[2]));
    const size_t all = slots + col * 3 * ((size_t)G.n[0] * G.n[1] * G.n[2]);
    parts = all > kScratchPart ? 2 : 1;
    return slots + line > kScratchPart ? 0 : std::min(kScratchPart, all);
}

cudaError_t launch_wilson_lines(const Geom &G, const void *links, int group, int prec, int Rmax, int Tmax,
                                const double *params, int twist, double *const parts[2], size_t part_bytes,
                                double *out, cudaStream_t s)
{
    if (prec) {
        Field<double> U{ (double4 *)links, G.pstride };
        return group == 3 ? wilson_lines<3, double>(U, G, Rmax, Tmax, params, twist, parts, part_bytes, out, s)
                          : wilson_lines<2, double>(U, G, Rmax, Tmax, params, twist, parts, part_bytes, out, s);
    }
    Field<float> U{ (float4 *)links, G.pstride };
    return group == 3 ? wilson_lines<3, float>(U, G, Rmax, Tmax, params, twist, parts, part_bytes, out, s)
                      : wilson_lines<2, float>(U, G, Rmax, Tmax, params, twist, parts, part_bytes, out, s);
}

}  // namespace qg
