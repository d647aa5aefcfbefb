// qg_update.cuh -- the checkerboard phase kernel: one thread per link of
// one (parity, direction) class; staple from the 18 neighbouring links,
// then Cabibbo-Marinari heatbath / overrelaxation (SU(3)) or Kennedy-
// Pendleton heatbath / reflection (SU(2)), stored in place.
// Restates update_{even,odd}_{X,Y,Z,T} (SU(N)/suncl/suncl.cl:399-975),
// lattice_staple_3 / lattice_staple_2 (su3_update_cl.cl:341-565,
// su2_update_cl.cl:206-431).
#pragma once
#include "qg_internal.h"
#include "qg_pair.cuh"

namespace qg {

template <typename Real>
struct Twist {
    int on;
    Real phi, omega;
    int xlast;
};

// Staple links by the read-only path (ld.global.nc) where the field allows it
// (RO).  It is defined only for data that nothing writes while the kernel is
// resident, so a kernel that takes it runs one phase and starts after the
// phase before has ended: k_phase is never a programmatic dependent
// (k_phase_split, which is, and the persistent half-sweep read with ordinary
// loads).  Ordinary loads and the early launch are not the faster pair: 32^4
// SU(3) FP64 heatbath 159 -> 173 us, FP32 overrelaxation in shape 1 50.5 -> 55.4.
template <typename Real, bool RO>
__device__ __forceinline__ G3<Real> load3t(const Field<Real, RO> &U, int dir, uint32_t e, int xc, const Twist<Real> &tw)
{
    G3<Real> m = U.ldg3(dir, e);
    if (tw.on && dir == 1 && xc == tw.xlast) m = twist3(m, tw.phi, tw.omega);
    return m;
}
template <typename Real, bool RO>
__device__ __forceinline__ R4<Real> load2t(const Field<Real, RO> &U, int dir, uint32_t e, int xc, const Twist<Real> &tw)
{
    R4<Real> m = U.ldg2(dir, e);
    if (tw.on && dir == 1 && xc == tw.xlast) {
        R4<Real> om = { RC<Real>::cs(tw.phi / 2), 0, RC<Real>::sn(tw.phi / 2), 0 };
        m = times2(om, m);
    }
    return m;
}

// the reference's fixed plane order: mu=X: Y,Z,T; Y: X,Z,T; Z: Y,X,T; T: Y,Z,X
__host__ __device__ constexpr int nu_of(int mu, int i)
{
    return (i == 0) ? (mu == 1 ? 0 : 1) : (i == 1) ? (mu == 2 ? 0 : 2) : (mu == 3 ? 0 : 3);
}

// Neighbour offsets in checkerboard half-index space.  With N2 even the
// half index of a site is h = (y>>1) + (N2/2)(z + N3 t + N3 N4 x), so a
// shift along one direction changes h by an amount that depends only on
// that direction's coordinate (and y's parity), and two shifts along
// different directions add: h(x - nu + mu) = h + dm[nu] + dp[mu].
struct Nbr {
    int32_t dp[4], dm[4];
    int x, xp, xm;          // x coordinates of the site and of its x neighbours
};

__device__ __forceinline__ Nbr neighbours(const Geom &G, const Crd &c)
{
    Nbr n;
    const int32_t Y2 = G.n[1] >> 1;
    const int32_t sz = Y2, st = Y2 * G.n[2], sx = st * G.n[3];
    // y: y+1 changes y>>1 by (y odd); the wrap from N2-1 to 0 by -(Y2-1)
    n.dp[1] = (c.y == G.n[1] - 1) ? -(Y2 - 1) : (c.y & 1);
    n.dm[1] = (c.y == 0) ? (Y2 - 1) : -((c.y & 1) ^ 1);
    n.dp[2] = (c.z == G.n[2] - 1) ? -sz * (G.n[2] - 1) : sz;
    n.dm[2] = (c.z == 0) ? sz * (G.n[2] - 1) : -sz;
    n.dp[3] = (c.t == G.n[3] - 1) ? -st * (G.n[3] - 1) : st;
    n.dm[3] = (c.t == 0) ? st * (G.n[3] - 1) : -st;
    n.dp[0] = (c.x == G.n[0] - 1) ? -sx * (G.n[0] - 1) : sx;
    n.dm[0] = (c.x == 0) ? sx * (G.n[0] - 1) : -sx;
    n.x = c.x;
    n.xp = (c.x == G.n[0] - 1) ? 0 : c.x + 1;
    n.xm = (c.x == 0) ? G.n[0] - 1 : c.x - 1;
    return n;
}

// staple of U_mu(x), lattice_staple_3 (su3_update_cl.cl:341-565): per
// plane nu the forward term U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+ and the
// backward term U_nu(x-nu+mu)^+ U_mu(x-nu)^+ U_nu(x-nu), summed as
// st = f0 + b0; st = b_i + (st + f_i)
template <int mu, typename Real, bool RO>
__device__ __forceinline__ M3<Real> staple3(const Field<Real, RO> &U, const Geom &G, uint32_t t, const Nbr &n, int p,
                                           const Twist<Real> &tw)
{
    const uint32_t own = (uint32_t)p * G.cb + t, opp = (uint32_t)(p ^ 1) * G.cb + t;
    const int xmu = (mu == 0) ? n.xp : n.x;
    M3<Real> st, s2;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int nu = nu_of(mu, i);
        const int xnp = (nu == 0) ? n.xp : n.x, xnm = (nu == 0) ? n.xm : n.x;
        const int xnmmu = (nu == 0) ? n.xm : xmu;
        M3<Real> fw = staple_fwd3(load3t(U, nu, opp + n.dp[mu], xmu, tw), load3t(U, mu, opp + n.dp[nu], xnp, tw),
                                  load3t(U, nu, own, n.x, tw));
        M3<Real> bw = staple_bwd3(load3t(U, nu, own + n.dm[nu] + n.dp[mu], xnmmu, tw),
                                  load3t(U, mu, opp + n.dm[nu], xnm, tw), load3t(U, nu, opp + n.dm[nu], xnm, tw));
        if (i == 0) {
            add3(st, fw, bw);
        } else {
            add3(s2, st, fw);
            add3(st, bw, s2);
        }
    }
    return st;
}

template <int mu, typename Real, bool RO>
__device__ __forceinline__ S2<Real> staple2(const Field<Real, RO> &U, const Geom &G, uint32_t t, const Nbr &n, int p,
                                           const Twist<Real> &tw)
{
    const uint32_t own = (uint32_t)p * G.cb + t, opp = (uint32_t)(p ^ 1) * G.cb + t;
    const int xmu = (mu == 0) ? n.xp : n.x;
    S2<Real> st, s2;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int nu = nu_of(mu, i);
        const int xnp = (nu == 0) ? n.xp : n.x, xnm = (nu == 0) ? n.xm : n.x;
        const int xnmmu = (nu == 0) ? n.xm : xmu;
        S2<Real> fw = staple_fwd2(load2t(U, nu, opp + n.dp[mu], xmu, tw), load2t(U, mu, opp + n.dp[nu], xnp, tw),
                                  load2t(U, nu, own, n.x, tw));
        S2<Real> bw = staple_bwd2(load2t(U, nu, own + n.dm[nu] + n.dp[mu], xnmmu, tw),
                                  load2t(U, mu, opp + n.dm[nu], xnm, tw), load2t(U, nu, opp + n.dm[nu], xnm, tw));
        if (i == 0) {
            st = add2(fw, bw);
        } else {
            s2 = add2(st, fw);
            st = add2(bw, s2);
        }
    }
    return st;
}

// ------------------------------------------ staple links through shared memory
// The staged form of staple3 (SU(3), FP32 links): each staple term's three
// links (nine 16-byte plane entries per thread) are copied global -> shared
// with cp.async two terms ahead of their use, so a warp keeps the next
// term's loads in flight while it multiplies the current one instead of
// holding them in registers.  A thread only reads back what it copied
// itself, so no block barrier is needed; the arithmetic is staple3's.
constexpr int kPhaseBlock = 128;

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// slots of 16 bytes x kPhaseBlock threads: two term buffers of 9 slots
// (3 links x 3 planes); the updated link itself goes into the forward
// buffer once the last forward term has been read (36 KB per block, so
// five blocks fit an SM with room to spare)
constexpr int kTermSlots = 9, kOwnSlot = 0, kStageSlots = 2 * kTermSlots;
using StageBuf = float4[kStageSlots][kPhaseBlock];

__device__ __forceinline__ void stage_link(const Field<float> &U, int dir, uint32_t e, StageBuf &sb, int slot)
{
#pragma unroll
    for (int c = 0; c < 3; c++) cp_async16(&sb[slot + c][threadIdx.x], U.p + (size_t)(dir + 4 * c) * U.pstride + e);
}
__device__ __forceinline__ G3<float> unstage_link(const StageBuf &sb, int slot)
{
    G3<float> m;
    float4 a = sb[slot][threadIdx.x], b = sb[slot + 1][threadIdx.x], d = sb[slot + 2][threadIdx.x];
    m.uv1 = { a.x, a.y, a.z, a.w };
    m.uv2 = { b.x, b.y, b.z, b.w };
    m.uv3 = { d.x, d.y, d.z, d.w };
    return m;
}

// the plane-nu neighbour offsets for a runtime nu (selects, no local memory)
__device__ __forceinline__ int32_t pick4(const int32_t (&a)[4], int k)
{
    return k == 0 ? a[0] : k == 1 ? a[1] : k == 2 ? a[2] : a[3];
}

// staple3 with staged loads, as a loop over the three planes (one copy of
// the forward and backward term code, so the kernel's instruction stream
// stays small); also brings in the updated link U_mu(x).  Term buffer 0
// holds the forward term of the plane, buffer 1 the backward term; the
// next plane's copies are issued as soon as a buffer has been read; on the
// last plane the forward buffer receives U_mu(x) instead, so its copy runs
// under the last backward term.  Every iteration commits one group per
// buffer (the last backward group is empty) so that wait_group 1 always
// means "this buffer has landed".
template <int mu>
__device__ __forceinline__ M3<float> staple3_staged(const Field<float> &U, const Geom &G, uint32_t t, const Nbr &n,
                                                   int p, const Twist<float> &tw, StageBuf &sb, G3<float> &m0)
{
    const uint32_t own = (uint32_t)p * G.cb + t, opp = (uint32_t)(p ^ 1) * G.cb + t;
    const int xmu = (mu == 0) ? n.xp : n.x;
    auto fwd_copy = [&](int nu) {
        stage_link(U, nu, opp + n.dp[mu], sb, 0);
        stage_link(U, mu, opp + pick4(n.dp, nu), sb, 3);
        stage_link(U, nu, own, sb, 6);
    };
    auto bwd_copy = [&](int nu) {
        const int32_t dmn = pick4(n.dm, nu);
        stage_link(U, nu, own + dmn + n.dp[mu], sb, kTermSlots);
        stage_link(U, mu, opp + dmn, sb, kTermSlots + 3);
        stage_link(U, nu, opp + dmn, sb, kTermSlots + 6);
    };
    auto get = [&](int slot, int dir, int xc) {
        G3<float> m = unstage_link(sb, slot);
        if (tw.on && dir == 1 && xc == tw.xlast) m = twist3(m, tw.phi, tw.omega);
        return m;
    };
    fwd_copy(nu_of(mu, 0));
    cp_async_commit();
    bwd_copy(nu_of(mu, 0));
    cp_async_commit();
    MR3 st, s2;
#pragma unroll 1
    for (int i = 0; i < 3; i++) {
        const int nu = nu_of(mu, i);
        const int xnp = (nu == 0) ? n.xp : n.x, xnm = (nu == 0) ? n.xm : n.x;
        const int xnmmu = (nu == 0) ? n.xm : xmu;
        cp_async_wait<1>();
        MR3 fw = staple_fwd3_rows(get(0, nu, xmu), get(3, mu, xnp), get(6, nu, n.x));
        if (i < 2)
            fwd_copy(nu_of(mu, i + 1));
        else
            stage_link(U, mu, own, sb, kOwnSlot);
        cp_async_commit();
        cp_async_wait<1>();
        MR3 bw = staple_bwd3_rows(get(kTermSlots, nu, xnmmu), get(kTermSlots + 3, mu, xnm),
                                  get(kTermSlots + 6, nu, xnm));
        if (i < 2) bwd_copy(nu_of(mu, i + 1));
        cp_async_commit();
        if (i == 0) {
            mr_add(st, fw, bw);
        } else {
            mr_add(s2, st, fw);
            mr_add(st, bw, s2);
        }
    }
    cp_async_wait<0>();
    m0 = unstage_link(sb, kOwnSlot);
    return mr_unpack(st);
}

__device__ __forceinline__ void grid_dependents_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// PRN source of thread t (PMODE 0 = RANLUX buffer, 1 = Philox, 2 = gid)
template <typename Real, int PMODE> struct PrnOf;
template <typename Real> struct PrnOf<Real, 0> {
    using T = PrnBuffer<Real>;
    __device__ static T make(const PhaseArgs &A, uint32_t t, uint32_t, uint64_t, const Geom &)
    {
        T p; p.prns = A.prns; p.idx = t; p.step = A.prngstep; return p;
    }
};
template <typename Real> struct PrnOf<Real, 1> {
    using T = PrnPhilox<Real>;
    __device__ static T make(const PhaseArgs &A, uint32_t t, uint32_t, uint64_t phase, const Geom &)
    {
        T p; p.key = A.key; p.t = (uint32_t)((int32_t)t + A.t_prn); p.k = 0; p.plo = (uint32_t)phase;
        p.phi = (uint32_t)(phase >> 32); return p;
    }
};
template <typename Real> struct PrnOf<Real, 2> {
    using T = PrnGid<Real>;
    __device__ static T make(const PhaseArgs &A, uint32_t, uint32_t site, uint64_t, const Geom &G)
    {
        T p; p.g = (double)(float)site; p.V = (double)G.V; p.nhit = A.nhit; return p;
    }
};

// the SU(2) group's update of link m0 with staple st: a Kennedy-Pendleton
// draw (m0 stays when no try is accepted) or the reflection
template <typename Real, bool OR, class Prn>
__device__ __forceinline__ R4<Real> su2_update(const S2<Real> &st, const R4<Real> &m0, Real beta, Prn &prn, int nhit)
{
    if (!OR) {
        S2<Real> a = st;
        if (kp_step<Real, false>(a, beta, prn, nhit)) return { a.u1.re, a.u2.re, a.u1.im, a.u2.im };
        return m0;
    }
    Real Mx = st.u1.re + st.v2.re, My = st.u1.im - st.v2.im;
    Real Mz = st.u2.re - st.v1.re, Mw = st.u2.im + st.v1.im;
    Real n2 = Mx * Mx;
    n2 = FMA(My, My, n2); n2 = FMA(Mz, Mz, n2); n2 = FMA(Mw, Mw, n2);
    Real id = (Real)1 / RC<Real>::sq(n2);
    R4<Real> aH = { Mx * id, -Mz * id, -My * id, -Mw * id };
    return times2(times2(aH, herm2(m0)), aH);
}

// MINB: minimum resident blocks of 128 threads per SM asked of the
// compiler (0 = its own register choice); the launch shapes the tuner picks
// The update of link U_mu(x) for thread t of a (parity, mu) phase: the
// body of update_{even,odd}_{X,Y,Z,T}.  STAGED: staple links through
// shared memory (staple3_staged; SU(3) FP32 links).
// TW: twisted boundaries possible (the launch has A.twist set); without it
// every twist test folds away at compile time (4 % of the phase's time)
// sb: the block's staging buffer (STAGED; declared by the kernel, so that a
// kernel running several directions holds one)
template <int NC, typename Real, int PMODE, bool OR, int mu, bool STAGED, bool TW = false, bool RO = true>
__device__ __forceinline__ void phase_site(const Field<Real, RO> &U, const Geom &G, const PhaseArgs &A, uint32_t t,
                                           StageBuf *sb)
{
    const int p = A.parity;
    Crd c = lex2crd(G, 2 * t);
    if (parity_of(c) != p) c.y += 1;                 // lattice_{even,odd}_gid
    const uint32_t site = 2 * t + (uint32_t)(c.y & 1);
    const uint32_t e0 = (uint32_t)p * G.cb + t;
    const Nbr nb = neighbours(G, c);
    Twist<Real> tw;
    tw.on = TW ? A.twist : 0;
    tw.xlast = G.n[0] - 1;
    tw.phi = (Real)(float)A.params[1]; tw.omega = (Real)(float)A.params[2];
    if (sizeof(Real) == 8) { tw.phi = (Real)A.params[1]; tw.omega = (Real)A.params[2]; }
    const Real beta = (Real)A.params[0];            // lattice_parameters[0] = BETA/N
    const uint64_t phase = (PMODE == 1) ? (*A.phase_base + A.phase_offset) : 0;
    auto prn = PrnOf<Real, PMODE>::make(A, t, site, phase, G);
    if (NC == 3) {
        G3<Real> m0;
        M3<Real> st;
        if constexpr (STAGED) {
            st = staple3_staged<mu>(Field<Real>{ U.p, U.pstride }, G, t, nb, p, tw, *sb, m0);
        } else {
            m0 = U.ld3(mu, e0);
            st = staple3<mu>(U, G, t, nb, p, tw);
        }
        if (tw.on && mu == 1 && c.x == tw.xlast) m0 = twist3(m0, tw.phi, tw.omega);
        G3<Real> mU;
        if constexpr (STAGED && OR)
            mU = cm3_or_rows(st, m0, A.nhitpar);
        else
            mU = cm3<Real, OR, decltype(prn), STAGED && !OR>(st, m0, beta, prn, A.nhit, A.nhitpar);
        U.st3(mu, e0, mU);
    } else {
        R4<Real> m0 = U.ld2(mu, e0);
        if (tw.on && mu == 1 && c.x == tw.xlast) {
            R4<Real> om = { RC<Real>::cs(tw.phi / 2), 0, RC<Real>::sn(tw.phi / 2), 0 };
            m0 = times2(om, m0);
        }
        S2<Real> st = staple2<mu>(U, G, t, nb, p, tw);
        U.st2(mu, e0, su2_update<Real, OR>(st, m0, beta, prn, A.nhit));
    }
}

template <int NC, typename Real, int PMODE, bool OR, int mu, int MINB, bool STAGED, bool TW>
__global__ void __launch_bounds__(kPhaseBlock, MINB) k_phase(Field<Real> U, Geom G, PhaseArgs A)
{
    const uint32_t t = A.t_begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= A.t_end) return;
    if constexpr (STAGED) {
        __shared__ __align__(16) StageBuf sb;
        phase_site<NC, Real, PMODE, OR, mu, STAGED, TW>(U, G, A, t, &sb);
    } else {
        phase_site<NC, Real, PMODE, OR, mu, STAGED, TW>(U, G, A, t, nullptr);
    }
}

// Overrelaxation of two links per thread (t and t + ceil(half/2)) with the
// packed FP32 algebra of qg_pair.cuh: each lane performs the scalar
// kernel's operations in the same order (bit-identical results) while one
// FFMA2 issue serves both links.  SU(3), FP32 links, periodic boundaries;
// the running staple sum is kept as s2 = st + f_i (f_0 alone for the first
// plane), then st = b_i + s2 -- the scalar order, with the first sum
// written b_0 + f_0 (addition commutes exactly).
template <int mu>
__global__ void __launch_bounds__(kPhaseBlock, 1) k_phase_or_pair(Field<float> U, Geom G, PhaseArgs A)
{
    const uint32_t H = (G.half + 1) >> 1;
    const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (t0 >= H) return;
    uint32_t t1 = t0 + H;
    const bool two = t1 < G.half;
    if (!two) t1 = t0;
    const int p = A.parity;
    Crd c0 = lex2crd(G, 2 * t0);
    if (parity_of(c0) != p) c0.y += 1;
    Crd c1 = lex2crd(G, 2 * t1);
    if (parity_of(c1) != p) c1.y += 1;
    const Nbr n0 = neighbours(G, c0), n1 = neighbours(G, c1);
    const uint32_t own0 = (uint32_t)p * G.cb + t0, opp0 = (uint32_t)(p ^ 1) * G.cb + t0;
    const uint32_t own1 = (uint32_t)p * G.cb + t1, opp1 = (uint32_t)(p ^ 1) * G.cb + t1;
    M32 st, s2;
#pragma unroll 1
    for (int i = 0; i < 3; i++) {
        const int nu = nu_of(mu, i);
        const int32_t dpn0 = pick4(n0.dp, nu), dpn1 = pick4(n1.dp, nu);
        const int32_t dmn0 = pick4(n0.dm, nu), dmn1 = pick4(n1.dm, nu);
        {
            M32 fw = pstaple_fwd3(gpair(U.ldg3(nu, opp0 + n0.dp[mu]), U.ldg3(nu, opp1 + n1.dp[mu])),
                                  gpair(U.ldg3(mu, opp0 + dpn0), U.ldg3(mu, opp1 + dpn1)),
                                  gpair(U.ldg3(nu, own0), U.ldg3(nu, own1)));
            if (i == 0) s2 = fw;
            else padd3(s2, st, fw);
        }
        M32 bw = pstaple_bwd3(gpair(U.ldg3(nu, own0 + dmn0 + n0.dp[mu]), U.ldg3(nu, own1 + dmn1 + n1.dp[mu])),
                              gpair(U.ldg3(mu, opp0 + dmn0), U.ldg3(mu, opp1 + dmn1)),
                              gpair(U.ldg3(nu, opp0 + dmn0), U.ldg3(nu, opp1 + dmn1)));
        padd3(st, bw, s2);
    }
    const G32 r = pcm3_or(st, gpair(U.ld3(mu, own0), U.ld3(mu, own1)), A.nhitpar);
    G3<float> r0, r1;
    gsplit(r, r0, r1);
    U.st3(mu, own0, r0);
    if (two) U.st3(mu, own1, r1);
}

// -------------------------------------------------- small lattices
// A phase of few links is bound by one link's chain of latencies (loads, six
// staple terms, three subgroup draws) and the launch, not by throughput.  SP = 6
// or 3 warps share 32 links here: each computes one staple term (warp w: plane
// w / 2, forward or backward) and its share of the sums, and the first one
// updates the links; in a heatbath the six also evaluate the functions of
// the first kSplitQuads random quads (logarithms, sines) ahead, so that the
// updating warp finds them in shared memory (it computes them itself for
// the rare later quads).  Operations and their order per value are those of
// phase_site.  In a sweep's graph the launches are programmatic dependents:
// a phase's indices and random numbers are computed under the end of the
// phase before it.  A phase lets the next one start before it waits itself, so
// a third may be resident while the first still writes; each waits for the end
// of the one before, which ends after its own wait, and reads links after that
// with ordinary loads only.
constexpr int kSplitQuads = 6;

// the functions of one quad that a Kennedy-Pendleton step uses, as a try
// (num = log(1-x) + cos^2(2 pi y) log(1-z), w2 = w^2) and as a direction
template <typename Real> struct QuadTry { double num; Real w2; };
template <typename Real> struct QuadDir { Real costh, sinth, sinphi, cosphi; };
template <typename Real>
__device__ __forceinline__ QuadTry<Real> quad_try(const R4<Real> &rnd)
{
    QuadTry<Real> q;
    Real cosrnd = RC<Real>::cs(RC<Real>::PI2 * rnd.y);
    double lx = qg_log(1.0 - (double)rnd.x), lz = qg_log(1.0 - (double)rnd.z);
    q.num = FMA((double)(cosrnd * cosrnd), lz, lx);
    q.w2 = rnd.w * rnd.w;
    return q;
}
template <typename Real>
__device__ __forceinline__ QuadDir<Real> quad_dir(const R4<Real> &rnd)
{
    QuadDir<Real> q;
    q.costh = (Real)FMA(2.0, (double)rnd.x, -1.0);
    q.sinth = (Real)sqrt(1.0 - (double)(q.costh * q.costh));
    Real phi = RC<Real>::PI2 * rnd.y;
    q.sinphi = RC<Real>::sn(phi);
    q.cosphi = RC<Real>::cs(phi);
    return q;
}
template <typename Real> struct QuadTable {
    QuadTry<Real> t[kSplitQuads][32];
    QuadDir<Real> d[kSplitQuads][32];
};
// quad k of the link's stream: a table entry, or computed from the source
template <typename Real, class Src> struct PrnTable {
    static constexpr bool GID = false;
    Src src;
    const QuadTable<Real> *tab;
    int k, lane;
    __device__ __forceinline__ R4<Real> quad(int n) { Src s = src; s.seek(n); return s.next(); }
    __device__ __forceinline__ QuadTry<Real> try_vals()
    {
        const int n = k++;
        return n < kSplitQuads ? tab->t[n][lane] : quad_try(quad(n));
    }
    __device__ __forceinline__ QuadDir<Real> dir_vals()
    {
        const int n = k++;
        return n < kSplitQuads ? tab->d[n][lane] : quad_dir(quad(n));
    }
    __device__ __forceinline__ void skip() { k++; }
};

// kp_step with the quads' functions at hand
template <typename Real, bool SU3PATH, class Src>
__device__ __forceinline__ bool kp_step(S2<Real> &a, Real beta, PrnTable<Real, Src> &prn, int nhit)
{
    R4<Real> aH;
    aH.x =  (a.u1.re + a.v2.re);
    aH.z = -(a.u1.im - a.v2.im);
    aH.y = -(a.u2.re - a.v1.re);
    aH.w = -(a.u2.im + a.v1.im);
    Real n2 = aH.x * aH.x;
    if (SU3PATH) {
        n2 = FMA(aH.y, aH.y, n2); n2 = FMA(aH.z, aH.z, n2); n2 = FMA(aH.w, aH.w, n2);
    } else {
        n2 = FMA(aH.z, aH.z, n2); n2 = FMA(aH.y, aH.y, n2); n2 = FMA(aH.w, aH.w, n2);
    }
    const Real det = RC<Real>::sq(n2);
    const Real id = (Real)1 / det;
    aH.x *= id; aH.z *= id; aH.y *= id; aH.w *= id;
    const Real bdet = beta * det;
    Real delta = 0;
    bool flag = false;
    for (int i = 0; i < nhit && !flag; i++) {
        const QuadTry<Real> q = prn.try_vals();
        delta = (Real)(-q.num / (double)bdet);
        if ((double)q.w2 <= FMA(-0.5, (double)delta, 1.0)) flag = true;
    }
    if (flag) {
        const QuadDir<Real> q = prn.dir_vals();
        Real cosal = (Real)(1.0 - (double)delta);
        Real sinal = (Real)sqrt(1.0 - (double)(cosal * cosal));
        R4<Real> c;
        c.x = cosal;
        c.z = sinal * q.costh;
        c.y = sinal * q.sinth * q.sinphi;
        c.w = sinal * q.sinth * q.cosphi;
        a = rec2(times2(c, aH));
        return true;
    }
    if (SU3PATH) {
        a.u1 = { (Real)1, (Real)0 }; a.u2 = { (Real)0, (Real)0 };
        a.v1 = { (Real)0, (Real)0 }; a.v2 = { (Real)1, (Real)0 };
        prn.skip();
    }
    return false;
}

template <int NC, typename Real, int PMODE, bool OR, int mu, int SP>
__global__ void __launch_bounds__(32 * SP) k_phase_split(Field<Real> U, Geom G, PhaseArgs A)
{
    constexpr int NT = NC == 3 ? 18 : 4;                // numbers of a term (SU(2): the quaternion)
    __shared__ Real term[6][NT][32];
    __shared__ QuadTable<Real> tab;                     // heatbath only
    grid_dependents_may_start();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t t = A.t_begin + blockIdx.x * 32 + lane;
    const bool on = t < A.t_end;
    const int p = A.parity;
    Crd c = lex2crd(G, 2 * (on ? t : A.t_begin));
    if (parity_of(c) != p) c.y += 1;
    const uint32_t site = 2 * t + (uint32_t)(c.y & 1);
    const Nbr n = neighbours(G, c);
    const uint32_t own = (uint32_t)p * G.cb + t, opp = (uint32_t)(p ^ 1) * G.cb + t;
    using PS = PrnOf<Real, PMODE>;
    typename PS::T src;
    auto fill = [&]() {
        for (int k = w; k < kSplitQuads; k += SP) {
            auto s = src;
            s.seek(k);
            const R4<Real> q = s.next();
            tab.t[k][lane] = quad_try(q);
            tab.d[k][lane] = quad_dir(q);
        }
    };
    if constexpr (!OR) {
        src = PS::make(A, t, site, PMODE == 1 ? *A.phase_base + A.phase_offset : 0, G);
        if (PMODE == 1) fill();                         // no memory of earlier phases is read
    }
    grid_dependency_wait();
    const Real beta = (Real)A.params[0];
    G3<Real> m0;
    R4<Real> q0;
    if (on) {
        if (w == 0) {
            if constexpr (NC == 3) m0 = U.ld3(mu, own);
            else q0 = U.ld2(mu, own);
        }
#pragma unroll
        for (int j = 0; j < 6 / SP; j++) {
            // forward U_nu(x+mu) U_mu(x+nu)^+ U_nu(x)^+, backward U_nu(x-nu+mu)^+ U_mu(x-nu)^+ U_nu(x-nu)
            const int k = w * (6 / SP) + j, nu = nu_of(mu, k >> 1);
            const bool bwd = k & 1;
            const int32_t d = bwd ? pick4(n.dm, nu) : pick4(n.dp, nu);
            const uint32_t ea = bwd ? own + d + n.dp[mu] : opp + n.dp[mu], eb = opp + d, ec = bwd ? opp + d : own;
            if constexpr (NC == 3) {
                const G3<Real> ga = U.ld3(nu, ea), gb = U.ld3(mu, eb), gc = U.ld3(nu, ec);
                M3<Real> T;
                if constexpr (sizeof(Real) == 4)
                    T = mr_unpack(bwd ? staple_bwd3_rows(ga, gb, gc) : staple_fwd3_rows(ga, gb, gc));
                else
                    T = bwd ? staple_bwd3(ga, gb, gc) : staple_fwd3(ga, gb, gc);
#pragma unroll
                for (int i = 0; i < 9; i++) {
                    term[k][2 * i][lane] = T.m[i / 3][i % 3].re;
                    term[k][2 * i + 1][lane] = T.m[i / 3][i % 3].im;
                }
            } else {
                const R4<Real> ga = U.ld2(nu, ea), gb = U.ld2(mu, eb), gc = U.ld2(nu, ec);
                const R4<Real> T =
                    bwd ? times2(times2(herm2(ga), herm2(gb)), gc) : times2(times2(ga, herm2(gb)), herm2(gc));
                term[k][0][lane] = T.x;
                term[k][1][lane] = T.y;
                term[k][2][lane] = T.z;
                term[k][3][lane] = T.w;
            }
        }
        if constexpr (!OR && PMODE == 0) fill();
    }
    __syncthreads();
    if (on) {                                           // st = f0 + b0; st = b_i + (st + f_i)
        for (int k = w; k < NT; k += SP) {
            Real st = term[0][k][lane] + term[1][k][lane];
            st = term[3][k][lane] + (st + term[2][k][lane]);
            st = term[5][k][lane] + (st + term[4][k][lane]);
            term[0][k][lane] = st;
        }
    }
    __syncthreads();
    if (w != 0 || !on) return;
    PrnTable<Real, typename PS::T> prn;
    if constexpr (!OR) {
        prn.src = src;
        prn.tab = &tab;
        prn.k = 0;
        prn.lane = lane;
    }
    if constexpr (NC == 3) {
        M3<Real> st;
#pragma unroll
        for (int i = 0; i < 9; i++) st.m[i / 3][i % 3] = { term[0][2 * i][lane], term[0][2 * i + 1][lane] };
        G3<Real> r;
        if constexpr (OR && sizeof(Real) == 4) r = cm3_or_rows(st, m0, A.nhitpar);
        else r = cm3<Real, OR>(st, m0, beta, prn, A.nhit, A.nhitpar);
        U.st3(mu, own, r);
    } else {
        const S2<Real> st = rec2(R4<Real>{ term[0][0][lane], term[0][1][lane], term[0][2][lane], term[0][3][lane] });
        U.st2(mu, own, su2_update<Real, OR>(st, q0, beta, prn, A.nhit));
    }
}

// a phase kernel; early: as the programmatic dependent of the phase before it
// in the graph (the kernels wait for that grid before they read links)
template <typename Real>
cudaError_t launch_after(void (*kern)(Field<Real>, Geom, PhaseArgs), unsigned nb, unsigned bs, bool early,
                         const Field<Real> &U, const Geom &G, const PhaseArgs &a, cudaStream_t s)
{
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nb);
    cfg.blockDim = dim3(bs);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, U, G, a);
}

// Launches k_phase_split with SP warps for 32 links; false where that is not
// the faster form.  A block's registers stay taken while its first warp alone
// updates the links, so the split pays while all blocks are resident with
// room to spare: SU(3) and the SU(2) heatbath with SP = 6 up to 3/4 (SU(2): 3/5)
// of the resident blocks, then with SP = 3 up to 3/4 (FP32 overrelaxation and
// RANLUX batches, whose generator wants the SMs too: 1/2; not the SU(2) FP64
// heatbath); the SU(2) overrelaxation, little more than its loads, up to 128
// blocks (FP64: 512).  Measured in the sweep graph, us a phase, heatbath /
// overrelaxation, one thread per link (the faster of its forms) -> split:
//   SU(3) FP32  8^4   8.9 / 4.4 -> 6.8 / 2.8    16^3 x 8   9.8 / 5.1 -> 8.5 / 4.2
//   SU(3) FP64  8^4  11.1 / 5.8 -> 6.9 / 3.9    12^3 x 8  11.8 / 6.4 -> 7.9 / 4.8
//   SU(2) FP32  8^4   4.1 / 2.0 -> 2.6 / 1.5    16^4       4.9       -> 4.4
//   SU(2) FP64  8^4   4.7 / 2.7 -> 2.7 / 1.7    16^3 x 8   5.1 / 2.8 -> 4.1 / 2.9
// and beyond the limits: SU(3) FP32 16^4 10.9 / 5.3 against 13.1 / 6.2 with
// SP = 3, FP64 14.3 / 8.4 against 16.9 / 11.2; SU(2) FP32 16^3 x 8
// overrelaxation 1.9 against 2.6 with SP = 6.  The early launch hides the
// Philox heatbath's random numbers (SU(2) 8^4: 4.1 -> 2.6 us); without them it
// only pays up to half a block per SM (the next phase's blocks crowd where
// the first slots come free: SU(3) FP32 12^3 x 8 overrelaxation 3.2 us
// without, 4.2 with it, 4^4 2.65 / 2.31).
template <int NC, typename Real, int PM, bool OR, int MU, int SP>
unsigned split_limit(unsigned nb)
{
    constexpr bool kF32 = sizeof(Real) == 4;
    if constexpr (NC == 2 && OR) return kF32 ? 128 : 512;
    // more than 64 warps per SM would hold: the driver is not asked (it would
    // load a kernel that a large lattice never launches, 0.1 ms each)
    if (nb > 148u * (64 / SP) * 3 / 4) return 0;
    static const int per_sm = [] {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_phase_split<NC, Real, PM, OR, MU, SP>, 32 * SP, 0) !=
            cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        return n;
    }();
    const unsigned resident = 148u * per_sm;
    if (SP == 6) return NC == 3 ? resident * 3 / 4 : resident * 3 / 5;
    return (OR && kF32) || (!OR && PM == 0) ? resident / 2 : resident * 3 / 4;
}

template <int NC, typename Real, int PM, bool OR, int MU, int SP>
bool try_split(const Field<Real> &U, const Geom &G, const PhaseArgs &a, cudaStream_t s, cudaError_t &e)
{
    if constexpr (SP == 3 && NC == 2 && (OR || sizeof(Real) == 8)) {
        return false;
    } else {
        const unsigned nb = (a.t_end - a.t_begin + 31) / 32;
        if (nb > split_limit<NC, Real, PM, OR, MU, SP>(nb)) return false;
        const bool early = a.after_phase && ((!OR && PM == 1) || nb <= 74);
        e = launch_after(k_phase_split<NC, Real, PM, OR, MU, SP>, nb, 32 * SP, early, U, G, a, s);
        return true;
    }
}

template <typename Real>
bool launch_phase_split(const Field<Real> &U, const Geom &G, int group, const PhaseArgs &a, cudaStream_t s,
                        cudaError_t &e)
{
#define QG_SPLIT1(NC, PM, OR, MU)                                                                       \
    return try_split<NC, Real, PM, OR, MU, 6>(U, G, a, s, e) || try_split<NC, Real, PM, OR, MU, 3>(U, G, a, s, e)
#define QG_SPLIT(NC, PM, OR)                            \
    switch (a.dir) {                                    \
    case 0: QG_SPLIT1(NC, PM, OR, 0);                   \
    case 1: QG_SPLIT1(NC, PM, OR, 1);                   \
    case 2: QG_SPLIT1(NC, PM, OR, 2);                   \
    default: QG_SPLIT1(NC, PM, OR, 3);                  \
    }
    if (group == 3) {
        if (a.prn_mode == -1) { QG_SPLIT(3, 0, true) }
        else if (a.prn_mode == 0) { QG_SPLIT(3, 0, false) }
        else { QG_SPLIT(3, 1, false) }
    } else {
        if (a.prn_mode == -1) { QG_SPLIT(2, 0, true) }
        else if (a.prn_mode == 0) { QG_SPLIT(2, 0, false) }
        else { QG_SPLIT(2, 1, false) }
    }
#undef QG_SPLIT
#undef QG_SPLIT1
}

template <typename Real>
cudaError_t launch_phase_T(const Geom &G, void *links, int group, const PhaseArgs &a, cudaStream_t s)
{
    Field<Real> U;
    U.p = reinterpret_cast<typename V4<Real>::T *>(links);
    U.pstride = G.pstride;
    const int bs = kPhaseBlock;
    const unsigned nb = (a.t_end - a.t_begin + bs - 1) / bs;
    const int pm = a.prn_mode;   // -1 selects overrelaxation (no PRNs)
    // shapes 3, 4 stage the staple through shared memory where that form
    // exists (SU(3), FP32 links); elsewhere they run shapes 0, 1
    constexpr bool kStage = sizeof(Real) == 4;
    // shape 5: overrelaxation two links per thread (SU(3), FP32, periodic,
    // the whole lattice); otherwise it runs shape 4
    if constexpr (sizeof(Real) == 4) {
        if (a.variant == 5 && group == 3 && pm == -1 && !a.twist && a.t_begin == 0 && a.t_end == G.half) {
            const unsigned nbp = ((G.half + 1) / 2 + bs - 1) / bs;
            switch (a.dir) {
            case 0: k_phase_or_pair<0><<<nbp, bs, 0, s>>>(U, G, a); break;
            case 1: k_phase_or_pair<1><<<nbp, bs, 0, s>>>(U, G, a); break;
            case 2: k_phase_or_pair<2><<<nbp, bs, 0, s>>>(U, G, a); break;
            default: k_phase_or_pair<3><<<nbp, bs, 0, s>>>(U, G, a); break;
            }
            return cudaGetLastError();
        }
    }
    // shape 0 of few links: six or three warps for 32 links (k_phase_split)
    cudaError_t e;
    if (a.variant == 0 && !a.twist && pm != 2 && launch_phase_split<Real>(U, G, group, a, s, e)) return e;
    // shape 0 otherwise: the compiler's registers, or the form held to five
    // blocks per SM (shape 1) where that is the faster: SU(3) FP32 (us a phase,
    // heatbath / overrelaxation: 20^4 19.2 / 10.2 -> 17.2 / 9.6, 24^4 31.4 / 16.5
    // -> 29.9 / 16.5, 32^4 93.7 / 58.9 -> 89.1 / 57.1) and SU(2) up to 100 000
    // links (FP32 16^4 5.6 / 3.1 -> 5.1 / 2.4, FP64 6.9 / 4.0 -> 5.7 / 3.4; at 32^4
    // the FP64 heatbath 39.6 against 44.4); SU(3) FP64 spills (16^4 14.4 / 8.4
    // against 17.8 / 11.0)
    const bool tight = group == 3 ? kStage : a.t_end - a.t_begin <= 100000;
    // twisted boundaries: shape 0's form with the twist tests compiled in
    // (any shape computes the same sequence); the others are compiled
    // without them
#define QG_LAUNCH2(NC, PM, OR, MU, MB, ST) k_phase<NC, Real, PM, OR, MU, MB, ST, false><<<nb, bs, 0, s>>>(U, G, a)
#define QG_LAUNCH1(NC, PM, OR, MU)                                                  \
    do {                                                                            \
        if (a.twist) k_phase<NC, Real, PM, OR, MU, 0, false, true><<<nb, bs, 0, s>>>(U, G, a); \
        else if (a.variant == 1) QG_LAUNCH2(NC, PM, OR, MU, 5, false);              \
        else if (a.variant == 2) QG_LAUNCH2(NC, PM, OR, MU, 6, false);              \
        else if (a.variant == 3) QG_LAUNCH2(NC, PM, OR, MU, 0, NC == 3 && kStage);  \
        else if (a.variant >= 4) QG_LAUNCH2(NC, PM, OR, MU, 5, NC == 3 && kStage);  \
        else if (tight) QG_LAUNCH2(NC, PM, OR, MU, 5, false);                       \
        else QG_LAUNCH2(NC, PM, OR, MU, NC == 3 && kStage ? 5 : 0, false);          \
    } while (0)
#define QG_LAUNCH(NC, PM, OR)                                     \
    do {                                                          \
        switch (a.dir) {                                          \
        case 0: QG_LAUNCH1(NC, PM, OR, 0); break;                 \
        case 1: QG_LAUNCH1(NC, PM, OR, 1); break;                 \
        case 2: QG_LAUNCH1(NC, PM, OR, 2); break;                 \
        default: QG_LAUNCH1(NC, PM, OR, 3); break;                \
        }                                                         \
    } while (0)
    if (group == 3) {
        if (pm == -1) QG_LAUNCH(3, 0, true);
        else if (pm == 0) QG_LAUNCH(3, 0, false);
        else if (pm == 1) QG_LAUNCH(3, 1, false);
        else QG_LAUNCH(3, 2, false);
    } else {
        if (pm == -1) QG_LAUNCH(2, 0, true);
        else if (pm == 0) QG_LAUNCH(2, 0, false);
        else if (pm == 1) QG_LAUNCH(2, 1, false);
        else QG_LAUNCH(2, 2, false);
    }
#undef QG_LAUNCH
#undef QG_LAUNCH1
#undef QG_LAUNCH2
    return cudaGetLastError();
}

}  // namespace qg
