// Adjoint kernels for one face precision; included once per precision by
// adjoint.cu (KT = double, with the forward FP64 kernels' -fmad=false) and
// adjoint_mixed.cu (KT = float, with the mixed kernels' flags), so every
// forward value the adjoint recomputes is the forward's own.
//
// Per Runge-Kutta stage s, with stage input X_s and residual R(X_s), the
// forward computes t_s = X_s + cfl * R(X_s). Backward, given the adjoint t_bar
// of t_s and mu = cfl * t_bar (FP64, per cell):
//   k_adj_flux   per edge: F_bar = mu_c2 - mu_c1 (the reference's -=/+=), the
//                VJP of both Gauss-point fluxes, reconstructions and ghost
//                states -> adjoints of the two cells' primitives and gradients
//   k_adj_gather per cell: sum of its faces' contributions (fixed order)
//   k_adj_cell   per cell: VJP of the Green-Gauss gradients (own and the three
//                neighbours' gradient adjoints), of the boundary ghosts and of
//                convertConsToPar; X_bar = t_bar + (dR/dX)^T mu in FP64; the
//                scheme's stage algebra gives the previous stage's t_bar
// Face-level products run in KT; everything accumulated per cell across stages
// and steps (t_bar, lambda, the boundary-parameter sums) is FP64. No atomics:
// every sum is a gather in a fixed order.
#pragma once
#include "adjoint.cuh"

namespace cfd2d {
namespace {

inline int adj_nblk(long n, int b) { return (int)((n + b - 1) / b); }

// One side's adjoints of an edge (12 values): primitives, then gradients.
template <typename T>
__device__ __forceinline__ void store_bars(T* o, const Prim<T>& q, const T* g) {
    st4(o, 0, q.r, q.u, q.v, q.p);
    st8(o + 4, 0, g);
}
__device__ __forceinline__ void store_bars(double* o, const Prim<xd>& q, const xd* g) {
    st4(o, 0, q.r.v, q.u.v, q.v.v, q.p.v);
    st8x(o + 4, 0, g);
}

// The flux VJP of an interior edge with FP64 faces and reconstruction, two lanes per edge: lane
// gp reverses Gauss point gp's flux (its states read from the forward's record with REC, else
// reconstructed), the pair exchanges the face states' adjoints, and each lane gathers the
// reconstruction's VJP of one side over both points, in the points' order: the same operations
// as adj_flux_edge's on the same values. One thread for an edge needs 160 registers (12 warps
// on an SM) and waits for its own chains. Called by whole warps.
template <int FLUX, int RECON, bool REC>
__device__ __forceinline__ void adj_flux_lane(const DevCase& c, const AdjCase& a, const FluxRec& rec, int e, int gp,
                                              bool live) {
    const size_t ne = c.ne;
    const xd nx(c.nx[e]), ny(c.ny[e]);
    const xd GAM = gam_of<xd>(c), IG1 = ig1_of<xd>(c);
    const int c1 = c.ec1[e], c2 = c.ec2[e];
    const double* __restrict__ DL = c.dl + e;
    unsigned codes = 0;
    Prim<xd> pL, pR, pb[2][2];  // adjoints of the face states: [point][side]
    {
        xd cL, cR;
        if constexpr (REC) {
            const double* v = static_cast<const double*>(rec.v) + (size_t)(10 * gp) * ne + e;
            pL = Prim<xd>{xd(v[0]), xd(v[ne]), xd(v[2 * ne]), xd(v[3 * ne])};
            pR = Prim<xd>{xd(v[4 * ne]), xd(v[5 * ne]), xd(v[6 * ne]), xd(v[7 * ne])};
            cL = xd(v[8 * ne]); cR = xd(v[9 * ne]);
            if (RECON == RECON_MINMOD) codes = rec.bits[e] >> (16 * gp);
        } else {
            pL = prim_as<xd>(load_prim(c.W64, c1));
            pR = prim_as<xd>(load_prim(c.W64, c2));
            Prim<xd> d = pL;
            if (RECON == RECON_MINMOD) d = Prim<xd>{pR.r - pL.r, pR.u - pL.u, pR.v - pL.v, pR.p - pL.p};
            const double* dl = DL + (size_t)(4 * gp) * ne;
            double g[8];
            ld8(c.G64, c1, g);
            codes = reconstruct<xd, RECON>(pL, g, xd(dl[0]), xd(dl[ne]), d);
            if (RECON == RECON_MINMOD) d = Prim<xd>{-d.r, -d.u, -d.v, -d.p};
            ld8(c.G64, c2, g);
            codes |= reconstruct<xd, RECON>(pR, g, xd(dl[2 * ne]), xd(dl[3 * ne]), d) << 8;
        }
        xd fb[4];
        {
            double m1[4], m2[4];
            ld4(a.mu, c1, m1);
            ld4(a.mu, c2, m2);
            // F = (sum over Gauss points of f) * l/2; R_c1 -= F, R_c2 += F
            const xd lh = half(xd(c.l[e]));
#pragma unroll
            for (int k = 0; k < 4; k++) fb[k] = (xd(m2[k]) - xd(m1[k])) * lh;
        }
        Prim<xd> Lb = zero_prim<xd>(), Rb = zero_prim<xd>();
        if constexpr (REC) vjp_hllc_c(pL, pR, cL, cR, nx, ny, GAM, IG1, fb, Lb, Rb);
        else vjp_flux<FLUX>(pL, pR, nx, ny, GAM, IG1, fb, Lb, Rb);
        pb[0][0] = Lb;
        pb[0][1] = Rb;
    }
    // both points' adjoints and branches in both lanes
    auto swap = [](xd x) { return xd(__shfl_xor_sync(0xffffffffu, x.v, 1)); };
    unsigned cd[2];
    {
        const unsigned oc = __shfl_xor_sync(0xffffffffu, codes, 1);
        cd[0] = gp ? oc : codes;
        cd[1] = gp ? codes : oc;
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const Prim<xd> m = pb[0][s], o{swap(m.r), swap(m.u), swap(m.v), swap(m.p)};
            pb[0][s] = gp ? o : m;
            pb[1][s] = gp ? m : o;
        }
    }
    if (!live) return;
    const int side = gp;  // this lane's side from here on
    xd qb[4], gb[8];
#pragma unroll
    for (int k = 0; k < 4; k++) qb[k] = acc0<xd>();
#pragma unroll
    for (int k = 0; k < 8; k++) gb[k] = acc0<xd>();
#pragma unroll
    for (int g = 0; g < 2; g++) {
        const double* dl = DL + (size_t)(4 * g + 2 * side) * ne;
        const xd dx(dl[0]), dy(dl[ne]);
        const Prim<xd>&l = pb[g][0], &r = pb[g][1];
        const xd lv[4] = {l.r, l.p, l.u, l.v}, rv[4] = {r.r, r.p, r.u, r.v};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const unsigned bl = RECON == RECON_LINEAR ? 1u : (cd[g] >> (2 * k)) & 3u;
            const unsigned br = RECON == RECON_LINEAR ? 1u : (cd[g] >> (8 + 2 * k)) & 3u;
            const xd own = side ? rv[k] : lv[k];
            if ((side ? br : bl) == 1u) {  // the projection: into the gradient
                gb[2 * k] = g == 0 ? own * dx : madd(gb[2 * k], own, dx);
                gb[2 * k + 1] = g == 0 ? own * dy : madd(gb[2 * k + 1], own, dy);
            }
            // the left face state's share, then the right one's: a side keeps its own state's
            // adjoint unless the difference was taken (2), which passes it to the other side
            if ((bl == 2u) == (side == 1)) qb[k] = qb[k] + lv[k];
            if ((br == 2u) == (side == 0)) qb[k] = qb[k] + rv[k];
        }
    }
    store_bars(static_cast<double*>(a.eq) + 24 * (size_t)e + 12 * side, Prim<xd>{qb[0], qb[2], qb[3], qb[1]}, gb);
}
// FP64 faces with reconstruction: the interior edges by lanes in the first n_lane blocks, the
// boundary edges (stored last) one thread each in the others
template <int RECON> constexpr bool kAdjLanes = RECON != RECON_NONE;

// SIDE: EDGE_ANY (interior or boundary, decided at run time), EDGE_INNER or EDGE_BOUNDARY (known at
// compile time: the interior instantiation carries no boundary code, which a warp would
// otherwise issue, predicated off, for every interior edge).
enum { EDGE_ANY = 0, EDGE_INNER = 1, EDGE_BOUNDARY = 2 };
template <int SIDE>
__device__ __forceinline__ bool edge_inner(const DevCase& c, int e) {
    return SIDE == EDGE_INNER ? true : (SIDE == EDGE_BOUNDARY ? false : e < c.n_int);
}

// A: the type the edge is computed in (adj_native)
template <typename T, int FLUX, int RECON, int SIDE, typename A>
__device__ __forceinline__ void adj_flux_edge(const DevCase& c, const AdjCase& a, int e);
template <typename T, int FLUX, int RECON, typename A = Arith<T>>
// FP32 faces: at most 128 registers (two 256-thread blocks' worth per SM), measured
// faster than the compiler's unconstrained choice. With FP64 faces interior and boundary edges
// (stored last) run their own instantiations.
__global__ void __launch_bounds__(sizeof(T) == 4 ? 256 : 128, sizeof(T) == 4 ? 2 : 4)
k_adj_flux(const DevCase c, const AdjCase a, int n_lane) {
    if constexpr (sizeof(T) == 8) {
        const int t = blockIdx.x * blockDim.x + threadIdx.x;
        if (kAdjLanes<RECON> && (int)blockIdx.x < n_lane) {
            const bool live = t < 2 * c.n_int;
            if constexpr (kAdjLanes<RECON>) adj_flux_lane<FLUX, RECON, false>(c, a, FluxRec{}, live ? t >> 1 : 0, t & 1, live);
            return;
        }
        const int e = t + (kAdjLanes<RECON> ? c.n_int - n_lane * (int)blockDim.x : 0);
        if (e >= c.ne) return;
        if (!kAdjLanes<RECON> && e < c.n_int) adj_flux_edge<T, FLUX, RECON, EDGE_INNER, A>(c, a, e);
        else adj_flux_edge<T, FLUX, RECON, EDGE_BOUNDARY, A>(c, a, e);
    } else {
        const int e = blockIdx.x * blockDim.x + threadIdx.x;
        if (e < c.ne) adj_flux_edge<T, FLUX, RECON, EDGE_ANY, A>(c, a, e);
    }
}
template <typename T, int FLUX, int RECON, int SIDE, typename A>
__device__ __forceinline__ void adj_flux_edge(const DevCase& c, const AdjCase& a, int e) {
    const int ne = c.ne;
    const T* W = W_of<T>(c);
    const T* G = G_of<T>(c);
    const T* DL = DL_of<T>(c);
    const A nx(NX_of<T>(c)[e]), ny(NY_of<T>(c)[e]), l(L_of<T>(c)[e]);
    const A GAM = gam_of<A>(c), IG1 = ig1_of<A>(c);
    const int c1 = c.ec1[e];
    const bool inner = edge_inner<SIDE>(c, e);
    const int c2 = inner ? c.ec2[e] : -1;
    const Prim<A> qL = prim_as<A>(load_prim(W, c1));
    Prim<A> qR = qL, gc = qL;
    DevBnd b{};
    A Tc = A(0), M = A(0), gm1 = A(0), Cv = A(0);
    A fb[4];
    {
        double m1[4], m2[4] = {0, 0, 0, 0};
        ld4(a.mu, c1, m1);
        if (inner) ld4(a.mu, c2, m2);
        // F = (sum over Gauss points of f) * l/2; R_c1 -= F, R_c2 += F. The difference is
        // formed in FP64 and rounded once into the face precision.
        const double lh = to_wide(l) * (RECON == RECON_NONE ? 1.0 : 0.5);
        for (int k = 0; k < 4; k++) fb[k] = to_face<A>((m2[k] - m1[k]) * lh);
    }
    if (inner) {
        qR = prim_as<A>(load_prim(W, c2));
    } else {
        b = c.bnds[c.ebnd[e]];
        const MatT<A> mt = matT_of<A>(c, c1);
        gm1 = mt.gm1; Cv = mt.Cv; M = mt.M;
        Tc = temperature(qL, gm1, Cv);
        if (RECON == RECON_MINMOD) gc = ghost_state(b, qL, Tc, nx, ny, M);
    }
    Prim<A> q1b = zero_prim<A>(), q2b = zero_prim<A>(), gcb = zero_prim<A>();
    A g1b[8], g2b[8], bp[4];
#pragma unroll
    for (int k = 0; k < 8; k++) { g1b[k] = acc0<A>(); g2b[k] = acc0<A>(); }
#pragma unroll
    for (int k = 0; k < 4; k++) bp[k] = acc0<A>();
    A Tcb = acc0<A>();
    const int ngp = RECON == RECON_NONE ? 1 : 2;
#pragma unroll 1
    for (int gp = 0; gp < ngp; gp++) {
        Prim<A> pL = qL, pR = qR;
        A aL[4] = {A(0), A(0), A(0), A(0)}, aR[4] = {A(0), A(0), A(0), A(0)};
        A dxL = A(0), dyL = A(0), dxR = A(0), dyR = A(0);
        if (RECON != RECON_NONE) {
            T g[8];
            dxL = A(DL[(4 * gp) * ne + e]); dyL = A(DL[(4 * gp + 1) * ne + e]);
            ld8(G, c1, g);
            project<RECON>(g, dxL, dyL, aL);
            pL = recon_a<RECON>(qL, aL, inner ? qR : gc);
            if (inner) {
                dxR = A(DL[(4 * gp + 2) * ne + e]); dyR = A(DL[(4 * gp + 3) * ne + e]);
                ld8(G, c2, g);
                project<RECON>(g, dxR, dyR, aR);
                pR = recon_a<RECON>(qR, aR, qL);
            }
        }
        if (!inner) pR = ghost_state(b, pL, Tc, nx, ny, M);
        Prim<A> pLb = zero_prim<A>(), pRb = zero_prim<A>();
        vjp_flux<FLUX>(pL, pR, nx, ny, GAM, IG1, fb, pLb, pRb);
        if (!inner) vjp_ghost(b, pL, Tc, nx, ny, M, pRb, pLb, Tcb, bp);
        if (RECON == RECON_NONE) {  // both Gauss points see the cell-centre states: one pass, twice the weight
            q1b.r += pLb.r; q1b.u += pLb.u; q1b.v += pLb.v; q1b.p += pLb.p;
            if (inner) { q2b.r += pRb.r; q2b.u += pRb.u; q2b.v += pRb.v; q2b.p += pRb.p; }
        } else if (inner) {
            vjp_reconstruct_a<RECON>(qL, aL, dxL, dyL, qR, pLb, q1b, g1b, q2b);
            vjp_reconstruct_a<RECON>(qR, aR, dxR, dyR, qL, pRb, q2b, g2b, q1b);
        } else {
            vjp_reconstruct_a<RECON>(qL, aL, dxL, dyL, gc, pLb, q1b, g1b, gcb);
        }
    }
    if (!inner) {
        if (RECON == RECON_MINMOD) vjp_ghost(b, qL, Tc, nx, ny, M, gcb, q1b, Tcb, bp);
        vjp_temperature(qL, gm1, Cv, Tcb, q1b);
        double* o = a.eb + 4 * (size_t)(e - c.n_int);  // this edge's own running sum over stages and steps
        o[0] += to_wide(bp[0]); o[1] += to_wide(bp[1]); o[2] += to_wide(bp[2]); o[3] += to_wide(bp[3]);
    }
    T* o = static_cast<T*>(a.eq) + 24 * (size_t)e;
    store_bars(o, q1b, g1b);
    store_bars(o + 12, q2b, g2b);
}

// The forward flux kernel of a recomputed stage that also keeps the evaluation's record
// (FluxRec: face states, sound speeds, minmod's branches) for k_adj_flux_rec. Compiled with
// the forward kernels' flags and the same code, so F is the forward's bit for bit.
template <typename T, int RECON>
__global__ void __launch_bounds__(128) k_flux_rec(const DevCase c, const FluxRec r) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if constexpr (FluxLanes<T, RECON>::n == 2) {
        const bool live = t < 2 * c.ne;
        if ((t & ~31) < 2 * c.ne) flux_lane<FLUX_HLLC, RECON, true>(c, live ? t >> 1 : c.ne - 1, t & 1, live, r);
    } else if (t < c.ne) {
        T out[4];
        flux_edge<T, FLUX_HLLC, RECON, true>(c, t, out, r);
        st4(F_of<T>(c), t, out[0], out[1], out[2], out[3]);
    }
}

// k_adj_flux (HLLC) reading the forward's record of each Gauss point instead of
// recomputing the reconstruction, the ghost state, the sound speeds and minmod's
// branches: the same reverse operations on the same values, so the same bits.
template <typename T, int RECON, int SIDE, typename A>
__device__ __forceinline__ void adj_flux_rec_edge(const DevCase& c, const AdjCase& a, const FluxRec& r, int e);
template <typename T, int RECON, typename A = Arith<T>>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 256 : 128, sizeof(T) == 4 ? 2 : 4)
k_adj_flux_rec(const DevCase c, const AdjCase a, const FluxRec r, int n_lane) {
    if constexpr (sizeof(T) == 8) {
        const int t = blockIdx.x * blockDim.x + threadIdx.x;
        if (kAdjLanes<RECON> && (int)blockIdx.x < n_lane) {
            const bool live = t < 2 * c.n_int;
            if constexpr (kAdjLanes<RECON>) adj_flux_lane<FLUX_HLLC, RECON, true>(c, a, r, live ? t >> 1 : 0, t & 1, live);
            return;
        }
        const int e = t + (kAdjLanes<RECON> ? c.n_int - n_lane * (int)blockDim.x : 0);
        if (e >= c.ne) return;
        if (!kAdjLanes<RECON> && e < c.n_int) adj_flux_rec_edge<T, RECON, EDGE_INNER, A>(c, a, r, e);
        else adj_flux_rec_edge<T, RECON, EDGE_BOUNDARY, A>(c, a, r, e);
    } else {
        const int e = blockIdx.x * blockDim.x + threadIdx.x;
        if (e < c.ne) adj_flux_rec_edge<T, RECON, EDGE_ANY, A>(c, a, r, e);
    }
}
template <typename T, int RECON, int SIDE, typename A>
__device__ __forceinline__ void adj_flux_rec_edge(const DevCase& c, const AdjCase& a, const FluxRec& r, int e) {
    const int ne = c.ne;
    const T* DL = DL_of<T>(c);
    const A nx(NX_of<T>(c)[e]), ny(NY_of<T>(c)[e]), l(L_of<T>(c)[e]);
    const A GAM = gam_of<A>(c), IG1 = ig1_of<A>(c);
    const int c1 = c.ec1[e];
    const bool inner = edge_inner<SIDE>(c, e);
    const int c2 = inner ? c.ec2[e] : -1;
    Prim<A> qL{};
    DevBnd b{};
    A Tc = A(0), M = A(0), gm1 = A(0), Cv = A(0);
    A fb[4];
    {
        double m1[4], m2[4] = {0, 0, 0, 0};
        ld4(a.mu, c1, m1);
        if (inner) ld4(a.mu, c2, m2);
        const double lh = to_wide(l) * (RECON == RECON_NONE ? 1.0 : 0.5);
        for (int k = 0; k < 4; k++) fb[k] = to_face<A>((m2[k] - m1[k]) * lh);
    }
    if (!inner) {
        qL = prim_as<A>(load_prim(W_of<T>(c), c1));
        b = c.bnds[c.ebnd[e]];
        const MatT<A> mt = matT_of<A>(c, c1);
        gm1 = mt.gm1; Cv = mt.Cv; M = mt.M;
        Tc = temperature(qL, gm1, Cv);
    }
    Prim<A> q1b = zero_prim<A>(), q2b = zero_prim<A>(), gcb = zero_prim<A>();
    A g1b[8], g2b[8], bp[4];
#pragma unroll
    for (int k = 0; k < 8; k++) { g1b[k] = acc0<A>(); g2b[k] = acc0<A>(); }
#pragma unroll
    for (int k = 0; k < 4; k++) bp[k] = acc0<A>();
    A Tcb = acc0<A>();
    const unsigned bits = RECON == RECON_MINMOD ? r.bits[e] : 0u;
    const int ngp = RECON == RECON_NONE ? 1 : 2;
#pragma unroll 1
    for (int gp = 0; gp < ngp; gp++) {
        const T* v = static_cast<const T*>(r.v) + (size_t)(10 * gp) * ne + e;
        const Prim<A> pL{A(v[0]), A(v[ne]), A(v[2 * (size_t)ne]), A(v[3 * (size_t)ne])};
        const Prim<A> pR{A(v[4 * (size_t)ne]), A(v[5 * (size_t)ne]), A(v[6 * (size_t)ne]), A(v[7 * (size_t)ne])};
        const A cL(v[8 * (size_t)ne]), cR(v[9 * (size_t)ne]);
        A dxL = A(0), dyL = A(0), dxR = A(0), dyR = A(0);
        if (RECON != RECON_NONE) {
            dxL = A(DL[(4 * gp) * ne + e]); dyL = A(DL[(4 * gp + 1) * ne + e]);
            if (inner) { dxR = A(DL[(4 * gp + 2) * ne + e]); dyR = A(DL[(4 * gp + 3) * ne + e]); }
        }
        Prim<A> pLb = zero_prim<A>(), pRb = zero_prim<A>();
        vjp_hllc_c(pL, pR, cL, cR, nx, ny, GAM, IG1, fb, pLb, pRb);
        if (!inner) vjp_ghost(b, pL, Tc, nx, ny, M, pRb, pLb, Tcb, bp);
        if (RECON == RECON_NONE) {
            q1b.r += pLb.r; q1b.u += pLb.u; q1b.v += pLb.v; q1b.p += pLb.p;
            if (inner) { q2b.r += pRb.r; q2b.u += pRb.u; q2b.v += pRb.v; q2b.p += pRb.p; }
        } else if (inner) {
            vjp_reconstruct_code<RECON>(bits >> (16 * gp), dxL, dyL, pLb, q1b, g1b, q2b);
            vjp_reconstruct_code<RECON>(bits >> (16 * gp + 8), dxR, dyR, pRb, q2b, g2b, q1b);
        } else {
            vjp_reconstruct_code<RECON>(bits >> (16 * gp), dxL, dyL, pLb, q1b, g1b, gcb);
        }
    }
    if (!inner) {
        if (RECON == RECON_MINMOD) vjp_ghost(b, qL, Tc, nx, ny, M, gcb, q1b, Tcb, bp);
        vjp_temperature(qL, gm1, Cv, Tcb, q1b);
        double* o = a.eb + 4 * (size_t)(e - c.n_int);
        o[0] += to_wide(bp[0]); o[1] += to_wide(bp[1]); o[2] += to_wide(bp[2]); o[3] += to_wide(bp[3]);
    }
    T* o = static_cast<T*>(a.eq) + 24 * (size_t)e;
    store_bars(o, q1b, g1b);
    store_bars(o + 12, q2b, g2b);
}

// The three faces' contributions summed exactly (SumAcc): the primitive adjoint is
// rounded once into FP64 (it is summed again in k_adj_cell), the gradient adjoint
// into the face precision and divided by the cell's area (it only enters products there).
template <typename T>
__global__ void __launch_bounds__(256) k_adj_gather(const DevCase c, const AdjCase a) {
    const int nc = c.nc;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nc) return;
    SumAcc<T> q[4], g[8];
    const T* eq = static_cast<const T*>(a.eq);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int f = c.face[k * nc + i];
        const T* s = eq + 24 * (size_t)(f >> 1) + ((f & 1) ? 12 : 0);
        T v[12];
        ld4(s, 0, v);
        ld8(s + 4, 0, v + 4);
#pragma unroll
        for (int m = 0; m < 4; m++) q[m].add(v[m]);
#pragma unroll
        for (int m = 0; m < 8; m++) g[m].add(v[4 + m]);
    }
    st4(a.qbar, i, q[0].value(), q[1].value(), q[2].value(), q[3].value());
    // kept divided by the cell's area: the Green-Gauss VJP (k_adj_cell) then needs no
    // per-face weights of its own and no products by 1/S
    const T iSi = invS_of<T>(c)[i];
    T gv[8];
#pragma unroll
    for (int m = 0; m < 8; m++) gv[m] = T(Arith<T>(g[m].face()) * Arith<T>(iSi));
    st8(static_cast<T*>(a.gbar), i, gv);
}

// coef_t / coef_acc: the scheme's stage algebra (the previous stage's t_bar and
// the step input's share); first: this is stage 0, write the step's lambda and,
// with (coef_t, coef_acc) the last stage's coefficients, start the step before it
// (t_bar, acc and mu from lambda: what k_adj_step_start does for the first step).
template <typename T>
__global__ void __launch_bounds__(256) k_adj_cell(const DevCase c, const AdjCase a, double coef_t, double coef_acc,
                                                  int first) {
    const int nc = c.nc;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nc) return;
    typedef Arith<T> A;
    typedef typename WideArith<T>::type D;
    const MatT<A> mt = matT_of<A>(c, i);
    const Prim<A> q = prim_as<A>(load_prim(W_of<T>(c), i));
    // h = the gradient adjoints divided by the area (k_adj_gather)
    const T* h = static_cast<const T*>(a.gbar);
    // the cell's primitive adjoint: the gathered FP64 value plus the sum of the
    // Green-Gauss products (r, u, v, p)
    SumAcc<T> qs[4];
    A Tcb = acc0<A>();
    Prim<A> qb = zero_prim<A>();  // ghost-path contributions (boundary faces only)
    // every load before the first branch and the first store: the faces and neighbours, then
    // their geometry, gradient adjoints and the cell's own state (one after another they took
    // two thirds of the FP32 form's time on a small mesh; with FP64 faces the neighbours'
    // gradient adjoints stay in the loop, 48 registers less)
    constexpr bool AHEAD = sizeof(T) == 4;
    int fc[3], nb[3];
    T ge[3][3], hv[AHEAD ? 3 : 1][8];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        fc[k] = c.face[k * nc + i];
        nb[k] = c.cf_nb[k * nc + i];
    }
    double q0[4], tb[4], ac[4];
    ld4(a.qbar, i, q0);  // r, u, v, p
#pragma unroll
    for (int k = 0; k < 4; k++) {
        tb[k] = a.tb[k * nc + i];
        ac[k] = a.acc[k * nc + i];
    }
    const double cfl = c.cfl[i];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int e = fc[k] >> 1;
        ge[k][0] = NX_of<T>(c)[e]; ge[k][1] = NY_of<T>(c)[e]; ge[k][2] = L_of<T>(c)[e];
        if (AHEAD) ld8(h, nb[k] >= 0 ? nb[k] >> 1 : i, hv[AHEAD ? k : 0]);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int e = fc[k] >> 1;
        const bool side2 = fc[k] & 1;
        const A nx(ge[k][0]), ny(ge[k][1]), l(ge[k][2]);
        // d g_i / d (neighbour or ghost value) = +-(l/2) n / S_i with n outward from c1; the
        // neighbour's gradient takes q_i with the opposite sign and its own 1/S_j. The own
        // value's direct terms, (1/S_i) sum_k (l_k/2) n_out,k over the three faces, are the
        // outward normals of a closed triangle weighted by their lengths: zero, and left out.
        const A w = neg_if(half(l), side2);
        const A wx = w * nx, wy = w * ny;
        if (!AHEAD) ld8(h, nb[k] >= 0 ? nb[k] >> 1 : i, hv[0]);
        const T* hj = hv[AHEAD ? k : 0];
        const A s0 = madd(wx * A(hj[0]), wy, A(hj[1])), s1 = madd(wx * A(hj[2]), wy, A(hj[3]));
        const A s2 = madd(wx * A(hj[4]), wy, A(hj[5])), s3 = madd(wx * A(hj[6]), wy, A(hj[7]));
        if (nb[k] >= 0) {
            qs[0].add(-s0);
            qs[3].add(-s1);
            qs[1].add(-s2);
            qs[2].add(-s3);
        } else {  // boundary face: the ghost of the unreconstructed centre state
            const DevBnd b = c.bnds[c.ebnd[e]];
            const A Tc = temperature(q, mt.gm1, mt.Cv);
            Prim<A> ob;
            ob.r = s0; ob.p = s1; ob.u = s2; ob.v = s3;
            A bp[4] = {acc0<A>(), acc0<A>(), acc0<A>(), acc0<A>()};
            vjp_ghost(b, q, Tc, nx, ny, mt.M, ob, qb, Tcb, bp);
            double* o = a.eb2 + 4 * (size_t)(e - c.n_int);
            o[0] += to_wide(bp[0]); o[1] += to_wide(bp[1]); o[2] += to_wide(bp[2]); o[3] += to_wide(bp[3]);
        }
    }
    if (to_wide(Tcb) != 0.0) vjp_temperature(q, mt.gm1, mt.Cv, Tcb, qb);
    {
        qs[0].add(qb.r); qs[1].add(qb.u); qs[2].add(qb.v); qs[3].add(qb.p);
        qb.r = to_face<A>(to_wide(D(q0[0]) + D(qs[0].value())));
        qb.u = to_face<A>(to_wide(D(q0[1]) + D(qs[1].value())));
        qb.v = to_face<A>(to_wide(D(q0[2]) + D(qs[2].value())));
        qb.p = to_face<A>(to_wide(D(q0[3]) + D(qs[3].value())));
    }
    A V[4] = {acc0<A>(), acc0<A>(), acc0<A>(), acc0<A>()};
    vjp_cons2prim_q(q, mt.gm1, qb, V);
    D ux[4];
    for (int k = 0; k < 4; k++) ux[k] = D(tb[k]) + D(to_wide(V[k]));
    const D cf(cfl), ct(coef_t), ca(coef_acc);
    double mu[4];
    for (int k = 0; k < 4; k++) {
        const size_t q4 = (size_t)k * nc + i;
        D t;
        if (first) {  // lambda of the step input, and (coef_t, coef_acc = the last stage's) the next step's start
            const D l = D(ac[k]) + ux[k];
            a.lam[q4] = to_wide(l);
            t = ct * l;
            a.acc[q4] = to_wide(ca * l);
        } else {
            t = ct * ux[k];
            a.acc[q4] = to_wide(D(ac[k]) + ca * ux[k]);
        }
        a.tb[q4] = to_wide(t);
        mu[k] = to_wide(cf * t);
    }
    st4(a.mu_out, i, mu[0], mu[1], mu[2], mu[3]);
}

// blocks of 128 threads for the flux VJP: n_lane for the interior edges' lanes, the rest one
// thread per edge
inline int adj_flux_grid(const DevCase& c, int recon, int& n_lane) {
    n_lane = sizeof(KT) == 8 && recon != RECON_NONE ? adj_nblk(2l * c.n_int, 128) : 0;
    return n_lane ? n_lane + adj_nblk(c.ne - c.n_int, 128) : adj_nblk(c.ne, 128);
}
// First order, FP64 faces, one thread per edge: on the FP64 unit (A = double) while the mesh has at
// most a warp for each of an SM's four schedulers, where an operation's latency counts and the
// unit waits for nobody; products on the integer pipes (A = xd, the same bits) from there on. A
// gradient (6 steps, SSP-RK3, 152 SMs: the line is at 19,456 edges), xd against double, us: 1,240
// edges HLLC 1,355 / 1,280, LAX 1,540 / 1,401; 19,360 edges 1,272 / 1,197, 1,396 / 1,278; 27,840
// edges 1,311 / 1,297, 1,450 / 1,440; 43,440 edges 1,533 / 1,580, 1,682 / 1,816.
inline bool adj_native(const DevCase& c) { return sizeof(KT) == 8 && c.ne <= 4 * 32 * c.sms; }
template <int FLUX>
void adj_flux_by_recon(const DevCase& c, const AdjCase& a, int recon, cudaStream_t s) {
    int n_lane;
    const int g = adj_flux_grid(c, recon, n_lane);
    if (recon == RECON_NONE && adj_native(c)) k_adj_flux<KT, FLUX, RECON_NONE, KT><<<g, 128, 0, s>>>(c, a, n_lane);
    else if (recon == RECON_NONE) k_adj_flux<KT, FLUX, RECON_NONE><<<g, 128, 0, s>>>(c, a, n_lane);
    else if (recon == RECON_LINEAR) k_adj_flux<KT, FLUX, RECON_LINEAR><<<g, 128, 0, s>>>(c, a, n_lane);
    else k_adj_flux<KT, FLUX, RECON_MINMOD><<<g, 128, 0, s>>>(c, a, n_lane);
}
}  // namespace

void KFN(adj_flux)(const DevCase& c, const AdjCase& a, int flux, int recon, cudaStream_t s) {
    if (flux == FLUX_HLLC) adj_flux_by_recon<FLUX_HLLC>(c, a, recon, s);
    else adj_flux_by_recon<FLUX_LAX>(c, a, recon, s);
}
void KFN(flux_rec)(const DevCase& c, int recon, const FluxRec& r, cudaStream_t s) {
    // 128-thread blocks: finer than 256 in registers, so more warps fit an SM
    const int g = adj_nblk(c.ne * (sizeof(KT) == 8 && recon != RECON_NONE ? 2 : 1), 128);
    if (recon == RECON_NONE) k_flux_rec<KT, RECON_NONE><<<g, 128, 0, s>>>(c, r);
    else if (recon == RECON_LINEAR) k_flux_rec<KT, RECON_LINEAR><<<g, 128, 0, s>>>(c, r);
    else k_flux_rec<KT, RECON_MINMOD><<<g, 128, 0, s>>>(c, r);
}
void KFN(adj_flux_rec)(const DevCase& c, const AdjCase& a, int recon, const FluxRec& r, cudaStream_t s) {
    int n_lane;
    const int g = adj_flux_grid(c, recon, n_lane);
    if (recon == RECON_NONE && adj_native(c)) k_adj_flux_rec<KT, RECON_NONE, KT><<<g, 128, 0, s>>>(c, a, r, n_lane);
    else if (recon == RECON_NONE) k_adj_flux_rec<KT, RECON_NONE><<<g, 128, 0, s>>>(c, a, r, n_lane);
    else if (recon == RECON_LINEAR) k_adj_flux_rec<KT, RECON_LINEAR><<<g, 128, 0, s>>>(c, a, r, n_lane);
    else k_adj_flux_rec<KT, RECON_MINMOD><<<g, 128, 0, s>>>(c, a, r, n_lane);
}
void KFN(adj_gather)(const DevCase& c, const AdjCase& a, cudaStream_t s) {
    k_adj_gather<KT><<<adj_nblk(c.nc, 128), 128, 0, s>>>(c, a);
}
void KFN(adj_cell)(const DevCase& c, const AdjCase& a, double coef_t, double coef_acc, int first, cudaStream_t s) {
    k_adj_cell<KT><<<adj_nblk(c.nc, 128), 128, 0, s>>>(c, a, coef_t, coef_acc, first);
}

}  // namespace cfd2d
