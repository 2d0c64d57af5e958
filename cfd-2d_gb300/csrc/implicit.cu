// FVM_TVD_IMPLICIT kernels that must equal the reference bit for bit: primitives,
// gradients, Gauss-point fluxes, the block-row assembly and the post-solve update
// (src/methods/fvm_tvd_implicit.cpp). Built with -fmad=false: no product is fused
// into a following sum, every expression is evaluated as the reference writes it.
#include "implicit.hpp"
#include "kernels.cuh"

namespace cfd2d {

namespace {

__device__ __forceinline__ const DevMat& imat(const ImpCase& c, int i) { return c.cmat ? c.mats[c.cmat[i]] : c.mat0; }

// FVM_TVD_IMPLICIT::boundaryCond, :963-1008. INLET: (T, P, Vx, Vy) then URS(2)
// rho = p M / (T gR); OUTLET: the cell state; WALL: the cell state with the normal
// velocity mirrored, u - 2 (u.n) n. Only r, u, v, p are consumed downstream.
__device__ __forceinline__ Prim<xd> imp_ghost(const DevBnd& b, const Prim<xd>& q, xd nx, xd ny, double M) {
    Prim<xd> g = q;
    if (b.kind == IBND_INLET) {
        g.u = xd(b.u); g.v = xd(b.v); g.p = xd(b.p);
        g.r = g.p * xd(M) / (xd(b.T) * xd(GAS_R));
    } else if (b.kind == IBND_WALL) {
        const xd Un = q.u * nx + q.v * ny;
        const xd Vx = nx * Un * xd(2.0), Vy = ny * Un * xd(2.0);
        g.u = q.u - Vx;
        g.v = q.v - Vy;
    }
    return g;
}

__global__ void __launch_bounds__(256) k_imp_prims(const ImpCase c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.nc) return;
    const int nc = c.nc;
    // convertConsToPar, :1058-1068 (URS(0): p = r e (gam - 1))
    const Prim<double> q = cons2prim<double>(c.A[i], c.A[nc + i], c.A[2 * nc + i], c.A[3 * nc + i], imat(c, i).gm1);
    store_prim(c.W, i, q);
    if (!(q.r > 0.0) || !(q.p > 0.0)) atomicOr(c.err, ERRBIT_NONPHYSICAL);  // non-positive or NaN: reported, not fixed
}

// calcGrad, :186-252: per cell over its faces in ascending edge order, the
// unreconstructed centre states and the implicit method's ghosts.
__global__ void __launch_bounds__(256) k_imp_grad(const ImpCase c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.nc) return;
    const int nc = c.nc;
    const Prim<xd> q = prim_as<xd>(load_prim(c.W, i));
    xd g[8];
#pragma unroll
    for (int m = 0; m < 8; m++) g[m] = xd(0.0);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int f = c.face[k * nc + i], e = f >> 1;
        const bool side2 = f & 1;
        const xd nx(c.nx[e]), ny(c.ny[e]), l(c.l[e]);
        Prim<xd> o;
        if (e < c.n_int) o = prim_as<xd>(load_prim(c.W, side2 ? c.ec1[e] : c.ec2[e]));
        else o = imp_ghost(c.bnds[c.ebnd[e]], q, nx, ny, imat(c, i).M);
        grad_face(g, q, o, nx, ny, l, side2);
    }
    const xd s(c.S[i]);
    const ip::Recip y = recip_of(s);
#pragma unroll
    for (int m = 0; m < 8; m++) g[m] = div_y(g[m], s, y);
    st8x(c.G, i, g);
}

// calcRoeAverage (:408-429) over roe_orig (src/global.cpp:407-441) with W = 0:
// the W terms add +0 to sums of squares and change no bit, so they are left out.
struct Roe { xd r, u, v, p, E, cz; };
__device__ __forceinline__ Roe roe_average(const Prim<xd>& L, const Prim<xd>& R, xd GAM) {
    const xd AGAM = GAM - xd(1.0);
    const xd fSB = t_sqrt(L.r), fSE = t_sqrt(R.r);
    const xd fS_ = xd(ip::rcp((fSB + fSE).v));
    Roe a;
    a.r = fSB * fSE;
    a.u = (fSB * L.u + fSE * R.u) * fS_;
    a.v = (fSB * L.v + fSE * R.v) * fS_;
    const xd EB = L.p / (L.r * AGAM), EE = R.p / (R.r * AGAM);
    const xd HB = EB + half(L.u * L.u + L.v * L.v) + L.p / L.r;
    const xd HE = EE + half(R.u * R.u + R.v * R.v) + R.p / R.r;
    const xd HI = (fSB * HB + fSE * HE) * fS_;
    a.p = (HI - half(a.u * a.u + a.v * a.v)) * a.r * (GAM - xd(1.0)) / GAM;
    const xd e = a.p / (a.r * AGAM);
    a.cz = t_sqrt(GAM * a.p / a.r);
    a.E = e + half(a.u * a.u + a.v * a.v);
    return a;
}

// The two Gauss-point fluxes of an edge times l/2 (run's loop, :612-633): interior
// faces reconstruct linearly from both centres (reconstruct(iFace, pL, pR, p),
// :444-476), boundary faces take the centre state and its ghost. Two lanes per edge, one
// Gauss point each (k_flux of the explicit method says why).
template <int FLUX>
__global__ void __launch_bounds__(128, 6) k_imp_flux(const ImpCase c) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if ((t & ~31) >= 2 * c.ne) return;
    const bool live = t < 2 * c.ne;
    const int e = live ? t >> 1 : c.ne - 1, gp = t & 1;
    const size_t ne = c.ne;
    const int c1 = c.ec1[e];
    const bool inner = e < c.n_int;
    const xd nx(c.nx[e]), ny(c.ny[e]), GAM(c.gam_flux);
    Prim<xd> pL = prim_as<xd>(load_prim(c.W, c1)), pR;
    if (inner) {
        const int c2 = c.ec2[e];
        const double* __restrict__ dl = c.dl + (size_t)(4 * gp) * ne + e;
        pR = prim_as<xd>(load_prim(c.W, c2));
        double g[8];
        ld8(c.G, c1, g);
        reconstruct<xd, RECON_LINEAR>(pL, g, xd(dl[0]), xd(dl[ne]), pL);
        ld8(c.G, c2, g);
        reconstruct<xd, RECON_LINEAR>(pR, g, xd(dl[2 * ne]), xd(dl[3 * ne]), pR);
    } else {  // both Gauss points see the same centre state and ghost
        pR = imp_ghost(c.bnds[c.ebnd[e]], pL, nx, ny, imat(c, c1).M);
    }
    xd f[4];
    bool hit = false;
    if constexpr (FLUX == FLUX_LAX) flux_lax(f, pL, pR, nx, ny, GAM, xd(c.ig1_flux), recip_of(pL.r), recip_of(pR.r));
    else hit = flux_godunov(f, pL, pR, nx, ny, c.rg_flux, c.newton_cap, recip_of(pL.r), recip_of(pR.r));
    if (hit && live) atomicOr(c.err, ERRBIT_NEWTON_CAP);
    const xd lh = half(xd(c.l[e]));  // right4 -= 0.5*l*fr, :623-633
    double out[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {  // the points' sum from +0, two components per lane
        double mine = gp ? f[2 + k].v : f[k].v;
        double other = __shfl_xor_sync(0xffffffffu, gp ? f[k].v : f[2 + k].v, 1);
        (gp ? other : mine) = ip::plus_zero(gp ? other : mine);
        out[k] = ((xd(mine) + xd(other)) * lh).v;
    }
    if (live) reinterpret_cast<double2*>(c.F)[2 * (size_t)e + gp] = make_double2(out[0], out[1]);
}

// calcRoeAverage of the edge's centre states (cellL = c1, cellR = c2 or the ghost,
// :553-554), for both cells' block rows
__global__ void __launch_bounds__(128) k_imp_roe(const ImpCase c) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= c.ne) return;
    const int c1 = c.ec1[e];
    const Prim<xd> qL = prim_as<xd>(load_prim(c.W, c1));
    const Prim<xd> qR = e < c.n_int ? prim_as<xd>(load_prim(c.W, c.ec2[e]))
                                    : imp_ghost(c.bnds[c.ebnd[e]], qL, xd(c.nx[e]), xd(c.ny[e]), imat(c, c1).M);
    const Roe a = roe_average(qL, qR, xd(c.gam_flux));
    st4(c.R, e, a.u.v, a.v.v, a.cz.v, (a.E + a.p / a.r).v);  // H of eigenValues' callers, :565
}

// (s * 0.5) * l as s * (0.5 l): halving is exact for |s| >= 2^-1021 (exponent field >= 2,
// decided on the integer pipe) and so is 0.5 l, so both round the same real number;
// a zero gives the same signed zero; smaller nonzero s take the two products (out of line,
// so that the common path is not evaluated beside them).
static __device__ __noinline__ double mul_half_l_tiny(double s, double l) { return (s * 0.5) * l; }
__device__ __forceinline__ xd mul_half_l(xd s, xd hl, xd l) {
    const long long b = __double_as_longlong(s.v);
    if (__builtin_expect(((b >> 52) & 0x7ff) >= 2 || (b << 1) == 0, 1)) return s * hl;  // (zeros: +-0 either way)
    return xd(mul_half_l_tiny(s.v, l.v));
}
__device__ __forceinline__ xd plus_zero(xd x) { return xd(ip::plus_zero(x.v)); }

// One block row of the system per cell (run's edge loop, :541-634, gathered per cell in
// ascending edge order, and the diagonal S/cTau of :640-664), four lanes per cell, one per row:
// per face the Roe average of its two centre states (k_imp_roe), A+ into the diagonal block, A-
// as the face's block, and the right-hand side -sum F l/2; steady also the spectral radius.
//
// A+- = 0.5 l R diag(lam+-) L (eigenValues / rightEigenVector / leftEigenVector / calcAP /
// calcAM, :335-406, scaled by l in run, :572-600), with the normal of the side being assembled.
// The reference forms R diag(lam+) and R diag(lam-) as full 4x4 products and multiplies each by
// L, summing four products from 0 per entry. An entry of R diag(lam+) is R[i][k] lam+_k or zero,
// and a zero term never changes such a sum (started from +0 it cannot become -0), so column k
// contributes to A+ only where lam_k > 0 and to A- only where lam_k < 0, in the reference's
// order of k: the same bits with half the products.
//
// One thread per cell held L, A- and the diagonal block (192 registers) in a body larger than
// the instruction cache; a lane holds one row of each, and the lanes divide L's quotients.
__global__ void __launch_bounds__(128) k_imp_assemble(const ImpCase c) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if ((t & ~31) >= 4 * c.nc) return;
    const bool live = t < 4 * c.nc;
    const int i = live ? t >> 2 : c.nc - 1, row = t & 3, nc = c.nc;
    const xd GAM(c.gam_flux), g1 = GAM - xd(1.0);
    xd dg[4] = {xd(0.0), xd(0.0), xd(0.0), xd(0.0)}, rhs(0.0), lsum(0.0);
#pragma unroll 1
    for (int k = 0; k < 3; k++) {
        const int f = c.face[k * nc + i], e = f >> 1;
        const bool side2 = f & 1;
        rhs = rhs + xd(neg_if(c.F[4 * (size_t)e + row], !side2));
        const xd nx(neg_if(c.nx[e], side2)), ny(neg_if(c.ny[e], side2)), l(c.l[e]), hl = half(l);
        double ra[4];  // the edge's Roe state
        ld4(c.R, e, ra);
        const xd u(ra[0]), v(ra[1]), cz(ra[2]), H(ra[3]);
        if (c.steady) lsum = lsum + (t_sqrt(u * u + v * v) + cz) * l;
        const xd qn = u * nx + v * ny, q2 = u * u + v * v;
        const xd lx = -ny, ly = nx, ql = u * lx + v * ly;
        // leftEigenVector's quotients: by c^2 in lanes 0-2, by c in lane 3
        const xd d = row == 3 ? cz : cz * cz;
        const ip::Recip y = recip_of(d);
        const xd n0 = row == 0 ? half(q2) * g1 : row == 1 ? g1 * u : row == 2 ? g1 * v : qn;
        const xd n1 = row == 0 ? half(g1) : row == 1 ? g1 : nx;
        const xd r0 = div_y(n0, d, y), r1 = div_y(n1, d, y), r2 = div_y(ny, d, y);
        auto from = [&](xd x, int lane) { return xd(__shfl_sync(0xffffffffu, x.v, lane, 4)); };
        const xd G0 = from(r1, 0), Hg = from(r1, 1), Cu = from(r0, 1), Ev = from(r0, 2), A0 = from(r0, 0);
        // A0 +- B0, Cu +- Dn, Ev +- Fn in lanes 0-2, 1 - A0 in lane 3
        const xd B0 = from(r0, 3), Dn = from(r1, 3), Fn = from(r2, 3);
        const xd x = row == 3 ? xd(1.0) : r0, z = row == 0 ? B0 : row == 1 ? Dn : row == 2 ? Fn : A0;
        const xd hp = half(x + z), dm = x - z, hm = half(dm);
        const xd L[16] = {from(hp, 0),  -from(hp, 1), -from(hp, 2), G0,
                          from(dm, 3),  Cu,           Ev,           -Hg,
                          from(hm, 0),  -from(hm, 1), -from(hm, 2), G0,
                          -ql,          lx,           ly,           xd(0.0)};
        const xd lam[4] = {qn - cz, qn, qn + cz, qn};
        // this lane's row of R
        const xd w = row == 1 ? nx : row == 2 ? ny : qn, b = row == 1 ? u : row == 2 ? v : H;
        const xd cw = cz * w;
        xd R[4] = {b - cw, b, b + cw, ly};
        if (row == 0) { R[0] = xd(1.0); R[1] = xd(1.0); R[2] = xd(1.0); R[3] = xd(0.0); }
        if (row == 1) R[3] = lx;
        if (row == 3) { R[1] = half(q2); R[3] = ql; }
        xd sp[4] = {xd(0.0), xd(0.0), xd(0.0), xd(0.0)}, sm[4] = {xd(0.0), xd(0.0), xd(0.0), xd(0.0)};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const xd s = R[q] * lam[q];
            // one sum, into the side the eigenvalue's sign names (cells of a warp differ in it)
            const bool plus = ip::positive(lam[q].v), minus = ip::positive((-lam[q]).v);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const xd t = (plus ? sp[j] : sm[j]) + s * L[4 * q + j];
                if (plus) sp[j] = t;
                if (minus) sm[j] = t;
            }
        }
        const bool inner = e < c.n_int;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            dg[j] = dg[j] + mul_half_l(sp[j], hl, l);
            const xd am = plus_zero(mul_half_l(sm[j], hl, l));
            if (live) c.O[oblk(nc, i, k, row, j)] = inner ? am.v : 0.0;
        }
    }
    const xd S(c.S[i]);
    xd tau;
    if (c.steady) {
        tau = xd(2.0) * xd(*c.cfl) * S / (lsum + xd(1.0e-100));
        if (live && row == 0) c.ctau[i] = tau.v;
    } else {
        tau = xd(c.ctau[i]);
    }
    const xd sd = S / tau;
    if (!live) return;
#pragma unroll
    for (int j = 0; j < 4; j++) c.D[dblk(nc, i, row, j)] = (j == row ? dg[j] + sd : plus_zero(dg[j])).v;  // + 0.0 off the diagonal
    c.b[4 * (size_t)i + row] = rhs.v;
}

__device__ __forceinline__ bool solve_ok(const GmresCtl* g) { return g->final_ && !g->restart && g->status == 0; }

// smoothingDelta, :790-808, for the four components at once (each pass reads and
// writes one component only): x2 = (x + a sum_nb x_nb) / (1 + a n_nb) over the
// unlimited neighbours in ascending edge order. (The reference indexes its
// neighbour sums with 4 i + shift instead of i, past their end; the sums of cell i
// are the evident intent and what is used here.)
__global__ void __launch_bounds__(256) k_imp_smooth(const ImpCase c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.nc || !solve_ok(c.ctl)) return;
    const int nc = c.nc;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    int n = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int f = c.face[k * nc + i], e = f >> 1;
        if (e >= c.n_int) continue;
        const int j = (f & 1) ? c.ec1[e] : c.ec2[e];
        if (c.flags[j] & 0x2u) continue;
        double xj[4];
        ld4(c.x, j, xj);
        for (int m = 0; m < 4; m++) s[m] = s[m] + xj[m];
        n++;
    }
    double xi[4];
    ld4(c.x, i, xi);
    const double a = c.smoothing_par;
    const double den = 1.0 + a * (double)n;
    st4(c.x2, i, (xi[0] + a * s[0]) / den, (xi[1] + a * s[1]) / den, (xi[2] + a * s[2]) / den,
        (xi[3] + a * s[3]) / den);
}

// The update of a solved system with the limits, :675-692.
__global__ void __launch_bounds__(256) k_imp_update(const ImpCase c, const double* __restrict__ dx) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool ok = solve_ok(c.ctl);
    bool lim = false;
    if (i < c.nc && ok && !(c.flags[i] & 0x2u)) {
        const int nc = c.nc;
        double d[4];
        ld4(dx, i, d);
        double U0 = c.A[i] + d[0], U1 = c.A[nc + i] + d[1], U2 = c.A[2 * nc + i] + d[2], U3 = c.A[3 * nc + i] + d[3];
        Prim<double> p = cons2prim<double>(U0, U1, U2, U3, imat(c, i).gm1);
        bool f = false;
        if (p.r > c.lim_rmax) { p.r = c.lim_rmax; f = true; }
        if (p.r < c.lim_rmin) { p.r = c.lim_rmin; f = true; }
        if (fabs(p.u) > c.lim_umax) { p.u = c.lim_umax * p.u / fabs(p.u); f = true; }
        if (fabs(p.v) > c.lim_umax) { p.v = c.lim_umax * p.v / fabs(p.v); f = true; }
        if (p.p > c.lim_pmax) { p.p = c.lim_pmax; f = true; }
        if (p.p < c.lim_pmin) { p.p = c.lim_pmin; f = true; }
        if (f) {  // par.e = p/((__GAM-1) r), convertParToCons
            const double e = p.p / ((1.4 - 1) * p.r);
            U0 = p.r;
            U1 = p.r * p.u;
            U2 = p.r * p.v;
            U3 = p.r * (e + 0.5 * (p.u * p.u + p.v * p.v));
            c.flags[i] |= 0x2u;
        }
        c.A[i] = U0; c.A[nc + i] = U1; c.A[2 * nc + i] = U2; c.A[3 * nc + i] = U3;
    }
    if (i < c.nc && ok) lim = (c.flags[i] & 0x2u) != 0;
    if (__syncthreads_or(lim) && threadIdx.x == 0) atomicAdd(c.n_lim, 1);
}

// FVM_TVD_IMPLICIT::remediateLimCells, :740-780: flagged cells in original order,
// one after another; the area-weighted mean of the cells across their faces, taken
// when those areas sum to at least TAU^2; flag aging.
__global__ void __launch_bounds__(1024) k_imp_remediate(const ImpCase c) {
    __shared__ int list[1024];
    __shared__ int cnt;
    __shared__ int wsum[32];
    const int nc = c.nc;
    if (*c.n_lim == 0 || !solve_ok(c.ctl)) return;
    for (int base = 0; base < nc; base += blockDim.x) {
        const int o = base + threadIdx.x;
        const int i = o < nc ? c.iperm[o] : -1;
        const bool fl = o < nc && (c.flags[i] & 0x2u);
        const unsigned ball = __ballot_sync(0xffffffffu, fl);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (lane == 0) wsum[warp] = __popc(ball);
        __syncthreads();
        if (threadIdx.x == 0) {
            int s = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) { int t = wsum[w]; wsum[w] = s; s += t; }
            cnt = s;
        }
        __syncthreads();
        if (fl) list[wsum[warp] + __popc(ball & ((1u << lane) - 1u))] = i;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 0; k < cnt; k++) {
                const int ci = list[k];
                double S = 0.0, a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
                for (int q = 0; q < 3; q++) {
                    const int f = c.face[q * nc + ci], e = f >> 1;
                    const int j = (f & 1) ? c.ec1[e] : c.ec2[e];
                    if (j >= 0) {
                        const double s = c.S[j];
                        S += s;
                        a0 += c.A[j] * s; a1 += c.A[nc + j] * s; a2 += c.A[2 * nc + j] * s; a3 += c.A[3 * nc + j] * s;
                    }
                }
                if (S >= c.tau_xml * c.tau_xml) {
                    c.A[ci] = a0 / S; c.A[nc + ci] = a1 / S; c.A[2 * nc + ci] = a2 / S; c.A[3 * nc + ci] = a3 / S;
                }
                unsigned f = c.flags[ci] + 0x010000u;
                if (f & 0x200000u) f &= 0x001110u;
                c.flags[ci] = f;
            }
        }
        __syncthreads();
    }
}

// getLimitedCellsCount, :782-788
__global__ void __launch_bounds__(256) k_imp_count(const ImpCase c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool lim = i < c.nc && (c.flags[i] & 0x2u);
    const int n = __syncthreads_count(lim);
    if (threadIdx.x == 0 && n && solve_ok(c.ctl)) atomicAdd(&c.ctl->n_lim, n);
}

// storage -> reference cell order of the block system: which 0 = D (16 per cell),
// 1 = O (48 per cell), 2 = b (4 per cell)
__global__ void __launch_bounds__(256) k_imp_permute(const ImpCase c, double* __restrict__ dst, int which) {
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= c.nc) return;
    const int i = c.iperm[o], nc = c.nc;
    if (which == 0)
        for (int m = 0; m < 16; m++) dst[16 * (size_t)o + m] = c.D[dblk(nc, i, m >> 2, m & 3)];
    else if (which == 1)
        for (int m = 0; m < 48; m++) dst[48 * (size_t)o + m] = c.O[oblk(nc, i, m >> 4, (m >> 2) & 3, m & 3)];
    else
        for (int m = 0; m < 4; m++) dst[4 * (size_t)o + m] = c.b[4 * (size_t)i + m];
}

inline int blocks(int n, int t) { return (n + t - 1) / t; }

}  // namespace

void imp_launch_prims(const ImpCase& c, cudaStream_t s) { k_imp_prims<<<blocks(c.nc, 256), 256, 0, s>>>(c); }
void imp_launch_grad(const ImpCase& c, cudaStream_t s) { k_imp_grad<<<blocks(c.nc, 256), 256, 0, s>>>(c); }
void imp_launch_flux(const ImpCase& c, cudaStream_t s) {
    if (c.flux == FLUX_LAX) k_imp_flux<FLUX_LAX><<<blocks(2 * c.ne, 128), 128, 0, s>>>(c);
    else k_imp_flux<FLUX_GODUNOV><<<blocks(2 * c.ne, 128), 128, 0, s>>>(c);
    k_imp_roe<<<blocks(c.ne, 128), 128, 0, s>>>(c);
}
void imp_launch_assemble(const ImpCase& c, cudaStream_t s) {
    k_imp_assemble<<<blocks(4 * c.nc, 128), 128, 0, s>>>(c);
}
void imp_launch_post(const ImpCase& c, cudaStream_t s) {
    const double* dx = c.x;
    if (c.smoothing) {
        k_imp_smooth<<<blocks(c.nc, 256), 256, 0, s>>>(c);
        dx = c.x2;
    }
    k_imp_update<<<blocks(c.nc, 256), 256, 0, s>>>(c, dx);
    k_imp_remediate<<<1, 1024, 0, s>>>(c);
    k_imp_count<<<blocks(c.nc, 256), 256, 0, s>>>(c);
}
void imp_launch_permute_blocks(const ImpCase& c, double* dst, int which, cudaStream_t s) {
    k_imp_permute<<<blocks(c.nc, 256), 256, 0, s>>>(c, dst, which);
}

}  // namespace cfd2d
