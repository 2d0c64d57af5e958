// GMRES on the implicit method's block system (the reference calls HYPRE's GMRES,
// src/methods/solvers/SolverHypreGmres.cpp: Krylov dimension 30, 20 iterations,
// relative tolerance 1e-7, x0 = 0, no preconditioner). Restarted GMRES with Givens
// rotations (Saad and Schultz 1986), stopping when the residual estimate
// |g_{j+1}| <= eps |b|, then checked against the true residual. The Arnoldi step
// orthogonalises with classical Gram-Schmidt: all inner products <w, v_i> in one pass
// over the basis, then w -= sum h_i v_i in a second, instead of modified Gram-Schmidt's
// j + 1 dependent passes (which the oracle and HYPRE use); in exact arithmetic both
// give the same Krylov iterate, and with the reference's at most 20 basis vectors the
// results agree with the oracle's to rounding. Krylov vectors are kept unscaled with
// their factors 1/|w|, so no normalisation pass runs.
//
// One solve is a fixed sequence of kernels (captured in the step's CUDA graph): every
// kernel first reads the control block and returns at once when the Arnoldi loop has
// ended, so iterations past convergence cost a launch each and no memory traffic. A column
// takes two kernels: k_gm_step (the end of the column before it, the block product and the
// inner products) and k_gm_orth; what a column's scalars need is reduced again by every block
// that reads them instead of by kernels of one block in between (four to nine microseconds
// each, more than the rest of a column on a small mesh).
// Reductions are deterministic: c.red partial sums (one per block), added in a fixed order.
// Built with FMA contraction (the solver is not part of the bit-exact path).
#include <cuda_runtime.h>

#include <algorithm>

#include "implicit.hpp"

namespace cfd2d {

namespace {

constexpr int kT = 256;  // threads of every grid-stride kernel

__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += sh[w];
    __syncthreads();
    return s;  // valid in thread 0
}

// sum of the n partials in a fixed order, by every block (thread 0's value broadcast)
__device__ __forceinline__ double total(const double* __restrict__ part, int n, double* sh) {
    double v = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) v += part[k];
    double s = block_sum(v, sh);
    if (threadIdx.x == 0) sh[32] = s;
    __syncthreads();
    s = sh[32];
    __syncthreads();
    return s;
}

__device__ __forceinline__ void put_partial(double v, double* part, double* sh) {
    const double s = block_sum(v, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// y = A x for the four rows of cell i: the diagonal block, then the faces' blocks in
// order, four independent accumulation chains. Every load is independent of the others
// but for the neighbours' x after their index; a boundary face's block is zero and
// points at the cell itself, so there is no branch. A block column (q) of the four rows
// is 32 contiguous bytes, so a warp's loads of it are one contiguous kilobyte.
__device__ __forceinline__ void row_matvec(const ImpCase& c, int i, const double* __restrict__ x, double y[4]) {
    const int nc = c.nc;
    const double2* x2 = reinterpret_cast<const double2*>(x);
    int nb[4];
    nb[0] = i;
    nb[1] = __ldg(c.nbr + i);
    nb[2] = __ldg(c.nbr + nc + i);
    nb[3] = __ldg(c.nbr + 2 * nc + i);
    double2 blk[4][4][2];  // [block: D, O0, O1, O2][column q][rows 0-1, 2-3]
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const double2* d = reinterpret_cast<const double2*>(c.D + dblk(nc, i, 0, q));
        blk[0][q][0] = __ldg(d);
        blk[0][q][1] = __ldg(d + 1);
    }
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double2* o = reinterpret_cast<const double2*>(c.O + oblk(nc, i, k, 0, q));
            blk[k + 1][q][0] = __ldg(o);
            blk[k + 1][q][1] = __ldg(o + 1);
        }
    double xv[4][4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double2 p = __ldg(x2 + 2 * (size_t)nb[k]), t = __ldg(x2 + 2 * (size_t)nb[k] + 1);
        xv[k][0] = p.x; xv[k][1] = p.y; xv[k][2] = t.x; xv[k][3] = t.y;
    }
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            s0 = fma(blk[k][q][0].x, xv[k][q], s0);
            s1 = fma(blk[k][q][0].y, xv[k][q], s1);
            s2 = fma(blk[k][q][1].x, xv[k][q], s2);
            s3 = fma(blk[k][q][1].y, xv[k][q], s3);
        }
    y[0] = s0; y[1] = s1; y[2] = s2; y[3] = s3;
}

// the same by one warp (the sum in lane 0)
__device__ __forceinline__ double warp_total(const double* __restrict__ part, int n) {
    double v = 0.0;
    for (int k = threadIdx.x & 31; k < n; k += 32) v += part[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
// partials of the inner products <w, V_i> and of the squared norms
__device__ __forceinline__ double* dot_part(const ImpCase& c, int i) { return c.part + (size_t)i * kRedBlocks; }
__device__ __forceinline__ double* norm_part(const ImpCase& c) { return dot_part(c, kGmresMaxKdim); }

__device__ __forceinline__ double* Vk(const ImpCase& c, int k) { return c.V + (size_t)k * 4 * c.nc; }

// The end of column j, by one warp: H[j+1][j] = |w|, s_{j+1} = 1/|w|, the Givens rotations
// (applied to the column as k_gm_orth left it in hraw), the residual estimate and whether the
// Arnoldi loop has ended. Every block that needs them runs it on what earlier kernels wrote;
// with `keep` (one block) the results go to the control block, in places the others do not read.
// Lane 0 returns the results.
struct ColEnd { double s; bool done; };
__device__ __forceinline__ ColEnd end_column(const ImpCase& c, int j, bool keep, double* col) {
    GmresCtl* g = c.ctl;
    const int lane = threadIdx.x & 31, m = c.kdim;
    double* cs = col + kGmresMaxKdim;
    double* sn = cs + kGmresMaxKdim;
    for (int i = lane; i <= j; i += 32) {
        col[i] = g->hraw[i];
        if (i < j) { cs[i] = g->cs[i]; sn[i] = g->sn[i]; }
    }
    const double hn = sqrt(warp_total(norm_part(c), c.red));
    __syncwarp();
    ColEnd r{0.0, false};
    if (lane == 0) {
        double a = col[0];
        for (int i = 0; i < j; i++) {  // a: row i after the rotations before it
            const double b = col[i + 1];
            col[i] = cs[i] * a + sn[i] * b;
            a = -sn[i] * a + cs[i] * b;
        }
        const double d = sqrt(a * a + hn * hn);
        const double cj = d == 0.0 ? 1.0 : a / d, sj = d == 0.0 ? 0.0 : hn / d;
        const double gj = g->g[j], rnorm = fabs(sj * gj);
        r.s = hn != 0.0 ? 1.0 / hn : 0.0;
        r.done = rnorm <= g->eps_abs || g->it0 + j + 1 >= c.maxit || j + 1 == m;
        if (keep) {
            for (int i = 0; i < j; i++) g->H[i * m + j] = col[i];
            g->H[j * m + j] = cj * a + sj * hn;
            g->cs[j] = cj; g->sn[j] = sj;
            g->gr[j] = cj * gj;       // the rotated right-hand side, for the back substitution
            g->g[j + 1] = -sj * gj;
            g->s[j + 1] = r.s;
            g->rnorm = rnorm;
            g->it = g->it0 + j + 1;
            g->cols = j + 1;
            if (r.done) g->done_col = j;
        }
    }
    return r;
}

// cycle start: counters, and |src|^2 partials (src = b on the first cycle, else r); x = 0 on the first
__global__ void __launch_bounds__(kT) k_gm_src_norm(const ImpCase c, int first) {
    __shared__ double sh[33];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        GmresCtl* g = c.ctl;
        if (first) { g->it = 0; g->final_ = 0; g->status = 0; g->cycle = 0; }
        g->it0 = g->it;
        g->cols = 0; g->done_col = kNotDone; g->restart = 0; g->cycle++;
        g->n_lim = 0;
        *c.n_lim = 0;
    }
    const double* src = first ? c.b : c.r;
    const size_t n = 4 * (size_t)c.nc;
    double v = 0.0;
    for (size_t q = blockIdx.x * (size_t)kT + threadIdx.x; q < n; q += (size_t)gridDim.x * kT) {
        const double s = src[q];
        v = fma(s, s, v);
        if (first) c.x[q] = 0.0;
    }
    put_partial(v, norm_part(c), sh);
}

__global__ void __launch_bounds__(kT) k_gm_v0(const ImpCase c, int first) {
    __shared__ double sh[33];
    GmresCtl* g = c.ctl;
    if (!first && g->final_) return;  // (the first cycle's start is the one that sets it)
    const double beta = sqrt(total(norm_part(c), c.red, sh));
    const double bnorm = first ? beta : g->bnorm;
    const double eps_abs = first ? c.eps * beta : g->eps_abs;
    const bool stop = beta <= eps_abs || g->it0 >= c.maxit;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (first) { g->bnorm = bnorm; g->eps_abs = eps_abs; }
        g->rnorm = beta;
        g->g[0] = beta;
        g->s[0] = 1.0;
        if (stop) {
            g->done_col = -2;
            if (first) {  // b = 0: x = 0 is the solution
                g->final_ = 1;
                g->rel = 0.0;
                g->status = 0;
            }
        }
    }
    if (stop) return;
    const double* src = first ? c.b : c.r;
    double* v0 = Vk(c, 0);
    const double ib = 1.0 / beta;
    const size_t n = 4 * (size_t)c.nc;
    for (size_t q = blockIdx.x * (size_t)kT + threadIdx.x; q < n; q += (size_t)gridDim.x * kT) v0[q] = src[q] * ib;
}

// Column j: the end of column j - 1 (by a warp of its own, while the others form their first
// rows), w = V_{j+1} = A (s_j V_j) and the partials of <w, V_i>, i < CNT. The Krylov vectors
// are kept unscaled with their factor 1/|w| in s (the scaling pass of every iteration is folded
// into its uses). The inner products read w from registers.
template <int CNT>
__global__ void __launch_bounds__(kT + 32, 3) k_gm_step(const ImpCase c, int j) {
    __shared__ double sh[CNT][kT / 32];
    __shared__ double col[3 * kGmresMaxKdim];
    __shared__ double s_j;
    __shared__ int ended;
    if (c.ctl->done_col < j - 1) return;  // (this kernel itself may set j - 1)
    const bool scalar = threadIdx.x >= kT;
    const double* vj = Vk(c, j);
    double2* w = reinterpret_cast<double2*>(Vk(c, j + 1));
    const double2* v0 = reinterpret_cast<const double2*>(c.V);
    const size_t n2 = 2 * (size_t)c.nc;
    // on a small mesh an equal share of the cells per block, else a sweep of the whole grid
    const int share = (c.nc + gridDim.x - 1) / gridDim.x;
    const bool small = share <= kT;
    int i = scalar || (small && (int)threadIdx.x >= share) ? c.nc
                                                           : (int)(blockIdx.x * (small ? share : kT) + threadIdx.x);
    double y[4];
    if (i < c.nc) row_matvec(c, i, vj, y);
    if (scalar) {
        ColEnd e{1.0, false};
        if (j > 0) e = end_column(c, j - 1, blockIdx.x == 0, col);
        if (threadIdx.x == kT) { s_j = e.s; ended = e.done; }
    }
    __syncthreads();
    if (ended) return;
    const double sj = s_j;
    double acc[CNT];
#pragma unroll
    for (int u = 0; u < CNT; u++) acc[u] = 0.0;
    while (i < c.nc) {
        const double2 a = make_double2(y[0] * sj, y[1] * sj), b = make_double2(y[2] * sj, y[3] * sj);
        w[2 * (size_t)i] = a;
        w[2 * (size_t)i + 1] = b;
#pragma unroll
        for (int u = 0; u < CNT; u++) {
            const double2 p = __ldg(v0 + (size_t)u * n2 + 2 * (size_t)i), q = __ldg(v0 + (size_t)u * n2 + 2 * (size_t)i + 1);
            acc[u] = fma(a.x, p.x, acc[u]);
            acc[u] = fma(a.y, p.y, acc[u]);
            acc[u] = fma(b.x, q.x, acc[u]);
            acc[u] = fma(b.y, q.y, acc[u]);
        }
        i = small ? c.nc : i + (int)gridDim.x * kT;
        if (i < c.nc) row_matvec(c, i, vj, y);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (!scalar)
#pragma unroll
        for (int u = 0; u < CNT; u++) {
            double v = acc[u];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) sh[u][warp] = v;
        }
    __syncthreads();
    if (threadIdx.x < CNT) {
        double t = 0.0;
        for (int k = 0; k < kT / 32; k++) t += sh[threadIdx.x][k];
        dot_part(c, threadIdx.x)[blockIdx.x] = t;
    }
}

// the partials of <w, V_i>, i = i0 .. i0 + CNT - 1, for the basis vectors past k_gm_step's
template <int CNT>
__global__ void __launch_bounds__(kT) k_gm_dots(const ImpCase c, int j, int i0) {
    __shared__ double sh[CNT][kT / 32];
    if (c.ctl->done_col < j) return;
    const double2* w = reinterpret_cast<const double2*>(Vk(c, j + 1));
    const double2* v0 = reinterpret_cast<const double2*>(Vk(c, i0));
    const size_t n2 = 2 * (size_t)c.nc;
    double acc[CNT];
#pragma unroll
    for (int u = 0; u < CNT; u++) acc[u] = 0.0;
    for (size_t q = blockIdx.x * (size_t)kT + threadIdx.x; q < n2; q += (size_t)gridDim.x * kT) {
        const double2 a = w[q];
        double2 b[CNT];
#pragma unroll
        for (int u = 0; u < CNT; u++) b[u] = v0[(size_t)u * n2 + q];
#pragma unroll
        for (int u = 0; u < CNT; u++) {
            acc[u] = fma(a.x, b[u].x, acc[u]);
            acc[u] = fma(a.y, b[u].y, acc[u]);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int u = 0; u < CNT; u++) {
        double v = acc[u];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) sh[u][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < CNT) {
        double t = 0.0;
        for (int k = 0; k < kT / 32; k++) t += sh[threadIdx.x][k];
        dot_part(c, i0 + threadIdx.x)[blockIdx.x] = t;
    }
}

// h_ij = s_i <w, V_i> from the partials (one warp per i, in a fixed order; one block keeps the
// column for its end), w -= sum_i h_ij s_i V_i, and the partials of |w|^2
__global__ void __launch_bounds__(kT) k_gm_orth(const ImpCase c, int j) {
    __shared__ double sh[33];
    __shared__ double hs[kGmresMaxKdim];
    GmresCtl* g = c.ctl;
    if (g->done_col < j) return;
    for (int i = threadIdx.x >> 5; i <= j; i += kT / 32) {
        const double v = warp_total(dot_part(c, i), c.red);
        if ((threadIdx.x & 31) == 0) {
            const double si = g->s[i], h = si * v;
            hs[i] = h * si;
            if (blockIdx.x == 0) g->hraw[i] = h;
        }
    }
    __syncthreads();
    double2* w = reinterpret_cast<double2*>(Vk(c, j + 1));
    const size_t n2 = 2 * (size_t)c.nc;
    double acc = 0.0;
    for (size_t q = blockIdx.x * (size_t)kT + threadIdx.x; q < n2; q += (size_t)gridDim.x * kT) {
        double2 a = w[q];
        for (int i = 0; i <= j; i++) {
            const double2 b = reinterpret_cast<const double2*>(Vk(c, i))[q];
            a.x = fma(-hs[i], b.x, a.x);
            a.y = fma(-hs[i], b.y, a.y);
        }
        w[q] = a;
        acc = fma(a.x, a.x, acc);
        acc = fma(a.y, a.y, acc);
    }
    put_partial(acc, norm_part(c), sh);
}

// the end of the last column if no later one has run it, and the back substitution H y = g over
// the cycle's columns, one warp: lane k holds rows k and k + 32
__global__ void __launch_bounds__(32) k_gm_solve(const ImpCase c, int last) {
    __shared__ double Hs[kGmresMaxKdim * kGmresMaxKdim];  // the n columns, row stride n
    GmresCtl* g = c.ctl;
    if (g->final_) return;
    if (g->done_col >= last) end_column(c, last, true, Hs);
    __threadfence_block();
    __syncwarp();
    const int m = c.kdim, n = g->cols, lane = threadIdx.x;
    for (int q = lane; q < n * n; q += 32) Hs[q] = g->H[(q / n) * m + q % n];
    double r0 = lane < n ? g->gr[lane] : 0.0, r1 = lane + 32 < n ? g->gr[lane + 32] : 0.0;
    __syncwarp();
    for (int i = n - 1; i >= 0; i--) {
        const double yi = __shfl_sync(0xffffffffu, (i < 32 ? r0 : r1) / Hs[i * n + i], i & 31);
        if (lane == 0) g->y[i] = yi;
        if (lane < i) r0 -= Hs[lane * n + i] * yi;
        if (lane + 32 < i) r1 -= Hs[(lane + 32) * n + i] * yi;
    }
}

// x += sum_k y_k s_k V_k
__global__ void __launch_bounds__(kT) k_gm_xupdate(const ImpCase c) {
    __shared__ double ys[kGmresMaxKdim];
    const GmresCtl* g = c.ctl;
    if (g->final_) return;
    const int n = g->cols;
    for (int k = threadIdx.x; k < n; k += kT) ys[k] = g->y[k] * g->s[k];
    __syncthreads();
    const size_t n2 = 2 * (size_t)c.nc;
    double2* x = reinterpret_cast<double2*>(c.x);
    const double2* V = reinterpret_cast<const double2*>(c.V);
    for (size_t q = blockIdx.x * (size_t)kT + threadIdx.x; q < n2; q += (size_t)gridDim.x * kT) {
        double2 s = x[q];
        for (int k = 0; k < n; k++) {
            const double2 v = V[(size_t)k * n2 + q];
            s.x = fma(ys[k], v.x, s.x);
            s.y = fma(ys[k], v.y, s.y);
        }
        x[q] = s;
    }
}

// r = b - A x and the partials of |r|^2
__global__ void __launch_bounds__(kT) k_gm_resid(const ImpCase c) {
    __shared__ double sh[33];
    if (c.ctl->final_) return;
    double acc = 0.0;
    for (int i = blockIdx.x * kT + threadIdx.x; i < c.nc; i += gridDim.x * kT) {
        double y[4];
        row_matvec(c, i, c.x, y);
        for (int k = 0; k < 4; k++) {
            const double r = c.b[4 * (size_t)i + k] - y[k];
            c.r[4 * (size_t)i + k] = r;
            acc = fma(r, r, acc);
        }
    }
    put_partial(acc, norm_part(c), sh);
}

// the true residual decides: final (with MatrixSolver's status bits) or another cycle
__global__ void __launch_bounds__(kT) k_gm_finish(const ImpCase c) {
    __shared__ double sh[33];
    GmresCtl* g = c.ctl;
    if (g->final_) return;
    const double rn = sqrt(total(norm_part(c), c.red, sh));
    if (threadIdx.x != 0) return;
    g->rnorm = rn;
    g->rel = g->bnorm > 0.0 ? rn / g->bnorm : 0.0;
    if (rn <= g->eps_abs || g->it >= c.maxit) {
        g->final_ = 1;
        g->restart = 0;
        int st = 0;
        if (g->it >= c.maxit) st |= SOLVE_MAX_ITER;
        if (!(g->rel < c.eps) || !isfinite(g->rel)) st |= SOLVE_CONVERG;
        g->status = st;
    } else {
        g->restart = 1;
    }
}

// inner products per kernel: 12 (registers: the accumulators beside the product's operands)
constexpr int kDotChunk = 12;

template <int N>
void step_n(const ImpCase& c, int j, int cnt, cudaStream_t s) {
    if constexpr (N > 0) {
        if (cnt == N) k_gm_step<N><<<c.red, kT + 32, 0, s>>>(c, j);
        else step_n<N - 1>(c, j, cnt, s);
    }
}
template <int N>
void dots_n(const ImpCase& c, int j, int i0, int cnt, cudaStream_t s) {
    if constexpr (N > 0) {
        if (cnt == N) k_gm_dots<N><<<c.red, kT, 0, s>>>(c, j, i0);
        else dots_n<N - 1>(c, j, i0, cnt, s);
    }
}

}  // namespace

// Blocks of the reductions, each a partial sum: what fits the chip at once, fewer (64 cells each)
// on a mesh that does not fill them.
int imp_red_blocks(int nc) { return std::max(1, std::min(kRedBlocks, (nc + 63) / 64)); }

void imp_launch_gmres_cycle(const ImpCase& c, bool first, cudaStream_t s) {
    const int f = first ? 1 : 0;
    k_gm_src_norm<<<c.red, kT, 0, s>>>(c, f);
    k_gm_v0<<<c.red, kT, 0, s>>>(c, f);
    const int jmax = c.kdim < c.maxit ? c.kdim : c.maxit;
    for (int j = 0; j < jmax; j++) {
        step_n<kDotChunk>(c, j, std::min(kDotChunk, j + 1), s);
        for (int i0 = kDotChunk; i0 <= j; i0 += kDotChunk) dots_n<kDotChunk>(c, j, i0, std::min(kDotChunk, j + 1 - i0), s);
        k_gm_orth<<<c.red, kT, 0, s>>>(c, j);
    }
    k_gm_solve<<<1, 32, 0, s>>>(c, jmax - 1);
    k_gm_xupdate<<<c.red, kT, 0, s>>>(c);
    k_gm_resid<<<c.red, kT, 0, s>>>(c);
    k_gm_finish<<<1, kT, 0, s>>>(c);
}

}  // namespace cfd2d
