// pcf_tiny.cuh -- the whole reference BiCGSTAB (apply_bicgstab!.jl:24-150
// with apply_preconditioner!.jl:40-124 and apply_operator!.jl:48-479) in ONE
// thread-block cluster, FP64, for grids of at most kTinyMaxCells cells.  On
// such grids (the periodic hill is 40 x 1 x 40) each of the multi-kernel
// solver's ~40 launches per iteration moves a few kB, so the solve is bound by
// launch and dependency latency; here an iteration is a sequence of phases
// separated by hardware barriers.
//
// Split: the columns are shared out over the kTinyCluster CTAs in equal runs,
// a thread holds one cell (up to eight on grids of few, tall columns) with its
// Krylov vectors and, with one cell, its 25 coefficients in registers.  Only
// what other threads read is in shared memory: the column solves' input and
// pivots, and the preconditioned vector, which the stencil reads across CTAs
// through distributed shared memory.  Ten cluster barriers per iteration:
// two per preconditioner application (its second pseudo-time step, the
// operator) and two per sum.  What bounds it: the four column solves'
// chains of 2 nz dependent FP64 steps, then the barriers.
// One CTA with the coefficients read from L2 took 40 us per iteration on the
// periodic hill (25 L2 loads per cell and apply, column sweeps waiting for
// shared memory at every level); this kernel takes 24, a solve 3.29 -> 2.13 ms
// (1.94 with the assembly's shorter blocks).
//
// Global sums run in the order of one 512-thread block (kTinySumThreads
// partial sums over cells t, t + 512, ..., a shuffle tree per warp, then one
// over the warps), shared out over the CTAs through distributed shared memory:
// the iteration counts and results do not depend on the split.
#pragma once

#include <cooperative_groups.h>

#include "pcf_kernels.cuh"

namespace pcf {

constexpr int kTinyMaxCells = 2048;
constexpr int kTinyThreads = 256;
constexpr int kTinyCluster = 8;  // 2048 cells in 256-thread CTAs, one cell a thread
constexpr int kTinySumThreads = 512;
constexpr int kTinySumWarps = kTinySumThreads / 32;

struct TinyArgs {
    int nx, ny, nz, n, plane;
    int ncol;            // columns per CTA
    const double *coef;  // 25 planes
    const double *fac;   // P, M, Q for deta
    const double *b;
    double *x;           // the solution (after the final x <- M x)
    double tol;
    int maxit, precond, pc_iters;
    double deta;
    KrylovScalars *scal;  // iter, converged, status, res, b_norm
    double *hist;
    int hist_cap;
};

// shared memory of a CTA: z twice, the column solves' input, P, M, Q, the
// vectors of a sum
inline size_t tiny_smem(int ncol, int nz) { return sizeof(double) * 8 * (size_t)ncol * nz; }

template <int CPT>
__global__ void __launch_bounds__(kTinyThreads) k_tiny_bicgstab(TinyArgs a) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) double tsm[];
    __shared__ double slot[3][kTinySumWarps][2];  // the warps' partial sums, one set per kind of sum
    const int rank = (int)cl.block_rank(), tid = threadIdx.x;
    const int size = a.ncol * a.nz;              // cells of a full CTA; the last may hold fewer columns
    const int col0 = rank * a.ncol, mycol = max(0, min(a.ncol, a.plane - col0));
    const int mine = mycol * a.nz;
    double *z[2] = {tsm, tsm + size}, *tmp = tsm + 2 * size, *P = tsm + 3 * size, *M = tsm + 4 * size,
           *Q = tsm + 5 * size, *va = tsm + 6 * size, *vb = tsm + 7 * size;

    // this thread's cells: local index q = local column + ncol k
    bool on[CPT];
    int lq[CPT], kk[CPT], gc[CPT];        // local index, level, index in the grid
    const double *zc[CPT][5];             // z[0] of the 5 columns (own, left, right, back, front) at level 0
    constexpr bool KEEP = CPT == 1;       // coefficients in registers
    double cf[KEEP ? PCF_NCOEF : 1];
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
        lq[c] = tid + c * kTinyThreads;
        kk[c] = lq[c] / a.ncol;
        const int lc = lq[c] - kk[c] * a.ncol;
        on[c] = kk[c] < a.nz && lc < mycol;
        const int col = on[c] ? col0 + lc : col0 < a.plane ? col0 : 0;
        if (!on[c]) kk[c] = 0;
        gc[c] = col + a.plane * kk[c];
        const int i = col % a.nx, j = col / a.nx;
        const int ip = i + 1 == a.nx ? 0 : i + 1, im = i == 0 ? a.nx - 1 : i - 1;
        const int jp = j + 1 == a.ny ? 0 : j + 1, jm = j == 0 ? a.ny - 1 : j - 1;
        const int nb[5] = {col, im + a.nx * j, ip + a.nx * j, i + a.nx * jm, i + a.nx * jp};
#pragma unroll
        for (int d = 0; d < 5; ++d) {
            const int owner = nb[d] / a.ncol;
            zc[c][d] = cl.map_shared_rank(tsm, owner) + (nb[d] - owner * a.ncol);
        }
    }
    if constexpr (KEEP) {
#pragma unroll
        for (int p = 0; p < PCF_NCOEF; ++p) cf[p] = on[0] ? __ldg(a.coef + (long long)p * a.n + gc[0]) : 0.0;
    }
    if (a.precond)
        for (int q = tid; q < mine; q += kTinyThreads) {
            const int k = q / mycol, lc = q - k * mycol;
            const long long g = col0 + lc + (long long)a.plane * k;
            P[lc + a.ncol * k] = __ldg(a.fac + g);
            M[lc + a.ncol * k] = __ldg(a.fac + a.n + g);
            Q[lc + a.ncol * k] = __ldg(a.fac + 2 * a.n + g);
        }

    // (A z)_c for z buffer w; HORIZ: its horizontal part
    auto apply = [&](int c, int w, bool horiz) -> double {
        auto K = [&](int p) { return KEEP ? cf[KEEP ? p : 0] : __ldg(a.coef + (long long)p * a.n + gc[c]); };
        const int off = w * size;
        auto S = [&](int d, int dk) -> double {
            const int k = kk[c] + dk;
            return (k < 0 || k >= a.nz) ? 0.0 : zc[c][d][off + a.ncol * k];
        };
        double v = 0.0;
        if (!horiz) v = K(PCF_AC) * S(0, 0) + K(PCF_AD) * S(0, -1) + K(PCF_AU) * S(0, 1);
        v += K(PCF_AL) * S(1, 0) + K(PCF_AR) * S(2, 0) + K(PCF_AB) * S(3, 0) + K(PCF_AF) * S(4, 0);
        v += K(PCF_ALD) * S(1, -1) + K(PCF_ALU) * S(1, 1) + K(PCF_ARD) * S(2, -1) + K(PCF_ARU) * S(2, 1) +
             K(PCF_ABD) * S(3, -1) + K(PCF_ABU) * S(3, 1) + K(PCF_AFD) * S(4, -1) + K(PCF_AFU) * S(4, 1);
        v += K(PCF_ADD) * S(0, -2) + K(PCF_AUU) * S(0, 2) + K(PCF_ALDD) * S(1, -2) + K(PCF_ALUU) * S(1, 2) +
             K(PCF_ARDD) * S(2, -2) + K(PCF_ARUU) * S(2, 2) + K(PCF_ABDD) * S(3, -2) + K(PCF_ABUU) * S(3, 2) +
             K(PCF_AFDD) * S(4, -2) + K(PCF_AFUU) * S(4, 2);
        return v;
    };
    // column solves of tmp into z[w], one thread per column; the loads of 8
    // levels are issued ahead of the chain that uses them
    auto columns = [&](double *out) {
        if (tid < mycol) {
            constexpr int D = 8;
            double y = 0.0;
            for (int k0 = 0; k0 < a.nz; k0 += D) {
                double r[D], p[D], m[D];
#pragma unroll
                for (int q = 0; q < D; ++q) {
                    const int o = tid + a.ncol * min(k0 + q, a.nz - 1);
                    r[q] = tmp[o];
                    p[q] = P[o];
                    m[q] = M[o];
                }
#pragma unroll
                for (int q = 0; q < D; ++q) {
                    if (k0 + q < a.nz) {
                        y = r[q] * p[q] + m[q] * y;
                        out[tid + a.ncol * (k0 + q)] = y;
                    }
                }
            }
            double xs = y;
            for (int k1 = a.nz - 2; k1 >= 0; k1 -= D) {
                double r[D], f[D];
#pragma unroll
                for (int q = 0; q < D; ++q) {
                    const int o = tid + a.ncol * max(k1 - q, 0);
                    r[q] = out[o];
                    f[q] = Q[o];
                }
#pragma unroll
                for (int q = 0; q < D; ++q) {
                    if (k1 - q >= 0) {
                        xs = r[q] + f[q] * xs;
                        out[tid + a.ncol * (k1 - q)] = xs;
                    }
                }
            }
        }
    };
    // M v (or v itself) into a z buffer, visible to the cluster; returns the
    // buffer.  A buffer is written again only after a later cluster barrier
    // than the one its readers passed before reading.
    auto precondition = [&](const double (&v)[CPT]) -> int {
        if (!a.precond) {
#pragma unroll
            for (int c = 0; c < CPT; ++c)
                if (on[c]) z[0][lq[c]] = v[c];
            cl.sync();
            return 0;
        }
        int w = 0;
        for (int it = 0; it < a.pc_iters; ++it) {
#pragma unroll
            for (int c = 0; c < CPT; ++c)
                if (on[c])
                    tmp[lq[c]] = it == 0 ? -a.deta * v[c]
                                         : z[w][lq[c]] + a.deta * (apply(c, w, true) - v[c]);
            if (it > 0) w ^= 1;
            __syncthreads();
            columns(z[w]);
            cl.sync();
        }
        return w;
    };
    // sum(a b) and, for TWO, sum(a a) over the grid, the same in every thread;
    // a and b are this thread's cells
    auto sum = [&](const double (&u)[CPT], const double (&w)[CPT], int kind, bool two, double &ab, double &aa) {
#pragma unroll
        for (int c = 0; c < CPT; ++c)
            if (on[c]) {
                va[lq[c]] = u[c];
                vb[lq[c]] = w[c];
            }
        cl.sync();
        // warp v of the sum, two per CTA: its lanes' cells, wherever they are
        constexpr int per = kTinySumWarps / kTinyCluster;
        const int warp = tid >> 5, lane = tid & 31;
        if (warp < per) {
            const int t = (rank * per + warp) * 32 + lane;
            double s0 = 0.0, s1 = 0.0;
            for (int c = t; c < a.n; c += kTinySumThreads) {
                const int k = c / a.plane, col = c - a.plane * k, owner = col / a.ncol;
                const double *base = cl.map_shared_rank(tsm, owner) + (col - owner * a.ncol) + a.ncol * k;
                const double x0 = base[6 * size], x1 = base[7 * size];
                s0 += x0 * x1;
                if (two) s1 += x0 * x0;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
            if (two)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            if (lane < kTinyCluster) {
                double(*d)[2] = cl.map_shared_rank(&slot[kind][0], lane);
                d[rank * per + warp][0] = s0;
                d[rank * per + warp][1] = s1;
            }
        }
        cl.sync();
        double s0 = lane < kTinySumWarps ? slot[kind][lane][0] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        ab = s0;
        if (two) {
            double s1 = lane < kTinySumWarps ? slot[kind][lane][1] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            aa = s1;
        }
    };

    // apply_bicgstab!.jl:44-67: x = 0, r = r0 = p = b
    double x[CPT], r[CPT], r0[CPT], p[CPT], v[CPT], s[CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
        r[c] = r0[c] = p[c] = on[c] ? a.b[gc[c]] : 0.0;
        x[c] = v[c] = s[c] = 0.0;
    }
    cl.sync();  // every CTA runs before its shared memory is read or written from another
    double rho, d0, d1;
    sum(r, r, 2, false, rho, d1);
    const double b_norm = sqrt(rho / a.n);
    double res = b_norm;
    int iter = 0, converged = 0, status = PCF_OK;
    if (!isfinite(b_norm)) status = PCF_ENONFINITE;
    else if (b_norm == 0.0 || res / b_norm <= a.tol) converged = 1;
    while (status == PCF_OK && !converged && iter < a.maxit) {
        iter += 1;
        // v = A M p; alpha = rho / <v, r0>   (:84-96)
        int w = precondition(p);
#pragma unroll
        for (int c = 0; c < CPT; ++c) v[c] = on[c] ? apply(c, w, false) : 0.0;
        sum(v, r0, 0, false, d0, d1);
        const double alpha = rho / d0;
        if (!isfinite(alpha)) {
            status = PCF_EBREAKDOWN;
            break;
        }
        // t = A M s; omega = <t, s> / <t, t>   (:98-109)
#pragma unroll
        for (int c = 0; c < CPT; ++c) s[c] = r[c] - alpha * v[c];
        w = precondition(s);
        double t[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) t[c] = on[c] ? apply(c, w, false) : 0.0;
        sum(t, s, 1, true, d0, d1);
        const double omega = d0 / d1;
        if (!isfinite(omega) || omega == 0.0) {
            status = PCF_EBREAKDOWN;
            break;
        }
        // x += alpha p + omega s; r = s - omega t; residual test, beta   (:110-143)
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
            x[c] += alpha * p[c] + omega * s[c];
            r[c] = s[c] - omega * t[c];
        }
        sum(r, r0, 2, true, d1, d0);  // <r, r0>, <r, r>
        res = sqrt(d0 / a.n);
        if (rank == 0 && tid == 0 && a.hist && iter - 1 < a.hist_cap) a.hist[iter - 1] = res / b_norm;
        if (!isfinite(res)) {
            status = PCF_ENONFINITE;
            break;
        }
        if (res / b_norm <= a.tol) {
            converged = 1;
            break;
        }
        const double beta = alpha / omega * d1 / rho;
        rho = d1;
        if (!isfinite(beta)) {
            status = PCF_EBREAKDOWN;
            break;
        }
#pragma unroll
        for (int c = 0; c < CPT; ++c) p[c] = r[c] + beta * (p[c] - omega * v[c]);
    }
    // solution = M(solution) on convergence (:132-135)
    if (converged && iter > 0 && a.precond) {
        const int w = precondition(x);
#pragma unroll
        for (int c = 0; c < CPT; ++c)
            if (on[c]) x[c] = z[w][lq[c]];
    }
#pragma unroll
    for (int c = 0; c < CPT; ++c)
        if (on[c]) a.x[gc[c]] = x[c];
    if (rank == 0 && tid == 0) {
        KrylovScalars *k = a.scal;
        k->iter = iter;
        k->converged = converged;
        k->status = status;
        k->res = res;
        k->b_norm = b_norm;
        k->done = 1;
    }
    cl.sync();  // no CTA leaves while another may still read its shared memory
}

}  // namespace pcf
