// pcf_flux.cuh -- the assembled operator in flux form, as the spectral solves
// apply it.
//
// compute_operator!.jl's 25 coefficients per cell are products of ten values
// per cell: the operator is the scaled divergence of the winds that the
// pressure corrects (correct!.jl:177-290 followed by compute_lhs!.jl:68-160),
//     (A s)_c = SC ( dx(JP U) + dy(JP V) + dz W ) + DG pi,   pi = s / fcscal,
// with, on the faces right of, in front of and above the cell,
//     U  = KU ( pi_r - pi + cx (M13 + M13_r) (E + E_r) ),     V likewise,
//     W  = KW3 (pi_u - pi) + KW ( m13 ax (q_r - q_l) + m23 ay (q_f - q_b) )
//          + BW ( TH T + (1 - TH) T_u ),
//     T  = M13 (U + U_l) + M23 (V + V_b),    q = TH pi + (1 - TH) pi_u,
// E the vertical difference pi_u - pi_d (one-sided at the walls: -3, 4, -1),
// m13, m23 the Jacobian-weighted means of M13, M23 at the upper face.
// Applying it from these values moves 10 words per cell where the coefficient
// planes take 25, and building them costs 7 divisions per cell where the
// planes take about 30 (512x512x192: 2.8 ms in a cold profile instead of 7.7).
// Whole solves: 512x512x192 38.1 -> 29.9 ms, 256x256x128 6.56 -> 5.41, 32
// ensemble members 46.7 -> 39.1, the 256x256x128 half step 8.42 -> 7.09.  A
// constant pi gives exactly zero in any precision,
// like the difference form (k_stencil, DIFF).
//
// The values live in the first planes of the handle's coefficient buffers
// (FP64 in coef64, FP32 in coefB32); the 25 planes are assembled when an entry
// point needs them (ensure_planes).
#pragma once

#include "pcf_kernels.cuh"

namespace pcf {

enum FluxPlane : int { FX_KU = 0, FX_KV, FX_JP, FX_M13, FX_M23, FX_TH, FX_KW, FX_KW3, FX_BW, FX_SC, FX_DG, FX_N };

struct FluxBuildArgs {
    int nx, ny, nz, nxx, nyy, nbx, nby, nbz, model, damp_h;
    int z0, z1;  // levels of this launch
    double dt, rf, rdx, rdy, rdz, gamma, kappa, rsp, pref;
    const double *jac, *met13, *met23, *met33, *pbar, *rhobar, *thetabar, *n2, *rho, *betar, *p, *rfch;
    double *f64;
    float *f32;
    unsigned *uneven;  // set where a halo column is not the periodic image
};

// The flux-form values of the cells of levels [z0, z1); one thread per cell,
// 64 x 4 threads.  The arithmetic is k_assemble's (which cites the reference
// line by line), in FP64; the FP32 copy is rounded from it.
__global__ void __launch_bounds__(256, 3) k_flux_build(FluxBuildArgs a) {
    const int i = blockIdx.x * 64 + threadIdx.x, j = blockIdx.y * 4 + threadIdx.y, k = a.z0 + blockIdx.z;
    if (i >= a.nx || j >= a.ny || k >= a.z1) return;
    const long long sy = a.nxx, sz = (long long)a.nxx * a.nyy, n = (long long)a.nx * a.ny * a.nz;
    const long long c = (i + a.nbx) + sy * (j + a.nby) + sz * (k + a.nbz), r = c + 1, f = c + sy, u = c + sz;
    if (!PCF_IN(u, sz * (a.nz + 2 * a.nbz), 701)) return;
    const long long q = i + (long long)a.nx * (j + (long long)a.ny * k);
    auto put = [&](int p, double v) {
        const long long o = (long long)p * n + q;
        if (!PCF_IN(o, (long long)FX_N * n, 702)) return;
        a.f64[o] = v;
        a.f32[o] = (float)v;
    };
    const double *J = a.jac, *P = a.pbar, *RB = a.rhobar, *RO = a.rho, *BR = a.betar;
    const double jc = J[c], ju = J[u], pc = P[c], pu = P[u];
    const double tc = RO[c] + RB[c], rouc = RO[u], rbuc = RB[u];
    auto face = [&](long long o) {  // P / (damping rho) at the face towards o
        const double fac = a.damp_h ? 1.0 + a.dt * 0.5 * (BR[c] + BR[o]) * a.rf : 1.0;
        return (pc + P[o]) / (fac * (tc + (RO[o] + RB[o])));
    };
    put(FX_KU, face(r) * a.rdx);
    put(FX_KV, face(f) * a.rdy);
    put(FX_JP, jc * pc);
    put(FX_M13, a.met13[c]);
    put(FX_M23, a.met23[c]);
    // the neighbours beyond the sides are taken from the interior's other end:
    // right only where the caller's halo columns hold the same values
    auto differs = [&](long long halo, long long image) {
        return J[halo] != J[image] || P[halo] != P[image] || RB[halo] != RB[image] || RO[halo] != RO[image] ||
               a.met13[halo] != a.met13[image] || a.met23[halo] != a.met23[image] ||
               (a.damp_h && BR[halo] != BR[image]);
    };
    if ((i == 0 && differs(c - 1, c + a.nx - 1)) || (i == a.nx - 1 && differs(c + 1, c - a.nx + 1)) ||
        (j == 0 && differs(c - sy, c + sy * (a.ny - 1))) || (j == a.ny - 1 && differs(c + sy, c - sy * (a.ny - 1))))
        *a.uneven = 1u;
    const double rfc = a.rfch[c];
    put(FX_SC, rfc / jc);
    if (k + 1 < a.nz) {
        const double rj = 1.0 / (jc + ju), th = ju * rj, tu = jc * rj;  // weights of this level and the next
        const double dt2 = a.dt * a.dt;
        double fw;
        const double den = ju * tc + jc * (rouc + rbuc);
        if (a.model == PCF_MODEL_COMPRESSIBLE)
            fw = (ju * pc / a.thetabar[c] + jc * pu / a.thetabar[u]) / den;
        else
            fw = (ju * RB[c] + jc * rbuc) / den;
        const double n2 = th * a.n2[c] + tu * a.n2[u];
        const double fac = 1.0 + a.dt * (th * BR[c] + tu * BR[u]) * a.rf;
        const double b = fw * n2 * dt2;
        const double g = jc * ju * (pc + pu) * rj * a.rdz / (fac + b);  // dz, mass factor and implicit factor
        const double rho = th * tc + tu * (rouc + rbuc);
        const double kw = g * (th * pc + tu * pu) / rho;
        put(FX_TH, th);
        put(FX_KW, kw);
        put(FX_KW3, kw * (th * a.met33[c] + tu * a.met33[u]) * a.rdz);
        put(FX_BW, g * b * 0.5);
    } else {  // no face above the top level
        put(FX_TH, 1.0);
        put(FX_KW, 0.0);
        put(FX_KW3, 0.0);
        put(FX_BW, 0.0);
    }
    if (a.model == PCF_MODEL_COMPRESSIBLE) {
        const double dpdpi = 1.0 / (a.gamma - 1.0) * pow(a.rsp / a.pref, 1.0 - a.gamma) * pow(a.p[c], 2.0 - a.gamma);
        put(FX_DG, -rfc * (dpdpi / a.dt) / (a.dt * a.rsp / a.kappa));
    }
}

template <typename T>
struct FluxArgs {
    const T *f;      // the planes (FluxPlane)
    const T *s;      // pi
    T *out;
    const T *w1;     // EPI_DOT1/2: second operand; EPI_RESID: b
    int nx, ny, nz;
    long long n;
    double rdx, rdy, rdz;
    int diag;        // FX_DG is set (Compressible)
    ReduceCtx red{};
    const KrylovScalars *guard = nullptr;
    int guard_update = 0;
};

// One thread per column, marching up a chunk of kc levels with the pressure of
// its own and the four neighbouring columns at three levels in registers; the
// neighbours' values come through L1, so there is neither shared memory nor a
// barrier.  A chunk starts one level early (without output) for the flux below
// its first cell.  Bound: memory, 10 values, pi, the second operand and the
// output once per cell.  Everything a pass of the loop reads is loaded one pass
// ahead into registers: 256x256x128 in FP32 154 us (52 bytes per cell, 2.8
// TB/s; 60 % issue), without the prefetch 217 us, and 329 us when the wall
// cases were selects instead of branches (the compiler then sank each load to
// its use); 512x512x192 704 us (3.7 TB/s) where the 25 planes took 963, FP64
// 1.32 ms instead of 1.81.
constexpr int kFluxTX = 32, kFluxTY = 4;

template <typename T, int EPI>
__global__ void __launch_bounds__(kFluxTX *kFluxTY, sizeof(T) == 4 ? 4 : 2) k_flux_apply(FluxArgs<T> a, int kc) {
    if (a.guard_update ? no_update_pending(a.guard) : krylov_done(a.guard)) return;
    const int x = blockIdx.x * kFluxTX + threadIdx.x, y = blockIdx.y * kFluxTY + threadIdx.y;
    double d0 = 0.0, d1 = 0.0;
    if (x < a.nx && y < a.ny) {
        const int k0 = blockIdx.z * kc, k1 = min(k0 + kc, a.nz), top = a.nz - 1;
        const int plane = a.nx * a.ny;
        const long long n = a.n;
        // the five columns: own, left, right, back, front
        const int row = a.nx * y;
        const int col[5] = {row + x, row + (x == 0 ? a.nx - 1 : x - 1), row + (x + 1 == a.nx ? 0 : x + 1),
                            x + a.nx * (y == 0 ? a.ny - 1 : y - 1), x + a.nx * (y + 1 == a.ny ? 0 : y + 1)};
        const T cx = (T)(0.125 * a.rdz / a.rdx), cy = (T)(0.125 * a.rdz / a.rdy);
        const T ax = (T)(0.5 * a.rdx), ay = (T)(0.5 * a.rdy);
        // byte offsets within a plane (n sizeof(T) < 2^32, checked by the host): a
        // 32-bit offset on a uniform base costs one instruction per load, 64-bit
        // indices three
        const unsigned lb = (unsigned)(plane * sizeof(T));
        unsigned cb[5];
#pragma unroll
        for (int d = 0; d < 5; ++d) cb[d] = (unsigned)(col[d] * sizeof(T));
        auto word = [&](const T *base, unsigned o) -> T {
            return PCF_IN(o / sizeof(T), n, 703) ? __ldg(reinterpret_cast<const T *>(reinterpret_cast<const char *>(base) + o))
                                                 : T(0);
        };
        // value of plane p, and pi, at column d, level k
        auto at = [&](int p, int d, int k) -> T { return word(a.f + p * n, cb[d] + lb * (unsigned)k); };
        auto pi = [&](int d, int k) -> T { return word(a.s, cb[d] + lb * (unsigned)k); };
        struct Level {  // what the horizontal fluxes of a level are formed from
            T m13[3], m23[3], jp[5], kul, kur, kvb, kvf;
        };
        auto load = [&](Level &L, int k) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                L.m13[d] = at(FX_M13, d, k);
                L.m23[d] = at(FX_M23, d == 0 ? 0 : d + 2, k);
            }
#pragma unroll
            for (int d = 0; d < 5; ++d) L.jp[d] = at(FX_JP, d, k);
            L.kul = at(FX_KU, 1, k);
            L.kur = at(FX_KU, 0, k);
            L.kvb = at(FX_KV, 3, k);
            L.kvf = at(FX_KV, 0, k);
        };
        T div, t;  // horizontal divergence and coupling term of a level with pressure pc, vertical difference e
        auto fluxes = [&](const Level &L, const T (&pc)[5], const T (&e)[5]) {
            const T ul = L.kul * (pc[0] - pc[1] + cx * (L.m13[1] + L.m13[0]) * (e[0] + e[1]));
            const T ur = L.kur * (pc[2] - pc[0] + cx * (L.m13[0] + L.m13[2]) * (e[0] + e[2]));
            const T vb = L.kvb * (pc[0] - pc[3] + cy * (L.m23[1] + L.m23[0]) * (e[0] + e[3]));
            const T vf = L.kvf * (pc[4] - pc[0] + cy * (L.m23[0] + L.m23[2]) * (e[0] + e[4]));
            div = ax * ((L.jp[0] + L.jp[2]) * ur - (L.jp[1] + L.jp[0]) * ul) +
                  ay * ((L.jp[0] + L.jp[4]) * vf - (L.jp[3] + L.jp[0]) * vb);
            t = L.m13[0] * (ul + ur) + L.m23[0] * (vb + vf);
        };
        struct Next {  // what a pass of the loop reads, loaded one pass ahead
            Level L;
            T up[5], th[5], kw, kw3, bw, sc, wv, dg;
        };
        // above the top level the loads repeat it and the face's factors are 0
        auto fetch = [&](Next &N, int k) {
            k = min(k, top);
            const int k2 = min(k + 2, top);
#pragma unroll
            for (int d = 0; d < 5; ++d) {
                N.up[d] = pi(d, k2);
                N.th[d] = at(FX_TH, d, k);
            }
            load(N.L, min(k + 1, top));
            N.kw = at(FX_KW, 0, k);
            N.kw3 = at(FX_KW3, 0, k);
            N.bw = at(FX_BW, 0, k);
            N.sc = at(FX_SC, 0, k);
            N.wv = word(a.w1, cb[0] + lb * (unsigned)k);
            N.dg = a.diag ? at(FX_DG, 0, k) : T(0);
        };
        const int ks = max(k0 - 1, 0);
        T pd[5], pc[5], pu[5], e[5];
        Next N;
        load(N.L, ks);
#pragma unroll
        for (int d = 0; d < 5; ++d) {
            pd[d] = pi(d, max(ks - 1, 0));
            pc[d] = pi(d, ks);
            pu[d] = pi(d, ks + 1);
            // ks < top (nz >= 4); one-sided at the bottom, as differences (-3, 4, -1
            // written out rounds 3 pi, so a constant would not give zero)
            e[d] = ks == 0 ? T(3) * (pu[d] - pc[d]) - (pi(d, 2) - pu[d]) : pu[d] - pd[d];
        }
        fluxes(N.L, pc, e);
        T m13k = N.L.m13[0], m23k = N.L.m23[0];
        fetch(N, ks);
        T below = 0;  // flux through the face below the cell
#pragma unroll 2
        for (int k = ks; k < k1; ++k) {
            const Next C = N;
            fetch(N, k + 1);
            const T dk = div, tk = t, own = pc[0], rise = pu[0] - pc[0];
            T q[5];
            const bool last = k + 2 > top;  // level k + 1 is the top one: one-sided
#pragma unroll
            for (int d = 0; d < 5; ++d) {
                const T up = pu[d] - pc[d];
                q[d] = pu[d] - C.th[d] * up;
                e[d] = last ? T(3) * up - (pc[d] - pd[d]) : C.up[d] - pc[d];
                pd[d] = pc[d];
                pc[d] = pu[d];
                pu[d] = C.up[d];
            }
            fluxes(C.L, pc, e);
            const T th = C.th[0];
            const T above = C.kw3 * rise +
                            C.kw * ((th * (m13k - C.L.m13[0]) + C.L.m13[0]) * ax * (q[2] - q[1]) +
                                    (th * (m23k - C.L.m23[0]) + C.L.m23[0]) * ay * (q[4] - q[3])) +
                            C.bw * (th * (tk - t) + t);
            const long long o = col[0] + (long long)plane * k;
            if (k >= k0 && PCF_IN(o, n, 707)) {
                T res = C.sc * (dk + (above - below)) + C.dg * own;
                if (EPI == EPI_RESID) {
                    res = C.wv - res;
                    d0 += (double)res * (double)res;
                } else {
                    d0 += (double)res * (double)C.wv;
                    if (EPI == EPI_DOT2) d1 += (double)res * (double)res;
                }
                a.out[o] = res;
            }
            below = above;
            m13k = C.L.m13[0];
            m23k = C.L.m23[0];
        }
    }
    if (EPI == EPI_DOT2) {
        double v[2] = {d0, d1};
        reduce_finalize<2>(a.red, v);
    } else {
        double v[1] = {d0};
        reduce_finalize<1>(a.red, v);
    }
}

// k_level_sums' five sums (pcf_spectral.cuh) from the flux-form values: the
// couplings of a cell with its neighbours' pressure without the metric's cross
// terms, whose level means all but vanish.
__global__ void __launch_bounds__(256) k_flux_sums(const float *__restrict__ f, int nx, int ny, long long n, float ax,
                                                   float ay, int diag, double *__restrict__ part, int max_blocks,
                                                   int nsum) {
    __shared__ double sh[5 * 32];
    const int k = blockIdx.y, plane = nx * ny;
    const float *b = f + (long long)plane * k;
    double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < plane; c += gridDim.x * blockDim.x) {
        if (!PCF_IN((long long)plane * k + c, n, 706)) break;
        const float sc = __ldg(b + FX_SC * n + c), jp = __ldg(b + FX_JP * n + c);
        // both faces of a direction have the same mean: twice this one
        s[0] += (double)(4.f * ax * sc * jp * __ldg(b + FX_KU * n + c));
        s[1] += (double)(4.f * ay * sc * jp * __ldg(b + FX_KV * n + c));
        if (k > 0) s[2] += (double)(sc * __ldg(b + FX_KW3 * n + c - plane));
        s[3] += (double)(sc * __ldg(b + FX_KW3 * n + c));
        if (diag) s[4] += (double)__ldg(b + FX_DG * n + c);
    }
    block_sum<5>(s, sh);
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < 5; ++q) part[((long long)k * max_blocks + blockIdx.x) * nsum + q] = s[q];
}

}  // namespace pcf
