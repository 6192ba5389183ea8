// pcf_spectral.cuh -- the spectral preconditioner of the mixed-precision
// solve (no reference counterpart): the exact inverse of the operator whose
// coefficients are averaged over each horizontal level.
//
// The FP32 loop works on pi = s / fcscal with the difference-form operator
//     (B pi)_c = d pi_c + sum_nb B_nb (pi_nb - pi_c).
// Averaging d and the six face couplings (left/right, back/front, down, up)
// over each level k gives a separable operator with the same null space:
//     cx_k (pi_i+1 - 2 pi + pi_i-1) + cy_k (pi_j+1 - 2 pi + pi_j-1)
//       + ad_k (pi_k-1 - pi) + au_k (pi_k+1 - pi) + d_k pi,
// periodic in x and y, whose inverse is a 2-D discrete Fourier transform, one
// tridiagonal system per wave number pair along z, and the transform back.
// The terrain's variation around the level means and the metric cross terms
// are what is left for the Krylov iteration: 4-5 iterations on the benchmark
// grids (the V-cycle takes 11-16), 10 on an 8 km mountain under a 20 km lid.
//
// One application is five launches: x transforms (the p or s update of the
// iteration formed on the way in), y transforms, column solves, y transforms
// back, x transforms back.  Each moves 8-20 bytes per cell, 52 in all (the
// V-cycle: about 330 and 60 launches).  Whole solves, V-cycle -> spectral (with
// the device-side loop and the flux form, pcf_flux.cuh): 64x64x32 3.97 -> 0.60
// ms, 150x90x45 25.3 -> 1.03 (the V-cycle's coarsening ends at 75x45),
// 128x128x64 9.33 -> 1.25, 256x256x128 30.0 -> 5.01, 512x512x192 158 -> 28.0,
// 32 ensemble members 185 -> 37.
// At 512x512x192 (cold, one by one): x transforms 186 us with the p update, 176
// with the s update, y 188 either way, column solves 174, x back 152, where
// their traffic takes 154, 123, 62, 69 and 62: index arithmetic, shared-memory
// passes and barriers.
//
// Layout of the transformed field (spec): rows of nxs floats, one per (j, k),
// holding npair complex values.  Pair i >= 1 of row j is the coefficient of
// wave number i in x; pair 0 holds the two real ones (wave number 0 and, for
// even nx, nx / 2).  After the y transform, row slot y of a pair i >= 1 is the
// wave number y (complex); each half of pair 0 is a real column, so it is
// stored as the real parts of wave numbers 0..ny/2 followed by the imaginary
// parts, number ny - y in slot y.  The eigenvalues are even in both wave
// numbers, so slot y always belongs to the number min(y, ny - y).
#pragma once

#include "pcf_kernels.cuh"

namespace pcf {

constexpr int kFftMaxStages = 16;
constexpr int kFftMaxLength = 4096;  // two lines' buffers of 64 KB
constexpr int kFftThreads = 256;

// floor(b / d) for b d < 2^32 (all indices of one block's transforms)
struct FastDiv {
    unsigned d, m;
    __host__ void set(unsigned v) {
        d = v;
        m = (unsigned)((0x100000000ull + v - 1) / v);
    }
    __device__ __forceinline__ unsigned div(unsigned b) const { return d == 1 ? b : __umulhi(b, m); }
};

// Mixed-radix transform of length n: radices 8, 7, 5, 4, 3, 2, and any other
// prime by its definition.
struct FftPlan {
    int n, nst;
    int radix[kFftMaxStages];
    FastDiv m[kFftMaxStages];   // n / radix: butterflies per line
    FastDiv ns[kFftMaxStages];  // product of the earlier radices
    const float2 *tw;           // exp(-2 pi i q / n), q < n
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// -i a (forward) or i a (inverse)
template <bool INV>
__device__ __forceinline__ float2 crot(float2 a) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c, float2 &d) {
    const float2 s = cadd(a, c), t = csub(a, c), u = cadd(b, d), v = crot<INV>(csub(b, d));
    a = cadd(s, u);
    b = cadd(t, v);
    c = csub(s, u);
    d = csub(t, v);
}

// cos and sin of 2 pi j / R for the odd radices
template <int R>
__host__ __device__ constexpr float odd_cos(int j) {
    constexpr float c3[3] = {1.f, -0.5f, -0.5f};
    constexpr float c5[5] = {1.f, 0.30901699437494742f, -0.80901699437494742f, -0.80901699437494742f,
                             0.30901699437494742f};
    constexpr float c7[7] = {1.f, 0.62348980185873353f, -0.22252093395631440f, -0.90096886790241913f,
                             -0.90096886790241913f, -0.22252093395631440f, 0.62348980185873353f};
    return R == 3 ? c3[j % 3] : R == 5 ? c5[j % 5] : c7[j % 7];
}
template <int R>
__host__ __device__ constexpr float odd_sin(int j) {
    constexpr float s3[3] = {0.f, 0.86602540378443865f, -0.86602540378443865f};
    constexpr float s5[5] = {0.f, 0.95105651629515357f, 0.58778525229247313f, -0.58778525229247313f,
                             -0.95105651629515357f};
    constexpr float s7[7] = {0.f, 0.78183148246802981f, 0.97492791218182361f, 0.43388373911755812f,
                             -0.43388373911755812f, -0.97492791218182361f, -0.78183148246802981f};
    return R == 3 ? s3[j % 3] : R == 5 ? s5[j % 5] : s7[j % 7];
}

// R-point transform in registers, natural order
template <int R, bool INV>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
    if constexpr (R == 2) {
        const float2 a = v[0];
        v[0] = cadd(a, v[1]);
        v[1] = csub(a, v[1]);
    } else if constexpr (R == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        constexpr float h = 0.70710678118654752f;  // sqrt(1/2)
        dft4<INV>(v[0], v[2], v[4], v[6]);
        dft4<INV>(v[1], v[3], v[5], v[7]);
        const float2 o1 = INV ? make_float2(h * (v[3].x - v[3].y), h * (v[3].x + v[3].y))
                              : make_float2(h * (v[3].x + v[3].y), h * (v[3].y - v[3].x));
        const float2 o2 = crot<INV>(v[5]);
        const float2 o3 = INV ? make_float2(-h * (v[7].x + v[7].y), h * (v[7].x - v[7].y))
                              : make_float2(h * (v[7].y - v[7].x), -h * (v[7].x + v[7].y));
        const float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
        v[0] = cadd(e0, o0);
        v[1] = cadd(e1, o1);
        v[2] = cadd(e2, o2);
        v[3] = cadd(e3, o3);
        v[4] = csub(e0, o0);
        v[5] = csub(e1, o1);
        v[6] = csub(e2, o2);
        v[7] = csub(e3, o3);
    } else {  // odd R: pairs (q, R - q) share the cosines and sines
        float2 s[R / 2], t[R / 2], a = v[0];
#pragma unroll
        for (int q = 0; q < R / 2; ++q) {
            s[q] = cadd(v[q + 1], v[R - 1 - q]);
            t[q] = crot<INV>(csub(v[q + 1], v[R - 1 - q]));
            a = cadd(a, s[q]);
        }
        const float2 v0 = v[0];
        v[0] = a;
#pragma unroll
        for (int k = 1; k <= R / 2; ++k) {
            float2 e = v0, o = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < R / 2; ++q) {
                const float c = odd_cos<R>((q + 1) * k), sn = odd_sin<R>((q + 1) * k);
                e = make_float2(e.x + c * s[q].x, e.y + c * s[q].y);
                o = make_float2(o.x + sn * t[q].x, o.y + sn * t[q].y);
            }
            v[k] = cadd(e, o);
            v[R - k] = csub(e, o);
        }
    }
}

// Shared-memory position of element i: one complex value of padding per 128
// bytes, so that the strided writes of a stage fall into different banks.
__device__ __forceinline__ int fpad(int i) { return i + (i >> 4); }
__host__ __device__ constexpr int fpad_size(int n) { return n + (n >> 4) + 1; }

// One stage over `lines` transforms in shared memory (Stockham: reads `in`,
// writes `out`, results of the last stage in natural order).  XMAJOR: line l
// is the n elements from l n on; otherwise element e of line l is e lines + l.
template <int R, bool INV, bool XMAJOR>
__device__ __forceinline__ void fft_stage(const FftPlan &P, int st, const float2 *in, float2 *out, int lines,
                                          FastDiv dl) {
    const int n = P.n, m = (int)P.m[st].d, Ns = (int)P.ns[st].d, step = m / Ns;  // n / (Ns R)
    for (int b = threadIdx.x; b < lines * m; b += blockDim.x) {
        int l, j;
        if (XMAJOR) {
            l = (int)P.m[st].div(b);
            j = b - l * m;
        } else {
            j = (int)dl.div(b);
            l = b - j * lines;
        }
        const int k = j - (int)P.ns[st].div(j) * Ns;
        const int o = (j - k) * R + k;
        float2 v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = in[fpad(XMAJOR ? l * n + j + q * m : (j + q * m) * lines + l)];
        if (Ns > 1) {
            // the twiddles are powers of one table entry: six loads fewer per butterfly
            float2 w[R];
            w[1] = __ldg(P.tw + k * step);
            if (INV) w[1].y = -w[1].y;
#pragma unroll
            for (int q = 2; q < R; ++q) w[q] = q % 2 == 0 ? cmul(w[q / 2], w[q / 2]) : cmul(w[q - 1], w[1]);
#pragma unroll
            for (int q = 1; q < R; ++q) v[q] = cmul(v[q], w[q]);
        }
        dft<R, INV>(v);
#pragma unroll
        for (int q = 0; q < R; ++q) out[fpad(XMAJOR ? l * n + o + q * Ns : (o + q * Ns) * lines + l)] = v[q];
    }
}

// A stage of any other prime radix: every output is the sum of its definition.
template <bool INV, bool XMAJOR>
__device__ __forceinline__ void fft_stage_prime(const FftPlan &P, int st, const float2 *in, float2 *out, int lines,
                                                FastDiv dl) {
    const int n = P.n, R = P.radix[st], m = (int)P.m[st].d, Ns = (int)P.ns[st].d, step = m / Ns;
    for (int b = threadIdx.x; b < lines * n; b += blockDim.x) {
        int l, e;
        if (XMAJOR) {
            l = b / n;
            e = b - l * n;
        } else {
            e = (int)dl.div(b);
            l = b - e * lines;
        }
        const int q = (int)P.m[st].div(e), j = e - q * m;  // output q of butterfly j
        const int k = j - (int)P.ns[st].div(j) * Ns;
        const int o = (j - k) * R + k;
        const int inc = k * step + q * m;  // twiddle index per input, below n: k step < m, q m <= n - m
        float2 acc = make_float2(0.f, 0.f);
        int t = 0;
        for (int r = 0; r < R; ++r) {
            const float2 v = in[fpad(XMAJOR ? l * n + j + r * m : (j + r * m) * lines + l)];
            float2 w = __ldg(P.tw + t);
            if (INV) w.y = -w.y;
            acc = cadd(acc, cmul(v, w));
            t += inc;
            if (t >= n) t -= n;
        }
        out[fpad(XMAJOR ? l * n + o + q * Ns : (o + q * Ns) * lines + l)] = acc;
    }
}

// All stages; the caller has synchronised after filling buf0.  Returns the
// buffer that holds the result (synchronised).
template <bool INV, bool XMAJOR>
__device__ __forceinline__ float2 *fft_lines(const FftPlan &P, float2 *buf0, float2 *buf1, int lines, FastDiv dl) {
    float2 *in = buf0, *out = buf1;
    for (int st = 0; st < P.nst; ++st) {
        switch (P.radix[st]) {
            case 2: fft_stage<2, INV, XMAJOR>(P, st, in, out, lines, dl); break;
            case 3: fft_stage<3, INV, XMAJOR>(P, st, in, out, lines, dl); break;
            case 4: fft_stage<4, INV, XMAJOR>(P, st, in, out, lines, dl); break;
            case 5: fft_stage<5, INV, XMAJOR>(P, st, in, out, lines, dl); break;
            case 7: fft_stage<7, INV, XMAJOR>(P, st, in, out, lines, dl); break;
            case 8: fft_stage<8, INV, XMAJOR>(P, st, in, out, lines, dl); break;
            default: fft_stage_prime<INV, XMAJOR>(P, st, in, out, lines, dl); break;
        }
        __syncthreads();
        float2 *w = in;
        in = out;
        out = w;
    }
    return in;
}

struct SpectralArgs {
    FftPlan fx, fy;
    int nx, ny, nz;
    int nxs, npair;       // floats per row of spec, complex values used of it
    long long n, nspec;   // cells, floats of spec
    long long rows;       // ny nz
    int lines;            // x kernels: row pairs per block; y kernels: pairs (columns) per block
    FastDiv dl;           // division by lines
    float *spec;
    const float *piv;     // (nz, ny / 2 + 1, nkx): reciprocal pivots
    const float *lad, *lau;  // level means of the down and up couplings
    int nkx, nky;
    FastDiv dper, dpair;  // division by nx / V (V values per load) and by npair
    // x transforms: input forming (ThomasIn modes) and the output
    const float *in, *r, *v;
    float *vec, *out;
    float scale;
    const KrylovScalars *scal;
};

// Forward x transforms of a.lines row pairs per block: two real rows are one
// complex line, separated after the transform.  MODE forms the input as the
// Thomas sweeps do: TH_B a.in; TH_PUPD p = r + beta (p - omega v); TH_SUPD
// s = r - alpha v, written back to a.vec.  VEC: nx % 4 == 0, 128-bit loads.
template <int MODE, bool VEC>
__global__ void __launch_bounds__(kFftThreads) k_spec_x(SpectralArgs a) {
    if (krylov_done(a.scal)) return;
    extern __shared__ float2 fft_sm[];
    const int n = a.nx, lines = a.lines;
    float2 *buf0 = fft_sm, *buf1 = fft_sm + fpad_size(lines * n);
    const long long row0 = 2LL * blockIdx.x * lines;
    float alpha = 0, beta = 0, omega = 0;
    if (MODE != TH_B) {
        alpha = (float)a.scal->alpha;
        beta = (float)a.scal->beta;
        omega = (float)a.scal->omega;
    }
    // the block's rows are contiguous in memory
    constexpr int V = VEC ? 4 : 1;
    const long long base = row0 * n;
    const int nrow = (int)min((long long)2 * lines, a.rows - row0);
    const int per = n / V;
    for (int e = threadIdx.x; e < 2 * lines * per; e += blockDim.x) {
        const int row = (int)a.dper.div(e);
        const int x = (e - row * per) * V;
        float u[V];
#pragma unroll
        for (int q = 0; q < V; ++q) u[q] = 0.f;
        const long long o = base + (long long)row * n + x;
        if (row < nrow && PCF_IN(o, a.n - (V - 1), 601)) {
            if (MODE == TH_B) {
                load_vec<float, V>(a.in + o, u);
            } else {
                float r[V], v[V];
                load_vec<float, V>(a.r + o, r);
                load_vec<float, V>(a.v + o, v);
                if (MODE == TH_PUPD) {
                    float p[V];
                    using VT = typename Vec<float, V>::type;
                    const VT pv = *reinterpret_cast<const VT *>(a.vec + o);
                    const float *pe = reinterpret_cast<const float *>(&pv);
#pragma unroll
                    for (int q = 0; q < V; ++q) p[q] = pe[q];
#pragma unroll
                    for (int q = 0; q < V; ++q) u[q] = r[q] + beta * (p[q] - omega * v[q]);
                } else {
#pragma unroll
                    for (int q = 0; q < V; ++q) u[q] = r[q] - alpha * v[q];
                }
                store_vec<float, V>(a.vec + o, u);
            }
        }
        float *dst = reinterpret_cast<float *>(buf0);
#pragma unroll
        for (int q = 0; q < V; ++q) dst[2 * fpad((row >> 1) * n + x + q) + (row & 1)] = u[q];
    }
    __syncthreads();
    const float2 *z = fft_lines<false, true>(a.fx, buf0, buf1, lines, a.dl);
    // rows a and b of line l: X_a = (Z_k + conj Z_-k) / 2, X_b = (Z_k - conj Z_-k) / (2 i)
    for (int e = threadIdx.x; e < lines * a.npair; e += blockDim.x) {
        const int l = (int)a.dpair.div(e), k = e - l * a.npair;
        const long long row = row0 + 2 * l;
        if (row >= a.rows) continue;
        float2 xa, xb;
        if (k == 0) {
            const float2 z0 = z[fpad(l * n)];
            const float2 zh = (n & 1) ? make_float2(0.f, 0.f) : z[fpad(l * n + n / 2)];
            xa = make_float2(z0.x, zh.x);
            xb = make_float2(z0.y, zh.y);
            if (n == 1) xa.y = xb.y = 0.f;
        } else {
            const float2 p = z[fpad(l * n + k)], m = z[fpad(l * n + n - k)];
            xa = make_float2(0.5f * (p.x + m.x), 0.5f * (p.y - m.y));
            xb = make_float2(0.5f * (p.y + m.y), 0.5f * (m.x - p.x));
        }
        const long long o = row * a.nxs + 2 * k;
        if (PCF_IN(o + 1, a.nspec, 602)) *reinterpret_cast<float2 *>(a.spec + o) = xa;
        if (row + 1 < a.rows && PCF_IN(o + a.nxs + 1, a.nspec, 603))
            *reinterpret_cast<float2 *>(a.spec + o + a.nxs) = xb;
    }
}

// Inverse x transforms into a.out (scaled by 1 / (nx ny)).
template <bool VEC>
__global__ void __launch_bounds__(kFftThreads) k_spec_xinv(SpectralArgs a) {
    if (krylov_done(a.scal)) return;
    extern __shared__ float2 fft_sm[];
    const int n = a.nx, lines = a.lines;
    float2 *buf0 = fft_sm, *buf1 = fft_sm + fpad_size(lines * n);
    const long long row0 = 2LL * blockIdx.x * lines;
    for (int e = threadIdx.x; e < lines * a.npair; e += blockDim.x) {
        const int l = (int)a.dpair.div(e), k = e - l * a.npair;
        const long long row = row0 + 2 * l;
        float2 xa = make_float2(0.f, 0.f), xb = xa;
        const long long o = row * a.nxs + 2 * k;
        if (row < a.rows && PCF_IN(o + 1, a.nspec, 604)) xa = *reinterpret_cast<const float2 *>(a.spec + o);
        if (row + 1 < a.rows && PCF_IN(o + a.nxs + 1, a.nspec, 605))
            xb = *reinterpret_cast<const float2 *>(a.spec + o + a.nxs);
        // Z_k = X_a + i X_b, Z_-k = conj X_a + i conj X_b
        if (k == 0) {
            buf0[fpad(l * n)] = make_float2(xa.x, xb.x);
            if (!(n & 1)) buf0[fpad(l * n + n / 2)] = make_float2(xa.y, xb.y);
        } else {
            buf0[fpad(l * n + k)] = make_float2(xa.x - xb.y, xa.y + xb.x);
            buf0[fpad(l * n + n - k)] = make_float2(xa.x + xb.y, xb.x - xa.y);
        }
    }
    __syncthreads();
    const float *z = reinterpret_cast<const float *>(fft_lines<true, true>(a.fx, buf0, buf1, lines, a.dl));
    constexpr int V = VEC ? 4 : 1;
    const long long base = row0 * n;
    const int nrow = (int)min((long long)2 * lines, a.rows - row0);
    const int per = n / V;
    for (int e = threadIdx.x; e < nrow * per; e += blockDim.x) {
        const int row = (int)a.dper.div(e);
        const int x = (e - row * per) * V;
        float u[V];
#pragma unroll
        for (int q = 0; q < V; ++q) u[q] = a.scale * z[2 * fpad((row >> 1) * n + x + q) + (row & 1)];
        const long long o = base + (long long)row * n + x;
        if (PCF_IN(o, a.n - (V - 1), 606)) store_vec<float, V>(a.out + o, u);
    }
}

// y transforms of a.lines pairs (blockIdx.x) of one level (blockIdx.y), in place.
template <bool INV>
__global__ void __launch_bounds__(kFftThreads) k_spec_y(SpectralArgs a) {
    if (krylov_done(a.scal)) return;
    extern __shared__ float2 fft_sm[];
    const int n = a.ny, lines = a.lines;
    float2 *buf0 = fft_sm, *buf1 = fft_sm + fpad_size(lines * n);
    const int i0 = blockIdx.x * lines;
    float *sp = a.spec + (long long)blockIdx.y * n * a.nxs;
    const long long left = a.nspec - (long long)blockIdx.y * n * a.nxs;
    auto at = [&](int y, int i) -> float2 {
        const long long o = (long long)y * a.nxs + 2 * i;
        return PCF_IN(o + 1, left, 607) ? *reinterpret_cast<const float2 *>(sp + o) : make_float2(0.f, 0.f);
    };
    for (int e = threadIdx.x; e < lines * n; e += blockDim.x) {
        const int y = (int)a.dl.div(e), i = i0 + e - y * lines;
        float2 w = make_float2(0.f, 0.f);
        if (i < a.npair) {
            w = at(y, i);
            if (INV && i == 0) {  // the two real columns' halves back into one complex column
                const int m = y == 0 ? 0 : n - y;
                if (m != y) {
                    const float2 h = at(m, 0);
                    w = y < m ? make_float2(w.x - h.y, h.x + w.y) : make_float2(h.x + w.y, h.y - w.x);
                }
            }
        }
        buf0[fpad(e)] = w;
    }
    __syncthreads();
    const float2 *z = fft_lines<INV, false>(a.fy, buf0, buf1, lines, a.dl);
    for (int e = threadIdx.x; e < lines * n; e += blockDim.x) {
        const int y = (int)a.dl.div(e), i = i0 + e - y * lines;
        if (i >= a.npair) continue;
        float2 w = z[fpad(e)];
        if (!INV && i == 0) {  // W = C_0 + i C_h of two real columns: their real and imaginary parts
            const int m = y == 0 ? 0 : n - y;
            const float2 h = z[fpad(m * lines)];
            w = y <= m ? make_float2(0.5f * (w.x + h.x), 0.5f * (w.y + h.y))
                       : make_float2(0.5f * (h.y - w.y), 0.5f * (w.x - h.x));
        }
        const long long o = (long long)y * a.nxs + 2 * i;
        if (PCF_IN(o + 1, left, 608)) *reinterpret_cast<float2 *>(sp + o) = w;
    }
}

// The column solves, in place: forward y_k = (r_k - ad_k y_k-1) P_k, back
// x_k = y_k - au_k P_k x_k+1.  As k_thomas_split: block (32, LPC), warp w holds
// the run of CH levels from w CH on of 32 neighbouring pairs, so every load is
// issued at once and a full line wide; the runs' affine maps are chained
// through shared memory by one warp.  A pair shares its pivots (except pair 0).
template <int CH>
__global__ void __launch_bounds__(1024) k_spec_z(SpectralArgs a) {
    if (krylov_done(a.scal)) return;
    __shared__ float4 sc[32][32];  // composite of a run: (A.x, A.y, B.x, B.y)
    __shared__ float2 sin[32][32];  // value entering a run
    const int lane = threadIdx.x, part = threadIdx.y, LPC = blockDim.y;
    const int i = blockIdx.x * 32 + lane, y = blockIdx.y;
    const bool valid = i < a.npair;
    const int ky = min(y, a.ny - y);
    const bool two = i == 0 && !(a.nx & 1);  // pair 0: wave numbers 0 and nx / 2
    const int kb = part * CH;
    float2 v[CH], P[CH];
    const long long lev = (long long)a.ny * a.nxs, plev = (long long)a.nky * a.nkx;
    float *sp = a.spec + (long long)y * a.nxs + 2 * i;
    const float *pp = a.piv + (long long)ky * a.nkx;
#pragma unroll
    for (int q = 0; q < CH; ++q) {
        const int k = kb + q;
        const bool on = valid && k < a.nz &&
                        PCF_IN((long long)k * lev + (long long)y * a.nxs + 2 * i + 1, a.nspec, 609);
        v[q] = on ? *reinterpret_cast<const float2 *>(sp + k * lev) : make_float2(0.f, 0.f);
        P[q].x = on ? __ldg(pp + k * plev + i) : 0.f;
        P[q].y = two && on ? __ldg(pp + k * plev + a.nx / 2) : P[q].x;
    }
    // forward: y_out = A + B y_in over the run
    float2 A = make_float2(0.f, 0.f), B = make_float2(1.f, 1.f);
#pragma unroll
    for (int q = 0; q < CH; ++q) {
        const int k = kb + q;
        if (k < a.nz) {
            const float ad = __ldg(a.lad + k);
            A = make_float2((v[q].x - ad * A.x) * P[q].x, (v[q].y - ad * A.y) * P[q].y);
            B = make_float2(-ad * P[q].x * B.x, -ad * P[q].y * B.y);
        }
    }
    sc[part][lane] = make_float4(A.x, A.y, B.x, B.y);
    __syncthreads();
    // one warp chains the runs: every warp for itself reads half of all composites
    float2 c = make_float2(0.f, 0.f);
    if (part == 0) {
#pragma unroll 8
        for (int w = 0; w < LPC; ++w) {
            const float4 f = sc[w][lane];
            sin[w][lane] = c;
            c = make_float2(f.x + f.z * c.x, f.y + f.w * c.y);
        }
    }
    __syncthreads();
    c = sin[part][lane];
#pragma unroll
    for (int q = 0; q < CH; ++q) {
        const int k = kb + q;
        if (k < a.nz) {
            const float ad = __ldg(a.lad + k);
            c = make_float2((v[q].x - ad * c.x) * P[q].x, (v[q].y - ad * c.y) * P[q].y);
            v[q] = c;
        }
    }
    // back: x_first = A + B x_in over the run
    A = make_float2(0.f, 0.f);
    B = make_float2(1.f, 1.f);
#pragma unroll
    for (int q = CH - 1; q >= 0; --q) {
        const int k = kb + q;
        if (k < a.nz) {
            const float au = __ldg(a.lau + k);
            P[q] = make_float2(-au * P[q].x, -au * P[q].y);
            A = make_float2(v[q].x + P[q].x * A.x, v[q].y + P[q].y * A.y);
            B = make_float2(P[q].x * B.x, P[q].y * B.y);
        }
    }
    sc[part][lane] = make_float4(A.x, A.y, B.x, B.y);
    __syncthreads();
    if (part == 0) {
        c = make_float2(0.f, 0.f);
#pragma unroll 8
        for (int w = LPC - 1; w >= 0; --w) {
            const float4 f = sc[w][lane];
            sin[w][lane] = c;
            c = make_float2(f.x + f.z * c.x, f.y + f.w * c.y);
        }
    }
    __syncthreads();
    c = sin[part][lane];
#pragma unroll
    for (int q = CH - 1; q >= 0; --q) {
        const int k = kb + q;
        if (k < a.nz) {
            c = make_float2(v[q].x + P[q].x * c.x, v[q].y + P[q].y * c.y);
            if (valid && PCF_IN((long long)k * lev + (long long)y * a.nxs + 2 * i + 1, a.nspec, 610))
                *reinterpret_cast<float2 *>(sp + k * lev) = c;
        }
    }
}

// --------------------------------------------------------------- set-up --

constexpr int kLevelSums = 5;      // AL + AR, AB + AF, AD, AU, defect
constexpr int kLevelBlocks = 64;   // partial sums per level, at most

// Sums of the difference-form planes over level blockIdx.y: block b of the
// level writes its partial sums to part[(k kLevelBlocks + b) kLevelSums + q]
// (a fixed split, so the sums are deterministic).
__global__ void __launch_bounds__(256) k_level_sums(const float *__restrict__ B, int plane, long long n,
                                                    double *__restrict__ part) {
    __shared__ double sh[kLevelSums * 32];
    const int k = blockIdx.y;
    const float *b = B + (long long)plane * k;
    double s[kLevelSums] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < plane; c += gridDim.x * blockDim.x) {
        if (!PCF_IN((long long)plane * k + c, n, 611)) break;
        s[0] += (double)__ldg(b + PCF_AL * n + c) + (double)__ldg(b + PCF_AR * n + c);
        s[1] += (double)__ldg(b + PCF_AB * n + c) + (double)__ldg(b + PCF_AF * n + c);
        s[2] += (double)__ldg(b + PCF_AD * n + c);
        s[3] += (double)__ldg(b + PCF_AU * n + c);
        s[4] += (double)__ldg(b + PCF_AC * n + c);
    }
    block_sum<kLevelSums>(s, sh);
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < kLevelSums; ++q) part[((long long)k * kLevelBlocks + blockIdx.x) * kLevelSums + q] = s[q];
}

// Level means from the partial sums: lev[q nz + k], and the FP32 copies of the
// vertical couplings; one thread per level and quantity.
__global__ void k_level_means(const double *__restrict__ part, int nblk, int plane, int nz, double *__restrict__ lev,
                              float *__restrict__ lad, float *__restrict__ lau) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= kLevelSums * nz) return;
    const int q = t / nz, k = t - q * nz;
    double s = 0.0;
    for (int b = 0; b < nblk; ++b) s += part[((long long)k * kLevelBlocks + b) * kLevelSums + q];
    s /= plane;
    if (q < 2) s *= 0.5;  // one face's share
    if ((q == 2 && k == 0) || (q == 3 && k == nz - 1)) s = 0.0;  // no coupling beyond the walls
    lev[(long long)q * nz + k] = s;
    if (q == 2) lad[k] = (float)s;
    if (q == 3) lau[k] = (float)s;
}

// Reciprocal pivots of every wave number pair (kx <= nx / 2, ky <= ny / 2).
// A vanishing last pivot (the constant mode of an operator without defect)
// becomes 0: that mode's free constant is set at the top level.
__global__ void __launch_bounds__(128) k_spec_pivots(const double *__restrict__ lev, int nx, int ny, int nz, int nkx,
                                                     int nky, float *__restrict__ piv) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nkx * nky) return;
    const int ky = t / nkx, kx = t - ky * nkx;
    const double ex = 2.0 * cospi(2.0 * kx / nx) - 2.0, ey = 2.0 * cospi(2.0 * ky / ny) - 2.0;
    const double *cx = lev, *cy = lev + nz, *ad = lev + 2 * nz, *au = lev + 3 * nz, *d = lev + 4 * nz;
    double ratio = 0.0;  // au / pivot of the level below
    for (int k = 0; k < nz; ++k) {
        const double diag = d[k] - ad[k] - au[k] + cx[k] * ex + cy[k] * ey;
        const double m = diag - ad[k] * ratio;
        const double p = fabs(m) > 1e-9 * fabs(diag) ? 1.0 / m : 0.0;
        ratio = au[k] * p;
        piv[(long long)k * nkx * nky + t] = (float)p;
    }
}

}  // namespace pcf
