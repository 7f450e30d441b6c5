// fp64.cu -- the double-precision state path (plan precision FULLMAG_FDM_PRECISION_DOUBLE).
//
// State, stage derivatives, fields, the FFT convolution and every reduction are FP64.
// The passes are those of the FP32 path -- a fused row pass and the column passes of the
// convolution, with this engine's own mixed-radix FP64 line transforms in shared memory (no
// cuFFT), the real, octant-unique demag kernel held in FP64, and the FP64 GPU Newell builder
// when the caller passes no spectra.  GB300 issues FP64 at a small fraction of its FP32 rate,
// so the work per point is chosen for the fewest FP64 instructions.
//
// Reference behaviour restated (paths in mzrptu/fullmag):
//   precision switch, plan validation          native/backends/fdm/src/api.cpp:97,324-395,533
//   exchange: mask clamp, region table          native/backends/fdm/src/exchange_fp64.cu:23-130
//   boundary tier T0 (face-link exchange)       native/backends/fdm/src/exchange_t0_fp64.cu:27-164
//   boundary tier T1 (boundary stencil)         native/backends/fdm/src/exchange_t1_fp64.cu:38-204
//   tier dispatch                               native/backends/fdm/src/exchange_fp64.cu:162-231
//   demag input phi Ms m, sparse correction      native/backends/fdm/src/demag_fp64.cu:55-90,440-545,
//                                               demag_boundary_fp64.cu:23-76
//   local terms, LLG right-hand side            native/backends/fdm/src/llg_fp64.cu
//   Heun / RK4 / DP45 / RK23 / ABM3 in FP64       llg_fp64.cu, llg_rk4_fp64.cu, llg_dp45_fp64.cu,
//                                               llg_rk23_fp64.cu, llg_abm3_fp64.cu
//   phi-weighted energies                        native/backends/fdm/src/reductions_fp64.cu:123-260,415-520
// Two kept differences from those kernels, both where the reference contradicts its own
// stated intent ("interior cells (phi = 1, f = 1) produce the standard exchange"):
//   * without region ids the T0 and T1 kernels scale by 2A/(mu0 Ms) and also weight
//     every face by A, so A enters twice; here A enters once, as in the standard kernel;
//   * cells with phi <= 0 (or m = 0) return before writing H there; here H = 0 there.
#include "fp64.h"

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "engine.h"

namespace fm {

namespace {

constexpr int kT = 256;
constexpr double kMu0d = 4.0 * M_PI * 1e-7;
constexpr int kMaxRadixStages = 32;
constexpr int kStats = 9;  // e_ex e_d e_ext e_uni e_cub | max|Heff|^2 max|Hd|^2 max|k|^2 max err^2
constexpr int kMaxBlocks = 1024;          // grid-stride conversions
constexpr size_t kMaxSmem = 227 * 1024;   // shared memory of one CTA

struct Plan64 {
    int n;
    int ns;
    int radix[kMaxRadixStages];
    const double2 *tw;  // n entries, e^{-2 pi i e / n}
};

__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zconj(double2 a) { return make_double2(a.x, -a.y); }
template <bool INV>
__device__ __forceinline__ double2 ztw(const double2 *tw, int e) {
    const double2 w = __ldg(tw + e);
    return INV ? zconj(w) : w;
}
// times -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ double2 zmi(double2 a) {
    return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// ---- FP64 line transforms ----
// GB300 issues FP64 at 1/64 of its FP32 rate, so these passes are bound by the number of
// FP64 instructions and by little else: shared-memory exchanges, index arithmetic and bank
// conflicts of 16-byte elements hide behind them.  Hence radix-8 butterflies (10.5
// instructions per point for three binary levels, twiddles included, against 7 for two with
// radix 4), odd radices as folded symmetric sums (R-1)^2 + O(R) multiply-adds instead of
// R^2 complex products, and half transforms where one half of a line is zero or unwanted.

// R-point DFT in place.  HIN: the upper R/2 inputs are zero; HOUT: only the lower R/2
// outputs are wanted.  tw: the table of the line's length n, W_R^e = tw[e n / R] (odd R).
template <int R, bool INV, bool HIN, bool HOUT>
__device__ __forceinline__ void dft64(double2 (&v)[R], const double2 *__restrict__ tw, int rs) {
    if constexpr (R == 2) {
        if constexpr (HIN) {
            v[1] = v[0];
        } else {
            const double2 a = v[0], b = v[1];
            v[0] = zadd(a, b);
            if constexpr (!HOUT) v[1] = zsub(a, b);
        }
    } else if constexpr (R == 4) {
        if constexpr (HIN) {
            const double2 a = v[0], b = v[1], ib = zmi<INV>(b);
            v[0] = zadd(a, b);
            v[2] = zsub(a, b);
            v[1] = zadd(a, ib);
            v[3] = zsub(a, ib);
        } else {
            const double2 a0 = zadd(v[0], v[2]), a1 = zsub(v[0], v[2]);
            const double2 b0 = zadd(v[1], v[3]), b1 = zmi<INV>(zsub(v[1], v[3]));
            v[0] = zadd(a0, b0);
            v[1] = zadd(a1, b1);
            if constexpr (!HOUT) {
                v[2] = zsub(a0, b0);
                v[3] = zsub(a1, b1);
            }
        }
    } else if constexpr (R == 8) {
        const double h = 0.70710678118654752440;
        double2 e[4], o[4];
        if constexpr (HOUT) {
            // decimation in time: y[t] = E[t] + W8^t O[t], t < 4
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                e[t] = v[2 * t];
                o[t] = v[2 * t + 1];
            }
            dft64<4, INV, false, false>(e, tw, rs);
            dft64<4, INV, false, false>(o, tw, rs);
            const double2 q1 = zmi<INV>(o[1]), q3 = zmi<INV>(o[3]);
            o[1] = make_double2(h * (o[1].x + q1.x), h * (o[1].y + q1.y));
            o[2] = zmi<INV>(o[2]);
            o[3] = make_double2(h * (q3.x - o[3].x), h * (q3.y - o[3].y));
#pragma unroll
            for (int t = 0; t < 4; ++t) v[t] = zadd(e[t], o[t]);
        } else {
            // decimation in frequency: even outputs from v[t] + v[t+4], odd ones from
            // W8^t (v[t] - v[t+4])
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                e[t] = HIN ? v[t] : zadd(v[t], v[t + 4]);
                o[t] = HIN ? v[t] : zsub(v[t], v[t + 4]);
            }
            const double2 q1 = zmi<INV>(o[1]), q3 = zmi<INV>(o[3]);
            o[1] = make_double2(h * (o[1].x + q1.x), h * (o[1].y + q1.y));
            o[2] = zmi<INV>(o[2]);
            o[3] = make_double2(h * (q3.x - o[3].x), h * (q3.y - o[3].y));
            dft64<4, INV, false, false>(e, tw, rs);
            dft64<4, INV, false, false>(o, tw, rs);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                v[2 * t] = e[t];
                v[2 * t + 1] = o[t];
            }
        }
    } else {
        // odd R: with s_t = v_t + v_{R-t}, d_t = v_t - v_{R-t},
        //   X_q, X_{R-q} = v_0 + sum_t cos(2 pi q t / R) s_t  -+ i sum_t sin(2 pi q t / R) d_t
        constexpr int H = (R - 1) / 2;
        double2 s[H], d[H];
        double2 x0 = v[0];
        const double2 v0 = v[0];
#pragma unroll
        for (int t = 0; t < H; ++t) {
            s[t] = zadd(v[1 + t], v[R - 1 - t]);
            d[t] = zsub(v[1 + t], v[R - 1 - t]);
            x0 = zadd(x0, s[t]);
        }
        v[0] = x0;
#pragma unroll
        for (int q = 1; q <= H; ++q) {
            double2 c = v0, z = make_double2(0.0, 0.0);
#pragma unroll
            for (int t = 0; t < H; ++t) {
                const double2 w = __ldg(tw + ((q * (t + 1)) % R) * rs);  // (cos, -sin)
                c.x += w.x * s[t].x;
                c.y += w.x * s[t].y;
                z.x += w.y * d[t].x;
                z.y += w.y * d[t].y;
            }
            // i z for the forward transform (w.y = -sin), -i z for the inverse
            const double2 iz = INV ? make_double2(z.y, -z.x) : make_double2(-z.y, z.x);
            v[q] = zadd(c, iz);
            v[R - q] = zsub(c, iz);
        }
    }
}

// One Stockham stage of radix R over nl lines of length n (line l at l * ls); twiddles on
// every stage but the first (Ns == 1).
template <int R, bool INV, bool HIN, bool HOUT>
__device__ __forceinline__ void stage64(const double2 *__restrict__ in, double2 *__restrict__ out, int nl, int ls, int n,
                                        int Ns, const double2 *__restrict__ tw) {
    const int nb = n / R, tws = n / (Ns * R);
    for (int idx = threadIdx.x; idx < nl * nb; idx += blockDim.x) {
        const int l = idx / nb, j = idx - l * nb;
        const int q = j / Ns, k = j - q * Ns;
        const double2 *src = in + l * ls + j;
        double2 *dst = out + l * ls + q * Ns * R + k;
        double2 v[R];
#pragma unroll
        for (int t = 0; t < (HIN ? R / 2 : R); ++t) v[t] = src[t * nb];
        if (!HIN && Ns > 1) {
#pragma unroll
            for (int t = 1; t < R; ++t) v[t] = zmul(v[t], ztw<INV>(tw, t * k * tws));
        }
        dft64<R, INV, HIN, HOUT>(v, tw, nb);
#pragma unroll
        for (int t = 0; t < (HOUT ? R / 2 : R); ++t) dst[t * Ns] = v[t];
    }
}

// prime radix above 13 (caller spectra or periodic extents with such a factor): O(R^2)
template <bool INV>
__device__ __noinline__ void stage64_generic(const double2 *__restrict__ in, double2 *__restrict__ out, int nl, int ls, int n,
                                             int Ns, int R, const double2 *__restrict__ tw) {
    const int nb = n / R, tws = n / (Ns * R);
    for (int idx = threadIdx.x; idx < nl * n; idx += blockDim.x) {
        const int l = idx / n, r = idx - l * n;
        const int q = r / nb, j = r - q * nb;  // output q of butterfly j
        const int k = j % Ns, o = (j / Ns) * Ns * R + k;
        const double2 *src = in + l * ls + j;
        double2 acc = make_double2(0.0, 0.0);
        int e = 0;  // (t q) mod R
        for (int t = 0; t < R; ++t) {
            double2 x = src[t * nb];
            if (Ns > 1 && t) x = zmul(x, ztw<INV>(tw, t * k * tws));
            acc = zadd(acc, zmul(x, ztw<INV>(tw, e * nb)));
            e += q;
            if (e >= R) e -= R;
        }
        out[l * ls + o + q * Ns] = acc;
    }
}

// nl lines of length p.n in shared memory (natural order in and out) by the whole CTA;
// returns the buffer that holds the result.  The radices run in plan order forwards and in
// reverse order backwards, so radix[0] is the first forward and the last inverse stage:
// with `prune` (an even radix[0], data in the lower half only) those two work on half
// lines.  Contains __syncthreads: every thread of the CTA calls it; the caller has
// synchronised the buffers.
template <bool INV>
__device__ __forceinline__ double2 *fft_lines64(double2 *a, double2 *b, int nl, int ls, const Plan64 &p, bool prune) {
    int Ns = 1;
    const int n = p.n;
    for (int s = 0; s < p.ns; ++s) {
        const int R = p.radix[INV ? p.ns - 1 - s : s];
        const bool half = prune && (INV ? s == p.ns - 1 : s == 0);
        switch (R) {
            case 8:
                if (half) stage64<8, INV, !INV, INV>(a, b, nl, ls, n, Ns, p.tw);
                else stage64<8, INV, false, false>(a, b, nl, ls, n, Ns, p.tw);
                break;
            case 4:
                if (half) stage64<4, INV, !INV, INV>(a, b, nl, ls, n, Ns, p.tw);
                else stage64<4, INV, false, false>(a, b, nl, ls, n, Ns, p.tw);
                break;
            case 2:
                if (half) stage64<2, INV, !INV, INV>(a, b, nl, ls, n, Ns, p.tw);
                else stage64<2, INV, false, false>(a, b, nl, ls, n, Ns, p.tw);
                break;
            case 3: stage64<3, INV, false, false>(a, b, nl, ls, n, Ns, p.tw); break;
            case 5: stage64<5, INV, false, false>(a, b, nl, ls, n, Ns, p.tw); break;
            case 7: stage64<7, INV, false, false>(a, b, nl, ls, n, Ns, p.tw); break;
            case 11: stage64<11, INV, false, false>(a, b, nl, ls, n, Ns, p.tw); break;
            case 13: stage64<13, INV, false, false>(a, b, nl, ls, n, Ns, p.tw); break;
            default: stage64_generic<INV>(a, b, nl, ls, n, Ns, R, p.tw); break;
        }
        __syncthreads();
        double2 *t = a;
        a = b;
        b = t;
        Ns *= R;
    }
    return a;
}

struct Conv64 {
    int nx, ny, nz, px, py, pz, nkx, nky, nkz, thin;
    long long n;
    int half;              // px / 2 when the x lines are packed (two real samples per complex one), else 0
    int xprune, yprune, zprune;  // half-line first / last stages (fft_lines64)
    Plan64 plx, ply, plz;  // plx: length half (packed) or px
    const double2 *xpost;  // packed: e^{-2 pi i k / px}, k <= half
    const double *kern;    // octant kernel scaled by Ms / P, and by 1/2 with packed x lines
    const double2 *kernc;  // periodic grids: complex kernel K[c][kz][ky][kx] (full ky, kz), else NULL
};

// U independent loads per thread in flight before the first is stored
template <int U, typename Load, typename Store>
__device__ __forceinline__ void copy64(int total, Load ld, Store st) {
    for (int base = threadIdx.x; base < total; base += U * blockDim.x) {
        double2 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int idx = base + u * (int)blockDim.x;
            if (idx < total) v[u] = ld(idx);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int idx = base + u * (int)blockDim.x;
            if (idx < total) st(idx, v[u]);
        }
    }
}

// ---- x lines of one batch: nl lines starting at line0 (line = 3 (row - row0) + c) ----
// Packed lines carry z[j] = s[2j] + i s[2j+1]; the forward split stores twice the spectrum
// (the factor is in the kernel), the inverse forms 2 Z[k] from X[k] and X[half - k].
__device__ __forceinline__ double2 *x_inverse_lines(const Conv64 &C, const double2 *__restrict__ X, int row0, int line0, int nl,
                                                    double2 *a, double2 *b, int ls) {
    const size_t nrows = (size_t)C.ny * C.nz;
    if (C.half) {
        const int half = C.half;
        for (int idx = threadIdx.x; idx < nl * half; idx += blockDim.x) {
            const int l = idx / half, k = idx - l * half;
            const int rr = (line0 + l) / 3, c = line0 + l - 3 * rr;
            const double2 *src = X + (c * nrows + row0 + rr) * C.nkx;
            const double2 p = src[k], q = src[half - k], w = __ldg(C.xpost + k);
            const double2 d = make_double2(p.x - q.x, p.y + q.y);  // X[k] - conj X[half-k]
            const double ox = d.x * w.x + d.y * w.y, oy = d.y * w.x - d.x * w.y;
            a[l * ls + k] = make_double2((p.x + q.x) - oy, (p.y - q.y) + ox);
        }
    } else {
        for (int idx = threadIdx.x; idx < nl * C.px; idx += blockDim.x) {
            const int l = idx / C.px, k = idx - l * C.px;
            const int rr = (line0 + l) / 3, c = line0 + l - 3 * rr;
            const double2 *src = X + (c * nrows + row0 + rr) * C.nkx;
            a[l * ls + k] = k < C.nkx ? src[k] : zconj(src[C.px - k]);
        }
    }
    __syncthreads();
    return fft_lines64<true>(a, b, nl, ls, C.plx, C.xprune != 0);
}

// samples H[(line0 + l) * nx + x] -> X rows
__device__ __forceinline__ void x_forward_lines(const Conv64 &C, double2 *__restrict__ X, const double *H, int row0, int line0,
                                                int nl, double2 *a, double2 *b, int ls) {
    const size_t nrows = (size_t)C.ny * C.nz;
    const int nx = C.nx, len = C.half ? C.half : C.px;
    const int lim = C.xprune ? len / 2 : len;  // the pruned first stage reads the lower half only
    for (int idx = threadIdx.x; idx < nl * lim; idx += blockDim.x) {
        const int l = idx / lim, j = idx - l * lim;
        const double *h = H + (size_t)(line0 + l) * nx;
        double2 v = make_double2(0.0, 0.0);
        if (C.half) {
            if (2 * j < nx) v.x = h[2 * j];
            if (2 * j + 1 < nx) v.y = h[2 * j + 1];
        } else if (j < nx) {
            v.x = h[j];
        }
        a[l * ls + j] = v;
    }
    __syncthreads();
    const double2 *r = fft_lines64<false>(a, b, nl, ls, C.plx, C.xprune != 0);
    for (int idx = threadIdx.x; idx < nl * C.nkx; idx += blockDim.x) {
        const int l = idx / C.nkx, k = idx - l * C.nkx;
        const int rr = (line0 + l) / 3, c = line0 + l - 3 * rr;
        double2 v;
        if (C.half) {
            const double2 p = r[l * ls + (k == C.half ? 0 : k)], q = r[l * ls + (k == 0 ? 0 : C.half - k)];
            const double2 w = __ldg(C.xpost + k);
            const double2 o = make_double2(p.y + q.y, q.x - p.x);  // -i (Z[k] - conj Z[half-k])
            v = make_double2((p.x + q.x) + (w.x * o.x - w.y * o.y), (p.y - q.y) + (w.x * o.y + w.y * o.x));
        } else {
            v = r[l * ls + k];
        }
        X[(c * nrows + row0 + rr) * C.nkx + k] = v;
    }
}

// Rows too long for the fused row pass's shared memory: one line per CTA, full-length lines.
__global__ void x_forward64(const Conv64 C, const double *__restrict__ m, const double *__restrict__ phi,
                            double2 *__restrict__ X) {
    extern __shared__ double2 sm64[];
    double2 *a = sm64, *b = sm64 + C.px;
    const int row = blockIdx.x, c = blockIdx.y;
    const size_t nrows = (size_t)C.ny * C.nz;
    const long long base = (long long)row * C.nx;
    for (int x = threadIdx.x; x < C.px; x += blockDim.x) {
        double v = 0.0;
        if (x < C.nx) {
            v = m[c * C.n + base + x];
            if (phi) v *= phi[base + x];
        }
        a[x] = make_double2(v, 0.0);
    }
    __syncthreads();
    const double2 *r = fft_lines64<false>(a, b, 1, C.px, C.plx, false);
    for (int k = threadIdx.x; k < C.nkx; k += blockDim.x) X[(c * nrows + row) * C.nkx + k] = r[k];
}
__global__ void x_inverse64(const Conv64 C, const double2 *__restrict__ X, double *__restrict__ hd) {
    extern __shared__ double2 sm64[];
    const int row = blockIdx.x, c = blockIdx.y;
    double2 *a = sm64, *b = sm64 + C.px;
    const size_t nrows = (size_t)C.ny * C.nz;
    const double2 *src = X + (c * nrows + row) * C.nkx;
    for (int k = threadIdx.x; k < C.px; k += blockDim.x) a[k] = k < C.nkx ? src[k] : zconj(src[C.px - k]);
    __syncthreads();
    const double2 *r = fft_lines64<true>(a, b, 1, C.px, C.plx, false);
    for (int x = threadIdx.x; x < C.nx; x += blockDim.x) hd[c * C.n + (long long)row * C.nx + x] = r[x].x;
}

// sign flip on the integer pipe
__device__ __forceinline__ double zneg_if(bool neg, double v) {
    return __longlong_as_double(__double_as_longlong(v) ^ (neg ? 0x8000000000000000ull : 0ull));
}

__device__ __forceinline__ double2 zmadd(double2 k, double2 m, double2 acc) {
    return make_double2(acc.x + k.x * m.x - k.y * m.y, acc.y + k.x * m.y + k.y * m.x);
}

// H(k) = -N(k) M(k) on three lines a[0..2] at (kx, ky, kz) of the octant kernel, or of the
// complex kernel of a periodic grid (components xx yy zz xy xz yz; 2-D: the first four)
__device__ __forceinline__ void multiply3(const Conv64 &C, double2 *mx, double2 *my, double2 *mz, int kx, int ky, int kz) {
    if (C.kernc) {
        const long long kc = (long long)C.pz * C.py * C.nkx;
        const double2 *K = C.kernc + ((long long)kz * C.py + ky) * C.nkx + kx;
        const double2 z0 = make_double2(0.0, 0.0);
        const double2 kxx = K[0], kyy = K[kc], kzz = K[2 * kc], kxy = K[3 * kc];
        const double2 kxz = C.thin ? z0 : K[4 * kc], kyz = C.thin ? z0 : K[5 * kc];
        const double2 a = *mx, b = *my, d = *mz;
        const double2 hx = zmadd(kxz, d, zmadd(kxy, b, zmadd(kxx, a, z0)));
        const double2 hy = zmadd(kyz, d, zmadd(kyy, b, zmadd(kxy, a, z0)));
        const double2 hz = zmadd(kzz, d, zmadd(kyz, b, zmadd(kxz, a, z0)));
        *mx = make_double2(-hx.x, -hx.y);
        *my = make_double2(-hy.x, -hy.y);
        *mz = make_double2(-hz.x, -hz.y);
        return;
    }
    const bool ny_ = ky > C.py / 2;  // mirrored frequencies: odd components change sign
    const int kym = ny_ ? C.py - ky : ky;
    const double2 a = *mx, b = *my, d = *mz;
    if (C.thin) {
        const long long kc = (long long)C.nky * C.nkx;
        const double *K = C.kern + (long long)kym * C.nkx + kx;
        const double kxx = __ldg(K), kyy = __ldg(K + kc), kzz = __ldg(K + 2 * kc), kxy = zneg_if(ny_, __ldg(K + 3 * kc));
        *mx = make_double2(-(kxx * a.x + kxy * b.x), -(kxx * a.y + kxy * b.y));
        *my = make_double2(-(kxy * a.x + kyy * b.x), -(kxy * a.y + kyy * b.y));
        *mz = make_double2(-kzz * d.x, -kzz * d.y);
        return;
    }
    const bool nz_ = kz > C.pz / 2;
    const int kzm = nz_ ? C.pz - kz : kz;
    const long long kc = (long long)C.nkz * C.nky * C.nkx;
    const double *K = C.kern + ((long long)kzm * C.nky + kym) * C.nkx + kx;
    const double kxx = __ldg(K), kyy = __ldg(K + kc), kzz = __ldg(K + 2 * kc);
    const double kxy = zneg_if(ny_, __ldg(K + 3 * kc)), kxz = zneg_if(nz_, __ldg(K + 4 * kc)),
                 kyz = zneg_if(ny_ != nz_, __ldg(K + 5 * kc));
    *mx = make_double2(-(kxx * a.x + kxy * b.x + kxz * d.x), -(kxx * a.y + kxy * b.y + kxz * d.y));
    *my = make_double2(-(kxy * a.x + kyy * b.x + kyz * d.x), -(kxy * a.y + kyy * b.y + kyz * d.y));
    *mz = make_double2(-(kxz * a.x + kyz * b.x + kzz * d.x), -(kxz * a.y + kyz * b.y + kzz * d.y));
}

// ---- column passes: a tile of tx kx columns per CTA ----
struct Col64 {
    Conv64 C;
    const double2 *in;
    double2 *out;
    int tx;
    int early;
};

// lines (c, col) at (c * ncol + col) * ls: elements e < cnt from src + c cs + e es + col,
// zeros up to lim
__device__ __forceinline__ void load_lines64(const double2 *__restrict__ src, size_t cs, size_t es, int nc, int cnt, int lim,
                                             int ncol, double2 *a, int ls) {
    copy64<4>(
        nc * cnt * ncol,
        [&](int idx) {
            const int r = idx / ncol, col = idx - r * ncol, c = r / cnt, e = r - c * cnt;
            return src[c * cs + e * es + col];
        },
        [&](int idx, double2 v) {
            const int r = idx / ncol, col = idx - r * ncol, c = r / cnt, e = r - c * cnt;
            a[(c * ncol + col) * ls + e] = v;
        });
    const int pad = lim - cnt;
    for (int idx = threadIdx.x; idx < nc * ncol * pad; idx += blockDim.x) {
        const int l = idx / pad;
        a[l * ls + cnt + (idx - l * pad)] = make_double2(0.0, 0.0);
    }
}
__device__ __forceinline__ void store_lines64(double2 *__restrict__ dst, size_t cs, size_t es, int nc, int cnt, int ncol,
                                              const double2 *a, int ls) {
    for (int idx = threadIdx.x; idx < nc * cnt * ncol; idx += blockDim.x) {
        const int r = idx / ncol, col = idx - r * ncol, c = r / cnt, e = r - c * cnt;
        dst[c * cs + e * es + col] = a[(c * ncol + col) * ls + e];
    }
}

constexpr int kTC = 128;  // threads of a column pass
// Line strides: one element of padding against bank conflicts, where shared memory holds it
__host__ __device__ inline int conv_ls64(int len) { return (size_t)6 * sizeof(double2) * (len + 1) <= kMaxSmem ? len + 1 : len; }
__host__ __device__ inline int y_ls64(const Conv64 &C, int tx) { return C.py + (tx > 1 ? 1 : 0); }  // one line fills the limit

// X[c][z][y < ny][kx] -> Y[c][z][ky][kx]
__global__ void __launch_bounds__(kTC) y_forward64(const Col64 P) {
    pdl_wait();
    if (P.early) pdl_trigger();
    extern __shared__ double2 sm64[];
    const Conv64 &C = P.C;
    const int kx0 = blockIdx.x * P.tx, ncol = min(P.tx, C.nkx - kx0), ls = y_ls64(C, P.tx);
    const size_t cz = (size_t)blockIdx.z * C.nz + blockIdx.y;
    double2 *a = sm64, *b = a + P.tx * ls;
    load_lines64(P.in + cz * C.ny * C.nkx + kx0, 0, C.nkx, 1, C.ny, C.yprune ? C.py / 2 : C.py, ncol, a, ls);
    __syncthreads();
    const double2 *r = fft_lines64<false>(a, b, ncol, ls, C.ply, C.yprune != 0);
    store_lines64(P.out + cz * C.py * C.nkx + kx0, 0, C.nkx, 1, C.py, ncol, r, ls);
}

// Y[c][z][ky][kx] -> X[c][z][y < ny][kx]
__global__ void __launch_bounds__(kTC) y_inverse64(const Col64 P) {
    pdl_wait();
    if (P.early) pdl_trigger();
    extern __shared__ double2 sm64[];
    const Conv64 &C = P.C;
    const int kx0 = blockIdx.x * P.tx, ncol = min(P.tx, C.nkx - kx0), ls = y_ls64(C, P.tx);
    const size_t cz = (size_t)blockIdx.z * C.nz + blockIdx.y;
    double2 *a = sm64, *b = a + P.tx * ls;
    load_lines64(P.in + cz * C.py * C.nkx + kx0, 0, C.nkx, 1, C.py, C.py, ncol, a, ls);
    __syncthreads();
    const double2 *r = fft_lines64<true>(a, b, ncol, ls, C.ply, C.yprune != 0);
    store_lines64(P.out + cz * C.ny * C.nkx + kx0, 0, C.nkx, 1, C.ny, ncol, r, ls);
}

// thin film (tile): forward y of the three components, multiply, inverse, rows y < ny;
// 3-D (tile, ky): the same along z.  In place.
template <bool THIN>
__global__ void __launch_bounds__(kTC) convolve64(const Col64 P) {
    pdl_wait();
    if (P.early) pdl_trigger();
    extern __shared__ double2 sm64[];
    const Conv64 &C = P.C;
    const int L = THIN ? C.py : C.pz, cnt = THIN ? C.ny : C.nz, ls = conv_ls64(L);
    const bool prune = (THIN ? C.yprune : C.zprune) != 0;
    const Plan64 &pl = THIN ? C.ply : C.plz;
    const int kx0 = blockIdx.x * P.tx, ncol = min(P.tx, C.nkx - kx0), ky = THIN ? 0 : blockIdx.y;
    const size_t es = THIN ? (size_t)C.nkx : (size_t)C.py * C.nkx, cs = cnt * es;
    const size_t base = (size_t)ky * C.nkx + kx0;
    double2 *a = sm64, *b = a + 3 * P.tx * ls;
    load_lines64(P.in + base, cs, es, 3, cnt, prune ? L / 2 : L, ncol, a, ls);
    __syncthreads();
    double2 *r = fft_lines64<false>(a, b, 3 * ncol, ls, pl, prune);
    for (int idx = threadIdx.x; idx < L * ncol; idx += blockDim.x) {
        const int k = idx / ncol, col = idx - k * ncol;
        double2 *q = r + col * ls + k;
        multiply3(C, q, q + ncol * ls, q + 2 * ncol * ls, kx0 + col, THIN ? k : ky, THIN ? 0 : k);
    }
    __syncthreads();
    const double2 *o = fft_lines64<true>(r, r == a ? b : a, 3 * ncol, ls, pl, prune);
    store_lines64(P.out + base, cs, es, 3, cnt, ncol, o, ls);
}

// H_corr(t) = -sum_s dN(t, s) (phi_s Ms m_s) at the target cells, which the row pass adds to
// H_d (demag_boundary_fp64.cu:23-76); the tensor row of (t, s) is xx xy xz yy yz zz.  hd is
// zero before the launch.
__global__ void demag_correction64(double *__restrict__ hd, const double *__restrict__ m, const double *__restrict__ phi,
                                   const int32_t *__restrict__ tidx, const int32_t *__restrict__ sidx,
                                   const double *__restrict__ tensor, double ms, long long n, uint32_t ntarget,
                                   uint32_t stencil) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < ntarget; t += gridDim.x * blockDim.x) {
        const int32_t ti = tidx[t];
        if (ti < 0) continue;
        double hx = 0.0, hy = 0.0, hz = 0.0;
        for (uint32_t s = 0; s < stencil; ++s) {
            const int32_t si = sidx[(size_t)t * stencil + s];
            if (si < 0) continue;
            const double *N = tensor + ((size_t)t * stencil + s) * 6;
            const double w = (phi ? phi[si] : 1.0) * ms;
            const double Mx = w * m[si], My = w * m[n + si], Mz = w * m[2 * n + si];
            hx -= N[0] * Mx + N[1] * My + N[2] * Mz;
            hy -= N[1] * Mx + N[3] * My + N[4] * Mz;
            hz -= N[2] * Mx + N[4] * My + N[5] * Mz;
        }
        hd[ti] += hx;
        hd[n + ti] += hy;
        hd[2 * n + ti] += hz;
    }
}

struct Field64 {
    int nx, ny, nz;
    long long n;
    const double *m;          // stage input; NULL: no right-hand side in this pass
    const double *hcorr;      // sparse demag correction at m (zero elsewhere) or NULL
    double *hex, *hd, *heff;  // observables; NULL: not written
    double *k;                // NULL: not stored
    const uint8_t *mask;
    const uint8_t *region;    // ids (< 256) or NULL
    const double *lut;        // 256 x 256 stiffness table (J/m)
    int tier;                 // 0 none, 1 T0 face links, 2 T1 boundary distances
    const double *phi;        // volume fractions (tiers 1, 2; also weights the energies)
    const double *face[6];    // +x -x +y -y +z -z
    const double *delta[6];
    double phi_floor, delta_min;
    int exchange;
    int per;                  // periodic axes (bit 0 x, 1 y, 2 z): neighbours wrap around
    double a_ex, dx, dy, dz;
    double inv2[3];           // 1 / d^2
    double ex_s;              // 2 / (mu0 Ms)
    int has_ext;
    double hext[3];
    int has_uni;
    double ku1, ku2, u[3];
    double ku1c, ku2c;        // 2 Ku1 / (mu0 Ms), 4 Ku2 / (mu0 Ms)
    int has_cub;
    double kc1, kc2, kc3, c1[3], c2[3], c3[3];
    double kc1c, kc2c, kc3c;  // -2 Kc1 / (mu0 Ms), -2 Kc2 / (mu0 Ms), -4 Kc3 / (mu0 Ms)
    double gbar, alpha, prec;
    double *partials;         // [block][kStats] or NULL
};

// exchange field at cell i (x, y, z); the neighbour offsets are +x -x +y -y +z -z
__device__ __forceinline__ void exchange64(const Field64 &P, long long i, int x, int y, int z, double e[3]) {
    e[0] = e[1] = e[2] = 0.0;
    if (!P.exchange) return;
    const double *m = P.m;
    const long long n = P.n, nxy = (long long)P.nx * P.ny;
    const bool has[6] = {x + 1 < P.nx, x > 0, y + 1 < P.ny, y > 0, z + 1 < P.nz, z > 0};
    const long long off[6] = {1, -1, P.nx, -(long long)P.nx, nxy, -nxy};
    const double c0[3] = {m[i], m[n + i], m[2 * n + i]};
    const int ri = P.region ? P.region[i] : 0;
    if (P.tier == 0) {
        // clamped neighbours: out of range or inactive -> the centre (no contribution); on a
        // periodic axis the neighbour wraps around (fdm_types.rs:126-132)
        const int ext[3] = {P.nx, P.ny, P.nz};
        for (int q = 0; q < 6; ++q) {
            long long j = has[q] ? i + off[q] : ((P.per >> (q >> 1)) & 1) ? i - off[q] * (ext[q >> 1] - 1) : i;
            if (P.mask && P.mask[j] == 0) j = i;
            if (j == i) continue;
            const double w = (P.region ? P.lut[ri * FULLMAG_FDM_MAX_EXCHANGE_REGIONS + P.region[j]] : P.a_ex) * P.inv2[q >> 1];
            for (int c = 0; c < 3; ++c) e[c] += w * (m[c * n + j] - c0[c]);
        }
    } else if (P.tier == 1) {
        // T0: face-link weights f
        for (int q = 0; q < 6; ++q) {
            if (q >= 4 && P.nz <= 1) continue;
            const double f = P.face[q][i];
            if (!(f > 0.0) || !has[q]) continue;
            const long long j = i + off[q];
            const double w = (P.region ? P.lut[ri * FULLMAG_FDM_MAX_EXCHANGE_REGIONS + P.region[j]] : P.a_ex) * f * P.inv2[q >> 1];
            for (int c = 0; c < 3; ++c) e[c] += w * (m[c * n + j] - c0[c]);
        }
    } else {
        // T1: neighbour at distance d across the face, boundary at the opposite distance
        // delta: 2 / (d (d + delta_opposite)) per face
        const double d[6] = {P.dx, P.dx, P.dy, P.dy, P.dz, P.dz};
        for (int q = 0; q < 6; ++q) {
            if (q >= 4 && P.nz <= 1) continue;
            const double dopp = fmax(P.delta[q ^ 1][i], P.delta_min);
            const double dsel = fmax(P.delta[q][i], P.delta_min);
            if (!has[q] || !(dsel > 0.0)) continue;
            const long long j = i + off[q];
            const double mj[3] = {m[j], m[n + j], m[2 * n + j]};
            if (mj[0] == 0.0 && mj[1] == 0.0 && mj[2] == 0.0) continue;
            const double w = (P.region ? P.lut[ri * FULLMAG_FDM_MAX_EXCHANGE_REGIONS + P.region[j]] : P.a_ex) * 2.0 /
                             (d[q] * (d[q] + dopp));
            for (int c = 0; c < 3; ++c) e[c] += w * (mj[c] - c0[c]);
        }
    }
    double s = P.ex_s;
    if (P.tier > 0) s /= fmax(P.phi[i], P.phi_floor);
    for (int c = 0; c < 3; ++c) e[c] *= s;
}

// exchange energy pairs of cell i with its forward neighbours (reductions_fp64.cu:123-210)
__device__ __forceinline__ double exchange_pairs64(const Field64 &P, long long i, int x, int y, int z, double phi_i) {
    if (!P.exchange) return 0.0;
    const double *m = P.m;
    const long long n = P.n, nxy = (long long)P.nx * P.ny;
    const bool has[3] = {x + 1 < P.nx, y + 1 < P.ny, z + 1 < P.nz};
    const long long off[3] = {1, P.nx, nxy};
    const int ext[3] = {P.nx, P.ny, P.nz};
    const int ri = P.region ? P.region[i] : 0;
    double e = 0.0;
    for (int a = 0; a < 3; ++a) {
        // forward pairs; on a periodic axis the last cell pairs with the first
        const bool wrap = !has[a] && ((P.per >> a) & 1);
        if (!has[a] && !wrap) continue;
        const long long j = has[a] ? i + off[a] : i - off[a] * (ext[a] - 1);
        if (j == i) continue;
        if (P.mask && P.mask[j] == 0) continue;
        if (P.phi && !(P.phi[j] > 0.0)) continue;
        const double A = P.region ? P.lut[ri * FULLMAG_FDM_MAX_EXCHANGE_REGIONS + P.region[j]] : P.a_ex;
        double s2 = 0.0;
        for (int c = 0; c < 3; ++c) {
            const double dm = m[c * n + j] - m[c * n + i];
            s2 += dm * dm;
        }
        e += A * phi_i * s2 * P.inv2[a];
    }
    return e;
}

__device__ __forceinline__ void block_stats(double (&v)[kStats], double *out) {
    __shared__ double red[kT / 32][kStats];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int s = 0; s < kStats; ++s)
        for (int o = 16; o > 0; o >>= 1) {
            const double w = __shfl_xor_sync(0xffffffffu, v[s], o);
            v[s] = s < 5 ? v[s] + w : fmax(v[s], w);
        }
    if (lane == 0)
        for (int s = 0; s < kStats; ++s) red[wid][s] = v[s];
    __syncthreads();
    if (threadIdx.x < kStats) {
        const int s = threadIdx.x;
        double acc = 0.0;
        for (int w = 0; w < kT / 32; ++w) acc = s < 5 ? acc + red[w][s] : fmax(acc, red[w][s]);
        out[blockIdx.x * kStats + s] = acc;
    }
}

// One fused pass over `rows` x-rows per CTA: inverse x-transform of the demag field at the
// stage input, exchange, local terms, torque, statistics, the adaptive error norm, the next
// stage input N(m0 + dt sum_j c_j k_j) and its forward x-transform.  The step is then a
// chain of two launches per evaluation on films and four on volumes; FP64 issue bounds it.
// 200x100x1 Heun: 511 us per step as one kernel per operation with strided radix-4 columns.
struct Row64 {
    Field64 f;
    Conv64 C;
    const double2 *x_in;  // NULL: no demag field from a spectrum in this pass
    double2 *x_out;       // NULL: no forward transform
    const double *hd_in;  // H_d from memory (rows too long for the fused transform) or NULL
    int rows;             // rows per CTA
    int lb;               // x lines transformed at a time: 3 rows or 1
    const double *m0;     // NULL: no combination
    int nk;
    const double *kk[8];  // NULL entry: the derivative of this pass
    double c[8];
    double dt;
    double *m_next;
    const double *m_fwd;  // forward-transform source without a combination
    int ne;               // error terms (0: none); NULL entry: the derivative of this pass
    const double *ek[8];
    double ec[8];
    int early;
};

__host__ __device__ inline int row_ls64(const Conv64 &C) { return (C.half ? C.half : C.px) + 1; }

__global__ void __launch_bounds__(kT, 2) row64(const Row64 R) {
    pdl_wait();
    if (R.early) pdl_trigger();
    extern __shared__ double2 sm64[];
    const Field64 &P = R.f;
    const int nx = P.nx, nrows = P.ny * P.nz, row0 = blockIdx.x * R.rows, rows = min(R.rows, nrows - row0);
    const bool fft = R.x_in || R.x_out;
    const int ls = fft ? row_ls64(R.C) : 0, lb = min(R.lb, rows * 3);
    double2 *a = sm64, *b = a + R.lb * ls;
    double *H = reinterpret_cast<double *>(b + R.lb * ls);  // line (row, c): H_d in, next input out
    if (R.x_in) {
        for (int l0 = 0; l0 < rows * 3; l0 += lb) {
            const int nl = min(lb, rows * 3 - l0);
            const double2 *r = x_inverse_lines(R.C, R.x_in, row0, l0, nl, a, b, ls);
            for (int idx = threadIdx.x; idx < nl * nx; idx += blockDim.x) {
                const int l = idx / nx, x = idx - l * nx;
                const double2 *q = r + l * ls;
                H[(size_t)l0 * nx + idx] = R.C.half ? ((x & 1) ? q[x >> 1].y : q[x >> 1].x) : q[x].x;
            }
            __syncthreads();
        }
    }
    double st[kStats] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const long long n = P.n;
    for (int idx = threadIdx.x; idx < rows * nx; idx += blockDim.x) {
        const int rr = idx / nx, x = idx - rr * nx, row = row0 + rr, z = row / P.ny, y = row - z * P.ny;
        const long long i = (long long)row * nx + x;
        const double phi_i = P.phi ? P.phi[i] : 1.0;
        double *hl = H + (size_t)rr * 3 * nx + x;
        double k[3] = {0, 0, 0};
        if (P.m) {
            const bool act = (P.mask == nullptr || P.mask[i] != 0) && (P.tier == 0 || phi_i > 0.0);
            double h[3] = {0, 0, 0}, ex[3] = {0, 0, 0}, hd[3] = {0, 0, 0};
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (act) hd[c] = R.x_in ? hl[c * nx] : R.hd_in ? R.hd_in[c * n + i] : 0.0;
                if (P.hcorr) hd[c] += P.hcorr[c * n + i];
                if (P.hd) P.hd[c * n + i] = hd[c];
            }
            if (act) {
                const double m0[3] = {P.m[i], P.m[n + i], P.m[2 * n + i]};
                exchange64(P, i, x, y, z, ex);
#pragma unroll
                for (int c = 0; c < 3; ++c) h[c] = ex[c] + hd[c] + (P.has_ext ? P.hext[c] : 0.0);
                double e_uni = 0.0, e_cub = 0.0;
                if (P.has_uni) {
                    const double mu = m0[0] * P.u[0] + m0[1] * P.u[1] + m0[2] * P.u[2], mu2 = mu * mu;
                    const double cf = mu * (P.ku1c + P.ku2c * mu2);
#pragma unroll
                    for (int c = 0; c < 3; ++c) h[c] += cf * P.u[c];
                    e_uni = mu2 * (P.ku1 + P.ku2 * mu2);
                }
                if (P.has_cub) {
                    const double a1 = m0[0] * P.c1[0] + m0[1] * P.c1[1] + m0[2] * P.c1[2];
                    const double a2 = m0[0] * P.c2[0] + m0[1] * P.c2[1] + m0[2] * P.c2[2];
                    const double a3 = m0[0] * P.c3[0] + m0[1] * P.c3[1] + m0[2] * P.c3[2];
                    const double s1 = a1 * a1, s2 = a2 * a2, s3 = a3 * a3;
                    const double sig = s1 * s2 + s2 * s3 + s1 * s3;
                    const double w = P.kc1c + P.kc3c * sig;
                    const double g1 = a1 * (w * (s2 + s3) + P.kc2c * s2 * s3);
                    const double g2 = a2 * (w * (s1 + s3) + P.kc2c * s1 * s3);
                    const double g3 = a3 * (w * (s1 + s2) + P.kc2c * s1 * s2);
#pragma unroll
                    for (int c = 0; c < 3; ++c) h[c] += g1 * P.c1[c] + g2 * P.c2[c] + g3 * P.c3[c];
                    e_cub = P.kc1 * sig + P.kc2 * s1 * s2 * s3 + P.kc3 * sig * sig;
                }
                const double p0 = m0[1] * h[2] - m0[2] * h[1], p1 = m0[2] * h[0] - m0[0] * h[2], p2 = m0[0] * h[1] - m0[1] * h[0];
                const double q0 = m0[1] * p2 - m0[2] * p1, q1 = m0[2] * p0 - m0[0] * p2, q2 = m0[0] * p1 - m0[1] * p0;
                k[0] = -P.gbar * (P.prec * p0 + P.alpha * q0);
                k[1] = -P.gbar * (P.prec * p1 + P.alpha * q1);
                k[2] = -P.gbar * (P.prec * p2 + P.alpha * q2);
                if (P.partials) {
                    st[0] += exchange_pairs64(P, i, x, y, z, phi_i);
                    st[1] += phi_i * (m0[0] * hd[0] + m0[1] * hd[1] + m0[2] * hd[2]);
                    if (P.has_ext) st[2] += phi_i * (m0[0] * P.hext[0] + m0[1] * P.hext[1] + m0[2] * P.hext[2]);
                    st[3] += phi_i * e_uni;
                    st[4] += phi_i * e_cub;
                    st[5] = fmax(st[5], h[0] * h[0] + h[1] * h[1] + h[2] * h[2]);
                    st[6] = fmax(st[6], hd[0] * hd[0] + hd[1] * hd[1] + hd[2] * hd[2]);
                    st[7] = fmax(st[7], k[0] * k[0] + k[1] * k[1] + k[2] * k[2]);
                }
            }
            if (R.ne > 0) {
                double e2 = 0.0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    double s = 0.0;
                    for (int t = 0; t < R.ne; ++t) s += R.ec[t] * (R.ek[t] ? R.ek[t][c * n + i] : k[c]);
                    s *= R.dt;
                    e2 += s * s;
                }
                st[8] = fmax(st[8], e2);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                if (P.hex) P.hex[c * n + i] = ex[c];
                if (P.heff) P.heff[c * n + i] = h[c];
                if (P.k) P.k[c * n + i] = k[c];
            }
        }
        double v[3] = {0, 0, 0};
        if (R.m0) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double s = 0.0;
                for (int t = 0; t < R.nk; ++t) s += R.c[t] * (R.kk[t] ? R.kk[t][c * n + i] : k[c]);
                v[c] = R.m0[c * n + i] + R.dt * s;
            }
            const double nn = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
            const double inv = nn > 0.0 ? 1.0 / sqrt(nn) : 0.0;  // a zero vector stays zero
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                v[c] *= inv;
                R.m_next[c * n + i] = v[c];
            }
        } else if (R.m_fwd) {
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c] = R.m_fwd[c * n + i];
        }
        if (R.x_out) {  // the convolution's input is phi m with a boundary tier
#pragma unroll
            for (int c = 0; c < 3; ++c) hl[c * nx] = P.phi ? v[c] * phi_i : v[c];
        }
    }
    if (P.partials) block_stats(st, P.partials);
    if (R.x_out) {
        __syncthreads();
        for (int l0 = 0; l0 < rows * 3; l0 += lb) {
            x_forward_lines(R.C, R.x_out, H, row0, l0, min(lb, rows * 3 - l0), a, b, ls);
            __syncthreads();
        }
    }
}

// sums / maxima of the block partials in a fixed order (one CTA of kT threads)
__global__ void __launch_bounds__(kT) finalize64(const double *__restrict__ partials, int nblocks, double *__restrict__ out,
                                                 int early) {
    pdl_wait();
    if (early) pdl_trigger();
    double v[kStats] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
        for (int s = 0; s < kStats; ++s) {
            const double w = partials[(size_t)b * kStats + s];
            v[s] = s < 5 ? v[s] + w : fmax(v[s], w);
        }
    block_stats(v, out);
}

__global__ void aos_to_soa64(const double *__restrict__ in, double *__restrict__ out, const uint8_t *__restrict__ mask,
                             const double *__restrict__ phi, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const bool act = (mask == nullptr || mask[i] != 0) && (phi == nullptr || phi[i] > 0.0);
        for (int c = 0; c < 3; ++c) out[c * n + i] = act ? in[3 * i + c] : 0.0;
    }
}

__global__ void soa_to_aos64(const double *__restrict__ in, double *__restrict__ out, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        for (int c = 0; c < 3; ++c) out[3 * i + c] = in[c * n + i];
}

unsigned blocks_for(long long n) { return (unsigned)std::min<long long>((n + kT - 1) / kT, kMaxBlocks); }

// radices 8 (4 or 2 for the remainder) first, then odd primes: the even radix in front
// carries the half-line stages
bool make_plan64(int n, std::vector<double2> &tw, std::vector<size_t> &off, Plan64 &p) {
    p.n = n;
    p.ns = 0;
    int r = n;
    for (int f : {8, 4, 2, 3, 5, 7}) {
        while (r % f == 0) {
            if (p.ns >= kMaxRadixStages) return false;
            p.radix[p.ns++] = f;
            r /= f;
        }
    }
    for (int f = 11; r > 1; f += 2) {
        while (r % f == 0) {
            if (p.ns >= kMaxRadixStages) return false;
            p.radix[p.ns++] = f;
            r /= f;
        }
    }
    off.push_back(tw.size());
    for (int e = 0; e < n; ++e) {
        const double a = 2.0 * M_PI * (double)e / (double)n;
        tw.push_back(make_double2(cos(a), -sin(a)));
    }
    p.tw = nullptr;
    return true;
}

// FP64 instructions per point of a transform of length n (twiddles included); 0 when n has
// a prime factor above 13, for which there is no butterfly
double fft_cost64(int n) {
    const struct {
        int r;
        double c;
    } cost[] = {{8, 10.5}, {4, 7.0}, {2, 4.0}, {3, 8.0}, {5, 12.0}, {7, 15.0}, {11, 19.0}, {13, 21.0}};
    double s = 0.0;
    for (const auto &f : cost)
        while (n % f.r == 0) {
            n /= f.r;
            s += f.c;
        }
    return n == 1 ? std::max(s, 1.0) : 0.0;
}

// Padded extent of an open axis of n cells when the engine builds the tensor: 2n, the
// reference's, when its factors are all 2..13; else the even extent above it whose
// transform issues the fewest instructions (a prime factor R > 13 costs 4R of them per
// point, so 2 x 157 takes 30 times the instructions of 320)
int pad_extent64(int n) {
    if (fft_cost64(2 * n) > 0.0) return 2 * n;
    int best = 2 * n;
    double bc = 1e30;
    for (int p = 2 * n + 2; p <= 2 * n + 2 + n / 2; p += 2) {
        const double c = fft_cost64(p) * p;
        if (c > 0.0 && c < bc) {
            bc = c;
            best = p;
        }
    }
    return best;
}

__host__ __device__ inline int axis_ls64(int p, int nl) { return p + (nl > 1 ? 1 : 0); }

// FP64 lines of length p along an axis of layout [outer][p][inner] (real input in_re with zero
// imaginary part, or complex c_in), nl per CTA: forward transform e^{-2 pi i k a / p}, the first
// nout outputs written to out[outer][nout][inner].  One line of 64 points has eight radix-8
// butterflies for 128 threads; with up to 16 lines a CTA every thread has one, and neighbouring
// lines are read together (periodic tensor of 128x128x30: create 5.2 -> 3.9 ms).
__global__ void fft_axis64_kernel(const double *__restrict__ in_re, const double2 *__restrict__ c_in,
                                  double2 *__restrict__ out, int p, int nout, int inner, unsigned lines, int nl,
                                  const Plan64 plan) {
    extern __shared__ double2 sm64[];
    const int ls = axis_ls64(p, nl);
    double2 *a = sm64, *b = sm64 + nl * ls;
    const unsigned line0 = blockIdx.x * (unsigned)nl;
    const int n = (int)min((unsigned)nl, lines - line0);
    for (int idx = threadIdx.x; idx < n * p; idx += blockDim.x) {
        // neighbouring threads on neighbouring addresses: along the line, or across the lines
        const int l = inner == 1 ? idx / p : idx % n, i = inner == 1 ? idx - l * p : idx / n;
        const unsigned o = (line0 + l) / inner, q = line0 + l - o * inner;
        const long long at = ((long long)o * p + i) * inner + q;
        a[l * ls + i] = in_re ? make_double2(in_re[at], 0.0) : c_in[at];
    }
    __syncthreads();
    const double2 *r = fft_lines64<false>(a, b, n, ls, plan, false);
    for (int idx = threadIdx.x; idx < n * nout; idx += blockDim.x) {
        const int l = inner == 1 ? idx / nout : idx % n, k = inner == 1 ? idx - l * nout : idx / n;
        const unsigned o = (line0 + l) / inner, q = line0 + l - o * inner;
        out[((long long)o * nout + k) * inner + q] = r[l * ls + k];
    }
}

}  // namespace

bool fft64_axis(const double *in_re, const double2 *c_in, double2 *out, long long outer, int p, int nout, int inner,
                cudaStream_t s, std::string &err) {
    std::vector<double2> tw;
    std::vector<size_t> off;
    Plan64 plan;
    if (!make_plan64(p, tw, off, plan)) return err = "FFT length has too many factors", false;
    const long long lines = outer * inner;
    if (sizeof(double2) * 2 * (size_t)p > kMaxSmem) return err = "FFT length too large for the double-precision lines", false;
    int nl = 16;
    auto bytes = [&](int k) { return sizeof(double2) * 2 * (size_t)k * axis_ls64(p, k); };
    while (nl > 1 && (bytes(nl) > 48 * 1024 || lines / nl < 304)) nl /= 2;
    const size_t smem = bytes(nl);
    double2 *dtw = nullptr;
    cudaError_t e = cudaMalloc(&dtw, sizeof(double2) * tw.size());
    if (e == cudaSuccess) e = cudaMemcpyAsync(dtw, tw.data(), sizeof(double2) * tw.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute((const void *)fft_axis64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) {
        plan.tw = dtw;
        fft_axis64_kernel<<<(unsigned)((lines + nl - 1) / nl), 128, smem, s>>>(in_re, c_in, out, p, nout, inner,
                                                                               (unsigned)lines, nl, plan);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(dtw);
    if (e != cudaSuccess) return err = std::string("fft64_axis: ") + cudaGetErrorString(e), false;
    return true;
}

struct Fp64Engine {
    // configuration
    int nx = 0, ny = 0, nz = 0;
    long long n = 0;
    double dx = 0, dy = 0, dz = 0, ms = 0, a_ex = 0, alpha = 0, gamma = 0;
    int integrator = FULLMAG_FDM_INTEGRATOR_HEUN;
    bool exchange = false, demag = false, has_ext = false, has_uni = false, has_cub = false, prec = true;
    double hext[3] = {0, 0, 0};
    double ku1 = 0, ku2 = 0, u[3] = {0, 0, 1}, kc1 = 0, kc2 = 0, kc3 = 0, c1[3] = {1, 0, 0}, c2[3] = {0, 1, 0}, c3[3] = {0, 0, 1};
    double max_error = 1e-5, dt_min = 1e-18, dt_max = 1e-10, headroom = 0.8;
    int tier = 0;
    double phi_floor = 0.0, delta_min = 0.0;
    int per = 0;                     // periodic axes (bit 0 x, 1 y, 2 z)
    uint32_t images[3] = {10, 10, 10};
    bool has_mask = false;
    std::vector<uint8_t> mask_host;
    uint32_t corr_targets = 0, corr_stencil = 0;
    // device
    int device = 0;
    cudaStream_t stream = nullptr;
    std::vector<void *> allocs;
    double *S[2] = {nullptr, nullptr}, *K[7] = {}, *A[2] = {nullptr, nullptr};
    double *hex = nullptr, *hd = nullptr, *heff = nullptr, *staging = nullptr;
    double *hcorr = nullptr;         // sparse demag correction (n targets among 3 n values)
    double *partials = nullptr, *dstats = nullptr, *hstats = nullptr;
    uint8_t *mask = nullptr, *region = nullptr;
    double *lut = nullptr, *phi = nullptr, *face[6] = {}, *delta[6] = {};
    int32_t *ctidx = nullptr, *csidx = nullptr;
    double *ctensor = nullptr;
    Conv64 conv{};
    double2 *X = nullptr, *Y = nullptr;
    double *kern = nullptr;
    double2 *kernc = nullptr;  // periodic grids: the complex image-sum kernel
    double2 *twid = nullptr;
    // launch shapes (choose_shapes)
    int rows = 1, lb = 3;            // rows per CTA of the row pass, x lines transformed at a time
    bool fused_x = true;             // the row pass holds the x-transforms
    int tx_y = 1, tx_c = 1;          // kx columns per CTA of the y passes and of the convolution pass
    bool early = false;              // programmatic early launch on small grids (engine.h)
    // state
    int cur = 0;
    double time = 0.0;
    uint64_t step_count = 0;
    bool k1_valid = false;
    bool fields_ok = false;  // hex / hd / heff hold the fields of the committed state
    fullmag_fdm_step_stats cur_stats{};
    double raw[kStats] = {};
    // ABM3 history (indices into K, rotated)
    int abm_startup = 0;
    double abm_last_dt = 0.0;
    int abm_hist[3] = {1, 2, 3}, abm_kf = 4;
    std::string err;

    ~Fp64Engine() {
        if (stream) cudaStreamSynchronize(stream);
        for (void *p : allocs) cudaFree(p);
        if (hstats) cudaFreeHost(hstats);
        if (stream) cudaStreamDestroy(stream);
    }

    bool fail(const char *what, cudaError_t e) {
        if (e == cudaSuccess) return false;
        cudaGetLastError();  // reported here: the next check is not to find it again
        err = std::string(what) + ": " + cudaGetErrorString(e);
        return true;
    }
    template <typename T>
    bool alloc(T *&p, size_t count) {
        void *q = nullptr;
        if (fail("cudaMalloc", cudaMalloc(&q, sizeof(T) * std::max<size_t>(count, 1)))) return false;
        allocs.push_back(q);
        p = static_cast<T *>(q);
        return true;
    }
    template <typename T>
    bool put(T *&p, const T *src, size_t count) {
        return alloc(p, count) &&
               !fail("cudaMemcpy", cudaMemcpyAsync(p, src, sizeof(T) * count, cudaMemcpyHostToDevice, stream));
    }

    bool setup(const fullmag_fdm_plan_desc *plan);
    bool upload(const double *m_xyz);

    // ---- one evaluation: the spectrum of its input lies in X, the column passes turn it into
    // the field's, and the row pass that evaluates it also forms and transforms the next input ----
    bool columns() {
        if (!demag) return true;
        const Conv64 &C = conv;
        Col64 P{};
        P.C = C;
        P.early = early;
        auto tiles = [&](int tx) { return (unsigned)((C.nkx + tx - 1) / tx); };
        cudaError_t e;
        if (C.thin) {
            P.tx = tx_c;
            P.in = X;
            P.out = X;
            e = launch_pdl(convolve64<true>, dim3(tiles(tx_c)), dim3(kTC), conv_smem(tx_c), stream, P);
        } else {
            P.tx = tx_y;
            P.in = X;
            P.out = Y;
            e = launch_pdl(y_forward64, dim3(tiles(tx_y), nz, 3), dim3(kTC), y_smem(tx_y), stream, P);
            P.tx = tx_c;
            P.in = Y;
            if (e == cudaSuccess) e = launch_pdl(convolve64<false>, dim3(tiles(tx_c), C.py), dim3(kTC), conv_smem(tx_c), stream, P);
            P.tx = tx_y;
            P.out = X;
            if (e == cudaSuccess) e = launch_pdl(y_inverse64, dim3(tiles(tx_y), nz, 3), dim3(kTC), y_smem(tx_y), stream, P);
        }
        return !fail("demag column passes", e);
    }
    size_t conv_smem(int tx) const { return sizeof(double2) * 6 * (size_t)tx * conv_ls64(conv.thin ? conv.py : conv.pz); }
    size_t y_smem(int tx) const { return sizeof(double2) * 2 * (size_t)tx * y_ls64(conv, tx); }
    size_t row_smem(int r, int l) const {
        if (!demag) return 0;
        return sizeof(double2) * 2 * (size_t)l * row_ls64(conv) + sizeof(double) * 3 * (size_t)r * nx;
    }

    // Tiles by the number of CTAs: FP64 issue is the bound, so a pass is as long as the SM
    // with the most lines.  Rows: one per CTA until 2 x 152 CTAs are there, then up to about
    // 256 cells; columns: the tile with the least ceil(CTAs / 152) x tile, the widest of equals
    // (64-byte segments from 4 columns on).
    bool choose_shapes() {
        constexpr size_t kSoft = 100 * 1024, kHard = kMaxSmem, kRow = kMaxSmem - 1024;  // row pass: static statistics
        const int nrows = ny * nz;
        rows = 1;
        lb = 3;
        fused_x = true;
        if (demag) {
            if (row_smem(1, 3) > kRow) lb = 1;
            fused_x = row_smem(1, lb) <= kRow;
        }
        if (!demag || row_smem(1, 3) <= kSoft) {
            while (rows < 8 && rows * nx < 256 && nrows / (2 * rows) >= 304 && row_smem(2 * rows, 6 * rows) <= kSoft) rows *= 2;
            lb = 3 * rows;
        }
        if (!demag) return true;
        auto pick = [&](long long outer, auto smem) {
            int best = 1;
            long long bc = 1LL << 60;
            for (int tx : {1, 2, 4, 8}) {
                if (tx > 1 && (tx > conv.nkx || smem(tx) > kSoft)) break;
                const long long ctas = ((conv.nkx + tx - 1) / tx) * outer, c = ((ctas + 151) / 152) * tx;
                if (c <= bc + bc / 16) {
                    best = tx;
                    bc = std::min(c, bc);
                }
            }
            return best;
        };
        tx_c = pick(conv.thin ? 1 : conv.py, [&](int tx) { return conv_smem(tx); });
        tx_y = conv.thin ? 1 : pick(3LL * nz, [&](int tx) { return y_smem(tx); });
        return conv_smem(tx_c) <= kHard && (conv.thin || y_smem(tx_y) <= kHard) &&
               (fused_x || sizeof(double2) * 2 * (size_t)conv.px <= kHard);
    }

    // the sparse correction at m, for the row pass that evaluates m
    bool correction(const double *m) {
        if (!demag || corr_targets == 0) return true;
        if (fail("correction memset", cudaMemsetAsync(hcorr, 0, sizeof(double) * 3 * n, stream))) return false;
        // the source weights phi_s are the volume fractions whenever the plan has them
        demag_correction64<<<std::max(1u, std::min(1024u, (corr_targets + kT - 1) / kT)), kT, 0, stream>>>(
            hcorr, m, phi, ctidx, csidx, ctensor, ms, n, corr_targets, corr_stencil);
        return !fail("demag correction", cudaGetLastError());
    }

    // one row pass: evaluation at m (NULL: none) into k, combination into out (NULL: none) or
    // the transform of fwd, statistics with the final evaluation of a step
    struct Terms {
        int nk = 0;
        const int *kidx = nullptr;  // -1: the derivative of this pass
        const double *coef = nullptr;
    };
    bool row_pass(const double *m, double *k, bool stats, const Terms &comb, double dt, double *out, const double *fwd,
                  const Terms &err_terms) {
        Row64 R{};
        R.f = field_base();
        R.C = conv;
        R.early = early;
        const bool to_x = demag && (out || fwd);
        if (m) {
            fields_ok = false;
            if (!correction(m)) return false;
            R.f.m = m;
            R.f.k = k;
            if (corr_targets > 0 && demag) R.f.hcorr = hcorr;
            if (stats) {
                R.f.partials = partials;
                R.f.hex = hex;
                R.f.hd = demag ? hd : nullptr;
                R.f.heff = heff;
            }
            if (demag && !fused_x) {
                x_inverse64<<<dim3(ny * nz, 3), kT, sizeof(double2) * 2 * conv.px, stream>>>(conv, X, hd);
                R.hd_in = hd;
            } else if (demag) {
                R.x_in = X;
            }
        }
        if (to_x && fused_x) R.x_out = X;
        R.rows = rows;
        R.lb = lb;
        R.dt = dt;
        if (out) {
            R.m0 = S[cur];
            R.m_next = out;
            R.nk = comb.nk;
            for (int t = 0; t < comb.nk; ++t) {
                R.kk[t] = comb.kidx[t] < 0 ? nullptr : K[comb.kidx[t]];
                R.c[t] = comb.coef[t];
            }
        }
        R.m_fwd = fwd;
        R.ne = err_terms.nk;
        for (int t = 0; t < err_terms.nk; ++t) {
            R.ek[t] = err_terms.kidx[t] < 0 ? nullptr : K[err_terms.kidx[t]];
            R.ec[t] = err_terms.coef[t];
        }
        const unsigned nb = (unsigned)((ny * nz + rows - 1) / rows);
        const bool fft = R.x_in || R.x_out;
        if (fail("row pass", launch_pdl(row64, dim3(nb), dim3(kT), fft ? row_smem(rows, lb) : 0, stream, R))) return false;
        if (to_x && !fused_x) {
            x_forward64<<<dim3(ny * nz, 3), kT, sizeof(double2) * 2 * conv.px, stream>>>(conv, out ? out : fwd,
                                                                                        tier > 0 ? phi : nullptr, X);
            if (fail("x forward", cudaGetLastError())) return false;
        }
        if (stats && fail("finalize", launch_pdl(finalize64, dim3(1), dim3(kT), 0, stream, partials, (int)nb, dstats, (int)early)))
            return false;
        return (out || fwd) ? columns() : true;
    }

    Field64 field_base() const {
        Field64 P{};
        P.nx = nx;
        P.ny = ny;
        P.nz = nz;
        P.n = n;
        P.mask = mask;
        P.region = region;
        P.lut = lut;
        P.tier = tier;
        P.phi = (tier > 0) ? phi : nullptr;
        for (int q = 0; q < 6; ++q) {
            P.face[q] = face[q];
            P.delta[q] = delta[q];
        }
        P.phi_floor = phi_floor;
        P.delta_min = delta_min;
        P.exchange = exchange;
        P.per = per;
        const double inv_mu0ms = 1.0 / (kMu0d * ms);
        P.a_ex = a_ex;
        P.dx = dx;
        P.dy = dy;
        P.dz = dz;
        P.inv2[0] = 1.0 / (dx * dx);
        P.inv2[1] = 1.0 / (dy * dy);
        P.inv2[2] = 1.0 / (dz * dz);
        P.ex_s = 2.0 / (kMu0d * ms);
        P.ku1c = 2.0 * inv_mu0ms * ku1;
        P.ku2c = 4.0 * inv_mu0ms * ku2;
        P.kc1c = -2.0 * kc1 * inv_mu0ms;
        P.kc2c = -2.0 * kc2 * inv_mu0ms;
        P.kc3c = -4.0 * kc3 * inv_mu0ms;
        P.has_ext = has_ext;
        for (int c = 0; c < 3; ++c) {
            P.hext[c] = hext[c];
            P.u[c] = u[c];
            P.c1[c] = c1[c];
            P.c2[c] = c2[c];
            P.c3[c] = c3[c];
        }
        P.has_uni = has_uni;
        P.ku1 = ku1;
        P.ku2 = ku2;
        P.has_cub = has_cub;
        P.kc1 = kc1;
        P.kc2 = kc2;
        P.kc3 = kc3;
        P.gbar = gamma / (1.0 + alpha * alpha);
        P.alpha = alpha;
        P.prec = prec ? 1.0 : 0.0;
        return P;
    }

    // first stage input of a step, N(m0 + dt sum c_j k_j), and its transforms
    bool first(int nk, const int *kidx, const double *coef, double dt, double *out) {
        return row_pass(nullptr, nullptr, false, {nk, kidx, coef}, dt, out, nullptr, {});
    }
    // derivative at m (into k, NULL: not stored) and the next input (index -1: this derivative)
    bool stage(const double *m, double *k, int nk, const int *kidx, const double *coef, double dt, double *out) {
        return row_pass(m, k, false, {nk, kidx, coef}, dt, out, nullptr, {});
    }
    // derivative at the proposed state with the statistics and optional error terms
    bool final_eval(const double *m, double *k, double dt, int ne = 0, const int *eidx = nullptr, const double *ecoef = nullptr) {
        return row_pass(m, k, true, {}, dt, nullptr, nullptr, {ne, eidx, ecoef});
    }

    bool read_stats() {
        if (fail("stats copy", cudaMemcpyAsync(hstats, dstats, sizeof(double) * kStats, cudaMemcpyDeviceToHost, stream)) ||
            fail("stream sync", cudaStreamSynchronize(stream)))
            return false;
        return true;
    }

    void fill_stats(const double *d) {
        const double V = dx * dy * dz;
        fullmag_fdm_step_stats &st = cur_stats;
        st.exchange_energy_joules = exchange ? V * d[0] : 0.0;
        st.demag_energy_joules = demag ? -0.5 * kMu0d * ms * V * d[1] : 0.0;
        st.external_energy_joules = has_ext ? -kMu0d * ms * V * d[2] : 0.0;
        st.anisotropy_energy_joules = has_uni ? -V * d[3] : 0.0;
        st.cubic_energy_joules = has_cub ? V * d[4] : 0.0;
        st.dmi_energy_joules = 0.0;
        st.total_energy_joules = st.exchange_energy_joules + st.demag_energy_joules + st.external_energy_joules +
                                 st.anisotropy_energy_joules + st.cubic_energy_joules;
        st.max_effective_field_amplitude = sqrt(d[5]);
        st.max_demag_field_amplitude = demag ? sqrt(d[6]) : 0.0;
        st.max_rhs_amplitude = sqrt(d[7]);
        st.step = step_count;
        st.time_seconds = time;
    }

    // k1 = f(S[cur]) with the statistics and observables of the committed state
    bool eval_state() {
        if (demag && !row_pass(nullptr, nullptr, false, {}, 0.0, nullptr, S[cur], {})) return false;
        if (!final_eval(S[cur], K[0], 0.0) || !read_stats()) return false;
        memcpy(raw, hstats, sizeof(raw));
        fill_stats(raw);
        k1_valid = true;
        fields_ok = true;
        return true;
    }

    bool poll_hit(fullmag_fdm_interrupt_poll_fn poll, void *user) { return poll && poll(user) != 0; }

    void commit(double dt) {
        cur = 1 - cur;
        step_count += 1;
        time += dt;
        memcpy(raw, hstats, sizeof(raw));
        fill_stats(raw);
        cur_stats.dt_seconds = dt;
        cur_stats.suggested_next_dt = 0.0;
        k1_valid = true;
        fields_ok = true;
    }

    // explicit Runge-Kutta stages from S[cur]: stage s input N(m0 + dt sum_j a_sj k_j),
    // k_s into K[s]; the proposal into S[1-cur]; its derivative into K[kfinal] with stats
    int rk_fixed(double dt, fullmag_fdm_interrupt_poll_fn poll, void *user) {
        const int nxt = 1 - cur;
        if (integrator == FULLMAG_FDM_INTEGRATOR_RK4) {
            const int k0[1] = {0}, self[1] = {-1}, kall[4] = {0, 1, 2, -1};
            const double h[1] = {0.5}, one[1] = {1.0}, b[4] = {1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0};
            if (!first(1, k0, h, dt, A[0])) return -1;
            if (poll_hit(poll, user)) return 1;
            if (!stage(A[0], K[1], 1, self, h, dt, A[1])) return -1;
            if (poll_hit(poll, user)) return 1;
            if (!stage(A[1], K[2], 1, self, one, dt, A[0])) return -1;
            if (poll_hit(poll, user)) return 1;
            if (!stage(A[0], nullptr, 4, kall, b, dt, S[nxt])) return -1;
        } else {  // Heun
            const int k0[1] = {0}, kb[2] = {0, -1};
            const double one[1] = {1.0}, half[2] = {0.5, 0.5};
            if (!first(1, k0, one, dt, A[0])) return -1;
            if (poll_hit(poll, user)) return 1;
            if (!stage(A[0], nullptr, 2, kb, half, dt, S[nxt])) return -1;
        }
        // k1 of the next step (the combination above was the last reader of K[0])
        k1_valid = false;
        if (!final_eval(S[nxt], K[0], dt) || !read_stats()) return -1;
        commit(dt);
        return 0;
    }

    // Dormand-Prince 5(4) or Bogacki-Shampine 3(2) attempt; 1 accepted, 0 rejected, -1 error, 2 interrupted
    int rk_adaptive_attempt(double dt, double &next_dt, fullmag_fdm_interrupt_poll_fn poll, void *user) {
        const int nxt = 1 - cur;
        int kfin;
        if (integrator == FULLMAG_FDM_INTEGRATOR_RK23) {
            static const double a2[1] = {0.5}, a3[1] = {0.75};
            static const double b[3] = {2.0 / 9.0, 1.0 / 3.0, 4.0 / 9.0};
            static const double e[4] = {-5.0 / 72.0, 1.0 / 12.0, 1.0 / 9.0, -1.0 / 8.0};
            const int k0[1] = {0}, self[1] = {-1}, kb[3] = {0, 1, -1}, ke[4] = {0, 1, 2, -1};
            if (!first(1, k0, a2, dt, A[0])) return -1;
            if (poll_hit(poll, user)) return 2;
            if (!stage(A[0], K[1], 1, self, a3, dt, A[1])) return -1;
            if (poll_hit(poll, user)) return 2;
            if (!stage(A[1], K[2], 3, kb, b, dt, S[nxt])) return -1;
            if (!final_eval(S[nxt], K[3], dt, 4, ke, e)) return -1;
            kfin = 3;
        } else {
            static const double a21[1] = {1.0 / 5.0};
            static const double a3[2] = {3.0 / 40.0, 9.0 / 40.0};
            static const double a4[3] = {44.0 / 45.0, -56.0 / 15.0, 32.0 / 9.0};
            static const double a5[4] = {19372.0 / 6561.0, -25360.0 / 2187.0, 64448.0 / 6561.0, -212.0 / 729.0};
            static const double a6[5] = {9017.0 / 3168.0, -355.0 / 33.0, 46732.0 / 5247.0, 49.0 / 176.0, -5103.0 / 18656.0};
            static const double b[5] = {35.0 / 384.0, 500.0 / 1113.0, 125.0 / 192.0, -2187.0 / 6784.0, 11.0 / 84.0};
            static const double e[6] = {71.0 / 57600.0, -71.0 / 16695.0, 71.0 / 1920.0, -17253.0 / 339200.0, 22.0 / 525.0,
                                        -1.0 / 40.0};
            const int k1[1] = {0}, k2[2] = {0, -1}, k3[3] = {0, 1, -1}, k4[4] = {0, 1, 2, -1}, k5[5] = {0, 1, 2, 3, -1};
            const int kb[5] = {0, 2, 3, 4, -1}, ke[6] = {0, 2, 3, 4, 5, -1};
            if (!first(1, k1, a21, dt, A[0])) return -1;
            if (poll_hit(poll, user)) return 2;
            if (!stage(A[0], K[1], 2, k2, a3, dt, A[1])) return -1;
            if (poll_hit(poll, user)) return 2;
            if (!stage(A[1], K[2], 3, k3, a4, dt, A[0])) return -1;
            if (poll_hit(poll, user)) return 2;
            if (!stage(A[0], K[3], 4, k4, a5, dt, A[1])) return -1;
            if (poll_hit(poll, user)) return 2;
            if (!stage(A[1], K[4], 5, k5, a6, dt, A[0])) return -1;
            if (poll_hit(poll, user)) return 2;
            if (!stage(A[0], K[5], 5, kb, b, dt, S[nxt])) return -1;
            if (!final_eval(S[nxt], K[6], dt, 6, ke, e)) return -1;
            kfin = 6;
        }
        if (!read_stats()) return -1;
        const double er = sqrt(hstats[8]);
        const double ex = integrator == FULLMAG_FDM_INTEGRATOR_RK23 ? 1.0 / 3.0 : 0.2;
        if (er <= max_error || dt <= dt_min) {
            double dtn = dt_max;
            if (er > 0.0) dtn = std::min(std::max(headroom * dt * pow(max_error / er, ex), dt_min), dt_max);
            std::swap(K[0], K[kfin]);  // first same as last
            commit(dt);
            cur_stats.suggested_next_dt = dtn;
            next_dt = dtn;
            return 1;
        }
        next_dt = std::min(std::max(headroom * dt * pow(max_error / er, ex), dt_min), dt_max);
        return 0;
    }

    // Adams-Bashforth-Moulton 3 as in the FP32 path: Heun steps build the history
    int abm3(double dt, fullmag_fdm_interrupt_poll_fn poll, void *user) {
        if (abm_last_dt > 0.0 && std::fabs(dt - abm_last_dt) / abm_last_dt > 0.1) abm_startup = 0;
        const int nxt = 1 - cur;
        if (abm_startup < 3) {
            const int saved = integrator;
            integrator = FULLMAG_FDM_INTEGRATOR_HEUN;
            const int rc = rk_fixed(dt, poll, user);
            integrator = saved;
            if (rc != 0) return rc;
            const int slot = abm_hist[2];
            abm_hist[2] = abm_hist[1];
            abm_hist[1] = abm_hist[0];
            abm_hist[0] = slot;
            if (fail("history copy", cudaMemcpyAsync(K[slot], K[0], sizeof(double) * 3 * n, cudaMemcpyDeviceToDevice, stream)))
                return -1;
            abm_startup += 1;
        } else {
            const int kp[3] = {abm_hist[0], abm_hist[1], abm_hist[2]};
            const double cp[3] = {23.0 / 12.0, -16.0 / 12.0, 5.0 / 12.0};
            if (!first(3, kp, cp, dt, A[0])) return -1;
            if (poll_hit(poll, user)) return 1;
            const int kc[3] = {-1, abm_hist[0], abm_hist[1]};
            const double cc[3] = {5.0 / 12.0, 8.0 / 12.0, -1.0 / 12.0};
            if (!stage(A[0], K[abm_kf], 3, kc, cc, dt, S[nxt])) return -1;
            if (poll_hit(poll, user)) return 1;
            k1_valid = false;
            if (!final_eval(S[nxt], K[0], dt) || !read_stats()) return -1;
            const int freed = abm_hist[2];
            abm_hist[2] = abm_hist[1];
            abm_hist[1] = abm_hist[0];
            abm_hist[0] = abm_kf;
            abm_kf = freed;
            commit(dt);
        }
        abm_last_dt = dt;
        return 0;
    }
};

bool Fp64Engine::setup(const fullmag_fdm_plan_desc *plan) {
    nx = (int)plan->grid.nx;
    ny = (int)plan->grid.ny;
    nz = (int)plan->grid.nz;
    n = (long long)nx * ny * nz;
    dx = plan->grid.dx;
    dy = plan->grid.dy;
    dz = plan->grid.dz;
    ms = plan->material.saturation_magnetisation;
    a_ex = plan->material.exchange_stiffness;
    alpha = plan->material.damping;
    gamma = plan->material.gyromagnetic_ratio;
    integrator = plan->integrator;
    exchange = plan->enable_exchange != 0;
    demag = plan->enable_demag != 0;
    prec = plan->disable_precession == 0;
    has_ext = plan->has_external_field != 0;
    for (int c = 0; c < 3; ++c) hext[c] = has_ext ? plan->external_field_am[c] : 0.0;
    max_error = plan->adaptive_max_error > 0 ? plan->adaptive_max_error : 1e-5;
    dt_min = plan->adaptive_dt_min > 0 ? plan->adaptive_dt_min : 1e-18;
    dt_max = plan->adaptive_dt_max > 0 ? plan->adaptive_dt_max : 1e-10;
    headroom = plan->adaptive_headroom > 0 ? plan->adaptive_headroom : 0.8;

    if (n == 0) return err = "grid has zero cells", false;
    if (plan->initial_magnetization_xyz == nullptr || plan->initial_magnetization_len != 3 * (uint64_t)n)
        return err = "initial_magnetization_len mismatch: expected " + std::to_string(3 * (uint64_t)n) + ", got " +
                     std::to_string(plan->initial_magnetization_len),
               false;
    if (plan->region_mask && plan->region_mask_len != (uint64_t)n)
        return err = "region_mask_len mismatch: expected " + std::to_string(n) + ", got " + std::to_string(plan->region_mask_len),
               false;
    if (plan->active_mask && plan->active_mask_len != (uint64_t)n)
        return err = "active_mask_len mismatch: expected " + std::to_string(n) + ", got " + std::to_string(plan->active_mask_len),
               false;
    if (!(dx > 0 && dy > 0 && dz > 0)) return err = "cell sizes must be positive", false;
    if (!(ms > 0)) return err = "saturation_magnetisation must be positive", false;
    if (integrator != FULLMAG_FDM_INTEGRATOR_HEUN && integrator != FULLMAG_FDM_INTEGRATOR_RK4 &&
        integrator != FULLMAG_FDM_INTEGRATOR_DP45 && integrator != FULLMAG_FDM_INTEGRATOR_RK23 &&
        integrator != FULLMAG_FDM_INTEGRATOR_ABM3)
        return err = "unsupported integrator", false;
    struct Feat {
        bool on;
        const char *what;
    };
    const Feat rejected[] = {
        {plan->has_interfacial_dmi != 0 || plan->has_bulk_dmi != 0, "DMI"},
        {plan->has_magnetoelastic != 0, "magnetoelastic coupling"},
        {plan->temperature > 0.0, "thermal noise"},
        {plan->current_density_x != 0.0 || plan->current_density_y != 0.0 || plan->current_density_z != 0.0,
         "spin-transfer torque"},
        {plan->has_sot != 0, "spin-orbit torque"},
        {plan->has_oersted_cylinder != 0, "Oersted field"},
        {plan->ku1_field || plan->ku2_field || plan->kc1_field || plan->kc2_field || plan->kc3_field,
         "per-cell anisotropy maps"},
    };
    for (const Feat &f : rejected)
        if (f.on) return err = std::string(f.what) + " is not available with double-precision state (use SINGLE)", false;

    has_uni = plan->has_uniaxial_anisotropy != 0;
    ku1 = plan->uniaxial_anisotropy_constant;
    ku2 = plan->uniaxial_anisotropy_k2;
    has_cub = plan->has_cubic_anisotropy != 0;
    kc1 = plan->cubic_Kc1;
    kc2 = plan->cubic_Kc2;
    kc3 = plan->cubic_Kc3;
    if (has_uni) {
        const double *a = plan->anisotropy_axis;
        const double nn = sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
        if (!(nn > 0)) return err = "anisotropy_axis must be non-zero", false;
        for (int c = 0; c < 3; ++c) u[c] = a[c] / nn;
    }
    if (has_cub) {
        const double *a = plan->cubic_axis1, *b = plan->cubic_axis2;
        const double na = sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]), nb = sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
        if (!(na > 0 && nb > 0)) return err = "cubic axes must be non-zero", false;
        for (int c = 0; c < 3; ++c) {
            c1[c] = a[c] / na;
            c2[c] = b[c] / nb;
        }
        c3[0] = c1[1] * c2[2] - c1[2] * c2[1];
        c3[1] = c1[2] * c2[0] - c1[0] * c2[2];
        c3[2] = c1[0] * c2[1] - c1[1] * c2[0];
    }

    // boundary tiers (exchange_fp64.cu:162-231): T0 needs the volume and face-link
    // fractions, T1 the volume fractions and boundary distances; without them the tier
    // falls back to the binary-mask exchange, as the reference's dispatch does
    tier = 0;
    if (plan->boundary_correction != FULLMAG_FDM_BOUNDARY_NONE && plan->volume_fraction) {
        if (plan->volume_fraction_len != (uint64_t)n)
            return err = "volume_fraction_len mismatch: expected " + std::to_string(n), false;
        if (plan->boundary_correction == FULLMAG_FDM_BOUNDARY_VOLUME && plan->face_link_xp && plan->face_link_xm &&
            plan->face_link_yp && plan->face_link_ym && plan->face_link_zp && plan->face_link_zm)
            tier = 1;
        else if (plan->boundary_correction == FULLMAG_FDM_BOUNDARY_FULL && plan->delta_xp && plan->delta_xm &&
                 plan->delta_yp && plan->delta_ym && plan->delta_zp && plan->delta_zm)
            tier = 2;
    }
    phi_floor = plan->boundary_phi_floor;
    delta_min = plan->boundary_delta_min;
    if (per && (tier > 0 || (plan->has_demag_boundary_corr && plan->demag_corr_target_count > 0)))
        return err = "boundary correction is not available with periodic boundaries", false;
    if (plan->has_demag_boundary_corr && plan->demag_corr_target_count > 0) {
        if (!plan->demag_corr_target_idx || !plan->demag_corr_source_idx || !plan->demag_corr_tensor ||
            plan->demag_corr_stencil_size == 0)
            return err = "demag boundary correction arrays are incomplete", false;
        corr_targets = plan->demag_corr_target_count;
        corr_stencil = plan->demag_corr_stencil_size;
        const size_t ns = (size_t)corr_targets * corr_stencil;
        for (uint32_t t = 0; t < corr_targets; ++t)
            if (plan->demag_corr_target_idx[t] >= (int64_t)n) return err = "demag correction target index out of range", false;
        for (size_t s = 0; s < ns; ++s)
            if (plan->demag_corr_source_idx[s] >= (int64_t)n) return err = "demag correction source index out of range", false;
    }

    // ---- device ----
    if (fail("cudaGetDevice", cudaGetDevice(&device))) return false;
    if (fail("cudaStreamCreate", cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking))) return false;
    const size_t v3 = 3 * (size_t)n;
    for (int s = 0; s < 2; ++s)
        if (!alloc(S[s], v3) || !alloc(A[s], v3)) return false;
    for (int s = 0; s < 7; ++s)
        if (!alloc(K[s], v3)) return false;
    if (!alloc(hex, v3) || !alloc(hd, v3) || !alloc(heff, v3) || !alloc(staging, v3) ||
        !alloc(partials, (size_t)ny * nz * kStats) || !alloc(dstats, kStats) || (corr_targets > 0 && !alloc(hcorr, v3)))
        return false;
    if (fail("cudaMemsetAsync", cudaMemsetAsync(hd, 0, sizeof(double) * v3, stream))) return false;
    if (fail("cudaMallocHost", cudaMallocHost((void **)&hstats, sizeof(double) * kStats))) return false;
    if (plan->active_mask) {
        has_mask = true;
        mask_host.assign(plan->active_mask, plan->active_mask + n);
        if (!put(mask, plan->active_mask, (size_t)n)) return false;
    }
    if (plan->region_mask) {
        std::vector<uint8_t> r((size_t)n);
        for (long long i = 0; i < n; ++i) {
            if (plan->region_mask[i] >= FULLMAG_FDM_MAX_EXCHANGE_REGIONS)
                return err = "region_mask ids must be below " + std::to_string(FULLMAG_FDM_MAX_EXCHANGE_REGIONS), false;
            r[i] = (uint8_t)plan->region_mask[i];
        }
        // the caller's table when it has 256 x 256 entries, else A on the diagonal (api.cpp:405-420)
        const size_t R = FULLMAG_FDM_MAX_EXCHANGE_REGIONS, R2 = R * R;
        std::vector<double> table(R2, 0.0);
        if (plan->exchange_lut && plan->exchange_lut_len == R2) std::copy(plan->exchange_lut, plan->exchange_lut + R2, table.begin());
        else
            for (size_t q = 0; q < R; ++q) table[q * R + q] = a_ex;
        if (!put(region, r.data(), r.size()) || !put(lut, table.data(), R2)) return false;
    }
    if (tier > 0 || corr_targets > 0) {
        if (plan->volume_fraction && plan->volume_fraction_len == (uint64_t)n) {
            if (!put(phi, plan->volume_fraction, (size_t)n)) return false;
        }
    }
    if (tier == 1) {
        const double *f[6] = {plan->face_link_xp, plan->face_link_xm, plan->face_link_yp,
                              plan->face_link_ym, plan->face_link_zp, plan->face_link_zm};
        for (int q = 0; q < 6; ++q)
            if (!put(face[q], f[q], (size_t)n)) return false;
    } else if (tier == 2) {
        const double *d[6] = {plan->delta_xp, plan->delta_xm, plan->delta_yp, plan->delta_ym, plan->delta_zp, plan->delta_zm};
        for (int q = 0; q < 6; ++q)
            if (!put(delta[q], d[q], (size_t)n)) return false;
    }
    if (corr_targets > 0) {
        const size_t ns = (size_t)corr_targets * corr_stencil;
        if (!put(ctidx, plan->demag_corr_target_idx, corr_targets) || !put(csidx, plan->demag_corr_source_idx, ns) ||
            !put(ctensor, plan->demag_corr_tensor, 6 * ns))
            return false;
    }

    // ---- demag: padded geometry P = 2n per axis (thin film: 2-D when nz == 1) ----
    if (demag) {
        Conv64 &C = conv;
        C.nx = nx;
        C.ny = ny;
        C.nz = nz;
        C.n = n;
        // periodic axes (fdm_fft.rs:140-160): unpadded, and the backend builds the tensor
        C.px = (per & 1) ? nx : 2 * nx;
        C.py = (per & 2) ? ny : 2 * ny;
        if (plan->demag_kernel_spectrum_len == 0) {
            if (!(per & 1)) C.px = pad_extent64(nx);
            if (!(per & 2)) C.py = pad_extent64(ny);
        }
        if (per && plan->demag_kernel_spectrum_len != 0)
            return err = "periodic boundaries: the backend builds the image-sum demag tensor, the plan must carry no spectra",
                   false;
        const uint64_t len3 = 2ull * (uint64_t)(2 * nx) * (2 * ny) * (2 * nz);
        const uint64_t len2 = 2ull * (uint64_t)(2 * nx) * (2 * ny);
        const bool given = plan->demag_kernel_spectrum_len != 0;
        bool thin = false;
        if (!given) {
            thin = nz == 1;
        } else {
            if (!plan->demag_kernel_xx_spectrum || !plan->demag_kernel_yy_spectrum || !plan->demag_kernel_zz_spectrum ||
                !plan->demag_kernel_xy_spectrum || !plan->demag_kernel_xz_spectrum || !plan->demag_kernel_yz_spectrum)
                return err = "demag kernel spectra pointers must all be present when demag_kernel_spectrum_len is set", false;
            if (nz == 1 && plan->demag_kernel_spectrum_len == len2) thin = true;
            else if (plan->demag_kernel_spectrum_len != len3)
                return err = "demag_kernel_spectrum_len mismatch: expected " + std::to_string(len3) + " (3D)" +
                             (nz == 1 ? " or " + std::to_string(len2) + " (thin-film 2D)" : std::string()) + ", got " +
                             std::to_string(plan->demag_kernel_spectrum_len),
                       false;
        }
        C.thin = thin;
        C.pz = thin ? 1 : (per & 4) ? nz : given ? 2 * nz : pad_extent64(nz);
        C.nkx = C.px / 2 + 1;
        C.nky = C.py / 2 + 1;
        C.nkz = C.pz / 2 + 1;
        // an even x extent is transformed at half its length, two real samples per complex one;
        // rows too long for the fused row pass take full lines of a pass of their own
        C.half = C.px % 2 == 0 ? C.px / 2 : 0;
        if (!choose_shapes()) {
            C.px = (per & 1) ? nx : 2 * nx;  // the least padding, then again
            C.py = (per & 2) ? ny : 2 * ny;
            C.pz = thin ? 1 : (per & 4) ? nz : 2 * nz;
            C.nkx = C.px / 2 + 1;
            C.nky = C.py / 2 + 1;
            C.nkz = C.pz / 2 + 1;
            C.half = C.px % 2 == 0 ? C.px / 2 : 0;
            if (!choose_shapes()) return err = "grid too large for the double-precision FFT lines", false;
        }
        if (!fused_x) C.half = 0;
        std::vector<double2> tw;
        std::vector<size_t> off;
        if (!make_plan64(C.half ? C.half : C.px, tw, off, C.plx) || !make_plan64(C.py, tw, off, C.ply) ||
            !make_plan64(C.pz, tw, off, C.plz))
            return err = "FFT length has too many factors", false;
        auto even = [](const Plan64 &p) { return p.ns > 0 && p.radix[0] % 2 == 0; };
        C.xprune = C.half && 2 * ((nx + 1) / 2) <= C.half && even(C.plx);
        C.yprune = 2 * ny <= C.py && even(C.ply);
        C.zprune = 2 * nz <= C.pz && even(C.plz);
        const size_t post = tw.size();
        for (int k = 0; k <= C.half; ++k) {
            const double a = 2.0 * M_PI * (double)k / (double)C.px;
            tw.push_back(make_double2(cos(a), -sin(a)));
        }
        if (!put(twid, tw.data(), tw.size())) return false;
        C.plx.tw = twid + off[0];
        C.ply.tw = twid + off[1];
        C.plz.tw = twid + off[2];
        C.xpost = twid + post;
        const int ncomp = thin ? 4 : 6;
        const size_t kper = per ? (size_t)C.pz * C.py * C.nkx : (size_t)C.nkz * C.nky * C.nkx;
        if (per ? !alloc(kernc, ncomp * kper) : !alloc(kern, ncomp * kper)) return false;
        if (!alloc(X, 3 * (size_t)nz * ny * C.nkx)) return false;
        if (!thin && !alloc(Y, 3 * (size_t)nz * C.py * C.nkx)) return false;
        const void *big[] = {(const void *)row64, (const void *)convolve64<true>, (const void *)convolve64<false>,
                             (const void *)x_forward64, (const void *)x_inverse64, (const void *)y_forward64,
                             (const void *)y_inverse64};
        for (const void *f : big)
            if (fail("cudaFuncSetAttribute", cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                                  (int)(f == big[0] ? kMaxSmem - 1024 : kMaxSmem))))
                return false;
        const double xs = C.half ? 0.5 : 1.0;  // the packed split stores twice the spectrum (exact)
        if (given) {
            const double *src[6] = {plan->demag_kernel_xx_spectrum, plan->demag_kernel_yy_spectrum, plan->demag_kernel_zz_spectrum,
                                    plan->demag_kernel_xy_spectrum, plan->demag_kernel_xz_spectrum, plan->demag_kernel_yz_spectrum};
            const double scale = xs * ms / ((double)C.px * C.py * C.pz);
            std::vector<double> h(ncomp * kper);
            for (int c = 0; c < ncomp; ++c)
                for (int kz = 0; kz < C.nkz; ++kz)
                    for (int ky = 0; ky < C.nky; ++ky)
                        for (int kx = 0; kx < C.nkx; ++kx) {
                            const size_t s = (size_t)kx + (size_t)C.px * (ky + (size_t)C.py * kz);
                            h[(size_t)c * kper + ((size_t)kz * C.nky + ky) * C.nkx + kx] = src[c][2 * s] * scale;
                        }
            if (fail("cudaMemcpy(kernel)", cudaMemcpyAsync(kern, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice, stream)) ||
                fail("kernel sync", cudaStreamSynchronize(stream)))
                return false;
        } else {
            Grid g{};
            g.nx = nx;
            g.ny = ny;
            g.nz = nz;
            g.n = n;
            g.px = C.px;
            g.py = C.py;
            g.pz = C.pz;
            g.half = C.px / 2;
            g.nkx = C.nkx;
            g.nky = C.nky;
            g.nkz = C.nkz;
            g.thin = thin;
            g.per = per;
            if (per ? !newell_periodic_spectrum_gpu(g, dx, dy, dz, xs * ms, images, nullptr, kernc, stream, err)
                    : !newell_spectrum_gpu64(g, dx, dy, dz, xs * ms, kern, stream, err))
                return false;
        }
        C.kern = kern;
        C.kernc = kernc;
    } else if (!choose_shapes()) {
        return err = "grid too large", false;
    }
    early = n <= 65536;
    return true;
}

bool Fp64Engine::upload(const double *m_xyz) {
    if (fail("cudaMemcpy(state)", cudaMemcpyAsync(staging, m_xyz, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, stream)))
        return false;
    aos_to_soa64<<<blocks_for(n), kT, 0, stream>>>(staging, S[cur], mask, tier > 0 ? phi : nullptr, n);
    if (fail("upload convert", cudaGetLastError())) return false;
    k1_valid = false;
    abm_startup = 0;
    abm_last_dt = 0.0;
    return eval_state();
}

bool fp64_refresh(Fp64Engine *e, std::string &err);

Fp64Engine *fp64_create(const fullmag_fdm_plan_desc *plan, std::string &err, int periodic, const uint32_t *images) {
    Fp64Engine *e = new (std::nothrow) Fp64Engine();
    if (!e) {
        err = "out of host memory";
        return nullptr;
    }
    e->per = periodic;
    if (images)
        for (int a = 0; a < 3; ++a) e->images[a] = images[a];
    if (!e->setup(plan) || !e->upload(plan->initial_magnetization_xyz)) {
        err = e->err;
        delete e;
        return nullptr;
    }
    e->cur_stats.step = 0;
    e->cur_stats.time_seconds = 0.0;
    return e;
}

void fp64_destroy(Fp64Engine *e) { delete e; }

int fp64_step(Fp64Engine *e, double dt, fullmag_fdm_step_stats *out, fullmag_fdm_interrupt_poll_fn poll, void *user,
              std::string &err) {
    const auto t0 = std::chrono::steady_clock::now();
    e->err.clear();
    int rc = 0;
    if (!e->k1_valid && !e->eval_state()) rc = -1;
    else if (e->poll_hit(poll, user)) rc = 1;
    else if (e->integrator == FULLMAG_FDM_INTEGRATOR_DP45 || e->integrator == FULLMAG_FDM_INTEGRATOR_RK23) {
        for (;;) {
            double next = dt;
            const int a = e->rk_adaptive_attempt(dt, next, poll, user);
            if (a < 0) {
                rc = -1;
                break;
            }
            if (a == 2) {
                rc = 1;
                break;
            }
            if (a == 1) break;
            dt = next;
        }
    } else if (e->integrator == FULLMAG_FDM_INTEGRATOR_ABM3) {
        rc = e->abm3(dt, poll, user);
    } else {
        rc = e->rk_fixed(dt, poll, user);
    }
    err = e->err;
    if (rc < 0) return FULLMAG_FDM_ERR_CUDA;
    *out = e->cur_stats;
    if (rc == 1) {
        out->dt_seconds = 0.0;
        out->wall_time_ns = 0;
        err = "interrupted";
        return FULLMAG_FDM_ERR_INTERRUPTED;
    }
    out->wall_time_ns =
        (uint64_t)std::chrono::duration_cast<std::chrono::nanoseconds>(std::chrono::steady_clock::now() - t0).count();
    e->cur_stats.wall_time_ns = out->wall_time_ns;
    return FULLMAG_FDM_OK;
}

bool fp64_download(Fp64Engine *e, int obs, double *out, std::string &err) {
    const long long n = e->n;
    if (obs == FULLMAG_FDM_OBSERVABLE_H_EXT) {
        for (long long i = 0; i < n; ++i) {
            const bool act = !e->has_mask || e->mask_host[i] != 0;
            for (int c = 0; c < 3; ++c) out[3 * i + c] = (e->has_ext && act) ? e->hext[c] : 0.0;
        }
        return true;
    }
    const double *src = nullptr;
    switch (obs) {
        case FULLMAG_FDM_OBSERVABLE_M: src = e->S[e->cur]; break;
        case FULLMAG_FDM_OBSERVABLE_H_EX: src = e->hex; break;
        case FULLMAG_FDM_OBSERVABLE_H_DEMAG: src = e->hd; break;
        case FULLMAG_FDM_OBSERVABLE_H_EFF: src = e->heff; break;
        default: err = "unknown observable " + std::to_string(obs); return false;
    }
    // the field buffers hold the last evaluation: after an interrupted step or a rejected
    // attempt that is not the committed state, which is evaluated again
    if (obs != FULLMAG_FDM_OBSERVABLE_M && !e->fields_ok && !fp64_refresh(e, err)) return false;
    soa_to_aos64<<<blocks_for(n), kT, 0, e->stream>>>(src, e->staging, n);
    if (e->fail("download convert", cudaGetLastError()) ||
        e->fail("cudaMemcpy(field)", cudaMemcpyAsync(out, e->staging, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, e->stream)) ||
        e->fail("download sync", cudaStreamSynchronize(e->stream))) {
        err = e->err;
        return false;
    }
    return true;
}

bool fp64_upload(Fp64Engine *e, const double *m_xyz, std::string &err) {
    const bool ok = e->upload(m_xyz);
    if (!ok) err = e->err;
    return ok;
}

bool fp64_refresh(Fp64Engine *e, std::string &err) {
    const fullmag_fdm_step_stats keep = e->cur_stats;
    const bool ok = e->eval_state();
    if (!ok) {
        err = e->err;
        return false;
    }
    e->cur_stats.dt_seconds = keep.dt_seconds;
    e->cur_stats.suggested_next_dt = keep.suggested_next_dt;
    e->cur_stats.wall_time_ns = keep.wall_time_ns;
    return true;
}

void fp64_stats(const Fp64Engine *e, fullmag_fdm_step_stats *out) { *out = e->cur_stats; }

void fp64_grid(const Fp64Engine *e, int &nx, int &ny, int &nz) {
    nx = e->nx;
    ny = e->ny;
    nz = e->nz;
}

int fp64_device(const Fp64Engine *e) { return e->device; }

void fp64_fft_shape(const Fp64Engine *e, uint32_t &px, uint32_t &py, uint32_t &pz) {
    px = e->demag ? (uint32_t)e->conv.px : 0;
    py = e->demag ? (uint32_t)e->conv.py : 0;
    pz = e->demag ? (uint32_t)e->conv.pz : 0;
}

}  // namespace fm
