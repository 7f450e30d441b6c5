// fft_smem.cuh -- shared-memory Stockham FFT used by every demag pass.
//
// A CTA transforms `nlines` complex lines of length n that sit in shared
// memory, ping-ponging between two buffers.  Element e of line l lives at
// buf[l * ls + sk(e)]: one float2 of padding after every 16 elements keeps the
// stride-R writes of the early Stockham stages off a single pair of banks
// (ls >= skewed_len(n)).  Each stage of radix R is one sweep of n/R butterflies
// per line; the Stockham index map keeps the result in natural order.
//
// Power-of-two lengths (every padded extent of the reference's 2n grids when n
// is a power of two) take a compile-time path: radix-16 stages where possible,
// then radix 8 or 4 (pow2_radix: never a lone radix-2 stage), all index
// arithmetic folded to shifts and masks.  Other lengths use the runtime path
// with radices 8, 4, 2, 3, 5, 7 and an O(R^2) loop for any other prime factor.  Twiddles are FP64-computed host-side and stored as
// float2 e^{-2 pi i e / n}; the inverse conjugates them.
//
// The passes over engine-built tensors take the two-level transforms further down at the
// lengths of two_level_length (2^a times 1, 5/4, 3/2 or 7/4).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fm {

constexpr int kMaxStages = 24;
constexpr int kMaxGenericRadix = 64;

struct FftPlan {
    int n;
    int nstages;
    int log2n;  // >= 0 when n is a power of two, else -1
    int radix[kMaxStages];
    const float2 *tw;  // n entries, e^{-2 pi i e / n}
};

// Division by a runtime divisor d >= 1 through a precomputed multiplier
// (round-up reciprocal method: q = (umulhi(n, m) + n) >> s with
// s = ceil(log2 d), m = floor(2^32 (2^s - d) / d) + 1), exact for n < 2^31.
struct FastDiv {
    uint32_t d = 1, m = 1, s = 0;
    FastDiv() = default;
    __host__ explicit FastDiv(uint32_t div) : d(div) {
        s = 0;
        while ((1ull << s) < div) ++s;
        m = (uint32_t)(((1ull << 32) * ((1ull << s) - div)) / div + 1);
    }
    __device__ __forceinline__ int div(int n) const {
        return (int)((__umulhi((uint32_t)n, m) + (uint32_t)n) >> s);
    }
    __device__ __forceinline__ int mod(int n, int q) const { return n - q * (int)d; }
};

__host__ __device__ __forceinline__ int sk(int e) { return e + (e >> 4); }

// Gather `total` elements: B independent loads per thread are issued before any of
// them is consumed, so each thread keeps B requests in flight (the passes are
// latency-bound otherwise: one outstanding load per thread at 2-4 CTAs per SM).
template <int B, typename Load, typename Store>
__device__ __forceinline__ void batched_copy(int total, Load ld, Store st) {
    for (int base = threadIdx.x; base < total; base += B * blockDim.x) {
        float2 v[B];
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int idx = base + u * (int)blockDim.x;
            if (idx < total) v[u] = ld(idx);
        }
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int idx = base + u * (int)blockDim.x;
            if (idx < total) st(idx, v[u]);
        }
    }
}

// Compensated float-float accumulation (Knuth TwoSum): hi + lo carries the sum of
// every added value with error ~ n * eps^2 instead of n * eps, using FP32 pipes only.
__device__ __forceinline__ void ff_add(float &hi, float &lo, float v) {
    const float s = hi + v;
    const float bb = s - hi;
    const float e = (hi - (s - bb)) + (v - bb);
    hi = s;
    lo += e;
}
__host__ __device__ constexpr int skewed_len(int n) {
    // odd, so that neighbouring lines start in different banks; lines of which one column fills the
    // shared memory keep the last element instead (a film of 4557 periodic rows needs it)
    return (n + (n >> 4) + 1) | (n <= 4096 ? 1 : 0);
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
// multiply by -i (forward) or +i (inverse)
__device__ __forceinline__ float2 mul_mi(float2 a, bool inv) {
    return inv ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

// ---- butterflies of radix 3, 5, 7 and of two coprime factors, on one complex line
// (float2) or on a pair of lines (cp2, fft_pair.cuh) ----
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return cadd(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return csub(a, b); }
__device__ __forceinline__ float2 vscale(float c, float2 a) { return make_float2(c * a.x, c * a.y); }
__device__ __forceinline__ float2 vfma(float c, float2 a, float2 b) {
    return make_float2(fmaf(c, a.x, b.x), fmaf(c, a.y, b.y));
}
__device__ __forceinline__ float2 vmul_mi(float2 a, bool inv) { return mul_mi(a, inv); }

// cos and sin of 2 pi m / P for P = 3, 5, 7 (m < P)
template <int P>
__device__ __forceinline__ constexpr float odd_cos(int m) {
    constexpr float c3 = -0.5f;
    constexpr float c5[2] = {0.30901699437494742410f, -0.80901699437494742410f};
    constexpr float c7[3] = {0.62348980185873353053f, -0.22252093395631440429f, -0.90096886790241912624f};
    const int q = m > P / 2 ? P - m : m;
    return q == 0 ? 1.f : P == 3 ? c3 : P == 5 ? c5[(q - 1) & 1] : c7[q - 1];
}
template <int P>
__device__ __forceinline__ constexpr float odd_sin(int m) {
    constexpr float s3 = 0.86602540378443864676f;
    constexpr float s5[2] = {0.95105651629515357212f, 0.58778525229247312917f};
    constexpr float s7[3] = {0.78183148246802980871f, 0.97492791218182360702f, 0.43388373911755812048f};
    const int q = m > P / 2 ? P - m : m;
    const float v = q == 0 ? 0.f : P == 3 ? s3 : P == 5 ? s5[(q - 1) & 1] : s7[q - 1];
    return m > P / 2 ? -v : v;
}

// Odd prime P: the inputs n and P - n are folded into a sum and a difference, so each
// output pair k, P - k takes P - 1 real-by-complex products.
template <int P, typename V>
__device__ __forceinline__ void dft_odd(V *v, bool inv) {
    constexpr int H = P / 2;
    V t[H], d[H];
#pragma unroll
    for (int j = 0; j < H; ++j) {
        t[j] = vadd(v[1 + j], v[P - 1 - j]);
        d[j] = vsub(v[1 + j], v[P - 1 - j]);
    }
    const V v0 = v[0];
    V sum = v0;
#pragma unroll
    for (int j = 0; j < H; ++j) sum = vadd(sum, t[j]);
    v[0] = sum;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        V m = vfma(odd_cos<P>(k % P), t[0], v0), n = vscale(odd_sin<P>(k % P), d[0]);
#pragma unroll
        for (int j = 1; j < H; ++j) {
            m = vfma(odd_cos<P>(((j + 1) * k) % P), t[j], m);
            n = vfma(odd_sin<P>(((j + 1) * k) % P), d[j], n);
        }
        n = vmul_mi(n, inv);
        v[k] = vadd(m, n);
        v[P - k] = vsub(m, n);
    }
}

template <int R>
__device__ __forceinline__ void dft_small(float2 *v, bool inv);
template <int R>
__device__ __forceinline__ void dft_v(float2 *v, bool inv) {
    dft_small<R>(v, inv);
}

// R = A B with A, B coprime (the prime-factor map n = B a + A b mod R, k -> (k mod A,
// k mod B)): an A x B transform without twiddles.
template <int A, int B, typename V>
__device__ __forceinline__ void dft_coprime(V *v, bool inv) {
    constexpr int R = A * B;
    V t[A][B];
#pragma unroll
    for (int a = 0; a < A; ++a) {
#pragma unroll
        for (int b = 0; b < B; ++b) t[a][b] = v[(B * a + A * b) % R];
        dft_v<B>(t[a], inv);
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
        V u[A];
#pragma unroll
        for (int a = 0; a < A; ++a) u[a] = t[a][b];
        dft_v<A>(u, inv);
#pragma unroll
        for (int a = 0; a < A; ++a) t[a][b] = u[a];
    }
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = t[k % A][k % B];
}

template <>
__device__ __forceinline__ void dft_small<1>(float2 *, bool) {}
template <>
__device__ __forceinline__ void dft_small<3>(float2 *v, bool inv) {
    dft_odd<3>(v, inv);
}
template <>
__device__ __forceinline__ void dft_small<5>(float2 *v, bool inv) {
    dft_odd<5>(v, inv);
}
template <>
__device__ __forceinline__ void dft_small<7>(float2 *v, bool inv) {
    dft_odd<7>(v, inv);
}

template <>
__device__ __forceinline__ void dft_small<2>(float2 *v, bool) {
    float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
}

template <>
__device__ __forceinline__ void dft_small<4>(float2 *v, bool inv) {
    float2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
    float2 b0 = cadd(v[1], v[3]), b1 = mul_mi(csub(v[1], v[3]), inv);
    v[0] = cadd(a0, b0);
    v[2] = csub(a0, b0);
    v[1] = cadd(a1, b1);
    v[3] = csub(a1, b1);
}

template <>
__device__ __forceinline__ void dft_small<8>(float2 *v, bool inv) {
    // radix-2 decimation in frequency, then two 4-point DFTs
    const float h = 0.70710678118654752440f;
    float2 a[4], b[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        a[t] = cadd(v[t], v[t + 4]);
        b[t] = csub(v[t], v[t + 4]);
    }
    // b[t] *= W8^t  (W8 = e^{-i pi/4} forward, conjugate for inverse)
    {
        float2 x = b[1];
        b[1] = inv ? make_float2(h * (x.x - x.y), h * (x.x + x.y)) : make_float2(h * (x.x + x.y), h * (x.y - x.x));
        b[2] = mul_mi(b[2], inv);
        x = b[3];
        b[3] = inv ? make_float2(-h * (x.x + x.y), h * (x.x - x.y)) : make_float2(h * (x.y - x.x), -h * (x.x + x.y));
    }
    dft_small<4>(a, inv);
    dft_small<4>(b, inv);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v[2 * q] = a[q];
        v[2 * q + 1] = b[q];
    }
}

template <>
__device__ __forceinline__ void dft_small<16>(float2 *v, bool inv) {
    // 16 = 4 x 4: x index 4*n1 + n2, output index k1 + 4*k2
    //   X[k1 + 4 k2] = sum_n2 W4^{n2 k2} W16^{n2 k1} sum_n1 x[4 n1 + n2] W4^{n1 k1}
    // cos / sin of 2 pi e / 16 for e = n2 * k1 in [0, 9]
    const float c16[10] = {1.0f, 0.92387953251128674f, 0.70710678118654752f, 0.38268343236508977f, 0.0f,
                           -0.38268343236508977f, -0.70710678118654752f, -0.92387953251128674f, -1.0f,
                           -0.92387953251128674f};
    const float s16[10] = {0.0f, 0.38268343236508977f, 0.70710678118654752f, 0.92387953251128674f, 1.0f,
                           0.92387953251128674f, 0.70710678118654752f, 0.38268343236508977f, 0.0f,
                           -0.38268343236508977f};
    float2 t[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
        float2 a[4] = {v[n2], v[4 + n2], v[8 + n2], v[12 + n2]};
        dft_small<4>(a, inv);
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            const int e = n2 * k1;
            if (e == 0) {
                t[n2][k1] = a[k1];
            } else {
                // W16^e = cos - i sin (forward), cos + i sin (inverse)
                const float2 w = make_float2(c16[e], inv ? s16[e] : -s16[e]);
                t[n2][k1] = cmul(a[k1], w);
            }
        }
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
        float2 b[4] = {t[0][k1], t[1][k1], t[2][k1], t[3][k1]};
        dft_small<4>(b, inv);
#pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = b[k2];
    }
}

template <>
__device__ __forceinline__ void dft_small<6>(float2 *v, bool inv) {
    dft_coprime<2, 3>(v, inv);
}
template <>
__device__ __forceinline__ void dft_small<10>(float2 *v, bool inv) {
    dft_coprime<2, 5>(v, inv);
}
template <>
__device__ __forceinline__ void dft_small<12>(float2 *v, bool inv) {
    dft_coprime<4, 3>(v, inv);
}
template <>
__device__ __forceinline__ void dft_small<14>(float2 *v, bool inv) {
    dft_coprime<2, 7>(v, inv);
}

template <>
__device__ __forceinline__ void dft_small<20>(float2 *v, bool inv) {
    dft_coprime<4, 5>(v, inv);
}
template <>
__device__ __forceinline__ void dft_small<24>(float2 *v, bool inv) {
    dft_coprime<8, 3>(v, inv);
}
template <>
__device__ __forceinline__ void dft_small<28>(float2 *v, bool inv) {
    dft_coprime<4, 7>(v, inv);
}
template <>
__device__ __forceinline__ void dft_small<32>(float2 *v, bool inv) {
    // even outputs from v[n] + v[n + 16], odd ones from (v[n] - v[n + 16]) W32^n
    const float c32[16] = {1.0f,           0.98078528040323043f,  0.92387953251128674f,  0.83146961230254524f,
                           0.70710678118654752f,  0.55557023301960218f,  0.38268343236508977f,  0.19509032201612825f,
                           0.0f,           -0.19509032201612825f, -0.38268343236508977f, -0.55557023301960218f,
                           -0.70710678118654752f, -0.83146961230254524f, -0.92387953251128674f, -0.98078528040323043f};
    float2 a[16], b[16];
#pragma unroll
    for (int n = 0; n < 16; ++n) {
        a[n] = cadd(v[n], v[n + 16]);
        const float2 d = csub(v[n], v[n + 16]);
        const float s = c32[n < 8 ? 8 - n : n - 8];  // sin(2 pi n / 32)
        b[n] = n == 0 ? d : n == 8 ? mul_mi(d, inv) : cmul(d, make_float2(c32[n], inv ? s : -s));
    }
    dft_small<16>(a, inv);
    dft_small<16>(b, inv);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        v[2 * k] = a[k];
        v[2 * k + 1] = b[k];
    }
}

// radix of the next power-of-two stage given the remaining length 2^m:
// radix 16 where possible, never a lone radix-2 stage (2^5 -> 8 x 4, 2^9 -> 16 x 8 x 4)
__host__ __device__ constexpr int pow2_radix(int rem) {
    return rem >= 16 && rem != 32 ? 16 : (rem >= 8 ? 8 : rem);
}

// ---- two-level transforms, N = N1 * N2 with N1 even ----
// With n = N2 n1 + n2 and k = k1 + N1 k2:
//   X[k1 + N1 k2] = sum_n2 W_N2^{n2 k2} W_N^{n2 k1} sum_n1 x[N2 n1 + n2] W_N1^{n1 k1}.
// Along an open axis inputs vanish for n >= N/2 (n1 >= N1/2) on the forward side and only
// n < N/2 is kept on the inverse side, so the outer N1-point passes run on half lines;
// along a periodic axis (no padding) they run on full ones.  tw holds the N twiddles
// e^{-2 pi i e / N}.
//
// Lengths: 2^a, 5/4 2^a, 3/2 2^a and 7/4 2^a from 16 to 1024, so that padding 2n - 1 samples
// up to the next one costs at most a quarter (11 % on average over log-uniform n) where a
// power of two costs up to a factor of two per axis.  A 150 x 150 x 10 box takes 320 x 320
// x 20 points instead of 512 x 512 x 32.
__host__ __device__ constexpr bool two_level_length(int n) {
    return n == 16 || n == 20 || n == 24 || n == 28 || n == 32 || n == 40 || n == 48 || n == 56 || n == 64 || n == 80 ||
           n == 96 || n == 112 || n == 128 || n == 160 || n == 192 || n == 224 || n == 256 || n == 320 || n == 384 ||
           n == 448 || n == 512 || n == 640 || n == 768 || n == 896 || n == 1024;
}
// Outer length N1 of a pass whose inner pass holds one line of N2 = n / N1 values a thread:
// both at most 16 (N1 counts half on open axes) up to n = 256, 32 beyond.
__host__ __device__ constexpr int split_line(int n) {
    return n <= 28 ? 4 : n <= 64 ? 8 : n <= 256 ? 16 : n <= 512 ? n / 16 : 32;
}
// The same for a convolution pass, whose inner pass holds three lines: N2 <= 8 up to 256.
__host__ __device__ constexpr int split_conv(int n) {
    return n <= 28 ? 4 : n <= 64 ? 8 : n <= 128 ? 16 : n <= 256 ? n / 8 : 32;
}

// N1-point DFT given as its even (e) and odd (o) halves -- inputs of the two N1/2-point
// DFTs that give the even and odd outputs -- times W_N^{n2 k1}, at line[sk(k1 * N2 + n2)].
template <int N1, int N2>
__device__ __forceinline__ void dft_halves_store(float2 (&e)[N1 / 2], float2 (&o)[N1 / 2], int n2, float2 *line,
                                                 const float2 *__restrict__ tw) {
    constexpr int H1 = N1 / 2;
    dft_small<H1>(e, false);
    dft_small<H1>(o, false);
#pragma unroll
    for (int u = 0; u < H1; ++u) {
        const int ka = 2 * u, kb = 2 * u + 1;
        line[sk(ka * N2 + n2)] = (n2 && ka) ? cmul(e[u], __ldg(tw + n2 * ka)) : e[u];
        line[sk(kb * N2 + n2)] = n2 ? cmul(o[u], __ldg(tw + n2 * kb)) : o[u];
    }
}

// Half-input N1-point DFT of e[0..N1/2).
template <int N1, int N2>
__device__ __forceinline__ void half_dft_store(float2 (&e)[N1 / 2], int n2, float2 *line, const float2 *__restrict__ tw) {
    constexpr int H1 = N1 / 2;
    float2 o[H1];
    o[0] = e[0];
#pragma unroll
    for (int n1 = 1; n1 < H1; ++n1) o[n1] = cmul(e[n1], __ldg(tw + n1 * N2));
    dft_halves_store<N1, N2>(e, o, n2, line, tw);
}

// Full N1-point DFT of e[0..N1/2) and f[0..N1/2) = x[N1/2 + n1], in one piece: fewer twiddle
// products than by its even and odd halves, and that much less rounding.
template <int N1, int N2>
__device__ __forceinline__ void full_dft_store(float2 (&e)[N1 / 2], float2 (&f)[N1 / 2], int n2, float2 *line,
                                               const float2 *__restrict__ tw) {
    constexpr int H1 = N1 / 2;
    float2 v[N1];
#pragma unroll
    for (int n1 = 0; n1 < H1; ++n1) {
        v[n1] = e[n1];
        v[H1 + n1] = f[n1];
    }
    dft_small<N1>(v, false);
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1)
        line[sk(k1 * N2 + n2)] = n2 && k1 ? cmul(v[k1], __ldg(tw + n2 * k1)) : v[k1];
}

// Inverse N1-point DFT over line[sk(k1 * N2 + n2)], k1 in [0, N1): y[n1] for n1 < N1/2 in e
// (two N1/2-point inverses combined with W_N1^{-n1}); FULL: y[N1/2 + n1] in f.
template <int N1, int N2, bool FULL>
__device__ __forceinline__ void idft_load(float2 (&e)[N1 / 2], float2 (&f)[N1 / 2], int n2, const float2 *line,
                                          const float2 *__restrict__ tw) {
    constexpr int H1 = N1 / 2;
    if constexpr (FULL) {
        float2 v[N1];
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) v[k1] = line[sk(k1 * N2 + n2)];
        dft_small<N1>(v, true);
#pragma unroll
        for (int n1 = 0; n1 < H1; ++n1) {
            e[n1] = v[n1];
            f[n1] = v[H1 + n1];
        }
    } else {
#pragma unroll
        for (int u = 0; u < H1; ++u) {
            e[u] = line[sk(2 * u * N2 + n2)];
            f[u] = line[sk((2 * u + 1) * N2 + n2)];
        }
        dft_small<H1>(e, true);
        dft_small<H1>(f, true);
#pragma unroll
        for (int n1 = 0; n1 < H1; ++n1) e[n1] = cadd(e[n1], n1 ? cmul(f[n1], cconj(__ldg(tw + n1 * N2))) : f[n1]);
    }
}
template <int N1, int N2>
__device__ __forceinline__ void half_idft_load(float2 (&e)[N1 / 2], int n2, const float2 *line,
                                               const float2 *__restrict__ tw) {
    float2 o[N1 / 2];
    idft_load<N1, N2, false>(e, o, n2, line, tw);
}

// case labels of the two-level lengths: F(n) for each (the long ones hold up to 32 complex values a thread)
#define FM_LENGTHS_TO_256(F) \
    F(16) F(20) F(24) F(28) F(32) F(40) F(48) F(56) F(64) F(80) F(96) F(112) F(128) F(160) F(192) F(224) F(256)
#define FM_LENGTHS_LONG(F) F(320) F(384) F(448) F(512) F(640) F(768) F(896) F(1024)

// ---- runtime-length path ----

template <int R>
__device__ __forceinline__ void stage_fixed(const float2 *__restrict__ in, float2 *__restrict__ out, int nlines, int ls,
                                            int n, int Ns, const float2 *__restrict__ tw, bool inv) {
    const int nb = n / R;
    const int total = nlines * nb;
    const int twstride = n / (Ns * R);
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int l = idx / nb;
        const int j = idx - l * nb;
        const float2 *src = in + (size_t)l * ls;
        float2 *dst = out + (size_t)l * ls;
        const int k = j % Ns;
        float2 v[R];
#pragma unroll
        for (int t = 0; t < R; ++t) v[t] = src[sk(j + t * nb)];
        if (Ns > 1) {
#pragma unroll
            for (int t = 1; t < R; ++t) {
                float2 w = __ldg(tw + t * k * twstride);
                if (inv) w.y = -w.y;
                v[t] = cmul(v[t], w);
            }
        }
        dft_small<R>(v, inv);
        const int o = (j / Ns) * Ns * R + k;
#pragma unroll
        for (int t = 0; t < R; ++t) dst[sk(o + t * Ns)] = v[t];
    }
}

__device__ __forceinline__ void stage_generic(const float2 *__restrict__ in, float2 *__restrict__ out, int nlines, int ls,
                                              int n, int Ns, int R, const float2 *__restrict__ tw, bool inv) {
    const int nb = n / R;
    const int total = nlines * nb;
    const int twstride = n / (Ns * R);
    const int rstride = n / R;  // W_R^e = tw[e * n / R]
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int l = idx / nb;
        const int j = idx - l * nb;
        const float2 *src = in + (size_t)l * ls;
        float2 *dst = out + (size_t)l * ls;
        const int k = j % Ns;
        const int o = (j / Ns) * Ns * R + k;
        for (int q = 0; q < R; ++q) {
            float2 acc = make_float2(0.f, 0.f);
            for (int t = 0; t < R; ++t) {
                float2 x = src[sk(j + t * nb)];
                if (Ns > 1 && t > 0) {
                    float2 w = __ldg(tw + t * k * twstride);
                    if (inv) w.y = -w.y;
                    x = cmul(x, w);
                }
                float2 w = __ldg(tw + ((t * q) % R) * rstride);
                if (inv) w.y = -w.y;
                acc = cadd(acc, cmul(x, w));
            }
            dst[sk(o + q * Ns)] = acc;
        }
    }
}

// ---- compile-time power-of-two path ----

template <int L, int R, int NS, bool INV>
__device__ __forceinline__ void stage_pow2(const float2 *__restrict__ in, float2 *__restrict__ out, int nlines, int ls,
                                           const float2 *__restrict__ tw) {
    constexpr int NB = L / R;
    constexpr int TWS = L / (NS * R);
    const int total = nlines * NB;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int l = idx / NB;
        const int j = idx % NB;
        const float2 *src = in + l * ls;
        float2 *dst = out + l * ls;
        const int k = j % NS;
        float2 v[R];
#pragma unroll
        for (int t = 0; t < R; ++t) v[t] = src[sk(j + t * NB)];
        if (NS > 1) {
#pragma unroll
            for (int t = 1; t < R; ++t) {
                float2 w = __ldg(tw + t * k * TWS);
                if (INV) w.y = -w.y;
                v[t] = cmul(v[t], w);
            }
        }
        dft_small<R>(v, INV);
        const int o = (j / NS) * NS * R + k;
#pragma unroll
        for (int t = 0; t < R; ++t) dst[sk(o + t * NS)] = v[t];
    }
}

template <int L, int NS, bool INV>
__device__ __forceinline__ float2 *stages_pow2(float2 *a, float2 *b, int nlines, int ls, const float2 *tw) {
    if constexpr (NS >= L) {
        return a;
    } else {
        constexpr int REM = L / NS;
        constexpr int R = pow2_radix(REM);
        stage_pow2<L, R, NS, INV>(a, b, nlines, ls, tw);
        __syncthreads();
        return stages_pow2<L, NS * R, INV>(b, a, nlines, ls, tw);
    }
}

template <bool INV>
__device__ __forceinline__ float2 *fft_pow2_dispatch(int log2n, float2 *a, float2 *b, int nlines, int ls,
                                                     const float2 *tw) {
    switch (log2n) {
        case 1: return stages_pow2<2, 1, INV>(a, b, nlines, ls, tw);
        case 2: return stages_pow2<4, 1, INV>(a, b, nlines, ls, tw);
        case 3: return stages_pow2<8, 1, INV>(a, b, nlines, ls, tw);
        case 4: return stages_pow2<16, 1, INV>(a, b, nlines, ls, tw);
        case 5: return stages_pow2<32, 1, INV>(a, b, nlines, ls, tw);
        case 6: return stages_pow2<64, 1, INV>(a, b, nlines, ls, tw);
        case 7: return stages_pow2<128, 1, INV>(a, b, nlines, ls, tw);
        case 8: return stages_pow2<256, 1, INV>(a, b, nlines, ls, tw);
        case 9: return stages_pow2<512, 1, INV>(a, b, nlines, ls, tw);
        case 10: return stages_pow2<1024, 1, INV>(a, b, nlines, ls, tw);
        case 11: return stages_pow2<2048, 1, INV>(a, b, nlines, ls, tw);
        case 12: return stages_pow2<4096, 1, INV>(a, b, nlines, ls, tw);
        default: return a;
    }
}

// Runs all stages; returns the buffer that holds the result (a or b).
// Must be called by every thread of the CTA (contains __syncthreads).
__device__ __forceinline__ float2 *fft_lines(float2 *a, float2 *b, int nlines, int ls, const FftPlan &p, bool inv) {
    if (p.log2n >= 1 && p.log2n <= 12) {
        return inv ? fft_pow2_dispatch<true>(p.log2n, a, b, nlines, ls, p.tw)
                   : fft_pow2_dispatch<false>(p.log2n, a, b, nlines, ls, p.tw);
    }
    int Ns = 1;
    for (int s = 0; s < p.nstages; ++s) {
        const int R = p.radix[s];
        if (R == 8) stage_fixed<8>(a, b, nlines, ls, p.n, Ns, p.tw, inv);
        else if (R == 4) stage_fixed<4>(a, b, nlines, ls, p.n, Ns, p.tw, inv);
        else if (R == 2) stage_fixed<2>(a, b, nlines, ls, p.n, Ns, p.tw, inv);
        else if (R == 3) stage_fixed<3>(a, b, nlines, ls, p.n, Ns, p.tw, inv);
        else if (R == 5) stage_fixed<5>(a, b, nlines, ls, p.n, Ns, p.tw, inv);
        else if (R == 7) stage_fixed<7>(a, b, nlines, ls, p.n, Ns, p.tw, inv);
        else stage_generic(a, b, nlines, ls, p.n, Ns, R, p.tw, inv);
        __syncthreads();
        float2 *t = a;
        a = b;
        b = t;
        Ns *= R;
    }
    return a;
}

}  // namespace fm
