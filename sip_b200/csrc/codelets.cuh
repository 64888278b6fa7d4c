// Register-resident DFT codelets and complex helpers for the sm_100a FFT kernels.
//
// Sign convention (the reference's, core/fft/fftcore/dft_core.cpp:88-97):
// FWD == true computes y[k] = sum_j a[j] * exp(-2*pi*i*j*k/R),
// FWD == false uses exp(+2*pi*i*j*k/R).  No scaling.
//
// Constants are evaluated at compile time in double from Taylor series
// (ccos/csin below) so no table or math-library call is needed in the
// butterflies; every codelet is fully unrolled into FMAs on registers.
//
// Every codelet runs on one transform (float2) or on two at once (cpx2): the
// kernels are bound by instruction issue, and sm_100's packed FP32 add,
// multiply and FMA do two transforms' arithmetic in one issue slot at the
// FP32 pipe's full rate (measured: 16 FFMA and 8 packed FMA take the same
// pipe time in half the slots).  Both run the same operations in the same
// order, so their results agree bit for bit, but for the composite radices (CompPrime).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// Codelets are host-callable as well so that a CPU test can check every radix
// against a direct DFT without a GPU.
#define SIPFFT_HD __host__ __device__ __forceinline__

namespace sipfft {

// ---------------------------------------------------------------- packed FP32 pairs
SIPFFT_HD float2 add2(float2 a, float2 b)
{
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
    return __fadd2_rn(a, b);
#else
    return make_float2(a.x + b.x, a.y + b.y);
#endif
}
SIPFFT_HD float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
SIPFFT_HD float2 sub2(float2 a, float2 b) { return add2(a, neg2(b)); }
SIPFFT_HD float2 mul2(float2 a, float2 b)
{
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
    return __fmul2_rn(a, b);
#else
    return make_float2(a.x * b.x, a.y * b.y);
#endif
}
SIPFFT_HD float2 fma2(float2 a, float2 b, float2 c)
{
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
    return __ffma2_rn(a, b, c);
#else
    return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
#endif
}
SIPFFT_HD float2 both(float s) { return make_float2(s, s); }

// One complex value of two transforms: re = (re 0, re 1), im = (im 0, im 1).
struct cpx2 {
    float2 re, im;
};
// interleaved complex values of the two transforms <-> cpx2
SIPFFT_HD cpx2 pair_of(float2 a, float2 b) { return {make_float2(a.x, b.x), make_float2(a.y, b.y)}; }
SIPFFT_HD float2 first_of(cpx2 v) { return make_float2(v.re.x, v.im.x); }
SIPFFT_HD float2 second_of(cpx2 v) { return make_float2(v.re.y, v.im.y); }

// ---------------------------------------------------------------- complex helpers
SIPFFT_HD float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
SIPFFT_HD float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
SIPFFT_HD float2 cmul(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// The product of the roots of unity 1 + l and 1 + h, given without their one, l of a
// small angle: values round at their own size and the smallest are added first, so that
// the product carries little more than its own rounding (two rounded roots multiplied:
// three roundings).
SIPFFT_HD float2 root_product(float2 l, float2 h)
{
    const float re = l.x + fmaf(l.x, h.x, -l.y * h.y), im = l.y + fmaf(l.x, h.y, l.y * h.x);
    return make_float2(1.f + (h.x + re), h.y + im);
}
SIPFFT_HD float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
SIPFFT_HD float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
SIPFFT_HD float2 cneg(float2 a) { return neg2(a); }
// acc + s * a, s real
SIPFFT_HD float2 caxpy(float s, float2 a, float2 acc) { return make_float2(fmaf(s, a.x, acc.x), fmaf(s, a.y, acc.y)); }
// acc + i s * a, s real
SIPFFT_HD float2 caxpy_i(float s, float2 a, float2 acc) { return make_float2(fmaf(-s, a.y, acc.x), fmaf(s, a.x, acc.y)); }
SIPFFT_HD float2 mul_i(float2 a) { return make_float2(-a.y, a.x); }
// a + i b, a - i b
SIPFFT_HD float2 cadd_i(float2 a, float2 b) { return make_float2(a.x - b.y, a.y + b.x); }
SIPFFT_HD float2 csub_i(float2 a, float2 b) { return make_float2(a.x + b.y, a.y - b.x); }

SIPFFT_HD cpx2 cadd(cpx2 a, cpx2 b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
SIPFFT_HD cpx2 csub(cpx2 a, cpx2 b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
SIPFFT_HD cpx2 cmul(cpx2 a, cpx2 b)
{
    return {fma2(a.re, b.re, neg2(mul2(a.im, b.im))), fma2(a.re, b.im, mul2(a.im, b.re))};
}
SIPFFT_HD cpx2 cmul(cpx2 a, float2 w) { return cmul(a, cpx2{both(w.x), both(w.y)}); }
SIPFFT_HD cpx2 cscale(cpx2 a, float s) { return {mul2(a.re, both(s)), mul2(a.im, both(s))}; }
SIPFFT_HD cpx2 cconj(cpx2 a) { return {a.re, neg2(a.im)}; }
SIPFFT_HD cpx2 cneg(cpx2 a) { return {neg2(a.re), neg2(a.im)}; }
SIPFFT_HD cpx2 caxpy(float s, cpx2 a, cpx2 acc) { return {fma2(both(s), a.re, acc.re), fma2(both(s), a.im, acc.im)}; }
SIPFFT_HD cpx2 caxpy_i(float s, cpx2 a, cpx2 acc) { return {fma2(both(-s), a.im, acc.re), fma2(both(s), a.re, acc.im)}; }
SIPFFT_HD cpx2 mul_i(cpx2 a) { return {neg2(a.im), a.re}; }
SIPFFT_HD cpx2 cadd_i(cpx2 a, cpx2 b) { return {sub2(a.re, b.im), add2(a.im, b.re)}; }
SIPFFT_HD cpx2 csub_i(cpx2 a, cpx2 b) { return {add2(a.re, b.im), sub2(a.im, b.re)}; }

// exp(sign * i * theta) with the direction's sign applied to a table entry
// that holds exp(-i * theta).
template <bool FWD, class V>
SIPFFT_HD V dir(V w)
{
    return FWD ? w : cconj(w);
}
// a + w b and a - w b for a quarter turn w = -i (FWD) or +i
template <bool FWD, class V>
SIPFFT_HD V add_quarter(V a, V b)
{
    return FWD ? csub_i(a, b) : cadd_i(a, b);
}
template <bool FWD, class V>
SIPFFT_HD V sub_quarter(V a, V b)
{
    return FWD ? cadd_i(a, b) : csub_i(a, b);
}

// ---------------------------------------------------------------- compile-time trig
constexpr double kPi = 3.141592653589793238462643383279502884;

constexpr double reduce_angle(double x)
{
    // bring x into [-pi, pi]
    while (x > kPi) x -= 2.0 * kPi;
    while (x < -kPi) x += 2.0 * kPi;
    return x;
}
constexpr double ccos(double x)
{
    x = reduce_angle(x);
    double term = 1.0, sum = 1.0;
    for (int k = 1; k < 30; k++) {
        term *= -x * x / ((2.0 * k - 1.0) * (2.0 * k));
        sum += term;
    }
    return sum;
}
constexpr double csin(double x)
{
    x = reduce_angle(x);
    double term = x, sum = x;
    for (int k = 1; k < 30; k++) {
        term *= -x * x / ((2.0 * k) * (2.0 * k + 1.0));
        sum += term;
    }
    return sum;
}
// cos / sin of 2*pi*j/R
template <int R, int J>
struct Root {
    static constexpr float c = static_cast<float>(ccos(2.0 * kPi * (J % R) / R));
    static constexpr float s = static_cast<float>(csin(2.0 * kPi * (J % R) / R));
};

// e + w a and e - w a, w = exp(-+ 2*pi*i*J/R) = c + i s, in six FMAs: with |c| >= |s|
// as e +- c u, u = a + i (s/c) a, else as e +- s u, u = (c/s) a + i a (two
// roundings a component instead of the three of product, sum and butterfly).
template <int R, int J, bool FWD, class V>
SIPFFT_HD void rot_butterfly(V e, V a, V &plus, V &minus)
{
    constexpr double t = 2.0 * kPi * (J % R) / R;
    constexpr double c = ccos(t), s = FWD ? -csin(t) : csin(t);
    constexpr bool wide = (c < 0 ? -c : c) >= (s < 0 ? -s : s);
    V u;
    if constexpr (wide)
        u = caxpy_i(static_cast<float>(s / c), a, a);
    else
        u = caxpy(static_cast<float>(c / s), a, mul_i(a));
    constexpr float m = static_cast<float>(wide ? c : s);
    plus = caxpy(m, u, e);
    minus = caxpy(-m, u, e);
}

// multiply a by exp(-+ 2*pi*i*J/R) with the trivial angles special-cased
template <int R, int J, bool FWD, class V>
SIPFFT_HD V rot(V a)
{
    constexpr int j = ((J % R) + R) % R;
    if constexpr (j == 0) {
        return a;
    } else if constexpr (4 * j == R) {
        return FWD ? cneg(mul_i(a)) : mul_i(a);
    } else if constexpr (2 * j == R) {
        return cneg(a);
    } else if constexpr (4 * j == 3 * R) {
        return FWD ? mul_i(a) : cneg(mul_i(a));
    } else {
        constexpr float c = Root<R, j>::c;
        constexpr float s = FWD ? -Root<R, j>::s : Root<R, j>::s;  // exp(+-i theta) = c + i*s
        return cmul(a, make_float2(c, s));
    }
}

// ---------------------------------------------------------------- power-of-two codelets
// Recursive radix-2 decimation in time on an array held in registers.
template <int R, bool FWD>
struct Pow2 {
    template <class V>
    SIPFFT_HD static void run(V *a)
    {
        V e[R / 2], o[R / 2];
#pragma unroll
        for (int i = 0; i < R / 2; i++) {
            e[i] = a[2 * i];
            o[i] = a[2 * i + 1];
        }
        Pow2<R / 2, FWD>::run(e);
        Pow2<R / 2, FWD>::run(o);
        combine<0>(a, e, o);
    }
    template <int K, class V>
    SIPFFT_HD static void combine(V *a, const V *e, const V *o)
    {
        if constexpr (K < R / 2) {
            if constexpr (4 * K == R) {
                a[K] = add_quarter<FWD>(e[K], o[K]);
                a[K + R / 2] = sub_quarter<FWD>(e[K], o[K]);
            } else if constexpr (K == 0) {
                a[0] = cadd(e[0], o[0]);
                a[R / 2] = csub(e[0], o[0]);
            } else {
                rot_butterfly<R, K, FWD>(e[K], o[K], a[K], a[K + R / 2]);
            }
            combine<K + 1>(a, e, o);
        }
    }
};
template <bool FWD>
struct Pow2<1, FWD> {
    template <class V>
    SIPFFT_HD static void run(V *)
    {
    }
};
template <bool FWD>
struct Pow2<2, FWD> {
    template <class V>
    SIPFFT_HD static void run(V *a)
    {
        const V t = a[1];
        a[1] = csub(a[0], t);
        a[0] = cadd(a[0], t);
    }
};
template <bool FWD>
struct Pow2<4, FWD> {
    template <class V>
    SIPFFT_HD static void run(V *a)
    {
        const V t0 = cadd(a[0], a[2]), t1 = csub(a[0], a[2]);
        const V t2 = cadd(a[1], a[3]), t3 = csub(a[1], a[3]);
        a[0] = cadd(t0, t2);
        a[2] = csub(t0, t2);
        a[1] = add_quarter<FWD>(t1, t3);
        a[3] = sub_quarter<FWD>(t1, t3);
    }
};

// ---------------------------------------------------------------- odd codelets
// Generic odd-length DFT using the conjugate-pair symmetry:
// for m = 1..H: y[m], y[R-m] = B_m -+ i*D_m with
// B_m = a0 + sum_k cos(2 pi k m / R) (a_k + a_{R-k}),
// D_m = sum_k sin(2 pi k m / R) (a_k - a_{R-k}).
template <int R, bool FWD>
struct Odd {
    static constexpr int H = (R - 1) / 2;
    template <class V>
    SIPFFT_HD static void run(V *a)
    {
        V tp[H], tm[H];
#pragma unroll
        for (int k = 1; k <= H; k++) {
            tp[k - 1] = cadd(a[k], a[R - k]);
            tm[k - 1] = csub(a[k], a[R - k]);
        }
        V y0 = a[0];
#pragma unroll
        for (int k = 0; k < H; k++) y0 = cadd(y0, tp[k]);
        V out[R];
        out[0] = y0;
        terms<1>(a[0], tp, tm, out);
#pragma unroll
        for (int i = 0; i < R; i++) a[i] = out[i];
    }
    template <int M, class V>
    SIPFFT_HD static void terms(V a0, const V *tp, const V *tm, V *out)
    {
        if constexpr (M <= H) {
            V b = a0, d = cscale(tm[0], Root<R, M % R>::s);
            accum<M, 1>(b, d, tp, tm);
            // forward: y_M = b - i d ; y_{R-M} = b + i d
            out[M] = add_quarter<FWD>(b, d);
            out[R - M] = sub_quarter<FWD>(b, d);
            terms<M + 1>(a0, tp, tm, out);
        }
    }
    template <int M, int K, class V>
    SIPFFT_HD static void accum(V &b, V &d, const V *tp, const V *tm)
    {
        if constexpr (K <= H) {
            b = caxpy(Root<R, (K * M) % R>::c, tp[K - 1], b);
            if constexpr (K > 1) d = caxpy(Root<R, (K * M) % R>::s, tm[K - 1], d);
            accum<M, K + 1>(b, d, tp, tm);
        }
    }
};

template <bool FWD>
struct Odd<3, FWD> {
    template <class V>
    SIPFFT_HD static void run(V *a)
    {
        constexpr float h = 0.86602540378443864676f;  // sqrt(3)/2
        const V s = cadd(a[1], a[2]);
        const V d = csub(a[1], a[2]);
        const V m = caxpy(-0.5f, s, a[0]);
        a[0] = cadd(a[0], s);
        // forward: y1 = m - i h d, y2 = m + i h d
        a[1] = caxpy_i(FWD ? -h : h, d, m);
        a[2] = caxpy_i(FWD ? h : -h, d, m);
    }
};

// ---------------------------------------------------------------- dispatch
template <int R>
constexpr bool is_pow2() { return R > 0 && (R & (R - 1)) == 0; }

constexpr int smallest_prime_factor(int r)
{
    for (int p = 2; p * p <= r; p++)
        if (r % p == 0) return p;
    return r;
}
// split of a composite radix R = A * B used by Comp: the power-of-two part
// first for even R, else the smallest prime factor
constexpr int comp_first(int r)
{
    if (r % 2 == 0) {
        int a = 1;
        while (r % (2 * a) == 0) a *= 2;
        return a;
    }
    return smallest_prime_factor(r);
}

template <int R, bool FWD, class V>
SIPFFT_HD void dft(V *a);

constexpr int common_divisor(int a, int b) { return b == 0 ? a : common_divisor(b, a % b); }
// x with x = 1 (mod a) and x = 0 (mod b), a and b coprime
constexpr int crt_unit(int a, int b)
{
    int x = b;
    while (x % a != 1) x += b;
    return x;
}

// Composite radix R = A*B in registers (Cooley-Tukey, decimation in time):
// B-point DFTs over the A interleaved sub-sequences, twiddles W_R^(n1*k2),
// then A-point DFTs; output index k = k2 + B*k1.
template <int A, int B, bool FWD>
struct Comp {
    static constexpr int R = A * B;
    template <class V>
    SIPFFT_HD static void run(V *a)
    {
        V y[A][B];
#pragma unroll
        for (int n1 = 0; n1 < A; n1++) {
#pragma unroll
            for (int n2 = 0; n2 < B; n2++) y[n1][n2] = a[n1 + A * n2];
            dft<B, FWD>(y[n1]);
        }
        twiddle<1, 1>(y);
#pragma unroll
        for (int k2 = 0; k2 < B; k2++) {
            V z[A];
#pragma unroll
            for (int n1 = 0; n1 < A; n1++) z[n1] = y[n1][k2];
            dft<A, FWD>(z);
#pragma unroll
            for (int k1 = 0; k1 < A; k1++) a[k2 + B * k1] = z[k1];
        }
    }
    template <int N1, int K2, class V>
    SIPFFT_HD static void twiddle(V (&y)[A][B])
    {
        if constexpr (N1 < A) {
            if constexpr (K2 < B) {
                y[N1][K2] = rot<R, N1 * K2, FWD>(y[N1][K2]);
                twiddle<N1, K2 + 1>(y);
            } else {
                twiddle<N1 + 1, 1>(y);
            }
        }
    }
};

// The same of coprime A and B (every composite radix of the kernels) on two transforms, in the
// prime-factor order: input B n1 + A n2 and output k = k1 (mod A) = k2 (mod B) need no twiddles.
// The pair tiles take larger radices than the one-transform tiles, and the twiddles' 2 to 8
// products would round more often (relative rms error of a radix, with them -> without:
// 6 4.5e-8 -> 3.9e-8, 10 5.7e-8 -> 5.1e-8, 12 5.2e-8 -> 4.8e-8, 14 6.0e-8 -> 5.5e-8,
// 15 6.3e-8 -> 5.7e-8; 1000-point rows 1.22e-7 -> 1.10e-7).  (The one-transform kernels, which
// hold every radix at a fixed register bound, lose 3 to 8 % in this order: r2c 9216 x 455
// 36.6 -> 38.2 us.)
template <int A, int B, bool FWD>
struct CompPrime {
    static constexpr int R = A * B, K1 = crt_unit(A, B), K2 = crt_unit(B, A);
    SIPFFT_HD static void run(cpx2 *a)
    {
        cpx2 y[A][B];
#pragma unroll
        for (int n1 = 0; n1 < A; n1++) {
#pragma unroll
            for (int n2 = 0; n2 < B; n2++) y[n1][n2] = a[(B * n1 + A * n2) % R];
            dft<B, FWD>(y[n1]);
        }
#pragma unroll
        for (int k2 = 0; k2 < B; k2++) {
            cpx2 z[A];
#pragma unroll
            for (int n1 = 0; n1 < A; n1++) z[n1] = y[n1][k2];
            dft<A, FWD>(z);
#pragma unroll
            for (int k1 = 0; k1 < A; k1++) a[(k1 * K1 + k2 * K2) % R] = z[k1];
        }
    }
};

template <int R, bool FWD, class V>
SIPFFT_HD void dft(V *a)
{
    if constexpr (is_pow2<R>()) {
        Pow2<R, FWD>::run(a);
    } else if constexpr (R % 2 == 0 || (smallest_prime_factor(R) != R && R > 13)) {
        constexpr int A = comp_first(R), B = R / A;
        if constexpr (sizeof(V) == sizeof(cpx2) && common_divisor(A, B) == 1)
            CompPrime<A, B, FWD>::run(a);
        else
            Comp<A, B, FWD>::run(a);
    } else {
        Odd<R, FWD>::run(a);
    }
}

}  // namespace sipfft
