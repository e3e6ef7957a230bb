// Register-resident DFTs of compile-time length, and the two-factor FFT of
// lines of length n = N1 N2 built from them.
//
// A line's transform runs as N2 DFTs of length N1 over elements j + N2 r, the
// twiddles exp(-2 pi i j k1 / n), and N1 DFTs of length N2 giving the
// elements k1 + N1 k2: one exchange through shared memory, with every
// radix, constant and index known at compile time.  The mixed-radix passes of
// gbk_fft.cuh take three to five exchanges for the same lines, with run-time
// index arithmetic in each; they remain for the lengths that no instantiation
// covers.
#pragma once

#include "gbk_fft.cuh"

namespace gbk {

// ---- compile-time cos and sin of 2 pi k / n -------------------------------------

// Taylor series on [0, pi/4]
__host__ __device__ constexpr double ct_sin_q(double x)
{
    double t = x, s = x;
    for (int i = 1; i < 10; ++i) {
        t *= -x * x / ((2 * i) * (2 * i + 1));
        s += t;
    }
    return s;
}
__host__ __device__ constexpr double ct_cos_q(double x)
{
    double t = 1.0, s = 1.0;
    for (int i = 1; i < 10; ++i) {
        t *= -x * x / ((2 * i - 1) * (2 * i));
        s += t;
    }
    return s;
}
__host__ __device__ constexpr double ct_cos(int k, int n)
{
    const double pi = 3.14159265358979323846;
    k %= n;
    if (k < 0) k += n;
    if (2 * k > n) k = n - k;
    double sign = 1.0;
    if (4 * k > n) {            // cos x = -cos(pi - x), pi - x = 2 pi (n - 2 k) / (2 n)
        sign = -1.0;
        k = n - 2 * k;
        n = 2 * n;
    }
    if (8 * k > n) return sign * ct_sin_q(2 * pi * (double)(n - 4 * k) / (4.0 * n));
    return sign * ct_cos_q(2 * pi * (double)k / (double)n);
}
__host__ __device__ constexpr double ct_sin(int k, int n)
{
    // sin x = cos(x - pi / 2)
    return ct_cos(4 * k - n, 4 * n);
}

// A convolution multiplies by a constant c on the way there and on the way
// back.  Rounded to the nearest fp32 both times, the errors add up, and most of the
// constants below lie under their value: a transform there and back lost 3 to
// 6 parts in 1e8 of every frequency.  The inverse takes the fp32 value next to
// c^2 / fp32(c) instead, so that the product is right to half an ulp (lost after
// it: 1.6 parts in 1e8 on average over the line lengths).
__host__ __device__ constexpr float tw_round(double c, bool inv)
{
    const float f = (float)c;
    return inv && f != 0.f ? (float)(c * c / (double)f) : f;
}
template<int R>
struct TwTable {
    float c[R], s[R];
};
template<int R, bool INV>
__host__ __device__ constexpr TwTable<R> make_tw_table()
{
    TwTable<R> t{};
    for (int k = 0; k < R; ++k) {
        t.c[k] = tw_round(ct_cos(k, R), INV);
        t.s[k] = tw_round(ct_sin(k, R), INV);
    }
    return t;
}

// x * exp(-+ 2 pi i e / R), e and R compile-time constants after unrolling
template<int R, bool INV>
__device__ __forceinline__ float2 tw_mul(float2 x, int e)
{
    constexpr TwTable<R> T = make_tw_table<R, INV>();
    e %= R;
    if (e == 0) return x;
    if (4 * e == R) return mul_mi(x, INV);
    if (2 * e == R) return make_float2(-x.x, -x.y);
    if (4 * e == 3 * R) return mul_mi(x, !INV);
    const float h = 0.70710678118654752f;
    if (8 * e == R)
        return INV ? make_float2(h * (x.x - x.y), h * (x.x + x.y))
                   : make_float2(h * (x.x + x.y), h * (x.y - x.x));
    if (8 * e == 3 * R)
        return INV ? make_float2(-h * (x.x + x.y), h * (x.x - x.y))
                   : make_float2(h * (x.y - x.x), -h * (x.x + x.y));
    const float c = T.c[e], s = INV ? T.s[e] : -T.s[e];
    return make_float2(x.x * c - x.y * s, x.x * s + x.y * c);
}

// ---- DFTs of compile-time length, in natural order ------------------------------

template<int R>
struct Split { static constexpr int A = 0; };        // prime: no split
template<> struct Split<6> { static constexpr int A = 2; };
template<> struct Split<8> { static constexpr int A = 2; };
template<> struct Split<9> { static constexpr int A = 3; };
template<> struct Split<10> { static constexpr int A = 2; };
template<> struct Split<12> { static constexpr int A = 4; };
template<> struct Split<14> { static constexpr int A = 2; };
template<> struct Split<15> { static constexpr int A = 3; };
template<> struct Split<16> { static constexpr int A = 4; };
template<> struct Split<18> { static constexpr int A = 2; };
template<> struct Split<20> { static constexpr int A = 4; };
template<> struct Split<21> { static constexpr int A = 3; };
template<> struct Split<22> { static constexpr int A = 2; };
template<> struct Split<24> { static constexpr int A = 4; };

template<int R, bool INV>
__device__ __forceinline__ void dft(float2 (&v)[R])
{
    if constexpr (R == 1) {
    } else if constexpr (R == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (R == 4) {
        const float2 s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
        const float2 s13 = cadd(v[1], v[3]), d13 = mul_mi(csub(v[1], v[3]), INV);
        v[0] = cadd(s02, s13);
        v[2] = csub(s02, s13);
        v[1] = cadd(d02, d13);
        v[3] = csub(d02, d13);
    } else if constexpr (Split<R>::A > 0) {
        constexpr int A = Split<R>::A, B = R / A;
#pragma unroll
        for (int b = 0; b < B; ++b) {
            float2 t[A];
#pragma unroll
            for (int a = 0; a < A; ++a) t[a] = v[b + B * a];
            dft<A, INV>(t);
#pragma unroll
            for (int k = 0; k < A; ++k) v[b + B * k] = tw_mul<R, INV>(t[k], b * k);
        }
        float2 o[R];
#pragma unroll
        for (int k = 0; k < A; ++k) {
            float2 u[B];
#pragma unroll
            for (int b = 0; b < B; ++b) u[b] = v[b + B * k];
            dft<B, INV>(u);
#pragma unroll
            for (int q = 0; q < B; ++q) o[k + A * q] = u[q];
        }
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = o[i];
    } else {
        // odd prime: the pairs v[j] +- v[R - j] against the cosines and sines
        constexpr TwTable<R> T = make_tw_table<R, INV>();
        constexpr int H = (R - 1) / 2;
        float2 sp[H], dm[H];
        float2 sum = v[0];
#pragma unroll
        for (int j = 0; j < H; ++j) {
            sp[j] = cadd(v[j + 1], v[R - 1 - j]);
            dm[j] = csub(v[j + 1], v[R - 1 - j]);
            sum = cadd(sum, sp[j]);
        }
        float2 o[R];
        o[0] = sum;
#pragma unroll
        for (int m = 1; m <= H; ++m) {
            float2 p = v[0], q = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 1; j <= H; ++j) {
                const float c = T.c[(j * m) % R], s = T.s[(j * m) % R];
                p.x += c * sp[j - 1].x;
                p.y += c * sp[j - 1].y;
                q.x += s * dm[j - 1].x;
                q.y += s * dm[j - 1].y;
            }
            // forward: X[m] = p - i q, X[R - m] = p + i q
            const float2 iq = INV ? make_float2(-q.y, q.x) : make_float2(q.y, -q.x);
            o[m] = cadd(p, iq);
            o[R - m] = csub(p, iq);
        }
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = o[i];
    }
}

// x * w or x * conj(w)
template<bool CONJ>
__device__ __forceinline__ float2 cmul_dir(float2 x, float2 w)
{
    return CONJ ? make_float2(x.x * w.x + x.y * w.y, x.y * w.x - x.x * w.y)
                : make_float2(x.x * w.x - x.y * w.y, x.x * w.y + x.y * w.x);
}

}  // namespace gbk
