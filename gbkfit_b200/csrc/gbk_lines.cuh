// Kernels of the 3-D real FFT convolution on the two-factor line transforms
// of gbk_dft.cuh, one instantiation per line length.
//
// The passes move each cube once in and once out; the mixed-radix kernels
// were bound by instruction issue (index arithmetic, three to five trips
// through shared memory per line).  Here a thread's loads, constants and
// addresses are compile-time and a line crosses shared memory once (the fused
// z pass twice), which leaves the passes bound by memory.  On a 320 x 320 x
// 160 grid (66 MB of spectrum), before -> after: x r2c 72 -> 33 us, y lines
// 58 -> 24 us each, z lines with the multiply 104 -> 55 us (198 MB of
// algorithmic traffic: 3.6 TB/s), x c2r 83 -> 29 us; on 128 x 128 x 96 the
// five passes 57 -> 23 us.  16 columns per block make each access a 128-byte
// segment; the spectra the library owns have rows padded to 16 values, so
// that those segments are whole lines.
#pragma once

#include "gbk_dft.cuh"

namespace gbk {

constexpr int FAST_LT = 16;      // columns (128 bytes) or rows per block

// Strided columns: element k of column (o, i) at o * so + i + k * sk, i in
// [0, inner).  A block holds 16 adjacent columns; a thread's DFT elements go
// from global memory to registers, once through shared memory, and back.
// MODE 0: forward, 1: inverse, 2: forward, multiply by spec (same strides)
// times scale, inverse (two exchanges, no spectrum in between).
template<int N1, int N2, int MODE>
__global__ void __launch_bounds__(FAST_LT * (N1 > N2 ? N1 : N2))
fast_lines_kernel(float2* data, int inner, int tiles, long long so, long long sk,
                  const float2* __restrict__ tw, const float2* __restrict__ spec, float scale)
{
    constexpr int n = N1 * N2, T = FAST_LT * (N1 > N2 ? N1 : N2);
    constexpr bool INV = MODE == 1;
    extern __shared__ float2 sm[];          // (N1, N2, 16) exchange, then n twiddles
    float2* s_tw = sm + n * FAST_LT;
    const int o = blockIdx.x / tiles, i0 = (blockIdx.x - o * tiles) * FAST_LT;
    const int l = threadIdx.x % FAST_LT, j = threadIdx.x / FAST_LT;
    const bool in = i0 + l < inner;
    float2* col = data + (long long)o * so + i0 + l;
    for (int i = threadIdx.x; i < n; i += T) s_tw[i] = tw[i];
    if (j < N2 && in) {
        float2 v[N1];
#pragma unroll
        for (int r = 0; r < N1; ++r) v[r] = col[(j + N2 * r) * sk];
        dft<N1, INV>(v);
#pragma unroll
        for (int k = 0; k < N1; ++k) sm[(k * N2 + j) * FAST_LT + l] = v[k];
    }
    __syncthreads();
    if (j < N1 && in) {                     // j is k1 here
        float2 v[N2];
#pragma unroll
        for (int r = 0; r < N2; ++r)
            v[r] = cmul_dir<INV>(sm[(j * N2 + r) * FAST_LT + l], s_tw[j * r]);
        dft<N2, INV>(v);
        if constexpr (MODE != 2) {
#pragma unroll
            for (int k = 0; k < N2; ++k) col[(j + N1 * k) * sk] = v[k];
        } else {
            const float2* sc = spec + (long long)o * so + i0 + l;
#pragma unroll
            for (int k = 0; k < N2; ++k) {
                const float2 w = __ldg(sc + (j + N1 * k) * sk);
                v[k] = make_float2((v[k].x * w.x - v[k].y * w.y) * scale,
                                   (v[k].x * w.y + v[k].y * w.x) * scale);
            }
            dft<N2, true>(v);
            // the elements this thread read
#pragma unroll
            for (int r = 0; r < N2; ++r)
                sm[(j * N2 + r) * FAST_LT + l] = cmul_dir<true>(v[r], s_tw[j * r]);
        }
    }
    if constexpr (MODE == 2) {
        __syncthreads();
        if (j < N2 && in) {
            float2 v[N1];
#pragma unroll
            for (int k = 0; k < N1; ++k) v[k] = sm[(k * N2 + j) * FAST_LT + l];
            dft<N1, true>(v);
#pragma unroll
            for (int r = 0; r < N1; ++r) col[(j + N2 * r) * sk] = v[r];
        }
    }
}

// Rows of the real cube (nx = 2 M even) as M = N1 N2 point complex transforms
// plus the even/odd split into M + 1 bins, at row pitch `pitch` of the
// spectrum.  16 rows per block.
template<int N1, int N2>
__global__ void __launch_bounds__(FAST_LT * (N1 > N2 ? N1 : N2))
fast_r2c_kernel(const float* __restrict__ in, float2* __restrict__ out, int rows, int pitch,
                const float2* __restrict__ tw, const float2* __restrict__ post)
{
    constexpr int M = N1 * N2, T = FAST_LT * (N1 > N2 ? N1 : N2), P2 = N2 + 1;
    extern __shared__ float2 sm[];          // 16 rows of N1 (N2 + 1), then M twiddles
    float2* s_tw = sm + FAST_LT * N1 * P2;
    const long long row0 = (long long)blockIdx.x * FAST_LT;
    for (int i = threadIdx.x; i < M; i += T) s_tw[i] = tw[i];
    if (threadIdx.x < FAST_LT * N2) {
        const int l = threadIdx.x / N2, j = threadIdx.x - l * N2;
        if (row0 + l < rows) {
            const float2* src = reinterpret_cast<const float2*>(in) + (row0 + l) * M + j;
            float2 v[N1];
#pragma unroll
            for (int r = 0; r < N1; ++r) v[r] = src[N2 * r];
            dft<N1, false>(v);
            float2* d = sm + l * N1 * P2 + j;
#pragma unroll
            for (int k = 0; k < N1; ++k) d[k * P2] = v[k];
        }
    }
    __syncthreads();
    {
        const int l = threadIdx.x / N1, k1 = threadIdx.x - l * N1;
        const bool on = l < FAST_LT;
        float2 v[N2];
        if (on) {
            const float2* s = sm + (l * N1 + k1) * P2;
#pragma unroll
            for (int r = 0; r < N2; ++r) v[r] = cmul_dir<false>(s[r], s_tw[k1 * r]);
            dft<N2, false>(v);
        }
        __syncthreads();
        if (on) {
            float2* d = sm + l * M + k1;    // rows of M from here on
#pragma unroll
            for (int k = 0; k < N2; ++k) d[N1 * k] = v[k];
        }
    }
    __syncthreads();
    constexpr int hx = M + 1;
    for (int e = threadIdx.x; e < FAST_LT * hx; e += T) {
        const int l = e / hx, k = e - l * hx;
        if (row0 + l >= rows) break;
        const float2 zk = sm[l * M + (k == M ? 0 : k)];
        const float2 zc = conjf2(sm[l * M + (k == 0 ? 0 : M - k)]);
        const float2 ev = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y + zc.y));
        const float2 od = make_float2(0.5f * (zk.x - zc.x), 0.5f * (zk.y - zc.y));
        // X = E + W^k (-i) O
        out[(row0 + l) * pitch + k] = cadd(ev, cmul(__ldg(post + k), make_float2(od.y, -od.x)));
    }
}

// The inverse of fast_r2c_kernel (unnormalised).
template<int N1, int N2>
__global__ void __launch_bounds__(FAST_LT * (N1 > N2 ? N1 : N2))
fast_c2r_kernel(const float2* __restrict__ in, float* __restrict__ out, int rows, int pitch,
                const float2* __restrict__ tw, const float2* __restrict__ post)
{
    constexpr int M = N1 * N2, T = FAST_LT * (N1 > N2 ? N1 : N2), P2 = N2 + 1;
    extern __shared__ float2 sm[];
    float2* s_tw = sm + FAST_LT * N1 * P2;
    const long long row0 = (long long)blockIdx.x * FAST_LT;
    for (int i = threadIdx.x; i < M; i += T) s_tw[i] = tw[i];
    if (threadIdx.x < FAST_LT * N2) {
        const int l = threadIdx.x / N2, j = threadIdx.x - l * N2;
        if (row0 + l < rows) {
            const float2* src = in + (row0 + l) * pitch;
            float2 v[N1];
#pragma unroll
            for (int r = 0; r < N1; ++r) {
                // Z[k] = (X[k] + conj X[M-k]) + i W^-k (X[k] - conj X[M-k])
                const int k = j + N2 * r;
                const float2 a = src[k], b = conjf2(src[M - k]);
                const float2 s = cadd(a, b), d = csub(a, b);
                const float2 t = cmul_dir<true>(d, __ldg(post + k));
                v[r] = make_float2(s.x - t.y, s.y + t.x);
            }
            dft<N1, true>(v);
            float2* d = sm + l * N1 * P2 + j;
#pragma unroll
            for (int k = 0; k < N1; ++k) d[k * P2] = v[k];
        }
    }
    __syncthreads();
    if (threadIdx.x < FAST_LT * N1) {
        const int l = threadIdx.x / N1, k1 = threadIdx.x - l * N1;
        if (row0 + l < rows) {
            const float2* s = sm + (l * N1 + k1) * P2;
            float2 v[N2];
#pragma unroll
            for (int r = 0; r < N2; ++r) v[r] = cmul_dir<true>(s[r], s_tw[k1 * r]);
            dft<N2, true>(v);
            float2* d = reinterpret_cast<float2*>(out) + (row0 + l) * M + k1;
#pragma unroll
            for (int k = 0; k < N2; ++k) d[N1 * k] = v[k];
        }
    }
}

// ---- the mixed-radix passes at compile-time lengths ------------------------------
// The same passes, twiddles and operations as fft_smem_t (gbk_fft.cuh), so the
// same values bit for bit, with the length, radices and strides known at compile
// time: the index arithmetic of the run-time form, its busiest pipe, folds
// away.  For the callers of the passes (gbkb200_ctx_set_fft), at the lengths
// of the padding rule; 128 x 128 x 96 38 us a convolution, 57 us before.

// factorize(): the p-th radix of n and the product of the radices before it
struct Radices {
    int nr, r[12];
};
__host__ __device__ constexpr Radices radices(int n)
{
    Radices f{0, {}};
    while (n % 8 == 0 && n > 8) { f.r[f.nr++] = 8; n /= 8; }
    while (n % 4 == 0) { f.r[f.nr++] = 4; n /= 4; }
    while (n % 2 == 0) { f.r[f.nr++] = 2; n /= 2; }
    for (int p = 3; p <= 7; p += 2)
        while (n % p == 0) { f.r[f.nr++] = p; n /= p; }
    return f;
}
template<int N, int P>
__host__ __device__ constexpr int radix_stride()
{
    int s = 1;
    for (int p = 0; p < P; ++p) s *= radices(N).r[p];
    return s;
}

template<int N, int P, int L, int SK, int SL, bool ROWS, bool INV>
__device__ __forceinline__ float2* mixed_passes(float2* src, float2* dst, const float2* tw)
{
    if constexpr (P == radices(N).nr) {
        return src;
    } else {
        constexpr int R = radices(N).r[P], Ns = radix_stride<N, P>(), nb = N / R;
        constexpr int twstep = N / (Ns * R);
        for (int u = threadIdx.x; u < nb * L; u += FFT_THREADS) {
            const int j = ROWS ? u % nb : u / L, l = ROWS ? u / nb : u % L;
            const int k = j % Ns;
            float2 v[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float2 x = src[(j + r * nb) * SK + l * SL];
                if (r > 0 && k > 0) {
                    float2 w = tw[r * k * twstep];
                    if (INV) w = conjf2(w);
                    x = cmul(x, w);
                }
                v[r] = x;
            }
            dft_small<R>(v, INV, tw, N);
            const int d0 = j / Ns * (Ns * R) + k;
#pragma unroll
            for (int m = 0; m < R; ++m) dst[(d0 + m * Ns) * SK + l * SL] = v[m];
        }
        __syncthreads();
        return mixed_passes<N, P + 1, L, SK, SL, ROWS, INV>(dst, src, tw);
    }
}

// as lines_kernel (fft.cu)
template<int N, int MODE>
__global__ void __launch_bounds__(FFT_THREADS)
mixed_lines_kernel(float2* data, int inner, int tiles, long long so, long long sk,
                   const float2* __restrict__ tw, const float2* __restrict__ spec, float scale)
{
    constexpr int LT = FAST_LT;
    extern __shared__ float2 sm[];
    float2 *b0 = sm, *b1 = sm + LT * N, *s_tw = sm + 2 * LT * N;
    load_twiddles(s_tw, tw, N);
    const int o = blockIdx.x / tiles, i0 = (blockIdx.x - o * tiles) * LT;
    const long long base = (long long)o * so + i0;
    staged_copy<8>(
        LT * N,
        [&](int e) {
            const int l = e % LT, k = e / LT;
            return (i0 + l < inner) ? data[base + l + k * sk] : make_float2(0.f, 0.f);
        },
        [&](int e, float2 v) { b0[e] = v; });
    __syncthreads();
    float2* res = mixed_passes<N, 0, LT, LT, 1, false, MODE == 1>(b0, b1, s_tw);
    if constexpr (MODE == 2) {
        staged_copy<8>(
            LT * N,
            [&](int e) {
                const int l = e % LT, k = e / LT;
                return (i0 + l < inner) ? spec[base + l + k * sk] : make_float2(0.f, 0.f);
            },
            [&](int e, float2 b) {
                if (i0 + e % LT < inner) {
                    const float2 a = res[e];
                    res[e] = make_float2((a.x * b.x - a.y * b.y) * scale,
                                         (a.x * b.y + a.y * b.x) * scale);
                }
            });
        __syncthreads();
        res = mixed_passes<N, 0, LT, LT, 1, false, true>(res, res == b0 ? b1 : b0, s_tw);
    }
    for (int e = threadIdx.x; e < LT * N; e += FFT_THREADS) {
        const int l = e % LT, k = e / LT;
        if (i0 + l < inner) data[base + l + k * sk] = res[k * LT + l];
    }
}

// as x_r2c_kernel and x_c2r_kernel (fft.cu), even row lengths 2 M
template<int M>
__global__ void __launch_bounds__(FFT_THREADS)
mixed_r2c_kernel(const float* __restrict__ in, float2* __restrict__ out, int rows, int pitch,
                 const float2* __restrict__ tw, const float2* __restrict__ post)
{
    constexpr int L = FAST_LT, hx = M + 1;
    extern __shared__ float2 sm[];
    float2 *b0 = sm, *b1 = sm + L * M, *s_tw = sm + 2 * L * M, *s_post = s_tw + M;
    load_twiddles(s_tw, tw, M);
    load_twiddles(s_post, post, hx);
    const long long row0 = (long long)blockIdx.x * L;
    staged_copy<8>(
        L * M,
        [&](int e) {
            const long long row = row0 + e / M;
            return row < rows ? reinterpret_cast<const float2*>(in)[row * M + e % M]
                              : make_float2(0.f, 0.f);
        },
        [&](int e, float2 v) { b0[e] = v; });
    __syncthreads();
    float2* z = mixed_passes<M, 0, L, 1, M, true, false>(b0, b1, s_tw);
    for (int e = threadIdx.x; e < L * hx; e += FFT_THREADS) {
        const int l = e / hx, k = e - l * hx;
        const long long row = row0 + l;
        if (row >= rows) continue;
        float2 zk = z[l * M + (k == M ? 0 : k)];
        float2 zc = conjf2(z[l * M + (k == 0 ? 0 : M - k)]);
        float2 ev = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y + zc.y));
        float2 od = make_float2(0.5f * (zk.x - zc.x), 0.5f * (zk.y - zc.y));
        float2 t = cmul(s_post[k], make_float2(od.y, -od.x));
        out[row * pitch + k] = cadd(ev, t);
    }
}

template<int M>
__global__ void __launch_bounds__(FFT_THREADS)
mixed_c2r_kernel(const float2* __restrict__ in, float* __restrict__ out, int rows, int pitch,
                 const float2* __restrict__ tw, const float2* __restrict__ post)
{
    constexpr int L = FAST_LT, hx = M + 1;
    extern __shared__ float2 sm[];
    float2 *b0 = sm, *b1 = sm + L * M, *s_tw = sm + 2 * L * M, *s_post = s_tw + M;
    load_twiddles(s_tw, tw, M);
    load_twiddles(s_post, post, hx);
    const long long row0 = (long long)blockIdx.x * L;
    staged_copy<8>(
        L * M,
        [&](int e) {
            const long long row = row0 + e / M;
            return row < rows ? in[row * pitch + e % M] : make_float2(0.f, 0.f);
        },
        [&](int e, float2 v) { b0[e] = v; });
    staged_copy<8>(
        L * M,
        [&](int e) {
            const long long row = row0 + e / M;
            return row < rows ? in[row * pitch + M - e % M] : make_float2(0.f, 0.f);
        },
        [&](int e, float2 v) { b1[e] = v; });
    __syncthreads();
    for (int e = threadIdx.x; e < L * M; e += FFT_THREADS) {
        const int k = e % M;
        const float2 a = b0[e], b = conjf2(b1[e]);
        const float2 s = cadd(a, b), d = csub(a, b);
        const float2 w = conjf2(s_post[k]);
        const float2 t = cmul(w, d);
        b0[e] = make_float2(s.x - t.y, s.y + t.x);
    }
    __syncthreads();
    float2* z = mixed_passes<M, 0, L, 1, M, true, true>(b0, b1, s_tw);
    for (int e = threadIdx.x; e < L * M; e += FFT_THREADS) {
        const long long row = row0 + e / M;
        if (row < rows) reinterpret_cast<float2*>(out)[row * M + e % M] = z[e];
    }
}

// ---- the instantiated lengths ---------------------------------------------------

typedef void (*FastLinesFn)(float2*, int, int, long long, long long, const float2*, const float2*,
                            float);
typedef void (*FastRowsFn)(const float*, float2*, int, int, const float2*, const float2*);
typedef void (*FastRowsInvFn)(const float2*, float*, int, int, const float2*, const float2*);

struct FastLines {
    FastLinesFn fn[3] = {nullptr, nullptr, nullptr};   // by MODE; null: no instantiation
    int threads = 0;
    size_t smem = 0;
};
struct FastRows {
    FastRowsFn fwd = nullptr;
    FastRowsInvFn inv = nullptr;
    int threads = 0;
    size_t smem = 0;
};
FastLines fast_lines(int n);
FastRows fast_rows(int M);
// the mixed-radix passes at compile-time lengths
FastLines mixed_lines(int n);
FastRows mixed_rows(int M);

}  // namespace gbk
