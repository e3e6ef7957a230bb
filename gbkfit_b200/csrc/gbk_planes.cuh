// Plane-wise FFT convolution of the batched evaluator, for PSFs that are not
// separable: the model kernel (gbk_batched.cuh) applies the LSF in registers
// and writes the LSF-convolved planes with their nonzero-column masks; each
// plane is then convolved with the PSF image by a 2-D real FFT in three
// passes on the two-factor line transforms of gbk_dft.cuh:
//   kp_rows   nonzero rows, 16 per block, two per complex transform;
//   kp_cols   16 kx columns of a plane per block: forward y transform,
//             multiply by the PSF's spectrum, inverse; only the crop's rows
//             are stored;
//   kp_resid  16 crop rows per block: inverse, residual, sum of r^2.
//
// The 3-D form (K1-K5 of batched.cu) transforms z as well, for an LSF of
// ten-odd taps: two more passes over a cube that left the L2, and run-time
// radices throughout.  64 sets of 128 x 128 x 96 with a Moffat PSF in waves of
// 16: 6420 us in the 3-D form, 920 us here (model and LSF 130, rows 153, columns
// 345, residual 275), bound by instruction issue (62-76 % of cycles, about 75
// instructions per spectrum value and pass).  The lines and the residual are
// those of the 3-D form, operation by operation, and r^2 is summed in fp64 (with
// ex2.approx lines and a residual weight made at creation 865 us, and chi^2 1.79e-7
// from its 64-bit value over 48 drawn batches, now 1.48e-7, the 3-D form 1.55e-7).
// Lines of 16 N1 points, so that a thread's elements lie 16 rows or columns apart and
// masks, addresses and zero row groups fold into compile-time offsets (with other
// factors the columns took 366-434 us), and two real rows per transform instead of
// the even/odd split (rows and residual 209 and 299 us with it, then 153 and 245).
#pragma once

#include "gbk_batched.cuh"
#include "gbk_dft.cuh"

namespace gbk {

constexpr int KP_L = 16;              // rows, or columns (128 bytes), per block
constexpr int KP_MAX_W = 384;         // longest window: 24 row groups, 12 chunks

struct PlaneArgs {
    int Nx, Ny, Nz, Wx, Wy, nch, pitch;    // pitch: of the planes (floats)
    int vec;                               // Nx % 4 == 0, data and model on 16 bytes: float4 rows
    int hxp, ngw, set0;                    // padded spectrum columns; window row groups
    const float* mplanes;                  // (sets, Nz, Wy, pitch)
    const int* xrt;                        // (sets, Nz, Wy, nch)
    float2* work;                          // (sets, Nz, hxp / 16, 16 ngw, 16)
    float2* conv;                          // (sets, Nz, Ny, hxp): crop rows of the convolution
    unsigned char* flags;                  // (sets, Nz, 32): row group holds a nonzero value
    // spec: (hxp / 16, Py, 16), of the PSF image shifted so that the crop starts
    // at the origin, scaled by 1 / (Px Py)
    const float2 *twx, *twy, *spec;
    const float *obs, *err, *msk;          // err, msk: may be null
    float weight;
    float* model;                          // optional (nsets, Nz, Ny, Nx)
    double* partials;                      // (nsets, Nz, ceil(Ny / 16))
};

// the plane's nonzero row groups as a bit mask (whole warps)
__device__ __forceinline__ unsigned plane_groups(const PlaneArgs& P, long long plane)
{
    const int lane = threadIdx.x & 31;
    const bool f = lane < P.ngw && P.flags[plane * 32 + lane] != 0;
    return __ballot_sync(0xffffffffu, f);
}

constexpr int KP_P = KP_L / 2;        // row pairs per block
// threads of the row kernels: whole warps (their sums shuffle across the warp)
__host__ __device__ constexpr int kp_threads(int n1)
{
    return (KP_P * (n1 > 16 ? n1 : 16) + 31) / 32 * 32;
}

// Rows [16 g, 16 g + 16) of a plane, two real rows as the real and imaginary
// part of one n = 16 N1 point transform:
//   X1[k] = (Z[k] + conj Z[n-k]) / 2,  X2[k] = (Z[k] - conj Z[n-k]) / (2 i).
// The planes hold values only in 4-column groups with a set mask bit (every
// column of those is written); a thread's columns lie 16 apart, so that the
// mask word of an element and its bit are known at compile time up to the lane.
template<int N1>
__global__ void __launch_bounds__(kp_threads(N1)) kp_rows(PlaneArgs P)
{
    constexpr int N2 = 16, n = N1 * N2, T = kp_threads(N1), P2 = N2 + 1;
    extern __shared__ float2 sm[];          // 8 pairs of N1 P2, then n twiddles
    float2* s_tw = sm + KP_P * N1 * P2;
    __shared__ int s_mask[KP_L * (KP_MAX_W / 32)];
    const int y0 = blockIdx.x * KP_L, rows = min(KP_L, P.Wy - y0);
    const long long plane = (long long)blockIdx.z * P.Nz + blockIdx.y;
    const int* xr = P.xrt + (plane * P.Wy + y0) * P.nch;
    int any = 0;
    for (int i = threadIdx.x; i < KP_L * P.nch; i += T) {
        const int m = i < rows * P.nch ? xr[i] : 0;     // rows past the window: zeros
        s_mask[i] = m;
        any |= m;
    }
    for (int i = threadIdx.x; i < n; i += T) s_tw[i] = P.twx[i];
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) P.flags[plane * 32 + blockIdx.x] = any != 0;
    if (!any) return;                       // whole block: the columns pass reads zeros
    const int p = threadIdx.x / KP_L, c = threadIdx.x % KP_L;
    if (p < KP_P) {
        const float* src = P.mplanes + (plane * P.Wy + y0 + 2 * p) * P.pitch + c;
        const int* m0 = s_mask + 2 * p * P.nch;
        const int* m1 = m0 + P.nch;
        float2 v[N1];
#pragma unroll
        for (int r = 0; r < N1; ++r) {
            // column c + 16 r: word r / 2, bit group c / 4 + 4 (r & 1)
            const unsigned g = 0xfu << (4 * (c >> 2) + 16 * (r & 1));
            const bool in = r / 2 < P.nch;
            v[r] = make_float2(0.f, 0.f);
            if (in && ((unsigned)m0[r / 2] & g)) v[r].x = __ldg(src + N2 * r);
            if (in && ((unsigned)m1[r / 2] & g)) v[r].y = __ldg(src + P.pitch + N2 * r);
        }
        dft<N1, false>(v);
        float2* d = sm + p * N1 * P2 + c;
#pragma unroll
        for (int k = 0; k < N1; ++k) d[k * P2] = v[k];
    }
    __syncthreads();
    {
        const int q = threadIdx.x / N1, k1 = threadIdx.x - q * N1;
        float2 v[N2];
        if (q < KP_P) {
            const float2* s = sm + (q * N1 + k1) * P2;
#pragma unroll
            for (int r = 0; r < N2; ++r) v[r] = cmul_dir<false>(s[r], s_tw[k1 * r]);
            dft<N2, false>(v);
        }
        __syncthreads();
        if (q < KP_P) {
            float2* d = sm + q * n + k1;    // transforms of n from here on
#pragma unroll
            for (int k = 0; k < N2; ++k) d[N1 * k] = v[k];
        }
    }
    __syncthreads();
    if (p < KP_P) {
        const int tile = KP_L * KP_L * P.ngw;           // a tile of 16 columns
        float2* out = P.work + plane * (P.hxp / KP_L) * tile + (y0 + 2 * p) * KP_L + c;
        const float2* z = sm + p * n;
#pragma unroll
        for (int t = 0; t <= n / 2 / KP_L; ++t) {
            const int k = KP_L * t + c;
            if (k > n / 2) break;
            const float2 a = z[k], b = z[k == 0 ? 0 : n - k];
            out[t * tile] = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
            out[t * tile + KP_L] = make_float2(0.5f * (a.y + b.y), 0.5f * (b.x - a.x));
        }
    }
}

// 16 columns of a plane's spectrum: y transform of n = 16 N1 points (zero
// beyond the window and in zero row groups), multiply, inverse; the crop's
// rows, the first Ny, are stored.  A thread's first elements lie 16 rows apart,
// one per row group, so that the groups' tests are uniform, and every address
// but the last stores' is an immediate offset.
template<int N1>
__global__ void __launch_bounds__(KP_L * (N1 > 16 ? N1 : 16)) kp_cols(PlaneArgs P, int hx)
{
    constexpr int N2 = 16, n = N1 * N2, T = KP_L * (N1 > N2 ? N1 : N2);
    extern __shared__ float2 sm[];          // (N1, 16, 16) exchange, then n twiddles
    float2* s_tw = sm + n * KP_L;
    const long long plane = (long long)blockIdx.z * P.Nz + blockIdx.y;
    const unsigned groups = plane_groups(P, plane);
    if (groups == 0u) return;               // whole block: an empty plane
    const int l = threadIdx.x % KP_L, j = threadIdx.x / KP_L;
    const bool in = blockIdx.x * KP_L + l < hx;
    for (int i = threadIdx.x; i < n; i += T) s_tw[i] = P.twy[i];
    if (j < N2 && in) {
        const float2* src = P.work + (plane * gridDim.x + blockIdx.x) * (KP_L * KP_L * P.ngw) +
                            j * KP_L + l;
        float2 v[N1];
#pragma unroll
        for (int r = 0; r < N1; ++r)
            v[r] = (groups >> r) & 1u ? src[r * N2 * KP_L] : make_float2(0.f, 0.f);
        dft<N1, false>(v);
#pragma unroll
        for (int k = 0; k < N1; ++k) sm[(k * N2 + j) * KP_L + l] = v[k];
    }
    __syncthreads();
    if (j < N1 && in) {                     // j is k1 here
        const float2* sc = P.spec + (blockIdx.x * n + j) * KP_L + l;
        float2 v[N2], w[N2];
#pragma unroll
        for (int k = 0; k < N2; ++k) w[k] = __ldg(sc + N1 * k * KP_L);
#pragma unroll
        for (int r = 0; r < N2; ++r) v[r] = cmul_dir<false>(sm[(j * N2 + r) * KP_L + l], s_tw[j * r]);
        dft<N2, false>(v);
#pragma unroll
        for (int k = 0; k < N2; ++k)
            v[k] = make_float2(v[k].x * w[k].x - v[k].y * w[k].y, v[k].x * w[k].y + v[k].y * w[k].x);
        dft<N2, true>(v);
#pragma unroll
        for (int r = 0; r < N2; ++r)
            sm[(j * N2 + r) * KP_L + l] = cmul_dir<true>(v[r], s_tw[j * r]);
    }
    __syncthreads();
    if (j < N2 && in) {
        float2 v[N1];
#pragma unroll
        for (int k = 0; k < N1; ++k) v[k] = sm[(k * N2 + j) * KP_L + l];
        dft<N1, true>(v);
        float2* dst = P.conv + (plane * P.Ny + j) * P.hxp + blockIdx.x * KP_L + l;
        const int step = N2 * P.hxp;
#pragma unroll
        for (int r = 0; r < N1; ++r)
            if (j + N2 * r < P.Ny) dst[r * step] = v[r];
    }
}

// Crop rows [16 g, 16 g + 16) of a plane: the inverse of kp_rows (Z = X1 + i X2,
// conj X1 + i conj X2 beyond n / 2), the first Nx columns, the residual
// (objective.hpp:7-31) and the block's sum of r^2.  Error and mask are read here,
// with the reference's division, so that a call meets them as they are (ten
// instructions per voxel more than a weight made once: 245 -> 272 us).
template<int N1>
__global__ void __launch_bounds__(kp_threads(N1)) kp_resid(PlaneArgs P)
{
    constexpr int N2 = 16, n = N1 * N2, T = kp_threads(N1), P2 = N2 + 1;
    extern __shared__ float2 sm[];          // 8 pairs of N1 P2, then n twiddles
    float2* s_tw = sm + KP_P * N1 * P2;
    __shared__ double s_part[T / 32];
    const int zo = blockIdx.y, y0 = blockIdx.x * KP_L, rows = min(KP_L, P.Ny - y0);
    const long long plane = (long long)blockIdx.z * P.Nz + zo;
    const int b = P.set0 + blockIdx.z;
    const long long v0 = ((long long)zo * P.Ny + y0) * P.Nx;       // the rows in the data cube
    float* model = P.model ? P.model + (long long)b * P.Nz * P.Ny * P.Nx + v0 : nullptr;
    const int p = threadIdx.x / KP_L, c = threadIdx.x % KP_L;
    double sum = 0.0;
    const bool empty = plane_groups(P, plane) == 0u;
    if (!empty) {
        for (int i = threadIdx.x; i < n; i += T) s_tw[i] = P.twx[i];
        if (p < KP_P && 2 * p < rows) {
            const float2* s0 = P.conv + (plane * P.Ny + y0 + 2 * p) * P.hxp;
            const float2* s1 = 2 * p + 1 < rows ? s0 + P.hxp : s0;
            float2 v[N1];
#pragma unroll
            for (int r = 0; r < N1; ++r) {
                // beyond n / 2 (known at compile time for all r but one)
                const int k = c + N2 * r;
                const bool up = N2 * r > n / 2 || (N2 * r + 15 > n / 2 && k > n / 2);
                const int kk = up ? n - k : k;
                float2 a = __ldg(s0 + kk), d = __ldg(s1 + kk);
                if (up) {
                    a.y = -a.y;
                    d.y = -d.y;
                }
                v[r] = make_float2(a.x - d.y, a.y + d.x);
            }
            dft<N1, true>(v);
            float2* d = sm + p * N1 * P2 + c;
#pragma unroll
            for (int k = 0; k < N1; ++k) d[k * P2] = v[k];
        }
        __syncthreads();
        const int q = threadIdx.x / N1, k1 = threadIdx.x - q * N1;
        const bool on = q < KP_P && 2 * q < rows;
        float2 v[N2];
        if (on) {
            const float2* s = sm + (q * N1 + k1) * P2;
#pragma unroll
            for (int r = 0; r < N2; ++r) v[r] = cmul_dir<true>(s[r], s_tw[k1 * r]);
            dft<N2, true>(v);
        }
        __syncthreads();
        if (on) {                           // the 16 rows of n values from here on
            float* d = reinterpret_cast<float*>(sm) + 2 * q * n + k1;
#pragma unroll
            for (int k = 0; k < N2; ++k) {
                d[N1 * k] = v[k].x;
                d[n + N1 * k] = v[k].y;
            }
        }
        __syncthreads();
    }
    auto residual = [&](float m, float o, float e, float k) {
        float r = m - o;
        if (P.err) r /= e;
        if (P.msk) r *= k;
        return r * P.weight;
    };
    for (int lr = p; lr < rows; lr += T / KP_L) {
        const float* ms = reinterpret_cast<const float*>(sm) + lr * n;
        const long long v = v0 + (long long)lr * P.Nx;
        const float* od = P.obs + v;
        const float* ed = P.err ? P.err + v : nullptr;
        const float* kd = P.msk ? P.msk + v : nullptr;
        float* md = model ? model + (long long)lr * P.Nx : nullptr;
        if (P.vec) {
            // the rows start on 16 bytes
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int x = 4 * c; x < P.Nx; x += 4 * KP_L) {
                const float4 o = __ldg(reinterpret_cast<const float4*>(od + x));
                const float4 e = ed ? __ldg(reinterpret_cast<const float4*>(ed + x)) : zero;
                const float4 k = kd ? __ldg(reinterpret_cast<const float4*>(kd + x)) : zero;
                const float4 m = empty ? zero : *reinterpret_cast<const float4*>(ms + x);
                const float r0 = residual(m.x, o.x, e.x, k.x), r1 = residual(m.y, o.y, e.y, k.y);
                const float r2 = residual(m.z, o.z, e.z, k.z), r3 = residual(m.w, o.w, e.w, k.w);
                sum += (double)((r0 * r0 + r1 * r1) + (r2 * r2 + r3 * r3));
                if (md) *reinterpret_cast<float4*>(md + x) = m;
            }
        } else {
            for (int x = c; x < P.Nx; x += KP_L) {
                const float m = empty ? 0.f : ms[x];
                const float r = residual(m, __ldg(od + x), ed ? __ldg(ed + x) : 0.f,
                                         kd ? __ldg(kd + x) : 0.f);
                sum += (double)(r * r);
                if (md) md[x] = m;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < T / 32; ++w) s += s_part[w];
        P.partials[((long long)b * P.Nz + zo) * gridDim.x + blockIdx.x] = s;
    }
}

typedef void (*KpFn)(PlaneArgs);
typedef void (*KpColsFn)(PlaneArgs, int);
struct PlaneRows {
    int n = 0, threads = 0;
    size_t smem = 0;
    KpFn rows = nullptr, resid = nullptr;
};
struct PlaneCols {
    int n = 0, threads = 0;
    size_t smem = 0;
    KpColsFn fn = nullptr;
};
// the shortest instantiated transforms of at least w points (null: none)
PlaneRows plane_rows(int w);
PlaneCols plane_cols(int w);

}  // namespace gbk
