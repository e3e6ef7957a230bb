// Batched evaluator: kernel arguments and the direct-convolution kernels
// (templates on the LSF and PSF FIR lengths, instantiated in their own
// translation units so that they compile in parallel).
#pragma once

#include "gbk_disk.cuh"
#include "gbk_fft.cuh"

#include <climits>

namespace gbk {

struct BatchKernelArgs {
    int Nx, Ny, Nz, Wx, Wy, Wz, Px, Py, Pz, hx, ex, ey, ez;
    int rows_k1;     // z rows per shared-memory group in K1
    int rows_k5;     // y rows per block in K5
    DiskArgs disk;   // per-set pointers are offset from set 0 by the strides
    int vstride[5];  // vsys, xpos, ypos, posa, incl values per set
    int pstride[9];  // trait parameter values per set, per kind
    AxisDev ax, ay, az;
    const float2* post;   // exp(-2 pi i k / Px), k in [0, Px/2]
    const float2* kspec;  // PSF x LSF spectrum (Pz, Py, hx)
    float scale;          // 1 / (Px Py Pz)
    const float *obs, *err, *msk;
    const float* iw;      // direct mode: mask * weight / error per voxel
    float weight;
    float2* work;         // (chunk, Wz, Py, hx)
    float* model;         // optional (nsets, Nz, Ny, Nx)
    double* partials;     // (nsets, Nz, ceil(Ny / rows_k5))
    int vec;              // Nx % 4 == 0 and obs, iw and model on 16 bytes: float4 rows
    int set0;
    // element counts of the buffers (bounds of the checked build)
    long long lim_work, lim_model, lim_part, lim_obs, lim_smem1, lim_smem5;
    // direct (separable) convolution
    int Kx, Ky, Kz;       // PSF (x, y) and LSF box sizes
    int K;                // FIR length of the PSF kernel (odd, >= Kx, Ky; zero-padded taps)
    int pitch;            // row pitch of the LSF-convolved planes in HBM (floats, % 32 == 0)
    int cap;              // shared-memory floats of a PSF block (rows of one pass)
    int band, nbands;     // output rows per PSF block, bands per plane
    // FIR coefficients in the parameter block (constant bank, uniform loads)
    float vr[33];         // (K): PSF x factor, reversed, zero-padded
    float ur[33];         // (K): PSF y factor, reversed, zero-padded
    float lsfr[33];       // (Kz): LSF reversed
    float* mplanes;       // (chunk, Nz, Wy, pitch): written where xr is not empty
    int nch;              // 32-column chunks per window row, ceil(Wx / 32)
    unsigned nch_inv;     // ceil(2^32 / nch), nch > 1: i / nch = umulhi(i, nch_inv) for
                          // i nch < 2^32
    int nwfast;           // the disk's traits are exactly rpt/vpt/dpt uid 101 (smdisk_spaxel_nw)
    int* xrt;             // (chunk, Nz, Wy, nch): the nonzero columns of each plane row
                          // chunk as a 32-bit mask (bit j: column 32 chunk + j; 0: the
                          // chunk is zero).  Every column of a 4-column group with a set
                          // bit is written; written by the model kernel, read by the
                          // PSF kernel
    const double* sat;    // (Nz, Ny + 1, Nx + 1): summed-area table of the zero-model r^2
    // executed-work counters (null unless enabled): what the direct-mode kernels
    // actually compute, for the roofline of the measured launches
    unsigned long long* counters;   // [GBK_CTR_*]
};

// counters[] slots (FMA = one fused multiply-add of one lane)
enum {
    GBK_CTR_KA_FMA = 0,     // LSF FIR taps of the model kernel
    GBK_CTR_KA_LINE = 1,    // line values (one exp each) of the model kernel
    GBK_CTR_KB_XFMA = 2,    // PSF x FIR taps
    GBK_CTR_KB_YFMA = 3,    // PSF y FIR taps
    GBK_CTR_KB_VOX = 4,     // residual voxels computed from the model box
    GBK_CTR_KA_SPAXEL = 5,  // spaxel evaluations
    GBK_CTR_N = 8
};

// set b's per-set inputs: pointers offset from set 0 by the strides
__device__ __forceinline__ DiskArgs set_disk(const BatchKernelArgs& P, int b)
{
    DiskArgs a = P.disk;
    if (a.vsys) a.vsys += (long long)b * P.vstride[0];
    a.xpos += (long long)b * P.vstride[1];
    a.ypos += (long long)b * P.vstride[2];
    a.posa += (long long)b * P.vstride[3];
    a.incl += (long long)b * P.vstride[4];
    TraitSet* ts[9] = {&a.rpt, &a.rht, &a.vpt, &a.vht, &a.dpt, &a.dht, &a.zpt, &a.spt, &a.wpt};
#pragma unroll
    for (int k = 0; k < 9; ++k)
        if (ts[k]->pv) ts[k]->pv += (long long)b * P.pstride[k];
    return a;
}

constexpr int KA_THREADS = 128;        // 4 independent (row, chunk) warps per block

// ---- direct convolution: LSF FIR per column, separable PSF FIR per plane ----
//
// Crop output (zo, yo, xo) of the reference's FFT convolution equals
//   sum_t sum_sy sum_sx  lsf[Kz-1-t] psf[Ky-1-sy][Kx-1-sx] model(zo+t, yo+sy, xo+sx)
// in window coordinates (the padded grid's first W indices): the kernel is
// PSF(x, y) x LSF(z), and PSF = u(y) v(x) (rank 1: a circular Gaussian's
// 8-sigma truncation corners are ~1e-14 of the peak).
//
// Sparsity: a line is exactly zero outside its +-5 sigma channel window and
// off the disk, so each LSF-convolved plane is nonzero only in a band of
// rows and columns.  The model kernel records each plane row chunk's nonzero
// columns; the PSF kernel convolves only the bounding box of its plane (sums
// of exact zeros are exact zeros, so results do not change) and takes the
// residual outside the box, where the model is exactly 0, from a summed-area
// table of ((0 - data) / error * mask * weight)^2 built once per data cube.

// KA: a warp per (set, window row y, 32-spaxel chunk of the row), no block
// synchronisation.  A lane evaluates its spaxel and then streams its
// LSF-convolved spectral column over the warp's output channel range: a
// sliding window of KZ line values in registers (compile-time rotation, KZ
// taps per output), each output plane row chunk stored as one coalesced
// 128-byte segment.  Per plane the chunk's nonzero-column mask is stored.
// Warp-wide transpose of a 32 x 32 bit matrix: lane i holds row i (bit j =
// column j) and receives column i (bit j = row j of lane j).  Five butterfly
// stages, each exchanging the off-diagonal blocks of the 2s x 2s sub-blocks
// (s = 16, 8, 4, 2, 1) with the partner lane i ^ s.
__device__ __forceinline__ unsigned warp_transpose32(unsigned v, int lane)
{
    constexpr unsigned M[5] = {0x0000ffffu, 0x00ff00ffu, 0x0f0f0f0fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int s = 16 >> k;
        const unsigned y = __shfl_xor_sync(0xffffffffu, v, s);
        v = (lane & s) ? ((v & ~M[k]) | ((y >> s) & M[k])) : ((v & M[k]) | ((y << s) & ~M[k]));
    }
    return v;
}

// The nonzero-lane masks of output planes [mz, mz + 32): lane j receives the
// mask of plane mz + j, bit l set when lane l's output range [olo, ohi]
// holds that plane (the per-plane ballots of the range test, for 32 planes
// at once).  A lane without a line passes olo > ohi.
__device__ __forceinline__ unsigned plane_masks32(int olo, int ohi, int mz, int lane)
{
    const int a = max(olo - mz, 0), e = min(ohi - mz, 31);
    const unsigned row = a <= e ? ((0xffffffffu >> (31 - e)) & (0xffffffffu << a)) : 0u;
    return warp_transpose32(row, lane);
}

template<int KZ>
__global__ void __launch_bounds__(KA_THREADS, (KZ <= 15 ? 8 : 4)) ka_lines_lsf(BatchKernelArgs P, int* status)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * (KA_THREADS / 32) + warp;
    if (item >= P.Wy * P.nch) return;                    // whole warp
    const int y = item / P.nch, chunk = item % P.nch;
    const int c = blockIdx.y, b = P.set0 + c;
    const DiskArgs a = set_disk(P, b);
    const DiskConst kc = disk_const(a);
    int bad = 0;
    const int x = chunk * 32 + lane;
    SpaxelOut o{};
    int lo = INT_MAX, hi = -1;
    float amp = 0.f, rinv = 0.f;
    const bool on = x < P.Wx && (P.nwfast ? smdisk_spaxel_nw(a, kc, x, y, o)
                                           : smdisk_spaxel(a, kc, x, y, 0, o, bad));
    if (on && line_window(o.vv, o.dv, P.Wz, a.spec_step, a.spec_zero, lo, hi)) {
        amp = o.orv * (1 / (o.dv * sqrtf(2 * GBK_PI)));
        // exp(-d^2 / (2 sigma^2)) as exp2(-d^2 * log2(e) / (2 sigma^2))
        rinv = 1.4426950408889634f / (2 * o.dv * o.dv);
    } else {
        lo = INT_MAX;
        hi = -1;
    }
    const float v = o.vv, z0 = a.spec_zero, dz = a.spec_step;
    // gmodels.hpp:109-115: the line at window channel z (0 outside [lo, hi]);
    // 2^x by the PTX ex2.approx instruction (relative error ~2^-22; the
    // argument is >= -18.1 inside the +-5 sigma window, far from underflow)
    // (one unsigned compare for z in [lo, hi]; a lane without a line has
    // amp = 0 and rinv = 0, so its value is 0 whatever the compare says)
    // zf: z as a float (exact: channel indices are far below 2^24)
    const unsigned wlen = (unsigned)hi - (unsigned)lo;
    auto line_f = [&](int z, float zf) {
        const float d = (z0 + zf * dz) - v;
        float e;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-(d * d) * rinv));
        return (unsigned)z - (unsigned)lo <= wlen ? amp * e : 0.f;
    };
    auto line = [&](int z) { return line_f(z, (float)z); };
    // the lane's and the warp's output channel ranges
    const bool lit = lo <= hi;
    const int olo = lit ? max(0, lo - KZ + 1) : INT_MAX, ohi = lit ? min(P.Nz - 1, hi) : -1;
    const unsigned olen = lit ? (unsigned)(ohi - olo) : 0u;
    int zlo = olo, zhi = ohi;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        zlo = min(zlo, __shfl_xor_sync(0xffffffffu, zlo, s));
        zhi = max(zhi, __shfl_xor_sync(0xffffffffu, zhi, s));
    }
    // the range table, plane-major (set, plane, row, chunk) as the PSF kernel
    // reads it: this warp's entry of plane z at xr[z * xs]
    const long long xs = (long long)P.Wy * P.nch;
    int* xr = P.xrt + ((long long)c * P.Nz * P.Wy + y) * P.nch + chunk;
    // planes outside [zlo, zhi] are empty for this chunk
    for (int zo = lane; zo < P.Nz; zo += 32)
        if (zo < zlo || zo > zhi) xr[zo * xs] = 0;
    if (zlo <= zhi) {
        float lz[KZ];
#pragma unroll
        for (int t = 0; t < KZ; ++t) lz[t] = P.lsfr[t];
        float w[KZ];
#pragma unroll
        for (int t = 0; t < KZ - 1; ++t) w[t] = line(zlo + t);
        const long long zstride = (long long)P.Wy * P.pitch;
        float* dp = P.mplanes + ((long long)c * P.Nz * P.Wy + y) * P.pitch + x + zlo * zstride;
        unsigned mm = 0u;
        // lane (zo - mz) keeps the ballot of plane zo; flushed at plane fl, every
        // 32 planes and at the last one
        int mz = zlo, own = zlo + lane, fl = min(zlo + 31, zhi);
        float zf = (float)(zlo + KZ - 1);       // the newest window channel, counted in float
        for (int zb = zlo; zb <= zhi; zb += KZ) {
#pragma unroll
            for (int k = 0; k < KZ; ++k) {
                const int zo = zb + k;
                if (zo > zhi) break;
                w[(k + KZ - 1) % KZ] = line_f(zo + KZ - 1, zf);
                zf += 1.f;
                // two independent accumulation chains (even and odd taps)
                float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
                for (int t = 0; t < KZ; t += 2) acc0 += lz[t] * w[(k + t) % KZ];
#pragma unroll
                for (int t = 1; t < KZ; t += 2) acc1 += lz[t] * w[(k + t) % KZ];
                *dp = acc0 + acc1;      // plane zo
                dp += zstride;
                // zo in [olo, ohi] (false for a lane without a line: olo = INT_MAX, ohi = -1)
                const unsigned m = __ballot_sync(0xffffffffu,
                                                 (unsigned)zo - (unsigned)olo <= olen);
                if (zo == own) mm = m;
                if (zo == fl) {
                    if (own <= zo) xr[own * xs] = (int)mm;
                    mz = zo + 1;
                    own = mz + lane;
                    fl = min(mz + 31, zhi);
                }
            }
        }
    }
    if (P.counters && lane == 0) {
        atomicAdd(&P.counters[GBK_CTR_KA_SPAXEL], 32ull);
        if (zlo <= zhi) {
            const unsigned long long n = (unsigned long long)(zhi - zlo + 1) * 32;
            atomicAdd(&P.counters[GBK_CTR_KA_FMA], n * KZ);
            atomicAdd(&P.counters[GBK_CTR_KA_LINE], n + (KZ - 1) * 32ull);
        }
    }
    if (bad) atomicOr(status, GBK_STATUS_BAD_TRAIT);
}

// The line's profile in ka_lines_lsf_t
enum {
    LINE_EX2,       // amp 2^(-d^2 rinv) by ex2.approx, as ka_lines_lsf
    LINE_SCALED,    // 2^(-t^2), t one multiply-add per channel
    LINE_EXP        // orv (amp expf(-d^2 / (2 sigma^2))), as the drop-in thin disk and K1
};

// KA on compact spaxel tiles: a block per (set, 4 window rows, 32-column
// chunk), its warp w on the 4 x 8 tile of columns [32 chunk + 8 w, + 8); lane
// l takes spaxel (32 chunk + 8 w + (l & 7), 4 rg + (l >> 3)).  The lines of
// nearby spaxels have close channel windows, and a 4 x 8 tile spans fewer
// velocities than a 32-spaxel row, so the warp's channel range (the union of
// its lanes' output ranges) is shorter: ~1.57 instead of ~2.11 times the
// lanes' own ranges for the 128 x 128 x 96 batch workload.  Each plane row
// store is a 32-byte segment.  A plane's 32 lanes are four rows' 8-column
// masks; each goes into byte w of that row chunk's entry (columns 8 w .. 8 w + 7)
// in shared memory (Nz x 4 entries, zero where no warp writes), and the block
// stores whole entries once all four warps are done.  The masks come after the
// channel loop, 32 planes at once: every lane forms its output range as a
// 32-bit row and the warp transposes the 32 rows (plane_masks32), a few
// instructions per group instead of a ballot and its bookkeeping per plane.
// The lines, the LSF FIR and its order of operations are those of
// ka_lines_lsf (identical values).
// LINE_SCALED: the exponent as -t^2 with t = zf (dz s) + (z0 - v) s and
// s = sqrt(log2(e) / (2 sigma^2)), one multiply-add and one multiply per
// channel instead of a multiply-add, an add and two multiplies; the same line
// up to fp32 rounding (not bit-identical to the other forms).
// LINE_EXP, for the plane-wise FFT mode: ex2.approx is 3.4e-8 low on average, which
// the transforms' rounding does not hide; 130 us instead of 105 for the lines and the
// LSF of 64 sets of 128 x 128 x 96 (eight blocks a SM; six and ten 134 and 132).
// Ten blocks a SM (48 registers, 36 bytes spilled before the channel loop): 512
// sets of 128 x 128 x 96 in 472 us, 490 with eight and 64 registers, 473 with
// nine, 480 with twelve; at 15 taps 67.5, 68.2, 71.4 and 70.6 us (16 sets of 256 x
// 240 x 128).
template<int KZ, int LF>
__global__ void __launch_bounds__(KA_THREADS, (KZ > 15 ? 4 : LF == LINE_EXP ? 8 : 10))
ka_lines_lsf_t(BatchKernelArgs P, int* status)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rg = blockIdx.x / P.nch, chunk = blockIdx.x % P.nch;   // grid: ceil(Wy / 4) nch
    extern __shared__ unsigned s_ent[];                               // (Nz, 4 rows)
    for (int i = threadIdx.x; i < 4 * P.Nz; i += KA_THREADS) s_ent[i] = 0u;
    __syncthreads();
    const int y = 4 * rg + (lane >> 3), x = chunk * 32 + 8 * warp + (lane & 7);
    const bool row_ok = y < P.Wy;
    const int c = blockIdx.y, b = P.set0 + c;
    const DiskArgs a = set_disk(P, b);
    const DiskConst kc = disk_const(a);
    int bad = 0;
    SpaxelOut o{};
    int lo = INT_MAX, hi = -1;
    float amp = 0.f, rinv = LF == LINE_EXP ? 1.f : 0.f;
    const bool on = row_ok && x < P.Wx &&
                    (P.nwfast ? smdisk_spaxel_nw(a, kc, x, y, o) : smdisk_spaxel(a, kc, x, y, 0, o, bad));
    if (on && line_window(o.vv, o.dv, P.Wz, a.spec_step, a.spec_zero, lo, hi)) {
        amp = 1 / (o.dv * sqrtf(2 * GBK_PI));
        if (LF == LINE_EXP) {
            rinv = 2 * o.dv * o.dv;             // the divisor
        } else {
            amp = o.orv * amp;
            rinv = 1.4426950408889634f / (2 * o.dv * o.dv);
        }
    } else {
        lo = INT_MAX;
        hi = -1;
    }
    const float v = o.vv, z0 = a.spec_zero, dz = a.spec_step;
    const unsigned wlen = (unsigned)hi - (unsigned)lo;
    const float sc = LF == LINE_SCALED ? sqrtf(rinv) : 0.f;
    const float dzs = dz * sc, cs = (z0 - v) * sc;
    auto line_f = [&](int z, float zf) {
        float e;
        if constexpr (LF == LINE_EXP) {
            const float d = (z0 + zf * dz) - v;
            return (unsigned)z - (unsigned)lo <= wlen ? o.orv * (amp * expf(-d * d / rinv)) : 0.f;
        } else if constexpr (LF == LINE_SCALED) {
            const float t = fmaf(zf, dzs, cs);
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-(t * t)));
        } else {
            const float d = (z0 + zf * dz) - v;
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-(d * d) * rinv));
        }
        return (unsigned)z - (unsigned)lo <= wlen ? amp * e : 0.f;
    };
    auto line = [&](int z) { return line_f(z, (float)z); };
    const bool lit = lo <= hi;
    const int olo = lit ? max(0, lo - KZ + 1) : INT_MAX, ohi = lit ? min(P.Nz - 1, hi) : -1;
    int zlo = olo, zhi = ohi;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        zlo = min(zlo, __shfl_xor_sync(0xffffffffu, zlo, s));
        zhi = max(zhi, __shfl_xor_sync(0xffffffffu, zhi, s));
    }
    // byte `warp` of the entries of plane z, rows 4 rg + r (r < 4)
    auto put = [&](int z, unsigned m) {
        unsigned char* e = reinterpret_cast<unsigned char*>(s_ent + 4 * z) + warp;
#pragma unroll
        for (int r = 0; r < 4; ++r) e[4 * r] = (unsigned char)(m >> (8 * r));
    };
    if (zlo <= zhi) {
        float lz[KZ];
#pragma unroll
        for (int t = 0; t < KZ; ++t) lz[t] = P.lsfr[t];
        float w[KZ];
#pragma unroll
        for (int t = 0; t < KZ - 1; ++t) w[t] = line(zlo + t);
        const long long zstride = (long long)P.Wy * P.pitch;
        float* dp = P.mplanes + ((long long)c * P.Nz * P.Wy + (row_ok ? y : 0)) * P.pitch + x +
                    zlo * zstride;
        float zf = (float)(zlo + KZ - 1);
        for (int zb = zlo; zb <= zhi; zb += KZ) {
#pragma unroll
            for (int k = 0; k < KZ; ++k) {
                const int zo = zb + k;
                if (zo > zhi) break;
                w[(k + KZ - 1) % KZ] = line_f(zo + KZ - 1, zf);
                zf += 1.f;
                float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
                for (int t = 0; t < KZ; t += 2) acc0 += lz[t] * w[(k + t) % KZ];
#pragma unroll
                for (int t = 1; t < KZ; t += 2) acc1 += lz[t] * w[(k + t) % KZ];
                if (row_ok) *dp = acc0 + acc1;      // plane zo
                dp += zstride;
            }
        }
        // lanes without a line: olo = INT_MAX, ohi = -1 (an empty row)
        for (int g = zlo; g <= zhi; g += 32) {
            const unsigned m = plane_masks32(olo, ohi, g, lane);
            if (g + lane <= zhi) put(g + lane, m);
        }
    }
    // the block's entries: every plane of its rows in the window
    __syncthreads();
    const int nrow = min(4, P.Wy - 4 * rg);
    const long long xs = (long long)P.Wy * P.nch;
    int* xr = P.xrt + ((long long)c * P.Nz * P.Wy + 4 * rg) * P.nch + chunk;
    for (int i = threadIdx.x; i < nrow * P.Nz; i += KA_THREADS) {
        const int z = i / nrow, r = i - z * nrow;
        xr[z * xs + r * P.nch] = (int)s_ent[4 * z + r];
    }
    if (P.counters && lane == 0) {
        atomicAdd(&P.counters[GBK_CTR_KA_SPAXEL], 32ull);
        if (zlo <= zhi) {
            const unsigned long long n = (unsigned long long)(zhi - zlo + 1) * 32;
            atomicAdd(&P.counters[GBK_CTR_KA_FMA], n * KZ);
            atomicAdd(&P.counters[GBK_CTR_KA_LINE], n + (KZ - 1) * 32ull);
        }
    }
    if (bad) atomicOr(status, GBK_STATUS_BAD_TRAIT);
}

// 16-byte copy to shared memory, or 16 zero bytes (gmem is not read then)
__device__ __forceinline__ void cp_async16_or_zero(void* smem, const void* gmem, bool on)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem),
                 "r"(on ? 16 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// sum of the summed-area table over rows [y0, y1) and columns [x0, x1)
__device__ __forceinline__ double sat_box(const double* T, int ld, int y0, int y1, int x0, int x1)
{
    return T[(long long)y1 * ld + x1] - T[(long long)y0 * ld + x1] - T[(long long)y1 * ld + x0] +
           T[(long long)y0 * ld + x0];
}

// zeros in rows [r0, r1) of a plane outside the box of rows [y0, y1) and columns
// [x0, x1) (multiples of 4, x1 possibly nx); a warp per row
__device__ __forceinline__ void kb_zero_rows(float* m, int nx, bool vec, int r0, int r1, int y0, int y1,
                                             int x0, int x1, int warp, int lane, int nwarps)
{
    for (int y = r0 + warp; y < r1; y += nwarps) {
        float* row = m + (long long)y * nx;
        const bool in = y >= y0 && y < y1;
        const int a = in ? x0 : nx, e = in ? x1 : nx;      // zero [0, a) and [e, nx)
        if (vec) {
            for (int x = 4 * lane; x < nx; x += 128)
                if (x < a || x >= e)
                    *reinterpret_cast<float4*>(row + x) = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
            for (int x = lane; x < nx; x += 32)
                if (x < a || x >= e) row[x] = 0.f;
        }
    }
}

// KB: one block per (set, output plane zo, band of output rows), sets fastest.  The block
// finds the bounding box of the band's nonzero input row chunks and works
// through its output rows in passes whose input rows fit the block's shared
// memory (box-relative row pitch; usually one pass):
//   - the rows' nonzero 4-column groups are loaded from HBM (cp.async), the rest of
//     the rows that the y FIR reads is zeroed;
//   - x FIR in place, a warp per row, its lanes on consecutive (row, strip)
//     pairs of its rows, 12 outputs per lane window;
//   - y FIR, 8 x 4 outputs per (8-row group, column) item in registers, in
//     place; then the crop, residual (objective.hpp:7-31) and r^2 against the
//     data.
// The zero-model residual outside the box comes from the summed-area table.
//
// Bound by issue (62 % of cycles) and shared-memory wavefronts (66 %) with 16
// warps a SM; a block's phases (cycles, 512 sets of 128 x 128 x 96): box 3.0k, to
// the loads 1.4k, loads 7.0k, x FIR 5.3k, y FIR 4.9k, residual 6.0k.  That batch:
// 1282 us with run-time divisions in the loads and outside the box and
// two-way bank conflicts in 8-column strips, 1037 now; 100 sets of 97 x 83 x 61
// 191 -> 106.  160 to 256 threads a block 1216-1300 us, 3, 5 or 6 blocks a SM
// 1141, 1090, 1199.
constexpr int KB_THREADS = 128;
constexpr int KB_XS = 12;       // output columns of an x FIR strip
constexpr int KB_NX_MAX = 512;  // widest data cube of the direct mode

template<int K>
__global__ void __launch_bounds__(KB_THREADS, 4) kb_psf_residual(BatchKernelArgs P)
{
    constexpr int NW = (K + KB_XS - 1 + 3) / 4;     // float4 slots of one x window
    constexpr int NT = KB_THREADS, NWARPS = NT / 32;
    extern __shared__ float4 sm4[];
    float* S = reinterpret_cast<float*>(sm4);                   // (rows of a pass, bp)
    int* const s_xr = reinterpret_cast<int*>(S + P.cap);        // (in1 - ob0, nch) range entries
    __shared__ float warp_part[NWARPS];
    __shared__ int s_box[4];
    __shared__ double s_sat[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ld = P.Nx + 1;
    // blockIdx.x the set, blockIdx.y the (plane, band): sets vary fastest, so
    // the blocks in flight share a few planes of the data
    const int c = blockIdx.x, b = P.set0 + c;
    const int zo = blockIdx.y / P.nbands, band = blockIdx.y % P.nbands;
    const int ob0 = band * P.band, ob1 = min(P.Ny, ob0 + P.band);  // output rows [ob0, ob1)
    const int in1 = min(P.Wy, ob1 + K - 1);                        // input rows [ob0, in1)
    const long long prow = ((long long)c * P.Nz + zo) * P.Wy;
    const int* xr = P.xrt + prow * P.nch;                          // (y, chunk) at [y nch + chunk]
    const double* T = P.sat + (long long)zo * (P.Ny + 1) * ld;
    if (threadIdx.x == 0) {
        s_box[0] = INT_MAX; s_box[1] = -1; s_box[2] = INT_MAX; s_box[3] = -1;
    }
    __syncthreads();
    // bounding box of the nonzero input row chunks, all of a thread's entries
    // requested at once
    {
        int y0 = INT_MAX, y1 = -1, x0 = INT_MAX, x1 = -1;
        const int* src = xr + ob0 * P.nch;
        const int n = (in1 - ob0) * P.nch;
        for (int i0 = threadIdx.x; i0 < n; i0 += 8 * NT) {
            int v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = i0 + u * NT < n ? src[i0 + u * NT] : 0;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int i = i0 + u * NT;
                if (i < n) s_xr[i] = v[u];
                if (v[u] != 0) {
                    const int r = P.nch == 1 ? i : (int)__umulhi((unsigned)i, P.nch_inv);
                    const int ch = i - r * P.nch;
                    y0 = min(y0, ob0 + r);
                    y1 = max(y1, ob0 + r);
                    x0 = min(x0, ch * 32 + __ffs(v[u]) - 1);
                    x1 = max(x1, ch * 32 + 31 - __clz(v[u]));
                }
            }
        }
        y0 = __reduce_min_sync(0xffffffffu, y0);
        y1 = __reduce_max_sync(0xffffffffu, y1);
        x0 = __reduce_min_sync(0xffffffffu, x0);
        x1 = __reduce_max_sync(0xffffffffu, x1);
        if (lane == 0 && y1 >= 0) {
            atomicMin(&s_box[0], y0);
            atomicMax(&s_box[1], y1);
            atomicMin(&s_box[2], x0);
            atomicMax(&s_box[3], x1);
        }
    }
    __syncthreads();
    const int y0 = s_box[0], y1 = s_box[1], x0 = s_box[2], x1 = s_box[3];
    const long long plane = (long long)P.Ny * P.Nx;
    float* model = P.model ? P.model + ((long long)b * P.Nz + zo) * plane : nullptr;
    const long long part = ((long long)b * P.Nz + zo) * P.nbands + band;
    if (y1 < 0) {   // nothing reaches this band: the model is 0 on it
        if (model)
            kb_zero_rows(model, P.Nx, P.vec, ob0, ob1, ob0, ob0, 0, 0, warp, lane, NWARPS);
        if (threadIdx.x == 0) P.partials[part] = sat_box(T, ld, ob0, ob1, 0, P.Nx);
        return;
    }
    // output box: x in 12-column strips [0, ns12) from the float4 slot sl0 on, rows
    // [yo_lo, yb_end) in 8-row groups
    const int sl0 = max(0, x0 - K + 1) >> 2;
    const int ns4 = (min(P.Nx - 1, x1) >> 2) - sl0 + 1;
    const int ns12 = (ns4 + KB_XS / 4 - 1) / (KB_XS / 4);
    const int yo_lo = max(ob0, y0 - K + 1), yo_hi = min(ob1 - 1, y1);
    const int yb_end = min(ob1, yo_lo + 8 * ((yo_hi - yo_lo + 8) / 8));
    const int xb0 = 4 * sl0, xb_end = min(P.Nx, xb0 + 4 * ns4);
    // the zero-model part: the corners of the band and of the box, copied to
    // shared memory beside the rows (thread 0 sums them at the end)
    if (threadIdx.x < 8) {
        const bool outer = threadIdx.x < 4;
        const int cy = threadIdx.x & 2 ? (outer ? ob1 : yb_end) : (outer ? ob0 : yo_lo);
        const int cx = threadIdx.x & 1 ? (outer ? P.Nx : xb_end) : (outer ? 0 : xb0);
        cp_async8(&s_sat[threadIdx.x], T + (long long)cy * ld + cx);
    }
    // box-relative rows: float4 slots [sl0, sl0 + nsl), pitch bp (% 32 == 4)
    const int nsl = KB_XS / 4 * (ns12 - 1) + NW;
    int bp = 4 * nsl;
    bp += ((4 - bp % 32) + 32) % 32;
    const int bp4 = bp / 4;
    const int bo = ((P.cap / bp - (K + 7)) / 8) * 8;        // output rows per pass (>= 8)
    const float4* src = reinterpret_cast<const float4*>(P.mplanes + prow * P.pitch);
    const int pbase = zo * P.Ny * P.Nx;       // the data cube has < 2^31 voxels
    float sum = 0.f;
    unsigned long long c_x = 0, c_y = 0, c_v = 0;    // executed work (thread 0)
    for (int ys = yo_lo; ys < yb_end; ys += bo) {
        const int ye = min(yb_end, ys + bo);                 // outputs [ys, ye)
        const int ng = (ye - ys + 7) / 8;
        const int rend = ys + 8 * ng + K - 1;                // rows [ys, rend) are read
        const int ly0 = max(y0, ys), ly1 = min(y1, rend - 1);
        if (P.counters && threadIdx.x == 0) {
            if (ly0 <= ly1) c_x += (unsigned long long)(ly1 - ly0 + 1) * ns12 * KB_XS * K;
            c_y += (unsigned long long)ng * ns4 * 32 * K;
            c_v += (unsigned long long)(ye - ys) * (xb_end - xb0);
        }
        // load rows [ly0, ly1], a warp per row and a lane per float4 slot: the
        // 4-column groups that hold a nonzero value (all written), zeros elsewhere
        for (int j = lane; j < nsl; j += 32) {
            const int sl = sl0 + j, ch = sl >> 3, sh = 4 * (sl & 7);
            const bool in = ch < P.nch;
            const int* m = s_xr + (ly0 + warp - ob0) * P.nch + (in ? ch : 0);
            const float4* g = src + (long long)(ly0 + warp) * (P.pitch / 4) + (in ? sl : 0);
            const long long gs = (long long)NWARPS * (P.pitch / 4);
            float4* d = sm4 + (ly0 + warp - ys) * bp4 + j;
#pragma unroll 4
            for (int y = ly0 + warp; y <= ly1; y += NWARPS) {
                cp_async16_or_zero(d, g, in && ((*m >> sh) & 0xf) != 0);
                m += NWARPS * P.nch;
                g += gs;
                d += NWARPS * bp4;
            }
        }
        // the other rows that the y FIR reads: zeros (whole rows, contiguous)
        {
            const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
            const int lo = ly0 <= ly1 ? (ly0 - ys) * bp4 : (rend - ys) * bp4;
            for (int i = threadIdx.x; i < lo; i += NT) sm4[i] = z;
            if (ly0 <= ly1)
                for (int i = (ly1 + 1 - ys) * bp4 + threadIdx.x; i < (rend - ys) * bp4; i += NT)
                    sm4[i] = z;
        }
        // a warp's x FIR reads only the rows that the warp has loaded
        cp_async_wait_all();
        __syncwarp();
        // x FIR in place: S[y][xo] = sum_s vr[s] S[y][xo + s].  A warp owns whole
        // rows (ly0 + warp, + NWARPS, ...); its lanes take consecutive (row,
        // strip) pairs of those rows, 32 per pass.  Strip g writes columns
        // [12 g, 12 g + 12) and reads columns >= 12 g, so a row's strips in increasing
        // order across passes, with loads before __syncwarp, never read a
        // column that an earlier store of the row has overwritten.  Strips of
        // 12: their float4 accesses lie 3 slots apart, which meets all banks
        // (8-column strips were 2 apart, two-way conflicts).
        if (ly0 <= ly1) {
            const int nr = ly1 - ly0 + 1;
            const int nri = warp < nr ? (nr - 1 - warp) / NWARPS + 1 : 0;   // rows of this warp
            const int npairs = nri * ns12;
            const int di = 32 / ns12, dg = 32 % ns12;
            int ri = lane / ns12, gi = lane % ns12;       // the lane's pair: row index, strip
            for (int q0 = 0; q0 < npairs; q0 += 32) {
                const bool act = q0 + lane < npairs;
                float4* row = sm4 + (ly0 + warp + NWARPS * ri - ys) * bp4 + KB_XS / 4 * gi;
                float w[4 * NW];
                if (act) {
#pragma unroll
                    for (int m = 0; m < NW; ++m) {
                        const float4 f = row[m];
                        w[4 * m] = f.x; w[4 * m + 1] = f.y; w[4 * m + 2] = f.z; w[4 * m + 3] = f.w;
                    }
                }
                __syncwarp();
                if (act) {
                    float o[KB_XS];
#pragma unroll
                    for (int q = 0; q < KB_XS; ++q) {
                        float acc = 0.f;
#pragma unroll
                        for (int s = 0; s < K; ++s) acc += P.vr[s] * w[q + s];
                        o[q] = acc;
                    }
#pragma unroll
                    for (int q = 0; q < KB_XS; q += 4)
                        row[q / 4] = make_float4(o[q], o[q + 1], o[q + 2], o[q + 3]);
                }
                __syncwarp();
                ri += di;
                gi += dg;
                if (gi >= ns12) {
                    gi -= ns12;
                    ++ri;
                }
            }
        }
        __syncthreads();
        // y FIR in place: model(yo, xo) = sum_t ur[t] S[yo + t][xo], written to S row yo.
        // Packed FP32 pairs (FFMA2: two lanes of fma, each rounded as fmaf),
        // columns (x, x+1) and (x+2, x+3) of a float4 per instruction.  Items
        // (row group, float4 column) in ascending order, NT per round, loads
        // before the round's barrier and stores after it: a column's group is
        // written only after every lower group of that column, the only
        // readers of its rows, has loaded them.
        {
            float2 u2[K];
#pragma unroll
            for (int t = 0; t < K; ++t) u2[t] = make_float2(P.ur[t], P.ur[t]);
            const int nitems = ng * ns4;
            for (int gr0 = 0; gr0 < nitems; gr0 += NT) {
                float2 acc[8][2];
                const int item = gr0 + threadIdx.x;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    acc[q][0] = make_float2(0.f, 0.f);
                    acc[q][1] = make_float2(0.f, 0.f);
                }
                const int rb = 8 * (item / ns4), s4 = item % ns4;
                if (item < nitems) {
                    const float4* colp = reinterpret_cast<const float4*>(S) + rb * bp4 + s4;
#pragma unroll
                    for (int m = 0; m < K + 7; ++m) {
                        const float4 p = colp[m * bp4];
                        const float2 pxy = make_float2(p.x, p.y), pzw = make_float2(p.z, p.w);
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const int t = m - q;
                            if (t >= 0 && t < K) {
                                acc[q][0] = __ffma2_rn(u2[t], pxy, acc[q][0]);
                                acc[q][1] = __ffma2_rn(u2[t], pzw, acc[q][1]);
                            }
                        }
                    }
                }
                __syncthreads();
                if (item < nitems) {
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (ys + rb + q < ye)
                            reinterpret_cast<float4*>(S)[(rb + q) * bp4 + s4] =
                                make_float4(acc[q][0].x, acc[q][0].y, acc[q][1].x, acc[q][1].y);
                }
                __syncthreads();
            }
        }
        // crop + residual over rows [ys, ye), columns [xb0, xb_end)
        if (P.vec) {
            // flat float4 index over the pass, stepped without divisions
            const int nv = (xb_end - xb0) >> 2;        // xb0 and xb_end are multiples of 4
            const int n = (ye - ys) * nv;
            const int dq = NT / nv, dr = NT % nv;
            int row = threadIdx.x / nv, col = threadIdx.x % nv;
            // running offsets: si in S (float4), vi in the data plane (float)
            int si = row * bp4 + col, vi = pbase + (ys + row) * P.Nx + xb0 + 4 * col;
            const int dsi = dq * bp4 + dr, dvi = dq * P.Nx + 4 * dr;
            float2 s2 = make_float2(0.f, 0.f);
#pragma unroll 4
            for (int i = threadIdx.x; i < n; i += NT) {
                const float4 m = reinterpret_cast<const float4*>(S)[si];
                const float4 o = *reinterpret_cast<const float4*>(P.obs + vi);
                const float4 w = *reinterpret_cast<const float4*>(P.iw + vi);
                // packed pairs: r = (m - o) w, s2 += r^2
                const float2 r01 = __fmul2_rn(__fadd2_rn(make_float2(m.x, m.y),
                                                         make_float2(-o.x, -o.y)),
                                              make_float2(w.x, w.y));
                const float2 r23 = __fmul2_rn(__fadd2_rn(make_float2(m.z, m.w),
                                                         make_float2(-o.z, -o.w)),
                                              make_float2(w.z, w.w));
                s2 = __ffma2_rn(r01, r01, s2);
                s2 = __ffma2_rn(r23, r23, s2);
                if (model) *reinterpret_cast<float4*>(model + (vi - pbase)) = m;
                col += dr;
                si += dsi;
                vi += dvi;
                if (col >= nv) {
                    col -= nv;
                    si += bp4 - nv;
                    vi += P.Nx - 4 * nv;
                }
            }
            sum += s2.x + s2.y;
        } else {
            // rows of any alignment: flat index over the pass, stepped without
            // divisions, several voxels in flight per thread
            const int nw = xb_end - xb0, n = (ye - ys) * nw;
            const int dq = NT / nw, dr = NT % nw;
            const int row = threadIdx.x / nw;
            int col = threadIdx.x % nw;
            int si = row * bp + col, vi = pbase + (ys + row) * P.Nx + xb0 + col;
            const int dsi = dq * bp + dr, dvi = dq * P.Nx + dr;
#pragma unroll 8
            for (int i = threadIdx.x; i < n; i += NT) {
                const float m = S[si];
                const float r0 = (m - P.obs[vi]) * P.iw[vi];
                sum += r0 * r0;
                if (model) model[vi - pbase] = m;
                col += dr;
                si += dsi;
                vi += dvi;
                if (col >= nw) {
                    col -= nw;
                    si += bp - nw;
                    vi += P.Nx - nw;
                }
            }
        }
        __syncthreads();    // S is reloaded by the next pass
    }
    if (model)
        kb_zero_rows(model, P.Nx, P.vec, ob0, ob1, yo_lo, yb_end, xb0, xb_end, warp, lane, NWARPS);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) warp_part[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int w = 0; w < NWARPS; ++w) s += warp_part[w];
        // corners [y1][x1] - [y0][x1] - [y1][x0] + [y0][x0], band minus box
        const double outside = (s_sat[3] - s_sat[1] - s_sat[2] + s_sat[0]) -
                               (s_sat[7] - s_sat[5] - s_sat[6] + s_sat[4]);
        P.partials[part] = (double)s + outside;
        if (P.counters) {
            atomicAdd(&P.counters[GBK_CTR_KB_XFMA], c_x);
            atomicAdd(&P.counters[GBK_CTR_KB_YFMA], c_y);
            atomicAdd(&P.counters[GBK_CTR_KB_VOX], c_v);
        }
    }
}

// The LSF FIR of given model cubes (any gmodel's output on the evaluation
// window, e.g. mcdisk's clouds) into the PSF kernel's input: the same
// planes and range table as ka_lines_lsf, so that the PSF FIR, residual and
// sum run unchanged.  cubes: (sets, Wz, Wy, Wx), set b = P.set0 + slot;
// one warp per (window row y, 32-column chunk), a lane per column, the
// channel axis walked with a KZ-deep register window (each cube value is
// read once).  A plane row chunk's mask marks its nonzero outputs (all
// outputs are written), so the PSF kernel skips exactly the zero ones.
template<int KZ>
__global__ void __launch_bounds__(KA_THREADS) kc_cube_lsf(BatchKernelArgs P,
                                                          const float* __restrict__ cubes)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * (KA_THREADS / 32) + warp;
    if (item >= P.Wy * P.nch) return;                    // whole warp
    const int y = item / P.nch, chunk = item % P.nch;
    const int c = blockIdx.y, b = P.set0 + c;
    const int x = chunk * 32 + lane;
    const bool in = x < P.Wx;
    const long long plane = (long long)P.Wy * P.Wx;
    const float* col = cubes + (long long)b * P.Wz * plane + (long long)y * P.Wx + (in ? x : 0);
    auto ld = [&](int z) { return in ? __ldg(col + z * plane) : 0.f; };
    float lz[KZ];
#pragma unroll
    for (int t = 0; t < KZ; ++t) lz[t] = P.lsfr[t];
    float w[KZ];
#pragma unroll
    for (int t = 0; t < KZ - 1; ++t) w[t] = ld(t);
    // the range table, plane-major: this warp's entry of plane z at xr[z * xs]
    const long long xs = (long long)P.Wy * P.nch;
    int* xr = P.xrt + ((long long)c * P.Nz * P.Wy + y) * P.nch + chunk;
    const long long zstride = (long long)P.Wy * P.pitch;
    float* dp = P.mplanes + ((long long)c * P.Nz * P.Wy + y) * P.pitch + x;
    unsigned mm = 0u;
    for (int zb = 0; zb < P.Nz; zb += KZ) {
#pragma unroll
        for (int k = 0; k < KZ; ++k) {
            const int zo = zb + k;
            if (zo >= P.Nz) break;
            w[(k + KZ - 1) % KZ] = ld(zo + KZ - 1);
            float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
            for (int t = 0; t < KZ; t += 2) acc0 += lz[t] * w[(k + t) % KZ];
#pragma unroll
            for (int t = 1; t < KZ; t += 2) acc1 += lz[t] * w[(k + t) % KZ];
            const float v = acc0 + acc1;
            *dp = v;        // plane zo
            dp += zstride;
            // lane (zo % 32) keeps the ballot of plane zo; written every 32
            // planes and at the last one
            const unsigned m = __ballot_sync(0xffffffffu, v != 0.f);
            if ((zo & 31) == lane) mm = m;
            if ((zo & 31) == 31 || zo == P.Nz - 1) {
                const int own = (zo & ~31) + lane;
                if (own <= zo) xr[own * xs] = (int)mm;
            }
        }
    }
    if (P.counters && lane == 0)
        atomicAdd(&P.counters[GBK_CTR_KA_FMA], (unsigned long long)P.Nz * 32 * KZ);
}

typedef void (*KaFn)(BatchKernelArgs, int*);
typedef void (*KbFn)(BatchKernelArgs);
constexpr int KA_KMAX = 33;                 // longest LSF of the direct path
constexpr int KB_KMIN = 5, KB_KMAX = 33;    // PSF FIR lengths (odd)
static_assert(KA_KMAX <= 33 && KB_KMAX <= 33, "coefficient arrays of BatchKernelArgs");
// fill t[Kz / 2] (model kernel) and t[(K - KB_KMIN) / 2] (PSF kernel)
void ka_register_short(KaFn* t);
void ka_register_long(KaFn* t);
// t[Kz / 2]: the model kernel on 4 x 8 spaxel tiles (ka_lines_lsf_t)
void ka_t_register(KaFn* t, int lf);
// t[Kz / 2]: the LSF FIR of given model cubes
typedef void (*KcFn)(BatchKernelArgs, const float*);
void kc_register(KcFn* t);
// t[(K - KB_KMIN) / 2]: the PSF kernel
void kb_register(KbFn* t);

}  // namespace gbk
