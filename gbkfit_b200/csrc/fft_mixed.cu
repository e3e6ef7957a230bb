// Instantiations of the mixed-radix FFT kernels at compile-time lengths: those
// that the padding rule of the drop-in path gives up to 256.
#include "gbk_lines.cuh"

namespace gbk {

template<int N>
static FastLines lines()
{
    FastLines f;
    f.fn[0] = mixed_lines_kernel<N, 0>;
    f.fn[1] = mixed_lines_kernel<N, 1>;
    f.fn[2] = mixed_lines_kernel<N, 2>;
    f.threads = FFT_THREADS;
    f.smem = (size_t)N * (2 * FAST_LT + 1) * sizeof(float2);
    return f;
}

FastLines mixed_lines(int n)
{
    switch (n) {
    case 32: return lines<32>();
    case 64: return lines<64>();
    case 96: return lines<96>();
    case 128: return lines<128>();
    case 160: return lines<160>();
    case 192: return lines<192>();
    case 224: return lines<224>();
    case 256: return lines<256>();
    default: return FastLines();
    }
}

template<int M>
static FastRows rows()
{
    FastRows f;
    f.fwd = mixed_r2c_kernel<M>;
    f.inv = mixed_c2r_kernel<M>;
    f.threads = FFT_THREADS;
    f.smem = (size_t)(2 * FAST_LT * M + 2 * M + 1) * sizeof(float2);
    return f;
}

FastRows mixed_rows(int M)
{
    switch (M) {
    case 16: return rows<16>();
    case 32: return rows<32>();
    case 48: return rows<48>();
    case 64: return rows<64>();
    case 80: return rows<80>();
    case 96: return rows<96>();
    case 112: return rows<112>();
    case 128: return rows<128>();
    default: return FastRows();
    }
}

}  // namespace gbk
