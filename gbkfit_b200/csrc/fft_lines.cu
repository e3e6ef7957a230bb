// Instantiations of the strided-column FFT kernels: the lengths that the
// padding rule of the drop-in path gives (multiples of 32).
#include "gbk_lines.cuh"

namespace gbk {

template<int N1, int N2>
static FastLines make()
{
    FastLines f;
    f.fn[0] = fast_lines_kernel<N1, N2, 0>;
    f.fn[1] = fast_lines_kernel<N1, N2, 1>;
    f.fn[2] = fast_lines_kernel<N1, N2, 2>;
    f.threads = FAST_LT * (N1 > N2 ? N1 : N2);
    f.smem = (size_t)(N1 * N2) * (FAST_LT + 1) * sizeof(float2);
    return f;
}

FastLines fast_lines(int n)
{
    switch (n) {
    case 32: return make<4, 8>();
    case 64: return make<8, 8>();
    case 96: return make<8, 12>();
    case 128: return make<8, 16>();
    case 160: return make<16, 10>();
    case 192: return make<16, 12>();
    case 224: return make<16, 14>();
    case 256: return make<16, 16>();
    case 288: return make<16, 18>();
    case 320: return make<16, 20>();
    case 352: return make<16, 22>();
    case 384: return make<16, 24>();
    default: return FastLines();
    }
}

}  // namespace gbk
