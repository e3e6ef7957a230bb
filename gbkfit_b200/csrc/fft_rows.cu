// Instantiations of the row FFT kernels: half the row lengths that the
// padding rule of the drop-in path gives (multiples of 16).
#include "gbk_lines.cuh"

namespace gbk {

template<int N1, int N2>
static FastRows make()
{
    FastRows f;
    f.fwd = fast_r2c_kernel<N1, N2>;
    f.inv = fast_c2r_kernel<N1, N2>;
    f.threads = FAST_LT * (N1 > N2 ? N1 : N2);
    f.smem = (size_t)(FAST_LT * N1 * (N2 + 1) + N1 * N2) * sizeof(float2);
    return f;
}

FastRows fast_rows(int M)
{
    switch (M) {
    case 16: return make<4, 4>();
    case 32: return make<4, 8>();
    case 48: return make<6, 8>();
    case 64: return make<8, 8>();
    case 80: return make<10, 8>();
    case 96: return make<12, 8>();
    case 112: return make<14, 8>();
    case 128: return make<16, 8>();
    case 144: return make<9, 16>();
    case 160: return make<10, 16>();
    case 176: return make<11, 16>();
    case 192: return make<12, 16>();
    default: return FastRows();
    }
}

}  // namespace gbk
