// Instantiations of the plane-wise FFT convolution kernels; a window is padded
// to the next line length.
#include "gbk_planes.cuh"

namespace gbk {

template<int N1>
static bool rows_fit(int w, PlaneRows& f)
{
    constexpr int n = N1 * 16;
    if (n < w) return false;
    f.n = n;
    f.threads = kp_threads(N1);
    f.smem = (size_t)(KP_P * N1 * 17 + n) * sizeof(float2);
    f.rows = kp_rows<N1>;
    f.resid = kp_resid<N1>;
    return true;
}

PlaneRows plane_rows(int w)
{
    PlaneRows f;
    (void)(rows_fit<2>(w, f) || rows_fit<3>(w, f) || rows_fit<4>(w, f) || rows_fit<5>(w, f) ||
           rows_fit<6>(w, f) || rows_fit<7>(w, f) || rows_fit<8>(w, f) || rows_fit<9>(w, f) ||
           rows_fit<10>(w, f) || rows_fit<11>(w, f) || rows_fit<12>(w, f) || rows_fit<14>(w, f) ||
           rows_fit<15>(w, f) || rows_fit<16>(w, f) || rows_fit<18>(w, f) || rows_fit<20>(w, f) ||
           rows_fit<22>(w, f) || rows_fit<24>(w, f));
    return f;
}

template<int N1>
static bool cols_fit(int w, PlaneCols& f)
{
    constexpr int n = N1 * 16;
    if (n < w) return false;
    f.n = n;
    f.threads = KP_L * (N1 > 16 ? N1 : 16);
    f.smem = (size_t)n * (KP_L + 1) * sizeof(float2);
    f.fn = kp_cols<N1>;
    return true;
}

PlaneCols plane_cols(int w)
{
    PlaneCols f;
    (void)(cols_fit<2>(w, f) || cols_fit<3>(w, f) || cols_fit<4>(w, f) || cols_fit<5>(w, f) ||
           cols_fit<6>(w, f) || cols_fit<7>(w, f) || cols_fit<8>(w, f) || cols_fit<9>(w, f) ||
           cols_fit<10>(w, f) || cols_fit<11>(w, f) || cols_fit<12>(w, f) || cols_fit<14>(w, f) ||
           cols_fit<15>(w, f) || cols_fit<16>(w, f) || cols_fit<18>(w, f) || cols_fit<20>(w, f) ||
           cols_fit<22>(w, f) || cols_fit<24>(w, f));
    return f;
}

}  // namespace gbk
