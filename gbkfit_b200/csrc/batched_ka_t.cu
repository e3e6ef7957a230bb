// Explicit instantiations of the model kernel on 4 x 8 spaxel tiles
// (ka_lines_lsf_t), one per odd LSF length of the FIR, by the form of the line.
#include "gbk_batched.cuh"

namespace gbk {

template<int KZ>
static void fill(KaFn* t, int lf)
{
    t[KZ / 2] = lf == LINE_EXP      ? ka_lines_lsf_t<KZ, LINE_EXP>
                : lf == LINE_SCALED ? ka_lines_lsf_t<KZ, LINE_SCALED>
                                    : ka_lines_lsf_t<KZ, LINE_EX2>;
    if constexpr (KZ + 2 <= KA_KMAX) fill<KZ + 2>(t, lf);
}

void ka_t_register(KaFn* t, int lf) { fill<1>(t, lf); }

}  // namespace gbk
