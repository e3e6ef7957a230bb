// Explicit instantiations of the model kernel on 4 x 8 spaxel tiles
// (ka_lines_lsf_t), one per odd LSF length of the direct path, with and
// without the scaled line exponent (sl).
#include "gbk_batched.cuh"

namespace gbk {

template<int KZ>
static void fill(KaFn* t, bool sl)
{
    t[KZ / 2] = sl ? ka_lines_lsf_t<KZ, true> : ka_lines_lsf_t<KZ, false>;
    if constexpr (KZ + 2 <= KA_KMAX) fill<KZ + 2>(t, sl);
}

void ka_t_register(KaFn* t, bool sl) { fill<1>(t, sl); }

}  // namespace gbk
