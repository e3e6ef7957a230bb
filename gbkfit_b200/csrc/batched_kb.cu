// Explicit instantiations of the batched PSF kernel, one per odd FIR length.
#include "gbk_batched.cuh"

namespace gbk {

template<int K>
static void fill(KbFn* t)
{
    t[(K - KB_KMIN) / 2] = kb_psf_residual<K>;
    if constexpr (K + 2 <= KB_KMAX) fill<K + 2>(t);
}

void kb_register(KbFn* t) { fill<KB_KMIN>(t); }

}  // namespace gbk
