// The vector node kernels' instances for f32 arenas.
#include "cfr_vec.cuh"

namespace gtob {

void vec_down_f32(const Dev& d, const Arenas& ar, const VecNodes& n, int nh, int mode, cudaStream_t s) {
    if (n.wide) down_t<kDevF32, kVKA>(d, ar, n, nh, mode, s);
    else down_t<kDevF32, kSKA>(d, ar, n, nh, mode, s);
}
void vec_mine_f32(const Dev& d, const Arenas& ar, const VecNodes& n, int p, int eval, cudaStream_t s) {
    if (n.wide) up_mine_t<kDevF32, kVKA>(d, ar, n, p, eval, s);
    else up_mine_t<kDevF32, kSKA>(d, ar, n, p, eval, s);
}

}  // namespace gtob
