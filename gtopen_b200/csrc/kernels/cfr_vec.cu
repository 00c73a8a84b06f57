// The vector node kernels' entry points, the opponent's nodes (no arenas) and
// the instances for FP8 arenas (nodes of at most 4 actions).
#include "cfr_vec.cuh"

namespace gtob {

void vec_down_f32(const Dev&, const Arenas&, const VecNodes&, int, int, cudaStream_t);
void vec_down_i16(const Dev&, const Arenas&, const VecNodes&, int, int, cudaStream_t);
void vec_mine_f32(const Dev&, const Arenas&, const VecNodes&, int, int, cudaStream_t);
void vec_mine_i16(const Dev&, const Arenas&, const VecNodes&, int, int, cudaStream_t);

void vec_down(const Dev& d, const Arenas& ar, int fmt, const VecNodes& n, int nh, int mode, cudaStream_t s) {
    if (!n.count) return;
    if (fmt == kDevF32) vec_down_f32(d, ar, n, nh, mode, s);
    else if (fmt == kDevI16) vec_down_i16(d, ar, n, nh, mode, s);
    else down_t<kDevFP8, kSKA>(d, ar, n, nh, mode, s);
}
void vec_up(const Dev& d, const Arenas& ar, int fmt, const VecNodes& n, bool mine, int p, int eval, cudaStream_t s) {
    if (!n.count) return;
    if (!mine) {
        if (n.wide) up_opp_t<kVKA>(d, n, p, s);
        else up_opp_t<kSKA>(d, n, p, s);
    } else if (fmt == kDevF32) {
        vec_mine_f32(d, ar, n, p, eval, s);
    } else if (fmt == kDevI16) {
        vec_mine_i16(d, ar, n, p, eval, s);
    } else {
        up_mine_t<kDevFP8, kSKA>(d, ar, n, p, eval, s);
    }
}

}  // namespace gtob
