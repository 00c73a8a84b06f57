// Host launchers of the vector node kernels (cfr_vec.cu).
#pragma once
#include <cuda_runtime.h>

#include "cfr_dev.cuh"

namespace gtob {

// Action nodes of one level and one actor, given as SNodeT<4> records or
// (wide) SNodeT<8> records.
struct VecNodes {
    const void* nodes;
    uint32_t count;
    bool wide;
};
// Down sweep: the actors' child reach vectors.  nh: hands of the records'
// actor (the larger player's when a launch mixes actors); mode 0: current
// strategies, else average strategies.
void vec_down(const Dev& d, const Arenas& ar, int fmt, const VecNodes& n, int nh, int mode, cudaStream_t s);
// Up sweep for traverser p: the traverser's nodes (mine) or the opponent's.
// eval < 0: the CFR update; 0 / 1: best response / average-strategy values.
void vec_up(const Dev& d, const Arenas& ar, int fmt, const VecNodes& n, bool mine, int p, int eval, cudaStream_t s);


}  // namespace gtob
