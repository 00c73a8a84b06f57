// Host launchers of the vector node kernels (cfr_vec.cu).
#pragma once
#include <cuda_runtime.h>

#include "cfr_dev.cuh"

namespace gtob {

// A launch of a kernel that starts with pdl_enter().
template <class... P, class... A>
void pdl_launch(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);  // an error stays for the caller's cudaGetLastError
}

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

// A sweep's showdowns in batches of `group` of one river board, one CTA each;
// a short batch is filled with items without a cfv slot.
struct ShowShape {
    int group = 8;      // showdowns per batch: 2, 4 or 8
    int threads = 64;   // per CTA
    int chunk = 4;      // scan entries per lane: 4, 8, 12 or 16
};
struct ShowGroups {
    const ShowItem* items = nullptr;  // count * group
    uint32_t count = 0;
    ShowShape shape[2];                   // per player whose hands are scanned (one group for both)
    int max_sorted[2] = {0, 0};           // per player: most hands on a board
    void* ranks[2] = {nullptr, nullptr};  // per traverser: every board's rank entries by hand
    void* img[2] = {nullptr, nullptr};    // per player: every board's scan entries
};
// The CTA for boards of at most max_sorted opponent hands: the fewest threads
// whose lanes hold the scan; false if none.
bool show_shape(int group, int max_sorted, ShowShape& sh);
size_t show_group_smem(const ShowShape& sh, int max_sorted, int nho);
const void* show_group_kernel(const ShowShape& sh);
size_t hand_rank_bytes();
size_t show_image_bytes(const ShowShape& sh, int max_sorted);
void build_show_tables(const Dev& d, const ShowGroups& sg, uint32_t slots, cudaStream_t s);
void vec_show(const Dev& d, const ShowGroups& sg, int p, cudaStream_t s);
// A sweep's fold summaries into d.folds: fold k's opponent vector is reach
// slot slots[k].
size_t fold_sum_bytes();
void fold_kernels(int nho, const void* (&fn)[2], size_t* smem);
void vec_folds(const Dev& d, const uint32_t* slots, uint32_t count, int p, cudaStream_t s);
// Chance nodes of one level (no runout terminals), and its chance edges' reach
// for the players of qmask.
void vec_chance(const Dev& d, const ChanceItem* items, uint32_t count, int p, cudaStream_t s);
void vec_edges(const Dev& d, const EdgeItem* items, uint32_t count, int qmask, cudaStream_t s);

}  // namespace gtob
