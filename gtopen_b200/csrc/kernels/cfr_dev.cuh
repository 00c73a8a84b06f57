// Device-side data layout and arithmetic shared by every engine kernel: the
// pointer tables of a plan on the device, the arenas, the node records of the
// staged engine, the exact terminal sums and the arenas' codecs.
#pragma once
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../host/plan.hpp"
#include "../host/solver.hpp"

namespace gtob {

enum ArenaFormatDev { kDevF32 = 0, kDevI16 = 1, kDevFP8 = 2 };

constexpr unsigned kSms = 148;  // a B200's SMs: the launch thresholds are multiples of it
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxHpt = 6;  // hands per thread in the runout kernel (nh <= 1536)

struct Dev {
    int nh[2];
    int nh_max;        // cfv slot stride (floats, a multiple of 4: 16-byte aligned slots)
    int rstr[2];       // reach slot stride per player (floats, a multiple of 4)
    int nh_pad;        // floats per staged hand vector (multiple of 4)
    int scr_elems;     // terminal scratch elements (4 * max_sorted + 105)
    int max_nterm;     // terminal children of one action node (fused smem layout)
    const uint8_t* c1[2];
    const uint8_t* c2[2];
    const uint64_t* mask[2];
    const uint32_t* same[2];
    const float* w[2];
    const uint16_t* hperm[2];
    const uint32_t* hcard_off[2];
    const uint16_t* hcard_idx[2];
    const uint32_t* sorted_off[2];
    const uint32_t* sorted_cnt[2];
    const uint16_t* sorted_idx[2];
    const uint32_t* ccard_off[2];
    const uint16_t* ccard_pos[2];
    const uint8_t* ccard_card[2];
    const uint32_t* bin_off[2];
    const uint16_t* bin_start[2];
    const uint32_t* rank_off[2];
    const uint32_t* rank_cnt[2];
    const RankEntry* rank[2];
    const uint32_t* zero_off[2];
    const uint16_t* zero_idx[2];
    const CardEntry* cards;
    const ChildRef* crefs;
    const TermInfo* terms;
    float* reach[2];
    float* cfv;
    const long long* lock_off[2];  // per sidx, -1 = unlocked
    const float* lock_sig;
    float* disc;  // pos, neg, strat
    unsigned* iter;
    double* dot;  // root dot products
    unsigned* err;  // device error bits (bounded waits that gave up, bad copies)
    // staged engine extras
    const uint32_t* hinfo[2];   // per hand: c1 | c2 << 6 | same << 16 (0xFFFF: no same combo)
    const struct FoldSum* folds;  // the sweep's fold summaries (vector kernels)
    const uint32_t* node_id[2];  // tree node id of each device action node (per player, by sidx)
    // river programs: per player o, the showdown table images of every river
    // board (river_tab_words words each) and their word offsets (num_slots + 1)
    const uint32_t* rtab[2];
    const uint32_t* rtab_off[2];
};
struct Arenas {
    void* reg[2];
    void* str[2];
    void* pred[2];  // PCFR+ only, else null
    float* rscale[2];
    float* sscale[2];
    float* pscale[2];
    int sr;  // 16-bit requantisation: 0 round to nearest even (store.rs), 1 stochastic rounding
};

// ----------------------------------------------------------- small helpers
// One player's entry of a kernel parameter's pair (a select: an indexed
// parameter would be copied to local memory).
template <class T>
__device__ __forceinline__ T pick(T const (&x)[2], int a) { return a ? x[1] : x[0]; }
// FP8 E4M3 arena values (the precision-study format): cvt with satfinite --
// round to nearest even, saturate to +-448 -- and the exact widening back.
__device__ __forceinline__ uint8_t f32_to_e4m3(float x) {
    return (uint8_t)__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ float e4m3_to_f32(uint8_t q) {
    return __half2float(__half(__nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)q, __NV_E4M3)));
}

// Rust `as i16` / `as u16` after round_ties_even (store.rs:178, 192): round to
// nearest even, saturate to the type's range, NaN -> 0.  One cvt.rni.sat each.
__device__ __forceinline__ int16_t sat_i16(float x) {
    short r;
    asm("cvt.rni.sat.s16.f32 %0, %1;" : "=h"(r) : "f"(x));
    return x != x ? (int16_t)0 : (int16_t)r;
}
__device__ __forceinline__ uint16_t sat_u16(float x) {
    unsigned short r;
    asm("cvt.rni.sat.u16.f32 %0, %1;" : "=h"(r) : "f"(x));
    return x != x ? (uint16_t)0 : (uint16_t)r;
}
// ------------------------------------------------ exact terminal sums
// Fold and showdown values need sums of opponent reach over hand subsets
// (game.rs:478-485, 512-575; the reference sums in f64 in one fixed order).
// Here the sums are exact, so any summation order gives the same bits: each
// reach value r (f32, >= 0) of one opponent vector goes on one fixed-point
// grid, q = round-half-even(r * 2^S) in an int64, with S = 51 - E for the
// vector's largest value < 2^E -- q < 2^51, and a sum of at most 1326 of
// them stays below 2^62.  Sums and differences are exact integer
// arithmetic; each difference becomes f32 once (correctly rounded, then
// scaled by 2^-S).  The grid step is 2^-51 of the vector's top power of two,
// about the rounding step of a running f64 sum.  Everything after the casts
// is the reference's f32 arithmetic.
__device__ __forceinline__ int fix_scale(float maxv) {
    const uint32_t u = __float_as_uint(maxv);
    const int e = (int)((u >> 23) & 0xFFu);
    const uint32_t m = u & 0x7FFFFFu;
    if (e == 0 && m == 0) return 0;
    const int E = e != 0 ? e - 126 : (32 - __clz((int)m)) - 149;  // maxv < 2^E
    return 51 - E;
}
__device__ __forceinline__ float pow2f(int k) { return __uint_as_float((uint32_t)(127 + k) << 23); }  // k in [-126,127]
__device__ __forceinline__ long long fix_q(float r, int S) {  // the scalings are exact
    float x = r;
    if (S > 100) {
        x = __fmul_rn(x, pow2f(100));
        S -= 100;
    }
    return __float2ll_rn(__fmul_rn(x, pow2f(S)));
}
__device__ __forceinline__ float fix_f(long long v, int S) {
    float y = __ll2float_rn(v);
    if (S > 100) {
        y = __fmul_rn(y, pow2f(-100));
        S -= 100;
    }
    return __fmul_rn(y, pow2f(-S));
}
// Accumulator types of the terminal sums: long long = the exact sums above
// (every engine), float = f32 sums like the reference GPU kernels (the
// fused32 engine).  q: one reach value onto the accumulator; f: a sum back
// to f32.  The scale argument is only used by the exact type.
template <class T>
struct Acc;
template <>
struct Acc<long long> {
    static constexpr bool kExact = true;
    __device__ static long long q(float r, int S) { return fix_q(r, S); }
    __device__ static float f(long long v, int S) { return fix_f(v, S); }
};
template <>
struct Acc<float> {
    static constexpr bool kExact = false;
    __device__ static float q(float r, int) { return r; }
    __device__ static float f(float v, int) { return v; }
};
__device__ __forceinline__ long long shfl_up_ll(long long v, int x) { return __shfl_up_sync(0xffffffffu, v, x); }

// Stochastic rounding of the 16-bit arenas' requantisation: x -> floor(x + u)
// with u in [0, 1) drawn from a hash of (tree node, iteration, hand, action),
// so the stored value is unbiased and increments below half a quantisation
// step still accumulate in expectation.  The hash is lowbias32 (Chris
// Wellons, "Hash Prospector", public domain): sr_base once per node and
// iteration, sr_bits per entry; the low 16 bits feed the regret, the high 16
// the strategy sum.  Deterministic: the oracle draws the same numbers.
__host__ __device__ __forceinline__ uint32_t lowbias32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}
__device__ __forceinline__ uint32_t sr_base(uint32_t node, uint32_t t) { return lowbias32(node ^ lowbias32(t)); }
__device__ __forceinline__ uint32_t sr_bits(uint32_t base, uint32_t hand, uint32_t action) {
    return lowbias32(base + ((hand << 4) | action) * 0x9E3779B9u);
}
__device__ __forceinline__ float sr_u_lo(uint32_t h) { return __fmul_rn((float)(h & 0xFFFFu), 0x1p-16f); }
__device__ __forceinline__ float sr_u_hi(uint32_t h) { return __fmul_rn((float)(h >> 16), 0x1p-16f); }
__device__ __forceinline__ int16_t sr_i16(float x, float u) {  // floor(x + u), saturated, NaN -> 0
    const float y = __fadd_rn(x, u);
    short r;
    asm("cvt.rmi.sat.s16.f32 %0, %1;" : "=h"(r) : "f"(y));
    return y != y ? (int16_t)0 : (int16_t)r;
}
__device__ __forceinline__ uint16_t sr_u16(float x, float u) {
    const float y = __fadd_rn(x, u);
    unsigned short r;
    asm("cvt.rmi.sat.u16.f32 %0, %1;" : "=h"(r) : "f"(y));
    return y != y ? (uint16_t)0 : (uint16_t)r;
}

// One entry's 16-bit requantisation after an update: store.rs's round to
// nearest even (sr = 0) or stochastic rounding (base = sr_base(tree node,
// iteration)).
__device__ __forceinline__ void requant16(float nr, float ns, float rk, float sk, int sr, uint32_t base, int i, int k,
                                          int16_t* rq, uint16_t* sq) {
    if (sr) {
        const uint32_t h = sr_bits(base, (uint32_t)i, (uint32_t)k);
        *rq = rk > 0.0f ? sr_i16(nr * rk, sr_u_lo(h)) : (int16_t)0;
        *sq = sk > 0.0f ? sr_u16(fmaxf(ns, 0.0f) * sk, sr_u_hi(h)) : (uint16_t)0;
    } else {
        *rq = rk > 0.0f ? sat_i16(nr * rk) : (int16_t)0;
        *sq = sk > 0.0f ? sat_u16(fmaxf(ns, 0.0f) * sk) : (uint16_t)0;
    }
}

constexpr int kSKA = 4;   // actions of a staged node record
constexpr int kVKA = 8;   // actions of the wide record (the vector kernels only)
// One action node as the node kernels read it: everything its loads need in
// one 80-byte record (112 bytes for the wide one).
template <int KA>
struct alignas(16) SNodeT {
    uint64_t aoff;             // arena offset (elements) in the actor's arena
    uint32_t cslot, rslot, oslot, sidx;
    uint32_t cs[KA];           // child cfv slots (the fold child: its fold's number)
    uint32_t rs[KA];           // child reach slots of the actor (down sweep; kNoSlot: none)
    uint32_t actor, na, fk;    // fk: the fold child's index, kNoSlot if none
    uint32_t folder;           // the folding player of the fold child
    float twin, tlose;         // fold payoffs
};
// Programmatic dependent launch: a kernel lets the next one on its stream
// take free SMs as soon as all its own CTAs run, and waits for the one before
// it to finish before it touches anything that one may write.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// One fold's opponent reach vector, summarised (game.rs:478-485) with exact
// sums: per card, in total, and the grid scale they are on.
struct alignas(16) FoldSum {
    long long S[52], T;
    int sc, pad;
};
using SNode = SNodeT<kSKA>;
static_assert(sizeof(SNode) == 80 && sizeof(SNodeT<kVKA>) == 112, "SNode layout");

// The two quantised arena formats: 16-bit (store.rs: i16 regrets, u16
// strategy sums) and FP8 E4M3 (both signed 8-bit), each with a per-node scale
// = the block's max magnitude, stored as value * (kR or kS) / scale.
template <int FMT>
struct QT {
    using R = int16_t;
    using S = uint16_t;
    static constexpr float kR = 32767.0f, kS = 65535.0f;
    __device__ static float dr(R q) { return (float)q; }
    __device__ static float ds(S q) { return (float)q; }
    __device__ static R er(float x) { return sat_i16(x); }
    __device__ static S es(float x) { return sat_u16(x); }
};
template <>
struct QT<kDevFP8> {
    using R = uint8_t;
    using S = uint8_t;
    static constexpr float kR = 448.0f, kS = 448.0f;
    __device__ static float dr(R q) { return e4m3_to_f32(q); }
    __device__ static float ds(S q) { return e4m3_to_f32(q); }
    __device__ static R er(float x) { return f32_to_e4m3(x); }
    __device__ static S es(float x) { return f32_to_e4m3(x); }
};
__host__ __device__ constexpr int fmt_bytes(int fmt) { return fmt == kDevF32 ? 4 : fmt == kDevFP8 ? 1 : 2; }


}  // namespace gtob
