// Vector node kernels: the level sweeps' action nodes (the default engine).
//
// A thread owns V consecutive hands of a node and keeps everything about
// them -- strategy, regrets, strategy sums, child values, new values -- in
// registers: arena blocks are hand-major ([hand * na + action]), so its
// entries are V * na consecutive elements, read and written with the widest
// aligned loads, and hand vectors (reach, child values) are read V floats at
// a time.  Nothing is staged in shared memory, and the only block-wide step is
// the node's maxima in the update of quantised arenas: a fold child's card
// sums come from the sweep's fold summaries (cfr_show.cu).
//
// What bounds them, and why this split: the bulk-copy kernels they replace
// kept each node's blocks in shared memory and touched every 16-bit entry
// with two-byte shared accesses, and a 128-thread CTA per node cost ~4.2 ns
// of the device whatever its size.  Here
//   * where a node's hands do not depend on one another -- the down sweep,
//     the opponent's nodes, evaluation sweeps, f32 updates -- a warp takes
//     32 V hands of one node, no barriers; V = 4 fills a load (470 v 647
//     hands: down 0.45 ms, V = 2 0.57, V = 1 0.69), V = 1 or 2 where the node
//     is smaller or the launch too small to fill the device;
//   * the update of quantised arenas takes the node's maxima first: a node of
//     up to 128 hands is one warp, a larger one a CTA of ceil(hands / 128)
//     warps (V = 4: half the warps, and half their per-warp work, of V = 2 --
//     1.52 against 2.35 ms for the traverser's nodes of a 470 v 647 flop).
// One iteration with only this changed, B200, bulk-copy kernels before ->
// after: flop of 284,901 nodes at 28 v 23 hands, f32 1.83 -> 1.05 ms; flop of
// 609,894 nodes at 64 v 39, 16-bit 3.58 -> 2.02 ms; flop of 346,255 nodes at
// 470 v 647, 16-bit 5.87 -> 5.29 ms; flop of 1,220,736 nodes at 243 v 321,
// f32 9.77 -> 8.62 ms; turn of 16,989 nodes with 5-action nodes (the
// warp-per-node engine before) 2.03 -> 0.73 ms.
// A tail thread's hands beyond the node read as zeros, and pads are written
// back as zeros: blocks are padded to whole groups of four hands
// (plan.cpp), hand vectors to four floats.
//
// Arithmetic is the other engines' (the same expressions in the same order,
// -fmad=false; terminal sums exact integers), so results are identical.
#pragma once
#include <type_traits>

#include "cfr_vec.hpp"

namespace gtob {
namespace {

// CTAs of 128 threads an SM must hold, for the forms that carry the large
// launches (V = 4, nodes of at most 4 actions): they wait for HBM, and more
// warps in flight are worth the spills of the rare 4-action body.  Down 16
// (32 registers), opponent 14, f32 update 8 (64); the quantised update's CTAs
// 56 registers a thread.  Registers as the compiler takes them -> capped, ms
// per iteration: 243 v 321 hands f32 down 0.96 -> 0.81, up 3.63 -> 3.03 (f32
// update 10 CTAs: 3.32); 470 v 647 16-bit down 0.50 -> 0.42, up 1.89 -> 1.59
// (64 registers: 1.67, 48: 1.64).
constexpr int kVDownCtas = 16, kVOppCtas = 14, kVMineCtas = 8, kVQuantRegs = 56;
constexpr int kVMaxWarps = 32;
constexpr uint64_t kVFillWarps = kSms * 16;  // warps that fill the device

// ------------------------------------------------------- register vectors
template <int B> struct Gran;
template <> struct Gran<1> { using T = uint8_t; };
template <> struct Gran<2> { using T = uint16_t; };
template <> struct Gran<4> { using T = uint32_t; };
template <> struct Gran<8> { using T = uint2; };
template <> struct Gran<16> { using T = uint4; };
constexpr int low_bit(int x) { return x & -x; }
constexpr int gran_bytes(int bytes) { return low_bit(bytes) < 16 ? low_bit(bytes) : 16; }
// N elements whose address is a multiple of the largest power of two
// dividing their size (at most 16)
template <class T, int N>
union Pack {
    static constexpr int G = gran_bytes(N * (int)sizeof(T));
    using GT = typename Gran<G>::T;
    static constexpr int NG = N * (int)sizeof(T) / G;
    T e[N];
    GT g[NG];
    __device__ Pack() {}
    __device__ void load(const void* p) {
#pragma unroll
        for (int k = 0; k < NG; k++) g[k] = ((const GT*)p)[k];
    }
    __device__ void store(void* p) const {
#pragma unroll
        for (int k = 0; k < NG; k++) ((GT*)p)[k] = g[k];
    }
    __device__ void zero() {
#pragma unroll
        for (int k = 0; k < N; k++) e[k] = T(0);
    }
    // entries from the live-th on are pads: zero them
    __device__ void keep(int live) {
#pragma unroll
        for (int k = 0; k < N; k++)
            if (k >= live) e[k] = T(0);
    }
};

// The thread's place in its node, and the node's scratch in shared memory.
struct Group {
    int t, W;       // thread within the node, warps of the node
    uint32_t* red;  // 3 * kVMaxWarps
};
// Maxima of non-negative floats over the node's threads (their bits order as
// unsigned integers): one redux per value and warp, one barrier.
template <bool WARP, int N>
__device__ __forceinline__ void group_max(const Group& g, float (&x)[N]) {
    uint32_t b[N];
#pragma unroll
    for (int k = 0; k < N; k++) b[k] = __reduce_max_sync(0xffffffffu, __float_as_uint(x[k]));
    if (!WARP) {
        const int w = g.t >> 5, lane = g.t & 31;
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < N; k++) g.red[k * kVMaxWarps + w] = b[k];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < N; k++)
            b[k] = __reduce_max_sync(0xffffffffu, lane < g.W ? g.red[k * kVMaxWarps + lane] : 0u);
    }
#pragma unroll
    for (int k = 0; k < N; k++) x[k] = __uint_as_float(b[k]);
}

// ------------------------------------------------------------- strategies
// One hand's regret-matching strategy (cfr.rs:240-292, 875-942) from its na
// stored entries.
template <int FMT, int NA, bool PRED, class T>
__device__ __forceinline__ void v_regret_sigma(const T* r, const T* pr, float kr, float kp, float (&sig)[NA]) {
    if constexpr (FMT == kDevI16 && !PRED) {
        // on the quants, whose scale cancels; in f32, where at most 8 of them add exactly
        float sum = 0.0f;
#pragma unroll
        for (int k = 0; k < NA; k++) {
            sig[k] = fmaxf((float)r[k], 0.0f);
            sum += sig[k];
        }
        const float inv = __frcp_rn(sum);
#pragma unroll
        for (int k = 0; k < NA; k++) sig[k] = sum > 0.0f ? sig[k] * inv : 1.0f / (float)NA;
    } else {
        float sum = 0.0f;
#pragma unroll
        for (int k = 0; k < NA; k++) {
            float v;
            if (FMT == kDevF32) v = PRED ? fmaxf((float)r[k], 0.0f) + (float)pr[k] : (float)r[k];
            else if (FMT == kDevI16) v = (float)max((int)r[k], 0) * kr + (float)pr[k] * kp;
            else v = PRED ? fmaxf(e4m3_to_f32(r[k]), 0.0f) * kr + e4m3_to_f32(pr[k]) * kp : e4m3_to_f32(r[k]);
            sig[k] = fmaxf(v, 0.0f);
            sum += sig[k];
        }
        const float inv = __frcp_rn(sum);
#pragma unroll
        for (int k = 0; k < NA; k++) sig[k] = sum > 1e-12f ? sig[k] * inv : 1.0f / (float)NA;
    }
}
// One entry's 16-bit requantisation: requant16's values in fewer
// instructions.  cvt from f32 to a 16-bit integer turns NaN into 0 by its
// definition; a zero scale (rk or sk = 0: nothing to store, and only zeros,
// infinities or NaN among the values) stores zeros; and the random fraction,
// a 16-bit integer times 2^-16, is exact, so one fused multiply-add rounds as
// the product's addition does.
__device__ __forceinline__ void v_requant_sr(float nr, float ns, float rk, float sk, uint32_t h, int16_t& q, uint16_t& w) {
    short a;
    unsigned short b;
    asm("cvt.rmi.sat.s16.f32 %0, %1;" : "=h"(a) : "f"(__fmaf_rn((float)(uint16_t)h, 0x1p-16f, nr * rk)));
    asm("cvt.rmi.sat.u16.f32 %0, %1;" : "=h"(b) : "f"(__fmaf_rn((float)(h >> 16), 0x1p-16f, fmaxf(ns, 0.0f) * sk)));
    q = rk > 0.0f ? a : (int16_t)0;
    w = sk > 0.0f ? b : (uint16_t)0;
}
__device__ __forceinline__ void v_requant(float nr, float ns, float rk, float sk, int16_t& q, uint16_t& w) {
    short a;
    unsigned short b;
    asm("cvt.rni.sat.s16.f32 %0, %1;" : "=h"(a) : "f"(nr * rk));
    asm("cvt.rni.sat.u16.f32 %0, %1;" : "=h"(b) : "f"(fmaxf(ns, 0.0f) * sk));
    q = rk > 0.0f ? a : (int16_t)0;
    w = sk > 0.0f ? b : (uint16_t)0;
}
// One hand's average strategy (cfr.rs:679-726).
template <int FMT, int NA, class T>
__device__ __forceinline__ void v_average_sigma(const T* s, float (&sig)[NA]) {
    if constexpr (FMT == kDevI16) {
        unsigned sum = 0, qv[NA];
#pragma unroll
        for (int k = 0; k < NA; k++) {
            qv[k] = (unsigned)s[k];
            sum += qv[k];
        }
        if (sum > 0) {
            const float inv = __frcp_rn((float)sum);
#pragma unroll
            for (int k = 0; k < NA; k++) sig[k] = (float)qv[k] * inv;
            return;
        }
    } else {
        double sum = 0.0;
        float v[NA];
#pragma unroll
        for (int k = 0; k < NA; k++) {
            v[k] = fmaxf(FMT == kDevF32 ? (float)s[k] : e4m3_to_f32((uint8_t)s[k]), 0.0f);
            sum += (double)v[k];
        }
        if (sum > 1e-12) {
#pragma unroll
            for (int k = 0; k < NA; k++) sig[k] = (float)((double)v[k] / sum);
            return;
        }
    }
#pragma unroll
    for (int k = 0; k < NA; k++) sig[k] = 1.0f / (float)NA;
}

// ------------------------------------------------------------- down sweep
// One warp per 32 V hands of a node: strategy x parent reach -> the children's
// reach (cfr.rs:469-531 push-down).  Bound by HBM: the strategy's source block
// and the parent's vector in, na vectors out.
enum VSrc { kVRegret = 0, kVPredicted = 1, kVAverage = 2 };
template <int FMT, int SRC, int NA, int V, class NODE>
__device__ __forceinline__ void v_down_node(const Dev& d, const Arenas& ar, const NODE& it, int i0) {
    using QR = std::conditional_t<FMT == kDevF32, float, typename QT<FMT == kDevFP8 ? kDevFP8 : kDevI16>::R>;
    using QS = std::conditional_t<FMT == kDevF32, float, typename QT<FMT == kDevFP8 ? kDevFP8 : kDevI16>::S>;
    const int a = (int)it.actor, nh = pick(d.nh, a);
    if (i0 >= nh) return;
    Pack<float, V> pr;
    pr.load(pick(d.reach, a) + (size_t)it.rslot * pick(d.rstr, a) + i0);
    const size_t e0 = it.aoff + (size_t)i0 * NA;
    Pack<QR, V * NA> r, pd;
    Pack<QS, V * NA> s;
    float kr = 0.0f, kp = 0.0f;
    if (SRC == kVAverage) {
        s.load((const QS*)pick(ar.str, a) + e0);
    } else {
        r.load((const QR*)pick(ar.reg, a) + e0);
        if (SRC == kVPredicted) {
            pd.load((const QR*)pick(ar.pred, a) + e0);
            if (FMT != kDevF32) {
                kr = pick(ar.rscale, a)[it.sidx] / QT<FMT == kDevFP8 ? kDevFP8 : kDevI16>::kR;
                kp = pick(ar.pscale, a)[it.sidx] / QT<FMT == kDevFP8 ? kDevFP8 : kDevI16>::kR;
            }
        }
    }
    const long long loff = pick(d.lock_off, a)[it.sidx];
    const int live = nh - i0;
    if (live < V) {
        pr.keep(live);
        r.keep(live * NA);
        pd.keep(live * NA);
        s.keep(live * NA);
    }
    Pack<float, V> out[NA];
#pragma unroll
    for (int u = 0; u < V; u++) {
        float sig[NA];
        if (loff >= 0) {
#pragma unroll
            for (int k = 0; k < NA; k++) sig[k] = u < live ? d.lock_sig[loff + (long long)k * nh + i0 + u] : 0.0f;
        } else if (SRC == kVAverage) {
            v_average_sigma<FMT, NA>(&s.e[u * NA], sig);
        } else {
            v_regret_sigma<FMT, NA, SRC == kVPredicted>(&r.e[u * NA], &pd.e[u * NA], kr, kp, sig);
        }
#pragma unroll
        for (int k = 0; k < NA; k++) out[k].e[u] = pr.e[u] * sig[k];
    }
#pragma unroll
    for (int k = 0; k < NA; k++)
        if (it.rs[k] != kNoSlot) out[k].store(pick(d.reach, a) + (size_t)it.rs[k] * pick(d.rstr, a) + i0);
}
template <int FMT, int SRC, int V, int KA>
__global__ void __launch_bounds__(128, V != 4 || KA != 4 || SRC == kVPredicted ? 1 : SRC == kVRegret ? kVDownCtas : 10) kv_down(Dev d, Arenas ar, const SNodeT<KA>* nodes, uint32_t count, uint32_t wn) {
    const uint32_t w = blockIdx.x * 4 + (threadIdx.x >> 5), n = w / wn;
    if (n >= count) return;
    const SNodeT<KA>& it = nodes[n];
    const uint32_t na = it.na;  // the record: constant, on its way while this waits
    pdl_enter();
    const int i0 = (int)((w - n * wn) * 32 + (threadIdx.x & 31)) * V;
#define V_CASE(NA)                                                                    \
    case NA:                                                                          \
        if (NA <= KA) v_down_node<FMT, SRC, NA <= KA ? NA : 1, V>(d, ar, it, i0);     \
        break;
    switch (na) {  // uniform per warp: one body per action count
        V_CASE(1) V_CASE(2) V_CASE(3) V_CASE(4) V_CASE(5) V_CASE(6) V_CASE(7) V_CASE(8)
    }
}

// --------------------------------------------------------------- up sweep
// The node's child values for this thread's hands: rows of cfv, and the fold
// child's value from its fold's summary (game.rs:487-496).
template <int NA, int V, class NODE>
__device__ __forceinline__ void v_children(const Dev& d, const NODE& it, int p, int i0, Pack<float, V> (&cv)[NA]) {
    const int nh = pick(d.nh, p), live = nh - i0, fk = (int)it.fk;
    if (live <= 0) {
#pragma unroll
        for (int k = 0; k < NA; k++) cv[k].zero();
        return;
    }
    uint32_t fold = 0, frs = 0;
#pragma unroll
    for (int k = 0; k < NA; k++) {
        if (k == fk) {
            cv[k].zero();
            fold = it.cs[k];
            frs = it.rs[k];
        } else {
            cv[k].load(d.cfv + (size_t)it.cs[k] * d.nh_max + i0);
        }
    }
    if (live < V) {
#pragma unroll
        for (int k = 0; k < NA; k++) cv[k].keep(live);
    }
    if (fk < 0) return;
    // the folding player's reach was written by the down sweep at an
    // opponent's node; at the traverser's it is the opponent's at the node
    const int o = 1 - p;
    const float* ro = pick(d.reach, o) + (size_t)((int)it.actor == p ? it.oslot : frs) * pick(d.rstr, o);
    const FoldSum* fs = d.folds + fold;
    const long long T = fs->T;
    const int sc = fs->sc;
    const float amount = (int)it.folder == p ? it.tlose : it.twin;
    Pack<uint32_t, V> hi;  // hand words are padded to whole groups of four
    hi.load(pick(d.hinfo, p) + i0);
#pragma unroll
    for (int u = 0; u < V; u++)
        if (u < live) {
            const uint32_t h = hi.e[u], sm = h >> 16;
            const float same_r = sm != 0xFFFFu ? ro[sm] : 0.0f;
            const float f = amount * (fix_f(T - fs->S[h & 63u] - fs->S[(h >> 6) & 63u], sc) + same_r);
#pragma unroll
            for (int k = 0; k < NA; k++)
                if (k == fk) cv[k].e[u] = f;
        }
}
template <int NA, int V, class NODE>
__device__ __forceinline__ void v_opp_node(const Dev& d, const NODE& it, int p, int i0) {
    if (i0 >= pick(d.nh, p)) return;
    Pack<float, V> cv[NA];
    v_children<NA, V>(d, it, p, i0, cv);
    Pack<float, V> out;
#pragma unroll
    for (int u = 0; u < V; u++) {
        float acc = 0.0f;
#pragma unroll
        for (int k = 0; k < NA; k++) acc += cv[k].e[u];
        out.e[u] = acc;
    }
    out.store(d.cfv + (size_t)it.cslot * d.nh_max + i0);
}
// The traverser's node: a locked node's value, an evaluation sweep's value
// (best_response.rs:69-121, 185-219), or the CFR update (cfr.rs:297-409) with
// the blocks and scales written back.
template <int FMT, int EVAL, bool PRED, bool WARP, int NA, int V, class NODE>
__device__ __forceinline__ void v_mine_node(const Dev& d, const Arenas& ar, const NODE& it, int p, int mode, int i0,
                                            const Group& g) {
    using Q = QT<FMT == kDevFP8 ? kDevFP8 : kDevI16>;
    using QR = std::conditional_t<FMT == kDevF32, float, typename Q::R>;
    using QS = std::conditional_t<FMT == kDevF32, float, typename Q::S>;
    const int nh = pick(d.nh, p), live = nh - i0;
    const bool on = live > 0;
    const size_t e0 = it.aoff + (size_t)i0 * NA;
    const long long loff = pick(d.lock_off, p)[it.sidx];
    Pack<QR, V * NA> r, pd;
    Pack<QS, V * NA> s;
    Pack<float, V> rp;
    r.zero();
    pd.zero();
    s.zero();
    rp.zero();
    float kr = 0.0f, kp = 0.0f, sscale = 0.0f;
    if (!EVAL) {
        if (on) {
            r.load((const QR*)pick(ar.reg, p) + e0);
            s.load((const QS*)pick(ar.str, p) + e0);
            if (PRED) pd.load((const QR*)pick(ar.pred, p) + e0);
            rp.load(pick(d.reach, p) + (size_t)it.rslot * pick(d.rstr, p) + i0);
        }
        if (FMT != kDevF32) {
            kr = pick(ar.rscale, p)[it.sidx] / Q::kR;
            if (PRED) kp = pick(ar.pscale, p)[it.sidx] / Q::kR;
            sscale = pick(ar.sscale, p)[it.sidx];
        }
    } else if (mode == 1 && on) {
        s.load((const QS*)pick(ar.str, p) + e0);
    }
    if (on && live < V) {
        r.keep(live * NA);
        pd.keep(live * NA);
        s.keep(live * NA);
        rp.keep(live);
    }
    Pack<float, V> cv[NA], out;
    v_children<NA, V>(d, it, p, i0, cv);
    float* outp = d.cfv + (size_t)it.cslot * d.nh_max + i0;
    if (loff >= 0 || EVAL) {
        if (!on) return;
#pragma unroll
        for (int u = 0; u < V; u++) {
            float acc = 0.0f;
            if (loff >= 0) {  // locked: fixed sigma, no update
                if (u < live) {
#pragma unroll
                    for (int k = 0; k < NA; k++) acc += d.lock_sig[loff + (long long)k * nh + i0 + u] * cv[k].e[u];
                }
            } else if (mode == 0) {
                acc = cv[0].e[u];
#pragma unroll
                for (int k = 1; k < NA; k++)
                    if (cv[k].e[u] > acc) acc = cv[k].e[u];
            } else {
                float sig[NA];
                v_average_sigma<FMT, NA>(&s.e[u * NA], sig);
#pragma unroll
                for (int k = 0; k < NA; k++) acc += sig[k] * cv[k].e[u];
            }
            out.e[u] = acc;
        }
        out.store(outp);
        return;
    }
    const float pos = d.disc[0], neg = d.disc[1], ds = d.disc[2];
    if (FMT == kDevF32) {
        if (!on) return;
#pragma unroll
        for (int u = 0; u < V; u++) {
            float sig[NA];
            v_regret_sigma<FMT, NA, PRED>(&r.e[u * NA], &pd.e[u * NA], 0.0f, 0.0f, sig);
            float o_ = 0.0f;
#pragma unroll
            for (int k = 0; k < NA; k++) o_ += sig[k] * cv[k].e[u];
#pragma unroll
            for (int k = 0; k < NA; k++) {
                const int b = u * NA + k;
                const float x = (float)r.e[b], dv = cv[k].e[u] - o_;
                r.e[b] = (QR)(x * (x > 0.0f ? pos : neg) + dv);
                s.e[b] = (QS)((float)s.e[b] * ds + rp.e[u] * sig[k]);
                if (PRED) pd.e[b] = (QR)dv;
            }
            out.e[u] = o_;
        }
        out.store(outp);
        r.store((QR*)pick(ar.reg, p) + e0);
        s.store((QS*)pick(ar.str, p) + e0);
        if (PRED) pd.store((QR*)pick(ar.pred, p) + e0);
        return;
    }
    // Quantised arenas (cfr.rs:350-407): the new f32 values stay in registers
    // between the maxima and the requantisation.
    const float kss = sscale / Q::kS * ds;
    float nr[V * NA], ns[V * NA], dv[V * NA];
    float mx[3] = {0.0f, 0.0f, 0.0f};
    if (on)
#pragma unroll
    for (int u = 0; u < V; u++) {
        float sig[NA];
        v_regret_sigma<FMT, NA, PRED>(&r.e[u * NA], &pd.e[u * NA], kr, kp, sig);
        float o_ = 0.0f;
#pragma unroll
        for (int k = 0; k < NA; k++) o_ += sig[k] * cv[k].e[u];
#pragma unroll
        for (int k = 0; k < NA; k++) {
            const int b = u * NA + k;
            const float x = Q::dr((typename Q::R)r.e[b]);  // the discount follows the stored sign
            const float dk = cv[k].e[u] - o_;
            nr[b] = x * kr * (x > 0.0f ? pos : neg) + dk;
            ns[b] = Q::ds((typename Q::S)s.e[b]) * kss + rp.e[u] * sig[k];
            if (PRED) dv[b] = dk;
            mx[0] = fmaxf(mx[0], fabsf(nr[b]));
            mx[1] = fmaxf(mx[1], ns[b]);
            if (PRED) mx[2] = fmaxf(mx[2], fabsf(dk));
        }
        out.e[u] = o_;
    }
    if (on) out.store(outp);
    if (PRED) {
        group_max<WARP>(g, mx);
    } else {
        float m2[2] = {mx[0], mx[1]};
        group_max<WARP>(g, m2);
        mx[0] = m2[0];
        mx[1] = m2[1];
    }
    const bool rok = mx[0] > 0.0f && isfinite(mx[0]), sok = mx[1] > 0.0f && isfinite(mx[1]),
               pok = mx[2] > 0.0f && isfinite(mx[2]);
    const float rk = rok ? Q::kR / mx[0] : 0.0f, sk = sok ? Q::kS / mx[1] : 0.0f, pk = pok ? Q::kR / mx[2] : 0.0f;
    const uint32_t sr_b = ar.sr ? sr_base(pick(d.node_id, p)[it.sidx], *d.iter) : 0u;
    if (on) {
#pragma unroll
        for (int u = 0; u < V; u++)
#pragma unroll
            for (int k = 0; k < NA; k++) {
                const int b = u * NA + k;
                if (FMT == kDevI16) {
                    int16_t q;
                    uint16_t w;
                    if (ar.sr) v_requant_sr(nr[b], ns[b], rk, sk, sr_bits(sr_b, (uint32_t)(i0 + u), (uint32_t)k), q, w);
                    else v_requant(nr[b], ns[b], rk, sk, q, w);
                    r.e[b] = (QR)q;
                    s.e[b] = (QS)w;
                } else {
                    r.e[b] = (QR)(rk > 0.0f ? Q::er(nr[b] * rk) : (typename Q::R)0);
                    s.e[b] = (QS)(sk > 0.0f ? Q::es(fmaxf(ns[b], 0.0f) * sk) : (typename Q::S)0);
                }
                if (PRED) pd.e[b] = (QR)(pk > 0.0f ? Q::er(dv[b] * pk) : (typename Q::R)0);
            }
        if (live < V) {
            r.keep(live * NA);
            s.keep(live * NA);
            if (PRED) pd.keep(live * NA);
        }
        r.store((QR*)pick(ar.reg, p) + e0);
        s.store((QS*)pick(ar.str, p) + e0);
        if (PRED) pd.store((QR*)pick(ar.pred, p) + e0);
    }
    if (g.t == 0) {
        pick(ar.rscale, p)[it.sidx] = rok ? mx[0] : 0.0f;
        pick(ar.sscale, p)[it.sidx] = sok ? mx[1] : 0.0f;
        if (PRED) pick(ar.pscale, p)[it.sidx] = pok ? mx[2] : 0.0f;
    }
}

// Nodes whose hands do not depend on one another (the opponent's nodes,
// evaluation sweeps, f32 arenas): one warp per 32 V hands, wn warps per node.
template <int V, int KA>
__global__ void __launch_bounds__(128, V == 4 && KA == 4 ? kVOppCtas : 1) kv_up_opp(Dev d, const SNodeT<KA>* nodes, uint32_t count, uint32_t wn, int p) {
    const uint32_t w = blockIdx.x * 4 + (threadIdx.x >> 5), n = w / wn;
    if (n >= count) return;
    const SNodeT<KA>& it = nodes[n];
    const uint32_t na = it.na;  // the record: constant, on its way while this waits
    pdl_enter();
    const int i0 = (int)((w - n * wn) * 32 + (threadIdx.x & 31)) * V;
#undef V_CASE
#define V_CASE(NA)                                                    \
    case NA:                                                          \
        if (NA <= KA) v_opp_node<NA <= KA ? NA : 1, V>(d, it, p, i0); \
        break;
    switch (na) {
        V_CASE(1) V_CASE(2) V_CASE(3) V_CASE(4) V_CASE(5) V_CASE(6) V_CASE(7) V_CASE(8)
    }
}
template <int FMT, int EVAL, bool PRED, int V, int KA>
__global__ void __launch_bounds__(128, V == 4 && KA == 4 && !PRED ? kVMineCtas : 1) kv_up_mine(Dev d, Arenas ar, const SNodeT<KA>* nodes, uint32_t count, uint32_t wn,
                                                  int p, int mode) {
    static_assert(EVAL || FMT == kDevF32, "a quantised update needs the node's maxima");
    const uint32_t w = blockIdx.x * 4 + (threadIdx.x >> 5), n = w / wn;
    if (n >= count) return;
    const SNodeT<KA>& it = nodes[n];
    const uint32_t na = it.na;  // the record: constant, on its way while this waits
    pdl_enter();
    const int i0 = (int)((w - n * wn) * 32 + (threadIdx.x & 31)) * V;
#undef V_CASE
#define V_CASE(NA)                                                                                               \
    case NA:                                                                                                     \
        if (NA <= KA) v_mine_node<FMT, EVAL, PRED, true, NA <= KA ? NA : 1, V>(d, ar, it, p, mode, i0, Group{}); \
        break;
    switch (na) {
        V_CASE(1) V_CASE(2) V_CASE(3) V_CASE(4) V_CASE(5) V_CASE(6) V_CASE(7) V_CASE(8)
    }
}
// Updates of quantised arenas: one warp per node (WARP), or one CTA of at most
// 11 warps (V = 4) or 21 (V = 2: 96 registers a thread still fit an SM).
template <int FMT, bool PRED, bool WARP, int V, int KA>
__global__ void __maxnreg__(WARP ? 168 : V == 2 ? 96 : KA == 4 ? kVQuantRegs : 160)
    kv_up_quant(Dev d, Arenas ar, const SNodeT<KA>* nodes, uint32_t count, int p) {
    __shared__ uint32_t red[WARP ? 1 : 3 * kVMaxWarps];
    const uint32_t n = WARP ? blockIdx.x * 4 + (threadIdx.x >> 5) : blockIdx.x;
    if (n >= count) return;
    const SNodeT<KA>& it = nodes[n];
    const uint32_t na = it.na;  // the record: constant, on its way while this waits
    pdl_enter();
    const Group g{(int)(WARP ? threadIdx.x & 31 : threadIdx.x), (int)(blockDim.x >> 5), red};
#undef V_CASE
#define V_CASE(NA)                                                                                        \
    case NA:                                                                                              \
        if (NA <= KA) v_mine_node<FMT, 0, PRED, WARP, NA <= KA ? NA : 1, V>(d, ar, it, p, 0, g.t * V, g); \
        break;
    switch (na) {
        V_CASE(1) V_CASE(2) V_CASE(3) V_CASE(4) V_CASE(5) V_CASE(6) V_CASE(7) V_CASE(8)
    }
}

template <int N>
using IntC = std::integral_constant<int, N>;
// Hands per lane of the forms whose warps are independent: four, unless the
// node is smaller, or the launch too small to fill the device with warps of
// 128 hands -- then fewer hands a lane shorten the one wave there is.
inline int lane_hands(int nh, uint32_t count) {
    if (nh <= 32) return 1;
    const uint64_t w4 = (uint64_t)count * (uint32_t)((nh + 127) / 128);
    if (w4 <= kVFillWarps / 4) return 1;
    if (nh <= 64 || w4 <= kVFillWarps / 2) return 2;
    return 4;
}
// f(V, warps per node, grid) for a launch of count nodes of nh hands
template <class F>
void with_lanes(int nh, uint32_t count, F f) {
    auto go = [&](auto V) {
        const uint32_t wn = (uint32_t)((nh + 32 * V() - 1) / (32 * V()));
        f(V, wn, (unsigned)(((uint64_t)count * wn + 3) / 4));
    };
    const int v = lane_hands(nh, count);
    if (v == 1) go(IntC<1>{});
    else if (v == 2) go(IntC<2>{});
    else go(IntC<4>{});
}

// The launches of one arena format.
template <int FMT, int KA>
void down_t(const Dev& d, const Arenas& ar, const VecNodes& n, int nh, int mode, cudaStream_t s) {
    const auto* nodes = (const SNodeT<KA>*)n.nodes;
    with_lanes(nh, n.count, [&](auto V, uint32_t wn, unsigned grid) {
        constexpr int v = V();
        if (mode) pdl_launch(kv_down<FMT, kVAverage, v, KA>, grid, 128, 0, s, d, ar, nodes, n.count, wn);
        else if (ar.pred[0]) pdl_launch(kv_down<FMT, kVPredicted, v, KA>, grid, 128, 0, s, d, ar, nodes, n.count, wn);
        else pdl_launch(kv_down<FMT, kVRegret, v, KA>, grid, 128, 0, s, d, ar, nodes, n.count, wn);
    });
}
template <int FMT, int KA>
void up_mine_t(const Dev& d, const Arenas& ar, const VecNodes& n, int p, int eval, cudaStream_t s) {
    const auto* nodes = (const SNodeT<KA>*)n.nodes;
    const int nh = d.nh[p];
    if (eval >= 0 || FMT == kDevF32) {
        with_lanes(nh, n.count, [&](auto V, uint32_t wn, unsigned grid) {
            constexpr int v = V();
            if (eval >= 0) {
                pdl_launch(kv_up_mine<FMT, 1, false, v, KA>, grid, 128, 0, s, d, ar, nodes, n.count, wn, p, eval);
            } else if constexpr (FMT == kDevF32) {
                if (ar.pred[0]) pdl_launch(kv_up_mine<FMT, 0, true, v, KA>, grid, 128, 0, s, d, ar, nodes, n.count, wn, p, 0);
                else pdl_launch(kv_up_mine<FMT, 0, false, v, KA>, grid, 128, 0, s, d, ar, nodes, n.count, wn, p, 0);
            }
        });
        return;
    }
    if constexpr (FMT != kDevF32) {
        auto go = [&](auto WP, auto V) {
            constexpr bool W = WP();
            constexpr int v = V();
            const unsigned grid = W ? (n.count + 3) / 4 : n.count;
            const unsigned block = W ? 128u : (unsigned)((nh + 32 * v - 1) / (32 * v)) * 32u;
            if (ar.pred[0]) pdl_launch(kv_up_quant<FMT, true, W, v, KA>, grid, block, 0, s, d, ar, nodes, n.count, p);
            else pdl_launch(kv_up_quant<FMT, false, W, v, KA>, grid, block, 0, s, d, ar, nodes, n.count, p);
        };
        // small launches: a CTA per node with fewer hands a thread
        const bool small = (uint64_t)n.count * (uint32_t)((nh + 127) / 128) <= kVFillWarps / 2;
        if (nh <= 32) go(std::true_type{}, IntC<1>{});
        else if (nh <= 64) go(std::true_type{}, IntC<2>{});
        else if (nh <= 128 && !small) go(std::true_type{}, IntC<4>{});
        else if (small) go(std::false_type{}, IntC<2>{});
        else go(std::false_type{}, IntC<4>{});
    }
}
template <int KA>
void up_opp_t(const Dev& d, const VecNodes& n, int p, cudaStream_t s) {
    with_lanes(d.nh[p], n.count, [&](auto V, uint32_t wn, unsigned grid) {
        constexpr int v = V();
        pdl_launch(kv_up_opp<v, KA>, grid, 128, 0, s, d, (const SNodeT<KA>*)n.nodes, n.count, wn, p);
    });
}
}  // namespace

}  // namespace gtob
