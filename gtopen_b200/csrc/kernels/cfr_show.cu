// Showdown and chance kernels of the level sweeps (the default engine).
//
// kv_show: one CTA evaluates G showdowns of one river board at once
// (game.rs:501-577 with the plan's rank tables), all of a sweep's showdowns
// in one launch -- they read only reach vectors, so no level waits for
// another.  Exact sums (cfr_dev.cuh), so the split changes no bits.
//
// What bounds it and why this layout: a hand's value needs eight prefix sums
// at positions of its own (strength order below / not above it, its two
// cards' lists likewise, the two cards' totals), i.e. eight scattered
// shared-memory reads, and shared-memory wavefronts and the instructions
// around them set the time (470 v 647 hands: LSU wavefronts 67% and issue 52%
// of their peaks, DRAM 9%).
//   * The G showdowns of a board use the same positions, so the prefixes lie
//     row by row with the G sums side by side and a lane takes two showdowns
//     (one 16-byte access): at G = 8 a quarter warp reads whole rows.
//   * The segmented scan over [strength order | card lists] keeps a lane's K
//     entries in registers (K up to 16) until its carry is known, so every
//     row is written once.
//   * The fewest threads whose lanes hold the scan, then the largest G: the
//     per-warp work (shuffles, carries, address set-up) is paid by fewer
//     warps.  Measured, ms per iteration for both sweeps (threads x G):
//     28 v 23 hands 32x8 0.070, 64x8 0.080, 128x8 0.111, 64x2 0.199; 64 v 39 hands 64x8
//     0.246, 128x8 0.288, 64x2 0.443; 243 v 321 64x2 2.35, 128x4 2.43, 256x8
//     2.70; 470 v 647 128x2 1.45, 256x4 1.65, 512x8 2.12.
// Showdowns of one iteration before (two at a time, one launch per level,
// chunks rewritten after the scan) -> after: 28 v 23 hands 0.41 -> 0.08 ms,
// 64 v 39 0.87 -> 0.25, 243 v 321 3.21 -> 2.35, 470 v 647 2.25 -> 1.45, a turn
// of 3,696 showdowns 0.43 -> 0.066, a river 0.14 -> 0.026.
//
// kv_chance, kv_edges: a chance node's value and its edges' reach, one hand
// (four, for the edges) per thread, so that a level of a few nodes still
// spreads over the chip: a node's 48 children used to be read one after the
// other by one CTA per node, 60-85 us a level however few its nodes.  Both
// are bound by the latency of their loads on small levels and by HBM on
// large ones.  One iteration, before -> after: chance values of a 564-hand
// turn 0.47 -> 0.09 ms, of a 470 v 647 flop 1.00 -> 0.26; the flop's edges
// 0.27 -> 0.19.
#include "cfr_vec.hpp"

#include <type_traits>

namespace gtob {
namespace {

// A board's scan entries: the opponent's hands in strength order (m), then
// card by card each list of the hands holding the card, in strength order
// (2 m); bit 15 marks the first entry of the strength order and of each list.
// Lanes scan K consecutive entries each; entry f's running sum goes to row
// f + 1 + f / K (a row left free per K entries spreads the lanes' stores over
// the banks), row 0 is zero: the empty prefix of every list.
__host__ __device__ inline int show_entries(int m, int K) { return (3 * m + K - 1) / K * K; }
__host__ __device__ inline int show_rows(int m, int K) { return show_entries(m, K) / K * (K + 1) + 1; }
__host__ __device__ inline int show_img_len(int msort, int K) { return (show_entries(msort, K) + 7) & ~7; }
__device__ __forceinline__ int show_row(int entries, int K) {  // the row of the sum of a list's entries up to `entries`
    return entries + (entries - 1) / K;
}
struct ShowLayout {
    unsigned o_r, o_img, total;
    __host__ __device__ ShowLayout(int G, int K, int msort, int nho_pad) {
        o_r = (unsigned)show_rows(msort, K) * (unsigned)G * 8u;
        o_img = o_r + (unsigned)nho_pad * (unsigned)G * 4u;  // nho_pad is a multiple of 4
        total = o_img + (unsigned)show_img_len(msort, K) * 2u;
    }
};

// Per board and traverser hand: the rows of its eight sums (strictly weaker
// and not stronger hands; the same for each of its cards' lists; the lists'
// totals); s1 of a blocked hand: 0xFFFF.
struct alignas(16) HandRank {
    uint16_t lb, ub, q1lo, q1hi, q2lo, q2hi, s1, s2;
};

// A vector's scaling onto its grid and back (fix_q, fix_f).  Up to S = 126
// one multiplication does what their two-step form does: the power of two is
// a normal number, the way to the grid is exact, and the way back rounds
// once.  BIG: some lane's vector is smaller than that.
struct Grid {
    int S;
    float up, down;
};
__device__ __forceinline__ Grid make_grid(float mx) {
    Grid g;
    g.S = fix_scale(mx);
    g.up = pow2f(min(g.S, 126));
    g.down = pow2f(-min(g.S, 126));
    return g;
}
template <bool BIG>
__device__ __forceinline__ long long grid_q(const Grid& g, float r) {
    return BIG ? fix_q(r, g.S) : __float2ll_rn(__fmul_rn(r, g.up));
}
template <bool BIG>
__device__ __forceinline__ float grid_f(const Grid& g, long long v) {
    return BIG ? fix_f(v, g.S) : __fmul_rn(__ll2float_rn(v), g.down);
}
struct ShowPay {
    float win, lose, tie;
};
// One hand's value from its integer sums (game.rs:560-575).
template <bool BIG>
__device__ __forceinline__ float show_value(const Grid& g, const ShowPay& pay, long long low, long long notabove,
                                            long long all, float same) {
    const float lower = grid_f<BIG>(g, low);
    const float higher = grid_f<BIG>(g, all - notabove);
    const float valid = grid_f<BIG>(g, all) + same;
    const float tied = valid - lower - higher;
    return pay.win * lower + pay.lose * higher + pay.tie * tied;
}
__device__ __forceinline__ longlong2 shfl_up2(const longlong2& v, int x) {
    return make_longlong2(__shfl_up_sync(0xffffffffu, v.x, x), __shfl_up_sync(0xffffffffu, v.y, x));
}

template <int G, int NT, int K, bool BIG>
__device__ __forceinline__ void show_group(const Dev& d, unsigned char* sm, const ShowLayout& SL, const ShowItem* s_it,
                                           longlong2* s_w, int* s_wf, const Grid& ga, const Grid& gb, int m, int nhp,
                                           const HandRank* hr, const uint32_t* hinfo) {
    constexpr int L = G / 2, NC = NT / L, NW = NT / 32;
    const int tid = (int)threadIdx.x, l = tid & (L - 1), c_ = tid / L, lane = tid & 31, warp = tid >> 5;
    longlong2* U = (longlong2*)sm + l;  // row k: U[k * L]
    const float2* r2 = (const float2*)(sm + SL.o_r) + l;
    // the lane's K entries: running sums since the last list head
    const bool on = c_ * K < 3 * m;
    longlong2 a = make_longlong2(0, 0), loc[K];
    int first = K;  // the first head among them
    if (on) {
        const uint2* ent = (const uint2*)(sm + SL.o_img) + c_ * (K / 4);
#pragma unroll
        for (int k = 0; k < K; k += 4) {
            const uint2 w = ent[k / 4];
            const uint32_t e[4] = {w.x & 0xFFFFu, w.x >> 16, w.y & 0xFFFFu, w.y >> 16};
            float2 x[4];
#pragma unroll
            for (int j = 0; j < 4; j++) x[j] = r2[(e[j] & 0x7FFFu) * L];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (e[j] & 0x8000u) {
                    a = make_longlong2(0, 0);
                    first = min(first, k + j);
                }
                a.x += grid_q<BIG>(ga, x[j].x);
                a.y += grid_q<BIG>(gb, x[j].y);
                loc[k + j] = a;
            }
        }
    }
    // scan of the lanes' (head seen, sum) pairs over the lanes with this l
    bool fl = first < K;
#pragma unroll
    for (int x = L; x < 32; x <<= 1) {
        const int fu = __shfl_up_sync(0xffffffffu, (int)fl, x);
        const longlong2 u = shfl_up2(a, x);
        if (lane >= x) {
            if (!fl) {
                a.x += u.x;
                a.y += u.y;
            }
            fl = fl || fu;
        }
    }
    longlong2 c = shfl_up2(a, L);  // what the warp's lanes before this one carry over
    bool cf = __shfl_up_sync(0xffffffffu, (int)fl, L) != 0;
    if (lane < L) {
        c = make_longlong2(0, 0);
        cf = false;
    }
    if (lane >= 32 - L) {
        s_w[warp * L + l] = a;
        if (l == 0) s_wf[warp] = (int)fl;
    }
    __syncthreads();
    if (!cf) {  // and the warps before it, back to the last head
#pragma unroll
        for (int w = NW - 2; w >= 0; w--) {
            if (w < warp && !cf) {
                const longlong2 u = s_w[w * L + l];
                c.x += u.x;
                c.y += u.y;
                cf = s_wf[w] != 0;
            }
        }
    }
    if (tid < L) *U = make_longlong2(0, 0);
    if (on) {
        longlong2* dst = U + (c_ * (K + 1) + 1) * L;
#pragma unroll
        for (int k = 0; k < K; k++) {
            longlong2 v = loc[k];
            if (k < first) {
                v.x += c.x;
                v.y += c.y;
            }
            dst[k * L] = v;
        }
    }
    __syncthreads();
    // values, in hand order: a warp's rows of output are whole sectors
    const ShowItem &ia = s_it[2 * l], &ib = s_it[2 * l + 1];
    float* outA = d.cfv + (size_t)ia.cslot * d.nh_max;
    float* outB = d.cfv + (size_t)ib.cslot * d.nh_max;
    const bool onA = ia.cslot != kNoSlot, onB = ib.cslot != kNoSlot;
    const ShowPay pa{ia.twin, ia.tlose, ia.ttie}, pb{ib.twin, ib.tlose, ib.ttie};
    const longlong2 T = U[m > 0 ? show_row(m, K) * L : 0];
    HandRank next;
    uint32_t nexth = 0;
    if (c_ < nhp) {
        next = hr[c_];
        nexth = hinfo[c_];
    }
    for (int i = c_; i < nhp; i += NC) {
        const HandRank e = next;
        const uint32_t same = nexth >> 16;
        if (i + NC < nhp) {  // in flight during this hand's sums
            next = hr[i + NC];
            nexth = hinfo[i + NC];
        }
        float vA = 0.0f, vB = 0.0f;  // a blocked hand's value
        if (e.s1 != 0xFFFFu) {
            const longlong2 plb = U[(int)e.lb * L], pub = U[(int)e.ub * L], q1l = U[(int)e.q1lo * L],
                            q1h = U[(int)e.q1hi * L], q2l = U[(int)e.q2lo * L], q2h = U[(int)e.q2hi * L],
                            s1 = U[(int)e.s1 * L], s2 = U[(int)e.s2 * L];
            float2 sr = make_float2(0.0f, 0.0f);
            if (same != 0xFFFFu) sr = r2[(int)same * L];
            vA = show_value<BIG>(ga, pa, plb.x - q1l.x - q2l.x, pub.x - q1h.x - q2h.x, T.x - s1.x - s2.x, sr.x);
            vB = show_value<BIG>(gb, pb, plb.y - q1l.y - q2l.y, pub.y - q1h.y - q2h.y, T.y - s1.y - s2.y, sr.y);
        }
        if (onA) outA[i] = vA;
        if (onB) outB[i] = vB;
    }
}

// A vector of a batch of G into the interleaved rows r[hand * G + g] (g the
// thread's vector), four hands a load; returns the largest value's bits over
// this thread's hands.
template <int G, int NT>
__device__ __forceinline__ uint32_t stage_interleaved(const float* src, bool live, int nho, int nho_pad, float* r) {
    const int q4 = nho_pad >> 2, tid = (int)threadIdx.x, g = tid & (G - 1);
    uint32_t mx = 0u;
    for (int q = tid / G; q < q4; q += NT / G) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live) v = ((const float4*)src)[q];
        const float x[4] = {v.x, 4 * q + 1 < nho ? v.y : 0.0f, 4 * q + 2 < nho ? v.z : 0.0f,
                            4 * q + 3 < nho ? v.w : 0.0f};
        mx = max(mx, __float_as_uint(fmaxf(fmaxf(fmaxf(x[0], 0.0f), x[1]), fmaxf(fmaxf(x[2], 0.0f), x[3]))));
#pragma unroll
        for (int j = 0; j < 4; j++) {  // rotated so that the warp's quads write different banks
            const int k = (j + q) & 3;
            const float y = k == 0 ? x[0] : k == 1 ? x[1] : k == 2 ? x[2] : x[3];
            r[(4 * q + k) * G + g] = y;
        }
    }
    return mx;
}

template <int G, int NT, int K>
__global__ void __launch_bounds__(NT) kv_show(Dev d, const ShowItem* items, const uint16_t* img, const HandRank* ranks,
                                              int p, int msort) {
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ longlong2 s_w[NT / 32 * (G / 2)];
    __shared__ int s_wf[NT / 32];
    __shared__ uint32_t s_mx[G];
    __shared__ ShowItem s_it[G];
    const int o = 1 - p, nho = pick(d.nh, o), nhp = pick(d.nh, p);
    const int nho_pad = (nho + 3) & ~3;
    const ShowLayout SL(G, K, msort, nho_pad);
    const int tid = (int)threadIdx.x, il = show_img_len(msort, K);
    const int g = tid & (G - 1);
    const ShowItem it = items[(size_t)blockIdx.x * G + g];  // (every thread: its own vector's; the slot is the batch's)
    if (tid < G) {
        s_mx[tid] = 0u;
        s_it[tid] = it;
    }
    const uint32_t slot = it.slot;
    const int m = (int)pick(d.sorted_cnt, o)[slot];
    {  // the board's entries
        const uint4* src = (const uint4*)(img + (size_t)slot * il);
        uint4* im = (uint4*)(sm + SL.o_img);
        for (int k = tid; k < il / 8; k += NT) im[k] = src[k];
    }
    pdl_enter();  // items, images and ranks are constant; reach is not
    uint32_t mx = stage_interleaved<G, NT>(pick(d.reach, o) + (size_t)it.rs[o] * pick(d.rstr, o), it.cslot != kNoSlot, nho,
                                           nho_pad, (float*)(sm + SL.o_r));
#pragma unroll
    for (int x = G; x < 32; x <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, x));
    __syncthreads();
    if ((tid & 31) < G) atomicMax(&s_mx[g], mx);
    __syncthreads();
    const int l = tid & (G / 2 - 1);
    const Grid ga = make_grid(__uint_as_float(s_mx[2 * l])), gb = make_grid(__uint_as_float(s_mx[2 * l + 1]));
    const HandRank* hr = ranks + (size_t)slot * nhp;
    // every warp holds every lane number l, so all warps agree
    if (__any_sync(0xffffffffu, ga.S > 126 || gb.S > 126))
        show_group<G, NT, K, true>(d, sm, SL, s_it, s_w, s_wf, ga, gb, m, nhp, hr, pick(d.hinfo, p));
    else
        show_group<G, NT, K, false>(d, sm, SL, s_it, s_w, s_wf, ga, gb, m, nhp, hr, pick(d.hinfo, p));
}

// ------------------------------------------------------------------- folds
// The sweep's fold summaries: G folds a CTA, their opponent vectors
// interleaved as in kv_show, a lane per card list and pair of folds.  Every
// fold of a player uses the same card lists, so a row of the interleaved
// vectors serves all of them.  Inside the up kernels these sums took three
// block barriers and a third of the traverser's instructions per node; as one
// launch beside the showdowns the opponent's nodes and f32 updates need no
// barrier at all.  470 v 647 hands, 85,413 folds: 0.13 and 0.15 ms a sweep (issue
// 73-75% of peak, 40 registers, 70% of the warps).  One iteration before -> after: that flop,
// 16-bit, 3.9 -> 3.7 ms; turn f32 0.364 -> 0.291; river f32 0.072 -> 0.058.
// threads: 52 card lists x 4 lanes (8 folds) x 2 halves of a list, and 26 x 16
// lanes (32 folds), are 416 -- every thread has a list; a launch that fills
// the device is faster without the halves' extra steps
template <int G, int PARTS>
constexpr int fold_threads() { return G == 8 && PARTS == 1 ? 256 : 416; }
// folds per CTA: short lists leave a CTA of 8 with more set-up than sums
inline int fold_group(int nho) { return nho <= 128 ? 32 : 8; }
template <int G, int PARTS>
__global__ void __launch_bounds__(fold_threads<G, PARTS>()) kv_folds(Dev d, const uint32_t* slots, uint32_t count, int p,
                                                         FoldSum* out) {
    constexpr int L = G / 2, NT = fold_threads<G, PARTS>(), NC = NT / L / PARTS;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ uint32_t s_mx[G];
    __shared__ longlong2 s_S[52 * L];
    const int o = 1 - p, nho = pick(d.nh, o), nho_pad = (nho + 3) & ~3;
    const int tid = (int)threadIdx.x, g = tid & (G - 1);
    const uint32_t f0 = blockIdx.x * G, fg = f0 + (uint32_t)g;
    if (tid < G) s_mx[tid] = 0u;
    const float* src = pick(d.reach, o) + (size_t)(fg < count ? slots[fg] : 0u) * pick(d.rstr, o);
    pdl_enter();
    uint32_t mx = stage_interleaved<G, NT>(src, fg < count, nho, nho_pad, (float*)sm);
#pragma unroll
    for (int x = G; x < 32; x <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, x));
    __syncthreads();
    if ((tid & 31) < G) atomicMax(&s_mx[g], mx);
    __syncthreads();
    const int l = tid & (L - 1), part = tid / L % PARTS, c_ = tid / (L * PARTS);
    const Grid ga = make_grid(__uint_as_float(s_mx[2 * l])), gb = make_grid(__uint_as_float(s_mx[2 * l + 1]));
    const uint32_t fa = f0 + 2 * (uint32_t)l;
    const bool onA = fa < count, onB = fa + 1 < count;
    const uint16_t* idx = pick(d.hcard_idx, o);
    for (int c = c_; c < 52; c += NC) {
        const uint32_t b = pick(d.hcard_off, o)[c], e = pick(d.hcard_off, o)[c + 1];
        const float2* r2 = (const float2*)sm + l;
        longlong2 a = make_longlong2(0, 0);
        const bool big = ga.S > 126 || gb.S > 126;
#pragma unroll 4
        for (uint32_t k = b + part; k < e; k += PARTS) {
            const float2 x = r2[(int)idx[k] * L];
            a.x += big ? grid_q<true>(ga, x.x) : grid_q<false>(ga, x.x);
            a.y += big ? grid_q<true>(gb, x.y) : grid_q<false>(gb, x.y);
        }
        if (PARTS == 2) {  // the other half's lane (every warp is whole here: one round)
            a.x += __shfl_xor_sync(0xffffffffu, a.x, L);
            a.y += __shfl_xor_sync(0xffffffffu, a.y, L);
        }
        if (part == 0) {
            s_S[c * L + l] = a;
            if (onA) out[fa].S[c] = a.x;
            if (onB) out[fa + 1].S[c] = a.y;
        }
    }
    __syncthreads();
    if (tid < 32) {  // every hand holds two cards: the total is half the card sums' sum
        longlong2 t = make_longlong2(0, 0);
        for (int k = tid / L; k < 52; k += 32 / L) {
            t.x += s_S[k * L + l].x;
            t.y += s_S[k * L + l].y;
        }
#pragma unroll
        for (int x = L; x < 32; x <<= 1) {
            t.x += __shfl_xor_sync(0xffffffffu, t.x, x);
            t.y += __shfl_xor_sync(0xffffffffu, t.y, x);
        }
        if (tid < L) {
            if (onA) {
                out[fa].T = t.x >> 1;
                out[fa].sc = ga.S;
            }
            if (onB) {
                out[fa + 1].T = t.y >> 1;
                out[fa + 1].sc = gb.S;
            }
        }
    }
}

// The boards' rank entries by hand, for kv_show (once per engine).
__global__ void k_hand_ranks(Dev d, int p, int K, HandRank* out) {
    const uint32_t slot = blockIdx.x;
    const int nh = pick(d.nh, p), o = 1 - p;
    HandRank* row = out + (size_t)slot * nh;
    for (int i = threadIdx.x; i < nh; i += blockDim.x) row[i] = HandRank{0, 0, 0, 0, 0, 0, 0xFFFF, 0};
    __syncthreads();
    const RankEntry* in = pick(d.rank, p) + pick(d.rank_off, p)[slot];
    const uint32_t cnt = pick(d.rank_cnt, p)[slot];
    const uint32_t* coff = pick(d.ccard_off, o) + (size_t)slot * 53;
    const int m = (int)pick(d.sorted_cnt, o)[slot];
    for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x) {
        const RankEntry e = in[k];
        const int c1 = e.cards & 0xFF, c2 = e.cards >> 8;
        auto strength = [&](int n) { return (uint16_t)(n ? show_row(n, K) : 0); };
        // the plan counts a card's prefixes from its offset + card number
        auto list = [&](int c, int n) { return (uint16_t)(n ? show_row(m + (int)(coff[c] - coff[0]) + n, K) : 0); };
        auto prefix = [&](int c, int q) { return list(c, q - (int)(coff[c] - coff[0]) - c); };
        auto total = [&](int c) { return list(c, (int)(coff[c + 1] - coff[c])); };
        row[e.idx] = HandRank{strength(e.lb),    strength(e.ub),    prefix(c1, e.q1lo), prefix(c1, e.q1hi),
                              prefix(c2, e.q2lo), prefix(c2, e.q2hi), total(c1),          total(c2)};
    }
}
// Every board's scan entries of player o's hands.
__global__ void k_show_images(Dev d, int o, int msort, int K, uint16_t* out) {
    const uint32_t slot = blockIdx.x;
    const int il = show_img_len(msort, K), m = (int)pick(d.sorted_cnt, o)[slot];
    uint16_t* im = out + (size_t)slot * il;
    const uint32_t* coff = pick(d.ccard_off, o) + (size_t)slot * 53;
    const uint16_t* order = pick(d.sorted_idx, o) + pick(d.sorted_off, o)[slot];
    const uint8_t* card = pick(d.ccard_card, o) + coff[0];
    const uint16_t* pos = pick(d.ccard_pos, o) + coff[0];
    for (int f = threadIdx.x; f < il; f += blockDim.x) {
        uint16_t e = 0;  // beyond the last list: read, never used
        if (f < m) {
            e = (uint16_t)(order[f] | (f == 0 ? 0x8000u : 0u));
        } else if (f < 3 * m) {
            const int t = f - m;
            e = (uint16_t)(order[pos[t]] | (t == 0 || card[t - 1] != card[t] ? 0x8000u : 0u));
        }
        im[f] = e;
    }
}

// ------------------------------------------------------------ chance nodes
// Chance node without runout terminals (cfr.rs:637-663): per hand the sum of
// its representatives' children in card order, times 1 / divisor.  One hand
// per lane, `chunks` CTAs per node; four threads load a hand's children, all 52
// cards' loads in flight, and one adds them in card order (a skipped card adds +0, which changes
// no bits of a sum that starts at +0).
constexpr int kChanceHands = 64, kChanceParts = 4;
__global__ void __launch_bounds__(kChanceHands* kChanceParts) kv_chance(Dev d, const ChanceItem* items, int p,
                                                                        uint32_t chunks) {
    constexpr int NT = kChanceHands * kChanceParts, N = 52 / kChanceParts;
    __shared__ CardEntry s_c[52];
    __shared__ float s_v[52][kChanceHands];
    const uint32_t nd = blockIdx.x / chunks;
    const ChanceItem c = items[nd];
    if (threadIdx.x < 52)
        s_c[threadIdx.x] = threadIdx.x < c.cc_count ? d.cards[c.cc_start + threadIdx.x] : CardEntry{0xFFu, 0, 0, 0};
    const int nh = pick(d.nh, p), h = (int)threadIdx.x % kChanceHands, part = (int)threadIdx.x / kChanceHands;
    const int i = (int)(blockIdx.x - nd * chunks) * kChanceHands + h;
    const uint64_t hm = i < nh ? pick(d.mask, p)[i] : ~0ull;
    const uint16_t* hp = pick(d.hperm, p);
    pdl_enter();
    __syncthreads();
    float v[N];
#pragma unroll
    for (int j = 0; j < N; j++) {
        const CardEntry e = s_c[part * N + j];
        const uint32_t card = e.card & 0xFF;
        v[j] = 0.0f;
        if (card < 52u && !(hm >> card & 1ull)) {
            const int src = e.perm ? (int)hp[(size_t)e.perm * nh + i] : i;
            v[j] = d.cfv[(size_t)e.child_cslot * d.nh_max + src];
        }
    }
#pragma unroll
    for (int j = 0; j < N; j++) s_v[part * N + j][h] = v[j];
    __syncthreads();
    if (part != 0 || i >= nh) return;
    float acc = 0.0f;
#pragma unroll
    for (int t = 0; t < 52; t++) acc += s_v[t][h];
    d.cfv[(size_t)c.cslot * d.nh_max + i] = acc * c.inv;
}
// Chance edges of player q: the parent's reach with the holders of the card
// zeroed; a thread takes four hands of one edge.
__global__ void __launch_bounds__(256) kv_edges(Dev d, const EdgeItem* items, uint32_t count, int q, uint32_t quads) {
    const uint64_t g = (uint64_t)blockIdx.x * 256u + threadIdx.x;
    const uint32_t e = (uint32_t)(g / quads), k = (uint32_t)(g - (uint64_t)e * quads);
    if (e >= count) return;
    const uint32_t card = items[e].card;
    pdl_enter();
    const size_t str = (size_t)pick(d.rstr, q);
    float* base = pick(d.reach, q);
    float4 v = ((const float4*)(base + (size_t)items[e].prs[q] * str))[k];
    const uint4 h = ((const uint4*)pick(d.hinfo, q))[k];
    auto keep = [&](uint32_t w) { return (w & 63u) != card && (w >> 6 & 63u) != card; };
    if (!keep(h.x)) v.x = 0.0f;
    if (!keep(h.y)) v.y = 0.0f;
    if (!keep(h.z)) v.z = 0.0f;
    if (!keep(h.w)) v.w = 0.0f;
    ((float4*)(base + (size_t)items[e].crs[q] * str))[k] = v;
}

template <class F>
bool with_show(const ShowShape& sh, F f) {
    auto by_k = [&](auto G, auto NT) {
        if (sh.chunk == 4) f(G, NT, std::integral_constant<int, 4>{});
        else if (sh.chunk == 8) f(G, NT, std::integral_constant<int, 8>{});
        else if (sh.chunk == 12) f(G, NT, std::integral_constant<int, 12>{});
        else if (sh.chunk == 16) f(G, NT, std::integral_constant<int, 16>{});
        else return false;
        return true;
    };
    using C8 = std::integral_constant<int, 8>;
    using C4 = std::integral_constant<int, 4>;
    using C2 = std::integral_constant<int, 2>;
    if (sh.threads == 32 && sh.group == 8) return by_k(C8{}, std::integral_constant<int, 32>{});
    if (sh.threads == 32 && sh.group == 4) return by_k(C4{}, std::integral_constant<int, 32>{});
    if (sh.threads == 32 && sh.group == 2) return by_k(C2{}, std::integral_constant<int, 32>{});
    if (sh.threads == 64 && sh.group == 8) return by_k(C8{}, std::integral_constant<int, 64>{});
    if (sh.threads == 64 && sh.group == 4) return by_k(C4{}, std::integral_constant<int, 64>{});
    if (sh.threads == 64 && sh.group == 2) return by_k(C2{}, std::integral_constant<int, 64>{});
    if (sh.threads == 128 && sh.group == 2) return by_k(C2{}, std::integral_constant<int, 128>{});
    if (sh.threads == 256 && sh.group == 2) return by_k(C2{}, std::integral_constant<int, 256>{});
    return false;
}
}  // namespace

bool show_shape(int group, int max_sorted, ShowShape& sh) {
    for (int threads = 32; threads <= (group == 2 ? 256 : 64); threads *= 2) {
        const int rows = threads / (group / 2), k = (3 * max_sorted + rows - 1) / rows;
        sh = {group, threads, k <= 4 ? 4 : (k + 3) / 4 * 4};
        if (sh.chunk <= 16) return true;
    }
    return false;
}
size_t show_group_smem(const ShowShape& sh, int max_sorted, int nho) {
    return ShowLayout(sh.group, sh.chunk, max_sorted, (nho + 3) & ~3).total;
}
const void* show_group_kernel(const ShowShape& sh) {
    const void* fn = nullptr;
    with_show(sh, [&](auto G, auto NT, auto K) { fn = (const void*)kv_show<G(), NT(), K()>; });
    return fn;
}
size_t hand_rank_bytes() { return sizeof(HandRank); }
size_t show_image_bytes(const ShowShape& sh, int max_sorted) { return (size_t)show_img_len(max_sorted, sh.chunk) * 2; }
void build_show_tables(const Dev& d, const ShowGroups& sg, uint32_t slots, cudaStream_t s) {
    if (!slots) return;
    for (int q = 0; q < 2; q++) {  // ranks of traverser q among the other player's entries
        k_hand_ranks<<<slots, 256, 0, s>>>(d, q, sg.shape[1 - q].chunk, (HandRank*)sg.ranks[q]);
        k_show_images<<<slots, 256, 0, s>>>(d, q, sg.max_sorted[q], sg.shape[q].chunk, (uint16_t*)sg.img[q]);
    }
}
void vec_show(const Dev& d, const ShowGroups& sg, int p, cudaStream_t s) {
    if (!sg.count) return;
    const int o = 1 - p;
    const size_t smem = show_group_smem(sg.shape[o], sg.max_sorted[o], d.nh[o]);
    with_show(sg.shape[o], [&](auto G, auto NT, auto K) {
        pdl_launch(kv_show<G(), NT(), K()>, sg.count, NT(), smem, s, d, sg.items, (const uint16_t*)sg.img[o],
                   (const HandRank*)sg.ranks[p], p, sg.max_sorted[o]);
    });
}
size_t fold_sum_bytes() { return sizeof(FoldSum); }
void fold_kernels(int nho, const void* (&fn)[2], size_t* smem) {
    const int G = fold_group(nho);
    *smem = (size_t)((nho + 3) & ~3) * G * 4;
    fn[0] = G == 8 ? (const void*)kv_folds<8, 1> : (const void*)kv_folds<32, 1>;
    fn[1] = G == 8 ? (const void*)kv_folds<8, 2> : fn[0];
}
void vec_folds(const Dev& d, const uint32_t* slots, uint32_t count, int p, cudaStream_t s) {
    if (!count) return;
    const int nho = d.nh[1 - p], G = fold_group(nho);
    const unsigned grid = (count + G - 1) / G, smem = (unsigned)((nho + 3) & ~3) * G * 4;
    FoldSum* out = const_cast<FoldSum*>(d.folds);
    if (G == 32) pdl_launch(kv_folds<32, 1>, grid, fold_threads<32, 1>(), smem, s, d, slots, count, p, out);
    else if (grid <= kSms * 3) pdl_launch(kv_folds<8, 2>, grid, fold_threads<8, 2>(), smem, s, d, slots, count, p, out);
    else pdl_launch(kv_folds<8, 1>, grid, fold_threads<8, 1>(), smem, s, d, slots, count, p, out);
}
void vec_chance(const Dev& d, const ChanceItem* items, uint32_t count, int p, cudaStream_t s) {
    if (!count) return;
    const uint32_t chunks = (uint32_t)((d.nh[p] + kChanceHands - 1) / kChanceHands);
    pdl_launch(kv_chance, count * chunks, kChanceHands * kChanceParts, 0, s, d, items, p, chunks);
}
void vec_edges(const Dev& d, const EdgeItem* items, uint32_t count, int qmask, cudaStream_t s) {
    if (!count) return;
    for (int q = 0; q < 2; q++) {
        if (!(qmask >> q & 1)) continue;
        const uint32_t quads = (uint32_t)(d.rstr[q] / 4);
        const uint64_t n = (uint64_t)count * quads;
        pdl_launch(kv_edges, (unsigned)((n + 255) / 256), 256, 0, s, d, items, count, q, quads);
    }
}

}  // namespace gtob
