// In-shared-memory NTT passes: radix-2^RB register blocks over a padded layout.
//
// The reference runs radix-2/4/8/16 stages over remainder trees with 16-point
// register leaves (src/transform/forward.rs:200-298, src/transform/stage.rs:34-175,
// src/arch/schedule/leaf.rs:28-82). Here one CTA transforms one or more vectors of
// n = 2^LOG_N points held in shared memory. Each thread loads 2^RB points spaced
// HQ apart into registers, runs RB butterfly levels there, and stores them back,
// so shared memory is touched twice per RB levels. The forward roots come from pass
// tables (one twiddle per block and level, ntt_arith.cuh), the inverse ones from a
// level-major table (entry h + j holds w_{2h}^-j), in shared or global memory.
//
// Every size is a template parameter, so the slot of point m of a register block
// is the block's base plus a compile-time offset and each twiddle load has an
// immediate offset from one per-block base: the only per-point instructions left
// are the loads, the stores and the butterflies themselves.
//
// Forward: natural order in, bit-reversed order out, in Cooley-Tukey butterflies (the
// same as the inverse's: fewer multiplier slots than the Gentleman-Sande form).
// Inverse: decimation in time, bit-reversed order in, natural order out.
#pragma once
#include "ntt_arith.cuh"

// Butterflies whose twiddle is 1 (the first of every group when a register block
// holds consecutive points) run without a product.
#ifndef NTT_UNIT_C0
#define NTT_UNIT_C0 1
#endif

// Shared-memory slot of logical index i: one pad word per 32 words.
__host__ __device__ constexpr int pad_index(int i) { return i + (i >> 5); }

// log2 of a power of two.
__host__ __device__ constexpr int ilog2(int n) { return n > 1 ? 1 + ilog2(n >> 1) : 0; }

// Padded words that hold one vector of n points.
__host__ __device__ constexpr int padded_len(int n) { return n + (n >> 5); }

// A product shorter than its transform: with the transform's T points in bit-reversed
// order, octant o of them (T/8 consecutive points) is the product modulo
// x^(T/8) - z_o, and l octants determine a product of at most l T/8 coefficients. So
// the passes compute only octants below l, 5 <= l <= 8 (shorter products take the next
// smaller transform), and the inverse column pass, which meets the octants in its last
// three levels, solves for the l T/8 coefficients (inv_tail). Eighths are the finest
// part the solve takes without products beyond those it replaces. Without and with the
// cut: 700,001 x 650,003 142.3 -> 120.4 us (6 octants), 2,800,000^2 636 -> 528 us
// (6), 11,000,000^2 2.93 -> 2.41 ms (6), 256 mixed products 408 -> 378 us.
constexpr int kOctants = 8;
__host__ __device__ inline int octants_of(u64 conv_len, int log_t) {
    const int l = (int)((conv_len + ((u64)1 << (log_t - 3)) - 1) >> (log_t - 3));
    return l < 5 ? 5 : l > kOctants ? kOctants : l;
}

// For a register block of 2^RB points spaced S apart whose first point i0 satisfies
// i0 mod 32 + (2^RB - 1) * S < 32 whenever 2^RB * S <= 32 (blocks are aligned), the
// slot of point m is pad_index(i0) + m*S + ((m*S) >> 5).
template <int S>
__device__ __forceinline__ constexpr int slot_offset(int m) {
    return m * S + ((m * S) >> 5);
}

// Vectors a thread transforms together: register blocks at the same position of
// two vectors share their twiddles, so each twiddle load serves both and the two
// butterfly chains interleave. Pairs are taken only while every thread still gets
// a block (2^LOG_GPV blocks per vector, NT threads).
template <int NV, int LOG_GPV, int NT>
__host__ __device__ constexpr int vectors_per_block() {
    return NV % 2 == 0 && ((NV / 2) << LOG_GPV) >= NT ? 2 : 1;
}

// RB forward levels on VP register blocks of 2^RB points. Sub-block b of level t has
// one twiddle, tw[((1 << t) + b - 1) * S] (ntt_arith.cuh, forward roots). FIRST: the
// blocks start at level 0, where sub-block 0 has twiddle 1 and the values come in
// below 2p; with HZ the upper half of every block is zero there, so the first level
// only copies: (x, 0) -> (x, x). With CUT (FIRST) only the octants below `octs` of
// the outputs are needed, and the levels from the third on skip the others.
template <class A, int RB, int S, int VP, bool FIRST = false, bool HZ = false, bool CUT = false, int START = 0>
__device__ __forceinline__ void fwd_levels(u32 (&x)[VP][1 << RB], const uint2* __restrict__ tw, Mod m,
                                           int octs = kOctants) {
    constexpr int E = 1 << RB;
    static_assert(FIRST || (!HZ && !CUT), "only the first pass has a known zero half or unused outputs");
    constexpr int TOP = CUT ? 3 : RB;  // levels of the whole block; the rest octant by octant
#pragma unroll
    for (int t = START; t < TOP; ++t) {
        const int half = E >> (t + 1);
#pragma unroll
        for (int b = 0; b < (1 << t); ++b) {
            if (FIRST && b == 0) {
#pragma unroll
                for (int q = 0; q < VP; ++q)
#pragma unroll
                    for (int c = 0; c < half; ++c) {
                        if (HZ && t == 0) x[q][c + half] = x[q][c];
                        else if (t == 0 || (HZ && t == 1)) A::bf_unit_2p(x[q][c], x[q][c + half], m);
                        else A::bf_unit(x[q][c], x[q][c + half], m);
                    }
                continue;
            }
            const uint2 w = tw[((1 << t) + b - 1) * S];
#pragma unroll
            for (int q = 0; q < VP; ++q)
#pragma unroll
                for (int c = 0; c < half; ++c) A::bf(x[q][2 * half * b + c], x[q][2 * half * b + c + half], w, m);
        }
    }
    if constexpr (CUT) {
#pragma unroll
        for (int o = 0; o < kOctants; ++o) {
            if (o >= octs) break;
#pragma unroll
            for (int t = TOP; t < RB; ++t) {
                const int half = E >> (t + 1);
#pragma unroll
                for (int b = o << (t - TOP); b < (o + 1) << (t - TOP); ++b) {
                    const uint2 w = tw[((1 << t) + b - 1) * S];
#pragma unroll
                    for (int q = 0; q < VP; ++q)
#pragma unroll
                        for (int c = 0; c < half; ++c) {
                            u32 &u = x[q][2 * half * b + c], &v = x[q][2 * half * b + c + half];
                            if (b == 0) A::bf_unit(u, v, m);
                            else A::bf(u, v, w, m);
                        }
                }
            }
        }
    }
}

// The same on a block whose outputs are all wanted times a constant c: f = (c and its
// companion, c * w and its companion) with w the twiddle of the first level, where
// x + w y becomes c x + (c w) y. That costs a product for half of the points.
template <class A, int RB, int S>
__device__ __forceinline__ void fwd_levels_scaled(u32 (&x)[1][1 << RB], uint4 f, const uint2* __restrict__ tw, Mod m) {
    constexpr int H = 1 << (RB - 1);
#pragma unroll
    for (int k = 0; k < H; ++k) {
        x[0][k] = A::mulc(x[0][k], make_uint2(f.x, f.y), m);
        A::bf_2p(x[0][k], x[0][k + H], make_uint2(f.z, f.w), m);
    }
    fwd_levels<A, RB, S, 1, false, false, false, 1>(x, tw, m);
}

// RB inverse levels on VP register blocks of 2^RB points spaced H apart. UNIT
// (H = 1: the first level's twiddle is 1) runs that level without products:
// 1 for inputs in [0, 4p) (A::bf_unit), 2 for inputs in [0, 2p) (A::bf_unit_2p).
template <class A, int RB, int H, int VP, int UNIT = 0>
__device__ __forceinline__ void dit_levels(u32 (&x)[VP][1 << RB], const uint2* __restrict__ twb, Mod m) {
    constexpr int E = 1 << RB;
    static_assert(UNIT == 0 || H == 1, "a product-free first level needs consecutive points");
#pragma unroll
    for (int t = 0; t < RB; ++t) {
        const int dist = 1 << t;
        if (UNIT && t == 0) {
#pragma unroll
            for (int q = 0; q < VP; ++q)
#pragma unroll
                for (int b = 0; b < E; b += 2) {
                    if (UNIT == 2) A::bf_unit_2p(x[q][b], x[q][b + 1], m);
                    else A::bf_unit(x[q][b], x[q][b + 1], m);
                }
            continue;
        }
#pragma unroll
        for (int c = 0; c < dist; ++c) {
            if (NTT_UNIT_C0 && H == 1 && c == 0) {  // twiddle 1: no product
#pragma unroll
                for (int q = 0; q < VP; ++q)
#pragma unroll
                    for (int b = 0; b < E; b += 2 * dist) A::bf_unit(x[q][b], x[q][b + dist], m);
                continue;
            }
            const uint2 w = twb[(H << t) + c * H];
#pragma unroll
            for (int q = 0; q < VP; ++q)
#pragma unroll
                for (int b = 0; b < E; b += 2 * dist) A::bf(x[q][b + c], x[q][b + c + dist], w, m);
        }
    }
}

// Start of register block gg of a pass whose blocks span 2^RB points H apart:
// i0 = a * H * 2^RB + j with j < H. With the plain order (j = gg mod H), a warp
// whose 32 blocks have 2 <= H <= 16 covers 32 / H values of a, whose starts are H/2
// banks apart in the padded layout: two-way conflicts. Taking H/2 values of j and
// 64/H values of a per warp instead spreads the 32 starts over distinct banks (the
// other half of j goes to the next warp).
template <int LOG_H, int RB, int LOG_GPV>
__device__ __forceinline__ int block_start(int gg, int& j) {
    constexpr int H = 1 << LOG_H;
    if constexpr (LOG_H >= 1 && LOG_H <= 4 && LOG_GPV >= 6) {
        constexpr int LOG_HH = LOG_H - 1;  // log2(H / 2)
        const int l = gg & 31, hi = gg >> 5;
        j = ((hi & 1) << LOG_HH) + (l & ((1 << LOG_HH) - 1));
        const int a = ((hi >> 1) << (6 - LOG_H)) + (l >> LOG_HH);
        return (a << (LOG_H + RB)) + j;
    } else {
        j = gg & (H - 1);
        return ((gg >> LOG_H) << (LOG_H + RB)) + j;
    }
}

// The last three inverse levels at one position of the octants when only l of them
// were transformed (5 <= l <= 7): u[o] is octant o there, unscaled, and the result is 8
// times coefficient q of the position (n1 = position + q R/8) in u[q], q < l; the
// coefficients from l on are zero. Octants 0..3 give s_q = c_q + c_(q+4) as usual. The
// others, untwisted by wc, are residues of d_q = c_q - c_(q+4) (q < 4) modulo
// y^2 - i (octants 4 and 5: g_q = d_q + i d_(q+2)), y - z (octant 4 alone) or
// y - z^3 (octant 6), z a primitive eighth root and i = z^2, and d_q = s_q wherever
// c_(q+4) = 0. Roots: wa of level one, wb of level two, wc[0..1] of level three
// and wc[2] = w_R^(-3 position) for octant 6; consts = small_inv.
template <class A>
__device__ __forceinline__ void inv_tail(u32 (&u)[kOctants], uint2 wa, uint2 wb0, uint2 wb1, const uint2 (&wc)[3],
                                         const uint2* __restrict__ consts, Mod m, int l) {
    const uint2 I = consts[3], Z = consts[5], Z3 = consts[7];  // i^-1, z^-1, z^-3
    A::bf(u[0], u[1], wa, m);
    A::bf(u[2], u[3], wa, m);
    A::bf(u[0], u[2], wb0, m);  // u[q] = 4 s_q
    A::bf(u[1], u[3], wb1, m);
    if (l == 5) {
        // 4 d_0 = 4 v_4 - i s_2 - z (s_1 + i s_3), s standing for 4 s
        u32 d = A::mulc(u[4], wc[0], m);
        d = A::add(d, d, m);
        d = A::add(d, d, m);
        d = A::add(d, A::mulc(u[2], I, m), m);
        d = A::add(d, A::mulc(A::sub(u[1], A::mulc(u[3], I, m), m), Z3, m), m);
        u[4] = A::sub(u[0], d, m);
        u[0] = A::add(u[0], d, m);
        u[1] = A::add(u[1], u[1], m);
        u[2] = A::add(u[2], u[2], m);
    } else {
        A::bf(u[4], u[5], wa, m);
        const u32 g0 = A::mulc(u[4], wc[0], m), g1 = A::mulc(u[5], wc[1], m);  // 2 g_q
        const u32 is3 = A::mulc(u[3], I, m);                                  // -4 i s_3
        const u32 d1 = A::add(A::add(g1, g1, m), is3, m);
        u32 d0;
        if (l == 6) {
            d0 = A::add(A::add(g0, g0, m), A::mulc(u[2], I, m), m);
            u[2] = A::add(u[2], u[2], m);
        } else {
            // h_q = d_q - i d_(q+2): 2 h_1 = g1 - 4 i s_3, 2 h_0 = 2 v_6 + 2 h_1 / z
            const u32 v6 = A::mulc(u[6], wc[2], m);
            const u32 h0 = A::add(A::add(v6, v6, m), A::mulc(A::add(g1, is3, m), Z, m), m);
            d0 = A::add(g0, h0, m);
            const u32 d2 = A::mulc(A::sub(g0, h0, m), I, m);
            u[6] = A::sub(u[2], d2, m);
            u[2] = A::add(u[2], d2, m);
        }
        u[4] = A::sub(u[0], d0, m);
        u[0] = A::add(u[0], d0, m);
        u[5] = A::sub(u[1], d1, m);
        u[1] = A::add(u[1], d1, m);
    }
    u[3] = A::add(u[3], u[3], m);
}

// The last RB inverse levels of a 2^LOG_N-point vector on a register block of points
// j0 + k H, k < 2^RB, of which only the octants below octs hold values (k < octs
// 2^RB / 8) and come out. twb = level-major table + j0.
template <class A, int RB, int H>
__device__ __forceinline__ void dit_levels_cut(u32 (&x)[1][1 << RB], const uint2* __restrict__ twb, int j0,
                                               const uint2* __restrict__ consts, Mod m, int octs) {
    constexpr int E = 1 << RB, W = E / kOctants;  // points per octant
    static_assert(RB >= 3, "the octants meet in the last three levels");
#pragma unroll
    for (int t = 0; t < RB; ++t) {
        if (t == RB - 3 && octs < kOctants) {
            constexpr int R8 = H * W;
#pragma unroll
            for (int j = 0; j < W; ++j) {
                const int p = j * H;
                uint2 wc[3] = {twb[4 * R8 + p], twb[4 * R8 + p + R8], make_uint2(0, 0)};
                if (octs == 7) wc[2] = twb[4 * R8 + 3 * p + 2 * j0];
                u32 u[kOctants];
#pragma unroll
                for (int o = 0; o < kOctants; ++o) u[o] = x[0][j + o * W];
                inv_tail<A>(u, twb[R8 + p], twb[2 * R8 + p], twb[2 * R8 + p + R8], wc, consts, m, octs);
#pragma unroll
                for (int o = 0; o < kOctants; ++o) x[0][j + o * W] = u[o];
            }
            break;
        }
        const int dist = 1 << t;
#pragma unroll
        for (int c = 0; c < dist; ++c) {
            const uint2 w = twb[(H << t) + c * H];
#pragma unroll
            for (int b = 0; b < E; b += 2 * dist) A::bf(x[0][b + c], x[0][b + c + dist], w, m);
        }
    }
}

// One pass of RB forward levels starting at LEVEL > 0 over NV vectors of 2^LOG_N points,
// VS words apart (a first pass reads global memory, in the kernels). Register block gg of
// a vector starts at block_start(gg) and spans 2^RB points HQ apart; tw is the pass table.
template <class A, int LOG_N, int LEVEL, int RB, int NT, int NV, int VS, bool CUT = false>
__device__ __forceinline__ void fwd_pass(u32* __restrict__ s, const uint2* __restrict__ tw, Mod m,
                                         int octs = kOctants) {
    static_assert(LEVEL > 0, "the first pass has twiddles of its own");
    constexpr int E = 1 << RB;
    constexpr int LOG_HQ = LOG_N - LEVEL - RB;
    constexpr int HQ = 1 << LOG_HQ;
    constexpr int LOG_GPV = LOG_N - RB;
    constexpr int VP = vectors_per_block<NV, LOG_GPV, NT>();
    constexpr int ITEMS = (NV / VP) << LOG_GPV;
#pragma unroll 1
    for (int it = threadIdx.x; it < ITEMS; it += NT) {
        const int v = (it >> LOG_GPV) * VP;
        const int gg = it & ((1 << LOG_GPV) - 1);
        int j0;
        const int i0 = block_start<LOG_HQ, RB, LOG_GPV>(gg, j0);
        if (CUT && i0 >= octs << (LOG_N - 3)) continue;
        u32* base = s + v * VS + pad_index(i0);
        u32 x[VP][E];
#pragma unroll
        for (int q = 0; q < VP; ++q)
#pragma unroll
            for (int k = 0; k < E; ++k) x[q][k] = base[q * VS + slot_offset<HQ>(k)];
        fwd_levels<A, RB, (1 << LEVEL), VP>(x, tw + (1 << LEVEL) + (i0 >> (LOG_HQ + RB)), m);
#pragma unroll
        for (int q = 0; q < VP; ++q)
#pragma unroll
            for (int k = 0; k < E; ++k) base[q * VS + slot_offset<HQ>(k)] = x[q][k];
    }
}

// One pass of RB inverse levels starting at LEVEL; block gg starts at
// block_start(gg) and spans 2^RB points HS = 2^LEVEL apart.
template <class A, int LOG_N, int LEVEL, int RB, int NT, int NV, int VS, bool CUT = false>
__device__ __forceinline__ void dit_pass(u32* __restrict__ s, const uint2* __restrict__ tw, Mod m,
                                         int octs = kOctants) {
    static_assert(!CUT || LEVEL + RB <= LOG_N - 3, "a register block lies in one octant");
    constexpr int E = 1 << RB;
    constexpr int HS = 1 << LEVEL;
    constexpr int LOG_GPV = LOG_N - RB;
    constexpr int VP = vectors_per_block<NV, LOG_GPV, NT>();
    constexpr int ITEMS = (NV / VP) << LOG_GPV;
#pragma unroll 1
    for (int it = threadIdx.x; it < ITEMS; it += NT) {
        const int v = (it >> LOG_GPV) * VP;
        const int gg = it & ((1 << LOG_GPV) - 1);
        int j0;
        const int i0 = block_start<LEVEL, RB, LOG_GPV>(gg, j0);
        if (CUT && i0 >= octs << (LOG_N - 3)) continue;
        u32* base = s + v * VS + pad_index(i0);
        u32 x[VP][E];
#pragma unroll
        for (int q = 0; q < VP; ++q)
#pragma unroll
            for (int k = 0; k < E; ++k) x[q][k] = base[q * VS + slot_offset<HS>(k)];
        dit_levels<A, RB, HS, VP>(x, tw + j0, m);
#pragma unroll
        for (int q = 0; q < VP; ++q)
#pragma unroll
            for (int k = 0; k < E; ++k) base[q * VS + slot_offset<HS>(k)] = x[q][k];
    }
}

// Levels per register block (2^RB points per thread and pass).
#ifndef NTT_MAX_RB
#define NTT_MAX_RB 4
#endif
constexpr int kMaxRB = NTT_MAX_RB;

// The forward passes of NV vectors of 2^LOG_N points, VS words apart, from LEVEL > 0 on,
// each followed by a barrier.
template <class A, int LOG_N, int NT, int NV, int VS, int LEVEL, bool CUT = false>
__device__ __forceinline__ void fwd_rest(u32* s, const uint2* tw, Mod m, int octs = kOctants) {
    static_assert(!CUT || LEVEL >= 3, "an octant's points lie in whole register blocks");
    if constexpr (LEVEL < LOG_N) {
        constexpr int RB = LOG_N - LEVEL >= kMaxRB ? kMaxRB : LOG_N - LEVEL;
        fwd_pass<A, LOG_N, LEVEL, RB, NT, NV, VS, CUT>(s, tw, m, octs);
        __syncthreads();
        fwd_rest<A, LOG_N, NT, NV, VS, LEVEL + RB, CUT>(s, tw, m, octs);
    }
}

// Forward passes of kMaxRB levels from LEVEL > 0 up to END (exclusive), each followed
// by a barrier.
template <class A, int LOG_N, int NT, int NV, int VS, int LEVEL, int END>
__device__ __forceinline__ void fwd_range(u32* s, const uint2* tw, Mod m) {
    if constexpr (LEVEL < END) {
        fwd_pass<A, LOG_N, LEVEL, kMaxRB, NT, NV, VS>(s, tw, m);
        __syncthreads();
        fwd_range<A, LOG_N, NT, NV, VS, LEVEL + kMaxRB, END>(s, tw, m);
    }
}

// Inverse passes of kMaxRB levels from LEVEL up to END (exclusive), each followed by
// a barrier.
template <class A, int LOG_N, int NT, int NV, int VS, int LEVEL, int END, bool CUT = false>
__device__ __forceinline__ void dit_range(u32* s, const uint2* tw, Mod m, int octs = kOctants) {
    if constexpr (LEVEL < END) {
        dit_pass<A, LOG_N, LEVEL, kMaxRB, NT, NV, VS, CUT>(s, tw, m, octs);
        __syncthreads();
        dit_range<A, LOG_N, NT, NV, VS, LEVEL + kMaxRB, END, CUT>(s, tw, m, octs);
    }
}
