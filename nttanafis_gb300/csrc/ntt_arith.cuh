// Modular arithmetic over 32-bit NTT primes, shared by every kernel.
//
// The reference multiplies in eight 50-bit prime fields held as integer-valued
// f64 (src/field/catalog.rs:67-76, src/arch/scalar/product.rs:99-109). GB300's
// FP64 rate is a small fraction of its 32-bit integer rate, so this library keeps
// every residue in a u32 and reduces with Shoup's precomputed-quotient product
// (one IMAD.HI, one IMUL, one IMAD) and Montgomery's product where neither factor
// is a constant. The integer product is unique, so the choice of primes does not
// change any output limb.
//
// Two residue domains exist, chosen per transform length by the planner:
//   Lazy  (p < 2^30): Harvey's lazy butterflies. Transform values lie in [0, 4p),
//                     packed limbs and stored spectra in [0, 2p); 4p < 2^32 keeps
//                     every sum in a u32.
//   Wide  (p < 2^31): values in [0, 2p), both terms of a butterfly reduced to [0, p)
//                     before its sums. Used where no prime below 2^30
//                     has the two-power roots of the transform (T >= 2^24), and
//                     at T = 2^22, 2^23 where five of them hold what six
//                     lazy primes would.
#pragma once
#include <stdint.h>

typedef uint32_t u32;
typedef uint64_t u64;

// A modulus p and its negative n = 2^32 - p. Both come from memory, so that a
// product is subtracted as a multiply-add by n: written as `- q * p`, the compiler
// multiplies, then subtracts, one instruction more on the path that bounds the
// transforms (10.2 against 11.5 register-only Gentleman-Sande butterflies per clock and SM).
struct Mod {
    u32 p, n;
};

// Returns x*w mod p in [0, 2p) for any x < 2^32, with wp = floor(w * 2^32 / p).
__device__ __forceinline__ u32 shoup_mul(u32 x, u32 w, u32 wp, Mod m) {
    const u32 q = __umulhi(x, wp);
    return q * m.n + x * w;
}
// a + (x*w mod p in [0, 2p)), the addition folded into the product's multiply-add.
__device__ __forceinline__ u32 shoup_mul_add(u32 a, u32 x, u32 w, u32 wp, Mod m) {
    const u32 q = __umulhi(x, wp);
    return q * m.n + (x * w + a);
}

// Returns x - m when x >= m, else x; valid when x < 2m and 2m <= 2^32.
__device__ __forceinline__ u32 sub_if_ge(u32 x, u32 m) { return min(x, x - m); }

// Montgomery product a*b*2^-32 mod p for a*b + 2^32 p < 2^64, below a*b / 2^32 + p: below
// 3p for a < 4p, b < 2p of a lazy prime, below 2p for a < 2p, b < p of a wide one (the
// largest, 2^31 - 2^24 + 1, leaves 1% of 2^64).
__device__ __forceinline__ u32 mont_mul(u32 a, u32 b, u32 p, u32 pneg_inv) {
    const u64 t = (u64)a * b;
    const u32 m = (u32)t * pneg_inv;
    const u64 u = t + (u64)m * p;
    return (u32)(u >> 32);
}

struct LazyArith {
    static constexpr bool kWide = false;
    // Butterfly of both directions (Cooley-Tukey form, the product before the sums):
    // x, y in [0, 4p) -> x + y*w, x - y*w in [0, 4p). With a = x below 2p, x' = a + y*w
    // keeps the multiply-adds whole and y' = 2a + 2p - x' is one three-input addition
    // more: 13.3 register-only butterflies per clock and SM, against 10.0 with y*w
    // formed first and 11.5 for the Gentleman-Sande form ((x - y) * w), with twiddles per
    // thread; probe.cu, whose twiddles are the same in every thread, runs this form at 14.3.
    static __device__ __forceinline__ void bf(u32& x, u32& y, uint2 w, Mod m) {
        const u32 a = sub_if_ge(x, m.p << 1);
        x = shoup_mul_add(a, y, w.x, w.y, m);
        y = a + a + (m.p << 1) - x;
    }
    // The same with x in [0, 2p).
    static __device__ __forceinline__ void bf_2p(u32& x, u32& y, uint2 w, Mod m) {
        const u32 a = x;
        x = shoup_mul_add(a, y, w.x, w.y, m);
        y = a + a + (m.p << 1) - x;
    }
    // The same with twiddle 1: no product.
    static __device__ __forceinline__ void bf_unit(u32& x, u32& y, Mod m) {
        const u32 a = sub_if_ge(x, m.p << 1), t = sub_if_ge(y, m.p << 1);
        x = a + t;
        y = a - t + (m.p << 1);
    }
    // Twiddle 1 and x, y already in [0, 2p) (packed limbs and what a pass over global
    // memory wrote) -> [0, 4p).
    static __device__ __forceinline__ void bf_unit_2p(u32& x, u32& y, Mod m) {
        const u32 s = x + y;
        y = x - y + (m.p << 1);
        x = s;
    }
    // Product by a constant with Shoup companion; any x < 2^32 -> [0, 2p).
    static __device__ __forceinline__ u32 mulc(u32 x, uint2 w, Mod m) { return shoup_mul(x, w.x, w.y, m); }
    // Transform value -> [0, 2p).
    static __device__ __forceinline__ u32 to_2p(u32 x, Mod m) { return sub_if_ge(x, m.p << 1); }
    // x + y and x - y of transform values.
    static __device__ __forceinline__ u32 add(u32 x, u32 y, Mod m) { return to_2p(x, m) + to_2p(y, m); }
    static __device__ __forceinline__ u32 sub(u32 x, u32 y, Mod m) { return to_2p(x, m) - to_2p(y, m) + (m.p << 1); }
    // Product of a transform value and one below 2p, times 2^-32 (below 3p).
    static __device__ __forceinline__ u32 pointwise(u32 a, u32 b, Mod m, u32 pni) { return mont_mul(a, b, m.p, pni); }
    // Transform value -> canonical [0, p).
    static __device__ __forceinline__ u32 canonical(u32 x, Mod m) { return sub_if_ge(sub_if_ge(x, m.p << 1), m.p); }
    // Sum of two values in [0, 2p) -> [0, 2p).
    static __device__ __forceinline__ u32 add_2p(u32 a, u32 b, Mod m) { return sub_if_ge(a + b, m.p << 1); }
};

struct WideArith {
    static constexpr bool kWide = true;
    static __device__ __forceinline__ u32 red(u32 x, Mod m) { return min(x, x + m.n); }
    // x, y in [0, 2p) -> x + y*w, x - y*w in [0, 2p): both terms reduced to [0, p), the
    // sums left open (2p < 2^32). 13.4 register-only butterflies per clock and SM in the
    // probe that runs the lazy ones at 14.3.
    static __device__ __forceinline__ void bf(u32& x, u32& y, uint2 w, Mod m) {
        const u32 a = red(x, m);
        const u32 t = red(shoup_mul(y, w.x, w.y, m), m);
        x = a + t;
        y = a - t + m.p;
    }
    static __device__ __forceinline__ void bf_2p(u32& x, u32& y, uint2 w, Mod m) { bf(x, y, w, m); }
    // The same with twiddle 1.
    static __device__ __forceinline__ void bf_unit(u32& x, u32& y, Mod m) {
        const u32 a = red(x, m), t = red(y, m);
        x = a + t;
        y = a - t + m.p;
    }
    static __device__ __forceinline__ void bf_unit_2p(u32& x, u32& y, Mod m) { bf_unit(x, y, m); }
    static __device__ __forceinline__ u32 mulc(u32 x, uint2 w, Mod m) {
        return shoup_mul(x, w.x, w.y, m);
    }
    // Transform value -> a factor of the pointwise product (here below p).
    static __device__ __forceinline__ u32 to_2p(u32 x, Mod m) { return sub_if_ge(x, m.p); }
    // x + y and x - y of transform values.
    static __device__ __forceinline__ u32 add(u32 x, u32 y, Mod m) { return red(x, m) + red(y, m); }
    static __device__ __forceinline__ u32 sub(u32 x, u32 y, Mod m) { return red(x, m) - red(y, m) + m.p; }
    // Product of a transform value and one below p, times 2^-32, in [0, 2p).
    static __device__ __forceinline__ u32 pointwise(u32 a, u32 b, Mod m, u32 pni) { return mont_mul(a, b, m.p, pni); }
    static __device__ __forceinline__ u32 canonical(u32 x, Mod m) { return sub_if_ge(x, m.p); }
    // Sum of two values in [0, 2p) -> [0, 2p).
    static __device__ __forceinline__ u32 add_2p(u32 a, u32 b, Mod m) {
        return sub_if_ge(a, m.p) + sub_if_ge(b, m.p);
    }
};

// Per-prime constants handed to every kernel.
struct PrimeParams {
    Mod mod;         // p and 2^32 - p
    u32 pni;         // -p^-1 mod 2^32 (Montgomery)
    u32 inv2_32;     // floor(2^32 / p): Shoup companion of w = 1
    u32 neg64;       // 2^64 mod p, subtracted for negative two's complement limbs
    uint2 r32;       // 2^32 mod p with its Shoup companion
    uint2 scale;     // small-path inverse scale T^-1 * (P/p)^-1 * 2^32 with companion
    const uint2* fwd;    // forward roots in pass order (kFwd4, kFwd5, kFwd6 below)
    const uint2* inv;    // level-major inverse roots: inv[h + j] = w_{2h}^-j
    const uint2* f4_a;   // forward four-step twiddles: per column-pass thread
    const uint2* f4_b;   //                              per column and sweep or register block
    const uint2* i4_lo;  // inverse four-step twiddles: per row, low digit of n2
    const uint2* i4_hi;  //                             per row, high digit, times the scale
    // Roots of the levels whose twiddles every thread shares (the first five forward
    // and the first five inverse ones), held in the kernel parameters, so that they
    // come from the constant cache: small_fwd[2^t + b] = w_{2^(t+1)}^brev_t(b) of block
    // b, small_inv[h + j] = inv[h + j].
    uint2 small_fwd[32];
    uint2 small_inv[32];
};

constexpr int kMaxPrimes = 8;

// Forward roots. The forward transform splits x^n - z^2 into (x^(n/2) - z)(x^(n/2) + z)
// level by level, so that level t has one twiddle per block, w_{2^(t+1)}^brev_t(block),
// whatever the position in the block. A pass of RB levels from LEVEL on gives each
// register block, of block a at LEVEL, 2^RB - 1 twiddles: entry
// 2^LEVEL * (2^t + b) + a is that of sub-block b at level LEVEL + t, so consecutive
// register blocks read consecutive entries. Four tables, by levels per pass, follow
// one another: 4 (every length up to 2^13, 2^7- and 2^8-point columns), 5 (2^9- and
// 2^10-point columns), 6 (2^12-point) and 3 (2^6-point).
constexpr int kFwd4Log = 13, kFwd5Log = 10, kFwd6Log = 12, kFwd3Log = 6;
constexpr int kFwd4 = 0, kFwd5 = kFwd4 + (1 << kFwd4Log), kFwd6 = kFwd5 + (1 << kFwd5Log);
constexpr int kFwd3 = kFwd6 + (1 << kFwd6Log);
constexpr int kFwdEntries = kFwd3 + (1 << kFwd3Log);

// Writes one of these tables (2^log_n entries; entry 0 is not read) from the
// level-major roots roots[h + j] = w_{2h}^j.
inline void forward_pass_table(const uint2* roots, uint2* out, int log_n, int rb) {
    out[0] = roots[0];
    for (int level = 0; level < log_n; level += rb)
        for (int t = 0; t < rb && level + t < log_n; ++t)
            for (u32 block = 0; block < (1u << (level + t)); ++block) {
                u32 rev = 0;
                for (int i = 0; i < level + t; ++i) rev |= ((block >> i) & 1u) << (level + t - 1 - i);
                const u32 a = block >> t, b = block & ((1u << t) - 1);
                out[((1u << t) + b << level) + a] = roots[(1u << (level + t)) + rev];
            }
}

struct PrimeSet {
    PrimeParams pr[kMaxPrimes];
};

// Reduces a 64-bit limb into the forward domain of its arithmetic.
template <class A>
__device__ __forceinline__ u32 reduce_limb(u64 x, const PrimeParams& pp) {
    const u32 lo = (u32)x, hi = (u32)(x >> 32);
    const u32 h = shoup_mul(hi, pp.r32.x, pp.r32.y, pp.mod);  // [0, 2p)
    const u32 l = lo + __umulhi(lo, pp.inv2_32) * pp.mod.n;   // [0, 2p)
    return A::add_2p(h, l, pp.mod);
}

// Reduces a two's complement 64-bit coefficient into the forward domain.
template <class A>
__device__ __forceinline__ u32 reduce_signed(u64 x, const PrimeParams& pp) {
    u32 r = reduce_limb<A>(x, pp);
    if ((int64_t)x < 0) {
        // value = x - 2^64: subtract 2^64 mod p, i.e. add p - neg64 in (0, p].
        r = A::add_2p(r, pp.mod.p - pp.neg64, pp.mod);
    }
    return r;
}
