// Transform-domain kernels: limb packing fused into the first forward pass, the
// pointwise product fused between the last forward and first inverse pass, and the
// inverse scale folded into the last twiddle multiply.
//
// Reference path (per prime): pack a and b (src/limb/packing.rs:113-292), forward
// transforms (src/transform/forward.rs:95-298), pointwise product (fused into the
// inverse leaves for long rows, src/multiply/schedule.rs:259-279), inverse with the
// N^-1 scale (src/transform/inverse.rs:52-218, src/multiply/schedule.rs:225-252).
//
// Layouts:
//  * one CTA per prime holds the whole transform (T <= 2^13): k_small and
//    k_small_fused, in small.cu;
//  * four-step for T = R*C >= 2^13: k_fwd_cols2 (pack + column transform + twiddle),
//    k_rows (row transforms of a and b, pointwise, inverse rows, inverse twiddle) and
//    k_inv_cols2 (inverse columns, canonical residues); 2^12-point columns take
//    k_fwd_cols4 and k_inv_cols4p, 2^11-point ones k_fwd_cols and k_inv_cols. The
//    spectrum order between the passes is
//    the four-step's transposed, bit-reversed order; only the inverse reads it, so
//    no transpose is ever materialised.
//  * k_step_tables builds the four-step factor tables of a transform length.
// Every kernel is instantiated per transform size so all shared-memory strides are
// compile-time constants.
#include "transform_common.cuh"

#include <algorithm>
#include <atomic>

namespace ntt {

#ifndef NTT_ROW_THREADS
#define NTT_ROW_THREADS 128
#endif
// Threads of a row-pass CTA: at least NTT_ROW_THREADS, and one per register block
// of the first pass (C / 16) up to 512, so that no pass loops twice over its
// blocks (two iterations made the compiler hold both in registers).
__host__ __device__ constexpr int row_threads(int log_c) {
    return (1 << (log_c - 4)) > NTT_ROW_THREADS ? ((1 << (log_c - 4)) < 512 ? (1 << (log_c - 4)) : 512)
                                                : NTT_ROW_THREADS;
}

// Padded words per column in shared memory: congruent to 32/G mod 32 (1 when G >=
// 32) so that a warp's G columns times 32/G rows fall in distinct banks.
__host__ __device__ constexpr int col_words_mod(int log_r) {
    return col_group_log(log_r) >= 5 ? 1 : 32 >> col_group_log(log_r);
}
__host__ __device__ constexpr int col_vstride(int log_r) {
    return padded_len(1 << log_r) + (((col_words_mod(log_r) - padded_len(1 << log_r)) % 32) + 32) % 32;
}

// Column pass of the forward four-step: G columns of R = 2^LOG_R points per CTA.
// grid = (C / G, np, operands). Coefficient n = n1*C + n2 sits at row n1, column n2.
// Column passes map thread t to column c = t mod G and rows r0 + k*RS (r0 = t / G,
// RS = 256 / G rows per sweep), so global addresses advance by a constant and the
// shared-memory slot of sweep k is a compile-time offset from the thread's first.
template <int LOG_R>
struct ColumnMap {
    static constexpr int LOG_G = col_group_log(LOG_R);
    static constexpr int G = 1 << LOG_G;
    static constexpr int VS = col_vstride(LOG_R);
    static constexpr int LOG_RS = col_log_rs(LOG_R);
    static constexpr int RS = kThreads / G;        // rows per sweep (power of two <= 32)
    static constexpr int SWEEPS = (1 << LOG_R) / RS;
    static constexpr int LOG_SW = LOG_R - (8 - LOG_G);
    __device__ static int col() { return threadIdx.x & (G - 1); }
    __device__ static int row0() { return threadIdx.x >> LOG_G; }
    __device__ static int slot0() { return col() * VS + pad_index(row0()); }
    // bit-reversed row index of sweep k, less that of row0 (the bits are disjoint)
    __device__ static constexpr u32 brev_sweep(int k) {
        u32 r = 0;
        for (int b = 0; b < LOG_SW; ++b) r |= ((u32)(k >> b) & 1u) << (LOG_SW - 1 - b);
        return r;
    }
};

// CHECK: a convolution's coefficients are checked against their bounds on the way
// in (column_votes); products are instantiated without the check.
template <class A, bool SIGNED, int LOG_R, bool CUT, bool CHECK = SIGNED>
__global__ void __launch_bounds__(kThreads) k_fwd_cols(const __grid_constant__ TransformArgs g) {
    extern __shared__ u32 sm[];
    using M = ColumnMap<LOG_R>;
    if (g.batch) wait_prior_grid();  // descriptors that the kernel before may write
    release_dependents();
    constexpr int B = M::SWEEPS < 8 ? M::SWEEPS : 8;  // sweeps per batch; B*RS is a multiple of 32
    static_assert(M::SWEEPS % B == 0 && (B * M::RS) % 32 == 0, "column batches");
    const int prime = (int)(blockIdx.x % (u32)g.np);  // prime fastest: see k_fwd_cols4
    const u32 group = blockIdx.x / (u32)g.np;
    // grid.z: operands (1 or 2) of one member, or per member in a batch (2, or 1
    // when the batch's other factor is a stored spectrum)
    const int op = g.batch ? (g.a_only ? 0 : blockIdx.z & 1) : blockIdx.z + g.op_base;
    const Member m = member_of(g, g.batch ? (g.a_only ? blockIdx.z : blockIdx.z >> 1) : 0, false);
    if (op && m.square) return;
    const int octs = CUT ? octants_of(m.conv_len, g.log_t) : kOctants;
    const PrimeParams& pp = g.ps.pr[prime];
    const u64* __restrict__ src = op ? m.b : m.a;
    const u64 len = op ? m.lb : m.la;
    u64 vmax = 0;
    u32* const votes =
        CHECK ? column_votes(g, g.batch ? (g.a_only ? blockIdx.z : blockIdx.z >> 1) : 0, op, prime, vmax) : nullptr;
    int bad = 0;
    const int log_c = g.log_c;
    const u32 col0 = group << M::LOG_G;
    const u32 col = col0 + M::col();
    const int r0 = M::row0();
    const u64 first = ((u64)r0 << log_c) + col;
    const u64 step = (u64)M::RS << log_c;
    u32* s = sm + M::slot0();
    uint2* tw = reinterpret_cast<uint2*>(sm + M::G * M::VS);
    load_table<LOG_R>(tw, pp.fwd + kFwd4);
    // Per-sweep four-step factors of the CTA's columns, rows padded to SW + 1 entries
    // so that the G columns of a warp read distinct banks.
    uint2* fb = tw + (1 << LOG_R);
    {
        const uint2* src = pp.f4_b + ((size_t)col0 << M::LOG_SW);
        for (int i = threadIdx.x; i < (M::G << M::LOG_SW); i += kThreads)
            fb[(i >> M::LOG_SW) * (M::SWEEPS + 1) + (i & (M::SWEEPS - 1))] = __ldg(src + i);
    }
    const uint2 fa = __ldg(pp.f4_a + ((size_t)col << M::LOG_RS) + (__brev((u32)r0) >> (32 - M::LOG_RS)));
    wait_prior_grid();  // the operands, and the last reader of the residues
    // First forward pass fused with the limb reduction (its roots are kernel
    // parameters; the shared table is published by the barrier after it). Item it takes
    // column c = it mod G and block gg = it / G (rows gg + k * HQ), so a warp loads
    // four rows of G consecutive limbs at a time and stores to distinct banks. When
    // len <= T/2 (every balanced product) rows R/2 and above hold no limb: their
    // loads are skipped and the first level only copies.
    {
        constexpr int RB = kMaxRB, LOG_HQ = LOG_R - RB, HQ = 1 << LOG_HQ, E = 1 << RB;
        const bool half = len <= ((u64)1 << (g.log_t - 1));
        const u64 kstep = (u64)HQ << log_c;
#pragma unroll 1
        for (int it = threadIdx.x; it < (M::G << LOG_HQ); it += kThreads) {
            const int c = it & (M::G - 1), gg = it >> M::LOG_G;
            const u64 n0 = ((u64)gg << log_c) + col0 + c;
            u32 x[1][E];
            if (half) {
#pragma unroll
                for (int k = 0; k < E / 2; ++k) {
                    const u64 n = n0 + k * kstep;
                    const u64 v = n < len ? __ldcg(src + n) : 0;
                    if (CHECK && votes) bad |= coefficient_over<SIGNED>(v, vmax);
                    x[0][k] = n < len ? reduce_coefficient<A, SIGNED>(v, pp) : 0u;
                }
                fwd_levels<A, RB, 1, 1, true, true, CUT>(x, pp.small_fwd + 1, pp.mod, octs);
            } else {
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    const u64 n = n0 + k * kstep;
                    const u64 v = n < len ? __ldcg(src + n) : 0;
                    if (CHECK && votes) bad |= coefficient_over<SIGNED>(v, vmax);
                    x[0][k] = n < len ? reduce_coefficient<A, SIGNED>(v, pp) : 0u;
                }
                fwd_levels<A, RB, 1, 1, true, false, CUT>(x, pp.small_fwd + 1, pp.mod, octs);
            }
            u32* base = sm + c * M::VS + pad_index(gg);
#pragma unroll
            for (int k = 0; k < E; ++k)
                if (!CUT || k < octs * (E / kOctants)) base[slot_offset<HQ>(k)] = x[0][k];
        }
    }
    if (CHECK && bad) votes[(blockIdx.x + threadIdx.x) % kAdmitSlots] = 1u;
    __syncthreads();
    fwd_rest<A, LOG_R, kThreads, M::G, M::VS, kMaxRB, CUT>(sm, tw, pp.mod, octs);
    // Four-step twiddle w_T^(col * brev(row)) = fa * fb[col][brev(k)], then the store.
    u32* dst = m.spec + ((size_t)(op * g.np + prime) << g.log_t) + first;
    const uint2* fbc = fb + M::col() * (M::SWEEPS + 1);
#pragma unroll 1
    for (int k0 = 0; k0 < (CUT ? octs * M::SWEEPS / kOctants : M::SWEEPS); k0 += B) {
        const uint2* fk = fbc + (__brev((u32)k0) >> (32 - M::LOG_SW));
        const u32* sk = s + slot_offset<M::RS>(k0);
#pragma unroll
        for (int u = 0; u < B; ++u) {
            if (CUT && k0 + u >= octs * M::SWEEPS / kOctants) break;
            u32 x = sk[slot_offset<M::RS>(u)];
            x = A::mulc(x, fk[M::brev_sweep(u)], pp.mod);
            x = A::mulc(x, fa, pp.mod);
            dst[u * step] = x;
        }
        dst += B * step;
    }
}

// Column passes for R = 2^6..2^10 in two register passes: one barrier and one round
// trip through shared memory per element. With EA = 2^RA points per thread in the
// forward pass 1 and EB = R / EA in pass 2, a thread owns column c = t mod G and
// register blocks of rows blk + EB k (blk < EB, k < EA) and rows EB blk + k (blk < EA,
// k < EB). Row EB k + b sits at slot (EB + 1) k + b of its column; EB + 1 is odd and the
// column stride 32 / G mod 32, so that both orders put a warp's G columns x 32 / G
// blocks on 32 distinct banks; both read or write global memory as rows of G
// consecutive columns. The forward four-step twiddle of row EB blk + k is
// w_T^(col * brev(row)) = f4_a[col][brev(k)] * f4_b[col][brev(blk)]. The limbs are
// reduced on the way into the first forward pass, f4_a is applied on the way out of the
// second and f4_b, one factor for a register block, on the way into it: its first level
// multiplies half of the points already, by a twiddle tabulated times f4_b, so that only
// the other half takes a product (4,000,000^2 638 -> 631 us, 1,048,576 x 100,003 103.1 ->
// 102.0; k_fwd_cols4, at its limit of registers, lost: 16M^2 3,004 -> 3,070 us). The last
// inverse pass writes canonical residues. Resident threads
// per SM asked for, by blocks of 32 points 1,024 (64 registers), of 8 and 16 points
// 1,536 (40 registers; 256 mixed products 333 us, 339 with 1,024 and 354 unasked). The
// lengths below 2^10 ran passes of four levels with sweeps for the load and the twiddle
// before: 256 mixed products 360 -> 333 us, 260,000^2 48.8 -> 45.1, 4,000^2 13.2 -> 10.6,
// 1,048,576 x 100,003 112.9 -> 103.7 us.
template <int LOG_R>
struct Columns {
    static constexpr int RA = col_first_log(LOG_R), RB = LOG_R - RA, EA = 1 << RA, EB = 1 << RB;
    static constexpr int LOG_G = LOG_R <= 8 ? 4 : 3, G = 1 << LOG_G;
    static constexpr int NT = G * EB, PITCH = EB + 1;
    static constexpr int VS = EA * PITCH + ((32 / G - EA * PITCH) % 32 + 32) % 32;
    static constexpr int MINB = (RA == 5 ? 1024 : 1536) / NT;
    static constexpr int FWD = RA == 3 ? kFwd3 : RA == 4 ? kFwd4 : kFwd5;  // roots of pass 2
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Whether the forward kernel of 2^10-point columns stages its second pass's roots in
// shared memory (8 KB): 1M^2 151.5 -> 150.0 us with the lazy arithmetic; with the wide one
// the pass gains 1% but 4M^2 as a whole loses as much (667 -> 674 us), so it reads
// them through L1.
template <class A, int LOG_R>
constexpr bool kStageCols2 = !A::kWide && LOG_R == 10;

// Four-step factor f4_b of column col and register block b, and its product with the
// twiddle of the block's first level.
__device__ __forceinline__ uint4 step_factors(const PrimeParams& pp, u32 col, int b, int log_blocks) {
    return __ldg(reinterpret_cast<const uint4*>(pp.f4_b) + ((size_t)col << log_blocks) +
                 (__brev((u32)b) >> (32 - log_blocks)));
}

// Starts the asynchronous copy of n table entries (n even) into shared memory.
template <int NT>
__device__ __forceinline__ void stage_table(uint2* dst, const uint2* src, int n) {
    for (int i = threadIdx.x; i < n / 2; i += NT) cp_async16(dst + 2 * i, src + 2 * i);
    cp_async_commit();
}

template <class A, bool SIGNED, int LOG_R, bool CUT, bool CHECK = SIGNED>
__global__ void __launch_bounds__(Columns<LOG_R>::NT, Columns<LOG_R>::MINB)
    k_fwd_cols2(const __grid_constant__ TransformArgs g) {
    extern __shared__ u32 sm[];
    if (g.batch) wait_prior_grid();  // descriptors that the kernel before may write
    release_dependents();
    using K = Columns<LOG_R>;
    constexpr int G = K::G, EA = K::EA, EB = K::EB;
    constexpr bool STAGE = kStageCols2<A, LOG_R>;
    const int prime = (int)(blockIdx.x % (u32)g.np);  // prime fastest: see k_fwd_cols4
    const u32 group = blockIdx.x / (u32)g.np;
    const int op = g.batch ? (g.a_only ? 0 : blockIdx.z & 1) : blockIdx.z + g.op_base;
    const Member m = member_of(g, g.batch ? (g.a_only ? blockIdx.z : blockIdx.z >> 1) : 0, false);
    if (op && m.square) return;
    const int octs = CUT ? octants_of(m.conv_len, g.log_t) : kOctants;
    const PrimeParams& pp = g.ps.pr[prime];
    const u64* __restrict__ src = op ? m.b : m.a;
    const u64 len = op ? m.lb : m.la;
    u64 vmax = 0;
    u32* const votes =
        CHECK ? column_votes(g, g.batch ? (g.a_only ? blockIdx.z : blockIdx.z >> 1) : 0, op, prime, vmax) : nullptr;
    int bad = 0;
    const int log_c = g.log_c;
    const u32 col0 = group * G;
    const int c = threadIdx.x & (G - 1), blk = threadIdx.x >> K::LOG_G;
    const u32 col = col0 + c;
    // f4_a rows of the CTA's columns, padded to EB + 1 entries per column.
    uint2* fa = reinterpret_cast<uint2*>(sm + G * K::VS);
    fa[c * (EB + 1) + blk] = __ldg(pp.f4_a + ((size_t)col << K::RB) + blk);
    uint2* const tw2 = fa + G * (EB + 1);  // staged roots of the second pass
    if constexpr (STAGE) stage_table<K::NT>(tw2, pp.fwd + K::FWD + EA, (EB - 1) * EA);
    wait_prior_grid();  // the operands, and the last reader of the residues
    // Pass 1: the first RA levels on rows blk + EB k, limbs reduced on the way in; rows
    // R/2 and above hold no limb when len <= T/2.
    {
        const bool half = len <= ((u64)1 << (g.log_t - 1));
        const u64* p0 = src + ((u64)blk << log_c) + col;
        const u64 n0 = ((u64)blk << log_c) + col, kstep = (u64)EB << log_c;
        u32 x[1][EA];
        if (half) {
#pragma unroll
            for (int k = 0; k < EA / 2; ++k) {
                const u64 v = n0 + k * kstep < len ? __ldcg(p0 + k * kstep) : 0;
                if (CHECK && votes) bad |= coefficient_over<SIGNED>(v, vmax);
                x[0][k] = n0 + k * kstep < len ? reduce_coefficient<A, SIGNED>(v, pp) : 0u;
            }
            fwd_levels<A, K::RA, 1, 1, true, true, CUT>(x, pp.small_fwd + 1, pp.mod, octs);
        } else {
#pragma unroll
            for (int k = 0; k < EA; ++k) {
                const u64 v = n0 + k * kstep < len ? __ldcg(p0 + k * kstep) : 0;
                if (CHECK && votes) bad |= coefficient_over<SIGNED>(v, vmax);
                x[0][k] = n0 + k * kstep < len ? reduce_coefficient<A, SIGNED>(v, pp) : 0u;
            }
            fwd_levels<A, K::RA, 1, 1, true, false, CUT>(x, pp.small_fwd + 1, pp.mod, octs);
        }
        u32* base = sm + c * K::VS + blk;
#pragma unroll
        for (int k = 0; k < EA; ++k)
            if (!CUT || k < octs * (EA / kOctants)) base[K::PITCH * k] = x[0][k];
    }
    if (CHECK && bad) votes[(blockIdx.x + threadIdx.x) % kAdmitSlots] = 1u;
    if constexpr (STAGE) cp_async_wait_all();
    const uint4 f0 = step_factors(pp, col, blk, K::RA);
    __syncthreads();
    // Pass 2: the other RB levels on rows EB b + k, four-step twiddle, store.
#pragma unroll
    for (int j = 0; j < EA / EB; ++j) {
        const int b = blk + j * EB;
        if (CUT && b >= octs * (EA / kOctants)) break;
        const u32* base = sm + c * K::VS + K::PITCH * b;
        u32 x[1][EB];
#pragma unroll
        for (int k = 0; k < EB; ++k) x[0][k] = base[k];
        const uint4 f = j == 0 ? f0 : step_factors(pp, col, b, K::RA);
        fwd_levels_scaled<A, K::RB, EA>(x, f, STAGE ? tw2 + b : pp.fwd + K::FWD + EA + b, pp.mod);
        const uint2* fac = fa + c * (EB + 1);
        u32* dst = m.spec + ((size_t)(op * g.np + prime) << g.log_t) + ((u64)(b * EB) << log_c) + col;
#pragma unroll
        for (int k = 0; k < EB; ++k) {
            dst[(u64)k << log_c] = A::mulc(x[0][k], fac[__brev((u32)k) >> (32 - K::RB)], pp.mod);
        }
    }
}

template <class A, int LOG_R, bool CUT>
__global__ void __launch_bounds__(Columns<LOG_R>::NT, Columns<LOG_R>::MINB)
    k_inv_cols2(const __grid_constant__ TransformArgs g) {
    extern __shared__ u32 sm[];
    using K = Columns<LOG_R>;
    constexpr int G = K::G, EA = K::EA, EB = K::EB;
    const int prime = blockIdx.y;
    const PrimeParams& pp = g.ps.pr[prime];
    release_dependents();
    const Member m = member_after(g, blockIdx.z, false);
    const int octs = CUT ? octants_of(m.conv_len, g.log_t) : kOctants;
    const int log_c = g.log_c;
    const int c = threadIdx.x & (G - 1), blk = threadIdx.x >> K::LOG_G;
    wait_prior_grid();  // the row pass's output
    // the CRT look-back flags of this product, cleared once every kernel before
    // this one has completed
    if (blockIdx.x == 0 && prime == 0) clear_flags(g, blockIdx.z);
    u32* const spec = m.spec + ((size_t)prime << g.log_t) + blockIdx.x * G + c;
    // Pass 1: the first RB levels on rows EB b + k (bit-reversed spectrum in).
#pragma unroll
    for (int j = 0; j < EA / EB; ++j) {
        const int b = blk + j * EB;
        if (CUT && b >= octs * (EA / kOctants)) break;
        const u32* q = spec + ((u64)(b * EB) << log_c);
        u32 x[1][EB];
#pragma unroll
        for (int k = 0; k < EB; ++k) x[0][k] = __ldcg(q + ((u64)k << log_c));
        dit_levels<A, K::RB, 1, 1, 2>(x, pp.small_inv, pp.mod);  // the row pass wrote [0, 2p)
        u32* base = sm + c * K::VS + K::PITCH * b;
#pragma unroll
        for (int k = 0; k < EB; ++k) base[k] = x[0][k];
    }
    __syncthreads();
    // Pass 2: the other RA levels on rows blk + EB k, canonical residues out.
    {
        const u32* base = sm + c * K::VS + blk;
        u32 x[1][EA];
#pragma unroll
        for (int k = 0; k < EA; ++k) x[0][k] = !CUT || k < octs * (EA / kOctants) ? base[K::PITCH * k] : 0u;
        if constexpr (CUT) dit_levels_cut<A, K::RA, EB>(x, pp.inv + blk, blk, pp.small_inv, pp.mod, octs);
        else dit_levels<A, K::RA, EB, 1>(x, pp.inv + blk, pp.mod);
        u32* q = spec + ((u64)blk << log_c);
#pragma unroll
        for (int k = 0; k < EA; ++k)
            if (!CUT || k < octs * (EA / kOctants)) q[(u64)(k * EB) << log_c] = A::canonical(x[0][k], pp.mod);
    }
}

// Column passes for R = 2^12 (the wide lengths T = 2^24 and 2^25) in two radix-64
// passes, the k_fwd_cols2 design at twice the block: G columns per CTA of 64 G
// threads, thread t owning column c = t mod G and either rows blk + 64k (pass 1)
// or rows 64 blk + k (pass 2), k < 64. Row r = 64a + b sits at slot 65a + b of its
// column, whose stride (32/G mod 32) puts a warp's G columns x 32/G blocks on 32
// distinct banks in both orders. The forward four-step twiddle of row 64 blk + k is
// w_T^(col * brev(row)) = f4_a[col][brev6(k)] * f4_b[col][brev6(blk)]. The roots
// of the first pass (shared by every thread) sit in shared memory, and those of the
// second pass are staged there by asynchronous copies while the limbs come in (32 KB;
// read through L1 level by level they cost 16M^2 1.125 instead of 1.082 ms forward
// and 0.530 instead of 0.512 ms inverse).
// G = 8 (512 threads of 128 registers, 167 KB) fills an SM with one CTA. G = 4
// (two CTAs per SM, so that one CTA's loads overlap the other's butterflies)
// measured slower on GB300 at T = 2^25: 1.58 against 1.20 ms forward, 0.76 against
// 0.57 ms inverse (16-byte row segments instead of whole 32-byte sectors).
#ifndef NTT_COLS4_LOG_G
#define NTT_COLS4_LOG_G 3
#endif
constexpr int kCol4LogG = NTT_COLS4_LOG_G, kCol4G = 1 << kCol4LogG, kCol4Threads = 64 * kCol4G;
constexpr int kCol4Vs = 65 * 64 + 32 / kCol4G;
static_assert(kCol4Vs % 32 == 32 / kCol4G && step_log_u(kCol4LogR) == 6, "radix-64 column layout");
static_assert(kCol4Threads * 128 * (kCol4LogG == 2 ? 2 : 1) <= 65536, "register budget of the column CTAs");

// SMs of the current device (persistent kernels launch one CTA per SM).
static int sm_count() {
    static std::atomic<int> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    int n = cached[dev].load(std::memory_order_relaxed);
    if (n > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 1;
    cached[dev].store(n, std::memory_order_relaxed);
    return n;
}

static size_t col4_smem(bool fwd) {
    return (size_t)kCol4G * kCol4Vs * sizeof(u32) + 64 * sizeof(uint2) + (fwd ? kCol4G * 65 * sizeof(uint2) + 63 * 64 * sizeof(uint2) : 0);
}

template <class A, bool SIGNED, bool CUT, bool CHECK = SIGNED>
__global__ void __launch_bounds__(kCol4Threads, kCol4LogG == 2 ? 2 : 1)
    k_fwd_cols4(const __grid_constant__ TransformArgs g) {
    extern __shared__ u32 sm[];
    if (g.batch) wait_prior_grid();  // descriptors that the kernel before may write
    release_dependents();
    constexpr int G = kCol4G, LOG_G = kCol4LogG, VS = kCol4Vs, E = 64;
    // grid.x runs over (column group, prime) with the prime fastest, so the np CTAs
    // that read the same limbs run together and all but the first read them from L2
    const int prime = (int)(blockIdx.x % (u32)g.np);
    const u32 group = blockIdx.x / (u32)g.np;
    const int op = g.batch ? (g.a_only ? 0 : blockIdx.z & 1) : blockIdx.z + g.op_base;
    const Member m = member_of(g, g.batch ? (g.a_only ? blockIdx.z : blockIdx.z >> 1) : 0, false);
    if (op && m.square) return;
    const int octs = CUT ? octants_of(m.conv_len, g.log_t) : kOctants;
    const PrimeParams& pp = g.ps.pr[prime];
    const u64* __restrict__ src = op ? m.b : m.a;
    const u64 len = op ? m.lb : m.la;
    u64 vmax = 0;
    u32* const votes =
        CHECK ? column_votes(g, g.batch ? (g.a_only ? blockIdx.z : blockIdx.z >> 1) : 0, op, prime, vmax) : nullptr;
    int bad = 0;
    const int log_c = g.log_c;
    const u32 col0 = group * G;
    const int c = threadIdx.x & (G - 1), blk = threadIdx.x >> LOG_G;
    const u32 col = col0 + c;
    uint2* tw = reinterpret_cast<uint2*>(sm + G * VS);
    uint2* fa = tw + 64;  // f4_a rows of the CTA's columns, 65 entries apart
    if (threadIdx.x < 64) tw[threadIdx.x] = __ldg(pp.fwd + kFwd6 + threadIdx.x);
    fa[c * (E + 1) + blk] = __ldg(pp.f4_a + ((size_t)col << 6) + blk);
    uint2* const tw2 = fa + G * (E + 1);  // roots of the second pass
    stage_table<kCol4Threads>(tw2, pp.fwd + kFwd6 + E, 63 * E);
    __syncthreads();  // the first pass reads tw
    wait_prior_grid();  // the operands, and the last reader of the residues
    // Pass 1: levels 0-5 on rows blk + 64k, limbs reduced on the way in; rows R/2
    // and above hold no limb when len <= T/2.
    {
        const bool half = len <= ((u64)1 << (g.log_t - 1));
        const u64* p0 = src + ((u64)blk << log_c) + col;
        const u64 n0 = ((u64)blk << log_c) + col, kstep = (u64)E << log_c;
        u32 x[1][E];
        if (half) {
#pragma unroll
            for (int k = 0; k < E / 2; ++k) {
                const u64 v = n0 + k * kstep < len ? __ldcg(p0 + k * kstep) : 0;
                if (CHECK && votes) bad |= coefficient_over<SIGNED>(v, vmax);
                x[0][k] = n0 + k * kstep < len ? reduce_coefficient<A, SIGNED>(v, pp) : 0u;
            }
            fwd_levels<A, 6, 1, 1, true, true, CUT>(x, tw + 1, pp.mod, octs);
        } else {
#pragma unroll
            for (int k = 0; k < E; ++k) {
                const u64 v = n0 + k * kstep < len ? __ldcg(p0 + k * kstep) : 0;
                if (CHECK && votes) bad |= coefficient_over<SIGNED>(v, vmax);
                x[0][k] = n0 + k * kstep < len ? reduce_coefficient<A, SIGNED>(v, pp) : 0u;
            }
            fwd_levels<A, 6, 1, 1, true, false, CUT>(x, tw + 1, pp.mod, octs);
        }
        u32* base = sm + c * VS + blk;
#pragma unroll
        for (int k = 0; k < E; ++k)
            if (!CUT || k < octs * (E / kOctants)) base[65 * k] = x[0][k];
    }
    if (CHECK && bad) votes[(blockIdx.x + threadIdx.x) % kAdmitSlots] = 1u;
    cp_async_wait_all();
    __syncthreads();
    // Pass 2: levels 6-11 on rows 64 blk + k, four-step twiddle, store.
    if (!CUT || blk < octs * (E / kOctants)) {
        const u32* base = sm + c * VS + 65 * blk;
        u32 x[1][E];
#pragma unroll
        for (int k = 0; k < E; ++k) x[0][k] = base[k];
        fwd_levels<A, 6, E, 1>(x, tw2 + blk, pp.mod);
        const uint2 fb = __ldg(pp.f4_b + ((size_t)col << 6) + (__brev((u32)blk) >> 26));
        const uint2* fac = fa + c * (E + 1);
        u32* dst = m.spec + ((size_t)(op * g.np + prime) << g.log_t) + ((u64)(blk * E) << log_c) + col;
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const u32 y = A::mulc(A::mulc(x[0][k], fac[__brev((u32)k) >> 26], pp.mod), fb, pp.mod);
            dst[(u64)k << log_c] = y;
        }
    }
}

template <class A, bool CUT>
__global__ void __launch_bounds__(kCol4Threads, kCol4LogG == 2 ? 2 : 1)
    k_inv_cols4(const __grid_constant__ TransformArgs g) {
    extern __shared__ u32 sm[];
    constexpr int G = kCol4G, LOG_G = kCol4LogG, VS = kCol4Vs, E = 64;
    const int prime = blockIdx.y;
    const PrimeParams& pp = g.ps.pr[prime];
    release_dependents();
    const Member m = member_after(g, blockIdx.z, false);
    const int octs = CUT ? octants_of(m.conv_len, g.log_t) : kOctants;
    const int log_c = g.log_c;
    const int c = threadIdx.x & (G - 1), blk = threadIdx.x >> LOG_G;
    uint2* tw = reinterpret_cast<uint2*>(sm + G * VS);
    if (threadIdx.x < 64) tw[threadIdx.x] = __ldg(pp.inv + threadIdx.x);
    __syncthreads();
    wait_prior_grid();  // the row pass's output
    // the CRT look-back flags of this product, cleared once every kernel before
    // this one has completed
    if (blockIdx.x == 0 && prime == 0) clear_flags(g, blockIdx.z);
    u32* const spec = m.spec + ((size_t)prime << g.log_t) + blockIdx.x * G + c;
    // Pass 1: levels 0-5 on rows 64 blk + k (bit-reversed spectrum in).
    if (!CUT || blk < octs * (E / kOctants)) {
        const u32* q = spec + ((u64)(blk * E) << log_c);
        u32 x[1][E];
#pragma unroll
        for (int k = 0; k < E; ++k) x[0][k] = __ldcg(q + ((u64)k << log_c));
        dit_levels<A, 6, 1, 1, 2>(x, tw, pp.mod);  // the row pass wrote [0, 2p)
        u32* base = sm + c * VS + 65 * blk;
#pragma unroll
        for (int k = 0; k < E; ++k) base[k] = x[0][k];
    }
    __syncthreads();
    // Pass 2: levels 6-11 on rows blk + 64k, canonical residues out.
    {
        const u32* base = sm + c * VS + blk;
        u32 x[1][E];
#pragma unroll
        for (int k = 0; k < E; ++k) x[0][k] = !CUT || k < octs * (E / kOctants) ? base[65 * k] : 0u;
        if constexpr (CUT) dit_levels_cut<A, 6, E>(x, pp.inv + blk, blk, pp.small_inv, pp.mod, octs);
        else dit_levels<A, 6, E, 1>(x, pp.inv + blk, pp.mod);
        u32* q = spec + ((u64)blk << log_c);
#pragma unroll
        for (int k = 0; k < E; ++k)
            if (!CUT || k < octs * (E / kOctants)) q[(u64)(k * E) << log_c] = A::canonical(x[0][k], pp.mod);
    }
}

// Persistent form of k_inv_cols4, for residues that start on a 16-byte boundary (a
// caller's scratch need not; k_inv_cols4 reads those): one CTA per SM loops over the
// (column group, prime, member) items. Once an item's second pass holds its points in
// registers, the shared buffer is free, and 16-byte cp.async copies
// bring the next item's residues into it while that pass computes and stores, so
// that the loads of one item overlap the butterflies of the one before. The copies
// land in a raw layout, row 64b + k of the 8 columns at word 520b + 8k: the first
// pass (rows 64 blk + k) reads it without bank conflicts, and it fits the buffer
// (64 x 520 <= 8 x kCol4Vs words). The first pass's inverse roots of every prime sit
// after it, then the roots of the current prime's second pass.
constexpr int kRawBlockWords = 520;
static_assert(kCol4G == 8 && 64 * kRawBlockWords <= kCol4G * kCol4Vs && kRawBlockWords % 32 == 8,
              "raw layout of the persistent inverse column pass");

static size_t col4p_smem(int np) {
    return (size_t)kCol4G * kCol4Vs * sizeof(u32) + ((size_t)np * 64 + 4096) * sizeof(uint2);
}

template <class A, bool CUT>
__global__ void __launch_bounds__(kCol4Threads, 1) k_inv_cols4p(const __grid_constant__ TransformArgs g) {
    extern __shared__ u32 sm[];
    constexpr int G = kCol4G, LOG_G = kCol4LogG, VS = kCol4Vs, E = 64, RB = kRawBlockWords;
    release_dependents();
    const int log_c = g.log_c;
    const u32 groups = 1u << (log_c - LOG_G), np = (u32)g.np;
    const u32 items = groups * np * (u32)(g.batch ? g.count : 1);
    const int c = threadIdx.x & (G - 1), blk = threadIdx.x >> LOG_G;
    uint2* tw = reinterpret_cast<uint2*>(sm + G * VS);  // [prime][64] inverse roots
    for (int i = threadIdx.x; i < g.np * 64; i += kCol4Threads) tw[i] = __ldg(g.ps.pr[i >> 6].inv + (i & 63));
    wait_prior_grid();  // the row pass's output
    // residues of item it: [prime][T] of its member, from column group * G
    auto source = [&](u32 it) -> u32* {
        const u32 group = it % groups, rest = it / groups;
        const Member mm = member_of(g, (int)(rest / np), false);
        return mm.spec + ((size_t)(rest % np) << g.log_t) + (size_t)group * G;
    };
    auto octants = [&](u32 it) {
        return CUT ? octants_of(member_of(g, (int)(it / groups / np), false).conv_len, g.log_t) : kOctants;
    };
    auto prefetch = [&](u32 it) {
        const u32* src = source(it);
        const int n = octants(it) * (2 * 4096 / kOctants);
        for (int j = threadIdx.x; j < n; j += kCol4Threads) {
            const int r = j >> 1, h = j & 1;
            cp_async16(sm + RB * (r >> 6) + 8 * (r & 63) + 4 * h, src + ((u64)r << log_c) + 4 * h);
        }
        cp_async_commit();
    };
    uint2* const tw2 = tw + g.np * 64;  // level-major roots of the current prime
    int staged = -1;
    if (blockIdx.x < items) prefetch(blockIdx.x);
    for (u32 it = blockIdx.x; it < items; it += gridDim.x) {
        const u32 group = it % groups, rest = it / groups;
        const int prime = (int)(rest % np), member = (int)(rest / np);
        const PrimeParams& pp = g.ps.pr[prime];
        // the CRT look-back flags of this product, cleared once every kernel before
        // this one has completed
        if (group == 0 && prime == 0) clear_flags(g, member);
        if (prime != staged) {  // every thread has used the last prime's (barrier at the loop's end)
            stage_table<kCol4Threads>(tw2, pp.inv, 4096);
            staged = prime;
        }
        cp_async_wait_all();
        __syncthreads();
        // Pass 1: levels 0-5 on rows 64 blk + k (bit-reversed spectrum in).
        const int octs = octants(it);
        const bool used = !CUT || blk < octs * (E / kOctants);
        u32 x[1][E];
        if (used) {
            const u32* raw = sm + RB * blk + c;
#pragma unroll
            for (int k = 0; k < E; ++k) x[0][k] = raw[8 * k];
            dit_levels<A, 6, 1, 1, 2>(x, tw + 64 * prime, pp.mod);  // [0, 2p) in
        }
        __syncthreads();  // every raw read is done before the padded layout overwrites it
        if (used) {
            u32* base = sm + c * VS + 65 * blk;
#pragma unroll
            for (int k = 0; k < E; ++k) base[k] = x[0][k];
        }
        __syncthreads();
        // Pass 2: levels 6-11 on rows blk + 64k, canonical residues out; the next
        // item's residues come in behind it.
        {
            const u32* base = sm + c * VS + blk;
#pragma unroll
            for (int k = 0; k < E; ++k) x[0][k] = !CUT || k < octs * (E / kOctants) ? base[65 * k] : 0u;
        }
        __syncthreads();
        if (it + gridDim.x < items) prefetch(it + gridDim.x);
        if constexpr (CUT) dit_levels_cut<A, 6, E>(x, tw2 + blk, blk, pp.small_inv, pp.mod, octs);
        else dit_levels<A, 6, E, 1>(x, tw2 + blk, pp.mod);
        u32* q = source(it) + c + ((u64)blk << log_c);
#pragma unroll
        for (int k = 0; k < E; ++k)
            if (!CUT || k < octs * (E / kOctants)) q[(u64)(k * E) << log_c] = A::canonical(x[0][k], pp.mod);
        __syncthreads();  // the staged roots may be replaced
    }
    cp_async_wait_all();
}

// Rows per CTA of the row pass: enough that every thread owns a register block of
// the first pass (2^(log_c - kMaxRB) blocks per row).
__host__ __device__ constexpr int row_log_rpc(int log_c) {
    return log_c - kMaxRB >= ilog2(row_threads(log_c)) ? 0 : ilog2(row_threads(log_c)) - (log_c - kMaxRB);
}

// Whether the row pass lets the inverse column pass in only after its own wait. Let in
// before, while the forward columns still drain, that pass's few CTAs (two per SM at
// T = 2^17 and 2^18) gather on the SMs that empty first and run unevenly: 90,000^2 33.4
// against 26.8 us, 130,000^2 36.1 and 31.5, 60,000^2 20.8 and 20.5. Shorter rows lose the
// overlap (4,000^2 10.8 against 11.4 us), longer ones have CTAs for every SM several
// times over (4M^2 638 against 643 us).
template <int LOG_C>
constexpr bool kRowsReleaseLate = LOG_C == 9 || LOG_C == 10;

// Row pass: forward rows of a (and b), pointwise product, inverse rows, inverse
// four-step twiddle with the 2^32 / T scale. grid = (R / RPC, np); writes over a's
// rows. A CTA owns RPC consecutive rows; shared memory holds vectors [RPC][a, b].
//
// Shared memory is touched as little as the register blocks allow: the first
// forward pass reads the rows from global memory, the last forward pass, the
// pointwise product and the first inverse pass run on the same registers (both
// work on blocks of 2^RBL consecutive points), and the last inverse pass applies
// the twiddle and writes global memory.
template <class A, int MODE, int LOG_C>
__global__ void __launch_bounds__(row_threads(LOG_C)) k_rows(const __grid_constant__ TransformArgs g) {
    constexpr int kRowThreads = row_threads(LOG_C);
    extern __shared__ u32 sm[];
    constexpr int C = 1 << LOG_C;
    constexpr int VS = padded_len(C);
    constexpr int NV = MODE == kRowMul ? 2 : 1;  // a (and b), transformed together
    constexpr int LOG_RPC = row_log_rpc(LOG_C);
    constexpr int RPC = 1 << LOG_RPC;
    constexpr int RB = kMaxRB;
    constexpr int RBL = LOG_C % RB ? LOG_C % RB : RB;  // levels of the fused middle pass
    constexpr int LL = LOG_C - RBL;              // its first forward level
    constexpr int NL = 1 << kRowTwLoBits, NH = C >> kRowTwLoBits;
    static_assert(LOG_C > RB && LOG_C > kRowTwLoBits, "at least two passes each way");
    const int prime = blockIdx.y;
    const int row0 = blockIdx.x << LOG_RPC;
    const PrimeParams& pp = g.ps.pr[prime];
    const Member m = member_after(g, blockIdx.z, NV == 1);
    if constexpr (!kRowsReleaseLate<LOG_C>) release_dependents();
    // rows of octants that the member's coefficients do not need (a CTA whose first row
    // is needed may hold unneeded ones as well: what it makes of them is not read)
    if (g.cut && row0 >= octants_of(m.conv_len, g.log_t) << (g.log_r - 3)) return;
    u32* ra = m.spec + ((size_t)prime << g.log_t) + ((size_t)row0 << LOG_C);
    const u32* rb = m.spec + ((size_t)(g.np + prime) << g.log_t) + ((size_t)row0 << LOG_C);
    // the stored spectrum of the rows (kRowFwd writes it, kRowPre multiplies by it)
    u32* rs = g.shared_spec + ((size_t)prime << g.log_t) + ((size_t)row0 << LOG_C);
    // The rows' inverse four-step factors: RPC x 64 low-digit entries, RPC x C/64 high.
    uint2* il = reinterpret_cast<uint2*>(sm + RPC * NV * VS);
    uint2* ih = il + RPC * NL;
    if constexpr (MODE != kRowFwd) {
        const uint2* lo = pp.i4_lo + (size_t)row0 * NL;
        const uint2* hi = pp.i4_hi + (size_t)row0 * NH;
        for (int i = threadIdx.x; i < RPC * (NL + NH); i += kRowThreads)
            il[i] = __ldg(i < RPC * NL ? lo + i : hi + (i - RPC * NL));
    }
    wait_prior_grid();  // the column pass's output
    if constexpr (kRowsReleaseLate<LOG_C>) release_dependents();
    // First forward pass: global -> shared. Block gg of a row holds points gg + k * HQ.
    {
        constexpr int LOG_HQ = LOG_C - RB;
        constexpr int HQ = 1 << LOG_HQ;
#pragma unroll 1
        for (int it = threadIdx.x; it < (RPC << LOG_HQ); it += kRowThreads) {
            const int r = it >> LOG_HQ, gg = it & (HQ - 1);
            const size_t off = ((size_t)r << LOG_C) + gg;
            u32 x[NV][1 << RB];
#pragma unroll
            for (int k = 0; k < (1 << RB); ++k) {
                x[0][k] = __ldcg(ra + off + k * HQ);
                if constexpr (NV == 2) x[NV - 1][k] = __ldcg(rb + off + k * HQ);
            }
            fwd_levels<A, RB, 1, NV, true>(x, pp.small_fwd + 1, pp.mod);
            u32* base = sm + r * NV * VS + pad_index(gg);
#pragma unroll
            for (int q = 0; q < NV; ++q)
#pragma unroll
                for (int k = 0; k < (1 << RB); ++k) base[q * VS + slot_offset<HQ>(k)] = x[q][k];
        }
    }
    __syncthreads();
    fwd_range<A, LOG_C, kRowThreads, RPC * NV, VS, RB, LL>(sm, pp.fwd + kFwd4, pp.mod);
    // Last forward pass, pointwise product, first inverse pass: blocks of 2^RBL
    // consecutive points (the inverse levels' twiddles are shared by all blocks).
    {
        constexpr int E = 1 << RBL;
#pragma unroll 1
        for (int it = threadIdx.x; it < (RPC << (LOG_C - RBL)); it += kRowThreads) {
            const int r = it >> (LOG_C - RBL), gg = it & ((C >> RBL) - 1);
            u32* base = sm + r * NV * VS + pad_index(gg << RBL);
            u32 x[NV][E];
#pragma unroll
            for (int q = 0; q < NV; ++q)
#pragma unroll
                for (int k = 0; k < E; ++k) x[q][k] = base[q * VS + k];
            // of the two factors, the Montgomery product takes one below 4p and one
            // below 2p; the product is below 3p, so the first inverse level
            // (twiddle 1) needs no products either
            u32 y[E];
            if constexpr (MODE == kRowPre) {  // the other factor is the stored spectrum
                const u32* in = rs + ((size_t)r << LOG_C) + (gg << RBL);
#pragma unroll
                for (int k = 0; k < E; ++k) y[k] = __ldcg(in + k);
            }
            fwd_levels<A, RBL, (1 << LL), NV>(x, pp.fwd + kFwd4 + (1 << LL) + gg, pp.mod);
            if constexpr (MODE != kRowPre) {
#pragma unroll
                for (int k = 0; k < E; ++k) y[k] = A::to_2p(x[NV - 1][k], pp.mod);
            }
            if constexpr (MODE == kRowFwd) {  // the reduced spectrum, stored
                u32* out = rs + ((size_t)r << LOG_C) + (gg << RBL);
#pragma unroll
                for (int k = 0; k < E; ++k) out[k] = y[k];
            } else {
#pragma unroll
                for (int k = 0; k < E; ++k) x[0][k] = A::pointwise(x[0][k], y[k], pp.mod, pp.pni);
                u32(&z)[1][E] = *reinterpret_cast<u32(*)[1][E]>(&x[0]);
                dit_levels<A, RBL, 1, 1, 1>(z, pp.small_inv, pp.mod);
#pragma unroll
                for (int k = 0; k < E; ++k) base[k] = x[0][k];
            }
        }
    }
    if constexpr (MODE == kRowFwd) return;
    __syncthreads();
    dit_range<A, LOG_C, kRowThreads, RPC, NV * VS, RBL, LOG_C - RB>(sm, pp.inv, pp.mod);
    // Last inverse pass: shared -> global, times the inverse four-step twiddle of
    // n2 = 64 hi + lo (i4_lo of lo, i4_hi of hi with the scale folded in).
    {
        constexpr int LOG_HS = LOG_C - RB;
        constexpr int HS = 1 << LOG_HS;
#pragma unroll 1
        for (int it = threadIdx.x; it < (RPC << LOG_HS); it += kRowThreads) {
            const int r = it >> LOG_HS, gg = it & (HS - 1);
            const u32* base = sm + r * NV * VS + pad_index(gg);
            u32 x[1][1 << RB];
#pragma unroll
            for (int k = 0; k < (1 << RB); ++k) x[0][k] = base[slot_offset<HS>(k)];
            dit_levels<A, RB, HS, 1>(x, pp.inv + gg, pp.mod);
            const uint2* lo = il + r * NL;
            const uint2* hi = ih + r * NH;
            u32* out = ra + ((size_t)r << LOG_C);
#pragma unroll
            for (int k = 0; k < (1 << RB); ++k) {
                const int n2 = gg + k * HS;
                out[n2] = A::mulc(A::mulc(x[0][k], lo[n2 & (NL - 1)], pp.mod), hi[n2 >> kRowTwLoBits], pp.mod);
            }
        }
    }
}

// Column pass of the inverse four-step: inverse columns, canonical residues in place.
template <class A, int LOG_R, bool CUT>
__global__ void __launch_bounds__(kThreads) k_inv_cols(const __grid_constant__ TransformArgs g) {
    extern __shared__ u32 sm[];
    using M = ColumnMap<LOG_R>;
    constexpr int B = M::SWEEPS < 8 ? M::SWEEPS : 8;
    static_assert(M::SWEEPS % B == 0 && (B * M::RS) % 32 == 0, "column batches");
    const int prime = blockIdx.y;
    const PrimeParams& pp = g.ps.pr[prime];
    release_dependents();
    const Member m = member_after(g, blockIdx.z, false);
    const int octs = CUT ? octants_of(m.conv_len, g.log_t) : kOctants;
    const u64 step = (u64)M::RS << g.log_c;
    u32* const base = m.spec + ((size_t)prime << g.log_t) + ((u64)M::row0() << g.log_c) +
                      (blockIdx.x << M::LOG_G) + M::col();
    u32* s = sm + M::slot0();
    uint2* tw = reinterpret_cast<uint2*>(sm + M::G * M::VS);
    load_table<LOG_R>(tw, pp.inv);
    wait_prior_grid();  // the row pass's output
    if (blockIdx.x == 0 && prime == 0) clear_flags(g, blockIdx.z);  // after every earlier kernel
    u32* q = base;
#pragma unroll 1
    for (int k0 = 0; k0 < (CUT ? octs * M::SWEEPS / kOctants : M::SWEEPS); k0 += B) {
        u32 x[B];
#pragma unroll
        for (int u = 0; u < B; ++u)
            x[u] = !CUT || k0 + u < octs * M::SWEEPS / kOctants ? __ldcg(q + u * step) : 0u;
        q += B * step;
        u32* sk = s + slot_offset<M::RS>(k0);
#pragma unroll
        for (int u = 0; u < B; ++u) sk[slot_offset<M::RS>(u)] = x[u];
    }
    __syncthreads();
    // Every inverse pass but the last in shared memory (the short one first) ...
    constexpr int RB = kMaxRB;
    constexpr int R0 = LOG_R % RB;
    if constexpr (R0 > 0) {
        dit_pass<A, LOG_R, 0, R0, kThreads, M::G, M::VS, CUT>(sm, tw, pp.mod, octs);
        __syncthreads();
    }
    dit_range<A, LOG_R, kThreads, M::G, M::VS, R0, LOG_R - RB, CUT>(sm, tw, pp.mod, octs);
    // ... and the last one straight to global memory as canonical residues. Item it
    // takes column c = it mod G and block gg = it / G (rows gg + k * HS), so a warp
    // reads distinct banks and writes four rows of G consecutive residues at a time.
    {
        constexpr int LOG_HS = LOG_R - RB, HS = 1 << LOG_HS;
        u32* const out0 = m.spec + ((size_t)prime << g.log_t) + (blockIdx.x << M::LOG_G);
        const u64 kstep = (u64)HS << g.log_c;
#pragma unroll 1
        for (int it = threadIdx.x; it < (M::G << LOG_HS); it += kThreads) {
            const int c = it & (M::G - 1), gg = it >> M::LOG_G;
            const u32* base = sm + c * M::VS + pad_index(gg);
            u32 x[1][1 << RB];
#pragma unroll
            for (int k = 0; k < (1 << RB); ++k)
                x[0][k] = !CUT || k < octs * ((1 << RB) / kOctants) ? base[slot_offset<HS>(k)] : 0u;
            if constexpr (CUT) dit_levels_cut<A, RB, HS>(x, tw + gg, gg, pp.small_inv, pp.mod, octs);
            else dit_levels<A, RB, HS, 1>(x, tw + gg, pp.mod);
            u32* out = out0 + ((u64)gg << g.log_c) + c;
#pragma unroll
            for (int k = 0; k < (1 << RB); ++k)
                if (!CUT || k < octs * ((1 << RB) / kOctants)) out[k * kstep] = A::canonical(x[0][k], pp.mod);
        }
    }
}

// ---------------------------------------------------------------------------------
// Four-step factor tables (layouts in launch.h). One thread per entry: the exponent
// of the entry, then the power as a product of the tabulated squares (Shoup
// products by constants), then its companion floor(x * 2^32 / p).

__device__ __forceinline__ u32 power_of(const uint2* pow2, u64 e, int bits, u32 p) {
    u32 x = 1;
    for (int i = 0; i < bits; ++i)
        if ((e >> i) & 1) x = sub_if_ge(shoup_mul(x, pow2[i].x, pow2[i].y, Mod{p, 0u - p}), p);
    return x;
}

__global__ void __launch_bounds__(256) k_step_tables(const __grid_constant__ StepTableBuild b) {
    u64 n[4];
    step_table_sizes(b.log_t, b.log_r, n);
    const u64 mask = ((u64)1 << b.log_t) - 1;
    const int log_rs = step_log_u(b.log_r), log_sw = b.log_r - log_rs, log_nh = b.log_c - kRowTwLoBits;
    const u64 total = n[0] + n[1] + n[2] + n[3];
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (u64)gridDim.x * blockDim.x) {
        u64 k = i;
        u32 x;
        uint2* out;
        if (k < n[0]) {  // w^(col * u * SW)
            const u64 col = k >> log_rs, u = k & ((1u << log_rs) - 1);
            x = power_of(b.fwd_pow, ((col * u) << log_sw) & mask, b.log_t, b.p);
            out = b.f4_a + k;
        } else if ((k -= n[0]) < n[1]) {  // w^(col * j), and w_(2 SW)^j times that
            const int pair = step_pairs(b.log_r);
            const u64 col = k >> (log_sw + pair), j = (k >> pair) & (((u64)1 << log_sw) - 1);
            const u64 level = pair && (k & 1) ? j << (b.log_t - log_sw - 1) : 0;
            x = power_of(b.fwd_pow, (col * j + level) & mask, b.log_t, b.p);
            out = b.f4_b + k;
        } else if ((k -= n[1]) < n[2]) {  // w^(-k1 * lo)
            const u64 row = k >> kRowTwLoBits, lo = k & ((1u << kRowTwLoBits) - 1);
            const u64 k1 = __brev((u32)row) >> (32 - b.log_r);
            x = power_of(b.inv_pow, (k1 * lo) & mask, b.log_t, b.p);
            out = b.i4_lo + k;
        } else {  // w^(-k1 * 64 * hi) * scale
            k -= n[2];
            const u64 row = k >> log_nh, hi = k & (((u64)1 << log_nh) - 1);
            const u64 k1 = __brev((u32)row) >> (32 - b.log_r);
            x = power_of(b.inv_pow, ((k1 * hi) << kRowTwLoBits) & mask, b.log_t, b.p);
            x = sub_if_ge(shoup_mul(x, b.scale.x, b.scale.y, Mod{b.p, 0u - b.p}), b.p);
            out = b.i4_hi + k;
        }
        *out = make_uint2(x, (u32)(((u64)x << 32) / b.p));
    }
}

cudaError_t launch_step_tables(const StepTableBuild& b, cudaStream_t st) {
    u64 n[4];
    step_table_sizes(b.log_t, b.log_r, n);
    const u64 total = n[0] + n[1] + n[2] + n[3];
    const unsigned blocks = (unsigned)std::min<u64>((total + 255) / 256, 152 * 16);
    k_step_tables<<<blocks, 256, 0, st>>>(b);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------
// Launchers: one instantiation per transform size. The lazy arithmetic covers
// T <= 2^23 (one-CTA sizes 2^4..2^13, columns 2^6..2^11, rows 2^7..2^13); the wide
// arithmetic covers T = 2^24, 2^25 (columns 2^12, rows 2^12..2^13) and T = 2^22,
// 2^23 when the wide primes save one (columns 2^10, rows 2^12..2^13).

// Column residues plus the level root table (8-byte entries, 16-byte aligned); the
// forward pass adds its per-sweep four-step factors (G rows of SW + 1 entries).
static size_t col_smem(int log_r, bool fwd) {
    const int log_g = col_group_log(log_r);
    const size_t words = (size_t)col_vstride(log_r) * (1 << log_g);
    const size_t sweeps = (size_t)1 << (log_r - col_log_rs(log_r));
    return ((words * sizeof(u32) + 15) & ~(size_t)15) + ((size_t)8 << log_r) +
           (fwd ? 8 * ((size_t)1 << log_g) * (sweeps + 1) : 0);
}

// Row residues (one or two vectors per row) plus the rows' inverse four-step factors.
static size_t row_smem(int log_c, int mode) {
    const size_t rpc = (size_t)1 << row_log_rpc(log_c);
    return rpc * ((size_t)(mode == kRowMul ? 2 : 1) * padded_len(1 << log_c) * sizeof(u32) +
                  8 * (((size_t)1 << kRowTwLoBits) + ((size_t)1 << (log_c - kRowTwLoBits))));
}

// Column data plus the f4_a rows (and staged roots) of the two-pass forward kernel.
template <class A, int LOG_R>
static size_t col2_smem(bool fwd) {
    using K = Columns<LOG_R>;
    const size_t roots = kStageCols2<A, LOG_R> ? (K::EB - 1) * K::EA : 0;
    return (size_t)K::G * K::VS * sizeof(u32) + (fwd ? (K::G * (K::EB + 1) + roots) * sizeof(uint2) : 0);
}

// One preference for the columns and rows that lengths up to 2^19 run, the driver's for
// longer ones (transform_common.cuh, kCarveout).
static constexpr int col_carveout(int log_r) { return log_r <= 9 ? kCarveout : -1; }
static constexpr int row_carveout(int log_c) { return log_c <= 10 ? kCarveout : -1; }

// The forward column kernel of a transform and its instantiations' attributes: unsigned
// convolutions take the checking one when they carry votes, signed ones always do (a
// product is never signed); CUT ones serve products shorter than their transform.
template <class A, int L, bool CUT>
static cudaError_t fwd_cols_cut(const TransformArgs& g, bool square, bool sign, cudaStream_t st, bool init) {
    const unsigned ops = g.op_count ? g.op_count : (square ? 1 : 2);
    const unsigned zdim = g.batch ? (g.a_only ? 1 : 2) * g.count + g.with_args : ops;
    const bool check = g.batch ? g.admit != 0 : g.votes != nullptr;
    void (*plain)(TransformArgs), (*checked)(TransformArgs), (*with_sign)(TransformArgs);
    int log_g = col_group_log(L), threads = kThreads;
    size_t smem;
    if constexpr (L <= 10) {
        plain = k_fwd_cols2<A, false, L, CUT>, checked = k_fwd_cols2<A, false, L, CUT, true>;
        with_sign = k_fwd_cols2<A, true, L, CUT>;
        smem = col2_smem<A, L>(true), log_g = Columns<L>::LOG_G, threads = Columns<L>::NT;
    } else if constexpr (L == kCol4LogR) {
        plain = k_fwd_cols4<A, false, CUT>, checked = k_fwd_cols4<A, false, CUT, true>;
        with_sign = k_fwd_cols4<A, true, CUT>;
        smem = col4_smem(true), log_g = kCol4LogG, threads = kCol4Threads;
    } else {
        plain = k_fwd_cols<A, false, L, CUT>, checked = k_fwd_cols<A, false, L, CUT, true>;
        with_sign = k_fwd_cols<A, true, L, CUT>;
        smem = col_smem(L, true);
    }
    if (init) {
        cudaError_t e = opt_in(plain, col_carveout(L));
        if (e == cudaSuccess) e = opt_in(checked, col_carveout(L));
        return e == cudaSuccess ? opt_in(with_sign, col_carveout(L)) : e;
    }
    const dim3 grid((1u << (g.log_c - log_g)) * (unsigned)g.np, 1, zdim);
    // an operand that arrives by an event (op_count) starts normally as well
    return launch_kernel(sign ? with_sign : check ? checked : plain, first_dependent(g), 0, grid, dim3(threads), smem, st, g);
}

template <class A, int L>
static cudaError_t fwd_cols_at(const TransformArgs& g, bool square, bool sign, cudaStream_t st, bool init) {
    if (init) {
        const cudaError_t e = fwd_cols_cut<A, L, false>(g, square, sign, st, true);
        return e == cudaSuccess ? fwd_cols_cut<A, L, true>(g, square, sign, st, true) : e;
    }
    return g.cut ? fwd_cols_cut<A, L, true>(g, square, sign, st, false)
                 : fwd_cols_cut<A, L, false>(g, square, sign, st, false);
}

template <class A, int L>
static cudaError_t rows_at(const TransformArgs& g, int mode, cudaStream_t st, bool init) {
    auto k = mode == kRowMul ? k_rows<A, kRowMul, L>
             : mode == kRowSqr ? k_rows<A, kRowSqr, L>
             : mode == kRowFwd ? k_rows<A, kRowFwd, L>
                               : k_rows<A, kRowPre, L>;
    if (init) return opt_in(k, row_carveout(L));
    // the rows of the octants that a single product needs; a batch's members decide theirs
    unsigned rows = 1u << g.log_r;
    if (g.cut && !g.batch) rows = (rows >> 3) * (unsigned)octants_of(g.conv_len, g.log_t);
    const dim3 grid((rows + (1u << row_log_rpc(L)) - 1) >> row_log_rpc(L), g.np, g.batch ? g.count : 1);
    const size_t smem = row_smem(L, mode);
    return launch_dependent(k, grid, dim3(row_threads(L)), smem, st, g);
}

template <class A, int L, bool CUT>
static cudaError_t inv_cols_cut(const TransformArgs& g, cudaStream_t st, bool init) {
    const int log_g = L == kCol4LogR ? kCol4LogG : L <= 10 ? Columns<L>::LOG_G : col_group_log(L);
    const dim3 grid(1u << (g.log_c - log_g), g.np, g.batch ? g.count : 1);
    if constexpr (L <= 10) {
        auto k = k_inv_cols2<A, L, CUT>;
        if (init) return opt_in(k, col_carveout(L));
        return launch_dependent(k, grid, dim3(Columns<L>::NT), col2_smem<A, L>(false), st, g);
    } else if constexpr (L == kCol4LogR) {
        auto p = k_inv_cols4p<A, CUT>;
        auto k = k_inv_cols4<A, CUT>;
        if (init) {
            const cudaError_t e = opt_in(p, col_carveout(L));
            return e == cudaSuccess ? opt_in(k, col_carveout(L)) : e;
        }
        // members of a batch start on 256-byte boundaries, blocks of a split product a
        // multiple of 256 bytes apart in the caller's scratch
        const u32* first = g.batch ? g.arena : g.spec;
        if ((reinterpret_cast<uintptr_t>(first) & 15) != 0)
            return launch_dependent(k, grid, dim3(kCol4Threads), col4_smem(false), st, g);
        const unsigned items = grid.x * grid.y * grid.z;
        return launch_dependent(p, dim3(std::min(items, (unsigned)sm_count())), dim3(kCol4Threads), col4p_smem(g.np),
                                st, g);
    } else {
        auto k = k_inv_cols<A, L, CUT>;
        if (init) return opt_in(k, col_carveout(L));
        return launch_dependent(k, grid, dim3(kThreads), col_smem(L, false), st, g);
    }
}

template <class A, int L>
static cudaError_t inv_cols_at(const TransformArgs& g, cudaStream_t st, bool init) {
    if (init) {
        const cudaError_t e = inv_cols_cut<A, L, false>(g, st, true);
        return e == cudaSuccess ? inv_cols_cut<A, L, true>(g, st, true) : e;
    }
    return g.cut ? inv_cols_cut<A, L, true>(g, st, false) : inv_cols_cut<A, L, false>(g, st, false);
}

static cudaError_t fwd_cols_any(const TransformArgs& g, bool square, bool sign, cudaStream_t st, bool init) {
    if (g.wide) {
        if (g.log_r == 12) return fwd_cols_at<WideArith, 12>(g, square, sign, st, init);
        if (g.log_r == 10) return fwd_cols_at<WideArith, 10>(g, square, sign, st, init);
        return cudaErrorInvalidValue;
    }
    switch (g.log_r) {
        case 6: return fwd_cols_at<LazyArith, 6>(g, square, sign, st, init);
        case 7: return fwd_cols_at<LazyArith, 7>(g, square, sign, st, init);
        case 8: return fwd_cols_at<LazyArith, 8>(g, square, sign, st, init);
        case 9: return fwd_cols_at<LazyArith, 9>(g, square, sign, st, init);
        case 10: return fwd_cols_at<LazyArith, 10>(g, square, sign, st, init);
        case 11: return fwd_cols_at<LazyArith, 11>(g, square, sign, st, init);
        default: return cudaErrorInvalidValue;
    }
}

static cudaError_t rows_any(const TransformArgs& g, int mode, cudaStream_t st, bool init) {
    if (g.wide) {
        if (g.log_c == 12) return rows_at<WideArith, 12>(g, mode, st, init);
        if (g.log_c == 13) return rows_at<WideArith, 13>(g, mode, st, init);
        return cudaErrorInvalidValue;
    }
    switch (g.log_c) {
        case 7: return rows_at<LazyArith, 7>(g, mode, st, init);
        case 8: return rows_at<LazyArith, 8>(g, mode, st, init);
        case 9: return rows_at<LazyArith, 9>(g, mode, st, init);
        case 10: return rows_at<LazyArith, 10>(g, mode, st, init);
        case 11: return rows_at<LazyArith, 11>(g, mode, st, init);
        case 12: return rows_at<LazyArith, 12>(g, mode, st, init);
        case 13: return rows_at<LazyArith, 13>(g, mode, st, init);
        default: return cudaErrorInvalidValue;
    }
}

static cudaError_t inv_cols_any(const TransformArgs& g, cudaStream_t st, bool init) {
    if (g.wide) {
        if (g.log_r == 12) return inv_cols_at<WideArith, 12>(g, st, init);
        if (g.log_r == 10) return inv_cols_at<WideArith, 10>(g, st, init);
        return cudaErrorInvalidValue;
    }
    switch (g.log_r) {
        case 6: return inv_cols_at<LazyArith, 6>(g, st, init);
        case 7: return inv_cols_at<LazyArith, 7>(g, st, init);
        case 8: return inv_cols_at<LazyArith, 8>(g, st, init);
        case 9: return inv_cols_at<LazyArith, 9>(g, st, init);
        case 10: return inv_cols_at<LazyArith, 10>(g, st, init);
        case 11: return inv_cols_at<LazyArith, 11>(g, st, init);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_fwd_cols(const TransformArgs& g, bool square, bool sign, cudaStream_t st) {
    return fwd_cols_any(g, square, sign, st, false);
}
cudaError_t launch_rows(const TransformArgs& g, int mode, cudaStream_t st) { return rows_any(g, mode, st, false); }
cudaError_t launch_inv_cols(const TransformArgs& g, cudaStream_t st) { return inv_cols_any(g, st, false); }

// Raises the dynamic shared-memory limit of every instantiation (both operand
// modes) on the current device.
cudaError_t init_transform_kernels() {
    cudaError_t e = init_small_kernels();
    TransformArgs g{};
    for (int sq = 0; sq < 2; ++sq)
        for (int sg = 0; sg < 2; ++sg) {
            for (int w = 0; w < 2; ++w) {
                g.wide = w;
                for (int l = 6; l <= 13 && e == cudaSuccess; ++l) {
                    g.log_r = l;
                    g.log_c = l;
                    const bool col_ok = w ? l == 12 || l == 10 : l <= 11;
                    const bool row_ok = w ? l >= 12 : l >= 7;
                    if (col_ok) e = fwd_cols_any(g, sq, sg, 0, true);
                    for (int mode = 0; mode < 4 && e == cudaSuccess && row_ok && sg == 0 && sq == 0; ++mode)
                        e = rows_any(g, mode, 0, true);
                    if (e == cudaSuccess && col_ok) e = inv_cols_any(g, 0, true);
                }
            }
        }
    return e;
}

}  // namespace ntt
