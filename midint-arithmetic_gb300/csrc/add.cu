// add.cu -- batched big-integer addition by carry-lookahead over thread groups.
//
// Counterpart of the reference's baddKer / a6pb10Ker (cuda/ker-addition.cu.h:
// 227-328).  The reference stages each operand global -> shared -> registers
// with 8-byte loads (cpGlb2Reg, cuda/ker-helpers.cu.h:121-144) and resolves the
// carries with a Hillis-Steele scan over volatile shared memory plus four block
// barriers (cuda/ker-addition.cu.h:88-134).  Here every thread loads its Q
// limbs straight into registers with 128-bit streaming loads, and the carries
// of a whole warp are resolved by two ballots and one 64-bit add
// (mi::group_carry); only integers wider than one warp touch shared memory, one
// word per warp.
//
// Mapping: a group of GS threads (power of two) owns one instance, thread t of
// the group owns limbs [t*Q, t*Q+Q).  GS*Q >= limbs; limbs beyond the instance
// are zero and never stored.  A block of max(256, GS) threads holds 256/GS
// groups and strides over the batch.  (Rows that allow no 16-byte access: the
// group's limbs are mostly dealt in rows instead, k_add_rows.)
#include <cstdio>

#include "common.cuh"
#include "kernels.h"

namespace mi {
namespace {

template <typename L>
struct Lim;
template <>
struct Lim<uint64_t> {
    using dev_t = unsigned long long;
};
template <>
struct Lim<uint32_t> {
    using dev_t = unsigned int;
};

// Streaming (evict-first) scalar load/store; every input limb is read once.
template <typename L>
__device__ __forceinline__ L ld_stream(const L* p) {
    using D = typename Lim<L>::dev_t;
    return (L)__ldcs(reinterpret_cast<const D*>(p));
}
template <typename L>
__device__ __forceinline__ void st_stream(L* p, L v) {
    using D = typename Lim<L>::dev_t;
    __stcs(reinterpret_cast<D*>(p), (D)v);
}

template <typename L, int Q>
__device__ __forceinline__ void unpack16(const uint4& t, L* v) {
    if constexpr (sizeof(L) == 8) {
        v[0] = (uint64_t(t.y) << 32) | t.x;
        v[1] = (uint64_t(t.w) << 32) | t.z;
    } else {
        v[0] = t.x;
        v[1] = t.y;
        v[2] = t.z;
        v[3] = t.w;
    }
}
template <typename L, int Q>
__device__ __forceinline__ uint4 pack16(const L* v) {
    uint4 t;
    if constexpr (sizeof(L) == 8) {
        t.x = uint32_t(v[0]);
        t.y = uint32_t(v[0] >> 32);
        t.z = uint32_t(v[1]);
        t.w = uint32_t(v[1] >> 32);
    } else {
        t.x = v[0];
        t.y = v[1];
        t.z = v[2];
        t.w = v[3];
    }
    return t;
}

// How a thread reaches its limbs: whole 16-byte words of a 16-byte aligned row,
// consecutive limbs one by one on other rows, or dealt in rows (k_add_rows).
enum Access : int { WORDS16, LIMBS, ROWS };

// Loads the chunk [start, start+Q) of one instance row, zero beyond m.
template <typename L, int Q, int ACCESS>
__device__ __forceinline__ void load_chunk(const L* __restrict__ row, uint32_t start, uint32_t m, bool valid,
                                           L (&v)[Q]) {
    constexpr int PER = 16 / sizeof(L);
    if (ACCESS == WORDS16 && valid && start + Q <= m) {
        const uint4* p = reinterpret_cast<const uint4*>(row + start);
#pragma unroll
        for (int k = 0; k < Q / PER; ++k) {
            const uint4 t = __ldcs(p + k);
            unpack16<L, Q>(t, &v[k * PER]);
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) v[q] = (valid && start + q < m) ? ld_stream(row + start + q) : L(0);
}

template <typename L, int Q, int ACCESS>
__device__ __forceinline__ void store_chunk(L* __restrict__ row, uint32_t start, uint32_t m, bool valid,
                                            const L (&v)[Q]) {
    constexpr int PER = 16 / sizeof(L);
    if (!valid) return;
    if (ACCESS == WORDS16 && start + Q <= m) {
        uint4* p = reinterpret_cast<uint4*>(row + start);
#pragma unroll
        for (int k = 0; k < Q / PER; ++k) __stcs(p + k, pack16<L, Q>(&v[k * PER]));
        return;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q)
        if (start + q < m) st_stream(row + start + q, v[q]);
}

// x + y over the group, result in r; returns the group's carry-out.
template <typename L, int Q, int GS>
__device__ __forceinline__ uint32_t group_add(const L (&x)[Q], const L (&y)[Q], L (&r)[Q], uint32_t* scratch) {
    bool g, p;
    chunk_add<L, Q>(x, y, r, g, p);
    uint32_t gc;
    const uint32_t cin = group_carry<GS>(g, p, 0u, &gc, scratch);
    chunk_inc<L, Q>(r, cin);
    return gc;
}

// The value v of thread t-1 of the group (0 for t == 0).  Groups wider than a
// warp pass the last lane's value through one shared word per warp.
template <int GS>
__device__ __forceinline__ uint64_t group_shift_up(uint64_t v, uint32_t t, uint64_t* xs) {
    if constexpr (GS <= 32) {
        const uint64_t u = __shfl_up_sync(group_lanes<GS>(), v, 1, GS);
        return t == 0 ? 0ull : u;
    } else {
        const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
        const uint64_t u = __shfl_up_sync(MI_FULL_MASK, v, 1);
        if (lane == 31) xs[warp] = v;
        __syncthreads();
        const uint64_t w = (lane == 0) ? ((t == 0) ? 0ull : xs[warp - 1]) : u;
        __syncthreads();
        return w;
    }
}

template <typename L, int Q, int GS, int ACCESS, int OP>
__global__ void __launch_bounds__(GS > 256 ? GS : 256)
    k_add(const L* __restrict__ a, const L* __restrict__ b, L* __restrict__ r, uint8_t* __restrict__ carry,
          uint32_t n, uint32_t m) {
    constexpr int BLOCK = GS > 256 ? GS : 256;
    constexpr int IPB = BLOCK / GS;
    __shared__ uint32_t scratch[BLOCK / 32];
    __shared__ uint64_t shift[OP == ADD_PLAIN ? 1 : BLOCK / 32];
    const uint32_t grp = threadIdx.x / GS;
    const uint32_t t = threadIdx.x % GS;
    const uint32_t start = t * Q;
    const uint64_t stride = uint64_t(gridDim.x) * IPB;
    pdl_wait();  // launched with launch_pdl
    pdl_trigger();
    // Uniform trip count per block: group_carry synchronises the block for GS > 32.
    for (uint64_t base = uint64_t(blockIdx.x) * IPB; base < n; base += stride) {
        const uint64_t inst = base + grp;
        const bool valid = inst < n;
        const uint64_t off = valid ? inst * m : 0;
        L x[Q], y[Q], s[Q];
        load_chunk<L, Q, ACCESS>(a + off, start, m, valid, x);
        load_chunk<L, Q, ACCESS>(b + off, start, m, valid, y);
        uint32_t gc;
        if constexpr (OP == ADD_PLAIN) {
            gc = group_add<L, Q, GS>(x, y, s, scratch);
        } else {
            // 6a + 10b mod 2^(64m), the value of a6pb10Ker's chain of six
            // additions (cuda/ker-addition.cu.h:304-324) with one carry pass:
            // per limb 6a_i + 10b_i = lo_i + hi_i*2^64 with hi_i <= 15, and
            // the result is lo + (hi shifted up one limb), whose limb sums
            // carry at most 1.
            static_assert(sizeof(L) == 8, "6a + 10b is defined on u64 limbs");
            L lo[Q], hi[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const L pa = x[q] * 6u, pb = y[q] * 10u;
                lo[q] = pa + pb;
                hi[q] = __umul64hi(x[q], 6u) + __umul64hi(y[q], 10u) + L(lo[q] < pa);
            }
            L sh[Q];
            sh[0] = group_shift_up<GS>(hi[Q - 1], t, shift);
#pragma unroll
            for (int q = 1; q < Q; ++q) sh[q] = hi[q - 1];
            gc = group_add<L, Q, GS>(lo, sh, s, scratch);
        }
        store_chunk<L, Q, ACCESS>(r + off, start, m, valid, s);
        if (OP == ADD_PLAIN && carry != nullptr && valid) {
            // The carry-out is the value left at limb position m (a padding
            // limb of zeros plus the carry), or the group's carry-out when the
            // instance fills the group exactly.
            if (m < uint32_t(GS * Q)) {
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    if (start + q == m) carry[inst] = uint8_t(s[q]);
            } else if (t == GS - 1) {
                carry[inst] = uint8_t(gc);
            }
        }
    }
}

// High word (at most 15) of the limb 6 a_i + 10 b_i.
__device__ __forceinline__ uint64_t six_hi(uint64_t ai, uint64_t bi) {
    const uint64_t pa = ai * 6u, pb = bi * 10u;
    return __umul64hi(ai, 6u) + __umul64hi(bi, 10u) + uint64_t(pa + pb < pa);
}

// The same for rows that allow no 16-byte access (odd lengths, 4-byte aligned
// rows).  With Q consecutive limbs per thread their loads would be Q strided
// single-limb accesses, each touching every line of the warp's span; here lane
// c of a warp's WL lanes of the group holds limb c of Q rows of WL consecutive
// limbs, so every access of the warp is contiguous.  A row's carries are one
// lookahead over its two ballots, the rows chained by their one-bit carry;
// groups wider than a warp do it twice, with the carry into the warp from a
// lookahead over one word per warp in between.  (2048 x 4095 limbs 60.4 ->
// 38.6 us, 8380 x 1001 42.7 -> 29.9, 16760 x 1001
// 32-bit limbs 67.1 -> 31.8, 2048 x 8191 116.5 -> 54.4.)
template <typename L, int Q, int GS, int OP>
__global__ void __launch_bounds__(GS > 256 ? GS : 256)
    k_add_rows(const L* __restrict__ a, const L* __restrict__ b, L* __restrict__ r, uint8_t* __restrict__ carry,
               uint32_t n, uint32_t m) {
    constexpr int BLOCK = GS > 256 ? GS : 256;
    constexpr int IPB = BLOCK / GS;
    constexpr int WL = GS < 32 ? GS : 32;  // lanes of the group in a warp
    constexpr int WARPS = GS / WL;         // warps of the group
    constexpr uint32_t MASK = WL == 32 ? MI_FULL_MASK : (1u << WL) - 1u;
    __shared__ uint32_t wflag[WARPS > 1 ? BLOCK / 32 : 1];  // bit 0 generate (carry-in 0), bit 1 propagate
    const uint32_t grp = threadIdx.x / GS, t = threadIdx.x % GS;
    const uint32_t c = t % WL, wig = t / WL, gb = (threadIdx.x & 31u) & ~uint32_t(WL - 1);
    const uint32_t start = wig * (WL * Q) + c;  // the thread's limb of row 0
    const uint64_t stride = uint64_t(gridDim.x) * IPB;
    pdl_wait();  // launched with launch_pdl
    pdl_trigger();
    for (uint64_t base = uint64_t(blockIdx.x) * IPB; base < n; base += stride) {
        const uint64_t inst = base + grp;
        const bool valid = inst < n;
        const uint64_t off = valid ? inst * m : 0;
        const uint32_t mm = valid ? m : 0;
        L x[Q], y[Q], s[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) x[k] = start + WL * k < mm ? ld_stream(a + off + start + WL * k) : L(0);
#pragma unroll
        for (int k = 0; k < Q; ++k) y[k] = start + WL * k < mm ? ld_stream(b + off + start + WL * k) : L(0);
        if constexpr (OP == ADD_SIX) {
            // 6a + 10b as lo + (hi shifted up one limb), as in k_add
            static_assert(sizeof(L) == 8, "6a + 10b is defined on u64 limbs");
            uint64_t before = 0;  // lane 0: the high word of the limb before the row
            if (WARPS > 1 && c == 0 && start > 0 && start - 1 < mm)
                before = six_hi(a[off + start - 1], b[off + start - 1]);
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                const uint64_t hi = six_hi(x[k], y[k]);
                x[k] = x[k] * 6u + y[k] * 10u;
                const uint64_t up = __shfl_up_sync(MI_FULL_MASK, hi, 1, WL);
                y[k] = c == 0 ? before : up;
                before = __shfl_sync(MI_FULL_MASK, hi, WL - 1, WL);
            }
        }
        uint32_t gc = 0;  // the group's carry-out
        if constexpr (WARPS == 1) {
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                s[k] = x[k] + y[k];
                const uint64_t Y = (__ballot_sync(MI_FULL_MASK, s[k] < x[k]) >> gb) & MASK;
                const uint64_t X = ((__ballot_sync(MI_FULL_MASK, s[k] == L(~L(0))) >> gb) & MASK) | Y;
                const uint64_t S = X + Y + gc;
                s[k] += L(((S ^ X ^ Y) >> c) & 1u);
                gc = uint32_t(S >> WL) & 1u;
            }
        } else {
            uint32_t G[Q], P[Q], cw = 0;
            bool ones = true;
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                s[k] = x[k] + y[k];
                G[k] = __ballot_sync(MI_FULL_MASK, s[k] < x[k]);
                P[k] = __ballot_sync(MI_FULL_MASK, s[k] == L(~L(0)));
                cw = uint32_t((uint64_t(G[k] | P[k]) + G[k] + cw) >> 32);
                ones = ones && P[k] == MI_FULL_MASK;
            }
            if (c == 0) wflag[threadIdx.x >> 5] = cw | (ones ? 2u : 0u);
            __syncthreads();
            const uint32_t f = c < WARPS ? wflag[grp * WARPS + c] : 0u;
            const uint64_t Y = __ballot_sync(MI_FULL_MASK, f & 1u);
            const uint64_t X = __ballot_sync(MI_FULL_MASK, (f & 2u) != 0) | Y, S = X + Y;
            gc = uint32_t(S >> WARPS) & 1u;
            cw = uint32_t((S ^ X ^ Y) >> wig) & 1u;  // into the warp
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                const uint64_t rx = G[k] | P[k], ry = G[k], rs = rx + ry + cw;
                s[k] += L(((rs ^ rx ^ ry) >> c) & 1u);
                cw = uint32_t(rs >> 32);
            }
            __syncthreads();  // the flags are rewritten by the next instance
        }
#pragma unroll
        for (int k = 0; k < Q; ++k)
            if (start + WL * k < mm) st_stream(r + off + start + WL * k, s[k]);
        if (OP == ADD_PLAIN && carry != nullptr && valid) {
            // as in k_add: the value left at limb position m, or the group's carry-out
            if (m < uint32_t(GS * Q)) {
#pragma unroll
                for (int k = 0; k < Q; ++k)
                    if (start + WL * k == m) carry[inst] = uint8_t(s[k]);
            } else if (t == GS - 1) {
                carry[inst] = uint8_t(gc);
            }
        }
    }
}

// --- instances wider than one block: decoupled look-back -------------------
//
// A tile is one 256-thread block over 64 bytes of each operand per thread
// (2048 u64 limbs).  Tiles take their index from an atomic counter in launch
// order, so every tile a tile waits for has already started and will finish
// (no dependence on the scheduler); the order goes round the instances, so
// that few tiles of one instance are in flight at a time.  A plain addition
// first reads the 32 limbs below its tile: the nearest one whose sum is not
// all ones gives the carry-in directly, which settles almost every tile of
// random data without waiting (the tile then only publishes its state).
// Otherwise, and for 6a + 10b, each tile adds its limbs with carry-in 0,
// publishes its state -- inclusive (its true carry-out) when it does not
// propagate a carry or is the first tile of its instance, otherwise an
// aggregate that says "passes the carry-in through" -- then it walks back
// over aggregates to the nearest inclusive tile, bounded by spin_limit polls
// of an unpublished one (then the error word is set and the tile carries on
// with carry-in 0, so the kernel always completes), publishes its own
// inclusive state, and the block redoes the carry pass with that carry-in.
//
// States are two bits per tile, 32 tiles to a 64-bit word (tile i of a word:
// bit 32 + i inclusive, bit i aggregate or, with bit 32 + i, a carry of one;
// neither: unpublished), added by the tile itself, so a warp's walk back reads
// 1024 tiles per step.  (One word per tile, 32 tiles per step, let a run of
// propagating tiles advance by 32 tiles per round trip to the L2: a number of
// 2^24 limbs that carries from end to end took 175-197 us; 128 words per step
// from every waiting tile took 227 us, the polls in each other's way.)  The
// words need no ordering with other memory, being all that a waiting tile
// reads of another: relaxed accesses (a release made every tile wait for a
// memory barrier before its stores: 16 x 2^20 limbs 66.7 us against 61.0).

__device__ __forceinline__ uint64_t ld_status(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void add_status(uint64_t* p, uint64_t v) {
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Within a tile, warp w owns 32 * Q consecutive limbs (Q = 64 bytes' worth) as
// R rows of 32 * V: lane i of row r holds V = 16 bytes of limbs on 16-byte
// aligned rows, V = 1 limb on others, so every load and store of a warp is
// one contiguous run whatever the alignment (with 64 bytes per thread, rows
// that allow no 16-byte access were read at a stride of 64 bytes: 16 x 1048573
// limbs 125 us).  A row's carries are one lookahead over its two ballots, the
// rows of a warp chained by their one-bit carry; the ballots are kept, so the
// second pass (with the warp's true carry-in) is integer work only.
template <typename L, int V>
__device__ __forceinline__ void load_row(const L* __restrict__ row, uint32_t i, uint32_t m, L (&v)[V]) {
    if constexpr (V > 1) {
        if (i + V <= m) {
            const uint4 q = __ldcs(reinterpret_cast<const uint4*>(row + i));
            unpack16<L, V>(q, v);
            return;
        }
    }
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = i + k < m ? ld_stream(row + i + k) : L(0);
}

template <typename L, int V>
__device__ __forceinline__ void store_row(L* __restrict__ row, uint32_t i, uint32_t m, const L (&v)[V]) {
    if constexpr (V > 1) {
        if (i + V <= m) {
            __stcs(reinterpret_cast<uint4*>(row + i), pack16<L, V>(v));
            return;
        }
    }
#pragma unroll
    for (int k = 0; k < V; ++k)
        if (i + k < m) st_stream(row + i + k, v[k]);
}

// What a tile needs of the limbs below it, as one byte.  Plain addition: its
// carry-in (0 or 1) where the nearest of the 32 limbs below whose sum is not
// all ones gives it, else 2.  6a + 10b: the high word of the limb below.  By
// the 32 lanes of a warp; i is the tile's first limb.
template <typename L, int OP>
__device__ __forceinline__ uint32_t tile_edge(const L* __restrict__ a, const L* __restrict__ b, uint64_t i,
                                              uint32_t lane) {
    if constexpr (OP == ADD_SIX) {
        return uint32_t(six_hi(a[i - 1], b[i - 1]));
    } else {
        const L ai = a[i - 1 - lane], bi = b[i - 1 - lane];  // lane 0 is the limb just below the tile
        const L si = ai + bi;
        const uint32_t settled = __ballot_sync(MI_FULL_MASK, si != L(~L(0)));
        const uint32_t gen = __ballot_sync(MI_FULL_MASK, si < ai);
        return settled ? (gen >> (__ffs(settled) - 1)) & 1u : 2u;
    }
}

// In-place calls: the edge bytes of every tile, taken before any tile
// overwrites the limbs below its neighbour.  One warp per tile.
template <typename L, int OP>
__global__ void __launch_bounds__(256)
    k_wide_edges(const L* __restrict__ a, const L* __restrict__ b, uint32_t m, uint32_t tiles_per, uint32_t n_tiles,
                 uint8_t* __restrict__ edges) {
    constexpr uint32_t W = 256u * (64 / uint32_t(sizeof(L)));
    pdl_wait();  // launched with launch_pdl
    const uint32_t tile = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (tile >= n_tiles || tile % tiles_per == 0) return;
    const uint64_t off = uint64_t(tile / tiles_per) * m;
    const uint32_t e = tile_edge<L, OP>(a + off, b + off, uint64_t(tile % tiles_per) * W, lane);
    if (lane == 0) edges[tile] = uint8_t(e);
}

// edges: the bytes of k_wide_edges when r is a or b, else null (each tile then
// reads the limbs below it itself).
template <typename L, int V, int OP>
__global__ void __launch_bounds__(256, sizeof(L) == 8 ? 4 : 2)
    k_add_wide(const L* __restrict__ a, const L* __restrict__ b, L* __restrict__ r, uint8_t* __restrict__ carry,
               uint32_t m, uint32_t tiles_per, uint32_t n_tiles, uint64_t* status, uint64_t* old, uint32_t old_words,
               unsigned long long* counter, uint32_t* err, uint32_t spin_limit, uint32_t withhold, uint64_t base,
               const uint8_t* __restrict__ edges) {
    constexpr int Q = 64 / int(sizeof(L));
    constexpr int R = Q / V;           // rows per warp
    constexpr uint32_t W = 256u * Q;   // limbs per tile
    __shared__ uint32_t wflag[8];      // per warp: bit 0 generate (carry-in 0), bit 1 propagate
    __shared__ uint32_t s_tile, s_cin;
    // a monotonic tile counter (this launch's tiles are base .. base+n_tiles-1)
    // and two arrays of state words, taken in turn: each launch clears the
    // words of the launch before it (old), so nothing is cleared in between
    pdl_wait();  // launched with launch_pdl: the previous launch has completed
    if (threadIdx.x == 0) s_tile = uint32_t(atomicAdd(counter, 1ull) - base);
    __syncthreads();
    if (s_tile >= n_tiles) return;  // (the grid has exactly n_tiles blocks)
    const uint32_t n_inst = n_tiles / tiles_per;
    const uint32_t inst = s_tile % n_inst, j = s_tile / n_inst;
    uint64_t* words = status + size_t(inst) * ((tiles_per + 31) / 32);  // the instance's states
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    for (uint32_t i = s_tile + n_tiles * t; i < old_words; i += n_tiles * 256) old[i] = 0;
    const uint64_t off = uint64_t(inst) * m;
    const uint32_t start = j * W + warp * (32 * Q) + lane * V;  // the thread's limbs of row 0; row r is 32 V r further
    L x[R][V], y[R][V], s[R][V];
#pragma unroll
    for (int k = 0; k < R; ++k) load_row<L, V>(a + off, start + 32 * V * k, m, x[k]);
#pragma unroll
    for (int k = 0; k < R; ++k) load_row<L, V>(b + off, start + 32 * V * k, m, y[k]);
    // Carry-in straight from the 32 limbs below the tile: the nearest limb
    // whose sum is not all ones decides it (generate: 1, kill: 0).  Random
    // limbs almost always settle it here and the tile never waits; only a
    // run of 32 all-ones sums falls back to the look-back.
    uint32_t local_cin = 0;
    bool local_ok = j == 0;
    if (OP == ADD_PLAIN && j > 0 && t < 32) {
        const uint32_t e = edges != nullptr ? edges[inst * tiles_per + j]
                                            : tile_edge<L, OP>(a + off, b + off, uint64_t(j) * W, lane);
        local_ok = e < 2;
        local_cin = e & 1u;
    }
    if constexpr (OP == ADD_SIX) {
        // 6a + 10b as lo + (hi shifted up one limb), as in k_add; lane 0 takes
        // the row before from lane 31, and for its first row recomputes the
        // high word of the limb before its warp's span
        static_assert(sizeof(L) == 8, "6a + 10b is defined on u64 limbs");
        uint64_t before = 0;
        if (lane == 0 && start > 0 && start - 1 < m)
            before = warp == 0 && edges != nullptr ? edges[inst * tiles_per + j]
                                                   : six_hi(a[off + start - 1], b[off + start - 1]);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            L hi[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                hi[v] = six_hi(x[k][v], y[k][v]);
                x[k][v] = x[k][v] * 6u + y[k][v] * 10u;
            }
            const uint64_t up = __shfl_up_sync(MI_FULL_MASK, uint64_t(hi[V - 1]), 1);
            y[k][0] = lane == 0 ? before : up;
#pragma unroll
            for (int v = 1; v < V; ++v) y[k][v] = hi[v - 1];
            before = __shfl_sync(MI_FULL_MASK, uint64_t(hi[V - 1]), 31);  // lane 0's next row
        }
    }
    uint32_t G[R], P[R], c = 0;  // each row's generate and propagate ballots
    bool ones = true;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        bool g, p;
        chunk_add<L, V>(x[k], y[k], s[k], g, p);
        G[k] = __ballot_sync(MI_FULL_MASK, g);
        P[k] = __ballot_sync(MI_FULL_MASK, p);
        c = uint32_t((uint64_t(G[k] | P[k]) + G[k] + c) >> 32);
        ones = ones && P[k] == MI_FULL_MASK;
    }
    if (lane == 0) wflag[warp] = c | (ones ? 2u : 0u);
    __syncthreads();
    // the tile's generate and propagate, and the carry into each warp: a
    // lookahead over the eight warps
    uint32_t WG = 0, WP = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        const uint32_t f = wflag[w];
        WG |= (f & 1u) << w;
        WP |= (f >> 1) << w;
    }
    const uint32_t gc0 = ((WG | WP) + WG) >> 8;
    const bool all = WP == 0xffu;  // the tile passes a carry-in through
    if (t < 32) {
        // warp 0 looks back 1024 tiles at a time: lane l reads the states of
        // word g - l; the carry-in is the value of the nearest inclusive tile,
        // valid once every tile between (all propagating aggregates) has
        // published
        const uint64_t agg = 1ull << (j & 31u), inc = agg << 32;  // the tile's own bits
        uint32_t cin = local_cin;
        if (!local_ok) {
            if (t == 0) add_status(words + (j >> 5), all ? agg : (gc0 ? inc + agg : inc));
            int32_t g = int32_t(j >> 5);
            uint32_t below = (1u << (j & 31u)) - 1u;  // the tiles of this tile's own word that precede it
            uint32_t spins = 0;
            for (;;) {
                const int32_t i = g - int32_t(t);
                const uint64_t w = i >= 0 ? ld_status(words + i) : 1ull << 63;  // (tile 0 is always inclusive)
                const uint32_t hi = uint32_t(w >> 32), lo = uint32_t(w);
                const uint32_t stop = ~(lo & ~hi) & (t == 0 ? below : MI_FULL_MASK);  // not aggregates
                const uint32_t top = 31u - __clz(stop);  // the nearest of them
                const bool known = stop != 0 && ((hi >> top) & 1u);
                const uint32_t found = __ballot_sync(MI_FULL_MASK, known);
                const uint32_t pending = __ballot_sync(MI_FULL_MASK, stop != 0 && !known);
                const uint32_t nearest = found ? uint32_t(__ffs(found) - 1) : 32u;
                const uint32_t nearer = nearest == 32u ? MI_FULL_MASK : ((1u << nearest) - 1u);
                if (pending & nearer) {
                    if (++spins > spin_limit) {
                        if (t == 0) atomicOr(err, 1u);
                        break;
                    }
                    __nanosleep(64);
                    continue;
                }
                if (found) {
                    cin = __shfl_sync(MI_FULL_MASK, (lo >> (top & 31u)) & 1u, int(nearest));
                    break;
                }
                g -= 32;
                below = MI_FULL_MASK;
            }
        }
        if (t == 0) {
            const uint32_t cout = gc0 | (all ? cin : 0u);
            if (local_ok) {
                if (!(withhold && j == 0)) add_status(words + (j >> 5), cout ? inc + agg : inc);
            } else if (all) {
                add_status(words + (j >> 5), cout ? inc : inc - agg);  // the aggregate becomes inclusive
            }
            s_cin = cin;
        }
    }
    __syncthreads();
    const uint32_t WX = WG | WP, WS = WX + WG + s_cin;
    c = ((WS ^ WX ^ WG) >> warp) & 1u;  // into the warp
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const uint64_t X = G[k] | P[k], Y = G[k], S = X + Y + c;
        chunk_inc<L, V>(s[k], uint32_t((S ^ X ^ Y) >> lane) & 1u);
        c = uint32_t(S >> 32);
        store_row<L, V>(r + off, start + 32 * V * k, m, s[k]);
    }
    if (OP == ADD_PLAIN && carry != nullptr && j == tiles_per - 1) {
        // carry-out: the value at limb m (zero padding plus the carry), or
        // the tile's carry-out when the instance ends with the tile
        if (m % W != 0) {
#pragma unroll
            for (int k = 0; k < R; ++k)
#pragma unroll
                for (int v = 0; v < V; ++v)
                    if (start + 32 * V * k + v == m) carry[inst] = uint8_t(s[k][v]);
        } else if (t == 255) {
            carry[inst] = uint8_t(WS >> 8);
        }
    }
}

// Rounds of whole instances, at most kWideTiles tiles each; every round takes
// the next n_tiles values of the tile counter and the other array of state
// words, clearing the words of the round before.  Under capture the graph clears
// the captured calls' area before each round instead, so that every replay starts
// from the same state.
template <typename L, bool VEC, int OP>
mi_status launch_wide(const L* a, const L* b, L* r, uint8_t* carry, uint32_t n, uint32_t m, WideState& w,
                      cudaStream_t st) {
    constexpr uint32_t W = 256u * (64 / uint32_t(sizeof(L)));
    constexpr int V = VEC ? 16 / int(sizeof(L)) : 1;  // limbs per access
    const uint32_t tiles_per = (m + W - 1) / W;
    const uint32_t cap = w.round_tiles < kWideTiles ? w.round_tiles : kWideTiles;
    if (tiles_per > cap) return set_error(MI_EINVAL, "add: %u limbs exceeds the multi-block maximum", m);
    const uint32_t per_round = cap / tiles_per;
    cudaStreamCaptureStatus capture;
    MI_CUDA_TRY(cudaStreamIsCapturing(st, &capture));
    const bool captured = capture != cudaStreamCaptureStatusNone;
    uint64_t* const area = w.status + (captured ? kWideBytes / 8 : 0);
    uint64_t* const counter = area + 2 * kWideWords;
    uint32_t* const err = reinterpret_cast<uint32_t*>(w.status + 2 * kWideWords + 1);
    for (uint32_t i0 = 0; i0 < n; i0 += per_round) {
        const uint32_t k = (n - i0) < per_round ? (n - i0) : per_round;
        const uint32_t n_tiles = k * tiles_per;
        const uint32_t words = k * ((tiles_per + 31) / 32);  // tiles_per >= 2, so at most kWideWords
        const uint64_t o = uint64_t(i0) * m;
        uint64_t *states = area + w.parity * kWideWords, *old = area + (w.parity ^ 1u) * kWideWords, base = w.issued;
        uint32_t old_words = w.old_words;
        if (captured) {  // the words right before the counter, cleared with it
            states = counter - words, base = 0, old_words = 0;
            MI_CUDA_TRY(cudaMemsetAsync(states, 0, (size_t(words) + 1) * 8, st));
        }
        uint8_t* edges = nullptr;
        if (r == a || r == b) {
            edges = reinterpret_cast<uint8_t*>(area + 2 * kWideWords + 2);
            MI_CUDA_TRY(launch_pdl(k_wide_edges<L, OP>, dim3((n_tiles + 7) / 8), dim3(256), 0, st, a + o, b + o, m,
                                   tiles_per, n_tiles, edges));
        }
        MI_CUDA_TRY(launch_pdl(k_add_wide<L, V, OP>, dim3(n_tiles), dim3(256), 0, st, a + o, b + o, r + o,
                               carry ? carry + i0 : nullptr, m, tiles_per, n_tiles, states, old, old_words,
                               reinterpret_cast<unsigned long long*>(counter), err, w.spin_limit, w.withhold, base,
                               edges));
        if (captured) continue;
        w.issued += n_tiles;  // every block of the launch takes one counter value
        w.old_words = words;
        w.parity ^= 1u;
    }
    return MI_OK;
}

template <typename L, int Q, int GS, int ACCESS, int OP>
mi_status launch_one(const L* a, const L* b, L* r, uint8_t* carry, uint32_t n, uint32_t m, cudaStream_t st) {
    constexpr int BLOCK = GS > 256 ? GS : 256;
    constexpr int IPB = BLOCK / GS;
    uint64_t blocks = (uint64_t(n) + IPB - 1) / IPB;
    // Enough blocks for full residency several times over; the kernel strides.
    const uint64_t cap = uint64_t(sm_count()) * 64;
    if (blocks > cap) blocks = cap;
    if constexpr (ACCESS == ROWS)
        MI_CUDA_TRY(
            launch_pdl(k_add_rows<L, Q, GS, OP>, dim3(uint32_t(blocks)), dim3(BLOCK), 0, st, a, b, r, carry, n, m));
    else
        MI_CUDA_TRY(launch_pdl(k_add<L, Q, GS, ACCESS, OP>, dim3(uint32_t(blocks)), dim3(BLOCK), 0, st, a, b, r, carry,
                               n, m));
    return MI_OK;
}

template <typename L, int ACCESS, int OP, int Q>
mi_status dispatch_gs(const L* a, const L* b, L* r, uint8_t* carry, uint32_t n, uint32_t m, uint32_t gs,
                      cudaStream_t st) {
    switch (gs) {
        case 1: return launch_one<L, Q, 1, ACCESS, OP>(a, b, r, carry, n, m, st);
        case 2: return launch_one<L, Q, 2, ACCESS, OP>(a, b, r, carry, n, m, st);
        case 4: return launch_one<L, Q, 4, ACCESS, OP>(a, b, r, carry, n, m, st);
        case 8: return launch_one<L, Q, 8, ACCESS, OP>(a, b, r, carry, n, m, st);
        case 16: return launch_one<L, Q, 16, ACCESS, OP>(a, b, r, carry, n, m, st);
        case 32: return launch_one<L, Q, 32, ACCESS, OP>(a, b, r, carry, n, m, st);
        case 64: return launch_one<L, Q, 64, ACCESS, OP>(a, b, r, carry, n, m, st);
        case 128: return launch_one<L, Q, 128, ACCESS, OP>(a, b, r, carry, n, m, st);
        case 256: return launch_one<L, Q, 256, ACCESS, OP>(a, b, r, carry, n, m, st);
        case 512: return launch_one<L, Q, 512, ACCESS, OP>(a, b, r, carry, n, m, st);
        case 1024: return launch_one<L, Q, 1024, ACCESS, OP>(a, b, r, carry, n, m, st);
        default: return set_error(MI_EINVAL, "add: %u limbs exceeds the single-group maximum", m);
    }
}

// k_add, 16-byte aligned rows: Q = thread_bytes / sizeof(L) limbs per thread
// (16, 32 or 64 bytes, raised until the group fits 1024 threads), GS =
// pow2ceil(m / Q) threads per instance.
template <typename L, int OP>
mi_status dispatch_vec(const L* a, const L* b, L* r, uint8_t* carry, uint32_t n, uint32_t m, uint32_t thread_bytes,
                       cudaStream_t st) {
    constexpr uint32_t QS = 16 / sizeof(L);  // limbs per 128-bit access
    uint32_t q = thread_bytes >= 64 ? 4 * QS : (thread_bytes >= 32 ? 2 * QS : QS);
    while (q < 4 * QS && pow2ceil((m + q - 1) / q) > 1024) q *= 2;
    const uint32_t gs = pow2ceil((m + q - 1) / q);
    if (q == QS) return dispatch_gs<L, WORDS16, OP, QS>(a, b, r, carry, n, m, gs, st);
    if (q == 2 * QS) return dispatch_gs<L, WORDS16, OP, 2 * QS>(a, b, r, carry, n, m, gs, st);
    return dispatch_gs<L, WORDS16, OP, 4 * QS>(a, b, r, carry, n, m, gs, st);
}

// Rows per thread of k_add_rows: four (two leave too little in flight, eight too
// few warps), or what pads less than the next power of two of threads does --
// five rows where 5/8 of it holds the row of limbs, three or six (the better by
// length) where 3/4 does.  Short u64 rows differ: with four rows a group of 4 or 8 lanes
// reads 32 or 64 contiguous bytes at a time, and five are better although they
// pad more.  us per 2^22 u64 or 2^23 u32 limbs with four rows against the
// pick: 15 limbs 20.9 -> 16.7, 27 17.6 -> 16.1, 65 17.0 -> 16.0, 95 16.9 -> 15.8, 129
// 20.8 -> 16.3, 513 18.3 -> 16.1; 33 words 24.6 -> 18.6, 65 23.3 -> 18.3, 129 29.8
// -> 17.5, 161 25.7 -> 17.0, 333 24.6 -> 20.0.  Eight where four would need a
// block of 1024 threads (4095 limbs 38.6 against 50.1).
template <typename L>
uint32_t rows_per_thread(uint32_t m) {
    const uint32_t slots = 4 * pow2ceil((m + 3) / 4);
    if (slots > 4 * 512) return 8;
    const bool half = 8 * m <= 5 * slots, three = 4 * m <= 3 * slots;
    if (sizeof(L) == 4) return m <= 4 ? 4 : half ? 5 : three ? (m < 256 ? 6 : 3) : 4;
    if (m <= 4 || (m >= 30 && m <= 32)) return 2;
    if ((m >= 13 && m <= 16) || (m >= 25 && m <= 29)) return 5;
    if (m <= 96) return three && (m < 9 || m > 12) ? 3 : 4;
    return half ? (m <= 160 ? 6 : 5) : 4;
}

template <typename L, int OP>
mi_status dispatch_rows(const L* a, const L* b, L* r, uint8_t* carry, uint32_t n, uint32_t m, uint32_t q,
                        cudaStream_t st) {
    const uint32_t gs = pow2ceil((m + q - 1) / q);
    switch (q) {
        case 2: return dispatch_gs<L, ROWS, OP, 2>(a, b, r, carry, n, m, gs, st);
        case 3: return dispatch_gs<L, ROWS, OP, 3>(a, b, r, carry, n, m, gs, st);
        case 4: return dispatch_gs<L, ROWS, OP, 4>(a, b, r, carry, n, m, gs, st);
        case 5: return dispatch_gs<L, ROWS, OP, 5>(a, b, r, carry, n, m, gs, st);
        case 6: return dispatch_gs<L, ROWS, OP, 6>(a, b, r, carry, n, m, gs, st);
        default: return dispatch_gs<L, ROWS, OP, 8>(a, b, r, carry, n, m, gs, st);
    }
}

// 6a + 10b on rows that allow no 16-byte access.  A row of k_add_rows costs two
// 64-bit shuffles more than in a plain addition, so lengths that fill the group
// well take consecutive limbs per thread instead (one shuffle per thread), two
// or four of them; the others three rows, or five where those pad less (us per
// 2^22 limbs with the rows of the plain addition against these: 13 limbs 22.3 ->
// 20.4, 29 21.5 -> 18.7, 63 20.2 -> 17.0, 99 23.1 -> 19.6, 127 23.1 -> 17.0, 129 26.2 -> 20.8,
// 191 26.4 -> 21.1, 255 23.8 -> 21.5, 333 29.4 -> 24.6, 385 27.4 -> 23.3, 511 24.5 -> 20.3, 641 26.5 ->
// 22.7, 1001 22.4 -> 19.9, 2049 46.4 -> 28.2, 4095 31.7 -> 29.6).
struct SixForm {
    uint32_t up_to;  // limbs
    int access;
    uint32_t q;      // rows, or limbs, per thread
};
constexpr SixForm kSixForms[] = {
    {2, ROWS, 2},    {3, ROWS, 3},     {4, ROWS, 2},     {6, ROWS, 3},    {8, ROWS, 4},    {12, ROWS, 3},
    {16, ROWS, 2},   {24, ROWS, 3},    {29, LIMBS, 4},   {32, ROWS, 2},   {48, ROWS, 3},   {64, LIMBS, 2},
    {88, ROWS, 3},   {128, LIMBS, 4},  {160, ROWS, 5},   {192, ROWS, 3},  {256, LIMBS, 2}, {384, ROWS, 3},
    {512, LIMBS, 2}, {768, ROWS, 3},   {1024, LIMBS, 4}, {1280, ROWS, 5}, {1536, ROWS, 3}, {2048, ROWS, 4},
    {2560, ROWS, 5}, {3072, ROWS, 3},  {kAddMaxLimbs64, ROWS, 4}};

mi_status dispatch_six(const uint64_t* a, const uint64_t* b, uint64_t* r, uint32_t n, uint32_t m, cudaStream_t st) {
    const SixForm* f = kSixForms;
    while (m > f->up_to) ++f;  // m <= kAddMaxLimbs64
    if (f->access == ROWS) return dispatch_rows<uint64_t, ADD_SIX>(a, b, r, nullptr, n, m, f->q, st);
    const uint32_t gs = pow2ceil((m + f->q - 1) / f->q);
    return f->q == 2 ? dispatch_gs<uint64_t, LIMBS, ADD_SIX, 2>(a, b, r, nullptr, n, m, gs, st)
                     : dispatch_gs<uint64_t, LIMBS, ADD_SIX, 4>(a, b, r, nullptr, n, m, gs, st);
}

// A plain addition on rows that allow no 16-byte access.  With operands over the
// host link and results in device memory (link) consecutive limbs, 16 bytes of
// them per thread, from 3 u64 or 13 u32 limbs on while they fit a group: the rows'
// short runs of lanes ask the link for the same 32 bytes more than once (us for
// 2^20 u64 or 2^21 u32 limbs with rows against these: 5 limbs 152 -> 144, 9 182 ->
// 144, 17 163 -> 143, 127 144 -> 142; 17 words 179 -> 143, 65 161 -> 143, 1001 155 -> 143;
// one limb 143 against 150, 9 words 142 against 144).  Results over the link want the
// rows' contiguous stores (1024 x 2047 words 141 against 301).
template <typename L>
mi_status dispatch_plain(const L* a, const L* b, L* r, uint8_t* carry, uint32_t n, uint32_t m, bool link,
                         cudaStream_t st) {
    constexpr uint32_t Q = 16 / sizeof(L);
    if (link && m >= (sizeof(L) == 8 ? 3 : 13) && m <= Q * 1024)
        return dispatch_gs<L, LIMBS, ADD_PLAIN, int(Q)>(a, b, r, carry, n, m, pow2ceil((m + Q - 1) / Q), st);
    if constexpr (sizeof(L) == 8) {
        // lengths a little above three quarters of a group of four rows, whose last
        // row is nearly empty (us for 2^22, 2^21 and 2^20 limbs with rows against four
        // limbs per thread: 99 16.7, 10.1, 6.3 against 16.2, 9.5, 5.8; 105 16.7, 10.1, 6.3
        // against 16.4, 9.7, 6.1; 109 16.6, 9.8, 5.8 against 16.5, 10.0, 6.2; 53 17.2, 10.6,
        // 6.7 against 17.2, 10.1, 6.2)
        if (m >= 50 && m <= 54) return launch_one<L, 4, 16, LIMBS, ADD_PLAIN>(a, b, r, carry, n, m, st);
        if (m >= 97 && m <= 107) return launch_one<L, 4, 32, LIMBS, ADD_PLAIN>(a, b, r, carry, n, m, st);
    }
    return dispatch_rows<L, ADD_PLAIN>(a, b, r, carry, n, m, rows_per_thread<L>(m), st);
}

}  // namespace

uint32_t add_size_class(uint64_t bytes) {
    const uint64_t limbs = (bytes + 7) / 8;
    uint32_t c = 0;
    while (c < 12 && (uint64_t(1) << c) < limbs) ++c;
    return c;
}

mi_status launch_add_u64(const uint64_t* a, const uint64_t* b, uint64_t* r, uint8_t* carry, uint32_t n,
                         uint32_t limbs, int op, uint32_t thread_bytes, cudaStream_t st, WideState* wide, bool link) {
    const bool vec = aligned16(a) && aligned16(b) && aligned16(r) && (limbs % 2 == 0);
    if (limbs > kAddMaxLimbs64) {
        if (wide == nullptr || wide->status == nullptr) return set_error(MI_EINVAL, "add: no multi-block state");
        if (op == ADD_SIX)
            return vec ? launch_wide<uint64_t, true, ADD_SIX>(a, b, r, nullptr, n, limbs, *wide, st)
                       : launch_wide<uint64_t, false, ADD_SIX>(a, b, r, nullptr, n, limbs, *wide, st);
        return vec ? launch_wide<uint64_t, true, ADD_PLAIN>(a, b, r, carry, n, limbs, *wide, st)
                   : launch_wide<uint64_t, false, ADD_PLAIN>(a, b, r, carry, n, limbs, *wide, st);
    }
    if (op == ADD_SIX)
        return vec ? dispatch_vec<uint64_t, ADD_SIX>(a, b, r, nullptr, n, limbs, thread_bytes, st)
                   : dispatch_six(a, b, r, n, limbs, st);
    return vec ? dispatch_vec<uint64_t, ADD_PLAIN>(a, b, r, carry, n, limbs, thread_bytes, st)
               : dispatch_plain<uint64_t>(a, b, r, carry, n, limbs, link, st);
}

mi_status launch_add_u32(const uint32_t* a, const uint32_t* b, uint32_t* r, uint8_t* carry, uint32_t n,
                         uint32_t limbs, uint32_t thread_bytes, cudaStream_t st, WideState* wide, bool link) {
    // An even number of u32 limbs on 8-byte aligned rows is the same bytes as
    // half as many u64 limbs, with the same carry-out.
    if (limbs % 2 == 0 && aligned8(a) && aligned8(b) && aligned8(r))
        return launch_add_u64(reinterpret_cast<const uint64_t*>(a), reinterpret_cast<const uint64_t*>(b),
                              reinterpret_cast<uint64_t*>(r), carry, n, limbs / 2, ADD_PLAIN, thread_bytes, st,
                              wide, link);
    if (limbs > 2 * kAddMaxLimbs64) {
        if (wide == nullptr || wide->status == nullptr) return set_error(MI_EINVAL, "add: no multi-block state");
        return launch_wide<uint32_t, false, ADD_PLAIN>(a, b, r, carry, n, limbs, *wide, st);
    }
    // Odd limb counts (or 4-byte aligned rows) cannot use 128-bit accesses.
    return dispatch_plain<uint32_t>(a, b, r, carry, n, limbs, link, st);
}

}  // namespace mi
