// mul_flex.cu -- batched classical products, full or low half, on groups of
// any number of lanes of a warp.
//
// The kernels of mul.cu and mul_lo.cu give an instance NT = pow2ceil(nb)
// threads (NT/2 for low halves) for its nb blocks of T limbs, so a product of
// 17 blocks keeps 17 of 32 lanes busy and a low half of 38 blocks 19.  Here a
// warp holds G instances on g lanes each, G g <= 32, and a lane owns R pairs of
// anti-diagonals, one per round: pair s is the anti-diagonals s and s + nb of a
// full product (nb tiles together), s and nb - 1 - s of a low half (nb + 1
// tiles).  Within a round a lane runs its pair's tiles as in mul_core.cuh (one
// parity-split accumulator, a snapshot where the first anti-diagonal
// completes) and leaves both values in its shared slots; after the last round
// the output blocks L_q + H_(q-1) + O_(q-2) are formed in rows of g, each row's
// carries one lookahead over the group's bits of two ballots.
//
// Bound by the integer multiply-add pipe and, between tiles, by the warp's own
// chain of loads, snapshot and carries: a step (64 wide multiply-adds) takes
// 390 to 430 cycles of a scheduler against 324 of the fully unrolled loop for
// 32 blocks in mul.cu.  Against the power-of-two groups (us, R): full products
// of 16384 x 68 limbs 81.3 -> 65.0 (2), x 80 94.8 -> 76.8 (2), x 96 109 -> 104 (3);
// 30000 x 40 49.4 -> 37.7 (1), 100000 x 16 49.1 -> 27.9 (1), 300000 x 4
// 72.8 -> 14.6 (1); low halves of 12000 x 301 u32 limbs 132 -> 106 (2), 40000 x
// 80 131 -> 90 (1), 200000 x 12 64.7 -> 27.5 (1).  Small groups gain most: their
// blocks of eight warps ran a loop whose lanes took their snapshots one
// group after another.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.h"
#include "mul_core.cuh"

namespace mi {
namespace {

using classic::ACC;
using classic::DiagAcc;
using classic::PAIRS;
using classic::T;

struct FlexShape {
    uint32_t nb, pairs, steps, rounds, lanes, groups, inv;  // inv: ceil(2^16 / lanes)
    uint32_t stride;                                        // words between the groups' operands
    size_t smem() const { return (size_t(groups) * stride + size_t(rounds) * 32 * 2 * PAIRS) * 4; }
};

// Unrolled twice, at up to 94 registers: two launches of 1500 products then fit
// the SMs at once and overlap (1500 x 68 limbs 12.4 us; unrolled four times, at
// more registers, 15.1, and the low halves of 12000 x 301 words 104 us instead
// of 106).
template <bool FULL, bool VEC>
__global__ void __launch_bounds__(32, 16)
    k_mul_flex(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint32_t* __restrict__ r, uint32_t n,
               uint32_t n32, FlexShape S) {
    extern __shared__ __align__(16) uint32_t smem[];
    const uint32_t lane = threadIdx.x, nb = S.nb, g = S.lanes;
    const bool idle = lane >= S.groups * g;  // repeats lane 0's work, stores nothing
    const uint32_t grp = idle ? 0u : lane / g, t = idle ? 0u : lane - grp * g, base = grp * g;
    uint32_t* gA = smem + grp * S.stride;                           // nb + 1 blocks (the last one zero)
    uint4* gB4 = reinterpret_cast<uint4*>(gA + (nb + 1) * T);       // two planes of nb + 1 halves
    uint2* slots = reinterpret_cast<uint2*>(smem + S.groups * S.stride) + lane;
    const uint64_t inst = uint64_t(blockIdx.x) * S.groups + grp;
    const bool valid = !idle && inst < n;
    const uint64_t off = valid ? inst * n32 : 0;
    pdl_wait();  // launched with launch_pdl
    pdl_trigger();
    if (!idle) {
        const uint32_t nv = 2 * (nb + 1);
#pragma unroll 1
        for (uint32_t v0 = t; v0 < nv; v0 += 4 * g) {
            uint4 qa[4], qb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t v = v0 + i * g;
                qa[i] = classic::load_slot<VEC>(a + off, v, n32, valid);
                qb[i] = classic::load_slot<VEC>(b + off, v, n32, valid);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t v = v0 + i * g;
                if (v < nv) {
                    reinterpret_cast<uint4*>(gA)[v] = qa[i];
                    gB4[(v & 1) * (nb + 1) + (v >> 1)] = qb[i];
                }
            }
        }
    }
    __syncwarp();
    const uint4* gA4 = reinterpret_cast<const uint4*>(gA);
#pragma unroll 1
    for (uint32_t rd = 0; rd < S.rounds; ++rd) {
        const uint32_t s0 = rd * g + t;
        const uint32_t s = FULL ? min(s0, nb - 1) : s0;  // past the pairs: repeats, or runs on the zero block
        const bool mirror = !FULL && s < S.pairs && s < nb - 1 - s;
        auto load = [&](uint32_t k, uint4 (&q)[4]) {
            uint32_t i, j;
            if (FULL) {
                i = k;
                j = k <= s ? s - k : s + nb - k;
            } else {
                const bool first = k <= s;
                i = first ? k : k - s - 1;
                j = first ? s - k : nb - k;
                if (first ? s >= S.pairs : !mirror) i = j = nb;
            }
            q[0] = gA4[2 * i];
            q[1] = gA4[2 * i + 1];
            q[2] = gB4[j];
            q[3] = gB4[nb + 1 + j];
        };
        DiagAcc acc;
#pragma unroll
        for (int w = 0; w < 2 * T; ++w) acc.a[w] = 0;
#pragma unroll
        for (int w = 0; w < 2 * T - 2; ++w) acc.b[w] = 0;
#pragma unroll
        for (int w = 0; w < T + 1; ++w) acc.cc[w] = 0;
        uint2* sl = slots + rd * PAIRS * 32;
        uint4 nq[4];
        load(0, nq);
#pragma unroll 2
        for (uint32_t k = 0; k < S.steps; ++k) {
            uint32_t A[T], B[T];
            A[0] = nq[0].x; A[1] = nq[0].y; A[2] = nq[0].z; A[3] = nq[0].w;
            A[4] = nq[1].x; A[5] = nq[1].y; A[6] = nq[1].z; A[7] = nq[1].w;
            B[0] = nq[2].x; B[1] = nq[2].y; B[2] = nq[2].z; B[3] = nq[2].w;
            B[4] = nq[3].x; B[5] = nq[3].y; B[6] = nq[3].z; B[7] = nq[3].w;
            if (k + 1 < S.steps) load(k + 1, nq);
            classic::tile_mac(A, B, acc);
            if (k == s) {
#pragma unroll
                for (int w = 0; w < T; ++w) sl[w * 32] = make_uint2(acc.a[2 * w], acc.a[2 * w + 1]);
#pragma unroll
                for (int w = 0; w < T - 1; ++w) sl[(T + w) * 32] = make_uint2(acc.b[2 * w], acc.b[2 * w + 1]);
#pragma unroll
                for (int w = 0; w < T / 2; ++w)
                    sl[(2 * T - 1 + w) * 32] = make_uint2(acc.cc[2 * w], acc.cc[2 * w + 1]);
                sl[(2 * T - 1 + T / 2) * 32] = make_uint2(acc.cc[T], 0u);
            }
        }
        uint32_t d1[ACC], d2[ACC], snap[2 * PAIRS];
#pragma unroll
        for (int w = 0; w < PAIRS; ++w) {
            const uint2 v = sl[w * 32];
            snap[2 * w] = v.x;
            snap[2 * w + 1] = v.y;
        }
        classic::fold(snap, snap + 2 * T, snap + 4 * T - 2, d1);
        classic::fold(acc.a, acc.b, acc.cc, d2);
        sub_cc(d2[0], d1[0]);
#pragma unroll
        for (int w = 1; w < ACC - 1; ++w) subc_cc(d2[w], d1[w]);
        subc(d2[ACC - 1], d1[ACC - 1]);
        // D1 in pairs 0..8, D2 in pairs 9..17 of the lane's slots of this round
#pragma unroll
        for (int w = 0; w < ACC / 2; ++w) {
            sl[w * 32] = make_uint2(d1[2 * w], d1[2 * w + 1]);
            sl[(9 + w) * 32] = make_uint2(d2[2 * w], d2[2 * w + 1]);
        }
        sl[(ACC / 2) * 32] = make_uint2(d1[ACC - 1], 0u);
        sl[(9 + ACC / 2) * 32] = make_uint2(d2[ACC - 1], 0u);
    }
    __syncwarp();
    // output blocks in rows of g
    const uint32_t total = FULL ? 2 * nb : nb, rlen = FULL ? 2 * n32 : n32;
    const uint2* all = reinterpret_cast<const uint2*>(smem + S.groups * S.stride) + base;
    // pair 0 of anti-diagonal sd's value, or null (those past the result are zero)
    auto diag = [&](uint32_t sd) -> const uint2* {
        if (sd >= total) return nullptr;  // (also sd = -1, -2)
        uint32_t s = sd, hi = 0;
        if (FULL) {
            if (sd >= nb) s = sd - nb, hi = 9;
        } else if (sd >= S.pairs) {
            s = nb - 1 - sd, hi = 9;
        }
        const uint32_t rd = (s * S.inv) >> 16;
        return all + (rd * PAIRS + hi) * 32 + (s - rd * g);
    };
    const uint32_t mask = g == 32 ? MI_FULL_MASK : (1u << g) - 1u;
    const uint32_t below = base + (t ? t - 1 : g - 1);  // the lane of the block before (t = 0: in the row before)
    uint32_t kprev = 0, cprev = 0;  // lane g-1's add3 carry and the lookahead's carry out of the row before
    uint32_t* rr = r + off * (FULL ? 2 : 1);
#pragma unroll 1
    for (uint32_t q0 = 0; q0 < total; q0 += g) {
        const uint32_t q = q0 + t;
        uint32_t L[T], H[T], v[T], O = 0;
        const uint2* p = diag(q);
#pragma unroll
        for (int w = 0; w < T / 2; ++w) {
            const uint2 x = p ? p[w * 32] : make_uint2(0, 0);
            L[2 * w] = x.x, L[2 * w + 1] = x.y;
        }
        p = diag(q - 1);
#pragma unroll
        for (int w = 0; w < T / 2; ++w) {
            const uint2 x = p ? p[(T / 2 + w) * 32] : make_uint2(0, 0);
            H[2 * w] = x.x, H[2 * w + 1] = x.y;
        }
        p = diag(q - 2);
        if (p) O = p[T * 32].x;
        const uint32_t k = classic::add3_block(L, H, O, v);
        const uint32_t kb = __shfl_sync(MI_FULL_MASK, k, int(below));
        const uint32_t e = classic::add_word_block(v, t ? kb : kprev);
        const uint32_t GB = __ballot_sync(MI_FULL_MASK, e != 0), PB = __ballot_sync(MI_FULL_MASK, classic::all_ones(v));
        const uint64_t X = ((GB | PB) >> base) & mask, Y = (GB >> base) & mask, sum = X + Y + cprev;
        classic::add_word_block(v, uint32_t((sum ^ X ^ Y) >> t) & 1u);
        cprev = uint32_t(sum >> g) & 1u;
        kprev = __shfl_sync(MI_FULL_MASK, k, int(base + g - 1));
        if (valid && q < total) classic::store_block<VEC>(rr, q * T, rlen, v);
    }
}

}  // namespace

// The shape for `rounds`, with at most 32 lanes per group.
static FlexShape flex_shape(uint32_t n32, bool full, uint32_t rounds) {
    FlexShape S;
    S.nb = (n32 + T - 1) / T;
    S.pairs = full ? S.nb : (S.nb + 1) / 2;
    S.steps = full ? S.nb : S.nb + 1;
    S.rounds = rounds;
    S.lanes = (S.pairs + rounds - 1) / rounds;
    S.groups = 32 / S.lanes;
    S.inv = (65536 + S.lanes - 1) / S.lanes;
    S.stride = 2 * (S.nb + 1) * T + 4;  // (the 4 words keep the groups' blocks on distinct banks)
    return S;
}

// The rule counts steps: a warp's steps times the warps a scheduler runs one
// after another (at least kLone, the cost of a warp on its own), times the
// measured cost of a step relative to the loops of mul.cu and mul_lo.cu at
// non-power-of-two sizes -- 1.05 to 1.08, 1.18 and 1.26 to 1.33 for one, two and three
// rounds (more rounds leave fewer warps per SM for the slots' shared memory).  Those
// loops run on 16 or more threads per product (32 or more blocks for low
// halves) only, 0.88 of a step where nb fills the group; below 16 warps per SM
// their launches overlap less, at 124 registers (full products of 1500 x 68
// limbs 14.1 us against 12.4), and blocks of eight warps spread badly (low
// halves of 1000 x 100 limbs 14.1 against 9.9).
uint32_t flex_rounds(uint32_t n, uint32_t n32, bool full) {
    constexpr double kLone = 1.2, kStep[2][4] = {{1.0, 1.05, 1.18, 1.26}, {1.0, 1.08, 1.18, 1.33}};  // [full][rounds]
    const double schedulers = 4.0 * sm_count();
    const uint32_t nb = (n32 + T - 1) / T, steps = full ? nb : nb + 1;
    uint32_t threads = 1;  // of a power-of-two group
    while (threads < (full ? nb : (nb + 1) / 2)) threads *= 2;
    double best = 1e300;
    uint32_t pick = 0;
    if (threads >= 16) {
        const double warps = double(n) * threads / 32;
        const bool fills = nb == (full ? threads : 2 * threads);
        best = steps * (fills ? 0.88 : kStep[full][0]) * std::max(kLone, warps / schedulers);
        if (warps < 16.0 * sm_count()) best *= full ? 1.15 : 1.3;
    }
    for (uint32_t rounds = 1; rounds <= 3; ++rounds) {
        const FlexShape S = flex_shape(n32, full, rounds);
        if (S.lanes > 32) continue;
        const double warps = std::ceil(double(n) / S.groups);
        const double cost = double(rounds) * steps * kStep[full][rounds] * std::max(kLone, warps / schedulers);
        if (cost < best) best = cost, pick = rounds;
    }
    return pick;
}

mi_status launch_mul_flex(const uint32_t* a, const uint32_t* b, uint32_t* r, uint32_t n, uint32_t n32, bool full,
                          uint32_t rounds, cudaStream_t st) {
    const bool vec = aligned16(a) && aligned16(b) && aligned16(r) && (n32 % 4 == 0);
    const FlexShape S = flex_shape(n32, full, rounds);
    auto kern = full ? (vec ? k_mul_flex<true, true> : k_mul_flex<true, false>)
                     : (vec ? k_mul_flex<false, true> : k_mul_flex<false, false>);
    MI_TRY(ensure_dyn_smem(kern, S.smem()));
    const uint64_t blocks = (uint64_t(n) + S.groups - 1) / S.groups;
    MI_CUDA_TRY(launch_pdl(kern, dim3(uint32_t(blocks)), dim3(32), S.smem(), st, a, b, r, n, n32, S));
    return MI_OK;
}

}  // namespace mi
