// mul_flex.cuh -- classical products on groups of any number of lanes of a
// warp: shapes, the rounds of tiles and the rows of output blocks, shared by
// the batched products (mul_flex.cu) and the fused composite (poly.cu).  What
// the shapes mean and why is told in mul_flex.cu.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "mul_core.cuh"

namespace mi {

struct FlexShape {
    uint32_t nb, pairs, steps, rounds, lanes, groups, inv;  // inv: ceil(2^16 / lanes)
    uint32_t stride;                                        // words between the groups' operands
    size_t smem() const { return (size_t(groups) * stride + size_t(rounds) * 32 * 2 * classic::PAIRS) * 4; }
};

// The shape for `rounds`, with at most 32 lanes per group (0 groups: it needs
// more); `numbers` is how many staged numbers of nb + 1 blocks a group keeps.
inline FlexShape flex_shape(uint32_t n32, bool full, uint32_t rounds, uint32_t numbers) {
    FlexShape S;
    S.nb = (n32 + classic::T - 1) / classic::T;
    S.pairs = full ? S.nb : (S.nb + 1) / 2;
    S.steps = full ? S.nb : S.nb + 1;
    S.rounds = rounds;
    S.lanes = (S.pairs + rounds - 1) / rounds;
    S.groups = 32 / S.lanes;
    S.inv = (65536 + S.lanes - 1) / S.lanes;
    S.stride = numbers * (S.nb + 1) * classic::T + 4;  // (the 4 words keep the groups' blocks on distinct banks)
    return S;
}

namespace flex {

using classic::ACC;
using classic::DiagAcc;
using classic::PAIRS;
using classic::T;

// A lane's place: its group, its index in the group and the group's first
// lane.  Lanes past the groups repeat lane 0's work and store nothing.
struct Place {
    uint32_t grp, t, base;
    bool idle;
    __device__ __forceinline__ explicit Place(const FlexShape& S) {
        const uint32_t lane = threadIdx.x;
        idle = lane >= S.groups * S.lanes;
        grp = idle ? 0u : lane / S.lanes;
        base = grp * S.lanes;
        t = idle ? 0u : lane - base;
    }
};

// Stages a row of n32 words as a number: two planes of nb + 1 16-byte halves
// (half h of block j at h (nb + 1) + j), block nb zero.  By the group's lanes.
template <bool VEC, int N>
__device__ __forceinline__ void stage(uint4* const (&g4)[N], const uint32_t* const (&row)[N], uint32_t n32, bool valid,
                                      const FlexShape& S, uint32_t t) {
    const uint32_t nv = 2 * (S.nb + 1);
#pragma unroll 1
    for (uint32_t v0 = t; v0 < nv; v0 += 4 * S.lanes) {
        uint4 q[N][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k = 0; k < N; ++k) q[k][i] = classic::load_slot<VEC>(row[k], v0 + i * S.lanes, n32, valid);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t v = v0 + i * S.lanes;
            if (v < nv) {
#pragma unroll
                for (int k = 0; k < N; ++k) g4[k][(v & 1) * (S.nb + 1) + (v >> 1)] = q[k][i];
            }
        }
    }
}

// The same for all instances of a warp, `count` of them from the rows on, which
// are consecutive in memory: the warp reads them as one run.  (stage() reads
// each row by its own lanes, a part of a 32-byte sector at a time; where the caches
// do not hold the sector until the next part is read, as over the host link, it
// is fetched again.)  By all lanes of the warp.
template <bool VEC, int N>
__device__ __forceinline__ void stage_run(uint32_t* smem, const uint32_t* const (&row)[N], uint32_t n32, uint32_t count,
                                          const FlexShape& S) {
    using E = std::conditional_t<VEC, uint4, uint32_t>;
    constexpr uint32_t PER = VEC ? 1 : 4;  // elements of a 16-byte half
    const uint32_t len = VEC ? n32 / 4 : n32, total = count * len, lane = threadIdx.x;
    const uint32_t inv = ((1u << 22) + len - 1) / len;  // u / len = u inv >> 22: u < 1536, len < 800
#pragma unroll 1
    for (uint32_t base = 0; base < total; base += 4 * 32) {
        E q[N][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k = 0; k < N; ++k)
                q[k][i] = __ldcs(reinterpret_cast<const E*>(row[k]) + min(base + lane + i * 32, total - 1));
        if (base == 0) {  // zeros past the rows, while the first loads are under way
            for (uint32_t v = lane; v < S.groups * S.stride / 4; v += 32)
                reinterpret_cast<uint4*>(smem)[v] = make_uint4(0, 0, 0, 0);
            __syncwarp();
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t u = base + lane + i * 32;
            if (u < total) {
                const uint32_t g = (u * inv) >> 22, e = u - g * len, h = e / PER;
#pragma unroll
                for (int k = 0; k < N; ++k)
                    reinterpret_cast<E*>(smem + g * S.stride + 8 * k * (S.nb + 1))
                        [((h & 1) * (S.nb + 1) + (h >> 1)) * PER + e % PER] = q[k][i];
            }
        }
    }
}

// The rounds of the product of the staged numbers A and B: every lane's pairs
// of anti-diagonal values, D1 in pairs 0..8 and D2 in pairs 9..17 of its slots
// of the round (slots: the lane's first).
template <bool FULL>
__device__ __forceinline__ void rounds(const uint4* gA4, const uint4* gB4, uint2* slots, const FlexShape& S,
                                       uint32_t t) {
    const uint32_t nb = S.nb;
#pragma unroll 1
    for (uint32_t rd = 0; rd < S.rounds; ++rd) {
        const uint32_t s0 = rd * S.lanes + t;
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
            q[0] = gA4[i];
            q[1] = gA4[nb + 1 + i];
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
}

// The output blocks of the product from its slots (the group's first lane's):
// row by row, the block of lane t is put(q, v) for q = t, g + t, ..., with
// block q of a number (z, as staged; null: none) added in.  By every lane of
// the warp, after a __syncwarp.
template <bool FULL, typename F>
__device__ __forceinline__ void rows(const uint2* all, const uint4* z, const FlexShape& S, const Place& L0, F put) {
    const uint32_t nb = S.nb, g = S.lanes, t = L0.t, base = L0.base;
    const uint32_t total = FULL ? 2 * nb : nb;
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
        uint32_t Z[T];
        if (z != nullptr) {
            const bool in = q < nb;
            const uint4 z0 = in ? z[q] : make_uint4(0, 0, 0, 0), z1 = in ? z[nb + 1 + q] : make_uint4(0, 0, 0, 0);
            Z[0] = z0.x, Z[1] = z0.y, Z[2] = z0.z, Z[3] = z0.w, Z[4] = z1.x, Z[5] = z1.y, Z[6] = z1.z, Z[7] = z1.w;
        }
        const uint32_t k = classic::add3_block(L, H, O, v, z != nullptr ? Z : nullptr);
        const uint32_t kb = __shfl_sync(MI_FULL_MASK, k, int(below));
        const uint32_t e = classic::add_word_block(v, t ? kb : kprev);
        const uint32_t GB = __ballot_sync(MI_FULL_MASK, e != 0), PB = __ballot_sync(MI_FULL_MASK, classic::all_ones(v));
        const uint64_t X = ((GB | PB) >> base) & mask, Y = (GB >> base) & mask, sum = X + Y + cprev;
        classic::add_word_block(v, uint32_t((sum ^ X ^ Y) >> t) & 1u);
        cprev = uint32_t(sum >> g) & 1u;
        kprev = __shfl_sync(MI_FULL_MASK, k, int(base + g - 1));
        if (!L0.idle && q < total) put(q, v);
    }
}

}  // namespace flex
}  // namespace mi
