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
// of 16384 x 68 limbs 81.3 -> 64.1 (2), x 80 94.8 -> 75.4 (2), x 96 109 -> 104 (3);
// 30000 x 40 49.4 -> 37.7 (1), 100000 x 16 49.1 -> 27.9 (1), 300000 x 4
// 72.8 -> 14.6 (1); low halves of 12000 x 301 u32 limbs 132 -> 105 (2), 40000 x
// 80 131 -> 90 (1), 200000 x 12 64.7 -> 27.5 (1).  Small groups gain most: their
// blocks of eight warps ran a loop whose lanes took their snapshots one
// group after another.
#include <algorithm>
#include <cmath>

#include "kernels.h"
#include "mul_flex.cuh"

namespace mi {
namespace {

using classic::T;

// MB: blocks per SM at least.  16 (100 registers) for batches that fill the
// GPU; 18 (96) below that, where two launches then fit the SMs at once and
// overlap (1500 x 68 limbs 11.5 us against 15.4; 16384 x 68 66.3 against 64.1,
// low halves of 12000 x 301 words 108 against 104.6).
// LINK: the operands are read over the host link, the warp's rows as one run
// (low halves between pinned buffers, us: 43690 x 24 limbs 190 -> 162, 131072 x
// 8 355 -> 232, 65536 x 4 43.8 -> 42.7; in device memory the run's index arithmetic
// costs more than it saves, 174762 x 3 limbs 8.7 against 11.4).
template <bool FULL, bool VEC, int MB, bool LINK = false>
__global__ void __launch_bounds__(32, MB)
    k_mul_flex(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint32_t* __restrict__ r, uint32_t n,
               uint32_t n32, FlexShape S) {
    extern __shared__ __align__(16) uint32_t smem[];
    const flex::Place L(S);
    uint4* gA4 = reinterpret_cast<uint4*>(smem + L.grp * S.stride);
    uint4* gB4 = gA4 + 2 * (S.nb + 1);
    uint2* slots = reinterpret_cast<uint2*>(smem + S.groups * S.stride);
    const uint64_t inst = uint64_t(blockIdx.x) * S.groups + L.grp;
    const bool valid = !L.idle && inst < n;
    const uint64_t off = valid ? inst * n32 : 0;
    pdl_wait();  // launched with launch_pdl
    pdl_trigger();
    if constexpr (LINK) {
        const uint64_t first = uint64_t(blockIdx.x) * S.groups;  // below n: the grid has no more blocks
        flex::stage_run<VEC, 2>(smem, {a + first * n32, b + first * n32}, n32,
                                uint32_t(min(uint64_t(S.groups), n - first)), S);
    } else if (!L.idle) {
        flex::stage<VEC, 2>({gA4, gB4}, {a + off, b + off}, n32, valid, S, L.t);
    }
    __syncwarp();
    flex::rounds<FULL>(gA4, gB4, slots + threadIdx.x, S, L.t);
    __syncwarp();
    uint32_t* rr = r + off * (FULL ? 2 : 1);
    const uint32_t rlen = FULL ? 2 * n32 : n32;
    flex::rows<FULL>(slots + L.base, nullptr, S, L, [&](uint32_t q, const uint32_t (&v)[T]) {
        if (valid) classic::store_block<VEC>(rr, q * T, rlen, v);
    });
}

}  // namespace

// Blocks of a shape resident per SM: 18 for the registers of the launches that
// do not fill the GPU, and what the shared memory allows.
static uint32_t flex_resident(const FlexShape& S) {
    return std::min<uint32_t>(18, uint32_t(228 * 1024 / (S.smem() + 1024)));
}

// The rule compares modelled times.  A launch's time is set by the warps of its
// busiest scheduler, k = ceil(warps per SM / 4): steps * (A + B k), A the
// latency of a step on its own, B its share of the scheduler (us
// per step: 0.164 for k_mul, which is 0.92 of that where nb
// fills the group, 0.173 and 0.178 for one round, 0.16 for two and 0.15 for
// three, whose steps share the staging).  k_mul_lo's blocks of eight warps come
// in pairs of warps per scheduler.  More rounds need more shared memory: a second wave of
// blocks costs its own latency.  Power-of-two groups of fewer than 16 threads
// serve no launches here.  Against what this replaced, the same with
// warps / 4 unrounded: 1824 x 177 words 24.4 -> 15.5, 3952 x 177 42.8 -> 30.0.
uint32_t flex_rounds(uint32_t n, uint32_t n32, bool full, double* us) {
    constexpr double kA[2] = {0.18, 0.145}, kB[2] = {0.166, 0.164};  // [full]: the power-of-two groups
    constexpr double kFlexA[2][4] = {{0, 0.16, 0.20, 0.19}, {0, 0.18, 0.18, 0.19}};  // [full][rounds]
    constexpr double kFlexB[2][4] = {{0, 0.178, 0.16, 0.15}, {0, 0.173, 0.158, 0.15}};
    const double sms = sm_count();
    const uint32_t nb = (n32 + T - 1) / T, steps = full ? nb : nb + 1;
    uint32_t threads = 1;  // of a power-of-two group
    while (threads < (full ? nb : (nb + 1) / 2)) threads *= 2;
    double best = 1e300;
    uint32_t pick = 0;
    if (threads >= 16) {
        const double w = std::ceil(double(n) * threads / 32) / sms;  // warps per SM
        double k = std::ceil(w / 4);
        if (!full) k = 2 * std::ceil(w / 8);
        best = steps * (kA[full] + kB[full] * k);
        if (nb == (full ? threads : 2 * threads)) best *= 0.92;
    }
    for (uint32_t rounds = 1; rounds <= 3; ++rounds) {
        const FlexShape S = flex_shape(n32, full, rounds, 2);
        if (S.lanes > 32) continue;
        const double w = std::ceil(double(n) / S.groups) / sms;
        const double waves = w > flex_resident(S) ? 2 : 1;
        const double cost = double(rounds) * steps * (kFlexA[full][rounds] * waves + kFlexB[full][rounds] * std::ceil(w / 4));
        if (cost < best) best = cost, pick = rounds;
    }
    *us = best;
    return pick;
}

mi_status launch_mul_flex(const uint32_t* a, const uint32_t* b, uint32_t* r, uint32_t n, uint32_t n32, bool full,
                          uint32_t rounds, cudaStream_t st, bool link, uint32_t max_per_sm) {
    // The batches whose rows in flight over the link outgrow the caches (us between
    // pinned buffers, each lane its rows against one run: 32768 x 8 limbs 82 and 58,
    // 10922 x 24 56 and 47, 131072 x 4 82 and 62).  Below, and for shorter rows, the
    // run's arithmetic costs a microsecond (21845 x 5 words 21.1 and 22.2).
    link = link && !full && n32 > 4 && uint64_t(n) * n32 * 4 >= (n32 <= 8 ? 3u << 20 : 1u << 20);
    const bool vec = aligned16(a) && aligned16(b) && aligned16(r) && (n32 % 4 == 0);
    const FlexShape S = flex_shape(n32, full, rounds, 2);
    const uint64_t blocks = (uint64_t(n) + S.groups - 1) / S.groups;
    using Kernel = void (*)(const uint32_t*, const uint32_t*, uint32_t*, uint32_t, uint32_t, FlexShape);
    static constexpr Kernel kernels[2][2][2] = {  // [few blocks][full][vec]
        {{k_mul_flex<false, false, 16>, k_mul_flex<false, true, 16>},
         {k_mul_flex<true, false, 16>, k_mul_flex<true, true, 16>}},
        {{k_mul_flex<false, false, 18>, k_mul_flex<false, true, 18>},
         {k_mul_flex<true, false, 18>, k_mul_flex<true, true, 18>}}};
    static constexpr Kernel link_kernels[2] = {k_mul_flex<false, false, 16, true>, k_mul_flex<false, true, 16, true>};
    const Kernel kern = link ? link_kernels[vec] : kernels[blocks <= 16u * uint64_t(sm_count())][full][vec];
    size_t smem = S.smem();
    // Over the link few resident blocks, as in mul.cu, for their results to leave
    // while the others' operands arrive: four warps for each of its blocks of
    // eight (with 4, 8, 12, 16 and 21 per SM, us: 43690 x 24 limbs 110, 127, 145, 161, 162; 262144
    // x 1 50.0, 38.8, 38.3, 38.3, 38.4).
    if (link)
        MI_TRY(capped_smem(smem, 4 * max_per_sm, &smem));
    else
        MI_TRY(balanced_smem(blocks, flex_resident(S), &smem));
    MI_TRY(ensure_dyn_smem(kern, smem));
    MI_CUDA_TRY(launch_pdl(kern, dim3(uint32_t(blocks)), dim3(32), smem, st, a, b, r, n, n32, S));
    return MI_OK;
}

}  // namespace mi
