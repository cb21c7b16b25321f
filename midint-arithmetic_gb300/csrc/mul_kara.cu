// mul_kara.cu -- batched full classical products of 25..32 blocks of T limbs
// with one level of Karatsuba.
//
// With h = ceil(nb / 2) blocks, a = a0 + a1 X and b = b0 + b1 X for X = B^h:
//
//   a b = P0 + (P0 + P2 - s |a0 - a1| |b0 - b1|) X + P2 X^2,   P0 = a0 b0, P2 = a1 b1,
//
// s the sign of (a0 - a1)(b0 - b1).  An instance runs on 16 lanes, two to a
// one-warp block; each lane owns one block of every half operand and the three
// half products are three square products of mul_core.cuh.  Each product leaves
// its 2 x 16 blocks where its operands were, and the result's 4 x 16 blocks are
// summed in four rows: a row's blocks take up to four addends each, their
// carries of 0..3 move up one lane, and the one-bit carries left are one
// lookahead over the row.  s = +1 adds the complement: every bit from block h
// up is flipped and one added there, and what leaves the top is dropped.  The
// tile loops are unrolled for each h of 13..16 (a loop of two steps: 16384 x 120
// limbs 131 us against 119).
//
// Bound by the integer multiply-add pipe in the products (3/4 of k_mul's wide
// multiply-adds) and, for a third of the time, by shared-memory traffic and
// carries around them.  Against k_mul and k_mul_flex (us, 16384 instances):
// 128 limbs 135.3 -> 123.1, 120 136.7 -> 118.6, 112 127.7 -> 112.6, 100 114.0 ->
// 105.5; 60000 x 128 482 -> 417.  With 24 blocks (96 limbs) it loses, 101.9
// against 105.5; with 33 and more the transforms win, 168 for 129..160 limbs.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.h"
#include "mul_core.cuh"

namespace mi {
namespace {

using classic::T;

constexpr int NT = 16;        // lanes per instance
constexpr int IPB = 32 / NT;  // instances per one-warp block
constexpr int W = NT * T;     // words of a half operand
// a0, b0, a1, b1, |a0 - a1|, |b0 - b1| (each pair then holds its product), and
// the snapshot slots of square_product
constexpr int GROUP = 6 * W + NT * classic::PER_T;
constexpr size_t SMEM = size_t(IPB) * GROUP * 4;

// |x - y| of two numbers of NT blocks (thread t holds block t of each), and
// whether x < y.  The borrows are one lookahead; x - y - 1 with the bits
// flipped is y - x, so the negative case only changes the borrow into block 0.
__device__ __forceinline__ bool abs_diff(const uint32_t (&x)[T], const uint32_t (&y)[T], uint32_t (&d)[T]) {
#pragma unroll
    for (int w = 0; w < T; ++w) d[w] = x[w];
    uint32_t br = 0;
    sub_cc(d[0], y[0]);
#pragma unroll
    for (int w = 1; w < T; ++w) subc_cc(d[w], y[w]);
    subc(br, 0u);
    uint32_t any = d[0];
#pragma unroll
    for (int w = 1; w < T; ++w) any |= d[w];
    const uint32_t lane = threadIdx.x & 31u, base = lane & ~uint32_t(NT - 1), vote = group_lanes<NT>();
    constexpr uint32_t mask = (1u << NT) - 1;
    const uint32_t G = __ballot_sync(vote, br != 0), P = __ballot_sync(vote, any == 0);
    const uint32_t X = ((G | P) >> base) & mask, Y = (G >> base) & mask;
    const bool neg = (X + Y) >> NT;
    const uint32_t in = (((X + Y + neg) ^ X ^ Y) >> (lane - base)) & 1u;
    sub_cc(d[0], in);
#pragma unroll
    for (int w = 1; w < T - 1; ++w) subc_cc(d[w], 0u);
    subc(d[T - 1], 0u);
    const uint32_t flip = neg ? MI_FULL_MASK : 0u;
#pragma unroll
    for (int w = 0; w < T; ++w) d[w] ^= flip;
    return neg;
}

// r += y, returns k plus the carry out
__device__ __forceinline__ uint32_t add_block(uint32_t (&r)[T], const uint32_t (&y)[T], uint32_t k) {
    add_cc(r[0], y[0]);
#pragma unroll
    for (int w = 1; w < T; ++w) addc_cc(r[w], y[w]);
    addc(k, 0u);
    return k;
}

__device__ __forceinline__ void lds_block(uint32_t (&v)[T], const uint32_t* p) {
    const uint4 a = reinterpret_cast<const uint4*>(p)[0], b = reinterpret_cast<const uint4*>(p)[1];
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
__device__ __forceinline__ void sts_block(uint32_t* p, const uint32_t (&v)[T]) {
    reinterpret_cast<uint4*>(p)[0] = make_uint4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<uint4*>(p)[1] = make_uint4(v[4], v[5], v[6], v[7]);
}

// Sixteen blocks per SM (126 registers).
template <uint32_t H, bool VEC>
__global__ void __launch_bounds__(32, 16)
    k_mul_kara(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint32_t* __restrict__ r, uint32_t n,
               uint32_t n32) {
    extern __shared__ __align__(16) uint32_t smem[];
    const uint32_t grp = threadIdx.x / NT, t = threadIdx.x % NT;
    uint32_t* gs = smem + grp * GROUP;
    uint2* slots = reinterpret_cast<uint2*>(gs + 6 * W);
    const uint64_t inst = uint64_t(blockIdx.x) * IPB + grp;
    const bool valid = inst < n;
    const uint64_t off = valid ? inst * n32 : 0;
    pdl_wait();  // launched with launch_pdl
    pdl_trigger();
    {  // the halves, in 16-byte slots; b's in the two planes of square_product
        uint4 q[8];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t v = t + i * NT;
            q[i] = classic::load_slot<VEC>(a + off, v, n32, valid && v < 2 * H);
            q[2 + i] = classic::load_slot<VEC>(b + off, v, n32, valid && v < 2 * H);
            q[4 + i] = classic::load_slot<VEC>(a + off, 2 * H + v, n32, valid);
            q[6 + i] = classic::load_slot<VEC>(b + off, 2 * H + v, n32, valid);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t v = t + i * NT, pl = (v & 1) * NT + (v >> 1);
            reinterpret_cast<uint4*>(gs)[v] = q[i];
            reinterpret_cast<uint4*>(gs + W)[pl] = q[2 + i];
            reinterpret_cast<uint4*>(gs + 2 * W)[v] = q[4 + i];
            reinterpret_cast<uint4*>(gs + 3 * W)[pl] = q[6 + i];
        }
    }
    group_sync<NT>();
    uint32_t M;  // all ones where the middle product is subtracted
    {
        uint32_t x[T], y[T], d[T];
        lds_block(x, gs + t * T);
        lds_block(y, gs + 2 * W + t * T);
        const bool na = abs_diff(x, y, d);
        sts_block(gs + 4 * W + t * T, d);
        const uint4* b0 = reinterpret_cast<const uint4*>(gs + W);
        const uint4* b1 = reinterpret_cast<const uint4*>(gs + 3 * W);
        uint4* bd = reinterpret_cast<uint4*>(gs + 5 * W);
        const uint4 x0 = b0[t], x1 = b0[NT + t], y0 = b1[t], y1 = b1[NT + t];
        x[0] = x0.x, x[1] = x0.y, x[2] = x0.z, x[3] = x0.w, x[4] = x1.x, x[5] = x1.y, x[6] = x1.z, x[7] = x1.w;
        y[0] = y0.x, y[1] = y0.y, y[2] = y0.z, y[3] = y0.w, y[4] = y1.x, y[5] = y1.y, y[6] = y1.z, y[7] = y1.w;
        const bool nbg = abs_diff(x, y, d);
        bd[t] = make_uint4(d[0], d[1], d[2], d[3]);
        bd[NT + t] = make_uint4(d[4], d[5], d[6], d[7]);
        M = na == nbg ? MI_FULL_MASK : 0u;
    }
    group_sync<NT>();
#pragma unroll 1
    for (int p = 0; p < 3; ++p) {
        uint32_t* gA = gs + 2 * p * W;
        uint32_t ulo[T], uhi[T];
        classic::square_product<NT, 1, H, true>(gA, reinterpret_cast<uint4*>(gA + W), slots, nullptr, t, ulo, uhi, H);
        group_sync<NT>();
        sts_block(gA + t * T, ulo);
        sts_block(gA + (NT + t) * T, uhi);
    }
    group_sync<NT>();
    // output block j: P0_j (j < 2h) or P2_(j-2h), plus P0_(j-H) + P2_(j-H) -+ Q_(j-H) from j = H on
    uint32_t v[4][T], k[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t j = i * NT + t;
        uint32_t y[T];
        const bool hi = j >= 2 * H;
        const uint32_t jb = hi ? j - 2 * H : j;
#pragma unroll
        for (int w = 0; w < T; ++w) v[i][w] = 0;
        if (jb < 2 * NT) lds_block(v[i], gs + (hi ? 2 * W : 0) + jb * T);
        k[i] = 0;
        if (j >= H) {
            const uint32_t jm = j - H;
            if (jm < 2 * NT) {
                lds_block(y, gs + jm * T);
                k[i] = add_block(v[i], y, k[i]);
                lds_block(y, gs + 2 * W + jm * T);
                k[i] = add_block(v[i], y, k[i]);
                lds_block(y, gs + 4 * W + jm * T);
            } else {
#pragma unroll
                for (int w = 0; w < T; ++w) y[w] = 0;
            }
#pragma unroll
            for (int w = 0; w < T; ++w) y[w] ^= M;
            k[i] = add_block(v[i], y, k[i]);
        }
    }
    // carries: 0..3 of each block to the next, then a one-bit ripple
    const uint32_t lanes = group_lanes<NT>();
    uint32_t in = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t up = __shfl_up_sync(lanes, k[i], 1, NT);
        const uint32_t top = __shfl_sync(lanes, k[i], NT - 1, NT);
        uint32_t c = t ? up : in;
        if (uint32_t(i) * NT + t == H) c += M & 1u;
        in = top;
        k[i] = classic::add_word_block(v[i], c);
    }
    uint32_t cin = 0;
    uint32_t* rr = r + off * 2;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t gc;
        const uint32_t c = group_carry<NT>(k[i] != 0, classic::all_ones(v[i]), cin, &gc, nullptr);
        cin = gc;
        classic::add_word_block(v[i], c);
        if (valid) classic::store_block<VEC>(rr, (i * NT + t) * T, 2 * n32, v[i]);
    }
}

}  // namespace

// A warp holds two instances where k_mul's holds one, so a batch that leaves
// the SMs partly empty waits longer for its warps.  The rule compares modelled
// times as flex_rounds does: the latency of the 3 h steps and, for each warp of
// the busiest scheduler, theirs and 2 us of staging and carries, against the
// form that it would replace (4 % of it in hand, 9 % on
// unaligned rows).  us against the other
// forms: 4257 x 128 limbs 39.4 against 41.4, 4000 x 128 39.5 against 37.7, 4257 x
// 100 33.8 against 35.2, 4000 x 100 34.1 against 31.8, 5000 x 128 48.5 against
// 46.9, 7000 x 128 56.3 against 61.6, 2280 x 120 21 against 23.7.
bool kara_pays(uint32_t n, uint32_t n32, bool vec, double* us) {
    if (n32 <= 24 * T || n32 > 2 * NT * T) return false;
    const double w = std::ceil(double(n) / IPB) / sm_count(), steps = 3 * ((n32 + 2 * T - 1) / (2 * T));
    // the first blocks of a second wave crowd the schedulers that free first
    const double k = w <= 16 ? std::ceil(w / 4) : std::max(6.0, std::ceil(w / 4 + 0.1));
    const double own = steps * 0.13 + 0.5 + k * (2.05 + 0.131 * steps);
    if (own >= (vec ? 0.96 : 0.91) * *us) return false;
    *us = own;
    return true;
}

mi_status launch_mul_kara(const uint32_t* a, const uint32_t* b, uint32_t* r, uint32_t n, uint32_t n32,
                          cudaStream_t st) {
    const bool vec = aligned16(a) && aligned16(b) && aligned16(r) && (n32 % 4 == 0);
    using Kernel = void (*)(const uint32_t*, const uint32_t*, uint32_t*, uint32_t, uint32_t);
    static constexpr Kernel kernels[4][2] = {{k_mul_kara<13, false>, k_mul_kara<13, true>},
                                             {k_mul_kara<14, false>, k_mul_kara<14, true>},
                                             {k_mul_kara<15, false>, k_mul_kara<15, true>},
                                             {k_mul_kara<16, false>, k_mul_kara<16, true>}};
    const uint32_t h = std::max((n32 + 2 * T - 1) / (2 * T), 13u);
    const Kernel kern = kernels[h - 13][vec];
    const uint32_t blocks = uint32_t((uint64_t(n) + IPB - 1) / IPB);
    MI_TRY(ensure_dyn_smem(kern, SMEM));
    MI_CUDA_TRY(launch_pdl(kern, dim3(blocks), dim3(32), SMEM, st, a, b, r, n, n32));
    return MI_OK;
}

}  // namespace mi
