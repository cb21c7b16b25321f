// poly_ntt.cu -- the fused polynomial composite ((a^2 + b)(b^2 + b) + ab) mod
// 2^(64m) on number-theoretic transforms, for operands from a few hundred u64
// limbs up, where a transform product is cheaper than the classical one.
//
// Counterpart of the reference's polyFttKer (cuda/ker-fft-mul.cu.h:456-509),
// which runs four FFT products and three additions on 16-bit digits in one
// kernel (and, like its bmulFFT, is exact only for tiny inputs).  The
// classical form of the same composite is poly.cu (polyKerQ).
//
// One CTA of L/8 threads owns an instance (L = pow2ceil(2m), the transform
// length of an m x m product, so the cyclic convolution never wraps into the
// low m coefficients).  The four products all keep only their low m limbs:
//   P3 = ab,  T1 = a^2 + b,  T2 = b^2 + b,  r = T1 T2 + P3   (all mod 2^(64m))
// The first three share the two forward transforms of a and b: per prime, the
// spectra X = F(a), Y = F(b) are taken in lockstep, the three pointwise
// products are X (Y 2^32/L), X (X 2^32/L), Y (Y 2^32/L) by two Shoup and three
// Montgomery products per point, and three inverse transforms leave the
// residues of the low L/2 coefficients of each.  Garner's recombination and
// the digit sums then give the thread's output limbs, the addend of the step
// (b or P3) is added into the digit sums, and one carry pass over the group
// leaves the m limbs in shared memory (T1, T2, P3) or, for the fourth product,
// in the result row: the intermediates never leave the chip.  Per prime 8
// transforms instead of the 12 of four separate products.  (When every product
// transformed its own operands, 10 per prime, 512 composites of 2048 limbs took
// 402 us against 311, 1000 of 1024 limbs 287 against 247, 2000 of 350 limbs
// 262 against 211; the multiply pipe and the issue rate bound both.)  Digit modes (64-bit digits on five
// primes, 48-bit ones on four where they fit the same length) as in
// ntt_mul.cuh.
#include <cstdio>

#include "common.cuh"
#include "kernels.h"
#include "ntt_host.h"
#include "ntt32.cuh"
#include "ntt_mul.cuh"

namespace mi {
namespace {

using ntt32::Field;
using ntt32::Plan;

// Shared memory of one CTA, in 32-bit words: exchange buffers (NX of LX words)
// and, per prime, the low-half residues of the three products (3 L/2 words).
// The intermediates T1, T2, P3 (m <= L/2 u64 limbs, so two pieces of L/2
// words) then take the pieces of their own product at the first two primes,
// and the fourth product's residues the space of the third prime on.  Where
// only one exchange buffer is kept (shorter transforms: three CTAs per SM
// need it), the second one of the forward transforms is the residue space of
// the last prime, which is written only after its own forward transforms.
template <int LG, bool D48>
struct PolySmem {
    static constexpr int L = 1 << LG, HALF = L / 2, NP = D48 ? 4 : ntt32::kPrimes;
    static constexpr int NX = LG == 12 ? 3 : 1;  // also the inverse transforms in lockstep
    static constexpr int SH = 0, RES = NX * Plan<LG>::LX;
    static constexpr size_t WORDS32 = size_t(RES) + size_t(3) * HALF * NP;
    static_assert(NX > 1 || 3 * HALF >= Plan<LG>::LX, "the second exchange buffer");
    static_assert(NP * HALF <= 3 * HALF * (NP - 2), "the fourth product's residues");
};

// Word w of intermediate X (0: T1, 1: T2, 2: P3) in the residue space.
template <int LG>
__device__ __forceinline__ uint32_t mid_word(int X, uint32_t w) {
    constexpr uint32_t HALF = Plan<LG>::L / 2;
    return uint32_t(X) * HALF + w + (w >= HALF ? 2 * HALF : 0u);
}

// Digit i of a number of `words` 32-bit words read through rd, as its low 32
// bits and its high ones; zero past the number.
template <bool D48, typename F>
__device__ __forceinline__ uint2 digit_of(F rd, uint32_t words, uint32_t i) {
    if constexpr (D48) {
        const uint32_t w = (3 * i) >> 1;
        const uint32_t w0 = w < words ? rd(w) : 0u;
        const uint32_t w1 = w + 1 < words ? rd(w + 1) : 0u;
        return (i & 1) ? make_uint2(__funnelshift_r(w0, w1, 16), w1 >> 16) : make_uint2(w0, w1 & 0xffffu);
    } else {
        return 2 * i < words ? make_uint2(rd(2 * i), rd(2 * i + 1)) : make_uint2(0u, 0u);
    }
}

// Recombines one product: Garner and the digit sums of the thread's 8
// coefficients (those of the low half only; the others reach limbs >= m or do
// not exist) from the residues at res[q * stride], plus limb i < m of
// `addend`, carried over the group; `put` receives limb i < m.  Every thread of
// the block calls this; it ends with a barrier.
template <int LG, bool D48, typename FA, typename FP>
__device__ __forceinline__ void recombine(const uint32_t* res, int stride, uint32_t m, const NttMulParams& P,
                                          uint32_t* sh, uint32_t* scr, FA addend, FP put) {
    using Pl = Plan<LG>;
    constexpr int HALF = Pl::L / 2, DM = D48 ? ntt32::DM48 : ntt32::DM64, NP = ntt32::Digits<DM>::NP;
    constexpr int OUT = ntt32::Digits<DM>::OUT, OVW = ntt32::Digits<DM>::OVW, SW = OUT + OVW;
    const uint32_t t = threadIdx.x % Pl::NT;
    uint64_t s[SW];
#pragma unroll
    for (int w = 0; w < SW; ++w) s[w] = 0;
    if (8 * t < HALF) {
        ntt32::DigitSum<DM> sum;
#pragma unroll
        for (int j = 0; j < 8; j += 4) {
            const uint32_t slot = ntt32::swz(8 * t + j);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                uint32_t y[NP], acc[5];
#pragma unroll
                for (int q = 0; q < NP; ++q) y[q] = res[q * stride + slot + h];
                ntt32::garner<NP>(y, P, acc);
                sum.add(j + h, acc);
            }
        }
        sum.get(s);
    }
    // the addend's limbs of the thread's block enter the digit sums
    const uint32_t o0 = OUT * t;
    {
        unsigned __int128 acc = 0;
#pragma unroll
        for (int w = 0; w < SW; ++w) {
            acc += s[w];
            if (w < OUT && o0 + w < m) acc += addend(o0 + w);
            s[w] = uint64_t(acc);
            acc >>= 64;
        }
    }
    // overflow words to the right neighbour, one carry pass, limbs below m out
    uint64_t* ov = reinterpret_cast<uint64_t*>(sh);
#pragma unroll
    for (int w = 0; w < OVW; ++w) ov[OVW * t + w] = s[OUT + w];
    __syncthreads();  // also: every residue of the product has been read
    uint64_t add[OUT], lo[OUT], blk[OUT];
#pragma unroll
    for (int w = 0; w < OUT; ++w) {
        add[w] = (w < OVW && t > 0) ? ov[OVW * (t - 1) + w] : 0ull;
        lo[w] = s[w];
    }
    bool g, p;
    chunk_add<uint64_t, OUT>(lo, add, blk, g, p);
    uint32_t gc;
    const uint32_t cin = group_carry<Pl::NT>(g, p, 0u, &gc, scr);
    chunk_inc<uint64_t, OUT>(blk, cin);
#pragma unroll
    for (int w = 0; w < OUT; ++w)
        if (o0 + w < m) put(o0 + w, blk[w]);
    __syncthreads();
}

// 768 threads per SM where shared memory allows (8.6 L words per CTA: three
// 256-thread CTAs for 2048-point transforms, one 512-thread CTA, with more
// buffers, for 4096); 512 for the 256-point ones, whose 48-bit digit mode
// spills at 80 registers
template <int LG, bool D48>
__global__ void __launch_bounds__((1 << LG) / 8, LG == 12 ? 1 : (LG == 8 ? 512 : 768) / ((1 << LG) / 8))
    k_poly_ntt(const uint64_t* __restrict__ a, const uint64_t* __restrict__ b, uint64_t* __restrict__ r, uint32_t n,
               uint32_t m, NttMulParams P) {
    using S = PolySmem<LG, D48>;
    using Pl = Plan<LG>;
    constexpr int HALF = S::HALF, NP = S::NP;
    extern __shared__ __align__(16) uint32_t smem32[];
    uint32_t* scr = smem32 + S::WORDS32;
    uint32_t* res = smem32 + S::RES;
    uint32_t* res4 = res + 2 * 3 * HALF;  // residues of the fourth product
    const uint32_t t = threadIdx.x;
    // exchange of two arrays: two buffers, or one and the last prime's residues
    uint32_t* const sh = smem32 + S::SH;
    constexpr int GAP = S::NX > 1 ? Pl::LX : S::RES + 3 * HALF * (NP - 1);  // of the second buffer
    pdl_wait();  // small batches are launched with launch_pdl
    pdl_trigger();
    for (uint64_t inst = blockIdx.x; inst < n; inst += gridDim.x) {
        const uint64_t* ai = a + inst * m;
        const uint64_t* bi = b + inst * m;
        uint64_t* ri = r + inst * m;
#pragma unroll 1
        for (int q = 0; q < NP; ++q) {
            const Field f{P.p[q], 2 * P.p[q], P.pinv[q]};
            const uint2 ka = P.ka[q], ks = P.ka_by_lg[q][LG - 8][1];
            uint32_t v[2][8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {  // m digits fit L/2: the upper halves are zero
                const uint2 da = digit_of<D48>(
                    [&](uint32_t w) { return __ldg(reinterpret_cast<const uint32_t*>(ai) + w); }, 2 * m, t + Pl::NT * j);
                const uint2 db = digit_of<D48>(
                    [&](uint32_t w) { return __ldg(reinterpret_cast<const uint32_t*>(bi) + w); }, 2 * m, t + Pl::NT * j);
                v[0][j] = f.digit(da.x, da.y, ka);
                v[1][j] = f.digit(db.x, db.y, ka);
            }
            ntt32::forward<LG, 2, true, GAP>(v, sh, P.tw[q], f);
            uint32_t z[3][8];  // a^2, b^2, ab
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t sa = f.shoup(v[0][j], ks), sb = f.shoup(v[1][j], ks);
                z[0][j] = f.mont(v[0][j], sa);
                z[1][j] = f.mont(v[1][j], sb);
                z[2][j] = f.mont(v[0][j], sb);
            }
            uint32_t* rq = res + q * 3 * HALF;
            if constexpr (S::NX > 1) {
                ntt32::inverse<LG, 3>(z, sh, P.itw[q], f);
#pragma unroll
                for (int x = 0; x < 3; ++x)
#pragma unroll
                    for (int j = 0; j < 4; ++j) rq[x * HALF + ntt32::swz(t + Pl::NT * j)] = f.reduce(z[x][j]);
            } else {
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    // an inverse transform begins with exchanges within warps and
                    // ends with one across them
                    if (x > 0) __syncthreads();
                    ntt32::inverse<LG>(z[x], sh, P.itw[q], f);
#pragma unroll
                    for (int j = 0; j < 4; ++j) rq[x * HALF + ntt32::swz(t + Pl::NT * j)] = f.reduce(z[x][j]);
                }
            }
        }
        __syncthreads();
        auto get = [&](int X, uint32_t i) -> uint64_t {
            return *reinterpret_cast<const uint64_t*>(res + mid_word<LG>(X, 2 * i));
        };
#pragma unroll 1
        for (int X = 0; X < 3; ++X)  // T1 = a^2 + b, T2 = b^2 + b, P3 = ab
            recombine<LG, D48>(
                res + X * HALF, 3 * HALF, m, P, sh, scr, [&](uint32_t i) { return X < 2 ? __ldg(bi + i) : 0ull; },
                [&](uint32_t i, uint64_t v) { *reinterpret_cast<uint64_t*>(res + mid_word<LG>(X, 2 * i)) = v; });
#pragma unroll 1
        for (int q = 0; q < NP; ++q) {
            const Field f{P.p[q], 2 * P.p[q], P.pinv[q]};
            // T1 unscaled, T2 times 2^32 / L
            const uint2 ka = P.ka[q], kb = P.kb_by_lg[q][LG - 8];
            uint32_t v[2][8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint2 d1 = digit_of<D48>([&](uint32_t w) { return res[mid_word<LG>(0, w)]; }, 2 * m, t + Pl::NT * j);
                const uint2 d2 = digit_of<D48>([&](uint32_t w) { return res[mid_word<LG>(1, w)]; }, 2 * m, t + Pl::NT * j);
                v[0][j] = f.digit(d1.x, d1.y, ka);
                v[1][j] = f.digit(d2.x, d2.y, kb);
            }
            ntt32::forward<LG, 2, true, GAP>(v, sh, P.tw[q], f);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[0][j] = f.mont(v[0][j], v[1][j]);
            ntt32::inverse<LG>(v[0], sh, P.itw[q], f);
#pragma unroll
            for (int j = 0; j < 4; ++j) res4[q * HALF + ntt32::swz(t + Pl::NT * j)] = f.reduce(v[0][j]);
        }
        __syncthreads();
        recombine<LG, D48>(res4, HALF, m, P, sh, scr, [&](uint32_t i) { return get(2, i); },
                           [&](uint32_t i, uint64_t v) { ri[i] = v; });  // r = T1 T2 + P3
    }
}

template <int LG, bool D48>
mi_status launch_lg(const uint64_t* a, const uint64_t* b, uint64_t* r, uint32_t n, uint32_t m, const NttMulParams& P,
                    cudaStream_t st) {
    constexpr int NT = (1 << LG) / 8;
    const size_t smem = PolySmem<LG, D48>::WORDS32 * 4 + size_t(NT / 32 + 1) * 4;
    auto kern = k_poly_ntt<LG, D48>;
    static ResidentBlocks site;
    int per_sm = 0;
    MI_TRY(site.get(kern, NT, smem, &per_sm));
    uint64_t blocks = uint64_t(sm_count()) * uint64_t(per_sm);
    if (blocks > n) blocks = n;
    if (ntt_dependent(n, per_sm)) {  // as the products do
        MI_CUDA_TRY(launch_pdl(kern, dim3(uint32_t(blocks)), dim3(NT), smem, st, a, b, r, n, m, P));
        return MI_OK;
    }
    kern<<<dim3(uint32_t(blocks)), dim3(NT), smem, st>>>(a, b, r, n, m, P);
    MI_CUDA_TRY(cudaGetLastError());
    return MI_OK;
}

}  // namespace

mi_status launch_poly_ntt(const uint64_t* a, const uint64_t* b, uint64_t* r, uint32_t n, uint32_t m,
                          const NttMulParams& P, cudaStream_t st) {
    uint32_t L = pow2ceil(2 * m);
    if (L < 256) L = 256;
    const bool d48 = 2 * ntt32::ntt_digits(m, true) <= L;
    switch (L) {
        case 256: return d48 ? launch_lg<8, true>(a, b, r, n, m, P, st) : launch_lg<8, false>(a, b, r, n, m, P, st);
        case 512: return d48 ? launch_lg<9, true>(a, b, r, n, m, P, st) : launch_lg<9, false>(a, b, r, n, m, P, st);
        case 1024: return d48 ? launch_lg<10, true>(a, b, r, n, m, P, st) : launch_lg<10, false>(a, b, r, n, m, P, st);
        case 2048: return d48 ? launch_lg<11, true>(a, b, r, n, m, P, st) : launch_lg<11, false>(a, b, r, n, m, P, st);
        case 4096: return d48 ? launch_lg<12, true>(a, b, r, n, m, P, st) : launch_lg<12, false>(a, b, r, n, m, P, st);
        default: return set_error(MI_EINVAL, "poly_ntt: %u limbs exceeds the maximum %u", m, kNttMaxLimbs);
    }
}

}  // namespace mi
