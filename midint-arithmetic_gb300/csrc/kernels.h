// kernels.h -- host launchers of the device kernels (internal to the library).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/midint.h"

namespace mi {

enum AddOp : int { ADD_PLAIN = 0, ADD_SIX = 1 };

// Device state of the additions wider than one block (decoupled look-back):
// `status` holds two arrays of kWideWords words of tile states (32 tiles per
// word, two bits each), then the tile counter, then the error word (set when
// a bounded wait gave up), then one byte per tile for in-place calls.  One per
// context; wide additions on one context must not overlap on the device.  The
// host side keeps which array the next launch takes, how many words of the
// other the last one used, and the counter values issued so far.  A call that is
// captured into a graph takes none of these, which a replay could not follow: it
// has a second such area, cleared by the graph itself (the error word is the
// first area's).
constexpr uint32_t kWideTiles = 1u << 16;  // per launch
constexpr uint32_t kWideWords = kWideTiles / 2;  // an instance has at least two tiles and starts a word
constexpr size_t kWideBytes = (2 * size_t(kWideWords) + 2) * 8 + kWideTiles;
struct WideState {
    uint64_t* status = nullptr;    // 2 kWideBytes: the area of direct calls, that of captured ones
    uint32_t parity = 0;           // array of the next launch
    uint32_t old_words = 0;        // words of the other array to clear
    uint64_t issued = 0;           // tile counter values taken by earlier launches
    uint32_t spin_limit = 1u << 20;  // polls of an unpublished predecessor before giving up
    uint32_t withhold = 0;         // tests only: first tiles never publish (makes the waits run out)
    uint32_t round_tiles = kWideTiles;  // tiles per launch (at most kWideTiles)
};

// Batched addition on u64 or u32 limbs (op = ADD_PLAIN or ADD_SIX).
// Arguments are already validated; n > 0, limbs > 0.
// thread_bytes: operand bytes each thread owns (16, 32 or 64; raised where the
// instance would need a group of more than 1024 threads).  Instances wider
// than one group (limbs above kAddMaxLimbs64 u64 limbs) take the multi-block
// kernel, which needs `wide`.  link: the operands are host memory, read over the
// host link, and the results are not.
mi_status launch_add_u64(const uint64_t* a, const uint64_t* b, uint64_t* r, uint8_t* carry, uint32_t n,
                         uint32_t limbs, int op, uint32_t thread_bytes, cudaStream_t st,
                         WideState* wide = nullptr, bool link = false);
mi_status launch_add_u32(const uint32_t* a, const uint32_t* b, uint32_t* r, uint8_t* carry, uint32_t n,
                         uint32_t limbs, uint32_t thread_bytes, cudaStream_t st, WideState* wide = nullptr,
                         bool link = false);
// Size class of an addition of `bytes` per operand: ceil(log2(u64 limbs)).
uint32_t add_size_class(uint64_t bytes);

// The form of a batch of classical products: the Karatsuba kernel, or `rounds` of
// the lane groups (0: the power-of-two groups), and its modelled time.
struct ClassicForm {
    bool known = false, kara = false;
    uint32_t rounds = 0;
    double us = 0;
};
ClassicForm classic_form(uint32_t n, uint32_t n32, bool full, bool vec);

// Classical multiplication on u32 limb views (a u64 buffer with m limbs is a
// u32 buffer with 2m limbs).  full: r has 2*n32 limbs per instance, else n32.
// max_per_sm > 0 caps the full-product kernel's resident blocks per SM (by
// its shared-memory request); link: the operands are read over the host link.
// form: that of classic_form, where the caller has it (unless max_per_sm > 0).
mi_status launch_mul_classic(const uint32_t* a, const uint32_t* b, uint32_t* r, uint32_t n, uint32_t n32,
                             bool full, cudaStream_t st, uint32_t max_per_sm = 0, bool link = false,
                             ClassicForm form = ClassicForm());

// Dynamic shared memory that leaves room for at most max_per_sm blocks of a
// kernel per SM (at least `smem`, at most the per-block maximum; 0: `smem`).
mi_status capped_smem(size_t smem, uint32_t max_per_sm, size_t* out);

// Dynamic shared memory (at least *smem) for a launch of one-warp blocks that
// keeps the next launch's early blocks from crowding one scheduler.
mi_status balanced_smem(uint64_t blocks, uint32_t resident, size_t* smem);

// The same products, full or low half, on groups of any number of lanes
// (mul_flex.cu): flex_rounds says with how many rounds (1..3), or 0 where the
// power-of-two groups are faster or hold the product alone; *us is the
// modelled time.
uint32_t flex_rounds(uint32_t n, uint32_t n32, bool full, double* us);
mi_status launch_mul_flex(const uint32_t* a, const uint32_t* b, uint32_t* r, uint32_t n, uint32_t n32, bool full,
                          uint32_t rounds, cudaStream_t st, bool link = false, uint32_t max_per_sm = 0);

// Full products of 25..32 blocks of 8 u32 limbs with one Karatsuba level
// (mul_kara.cu), and the batches for which that is faster than the other forms'
// modelled *us, which then becomes its own.
bool kara_pays(uint32_t n, uint32_t n32, bool vec, double* us);
mi_status launch_mul_kara(const uint32_t* a, const uint32_t* b, uint32_t* r, uint32_t n, uint32_t n32,
                          cudaStream_t st);

// Low n32 limbs of a*b per instance (u32 limb views) on power-of-two groups, n32 > 128.
mi_status launch_mul_lo(const uint32_t* a, const uint32_t* b, uint32_t* r, uint32_t n, uint32_t n32, cudaStream_t st);

// ((a^2 + b)(b^2 + b) + ab) mod 2^(32*n32) per instance (u32 limb views).
mi_status launch_poly(const uint32_t* a, const uint32_t* b, uint32_t* r, uint32_t n, uint32_t n32, cudaStream_t st);

// GMP word-format conversions (convert.cu): fields of `words` words of `size`
// bytes (1, 2, 4, 8), order 1 / -1, endian 1 (big) / 0, -1 (little).
mi_status launch_import(const void* src, uint64_t* dst, uint32_t n, uint32_t words, uint32_t size, int order,
                        int endian, uint32_t limbs, cudaStream_t st);
mi_status launch_export(const uint64_t* src, void* dst, uint32_t n, uint32_t limbs, uint32_t words, uint32_t size,
                        int order, int endian, uint32_t* counts, cudaStream_t st);

// Ragged batches (ragged.cu): device scratch words for n_ops, the word that
// counts skipped ops, the one-time per-device setup (call outside stream
// capture) and the asynchronous launch sequence.
size_t ragged_scratch_words(uint32_t n_ops);
size_t ragged_invalid_word();
mi_status ragged_prepare();
mi_status ragged_launch(mi_ctx ctx, const mi_op* ops, uint32_t n_ops, const uint64_t* in, uint64_t* out,
                        uint8_t* carry, void* scratch, size_t scratch_bytes, uint32_t ntt_min, cudaStream_t st);

// Largest u32 limb count the classical kernel takes per instance.
constexpr uint32_t kMulMaxN32 = 4096;
// Largest u64 limb count the addition kernels take per instance (one group of
// at most 1024 threads, 4 limbs each).
constexpr uint32_t kAddMaxLimbs64 = 4096;
// Largest u64 limb count of one instance of the multi-block addition.
constexpr uint32_t kAddWideMaxLimbs64 = 1u << 26;

}  // namespace mi
