// places.h -- shared-memory requests that set how many blocks of a kernel an
// SM holds (host code without CUDA, so that it is checked without a GPU).
#pragma once

#include <cstddef>
#include <cstdint>

namespace mi {

// Shared memory of a device, in bytes: per SM, what each block reserves beside
// its own, and the most one block may ask for.
struct SmemLimits {
    size_t per_sm, reserved, per_block;
};

// The unit in which an SM allots shared memory to blocks.
constexpr size_t kSmemUnit = 128;

// Blocks of `smem` bytes that an SM's shared memory holds.
constexpr uint32_t smem_places(const SmemLimits& L, size_t smem) {
    return uint32_t(L.per_sm / ((smem + L.reserved + kSmemUnit - 1) / kSmemUnit * kSmemUnit));
}

// The request (at least `smem`, at most the per-block maximum) that leaves room
// for at most `places` blocks per SM -- one more would overflow it by 1 KB -- and
// for that many where `smem` itself allows them: 16 blocks of an even share of
// the SM and that 1 KB would be 15.
constexpr size_t smem_for_places(const SmemLimits& L, size_t smem, uint32_t places) {
    const size_t share = L.per_sm / places / kSmemUnit * kSmemUnit;
    size_t block = L.per_sm / (places + 1) + 1024;
    if (block > share) block = share;
    const size_t need = block > L.reserved ? block - L.reserved : 0;
    const size_t want = need > smem ? need : smem;
    return want < L.per_block || smem > L.per_block ? want : L.per_block;
}

}  // namespace mi
