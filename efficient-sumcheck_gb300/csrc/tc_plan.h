// tc_plan.h -- how the tensor-core start of many proofs shares a launch's
// blocks, and the words its blocks' sums take.  Plain C++, compiled and tested
// without a GPU.
#pragma once
#include <cstddef>
#include <cstdint>

namespace effsc {

// Tiles a block takes where `total` tiles share a launch: about 5/2 blocks per
// SM, at least 16 tiles each and at most what a block's accumulators hold.
constexpr uint64_t tc_tiles_per_block(uint64_t total, uint64_t sms, uint64_t max_tiles) {
    const uint64_t blocks = sms * 5 / 2, t = (total + blocks - 1) / blocks;
    return t < 16 ? 16 : t > max_tiles ? max_tiles : t;
}
// The most blocks of a launch over at most `total` tiles of at most n proofs
// (each proof's last block may be short).
constexpr uint64_t tc_blocks_most(uint64_t total, uint64_t n, uint64_t sms, uint64_t max_tiles) {
    const uint64_t blocks = sms * 5 / 2, full = total / max_tiles;
    return (full > blocks ? full : blocks) + n;
}

// Words of a prover's block sums, `grid` being the largest grid of a round
// kernel (eight blocks per SM; 12 words each).  InnerProduct: 256 for each SM's
// block of k_ip_gram; Coefficient: 108 for each of k_c3_gram.
constexpr size_t partial_words(bool inner_product, bool coefficient, size_t grid) {
    return grid * (inner_product ? 32 : coefficient ? 14 : 12);
}

}  // namespace effsc
