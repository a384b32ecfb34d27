// Runs of blocks whose codewords are packed together.
#pragma once
#include <cstdint>

namespace gb {

// The run of blocks from `first` whose codewords, each rounded up to whole words, fit in `limit`
// bytes together (one block at least): returns its end and their bytes. info4: 4 words per block,
// the codeword's bytes last. Packed offsets are 32 bits (compact.cuh), so limit is below 2^32.
inline uint32_t packedRun(const uint32_t* info4, uint32_t first, uint32_t n, uint64_t limit, uint64_t& bytes) {
    uint32_t end = first;
    bytes = 0;
    for (; end < n; ++end) {
        const uint64_t len = ((uint64_t)info4[4 * (uint64_t)end + 3] + 3u) & ~3ull;
        if (end > first && bytes + len > limit) break;
        bytes += len;
    }
    return end;
}

}  // namespace gb
