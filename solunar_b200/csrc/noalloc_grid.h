// noalloc_grid.h -- the grid of the cell sort without allocation (host arithmetic only).
#pragma once

#include <algorithm>
#include <cstdint>

namespace slf {

constexpr uint32_t kNoAllocThreads = 512;
constexpr uint32_t kNoAllocItems = 4;     // particles a thread keeps in registers from pass to pass
constexpr uint32_t kNoAllocBlocks = 256;  // most blocks of the sort's grid

struct NoAllocGrid {
    uint32_t blocks;
    bool held;  // the threads' registers hold every particle; else the threads stride over them
};

// The grid for n >= 1 particles where `room` blocks run at once (the blocks wait for one another).  A
// block for each 256 particles while there is room, so that small calls spread over the SMs; with a
// block on each of 148 SMs the registers hold all that the scratch array does.
inline NoAllocGrid noalloc_grid(uint32_t n, uint32_t room) {
    const uint32_t most = std::max(1u, std::min(room, kNoAllocBlocks));
    const uint32_t blocks = std::min(most, (n + 255u) / 256u);
    return NoAllocGrid{blocks, uint64_t(blocks) * kNoAllocThreads * kNoAllocItems >= n};
}

}  // namespace slf
