// Index arithmetic of the cell sort's bins and of its scan. Each slab of a cell
// has two bins, its free and its fixed particles: at the limit of cells with the
// finest split there are 2^31, so bins are counted in unsigned ints (their sums,
// particle counts below 2^26, stay ints).
#pragma once

#include "psph_common.cuh"

namespace psph {

constexpr long long kMaxCells = 1LL << 28;  // of all instances' grids together
constexpr int kMaxXsub = 4;                 // x-slabs per cell at most

// The bin of the free particles of a cell's slab; the fixed ones' is the next.
PSPH_HD unsigned sort_bin(int cell, int xsub, int slab) { return 2u * ((unsigned)cell * (unsigned)xsub + (unsigned)slab); }

// The scan: a thread takes kScanPer consecutive entries, a block of 1,024 threads kScanBlock.
constexpr unsigned kScanPer = 8, kScanBlock = 1024 * kScanPer;
PSPH_HD unsigned scan_first(unsigned block, unsigned thread) { return block * kScanBlock + thread * kScanPer; }
PSPH_HD bool scan_full(unsigned first, unsigned per, unsigned len) { return first + per <= len; }
PSPH_HD unsigned scan_blocks_for(unsigned len) { return len > kScanBlock ? (len - 1) / kScanBlock + 1 : 1; }

// The largest index that any of it forms: the end of the last scan block.
static_assert(2 * kMaxCells * kMaxXsub + 2 + kScanBlock < 1LL << 32, "bin indices fit 32 bits");

}  // namespace psph
