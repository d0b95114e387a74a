// blocks.h — how the analysis asks the driver for its arrays.
//
// cudaMalloc serves a block of up to 1 MB from 2-MB chunks that blocks share, a
// larger one by itself.  A chunk that is new and every larger block cost 0.34 ms,
// and 0.28 ms again when they go, whatever their size; a place in a chunk that is
// there costs about 1 us (measured, 0.1 to 16 MB, 1 to 13 blocks).  So arrays
// share a block where they are small (one call instead of several) and where three
// of them would overfill a chunk; between the two they stay apart and fill the
// chunks.  Analyses of 32-row blocks, us, all apart / three arrays in a block / as
// here: n = 60,000 302 / 264 / 264, 100,000 910 / 973 / 910, 130,000 950 / 1633 /
// 960, 200,000 2300 / 1650 / 1520, 400,000 4700 / 2200 / 2150.
#pragma once

namespace sptrsv {

// bytes of a small shared block: of the arrays with one entry a row, which come first, and of
// the others, which are to fit beside them
constexpr long long kRowShare = 768 * 1024, kOtherShare = 256 * 1024;
constexpr long long kThirdOfChunk = (2048 * 1024 - 64 * 1024) / 3;  // with room for the smallest beside three

inline long long block_part(long long ints) { return (ints + 63) / 64 * 64; }  // 256-byte aligned

// Do k arrays of so many ints share one block?  small: the bytes up to which they always do.
inline bool share_block(const long long* ints, int k, long long small)
{
    long long sum = 0, most = 0;
    for (int i = 0; i < k; i++) {
        const long long bytes = 4 * block_part(ints[i]);
        sum += bytes;
        most = bytes > most ? bytes : most;
    }
    return sum <= small || most > kThirdOfChunk;
}

}  // namespace sptrsv
