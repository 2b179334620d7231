// mma_layout.h -- word offsets of one hash's tables (mma_tables.h, hash_mma.cuh).
#pragma once

namespace zk {

enum : unsigned {
    MMA_KB = 2 * 32 * 4,              // words of one k-block of one output group: 2 pairs of column tiles x 32 threads x 4
    MMA_GROUP = 4 * 4 * 4,            // starting sums of one output group: 4 byte pairs x 4 threads x 4
    MMA_FULL = 0,                     // full-round matrix [group 3], one k-block per pair of columns
    MMA_Y = MMA_FULL + 3 * MMA_KB,    // lane 0 before partial rounds 4 b .. 4 b + 3, b < 6 [k-block 3 + b]
    MMA_W = MMA_Y + 33 * MMA_KB,      // lanes after the partial rounds [group 3][k-block 9]
    MMA_CONST = MMA_W + 27 * MMA_KB,  // starting sums of 9 layers, 3 groups each
    MMA_YCONST = MMA_CONST + 27 * MMA_GROUP,  // of the 6 blocks of partial rounds
    MMA_WORDS = MMA_YCONST + 6 * MMA_GROUP,
    // Monolith: its matrix and the starting sums of its 7 layers
    MMA_MONO_CONST = MMA_FULL + 3 * MMA_KB,
    MMA_MONO_WORDS = MMA_MONO_CONST + 21 * MMA_GROUP
};

}  // namespace zk
