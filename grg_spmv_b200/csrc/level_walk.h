// The row walk of default-mode level launches (level_walk.cu) and of mixed storage (level_walk_mixed.cu).
#ifndef GRG_B200_LEVEL_WALK_H
#define GRG_B200_LEVEL_WALK_H

#include "level_common.cuh"

// Whether level_walk serves this launch: padded lists, no error word, no init inside the
// traversal, 32-bit leading dimensions.
bool walk_serves(const LevelArgs& la, int init_mode, bool exact);

// Launches one level: its very long rows (if any) over clusters, then every other row.
// `long_counts[i]` rows of the level hold more than GRG_B200_LONG_ROW << i entries and are
// listed first in heavy_rows; nullptr when the level does not say.
template <typename T>
int launch_walk(const LevelArgs& la, int64_t num_entries, const int64_t* long_counts, bool pdl, cudaStream_t s);

// The same over mixed storage, for every launch of that dtype (any init, with or without an error
// word).
int launch_walk_mixed(const LevelArgs& la, int init_mode, int64_t num_entries, const int64_t* long_counts, bool pdl, cudaStream_t s);

#endif  // GRG_B200_LEVEL_WALK_H
