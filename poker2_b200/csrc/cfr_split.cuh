// Iteration passes of a solve as two kernels a pass, each parallel over the whole batch (cfr_split.cu).
#pragma once

#include "cfr.cuh"

namespace p2b {

constexpr int kSplitMaxDepth = 16;  // levels of a tree below its root; deeper trees stay in the general kernel

// Floats of work space the passes need: per row the current policy, the opponent-conditioned policy, the regret
// weights and the values of both players, then one record per internal node and the level bounds per subgame.
long long split_scratch_floats(int num_subgames, long long rows);
// True if the passes of such a batch can run here: the work space fits and no tree is too deep or too wide.
bool split_applies(const CfrParams& p, int max_children, long long scratch_floats);

// Passes pass_begin .. pass_end (iteration passes only) on the work space at p.scratch, which holds nothing else
// between the calls.  `down`: the call starts with the first half of pass_begin (beliefs, cross-hand work), for
// which it derives the work space anew; otherwise with its second half.  `up`: the call ends with the second half
// of pass_end, otherwise with its first half.
int launch_split_passes(const CfrParams& p, int max_children, int pass_begin, int pass_end, bool down, bool up,
                        cudaStream_t stream);

}  // namespace p2b
