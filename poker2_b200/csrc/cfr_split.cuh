// Iteration passes of a solve as two kernels a pass, each parallel over the whole batch (cfr_split.cu).
#pragma once

#include "cfr.cuh"

namespace p2b {

constexpr int kSplitMaxDepth = 16;  // levels of a tree below its root; deeper trees stay in the general kernel

// Floats of work space the passes need: seven rows a node (the current policy, the policy as the other player sees it, the
// regret weights, the values of both players, the acting player's reach under the current and the old average
// policy), one record per internal node and the level bounds per subgame.
long long split_scratch_floats(int num_subgames, long long rows);
// True if the passes of such a batch can run here: the work space fits and no tree is too deep or too wide.
bool split_applies(const CfrParams& p, int max_children, long long scratch_floats);

// Passes pass_begin .. pass_end (iteration passes only) on the work space at p.scratch, which holds nothing else
// between the calls.  `down`: the call starts with the first half of pass_begin (beliefs, cross-hand work), for which it
// derives the work space anew unless it is `continued` from the start pass with its root advanced; otherwise with its
// second half.  `up`: the call ends with the second half of pass_end, otherwise with its first half.
int launch_split_passes(const CfrParams& p, int max_children, int pass_begin, int pass_end, bool down, bool up, bool continued,
                        cudaStream_t stream);
// The start pass, its first half (`down`) and/or its second (`up`); `advance`: pass 0 follows without the caller doing anything
// in between.  Leaves nothing for a `model_br` warm start, which needs the general kernel's start pass.
int launch_split_start(const CfrParams& p, int max_children, bool down, bool up, bool advance, cudaStream_t stream);
// The final pass, its halves as above, and the best responses from the state it left.
int launch_split_final(const CfrParams& p, int max_children, bool down, bool up, bool best_responses, cudaStream_t stream);

}  // namespace p2b
