// pearl_uniform.hpp — when the threads of a block may read the proposal that
// its leading thread left in shared memory (Uniform) for its uniform tiles.
//
// The walk has one block barrier per tile, the vote on whether all its cells
// equal the reference cell.  The leader writes the proposal in a tile of its own
// uniform cells, before that tile's vote, and no more once a vote was unanimous;
// the others read it only after such a vote, in which the leader took part.  So
// every write is before a barrier that every read is after, and each thread knows
// this from the votes alone.  (A flag in shared memory that the threads read
// after the vote is not enough: the leader may already be in the next tile.)
#pragma once

#ifdef __CUDACC__
#define PEARL_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define PEARL_HOST_DEVICE inline
#endif

namespace pearl_gpu {

// One thread's view of it.
struct FilledByVote {
    bool filled = false;  // the same in all threads between two votes
    // this thread's cells are uniform: it takes the proposal instead of forming one
    PEARL_HOST_DEVICE bool takes(bool same) const { return same && filled; }
    // it leaves the one that it formed
    PEARL_HOST_DEVICE bool fills(bool same, bool leader) const { return same && leader && !filled; }
    PEARL_HOST_DEVICE void vote(bool unanimous) { filled = filled || unanimous; }
};

}  // namespace pearl_gpu
