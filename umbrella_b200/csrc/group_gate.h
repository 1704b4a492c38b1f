// The steps that the warps of a group take together, each behind a barrier that says whether all of them go on.
//
// Every warp of the group comes to the same barriers in the same order until one of them fails, which all of its warps learn from the barrier itself.
// Behind that none of them may come to another: a warp that gave up on a wait has left the loop that the others are still in, and meets them at whichever
// barrier is theirs next, so that they have one barrier more in front of them than it has, which it would never join.
#pragma once
#ifdef __CUDACC__
#define UMB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define UMB_HOST_DEVICE inline
#endif

namespace umb {

struct GroupGate {
    bool open = true;
    // all_of(ok): the barrier, true where it was true of every warp
    template <typename F> UMB_HOST_DEVICE bool pass(bool ok, F&& all_of) {
        if (open) open = all_of(ok);
        return open;
    }
};

}  // namespace umb
