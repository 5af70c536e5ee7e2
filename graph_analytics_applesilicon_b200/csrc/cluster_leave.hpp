// cluster_leave.hpp -- how the blocks of a cluster that use one another's shared
// memory end together when a wait of one of them has run out.
//
// A cluster barrier only counts arrivals: the barrier with which a block that
// gave up would leave also releases blocks that meet in the middle of a level,
// and those would then use the shared memory of a block that is gone.  So a
// block that gives up first raises a flag in every block, and a block that
// comes out of a barrier looks at its own flag before it touches another's
// memory: all that was raised before the last arrival is seen by every block.
// A block leaves only after a barrier that it entered with its own mind made up,
// so nobody that has not seen the flag is still to come.  (A barrier waits for
// the threads that have not exited, so blocks may leave one barrier apart.)
//
// C is the cluster as one block sees it:
//   sync()    the cluster barrier: what was written before it is seen after it
//   raise()   sets the flag of every block
//   raised()  this block's flag, the same for all its threads
//   settle()  waits until what the others sent before the barrier has arrived
#pragma once

#ifdef __CUDACC__
#define GB_CLUSTER_FN __device__ __forceinline__
#else
#define GB_CLUSTER_FN inline
#endif

namespace gb {

// A barrier within the traversal; false: a block gave up, go to clusterLeave.
template <class C>
GB_CLUSTER_FN bool clusterMeet(C& c) {
    c.sync();
    return !c.raised();
}

// The last barrier; true when any block gave up.
template <class C>
GB_CLUSTER_FN bool clusterLeave(C& c, bool gaveUp) {
    if (gaveUp) c.raise();
    c.sync();
    const bool raised = c.raised();
    if (raised) c.settle();
    return raised;
}

}  // namespace gb
