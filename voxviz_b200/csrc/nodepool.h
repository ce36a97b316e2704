// nodepool.h - a node pool as the kernels take it.
#pragma once

#include <cuda_runtime.h>

namespace vv {

// A node pool on the device: the words, block-linear (8 nodes of a 2x2x2 cell
// contiguous), and the same nodes as the unit box's walk reads them
// (walknode.h).  The records take as much memory again and are left out (null)
// where it is not to be had: the draws then walk the words, as other boxes do.
struct NodePool {
    uint2* words;
    uint2* walk;
    int dim[3];
};

}  // namespace vv
