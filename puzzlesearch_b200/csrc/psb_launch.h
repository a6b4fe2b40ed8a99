// psb_launch.h -- what a failed launch means to its caller (host code only).
#pragma once

#include <driver_types.h>

namespace psb {

// Did the device have no room for the launch: for a cluster of its size
// (fewer SMs free of a cluster's kind than it has blocks, as on a partition of
// a GPU), its shared memory and registers, or the memory that loading the
// kernel takes?  Smaller launches may still run.  Any other error, a bad
// argument or an earlier kernel's fault, is no reason to try them.
constexpr bool launch_has_no_room(cudaError_t e) {
    return e == cudaErrorInvalidClusterSize || e == cudaErrorInvalidConfiguration ||
           e == cudaErrorLaunchOutOfResources || e == cudaErrorMemoryAllocation || e == cudaErrorNotSupported;
}

}  // namespace psb
