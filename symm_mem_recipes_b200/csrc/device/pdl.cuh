// Programmatic dependent launch (griddepcontrol).  A kernel launched with
// cudaLaunchAttributeProgrammaticStreamSerialization may start while its predecessor in the stream still
// runs; `pdl_wait` returns once every earlier kernel has finished and its writes are visible, and
// `pdl_launch_dependents` lets the successor start early.  Both do nothing in an ordinary launch.
//
// Ordering over a chain: a kernel that calls pdl_wait before its first dependent access and before its
// first store finishes after everything that precedes it, so one pdl_wait covers all predecessors as long
// as every kernel of the chain calls it.  What a kernel reads BEFORE pdl_wait must not have been written by
// any kernel since the last ordinary (fully ordered) launch.
#pragma once

namespace smr {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace smr
