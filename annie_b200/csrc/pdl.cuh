// Programmatic dependent launch: the kernels of a squaring are launched so that
// the next one on the stream may be scheduled while the current one is still
// running.  Until griddep_wait() a kernel reads only what no earlier work of
// the stream writes (twiddles, images of N and N^-1, its launch parameters; the
// passes also the per-slot control words, uploaded before a graph launch) and
// writes only shared memory; griddep_wait() returns once the previous kernel of
// the stream has completed and its writes are visible.
//
// The passes do not call griddep_launch(): their successor is scheduled as
// their CTAs exit.  Triggered earlier it holds SM resources that the running
// pass and the other stream need (33.2 M bits: 221.7 us per squaring right
// after griddep_wait, 233.3 before the final stores, 210.1 without; without
// programmatic launch 218.9).  A resident run calls it in its last step, for
// the next run's tables.
#pragma once

namespace ab
{

__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

} // namespace ab
