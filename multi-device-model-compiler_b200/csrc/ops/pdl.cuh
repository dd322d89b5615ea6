// Programmatic dependent launch, device side (the host side is launch_chain in ops_common.h).
#pragma once

namespace mdc {

// Blocks until the grid this one was made dependent on has completed and its writes are
// visible; returns at once for a kernel launched without the attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the NEXT kernel of the chain be set up now: once every CTA of this grid has executed
// this (or exited), the dependent grid's CTAs are placed on whatever SM resources are free
// and run their prologue (barrier init, tensor-memory allocation, descriptor prefetch) up to
// their own pdl_wait(), which still holds them until this whole grid has finished and its
// writes are visible.  Called first thing in every chain kernel, so nothing of the next
// kernel's launch and set-up latency is left exposed between two kernels; a conversion launched
// `late` calls it after its own pdl_wait(), so that all it waited for is complete for the next kernel.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace mdc
