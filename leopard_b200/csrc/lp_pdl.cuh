// leopard_b200 — programmatic dependent launch, device side.
#pragma once
#ifdef __CUDACC__
namespace lp {
// No-ops when the kernel was launched without the attribute.  `wait` blocks until every prerequisite grid has completed and its memory
// is visible: it must precede the first dependent global access, and every kernel launched with the attribute has to call it, because a kernel
// that ends early would let the one after it start before the one before it has finished.  `launch_dependents` lets the next kernel's CTAs be
// scheduled as soon as this grid's resources free up.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
}  // namespace lp
#endif
