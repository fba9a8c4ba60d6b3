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
// ... of a kernel whose grid may be large.  Asking costs 0.5 ns a CTA (us, with it and without: 26,584 CTAs 112, 95; 3,479 of 128 threads 4.2, 2.9), and what comes after many CTAs
// has no launch to hide: up to four CTAs an SM ask.
constexpr unsigned PDL_ASKING_CTAS = 4 * 148;
__device__ __forceinline__ void pdl_launch_next() {
  if ((unsigned long long)gridDim.x * gridDim.y * gridDim.z <= PDL_ASKING_CTAS) pdl_launch_dependents();
}
}  // namespace lp
#endif
