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
// ... of a kernel whose grid may be large: a CTA that has ended need not have asked, so only the last of them do, as many as are resident together
// (asking costs 0.5 ns a CTA; us, where all asked, none did and so: 26,584 CTAs 112, 95, 97; 3,479 of 128 threads 4.2, 2.9, 3.5.  With none asking, a norm, two products and a
// gated unit of 1,500 rows of 2,048 columns took 163 us for 158).
constexpr unsigned PDL_ASKING_CTAS = 8 * 148;
__device__ __forceinline__ void pdl_launch_next() {
  if (blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z) + PDL_ASKING_CTAS >= gridDim.x * gridDim.y * gridDim.z) pdl_launch_dependents();
}
// ... of a kernel that asks when its grid is small, for loops whose registers the place of a CTA in the grid would cost (window attention of 24 rows 42 us, with the line above 57)
__device__ __forceinline__ void pdl_launch_next_of_few() {
  if ((unsigned long long)gridDim.x * gridDim.y * gridDim.z <= 4 * 148) pdl_launch_dependents();
}
}  // namespace lp
#endif
