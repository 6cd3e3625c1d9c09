/*
 * The dynamic shared memory that a kernel may ask for is an attribute of the
 * function, common to all threads and streams that launch it.  A launcher
 * whose size depends on the call therefore sets the kernel's one upper bound,
 * never the size at hand: a smaller bound set by another thread between this
 * call and the launch would refuse it.
 */
#ifndef SXS_SMEM_CUH
#define SXS_SMEM_CUH

#define SXS_SMEM_MAX (227 * 1024)   /* of a block: static and dynamic */

/* before a launch with smem bytes of dynamic shared memory; bound the same in
 * every launch of the kernel.  (2 KB: what kernels have beside it) */
template <typename... P>
inline cudaError_t smem_bound(void (*kern)(P...), size_t smem, size_t bound)
{
	if (smem + 2048 <= 48 * 1024) return cudaSuccess;
	return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bound);
}

#endif
