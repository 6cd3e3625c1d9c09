/*
 * Chains of launches that do not depend on one another (the translation's
 * one launch per class of n, each with a short last wave): every kernel of
 * the chain lets the next one start once all its own blocks have started,
 * and ends only after the one before it has, so that what follows the chain
 * in the stream finds all of it done.  Only the first waits for the stream's
 * earlier work, which the others read too.  Mixed translation: 1.96 -> 1.87
 * ms at L = 20, Q = 101 with 18,000 combos, 1.23 -> 1.14 with 8,500, 0.284 ->
 * 0.250 at L = 15, Q = 51, 10,000 poses; eight dimers' pieces of one batch
 * likewise.  The order of the classes makes no difference.
 */
#ifndef SXS_CHAIN_CUH
#define SXS_CHAIN_CUH

/* first and last statement of a kernel of a chain; nothing in other launches */
__device__ __forceinline__ void chain_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_end() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

/* launch behind the chain's last kernel (linked), or start a chain */
template <typename... P, typename... A>
inline cudaError_t chain_launch(void (*kern)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t s,
                                bool linked, A... args)
{
	cudaLaunchAttribute at[1];
	at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[0].val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t c = {};
	c.gridDim = dim3(grid);
	c.blockDim = dim3(threads);
	c.dynamicSmemBytes = smem;
	c.stream = s;
	c.attrs = at;
	c.numAttrs = linked ? 1 : 0;
	return cudaLaunchKernelEx(&c, kern, static_cast<P>(args)...);
}

#endif
