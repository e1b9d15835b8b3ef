/*
 * jn_pdl.cuh — programmatic dependent launch between the kernels of one
 * product: a kernel whose stream predecessor is another kernel of the same
 * product is set up and made resident while that one still runs, and waits
 * on the device for its completion (and for all its writes) before it reads
 * anything that it wrote.
 */
#ifndef JN_PDL_CUH
#define JN_PDL_CUH

#include <cuda_runtime.h>

/* waits until the kernels this one depends on have completed and their
 * writes are visible; returns at once in a kernel launched without the attribute */
__device__ __forceinline__ void pdl_wait(void) { asm volatile("griddepcontrol.wait;" ::: "memory"); }

/* lets the next kernel of the product become resident (its own pdl_wait still
 * waits for this kernel's end) */
__device__ __forceinline__ void pdl_trigger(void) { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

/* a pointer to data of the preceding kernel, to be used after pdl_wait: no
 * load through it can be moved above the wait, also not one through the
 * read-only path */
template <typename T> __device__ __forceinline__ T *pdl_after(T *p)
{
	unsigned long long a = (unsigned long long)p;
	asm volatile("" : "+l"(a)::"memory");
	return (T *)a;
}

/* kernel<<<grid, block, smem, st>>>(args...), overlapped with the stream's
 * preceding kernel when `overlap` (the operation before it on the stream is
 * then a kernel of the same product) */
template <typename... P, typename... A>
static inline void pdl_launch(int overlap, void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t st, A... args)
{
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = grid;
	cfg.blockDim = dim3((unsigned int)block);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = st;
	cudaLaunchAttribute at = {};
	at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at.val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = &at;
	cfg.numAttrs = overlap ? 1 : 0;
	cudaLaunchKernelEx(&cfg, kernel, (P)args...);
}

#endif
