/*
 * jn_ortho.cuh — dot products of a vector with a Krylov basis, shared by the
 * single solve (jn_lanczos.cu) and the batched solve (jn_batch.cu).
 */
#ifndef JN_ORTHO_CUH
#define JN_ORTHO_CUH

#include <stdint.h>

#define ORTHO_WARPS 8           /* warps of the CTAs that call it */
#define ORTHO_GROUP 16          /* vectors a warp sums at once */
#define ORTHO_SPLIT_VECTORS 512 /* up to this many vectors the warps may share a group's elements */

#define ORTHO_THREADS (ORTHO_WARPS * 32)

/* Sum over the CTA's threads in a fixed order, on every thread.  One warp adds
 * all of it, 12 FP64 instructions: a shuffle tree in each of the eight warps
 * takes 40 and the eight warps' own sums of the results 56, at 19 cycles of
 * the SM's FP64 pipe each.  sh: ORTHO_THREADS doubles. */
__device__ __forceinline__ double ortho_cta_sum(double v, double *sh)
{
	__syncthreads();
	sh[threadIdx.x] = v;
	__syncthreads();
	if (threadIdx.x < 32) {
		double s = sh[threadIdx.x];
#pragma unroll
		for (int i = 1; i < ORTHO_WARPS; i++) s += sh[threadIdx.x + 32 * i];
		for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
		__syncwarp();
		if (threadIdx.x == 0) sh[0] = s;
	}
	__syncthreads();
	return sh[0];
}

/* sum of n partials from L2, by one warp (every lane gets it) */
__device__ __forceinline__ double ortho_partials(const double *part, int n)
{
	double s = 0.0;
	for (int b = threadIdx.x & 31; b < n; b += 32) s += __ldcg(part + b);
	for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
	return s;
}

/* the same on every thread of the CTA, added by its first warp (word: one
 * double that nothing else uses) */
__device__ __forceinline__ double ortho_cta_partials(const double *part, int n, double *word)
{
	if (threadIdx.x < 32) {
		const double s = ortho_partials(part, n);
		if (threadIdx.x == 0) *word = s;
	}
	__syncthreads();
	return *word;
}

/* How many ways the elements of a slice are shared out: the warps take
 * ng x split tasks in rounds, a task costs its multiply-adds and 16 adds of
 * the fold; the cheapest of 1, 2, 4, 8 keeps the eight warps busy whatever
 * the number of vectors (figures at kb_recur_dots). */
__device__ __forceinline__ int ortho_split(int nvec, int64_t elements)
{
	if (nvec > ORTHO_SPLIT_VECTORS) return 1;
	const int ng = (nvec + ORTHO_GROUP - 1) / ORTHO_GROUP, iters = (int)((elements + 31) / 32);
	int best = 1, cost = 0x7fffffff;
	for (int split = 1; split <= ORTHO_WARPS; split *= 2) {
		const int c = (ng * split + ORTHO_WARPS - 1) / ORTHO_WARPS * ((iters + split - 1) / split + 1);
		if (c < cost) { cost = c; best = split; }
	}
	return best;
}

/* out[j out_ld] = V_j . w over elements [i0, i1), j < nvec, by one CTA of
 * ORTHO_WARPS warps.  A warp takes 16 vectors, its lanes the elements
 * (coalesced rows of V), 16 sums in registers; the sums are then folded
 * across the lanes by halves, 16 adds for the 16 vectors where a butterfly
 * per vector takes 80 (GB300's FP64 pipe charges 64 cycles each).  ps: one
 * row of ORTHO_SPLIT_VECTORS sums for each share.  The order of every sum
 * depends on the sizes only.  w must be visible to the whole CTA. */
__device__ __forceinline__ void ortho_dots(const double *__restrict__ V, int64_t D, int nvec, const double *w, int64_t i0,
					   int64_t i1, double *__restrict__ out, int64_t out_ld,
					   double (*ps)[ORTHO_SPLIT_VECTORS])
{
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int ng = (nvec + ORTHO_GROUP - 1) / ORTHO_GROUP, split = ortho_split(nvec, i1 - i0);
	const int64_t sub = ((i1 - i0 + split - 1) / split + 31) & ~31ll;
	for (int task = warp; task < ng * split; task += ORTHO_WARPS) {
		const int g = task % ng, sp = task / ng, j0 = g * ORTHO_GROUP;
		const int64_t e0 = i0 + sp * sub, e1 = min(i1, e0 + sub);
		double acc[ORTHO_GROUP];
#pragma unroll
		for (int u = 0; u < ORTHO_GROUP; u++) acc[u] = 0.0;
		const double *v = V + (int64_t)j0 * D;
		if (j0 + ORTHO_GROUP <= nvec) {
			for (int64_t e = e0 + lane; e < e1; e += 32) {
				const double we = w[e];
#pragma unroll
				for (int u = 0; u < ORTHO_GROUP; u++) acc[u] = fma(v[u * D + e], we, acc[u]);
			}
		} else {
			for (int64_t e = e0 + lane; e < e1; e += 32) {
				const double we = w[e];
#pragma unroll
				for (int u = 0; u < ORTHO_GROUP; u++)
					if (j0 + u < nvec) acc[u] = fma(v[u * D + e], we, acc[u]);
			}
		}
#pragma unroll
		for (int h = ORTHO_GROUP / 2; h; h >>= 1) {
			const bool up = (lane & (2 * h)) != 0;
#pragma unroll
			for (int u = 0; u < h; u++) {
				const double give = up ? acc[u] : acc[u + h], keep = up ? acc[u + h] : acc[u];
				acc[u] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * h);
			}
		}
		acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
		const int j = j0 + (lane >> 1);
		if (!(lane & 1) && j < nvec) {
			if (split > 1) ps[sp][j] = acc[0];
			else out[j * out_ld] = acc[0];
		}
	}
	if (split > 1) {
		__syncthreads();
		for (int j = threadIdx.x; j < nvec; j += blockDim.x) {
			double s = ps[0][j];
			for (int sp = 1; sp < split; sp++) s += ps[sp][j];
			out[j * out_ld] = s;
		}
	}
}

#endif
