/*
 * jn_lanczos.cu — the Lanczos eigensolver of Bacchus on the GPU, in FP64.
 *
 * Reference: src/Bacchus/lanczos/lanczos.c.  One iteration
 * (lanczos_iteration, :74-153) is
 *     w = H v_k;  alpha_k = <v_k|w>;  w -= alpha_k v_k + beta_{k-1} v_{k-1};
 *     beta_k = |w|;  v_{k+1} = w / beta_k
 * followed by reorthogonalisation (orthogonalize_krylow_basis, :155-169) and
 * the eigen-decomposition of the tridiagonal matrix (diagonalize, :171-253;
 * dsteqr in src/Bacchus/diagonalization/diagonalization.c:16-68).
 *
 * Two modes:
 *   JN_LANCZOS_REFERENCE  the reference's choices: start vector e_0
 *                         (lanczos.c:60-72), reorthogonalisation of
 *                         v_{k+1} against v_0..v_{k-3} only, without
 *                         renormalising (lanczos.c:155-169,
 *                         vector.c:461-476), convergence when the target
 *                         (ground-state) Ritz value moves by less than the
 *                         tolerance (lanczos.c:199-235).
 *   JN_LANCZOS_FULL       full reorthogonalisation (classical Gram-Schmidt
 *                         after the recurrence, again where it cancels) and
 *                         convergence when the error
 *                         bound min(r, r^2/gap) of each of the lowest `nev`
 *                         Ritz values is below the tolerance, r being the
 *                         residual norm beta_k |s_{k,i}|.
 *
 * The Krylov basis stays in HBM.  Every reduction is a two-pass fixed-order
 * reduction, so two runs give bit-identical alpha/beta.  In full mode one
 * cooperative kernel (k_orthonormalize) takes w = H v_k to v_{k+1}.  The
 * convergence check (k_tri_check: eigenvalues of T by multisection and their
 * eigenvectors, jn_tridiag.cuh) runs on its own stream beside the next
 * steps' products: the host enqueues step k + 1 (and k + 2, where steps are
 * short), then reads the check of step k.  The final Ritz vectors are refined by FP64 products (Rayleigh
 * quotient and residual norm).
 */
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/stat.h>
#include <sys/types.h>
#include <time.h>

#include <vector>

#include <cooperative_groups.h>

#include "jn_internal.h"
#include "jn_ortho.cuh"
#include "jn_tridiag.cuh"

#define RED_BLOCKS 304      /* 2 x 152 SMs */
#define RED_THREADS 256

/* Checks in flight at most, one more than the steps by which the host reads
 * them behind: it enqueues steps k + 1 and k + 2, then reads check k.  A check
 * takes about as long as a small basis's product (83 against 96 us for 4He
 * Nmax 6), and one step behind left the host no time to enqueue the next
 * before the device ran out: 165 steps with a check each 23.1 -> 21.1 ms, where
 * a check every tenth takes 20.7.  The steps behind are run for nothing once a
 * solve has converged, so where a step takes twice a check and more, from
 * about 1.5e8 multiply-adds a product on (300 us), it is one: 6Li Nmax 6,
 * 3.5 ms a step, ends a step sooner; 6Li Nmax 4 with 3NF (5.6e7, 190 us a
 * step) stays at two. */
#define CHECKS 3
#define LONG_STEP 1.5e8

struct jn_lanczos_state {
	int64_t D;
	int mmax;               /* allocated Krylov dimension (vectors mmax+1) */
	int k;                  /* Lanczos steps done */
	int nev;
	double *d_V;            /* (mmax+1) x D */
	double *d_w;
	double *d_alpha, *d_beta;
	double *d_part;         /* RED_BLOCKS x (mmax+2) partials */
	double *d_h;            /* mmax+2 coefficients */
	double *d_scalar;       /* 4 scalars */
	double *d_theta;        /* Ritz values (ascending), mmax */
	double *d_Z;            /* nev_cap x mmax tridiagonal eigenvectors */
	double *d_work;         /* scratch of k_tri_check above JN_TRI_SMEM_ROWS rows, else NULL */
	unsigned int *d_done;   /* finished CTAs of k_tri_check */
	double *d_pack;         /* a check's results: Ritz values, bottom components, beta */
	double *d_ritz;         /* nev x D Ritz vectors */
	double *d_hritz;        /* and H times them */
	double *d_rr;           /* Rayleigh quotients, residual norms (2 nev_cap) */
	double *h_pack[CHECKS]; /* pinned copies of d_pack: a check is read while the next ones run */
	cudaStream_t check;     /* the checks' stream */
	cudaEvent_t stepped, begun, checked[CHECKS];
	int guesses;            /* entries of d_theta that hold eigenvalues of the last T of this solve */
	int nev_cap;
	int have_ritz;
	double *h_rq, *h_res;   /* refined Rayleigh quotients and residual norms */
};

void jn_lanczos_release(jn_ctx *c)
{
	struct jn_lanczos_state *s = c->lz;
	if (!s) return;
	cudaFree(s->d_V); cudaFree(s->d_w); cudaFree(s->d_alpha); cudaFree(s->d_beta); cudaFree(s->d_part);
	cudaFree(s->d_h); cudaFree(s->d_scalar); cudaFree(s->d_theta); cudaFree(s->d_Z); cudaFree(s->d_ritz);
	cudaFree(s->d_work); cudaFree(s->d_done); cudaFree(s->d_pack); cudaFree(s->d_hritz); cudaFree(s->d_rr);
	for (int i = 0; i < CHECKS; i++) {
		if (s->h_pack[i]) cudaFreeHost(s->h_pack[i]);
		if (s->checked[i]) cudaEventDestroy(s->checked[i]);
	}
	if (s->stepped) cudaEventDestroy(s->stepped);
	if (s->begun) cudaEventDestroy(s->begun);
	if (s->check) cudaStreamDestroy(s->check);
	free(s->h_rq); free(s->h_res);
	free(s);
	c->lz = NULL;
}

/* ------------------------------------------------------------------ */
/* BLAS-1/2 kernels with fixed reduction order                         */
/* ------------------------------------------------------------------ */

/* part[b*ncol + j] = sum over this block's slice of V[j] . w, j < nvec:
 * warp j % (warps) owns vector j and reduces it with shuffles in a fixed
 * order, so the vectors run side by side with no CTA-wide barrier */
__global__ void __launch_bounds__(RED_THREADS) k_gemv_t(const double *__restrict__ V, int64_t D, int nvec,
							 const double *__restrict__ w, double *__restrict__ part, int ncol)
{
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
	const int64_t chunk = (D + gridDim.x - 1) / gridDim.x;
	const int64_t i0 = (int64_t)blockIdx.x * chunk, i1 = min(D, i0 + chunk);
	for (int j = warp; j < nvec; j += nwarps) {
		const double *v = V + (int64_t)j * D;
		double s = 0.0;
		for (int64_t i = i0 + lane; i < i1; i += 32) s = fma(v[i], w[i], s);
		for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
		if (lane == 0) part[(int64_t)blockIdx.x * ncol + j] = s;
	}
}

/* out[j] = sum_b part[b*ncol + j], one warp per j: lane l sums blocks
 * l, l + 32, ... in order, then the lanes' sums are added by a fixed
 * shuffle tree (the partials' loads are in flight together) */
__global__ void k_finish(const double *__restrict__ part, int nblk, int ncol, int nvec, double *__restrict__ out)
{
	const int j = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
	if (j >= nvec) return;          /* warp-uniform */
	double s = 0.0;
	for (int b = lane; b < nblk; b += 32) s += part[(int64_t)b * ncol + j];
	for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
	if (lane == 0) out[j] = s;
}

/* w -= a*v + b*u (reads a = *pa, b = *pb on the device; u may be NULL) */
__global__ void k_three_term(double *__restrict__ w, const double *__restrict__ v, const double *__restrict__ u,
			     const double *pa, const double *pb, int64_t D)
{
	const double a = *pa, b = pb ? *pb : 0.0;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D; i += (int64_t)gridDim.x * blockDim.x) {
		double r = w[i] - a * v[i];
		if (u) r -= b * u[i];
		w[i] = r;
	}
}

/* dst = src / sqrt(*nrm2) ; beta_out = sqrt(*nrm2) */
__global__ void k_normalize(double *__restrict__ dst, const double *__restrict__ src, const double *nrm2,
			    double *beta_out, int64_t D)
{
	const double b = sqrt(*nrm2);
	if (blockIdx.x == 0 && threadIdx.x == 0 && beta_out) *beta_out = b;
	const double inv = 1.0 / b;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D; i += (int64_t)gridDim.x * blockDim.x)
		dst[i] = src[i] * inv;
}

__global__ void k_axpy_neg(double *__restrict__ y, const double *__restrict__ x, const double *pa, int64_t D)
{
	const double a = *pa;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D; i += (int64_t)gridDim.x * blockDim.x)
		y[i] -= a * x[i];
}

/* ------------------------------------------------------------------ */
/* full reorthogonalisation                                            */
/* ------------------------------------------------------------------ */
#define ORTHO_H 1024            /* coefficients staged at a time in the subtraction */

/* h[j] = sum over the CTAs' partials of vector j, one warp of the grid per j */
__device__ __forceinline__ void ortho_reduce(const double *part, int nvec, double *h)
{
	const int lane = threadIdx.x & 31;
	for (int j = blockIdx.x * ORTHO_WARPS + (threadIdx.x >> 5); j < nvec; j += gridDim.x * ORTHO_WARPS) {
		const double s = ortho_partials(part + (int64_t)j * gridDim.x, gridDim.x);
		if (lane == 0) h[j] = s;
	}
}

/* w -= sum_j V_j h_j over [i0, i1): a warp's lanes are 32 elements; the warps
 * share the vectors where the slice has fewer than 8 x 32 elements */
__device__ __forceinline__ void ortho_subtract(const double *__restrict__ V, int64_t D, int nvec, const double *h, double *w,
					       int64_t i0, int64_t i1, double *hs, double (*ps)[32])
{
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int64_t tiles = (i1 - i0 + 31) / 32;
	const int split = tiles < ORTHO_WARPS ? ORTHO_WARPS / (int)max(tiles, (int64_t)1) : 1;
	for (int c0 = 0; c0 < nvec; c0 += ORTHO_H) {
		const int nc = min(ORTHO_H, nvec - c0);
		__syncthreads();
		for (int j = threadIdx.x; j < nc; j += blockDim.x) hs[j] = __ldcg(h + c0 + j);
		__syncthreads();
		const int sub = (nc + split - 1) / split;
		for (int64_t task = warp; task < tiles * split; task += ORTHO_WARPS) {
			const int64_t tile = task % tiles;
			const int sp = (int)(task / tiles), ja = sp * sub, jb = min(nc, ja + sub);
			const int64_t e = i0 + tile * 32 + lane;
			double s = 0.0;
			if (e < i1) {
				const double *v = V + (int64_t)(c0 + ja) * D + e;
#pragma unroll 8
				for (int j = ja; j < jb; j++, v += D) s = fma(*v, hs[j], s);
			}
			if (split > 1) ps[task][lane] = s;
			else if (e < i1) w[e] -= s;
		}
		if (split > 1) {
			__syncthreads();
			for (int64_t task = warp; task < tiles; task += ORTHO_WARPS) {
				const int64_t e = i0 + task * 32 + lane;
				double s = ps[task][lane];
				for (int sp = 1; sp < split; sp++) s += ps[task + sp * tiles][lane];
				if (e < i1) w[e] -= s;
			}
		}
	}
	__syncthreads();
}

/* One Lanczos step's vector work: from w = H v_k, with v_0 .. v_k the
 * orthonormal basis,
 *     alpha_k = <v_k|w>;  w -= alpha_k v_k + beta_{k-1} v_{k-1};
 *     w -= V (V^T w);  beta_k = |w|;  v_{k+1} = w / beta_k.
 * After the recurrence w is orthogonal to the basis but for rounding, so one
 * Gram-Schmidt pass restores full orthogonality (max |V^T V - 1| 7e-16 over
 * 200 steps, as with two passes) unless the pass took most of w away: |w|
 * below 0.7 of what it was, which happens only when the Krylov space closes;
 * then there is a second pass.  A cooperative launch, one CTA an SM, a slice
 * of the vectors to each; the CTAs meet at four grid-wide barriers.  Bound by
 * the barriers (1.1 us each) and the FP64 pipe (2 multiply-adds per element
 * and vector): 31 us a step at D = 7 916, k = 25 to 125.  As thirteen
 * kernels in a row, with two passes, the same work took 130 us at k = 45,
 * most of it launches and a subtraction on 31 CTAs; with two passes in one
 * launch, 34 us. */
__global__ void __launch_bounds__(ORTHO_WARPS * 32)
	k_orthonormalize(double *__restrict__ V, int64_t D, int64_t chunk, int k, double *w, double *part, double *h,
			 double *__restrict__ alpha, double *__restrict__ beta)
{
	__shared__ double ps[ORTHO_WARPS][ORTHO_SPLIT_VECTORS];
	__shared__ double pt[ORTHO_WARPS][32];
	__shared__ double hs[ORTHO_H];
	__shared__ double sh[ORTHO_THREADS], word[4];
	namespace cg = cooperative_groups;
	cg::grid_group grid = cg::this_grid();
	const int nvec = k + 1;
	const int64_t i0 = (int64_t)blockIdx.x * chunk, i1 = min(D, i0 + chunk);
	/* partial sums of alpha and, later, of |w|^2 after a pass; of |w|^2 before it */
	double *pa = part + (int64_t)nvec * gridDim.x, *pb = pa + gridDim.x;
	const double *vk = V + (int64_t)k * D, *u = k > 0 ? vk - D : vk;
	double s = 0.0;
	for (int64_t e = i0 + threadIdx.x; e < i1; e += blockDim.x) s = fma(vk[e], w[e], s);
	s = ortho_cta_sum(s, sh);
	if (threadIdx.x == 0) pa[blockIdx.x] = s;
	grid.sync();
	const double a = ortho_cta_partials(pa, gridDim.x, word), b0 = k > 0 ? beta[k - 1] : 0.0;
	if (blockIdx.x == 0 && threadIdx.x == 0) alpha[k] = a;
	s = 0.0;
	for (int64_t e = i0 + threadIdx.x; e < i1; e += blockDim.x) {
		double r = w[e] - a * vk[e];
		if (k > 0) r -= b0 * u[e];
		w[e] = r;
		s = fma(r, r, s);
	}
	s = ortho_cta_sum(s, sh);       /* its barriers also publish w to the CTA */
	if (threadIdx.x == 0) pb[blockIdx.x] = s;
	double n2, n0 = 0.0;
	for (int pass = 0;; pass++) {
		ortho_dots(V, D, nvec, w, i0, i1, part + blockIdx.x, gridDim.x, ps);
		grid.sync();
		ortho_reduce(part, nvec, h);
		if (pass == 0) n0 = ortho_cta_partials(pb, gridDim.x, word + 2);
		grid.sync();
		ortho_subtract(V, D, nvec, h, w, i0, i1, hs, pt);
		s = 0.0;
		for (int64_t e = i0 + threadIdx.x; e < i1; e += blockDim.x) s = fma(w[e], w[e], s);
		s = ortho_cta_sum(s, sh);
		if (threadIdx.x == 0) pa[blockIdx.x] = s;
		grid.sync();
		n2 = ortho_cta_partials(pa, gridDim.x, word + 1);
		/* every CTA decides alike */
		if (pass == 1 || n2 >= 0.49 * n0) break;
		__syncthreads();
	}
	if (threadIdx.x == 0) {
		const double b = sqrt(n2);
		word[3] = b > 0.0 ? 1.0 / b : 0.0;
		if (blockIdx.x == 0) beta[k] = b;
	}
	__syncthreads();
	const double inv = word[3];
	double *v = V + (int64_t)(k + 1) * D;
	for (int64_t e = i0 + threadIdx.x; e < i1; e += blockDim.x) v[e] = w[e] * inv;
}

/* X[i] = sum_j Z[i][j] V[j], i < want: an element of each V_j is read once
 * for 8 Ritz vectors */
#define RITZ_ROWS 8
#define RITZ_J 256
__global__ void __launch_bounds__(128) k_ritz_vectors(const double *__restrict__ V, int64_t D, int n, const double *__restrict__ Z,
						       int ldz, int want, double *__restrict__ X)
{
	__shared__ double zs[RITZ_ROWS][RITZ_J];
	const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	const int i0 = blockIdx.y * RITZ_ROWS, ni = min(RITZ_ROWS, want - i0);
	double acc[RITZ_ROWS];
#pragma unroll
	for (int i = 0; i < RITZ_ROWS; i++) acc[i] = 0.0;
	for (int j0 = 0; j0 < n; j0 += RITZ_J) {
		const int nj = min(RITZ_J, n - j0);
		__syncthreads();
		for (int t = threadIdx.x; t < RITZ_ROWS * nj; t += blockDim.x)
			zs[t / nj][t % nj] = t / nj < ni ? Z[(int64_t)(i0 + t / nj) * ldz + j0 + t % nj] : 0.0;
		__syncthreads();
		if (e < D) {
			const double *v = V + (int64_t)j0 * D + e;
#pragma unroll 4
			for (int j = 0; j < nj; j++, v += D) {
				const double x = *v;
#pragma unroll
				for (int i = 0; i < RITZ_ROWS; i++) acc[i] = fma(x, zs[i][j], acc[i]);
			}
		}
	}
	if (e < D)
#pragma unroll
		for (int i = 0; i < RITZ_ROWS; i++)
			if (i < ni) X[(int64_t)(i0 + i) * D + e] = acc[i];
}

/* CTA i: rr[i] = x.w / x.x (the Rayleigh quotient of x = X_i, w = H x), rr[n + i] = |w - rr[i] x| / |x| */
__global__ void __launch_bounds__(512) k_rayleigh(const double *__restrict__ X, const double *__restrict__ HX, int64_t D, int n,
						   double *__restrict__ rr)
{
	__shared__ double sh[512];
	const double *x = X + (int64_t)blockIdx.x * D, *w = HX + (int64_t)blockIdx.x * D;
	double xw = 0.0, xx = 0.0;
	for (int64_t e = threadIdx.x; e < D; e += blockDim.x) {
		xw = fma(x[e], w[e], xw);
		xx = fma(x[e], x[e], xx);
	}
	xw = jn_block_sum(xw, sh);
	xx = jn_block_sum(xx, sh);
	const double q = xw / xx;
	double r2 = 0.0;
	for (int64_t e = threadIdx.x; e < D; e += blockDim.x) {
		const double r = w[e] - q * x[e];
		r2 = fma(r, r, r2);
	}
	r2 = jn_block_sum(r2, sh);
	if (threadIdx.x == 0) {
		rr[blockIdx.x] = q;
		rr[n + blockIdx.x] = sqrt(r2 / xx);
	}
}

/* ------------------------------------------------------------------ */
/* tridiagonal eigenproblem                                            */
/* ------------------------------------------------------------------ */
#define TRI_THREADS 128
#define TRI_WAVE 256            /* eigenvalues at a time where the scratch is in global memory */

/* The `want` lowest eigenvalues of T_n, CTA i the (first + i)-th, and the eigenvectors
 * of the lowest `nvec` (rows of Z).  The CTA that finishes last makes the
 * vectors orthogonal among themselves and packs the results for one copy to
 * the host: theta (want), the vectors' bottom components (nvec), beta_{n-1}.
 * The first `guesses` entries of theta hold an earlier check's eigenvalues.
 * exact: to the last bit of each eigenvalue.
 * Scratch: shared memory, or `work` (JN_TRI_VECTOR_DOUBLES(n) a CTA) above
 * JN_TRI_SMEM_ROWS rows.  Bound by the FP64 chains of a warp (about five
 * rounds of 1.5 n instructions, then 2 n for the vector, 64 cycles each): 100
 * us for 11 pairs at n = 25 to 125 (125 us with one warp to a count), where bisection, inverse iteration and
 * Gram-Schmidt as three kernels took 700 us at n = 45. */
__global__ void __launch_bounds__(TRI_THREADS)
	k_tri_check(const double *__restrict__ a, const double *__restrict__ b, int n, int want, int nvec,
		    double *__restrict__ theta, double *Z, int ldz, double *work, unsigned int *__restrict__ done,
		    double *__restrict__ pack, int first, int exact, int guesses)
{
	extern __shared__ double sbuf[];
	__shared__ jn_tri_exchange ex;
	__shared__ unsigned int last;
	const int i = first + blockIdx.x;
	double *as = work ? work + (size_t)blockIdx.x * JN_TRI_VECTOR_DOUBLES(n) : sbuf, *b2 = as + n;
	double lo, hi, sc = 0.0, guess = 0.0;
	if (threadIdx.x < 64) {
		sc = jn_tri_scale(a, b, n, &lo, &hi);
		if (threadIdx.x < 32) jn_tri_stage(a, b, n, sc, as, b2);
		if (i < guesses) guess = theta[i] * sc;
	}
	__syncthreads();
	if (threadIdx.x < 64) {
		const double x = jn_tri_multisect(as, b2, n, i, lo, hi, exact, i < guesses, guess, &ex);
		if (threadIdx.x == 0) theta[i] = x / sc;
		if (i < nvec && threadIdx.x < 32) jn_tri_vector_warp(as, b2, n, x, Z + (int64_t)i * ldz, b2 + n);
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		__threadfence();
		last = atomicAdd(done, 1u) == gridDim.x - 1;
	}
	__syncthreads();
	if (!last) return;
	__threadfence();
	if (nvec > 0) jn_tri_mgs(Z, ldz, n, nvec);
	for (int j = threadIdx.x; j < want; j += blockDim.x) pack[j] = __ldcg(theta + j);
	for (int j = threadIdx.x; j < nvec; j += blockDim.x) pack[want + j] = Z[(int64_t)j * ldz + n - 1];
	if (threadIdx.x == 0) {
		pack[want + nvec] = b[n - 1];
		*done = 0;
	}
}

/* ------------------------------------------------------------------ */
/* host driver                                                         */
/* ------------------------------------------------------------------ */
static double seconds_now(void)
{
	struct timespec t;
	clock_gettime(CLOCK_MONOTONIC, &t);
	return (double)t.tv_sec + 1e-9 * (double)t.tv_nsec;
}

static int grid_for(int64_t D) { int64_t g = (D + 255) / 256; return (int)(g < 4096 ? (g > 0 ? g : 1) : 4096); }

/* res = <x|y> into device scalar */
static void dot_dev(jn_ctx *c, const double *x, const double *y, double *res)
{
	struct jn_lanczos_state *s = c->lz;
	k_gemv_t<<<RED_BLOCKS, RED_THREADS, 0, c->stream>>>(x, s->D, 1, y, s->d_part, 1);
	k_finish<<<1, 32, 0, c->stream>>>(s->d_part, RED_BLOCKS, 1, 1, res);
}

static jn_status ensure_state(jn_ctx *c, int mmax, int nev)
{
	struct jn_lanczos_state *s = c->lz;
	int64_t D = c->plan.dim;
	if (s && s->mmax >= mmax && s->nev_cap >= nev) return JN_OK;
	jn_lanczos_release(c);
	s = (struct jn_lanczos_state *)calloc(1, sizeof *s);
	c->lz = s;
	s->D = D; s->mmax = mmax; s->nev_cap = nev;
	size_t ncol = (size_t)mmax + 2;
	const size_t packed = (size_t)mmax + nev + 4;
	cudaError_t e = cudaSuccess;
#define DALLOC(ptr, n) if (e == cudaSuccess) e = cudaMalloc((void **)&(ptr), (size_t)(n) * sizeof(*(ptr)))
	DALLOC(s->d_V, (size_t)(mmax + 1) * D);
	DALLOC(s->d_w, D);
	DALLOC(s->d_alpha, mmax + 1);
	DALLOC(s->d_beta, mmax + 1);
	DALLOC(s->d_part, RED_BLOCKS * ncol);
	DALLOC(s->d_h, ncol);
	DALLOC(s->d_scalar, 8);
	DALLOC(s->d_theta, mmax + 1);
	DALLOC(s->d_Z, (size_t)nev * (mmax + 1));
	/* one CTA for each of nev + 1 eigenvalues of a check; all the eigenvalues come TRI_WAVE at a time */
	if (mmax > JN_TRI_SMEM_ROWS)
		DALLOC(s->d_work, (size_t)(nev + 1 > TRI_WAVE ? nev + 1 : TRI_WAVE) * JN_TRI_VECTOR_DOUBLES(mmax));
	DALLOC(s->d_done, 1);
	DALLOC(s->d_pack, packed);
	DALLOC(s->d_ritz, (size_t)nev * D);
	DALLOC(s->d_hritz, (size_t)nev * D);
	DALLOC(s->d_rr, 2 * (size_t)nev);
#undef DALLOC
	for (int i = 0; i < CHECKS; i++) {
		if (e == cudaSuccess) e = cudaMallocHost((void **)&s->h_pack[i], packed * sizeof(double));
		if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->checked[i], cudaEventDisableTiming);
	}
	if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->stepped, cudaEventDisableTiming);
	if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->begun, cudaEventDisableTiming);
	/* the checks' few CTAs are scheduled before the product's thousands */
	int least = 0, greatest = 0;
	if (e == cudaSuccess) e = cudaDeviceGetStreamPriorityRange(&least, &greatest);
	if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&s->check, cudaStreamNonBlocking, greatest);
	if (e == cudaSuccess) e = cudaMemsetAsync(s->d_done, 0, sizeof(unsigned int), s->check);
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(k_tri_check, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)JN_TRI_SMEM(JN_TRI_SMEM_ROWS));
	if (e != cudaSuccess) {
		jn_lanczos_release(c);
		return jn_fail(JN_ERR_NOMEM, "Lanczos workspace (%d vectors of %lld): %s", mmax + 1, (long long)D,
			       cudaGetErrorString(e));
	}
	s->h_rq = (double *)calloc(nev + 1, sizeof(double));
	s->h_res = (double *)calloc(nev + 1, sizeof(double));
	return JN_OK;
}

/* k_tri_check for the `want` lowest eigenvalues of T_n */
static void tri_launch(cudaStream_t st, const double *a, const double *b, int n, int want, int nvec, double *theta, double *Z,
		       int ldz, double *work, unsigned int *done, double *pack, int exact, int guesses)
{
	const int in_smem = n <= JN_TRI_SMEM_ROWS;
	/* TRI_WAVE at a time: all eigenvalues of a T_n whose rows do not fit shared memory */
	for (int i = 0; i < want; i += TRI_WAVE)
		if (in_smem || want <= TRI_WAVE) {
			k_tri_check<<<want, TRI_THREADS, in_smem ? JN_TRI_SMEM(n) : 0, st>>>(a, b, n, want, nvec, theta, Z, ldz,
											     in_smem ? NULL : work, done, pack, 0, exact, guesses);
			break;
		} else {
			k_tri_check<<<want - i < TRI_WAVE ? want - i : TRI_WAVE, TRI_THREADS, 0, st>>>(
				a, b, n, want, nvec, theta, Z, ldz, work, done, pack, i, exact, guesses);
		}
}

/* Enqueue, behind the work now on the context's stream, the lowest `want`
 * eigenvalues of T_n and the eigenvectors of the lowest `nvec` (rows of d_Z)
 * on the checks' stream.  exact: to the last bit and from T_n alone, whatever
 * was checked before; else to 2^-54 of the span, from the last check's values
 * on.  h_pack[slot] receives theta (want), the bottom
 * components (nvec) and beta_{n-1} once checked[slot] has happened. */
static jn_status tri_enqueue(jn_ctx *c, int n, int want, int nvec, int exact, int slot)
{
	struct jn_lanczos_state *s = c->lz;
	CUDA_TRY(cudaEventRecord(s->stepped, c->stream));
	CUDA_TRY(cudaStreamWaitEvent(s->check, s->stepped, 0));
	if (exact) CUDA_TRY(cudaEventRecord(s->begun, s->check));
	tri_launch(s->check, s->d_alpha, s->d_beta, n, want, nvec, s->d_theta, s->d_Z, s->mmax + 1, s->d_work, s->d_done, s->d_pack,
		   exact, exact ? 0 : s->guesses);
	s->guesses = want;
	CUDA_TRY(cudaGetLastError());
	CUDA_TRY(cudaMemcpyAsync(s->h_pack[slot], s->d_pack, (size_t)(want + nvec + 1) * sizeof(double), cudaMemcpyDeviceToHost,
				 s->check));
	CUDA_TRY(cudaEventRecord(s->checked[slot], s->check));
	return JN_OK;
}

/* each eigenvalue is found by itself: those of a cluster may cross by a rounding */
static void ascending(double *v, int n)
{
	for (int i = 1; i < n; i++)
		if (v[i] < v[i - 1]) v[i] = v[i - 1];
}

/* wait for the results in h_pack[0] */
static jn_status tri_wait(jn_ctx *c, int want)
{
	struct jn_lanczos_state *s = c->lz;
	CUDA_TRY(cudaEventSynchronize(s->checked[0]));
	ascending(s->h_pack[0], want);
	return JN_OK;
}

/* the same, exact and waited for, into h_pack[0] */
static jn_status tri_eig(jn_ctx *c, int n, int want, int nvec)
{
	jn_status st = tri_enqueue(c, n, want, nvec, 1, 0);
	return st ? st : tri_wait(c, want);
}

extern "C" jn_status jn_tridiagonal(const double *a, const double *b, int n, int num_values, double *values, int num_vectors,
				    double *vectors)
{
	if (!a || (!b && n > 1) || !values || n < 1 || num_values < 1 || num_values > n || num_vectors < 0 || num_vectors > num_values ||
	    (num_vectors && !vectors))
		return jn_fail(JN_ERR_INVALID, "bad argument");
	const size_t wave = num_values < TRI_WAVE ? num_values : TRI_WAVE;
	const size_t nv = (size_t)num_vectors * n, nw = n > JN_TRI_SMEM_ROWS ? wave * JN_TRI_VECTOR_DOUBLES(n) : 0;
	const size_t np = (size_t)num_values + num_vectors + 1;
	double *d = NULL;
	cudaStream_t st = NULL;
	/* the matrix (2 n), the values, the vectors, the scratch, the packed results, the counter */
	const size_t bytes = (2 * (size_t)n + num_values + nv + nw + np + 1) * sizeof(double);
	cudaError_t e = cudaMalloc((void **)&d, bytes);
	if (e != cudaSuccess) {
		cudaGetLastError();
		return jn_fail(JN_ERR_NOMEM, "tridiagonal matrix of %d rows: %s", n, cudaGetErrorString(e));
	}
	double *theta = d + 2 * (size_t)n, *Z = theta + num_values, *work = Z + nv, *pack = work + nw;
	e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(k_tri_check, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)JN_TRI_SMEM(JN_TRI_SMEM_ROWS));
	if (e == cudaSuccess) e = cudaMemsetAsync(d, 0, bytes, st);
	if (e == cudaSuccess) e = cudaMemcpyAsync(d, a, n * sizeof(double), cudaMemcpyHostToDevice, st);
	if (e == cudaSuccess && n > 1) e = cudaMemcpyAsync(d + n, b, (n - 1) * sizeof(double), cudaMemcpyHostToDevice, st);
	if (e == cudaSuccess) {
		tri_launch(st, d, d + n, n, num_values, num_vectors, theta, Z, n, work, (unsigned int *)(pack + np), pack, 1, 0);
		e = cudaGetLastError();
	}
	if (e == cudaSuccess) e = cudaMemcpyAsync(values, pack, num_values * sizeof(double), cudaMemcpyDeviceToHost, st);
	if (e == cudaSuccess && nv) e = cudaMemcpyAsync(vectors, Z, nv * sizeof(double), cudaMemcpyDeviceToHost, st);
	if (st) {
		const cudaError_t es = cudaStreamSynchronize(st);
		if (e == cudaSuccess) e = es;
		cudaStreamDestroy(st);
	}
	cudaFree(d);
	if (e != cudaSuccess) return jn_fail(JN_ERR_CUDA, "tridiagonal matrix: %s", cudaGetErrorString(e));
	ascending(values, num_values);
	/* the kernels take couplings >= 0, as a recurrence makes them; the others' signs go into the components */
	int negative = 0;
	for (int i = 1; i < n; i++) {
		negative ^= b[i - 1] < 0.0;
		for (int k = 0; k < num_vectors && negative; k++) vectors[(size_t)k * n + i] = -vectors[(size_t)k * n + i];
	}
	return JN_OK;
}

extern "C" jn_status jn_lanczos(jn_ctx *c, const jn_lanczos_options *opt, jn_lanczos_result *res)
{
	if (!c || !opt || !res) return jn_fail(JN_ERR_INVALID, "null argument");
	const int64_t D = c->plan.dim;
	int m = opt->max_iterations > 0 ? opt->max_iterations : 200;
	if ((int64_t)m > D) m = (int)D;               /* lanczos.c:181-185 */
	int nev = opt->num_eigenvalues > 0 ? opt->num_eigenvalues : 10;
	if (nev > JN_MAX_REPORTED) nev = JN_MAX_REPORTED;
	if (nev > m) nev = m;
	const int reference_mode = opt->mode == JN_LANCZOS_REFERENCE;
	const int check_every = opt->check_every > 0 ? opt->check_every : 1;
	jn_status st = ensure_state(c, m, nev < 1 ? 1 : nev);
	if (st) return st;
	struct jn_lanczos_state *s = c->lz;
	s->nev = nev;
	s->have_ritz = 0;
	s->guesses = 0;
	cudaStream_t q = c->stream;
	const int g = grid_for(D);
	double *V = s->d_V;

	/* v_0 */
	if (opt->start_vector) {
		CUDA_TRY(cudaMemcpyAsync(s->d_w, opt->start_vector, D * sizeof(double), cudaMemcpyHostToDevice, q));
		dot_dev(c, s->d_w, s->d_w, s->d_scalar);
		k_normalize<<<g, 256, 0, q>>>(V, s->d_w, s->d_scalar, NULL, D);
	} else {
		CUDA_TRY(cudaMemsetAsync(V, 0, D * sizeof(double), q));
		double one = 1.0;
		CUDA_TRY(cudaMemcpyAsync(V, &one, sizeof(double), cudaMemcpyHostToDevice, q));
		CUDA_TRY(cudaStreamSynchronize(q));
	}

	/* the step's vector work: one CTA an SM, at least 32 elements each */
	int64_t chunk = (D + c->num_sms - 1) / c->num_sms;
	chunk = (chunk < 32 ? 32 : chunk + 3) & ~3ll;
	const int og = (int)((D + chunk - 1) / chunk);

	double prev = 0.0;
	int k, converged = 0;
	const int behind = c->plan.visits >= LONG_STEP ? 1 : CHECKS - 1;
	int pending[CHECKS], npending = 0;      /* rows of the checks that are still to be read, oldest first */
	/* the eigenvector criterion keeps the previous step's vector (and the current one after it) */
	const int by_vector = reference_mode && opt->criterion == JN_CONVERGE_EIGENVECTORS;
	std::vector<double> zbuf;
	try {
		zbuf.resize(by_vector ? 2 * (size_t)(m + 1) : 0);
	} catch (const std::bad_alloc &) {
		return jn_fail(JN_ERR_NOMEM, "out of host memory");
	}
	double *zprev = zbuf.data();
	res->iterations = 0;
	res->iteration_seconds = res->refinement_seconds = 0.0;
	const double t_loop = seconds_now();
	/* the convergence test of T_n from its check's results: 1 converged, 0 not, -1 on an error (in st) */
	auto test_full = [&](int n) -> int {
		const int slot = n % CHECKS, wv = nev < n ? nev : n, wt = wv + (wv < n ? 1 : 0);
		const cudaError_t e = cudaEventSynchronize(s->checked[slot]);
		if (e != cudaSuccess) {
			st = jn_fail(JN_ERR_CUDA, "convergence check: %s", cudaGetErrorString(e));
			return -1;
		}
		const double *theta = s->h_pack[slot], *zlast = theta + wt, beta = zlast[wv];
		int ok = n >= nev;
		for (int i = 0; i < wv && ok; i++) {
			double r = fabs(beta * zlast[i]);
			double gap = 1e300;
			if (i > 0) gap = fmin(gap, theta[i] - theta[i - 1]);
			if (i + 1 < wt) gap = fmin(gap, theta[i + 1] - theta[i]);
			double bound = fmin(r, r * r / fmax(gap, 1e-300));
			if (!(bound < opt->tolerance)) ok = 0;
		}
		if (opt->verbose)
			printf("Lanczos iteration %d: lowest Ritz value %.17lg, beta %lg\n", n, theta[0], beta);
		return ok || beta == 0.0;
	};
	for (k = 0; k < m; k++) {
		double *vk = V + (int64_t)k * D, *vk1 = V + (int64_t)(k + 1) * D;
		st = jn_launch_matvec(c, vk, s->d_w, 0, q);
		if (st) return st;
		if (!reference_mode) {
			int64_t Dl = D;
			void *args[] = { &V, &Dl, &chunk, &k, &s->d_w, &s->d_part, &s->d_h, &s->d_alpha, &s->d_beta };
			CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_orthonormalize, dim3(og), dim3(ORTHO_WARPS * 32), args, 0, q));
		} else {
			dot_dev(c, vk, s->d_w, s->d_alpha + k);
			k_three_term<<<g, 256, 0, q>>>(s->d_w, vk, k ? V + (int64_t)(k - 1) * D : NULL, s->d_alpha + k,
						       k ? s->d_beta + k - 1 : NULL, D);
			dot_dev(c, s->d_w, s->d_w, s->d_scalar);
			k_normalize<<<g, 256, 0, q>>>(vk1, s->d_w, s->d_scalar, s->d_beta + k, D);
			/* MGS of v_{k+1} against v_0..v_{k-3}, no renormalisation (vector.c:461-476) */
			for (int j = 0; j + 2 < k; j++) {
				dot_dev(c, vk1, V + (int64_t)j * D, s->d_scalar + 1);
				k_axpy_neg<<<g, 256, 0, q>>>(vk1, V + (int64_t)j * D, s->d_scalar + 1, D);
			}
			CUDA_TRY(cudaGetLastError());
		}
		const int n = k + 1, check = !(n % check_every) || n == m;
		if (reference_mode) {
			if (!check) continue;
			st = tri_eig(c, n, 1, by_vector);
			if (st) return st;
			const double theta0 = s->h_pack[0][0];
			double diff;
			if (by_vector) {
				/* the lowest eigenvector of T_n against the previous step's (lanczos.c:210-215, 276-287) */
				CUDA_TRY(cudaMemcpy(zprev + (m + 1), s->d_Z, n * sizeof(double), cudaMemcpyDeviceToHost));
				double *z = zprev + (m + 1);
				if (z[0] < 0.0)
					for (int i = 0; i < n; i++) z[i] = -z[i];
				double d2 = z[n - 1] * z[n - 1];
				for (int i = 0; i + 1 < n; i++) d2 += (z[i] - zprev[i]) * (z[i] - zprev[i]);
				diff = sqrt(d2);
				memcpy(zprev, z, n * sizeof(double));
			} else {
				diff = fabs(theta0 - prev);
			}
			prev = theta0;
			if (opt->verbose)
				printf("Lanczos iteration %d: lowest Ritz value %.17lg, difference %lg\n", n, theta0, diff);
			if (diff < opt->tolerance) { converged = 1; k++; break; }
			continue;
		}
		/* full mode: this step's check is enqueued, then the one `behind` steps
		   before it is read, so the device always holds work; a solve that has
		   converged has as many steps too many in flight, which nothing reads */
		if (check) {
			const int wv = nev < n ? nev : n;
			st = tri_enqueue(c, n, wv + (wv < n ? 1 : 0), wv, 0, n % CHECKS);
			if (st) return st;
			pending[npending++] = n;
		}
		if (npending && pending[0] <= n - behind) {
			const int t = test_full(pending[0]);
			if (t < 0) return st;
			if (t) { converged = 1; k = pending[0]; npending = 0; break; }
			npending--;
			for (int i = 0; i < npending; i++) pending[i] = pending[i + 1];
		}
	}
	for (int i = 0; i < npending && !converged; i++) {
		const int t = test_full(pending[i]);
		if (t < 0) return st;
		converged = t;
		k = pending[i];
	}
	s->k = k;
	res->iterations = k;
	res->converged = converged;
	/* final decomposition of T_k: the Ritz values and vectors of the lowest nev */
	int want = nev < k ? nev : k;
	res->num_ritz_values = k;
	st = tri_enqueue(c, k, want, want, 1, 0);
	if (st) return st;
	/* the steps and checks under way when convergence was read end before it begins */
	CUDA_TRY(cudaEventSynchronize(s->begun));
	const double t_final = seconds_now();
	res->iteration_seconds = t_final - t_loop;
	st = tri_wait(c, want);
	if (st) return st;
	/* Ritz vectors x_i = sum_j z_i[j] v_j and their FP64 refinement */
	k_ritz_vectors<<<dim3((unsigned int)((D + 127) / 128), (want + RITZ_ROWS - 1) / RITZ_ROWS), 128, 0, q>>>(
		V, D, k, s->d_Z, s->mmax + 1, want, s->d_ritz);
	s->have_ritz = 1;
	/* the refinement's products are FP64-grade whatever the iteration's precision */
	const int prec0 = c->precision, engine0 = c->engine;
	c->precision = 64;
	c->engine = c->engine_of[0];
	st = jn_enqueue_many(c, s->d_ritz, s->d_hritz, want, q);
	c->precision = prec0;
	c->engine = engine0;
	if (st) return st;
	k_rayleigh<<<want, 512, 0, q>>>(s->d_ritz, s->d_hritz, D, want, s->d_rr);
	CUDA_TRY(cudaGetLastError());
	CUDA_TRY(cudaMemcpyAsync(s->h_pack[1], s->d_rr, 2 * (size_t)want * sizeof(double), cudaMemcpyDeviceToHost, q));
	CUDA_TRY(cudaStreamSynchronize(q));
	for (int i = 0; i < want; i++) {
		s->h_rq[i] = s->h_pack[1][i];
		s->h_res[i] = s->h_pack[1][want + i];
	}
	res->refinement_seconds = seconds_now() - t_final;
	res->num_eigenvalues = want;
	for (int i = 0; i < want && i < JN_MAX_REPORTED; i++) {
		res->eigenvalues[i] = s->h_rq[i];
		res->ritz_values[i] = s->h_pack[0][i];
		res->residual_norms[i] = s->h_res[i];
	}
	return converged ? JN_OK : (opt->mode == JN_LANCZOS_REFERENCE ? JN_OK : jn_fail(JN_ERR_NOT_CONVERGED,
		"Lanczos did not converge in %d iterations", k));
}

extern "C" jn_status jn_lanczos_ritz_values(jn_ctx *c, double *out, int capacity, int *count)
{
	if (!c || !c->lz || !out) return jn_fail(JN_ERR_INVALID, "no Lanczos solve on this context");
	struct jn_lanczos_state *s = c->lz;
	jn_status st = tri_eig(c, s->k, s->k, 0);
	if (st) return st;
	int n = s->k < capacity ? s->k : capacity;
	memcpy(out, s->h_pack[0], n * sizeof(double));
	if (count) *count = s->k;
	return JN_OK;
}

extern "C" jn_status jn_lanczos_eigenvector(jn_ctx *c, int i, double *host_out)
{
	if (!c || !c->lz || !c->lz->have_ritz || !host_out) return jn_fail(JN_ERR_INVALID, "no Ritz vectors on this context");
	struct jn_lanczos_state *s = c->lz;
	if (i < 0 || i >= s->nev || i >= s->k) return jn_fail(JN_ERR_INVALID, "eigenvector index out of range");
	CUDA_TRY(cudaMemcpyAsync(host_out, s->d_ritz + (size_t)i * s->D, s->D * sizeof(double), cudaMemcpyDeviceToHost,
				 c->stream));
	CUDA_TRY(cudaStreamSynchronize(c->stream));
	return JN_OK;
}

extern "C" jn_status jn_lanczos_save_eigenvectors(jn_ctx *c, const char *directory, int count)
{
	if (!c || !directory) return jn_fail(JN_ERR_INVALID, "null argument");
	const jn_plan_t *p = &c->plan;
	double *buf = (double *)malloc((p->dim ? p->dim : 1) * sizeof(double));
	jn_status st = JN_OK;
	mkdir(directory, 0755);
	for (int i = 0; i < count && !st; i++) {
		st = jn_lanczos_eigenvector(c, i, buf);
		if (st) break;
		char dir[8192];
		snprintf(dir, sizeof dir, "%s/eigenvector_%d", directory, i + 1);   /* bacchus.c:68-87 */
		mkdir(dir, 0755);
		for (int b = 0; b < p->nblocks && !st; b++) {
			char path[8300];
			snprintf(path, sizeof path, "%s/vec_%d", dir, b + 1);            /* vector.c:538-555 */
			FILE *f = fopen(path, "wb");
			if (!f) { st = jn_fail(JN_ERR_IO, "Could not open %s", path); break; }
			size_t n = (size_t)(p->blocks[b].Np * p->blocks[b].Nn);
			if (fwrite(buf + p->blocks[b].offset, sizeof(double), n, f) != n) st = jn_fail(JN_ERR_IO, "write %s", path);
			fclose(f);
		}
	}
	free(buf);
	return st;
}

extern "C" void jn_print_eigensystem(const double *ev, int n)
{
	printf("eigensystem:\n{\n");
	printf("\tnum_eigenvalues = %d;\n", n);
	printf("\teigenvalues = ( ");
	for (int i = 0; i < n; i++) printf("%.17lg%s ", ev[i], i == n - 1 ? "" : ",");
	printf(");\n}\n");
	fflush(stdout);
}
