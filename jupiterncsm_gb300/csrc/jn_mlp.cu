/*
 * jn_mlp.cu — the learned warm start: a small MLP, trained and run with
 * hand-written kernels, that maps the couplings c of H(c) = H0 + sum c_i H_i
 * to coefficients over a reduced basis of snapshot eigenvectors.  The
 * expanded vector is the Lanczos start vector.  No counterpart in the
 * reference.
 *
 * Network (FP32): x (n_in) -> h1 = gelu(W1 x + b1) (H) -> h2 = gelu(W2 h1 + b2)
 * (H) -> y = W3 h2 + b3 (n_out), gelu(a) = a/2 (1 + erf(a/sqrt 2)).
 * Loss: sum over samples and outputs of (y - t)^2 / (2 N).  Parameters are
 * one flat array [W1 (H x n_in), b1, W2 (H x H), b2, W3 (n_out x H), b3],
 * row-major with the output index first.  Gradients are summed over samples
 * in sample order (no atomics), so training is deterministic.  Adam updates
 * the parameters.
 */
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <cooperative_groups.h>

#include "jn_internal.h"
#include "jn_tridiag.cuh"

struct jn_mlp {
	int nin, nh, nout;
	int num_sms;
	int64_t np;                     /* parameters */
	float *d_p, *d_g, *d_m, *d_v;   /* parameters (the allocation), gradient, Adam moments */
	int64_t t;                      /* Adam steps taken */
	int cap;                        /* samples the activation buffers hold */
	/* activations, one allocation (d_x): sample by sample, or unit by unit on the fused path */
	float *d_x, *d_t, *d_a1, *d_h1, *d_a2, *d_h2, *d_y, *d_d1, *d_d2, *d_d3, *d_loss;
	float *d_corr;                  /* the fused path's bias corrections, then its two status words */
	float *d_image;                 /* and its image of the weights */
	int polls;                      /* limit of a wait for a copy of it */
	cudaStream_t stream;
};

struct mlp_off {
	int64_t w1, b1, w2, b2, w3, b3;
};

__host__ __device__ static inline mlp_off offsets(int nin, int nh, int nout)
{
	mlp_off o;
	o.w1 = 0;
	o.b1 = o.w1 + (int64_t)nh * nin;
	o.w2 = o.b1 + nh;
	o.b2 = o.w2 + (int64_t)nh * nh;
	o.w3 = o.b2 + nh;
	o.b3 = o.w3 + (int64_t)nout * nh;
	return o;
}

__device__ __forceinline__ float gelu(float a) { return 0.5f * a * (1.0f + erff(a * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float a)
{
	return 0.5f * (1.0f + erff(a * 0.70710678118654752f)) + a * 0.39894228040143268f * expf(-0.5f * a * a);
}

/* one CTA per sample, blockDim >= max(nh, nout) */
__global__ void mlp_forward(const float *__restrict__ P, int nin, int nh, int nout, int n, const float *__restrict__ X,
			    float *__restrict__ A1, float *__restrict__ H1, float *__restrict__ A2, float *__restrict__ H2,
			    float *__restrict__ Y)
{
	extern __shared__ float sm[];
	float *x = sm, *h1 = x + nin, *h2 = h1 + nh;
	const int s = blockIdx.x, j = threadIdx.x;
	if (s >= n) return;
	const mlp_off o = offsets(nin, nh, nout);
	for (int i = j; i < nin; i += blockDim.x) x[i] = X[(int64_t)s * nin + i];
	__syncthreads();
	if (j < nh) {
		float a = P[o.b1 + j];
		for (int i = 0; i < nin; i++) a = fmaf(P[o.w1 + (int64_t)j * nin + i], x[i], a);
		A1[(int64_t)s * nh + j] = a;
		h1[j] = H1[(int64_t)s * nh + j] = gelu(a);
	}
	__syncthreads();
	if (j < nh) {
		float a = P[o.b2 + j];
		for (int k = 0; k < nh; k++) a = fmaf(P[o.w2 + (int64_t)j * nh + k], h1[k], a);
		A2[(int64_t)s * nh + j] = a;
		h2[j] = H2[(int64_t)s * nh + j] = gelu(a);
	}
	__syncthreads();
	if (j < nout) {
		float a = P[o.b3 + j];
		for (int k = 0; k < nh; k++) a = fmaf(P[o.w3 + (int64_t)j * nh + k], h2[k], a);
		Y[(int64_t)s * nout + j] = a;
	}
}

/* per sample: output error and the back-propagated deltas; loss partial per sample */
__global__ void mlp_deltas(const float *__restrict__ P, int nin, int nh, int nout, int n, const float *__restrict__ T,
			   const float *__restrict__ Y, const float *__restrict__ A1, const float *__restrict__ A2,
			   float *__restrict__ D1, float *__restrict__ D2, float *__restrict__ D3, float *__restrict__ lossp)
{
	extern __shared__ float sm[];
	float *d3 = sm, *d2 = d3 + nout;
	const int s = blockIdx.x, j = threadIdx.x;
	if (s >= n) return;
	const mlp_off o = offsets(nin, nh, nout);
	const float inv = 1.0f / (float)n;
	if (j < nout) {
		const float e = Y[(int64_t)s * nout + j] - T[(int64_t)s * nout + j];
		d3[j] = D3[(int64_t)s * nout + j] = e * inv;
	}
	__syncthreads();
	if (j == 0) {
		float l = 0.0f;
		for (int q = 0; q < nout; q++) {
			const float e = Y[(int64_t)s * nout + q] - T[(int64_t)s * nout + q];
			l = fmaf(e, e, l);
		}
		lossp[s] = 0.5f * l * inv;
	}
	if (j < nh) {
		float g = 0.0f;
		for (int q = 0; q < nout; q++) g = fmaf(P[o.w3 + (int64_t)q * nh + j], d3[q], g);
		d2[j] = D2[(int64_t)s * nh + j] = g * gelu_grad(A2[(int64_t)s * nh + j]);
	}
	__syncthreads();
	if (j < nh) {
		float g = 0.0f;
		for (int k = 0; k < nh; k++) g = fmaf(P[o.w2 + (int64_t)k * nh + j], d2[k], g);
		D1[(int64_t)s * nh + j] = g * gelu_grad(A1[(int64_t)s * nh + j]);
	}
}

/* one thread per parameter: the gradient summed over samples in order */
__global__ void mlp_gradients(int nin, int nh, int nout, int n, const float *__restrict__ X, const float *__restrict__ H1,
			      const float *__restrict__ H2, const float *__restrict__ D1, const float *__restrict__ D2,
			      const float *__restrict__ D3, float *__restrict__ G)
{
	const mlp_off o = offsets(nin, nh, nout);
	const int64_t np = o.b3 + nout;
	const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= np) return;
	const float *delta, *act;
	int dn, an, row, col;
	if (p < o.b1) { delta = D1; dn = nh; act = X; an = nin; row = (int)((p - o.w1) / nin); col = (int)((p - o.w1) % nin); }
	else if (p < o.w2) { delta = D1; dn = nh; act = NULL; an = 0; row = (int)(p - o.b1); col = 0; }
	else if (p < o.b2) { delta = D2; dn = nh; act = H1; an = nh; row = (int)((p - o.w2) / nh); col = (int)((p - o.w2) % nh); }
	else if (p < o.w3) { delta = D2; dn = nh; act = NULL; an = 0; row = (int)(p - o.b2); col = 0; }
	else if (p < o.b3) { delta = D3; dn = nout; act = H2; an = nh; row = (int)((p - o.w3) / nh); col = (int)((p - o.w3) % nh); }
	else { delta = D3; dn = nout; act = NULL; an = 0; row = (int)(p - o.b3); col = 0; }
	float g = 0.0f;
	for (int s = 0; s < n; s++) {
		const float d = delta[(int64_t)s * dn + row];
		g = act ? fmaf(d, act[(int64_t)s * an + col], g) : g + d;
	}
	G[p] = g;
}

/* out[n] = the samples' losses summed in order (staged, then one thread adds) */
__global__ void __launch_bounds__(256) mlp_loss_sum(const float *__restrict__ lossp, int n, float *__restrict__ out)
{
	__shared__ float buf[1024];
	float l = 0.0f;
	for (int s0 = 0; s0 < n; s0 += 1024) {
		const int ns = min(1024, n - s0);
		__syncthreads();
		for (int s = threadIdx.x; s < ns; s += blockDim.x) buf[s] = lossp[s0 + s];
		__syncthreads();
		if (threadIdx.x == 0)
			for (int s = 0; s < ns; s++) l += buf[s];
	}
	if (threadIdx.x == 0) out[n] = l;
}

__device__ __forceinline__ void mlp_adam_one(float &p, float &m, float &v, float g, float lr, float b1, float b2, float eps,
					     float c1, float c2)
{
	/* the contractions are spelt out: both paths round alike */
	m = fmaf(1.0f - b1, g, b1 * m);
	v = fmaf((1.0f - b2) * g, g, b2 * v);
	p -= lr * (m / c1) / (sqrtf(v / c2) + eps);
}

__global__ void mlp_adam(float *__restrict__ P, const float *__restrict__ G, float *__restrict__ M, float *__restrict__ V,
			 int64_t np, float lr, float b1, float b2, float eps, float c1, float c2)
{
	const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (p < np) mlp_adam_one(P[p], M[p], V[p], G[p], lr, b1, b2, eps, c1, c2);
}

static int threads_for(const jn_mlp *m)
{
	int t = m->nh > m->nout ? m->nh : m->nout;
	return (t + 31) / 32 * 32;
}

#define FUSED_SMEM_LIMIT (220 * 1024)
/* ------------------------------------------------------------------ */
/* fused path: whole training runs in one launch                        */
/* ------------------------------------------------------------------ */
/* Networks whose weights fit an SM's shared memory (hidden widths up to
 * about 200) run here: one cooperative launch, one CTA an SM, for up to
 * FUSED_STEPS Adam steps.  Per step, phase A: every CTA loads the weights
 * (L2 to shared memory, bulk copies) and takes SP samples
 * through the forward pass and the deltas, a thread per unit; phase B: every
 * CTA takes 16 x 16 tiles of (weight matrix | bias), sums their gradient
 * over the samples and updates its parameters.  Two grid-wide barriers a step.
 * Every sum runs in the order of the kernel-per-pass path above (bias, then
 * inputs ascending; samples ascending), so the results are the same bits.
 * What bounds it: shared-memory reads (a wavefront for every 128 bytes that
 * a warp's lanes take in, equal or not) and the two barriers (1.1 us each).
 * 4-128-128-32 on 256 samples: 11.7 us a step, where the five kernels of the
 * other path take 102 us, 90 of them in strided reads of weights and
 * activations.  The weights as 8 bulk copies a CTA; measured with the CTAs in
 * clusters of 8, which do not fill all SMs, that takes 12.9 us a step, 32 copies 13.3, 16-byte
 * asynchronous copies by all threads 14.0, and an eighth from L2 with the rest
 * from the shared memory of seven neighbours 17.6 to 17.9. */
#define FUSED_STEPS 1024
#define FUSED_THREADS 512       /* at most: 128 registers a thread */
#define FUSED_TILE 16
#define FUSED_CHUNK 256         /* samples staged at a time in phase B */
#define FUSED_PITCH (FUSED_CHUNK + 4)
#define FUSED_PARTS 8           /* copies of a fetch of the weights */

/* row pitch in floats: a multiple of 4, 4 modulo 32, so that 16-byte reads
 * of one column group by 8 neighbouring rows touch all 32 banks */
__host__ __device__ static inline int fused_pitch(int n) { return n <= 4 ? 4 : (n - 4 + 31) / 32 * 32 + 4; }
__host__ __device__ static inline int round4(int n) { return (n + 3) & ~3; }

struct fused_args {
	int nin, nh, nout, n, ldn;      /* ldn: samples a unit's row of XT, H1T, ... holds (a multiple of 4) */
	int steps;                      /* Adam steps */
	int grad;                       /* after them: the gradient at the parameters (into G) */
	int eval;                       /* after them: a forward pass; 1 losses per sample, 2 outputs, 0 none */
	float *P, *G, *M, *V;
	const float *X, *T;             /* n x nin, n x nout */
	float *XT, *H1T, *H2T, *D1T, *D2T, *D3T;        /* unit by unit: inputs, activations, deltas */
	float *Y, *lossp;
	const float *corr;              /* the steps' bias corrections, c1 and c2 of each */
	float *image;                   /* the weights in the shared-memory layout */
	unsigned int *status;           /* set when a wait gave up; Adam steps taken, `before` and this launch's */
	int before;
	int polls;
	float lr, b1, b2, eps;
};

/* words of the weights' image: W1, W2 and W3 with padded rows, in FUSED_PARTS equal parts of 16-byte units */
__host__ __device__ static inline size_t fused_words(int nin, int nh, int nout)
{
	const size_t w = (size_t)nh * fused_pitch(nin) + (size_t)(nh + nout) * fused_pitch(nh), unit = 4 * FUSED_PARTS;
	return (w + unit - 1) / unit * unit;
}

static size_t fused_smem(int nin, int nh, int nout, int sp)
{
	const size_t weights = fused_words(nin, nh, nout);
	const size_t tiles = 2 * FUSED_TILE * FUSED_PITCH;
	const size_t units = (size_t)sp * (round4(nin) + 3 * round4(nh) + 2 * round4(nout));
	return ((weights > tiles ? weights : tiles) + units) * sizeof(float);
}

/* The weights' image (the shared-memory layout, kept in global memory beside
 * the parameters) into the CTA's shared memory: FUSED_PARTS bulk copies that
 * complete on its barrier, by its first warp.  Each CTA starts at another
 * part, so that the CTAs do not all ask L2 for the same lines at once. */
__device__ __forceinline__ void fused_fetch(const float *image, int words, float *s, unsigned int bar)
{
	if (threadIdx.x == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(words * 4) : "memory");
	__syncwarp();
	if (threadIdx.x < FUSED_PARTS) {
		const int part = words / FUSED_PARTS, at = (int)((threadIdx.x + blockIdx.x) % FUSED_PARTS) * part;
		const unsigned int dst = (unsigned int)__cvta_generic_to_shared(s + at);
		asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
			     ::"r"(dst), "l"(image + at), "r"(part * 4), "r"(bar)
			     : "memory");
	}
}

/* wait for phase `parity` of the barrier, at most `polls` times up to a microsecond; false if it gave up */
#define FUSED_POLLS (1 << 20)
__device__ __forceinline__ bool fused_wait(unsigned int bar, unsigned int parity, int polls)
{
	for (int i = 0; i < polls; i++) {
		unsigned int done;
		asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\tselp.u32 %0, 1, 0, p;\n\t}"
			     : "=r"(done)
			     : "r"(bar), "r"(parity)
			     : "memory");
		if (done) return true;
	}
	return false;
}

/* The wait for the weights.  If it gives up, the status word is set and the
 * copies are waited for once more, so that none lands after the CTA has gone
 * on; the grid leaves the step loop in the phase B that follows, before any
 * parameter is changed. */
__device__ __forceinline__ void fused_land(const fused_args &a, unsigned int bar, unsigned int parity)
{
	if (fused_wait(bar, parity, a.polls)) return;
	*a.status = 1;
	fused_wait(bar, parity, FUSED_POLLS);
}

/* acc[s] += sum_k w[k] v[s][k], k ascending (w a padded shared row, v at
 * pitch ldv); 16 columns' reads are issued before their multiply-adds */
template <int SP>
__device__ __forceinline__ void fused_row(float *acc, const float *w, const float *v, int ldv, int n)
{
	constexpr int U = SP <= 2 ? 4 : 2;
	int k = 0;
	for (; k + 4 * U <= n; k += 4 * U) {
		float4 a[U], b[U][SP];
#pragma unroll
		for (int u = 0; u < U; u++) {
			a[u] = *(const float4 *)(w + k + 4 * u);
#pragma unroll
			for (int s = 0; s < SP; s++) b[u][s] = *(const float4 *)(v + s * ldv + k + 4 * u);
		}
#pragma unroll
		for (int u = 0; u < U; u++)
#pragma unroll
			for (int s = 0; s < SP; s++) {
				acc[s] = fmaf(a[u].x, b[u][s].x, acc[s]);
				acc[s] = fmaf(a[u].y, b[u][s].y, acc[s]);
				acc[s] = fmaf(a[u].z, b[u][s].z, acc[s]);
				acc[s] = fmaf(a[u].w, b[u][s].w, acc[s]);
			}
	}
	for (; k < n; k++)
#pragma unroll
		for (int s = 0; s < SP; s++) acc[s] = fmaf(w[k], v[s * ldv + k], acc[s]);
}

/* acc[s] += sum_k w[k pitch] v[s][k], k ascending */
template <int SP>
__device__ __forceinline__ void fused_col(float *acc, const float *w, int pitch, const float *v, int ldv, int n)
{
	constexpr int U = SP <= 2 ? 4 : 2;
	int k = 0;
	for (; k + 4 * U <= n; k += 4 * U) {
		float a[4 * U];
		float4 b[U][SP];
#pragma unroll
		for (int u = 0; u < 4 * U; u++) a[u] = w[(k + u) * pitch];
#pragma unroll
		for (int u = 0; u < U; u++)
#pragma unroll
			for (int s = 0; s < SP; s++) b[u][s] = *(const float4 *)(v + s * ldv + k + 4 * u);
#pragma unroll
		for (int u = 0; u < U; u++)
#pragma unroll
			for (int s = 0; s < SP; s++) {
				acc[s] = fmaf(a[4 * u], b[u][s].x, acc[s]);
				acc[s] = fmaf(a[4 * u + 1], b[u][s].y, acc[s]);
				acc[s] = fmaf(a[4 * u + 2], b[u][s].z, acc[s]);
				acc[s] = fmaf(a[4 * u + 3], b[u][s].w, acc[s]);
			}
	}
	for (; k < n; k++)
#pragma unroll
		for (int s = 0; s < SP; s++) acc[s] = fmaf(w[k * pitch], v[s * ldv + k], acc[s]);
}

/* phase A: forward pass of every sample; with deltas, also back-propagation
 * and the activations that phase B reads.  round: how often the launch has
 * been here (the barrier's phase).  A CTA without samples fetches the
 * weights as well, so that all barriers keep the same phase. */
template <int SP>
__device__ __forceinline__ void fused_samples(const fused_args &a, const mlp_off &o, float *sm, size_t weights, unsigned int bar, unsigned int round,
					      bool deltas, int eval)
{
	const int nin = a.nin, nh = a.nh, nout = a.nout, j = threadIdx.x;
	const int p1 = fused_pitch(nin), p2 = fused_pitch(nh), lx = round4(nin), lh = round4(nh), lo = round4(nout);
	float *w1 = sm, *w2 = w1 + (size_t)nh * p1, *w3 = w2 + (size_t)nh * p2;
	float *x = sm + weights, *h1 = x + SP * lx, *h2 = h1 + SP * lh, *d2 = h2 + SP * lh, *e3 = d2 + SP * lh, *d3 = e3 + SP * lo;
	const int groups = (a.n + SP - 1) / SP;
	if (threadIdx.x < 32) fused_fetch(a.image, (int)fused_words(nin, nh, nout), sm, bar);
	const float *P = a.P;
	/* the outputs of the CTA's samples, one sample a thread where they fit */
	const bool spread = SP * nout <= (int)blockDim.x;
	const int jo = spread ? j % nout : j, so = spread ? j / nout : 0;
	const float bias1 = j < nh ? __ldcg(P + o.b1 + j) : 0.0f, bias2 = j < nh ? __ldcg(P + o.b2 + j) : 0.0f,
		    bias3 = jo < nout ? __ldcg(P + o.b3 + jo) : 0.0f;
	const float inv = 1.0f / (float)a.n;
	bool landed = false;
	for (int g = blockIdx.x; g < groups; g += gridDim.x) {
		const int s0 = g * SP, ns = min(SP, a.n - s0);
		float target = 0.0f;
		if (spread && so < ns && (deltas || eval == 1)) target = a.T[(int64_t)(s0 + so) * nout + jo];
		for (int t = j; t < SP * nin; t += blockDim.x) {
			const int s = t / nin, i = t - s * nin;
			x[s * lx + i] = s < ns ? a.X[(int64_t)(s0 + s) * nin + i] : 0.0f;
		}
		if (!landed) {
			landed = true;
			fused_land(a, bar, round & 1);
		}
		__syncthreads();
		float z1[SP], z2[SP], acc[SP];
		if (j < nh) {
#pragma unroll
			for (int s = 0; s < SP; s++) z1[s] = bias1;
			fused_row<SP>(z1, w1 + (size_t)j * p1, x, lx, nin);
#pragma unroll
			for (int s = 0; s < SP; s++) {
				const float h = gelu(z1[s]);
				h1[s * lh + j] = h;
				if (deltas && s < ns) a.H1T[(int64_t)j * a.ldn + s0 + s] = h;
			}
		}
		__syncthreads();
		if (j < nh) {
#pragma unroll
			for (int s = 0; s < SP; s++) z2[s] = bias2;
			fused_row<SP>(z2, w2 + (size_t)j * p2, h1, lh, nh);
#pragma unroll
			for (int s = 0; s < SP; s++) {
				const float h = gelu(z2[s]);
				h2[s * lh + j] = h;
				if (deltas && s < ns) a.H2T[(int64_t)j * a.ldn + s0 + s] = h;
			}
		}
		__syncthreads();
		auto output = [&](int s, float y, float t) {
			float e = 0.0f;
			if (s < ns) {
				if (eval == 2) a.Y[(int64_t)(s0 + s) * nout + jo] = y;
				e = y - t;
				if (deltas) a.D3T[(int64_t)jo * a.ldn + s0 + s] = e * inv;
			}
			e3[s * lo + jo] = e;
			d3[s * lo + jo] = e * inv;
		};
		if (spread) {
			if (so < SP) {
				float y = bias3;
				fused_row<1>(&y, w3 + (size_t)jo * p2, h2 + so * lh, lh, nh);
				output(so, y, target);
			}
		} else if (j < nout) {
#pragma unroll
			for (int s = 0; s < SP; s++) acc[s] = bias3;
			fused_row<SP>(acc, w3 + (size_t)j * p2, h2, lh, nh);
#pragma unroll
			for (int s = 0; s < SP; s++)
				output(s, acc[s], s < ns && (deltas || eval == 1) ? a.T[(int64_t)(s0 + s) * nout + j] : 0.0f);
		}
		__syncthreads();
		if (eval == 1 && j < ns) {
			float l = 0.0f;
			for (int q = 0; q < nout; q++) l = fmaf(e3[j * lo + q], e3[j * lo + q], l);
			a.lossp[s0 + j] = 0.5f * l * inv;
		}
		if (deltas) {
			if (j < nh) {
#pragma unroll
				for (int s = 0; s < SP; s++) acc[s] = 0.0f;
				fused_col<SP>(acc, w3 + j, p2, d3, lo, nout);
#pragma unroll
				for (int s = 0; s < SP; s++) {
					const float d = acc[s] * gelu_grad(z2[s]);
					d2[s * lh + j] = d;
					if (s < ns) a.D2T[(int64_t)j * a.ldn + s0 + s] = d;
				}
			}
			__syncthreads();
			if (j < nh) {
#pragma unroll
				for (int s = 0; s < SP; s++) acc[s] = 0.0f;
				fused_col<SP>(acc, w2 + j, p2, d2, lh, nh);
#pragma unroll
				for (int s = 0; s < SP; s++)
					if (s < ns) a.D1T[(int64_t)j * a.ldn + s0 + s] = acc[s] * gelu_grad(z1[s]);
			}
		}
		__syncthreads();        /* the next samples overwrite x, h1, ... */
	}
	/* no CTA goes on with copies in flight */
	/* no CTA goes on with copies in flight */
	if (!landed) fused_land(a, bar, round & 1);
}

/* one parameter's Adam update, or its gradient: p in the parameter array, at
 * in the image (-1: a bias, which the image does not hold) */
__device__ __forceinline__ void fused_update(const fused_args &a, int64_t p, int at, float g, bool adam, float c1, float c2, float pv,
					     float mv, float vv)
{
	if (!adam) {
		a.G[p] = g;
		return;
	}
	mlp_adam_one(pv, mv, vv, g, a.lr, a.b1, a.b2, a.eps, c1, c2);
	a.P[p] = pv;
	if (at >= 0) a.image[at] = pv;
	a.M[p] = mv;
	a.V[p] = vv;
}

/* phase B: the gradient of 16 x 16 tiles of W, a parameter a thread, and
 * with a matrix's first column tile of its bias; with adam the update.  Nothing
 * is written if a wait gave up. */
__device__ __forceinline__ void fused_parameters(const fused_args &a, const mlp_off &o, float *sm, bool adam, float c1, float c2, unsigned int gave_up)
{
	float *ds = sm, *as = sm + FUSED_TILE * FUSED_PITCH;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = threadIdx.x;
	const int row = (warp >> 1) * 4 + (lane >> 3), col = (warp & 1) * 8 + (lane & 7);
	const int p1 = fused_pitch(a.nin), p2 = fused_pitch(a.nh);
	const int rt = (a.nh + FUSED_TILE - 1) / FUSED_TILE, ct1 = (a.nin + FUSED_TILE - 1) / FUSED_TILE;
	const int n1 = rt * ct1, n2 = n1 + rt * rt, n3 = n2 + (a.nout + FUSED_TILE - 1) / FUSED_TILE * rt;
	for (int tile = blockIdx.x; tile < n3; tile += gridDim.x) {
		const float *delta, *act;
		int rows, cols, k, ct, image, pitch;
		int64_t w, b;
		if (tile < n1) {
			delta = a.D1T; act = a.XT; rows = a.nh; cols = a.nin; w = o.w1; b = o.b1; k = tile; ct = ct1; image = 0; pitch = p1;
		} else if (tile < n2) {
			delta = a.D2T; act = a.H1T; rows = a.nh; cols = a.nh; w = o.w2; b = o.b2; k = tile - n1; ct = rt;
			image = a.nh * p1; pitch = p2;
		} else {
			delta = a.D3T; act = a.H2T; rows = a.nout; cols = a.nh; w = o.w3; b = o.b3; k = tile - n2; ct = rt;
			image = a.nh * (p1 + p2); pitch = p2;
		}
		const int r0 = k / ct * FUSED_TILE, c0 = k % ct * FUSED_TILE, r = r0 + row, c = c0 + col;
		const bool mine = t < FUSED_TILE * FUSED_TILE && r < rows && c < cols, bias = mine && c == 0;
		const int64_t p = w + (int64_t)r * cols + c, pb = b + r;
		/* the parameters' state, on its way while the gradient is summed */
		float pv = 0.0f, mv = 0.0f, vv = 0.0f, pbv = 0.0f, mbv = 0.0f, vbv = 0.0f, g = 0.0f, gb = 0.0f;
		if (mine && adam) { pv = a.P[p]; mv = a.M[p]; vv = a.V[p]; }
		if (bias && adam) { pbv = a.P[pb]; mbv = a.M[pb]; vbv = a.V[pb]; }
		for (int s0 = 0; s0 < a.n; s0 += FUSED_CHUNK) {
			const int ns = min(FUSED_CHUNK, a.n - s0), n4 = round4(ns) / 4;
			__syncthreads();
			/* rows of delta, then of the activations, 4 samples a copy */
			const int q = t % (FUSED_CHUNK / 4);
			for (int i = t / (FUSED_CHUNK / 4); i < 2 * FUSED_TILE; i += blockDim.x / (FUSED_CHUNK / 4)) {
				const bool d = i < FUSED_TILE;
				const int u = d ? r0 + i : c0 + i - FUSED_TILE;
				if (q < n4 && u < (d ? rows : cols)) {
					const float *src = (d ? delta : act) + (int64_t)u * a.ldn + s0 + 4 * q;
					const unsigned int dst = (unsigned int)__cvta_generic_to_shared(sm + i * FUSED_PITCH + 4 * q);
					asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
				}
			}
			asm volatile("cp.async.wait_all;" ::: "memory");
			__syncthreads();
			if (t < FUSED_TILE * FUSED_TILE) {
				const float *d = ds + row * FUSED_PITCH, *x = as + col * FUSED_PITCH;
				int s = 0;
#pragma unroll 4
				for (; s + 4 <= ns; s += 4) {
					const float4 u = *(const float4 *)(d + s), v = *(const float4 *)(x + s);
					g = fmaf(u.x, v.x, g);
					g = fmaf(u.y, v.y, g);
					g = fmaf(u.z, v.z, g);
					g = fmaf(u.w, v.w, g);
					gb += u.x;
					gb += u.y;
					gb += u.z;
					gb += u.w;
				}
				for (; s < ns; s++) {
					g = fmaf(d[s], x[s], g);
					gb += d[s];
				}
			}
		}
		if (gave_up) break;
		if (mine) fused_update(a, p, image + r * pitch + c, g, adam, c1, c2, pv, mv, vv);
		if (bias) fused_update(a, pb, -1, gb, adam, c1, c2, pbv, mbv, vbv);
	}
	/* the next phase A reads the image and fills this shared memory through the asynchronous proxy */
	asm volatile("fence.proxy.async;" ::: "memory");
	__syncthreads();
}

template <int SP>
__global__ void __launch_bounds__(FUSED_THREADS) mlp_fused(const fused_args a)
{
	extern __shared__ __align__(16) float sm[];
	__shared__ __align__(8) unsigned long long mbar;
	namespace cg = cooperative_groups;
	cg::grid_group grid = cg::this_grid();
	if (__ldcg(a.status)) return;   /* an earlier launch of the call gave up */
	const mlp_off o = offsets(a.nin, a.nh, a.nout);
	const size_t w = fused_words(a.nin, a.nh, a.nout), weights = w > 2 * FUSED_TILE * FUSED_PITCH ? w : 2 * FUSED_TILE * FUSED_PITCH;
	const unsigned int bar = (unsigned int)__cvta_generic_to_shared(&mbar);
	const int64_t q0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, dq = (int64_t)gridDim.x * blockDim.x;
	if (threadIdx.x == 0) {
		asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	/* the image of the parameters, and the transposed inputs */
	const int p1 = fused_pitch(a.nin), p2 = fused_pitch(a.nh);
	for (int64_t q = q0; q < (int64_t)a.nh * a.nin; q += dq) a.image[q / a.nin * p1 + q % a.nin] = a.P[o.w1 + q];
	for (int64_t q = q0; q < (int64_t)a.nh * a.nh; q += dq) a.image[a.nh * p1 + q / a.nh * p2 + q % a.nh] = a.P[o.w2 + q];
	for (int64_t q = q0; q < (int64_t)a.nout * a.nh; q += dq) a.image[a.nh * (p1 + p2) + q / a.nh * p2 + q % a.nh] = a.P[o.w3 + q];
	if (a.steps || a.grad)
		for (int64_t q = q0; q < (int64_t)a.n * a.nin; q += dq) a.XT[q % a.nin * a.ldn + q / a.nin] = a.X[q];
	asm volatile("fence.proxy.async;" ::: "memory");
	grid.sync();
	unsigned int round = 0;
	int it = 0;
	unsigned int gave_up = 0;
	for (; it < a.steps + (a.grad ? 1 : 0); it++) {
		fused_samples<SP>(a, o, sm, weights, bar, round++, true, it == a.steps ? a.eval : 0);
		grid.sync();
		/* all CTAs alike: the word is set in phase A only.  It is on its way while the gradients are summed */
		gave_up = __ldcg(a.status);
		const bool adam = it < a.steps;
		fused_parameters(a, o, sm, adam, adam ? a.corr[2 * it] : 1.0f, adam ? a.corr[2 * it + 1] : 1.0f, gave_up);
		if (gave_up) break;
		grid.sync();
	}
	if (blockIdx.x == 0 && threadIdx.x == 0) a.status[1] = a.before + min(it, a.steps);
	if (!a.grad && a.eval && !gave_up) fused_samples<SP>(a, o, sm, weights, bar, round++, false, a.eval);
}

/* the fused launch for n samples and its grid, or NULL where the network does not fit it */
typedef void (*fused_kernel)(const fused_args);
static int fused_threads(const jn_mlp *m) { return threads_for(m) > 256 ? threads_for(m) : 256; }
static fused_kernel fused_for(const jn_mlp *m, int n, size_t *smem, int *grid)
{
	/* the fewest samples a CTA (the shortest phase A) for which one round of CTAs takes them all */
	int sp = 1;
	while (sp < 8 && (int64_t)m->num_sms * sp < n) sp *= 2;
	*smem = fused_smem(m->nin, m->nh, m->nout, sp);
	if (*smem > FUSED_SMEM_LIMIT || threads_for(m) > FUSED_THREADS) return NULL;
	fused_kernel f = sp == 1 ? mlp_fused<1> : sp == 2 ? mlp_fused<2> : sp == 4 ? mlp_fused<4> : mlp_fused<8>;
	/* the grid must be resident at once: one CTA an SM */
	int per_sm = 0;
	if (cudaFuncSetAttribute((const void *)f, cudaFuncAttributeMaxDynamicSharedMemorySize, FUSED_SMEM_LIMIT) != cudaSuccess ||
	    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)f, fused_threads(m), *smem) != cudaSuccess || per_sm < 1) {
		cudaGetLastError();
		return NULL;
	}
	*grid = m->num_sms;
	return f;
}

/* Whether the kernels of a pass take one forward pass (or one gradient) in less
 * time than the cooperative launch, which costs about 20 us more to start and
 * needs two grid barriers for a gradient; it wins where the passes' strided reads of the weights
 * take longer than that.  Calls, kernels of a pass against cooperative, us:
 * predict 2-8-8-4 on 1 / 1000 / 100 000 samples 19 / 21 / 119 against 37 / 41 / 199,
 * 4-32-32-8 on 1 / 1000 / 10 000 21 / 31 / 87 against 37 / 41 / 69, 4-64-64-16 on 256 / 1000
 * 30 / 44 against 39 / 40, 4-128-128-32 on 64 / 256 35 / 45 against 39 / 40,
 * 8-160-160-40 on 1 / 64 41 / 43 against 39 / 39; gradient 4-16-16-8 on 1 / 16 / 64
 * 45 / 47 / 58 against 55 / 53 / 54, 4-32-32-8 47 / 47 / 61 against 53 / 53 / 54,
 * 4-64-64-16 on 1 58 against 55. */
static int short_pass(const jn_mlp *m, int n, int gradient)
{
	const int64_t w = (int64_t)m->nh * (m->nin + m->nh + m->nout);
	if (gradient) return w <= 2048 && n <= 32;
	return w <= 512 || (w <= 24576 && n * w <= 1 << 21);
}

static const float ADAM_B1 = 0.9f, ADAM_B2 = 0.999f, ADAM_EPS = 1e-8f;

static jn_status ensure_capacity(jn_mlp *m, int n)
{
	if (n <= m->cap) return JN_OK;
	float **bufs[] = { &m->d_x, &m->d_t, &m->d_a1, &m->d_h1, &m->d_a2, &m->d_h2, &m->d_y, &m->d_d1, &m->d_d2, &m->d_d3,
			   &m->d_loss };
	/* d_a1 also takes the transposed inputs of the fused path */
	const int64_t w[] = { m->nin, m->nout, m->nh > m->nin ? m->nh : m->nin, m->nh, m->nh, m->nh, m->nout, m->nh, m->nh,
			      m->nout, 1 };
	const int64_t rows = ((int64_t)n + 4) & ~3ll;
	int64_t total = 0;
	for (size_t i = 0; i < sizeof w / sizeof w[0]; i++) total += rows * w[i];
	cudaFree(m->d_x);
	m->cap = 0;
	if (cudaMalloc((void **)&m->d_x, (size_t)total * sizeof(float)) != cudaSuccess) {
		m->d_x = NULL;
		return jn_fail(JN_ERR_NOMEM, "MLP activations for %d samples", n);
	}
	for (size_t i = 1; i < sizeof w / sizeof w[0]; i++) *bufs[i] = *bufs[i - 1] + rows * w[i - 1];
	m->cap = n;
	return JN_OK;
}

extern "C" jn_status jn_mlp_set_wait_limit(jn_mlp *m, int polls)
{
	if (!m || polls < 0) return jn_fail(JN_ERR_INVALID, "bad argument");
	m->polls = polls;
	return JN_OK;
}

extern "C" void jn_mlp_destroy(jn_mlp *m)
{
	if (!m) return;
	cudaFree(m->d_p);
	cudaFree(m->d_x);
	if (m->stream) cudaStreamDestroy(m->stream);
	free(m);
}

extern "C" jn_status jn_mlp_create(int nin, int nh, int nout, uint64_t seed, jn_mlp **out)
{
	if (!out || nin < 1 || nh < 1 || nout < 1 || nh > 1024 || nout > 1024 || nin > 1024)
		return jn_fail(JN_ERR_INVALID, "MLP sizes must be in 1..1024");
	*out = NULL;
	jn_mlp *m = (jn_mlp *)calloc(1, sizeof *m);
	m->nin = nin; m->nh = nh; m->nout = nout;
	const mlp_off o = offsets(nin, nh, nout);
	m->np = o.b3 + nout;
	m->polls = FUSED_POLLS;
	float *h = (float *)calloc(m->np, sizeof(float));
	/* seeded uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights, zero biases */
	uint64_t z = seed;
	auto unif = [&z]() {
		z += 0x9E3779B97F4A7C15ull;
		uint64_t v = z;
		v = (v ^ (v >> 30)) * 0xBF58476D1CE4E5B9ull;
		v = (v ^ (v >> 27)) * 0x94D049BB133111EBull;
		v ^= v >> 31;
		return (double)(v >> 11) * 0x1.0p-53 * 2.0 - 1.0;
	};
	for (int64_t i = 0; i < (int64_t)nh * nin; i++) h[o.w1 + i] = (float)(unif() / sqrt((double)nin));
	for (int64_t i = 0; i < (int64_t)nh * nh; i++) h[o.w2 + i] = (float)(unif() / sqrt((double)nh));
	for (int64_t i = 0; i < (int64_t)nout * nh; i++) h[o.w3 + i] = (float)(unif() / sqrt((double)nh));
	jn_status st = JN_OK;
	const int64_t np4 = (m->np + 3) & ~3ll;
	int device = 0;
	const size_t words = 4 * np4 + 2 * FUSED_STEPS + 4 + fused_words(nin, nh, nout);
	if (cudaMalloc((void **)&m->d_p, words * sizeof(float)) != cudaSuccess ||
	    cudaMemset(m->d_p, 0, words * sizeof(float)) != cudaSuccess || cudaGetDevice(&device) != cudaSuccess ||
	    cudaDeviceGetAttribute(&m->num_sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
		st = jn_fail(JN_ERR_NOMEM, "MLP parameters");
	m->d_g = m->d_p + np4;
	m->d_m = m->d_g + np4;
	m->d_v = m->d_m + np4;
	m->d_corr = m->d_v + np4;
	m->d_image = m->d_corr + 2 * FUSED_STEPS + 4;
	if (!st && cudaMemcpy(m->d_p, h, m->np * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess)
		st = jn_fail(JN_ERR_CUDA, "MLP parameter upload");
	if (!st && cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess)
		st = jn_fail(JN_ERR_CUDA, "MLP stream");
	free(h);
	if (st) { jn_mlp_destroy(m); return st; }
	*out = m;
	return JN_OK;
}

extern "C" size_t jn_mlp_num_params(const jn_mlp *m) { return m ? (size_t)m->np : 0; }

extern "C" jn_status jn_mlp_get_params(const jn_mlp *m, float *params)
{
	if (!m || !params) return jn_fail(JN_ERR_INVALID, "null argument");
	CUDA_TRY(cudaMemcpy(params, m->d_p, m->np * sizeof(float), cudaMemcpyDeviceToHost));
	return JN_OK;
}

extern "C" jn_status jn_mlp_set_params(jn_mlp *m, const float *params)
{
	if (!m || !params) return jn_fail(JN_ERR_INVALID, "null argument");
	CUDA_TRY(cudaMemcpy(m->d_p, params, m->np * sizeof(float), cudaMemcpyHostToDevice));
	return JN_OK;
}

static jn_status forward(jn_mlp *m, int n)
{
	const int th = threads_for(m);
	mlp_forward<<<n, th, (m->nin + 2 * m->nh) * sizeof(float), m->stream>>>(m->d_p, m->nin, m->nh, m->nout, n, m->d_x,
										m->d_a1, m->d_h1, m->d_a2, m->d_h2, m->d_y);
	return cudaGetLastError() == cudaSuccess ? JN_OK : jn_fail(JN_ERR_CUDA, "MLP forward launch");
}

static jn_status backward(jn_mlp *m, int n)
{
	const int th = threads_for(m);
	mlp_deltas<<<n, th, (m->nout + m->nh) * sizeof(float), m->stream>>>(m->d_p, m->nin, m->nh, m->nout, n, m->d_t,
									      m->d_y, m->d_a1, m->d_a2, m->d_d1, m->d_d2,
									      m->d_d3, m->d_loss);
	mlp_loss_sum<<<1, 256, 0, m->stream>>>(m->d_loss, n, m->d_loss);
	mlp_gradients<<<(int)((m->np + 255) / 256), 256, 0, m->stream>>>(m->nin, m->nh, m->nout, n, m->d_x, m->d_h1, m->d_h2,
									  m->d_d1, m->d_d2, m->d_d3, m->d_g);
	return cudaGetLastError() == cudaSuccess ? JN_OK : jn_fail(JN_ERR_CUDA, "MLP backward launch");
}

/* the fused launch over the loaded samples: `steps` Adam steps (the bias
 * corrections in d_corr; the call's `before` are behind it), then the gradient (grad) and a pass for the losses
 * (eval 1) or the outputs (eval 2) */
static jn_status fused_run(jn_mlp *m, fused_kernel f, size_t smem, int grid, int n, int before, int steps, float lr, int grad, int eval)
{
	fused_args a;
	memset(&a, 0, sizeof a);
	a.nin = m->nin; a.nh = m->nh; a.nout = m->nout;
	a.n = n;
	a.ldn = round4(n);
	a.steps = steps; a.grad = grad; a.eval = eval;
	a.P = m->d_p; a.G = m->d_g; a.M = m->d_m; a.V = m->d_v;
	a.X = m->d_x; a.T = m->d_t;
	a.XT = m->d_a1; a.H1T = m->d_h1; a.H2T = m->d_h2; a.D1T = m->d_d1; a.D2T = m->d_d2; a.D3T = m->d_d3;
	a.image = m->d_image;
	a.status = (unsigned int *)(m->d_corr + 2 * FUSED_STEPS);
	a.before = before;
	a.polls = m->polls;
	a.Y = m->d_y; a.lossp = m->d_loss;
	a.corr = m->d_corr;
	a.lr = lr; a.b1 = ADAM_B1; a.b2 = ADAM_B2; a.eps = ADAM_EPS;
	void *args[] = { &a };
	CUDA_TRY(cudaLaunchCooperativeKernel((const void *)f, dim3(grid), dim3(fused_threads(m)), args, smem, m->stream));
	return JN_OK;
}

/* A wait of the call's launches gave up: the parameters and moments are those
 * after status[1] of its steps, t0 + status[1] in all; the call's other results
 * are not valid. */
static jn_status fused_check(jn_mlp *m, const unsigned int *status, int64_t t0)
{
	if (!status[0]) return JN_OK;
	m->t = t0 + status[1];
	CUDA_TRY(cudaMemset(m->d_corr + 2 * FUSED_STEPS, 0, sizeof(unsigned int)));
	return jn_fail(JN_ERR_TIMEOUT, "MLP: a wait for the weights' copy gave up");
}

static jn_status load(jn_mlp *m, const float *x, const float *t, int n)
{
	jn_status s = ensure_capacity(m, n);
	if (s) return s;
	CUDA_TRY(cudaMemcpyAsync(m->d_x, x, (size_t)n * m->nin * sizeof(float), cudaMemcpyHostToDevice, m->stream));
	if (t) CUDA_TRY(cudaMemcpyAsync(m->d_t, t, (size_t)n * m->nout * sizeof(float), cudaMemcpyHostToDevice, m->stream));
	return JN_OK;
}

extern "C" jn_status jn_mlp_loss_and_gradient(jn_mlp *m, const float *x, const float *t, int n, float *loss, float *grad)
{
	if (!m || !x || !t || n < 1) return jn_fail(JN_ERR_INVALID, "bad argument");
	jn_status s = load(m, x, t, n);
	size_t smem;
	int grid;
	unsigned int status[2] = { 0, 0 };
	const int64_t t0 = m->t;
	fused_kernel f = short_pass(m, n, 1) ? NULL : fused_for(m, n, &smem, &grid);
	if (!s && f) {
		s = fused_run(m, f, smem, grid, n, 0, 0, 0.0f, 1, 1);
		if (!s) mlp_loss_sum<<<1, 256, 0, m->stream>>>(m->d_loss, n, m->d_loss);
	} else {
		if (!s) s = forward(m, n);
		if (!s) s = backward(m, n);
	}
	if (s) return s;
	if (loss) CUDA_TRY(cudaMemcpyAsync(loss, m->d_loss + n, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
	if (grad) CUDA_TRY(cudaMemcpyAsync(grad, m->d_g, m->np * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
	if (f) CUDA_TRY(cudaMemcpyAsync(status, m->d_corr + 2 * FUSED_STEPS, sizeof status, cudaMemcpyDeviceToHost, m->stream));
	CUDA_TRY(cudaStreamSynchronize(m->stream));
	return fused_check(m, status, t0);
}

extern "C" jn_status jn_mlp_train(jn_mlp *m, const float *x, const float *t, int n, int steps, float lr, float *final_loss)
{
	if (!m || !x || !t || n < 1 || steps < 0) return jn_fail(JN_ERR_INVALID, "bad argument");
	jn_status s = load(m, x, t, n);
	size_t smem;
	int grid;
	unsigned int status[2] = { 0, 0 };
	const int64_t t0 = m->t;
	fused_kernel f = fused_for(m, n, &smem, &grid);
	if (!s && f) {
		float corr[2 * FUSED_STEPS];
		for (int it = 0; (it < steps || it == 0) && !s; it += FUSED_STEPS) {
			const int run = steps - it < FUSED_STEPS ? steps - it : FUSED_STEPS;
			for (int i = 0; i < run; i++) {
				m->t++;
				corr[2 * i] = 1.0f - powf(ADAM_B1, (float)m->t);
				corr[2 * i + 1] = 1.0f - powf(ADAM_B2, (float)m->t);
			}
			/* pageable memory: the copy has left `corr` when the call returns */
			if (run) CUDA_TRY(cudaMemcpyAsync(m->d_corr, corr, 2 * run * sizeof(float), cudaMemcpyHostToDevice, m->stream));
			/* the last launch also takes the loss of the final parameters */
			s = fused_run(m, f, smem, grid, n, it, run, lr, 0, it + FUSED_STEPS >= steps);
		}
		if (!s) mlp_loss_sum<<<1, 256, 0, m->stream>>>(m->d_loss, n, m->d_loss);
	} else {
		for (int it = 0; it < steps && !s; it++) {
			s = forward(m, n);
			if (!s) s = backward(m, n);
			m->t++;
			const float c1 = 1.0f - powf(ADAM_B1, (float)m->t), c2 = 1.0f - powf(ADAM_B2, (float)m->t);
			if (!s) mlp_adam<<<(int)((m->np + 255) / 256), 256, 0, m->stream>>>(m->d_p, m->d_g, m->d_m, m->d_v, m->np, lr,
											       ADAM_B1, ADAM_B2, ADAM_EPS, c1, c2);
		}
		/* loss of the final parameters */
		if (!s) s = forward(m, n);
		if (!s) s = backward(m, n);
	}
	if (s) return s;
	if (final_loss) CUDA_TRY(cudaMemcpyAsync(final_loss, m->d_loss + n, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
	if (f) CUDA_TRY(cudaMemcpyAsync(status, m->d_corr + 2 * FUSED_STEPS, sizeof status, cudaMemcpyDeviceToHost, m->stream));
	CUDA_TRY(cudaStreamSynchronize(m->stream));
	CUDA_TRY(cudaGetLastError());
	return fused_check(m, status, t0);
}

extern "C" jn_status jn_mlp_predict(jn_mlp *m, const float *x, int n, float *y)
{
	if (!m || !x || !y || n < 1) return jn_fail(JN_ERR_INVALID, "bad argument");
	jn_status s = load(m, x, NULL, n);
	size_t smem;
	int grid;
	unsigned int status[2] = { 0, 0 };
	const int64_t t0 = m->t;
	fused_kernel f = short_pass(m, n, 0) ? NULL : fused_for(m, n, &smem, &grid);
	if (!s) s = f ? fused_run(m, f, smem, grid, n, 0, 0, 0.0f, 0, 2) : forward(m, n);
	if (s) return s;
	CUDA_TRY(cudaMemcpyAsync(y, m->d_y, (size_t)n * m->nout * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
	if (f) CUDA_TRY(cudaMemcpyAsync(status, m->d_corr + 2 * FUSED_STEPS, sizeof status, cudaMemcpyDeviceToHost, m->stream));
	CUDA_TRY(cudaStreamSynchronize(m->stream));
	return fused_check(m, status, t0);
}


/* ------------------------------------------------------------------ */
/* warm start: reduced basis of solver snapshots + MLP coordinates      */
/* ------------------------------------------------------------------ */
#define WT 256

/* out[row] = A_row . V_row with A_row = A + row * lda, V_row = V + row * ldv
 * (ldv = 0: one vector for all rows); one CTA per row, fixed order */
__global__ void __launch_bounds__(WT) ws_dots(const double *__restrict__ A, int64_t lda, const double *__restrict__ V,
					      int64_t ldv, int64_t dim, double *__restrict__ out)
{
	__shared__ double sh[WT];
	const double *a = A + (int64_t)blockIdx.x * lda, *v = V + (int64_t)blockIdx.x * ldv;
	double s = 0.0;
	for (int64_t i = threadIdx.x; i < dim; i += WT) s = fma(a[i], v[i], s);
	s = jn_block_sum(s, sh);
	if (threadIdx.x == 0) out[blockIdx.x] = s;
}

/* out = sum_{r < nrows} coef[r] A_r (coef on the device), or out -= it when sub */
__global__ void ws_combine(const double *__restrict__ A, int64_t lda, int nrows, const double *__restrict__ coef,
			   int64_t dim, double *__restrict__ out, int sub)
{
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += (int64_t)gridDim.x * blockDim.x) {
		double s = 0.0;
		for (int r = 0; r < nrows; r++) s = fma(coef[r], A[(int64_t)r * lda + i], s);
		out[i] = sub ? out[i] - s : s;
	}
}

/* row = blockIdx.y: A_row *= 1 / sqrt(nrm2[row]) */
__global__ void ws_scale(double *__restrict__ A, int64_t lda, const double *__restrict__ nrm2, int64_t dim)
{
	double *a = A + (int64_t)blockIdx.y * lda;
	const double inv = 1.0 / sqrt(nrm2[blockIdx.y]);
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += (int64_t)gridDim.x * blockDim.x)
		a[i] *= inv;
}

/* sample s = blockIdx.y: out_s = sum_j coef[s][j] Q_j + noise * r */
__global__ void ws_expand(const double *__restrict__ Q, int k, const double *__restrict__ coef,
			  const double *__restrict__ r, double noise, int64_t dim, double *__restrict__ out)
{
	const int s = blockIdx.y;
	const double *c = coef + (int64_t)s * k;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += (int64_t)gridDim.x * blockDim.x) {
		double v = noise * r[i];
		for (int j = 0; j < k; j++) v = fma(c[j], Q[(int64_t)j * dim + i], v);
		out[(int64_t)s * dim + i] = v;
	}
}

struct jn_warm_start {
	int64_t dim;
	int nc, k;
	double noise;
	double *mean, *scale;   /* input standardisation (host, nc) */
	jn_mlp *mlp;
	double *d_Q;            /* reduced basis, k x dim, orthonormal */
	double *d_r;            /* the default start vector, normalised */
};

extern "C" void jn_default_start_vector(int64_t dim, double *out)
{
	/* SplitMix64 stream, uniform in [-0.5, 0.5) */
	uint64_t z = 0x9E3779B97F4A7C15ull;
	for (int64_t e = 0; e < dim; e++) {
		z += 0x9E3779B97F4A7C15ull;
		uint64_t v = z;
		v = (v ^ (v >> 30)) * 0xBF58476D1CE4E5B9ull;
		v = (v ^ (v >> 27)) * 0x94D049BB133111EBull;
		v ^= v >> 31;
		out[e] = (double)(v >> 11) * 0x1.0p-53 - 0.5;
	}
}

extern "C" void jn_warm_start_destroy(jn_warm_start *w)
{
	if (!w) return;
	jn_mlp_destroy(w->mlp);
	cudaFree(w->d_Q);
	cudaFree(w->d_r);
	free(w->mean);
	free(w->scale);
	free(w);
}

static int grid_for(int64_t dim)
{
	int64_t g = (dim + 255) / 256;
	return (int)(g < 1 ? 1 : g > 256 ? 256 : g);
}

extern "C" jn_status jn_warm_start_fit(const jn_warm_start_options *o, int64_t dim, int nc, int S, const double *cpl,
				       int nv, const double *const *eig, jn_warm_start **out, float *final_loss)
{
	if (!o || !cpl || !eig || !out) return jn_fail(JN_ERR_INVALID, "null argument");
	*out = NULL;
	const int hidden = o->hidden > 0 ? o->hidden : 128;
	int k = o->basis_size > 0 ? o->basis_size : 32;
	const int steps = o->train_steps > 0 ? o->train_steps : 3000;
	const float lr = o->learning_rate > 0 ? o->learning_rate : 1e-3f;
	if (dim < 1 || nc < 1 || nc > 1024 || S < 1 || S > 2048 || nv < 1 || o->noise < 0)
		return jn_fail(JN_ERR_INVALID, "warm start: need dim >= 1, 1..1024 couplings, 1..2048 samples, "
					       "num_vectors >= 1, noise >= 0");
	if (k > S) k = S;
	if (k > 1024) k = 1024;
	for (int s = 0; s < S; s++)
		if (!eig[s]) return jn_fail(JN_ERR_INVALID, "eigenvectors[%d] is NULL", s);
	jn_warm_start *w = (jn_warm_start *)calloc(1, sizeof *w);
	w->dim = dim;
	w->nc = nc;
	w->noise = o->noise > 0 ? o->noise : 0.01;
	w->mean = (double *)calloc(nc, sizeof(double));
	w->scale = (double *)calloc(nc, sizeof(double));
	jn_status st = JN_OK;
	double *d_E = NULL, *d_U = NULL, *d_c = NULL, *d_d = NULL;
	double *hr = (double *)malloc(dim * sizeof(double)), *hd = (double *)malloc(S * sizeof(double));
	double *T = (double *)calloc((size_t)S * k, sizeof(double)), *res = (double *)malloc(S * sizeof(double));
	char *used = (char *)calloc(S, 1);
	cudaStream_t q = NULL;
	if (cudaMalloc((void **)&w->d_r, dim * sizeof(double)) != cudaSuccess ||
	    cudaMalloc((void **)&w->d_Q, (size_t)k * dim * sizeof(double)) != cudaSuccess ||
	    cudaMalloc((void **)&d_E, (size_t)nv * dim * sizeof(double)) != cudaSuccess ||
	    cudaMalloc((void **)&d_U, (size_t)S * dim * sizeof(double)) != cudaSuccess ||
	    cudaMalloc((void **)&d_c, (size_t)(S > nv ? S : nv) * sizeof(double) + (size_t)k * sizeof(double)) != cudaSuccess ||
	    cudaMalloc((void **)&d_d, (size_t)(S > k ? S : k) * sizeof(double)) != cudaSuccess)
		st = jn_fail(JN_ERR_NOMEM, "warm start: device buffers for %d samples of dimension %lld", S, (long long)dim);
	if (!st) st = jn_mlp_create(nc, hidden, k, o->seed, &w->mlp);
	if (!st) q = w->mlp->stream;
	const int g = grid_for(dim);
	/* r / |r| */
	if (!st) {
		jn_default_start_vector(dim, hr);
		double n2 = 0.0;
		for (int64_t i = 0; i < dim; i++) n2 += hr[i] * hr[i];
		const double inv = 1.0 / sqrt(n2);
		for (int64_t i = 0; i < dim; i++) hr[i] *= inv;
		if (cudaMemcpy(w->d_r, hr, dim * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
			st = jn_fail(JN_ERR_CUDA, "warm start: upload");
	}
	/* u_s = sum_e v_e (v_e . r), normalised */
	for (int s = 0; s < S && !st; s++) {
		if (cudaMemcpyAsync(d_E, eig[s], (size_t)nv * dim * sizeof(double), cudaMemcpyHostToDevice, q) != cudaSuccess) {
			st = jn_fail(JN_ERR_CUDA, "warm start: upload of snapshot %d", s);
			break;
		}
		ws_dots<<<nv, WT, 0, q>>>(d_E, dim, w->d_r, 0, dim, d_c);
		ws_combine<<<g, 256, 0, q>>>(d_E, dim, nv, d_c, dim, d_U + (size_t)s * dim, 0);
		/* the staging buffer is reused by the next sample's copy */
		if (cudaStreamSynchronize(q) != cudaSuccess) st = jn_fail(JN_ERR_CUDA, "warm start: snapshot %d", s);
	}
	if (!st) {
		ws_dots<<<S, WT, 0, q>>>(d_U, dim, d_U, dim, dim, d_d);
		if (cudaMemcpyAsync(hd, d_d, S * sizeof(double), cudaMemcpyDeviceToHost, q) != cudaSuccess ||
		    cudaStreamSynchronize(q) != cudaSuccess)
			st = jn_fail(JN_ERR_CUDA, "warm start: snapshot norms");
		for (int s = 0; s < S && !st; s++)
			if (!(hd[s] > 0.0) || !isfinite(hd[s]))
				st = jn_fail(JN_ERR_INVALID, "warm start: snapshot %d has no component along the start vector", s);
		if (!st) ws_scale<<<dim3(g, S), 256, 0, q>>>(d_U, dim, d_d, dim);
	}
	/* greedy reduced basis: the snapshot with the largest residual, CGS2 */
	for (int s = 0; s < S; s++) res[s] = 1.0;
	int kk = 0;
	for (int j = 0; j < k && !st; j++) {
		int best = -1;
		for (int s = 0; s < S; s++)
			if (!used[s] && (best < 0 || res[s] > res[best])) best = s;
		if (best < 0 || res[best] < 1e-12) break;  /* residual norm below 1e-6 */
		used[best] = 1;
		double *qj = w->d_Q + (size_t)j * dim;
		cudaMemcpyAsync(qj, d_U + (size_t)best * dim, dim * sizeof(double), cudaMemcpyDeviceToDevice, q);
		for (int pass = 0; pass < 2 && j > 0; pass++) {
			ws_dots<<<j, WT, 0, q>>>(w->d_Q, dim, qj, 0, dim, d_c);
			ws_combine<<<g, 256, 0, q>>>(w->d_Q, dim, j, d_c, dim, qj, 1);
		}
		ws_dots<<<1, WT, 0, q>>>(qj, dim, qj, 0, dim, d_c);
		ws_scale<<<dim3(g, 1), 256, 0, q>>>(qj, dim, d_c, dim);
		ws_dots<<<S, WT, 0, q>>>(d_U, dim, qj, 0, dim, d_d);
		if (cudaMemcpyAsync(hd, d_d, S * sizeof(double), cudaMemcpyDeviceToHost, q) != cudaSuccess ||
		    cudaStreamSynchronize(q) != cudaSuccess) {
			st = jn_fail(JN_ERR_CUDA, "warm start: reduced basis");
			break;
		}
		for (int s = 0; s < S; s++) {
			T[(size_t)s * k + j] = hd[s];
			res[s] -= hd[s] * hd[s];
		}
		kk = j + 1;
	}
	if (!st && kk < 1) st = jn_fail(JN_ERR_INVALID, "warm start: the snapshots span nothing");
	/* a rank-deficient snapshot set gives a smaller basis: rebuild the MLP with kk outputs */
	if (!st && kk < k) {
		jn_mlp_destroy(w->mlp);
		w->mlp = NULL;
		st = jn_mlp_create(nc, hidden, kk, o->seed, &w->mlp);
	}
	w->k = kk;
	/* train on standardised couplings */
	float *X = NULL, *Y = NULL;
	if (!st) {
		for (int i = 0; i < nc; i++) {
			double m = 0.0, v = 0.0;
			for (int s = 0; s < S; s++) m += cpl[(size_t)s * nc + i];
			m /= S;
			for (int s = 0; s < S; s++) v += (cpl[(size_t)s * nc + i] - m) * (cpl[(size_t)s * nc + i] - m);
			v = sqrt(v / S);
			w->mean[i] = m;
			w->scale[i] = v > 1e-12 ? 1.0 / v : 1.0;
		}
		X = (float *)malloc((size_t)S * nc * sizeof(float));
		Y = (float *)malloc((size_t)S * kk * sizeof(float));
		for (int s = 0; s < S; s++) {
			for (int i = 0; i < nc; i++) X[(size_t)s * nc + i] = (float)((cpl[(size_t)s * nc + i] - w->mean[i]) * w->scale[i]);
			for (int j = 0; j < kk; j++) Y[(size_t)s * kk + j] = (float)T[(size_t)s * k + j];
		}
		st = jn_mlp_train(w->mlp, X, Y, S, steps, lr, final_loss);
	}
	free(X); free(Y);
	cudaFree(d_E); cudaFree(d_U); cudaFree(d_c); cudaFree(d_d);
	free(hr); free(hd); free(T); free(res); free(used);
	if (st) {
		jn_warm_start_destroy(w);
		return st;
	}
	*out = w;
	return JN_OK;
}

extern "C" jn_status jn_warm_start_vectors(jn_warm_start *w, int n, const double *cpl, double *const *vec)
{
	if (!w || !cpl || !vec || n < 1) return jn_fail(JN_ERR_INVALID, "bad argument");
	const int nc = w->nc, k = w->k;
	const int64_t dim = w->dim;
	float *X = (float *)malloc((size_t)n * nc * sizeof(float)), *Y = (float *)malloc((size_t)n * k * sizeof(float));
	double *C = (double *)malloc((size_t)n * k * sizeof(double));
	for (int s = 0; s < n; s++)
		for (int i = 0; i < nc; i++) X[(size_t)s * nc + i] = (float)((cpl[(size_t)s * nc + i] - w->mean[i]) * w->scale[i]);
	jn_status st = jn_mlp_predict(w->mlp, X, n, Y);
	/* unit coordinates: |Q y| = |y| for an orthonormal basis */
	for (int s = 0; s < n && !st; s++) {
		double n2 = 0.0;
		for (int j = 0; j < k; j++) n2 += (double)Y[(size_t)s * k + j] * Y[(size_t)s * k + j];
		const double inv = n2 > 0.0 ? 1.0 / sqrt(n2) : 0.0;
		for (int j = 0; j < k; j++) C[(size_t)s * k + j] = Y[(size_t)s * k + j] * inv;
	}
	double *d_C = NULL, *d_o = NULL;
	cudaStream_t q = w->mlp->stream;
	if (!st && (cudaMalloc((void **)&d_C, (size_t)n * k * sizeof(double)) != cudaSuccess ||
		    cudaMalloc((void **)&d_o, (size_t)n * dim * sizeof(double)) != cudaSuccess))
		st = jn_fail(JN_ERR_NOMEM, "warm start: %d vectors of dimension %lld", n, (long long)dim);
	if (!st && cudaMemcpyAsync(d_C, C, (size_t)n * k * sizeof(double), cudaMemcpyHostToDevice, q) != cudaSuccess)
		st = jn_fail(JN_ERR_CUDA, "warm start: upload");
	if (!st) {
		ws_expand<<<dim3(grid_for(dim), n), 256, 0, q>>>(w->d_Q, k, d_C, w->d_r, w->noise, dim, d_o);
		if (cudaGetLastError() != cudaSuccess) st = jn_fail(JN_ERR_CUDA, "warm start: expansion launch");
	}
	for (int s = 0; s < n && !st; s++)
		if (vec[s] && cudaMemcpyAsync(vec[s], d_o + (size_t)s * dim, dim * sizeof(double), cudaMemcpyDeviceToHost, q) !=
				      cudaSuccess)
			st = jn_fail(JN_ERR_CUDA, "warm start: copy of vector %d", s);
	if (!st && cudaStreamSynchronize(q) != cudaSuccess) st = jn_fail(JN_ERR_CUDA, "warm start: expansion");
	cudaFree(d_C);
	cudaFree(d_o);
	free(X); free(Y); free(C);
	return st;
}

extern "C" int jn_warm_start_basis_size(const jn_warm_start *w) { return w ? w->k : 0; }

extern "C" jn_status jn_warm_start_basis(const jn_warm_start *w, double *basis)
{
	if (!w || !basis) return jn_fail(JN_ERR_INVALID, "null argument");
	CUDA_TRY(cudaMemcpy(basis, w->d_Q, (size_t)w->k * w->dim * sizeof(double), cudaMemcpyDeviceToHost));
	return JN_OK;
}
