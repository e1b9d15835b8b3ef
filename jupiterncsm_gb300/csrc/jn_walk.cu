/*
 * jn_walk.cu — the walk engine (engine 5): the index-list product with the
 * contributions summed in registers before they reach memory (host plan in
 * jn_walk.c, layout in jn_problem.h).
 *
 * Semantics are the reference Minerva kernels'
 * (src/Minerva/matrix_vector_multiplication/matrix_vector_multiplication.c:
 * n list :20-77, p list :79-132, n x p lists :134-210, off-diagonal
 * transposes :212-462, |M| < 1e-12 skip of single-species terms :52-53).
 *
 * GB300 organisation.  A warp task is 32 lane chunks (up to U = 8, 4 or 2
 * entries of one walk each: one destination column; a walk's entries are
 * dealt to its lanes in turn) times the rows of a piece.  The rows are
 * grouped by their connection index: a group reads one contiguous row of its
 * matrix-element block (of its transposed copy for proton walks), so a lane
 * gathers the coefficients of its chunk from that row once per group,
 * through L1, and reuses them for every row of the group.  Warps take tasks
 * from a counter, so the tasks in flight are a narrow window of the plan's
 * order, which keeps the instructions that share a block together: L2 serves
 * each element to all of them.  For each row the lane gathers its chunk's x
 * values, sums the U products in registers, rounds the sum once to the
 * 64-bit fixed-point unit and adds it into its own slot (destination row,
 * lane) in shared memory: no atomics, no bank conflicts.  After the task a
 * lane sums the slots of one walk and gives one global add per
 * (destination row, walk).  A CTA is one warp, so the register file alone
 * sets how many warps an SM holds.
 *
 * Arithmetic (the template parameter MODE):
 *   32  FP32 coefficients and x, fused multiply-adds in entry order;
 *   64  FP64 coefficients and x, fused multiply-adds (GB300's FP64 pipe is
 *       narrow: this mode is bound by it);
 *   1   exact integers: coefficients and x as 52-bit fixed-point integers
 *       (each matrix-element block scaled to its own max|M|, x to max|x|)
 *       split into a signed high part (28 bits) and a low part (24 bits);
 *       c x = ch xh 2^48 + (ch xl + cl xh) 2^24 + cl xl, summed over the
 *       chunk in two 64-bit registers with three 32 x 32 -> 64-bit integer
 *       multiply-adds per contribution (cl xl < 2^48 is dropped), and the
 *       sum rounded once to the nearest output unit.  This is the FP64-grade
 *       product: its inputs keep 52 bits against their block's max|c| and
 *       against max|x|, every
 *       sum is exact, and it runs on the integer pipe.
 * Every row sum is rounded once, at a place fixed by the plan, and the
 * rounded sums are added as integers: the result is bit-identical from run
 * to run and independent of the grid.
 */
#include "jn_internal.h"
#include "jn_fixed.cuh"
#include "jn_pdl.cuh"

#include <type_traits>

#define WALK_WARPS 1     /* one warp a CTA: the register file alone sets how many an SM holds */
#define WALK_THREADS (WALK_WARPS * 32)
#define WALK_PITCH 33    /* words of a slot row: lanes on different rows of one column hit different banks */
#define WALK_SLOTS (JN_WALK_RS * WALK_PITCH)    /* per warp: one 64-bit slot per (destination row, lane) */
#define WALK_SMEM ((size_t)WALK_WARPS * (WALK_SLOTS * sizeof(unsigned long long) + 32 * sizeof(uint32_t)))

static_assert(sizeof(jn_wtask_t) == 16 && sizeof(jn_wpiece_t) == 32, "tasks are read as one uint4, pieces as two");

/* exponent of the 52-bit fixed-point x: |x| 2^Sx < 2^52 for the bound max|x| in xmax_bits */
__device__ __forceinline__ int walk_x_exponent(unsigned int xmax_bits)
{
	if (!(xmax_bits & 0x7fffffffu)) return 0;
	return 52 - ((int)((xmax_bits >> 23) & 0xff) - 126);
}

/* The output unit 2^-S and, for the integer path, the shift of a row sum
 * A 2^48 + B 2^24 (in units of 2^-(Sc + Sx)) down to it: S is the usual
 * fixed-point exponent (|y| 2^S < 2^62), lowered where needed so that the
 * shift is at least 49 bits (48 + sh, sh >= 1). */
__device__ __forceinline__ void walk_scales(unsigned int xmax_bits, double abs_bound, int Sc, int mode, int *S, int *sh)
{
	int s = fixed_exponent(xmax_bits, abs_bound), k = 0;
	if (mode == 1) {
		const int Sx = walk_x_exponent(xmax_bits);
		if (Sc + Sx - s < 49) s = Sc + Sx - 49;
		k = Sc + Sx - s - 48;
		if (k > 63) k = 63;
	}
	*S = s;
	*sh = k;
}

template <int MODE> struct WalkT;
template <> struct WalkT<32> { typedef float C; typedef float X; };
template <> struct WalkT<64> { typedef double C; typedef double X; };
template <> struct WalkT<1> { typedef int2 C; typedef int2 X; };

/* the sum of one row over a lane's chunk, rounded once to a 64-bit integer in output units */
template <int MODE, int U>
__device__ __forceinline__ long long walk_row(const typename WalkT<MODE>::C *c, const typename WalkT<MODE>::X *xv, uint32_t row,
					      int sh, float scalef, double scale)
{
	long long v;
	if constexpr (MODE == 1) {
		long long A = 0, B = 0;
#pragma unroll
		for (int u = 0; u < U; u++) {
			A += (long long)c[u].x * xv[u].x;
			B += (long long)c[u].x * xv[u].y;
			B += (long long)c[u].y * xv[u].x;
		}
		/* A 2^48 + B 2^24 rounded to the nearest multiple of 2^(48 + sh), sh >= 1
		   (ties up), then given the row's sign */
		const long long q = A + (B >> 24), m = (long long)((int)row >> 31);
		v = (((q + (1ll << (sh - 1))) >> sh) ^ m) - m;
	} else if constexpr (MODE == 32) {
		float acc = 0.0f;
#pragma unroll
		for (int u = 0; u < U; u++) acc = __fmaf_rn(c[u], xv[u], acc);
		v = __float2ll_rn(acc * ((row >> 31) ? -scalef : scalef));
	} else {
		double acc = 0.0;
#pragma unroll
		for (int u = 0; u < U; u++) acc = __fma_rn(c[u], xv[u], acc);
		v = __double2ll_rn(acc * ((row >> 31) ? -scale : scale));
	}
	return v;
}

/* the coefficient of lane entry u from its raw element and the lane's
 * multipliers (2 bits per entry, a two's complement: +1, -1, or 0 for
 * padding) */
template <int MODE>
__device__ __forceinline__ typename WalkT<MODE>::C walk_coef(typename WalkT<MODE>::C v, uint32_t mul, int u)
{
	const int m = (int)(mul << (30 - 2 * u)) >> 30;
	if constexpr (MODE == 1) {
		return make_int2(v.x * m, v.y * m);
	} else {
		if (!m) v = 0;
		return m < 0 ? -v : v;
	}
}

/* one warp task with chunks of U entries (see the file comment).  Rows are
 * taken two at a time, so that two rows' gathers of x are in flight at once;
 * up to two words after a group's last row are read ahead (the plan keeps
 * JN_WALK_ROW_SPARE zero words after the last row) and not used.  A group's first row pair issues its
 * gathers of x before the coefficients (loaded at the top of the group) are
 * first used, so the two latencies overlap. */
template <int MODE, int U>
__device__ __forceinline__ void walk_task(const uint4 ta, const uint4 pa, const uint4 pb, const uint32_t *__restrict__ lanes,
					  const uint32_t *__restrict__ walks, const uint32_t *__restrict__ rows,
					  const uint32_t *__restrict__ rdst, const uint32_t *__restrict__ groups,
					  const uint8_t *__restrict__ gshift, const typename WalkT<MODE>::C *__restrict__ elem,
					  const typename WalkT<MODE>::X *__restrict__ x, const typename WalkT<MODE>::X *__restrict__ xt,
					  unsigned long long *__restrict__ gacc, unsigned long long *__restrict__ slots, uint32_t *__restrict__ tab, int lane,
					  int sh, float scalef, double scale)
{
	typedef typename WalkT<MODE>::C C;
	typedef typename WalkT<MODE>::X X;
	const int src_off = (int)pa.x, dst_off = (int)pa.y, stride = (int)pa.z, Nn_dst = (int)pa.w;
	const int rs = (int)(pb.w & 0xffu), wp = (int)((pb.w >> 8) & 1u), ngroups = (int)(pb.w >> 9);
	const uint32_t *__restrict__ L = lanes + ta.y + lane;
	const uint32_t head = __ldg(L);
	const int ws = (int)(head & 0xffffu);
	const uint32_t mul = head >> 16;
	int off[U];
#pragma unroll
	for (int k = 0; k < U / 2; k++) {
		const uint32_t w = __ldg(L + (1 + k) * 32);
		off[2 * k] = (int)(w & 0xffffu);
		off[2 * k + 1] = (int)(w >> 16);
	}
	/* proton walks read the transposed view: a row's entries index one row of the source block */
	const X *__restrict__ xs = (wp ? xt : x) + src_off;
	int j = (int)pb.x;
	uint32_t row = __ldg(rows + j);
	for (int g = 0; g < ngroups; g++) {
		const C *__restrict__ er = elem + __ldg(groups + (int)pb.z + g);
		/* the integer path scales each block by its own exponent: its rows shift further */
		int shg = sh;
		if constexpr (MODE == 1) {
			shg += (int)__ldg(gshift + (int)pb.z + g);
			if (shg > 62) shg = 62;
		}
		C c[U];
#pragma unroll
		for (int u = 0; u < U; u++) c[u] = __ldg(er + (__ldg(L + (1 + U / 2 + u) * 32) & 0x3fffffffu));
		for (bool first = true;; first = false) {
			/* this row and the next one of the group (if any) */
			const uint32_t row2 = __ldg(rows + j + 1);
			const bool two = !(row & JN_WALK_GROUP_END);
			const X *__restrict__ xb = xs + (int)(row & 0xffffu) * stride;
			const X *__restrict__ xb2 = xs + (two ? (int)(row2 & 0xffffu) * stride : 0);
			X xv[U], xv2[U];
#pragma unroll
			for (int u = 0; u < U; u++) xv[u] = __ldg(xb + off[u]);
#pragma unroll
			for (int u = 0; u < U; u++) xv2[u] = __ldg(xb2 + off[u]);
			const uint32_t next = __ldg(rows + j + 2);
			/* the coefficients' multipliers, applied after this pair's gathers are issued */
			if (first) {
#pragma unroll
				for (int u = 0; u < U; u++) c[u] = walk_coef<MODE>(c[u], mul, u);
			}
			slots[(int)((row >> 16) & 31u) * WALK_PITCH + lane] += (unsigned long long)walk_row<MODE, U>(c, xv, row, shg, scalef, scale);
			if (two)
				slots[(int)((row2 >> 16) & 31u) * WALK_PITCH + lane] +=
					(unsigned long long)walk_row<MODE, U>(c, xv2, row2, shg, scalef, scale);
			const bool end = !two || (row2 & JN_WALK_GROUP_END);
			j += two ? 2 : 1;
			row = two ? next : row2;
			if (end) break;
		}
	}
	__syncwarp();
	/* The task's slots into the global accumulator; slots are left zero.  The
	   lanes of one walk are a run of neighbouring lanes: a lane takes a
	   (destination row, walk) pair and sums its run's slots, so the pairs of
	   all rows share a warp's instructions (a segmented shuffle sum, row by
	   row, takes about three times as many, and as many passes of the
	   shared-memory pipe, which bounds the large products: 6Li Nmax 6 3492 ->
	   3419 us, FP32 2794 -> 2657; 7Li Nmax 4 with 3NF 88.2 -> 84.2; 4He Nmax 4
	   16.4 -> 14.4).  Lanes past the view's chunks carry walk slot 0 after a
	   higher one and hold zeros. */
	const int ws_prev = __shfl_up_sync(0xffffffffu, ws, 1);     /* every lane takes part */
	const unsigned int starts = __ballot_sync(0xffffffffu, lane == 0 || ws != ws_prev);
	const unsigned int after = lane == 31 ? 0u : starts >> (lane + 1);
	const int end = after ? lane + __ffs(after) : 32;
	if (lane == 0 || ws > ws_prev) tab[ws] = __ldg(walks + ta.z + ws) | ((uint32_t)lane << 16) | ((uint32_t)end << 21);
	const uint32_t dr_of = lane < rs ? __ldg(rdst + (int)pb.y + lane) : 0u;
	__syncwarp();
	const int nw = (int)(ta.w & 0xffu), total = rs * nw;
	const float per = __frcp_rn((float)nw);
	for (int p0 = 0; p0 < total; p0 += 32) {
		const int p = p0 + lane;
		int r = (int)(((float)p + 0.5f) * per);         /* p / nw: p < 512 */
		const int w = p - r * nw;
		const uint32_t dr = __shfl_sync(0xffffffffu, dr_of, r & 31);
		if (p < total) {
			const uint32_t t = tab[w];
			unsigned long long v = 0ull, *slot = slots + r * WALK_PITCH;
			const int last = (int)(t >> 21);
			for (int q = (int)((t >> 16) & 31u); q < last; q++) {
				v += slot[q];
				slot[q] = 0ull;
			}
			const int dw = (int)(t & 0xffffu);
			if (v) atomicAdd(gacc + dst_off + (wp ? dw * Nn_dst + (int)dr : (int)dr * Nn_dst + dw), v);
		}
	}
	__syncwarp();
}

/* FP32: 32 warps an SM (64 registers); the 64-bit paths 28 (the integer path
 * uses 68).  With 64 registers and 32 warps the integer path's warps have less
 * L1 each: 6Li Nmax 6 takes 3524 us, not 3420; with 20 warps 3726. */
template <int MODE, bool MANY>
__global__ void __launch_bounds__(WALK_THREADS, MODE == 32 ? 32 : 28)
	jn_walk_kernel(const uint4 *__restrict__ tasks, const uint4 *__restrict__ pieces, const uint32_t *__restrict__ lanes,
		       const uint32_t *__restrict__ walks, const uint32_t *__restrict__ rows,
		       const uint32_t *__restrict__ rdst, const uint32_t *__restrict__ groups,
		       const uint8_t *__restrict__ gshift, const typename WalkT<MODE>::C *__restrict__ elem,
		       const typename WalkT<MODE>::X *__restrict__ x, const typename WalkT<MODE>::X *__restrict__ xt,
		       unsigned long long *__restrict__ gacc, unsigned int *__restrict__ ctrl, long long ntasks,
		       double abs_bound, int Sc, unsigned int nvec, long long dim)
{
	extern __shared__ unsigned long long wslots[];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	unsigned long long *slots = wslots + warp * WALK_SLOTS;
	uint32_t *tab = (uint32_t *)(wslots + WALK_WARPS * WALK_SLOTS) + warp * 32;
	for (int i = lane; i < WALK_SLOTS; i += 32) slots[i] = 0ull;
	__syncwarp();
	/* from here on the kernel reads what the x view kernel wrote */
	pdl_wait();
	pdl_trigger();
	ctrl = pdl_after(ctrl);
	x = pdl_after(x);
	xt = pdl_after(xt);
	/* MANY: lane v keeps the scales of vector v */
	int S, sh;
	walk_scales(ctrl[MANY && (unsigned int)lane < nvec ? 2 * lane : 0], abs_bound, Sc, MODE, &S, &sh);
	const int Sv = S, shv = sh;
	float scalef = MODE == 32 ? __int_as_float((127 + (S < -126 ? -126 : (S > 127 ? 127 : S))) << 23) : 0.0f;
	double scale = MODE == 64 ? ldexp(1.0, S) : 0.0;
	const typename WalkT<MODE>::X *x0 = x, *xt0 = xt;
	unsigned long long *gacc0 = gacc;
	/* warps take the next task from a counter (ctrl[1], zero at launch), so
	   the tasks in flight stay a window of about two tasks per warp: the
	   instructions that read one matrix-element block run together and L2
	   serves the block's rows to all of them (a fixed assignment lets warps
	   drift apart by many tasks, and the window with them) */
	unsigned int t = 0, tn = 0;
	if (lane == 0) t = atomicAdd(ctrl + 1, 1u);
	t = __shfl_sync(0xffffffffu, t, 0);
	for (; (long long)t < ntasks; t = __shfl_sync(0xffffffffu, tn, 0)) {
		if (lane == 0) tn = atomicAdd(ctrl + 1, 1u);
		if (MANY) {
			const unsigned int q = t / nvec, v = t - q * nvec;
			t = q;
			x = x0 + v * dim;
			xt = xt0 + v * dim;
			gacc = gacc0 + v * dim;
			sh = __shfl_sync(0xffffffffu, shv, v);
			if (MODE != 1) S = __shfl_sync(0xffffffffu, Sv, v);
			if (MODE == 32) scalef = __int_as_float((127 + (S < -126 ? -126 : (S > 127 ? 127 : S))) << 23);
			if (MODE == 64) scale = ldexp(1.0, S);
		}
		const uint4 ta = __ldg(tasks + t);
		const uint4 pa = __ldg(pieces + 2 * ta.x), pb = __ldg(pieces + 2 * ta.x + 1);
		const uint32_t U = (ta.w >> 8) & 0xffu;
		if (U == 8)
			walk_task<MODE, 8>(ta, pa, pb, lanes, walks, rows, rdst, groups, gshift, elem, x, xt, gacc, slots, tab, lane, sh,
					       scalef, scale);
		else if (U == 4)
			walk_task<MODE, 4>(ta, pa, pb, lanes, walks, rows, rdst, groups, gshift, elem, x, xt, gacc, slots, tab, lane, sh,
					       scalef, scale);
		else
			walk_task<MODE, 2>(ta, pa, pb, lanes, walks, rows, rdst, groups, gshift, elem, x, xt, gacc, slots, tab, lane, sh,
					       scalef, scale);
	}
}

/* x as 52-bit fixed-point integers {high 28 bits (signed), low 24 bits} */
__device__ __forceinline__ int2 walk_xsplit(double v, double s)
{
	const long long q = __double2ll_rn(v * s);
	return make_int2((int)(q >> 24), (int)(q & 0xffffff));
}

/* max|x| of each vector (blockIdx.y) as an FP32 bound into ctrl[2 v], zero before */
__global__ void jn_walk_max_kernel(const double *__restrict__ x, int64_t n, unsigned int *__restrict__ ctrl)
{
	x += blockIdx.y * n;
	float m = 0.0f;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
		m = fmaxf(m, (float)fabs(x[i]) * 1.0000002f);   /* round-up margin of the FP32 conversion */
	for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
	if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(ctrl + 2 * blockIdx.y, __float_as_uint(m));
}

/* the x views the walk kernel reads in the arithmetic MODE, of each vector
 * (blockIdx.y): the converted copy of x (split integers, MODE 1; FP32, MODE
 * 32), and, where proton walks exist (perm != NULL), the transposed view
 * xT[i] = x[perm[i]] */
template <int MODE>
__global__ void jn_walk_xview_kernel(const double *__restrict__ x, const int32_t *__restrict__ perm,
				     typename WalkT<MODE>::X *__restrict__ xv, typename WalkT<MODE>::X *__restrict__ xt, int64_t n,
				     const unsigned int *__restrict__ ctrl)
{
	pdl_wait();
	pdl_trigger();
	x += blockIdx.y * n;
	if (MODE != 64) xv += blockIdx.y * n;
	if (perm) xt += blockIdx.y * n;
	ctrl = pdl_after(ctrl) + 2 * blockIdx.y;
	const double s = MODE == 1 ? ldexp(1.0, walk_x_exponent(ctrl[0])) : 1.0;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		if constexpr (MODE == 1) {
			xv[i] = walk_xsplit(x[i], s);
			if (perm) xt[i] = walk_xsplit(__ldg(x + __ldg(perm + i)), s);
		} else {
			if (MODE == 32) xv[i] = (typename WalkT<MODE>::X)x[i];
			if (perm) xt[i] = (typename WalkT<MODE>::X)__ldg(x + __ldg(perm + i));
		}
	}
}

/* Everything before the walk kernel in one launch, for a small basis: every
 * CTA takes max|x| over the whole of x and converts its
 * own states (of vector blockIdx.y); its first CTA sets ctrl[0], and the task
 * counter ctrl[1] to zero.
 * Bound by latency; it stands for a memset and two kernels.  Up to 12 288
 * states reading x once per CTA costs less than those launches: products back
 * to back at D = 59 / 952 / 7916 / 10 817 take 7.8 / 13.5 / 93.3 / 82.4 us with
 * it and 13.3 / 17.5 / 96.0 / 85.2 us without; at 15 764 the two took the same.
 * (A cluster of eight CTAs that meets over the maximum was slower than either at
 * all of these.) */
#define WALK_SMALL_THREADS 256
#define WALK_SMALL_DIM 12288
template <int MODE>
__global__ void __launch_bounds__(WALK_SMALL_THREADS)
	jn_walk_small_x_kernel(const double *__restrict__ x, const int32_t *__restrict__ perm,
			       typename WalkT<MODE>::X *__restrict__ xv, typename WalkT<MODE>::X *__restrict__ xt, int n,
			       unsigned int *__restrict__ ctrl)
{
	typedef typename WalkT<MODE>::X X;
	__shared__ unsigned long long wmax[WALK_SMALL_THREADS / 32];
	/* x, and the product before this one, which reads the views and ctrl */
	pdl_wait();
	pdl_trigger();
	x = pdl_after(x);
	x += (int64_t)blockIdx.y * n;
	if (MODE != 64) xv += (int64_t)blockIdx.y * n;
	if (perm) xt += (int64_t)blockIdx.y * n;
	ctrl += 2 * blockIdx.y;
	const int i = blockIdx.x * WALK_SMALL_THREADS + threadIdx.x;
	const double v = i < n ? x[i] : 0.0, t = perm && i < n ? x[__ldg(perm + i)] : 0.0;
	const unsigned int bound = x_bound_of_all<WALK_SMALL_THREADS>(x, n, wmax);
	if (i == 0) {
		ctrl[0] = bound;
		ctrl[1] = 0u;
	}
	if (i >= n) return;
	if constexpr (MODE == 1) {
		const double s = ldexp(1.0, walk_x_exponent(bound));
		xv[i] = walk_xsplit(v, s);
		if (perm) xt[i] = walk_xsplit(t, s);
	} else {
		if (MODE == 32) xv[i] = (X)v;
		if (perm) xt[i] = (X)t;
	}
}

/* y (+)= acc 2^-S with the integer path's unit; the accumulator is cleared */
__global__ void jn_walk_finalize_kernel(unsigned long long *__restrict__ gacc, double *__restrict__ y, int64_t n,
					const unsigned int *__restrict__ ctrl, double abs_bound, int Sc, int mode,
					int accumulate)
{
	pdl_wait();
	pdl_trigger();
	ctrl = pdl_after(ctrl) + 2 * blockIdx.y;
	gacc = pdl_after(gacc) + blockIdx.y * n;
	y += blockIdx.y * n;
	int S, sh;
	walk_scales(ctrl[0], abs_bound, Sc, mode, &S, &sh);
	const double unit = ldexp(1.0, -S);
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		const double v = (double)(long long)gacc[i] * unit;
		y[i] = accumulate ? y[i] + v : v;
		gacc[i] = 0ull;
	}
}

/* the walk element array in FP32 */
__global__ void jn_walk_f32_kernel(const double *__restrict__ a, int64_t n, float *__restrict__ out)
{
	for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
		out[e] = (float)a[e];
}

/* ------------------------------------------------------------------ */
/* host side                                                           */
/* ------------------------------------------------------------------ */
template <typename T>
static jn_status wupload(T **dst, const void *src, size_t n)
{
	size_t bytes = (n ? n : 1) * sizeof(T);
	cudaError_t e = cudaMalloc((void **)dst, bytes);
	if (e != cudaSuccess) return jn_fail(JN_ERR_NOMEM, "cudaMalloc(%zu bytes) failed: %s", bytes, cudaGetErrorString(e));
	if (n && src) {
		e = cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice);
		if (e != cudaSuccess) return jn_fail(JN_ERR_CUDA, "cudaMemcpy failed: %s", cudaGetErrorString(e));
	}
	return JN_OK;
}

static int walk_mode(const jn_ctx *c) { return c->precision == 32 ? 32 : (c->walk_fp64 ? 64 : 1); }
static int walk_slot(int mode) { return mode == 32 ? 0 : (mode == 64 ? 1 : 2); }

void jn_walk_release(jn_ctx *c)
{
	cudaFree(c->d_wtasks); cudaFree(c->d_wpieces); cudaFree(c->d_wlanes); cudaFree(c->d_wwalks); cudaFree(c->d_wrows);
	cudaFree(c->d_wmany);
	c->d_wmany = NULL;
	c->walk_many = 0;
	cudaFree(c->d_wrdst); cudaFree(c->d_wgroups); cudaFree(c->d_wgshift); cudaFree(c->d_wx); cudaFree(c->d_wxt);
	cudaFree(c->d_wxperm);
	for (int i = 0; i < 3; i++) cudaFree(c->d_welem[i]);
	c->d_wtasks = NULL; c->d_wpieces = NULL; c->d_wlanes = NULL; c->d_wwalks = NULL; c->d_wrows = NULL;
	c->d_wrdst = NULL; c->d_wgroups = NULL; c->d_wgshift = NULL; c->d_wx = NULL; c->d_wxt = NULL; c->d_wxperm = NULL;
	for (int i = 0; i < 3; i++) c->d_welem[i] = NULL;
	c->walk_ready = 0;
}

void jn_walk_invalidate(jn_ctx *c)
{
	for (int i = 0; i < 3; i++) {
		cudaFree(c->d_welem[i]);
		c->d_welem[i] = NULL;
	}
}

jn_status jn_walk_setup(jn_ctx *c)
{
	if (c->walk_ready) return JN_OK;
	jn_plan_t *p = &c->plan;
	char err[512] = { 0 };
	if (jn_walk_build(p, err, sizeof err)) return jn_fail(JN_ERR_NOMEM, "walk plan: %s", err);
	jn_status s;
	if ((s = wupload(&c->d_wtasks, p->wtasks, (size_t)p->nwtasks)) ||
	    (s = wupload(&c->d_wpieces, p->wpieces, (size_t)p->nwpieces * 2)) ||
	    (s = wupload(&c->d_wlanes, p->wlanes, (size_t)p->n_wlanes)) ||
	    (s = wupload(&c->d_wwalks, p->wwalks, (size_t)p->n_wwalks)) ||
	    (s = wupload(&c->d_wrows, p->wrows, (size_t)p->n_wrows + JN_WALK_ROW_SPARE)) ||
	    (s = wupload(&c->d_wrdst, p->wrdst, (size_t)p->n_wrdst)) ||
	    (s = wupload(&c->d_wgroups, p->wgroups, (size_t)p->n_wgroups)) ||
	    (s = wupload(&c->d_wx, (const void *)NULL, (size_t)(p->dim ? p->dim : 1))) ||
	    (p->wxt && (s = wupload(&c->d_wxt, (const void *)NULL, (size_t)(p->dim ? p->dim : 1)))) ||
	    (p->wxt && (s = wupload(&c->d_wxperm, p->wxperm, (size_t)p->dim)))) {
		jn_walk_release(c);
		return s;
	}
	int per[3] = { 0, 0, 0 };
	cudaError_t e = cudaFuncSetAttribute(jn_walk_kernel<32, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WALK_SMEM);
	if (e == cudaSuccess) e = cudaFuncSetAttribute(jn_walk_kernel<64, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WALK_SMEM);
	if (e == cudaSuccess) e = cudaFuncSetAttribute(jn_walk_kernel<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WALK_SMEM);
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[0], jn_walk_kernel<32, false>, WALK_THREADS, WALK_SMEM);
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[1], jn_walk_kernel<64, false>, WALK_THREADS, WALK_SMEM);
	if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per[2], jn_walk_kernel<1, false>, WALK_THREADS, WALK_SMEM);
	if (e != cudaSuccess) {
		jn_walk_release(c);
		return jn_fail(JN_ERR_CUDA, "walk kernel set-up: %s", cudaGetErrorString(e));
	}
	for (int i = 0; i < 3; i++) {
		if (per[i] < 1) {
			jn_walk_release(c);
			return jn_fail(JN_ERR_CUDA, "the walk kernel does not fit on an SM");
		}
		c->walk_per_sm[i] = per[i];
	}
	c->walk_ready = 1;
	return JN_OK;
}

/* the walk element array of the current matrix elements for one arithmetic
 * (built on first use and after the matrix elements change): FP64
 * (arithmetic 64) from the FP64 array built on the host; FP32, converted on
 * the device from the FP64 copy when that exists, else on the host; the
 * integer path's split 52-bit values with their per-group shifts, formed on
 * the host straight from the plan's elements (only these reach the device
 * for it) */
static jn_status walk_elements(jn_ctx *c, int mode)
{
	const jn_plan_t *p = &c->plan;
	const int slot = walk_slot(mode);
	if (c->d_welem[slot]) return JN_OK;
	const int64_t n = p->n_wme;
	if (mode == 32 && c->d_welem[1]) {
		const double *a = (const double *)c->d_welem[1];
		cudaError_t e = cudaMalloc(&c->d_welem[0], (size_t)(n ? n : 1) * sizeof(float));
		if (e != cudaSuccess) {
			c->d_welem[0] = NULL;
			return jn_fail(JN_ERR_NOMEM, "cudaMalloc of %lld walk matrix elements: %s", (long long)n, cudaGetErrorString(e));
		}
		const int g = (int)(n / 256 + 1 < 4096 ? n / 256 + 1 : 4096);
		if (n) jn_walk_f32_kernel<<<g, 256, 0, c->stream>>>(a, n, (float *)c->d_welem[0]);
		e = cudaGetLastError();
		if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
		if (e != cudaSuccess) return jn_fail(JN_ERR_CUDA, "walk matrix elements: %s", cudaGetErrorString(e));
		return JN_OK;
	}
	/* the exact integer path splits the plan's elements directly; the FP64
	   and FP32 paths start from the FP64 walk element array */
	double *h = NULL;
	if (mode == 64 || mode == 32) {
		h = (double *)malloc((size_t)(n ? n : 1) * sizeof(double));
		if (!h) return jn_fail(JN_ERR_NOMEM, "out of host memory for %lld walk matrix elements", (long long)n);
		jn_walk_elements(p, p->me, h);
	}
	jn_status s = JN_OK;
	if (mode == 64) {
		double *d = NULL;
		if (!(s = wupload(&d, h, (size_t)n))) c->d_welem[1] = d;
	} else if (mode == 32) {
		float *f = (float *)malloc((size_t)(n ? n : 1) * sizeof(float));
		if (!f) {
			s = jn_fail(JN_ERR_NOMEM, "out of host memory for %lld walk matrix elements", (long long)n);
		} else {
			for (int64_t e = 0; e < n; e++) f[e] = (float)h[e];
			float *d = NULL;
			if (!(s = wupload(&d, f, (size_t)n))) c->d_welem[0] = d;
			free(f);
		}
	} else {
		/* per-block exponents: every block keeps 52 bits against its own max|A| */
		int32_t *sp = (int32_t *)malloc((size_t)(n ? n : 1) * 2 * sizeof(int32_t));
		uint8_t *gs = (uint8_t *)malloc((size_t)(p->n_wgroups ? p->n_wgroups : 1));
		if (!sp || !gs) {
			s = jn_fail(JN_ERR_NOMEM, "out of host memory for %lld walk matrix elements", (long long)n);
		} else {
			jn_walk_int_elements(p, p->me, sp, gs, &c->walk_sc);
			int2 *d = NULL;
			s = wupload(&d, sp, (size_t)n);
			if (!s) {
				c->d_welem[2] = d;
				cudaFree(c->d_wgshift);
				c->d_wgshift = NULL;
				s = wupload(&c->d_wgshift, gs, (size_t)p->n_wgroups);
			}
		}
		free(sp); free(gs);
	}
	free(h);
	return s;
}

/* nvec products Y (+)= H X (vectors of length D one after another) on the
 * walk engine: max|x| and the converted copies of x, the walk kernel, the
 * conversion of the accumulators into Y.  Each kernel is set up while the one
 * before it still runs (jn_pdl.cuh): without that overlap the gaps and
 * launches cost 6 us more at any size, and where the first kernel overlaps the
 * product before it as well (up to WALK_SMALL_DIM states), 2 us more: products
 * back to back at D = 59 / 952 / 10 817 / 7916 10.3 / 14.4 / 84.1 / 96.6 -> 8.1 /
 * 13.1 / 82.1 / 93.9 us.  xv, xt, gacc and ctrl hold nvec
 * vectors (control words 2 v). */
template <int MODE>
static jn_status walk_launch(jn_ctx *c, const double *d_x, double *d_y, int nvec, int accumulate, int2 *wx, int2 *wxt,
			     unsigned long long *gacc, unsigned int *ctrl, cudaStream_t st, cudaEvent_t pre, cudaEvent_t mid)
{
	typedef typename WalkT<MODE>::X X;
	typedef typename WalkT<MODE>::C C;
	const jn_plan_t *p = &c->plan;
	const int slot = walk_slot(MODE), Sc = MODE == 1 ? c->walk_sc : 0;
	const int32_t *perm = p->wxt ? c->d_wxperm : NULL;
	X *xv = MODE == 64 ? NULL : (X *)wx, *xt = (X *)wxt;
	int g = (int)((p->dim + 255) / 256);
	if (g > 1024) g = 1024;
	/* what precedes the walk kernel on the stream is a kernel of this product
	   unless an event was recorded in between */
	int overlap = 1;
	if (p->dim <= WALK_SMALL_DIM) {
		/* overlaps whatever kernel precedes it on the stream (back to back that
		   is the last product's conversion), except in a capture, where what
		   precedes it may be no kernel */
		cudaStreamCaptureStatus cs = cudaStreamCaptureStatusActive;
		const int first = !pre && cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone;
		pdl_launch(first, jn_walk_small_x_kernel<MODE>,
			   dim3((unsigned int)((p->dim + WALK_SMALL_THREADS - 1) / WALK_SMALL_THREADS), nvec), WALK_SMALL_THREADS, 0, st,
			   d_x, perm, xv, xt, (int)p->dim, ctrl);
	} else {
		CUDA_TRY(cudaMemsetAsync(ctrl, 0, (size_t)nvec * 2 * sizeof(unsigned int), st));
		jn_walk_max_kernel<<<dim3(g, nvec), 256, 0, st>>>(d_x, p->dim, ctrl);
		if (perm || MODE != 64)
			pdl_launch(1, jn_walk_xview_kernel<MODE>, dim3(g, nvec), 256, 0, st, d_x, perm, xv, xt, p->dim, ctrl);
	}
	if (pre) {
		cudaEventRecord(pre, st);
		overlap = 0;
	}
	if (p->nwtasks) {
		const long long n = p->nwtasks * nvec;
		const int resident = c->num_sms * c->walk_per_sm[slot];
		const dim3 grid(n < resident ? (unsigned int)n : (unsigned int)resident);
		pdl_launch(overlap, nvec > 1 ? jn_walk_kernel<MODE, true> : jn_walk_kernel<MODE, false>, grid, WALK_THREADS, WALK_SMEM, st,
			   (const uint4 *)c->d_wtasks, (const uint4 *)c->d_wpieces, c->d_wlanes, c->d_wwalks, c->d_wrows, c->d_wrdst,
			   c->d_wgroups, MODE == 1 ? c->d_wgshift : NULL, (const C *)c->d_welem[slot],
			   MODE == 64 ? (const X *)d_x : (const X *)wx, (const X *)wxt, gacc, ctrl, n, p->abs_bound, Sc,
			   (unsigned int)nvec, p->dim);
		overlap = 1;
	}
	if (mid) {
		cudaEventRecord(mid, st);
		overlap = 0;
	}
	pdl_launch(overlap, jn_walk_finalize_kernel, dim3(g, nvec), 256, 0, st, gacc, d_y, p->dim, ctrl, p->abs_bound, Sc, MODE,
		   accumulate);
	cudaError_t e = cudaGetLastError();
	if (e != cudaSuccess) return jn_fail(JN_ERR_CUDA, "walk product launch: %s", cudaGetErrorString(e));
	return JN_OK;
}

int jn_walk_kernels(const jn_ctx *c)
{
	const jn_plan_t *p = &c->plan;
	if (!p->dim) return 0;
	/* before the walk kernel: all in one, or max|x| and, where there is one to make, the converted copy of x */
	const int views = p->dim <= WALK_SMALL_DIM ? 1 : p->wxt || walk_mode(c) != 64 ? 2 : 1;
	return views + (p->nwtasks > 0) + 1;
}

/* y (+)= H x on the walk engine */
jn_status jn_enqueue_walk(jn_ctx *c, const double *d_x, double *d_y, int accumulate, cudaStream_t st, cudaEvent_t pre,
			  cudaEvent_t mid)
{
	jn_status s = jn_walk_setup(c);
	const int mode = walk_mode(c);
	if (!s) s = walk_elements(c, mode);
	if (s) return s;
	if (!c->plan.dim) {
		if (pre) cudaEventRecord(pre, st);
		if (mid) cudaEventRecord(mid, st);
		return JN_OK;
	}
	return (mode == 1 ? walk_launch<1> : mode == 32 ? walk_launch<32> : walk_launch<64>)(
		c, d_x, d_y, 1, accumulate, c->d_wx, c->d_wxt, c->d_gacc, c->d_xmax, st, pre, mid);
}

/* Y = H X for n vectors of length D one after another.  On the walk engine up
 * to WALK_MANY of them share one launch: their tasks form one list (the same
 * task of all vectors in a row, so the lists and matrix elements are read
 * from the caches for all but the first), without the ramps and the gaps of
 * separate products.  The workspace, at most WALK_MANY_BYTES, stays with the
 * context; without it, and on the other engines, the products run one by one.
 * The bits are the single products'.  Measured (subspace matrices of 32
 * vectors, one by one -> together): D = 952 1.15 -> 0.23 ms, 15 764 (6Li Nmax
 * 4, 2NF) 2.33 -> 1.39 ms, 10 817 (7Li Nmax 4, 2NF + 3NF) 4.5 -> 2.86 ms; two
 * vectors at D = 186 894 take as long either way (7.7 ms), where the walk
 * kernel is bound by the L1 data banks (82 %). */
#define WALK_MANY 32
#define WALK_MANY_BYTES ((size_t)64 << 20)
jn_status jn_enqueue_many(jn_ctx *c, const double *d_x, double *d_y, int n, cudaStream_t st)
{
	const int64_t D = c->plan.dim;
	jn_status s = JN_OK;
	if (c->engine == 5 && n > 1 && D > 0) {
		s = jn_walk_setup(c);
		const int mode = walk_mode(c);
		if (!s) s = walk_elements(c, mode);
		if (s) return s;
		const size_t per = (size_t)D * (2 * sizeof(int2) + sizeof(unsigned long long));
		int cap = (int)(WALK_MANY_BYTES / per < WALK_MANY ? WALK_MANY_BYTES / per : WALK_MANY);
		/* the task counter is one 32-bit word */
		while (cap > 1 && c->plan.nwtasks * cap + (1 << 20) > 0xffffffffll) cap--;
		if (cap > n) cap = n;
		if (cap > 1 && c->walk_many < cap) {
			cudaFree(c->d_wmany);
			c->walk_many = 0;
			c->d_wmany = NULL;
			const size_t bytes = (size_t)cap * (per + 2 * sizeof(unsigned int));
			if (cudaMalloc(&c->d_wmany, bytes) == cudaSuccess && cudaMemsetAsync(c->d_wmany, 0, bytes, st) == cudaSuccess) {
				c->walk_many = cap;
			} else {
				cudaGetLastError();
				cap = 1;
			}
		}
		if (cap > 1) {
			const int parts = (n + cap - 1) / cap;
			unsigned long long *gacc = (unsigned long long *)c->d_wmany;
			int2 *wx = (int2 *)(gacc + (size_t)c->walk_many * D), *wxt = wx + (size_t)c->walk_many * D;
			unsigned int *ctrl = (unsigned int *)(wxt + (size_t)c->walk_many * D);
			for (int k = 0; k < parts && !s; k++) {
				const int i0 = (int)((int64_t)n * k / parts), i1 = (int)((int64_t)n * (k + 1) / parts);
				s = (mode == 1 ? walk_launch<1> : mode == 32 ? walk_launch<32> : walk_launch<64>)(
					c, d_x + i0 * D, d_y + i0 * D, i1 - i0, 0, wx, wxt, gacc, ctrl, st, NULL, NULL);
			}
			return s;
		}
	}
	for (int i = 0; i < n && !s; i++) s = jn_launch_matvec(c, d_x + i * D, d_y + i * D, 0, st);
	return s;
}

/* ------------------------------------------------------------------ */
/* batched products over instances of several bases                    */
/* ------------------------------------------------------------------ */
/* One instance of a batched walk product: its basis's plan (on the
 * basis's context), its own walk element arrays, x views, accumulator and
 * scale bound, and its range of the batch's task list (128 bytes). */
struct jn_walk_inst {
	const uint4 *tasks, *pieces;
	const uint32_t *lanes, *walks, *rows, *rdst, *groups;
	const double *elem64;
	const float *elem32;
	float *x32;                     /* FP32 copy of the instance's x (arithmetic 32) */
	void *xt;                       /* transposed view of x in the arithmetic's type, NULL without proton walks */
	const int32_t *perm;            /* position in x of each element of that view */
	unsigned long long *gacc;
	int64_t dim;
	double abs_bound;               /* |H x| <= abs_bound max|x| */
	uint32_t task0, ntasks;         /* the instance's tasks in the batch's list */
};
static_assert(sizeof(jn_walk_inst) == 128, "one descriptor is 128 bytes");

struct jn_walk_batch {
	int B;
	jn_walk_inst *h, *d;
	uint32_t *d_task0;              /* B + 1 task offsets */
	uint32_t total;
	unsigned int *d_ctrl;           /* max|x| bits of instance i at 2 i; the task counter at 2 B */
	int num_sms, per_sm[2];         /* resident one-warp CTAs an SM: arithmetic 32, 64 */
	int has32;
};

/* max|x_i| into ctrl[2 i], the FP32 copy of x_i (MODE 32) and the
 * transposed view; x_i = src + i src_ld + (*sel) sel_ld */
template <int MODE>
__global__ void jn_walk_multi_prep_kernel(const jn_walk_inst *__restrict__ I, const double *__restrict__ src,
					  int64_t src_ld, const int *__restrict__ sel, int64_t sel_ld,
					  unsigned int *__restrict__ ctrl, const int *__restrict__ active)
{
	const int inst = blockIdx.y;
	if (active && !active[inst]) return;
	const jn_walk_inst d = I[inst];
	const double *x = src + inst * src_ld + (sel ? (int64_t)(*sel) * sel_ld : 0);
	typedef typename WalkT<MODE>::X X;
	X *xt = (X *)d.xt;
	float m = 0.0f;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < d.dim; i += (int64_t)gridDim.x * blockDim.x) {
		const double v = x[i];
		if (MODE == 32) d.x32[i] = (float)v;
		if (xt) xt[i] = (X)x[d.perm[i]];
		m = fmaxf(m, (float)fabs(v) * 1.0000002f);     /* round-up margin of the FP32 conversion */
	}
	for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
	if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(ctrl + 2 * inst, __float_as_uint(m));
}

/* All instances' tasks in one persistent launch: a warp takes task t of
 * the batch's list from the counter, finds its instance (binary search of
 * the task offsets) and runs it with that instance's plan, elements, x
 * views and accumulator. */
template <int MODE>
__global__ void __launch_bounds__(WALK_THREADS, MODE == 32 ? 32 : 28)
	jn_walk_multi_kernel(const jn_walk_inst *__restrict__ I, const uint32_t *__restrict__ task0, int B, uint32_t total,
			     unsigned int *__restrict__ ctrl, const double *__restrict__ src, int64_t src_ld,
			     const int *__restrict__ sel, int64_t sel_ld, const int *__restrict__ active)
{
	extern __shared__ unsigned long long wslots[];
	const int lane = threadIdx.x & 31;
	unsigned long long *slots = wslots;
	uint32_t *tab = (uint32_t *)(wslots + WALK_SLOTS);
	for (int i = lane; i < WALK_SLOTS; i += 32) slots[i] = 0ull;
	__syncwarp();
	const int64_t k = sel ? (int64_t)(*sel) : 0;
	unsigned int t = 0, tn = 0;
	if (lane == 0) t = atomicAdd(ctrl + 2 * B, 1u);
	t = __shfl_sync(0xffffffffu, t, 0);
	for (; t < total; t = __shfl_sync(0xffffffffu, tn, 0)) {
		if (lane == 0) tn = atomicAdd(ctrl + 2 * B, 1u);
		int lo = 0, hi = B;             /* task0[lo] <= t < task0[hi] */
		while (hi - lo > 1) {
			const int mid = (lo + hi) >> 1;
			if (__ldg(task0 + mid) <= t) lo = mid;
			else hi = mid;
		}
		if (active && !active[lo]) continue;
		const jn_walk_inst *d = I + lo;
		int S, sh;
		walk_scales(ctrl[2 * lo], d->abs_bound, 0, MODE, &S, &sh);
		const float scalef = MODE == 32 ? __int_as_float((127 + (S < -126 ? -126 : (S > 127 ? 127 : S))) << 23) : 0.0f;
		const double scale = MODE == 64 ? ldexp(1.0, S) : 0.0;
		typedef typename WalkT<MODE>::C C;
		typedef typename WalkT<MODE>::X X;
		const C *elem;
		const X *x;
		if constexpr (MODE == 32) {
			elem = d->elem32;
			x = d->x32;
		} else {
			elem = d->elem64;
			x = src + lo * src_ld + k * sel_ld;
		}
		const X *xt = (const X *)d->xt;
		const uint4 ta = __ldg(d->tasks + (t - __ldg(task0 + lo)));
		const uint4 pa = __ldg(d->pieces + 2 * ta.x), pb = __ldg(d->pieces + 2 * ta.x + 1);
		const uint32_t U = (ta.w >> 8) & 0xffu;
		if (U == 8)
			walk_task<MODE, 8>(ta, pa, pb, d->lanes, d->walks, d->rows, d->rdst, d->groups, NULL, elem, x, xt, d->gacc,
					   slots, tab, lane, sh, scalef, scale);
		else if (U == 4)
			walk_task<MODE, 4>(ta, pa, pb, d->lanes, d->walks, d->rows, d->rdst, d->groups, NULL, elem, x, xt, d->gacc,
					   slots, tab, lane, sh, scalef, scale);
		else
			walk_task<MODE, 2>(ta, pa, pb, d->lanes, d->walks, d->rows, d->rdst, d->groups, NULL, elem, x, xt, d->gacc,
					   slots, tab, lane, sh, scalef, scale);
	}
}

/* y_i = acc_i 2^-S_i (y + i y_ld); the accumulators are cleared */
template <int MODE>
__global__ void jn_walk_multi_finalize_kernel(const jn_walk_inst *__restrict__ I, double *__restrict__ y, int64_t y_ld,
					      const unsigned int *__restrict__ ctrl, const int *__restrict__ active)
{
	const int inst = blockIdx.y;
	if (active && !active[inst]) return;
	const jn_walk_inst d = I[inst];
	int S, sh;
	walk_scales(ctrl[2 * inst], d.abs_bound, 0, MODE, &S, &sh);
	const double unit = ldexp(1.0, -S);
	double *yy = y + inst * y_ld;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < d.dim; i += (int64_t)gridDim.x * blockDim.x) {
		yy[i] = (double)(long long)d.gacc[i] * unit;
		d.gacc[i] = 0ull;
	}
}

void jn_walk_batch_free(jn_walk_batch *wb)
{
	if (!wb) return;
	if (wb->h)
		for (int i = 0; i < wb->B; i++) {
			cudaFree((void *)wb->h[i].elem64);
			cudaFree((void *)wb->h[i].elem32);
			cudaFree(wb->h[i].x32);
			cudaFree(wb->h[i].xt);
			cudaFree(wb->h[i].gacc);
		}
	free(wb->h);
	cudaFree(wb->d);
	cudaFree(wb->d_task0);
	cudaFree(wb->d_ctrl);
	free(wb);
}

jn_status jn_walk_batch_create(jn_ctx *const *ctxs, const int *inst_ctx, int B, const double *const *me, int want32,
			       jn_walk_batch **out)
{
	*out = NULL;
	if (B < 1 || B > 65535) return jn_fail(JN_ERR_INVALID, "batch of %d instances", B);
	jn_walk_batch *wb = (jn_walk_batch *)calloc(1, sizeof *wb);
	if (!wb) return jn_fail(JN_ERR_NOMEM, "out of host memory");
	wb->B = B;
	wb->has32 = want32;
	wb->h = (jn_walk_inst *)calloc((size_t)B, sizeof(jn_walk_inst));
	uint32_t *task0 = (uint32_t *)malloc((size_t)(B + 1) * sizeof(uint32_t));
	jn_status s = (!wb->h || !task0) ? jn_fail(JN_ERR_NOMEM, "out of host memory") : JN_OK;
	double *hbuf = NULL;
	int64_t hcap = 0;
	uint64_t total = 0;
	for (int i = 0; i < B && !s; i++) {
		jn_ctx *c = ctxs[inst_ctx[i]];
		if ((s = jn_walk_setup(c))) break;
		const jn_plan_t *p = &c->plan;
		jn_walk_inst *d = &wb->h[i];
		d->tasks = (const uint4 *)c->d_wtasks;
		d->pieces = (const uint4 *)c->d_wpieces;
		d->lanes = c->d_wlanes;
		d->walks = c->d_wwalks;
		d->rows = c->d_wrows;
		d->rdst = c->d_wrdst;
		d->groups = c->d_wgroups;
		d->perm = p->wxt ? c->d_wxperm : NULL;
		d->dim = p->dim;
		d->abs_bound = jn_plan_abs_bound(p, me[i]);
		d->task0 = (uint32_t)total;
		d->ntasks = (uint32_t)p->nwtasks;
		task0[i] = (uint32_t)total;
		total += (uint64_t)p->nwtasks;
		if (total > 0xf0000000ull) { s = jn_fail(JN_ERR_INVALID, "the batch has too many walk tasks"); break; }
		/* the instance's walk element arrays: FP64 built on the host, FP32 converted on the device */
		const int64_t n = p->n_wme;
		if (n > hcap) {
			free(hbuf);
			hcap = n;
			hbuf = (double *)malloc((size_t)hcap * sizeof(double));
			if (!hbuf) { s = jn_fail(JN_ERR_NOMEM, "out of host memory"); break; }
		}
		if (n) jn_walk_elements(p, me[i], hbuf);
		double *e64 = NULL;
		if ((s = wupload(&e64, hbuf, (size_t)n))) break;
		d->elem64 = e64;
		if (want32) {
			float *e32 = NULL;
			if ((s = wupload(&e32, (const void *)NULL, (size_t)n))) break;
			d->elem32 = e32;
			const int g = (int)(n / 256 + 1 < 4096 ? n / 256 + 1 : 4096);
			if (n) jn_walk_f32_kernel<<<g, 256, 0, c->stream>>>(e64, n, e32);
			float *x32 = NULL;
			if ((s = wupload(&x32, (const void *)NULL, (size_t)p->dim))) break;
			d->x32 = x32;
		}
		if (p->wxt) {
			double *xt = NULL;
			if ((s = wupload(&xt, (const void *)NULL, (size_t)p->dim))) break;
			d->xt = xt;
		}
		unsigned long long *g = NULL;
		if ((s = wupload(&g, (const void *)NULL, (size_t)p->dim))) break;
		if (cudaMemset(g, 0, (size_t)(p->dim ? p->dim : 1) * sizeof(unsigned long long)) != cudaSuccess)
			s = jn_fail(JN_ERR_CUDA, "cudaMemset of a batch accumulator");
		d->gacc = g;
		if (!wb->num_sms) {
			wb->num_sms = c->num_sms;
			wb->per_sm[0] = c->walk_per_sm[0];
			wb->per_sm[1] = c->walk_per_sm[1];
		}
	}
	free(hbuf);
	if (!s) {
		task0[B] = (uint32_t)total;
		wb->total = (uint32_t)total;
		if ((s = wupload(&wb->d, wb->h, (size_t)B)) || (s = wupload(&wb->d_task0, task0, (size_t)B + 1)) ||
		    (s = wupload(&wb->d_ctrl, (const void *)NULL, (size_t)2 * B + 1)))
			;
	}
	free(task0);
	if (!s) {
		cudaError_t e = cudaFuncSetAttribute(jn_walk_multi_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
						     (int)WALK_SMEM);
		int per = 0;
		if (e == cudaSuccess) e = cudaFuncSetAttribute(jn_walk_multi_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
							       (int)WALK_SMEM);
		if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, jn_walk_multi_kernel<32>, WALK_THREADS, WALK_SMEM);
		if (e == cudaSuccess) wb->per_sm[0] = per;
		if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, jn_walk_multi_kernel<64>, WALK_THREADS, WALK_SMEM);
		if (e == cudaSuccess) wb->per_sm[1] = per;
		if (e == cudaSuccess) e = cudaDeviceSynchronize();
		if (e != cudaSuccess) s = jn_fail(JN_ERR_CUDA, "batched walk set-up: %s", cudaGetErrorString(e));
		else if (wb->per_sm[0] < 1 || wb->per_sm[1] < 1) s = jn_fail(JN_ERR_CUDA, "the batched walk kernel does not fit on an SM");
	}
	if (s) {
		jn_walk_batch_free(wb);
		return s;
	}
	*out = wb;
	return JN_OK;
}

jn_status jn_walk_batch_enqueue(jn_walk_batch *wb, int mode, const double *src, int64_t src_ld, const int *d_sel,
				int64_t sel_ld, double *y, int64_t y_ld, const int *d_active, int64_t max_dim, cudaStream_t st)
{
	if (mode != 32 && mode != 64) return jn_fail(JN_ERR_INVALID, "batched walk arithmetic %d", mode);
	if (mode == 32 && !wb->has32) return jn_fail(JN_ERR_INVALID, "the batch has no FP32 elements");
	const int B = wb->B;
	int g = (int)((max_dim + 255) / 256);
	if (g > 256) g = 256;
	if (g < 1) g = 1;
	CUDA_TRY(cudaMemsetAsync(wb->d_ctrl, 0, (size_t)(2 * B + 1) * sizeof(unsigned int), st));
	const int grid = wb->num_sms * wb->per_sm[mode == 32 ? 0 : 1];
	if (mode == 32) {
		jn_walk_multi_prep_kernel<32><<<dim3(g, B), 256, 0, st>>>(wb->d, src, src_ld, d_sel, sel_ld, wb->d_ctrl, d_active);
		if (wb->total)
			jn_walk_multi_kernel<32><<<grid, WALK_THREADS, WALK_SMEM, st>>>(wb->d, wb->d_task0, B, wb->total, wb->d_ctrl,
											 src, src_ld, d_sel, sel_ld, d_active);
		jn_walk_multi_finalize_kernel<32><<<dim3(g, B), 256, 0, st>>>(wb->d, y, y_ld, wb->d_ctrl, d_active);
	} else {
		jn_walk_multi_prep_kernel<64><<<dim3(g, B), 256, 0, st>>>(wb->d, src, src_ld, d_sel, sel_ld, wb->d_ctrl, d_active);
		if (wb->total)
			jn_walk_multi_kernel<64><<<grid, WALK_THREADS, WALK_SMEM, st>>>(wb->d, wb->d_task0, B, wb->total, wb->d_ctrl,
											 src, src_ld, d_sel, sel_ld, d_active);
		jn_walk_multi_finalize_kernel<64><<<dim3(g, B), 256, 0, st>>>(wb->d, y, y_ld, wb->d_ctrl, d_active);
	}
	cudaError_t e = cudaGetLastError();
	if (e != cudaSuccess) return jn_fail(JN_ERR_CUDA, "batched walk product launch: %s", cudaGetErrorString(e));
	return JN_OK;
}

extern "C" jn_status jn_set_walk_arithmetic(jn_ctx *c, int fp64_fma)
{
	if (!c) return jn_fail(JN_ERR_INVALID, "null argument");
	if (fp64_fma != 0 && fp64_fma != 1) return jn_fail(JN_ERR_INVALID, "walk arithmetic %d: must be 0 (exact integers) or 1 (FP64)", fp64_fma);
	c->walk_fp64 = fp64_fma;
	return JN_OK;
}

extern "C" jn_status jn_walk_stats(jn_ctx *c, double *out)
{
	if (!c || !out) return jn_fail(JN_ERR_INVALID, "null argument");
	jn_status s = jn_walk_setup(c);
	if (s) return s;
	const jn_plan_t *p = &c->plan;
	out[0] = (double)p->nwtasks;
	out[1] = (double)p->nwpieces;
	out[2] = (double)p->n_wgroups;
	out[3] = p->wvisits;
	out[4] = p->wlane_slots;
	out[5] = (double)p->n_wme;
	out[6] = (double)(c->num_sms * c->walk_per_sm[walk_slot(walk_mode(c))]);
	return JN_OK;
}
