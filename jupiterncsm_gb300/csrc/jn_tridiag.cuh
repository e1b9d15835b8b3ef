/*
 * jn_tridiag.cuh — device routines for the symmetric tridiagonal
 * eigenproblem of Lanczos (diagonal a[0..n), off-diagonal b[0..n-1)),
 * shared by the single solve (jn_lanczos.cu) and the batched solve
 * (jn_batch.cu).  They replace LAPACK dsteqr in the reference
 * (src/Bacchus/diagonalization/diagonalization.c:16-68).
 *
 * What bounds them: GB300's FP64 pipe, one warp instruction in 64 cycles on
 * an SM sub-partition however few lanes take part (measured; dependent and
 * independent multiply-adds alike), and one division is about ten of them
 * (641 cycles measured for a - b/x).  So the serial chains hold no division:
 * Sturm counts come from the leading principal minors
 *     p_i = (a_i - x) p_{i-1} - b_{i-1}^2 p_{i-2}
 * (three FP64 instructions a step; the exponents are kept in range by integer
 * work every eighth step), taken from both ends of the matrix at once by two
 * warps, and an eigenvector from the leading and trailing
 * minors at the eigenvalue, joined where their product is largest (the
 * twisted factorisation, in minors instead of quotients).  The quotient form
 * of the counts and inverse iteration by an LU factorisation with divisions
 * in its chain took 380 and 230 us for 11 pairs at n = 45 (SM clock 2.07
 * GHz).
 */
#ifndef JN_TRIDIAG_CUH
#define JN_TRIDIAG_CUH

#include <stdint.h>

/* doubles of scratch one warp needs for n rows: the staged matrix and the
 * work space of one vector */
#define JN_TRI_VECTOR_DOUBLES(n) (8 * (size_t)(n) + 8)
/* rows up to which that scratch is taken in shared memory (204 KB) */
#define JN_TRI_SMEM_ROWS 3192
#define JN_TRI_SMEM(n) (JN_TRI_VECTOR_DOUBLES(n) * sizeof(double))

/* bits of the unbiased exponent field; 0 for zero and subnormals */
__device__ __forceinline__ int jn_expo(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

/* v 2^-k by the exponent field, flushed to zero below the normal range */
__device__ __forceinline__ double jn_shift_expo(double v, int k)
{
	const int e = jn_expo(v);
	if (e == 0 || e - k <= 0) return 0.0;
	return __hiloint2double(__double2hiint(v) - k * 0x100000, __double2loint(v));
}

/* bring the larger of p1, p2 to exponent 0 (values in [1, 2)); returns the shift */
__device__ __forceinline__ int jn_rescale(double &p1, double &p2)
{
	const int k = max(jn_expo(p1), jn_expo(p2)) - 1023;
	if (k == -1023) return 0;
	p1 = jn_shift_expo(p1, k);
	p2 = jn_shift_expo(p2, k);
	return k;
}

/* the power of two 2^k with |T| 2^k <= 1 (Gershgorin), found by one warp */
__device__ __forceinline__ double jn_tri_scale(const double *a, const double *b, int n, double *lo, double *hi)
{
	const int lane = threadIdx.x & 31;
	double l = 1e300, h = -1e300;
	for (int j = lane; j < n; j += 32) {
		const double r = (j > 0 ? fabs(b[j - 1]) : 0.0) + (j < n - 1 ? fabs(b[j]) : 0.0);
		l = fmin(l, a[j] - r);
		h = fmax(h, a[j] + r);
	}
	for (int o = 16; o; o >>= 1) {
		l = fmin(l, __shfl_xor_sync(0xffffffffu, l, o));
		h = fmax(h, __shfl_xor_sync(0xffffffffu, h, o));
	}
	const double span = fmax(fabs(l), fabs(h));
	const int e = jn_expo(span);
	const double sc = e > 1 && e < 2045 ? __hiloint2double((2045 - e) << 20, 0) : 1.0;       /* span sc in [1/2, 1) */
	*lo = l * sc - 1e-12;
	*hi = h * sc + 1e-12;
	return sc;
}

/* one warp: a sc into as, (b sc)^2 into b2; couplings below 2^-110 of the
 * span are raised to it, so that the minors cannot stay at zero (eight steps
 * of such couplings keep a minor above 2^-880).  A floor at the rounding of
 * the span, 2^-53, moves the small eigenvalues of a graded matrix: of
 * diag(2^-5i) with couplings of 2^-(5i+8), n = 14, the smallest came out 10^4 times off. */
__device__ __forceinline__ void jn_tri_stage(const double *a, const double *b, int n, double sc, double *as, double *b2)
{
	for (int j = threadIdx.x & 31; j < n; j += 32) {
		as[j] = a[j] * sc;
		const double v = j < n - 1 ? fmax(fabs(b[j]) * sc, 0x1p-110) : 0.0;
		b2[j] = v * v;
	}
	__syncwarp();
}

/* one end's minors of T - x: the last two (times 2^e), the sign changes up to
 * the last, and the signs of the last two (bit 0 and 1; a zero minor takes
 * its predecessor's sign) */
struct jn_minors {
	double last, prev;
	int e, changes, signs;
};

/* what the two warps of a pair exchange in a round */
struct jn_tri_exchange {
	jn_minors m[2][2][32];          /* [round parity][warp][lane] */
};

__device__ __forceinline__ int jn_sign_or(double v, int s) { return ((__double2hiint(v) << 1) | __double2loint(v)) != 0 ? (__double2hiint(v) >> 31) & 1 : s; }

/* `steps` minors from row `row` in direction dir (1: leading, -1: trailing) */
__device__ __forceinline__ jn_minors jn_minor_chain(const double *as, const double *b2, int row, int dir, int steps, double x)
{
	jn_minors r = { 1.0, 0.0, 0, 0, 0 };
	int s = 0, sp = 0;
	double p2 = 0.0, p1 = 1.0;
	/* the coupling to the row before: b2[row - 1] going down, b2[row] going up */
	const double *a = as + row, *c = b2 + (dir > 0 ? row - 1 : row);
	for (int i = 0; i < steps;) {
		const int stop = min(steps, i + 8);
		for (; i < stop; i++) {
			const double p = fma(a[i * dir] - x, p1, i > 0 ? -(c[i * dir] * p2) : 0.0);
			sp = s;
			s = jn_sign_or(p, s);
			r.changes += s ^ sp;
			p2 = p1;
			p1 = p;
		}
		r.e += jn_rescale(p1, p2);
	}
	r.last = p1;
	r.prev = p2;
	r.signs = s | (sp << 1);
	return r;
}

/* Number of eigenvalues below x, by two warps w = 0, 1 (the same x on lane l
 * of both): warp 0 takes the leading minors of rows 0 .. m-1, warp 1 the
 * trailing ones of rows n-1 .. m, half of the chain each, and both put them
 * together: eliminating rows 0 .. m-2 from the top and n-1 .. m from the
 * bottom leaves the pivot det / (p_{m-1} q_m) in row m-1.  pm 2^pe is
 * det(T - x). */
__device__ __forceinline__ int jn_sturm_count(const double *as, const double *b2, int n, double x, jn_tri_exchange *ex, int round,
					      double *pm, int *pe)
{
	const int w = (threadIdx.x >> 5) & 1, lane = threadIdx.x & 31, m = (n + 1) / 2;
	const jn_minors mine = w == 0 ? jn_minor_chain(as, b2, 0, 1, m, x) : jn_minor_chain(as, b2, n - 1, -1, n - m, x);
	ex->m[round & 1][w][lane] = mine;
	asm volatile("bar.sync 1, 64;" ::: "memory");
	const jn_minors p = ex->m[round & 1][0][lane], q = ex->m[round & 1][1][lane];
	/* b2[m-1] couples the halves (0 when there is one row); q.prev is 0 when the lower half is empty */
	const double det = fma(p.last, q.last, -(b2[m - 1] * (p.prev * q.prev)));
	const int sp = p.signs >> 1, sq = q.signs & 1, sd = jn_sign_or(det, sp ^ sq);
	*pm = det;
	*pe = p.e + q.e;
	return p.changes - ((p.signs ^ (p.signs >> 1)) & 1) + q.changes + (sd ^ sp ^ sq);
}

/* The i-th smallest eigenvalue of the staged matrix (in its units) by
 * multisection, two warps (see jn_sturm_count; both must call): each round
 * the lanes count at 32 points of the bracket [lo, hi].  Points are
 * equidistant until the bracket holds this
 * eigenvalue alone and det(T - x) is known at both its ends; then they lie
 * at geometric distances around the secant estimate, whose error shrinks
 * quadratically: 6 to 8 rounds in all, where equidistant points take 11.
 * A guess (the same eigenvalue of an earlier, smaller T of the solve) takes
 * the estimate's place in the first round.  The counts alone decide the
 * bracket, so a poor estimate costs a round and nothing else.  It ends at
 * 2^-54 of the span or, `exact`, of the eigenvalue where that is smaller, two or three
 * rounds later: a convergence check compares errors far above either.  Every lane returns the same value. */
__device__ __forceinline__ double jn_tri_multisect(const double *as, const double *b2, int n, int i, double lo, double hi,
						    bool exact, bool guessed, double guess, jn_tri_exchange *ex)
{
	const int lane = threadIdx.x & 31;
	int cl = 0, ch = n, el = 0, eh = 0, known = 0;          /* known: 1 det at lo, 2 det at hi */
	double pl = 0.0, ph = 0.0;
	int geo_ok = 1;
	for (int round = 0; round < 96; round++) {
		/* 2^-54 to 2^-53 of the larger end, in integer work */
		const int e2 = exact ? max(min(max(jn_expo(lo), jn_expo(hi)) - 53, 1023 - 54), 1) : 1023 - 54;
		if (!(hi - lo > __hiloint2double(e2 << 20, 0))) break;
		const double w = hi - lo;
		const int first = guessed && round == 0;
		const int geo = first || (geo_ok && known == 3 && cl == i && ch == i + 1 && pl != 0.0);
		double x;
		if (geo) {
			double c = guess;
			if (!first) {
				const int de = min(max(eh - el, -900), 900);
				const double q = fabs(ph / pl) * __hiloint2double((1023 + de) << 20, 0);
				c = lo + w / (1.0 + q);
			}
			const int k = lane < 16 ? lane : 31 - lane;
			double d = w * __hiloint2double((1023 - 1 - k - (k >> 1)) << 20, 0);
			if (k & 1) d *= 0.70710678118654752;
			x = fmin(fmax(lane < 16 ? c - d : c + d, lo), hi);
		} else {
			x = lane == 31 ? hi : lo + (double)(lane + 1) * (w * (1.0 / 32.0));
		}
		double p;
		int e;
		const int cnt = jn_sturm_count(as, b2, n, x, ex, round, &p, &e);
		const unsigned int above = __ballot_sync(0xffffffffu, cnt > i);
		const int f = above ? __ffs(above) - 1 : 32, fl = f > 0 ? f - 1 : 0, fh = f < 32 ? f : 31;
		const double nlo = __shfl_sync(0xffffffffu, x, fl), nhi = __shfl_sync(0xffffffffu, x, fh);
		const double npl = __shfl_sync(0xffffffffu, p, fl), nph = __shfl_sync(0xffffffffu, p, fh);
		const int nel = __shfl_sync(0xffffffffu, e, fl), neh = __shfl_sync(0xffffffffu, e, fh);
		const int ncl = __shfl_sync(0xffffffffu, cnt, fl), nch = __shfl_sync(0xffffffffu, cnt, fh);
		const double lo0 = lo, hi0 = hi;
		if (f > 0) { lo = nlo; pl = npl; el = nel; cl = ncl; known |= 1; }
		if (f < 32) { hi = nhi; ph = nph; eh = neh; ch = nch; known |= 2; }
		if (!(lo > lo0 || hi < hi0) && !geo) break;     /* the bracket no longer shrinks: converged */
		geo_ok = !geo || hi - lo < 0.125 * w;
	}
	return 0.5 * (lo + hi);
}

/* The unit eigenvector z[0..n) of the staged matrix for its eigenvalue x,
 * by one warp, z[0] >= 0 as diagonalization.c:55-58 makes it.  Lanes 0, 1
 * and 2 run the chains of the leading minors p_t, the trailing minors q_t
 * and the products c_t of the couplings, one shared instruction stream;
 * then, with r where |p_r q_{n-1-r}| (the r-th diagonal element of the
 * adjugate of T - x, so |z_r|^2 up to a factor) is largest,
 *     z_i / z_r = (-1)^(r-i) (p_i / c_i) / (p_r / c_r)               i <= r
 *     z_i / z_r = (-1)^(r-i) (q_{n-1-i} c_i) / (q_{n-1-r} c_r)       i >= r.
 * buf: 5 n doubles and 3 (n/8 + 1) ints: n for d, n for the couplings' roots
 * and the three chains; as and b2 are read. */
__device__ __forceinline__ double jn_split(double v, int *e)
{
	const int k = jn_expo(v);
	if (k == 0) { *e = -100000; return 0.0; }
	*e = k - 1023;
	return __hiloint2double((__double2hiint(v) & 0x800fffff) | 0x3ff00000, __double2loint(v));
}

__device__ __forceinline__ double jn_scale2(double v, int e)
{
	if (e < -1000) return 0.0;
	return v * __hiloint2double((1023 + min(e, 1000)) << 20, 0);
}

__device__ __forceinline__ void jn_tri_vector_warp(const double *as, const double *b2, int n, double x, double *z, double *buf)
{
	const int lane = threadIdx.x & 31, ne = n / 8 + 1;
	double *d = buf, *bs = d + n, *ch = bs + n;
	int *ex = (int *)(ch + 3 * (size_t)n);
	for (int j = lane; j < n; j += 32) {
		d[j] = as[j] - x;
		bs[j] = sqrt(b2[j]);
	}
	__syncwarp();
	if (lane < 3) {
		double *v = ch + (size_t)lane * n;
		int *ev = ex + lane * ne;
		double p2 = 0.0, p1 = 1.0;
		int e = 0;
		v[0] = 1.0;
		ev[0] = 0;
		for (int t = 1; t < n; t++) {
			if ((t & 7) == 0) {
				e += jn_rescale(p1, p2);
				ev[t >> 3] = e;
			}
			const double A = lane == 0 ? d[t - 1] : lane == 1 ? d[n - t] : bs[t - 1];
			const double B = lane == 2 || t < 2 ? 0.0 : lane == 0 ? b2[t - 2] : b2[n - t];
			const double p = fma(A, p1, -(B * p2));
			v[t] = p;
			p2 = p1;
			p1 = p;
		}
	}
	__syncwarp();
	const double *P = ch, *Q = ch + n, *C = ch + 2 * (size_t)n;
	const int *EP = ex, *EQ = ex + ne, *EC = ex + 2 * ne;
	/* r: the largest |p_r q_{n-1-r}| (lowest index on ties) */
	float best = -3e38f;
	int r = 0;
	for (int i = lane; i < n; i += 32) {
		int e1, e2;
		const double m1 = jn_split(P[i], &e1), m2 = jn_split(Q[n - 1 - i], &e2);
		const float key = (float)(e1 + e2 + EP[i >> 3] + EQ[(n - 1 - i) >> 3]) +
				  __log2f(fmaxf((float)fabs(m1) * (float)fabs(m2), 1e-30f));
		if (key > best) { best = key; r = i; }
	}
	for (int o = 16; o; o >>= 1) {
		const float kb = __shfl_xor_sync(0xffffffffu, best, o);
		const int rb = __shfl_xor_sync(0xffffffffu, r, o);
		if (kb > best || (kb == best && rb < r)) { best = kb; r = rb; }
	}
	int epr, eqr, ecr;
	const double pr = jn_split(P[r], &epr), qr = jn_split(Q[n - 1 - r], &eqr), cr = jn_split(C[r], &ecr);
	epr += EP[r >> 3];
	eqr += EQ[(n - 1 - r) >> 3];
	ecr += EC[r >> 3];
	const double fp = cr / pr, fq = 1.0 / (qr * cr);
	double s = 0.0;
	for (int i = lane; i < n; i += 32) {
		int em, ec;
		const double c = jn_split(C[i], &ec);
		ec += EC[i >> 3];
		double v;
		if (i <= r) {
			v = jn_split(P[i], &em) * fp / c;
			v = jn_scale2(v, em + EP[i >> 3] - ec + ecr - epr);
		} else {
			v = jn_split(Q[n - 1 - i], &em) * fq * c;
			v = jn_scale2(v, em + EQ[(n - 1 - i) >> 3] + ec - eqr - ecr);
		}
		if ((i ^ r) & 1) v = -v;
		z[i] = v;
		s = fma(v, v, s);
	}
	for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
	__syncwarp();
	double inv = 1.0 / sqrt(s);
	if (z[0] < 0.0) inv = -inv;
	__syncwarp();
	for (int i = lane; i < n; i += 32) z[i] *= inv;
	__syncwarp();
}

/* fixed-order sum over the CTA (blockDim.x a power of two, sh of blockDim.x) */
__device__ __forceinline__ double jn_block_sum(double v, double *sh)
{
	const int t = threadIdx.x;
	sh[t] = v;
	__syncthreads();
	for (int s = blockDim.x / 2; s > 0; s >>= 1) {
		if (t < s) sh[t] += sh[t + s];
		__syncthreads();
	}
	double r = sh[0];
	__syncthreads();
	return r;
}

/* modified Gram-Schmidt among `want` vectors of length n (rows of Z), by one
 * CTA: repairs the vectors of close eigenvalues.  Each finished vector is
 * taken out of all later ones at once, a warp per vector, which are the
 * operations of the vector-by-vector order with one CTA barrier a vector. */
__device__ __forceinline__ void jn_tri_mgs(double *Z, int ldz, int n, int want)
{
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
	for (int i = 0; i < want; i++) {
		double *zi = Z + (int64_t)i * ldz;
		if (warp == 0) {
			double s = 0.0;
			for (int t = lane; t < n; t += 32) s = fma(zi[t], zi[t], s);
			for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
			double inv = 1.0 / sqrt(s);
			if (zi[0] < 0.0) inv = -inv;
			__syncwarp();
			for (int t = lane; t < n; t += 32) zi[t] *= inv;
		}
		__syncthreads();
		for (int j = i + 1 + warp; j < want; j += nwarps) {
			double *zj = Z + (int64_t)j * ldz;
			double s = 0.0;
			for (int t = lane; t < n; t += 32) s = fma(zj[t], zi[t], s);
			for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
			for (int t = lane; t < n; t += 32) zj[t] -= s * zi[t];
		}
		__syncthreads();
	}
}

#endif
