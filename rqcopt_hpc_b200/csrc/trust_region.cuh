// FP64 device arithmetic of truncated CG and of the trust-region ratio test
// (src/trust_region.c:14-65, 159-217, 336-352): dot products and axpys with
// explicitly rounded multiplies and adds in index order (no fused multiply-add),
// the arithmetic of a sequential BLAS level-1 loop.  Shared by the single-problem
// optimiser and the batched one.
#pragma once
#include <math.h>

namespace rqc {

enum TcgStatus { TCG_CONTINUE = 0, TCG_BOUNDARY = 1, TCG_CONVERGED = 2 };

struct TcgState
{
	double rsq, stoptol, radius;
	int status;
};

struct RtrState
{
	double radius, rho, fx, fnext, maxradius, rho_trust;
	int accept;
};

__device__ inline double dot_seq(int n, const double* a, const double* b)
{
	double s = 0;
	for (int k = 0; k < n; k++) s = __dadd_rn(s, __dmul_rn(a[k], b[k]));
	return s;
}

// t > 0 with ||z + t d|| = radius (src/trust_region.c:14-65)
__device__ inline double to_boundary(int n, const double* z, const double* d, double radius)
{
	const double dsq = dot_seq(n, d, d);
	if (dsq == 0) return 0;
	const double p = __ddiv_rn(dot_seq(n, z, d), dsq);
	const double q = __ddiv_rn(__dsub_rn(dot_seq(n, z, z), __dmul_rn(radius, radius)), dsq);
	if (p == 0) return sqrt(-q);
	const double a = -__dadd_rn(p, copysign(1.0, p) * sqrt(__dsub_rn(__dmul_rn(p, p), q)));
	const double b = __ddiv_rn(q, a);
	return a <= b ? b : a;
}

// r = grad, rsq, stop tolerance, z = 0, d = -r (src/trust_region.c:161-175)
__device__ inline void tcg_init_dev(int n, const double* grad, double* r, double* d, double* z, TcgState* st,
                                    double radius, double abstol, double reltol)
{
	for (int k = 0; k < n; k++) { r[k] = grad[k]; z[k] = 0; d[k] = -grad[k]; }
	st->rsq = dot_seq(n, r, r);
	st->stoptol = fmax(abstol, reltol * sqrt(st->rsq));
	st->radius = radius;
	st->status = TCG_CONTINUE;
}

// One tCG step after Hd = H d (src/trust_region.c:181-209)
__device__ inline void tcg_step_dev(int n, double* d, const double* hd, double* z, double* r, TcgState* st)
{
	const double dhd = dot_seq(n, d, hd);
	const double t = to_boundary(n, z, d, st->radius);
	const double alpha = __ddiv_rn(st->rsq, dhd);
	if (dhd <= 0 || alpha > t) {
		for (int k = 0; k < n; k++) z[k] = __dadd_rn(z[k], __dmul_rn(t, d[k]));
		st->status = TCG_BOUNDARY;
		return;
	}
	for (int k = 0; k < n; k++) r[k] = __dadd_rn(r[k], __dmul_rn(alpha, hd[k]));
	for (int k = 0; k < n; k++) z[k] = __dadd_rn(z[k], __dmul_rn(alpha, d[k]));
	const double rsq_next = dot_seq(n, r, r);
	if (sqrt(rsq_next) <= st->stoptol) {
		st->status = TCG_CONVERGED;
		return;
	}
	const double beta = __ddiv_rn(rsq_next, st->rsq);
	for (int k = 0; k < n; k++) d[k] = __dadd_rn(__dmul_rn(beta, d[k]), -r[k]);
	st->rsq = rsq_next;
	st->status = TCG_CONTINUE;
}

// Ratio test and radius update (src/trust_region.c:336-352); st->fx, st->fnext set
__device__ inline void rtr_rho_dev(int n, const double* grad, const double* eta, const double* heta, RtrState* st,
                                   int on_boundary)
{
	const double den = __dadd_rn(dot_seq(n, grad, eta), __dmul_rn(0.5, dot_seq(n, eta, heta)));
	const double rho = __ddiv_rn(__dsub_rn(st->fnext, st->fx), den);
	if (rho < 0.25) st->radius = __dmul_rn(st->radius, 0.25);
	else if (rho > 0.75 && on_boundary) st->radius = fmin(2 * st->radius, st->maxradius);
	st->rho = rho;
	st->accept = rho > st->rho_trust;
}

// The same steps by a whole block.  What must stay in order are the additions of the dot
// products; the loads, the multiplications and the vector updates are independent.  So all
// threads fill the products of up to four dot products into shared memory and one lane each
// adds them up in index order: bit for bit the results of the single-thread forms above, whose
// chains of dependent global loads took 30-50 us at n = 288 (here 4-7 us).
constexpr int TR_THREADS = 256;
constexpr int TR_CHUNK = 1024;

struct BlockDots
{
	double prod[4][TR_CHUNK + 1];   // odd pitch: the four adding lanes read four banks
	double sum[4];
};

// w.sum[j] = dot product of a[j] and b[j], j < M
template <int M>
__device__ inline void block_dots(int n, const double* const (&a)[M], const double* const (&b)[M], BlockDots& w)
{
	double s = 0;
	for (int k0 = 0; k0 < n; k0 += TR_CHUNK) {
		const int m = min(TR_CHUNK, n - k0);
		__syncthreads();
		for (int i = threadIdx.x; i < m; i += blockDim.x)
#pragma unroll
			for (int j = 0; j < M; j++) w.prod[j][i] = __dmul_rn(a[j][k0 + i], b[j][k0 + i]);
		__syncthreads();
		if (threadIdx.x < M) {
			const double* p = w.prod[threadIdx.x];
#pragma unroll 8
			for (int i = 0; i < m; i++) s = __dadd_rn(s, p[i]);
		}
	}
	if (threadIdx.x < M) w.sum[threadIdx.x] = s;
	__syncthreads();
}

__device__ inline void tcg_init_blk(int n, const double* grad, double* r, double* d, double* z, TcgState* st,
                                    double radius, double abstol, double reltol, BlockDots& w)
{
	for (int k = threadIdx.x; k < n; k += blockDim.x) { r[k] = grad[k]; z[k] = 0; d[k] = -grad[k]; }
	block_dots<1>(n, {grad}, {grad}, w);
	if (threadIdx.x == 0) {
		st->rsq = w.sum[0];
		st->stoptol = fmax(abstol, reltol * sqrt(st->rsq));
		st->radius = radius;
		st->status = TCG_CONTINUE;
	}
	__syncthreads();
}

__device__ inline void tcg_step_blk(int n, double* d, const double* hd, double* z, double* r, TcgState* st, BlockDots& w)
{
	block_dots<4>(n, {d, d, z, z}, {hd, d, d, z}, w);
	const double dhd = w.sum[0], dsq = w.sum[1], zd = w.sum[2], zz = w.sum[3];
	const double radius = st->radius, rsq = st->rsq, stoptol = st->stoptol;
	double t = 0;
	if (dsq != 0) {
		const double p = __ddiv_rn(zd, dsq);
		const double q = __ddiv_rn(__dsub_rn(zz, __dmul_rn(radius, radius)), dsq);
		if (p == 0) {
			t = sqrt(-q);
		} else {
			const double a = -__dadd_rn(p, copysign(1.0, p) * sqrt(__dsub_rn(__dmul_rn(p, p), q)));
			const double b = __ddiv_rn(q, a);
			t = a <= b ? b : a;
		}
	}
	const double alpha = __ddiv_rn(rsq, dhd);
	__syncthreads();   // every thread has read *st and w.sum
	if (dhd <= 0 || alpha > t) {
		for (int k = threadIdx.x; k < n; k += blockDim.x) z[k] = __dadd_rn(z[k], __dmul_rn(t, d[k]));
		if (threadIdx.x == 0) st->status = TCG_BOUNDARY;
		__syncthreads();
		return;
	}
	for (int k = threadIdx.x; k < n; k += blockDim.x) {
		r[k] = __dadd_rn(r[k], __dmul_rn(alpha, hd[k]));
		z[k] = __dadd_rn(z[k], __dmul_rn(alpha, d[k]));
	}
	block_dots<1>(n, {r}, {r}, w);
	const double rsq_next = w.sum[0];
	if (sqrt(rsq_next) <= stoptol) {
		if (threadIdx.x == 0) st->status = TCG_CONVERGED;
		__syncthreads();
		return;
	}
	const double beta = __ddiv_rn(rsq_next, rsq);
	for (int k = threadIdx.x; k < n; k += blockDim.x) d[k] = __dadd_rn(__dmul_rn(beta, d[k]), -r[k]);
	if (threadIdx.x == 0) {
		st->rsq = rsq_next;
		st->status = TCG_CONTINUE;
	}
	__syncthreads();
}

__device__ inline void rtr_rho_blk(int n, const double* grad, const double* eta, const double* heta, RtrState* st,
                                   int on_boundary, BlockDots& w)
{
	block_dots<2>(n, {grad, eta}, {eta, heta}, w);
	if (threadIdx.x == 0) {
		const double den = __dadd_rn(w.sum[0], __dmul_rn(0.5, w.sum[1]));
		const double rho = __ddiv_rn(__dsub_rn(st->fnext, st->fx), den);
		if (rho < 0.25) st->radius = __dmul_rn(st->radius, 0.25);
		else if (rho > 0.75 && on_boundary) st->radius = fmin(2 * st->radius, st->maxradius);
		st->rho = rho;
		st->accept = rho > st->rho_trust;
	}
}

}  // namespace rqc
