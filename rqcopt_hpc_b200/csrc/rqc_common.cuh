// Shared device helpers: complex arithmetic on double2/float2 and the
// amplitude-group index arithmetic of a two-qubit gate.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "orbits.h"

namespace rqc {

// ---------------------------------------------------------------- complex types

template <typename T> struct cplx_t;
template <> struct cplx_t<double> { using type = double2; };
template <> struct cplx_t<float>  { using type = float2; };
template <typename T> using cplx = typename cplx_t<T>::type;

template <typename T> __host__ __device__ __forceinline__ cplx<T> mk(T re, T im) { cplx<T> z; z.x = re; z.y = im; return z; }

// a * b + c
template <typename V> __host__ __device__ __forceinline__ V cfma(V a, V b, V c)
{
	V r;
	r.x = fma(a.x, b.x, fma(-a.y, b.y, c.x));
	r.y = fma(a.x, b.y, fma(a.y, b.x, c.y));
	return r;
}
template <typename V> __host__ __device__ __forceinline__ V cmul(V a, V b)
{
	V r;
	r.x = a.x * b.x - a.y * b.y;
	r.y = a.x * b.y + a.y * b.x;
	return r;
}
template <typename V> __host__ __device__ __forceinline__ V cadd(V a, V b) { V r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename V> __host__ __device__ __forceinline__ V csub(V a, V b) { V r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
template <typename V> __host__ __device__ __forceinline__ V cneg_conj(V a) { V r; r.x = -a.x; r.y = a.y; return r; }
template <typename V> __host__ __device__ __forceinline__ V czero() { V r; r.x = 0; r.y = 0; return r; }

__device__ __forceinline__ double2 to_d(double2 a) { return a; }
__device__ __forceinline__ double2 to_d(float2 a) { return make_double2(a.x, a.y); }

// ---------------------------------------------------------------- gates as kernel arguments

// One 4x4 gate in arithmetic precision T, row-major (row = 2*b_i + b_j).
template <typename T> struct Gate4 { cplx<T> m[16]; };

// ---------------------------------------------------------------- basis columns

// Where the columns of a chunk come from.  Column c of the chunk is number b0 + c: entry of
// tab if there is one, otherwise basis state b0 + c (paired with b0 + c + pair_half if that
// is not 0).  Columns at or beyond end are zero (they add nothing to any sum).  The weights
// multiply the input of the target passes (weighted), so that phi carries them into every
// sum, all of which are linear in phi.
struct ColumnSource
{
	const BasisCol* tab = nullptr;
	int64_t b0 = 0, end = INT64_MAX, pair_half = 0;
	int weighted = 0;
};

// amplitude `row` of column c of the chunk
template <typename T>
__device__ __forceinline__ cplx<T> basis_amp(const ColumnSource& s, int64_t row, int64_t c)
{
	const int64_t k = s.b0 + c;
	cplx<T> v = mk<T>(T(0), T(0));
	if (k >= s.end) return v;
	if (s.tab) {
		const BasisCol e = s.tab[k];
		if (row == e.re) v.x = s.weighted ? (T)e.wre : T(1);
		if (row == e.im) v.y = s.weighted ? (T)e.wim : T(1);
	} else {
		if (row == k) v.x = T(1);
		if (s.pair_half != 0 && row == k + s.pair_half) v.y = T(1);
	}
	return v;
}

// amplitude `row` of U applied to (weighted) column c of the chunk, U a dense row-major 2^L x 2^L
// matrix
__device__ __forceinline__ double2 dense_amp(const double2* __restrict__ u, int L, const ColumnSource& s, int64_t row,
                                             int64_t c)
{
	const int64_t k = s.b0 + c;
	double2 v = make_double2(0, 0);
	if (k >= s.end) return v;
	const int64_t re = s.tab ? s.tab[k].re : k;
	const int64_t im = s.tab ? s.tab[k].im : (s.pair_half ? k + s.pair_half : -1);
	const double wre = s.tab ? s.tab[k].wre : 1.0, wim = s.tab ? s.tab[k].wim : 1.0;
	const double2 x = u[(row << L) + re];
	v = make_double2(wre * x.x, wre * x.y);
	if (im >= 0) {
		const double2 y = u[(row << L) + im];
		v.x -= wim * y.y;
		v.y += wim * y.x;
	}
	return v;
}

// ---------------------------------------------------------------- amplitude groups

// Wire pair of a gate acting on an L-qubit register: bit positions of the two
// wires (qubit q <-> index bit L-1-q) and the two positions sorted, for the
// insertion of zero bits into a rest index.
struct WirePair
{
	int64_t si, sj;   // strides of wire i and wire j
	int plo, phi;     // sorted bit positions
};

__host__ __device__ __forceinline__ WirePair make_pair_(int L, int i, int j)
{
	WirePair w;
	const int pi = L - 1 - i, pj = L - 1 - j;
	w.si = (int64_t)1 << pi;
	w.sj = (int64_t)1 << pj;
	w.plo = pi < pj ? pi : pj;
	w.phi = pi < pj ? pj : pi;
	return w;
}

// Base index (both wire bits zero) of the rest index r in [0, 2^(L-2)).
__host__ __device__ __forceinline__ int64_t group_base(int64_t r, const WirePair& w)
{
	const int64_t mlo = ((int64_t)1 << w.plo) - 1;
	r = ((r & ~mlo) << 1) | (r & mlo);
	const int64_t mhi = ((int64_t)1 << w.phi) - 1;
	r = ((r & ~mhi) << 1) | (r & mhi);
	return r;
}

// Offsets of the four group members in the order of the gate's row index.
__host__ __device__ __forceinline__ void group_offsets(const WirePair& w, int64_t off[4])
{
	off[0] = 0;
	off[1] = w.sj;
	off[2] = w.si;
	off[3] = w.si + w.sj;
}

// ---------------------------------------------------------------- 4x4 actions on a group

// y = G x
template <typename T>
__device__ __forceinline__ void gate_apply(const Gate4<T>& g, const cplx<T> x[4], cplx<T> y[4])
{
#pragma unroll
	for (int r = 0; r < 4; r++) {
		cplx<T> s = cmul(g.m[4*r], x[0]);
#pragma unroll
		for (int c = 1; c < 4; c++) s = cfma(g.m[4*r + c], x[c], s);
		y[r] = s;
	}
}

// y = G^T x
template <typename T>
__device__ __forceinline__ void gate_apply_t(const Gate4<T>& g, const cplx<T> x[4], cplx<T> y[4])
{
#pragma unroll
	for (int c = 0; c < 4; c++) {
		cplx<T> s = cmul(g.m[c], x[0]);
#pragma unroll
		for (int r = 1; r < 4; r++) s = cfma(g.m[4*r + c], x[r], s);
		y[c] = s;
	}
}

// y += G x
template <typename T>
__device__ __forceinline__ void gate_apply_acc(const Gate4<T>& g, const cplx<T> x[4], cplx<T> y[4])
{
#pragma unroll
	for (int r = 0; r < 4; r++) {
		cplx<T> s = y[r];
#pragma unroll
		for (int c = 0; c < 4; c++) s = cfma(g.m[4*r + c], x[c], s);
		y[r] = s;
	}
}

// y += G^T x
template <typename T>
__device__ __forceinline__ void gate_apply_t_acc(const Gate4<T>& g, const cplx<T> x[4], cplx<T> y[4])
{
#pragma unroll
	for (int c = 0; c < 4; c++) {
		cplx<T> s = y[c];
#pragma unroll
		for (int r = 0; r < 4; r++) s = cfma(g.m[4*r + c], x[r], s);
		y[c] = s;
	}
}

// acc[r][c] += a[r] * b[c]  (no conjugation)
template <typename A, typename V>
__device__ __forceinline__ void outer_acc(A acc[16], const V a[4], const V b[4])
{
#pragma unroll
	for (int r = 0; r < 4; r++)
#pragma unroll
		for (int c = 0; c < 4; c++) {
			A p;
			p.x = a[r].x * b[c].x - a[r].y * b[c].y;
			p.y = a[r].x * b[c].y + a[r].y * b[c].x;
			acc[4*r + c].x += p.x;
			acc[4*r + c].y += p.y;
		}
}

// ---------------------------------------------------------------- reductions

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}

// Compensated sum of p[b * stride], b = 0 .. n-1, by the threads of a block: the block's
// RED_GROUPS groups of NV threads take every RED_GROUPS-th term each (a serial chain over a
// few hundred blocks' partials took 50-60 us; eight chains an eighth of it), then thread v < NV
// of group 0 adds the groups' sums in order and gets the result of its own p.
constexpr int RED_GROUPS = 8;

template <int NV>
__device__ __forceinline__ double block_column_sum(const double* __restrict__ p, int n, size_t stride,
                                                   double (*red)[NV])
{
	const int v = threadIdx.x % NV, g = threadIdx.x / NV;
	double sum = 0, comp = 0;
	for (int b = g; b < n; b += RED_GROUPS) {
		const double y = p[(size_t)b * stride] - comp;
		const double u = sum + y;
		comp = (u - sum) - y;
		sum = u;
	}
	red[g][v] = sum;
	__syncthreads();
	if (g != 0) return 0;
	comp = 0;
	for (int k = 1; k < RED_GROUPS; k++) {
		const double y = red[k][v] - comp;
		const double u = sum + y;
		comp = (u - sum) - y;
		sum = u;
	}
	return sum;
}

}  // namespace rqc
