// Full-Hessian engine (see hess.h).
//
// Per basis column b (or for one given state) let psi_q be the input state of
// sequential gate q and phi_q the cotangent at its output: phi_{G-1} is the
// target column -conj(U e_b) (or the given output cotangent) and
// phi_{q-1} = G_q^T phi_q.  f = phi_{G-1} . psi_G is linear in every gate
// occurrence, so its second derivative in entry x of occurrence q and entry y of
// an earlier occurrence p is
//     sum over the gate group of  phi_q[x_r] * (G_{q-1} ... G_{p+1} E_y psi_p)[x_c]
// with E_y the unit 4x4 gate with entry y = 4 r + c at p's wires.
//
// The engine stores phi_q for all gates (one reverse chain of G^T applications)
// and then sweeps forward once.  For every layer l already reached and every
// entry y it carries one tangent state
//     T_{l,y} = sum over occurrences p of layer l (before the current gate) of
//               G_{q-1} ... G_{p+1} E_y psi_p,
// so the L/2 occurrences of a layer share one state per entry.  At gate q of
// layer a, one kernel launch (k_hsweep) takes every active state s -- psi_q
// itself and the 16 (a + 1) tangents -- contracts it with phi_q (the outer
// product of a gate gradient: 16 complex numbers, summed per layer), then
// carries it through G_q; the tangents of layer a also gain the placeholder
// E_y psi_q.  The contraction of psi_q is the gate gradient; the contraction of
// T_{l,y} at layer a is the Hessian block (a, l) for l < a, and for l = a the
// pairs p < q of the same layer, which the reference symmetrises
// (src/brickwall_circuit.c:229-237).  This replaces the reference's propagation
// of 16 placeholder states per occurrence (src/brickwall_circuit.c:186-224):
// each gate moves 16 (a + 1) + 1 states instead of 16 times the number of
// earlier occurrences.
//
// That is the general sweep (any gates; one state; k_hsweep, k_hlayer).  For unitary gates the
// column sums take the layer sweep (below, "layer sweep"), which moves whole layers, where a
// column of it fits the workspace and it is not the slower one (latency_bound).
//
// Sums: each block reduces its 16 complex products per state (warp transpose
// reduction, then over warps) and adds them to its own slot of a partial-sum
// array, [layer][state][32 doubles][block]; the launches of a layer and the
// column chunks add into the same slots in stream order, and one final kernel
// sums the slots over blocks in index order, so results are deterministic.
#include "hess.h"

#include <math.h>
#include <stdio.h>
#include <string.h>
#include <algorithm>
#include <vector>

#include "layer_pass.h"
#include "manifold.cuh"
#include "rqc_common.cuh"
#include "rqcopt_gpu.h"
#include "sampling.h"
#include "trust_region.cuh"

namespace rqc {

namespace {

constexpr int HT = 256;       // threads per block of the sweep and array kernels
constexpr int HMAXBX = 64;    // blocks per state and launch (partial-sum slots)

// Lane l returns the warp sum of v[l] (31 shuffles for 32 values).
__device__ __forceinline__ double transpose_sum32(double (&v)[32], int lane)
{
#pragma unroll
	for (int o = 16; o >= 1; o >>= 1) {
		const bool up = (lane & o) != 0;
#pragma unroll
		for (int k = 0; k < o; k++) {
			const double send = up ? v[k] : v[k + o];
			const double keep = up ? v[k + o] : v[k];
			v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
		}
	}
	return v[0];
}

// Block sum of acc[32] added to out[c * stride], c = 0..31 (one thread per c).
__device__ __forceinline__ void block_add32(double (&acc)[32], double* __restrict__ out, size_t stride, bool add)
{
	__shared__ double red[HT / 32][32];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	red[warp][lane] = transpose_sum32(acc, lane);
	__syncthreads();
	if (threadIdx.x < 32) {
		double s = 0;
#pragma unroll
		for (int k = 0; k < HT / 32; k++) s += red[k][threadIdx.x];
		double* o = out + (size_t)threadIdx.x * stride;
		*o = add ? *o + s : s;
	}
}

// acc[2 (4 r + c) + {0, 1}] += p[r] * x[c]
__device__ __forceinline__ void contract(double (&acc)[32], const double2 p[4], const double2 x[4])
{
#pragma unroll
	for (int r = 0; r < 4; r++)
#pragma unroll
		for (int c = 0; c < 4; c++) {
			acc[2 * (4 * r + c)] = fma(p[r].x, x[c].x, fma(-p[r].y, x[c].y, acc[2 * (4 * r + c)]));
			acc[2 * (4 * r + c) + 1] = fma(p[r].x, x[c].y, fma(p[r].y, x[c].x, acc[2 * (4 * r + c) + 1]));
		}
}

// One gate of the forward sweep (see the file comment).  Block (s, bx): state s
// (0: psi, 1 + t: tangent t of layer t / 16, entry t % 16), column range bx.
//   basis: psi_in is basis column c of src for chunk column c
//   fresh:  the tangents of `layer` are zero before this gate
//   carry:  carry the tangents through the gate (0 at the last gate)
//   psi_out: G psi_in, or null where the next input state is given (one-state pass)
//   fpart:  non-null at the last gate of a target sum: f += phi . (G psi)
__global__ void __launch_bounds__(HT, 2)
k_hsweep(const double2* __restrict__ psi_in, int basis, ColumnSource src, double2* __restrict__ psi_out,
         const double2* __restrict__ phi, double2* __restrict__ tan, Gate4<double> g, WirePair w, int L,
         int64_t ngroups, int64_t sstride, int layer, int fresh, int carry, double* __restrict__ part, int S,
         double2* __restrict__ fpart)
{
	const int s = blockIdx.x, bx = blockIdx.y, nbx = gridDim.y;
	const int t = s - 1;
	const bool own = s > 0 && (t >> 4) == layer;
	const bool zero_in = own && fresh;
	const int er = (t & 15) >> 2, ec = t & 3;   // placeholder entry (row, column)
	double2* __restrict__ T = s > 0 ? tan + (int64_t)t * sstride : nullptr;
	const int lg = L - 2;
	const int64_t gmask = ((int64_t)1 << lg) - 1;
	int64_t off[4];
	group_offsets(w, off);
	double acc[32];
#pragma unroll
	for (int k = 0; k < 32; k++) acc[k] = 0;
	double fx = 0, fy = 0;
	for (int64_t gi = (int64_t)bx * HT + threadIdx.x; gi < ngroups; gi += (int64_t)nbx * HT) {
		const int64_t c = gi >> lg;
		const int64_t loc = group_base(gi & gmask, w);
		const int64_t base = (c << L) + loc;
		double2 p[4], x[4], y[4];
#pragma unroll
		for (int m = 0; m < 4; m++) p[m] = phi[base + off[m]];
		if (s == 0) {
#pragma unroll
			for (int m = 0; m < 4; m++)
				x[m] = basis ? basis_amp<double>(src, loc + off[m], c) : psi_in[base + off[m]];
		} else if (zero_in) {
#pragma unroll
			for (int m = 0; m < 4; m++) x[m] = make_double2(0, 0);
		} else {
#pragma unroll
			for (int m = 0; m < 4; m++) x[m] = T[base + off[m]];
		}
		if (!zero_in) contract(acc, p, x);
		if (s == 0) {
			// psi_out is null where the input states are given (one-state backward pass)
			if (psi_out || fpart) gate_apply(g, x, y);
			if (psi_out) {
#pragma unroll
				for (int m = 0; m < 4; m++) psi_out[base + off[m]] = y[m];
			}
			if (fpart) {
#pragma unroll
				for (int m = 0; m < 4; m++) {
					fx += p[m].x * y[m].x - p[m].y * y[m].y;
					fy += p[m].x * y[m].y + p[m].y * y[m].x;
				}
			}
		} else if (carry) {
			if (zero_in) {
#pragma unroll
				for (int m = 0; m < 4; m++) y[m] = make_double2(0, 0);
			} else {
				gate_apply(g, x, y);
			}
			if (own) {
				const double2 v = basis ? basis_amp<double>(src, loc + off[ec], c) : psi_in[base + off[ec]];
				y[er].x += v.x;
				y[er].y += v.y;
			}
#pragma unroll
			for (int m = 0; m < 4; m++) T[base + off[m]] = y[m];
		}
	}
	const size_t slot = (size_t)layer * S + s;
	block_add32(acc, part + slot * 32 * nbx + bx, nbx, true);
	if (s == 0 && fpart) {
		__shared__ double fr[2][HT / 32];
		fx = warp_sum(fx);
		fy = warp_sum(fy);
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
		if (lane == 0) { fr[0][warp] = fx; fr[1][warp] = fy; }
		__syncthreads();
		if (threadIdx.x == 0) {
			double sx = 0, sy = 0;
			for (int k = 0; k < HT / 32; k++) { sx += fr[0][k]; sy += fr[1][k]; }
			fpart[bx].x += sx;
			fpart[bx].y += sy;
		}
	}
}

constexpr int HTILE = 4096;   // amplitudes per shared-memory tile of the layer kernel (64 KB)
constexpr int HMAXPER = 6;    // gates per layer of the layer kernel (L <= 12)

// The wire pairs of one brickwall layer (every position holds the layer gate).
struct LayerGates
{
	WirePair w[HMAXPER];
	int q0, per;
};

// One whole layer of the forward sweep with each tangent's column tiles held in
// shared memory (L <= 12): the gates of a brickwall layer act on disjoint wires,
// so a block loads HTILE amplitudes of a tangent (cb = HTILE / 2^L columns) once,
// runs the layer's L/2 gates on them -- contraction with phi_q, G_q, placeholder --
// and writes them back once; one thread per amplitude group and gate.  Block
// (s, bx): state s as in k_hsweep, column blocks bx, bx + nbx, ...  psi_q comes
// from the forward cache psi + q * sstride, except psi_0 of a basis-column sum
// (from_basis), which is basis column c of src.  The tangents of
// `layer` start at zero (they are created at its first gate).  last: the layer
// holds the circuit's last gate (no G at that gate, no store of the tiles, f
// summed by the psi blocks).
__global__ void __launch_bounds__(HT, 2)
k_hlayer(const double2* __restrict__ psi, int from_basis, ColumnSource src, const double2* __restrict__ phi, double2* __restrict__ tan,
         Gate4<double> g, LayerGates lgts, int L, int64_t ncols, int64_t sstride, int layer, int last,
         double* __restrict__ part, int S, double2* __restrict__ fpart)
{
	extern __shared__ double2 tile[];
	__shared__ WirePair sw[HMAXPER];
	if (threadIdx.x < lgts.per) sw[threadIdx.x] = lgts.w[threadIdx.x];
	__syncthreads();
	const int s = blockIdx.x, bx = blockIdx.y, nbx = gridDim.y;
	const int t = s - 1;
	const bool own = s > 0 && (t >> 4) == layer;
	const int er = (t & 15) >> 2, ec = t & 3;
	double2* __restrict__ T = s > 0 ? tan + (int64_t)t * sstride : nullptr;
	const int lg = L - 2;
	const int64_t gmask = ((int64_t)1 << lg) - 1;
	const int cb = HTILE >> L;                               // columns per tile
	const int64_t nblk = (ncols + cb - 1) / cb;
	double acc[32];
#pragma unroll
	for (int k = 0; k < 32; k++) acc[k] = 0;
	double fx = 0, fy = 0;
	for (int64_t blk = bx; blk < nblk; blk += nbx) {
		const int64_t col0 = blk * cb;
		const int cbn = (int)min((int64_t)cb, ncols - col0);
		const int n = cbn << L;                               // amplitudes of this tile
		const int64_t gofs = col0 << L;
		if (s > 0 && !own) {
			for (int e = threadIdx.x; e < n; e += HT) tile[e] = T[gofs + e];
			__syncthreads();
		}
		const int ngr = n >> 2;
		for (int k = 0; k < lgts.per; k++) {
			const int q = lgts.q0 + k;
			const WirePair w = sw[k];
			int64_t off[4];
			group_offsets(w, off);
			const bool final_gate = last && k == lgts.per - 1;
			const double2* __restrict__ ph = phi + (int64_t)q * sstride + gofs;
			const double2* __restrict__ ps = psi + (int64_t)q * sstride + gofs;
			const bool zero_in = own && k == 0;
			const bool basis = q == 0 && from_basis;
			const int64_t offc = ((ec & 2) ? w.si : 0) + ((ec & 1) ? w.sj : 0);
			for (int gi = threadIdx.x; gi < ngr; gi += HT) {
				const int cc = gi >> lg;
				const int64_t loc = group_base(gi & gmask, w);
				const int64_t li = ((int64_t)cc << L) + loc;      // index within the tile
				double2 p[4], x[4];
#pragma unroll
				for (int m = 0; m < 4; m++) p[m] = ph[li + off[m]];
				if (s == 0) {
#pragma unroll
					for (int m = 0; m < 4; m++)
						x[m] = basis ? basis_amp<double>(src, loc + off[m], col0 + cc) : ps[li + off[m]];
				} else if (zero_in) {
#pragma unroll
					for (int m = 0; m < 4; m++) x[m] = make_double2(0, 0);
				} else {
#pragma unroll
					for (int m = 0; m < 4; m++) x[m] = tile[li + off[m]];
				}
				if (!zero_in) {
#pragma unroll
					for (int r = 0; r < 4; r++)
#pragma unroll
						for (int c = 0; c < 4; c++) {
							acc[2 * (4 * r + c)] = fma(p[r].x, x[c].x, fma(-p[r].y, x[c].y, acc[2 * (4 * r + c)]));
							acc[2 * (4 * r + c) + 1] = fma(p[r].x, x[c].y, fma(p[r].y, x[c].x, acc[2 * (4 * r + c) + 1]));
						}
				}
				if (s == 0) {
					if (final_gate) {
						double2 y[4];
						gate_apply(g, x, y);
#pragma unroll
						for (int m = 0; m < 4; m++) {
							fx += p[m].x * y[m].x - p[m].y * y[m].y;
							fy += p[m].x * y[m].y + p[m].y * y[m].x;
						}
					}
				} else if (!final_gate) {
					double2 y[4];
					if (zero_in) {
#pragma unroll
						for (int m = 0; m < 4; m++) y[m] = make_double2(0, 0);
					} else {
						gate_apply(g, x, y);
					}
					if (own) {
						const double2 v = basis ? basis_amp<double>(src, loc + offc, col0 + cc) : ps[li + offc];
						y[er].x += v.x;
						y[er].y += v.y;
					}
#pragma unroll
					for (int m = 0; m < 4; m++) tile[li + off[m]] = y[m];
				}
			}
			__syncthreads();
		}
		if (s > 0 && !last) {
			for (int e = threadIdx.x; e < n; e += HT) T[gofs + e] = tile[e];
			__syncthreads();
		}
	}
	const size_t slot = (size_t)layer * S + s;
	block_add32(acc, part + slot * 32 * nbx + bx, nbx, true);
	if (s == 0 && fpart) {
		__shared__ double fr[2][HT / 32];
		fx = warp_sum(fx);
		fy = warp_sum(fy);
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
		if (lane == 0) { fr[0][warp] = fx; fr[1][warp] = fy; }
		__syncthreads();
		if (threadIdx.x == 0) {
			double sx = 0, sy = 0;
			for (int k = 0; k < HT / 32; k++) { sx += fr[0][k]; sy += fr[1][k]; }
			fpart[bx].x += sx;
			fpart[bx].y += sy;
		}
	}
}

// ------------------------------------------------------------------ block encoding

// full-register index of half-register basis state b: bit i of b at bit 2 i + 1
// (src/target.c:1148-1157)
__host__ __device__ __forceinline__ int64_t blockenc_index(int64_t b, int half)
{
	int64_t c = 0;
	for (int i = 0; i < half; i++) c |= ((b >> i) & 1) << (2 * i + 1);
	return c;
}

// half-register basis state and weight of column k (tab null: state k, weight 1)
__device__ __forceinline__ int64_t benc_state(const BasisCol* tab, int64_t k) { return tab ? tab[k].re : k; }
__device__ __forceinline__ double benc_weight(const BasisCol* tab, int64_t k) { return tab ? tab[k].wre : 1.0; }

// psi_0 of columns b0 .. b0 + ncols - 1: the basis states P e_b
__global__ void k_benc_init(double2* __restrict__ states, int L, const BasisCol* __restrict__ tab, int64_t b0, int64_t ncols)
{
	const int64_t N = (int64_t)1 << L;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ncols * N; i += (int64_t)gridDim.x * blockDim.x) {
		const int64_t c = i >> L, a = i & (N - 1);
		states[i] = make_double2(a == blockenc_index(benc_state(tab, b0 + c), L / 2) ? 1.0 : 0.0, 0.0);
	}
}

// residual d = P^dag W P e_b - H e_b on the P rows: f += w |d|^2 / 2 (per block), chi = w P conj(d)
// (zero elsewhere: chi is cleared before), w the column's weight.  hneg[b][a] = -conj((H e_b)[a]).
__global__ void k_benc_residual(const double2* __restrict__ wout, const double2* __restrict__ hneg, int L,
                                const BasisCol* __restrict__ tab, int64_t b0, int64_t ncols, double2* __restrict__ chi,
                                double2* __restrict__ fpart)
{
	__shared__ double red[HT / 32];
	const int half = L / 2;
	const int64_t s = (int64_t)1 << half;
	double acc = 0;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ncols * s; i += (int64_t)gridDim.x * blockDim.x) {
		const int64_t c = i >> half, a = i & (s - 1);
		const int64_t idx = (c << L) + blockenc_index(a, half);
		const double2 hn = hneg[benc_state(tab, b0 + c) * s + a];
		const double wt = benc_weight(tab, b0 + c);
		const double2 w = wout[idx];
		const double dx = w.x + hn.x, dy = w.y - hn.y;   // w - H e_b with H e_b = -conj(hn)
		acc += 0.5 * wt * (dx * dx + dy * dy);
		if (chi) chi[idx] = make_double2(wt * dx, -wt * dy);
	}
	acc = warp_sum(acc);
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
	__syncthreads();
	if (threadIdx.x == 0) {
		double t = 0;
		for (int k = 0; k < HT / 32; k++) t += red[k];
		fpart[blockIdx.x].x += t;
	}
}

// Jacobian rows on the P rows: jac[t][c * s + a] = tan_t[c][P a]
__global__ void k_benc_gather(const double2* __restrict__ tan, int L, int64_t ncols, int64_t sstride, int m,
                              double2* __restrict__ jac)
{
	const int half = L / 2;
	const int64_t s = (int64_t)1 << half, K = ncols * s;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)m * K; i += (int64_t)gridDim.x * blockDim.x) {
		const int64_t t = i / K, r = i % K;
		jac[i] = tan[t * sstride + ((r >> half) << L) + blockenc_index(r & (s - 1), half)];
	}
}

// Gauss-Newton term: part2[(l i), (k j)] += sum_r w conj(jac[l i][r]) jac[k j][r] for layer l >= k
// (src/target.c:1570-1580), row r belonging to column b0 + (r >> half) of weight w; one block per entry
__global__ void k_benc_gram(const double2* __restrict__ jac, int64_t K, int nl, const BasisCol* __restrict__ tab, int64_t b0,
                            int half, double2* __restrict__ part2)
{
	__shared__ double red[2][HT / 32];
	const int m = 16 * nl;
	const int e = blockIdx.x;
	const int row = e / m, col = e % m;
	if ((row >> 4) < (col >> 4)) return;
	const double2* __restrict__ x = jac + (int64_t)row * K;
	const double2* __restrict__ y = jac + (int64_t)col * K;
	double sx = 0, sy = 0;
	for (int64_t r = threadIdx.x; r < K; r += HT) {
		const double2 a = x[r], b = y[r];
		const double wt = benc_weight(tab, b0 + (r >> half));
		sx += wt * (a.x * b.x + a.y * b.y);     // conj(a) b
		sy += wt * (a.x * b.y - a.y * b.x);
	}
	sx = warp_sum(sx);
	sy = warp_sum(sy);
	if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = sx; red[1][threadIdx.x >> 5] = sy; }
	__syncthreads();
	if (threadIdx.x == 0) {
		double tx = 0, ty = 0;
		for (int k = 0; k < HT / 32; k++) { tx += red[0][k]; ty += red[1][k]; }
		part2[e].x += tx;
		part2[e].y += ty;
	}
}

// hess2 from the lower blocks, upper blocks by conjugate symmetry; f from the residual parts
__global__ void k_benc_finish(const double2* __restrict__ part2, int nl, const double2* __restrict__ fres, int nres,
                              double2* __restrict__ rec, double2* __restrict__ hess2)
{
	const int m = 16 * nl;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)m * m; i += (int64_t)gridDim.x * blockDim.x) {
		const int row = (int)(i / m), col = (int)(i % m);
		if (!hess2) break;
		if ((row >> 4) >= (col >> 4)) hess2[i] = part2[i];
		else {
			const double2 v = part2[(int64_t)col * m + row];
			hess2[i] = make_double2(v.x, -v.y);
		}
	}
	if (blockIdx.x == 0 && threadIdx.x == 0) {
		double t = 0;
		for (int k = 0; k < nres; k++) t += fres[k].x;
		rec[0] = make_double2(t, 0.0);
	}
}

// Sum over the blocks of partial slot (slot, entry e)
__device__ __forceinline__ double2 slot_sum(const double* __restrict__ part, int nbx, size_t slot, int e)
{
	const double* re = part + (slot * 32 + 2 * e) * nbx;
	const double* im = re + nbx;
	double sx = 0, sy = 0;
	for (int b = 0; b < nbx; b++) { sx += re[b]; sy += im[b]; }
	return make_double2(sx, sy);
}

// Record: f, per-layer gradients, symmetric complex Hessian (row (a, x), column (b, y)).
__global__ void k_hassemble(const double* __restrict__ part, int nbx, int nl, int S, const double2* __restrict__ fpart,
                            double2* __restrict__ rec)
{
	const int m = 16 * nl;
	const int64_t n = 1 + 16 * (int64_t)nl + (int64_t)m * m;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		if (i == 0) {
			double sx = 0, sy = 0;
			for (int b = 0; b < nbx; b++) { sx += fpart[b].x; sy += fpart[b].y; }
			rec[0] = make_double2(sx, sy);
		} else if (i <= 16 * nl) {
			const int l = (int)(i - 1) >> 4, e = (int)(i - 1) & 15;
			rec[i] = slot_sum(part, nbx, (size_t)l * S, e);
		} else {
			const int64_t h = i - 1 - 16 * (int64_t)nl;
			const int row = (int)(h / m), col = (int)(h % m);
			const int a = row >> 4, x = row & 15, b = col >> 4, y = col & 15;
			double2 v;
			if (a < b) {
				v = slot_sum(part, nbx, (size_t)b * S + 1 + 16 * a + x, y);
			} else if (a > b) {
				v = slot_sum(part, nbx, (size_t)a * S + 1 + 16 * b + y, x);
			} else {
				const double2 u = slot_sum(part, nbx, (size_t)a * S + 1 + 16 * a + x, y);
				const double2 u2 = slot_sum(part, nbx, (size_t)a * S + 1 + 16 * a + y, x);
				v = make_double2(u.x + u2.x, u.y + u2.y);
			}
			rec[i] = v;
		}
	}
}

// out = G in over `ngroups` groups of consecutive 2^L-amplitude states
//   basis: `in` is basis column c of src
__global__ void __launch_bounds__(HT) k_happly(const double2* __restrict__ in, double2* __restrict__ out, Gate4<double> g,
                                               WirePair w, int L, int64_t ngroups, int basis = 0,
                                               ColumnSource src = ColumnSource{})
{
	const int lg = L - 2;
	const int64_t gmask = ((int64_t)1 << lg) - 1;
	int64_t off[4];
	group_offsets(w, off);
	for (int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gi < ngroups; gi += (int64_t)gridDim.x * blockDim.x) {
		const int64_t c = gi >> lg, loc = group_base(gi & gmask, w);
		const int64_t base = (c << L) + loc;
		double2 x[4], y[4];
#pragma unroll
		for (int m = 0; m < 4; m++)
			x[m] = basis ? basis_amp<double>(src, loc + off[m], c) : in[base + off[m]];
		gate_apply(g, x, y);
#pragma unroll
		for (int m = 0; m < 4; m++) out[base + off[m]] = y[m];
	}
}

// Column (b, k) entries of the real Hessian for layers a <= b (src/target.c:937-987), and
// the gradient vector (src/target.c:1025-1030).  rec as written by k_hassemble.
__global__ void k_hproject(int nl, const double2* __restrict__ ug, const double2* __restrict__ rec,
                           const double2* __restrict__ hess2, double* __restrict__ grad, double* __restrict__ H)
{
	const int m = 16 * nl;
	const int npairs = nl * (nl + 1) / 2;
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	const double2* dv = rec + 1;
	const double2* hess = rec + 1 + 16 * nl;
	if (i < nl) {
		M4 v, d;
		for (int e = 0; e < 16; e++) { v.a[e] = ug[16 * i + e]; d.a[e] = c_conj(dv[16 * i + e]); }
		m4_tangent_to_real(v, d, grad + 16 * i);
	}
	if (i >= npairs * 16) return;
	const int k = i & 15;
	int pr = i >> 4, a = 0;
	while (pr >= nl - a) { pr -= nl - a; a++; }
	const int b = a + pr;
	M4 va, vb, z, g;
	for (int e = 0; e < 16; e++) { va.a[e] = ug[16 * a + e]; vb.a[e] = ug[16 * b + e]; }
	double r[16];
	for (int e = 0; e < 16; e++) r[e] = 0;
	r[k] = 1;
	m4_real_to_tangent(r, vb, z);
	for (int x = 0; x < 16; x++) {
		const double2* row = hess + (size_t)(16 * a + x) * m + 16 * b;
		double2 s = c_(0, 0);
		for (int y = 0; y < 16; y++) s = c_add(s, c_mul(row[y], z.a[y]));
		g.a[x] = c_conj(s);
		if (hess2) {   // block encoding: conj(hess1 Z) + hess2 Z (src/target.c:1673-1683)
			const double2* row2 = hess2 + (size_t)(16 * a + x) * m + 16 * b;
			double2 s2 = c_(0, 0);
			for (int y = 0; y < 16; y++) s2 = c_add(s2, c_mul(row2[y], z.a[y]));
			g.a[x] = c_add(g.a[x], s2);
		}
	}
	if (a == b) {
		M4 p, dc, gh, t;
		m4_project_tangent(va, g, p);
		for (int e = 0; e < 16; e++) dc.a[e] = c_conj(dv[16 * a + e]);
		m4_adjoint(dc, gh);
		m4_symmetric_triple(z, gh, va, t);
		for (int e = 0; e < 16; e++) g.a[e] = c_sub(p.a[e], t.a[e]);
	}
	m4_tangent_to_real(va, g, r);
	for (int x = 0; x < 16; x++) H[(size_t)(16 * a + x) * m + 16 * b + k] = r[x];
}

// rec *= scale (the 2^L / nsamples normalisation of the sampling estimator,
// src/target.c:904-915)
__global__ void k_scale_rec(double2* __restrict__ rec, int64_t n, double scale)
{
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
		rec[i] = make_double2(rec[i].x * scale, rec[i].y * scale);
}

// lower triangle from the upper one (src/target.c:981-986)
__global__ void k_hmirror(int m, double* __restrict__ H)
{
	const int64_t n = (int64_t)m * m;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		const int row = (int)(i / m), col = (int)(i % m);
		if (row > col) H[i] = H[(size_t)col * m + row];
	}
}

// Truncated CG with a dense Hessian (src/trust_region.c:83-141): the matrix-vector
// product by rows in parallel, the other steps with dot products in index order
// (trust_region.cuh).
__global__ void __launch_bounds__(HT) k_tcg_hmat(int n, const double* __restrict__ grad, const double* __restrict__ hess,
                                                 double radius, int maxiter, double abstol, double reltol, double* r,
                                                 double* d, double* hd, double* z, int* status)
{
	__shared__ TcgState st;
	__shared__ BlockDots dots;
	tcg_init_blk(n, grad, r, d, z, &st, radius, abstol, reltol, dots);
	for (int it = 0; it < maxiter; it++) {
		for (int row = threadIdx.x; row < n; row += blockDim.x) hd[row] = dot_seq(n, hess + (size_t)row * n, d);
		__syncthreads();
		tcg_step_blk(n, d, hd, z, r, &st, dots);
		if (st.status != TCG_CONTINUE) break;
	}
	if (threadIdx.x == 0) status[0] = st.status == TCG_BOUNDARY ? 1 : 0;
}

__global__ void k_gemv(int n, const double* __restrict__ a, const double* __restrict__ x, double* __restrict__ y)
{
	const int row = blockIdx.x * blockDim.x + threadIdx.x;
	if (row < n) y[row] = dot_seq(n, a + (size_t)row * n, x);
}

// ------------------------------------------------------------------ layer sweep
//
// The gates of a layer commute, so everything the sweep needs can be taken at the layer's OUTPUT.
// With psi, phi the state and cotangent there and T any tangent carried through the whole layer,
// the contraction at gate q is the raw sum R_q[i][j] = sum phi[.. i at q ..] T[.. j at q ..] times
// conj(G) (G unitary).  Summed over the layer's gates that is ONE inner product with states made
// from phi,
//     R[i][j] = sum_q R_q[i][j] = <Phi_{ij}, T>,   Phi_{ij}[a] = sum over q with bits_q(a) = j of phi[a, i at q],
// so the layer's Hessian blocks are a complex matrix product of 16 cotangent states with the
// 16 (a + 1) tangents over all amplitudes and columns (k_hgemm): 16 multiply-adds per amplitude
// and tangent whatever the layer's length, in FP64 MMAs whose operands come straight from memory.
// The layer's own tangents at its output are T_{rc}[a] = sum over q with bits_q(a) = r of
// (row c of G_q^+ psi at q)[a], and the pairs p = q that the product with them contains are
//     dV[i][yc] conj(G[yr][xc])          (x = (i, xc), y = (yr, yc))
// with dV the layer's gradient, taken off in k_hrecord.  What is left per layer: carry the
// earlier tangents (layer_pass.cu), 32 new states (k_hstates) and the product.  Against the
// general layer kernel this is a third of the flops at L = 12, 1-2 memory round trips a layer
// instead of two tiles' worth of shared-memory traffic per gate; L = 10, depth 7, one column
// per orbit: 3.8 -> 1.7 ms (see the figures at k_hgemm).

// T_{rc} (own tangents) and Phi_{ij} at a layer's output, 16 states each, from psi and phi
struct LayerWires
{
	int n;
	int8_t bi[16], bj[16];   // state bits of the pairs
	Gate4<double> g;
};

// a thread per amplitude and column; own: write the tangents (not where only the gradient is
// wanted); fpart (the circuit's last layer): f = phi . psi, per block
__global__ void __launch_bounds__(256) k_hstates(const double2* __restrict__ psi, const double2* __restrict__ phi,
                                                 const __grid_constant__ LayerWires w, int64_t n,
                                                 double2* __restrict__ own, double2* __restrict__ cot,
                                                 double2* __restrict__ fpart)
{
	double fx = 0, fy = 0;
	for (int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += (int64_t)gridDim.x * blockDim.x) {
		double2 t[16];
		if (own) {
#pragma unroll
			for (int e = 0; e < 16; e++) t[e] = make_double2(0, 0);
			for (int q = 0; q < w.n; q++) {
				const int64_t si = (int64_t)1 << w.bi[q], sj = (int64_t)1 << w.bj[q];
				const int r = ((a & si) ? 2 : 0) | ((a & sj) ? 1 : 0);
				const int64_t b = a & ~(si | sj);
				const double2 x[4] = {psi[b], psi[b | sj], psi[b | si], psi[b | si | sj]};
#pragma unroll
				for (int c = 0; c < 4; c++) {
					double2 v = make_double2(0, 0);
#pragma unroll
					for (int m = 0; m < 4; m++) v = cfma(make_double2(w.g.m[4 * m + c].x, -w.g.m[4 * m + c].y), x[m], v);
#pragma unroll
					for (int k = 0; k < 4; k++)
						if (k == r) t[4 * k + c] = cadd(t[4 * k + c], v);
				}
			}
#pragma unroll
			for (int e = 0; e < 16; e++) own[e * n + a] = t[e];
		}
#pragma unroll
		for (int e = 0; e < 16; e++) t[e] = make_double2(0, 0);
		for (int q = 0; q < w.n; q++) {
			const int64_t si = (int64_t)1 << w.bi[q], sj = (int64_t)1 << w.bj[q];
			const int j = ((a & si) ? 2 : 0) | ((a & sj) ? 1 : 0);
			const int64_t b = a & ~(si | sj);
			const double2 x[4] = {phi[b], phi[b | sj], phi[b | si], phi[b | si | sj]};
#pragma unroll
			for (int k = 0; k < 4; k++)
				if (k == j)
#pragma unroll
					for (int i = 0; i < 4; i++) t[4 * i + k] = cadd(t[4 * i + k], x[i]);
		}
#pragma unroll
		for (int e = 0; e < 16; e++) cot[e * n + a] = t[e];
		if (fpart) {
			const double2 p = phi[a], v = psi[a];
			fx += p.x * v.x - p.y * v.y;
			fy += p.x * v.y + p.y * v.x;
		}
	}
	if (fpart) {
		__shared__ double fr[2][8];
		fx = warp_sum(fx);
		fy = warp_sum(fy);
		if ((threadIdx.x & 31) == 0) { fr[0][threadIdx.x >> 5] = fx; fr[1][threadIdx.x >> 5] = fy; }
		__syncthreads();
		if (threadIdx.x == 0) {
			double sx = 0, sy = 0;
			for (int k = 0; k < 8; k++) { sx += fr[0][k]; sy += fr[1][k]; }
			fpart[blockIdx.x].x += sx;
			fpart[blockIdx.x].y += sy;
		}
	}
}

__device__ __forceinline__ void hdmma(double (&d)[2], double a, double b)
{
	asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
	    : "+d"(d[0]), "+d"(d[1])
	    : "d"(a), "d"(b));
}

constexpr int GW = 4;               // warps per block of the product
constexpr int GN = 32;              // tangents per block: two layers
constexpr int GSLOT = 16 * GN;      // complex sums per block
constexpr int GRUN = 64;            // amplitudes a warp takes in a row: 1 KB of each state
constexpr int GDEPTH = 5;           // steps of four amplitudes in a warp's queue
constexpr int GSMEM = GW * (GDEPTH * 6 * 32 > GSLOT ? GDEPTH * 6 * 32 : GSLOT) * (int)sizeof(double2);

// R[m][n] += sum_k A[m][k] B[n][k] (no conjugation) for 16 cotangent states A and the ntan tangents
// B, then psi as column ntan.  Block x takes four fragments of eight columns, K amplitudes per
// state; blockIdx.y and the block's warps split them in runs of GRUN.  FP64 MMAs m8n8k4 on the real
// and imaginary parts (four per complex 8 x 8 x 4 product): a lane's operand is the complex number
// it loads, rows of four consecutive amplitudes (64 B), so the fragments come from memory as they
// are, six 16-byte loads for 32 MMAs.  Bound: the FP64 pipe (32 MMAs per 3 KB), at few tangents the read from HBM.
//
// The operands wait in shared memory only as a queue: each lane copies its own six numbers of a
// step (cp.async, GDEPTH - 1 steps ahead) and reads them back itself.  With the next step's in
// registers instead, the warps waited for memory half the time (FP64 MMA pipe 47 % busy).
__global__ void __launch_bounds__(32 * GW, 3)
k_hgemm(const double2* __restrict__ A, const double2* __restrict__ B, const double2* __restrict__ psi, int64_t K, int ntan,
        double2* __restrict__ part, int add)
{
	extern __shared__ __align__(16) double2 hsm[];   // queue [GW][GDEPTH][6][32], then the block's sums [GW][GSLOT]
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int row = lane >> 2, kk = lane & 3;
	const int nt = ntan / 8, f0 = 4 * blockIdx.x;   // fragments of tangents; this block's first
	const int nf = min(4, nt + 1 - f0);
	const double2* p[6] = {A + row * K + kk, A + (row + 8) * K + kk};
	bool live[6] = {true, true};
#pragma unroll
	for (int f = 0; f < 4; f++) {
		const bool tangent = f0 + f < nt;
		p[2 + f] = tangent ? B + (int64_t)(8 * (f0 + f) + row) * K + kk : psi + kk;
		live[2 + f] = tangent || (f0 + f == nt && row == 0);
	}
	double re[2][4][2], im[2][4][2];
#pragma unroll
	for (int m = 0; m < 2; m++)
#pragma unroll
		for (int f = 0; f < 4; f++) re[m][f][0] = re[m][f][1] = im[m][f][0] = im[m][f][1] = 0;
	const int64_t nrun = (K + GRUN - 1) / GRUN, stride = (int64_t)gridDim.y * GW;
	const int64_t first = (int64_t)blockIdx.y * GW + warp;
	const int nstep = first < nrun ? (int)((nrun - first + stride - 1) / stride) * (GRUN / 4) : 0;
	double2* queue = hsm + (size_t)warp * GDEPTH * 6 * 32 + lane;
	const unsigned qaddr = (unsigned)__cvta_generic_to_shared(queue);
	int64_t knext = first * GRUN;   // amplitude of the next step to copy
	auto fetch = [&](int n) {
		if (n < nstep) {
			const bool in = knext + kk < K;
			const unsigned d = qaddr + (n % GDEPTH) * 6 * 32 * 16;
#pragma unroll
			for (int f = 0; f < 6; f++) {
				if (f - 2 >= nf) break;
				const bool on = in && live[f];
				const double2* src = on ? p[f] + knext : A;
				asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d + f * 32 * 16), "l"(src), "r"(on ? 16 : 0)
				             : "memory");
			}
			knext += (n % (GRUN / 4)) == GRUN / 4 - 1 ? (stride - 1) * GRUN + 4 : 4;
		}
		asm volatile("cp.async.commit_group;\n" ::: "memory");
	};
#pragma unroll
	for (int n = 0; n < GDEPTH - 1; n++) fetch(n);
	for (int n = 0; n < nstep; n++) {
		asm volatile("cp.async.wait_group %0;\n" ::"n"(GDEPTH - 2) : "memory");
		const double2* q = queue + (n % GDEPTH) * 6 * 32;
		const double2 x[2] = {q[0], q[32]};
		double2 y[4];
#pragma unroll
		for (int f = 0; f < 4; f++) y[f] = f < nf ? q[(2 + f) * 32] : make_double2(0, 0);
		fetch(n + GDEPTH - 1);   // into the slot read one step ago
		// the two products into one accumulator sixteen MMAs apart
		if (nf == 4) {
#pragma unroll
			for (int f = 0; f < 4; f++)
#pragma unroll
				for (int m = 0; m < 2; m++) {
					hdmma(re[m][f], x[m].x, y[f].x);
					hdmma(im[m][f], x[m].x, y[f].y);
				}
#pragma unroll
			for (int f = 0; f < 4; f++)
#pragma unroll
				for (int m = 0; m < 2; m++) {
					hdmma(re[m][f], -x[m].y, y[f].y);
					hdmma(im[m][f], x[m].y, y[f].x);
				}
		} else {
#pragma unroll
			for (int f = 0; f < 3; f++) {
				if (f >= nf) break;
#pragma unroll
				for (int m = 0; m < 2; m++) {
					hdmma(re[m][f], x[m].x, y[f].x);
					hdmma(im[m][f], x[m].x, y[f].y);
					hdmma(re[m][f], -x[m].y, y[f].y);
					hdmma(im[m][f], x[m].y, y[f].x);
				}
			}
		}
	}
	asm volatile("cp.async.wait_group 0;\n" ::: "memory");
	__syncthreads();
	double2 (*red)[GSLOT] = reinterpret_cast<double2 (*)[GSLOT]>(hsm);
	// lane: rows row (+ 8 m), columns 8 f + 2 kk, + 1
#pragma unroll
	for (int m = 0; m < 2; m++)
#pragma unroll
		for (int f = 0; f < 4; f++)
#pragma unroll
			for (int c = 0; c < 2; c++)
				red[warp][(row + 8 * m) * GN + 8 * f + 2 * kk + c] = make_double2(re[m][f][c], im[m][f][c]);
	__syncthreads();
	double2* o = part + ((int64_t)blockIdx.x * gridDim.y + blockIdx.y) * GSLOT;
	for (int e = threadIdx.x; e < GSLOT; e += blockDim.x) {
		double2 v = red[0][e];
#pragma unroll
		for (int w = 1; w < GW; w++) v = cadd(v, red[w][e]);
		o[e] = add ? cadd(o[e], v) : v;
	}
}

// where a layer's partial sums lie: tile x of split s at off + (x * nsplit + s) * GSLOT
struct LayerParts
{
	int64_t off;
	int nsplit, ntile;   // 16 (a + 1) tangents (none without a Hessian), then psi, 32 columns a tile
};

// Sums of tile blockIdx.x of layer blockIdx.y over the splits, into the tile's first split: 32
// complex entries a block at a time, eight groups of threads sharing the splits.
__global__ void __launch_bounds__(256) k_hsum(double2* __restrict__ part, const LayerParts* __restrict__ parts)
{
	__shared__ double2 red[8][32];
	const LayerParts p = parts[blockIdx.y];
	if ((int)blockIdx.x >= p.ntile) return;
	const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
	double2* q = part + p.off + (int64_t)blockIdx.x * p.nsplit * GSLOT + 32 * blockIdx.z + lane;
	double2 s = make_double2(0, 0);
	for (int k = g; k < p.nsplit; k += 8) s = cadd(s, q[(int64_t)k * GSLOT]);
	red[g][lane] = s;
	__syncthreads();
	if (g != 0) return;
	for (int k = 1; k < 8; k++) s = cadd(s, red[k][lane]);
	q[0] = s;
}

// Record of the layer sweep from k_hsum's sums: block b handles the layer pair (a, l <= a) in
// row-major order of the lower triangle; fpart: partial sums of f, or null
__global__ void __launch_bounds__(256) k_hrecord(const double2* __restrict__ part, const LayerParts* __restrict__ parts,
                                                 const double2* __restrict__ ug, int nl, const double2* __restrict__ fpart,
                                                 int nfpart, int hess, double2* __restrict__ rec)
{
	__shared__ double2 R[256], V[16], D[16], H[256];
	int a = 0, l = blockIdx.x;
	if (hess) while (l > a) l -= ++a;
	else { a = l; }
	const int t = threadIdx.x, m = 16 * nl;
	const LayerParts p = parts[a];
	auto sum_at = [&](int x, int e) { return part[p.off + (int64_t)x * p.nsplit * GSLOT + e]; };
	if (t < 16) {
		V[t] = ug[16 * a + t];
		if (l == a) {
			const int n = hess ? 16 * (a + 1) : 0;   // psi's column
			R[t] = sum_at(n / GN, t * GN + n % GN);
		}
	}
	if (blockIdx.x == 0 && fpart) {
		double fx = 0, fy = 0;
		for (int k = t; k < nfpart; k += 256) { fx += fpart[k].x; fy += fpart[k].y; }
		__shared__ double fr[2][8];
		fx = warp_sum(fx);
		fy = warp_sum(fy);
		if ((t & 31) == 0) { fr[0][t >> 5] = fx; fr[1][t >> 5] = fy; }
		__syncthreads();
		if (t < 2) {
			double s = 0;
			for (int k = 0; k < 8; k++) s += fr[t][k];
			reinterpret_cast<double*>(rec)[t] = s;
		}
	}
	__syncthreads();
	auto times_conj = [&](const double2* r, int stride, int i, int c) {   // sum_j r[(i, j)] conj(G[j][c])
		double2 s = make_double2(0, 0);
		for (int j = 0; j < 4; j++) s = cfma(r[(4 * i + j) * stride], make_double2(V[4 * j + c].x, -V[4 * j + c].y), s);
		return s;
	};
	if (l == a) {
		if (t < 16) {
			D[t] = times_conj(R, 1, t >> 2, t & 3);
			rec[1 + 16 * a + t] = D[t];
		}
		__syncthreads();
	}
	if (!hess) return;
	const int x = t >> 4, y = t & 15;
	R[t] = sum_at(l / 2, x * GN + 16 * (l & 1) + y);   // column y of layer l in its tile
	__syncthreads();
	double2 h = times_conj(R + y, 16, x >> 2, x & 3);
	double2* out = rec + 1 + 16 * nl;
	if (l == a) {
		// the pairs p = q: dV[i][yc] conj(G[yr][xc])
		const double2 g = V[4 * (y >> 2) + (x & 3)];
		h = csub(h, cmul(D[4 * (x >> 2) + (y & 3)], make_double2(g.x, -g.y)));
		H[t] = h;
		__syncthreads();
		const double2 ht = H[16 * y + x];
		h = make_double2(0.5 * (h.x + ht.x), 0.5 * (h.y + ht.y));
		out[(int64_t)(16 * a + x) * m + 16 * a + y] = h;
	} else {
		out[(int64_t)(16 * a + x) * m + 16 * l + y] = h;
		out[(int64_t)(16 * l + y) * m + 16 * a + x] = h;
	}
}

// ------------------------------------------------------------------ interleaved arrays

__global__ void __launch_bounds__(HT) k_gate_array(const double2* __restrict__ in, double2* __restrict__ out,
                                                   Gate4<double> g, WirePair w, int ns, int64_t n)
{
	int64_t off[4];
	group_offsets(w, off);
	for (int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gi < n; gi += (int64_t)gridDim.x * blockDim.x) {
		const int64_t s = gi % ns, base = group_base(gi / ns, w);
		double2 x[4], y[4];
#pragma unroll
		for (int m = 0; m < 4; m++) x[m] = in[(base + off[m]) * ns + s];
		gate_apply(g, x, y);
#pragma unroll
		for (int m = 0; m < 4; m++) out[(base + off[m]) * ns + s] = y[m];
	}
}

// block (s, bx): partial sums of dout (x) psi_s over the groups of column range bx
__global__ void __launch_bounds__(HT) k_gate_backward_array(const double2* __restrict__ psi, const double2* __restrict__ dout,
                                                            WirePair w, int ns, int64_t ngroups, double* __restrict__ part)
{
	const int s = blockIdx.x, bx = blockIdx.y, nbx = gridDim.y;
	int64_t off[4];
	group_offsets(w, off);
	double acc[32];
#pragma unroll
	for (int k = 0; k < 32; k++) acc[k] = 0;
	for (int64_t gi = (int64_t)bx * HT + threadIdx.x; gi < ngroups; gi += (int64_t)nbx * HT) {
		const int64_t base = group_base(gi, w);
		double2 p[4], x[4];
#pragma unroll
		for (int m = 0; m < 4; m++) { p[m] = dout[base + off[m]]; x[m] = psi[(base + off[m]) * ns + s]; }
		contract(acc, p, x);
	}
	block_add32(acc, part + (size_t)s * 32 * nbx + bx, nbx, false);
}

__global__ void k_array_sum(const double* __restrict__ part, int ns, int nbx, double2* __restrict__ dgates)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < 16 * ns) dgates[i] = slot_sum(part, nbx, (size_t)(i >> 4), i & 15);
}

__global__ void __launch_bounds__(HT) k_placeholder(const double2* __restrict__ psi, double2* __restrict__ out, WirePair w,
                                                    int64_t ngroups)
{
	int64_t off[4];
	group_offsets(w, off);
	for (int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gi < ngroups; gi += (int64_t)gridDim.x * blockDim.x) {
		const int64_t base = group_base(gi, w);
		double2 x[4];
#pragma unroll
		for (int m = 0; m < 4; m++) x[m] = psi[base + off[m]];
#pragma unroll
		for (int m = 0; m < 4; m++) {
			double2* o = out + (base + off[m]) * 16;
#pragma unroll
			for (int e = 0; e < 16; e++) o[e] = (e >> 2) == m ? x[e & 3] : make_double2(0, 0);
		}
	}
}

// ------------------------------------------------------------------ host helpers

Gate4<double> gate_of(const double2* g, bool transposed)
{
	Gate4<double> r;
	for (int a = 0; a < 4; a++)
		for (int b = 0; b < 4; b++) r.m[4 * a + b] = transposed ? g[4 * b + a] : g[4 * a + b];
	return r;
}

int grid_of(const Runtime& rt, int64_t items, int per_sm)
{
	const int64_t want = (items + HT - 1) / HT;
	return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)rt.num_sms * per_sm));
}

int checked(Runtime& rt)
{
	rt.launches++;
	return RQC_CUDA(cudaGetLastError());
}

// blocks per state: enough for four groups per thread, at most HMAXBX
int blocks_per_state(int64_t ngroups)
{
	return (int)std::max<int64_t>(1, std::min<int64_t>(HMAXBX, ngroups / (4 * HT)));
}

struct Sweep
{
	Runtime& rt;
	const HessCircuit& c;
	int L, nl, per, G, S, nbx;
	double* part = nullptr;
	double2* fpart = nullptr;
	std::vector<Gate4<double>> gg, gt;
	std::vector<WirePair> gw;

	bool keep_final = false;   // carry the tangents through the last gate and store them (block encoding)
	bool psi_only = false;     // gradient only: the psi blocks of the sweep
	ColumnSource src;          // basis columns of the chunk

	Sweep(Runtime& r, const HessCircuit& hc) : rt(r), c(hc), L(hc.L), nl(hc.nlayers), per(hc.L / 2),
	                                           G(hc.nlayers * (hc.L / 2)), S(1 + 16 * hc.nlayers), nbx(1) {}

	// blocks per state: by groups for the per-gate kernel, by column tiles for the layer kernel
	int init(int64_t ngroups_per_state, int64_t layer_tiles = 0)
	{
		nbx = layer_tiles > 0 ? (int)std::min<int64_t>(HMAXBX, layer_tiles) : blocks_per_state(ngroups_per_state);
		gg.resize(nl);
		gt.resize(nl);
		for (int l = 0; l < nl; l++) {
			gg[l] = gate_of(c.ugates + 16 * l, false);
			gt[l] = gate_of(c.ugates + 16 * l, true);
		}
		gw.resize(G);
		for (int q = 0; q < G; q++) gw[q] = make_pair_(L, c.wires[2 * q], c.wires[2 * q + 1]);
		const size_t doubles = (size_t)nl * S * 32 * nbx + 2 * (size_t)nbx;
		int ret = ensure_device(rt.partials, doubles * sizeof(double));
		if (ret) return ret;
		part = reinterpret_cast<double*>(rt.partials.ptr);
		fpart = reinterpret_cast<double2*>(part + (size_t)nl * S * 32 * nbx);
		return RQC_CUDA(cudaMemsetAsync(part, 0, doubles * sizeof(double), rt.stream));
	}

	// phi_{q-1} = G_q^T phi_q for q = G-1 .. 1 (phi_at(G-1) given), and optionally the
	// cotangent of the circuit input
	template <typename PhiAt>
	int reverse_chain(PhiAt phi_at, int64_t ngroups, double2* dpsi_in)
	{
		const int grid = grid_of(rt, ngroups, 8);
		for (int q = G - 1; q >= 1; q--) {
			cudaEvent_t ev;
			launch_begin(rt, KC_APPLY, &ev);
			k_happly<<<grid, HT, 0, rt.stream>>>(phi_at(q), phi_at(q - 1), gt[q / per], gw[q], L, ngroups);
			launch_end(rt, KC_APPLY, ev);   // launch_begin counted the launch
			if (int e = RQC_CUDA(cudaGetLastError())) return e;
		}
		if (dpsi_in) {
			k_happly<<<grid, HT, 0, rt.stream>>>(phi_at(0), dpsi_in, gt[0], gw[0], L, ngroups);
			if (int e = checked(rt)) return e;
		}
		return OK;
	}

	// one gate of the forward sweep
	// basis: psi_in is the basis columns of the chunk (psi_0 of a column sum)
	int gate(int q, const double2* psi_in, int basis, double2* psi_out, const double2* phi, double2* tan,
	         int64_t ngroups, int64_t sstride, bool with_f)
	{
		const int a = q / per;
		const bool last = q == G - 1;
		const dim3 grid(psi_only ? 1 : 1 + 16 * (a + 1), nbx);
		cudaEvent_t ev;
		launch_begin(rt, KC_HESS, &ev);
		k_hsweep<<<grid, HT, 0, rt.stream>>>(psi_in, basis, src, last ? nullptr : psi_out, phi, tan, gg[a], gw[q], L,
		                                     ngroups, sstride, a, q % per == 0 ? 1 : 0, (last && !keep_final) ? 0 : 1, part,
		                                     S, (with_f && last) ? fpart : nullptr);
		launch_end(rt, KC_HESS, ev);
		return RQC_CUDA(cudaGetLastError());
	}

	// psi_q = G_{q-1} psi_{q-1} for q = 1 .. G-1 into psi_at(q); psi_0 the chunk's basis columns (basis) or psi_at(0)
	template <typename PsiAt>
	int forward_chain(PsiAt psi_at, int64_t ngroups, int basis)
	{
		const int grid = grid_of(rt, ngroups, 8);
		for (int q = 1; q < G; q++) {
			cudaEvent_t ev;
			launch_begin(rt, KC_APPLY, &ev);
			k_happly<<<grid, HT, 0, rt.stream>>>(psi_at(q - 1), psi_at(q), gg[(q - 1) / per], gw[q - 1], L, ngroups,
			                                     q == 1 ? basis : 0, src);
			launch_end(rt, KC_APPLY, ev);
			if (int e = RQC_CUDA(cudaGetLastError())) return e;
		}
		return OK;
	}

	// one layer with shared-memory tiles (L <= 12)
	int layer(int a, const double2* psi, int basis, const double2* phi, double2* tan, int64_t ncols,
	          int64_t sstride, bool with_f)
	{
		static PerDevice prepared;
		int& smem_set = prepared[rt];
		if (!smem_set) {
			if (int e = RQC_CUDA(cudaFuncSetAttribute(k_hlayer, cudaFuncAttributeMaxDynamicSharedMemorySize,
			                                          (int)(HTILE * sizeof(double2)))))
				return e;
			smem_set = true;
		}
		LayerGates lgts;
		lgts.q0 = a * per;
		lgts.per = per;
		for (int k = 0; k < per; k++) lgts.w[k] = gw[a * per + k];
		const bool last = a == nl - 1 && !keep_final;
		const dim3 grid(psi_only ? 1 : 1 + 16 * (a + 1), nbx);
		cudaEvent_t ev;
		launch_begin(rt, KC_HESS, &ev);
		k_hlayer<<<grid, HT, HTILE * sizeof(double2), rt.stream>>>(psi, basis, src, phi, tan, gg[a], lgts, L, ncols, sstride, a,
		                                                             last ? 1 : 0, part, S,
		                                                             (with_f && last) ? fpart : nullptr);
		launch_end(rt, KC_HESS, ev);
		return RQC_CUDA(cudaGetLastError());
	}

	int assemble(double2* d_rec)
	{
		const int m = 16 * nl;
		const int64_t n = 1 + 16 * (int64_t)nl + (int64_t)m * m;
		k_hassemble<<<grid_of(rt, n, 4), HT, 0, rt.stream>>>(part, nbx, nl, S, fpart, d_rec);
		return checked(rt);
	}
};

// every layer gate unitary to 1e-14 and every layer's pairs on wires of their own; with one pair
// a layer the diagonal blocks are exactly zero, which the difference in k_hrecord is not
bool layer_sweep_ok(const HessCircuit& c)
{
	const int per = c.L / 2;
	if (per < 2 || per > 16) return false;
	for (int l = 0; l < c.nlayers; l++) {
		const double2* g = c.ugates + 16 * l;
		for (int r = 0; r < 4; r++)
			for (int k = 0; k < 4; k++) {
				double re = 0, im = 0;
				for (int q = 0; q < 4; q++) {
					const double2 x = g[4 * q + r], y = g[4 * q + k];
					re += x.x * y.x + x.y * y.y;
					im += x.x * y.y - x.y * y.x;
				}
				if (!(fabs(re - (r == k ? 1.0 : 0.0)) <= 1e-14 && fabs(im) <= 1e-14)) return false;
			}
		std::vector<LayerGate> gates;
		for (int p = 0; p < per; p++)
			gates.push_back({g, c.wires[2 * (l * per + p)], c.wires[2 * (l * per + p) + 1]});
		if (!gates_disjoint(c.L, gates)) return false;
	}
	return true;
}

struct LayerSweep
{
	Runtime& rt;
	const HessCircuit& c;
	int L, nl, per;
	bool hess = true;
	std::vector<std::vector<LayerGate>> layers;
	std::vector<LayerParts> parts;
	double2* d_part = nullptr;
	const double2* d_ug = nullptr;
	double2* d_f = nullptr;
	int nf = 0, most_tiles = 1;
	const LayerParts* d_parts = nullptr;

	LayerSweep(Runtime& r, const HessCircuit& hc, bool with_hess)
		: rt(r), c(hc), L(hc.L), nl(hc.nlayers), per(hc.L / 2), hess(with_hess), layers(hc.nlayers)
	{
		for (int l = 0; l < nl; l++)
			for (int p = 0; p < per; p++)
				layers[l].push_back({c.ugates + 16 * l, c.wires[2 * (l * per + p)], c.wires[2 * (l * per + p) + 1]});
	}

	// partial-sum slots for chunks of up to K amplitudes per state: enough splits to fill the
	// GPU (three blocks of four warps per SM), of one run per warp at least (of two: L = 6, 8
	// layers, 15 samples 617 us, now 424; L = 8, 5 layers, all columns 355 us, now 321)
	int init(int64_t K)
	{
		static PerDevice prepared;
		int& smem_set = prepared[rt];
		if (!smem_set) {
			if (int e = RQC_CUDA(cudaFuncSetAttribute(k_hgemm, cudaFuncAttributeMaxDynamicSharedMemorySize, GSMEM))) return e;
			smem_set = true;
		}
		int64_t off = 0;
		parts.resize(nl);
		for (int a = 0; a < nl; a++) {
			const int ntile = hess ? (16 * (a + 1) + 1 + GN - 1) / GN : 1;
			const int64_t fill = (3 * (int64_t)rt.num_sms + ntile - 1) / ntile, most = (K + GRUN * GW - 1) / (GRUN * GW);
			most_tiles = std::max(most_tiles, ntile);
			parts[a] = {off, (int)std::max<int64_t>(1, std::min(fill, most)), ntile};
			off += (int64_t)ntile * parts[a].nsplit * GSLOT;
		}
		// sums | unit gates | parts of f | slots
		nf = grid_of(rt, K, 8);
		const size_t bytes = ((size_t)off + 16 * (size_t)nl + nf) * sizeof(double2) + nl * sizeof(LayerParts);
		int ret = ensure_device(rt.partials, bytes);
		if (ret) return ret;
		d_part = static_cast<double2*>(rt.partials.ptr);
		double2* ug = d_part + off;
		d_f = ug + 16 * nl;
		LayerParts* lp = reinterpret_cast<LayerParts*>(d_f + nf);
		if ((ret = RQC_CUDA(cudaMemsetAsync(d_f, 0, nf * sizeof(double2), rt.stream)))) return ret;
		d_ug = ug;
		d_parts = lp;
		if ((ret = RQC_CUDA(cudaMemcpyAsync(ug, c.ugates, 16 * (size_t)nl * sizeof(double2), cudaMemcpyHostToDevice, rt.stream))))
			return ret;
		return RQC_CUDA(cudaMemcpyAsync(lp, parts.data(), nl * sizeof(LayerParts), cudaMemcpyHostToDevice, rt.stream));
	}

	// psi at every layer's output (psi + a K); psi_0 in `in`, or the basis columns of *src
	int forward(const double2* in, const ColumnSource* src, double2* psi, int64_t ncols)
	{
		const int64_t K = ncols << L;
		for (int a = 0; a < nl; a++)
			if (int e = layer_apply(rt, L, layers[a], false, a == 0 ? in : psi + (a - 1) * K, psi + a * K, ncols,
			                        a == 0 ? src : nullptr))
				return e;
		return OK;
	}

	// phi at every layer's output from that of the last
	int reverse(double2* phi, int64_t ncols)
	{
		const int64_t K = ncols << L;
		for (int a = nl - 1; a >= 1; a--)
			if (int e = layer_apply(rt, L, layers[a], true, phi + a * K, phi + (a - 1) * K, ncols)) return e;
		return OK;
	}

	// tangents and sums of one chunk; tan: 16 states per layer, cot: 16 states.  At the end the
	// tangents are at the circuit's output.
	int sweep(const double2* psi, const double2* phi, double2* tan, double2* cot, int64_t ncols, bool add)
	{
		const int64_t K = ncols << L;
		for (int a = 0; a < nl; a++) {
			if (hess && a > 0)
				if (int e = layer_apply(rt, L, layers[a], false, tan, tan, 16 * a * ncols)) return e;
			LayerWires w;
			w.n = per;
			for (int q = 0; q < per; q++) {
				w.bi[q] = (int8_t)(L - 1 - layers[a][q].i);
				w.bj[q] = (int8_t)(L - 1 - layers[a][q].j);
			}
			w.g = gate_of(c.ugates + 16 * a, false);
			k_hstates<<<std::min(nf, grid_of(rt, K, 8)), 256, 0, rt.stream>>>(psi + a * K, phi + a * K, w, K, hess ? tan + 16 * a * K : nullptr, cot,
			                                                    a == nl - 1 ? d_f : nullptr);
			if (int e = checked(rt)) return e;
			cudaEvent_t ev;
			launch_begin(rt, KC_HESS, &ev);
			k_hgemm<<<dim3(parts[a].ntile, parts[a].nsplit), 32 * GW, GSMEM, rt.stream>>>(
				cot, tan, psi + a * K, K, hess ? 16 * (a + 1) : 0, d_part + parts[a].off, add ? 1 : 0);
			launch_end(rt, KC_HESS, ev);
			if (int e = RQC_CUDA(cudaGetLastError())) return e;
		}
		return OK;
	}

	int record(double2* d_rec, bool with_f)
	{
		const int blocks = hess ? nl * (nl + 1) / 2 : nl;
		k_hsum<<<dim3(most_tiles, nl, GSLOT / 32), 256, 0, rt.stream>>>(d_part, d_parts);
		if (int e = checked(rt)) return e;
		k_hrecord<<<blocks, 256, 0, rt.stream>>>(d_part, d_parts, d_ug, nl, with_f ? d_f : nullptr, nf, hess ? 1 : 0, d_rec);
		return checked(rt);
	}
};

// Hessians of so few amplitudes that either sweep waits for its launches: the layer sweep makes five a layer,
// of which the product takes longer with every tangent tile, the general sweep two a gate and one a layer.
// General against layer sweep (samples unless named): L = 4, 8 layers, 8: 268 us and 394 us, 128: 353 us and
// 425 us, 512: 436 us and 435 us, all columns 257 us and 382 us; 2 layers, 8: 135 us and 170 us.  L = 6, 8 layers,
// 4: 337 us and 432 us, 16: 403 us and 433 us, 64: 502 us and 446 us, one column per orbit (24) 417 us and
// 421 us.  L = 8, 8 layers, 1: 399 us and 438 us, 2: 437 us and 437 us, 4: 485 us and 437 us.  L = 10, 8 layers,
// 1: 566 us and 458 us.
bool latency_bound(int L, int64_t ncols) { return L <= 8 && ncols <= (1 << 16) >> (2 * L); }

// States of the layer sweep per column: psi and phi at every layer's output, 16 tangents per
// layer (before that a scratch state of the target), 16 cotangent states, the sample states.
// (The general sweep holds fewer for short circuits: 16 nl + 2 G + 2 up to L = 12.)
size_t layer_column_bytes(int L, int nl, bool samp)
{
	return (size_t)(2 * nl + 16 * nl + 16 + (samp ? 1 : 0)) * sizeof(double2) << L;
}

// hessian_target_device for unitary gates: the layer sweep over column chunks
int hessian_layers(Runtime& rt, const HessCircuit& c, const TargetSpec& t, double2* d_rec, const SampleSpec* samp)
{
	const int L = c.L, nl = c.nlayers;
	const int64_t N = (int64_t)1 << L;
	const int64_t ncols = samp ? samp->nsamples : (c.columns ? c.ncolumns : N);
	const size_t col_bytes = layer_column_bytes(L, nl, samp != nullptr);
	int64_t C = ncols;
	if (rt.column_chunk > 0) C = std::min<int64_t>(C, rt.column_chunk);
	if (t.ufunc) C = std::min<int64_t>(C, std::max<int64_t>(1, ((int64_t)256 << 20) / (N * 16)));
	C = std::min<int64_t>(C, (int64_t)(workspace_budget(rt, C * col_bytes) / col_bytes));
	if (C < 1) return E_ALLOC;   // (the caller has seen that a column fits)
	int ret = ensure_device(rt.work, (size_t)C * col_bytes);
	if (ret) return ret;
	LayerSweep sw(rt, c, true);
	if ((ret = sw.init(C * N))) return ret;
	for (int64_t b0 = 0; b0 < ncols; b0 += C) {
		const int64_t Cc = std::min(C, ncols - b0), K = Cc * N;
		double2* psi = static_cast<double2*>(rt.work.ptr);
		double2* phi = psi + nl * K;
		double2* tan = phi + nl * K;
		double2* cot = tan + 16 * nl * K;
		double2* states = cot + 16 * K;
		double2* last = phi + (nl - 1) * K;
		ColumnSource src;
		src.tab = c.columns;
		src.b0 = b0;
		src.end = ncols;
		if (samp) {
			if ((ret = haar_states_device(rt, *samp, L, b0, Cc, states))) return ret;
			if ((ret = target_states_device(rt, t, L, states, Cc, last, tan))) return ret;
		} else {
			ColumnSource tsrc = src;
			tsrc.weighted = 1;
			if ((ret = target_columns_device(rt, t, L, tsrc, Cc, last, tan))) return ret;
		}
		if ((ret = sw.forward(samp ? states : nullptr, samp ? nullptr : &src, psi, Cc))) return ret;
		if ((ret = sw.reverse(phi, Cc))) return ret;
		if ((ret = sw.sweep(psi, phi, tan, cot, Cc, b0 > 0))) return ret;
	}
	if ((ret = sw.record(d_rec, true))) return ret;
	if (samp) {
		const int64_t n = (int64_t)hess_record_count(nl);
		k_scale_rec<<<grid_of(rt, n, 4), HT, 0, rt.stream>>>(d_rec, n, (double)N / (double)samp->nsamples);
		ret = checked(rt);
	}
	return ret;
}

}  // namespace

// ------------------------------------------------------------------ engine entry points

int hessian_target_device(Runtime& rt, const HessCircuit& c, const TargetSpec& t, double2* d_rec, const SampleSpec* samp)
{
	const int L = c.L, nl = c.nlayers;
	if (L < 2 || L % 2 || nl < 1) return E_ARG;
	if (samp && samp->nsamples < 1) return E_ARG;
	const int per = L / 2, G = nl * per;
	const int64_t N = (int64_t)1 << L;
	const int64_t ncols = samp ? samp->nsamples : (c.columns ? c.ncolumns : N);   // basis columns, or sample states
	const size_t layer_bytes = layer_column_bytes(L, nl, samp != nullptr);
	if (layer_sweep_ok(c) && !latency_bound(L, ncols) && layer_bytes <= workspace_budget(rt, layer_bytes))
		return hessian_layers(rt, c, t, d_rec, samp);
	// layer kernel (shared-memory tiles) up to L = 12, one kernel per gate beyond
	const bool layered = L <= 12 && per <= HMAXPER;
	// states per column: phi_q of every gate, psi_q of every gate (layered) or two psi
	// buffers, 16 tangents per layer; sampled: the sample states (layered: psi_0) and a target
	// scratch state besides
	const int64_t nstates = G + (layered ? G : 2) + 16 * (int64_t)nl + (samp ? (layered ? 1 : 2) : 0);
	const size_t col_bytes = (size_t)nstates * N * sizeof(double2);
	int64_t C = ncols;
	if (rt.column_chunk > 0) C = std::min<int64_t>(C, rt.column_chunk);
	if (t.ufunc) C = std::min<int64_t>(C, std::max<int64_t>(1, ((int64_t)256 << 20) / (N * 16)));
	C = std::min<int64_t>(C, (int64_t)(workspace_budget(rt, C * col_bytes) / col_bytes));
	if (C < 1) {
		fprintf(stderr, "rqcopt_gpu: one basis column of the Hessian sweep needs %zu bytes of workspace, more than the limit\n",
		        col_bytes);
		return E_ALLOC;
	}
	int ret = ensure_device(rt.work, (size_t)nstates * C * N * sizeof(double2));
	if (ret) return ret;
	double2* phi = reinterpret_cast<double2*>(rt.work.ptr);
	const int64_t cs = C * N;   // elements per chunk state
	double2* P[2] = { phi + (int64_t)G * cs, phi + (int64_t)(G + 1) * cs };
	double2* psi = phi + (int64_t)G * cs;                              // layered: psi_q at psi + q cs
	double2* tan = phi + (int64_t)(G + (layered ? G : 2)) * cs;
	double2* extra = tan + 16 * (int64_t)nl * cs;                       // sampled: scratch (and states)
	double2* states = samp ? (layered ? psi : extra + cs) : nullptr;
	double2* tscratch = samp ? extra : P[0];                            // target scratch
	auto phi_at = [&](int q) { return phi + (int64_t)q * cs; };
	auto psi_at = [&](int q) { return psi + (int64_t)q * cs; };

	Sweep sw(rt, c);
	if ((ret = sw.init(cs / 4, layered ? (C + (HTILE >> L) - 1) / (HTILE >> L) : 0))) return ret;
	for (int64_t b0 = 0; b0 < ncols; b0 += C) {
		const int64_t Cc = std::min(C, ncols - b0);
		const int64_t ngroups = Cc * (N / 4);
		const int basis = samp ? 0 : 1;
		sw.src.tab = c.columns;
		sw.src.b0 = b0;
		sw.src.end = ncols;
		ColumnSource tsrc = sw.src;
		tsrc.weighted = 1;
		if (samp) {
			if ((ret = haar_states_device(rt, *samp, L, b0, Cc, states))) return ret;
			if ((ret = target_states_device(rt, t, L, states, Cc, phi_at(G - 1), tscratch))) return ret;
		} else if ((ret = target_columns_device(rt, t, L, tsrc, Cc, phi_at(G - 1), tscratch))) {
			return ret;
		}
		if ((ret = sw.reverse_chain(phi_at, ngroups, nullptr))) return ret;
		if (layered) {
			if ((ret = sw.forward_chain(psi_at, ngroups, basis))) return ret;
			for (int a = 0; a < nl; a++)
				if ((ret = sw.layer(a, psi, basis, phi, tan, Cc, cs, true))) return ret;
			continue;
		}
		for (int q = 0; q < G; q++) {
			const double2* in = q == 0 ? states : P[(q - 1) & 1];
			if ((ret = sw.gate(q, in, q == 0 ? basis : 0, P[q & 1], phi_at(q), tan, ngroups, cs, true))) return ret;
		}
	}
	if ((ret = sw.assemble(d_rec))) return ret;
	if (samp) {
		const int64_t n = (int64_t)hess_record_count(nl);
		k_scale_rec<<<grid_of(rt, n, 4), HT, 0, rt.stream>>>(d_rec, n, (double)N / (double)samp->nsamples);
		ret = checked(rt);
	}
	return ret;
}

int hessian_single_device(Runtime& rt, const HessCircuit& c, const double2* d_cache, const double2* d_dout,
                          double2* d_dpsi, double2* d_rec)
{
	const int L = c.L, nl = c.nlayers;
	if (L < 2 || L % 2 || nl < 1) return E_ARG;
	const int per = L / 2, G = nl * per;
	const int64_t N = (int64_t)1 << L;
	const bool layered = L <= 12 && per <= HMAXPER;
	// phi_0 .. phi_{G-1} (the last a copy of d_dout) and 16 tangents per layer
	const int64_t nstates = G + 16 * (int64_t)nl;
	int ret = ensure_device(rt.work, (size_t)nstates * N * sizeof(double2));
	if (ret) return ret;
	double2* phi = reinterpret_cast<double2*>(rt.work.ptr);
	double2* tan = phi + (int64_t)G * N;
	auto phi_at = [&](int q) { return phi + (int64_t)q * N; };
	if ((ret = RQC_CUDA(cudaMemcpyAsync(phi_at(G - 1), d_dout, N * sizeof(double2), cudaMemcpyDeviceToDevice, rt.stream))))
		return ret;
	Sweep sw(rt, c);
	if ((ret = sw.init(N / 4, layered ? 1 : 0))) return ret;
	if ((ret = sw.reverse_chain(phi_at, N / 4, d_dpsi))) return ret;
	if (layered) {
		for (int a = 0; a < nl; a++)
			if ((ret = sw.layer(a, d_cache, 0, phi, tan, 1, N, false))) return ret;
	} else {
		for (int q = 0; q < G; q++)
			if ((ret = sw.gate(q, d_cache + (int64_t)q * N, 0, nullptr, phi_at(q), tan, N / 4, N, false))) return ret;
	}
	return sw.assemble(d_rec);
}

int blockenc_device(Runtime& rt, const HessCircuit& c, const TargetSpec& t, int mode, double2* d_rec, double2* d_hess2)
{
	const int L = c.L, nl = c.nlayers;
	if (L < 2 || L % 2 || nl < 1 || mode < 0 || mode > 2) return E_ARG;
	const int per = L / 2, G = nl * per, half = L / 2, m = 16 * nl;
	const int64_t N = (int64_t)1 << L, s = (int64_t)1 << half;
	const bool hess = mode == 2;
	const bool layered = L <= 12 && per <= HMAXPER;
	// layer sweep, states per column: the input states, psi and phi at every layer's output, 16
	// cotangent states, the tangents (Hessian only).
	// General sweep (also where the workspace does not hold a column of the layer sweep): phi_q of
	// every gate; psi_q of every gate (layered) or two psi buffers and the input states; W P e_b;
	// the tangents (Hessian only)
	const int64_t layer_states = 1 + 2 * nl + 16 + (hess ? 16 * (int64_t)nl : 0);
	const size_t layer_bytes = (size_t)layer_states * N * sizeof(double2);
	const int64_t ncols = c.columns ? c.ncolumns : s;
	const bool sweep = layer_sweep_ok(c) && !(hess && latency_bound(L, ncols)) && layer_bytes <= workspace_budget(rt, layer_bytes);
	const int64_t nstates = sweep ? layer_states : G + (layered ? G : 3) + 1 + (hess ? 16 * (int64_t)nl : 0);
	const size_t col_bytes = (size_t)nstates * N * sizeof(double2);
	int64_t C = ncols;
	if (rt.column_chunk > 0) C = std::min<int64_t>(C, rt.column_chunk);
	C = std::min<int64_t>(C, (int64_t)(workspace_budget(rt, C * col_bytes) / col_bytes));
	if (C < 1) return E_ALLOC;
	int ret = ensure_device(rt.work, (size_t)nstates * C * N * sizeof(double2));
	if (ret) return ret;
	double2* phi = reinterpret_cast<double2*>(rt.work.ptr);
	const int64_t cs = C * N;
	double2* P[2] = { phi + (int64_t)G * cs, phi + (int64_t)(G + 1) * cs };
	double2* psi = phi + (int64_t)G * cs;
	double2* states = layered ? psi : phi + (int64_t)(G + 2) * cs;
	double2* wout = phi + (int64_t)(G + (layered ? G : 3)) * cs;
	double2* tan = wout + cs;
	auto phi_at = [&](int q) { return phi + (int64_t)q * cs; };
	auto psi_at = [&](int q) { return psi + (int64_t)q * cs; };
	// per evaluation: -conj(H e_b) for all b, target scratch, Jacobian rows, Gauss-Newton parts, f parts
	const int nres = rt.num_sms * 2;
	const size_t abytes = (2 * (size_t)s * s + (hess ? (size_t)m * C * s + (size_t)m * m : 0) + nres) * sizeof(double2);
	if ((ret = ensure_device(rt.arrays, abytes))) return ret;
	double2* hneg = static_cast<double2*>(rt.arrays.ptr);
	double2* scratch = hneg + s * s;
	double2* jac = scratch + s * s;
	double2* part2 = hess ? jac + (size_t)m * C * s : jac;
	double2* fres = hess ? part2 + (size_t)m * m : jac;
	if ((ret = RQC_CUDA(cudaMemsetAsync(fres, 0, nres * sizeof(double2), rt.stream)))) return ret;
	if (hess && (ret = RQC_CUDA(cudaMemsetAsync(part2, 0, (size_t)m * m * sizeof(double2), rt.stream)))) return ret;
	if ((ret = target_columns_device(rt, t, half, ColumnSource{}, s, hneg, scratch))) return ret;

	if (sweep) {
		LayerSweep ls(rt, c, hess);
		if ((ret = ls.init(C * N))) return ret;
		for (int64_t b0 = 0; b0 < ncols; b0 += C) {
			const int64_t Cc = std::min(C, ncols - b0), K = Cc * N;
			double2* in = phi;
			double2* psi_l = in + K;
			double2* phi_l = psi_l + nl * K;
			double2* cot = phi_l + nl * K;
			double2* tan_l = cot + 16 * K;
			double2* chi = phi_l + (nl - 1) * K;
			k_benc_init<<<grid_of(rt, K, 8), HT, 0, rt.stream>>>(in, L, c.columns, b0, Cc);
			if ((ret = checked(rt))) return ret;
			if ((ret = ls.forward(in, nullptr, psi_l, Cc))) return ret;
			if (mode >= 1 && (ret = RQC_CUDA(cudaMemsetAsync(chi, 0, (size_t)K * sizeof(double2), rt.stream)))) return ret;
			k_benc_residual<<<nres, HT, 0, rt.stream>>>(psi_l + (nl - 1) * K, hneg, L, c.columns, b0, Cc,
			                                            mode >= 1 ? chi : nullptr, fres);
			if ((ret = checked(rt))) return ret;
			if (mode == 0) continue;
			if ((ret = ls.reverse(phi_l, Cc))) return ret;
			if ((ret = ls.sweep(psi_l, phi_l, tan_l, cot, Cc, b0 > 0))) return ret;
			if (hess) {
				k_benc_gather<<<grid_of(rt, (int64_t)m * Cc * s, 8), HT, 0, rt.stream>>>(tan_l, L, Cc, K, m, jac);
				if ((ret = checked(rt))) return ret;
				k_benc_gram<<<m * m, HT, 0, rt.stream>>>(jac, Cc * s, nl, c.columns, b0, half, part2);
				if ((ret = checked(rt))) return ret;
			}
		}
		if (mode >= 1 && (ret = ls.record(d_rec, false))) return ret;
		k_benc_finish<<<grid_of(rt, (int64_t)m * m, 4), HT, 0, rt.stream>>>(part2, nl, fres, nres, d_rec,
		                                                                     hess ? d_hess2 : nullptr);
		return checked(rt);
	}

	Sweep sw(rt, c);
	sw.keep_final = hess;
	sw.psi_only = mode == 1;
	if (mode >= 1 && (ret = sw.init(cs / 4, layered ? (C + (HTILE >> L) - 1) / (HTILE >> L) : 0))) return ret;
	if (mode == 0) {   // the gates and wires of the forward passes
		sw.gg.resize(nl);
		for (int l = 0; l < nl; l++) sw.gg[l] = gate_of(c.ugates + 16 * l, false);
		sw.gw.resize(G);
		for (int q = 0; q < G; q++) sw.gw[q] = make_pair_(L, c.wires[2 * q], c.wires[2 * q + 1]);
	}
	for (int64_t b0 = 0; b0 < ncols; b0 += C) {
		const int64_t Cc = std::min(C, ncols - b0);
		const int64_t ngroups = Cc * (N / 4);
		const int agrid = grid_of(rt, ngroups, 8);
		k_benc_init<<<grid_of(rt, Cc * N, 8), HT, 0, rt.stream>>>(states, L, c.columns, b0, Cc);
		if ((ret = checked(rt))) return ret;
		// forward pass to W P e_b
		if (layered && mode >= 1) {
			if ((ret = sw.forward_chain(psi_at, ngroups, 0))) return ret;
			k_happly<<<agrid, HT, 0, rt.stream>>>(psi_at(G - 1), wout, sw.gg[(G - 1) / per], sw.gw[G - 1], L, ngroups);
			if ((ret = checked(rt))) return ret;
		} else {
			const double2* in = states;
			for (int q = 0; q < G; q++) {
				double2* o = q == G - 1 ? wout : P[q & 1];
				k_happly<<<agrid, HT, 0, rt.stream>>>(in, o, sw.gg[q / per], sw.gw[q], L, ngroups);
				if ((ret = checked(rt))) return ret;
				in = o;
			}
		}
		double2* chi = mode >= 1 ? phi_at(G - 1) : nullptr;
		if (chi && (ret = RQC_CUDA(cudaMemsetAsync(chi, 0, (size_t)Cc * N * sizeof(double2), rt.stream)))) return ret;
		k_benc_residual<<<nres, HT, 0, rt.stream>>>(wout, hneg, L, c.columns, b0, Cc, chi, fres);
		if ((ret = checked(rt))) return ret;
		if (mode == 0) continue;
		if ((ret = sw.reverse_chain(phi_at, ngroups, nullptr))) return ret;
		if (layered) {
			for (int a = 0; a < nl; a++)
				if ((ret = sw.layer(a, psi, 0, phi, tan, Cc, cs, false))) return ret;
		} else {
			for (int q = 0; q < G; q++) {
				const double2* in = q == 0 ? states : P[(q - 1) & 1];
				if ((ret = sw.gate(q, in, 0, P[q & 1], phi_at(q), tan, ngroups, cs, false))) return ret;
			}
		}
		if (hess) {
			k_benc_gather<<<grid_of(rt, (int64_t)m * Cc * s, 8), HT, 0, rt.stream>>>(tan, L, Cc, cs, m, jac);
			if ((ret = checked(rt))) return ret;
			k_benc_gram<<<m * m, HT, 0, rt.stream>>>(jac, Cc * s, nl, c.columns, b0, half, part2);
			if ((ret = checked(rt))) return ret;
		}
	}
	if (mode >= 1 && (ret = sw.assemble(d_rec))) return ret;
	k_benc_finish<<<grid_of(rt, (int64_t)m * m, 4), HT, 0, rt.stream>>>(part2, nl, fres, nres, d_rec,
	                                                                     hess ? d_hess2 : nullptr);
	return checked(rt);
}

int project_hessian_device(Runtime& rt, int nlayers, const double2* d_ugates, const double2* d_rec, double* d_grad,
                           double* d_H, const double2* d_hess2)
{
	const int m = 16 * nlayers;
	const int n = std::max(nlayers, 16 * nlayers * (nlayers + 1) / 2);
	k_hproject<<<(n + 63) / 64, 64, 0, rt.stream>>>(nlayers, d_ugates, d_rec, d_hess2, d_grad, d_H);
	int ret = checked(rt);
	if (ret) return ret;
	k_hmirror<<<grid_of(rt, (int64_t)m * m, 4), HT, 0, rt.stream>>>(m, d_H);
	return checked(rt);
}

int tcg_hmat_device(Runtime& rt, int n, const double* d_grad, const double* d_hess, double radius, int maxiter,
                    double abstol, double reltol, double* d_work, double* d_z, int* d_status)
{
	k_tcg_hmat<<<1, HT, 0, rt.stream>>>(n, d_grad, d_hess, radius, maxiter, abstol, reltol, d_work, d_work + n,
	                                    d_work + 2 * n, d_z, d_status);
	return checked(rt);
}

int gemv_device(Runtime& rt, int n, const double* d_a, const double* d_x, double* d_y)
{
	k_gemv<<<(n + 127) / 128, 128, 0, rt.stream>>>(n, d_a, d_x, d_y);
	return checked(rt);
}

int gate_to_array_device(Runtime& rt, int L, int ns, const double2* gate, int i, int j, const double2* d_in,
                         double2* d_out)
{
	const int64_t n = ((int64_t)1 << (L - 2)) * ns;
	k_gate_array<<<grid_of(rt, n, 8), HT, 0, rt.stream>>>(d_in, d_out, gate_of(gate, false), make_pair_(L, i, j), ns, n);
	return checked(rt);
}

int gate_backward_array_device(Runtime& rt, int L, int ns, int i, int j, const double2* d_psi, const double2* d_dout,
                               double2* d_dgates)
{
	const int64_t ngroups = (int64_t)1 << (L - 2);
	const int nbx = blocks_per_state(ngroups);
	int ret = ensure_device(rt.partials, (size_t)ns * 32 * nbx * sizeof(double));
	if (ret) return ret;
	double* part = reinterpret_cast<double*>(rt.partials.ptr);
	k_gate_backward_array<<<dim3(ns, nbx), HT, 0, rt.stream>>>(d_psi, d_dout, make_pair_(L, i, j), ns, ngroups, part);
	if ((ret = checked(rt))) return ret;
	k_array_sum<<<(16 * ns + 127) / 128, 128, 0, rt.stream>>>(part, ns, nbx, d_dgates);
	return checked(rt);
}

int gate_placeholder_device(Runtime& rt, int L, int i, int j, const double2* d_psi, double2* d_out)
{
	const int64_t ngroups = (int64_t)1 << (L - 2);
	k_placeholder<<<grid_of(rt, ngroups, 8), HT, 0, rt.stream>>>(d_psi, d_out, make_pair_(L, i, j), ngroups);
	return checked(rt);
}

}  // namespace rqc
