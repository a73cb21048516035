// Small evaluations: f, gradient and Hessian-vector product of a circuit whose basis
// columns fit a block's shared memory, in two launches.
//
// An evaluation of a few qubits is bound by latency: as passes (engine_fused.cu) it is a
// dozen or more launches of which each does a microsecond of work (L = 6, depth 5: 13
// launches, 165 us on the device, 207 us a call; here 2 launches).  k_small runs the whole
// evaluation of a column in one block: phi = -conj(U e_b) (target gates, or a column of a
// dense U), the forward sweep of psi and dpsi, f, and the reverse sweep, with the four states
// in shared memory throughout.  Four threads share an amplitude group; thread q computes
// component q of every product and owns row q of the outer sums, so that a group's exchange
// stays inside a warp and each gate costs one block barrier.
//
// The forward sweep leaves the state entering each gate in a scratch array (in L2 up to a
// quarter of SMALL_MAX_WORK); the reverse sweep brings the next gate's by cp.async into a
// second pair of tiles while it works on the current one, so that a gate's outer sums
//   dG += phi (x) psi,   HZ += phi (x) dpsi + dphi (x) psi
// and its moves phi <- G^T phi, dphi <- G^T dphi + Z^T phi are all independent.  (Rebuilding
// the states with adjoint gates instead, 12 more products per group and gate, measured the
// same time at L = 6 and 2.5 times the rounding error.)  The gates of a brickwall layer are
// copies of one, so the sums add up over the layer.  Sums per block go to fixed slots that
// k_small_post adds in block order (compensated), so results are deterministic.
#include "engine_small.h"

#include <string.h>
#include <algorithm>

#include "rqc_common.cuh"

namespace rqc {

namespace {

constexpr int SMALL_THREADS = 384;     // most threads per block (three roles of 128)
constexpr int SMALL_MAX_L = 10;        // eight tiles of a column: 128 KB
constexpr int SMALL_MAX_UNITS = 128;   // gate tables in shared memory: 512 B per unit
constexpr size_t SMALL_SMEM = 200 * 1024;
// Amplitudes of all columns up to which an evaluation runs here: a block takes its column at the rate of its
// chain of barriers, and beyond a wave or two of blocks the pass engine is the faster one; HVPs, with twice
// the tiles a block, from half as many.  Small engine against passes: L = 8, 256 columns, 60 gates f 72 and
// 167 us, gradient 140 and 346 us, HVP 271 and 461 us; L = 9, 512 columns, 40 gates 99 and 146, 235 and 279, 483
// and 419 us; in 256 paired columns gradient 130 and 263, HVP 260 and 344 us; L = 10, 208 columns, 45 gates 127
// and 214, 232 and 356, 467 and 496 us; 512 paired columns, 30 gates gradient 275 and 302, HVP 586 and 481 us;
// 1024 columns, 30 gates 187 and 165, 472 and 386, 1007 and 698 us.
constexpr int64_t SMALL_MAX_AMPS = 1 << 19, SMALL_MAX_AMPS_HVP = (1 << 18) - 1;
// Beyond, evaluations of so few gates (the target's included) that launches weigh more: HVP of 12 gates at L = 9
// 162 and 169 us.  On 1024 columns up to nine gates stay in two launches though the passes are a little faster
// (seven gates: f 89 and 82 us, gradient 137 and 127 us, HVP 244 and 195 us).
constexpr int SMALL_FEW_GATES = 15, SMALL_FEW_GATES_1024 = 9;
// Amplitude x gate updates: 512 MB of states
constexpr double SMALL_MAX_WORK = 1 << 24;
constexpr int SLOT = 64;               // doubles per unit and block: row q of dG (8), of HZ (8)

struct SmallArgs
{
	int L, G, per, nunits, Gt;
	int cb;                  // columns per block
	int real;                // paired real columns: clear the imaginary parts of the sums
	ColumnSource src;
	const double2* ug;       // [nunits][16]
	const double2* uz;
	const int* bits;         // [2 (G + Gt)] state bits of the gates' wires, circuit then target
	const double2* tg;       // [Gt][16]
	const double2* dense;    // U row-major, or null
	double* part;            // [blocks][2 + SLOT nunits]
	double2* states;         // [blocks][G - 1][psi, dpsi][cb 2^L]: the states entering gates 1 .. G-1
};

// place of amplitude i in shared memory: 16-byte words of a 128-byte line permuted so that
// group members at strides of 4 and 8 amplitudes fall into different banks
__device__ __forceinline__ int swz(int i) { return i ^ ((i >> 3) & 7); }

// The groups of one gate.  swz is linear over XOR, so a member's place is the group's base
// place XOR the member's own, both fixed per gate and per task.
struct Group
{
	int lo, hi, m[4];
	__device__ __forceinline__ explicit Group(int2 w) : lo(min(w.x, w.y)), hi(max(w.x, w.y))
	{
		m[0] = 0;
		m[1] = swz(1 << w.y);
		m[2] = swz(1 << w.x);
		m[3] = m[1] ^ m[2];
	}
	// place of member 0 of group gi (over all columns of the block)
	__device__ __forceinline__ int base(int gi, int lg, int L) const
	{
		int g = gi & ((1 << lg) - 1);
		g = ((g >> lo) << (lo + 1)) | (g & ((1 << lo) - 1));
		g = ((g >> hi) << (hi + 1)) | (g & ((1 << hi) - 1));
		return swz(((gi >> lg) << L) | g);
	}
};

// sum of a[m] x[m]: the two products of each component in chains of their own (a single warp
// waits for each dependent FMA)
__device__ __forceinline__ double2 dot4(const double2 a[4], const double2 x[4])
{
	double rr = a[0].x * x[0].x, ii = a[0].y * x[0].y, ri = a[0].x * x[0].y, ir = a[0].y * x[0].x;
#pragma unroll
	for (int m = 1; m < 4; m++) {
		rr = fma(a[m].x, x[m].x, rr);
		ii = fma(a[m].y, x[m].y, ii);
		ri = fma(a[m].x, x[m].y, ri);
		ir = fma(a[m].y, x[m].x, ir);
	}
	return make_double2(rr - ii, ri + ir);
}

// sums of v[k] over the lanes that share q = lane & 3: lane l gets that of entry
// 4 (l >> 4 & 1) + 2 (l >> 3 & 1) + (l >> 2 & 1)
__device__ __forceinline__ double row_sums(double (&v)[8], int lane)
{
#pragma unroll
	for (int o = 16, h = 4; o >= 4; o >>= 1, h >>= 1) {
		const bool up = (lane & o) != 0;
#pragma unroll
		for (int k = 0; k < h; k++) {
			const double send = up ? v[k] : v[k + h];
			const double keep = up ? v[k + h] : v[k];
			v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
		}
	}
	return v[0];
}

// acc[c] += p x[c] (complex, c < 4)
__device__ __forceinline__ void outer_row(double (&acc)[8], double2 p, const double2 x[4])
{
#pragma unroll
	for (int c = 0; c < 4; c++) {
		const double2 v = cfma(p, x[c], make_double2(acc[2 * c], acc[2 * c + 1]));
		acc[2 * c] = v.x;
		acc[2 * c + 1] = v.y;
	}
}

__device__ __forceinline__ void copy16(double2* smem, const double2* gmem)
{
	const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem) : "memory");
}

// Threads: `nb` per role.  With one role every thread does all of a gate's work on its groups;
// with ROLES = 3 (columns too small to fill a block) the warps of role 0 take the value part
// (psi, dG, phi), those of role 1 the tangent of psi and HZ, those of role 2 the copies of
// forward states and the tangent of phi.  All states have two tiles, read and written in turn,
// so that a gate costs one barrier whatever the roles.
template <int MODE, int ROLES>
__global__ void __launch_bounds__(SMALL_THREADS) k_small(SmallArgs a, int nb)
{
	constexpr bool TAN = MODE == EVAL_HVP;
	extern __shared__ __align__(16) double2 sm[];
	__shared__ double red[2][2][SMALL_THREADS / 32][32];   // units in turn: dG, HZ: per warp
	__shared__ double fred[2][SMALL_THREADS / 32];
	const int L = a.L, N = 1 << L, T = a.cb << L;
	double2* Psi = sm;                       // [2]
	double2* Phi = sm + 2 * T;               // [2]
	double2* dPsi = TAN ? sm + 4 * T : nullptr;
	double2* dPhi = TAN ? sm + 6 * T : nullptr;
	double2* tab = sm + (TAN ? 8 : 4) * T;   // per unit: G, and for HVPs Z
	constexpr int US = TAN ? 32 : 16;
	double2* ttab = tab + US * a.nunits;     // the target's gates, conjugated
	int2* bits = reinterpret_cast<int2*>(ttab + 16 * a.Gt);
	int2* tbits = bits + a.G;
	constexpr int NS = TAN ? 2 : 1;
	double2* states = MODE == EVAL_F ? nullptr : a.states + (size_t)blockIdx.x * (a.G - 1) * NS * T;
	const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
	const int role = ROLES == 1 ? 0 : tid / nb, rt = ROLES == 1 ? tid : tid - role * nb;
	const bool value = ROLES == 1 || role == 0, tanp = TAN && (ROLES == 1 || role == 1);
	const bool third = ROLES == 1 || role == 2;
	const int q = tid & 3;
	const int lg = L - 2, ntasks = a.cb << L;   // four threads per group: one task per amplitude
	const int64_t col0 = (int64_t)blockIdx.x * a.cb;
	double* part = a.part + (size_t)blockIdx.x * (2 + SLOT * (size_t)a.nunits);

	for (int e = tid; e < 16 * a.nunits; e += nt) {
		const int u = e >> 4, w = e & 15;
		tab[u * US + w] = a.ug[e];
		if (TAN) tab[u * US + 16 + w] = a.uz[e];
	}
	for (int e = tid; e < 16 * a.Gt; e += nt) ttab[e] = make_double2(a.tg[e].x, -a.tg[e].y);
	for (int e = tid; e < a.G + a.Gt; e += nt) bits[e] = make_int2(a.bits[2 * e], a.bits[2 * e + 1]);
	ColumnSource wsrc = a.src;
	wsrc.weighted = 1;
	int ph = a.dense ? 0 : a.Gt & 1;   // the tile that holds phi once the target is done
	for (int e = tid; e < T; e += nt) {
		const int c = e >> L, row = e & (N - 1), p = swz(e);
		Psi[p] = basis_amp<double>(a.src, row, col0 + c);
		if (TAN) {
			dPsi[p] = make_double2(0, 0);
			dPhi[p] = make_double2(0, 0);
			dPhi[T + p] = make_double2(0, 0);
		}
		if (a.dense) Phi[p] = cneg_conj(dense_amp(a.dense, L, a.src, row, col0 + c));
		else Phi[p] = cneg_conj(basis_amp<double>(wsrc, row, col0 + c));
	}
	__syncthreads();

	// phi = -conj(U e): the conjugate gates on the negated conjugate column
	if (!a.dense) {
		for (int k = 0; k < a.Gt; k++) {
			const Group gr(tbits[k]);
			const int mq = q == 0 ? 0 : q == 1 ? gr.m[1] : q == 2 ? gr.m[2] : gr.m[3];
			const double2* in = Phi + (k & 1) * T;
			double2* out = Phi + (~k & 1) * T;
			double2 g[4];
#pragma unroll
			for (int m = 0; m < 4; m++) g[m] = ttab[16 * k + 4 * q + m];
			for (int t = tid; t < ntasks; t += nt) {
				const int at = gr.base(t >> 2, lg, L);
				double2 x[4];
#pragma unroll
				for (int m = 0; m < 4; m++) x[m] = in[at ^ gr.m[m]];
				out[at ^ mq] = dot4(g, x);
			}
			__syncthreads();
		}
	}

	// forward
	int cur = 0;   // the tile that holds psi, dpsi
	for (int k = 0, u = 0, r = 0; k < a.G; k++, cur ^= 1) {
		const Group gr(bits[k]);
		const int mq = q == 0 ? 0 : q == 1 ? gr.m[1] : q == 2 ? gr.m[2] : gr.m[3];
		const double2* gt = tab + u * US + 4 * q;
		const double2* in = Psi + cur * T;
		const double2* din = TAN ? dPsi + cur * T : nullptr;
		double2* out = Psi + (cur ^ 1) * T;
		double2* dout = TAN ? dPsi + (cur ^ 1) * T : nullptr;
		if (MODE != EVAL_F && k > 0 && third) {
			double2* st = states + (size_t)(k - 1) * NS * T;
			for (int e = rt; e < T; e += nb) {
				st[e] = in[e];
				if (TAN) st[T + e] = din[e];
			}
		}
		if (value || tanp) {
			double2 g[4], z[4];
#pragma unroll
			for (int m = 0; m < 4; m++) {
				g[m] = gt[m];
				if (tanp) z[m] = gt[16 + m];
			}
			for (int t = rt; t < ntasks; t += nb) {
				const int at = gr.base(t >> 2, lg, L);
				double2 x[4], dx[4];
#pragma unroll
				for (int m = 0; m < 4; m++) {
					x[m] = in[at ^ gr.m[m]];
					if (tanp) dx[m] = din[at ^ gr.m[m]];
				}
				if (value) out[at ^ mq] = dot4(g, x);
				if (tanp) dout[at ^ mq] = cadd(dot4(z, x), dot4(g, dx));
			}
		}
		if (++r == a.per) { r = 0; u++; }
		__syncthreads();
	}

	// f = phi . psi
	{
		double fx = 0, fy = 0;
		for (int e = tid; e < T; e += nt) {
			const double2 p = Phi[ph * T + e], v = Psi[cur * T + e];
			fx += p.x * v.x - p.y * v.y;
			fy += p.x * v.y + p.y * v.x;
		}
		fx = warp_sum(fx);
		fy = warp_sum(fy);
		if (lane == 0) { fred[0][warp] = fx; fred[1][warp] = fy; }
		__syncthreads();
		if (tid < 2) {
			double s = 0;
			for (int w = 0; w < nwarps; w++) s += fred[tid][w];
			part[tid] = s;
		}
	}
	if (MODE == EVAL_F) return;

	// the state entering gate k into tile b of psi, dpsi
	auto fetch = [&](int k, int b, int from, int step) {
		double2* p = Psi + b * T;
		double2* d = TAN ? dPsi + b * T : nullptr;
		if (k > 0) {
			const double2* st = states + (size_t)(k - 1) * NS * T;
			for (int e = from; e < T; e += step) {
				copy16(p + e, st + e);
				if (TAN) copy16(d + e, st + T + e);
			}
		} else if (k == 0) {
			for (int e = from; e < T; e += step) {
				p[swz(e)] = basis_amp<double>(a.src, e & (N - 1), col0 + (e >> L));
				if (TAN) d[e] = make_double2(0, 0);
			}
		}
		asm volatile("cp.async.commit_group;\n" ::: "memory");
	};
	auto arrived = [] { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); };

	// reverse
	double ag[8], ah[8];
#pragma unroll
	for (int e = 0; e < 8; e++) ag[e] = ah[e] = 0;
	fetch(a.G - 1, cur ^ 1, tid, nt);   // psi at the output (tile cur) is still being read for f
	arrived();
	__syncthreads();
	cur ^= 1;
	for (int k = a.G - 1, u = a.nunits - 1, r = a.per - 1; k >= 0; k--, cur ^= 1, ph ^= 1) {
		if (third) fetch(k - 1, cur ^ 1, rt, nb);   // that tile's last readers are behind the barrier
		const double2* X = Psi + cur * T;
		const double2* dX = TAN ? dPsi + cur * T : nullptr;
		const double2* P = Phi + ph * T;
		const double2* dP = TAN ? dPhi + ph * T : nullptr;
		double2* Po = Phi + (ph ^ 1) * T;
		double2* dPo = TAN ? dPhi + (ph ^ 1) * T : nullptr;
		const Group gr(bits[k]);
		const int mq = q == 0 ? 0 : q == 1 ? gr.m[1] : q == 2 ? gr.m[2] : gr.m[3];
		const double2* gt = tab + u * US + q;
		double2 g[4], z[4];   // column q of G and Z
#pragma unroll
		for (int m = 0; m < 4; m++) {
			if (value || third) g[m] = gt[4 * m];
			if (TAN && third) z[m] = gt[16 + 4 * m];
		}
		for (int t = rt; t < ntasks; t += nb) {
			const int at = gr.base(t >> 2, lg, L), own = at ^ mq;
			double2 x[4], p[4], dp[4];
			if (value || tanp) {
#pragma unroll
				for (int m = 0; m < 4; m++) x[m] = X[at ^ gr.m[m]];
			}
			if (value || (TAN && third)) {
#pragma unroll
				for (int m = 0; m < 4; m++) p[m] = P[at ^ gr.m[m]];
			}
			if (value) {
				outer_row(ag, P[own], x);
				Po[own] = dot4(g, p);
			}
			if (tanp) {
				double2 dx[4];
#pragma unroll
				for (int m = 0; m < 4; m++) dx[m] = dX[at ^ gr.m[m]];
				outer_row(ah, P[own], dx);
				outer_row(ah, dP[own], x);
			}
			if (TAN && third) {
#pragma unroll
				for (int m = 0; m < 4; m++) dp[m] = dP[at ^ gr.m[m]];
				dPo[own] = cadd(dot4(z, p), dot4(g, dp));
			}
		}
		const bool done = r == 0;   // the unit's last gate of the sweep
		if (done) {
			const int e = 8 * q + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
			if (value) red[u & 1][0][warp][e] = row_sums(ag, lane);
			if (tanp) red[u & 1][1][warp][e] = row_sums(ah, lane);
#pragma unroll
			for (int i = 0; i < 8; i++) ag[i] = ah[i] = 0;
		}
		arrived();
		__syncthreads();
		if (done) {
			// warp 0 adds up dG, warp 1 (or 0) HZ, over the warps that hold them; this half of red is
			// written again two units on, behind the next barrier
			const int nw = nb >> 5;
			double* o = part + 2 + SLOT * (size_t)u;
			const int row = lane >> 3, v = lane & 7;
			if (warp == 0) {
				double s = 0;
				for (int w = 0; w < nw; w++) s += red[u & 1][0][w][lane];
				o[16 * row + v] = s;
			}
			if (TAN && warp == (nwarps > 1 ? 1 : 0)) {
				double s = 0;
				for (int w = 0; w < nw; w++) s += red[u & 1][1][(ROLES == 1 ? 0 : nw) + w][lane];
				o[16 * row + 8 + v] = s;
			}
			if (!TAN && warp == 0) o[16 * row + 8 + v] = 0;
			r = a.per;
			u--;
		}
		r--;
	}
}

// Unit u (one block each): the sums dG, HZ over blocks and their projection (src/target.c:410-430),
// a thread per matrix entry; the last block sums f.
__global__ void __launch_bounds__(RED_GROUPS * SLOT) k_small_post(SmallArgs a, int nblk, int mode, SmallOut out)
{
	__shared__ double red[RED_GROUPS][SLOT];
	__shared__ double raw[SLOT];
	__shared__ double2 V[16], Z[16], D[16], H[16], A[16], B[16], X[16];
	const int u = blockIdx.x, t = threadIdx.x;
	const size_t stride = 2 + SLOT * (size_t)a.nunits;
	if (u == a.nunits) {
		const double s = block_column_sum<SLOT>(a.part + (t & 1), nblk, stride, red);
		if (t < 2 && out.f) reinterpret_cast<double*>(out.f)[t] = a.real && t == 1 ? 0.0 : s;
		return;
	}
	if (mode == EVAL_F) return;
	const bool tan = mode == EVAL_HVP;
	const double s = block_column_sum<SLOT>(a.part + 2 + SLOT * (size_t)u + (t % SLOT), nblk, stride, red);
	if (t < SLOT) raw[t] = a.real && (t & 1) ? 0.0 : s;
	if (t < 16) {
		V[t] = a.ug[16 * u + t];
		Z[t] = tan ? a.uz[16 * u + t] : make_double2(0, 0);
	}
	__syncthreads();
	if (t >= 16) return;
	const unsigned mask = 0xffffu;
	const int r = t >> 2, c = t & 3;
	auto conj = [](double2 v) { return make_double2(v.x, -v.y); };
	const double2 dg = make_double2(raw[16 * r + 2 * c], raw[16 * r + 2 * c + 1]);
	const double2 hz = make_double2(raw[16 * r + 8 + 2 * c], raw[16 * r + 9 + 2 * c]);
	if (out.dunits) out.dunits[16 * u + t] = dg;
	if (out.hunits && tan) out.hunits[16 * u + t] = hz;
	D[t] = conj(dg);
	__syncwarp(mask);
	// x = Re + Im of the anti-Hermitian part of V^+ M
	auto tangent = [&](const double2* M, double* x) {
		double2 w = make_double2(0, 0);
		for (int m = 0; m < 4; m++) w = cfma(conj(V[4 * m + r]), M[4 * m + c], w);
		X[t] = w;
		__syncwarp(mask);
		const double2 wt = X[4 * c + r];
		if (x) x[16 * u + t] = 0.5 * (w.x - wt.x) + 0.5 * (w.y + wt.y);
		__syncwarp(mask);
	};
	if (out.grad) tangent(D, out.grad);
	if (!tan || !out.hvp) return;
	// minus (Z D^+ V + V D^+ Z) / 2
	double2 av = make_double2(0, 0), bz = make_double2(0, 0);
	for (int m = 0; m < 4; m++) {
		av = cfma(conj(D[4 * m + r]), V[4 * m + c], av);
		bz = cfma(conj(D[4 * m + r]), Z[4 * m + c], bz);
	}
	A[t] = av;
	B[t] = bz;
	__syncwarp(mask);
	double2 pd = make_double2(0, 0);
	for (int i = 0; i < 4; i++) {
		pd = cfma(Z[4 * r + i], A[4 * i + c], pd);
		pd = cfma(V[4 * r + i], B[4 * i + c], pd);
	}
	H[t] = make_double2(hz.x - 0.5 * pd.x, -hz.y - 0.5 * pd.y);
	__syncwarp(mask);
	tangent(H, out.hvp);
}

// columns per block: enough groups to fill a warp
int columns_per_block(int L) { return L >= 5 ? 1 : 32 >> L; }

int block_count(int L, int64_t ncols) { return (int)((ncols + columns_per_block(L) - 1) / columns_per_block(L)); }

// bytes of the states entering gates 1 .. G-1, of all blocks
size_t states_bytes(int L, int G, int64_t ncols, int mode)
{
	if (mode == EVAL_F) return 0;
	return (size_t)block_count(L, ncols) * (G - 1) * (mode == EVAL_HVP ? 2 : 1) * ((size_t)columns_per_block(L) << L) * sizeof(double2);
}

size_t small_smem(int L, int nunits, int G, int Gt, bool tan)
{
	return ((tan ? 8 : 4) * ((size_t)columns_per_block(L) << L) + (size_t)nunits * (tan ? 32 : 16) + 16 * (size_t)Gt) * sizeof(double2) +
	       (size_t)(G + Gt) * sizeof(int2);
}

template <int MODE, int ROLES>
int launch_small_as(Runtime& rt, const SmallArgs& a, int blocks, int nb)
{
	static PerDevice prepared;
	int& ready = prepared[rt];
	if (!ready) {
		if (int e = RQC_CUDA(cudaFuncSetAttribute(k_small<MODE, ROLES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                                          (int)SMALL_SMEM)))
			return e;
		ready = true;
	}
	cudaEvent_t ev;
	launch_begin(rt, KC_FUSED, &ev);
	k_small<MODE, ROLES><<<blocks, ROLES * nb, small_smem(a.L, a.nunits, a.G, a.Gt, MODE == EVAL_HVP), rt.stream>>>(a, nb);
	launch_end(rt, KC_FUSED, ev);
	return RQC_CUDA(cudaGetLastError());
}

// A thread per amplitude of the block's columns, up to 256.  Up to 128 (L <= 7) three roles share
// a gate's work: a warp or two per SM sub-partition wait out every latency in turn.
template <int MODE>
int launch_small(Runtime& rt, const SmallArgs& a, int blocks)
{
	const int nb = std::max(32, std::min(256, a.cb << a.L));
	if (MODE == EVAL_HVP && nb <= 128) return launch_small_as<MODE, 3>(rt, a, blocks, nb);
	return launch_small_as<MODE, 1>(rt, a, blocks, nb);
}

}  // namespace

bool SmallEval::fits(Runtime& rt, const Problem& pb, const TargetHolder& th, int64_t ncols, int mode)
{
	if (rt.pin_gpp || rt.pin_chunk || rt.pin_recon || rt.col_begin != 0 || rt.col_end != 0) return false;
	if (pb.L < 2 || pb.L > SMALL_MAX_L || pb.nunits > SMALL_MAX_UNITS || ncols < 1) return false;
	if (th.spec.ufunc || (!th.spec.dense && th.spec.ngates < 1)) return false;
	const int64_t amps = ncols << pb.L;
	const int gates = pb.G + th.spec.ngates;
	if ((double)amps * gates >= SMALL_MAX_WORK) return false;
	if (amps > (mode == EVAL_HVP ? SMALL_MAX_AMPS_HVP : SMALL_MAX_AMPS) &&
	    gates > (amps <= SMALL_MAX_AMPS ? SMALL_FEW_GATES : SMALL_FEW_GATES_1024))
		return false;
	if (small_smem(pb.L, pb.nunits, pb.G, th.spec.ngates, true) > SMALL_SMEM) return false;
	// the pass engine splits its columns where the workspace does not hold all of them
	const size_t states = states_bytes(pb.L, pb.G, ncols, mode);
	return !states || states <= workspace_budget(rt, states);
}

int SmallEval::reserve(Runtime& rt, int mode)
{
	int ret = ensure_device(rt.partials, (size_t)block_count(L_, ncols_) * (2 + SLOT * (size_t)nunits_) * sizeof(double));
	if (!ret) ret = ensure_device(rt.work, states_bytes(L_, G_, ncols_, mode));
	return ret;
}

int SmallEval::prepare(Runtime& rt, const Problem& pb, const TargetHolder& th, const std::vector<BasisCol>& cols, int mode,
                       const double2* ugates, const double2* udirs)
{
	const int64_t N = (int64_t)1 << pb.L;
	L_ = pb.L;
	G_ = pb.G;
	nunits_ = pb.nunits;
	per_ = pb.per;
	Gt_ = th.spec.dense ? 0 : th.spec.ngates;
	src_ = ColumnSource{};
	if (cols.empty()) {
		const int64_t all = rt.real_pairs ? N / 2 : N;
		src_.end = all;
		src_.pair_half = rt.real_pairs ? N / 2 : 0;
	} else {
		src_.end = (int64_t)cols.size();
	}
	ncols_ = src_.end - src_.b0;
	// one staged copy: unit gates | directions | target gates | columns | wire bits
	const size_t nug = ugates ? 16 * (size_t)nunits_ : 0, nuz = udirs ? 16 * (size_t)nunits_ : 0, ntg = 16 * (size_t)Gt_;
	const size_t gates_b = (nug + nuz + ntg) * sizeof(double2), cols_b = cols.size() * sizeof(BasisCol);
	const size_t bytes = gates_b + cols_b + 2 * (size_t)(G_ + Gt_) * sizeof(int);
	int ret = ensure_host_pinned(rt.small_host, bytes);
	if (!ret) ret = ensure_device(rt.small_dev, bytes);
	if (!ret) ret = reserve(rt, mode);
	if (ret) return ret;
	char* h = static_cast<char*>(rt.small_host.ptr);
	double2* hg = reinterpret_cast<double2*>(h);
	if (nug) memcpy(hg, ugates, nug * sizeof(double2));
	if (nuz) memcpy(hg + nug, udirs, nuz * sizeof(double2));
	if (ntg) memcpy(hg + nug + nuz, th.spec.gates, ntg * sizeof(double2));
	if (cols_b) memcpy(h + gates_b, cols.data(), cols_b);
	int* hb = reinterpret_cast<int*>(h + gates_b + cols_b);
	for (int k = 0; k < 2 * G_; k++) hb[k] = L_ - 1 - pb.wires[k];
	for (int k = 0; k < 2 * Gt_; k++) hb[2 * G_ + k] = L_ - 1 - th.wires[k];
	if ((ret = RQC_CUDA(cudaMemcpyAsync(rt.small_dev.ptr, h, bytes, cudaMemcpyHostToDevice, rt.stream)))) return ret;
	const char* d = static_cast<const char*>(rt.small_dev.ptr);
	const double2* dg = reinterpret_cast<const double2*>(d);
	ug_ = nug ? dg : nullptr;
	uz_ = nuz ? dg + nug : nullptr;
	tg_ = dg + nug + nuz;
	if (!cols.empty()) src_.tab = reinterpret_cast<const BasisCol*>(d + gates_b);
	bits_ = reinterpret_cast<const int*>(d + gates_b + cols_b);
	dense_ = th.spec.dense;
	return OK;
}

int SmallEval::eval(Runtime& rt, int mode, const double2* ugates, const double2* udirs, const SmallOut& out)
{
	SmallArgs a;
	a.L = L_;
	a.G = G_;
	a.per = per_;
	a.nunits = nunits_;
	a.Gt = Gt_;
	a.cb = columns_per_block(L_);
	a.real = rt.real_pairs;
	a.src = src_;
	a.ug = ugates ? ugates : ug_;
	a.uz = udirs ? udirs : uz_;
	a.bits = bits_;
	a.tg = tg_;
	a.dense = dense_;
	const int blocks = block_count(L_, ncols_);
	int ret = reserve(rt, mode);   // (other work of an optimiser may have taken the buffers)
	if (ret) return ret;
	a.part = static_cast<double*>(rt.partials.ptr);
	a.states = static_cast<double2*>(rt.work.ptr);
	if (mode == EVAL_HVP) ret = launch_small<EVAL_HVP>(rt, a, blocks);
	else if (mode == EVAL_GRAD) ret = launch_small<EVAL_GRAD>(rt, a, blocks);
	else ret = launch_small<EVAL_F>(rt, a, blocks);
	if (ret) return ret;
	k_small_post<<<nunits_ + 1, RED_GROUPS * SLOT, 0, rt.stream>>>(a, blocks, mode, out);
	rt.launches++;
	rt.last_choice = {rt.gates_per_pass, rt.column_chunk, rt.recon_c128, rt.c64_ffma, 0.0, 0};
	return RQC_CUDA(cudaGetLastError());
}

}  // namespace rqc
