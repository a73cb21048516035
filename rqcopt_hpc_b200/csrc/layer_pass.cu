// Gates on disjoint wires applied to many complex128 states, up to six per memory round trip.
//
// The full-Hessian sweep carries 16 tangent states per layer and column through every later
// layer; a layer's gates act on disjoint wires.  A block holds a tile of 2^11 (or 2^12)
// amplitudes over the gates' bits and the lowest others in shared memory and takes two gates
// per round: a thread's 16 amplitudes are closed under both, so they pass through registers
// once for 512 FMAs, with the gate entries as constant operands.  What bounds it is close to
// balanced: at four gates a tile moves 2 x 16 B per amplitude to and from memory and does 64
// complex multiply-adds (8 flop per byte; 6.5 TB/s against 34 TFLOP/s of DFMA is 5.2), and
// shared memory moves a quarter-warp per cycle for two thirds of the FMA time.  One gate per
// launch (k_happly) needs 1.3 flop per byte.  The tile's words are permuted within 128-byte
// lines (swz) and the lanes' bits chosen per round so that a quarter-warp's 16-byte accesses
// fall into different banks.
#include "layer_pass.h"

#include <algorithm>

namespace rqc {

namespace {

constexpr int MAXG = 6;         // gates per pass
constexpr int ROUNDS = MAXG / 2;

struct PassArgs
{
	Gate4<double> g[MAXG];
	int K, L;
	int8_t bit[ROUNDS][4];      // tile bits of wires i, j of the round's first and second gate (or fillers)
	int8_t pos[ROUNDS][8];      // tile bits of a thread's index bits
	int8_t tbit[12];            // index bit of tile bit b
	uint64_t rest;              // index bits that are not tile bits
	int64_t total, ntiles;      // amplitudes, tiles
	ColumnSource src;
};

// place of tile amplitude i: its 16-byte word within a 128-byte line XORed with the bits above
__device__ __forceinline__ int swz(int i) { return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9)) & 7); }

__device__ __forceinline__ int64_t deposit64(int64_t v, uint64_t mask)
{
	int64_t r = 0;
	while (v && mask) {
		const uint64_t low = mask & (0 - mask);
		if (v & 1) r |= (int64_t)low;
		v >>= 1;
		mask ^= low;
	}
	return r;
}

// the 4x4 gate on the four amplitudes x[0], x[s], x[2 s], x[3 s]
template <int S>
__device__ __forceinline__ void apply4(const Gate4<double>& g, double2* x)
{
	double2 y[4];
#pragma unroll
	for (int r = 0; r < 4; r++) {
		y[r] = cmul(g.m[4 * r], x[0]);
#pragma unroll
		for (int c = 1; c < 4; c++) y[r] = cfma(g.m[4 * r + c], x[c * S], y[r]);
	}
#pragma unroll
	for (int r = 0; r < 4; r++) x[r * S] = y[r];
}

// Tiles of 2^11 amplitudes are double-buffered: three blocks per SM, each with the next tile's
// loads (32 KB) in flight while it works on the current one; 2^12 ones alternate between two
// blocks per SM.
template <int TB, int IN, int OUT>
__global__ void __launch_bounds__(1 << (TB - 4), TB == 11 ? 3 : 2)
k_lpass(const double2* in, double2* out, const __grid_constant__ PassArgs a)
{
	constexpr int NT = 1 << (TB - 4);
	constexpr int NBUF = TB == 11 ? 2 : 1;
	extern __shared__ __align__(16) double2 tiles[];
	__shared__ uint32_t lo[64], hi[64];
	const int tid = threadIdx.x;
	if (tid < 64) {
		uint32_t o = 0, p = 0;
		for (int b = 0; b < 6; b++)
			if ((tid >> b) & 1) {
				o |= 1u << a.tbit[b];
				if (6 + b < TB) p |= 1u << a.tbit[6 + b];
			}
		lo[tid] = o;
		hi[tid] = p;
	}
	// first amplitude (place) of this thread's set in each round
	int base[ROUNDS];
#pragma unroll
	for (int r = 0; r < ROUNDS; r++) {
		int v = 0;
		if (2 * r < a.K)
#pragma unroll
			for (int b = 0; b < TB - 4; b++) v |= ((tid >> b) & 1) << a.pos[r][b];
		base[r] = swz(v);
	}
	__syncthreads();
	const int64_t mask = ((int64_t)1 << a.L) - 1;
	// tile t into buffer `tile`
	auto fetch = [&](int64_t t, double2* tile) {
		if (t < a.ntiles) {
			const int64_t at = deposit64(t, a.rest);
#pragma unroll
			for (int k = 0; k < 16; k++) {
				const int i = tid + k * NT;
				const int64_t e = at + lo[i & 63] + hi[i >> 6];
				if (IN == 0) {
					const unsigned d = (unsigned)__cvta_generic_to_shared(tile + swz(i));
					if (e < a.total) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(in + e) : "memory");
				} else {
					tile[swz(i)] = basis_amp<double>(a.src, e & mask, e >> a.L);
				}
			}
		}
		if (IN == 0) asm volatile("cp.async.commit_group;\n" ::: "memory");
	};
	if (NBUF == 2) fetch(blockIdx.x, tiles);
	int buf = 0;
	for (int64_t t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
		double2* tile = tiles + ((size_t)buf << TB);
		if (NBUF == 1) fetch(t, tile);
		if (IN == 0) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
		// this tile has landed, and every thread is done with the other buffer
		__syncthreads();
		if (NBUF == 2) {
			buf ^= 1;
			fetch(t + gridDim.x, tiles + ((size_t)buf << TB));
		}
		const int64_t at = deposit64(t, a.rest);
#pragma unroll
		for (int r = 0; r < ROUNDS; r++) {
			if (2 * r < a.K) {
				const int i0 = swz(1 << a.bit[r][0]), j0 = swz(1 << a.bit[r][1]);
				const int i1 = swz(1 << a.bit[r][2]), j1 = swz(1 << a.bit[r][3]);
				double2 x[16];   // [member of the first gate][member of the second]
#pragma unroll
				for (int m = 0; m < 16; m++)
					x[m] = tile[base[r] ^ (m & 8 ? i0 : 0) ^ (m & 4 ? j0 : 0) ^ (m & 2 ? i1 : 0) ^ (m & 1 ? j1 : 0)];
#pragma unroll
				for (int m = 0; m < 4; m++) apply4<4>(a.g[2 * r], x + m);
				if (2 * r + 1 < a.K)
#pragma unroll
					for (int m = 0; m < 4; m++) apply4<1>(a.g[2 * r + 1], x + 4 * m);
#pragma unroll
				for (int m = 0; m < 16; m++)
					tile[base[r] ^ (m & 8 ? i0 : 0) ^ (m & 4 ? j0 : 0) ^ (m & 2 ? i1 : 0) ^ (m & 1 ? j1 : 0)] = x[m];
				__syncthreads();
			}
		}
#pragma unroll
		for (int k = 0; k < 16; k++) {
			const int i = tid + k * NT;
			const int64_t e = at + lo[i & 63] + hi[i >> 6];
			if (e < a.total) out[e] = OUT == 1 ? cneg_conj(tile[swz(i)]) : tile[swz(i)];
		}
		if (NBUF == 1) __syncthreads();
	}
}

template <int TB, int IN, int OUT>
int launch(Runtime& rt, const double2* in, double2* out, const PassArgs& a)
{
	constexpr int smem = (TB == 11 ? 2 : 1) * (1 << TB) * (int)sizeof(double2);
	static int per_sm = 0;
	if (!per_sm) {
		if (int e = RQC_CUDA(cudaFuncSetAttribute(k_lpass<TB, IN, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)))
			return e;
		if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lpass<TB, IN, OUT>, 1 << (TB - 4), smem) != cudaSuccess ||
		    per_sm < 1) {
			cudaGetLastError();
			per_sm = 1;
		}
	}
	const int grid = (int)std::min<int64_t>(a.ntiles, (int64_t)rt.num_sms * per_sm);
	cudaEvent_t ev;
	launch_begin(rt, KC_APPLY, &ev);
	k_lpass<TB, IN, OUT><<<grid, 1 << (TB - 4), smem, rt.stream>>>(in, out, a);
	launch_end(rt, KC_APPLY, ev);
	return RQC_CUDA(cudaGetLastError());
}

template <int TB>
int launch_any(Runtime& rt, int in_mode, int out_mode, const double2* in, double2* out, const PassArgs& a)
{
	if (in_mode == 0) return out_mode == 0 ? launch<TB, 0, 0>(rt, in, out, a) : launch<TB, 0, 1>(rt, in, out, a);
	return out_mode == 0 ? launch<TB, 1, 0>(rt, in, out, a) : launch<TB, 1, 1>(rt, in, out, a);
}

}  // namespace

bool gates_disjoint(int L, const std::vector<LayerGate>& gates)
{
	uint64_t used = 0;
	for (const LayerGate& g : gates) {
		if (g.i < 0 || g.j < 0 || g.i >= L || g.j >= L || g.i == g.j) return false;
		const uint64_t w = ((uint64_t)1 << g.i) | ((uint64_t)1 << g.j);
		if (used & w) return false;
		used |= w;
	}
	return true;
}

int layer_apply(Runtime& rt, int L, const std::vector<LayerGate>& gates, bool transposed, const double2* in, double2* out,
                int64_t ncols, const ColumnSource* columns, bool neg_conj)
{
	const int n = (int)gates.size();
	// tiles of 2^11 amplitudes hold five gates' bits; 2^12 where that saves a pass (L = 12: the
	// whole column, six gates)
	const int TB = L == 12 && n == 6 ? 12 : 11;
	const int most = TB / 2, npass = std::max(1, (n + most - 1) / most);
	for (int p = 0, first = 0; p < npass; p++) {
		const int K = (n - first + npass - p - 1) / (npass - p);
		PassArgs a;
		a.K = K;
		a.L = L;
		a.total = ncols << L;
		uint64_t bits = 0;
		for (int k = 0; k < K; k++) {
			const LayerGate& g = gates[first + k];
			for (int e = 0; e < 16; e++) a.g[k].m[e] = transposed ? g.m[4 * (e & 3) + (e >> 2)] : g.m[e];
			bits |= ((uint64_t)1 << (L - 1 - g.i)) | ((uint64_t)1 << (L - 1 - g.j));
		}
		// the lowest other bits (for L < TB those of the column number among them)
		for (int b = 0; __builtin_popcountll(bits) < TB; b++) bits |= (uint64_t)1 << b;
		int local[64], nb = 0;
		for (int b = 0; nb < TB; b++)
			if ((bits >> b) & 1) {
				local[b] = nb;
				a.tbit[nb++] = (int8_t)b;
			}
		a.rest = ~bits;
		const int64_t tile = (int64_t)1 << TB;
		a.ntiles = (a.total + tile - 1) / tile;
		for (int r = 0; 2 * r < K; r++) {
			uint32_t used = 0;
			auto take = [&](int slot, int wire) {
				a.bit[r][slot] = (int8_t)local[L - 1 - wire];
				used |= 1u << a.bit[r][slot];
			};
			take(0, gates[first + 2 * r].i);
			take(1, gates[first + 2 * r].j);
			if (2 * r + 1 < K) {
				take(2, gates[first + 2 * r + 1].i);
				take(3, gates[first + 2 * r + 1].j);
			} else {   // a gate alone: the set takes the two highest other bits
				for (int s = 2, b = TB - 1; s < 4; b--)
					if (!((used >> b) & 1)) {
						a.bit[r][s++] = (int8_t)b;
						used |= 1u << b;
					}
			}
			// thread index bits: first three of different residues mod 3 (different lines of swz), then the rest
			int m = 0;
			uint32_t left = ((1u << TB) - 1) & ~used;
			for (int c = 0; c < 3; c++)
				for (int b = c; b < TB; b += 3)
					if ((left >> b) & 1) {
						a.pos[r][m++] = (int8_t)b;
						left &= ~(1u << b);
						break;
					}
			for (int b = 0; b < TB; b++)
				if ((left >> b) & 1) a.pos[r][m++] = (int8_t)b;
		}
		const bool first_pass = p == 0, last_pass = p == npass - 1;
		int in_mode = 0;
		if (first_pass && columns) {
			in_mode = 1;
			a.src = *columns;
		}
		const int out_mode = last_pass && neg_conj ? 1 : 0;
		const double2* src = first_pass ? in : out;
		const int ret = TB == 12 ? launch_any<12>(rt, in_mode, out_mode, src, out, a) : launch_any<11>(rt, in_mode, out_mode, src, out, a);
		if (ret) return ret;
		first += K;
	}
	return OK;
}

int circuit_apply(Runtime& rt, int L, int ngates, const double2* gates, const int* wires, const double2* in, double2* out,
                  double2* scratch, int64_t ncols, const ColumnSource* columns, bool neg_conj)
{
	// runs of gates on wires of their own
	std::vector<std::vector<LayerGate>> runs;
	uint64_t used = 0;
	for (int k = 0; k < ngates; k++) {
		const int i = wires[2 * k], j = wires[2 * k + 1];
		const uint64_t w = ((uint64_t)1 << i) | ((uint64_t)1 << j);
		if (runs.empty() || (used & w)) {
			runs.emplace_back();
			used = 0;
		}
		runs.back().push_back({gates + 16 * (size_t)k, i, j});
		used |= w;
	}
	const int n = (int)runs.size();
	const double2* src = in;
	for (int r = 0; r < n; r++) {
		double2* dst = (n - 1 - r) % 2 == 0 ? out : scratch;
		const bool last = r == n - 1;
		if (int e = layer_apply(rt, L, runs[r], false, src, dst, ncols, r == 0 ? columns : nullptr, last && neg_conj)) return e;
		src = dst;
	}
	return OK;
}

}  // namespace rqc
