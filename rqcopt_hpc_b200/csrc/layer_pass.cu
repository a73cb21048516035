// Gates on disjoint wires applied to many complex128 states, up to six per memory round trip.
//
// The full-Hessian sweep carries 16 tangent states per layer and column through every later
// layer; a layer's gates act on disjoint wires.  A block holds a tile of 2^11 (or 2^12)
// amplitudes over the gates' bits and the lowest others in shared memory and takes two gates
// per round, so that the amplitudes pass through registers once for both.  The first gate runs on
// the FP64 MMA (m8n8k4) with the amplitude's real and imaginary parts as two operands: a lane's
// operand is then one amplitude of its group, and the result comes back as the same amplitude of
// the same group, so nothing is exchanged.  The second gate's four amplitudes lie in the thread's
// own 16 and take FMAs with the gate's entries as constant operands.  Both run on the one FP64
// pipe; the MMAs are there because an FP64 FMA holds the issue port for two cycles.
//
// What bounds it is close to balanced: at four gates a tile moves 2 x 16 B per amplitude to and
// from memory and does 64 complex multiply-adds (8 flop per byte; 6.5 TB/s against 36 TFLOP/s is
// 5.5).  One gate per launch (k_happly) needs 1.3 flop per byte.  Measured on 2^26 amplitudes (2 GB
// read and written a pass): one or two gates 5.7 TB/s; four 5.3 TB/s, 21 TFLOP/s; five at L = 10
// 4.7 TB/s, 23 TFLOP/s.  Both gates in FMAs: 4.8 TB/s and 4.1 TB/s; with 64-bit index arithmetic per
// shared-memory access besides, 18 TFLOP/s.  Four blocks per SM at 128 registers; five spill and
// lose 12 %, three with the next tile prefetched gain 2 % at four gates and lose 5 % at five.
//
// The tile's words are permuted within 128-byte lines (swz) and the lanes' bits chosen per round
// so that a quarter-warp's 16-byte accesses fall into different banks.
#include "layer_pass.h"
#include "pass_tile.cuh"

#include <algorithm>

namespace rqc {

namespace {

constexpr int MAXG = 6;         // gates per pass
constexpr int ROUNDS = MAXG / 2;

struct PassArgs
{
	Gate4<double> g[MAXG];
	int K, L;
	int step[ROUNDS][4];        // places (bytes) of the tile bits of a thread's 16 amplitudes: two others, wires i, j of the
	                            // round's second gate (or two more others)
	int8_t pos[ROUNDS][8];      // tile bits of a thread's index bits (0, 1: wires j, i of the round's first gate)
	int8_t tbit[12];            // index bit of tile bit b
	uint32_t koff[16];          // index bits of the tile's top four bits
	// tile number to index bits outside the tile: nseg runs of consecutive bits, bits seg_from ..
	// of the number to bits seg_to .. of the index, seg_mask wide
	int nseg;
	int8_t seg_from[13], seg_to[13];
	uint64_t seg_mask[13];
	int64_t total, ntiles;      // amplitudes, tiles
	ColumnSource src;
};

__device__ __forceinline__ int64_t tile_base(const PassArgs& a, int64_t t)
{
	int64_t r = 0;
	for (int k = 0; k < a.nseg; k++) r |= (int64_t)(((uint64_t)t >> a.seg_from[k]) & a.seg_mask[k]) << a.seg_to[k];
	return r;
}

// Shared-memory addresses are byte offsets into the tile (places * 16), so that a member's is one
// XOR away from its neighbour's.
template <int TB, int IN, int OUT>
__global__ void __launch_bounds__(1 << (TB - 4), TB == 11 ? 4 : 2)
k_lpass(const double2* in, double2* out, const __grid_constant__ PassArgs a)
{
	constexpr int NT = 1 << (TB - 4);
	extern __shared__ __align__(16) char tile[];
	const int tid = threadIdx.x;
	auto at_smem = [&](int byte) -> double2& { return *reinterpret_cast<double2*>(tile + byte); };
	// this thread's amplitudes of a tile are tid + k NT: index offset own + a.koff[k], place swz(tid) ^ swz(k NT)
	uint32_t own = 0;
#pragma unroll
	for (int b = 0; b < TB - 4; b++) own |= (uint32_t)((tid >> b) & 1) << a.tbit[b];
	const int place = swz(tid) << 4;
	// first amplitude of this thread's set in each round
	int base[ROUNDS];
#pragma unroll
	for (int r = 0; r < ROUNDS; r++) {
		int v = 0;
		if (2 * r < a.K)
#pragma unroll
			for (int b = 0; b < TB - 4; b++) v |= ((tid >> b) & 1) << a.pos[r][b];
		base[r] = swz(v) << 4;
	}
	// operand of the rounds' first gates: for input amplitude k = lane & 3 and output part n = lane >> 2
	double bre[ROUNDS], bim[ROUNDS];
#pragma unroll
	for (int r = 0; r < ROUNDS; r++) {
		const int lane = tid & 31;
		const double2 g = 2 * r < a.K ? a.g[2 * r].m[4 * (lane >> 3) + (lane & 3)] : make_double2(0, 0);
		bre[r] = lane & 4 ? g.y : g.x;
		bim[r] = lane & 4 ? g.x : -g.y;
	}
	auto load = [&](int64_t t) {
		const int64_t at = tile_base(a, t) + own;
		if (IN == 0) {
			const bool whole = at + a.koff[15] < a.total;   // only tiles of contiguous columns can be cut off
			const double2* src = in + at;
			const unsigned dst = (unsigned)__cvta_generic_to_shared(tile);
#pragma unroll
			for (int k = 0; k < 16; k++)
				if (whole || at + a.koff[k] < a.total)
					asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + (place ^ (swz(k * NT) << 4))),
					             "l"(src + a.koff[k])
					             : "memory");
			asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
		} else {
			const int64_t mask = ((int64_t)1 << a.L) - 1;
#pragma unroll
			for (int k = 0; k < 16; k++) {
				const int64_t e = at + a.koff[k];
				at_smem(place ^ (swz(k * NT) << 4)) = basis_amp<double>(a.src, e & mask, e >> a.L);
			}
		}
	};
	for (int64_t t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
		load(t);
		__syncthreads();
#pragma unroll
		for (int r = 0; r < ROUNDS; r++) {
			if (2 * r < a.K) {
				const int s0 = a.step[r][0], s1 = a.step[r][1], s2 = a.step[r][2], s3 = a.step[r][3];
				auto mem = [&](int k) { return base[r] ^ (k & 8 ? s0 : 0) ^ (k & 4 ? s1 : 0) ^ (k & 2 ? s2 : 0) ^ (k & 1 ? s3 : 0); };
				double2 x[16];
#pragma unroll
				for (int k = 0; k < 16; k++) x[k] = at_smem(mem(k));
#pragma unroll
				for (int k = 0; k < 16; k++) {
					double2 y = make_double2(0, 0);
					dmma_amp(y, x[k].x, bre[r]);
					dmma_amp(y, x[k].y, bim[r]);
					x[k] = y;
				}
				if (2 * r + 1 < a.K)
#pragma unroll
					for (int k = 0; k < 4; k++) apply4<1>(a.g[2 * r + 1], x + 4 * k);
#pragma unroll
				for (int k = 0; k < 16; k++) at_smem(mem(k)) = x[k];
				__syncthreads();
			}
		}
		// (the tile's base again: held through the rounds it costs spills)
		const int64_t at = tile_base(a, t) + own;
		const bool whole = at + a.koff[15] < a.total;
		double2* dst = out + at;
#pragma unroll
		for (int k = 0; k < 16; k++) {
			const double2 v = at_smem(place ^ (swz(k * NT) << 4));
			if (whole || at + a.koff[k] < a.total) dst[a.koff[k]] = OUT == 1 ? cneg_conj(v) : v;
		}
		__syncthreads();
	}
}

template <int TB, int IN, int OUT>
int launch(Runtime& rt, const double2* in, double2* out, const PassArgs& a)
{
	constexpr int smem = (1 << TB) * (int)sizeof(double2);
	static PerDevice blocks;
	int& per_sm = blocks[rt];
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
	// Tiles of 2^11 amplitudes hold five gates' bits.  2^12 hold six, which pays where these are the lowest
	// bits, so that a tile is one run in memory: 2^26 amplitudes, L = 12, one pass 598 us and two 704 us; on
	// the first wires instead (runs of four amplitudes and less) L = 14 824 us and 704 us, L = 24 1340 us and
	// 724 us, 12 gates 1938 us and 1215 us.
	int low = 0;
	for (const LayerGate& g : gates) low += std::min(g.i, g.j) >= L - 12;
	const int TB = n == 6 && low == 6 ? 12 : 11;
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
		for (int k = 0; k < 16; k++) {
			a.koff[k] = 0;
			for (int b = 0; b < 4; b++)
				if ((k >> b) & 1) a.koff[k] |= 1u << a.tbit[TB - 4 + b];
		}
		a.nseg = 0;
		for (int b = 0, from = 0; b < 64;) {
			if ((bits >> b) & 1) {
				b++;
				continue;
			}
			int e = b;
			while (e < 64 && !((bits >> e) & 1)) e++;
			a.seg_from[a.nseg] = (int8_t)from;
			a.seg_to[a.nseg] = (int8_t)b;
			a.seg_mask[a.nseg++] = e - b >= 64 ? ~(uint64_t)0 : ((uint64_t)1 << (e - b)) - 1;
			from += e - b;
			b = e;
		}
		const int64_t tile = (int64_t)1 << TB;
		a.ntiles = (a.total + tile - 1) / tile;
		for (int r = 0; 2 * r < K; r++) {
			// thread index bits 0 and 1: the first gate's wires j and i (the lanes of an MMA's amplitude);
			// 16 amplitudes per thread: the second gate's wires and two other bits
			uint32_t used = 0;
			auto bit_of = [&](int wire) {
				const int b = local[L - 1 - wire];
				used |= 1u << b;
				return b;
			};
			const LayerGate& g0 = gates[first + 2 * r];
			a.pos[r][0] = (int8_t)bit_of(g0.j);
			a.pos[r][1] = (int8_t)bit_of(g0.i);
			int slot = 2;
			if (2 * r + 1 < K) {
				const LayerGate& g1 = gates[first + 2 * r + 1];
				a.step[r][2] = swz(1 << bit_of(g1.i)) << 4;
				a.step[r][3] = swz(1 << bit_of(g1.j)) << 4;
			} else {
				slot = 4;
			}
			// thread bit 2: of the residue mod 3 that the gate's two bits leave (a quarter-warp's accesses
			// then fall into different banks), if there is one
			int third = -1;
			for (int b = 0; b < TB && third < 0; b++)
				if (!((used >> b) & 1) && b % 3 != a.pos[r][0] % 3 && b % 3 != a.pos[r][1] % 3) third = b;
			for (int b = 0; b < TB && third < 0; b++)
				if (!((used >> b) & 1)) third = b;
			a.pos[r][2] = (int8_t)third;
			used |= 1u << third;
			// the remaining bits: the highest to the thread's own amplitudes, the others to the thread index
			for (int b = TB - 1, s = 0; s < slot; b--)
				if (!((used >> b) & 1)) {
					a.step[r][s++] = swz(1 << b) << 4;
					used |= 1u << b;
				}
			int m = 3;
			for (int b = 0; b < TB; b++)
				if (!((used >> b) & 1)) a.pos[r][m++] = (int8_t)b;
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

std::vector<std::vector<int>> reordered_passes(int L, int ngates, const int* wires, int most)
{
	// A gate waits for the last gates before it on its two wires; gates that wait for none commute
	// and act on wires of their own.  Each pass takes the `most` of them with the longest chains of
	// gates behind them: taken in the order of the circuit, chains are left over at the end that
	// cost a pass per gate or two (64 gates on random pairs of 27 wires: the least number of passes,
	// 16 of four gates, for three draws in four).
	std::vector<int> waits(ngates, 0), height(ngates, 1), last(L, -1);
	std::vector<std::vector<int>> next(ngates);
	for (int k = 0; k < ngates; k++)
		for (int e = 0; e < 2; e++) {
			const int w = wires[2 * k + e];
			if (last[w] >= 0) {
				next[last[w]].push_back(k);
				waits[k]++;
			}
			last[w] = k;
		}
	for (int k = ngates - 1; k >= 0; k--)
		for (int m : next[k]) height[k] = std::max(height[k], height[m] + 1);
	std::vector<int> ready;
	for (int k = 0; k < ngates; k++)
		if (!waits[k]) ready.push_back(k);
	std::vector<std::vector<int>> passes;
	while (!ready.empty()) {
		std::stable_sort(ready.begin(), ready.end(), [&](int x, int y) { return height[x] > height[y]; });
		const int n = std::min<int>(most, (int)ready.size());
		passes.emplace_back(ready.begin(), ready.begin() + n);
		ready.erase(ready.begin(), ready.begin() + n);
		for (int k : passes.back())
			for (int m : next[k])
				if (--waits[m] == 0) ready.push_back(m);
	}
	return passes;
}

int circuit_apply_passes(Runtime& rt, int L, const std::vector<std::vector<int>>& passes, const double2* gates,
                         const int* wires, const double2* in, double2* out)
{
	const double2* src = in;
	for (const std::vector<int>& pass : passes) {
		std::vector<LayerGate> list;
		for (int k : pass) list.push_back({gates + 16 * (size_t)k, wires[2 * k], wires[2 * k + 1]});
		if (int e = layer_apply(rt, L, list, false, src, out, 1)) return e;
		src = out;
	}
	return OK;
}

}  // namespace rqc
