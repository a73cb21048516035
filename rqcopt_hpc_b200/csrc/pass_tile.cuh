// Parts shared by the complex128 passes that hold a tile of amplitudes in shared memory.
#pragma once

#include "rqc_common.cuh"

namespace rqc {

// place of tile amplitude i: its 16-byte word within a 128-byte line XORed with the bits above
__host__ __device__ __forceinline__ constexpr int swz(int i) { return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9)) & 7); }

// D (8 groups x [re, im of 4 amplitudes]) += a (8 groups x 4) b: a lane's a is one part of amplitude
// lane & 3 of group lane >> 2, and its D are the parts of that same amplitude
__device__ __forceinline__ void dmma_amp(double2& d, double a, double b)
{
	asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
	    : "+d"(d.x), "+d"(d.y)
	    : "d"(a), "d"(b));
}

// the 4x4 gate on the four amplitudes x[0], x[s], x[2 s], x[3 s]
template <int S>
__device__ __forceinline__ void apply4(const Gate4<double>& g, double2* x)
{
	// eight sums side by side, each touched every eighth FMA
	double2 y[4];
#pragma unroll
	for (int r = 0; r < 4; r++) y[r] = make_double2(g.m[4 * r].x * x[0].x, g.m[4 * r].x * x[0].y);
#pragma unroll
	for (int r = 0; r < 4; r++) {
		y[r].x = fma(-g.m[4 * r].y, x[0].y, y[r].x);
		y[r].y = fma(g.m[4 * r].y, x[0].x, y[r].y);
	}
#pragma unroll
	for (int c = 1; c < 4; c++) {
#pragma unroll
		for (int r = 0; r < 4; r++) {
			y[r].x = fma(g.m[4 * r + c].x, x[c * S].x, y[r].x);
			y[r].y = fma(g.m[4 * r + c].x, x[c * S].y, y[r].y);
		}
#pragma unroll
		for (int r = 0; r < 4; r++) {
			y[r].x = fma(-g.m[4 * r + c].y, x[c * S].y, y[r].x);
			y[r].y = fma(g.m[4 * r + c].y, x[c * S].x, y[r].y);
		}
	}
#pragma unroll
	for (int r = 0; r < 4; r++) x[r * S] = y[r];
}

}  // namespace rqc
