// Gates on disjoint wires applied to many states in one pass (see layer_pass.cu).
#pragma once

#include <vector>

#include "rqc_common.cuh"
#include "rqc_runtime.h"

namespace rqc {

struct LayerGate
{
	const double2* m;   // 16 entries, row-major (host)
	int i, j;           // wires
};

// Whether the gates act on wires of their own.
bool gates_disjoint(int L, const std::vector<LayerGate>& gates);

// out = (the gates) in for ncols complex128 states of 2^L amplitudes one after another (device;
// in place where in == out).  The gates act on disjoint wires; transposed: their transposes.
//   columns: non-null: in is ignored, state c is (weighted) column c of *columns
//   neg_conj: out = -conj(...)
int layer_apply(Runtime& rt, int L, const std::vector<LayerGate>& gates, bool transposed, const double2* in, double2* out,
                int64_t ncols, const ColumnSource* columns = nullptr, bool neg_conj = false);

// The gates of a circuit in passes of up to `most` (<= 5; 4 measured best: a fifth leaves tiles short
// runs) on wires of their own, reordered where they commute.
std::vector<std::vector<int>> reordered_passes(int L, int ngates, const int* wires, int most);

// out = C in for one state (out may be in), a layer_apply per pass.
int circuit_apply_passes(Runtime& rt, int L, const std::vector<std::vector<int>>& passes, const double2* gates,
                         const int* wires, const double2* in, double2* out);

}  // namespace rqc
