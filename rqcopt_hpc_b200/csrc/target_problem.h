// Host description of an optimisation problem: the sequential circuit the
// engine evaluates, its optimisation units (one gate per brickwall layer, or
// every gate of a general circuit) and the target.
#pragma once

#include <vector>

#include "engine.h"
#include "rqcopt_gpu.h"

namespace rqc {

struct Problem
{
	int L = 0;
	int G = 0;        // sequential gates
	int nunits = 0;   // optimisation units
	int per = 1;      // sequential gates per unit (brickwall: L/2 copies of the layer gate)
	bool brickwall = false;
	std::vector<double2> gates, dirs;     // [G][16]
	std::vector<int> wires;               // [2G]
	std::vector<double2> ugates, udirs;   // [nunits][16]

	bool set_brickwall(int L, int nlayers, const struct mat4x4* vlist, const struct mat4x4* vdirs, const int* const* perms);
	bool set_circuit(int L, int ngates, const struct mat4x4* gates, const struct mat4x4* dirs, const int* wires);
	bool valid() const;
	void set_gates_from_units(const double2* ugates);
	void set_dirs_from_units(const double2* udirs);
};

// Target of the basis-column sums: a device-native brickwall / circuit, or a host callback.
struct TargetHolder
{
	std::vector<double2> gates;
	std::vector<int> wires;
	TargetSpec spec;
	// dense target (rqcopt_dense_ufunc): host matrix, to be laid out on the device
	const double2* dense_host = nullptr;
	int dense_L = 0;
	bool set(linear_func ufunc, void* udata, int L);
	// Copies a dense target to the device for the evaluations of this call (up to 1 GiB and within
	// the workspace limit; others stay a host callback, one column at a time).  ranged: the call sums
	// over the column range set by the caller.
	int to_device(Runtime& rt, bool ranged = false);
};

// Sum over the orbits of the wire relabellings that circuit and target share, instead of
// over all basis states (orbits.h): a brickwall against a device-native brickwall whose
// results are per-layer sums, over all columns.  Sets *columns and *ncolumns where there is
// such a symmetry; the list lies in rt.columns (held until the next call).  orbits_of: the list
// itself, empty where there is none.  evaluation_columns: that of f, gradient and Hessian-vector
// product evaluations, which take the columns of a real problem in pairs (rt.real_pairs); the
// full-Hessian sums keep imaginary parts and never do.
int upload_columns(Runtime& rt, const std::vector<BasisCol>& cols, const BasisCol** columns, int64_t* ncolumns);
std::vector<BasisCol> orbits_of(const Runtime& rt, int L, int nlayers, const int* wires, const TargetHolder& th);
std::vector<BasisCol> evaluation_columns(const Runtime& rt, const Problem& pb, const TargetHolder& th);
int use_orbits(Runtime& rt, int L, int nlayers, const int* wires, const TargetHolder& th, const BasisCol** columns,
               int64_t* ncolumns);
// The same for the block encoding of a brickwall on L/2 qubits (the target) by one on L: the
// relabellings keep the wires of the half register (0, 2, 4, ...) among themselves; columns
// of the half register.
int use_orbits_blockenc(Runtime& rt, int L, int nlayers, const int* wires, const TargetHolder& th,
                        const BasisCol** columns, int64_t* ncolumns);

int post_launch(Runtime& rt, const double2* d_res, const Problem& pb, const double2* d_ugates, const double2* d_udirs,
                int with_hvp, double2* d_dunits, double2* d_hunits, double* d_grad, double* d_hvp);

int run_target(const Problem& pb, TargetHolder& th, int mode, numeric* fval, struct mat4x4* dunits,
               struct mat4x4* hunits, double* grad_vec, double* hvp_vec);

}  // namespace rqc
