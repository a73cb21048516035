// Evaluation of small problems in two launches (see engine_small.cu).
#pragma once

#include <vector>

#include "engine.h"
#include "target_problem.h"

namespace rqc {

// Where an evaluation's results go (device or pinned host memory; any may be null): f, the
// per-unit sums dG and HZ ([nunits][16]) and the projected vectors (16 reals per unit).
struct SmallOut
{
	double2* f = nullptr;
	double2* dunits = nullptr;
	double2* hunits = nullptr;
	double* grad = nullptr;
	double* hvp = nullptr;
};

class SmallEval
{
public:
	// Whether evaluations of the problem (mode: the largest, as EvalMode) run here: complex128, a
	// target that lives on the device, few enough amplitude updates, states within the workspace
	// limit and no engine setting fixed by the caller.
	static bool fits(Runtime& rt, const Problem& pb, const TargetHolder& th, int64_t ncols, int mode);

	// Lays the target, the wires and the columns (all basis states if cols is empty) out on
	// the device, in one copy, with the unit gates and directions if given, and takes the memory
	// of evaluations up to `mode`.  The layout is held in the runtime until the next call's.
	// E_ALLOC: there is no room; the pass engine may do with less.
	int prepare(Runtime& rt, const Problem& pb, const TargetHolder& th, const std::vector<BasisCol>& cols, int mode,
	            const double2* ugates = nullptr, const double2* udirs = nullptr);

	// mode as EvalMode; ugates / udirs: unit gates and directions on the device (null: those
	// given to prepare)
	int eval(Runtime& rt, int mode, const double2* ugates, const double2* udirs, const SmallOut& out);

private:
	int reserve(Runtime& rt, int mode);

	int L_ = 0, G_ = 0, nunits_ = 0, per_ = 1, Gt_ = 0;
	int64_t ncols_ = 0;
	ColumnSource src_;
	const double2 *ug_ = nullptr, *uz_ = nullptr, *tg_ = nullptr, *dense_ = nullptr;
	const int* bits_ = nullptr;
};

}  // namespace rqc
