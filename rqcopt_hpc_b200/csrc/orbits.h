// Basis columns of a brickwall problem up to its wire symmetry.
//
// Every layer of a brickwall applies ONE gate to all its pairs, so a relabelling s of
// the wires that maps each layer's set of (ordered) pairs onto itself, in the circuit and
// in the target, commutes with both: C S = S C, U S = S U for the permutation matrix S of
// s.  Then the column of basis state s(b) contributes to f, to the sums over a layer's
// gates and to their tangents exactly what the column of b contributes (the gates of a
// layer trade places), and the sum over all 2^L columns is the sum over one column per
// orbit, weighted by the orbit's size.  The periodic brickwall has the L/2 shifts by two
// wires: L/2 times fewer columns (up to the orbits shorter than L/2).
#pragma once

#include <stdint.h>
#include <vector>

namespace rqc {

// One column of an evaluation: the basis state re, or with im >= 0 the paired real columns
// e_re + i e_im, with the weights of the two in the sums.
struct BasisCol
{
	int32_t re, im;
	double wre, wim;
};

// The relabellings that preserve every layer, the identity first: entry [L * g + q] is the
// image of wire q.  layers: one array of L wires (pairs 2p, 2p + 1) per layer.  Only the
// identity if a layer does not cover each wire once, or if the pairs of all layers together
// do not connect the wires (a relabelling is then not fixed by the image of one wire).
std::vector<int> wire_symmetries(int L, const std::vector<const int*>& layers);

// Whether the relabelling s (L wires) preserves every layer; false if a layer does not cover
// each wire once.
bool preserves_layers(int L, const std::vector<const int*>& layers, const int* s);

// The least state of every orbit under the relabellings sym, in ascending order, with the size
// of its orbit as weight (im = -1: no second state).
std::vector<BasisCol> orbit_columns(int L, const std::vector<int>& sym);

// Two real columns per complex one (real gates and target): states 2k and 2k + 1 of the
// list as real and imaginary part.
std::vector<BasisCol> pair_columns(const std::vector<BasisCol>& cols);

}  // namespace rqc
