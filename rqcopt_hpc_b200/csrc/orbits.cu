// Wire symmetries of a brickwall and the basis-state orbits under them (orbits.h).
#include "orbits.h"

namespace rqc {

std::vector<int> wire_symmetries(int L, const std::vector<const int*>& layers)
{
	std::vector<int> sym(L);
	for (int q = 0; q < L; q++) sym[q] = q;
	const int n = (int)layers.size();
	// partner and position (first or second wire of its pair) of every wire in every layer
	std::vector<int> partner((size_t)n * L, -1), second((size_t)n * L, 0);
	for (int l = 0; l < n; l++)
		for (int p = 0; p < L / 2; p++) {
			const int i = layers[l][2 * p], j = layers[l][2 * p + 1];
			if (i < 0 || j < 0 || i >= L || j >= L || i == j) return sym;
			if (partner[(size_t)l * L + i] >= 0 || partner[(size_t)l * L + j] >= 0) return sym;
			partner[(size_t)l * L + i] = j;
			partner[(size_t)l * L + j] = i;
			second[(size_t)l * L + j] = 1;
		}
	std::vector<int> s(L), queue;
	for (int y = 1; y < L; y++) {
		// a relabelling with s(0) = y: follow the pairs of all layers from wire 0
		s.assign(L, -1);
		s[0] = y;
		queue.assign(1, 0);
		bool ok = true;
		for (size_t at = 0; at < queue.size() && ok; at++) {
			const int x = queue[at];
			for (int l = 0; l < n && ok; l++) {
				const size_t o = (size_t)l * L;
				const int px = partner[o + x], image = partner[o + s[x]];
				if (second[o + x] != second[o + s[x]]) ok = false;
				else if (s[px] < 0) { s[px] = image; queue.push_back(px); }
				else if (s[px] != image) ok = false;
			}
		}
		if ((int)queue.size() < L) {
			if (ok) return std::vector<int>(sym.begin(), sym.begin() + L);   // not connected
			continue;
		}
		std::vector<char> seen(L, 0);
		for (int q = 0; q < L && ok; q++) {
			ok = !seen[s[q]];
			seen[s[q]] = 1;
		}
		if (ok) sym.insert(sym.end(), s.begin(), s.end());
	}
	return sym;
}

bool preserves_layers(int L, const std::vector<const int*>& layers, const int* s)
{
	for (const int* w : layers) {
		std::vector<int> after(L, -1);   // second wire of the pair that begins with a wire
		std::vector<char> seen(L, 0);
		for (int p = 0; p < L / 2; p++) {
			const int i = w[2 * p], j = w[2 * p + 1];
			if (i < 0 || j < 0 || i >= L || j >= L || i == j || seen[i] || seen[j]) return false;
			seen[i] = seen[j] = 1;
			after[i] = j;
		}
		for (int p = 0; p < L / 2; p++)
			if (after[s[w[2 * p]]] != s[w[2 * p + 1]]) return false;
	}
	return true;
}

std::vector<BasisCol> orbit_columns(int L, const std::vector<int>& sym)
{
	const int ng = (int)sym.size() / L, nbytes = (L + 7) / 8;
	// image of a basis state under relabelling g, a byte of it at a time (wire q is bit L-1-q)
	std::vector<int32_t> table((size_t)ng * nbytes * 256, 0);
	for (int g = 0; g < ng; g++)
		for (int k = 0; k < nbytes; k++) {
			int32_t* t = &table[((size_t)g * nbytes + k) * 256];
			for (int b = 0; b < 8 && 8 * k + b < L; b++) {
				const int32_t image = (int32_t)1 << (L - 1 - sym[(size_t)g * L + (L - 1 - (8 * k + b))]);
				for (int v = 0; v < 1 << b; v++) t[(1 << b) + v] = t[v] | image;
			}
		}
	std::vector<BasisCol> out;
	for (int32_t b = 0; b < (int32_t)1 << L; b++) {
		int fixed = 1;
		bool least = true;
		for (int g = 1; g < ng && least; g++) {
			int32_t r = 0;
			for (int k = 0; k < nbytes; k++) r |= table[((size_t)g * nbytes + k) * 256 + ((b >> (8 * k)) & 255)];
			least = r >= b;
			fixed += r == b;
		}
		if (least) out.push_back({b, -1, (double)(ng / fixed), 0.0});
	}
	return out;
}

std::vector<BasisCol> pair_columns(const std::vector<BasisCol>& cols)
{
	std::vector<BasisCol> out;
	for (size_t k = 0; k < cols.size(); k += 2) {
		BasisCol c = cols[k];
		if (k + 1 < cols.size()) {
			c.im = cols[k + 1].re;
			c.wim = cols[k + 1].wre;
		}
		out.push_back(c);
	}
	return out;
}

}  // namespace rqc
