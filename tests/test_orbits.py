"""Sums over the orbits of a brickwall's wire symmetries (csrc/orbits.cu) against sums over
all basis columns: the column lists on the CPU, the evaluations on the GPU (a column range
over all columns takes the plain path)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from helpers import brickwall_instance, haar_unitary, periodic_perms, random_tangent_dirs, real_to_antisymm, rel_err

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rqcopt_hpc_b200", "csrc")
WRAP = """
#include "orbits.h"
extern "C" long columns(int L, int n, const int* perms, int pairs, int* re, int* im, double* wre, double* wim)
{
	std::vector<const int*> layers;
	for (int l = 0; l < n; l++) layers.push_back(perms + l * L);
	std::vector<rqc::BasisCol> c = rqc::orbit_columns(L, rqc::wire_symmetries(L, layers));
	if (pairs) c = rqc::pair_columns(c);
	for (size_t k = 0; k < c.size(); k++) { re[k] = c[k].re; im[k] = c[k].im; wre[k] = c[k].wre; wim[k] = c[k].wim; }
	return (long)c.size();
}
"""


def _layers(kind, L, n, seed=0):
    """Layer layouts: the periodic brickwall, one with its wires renamed, one with a pair of
    one layer reversed (no common symmetry but those that keep it), one with arbitrary
    layers, one whose layers do not connect the wires, one that is not a permutation."""
    rng = np.random.default_rng(seed)
    p = periodic_perms(L, n)
    if kind == "renamed":
        p = rng.permutation(L).astype(np.int32)[p]
    elif kind == "reversed":
        p = p.copy()
        p[n - 1, :2] = p[n - 1, 1::-1]
    elif kind == "any":
        p = np.stack([rng.permutation(L) for _ in range(n)]).astype(np.int32)
    elif kind == "even":
        p = np.stack([p[0]] * n)
    return np.ascontiguousarray(p, np.int32)


@pytest.fixture(scope="module")
def columns(tmp_path_factory):
    d = tmp_path_factory.mktemp("orbits")
    (d / "wrap.cpp").write_text(WRAP)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + CSRC, "-o", str(d / "orbits.so"), "-x", "c++",
                    str(d / "wrap.cpp"), os.path.join(CSRC, "orbits.cu")], check=True)
    f = ctypes.CDLL(str(d / "orbits.so")).columns
    f.restype = ctypes.c_long

    def call(L, perms, pairs=False):
        n = 1 << L
        re, im, wre, wim = np.zeros(n, np.int32), np.zeros(n, np.int32), np.zeros(n), np.zeros(n)
        k = f(L, len(perms), np.ascontiguousarray(perms, np.int32).ctypes.data_as(ctypes.c_void_p), int(pairs),
              *(a.ctypes.data_as(ctypes.c_void_p) for a in (re, im, wre, wim)))
        return re[:k], im[:k], wre[:k], wim[:k]
    return call


@pytest.mark.parametrize("L", [2, 4, 6, 8, 10])
@pytest.mark.parametrize("kind", ["ring", "renamed", "reversed", "any", "even"])
def test_orbit_sums_equal_sums_over_all_columns(columns, oracle, L, kind):
    n, nt = 3, 2
    perms = np.concatenate([_layers(kind, L, n, L), _layers(kind, L, n, L)[:nt]])
    re, im, w, _ = columns(L, perms)
    assert np.sum(w) == 1 << L and np.all(im == -1) and np.all(np.diff(re) > 0)
    expected = L // 2 if kind in ("ring", "renamed") and L > 2 else 1
    if expected > 1:
        assert len(re) < (1 << L) / expected * 2
    if kind == "even" or L == 2:
        assert len(re) == 1 << L
    # a function of a column that is what the engine sums: <U e_b, C e_b>, and the gradient of a layer
    rng = np.random.default_rng(L)
    v = [haar_unitary(rng) for _ in range(n + nt)]

    def apply(layers, gates, x):
        for p, g in zip(layers, gates):
            for q in range(L // 2):
                i, j = int(p[2 * q]), int(p[2 * q + 1])
                t = np.moveaxis(x.reshape((2,) * L + (-1,)), (i, j), (0, 1))
                t = (g @ t.reshape(4, -1)).reshape(t.shape)
                x = np.moveaxis(t, (0, 1), (i, j)).reshape(1 << L, -1)
        return x
    if L <= 8:
        e = np.eye(1 << L, dtype=complex)
        f = np.sum(apply(perms[n:], v[n:], e).conj() * apply(perms[:n], v[:n], e), axis=0)
        assert abs(np.sum(w * f[re]) - np.sum(f)) <= 1e-12 * np.sum(np.abs(f))
    # paired columns hold every entry once
    pre, pim, pw, pv = columns(L, perms, pairs=True)
    got = np.zeros(1 << L)
    got[pre] += pw
    got[pim[pim >= 0]] += pv[pim >= 0]
    ref = np.zeros(1 << L)
    ref[re] = w
    assert np.array_equal(got, ref)


def test_layers_that_are_no_permutation_have_no_symmetry(columns):
    p = _layers("ring", 6, 2)
    p[1] = [0, 1, 1, 2, 3, 4]
    assert len(columns(6, p)[0]) == 64


@pytest.mark.gpu
@pytest.mark.parametrize("L,kind", [(4, "ring"), (6, "renamed"), (8, "ring"), (8, "reversed"), (8, "any"), (10, "renamed"),
                                    (12, "ring")])
@pytest.mark.parametrize("gpp", [4, 1])
def test_orbit_evaluations_equal_plain_ones(gpu, L, kind, gpp):
    vlist, _, tvlist, _ = brickwall_instance(L, 4, L, 3, L + 1)
    perms = _layers(kind, L, 4, L)
    r = random_tangent_dirs(vlist, 2)
    z = np.stack([vlist[k] @ real_to_antisymm(r[k]) for k in range(len(vlist))])
    t = gpu.Target(brickwall=(tvlist, perms[:3]))

    def run():
        return (gpu.brickwall_unitary_target(t, vlist, perms, L),
                *gpu.brickwall_unitary_target_and_gradient(t, vlist, perms, L),
                *gpu.brickwall_unitary_target_hessian_vector_product(t, vlist, z, perms, L))

    try:
        gpu.set_gates_per_pass(gpp)
        for precision, tol in ((gpu.PRECISION_C128, 1e-12), (gpu.PRECISION_C64, 2e-5)):
            gpu.set_precision(precision)
            got = run()
            gpu.set_column_range(0, 1 << L)
            ref = run()
            gpu.set_column_range(0, 0)
            # f may nearly cancel: bound it by the size of its terms
            assert abs(got[0] - ref[0]) <= tol * 2 ** (L / 2)
            for a, b in zip(got[2:], ref[2:]):
                if np.ndim(a):
                    assert rel_err(a, b) <= tol
    finally:
        gpu.set_column_range(0, 0)
        gpu.set_precision(gpu.PRECISION_C128)
        gpu.set_autotune(True)


@pytest.mark.gpu
@pytest.mark.parametrize("L,kind", [(4, "ring"), (6, "ring"), (8, "renamed"), (8, "any")])
def test_real_orbit_evaluations_equal_plain_ones(gpu, L, kind):
    from rqcopt_hpc_b200 import real
    rng = np.random.default_rng(L)
    v = np.stack([np.linalg.qr(rng.standard_normal((4, 4)))[0] for _ in range(5)])
    perms = _layers(kind, L, 3, L)
    d = np.stack([real.real_to_tangent(rng.standard_normal(6), v[k]) for k in range(3)])
    t = real.Target(brickwall=(v[3:], perms[:2]))
    ref_t = real.Target(fn=lambda x: real.apply_brickwall_unitary(v[3:], perms[:2], x))
    got = real.brickwall_unitary_target_projected_hessian_vector_product(t, v[:3], d, perms, L)
    ref = real.brickwall_unitary_target_projected_hessian_vector_product(ref_t, v[:3], d, perms, L)
    assert abs(got[0] - ref[0]) <= 1e-12 * 2 ** (L / 2)
    assert rel_err(got[1], ref[1]) <= 1e-12 and rel_err(got[2], ref[2]) <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("L,kind", [(4, "ring"), (6, "renamed"), (8, "ring"), (8, "reversed"), (8, "any"), (14, "ring")])
@pytest.mark.parametrize("chunk", [0, 7])
def test_orbit_hessians_equal_plain_ones(gpu, L, kind, chunk):
    depth = 2 if L == 14 else 3
    vlist, _, tvlist, _ = brickwall_instance(L, depth, L, 2, L + 1)
    perms = _layers(kind, L, depth, L)
    t = gpu.Target(brickwall=(tvlist, perms[:2]))
    if L == 14 and chunk:
        chunk = 700
    try:
        gpu.set_column_chunk(chunk)
        got = gpu.brickwall_unitary_target_gradient_hessian(t, vlist, perms, L)
        gpu.set_column_range(0, 1 << L)
        ref = gpu.brickwall_unitary_target_gradient_hessian(t, vlist, perms, L)
    finally:
        gpu.set_column_range(0, 0)
        gpu.set_autotune(True)
    assert abs(got[0] - ref[0]) <= 1e-12 * 2 ** (L / 2)
    assert rel_err(got[1], ref[1]) <= 1e-12 and rel_err(got[2], ref[2]) <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("L,depth,hdepth", [(4, 2, 1), (8, 3, 1), (8, 3, 2), (12, 3, 3)])
def test_orbit_block_encodings_equal_plain_ones(gpu, L, depth, hdepth):
    vlist, perms, _, _ = brickwall_instance(L, depth, L, 1, L + 1)
    hv, hp, _, _ = brickwall_instance(L // 2, hdepth, 3, 1, 4)
    dev = gpu.Target(brickwall=(hv, hp))
    host = gpu.Target(fn=lambda x: gpu.apply_brickwall_unitary(hv, hp, x))   # a callback: all columns
    for fn in (gpu.brickwall_blockenc_target_and_gradient, gpu.brickwall_blockenc_target_gradient_hessian,
               gpu.brickwall_blockenc_target_gradient_vector_hessian_matrix):
        got, ref = fn(dev, vlist, perms, L), fn(host, vlist, perms, L)
        assert abs(got[0] - ref[0]) <= 1e-12 * abs(ref[0])
        for a, b in zip(got[1:], ref[1:]):
            assert rel_err(a, b) <= 1e-12
    assert abs(gpu.brickwall_blockenc_target(dev, vlist, perms, L) - ref[0]) <= 1e-12 * abs(ref[0])


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("PRECISION_C128", 1e-12), ("PRECISION_MIXED", 1e-4), ("PRECISION_C64", 1e-4)])
def test_batches_of_problems_with_and_without_symmetries(gpu, precision, tol):
    """One column per orbit where a problem has wire symmetries and its rounds are complex128, against
    sums over all columns of one problem at a time; columns that do not fill the last tile."""
    from rqcopt_hpc_b200 import batch
    probs, dirs, ref = [], [], []
    for L, kind, n in [(8, "ring", 4), (6, "any", 3), (10, "renamed", 3), (4, "ring", 3), (12, "ring", 2), (8, "reversed", 4),
                       (2, "ring", 2), (14, "ring", 2)]:
        vlist, _, tvlist, _ = brickwall_instance(L, n, L, 2, L + 1)
        perms = _layers(kind, L, n, L)
        r = random_tangent_dirs(vlist, 2)
        z = np.stack([vlist[k] @ real_to_antisymm(r[k]) for k in range(n)])
        probs.append((L, vlist, perms, tvlist, perms[:2]))
        dirs.append(z)
        try:
            gpu.set_column_range(0, 1 << L)
            ref.append(gpu.brickwall_unitary_target_projected_hessian_vector_product(gpu.Target(brickwall=(tvlist, perms[:2])),
                                                                                     vlist, z, perms, L))
        finally:
            gpu.set_column_range(0, 0)
            gpu.set_autotune(True)
    f, g, h = batch.evaluate(probs, dirs, batch.EVAL_HVP, getattr(gpu, precision))
    for k, (f0, g0, h0) in enumerate(ref):
        assert abs(f[k] - f0) <= tol * 2 ** (probs[k][0] / 2)
        assert rel_err(g[k], g0) <= tol
        assert rel_err(h[k], h0) <= tol
