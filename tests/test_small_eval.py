"""Evaluations of small problems in one block per column (csrc/engine_small.cu) against the
oracle: qubit counts at which columns share a block, fill a warp and loop over threads, gates in
either wire order, every mode, circuit, brickwall and dense targets, real-orthogonal problems.
Rounding bound: sums of 2^L columns of at most ~G products each stay below 1e-13 of their
largest entry here; the bar is the complex128 bar of the other engines, 1e-12."""
import numpy as np
import pytest

from helpers import brickwall_instance, crandn, haar_unitary, random_tangent_dirs, real_to_antisymm, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _no_fixed_settings(gpu):
    gpu.set_precision(gpu.PRECISION_C128)
    gpu.set_autotune(True)   # settings that another test fixed keep evaluations on the pass engine


def _check(got, ref, L):
    # f may nearly cancel: bound it by the size of its terms
    assert abs(got[0] - ref[0]) <= 1e-12 * 2 ** (L / 2)
    for a, b in zip(got[1:], ref[1:]):
        assert rel_err(a, b) <= 1e-12


@pytest.mark.parametrize("L,G", [(2, 1), (2, 5), (3, 4), (4, 7), (5, 18), (6, 9), (7, 11), (8, 12), (9, 6), (10, 5)])
@pytest.mark.parametrize("kind", ["circuit", "dense"])
def test_circuits(gpu, oracle, L, G, kind):
    rng = np.random.default_rng(100 * L + G)
    gates = np.stack([haar_unitary(rng) for _ in range(G)])
    wires = np.array([rng.choice(L, 2, replace=False) for _ in range(G)], np.int32)
    dirs = crandn((G, 4, 4), rng)   # not tangent: the sums themselves
    tg = np.stack([haar_unitary(rng) for _ in range(4)])
    tw = np.array([rng.choice(L, 2, replace=False) for _ in range(4)], np.int32)
    u = np.eye(1 << L, dtype=complex)
    for g, w in zip(tg, tw):
        u = np.stack([oracle.apply_quantum_circuit(g[None], w[None], np.ascontiguousarray(c)) for c in u.T], 1)
    target = gpu.Target(circuit=(tg, tw)) if kind == "circuit" else gpu.Target(dense=np.ascontiguousarray(u))
    ot = oracle.target("dense", np.ascontiguousarray(u))
    gpu.reset_launch_count()
    got = gpu.circuit_unitary_target_hessian_vector_product(target, gates, dirs, wires, L)
    assert gpu.launch_count() == 2
    _check(got, oracle.circuit_unitary_target_hessian_vector_product(ot, gates, dirs, wires, L), L)
    _check(gpu.circuit_unitary_target_projected_hessian_vector_product(target, gates, dirs, wires, L),
           oracle.circuit_unitary_target_projected_hessian_vector_product(ot, gates, dirs, wires, L), L)
    _check(gpu.circuit_unitary_target_and_gradient(target, gates, wires, L),
           oracle.circuit_unitary_target_and_gradient(ot, gates, wires, L), L)
    _check(gpu.circuit_unitary_target_and_projected_gradient(target, gates, wires, L),
           oracle.circuit_unitary_target_and_projected_gradient(ot, gates, wires, L), L)
    _check([gpu.circuit_unitary_target(target, gates, wires, L)], [oracle.circuit_unitary_target(ot, gates, wires, L)], L)


@pytest.mark.parametrize("L,depth", [(2, 3), (4, 2), (6, 5), (8, 4), (10, 2)])
@pytest.mark.parametrize("dense", [False, True])
def test_brickwalls(gpu, oracle, L, depth, dense):
    vlist, perms, tvlist, tperms = brickwall_instance(L, depth, L, 2, L + 1)
    r = random_tangent_dirs(vlist, 2)
    z = np.stack([vlist[k] @ real_to_antisymm(r[k]) for k in range(depth)])
    target, ot = gpu.Target(brickwall=(tvlist, tperms)), oracle.target("brickwall", (tvlist, tperms))
    if dense:
        rng = np.random.default_rng(L)
        u = haar_unitary(rng, 1 << L)
        target, ot = gpu.Target(dense=u), oracle.target("dense", u)
    _check(gpu.brickwall_unitary_target_hessian_vector_product(target, vlist, z, perms, L),
           oracle.brickwall_unitary_target_hessian_vector_product(ot, vlist, z, perms, L), L)
    _check(gpu.brickwall_unitary_target_projected_hessian_vector_product(target, vlist, z, perms, L),
           oracle.brickwall_unitary_target_projected_hessian_vector_product(ot, vlist, z, perms, L), L)
    _check(gpu.brickwall_unitary_target_and_gradient(target, vlist, perms, L),
           oracle.brickwall_unitary_target_and_gradient(ot, vlist, perms, L), L)
    _check([gpu.brickwall_unitary_target(target, vlist, perms, L)],
           [oracle.brickwall_unitary_target(ot, vlist, perms, L)], L)


@pytest.mark.parametrize("L", [2, 3, 5, 6])
def test_real_circuits_run_on_paired_columns(gpu, oracle, L):
    from oracle.oracle import RealOracle
    from rqcopt_hpc_b200 import real
    rng = np.random.default_rng(L)
    g = np.stack([np.linalg.qr(rng.standard_normal((4, 4)))[0] for _ in range(6)])
    w = np.array([rng.choice(L, 2, replace=False) for _ in range(6)], np.int32)
    d = np.stack([real.real_to_tangent(rng.standard_normal(6), g[k]) for k in range(4)])
    ro = RealOracle()
    u = np.eye(1 << L)
    for k in (4, 5):
        u = np.stack([ro.apply_quantum_circuit(g[k:k + 1], w[k:k + 1], np.ascontiguousarray(c)) for c in u.T], 1)
    got = real.circuit_unitary_target_projected_hessian_vector_product(real.Target(circuit=(g[4:], w[4:])), g[:4], d, w[:4], L)
    ref = ro.circuit_unitary_target_projected_hessian_vector_product(ro.target("dense", np.ascontiguousarray(u)), g[:4], d,
                                                                     w[:4], L)
    _check(got, ref, L)


def test_gates_that_are_not_unitary(gpu, oracle):
    L, G = 4, 3
    rng = np.random.default_rng(5)
    gates, dirs = crandn((G, 4, 4), rng), crandn((G, 4, 4), rng)
    wires = np.array([rng.choice(L, 2, replace=False) for _ in range(G)], np.int32)
    u = crandn((16, 16), rng)
    got = gpu.circuit_unitary_target_hessian_vector_product(gpu.Target(dense=u), gates, dirs, wires, L)
    _check(got, oracle.circuit_unitary_target_hessian_vector_product(oracle.target("dense", u), gates, dirs, wires, L), 12)


@pytest.mark.parametrize("L,ns", [(2, 3), (6, 5), (8, 9)])
def test_dense_target_on_sample_states(gpu, oracle, L, ns):
    vlist, perms, _, _ = brickwall_instance(L, 3, 1, 1, 2)
    u = haar_unitary(np.random.default_rng(L), 1 << L)
    got = gpu.brickwall_unitary_target_gradient_hessian_sampling(gpu.Target(dense=u), vlist, perms, L, ns, gpu.seed_rng_state(7))
    ref = oracle.brickwall_unitary_target_gradient_hessian_sampling(oracle.target("dense", u), vlist, perms, L, ns,
                                                                    oracle.seed_rng_state(7))
    _check(got, ref, L)


@pytest.mark.parametrize("n", [1, 16, 255, 1024, 1025, 3001])
def test_tcg_steps_by_a_block_match_the_oracle(gpu, oracle, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal(n)
    h = np.abs(rng.standard_normal(n)) + 0.5 if n % 2 else rng.standard_normal(n)
    hvp = lambda v: h * v + 0.1 * np.roll(v, 1) + 0.1 * np.roll(v, -1)   # noqa: E731
    z, b = gpu.truncated_cg_hvp(a, hvp, 3.0)
    zo, bo = oracle.truncated_cg_hvp(a, hvp, 3.0)
    assert b == bo and rel_err(z, zo) <= 1e-14
