"""Passes over complex128 states with gates on wires of their own (csrc/layer_pass.cu): tiles larger
and smaller than the state, passes of one to six gates, reordering where gates commute and not
where they do not.  Each gate adds at most a few units of 1.1e-16 of the state's norm: the bar of
1e-13 holds for the at most 40 gates here with two orders to spare."""
import numpy as np
import pytest

from helpers import brickwall_instance, crandn, haar_unitary, periodic_perms

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _no_fixed_settings(gpu):
    gpu.set_autotune(True)
    yield
    gpu.set_autotune(True)


@pytest.mark.parametrize("L", [10, 11, 12, 13, 14])
@pytest.mark.parametrize("G,near", [(1, False), (2, False), (17, False), (40, False), (23, True)])
@pytest.mark.parametrize("per_pass", [0, 2, 3])
def test_circuits_match_the_oracle(gpu, oracle, L, G, near, per_pass):
    rng = np.random.default_rng(100 * L + G)
    gates = np.stack([haar_unitary(rng) for _ in range(G)])
    pool = 4 if near else L   # near: every gate shares wires with its neighbours in the sequence
    wires = np.array([rng.choice(pool, 2, replace=False) for _ in range(G)], np.int32)
    psi = crandn(1 << L, rng)
    if per_pass:
        gpu.set_gates_per_pass(per_pass)
    got = gpu.apply_quantum_circuit(gates, wires, psi)
    ref = oracle.apply_quantum_circuit(gates, wires, psi)
    assert np.linalg.norm(got - ref) <= 1e-13 * np.linalg.norm(ref)


@pytest.mark.parametrize("L", [2, 4, 6, 8, 10, 12, 14])
@pytest.mark.parametrize("ns", [1, 3])
def test_sampled_sums_take_layers_of_every_length(gpu, oracle, L, ns):
    vlist, perms, tvlist, tperms = brickwall_instance(L, 2, L, 2, L + 1)
    got = gpu.brickwall_unitary_target_gradient_hessian_sampling(gpu.Target(brickwall=(tvlist, tperms)), vlist, perms, L, ns,
                                                                 gpu.seed_rng_state(3))
    ref = oracle.brickwall_unitary_target_gradient_hessian_sampling(oracle.target("brickwall", (tvlist, tperms)), vlist, perms,
                                                                    L, ns, oracle.seed_rng_state(3))
    assert abs(got[0] - ref[0]) <= 1e-12 * 2 ** L
    for a, b in zip(got[1:], ref[1:]):
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)


def test_hessians_of_gates_that_are_not_unitary(gpu, oracle):
    rng = np.random.default_rng(1)
    v, tv, perms = crandn((3, 4, 4), rng), crandn((2, 4, 4), rng), periodic_perms(6, 3)
    got = gpu.brickwall_unitary_target_gradient_hessian(gpu.Target(brickwall=(tv, perms[:2])), v, perms, 6)
    ref = oracle.brickwall_unitary_target_gradient_hessian(oracle.target("brickwall", (tv, perms[:2])), v, perms, 6)
    for a, b in zip(got, ref):
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)


@pytest.mark.parametrize("L,G", [(11, 9), (11, 40), (12, 17), (13, 6)])
@pytest.mark.parametrize("near", [False, True])
@pytest.mark.parametrize("per_pass", [4, 3, 2])
def test_circuit_sums_in_passes_of_several_groups(gpu, L, G, near, per_pass):
    """Reordered passes, with gates that share wires in one pass, against one gate per pass.  Column
    sums of the same products in another order: 1e-12, the bar between the engines."""
    rng = np.random.default_rng(10 * L + G)
    gates = np.stack([haar_unitary(rng) for _ in range(G)])
    pool = 5 if near else L
    wires = np.array([rng.choice(pool, 2, replace=False) for _ in range(G)], np.int32)
    dirs = crandn((G, 4, 4), rng)
    t = gpu.Target(circuit=(gates[:3], wires[:3][:, ::-1].copy()))
    run = lambda: gpu.circuit_unitary_target_hessian_vector_product(t, gates, dirs, wires, L)   # noqa: E731
    try:
        gpu.set_column_range(3, 40)
        gpu.set_gates_per_pass(per_pass)
        got, grad = run(), gpu.circuit_unitary_target_and_gradient(t, gates, wires, L)
        gpu.set_gates_per_pass(1)
        ref = run()
    finally:
        gpu.set_column_range(0, 0)
    for a, b in zip(got, ref):
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
    assert np.linalg.norm(grad[1] - ref[1]) <= 1e-12 * np.linalg.norm(ref[1])


@pytest.mark.parametrize("L", [4, 5, 7, 8, 9, 11])
@pytest.mark.parametrize("near", [False, True])
@pytest.mark.parametrize("unitary", [False, True])
@pytest.mark.parametrize("first,last", [(0, 0), (1, 2), (3, 14)])
def test_forward_passes_on_ragged_columns(gpu, L, near, unitary, first, last):
    """Forward passes with and without tangents, column ranges that end inside a tile, gates that
    share wires: against one kernel per gate, 1e-12 as between the engines."""
    rng = np.random.default_rng(L)
    make = (lambda: haar_unitary(rng)) if unitary else (lambda: crandn((4, 4), rng) / 4)
    gates, target = (np.stack([make() for _ in range(n)]) for n in (9, 5))
    pool = 4 if near else L
    wires, twires = (np.array([rng.choice(pool, 2, replace=False) for _ in range(n)], np.int32) for n in (9, 5))
    dirs = crandn((9, 4, 4), rng)
    t = gpu.Target(circuit=(target, twires))

    def run(per_pass):
        gpu.set_gates_per_pass(per_pass)
        return (*gpu.circuit_unitary_target_hessian_vector_product(t, gates, dirs, wires, L),
                *gpu.circuit_unitary_target_and_gradient(t, gates, wires, L))

    try:
        gpu.set_column_range(first, last)
        ref = run(1)
        for per_pass in (4, 3):
            for a, b in zip(run(per_pass), ref):
                assert np.linalg.norm(a - b) <= 1e-12 * (np.linalg.norm(b) + np.linalg.norm(ref[1]))
    finally:
        gpu.set_column_range(0, 0)


@pytest.mark.parametrize("L,depth", [(4, 1), (6, 2), (8, 3), (6, 4), (8, 5), (4, 9), (6, 13)])
def test_hessian_products_of_every_last_tile(gpu, oracle, L, depth):
    """Layers whose last tile of tangents holds one fragment or three, alone or after whole tiles."""
    vlist, perms, tvlist, tperms = brickwall_instance(L, depth, L, 2, L + depth)
    got = gpu.brickwall_unitary_target_gradient_hessian(gpu.Target(brickwall=(tvlist, tperms)), vlist, perms, L)
    ref = oracle.brickwall_unitary_target_gradient_hessian(oracle.target("brickwall", (tvlist, tperms)), vlist, perms, L)
    for a, b in zip(got[1:], ref[1:]):
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
