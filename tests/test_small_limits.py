"""Where evaluations leave the small engine: by the amplitudes of all columns, and the gates beyond.
Either side of each line against the oracle, and the launches that tell which engine ran (two for the
small one)."""
import numpy as np
import pytest

from helpers import brickwall_instance, haar_unitary, random_tangent_dirs, real_to_antisymm, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _settings(gpu):
    gpu.set_precision(gpu.PRECISION_C128)
    gpu.set_autotune(True)
    yield
    gpu.set_autotune(True)


def _check(got, ref, L):
    assert abs(got[0] - ref[0]) <= 1e-12 * 2 ** (L / 2)
    for a, b in zip(got[1:], ref[1:]):
        assert rel_err(a, b) <= 1e-12


@pytest.mark.parametrize("L,G,hvp_small,grad_small", [(8, 60, True, True), (9, 12, True, True), (9, 13, False, True),
                                                      (9, 40, False, True), (10, 6, True, True), (10, 7, False, False)])
def test_circuits_on_either_side(gpu, oracle, L, G, hvp_small, grad_small):
    rng = np.random.default_rng(L + G)
    gates = np.stack([haar_unitary(rng) for _ in range(G)])
    wires = np.array([rng.choice(L, 2, replace=False) for _ in range(G)], np.int32)
    dirs = np.stack([g @ real_to_antisymm(rng.standard_normal(16)) for g in gates])
    target = gpu.Target(circuit=(gates[:3], wires[:3]))   # three gates of the target count too
    u = np.eye(1 << L, dtype=complex)
    for g, w in zip(gates[:3], wires[:3]):
        t = np.moveaxis(u.reshape((2,) * L + (-1,)), w, (0, 1))
        u = np.moveaxis((g @ t.reshape(4, -1)).reshape(t.shape), (0, 1), w).reshape(1 << L, -1)
    ot = oracle.target("dense", np.ascontiguousarray(u))
    gpu.reset_launch_count()
    got = gpu.circuit_unitary_target_projected_hessian_vector_product(target, gates, dirs, wires, L)
    assert (gpu.launch_count() == 2) == hvp_small
    _check(got, oracle.circuit_unitary_target_projected_hessian_vector_product(ot, gates, dirs, wires, L), L)
    gpu.reset_launch_count()
    got = gpu.circuit_unitary_target_and_projected_gradient(target, gates, wires, L)
    assert (gpu.launch_count() == 2) == grad_small
    _check(got, oracle.circuit_unitary_target_and_projected_gradient(ot, gates, wires, L), L)


def test_one_column_per_orbit_keeps_ten_qubits_small(gpu, oracle):
    L, depth = 10, 6
    v, p, tv, tp = brickwall_instance(L, depth, 1, 3, 2)
    r = random_tangent_dirs(v, 3)
    z = np.stack([v[k] @ real_to_antisymm(r[k]) for k in range(depth)])
    gpu.reset_launch_count()
    got = gpu.brickwall_unitary_target_projected_hessian_vector_product(gpu.Target(brickwall=(tv, tp)), v, z, p, L)
    assert gpu.launch_count() == 2
    _check(got, oracle.brickwall_unitary_target_projected_hessian_vector_product(oracle.target("brickwall", (tv, tp)), v, z, p,
                                                                                 L), L)
