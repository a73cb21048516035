"""rqcopt_gpu_set_workspace_limit bounds what an evaluation takes for states: one that does not fit
the small engine runs in passes over chunks of columns, with the same results, and a limit below
those of one column is an error."""
import numpy as np
import pytest

from helpers import brickwall_instance, crandn, haar_unitary, rel_err

pytestmark = pytest.mark.gpu

STATE = 16   # bytes of an amplitude


@pytest.fixture(autouse=True)
def _settings(gpu):
    gpu.set_precision(gpu.PRECISION_C128)
    gpu.set_autotune(True)
    yield
    gpu.set_workspace_limit(0)


def _circuit(L, G, seed=0):
    rng = np.random.default_rng(seed)
    gates = np.stack([haar_unitary(rng) for _ in range(G)])
    wires = np.array([rng.choice(L, 2, replace=False) for _ in range(G)], np.int32)
    return gates, wires, crandn((G, 4, 4), rng), haar_unitary(rng, 1 << L)


def _check(got, ref, L):
    assert abs(got[0] - ref[0]) <= 1e-12 * 2 ** (L / 2)
    for a, b in zip(got[1:], ref[1:]):
        assert rel_err(a, b) <= 1e-12


@pytest.mark.parametrize("L,G,limit", [(8, 120, 4 << 20), (5, 18, 200 << 10), (4, 7, 20 << 10)])
def test_small_evaluations_keep_within_the_limit(gpu, oracle, L, G, limit):
    """States entering G gates, with tangents, of all columns: more than the limit each time."""
    assert 2 * G * STATE << (2 * L) > limit
    gates, wires, dirs, u = _circuit(L, G)
    target, ot = gpu.Target(circuit=(gates[:3], wires[:3])), None
    ref_u = np.eye(1 << L, dtype=complex)
    for g, w in zip(gates[:3], wires[:3]):
        ref_u = np.stack([oracle.apply_quantum_circuit(g[None], w[None], np.ascontiguousarray(c)) for c in ref_u.T], 1)
    ot = oracle.target("dense", np.ascontiguousarray(ref_u))
    gpu.set_workspace_limit(limit)
    gpu.reset_launch_count()
    got = gpu.circuit_unitary_target_hessian_vector_product(target, gates, dirs, wires, L)
    assert gpu.launch_count() > 2   # passes over chunks of columns, not the small engine's two launches
    _check(got, oracle.circuit_unitary_target_hessian_vector_product(ot, gates, dirs, wires, L), L)
    _check(gpu.circuit_unitary_target_and_gradient(target, gates, wires, L),
           oracle.circuit_unitary_target_and_gradient(ot, gates, wires, L), L)


def test_a_limit_below_one_column_is_an_error(gpu):
    gates, wires, dirs, _ = _circuit(6, 9)
    target = gpu.Target(circuit=(gates[:3], wires[:3]))
    gpu.set_workspace_limit(1 << 10)
    with pytest.raises(gpu.RqcError):
        gpu.circuit_unitary_target_hessian_vector_product(target, gates, dirs, wires, 6)


def test_optimisers_keep_within_the_limit(gpu):
    L, G = 5, 18
    gates, wires, _, u = _circuit(L, G, 3)
    target = gpu.Target(circuit=(gates[:4], wires[:4]))
    ref = gpu.optimize_quantum_circuit(target, gates, wires, L, 3)
    gpu.set_workspace_limit(200 << 10)
    gpu.reset_launch_count()
    got = gpu.optimize_quantum_circuit(target, gates, wires, L, 3)
    # the same iterates: rounding of f (at most 2^L) through three trust-region iterations
    assert np.all(np.abs(np.asarray(got[0]) - np.asarray(ref[0])) <= 1e-10 * 2 ** L)


def test_a_dense_target_is_not_copied_beyond_the_limit(gpu, oracle):
    L = 8
    gates, wires, _, u = _circuit(L, 1)
    target, ot = gpu.Target(dense=u), oracle.target("dense", u)
    ref = oracle.circuit_unitary_target_and_gradient(ot, gates, wires, L)
    gpu.set_workspace_limit((STATE << (2 * L)) - 1)
    gpu.reset_launch_count()
    _check(gpu.circuit_unitary_target_and_gradient(target, gates, wires, L), ref, L)
    assert gpu.launch_count() > 2
