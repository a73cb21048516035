"""Six gates on the lowest twelve wires share one pass over the states, whatever the register's
size; six gates elsewhere take two: the same states as the oracle's."""
import numpy as np
import pytest

from helpers import haar_unitary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,shift,passes", [(12, 0, 1), (13, 1, 1), (14, 2, 1), (13, 0, 2), (14, 0, 2), (14, 1, 2)])
def test_six_gates_on_wires_of_their_own(gpu, oracle, L, shift, passes):
    rng = np.random.default_rng(L + shift)
    tg = np.stack([haar_unitary(rng) for _ in range(6)])
    order = rng.permutation(12) + shift
    tw = np.ascontiguousarray(order.reshape(6, 2), np.int32)
    g, w = haar_unitary(rng)[None], np.array([[1, L - 1]], np.int32)

    def run(k):
        gpu.enable_kernel_timing(True)
        f = gpu.circuit_unitary_target_sampling(gpu.Target(circuit=(tg[:k], tw[:k])), g, w, L, 2, gpu.seed_rng_state(3))
        n = gpu.kernel_time(0)[1]
        gpu.enable_kernel_timing(False)
        return f, n
    got, n6 = run(6)
    _, n5 = run(5)
    assert n6 - n5 == passes - 1
    rng_state = oracle.seed_rng_state(3)
    ref = 0
    for _ in range(2):
        psi = oracle.haar_random_statevector(L, rng_state)
        ref -= np.vdot(oracle.apply_quantum_circuit(tg, tw, psi), oracle.apply_quantum_circuit(g, w, psi)) * 2 ** L / 2
    assert abs(got - ref) <= 1e-12 * 2 ** L
