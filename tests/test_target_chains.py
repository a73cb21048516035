"""Targets whose gates share wires: runs of one gate and runs of several, odd and even numbers of
them, on basis columns (full Hessians) and on sample states, against the oracle."""
import numpy as np
import pytest

from helpers import brickwall_instance, haar_unitary

pytestmark = pytest.mark.gpu

# wires of the target's gates; runs of gates on wires of their own in brackets
CHAINS = {"one": [(0, 1)],                                        # [1]
          "chain": [(0, 1), (1, 2), (2, 0), (0, 1)],              # [1] [1] [1] [1]
          "odd": [(0, 1), (1, 2), (2, 3)],                        # [1] [1] [1]
          "mixed": [(0, 1), (2, 3), (1, 2), (3, 0), (0, 2)],      # [2] [2] [1]
          "ends": [(0, 2), (0, 1), (3, 2), (1, 3)]}               # [1] [2] [1]


@pytest.mark.parametrize("L", [4, 6, 8])
@pytest.mark.parametrize("kind", sorted(CHAINS))
@pytest.mark.parametrize("samples", [0, 3])
def test_chains_of_gates_as_targets(gpu, oracle, L, kind, samples):
    rng = np.random.default_rng(L)
    tw = np.array(CHAINS[kind], np.int32) + (L - 4)
    tg = np.stack([haar_unitary(rng) for _ in tw])
    u = np.eye(1 << L, dtype=complex)
    for g, w in zip(tg, tw):
        t = np.moveaxis(u.reshape((2,) * L + (-1,)), w, (0, 1))
        u = np.moveaxis((g @ t.reshape(4, -1)).reshape(t.shape), (0, 1), w).reshape(1 << L, -1)
    v, p, _, _ = brickwall_instance(L, 2, 3, 1, 4)
    target, ot = gpu.Target(circuit=(tg, tw)), oracle.target("dense", np.ascontiguousarray(u))
    if samples:
        got = gpu.brickwall_unitary_target_gradient_hessian_sampling(target, v, p, L, samples, gpu.seed_rng_state(2))
        ref = oracle.brickwall_unitary_target_gradient_hessian_sampling(ot, v, p, L, samples, oracle.seed_rng_state(2))
    else:
        got = gpu.brickwall_unitary_target_gradient_hessian(target, v, p, L)
        ref = oracle.brickwall_unitary_target_gradient_hessian(ot, v, p, L)
    assert abs(got[0] - ref[0]) <= 1e-12 * 2 ** L
    for a, b in zip(got[1:], ref[1:]):
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
