"""Circuits of one gate per layer: f is linear in each gate, so the diagonal blocks of the Hessian
are exactly zero, not the rounding of a difference."""
import numpy as np
import pytest

from helpers import brickwall_instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [1, 3])
@pytest.mark.parametrize("kind", ["columns", "samples"])
def test_one_gate_per_layer_has_no_diagonal_blocks(gpu, oracle, depth, kind):
    v, p, tv, tp = brickwall_instance(2, depth, 3, 2, 4)
    target, ot = gpu.Target(brickwall=(tv, tp)), oracle.target("brickwall", (tv, tp))
    if kind == "columns":
        h = gpu.brickwall_unitary_target_gradient_hessian(target, v, p, 2)[2]
        ref = oracle.brickwall_unitary_target_gradient_hessian(ot, v, p, 2)[2]
    else:
        h = gpu.brickwall_unitary_target_gradient_hessian_sampling(target, v, p, 2, 5, gpu.seed_rng_state(1))[2]
        ref = oracle.brickwall_unitary_target_gradient_hessian_sampling(ot, v, p, 2, 5, oracle.seed_rng_state(1))[2]
    h, ref = h.reshape(16 * depth, 16 * depth), ref.reshape(16 * depth, 16 * depth)
    for l in range(depth):
        assert not np.any(ref[16 * l:16 * l + 16, 16 * l:16 * l + 16])
        assert not np.any(h[16 * l:16 * l + 16, 16 * l:16 * l + 16])
