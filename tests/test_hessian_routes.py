"""Full Hessians of few amplitudes take the general sweep, others the layer sweep: both sides of the
rule (256 columns or samples at L = 4, 16 at L = 6, one at L = 8) against the oracle, and the gate
launches that tell which sweep ran."""
import numpy as np
import pytest

from helpers import brickwall_instance

pytestmark = pytest.mark.gpu


def _general(L, depth):
    return 2 + 2 * (depth * (L // 2) - 1)      # two target layers, states and cotangents gate by gate


def _layers(depth):
    return 2 + depth + 2 * (depth - 1)         # two target layers, states, cotangents, tangents


def _launches(gpu, call):
    gpu.enable_kernel_timing(True)
    out = call()
    n = gpu.kernel_time(0)[1]
    gpu.enable_kernel_timing(False)
    return out, n


@pytest.mark.parametrize("L,depth,ns,general", [(2, 1, 0, True), (4, 1, 0, True), (4, 6, 0, True), (4, 3, 256, True),
                                                (4, 3, 257, False), (6, 3, 0, False), (6, 3, 16, True), (6, 3, 17, False),
                                                (8, 3, 1, True), (8, 3, 2, False), (10, 2, 1, False)])
def test_hessians_on_either_side_of_the_rule(gpu, oracle, L, depth, ns, general):
    v, p, tv, tp = brickwall_instance(L, depth, L, 2, L + 1)
    target, ot = gpu.Target(brickwall=(tv, tp)), oracle.target("brickwall", (tv, tp))
    if ns:
        got, n = _launches(gpu, lambda: gpu.brickwall_unitary_target_gradient_hessian_sampling(target, v, p, L, ns,
                                                                                               gpu.seed_rng_state(1)))
        ref = oracle.brickwall_unitary_target_gradient_hessian_sampling(ot, v, p, L, ns, oracle.seed_rng_state(1))
    else:
        got, n = _launches(gpu, lambda: gpu.brickwall_unitary_target_gradient_hessian(target, v, p, L))
        ref = oracle.brickwall_unitary_target_gradient_hessian(ot, v, p, L)
    assert n == (_general(L, depth) if general else _layers(depth))
    assert abs(got[0] - ref[0]) <= 1e-12 * 2 ** L
    for a, b in zip(got[1:], ref[1:]):
        assert np.linalg.norm(a - b) <= 1e-12 * max(np.linalg.norm(b), np.linalg.norm(ref[1]))


@pytest.mark.parametrize("L,depth", [(4, 1), (4, 5), (8, 2), (8, 5)])
def test_block_encodings_on_either_side_of_the_rule(gpu, oracle, L, depth):
    v, p, tv, _ = brickwall_instance(L, depth, L, 2, L + 1)
    half = np.stack([np.roll(np.arange(L // 2), -(k % 2)) for k in range(2)]).astype(np.int32)
    got = gpu.brickwall_blockenc_target_gradient_hessian(gpu.Target(brickwall=(tv, half)), v, p, L)
    ref = oracle.brickwall_blockenc_target_gradient_hessian(oracle.target("brickwall", (tv, half)), v, p, L)
    for a, b in zip(got, ref):
        assert np.linalg.norm(np.asarray(a) - b) <= 1e-12 * max(1.0, np.linalg.norm(b))
