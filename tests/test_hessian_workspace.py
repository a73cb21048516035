"""rqcopt_gpu_set_workspace_limit and the full Hessians: a limit that the layer sweep's states of a
column exceed and the general sweep's do not is served by the general sweep."""
import numpy as np
import pytest

from helpers import brickwall_instance

pytestmark = pytest.mark.gpu

STATE = 16   # bytes of an amplitude


@pytest.fixture(autouse=True)
def _settings(gpu):
    gpu.set_autotune(True)
    yield
    gpu.set_workspace_limit(0)


# states a column of the general Hessian sweep holds (phi and psi of every gate, 16 tangents a layer, samples
# and a scratch state) and of the layer sweep (psi, phi and 16 tangents a layer, 16
# cotangent states, the sample state): the limits lie between the two
@pytest.mark.parametrize("L,depth,states", [(2, 1, 21), (4, 1, 24), (4, 2, 45), (8, 1, 30), (8, 2, 51), (14, 1, 30)])
@pytest.mark.parametrize("samples", [False, True])
def test_hessians_take_the_sweep_that_fits(gpu, L, depth, states, samples):
    if L == 14 and not samples:
        pytest.skip("all columns of a large register")
    v, p, tv, tp = brickwall_instance(L, depth, L, 2, L + 1)
    target = gpu.Target(brickwall=(tv, tp))

    def run():
        if samples:
            return gpu.brickwall_unitary_target_gradient_hessian_sampling(target, v, p, L, 3, gpu.seed_rng_state(1))
        return gpu.brickwall_unitary_target_gradient_hessian(target, v, p, L)
    ref = run()
    gpu.set_workspace_limit(states * STATE << L)
    got = run()
    assert abs(got[0] - ref[0]) <= 1e-12 * 2 ** L
    # one gate in one layer: the Hessian is zero
    for a, b in zip(got[1:], ref[1:]):
        assert np.linalg.norm(a - b) <= 1e-12 * max(np.linalg.norm(b), np.linalg.norm(ref[1]))


@pytest.mark.parametrize("L,depth", [(4, 1), (4, 2), (8, 1), (8, 2)])
@pytest.mark.parametrize("what", ["target", "gradient", "hessian"])
def test_block_encodings_take_the_sweep_that_fits(gpu, L, depth, what):
    G = depth * (L // 2)
    v, p, tv, tp = brickwall_instance(L, depth, 5, 1, 6)
    target = gpu.Target(brickwall=(tv, np.arange(L // 2, dtype=np.int32)[None]))
    call = {"target": gpu.brickwall_blockenc_target, "gradient": gpu.brickwall_blockenc_target_and_gradient,
            "hessian": gpu.brickwall_blockenc_target_gradient_hessian}[what]
    ref = np.atleast_1d(call(target, v, p, L)) if what == "target" else call(target, v, p, L)
    # the general sweep's states of one column, and one more
    gpu.set_workspace_limit((2 * G + 1 + (16 * depth if what == "hessian" else 0) + 1) * STATE << L)
    got = np.atleast_1d(call(target, v, p, L)) if what == "target" else call(target, v, p, L)
    for a, b in zip(got, ref):
        assert np.linalg.norm(np.asarray(a) - b) <= 1e-12 * max(1.0, np.linalg.norm(b))
