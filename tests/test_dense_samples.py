"""Dense targets on sample states, on either side of a launch dimension's limit."""
import numpy as np
import pytest

from helpers import brickwall_instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [4 * 65535, 4 * 65535 + 1])
def test_dense_targets_take_any_number_of_samples(gpu, ns):
    """The dense matrix of a brickwall against the brickwall, on either side of 65535 groups of
    four states.  f is a mean of terms of size at most 2^(L/2) each."""
    L = 4
    v, p, tv, tp = brickwall_instance(L, 2, 1, 2, 2)
    u = np.stack([gpu.apply_brickwall_unitary(tv, tp, np.ascontiguousarray(c)) for c in np.eye(1 << L, dtype=complex)], 1)
    got = gpu.brickwall_unitary_target_sampling(gpu.Target(dense=np.ascontiguousarray(u)), v, p, L, ns, gpu.seed_rng_state(5))
    ref = gpu.brickwall_unitary_target_sampling(gpu.Target(brickwall=(tv, tp)), v, p, L, ns, gpu.seed_rng_state(5))
    assert abs(got - ref) <= 1e-12 * 2 ** L
