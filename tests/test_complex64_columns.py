"""complex64 sums run over every basis column, whatever the symmetry of the layers: the same bits
as with the column range given in full, which never takes a list of orbits."""
import numpy as np
import pytest

from helpers import brickwall_instance, random_tangent_dirs, real_to_antisymm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [4, 8, 12])
@pytest.mark.parametrize("ffma", [0, 1])
def test_complex64_sums_keep_their_bits(gpu, L, ffma):
    v, p, tv, tp = brickwall_instance(L, 4, L, 3, L + 1)
    r = random_tangent_dirs(v, 2)
    z = np.stack([v[k] @ real_to_antisymm(r[k]) for k in range(4)])
    target = gpu.Target(brickwall=(tv, tp))
    run = lambda: gpu.brickwall_unitary_target_hessian_vector_product(target, v, z, p, L)   # noqa: E731
    try:
        gpu.set_precision(gpu.PRECISION_C64)
        gpu.set_gates_per_pass(4)
        gpu.set_column_chunk(64)
        gpu.set_c64_fp32_pipe(bool(ffma))
        got = run()
        gpu.set_column_range(0, 1 << L)
        ref = run()
    finally:
        gpu.set_column_range(0, 0)
        gpu.set_precision(gpu.PRECISION_C128)
        gpu.set_autotune(True)
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)
