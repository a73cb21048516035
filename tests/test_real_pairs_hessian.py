"""Paired columns (rqcopt_gpu_set_real_pairs) are a form of the f / gradient / HVP sums: full
Hessians, which keep imaginary parts, run on plain columns in either state of the switch."""
import numpy as np
import pytest

from helpers import periodic_perms

pytestmark = pytest.mark.gpu


def _real_instance(L, depth, seed):
    rng = np.random.default_rng(seed)
    v = np.stack([np.linalg.qr(rng.standard_normal((4, 4)))[0] for _ in range(depth + 2)]).astype(complex)
    return v[:depth], periodic_perms(L, depth), v[depth:], periodic_perms(L, 2)


@pytest.mark.parametrize("L", [4, 6, 8])
def test_paired_columns_leave_full_hessians_alone(gpu, L):
    v, p, tv, tp = _real_instance(L, 3, L)
    target = gpu.Target(brickwall=(tv, tp))
    ref = gpu.brickwall_unitary_target_gradient_hessian(target, v, p, L)
    vec = gpu.brickwall_unitary_target_gradient_vector_hessian_matrix(target, v, p, L)
    opt = gpu.optimize_brickwall_circuit_hmat(target, v, p, L, 3)
    try:
        gpu.lib().rqcopt_gpu_set_real_pairs(1)
        got = gpu.brickwall_unitary_target_gradient_hessian(target, v, p, L)
        got_vec = gpu.brickwall_unitary_target_gradient_vector_hessian_matrix(target, v, p, L)
        got_opt = gpu.optimize_brickwall_circuit_hmat(target, v, p, L, 3)
    finally:
        gpu.lib().rqcopt_gpu_set_real_pairs(0)
    for a, b in zip((*got, *got_vec), (*ref, *vec)):
        assert np.array_equal(a, b)
    # f of a candidate may run on other columns: the rounding of 2^L unit vectors' sums
    assert np.all(np.abs(np.asarray(got_opt[0]) - np.asarray(opt[0])) <= 1e-12 * 2 ** L)
