"""Circuits on one complex128 state take tiles of consecutive gates or passes of gates on wires of
their own, by the number of passes each needs: the same states as gate by gate, on either side of
the rule and of its changes with the size, in as many launches as the better form has passes."""
import ctypes as C

import numpy as np
import pytest

from helpers import haar_unitary

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _settings(gpu):
    gpu.set_autotune(True)
    yield
    gpu.set_autotune(True)


def _circuit(L, G, pool):
    rng = np.random.default_rng(L + G)
    gates = np.stack([haar_unitary(rng) for _ in range(G)])
    return gates, np.array([rng.choice(pool, 2, replace=False) for _ in range(G)], np.int32)


@pytest.mark.parametrize("L", [10, 11, 12, 14, 22, 23])
@pytest.mark.parametrize("G,pool", [(1, 2), (4, 2), (9, 3), (9, 6), (16, 10)])
def test_both_routes_match_gate_by_gate(gpu, L, G, pool):
    import torch
    from rqcopt_hpc_b200.abi import Statevector
    gates, wires = _circuit(L, G, pool)
    psi = torch.randn(1 << L, dtype=torch.complex128, device="cuda", generator=torch.Generator("cuda").manual_seed(L))
    out = [torch.empty_like(psi), torch.empty_like(psi)]
    torch.cuda.synchronize()

    def run(a, b):
        assert gpu.lib().apply_quantum_circuit(gates.ctypes.data, G, wires.ctypes.data, C.byref(Statevector(a.data_ptr(), L)),
                                               C.byref(Statevector(b.data_ptr(), L))) == 0
    run(psi, out[0])
    gpu.set_gates_per_pass(1)
    run(psi, out[1])
    # G products of unitaries in another order: a few roundings each
    norm = torch.linalg.vector_norm(psi)
    assert torch.linalg.vector_norm(out[0] - out[1]) <= 4e-16 * 8 * G * norm


@pytest.mark.parametrize("L,G,pool,launches", [(10, 12, 3, 3), (11, 40, 11, 10), (14, 12, 3, 3), (18, 16, 3, 4),
                                               (23, 12, 3, 3), (24, 16, 5, 4)])
def test_gates_that_share_wires_run_in_tiles(gpu, L, G, pool, launches):
    gates, wires = _circuit(L, G, pool)
    psi = np.zeros(1 << L, complex)
    psi[1] = 1
    gpu.reset_launch_count()
    gpu.apply_quantum_circuit(gates, wires, psi)
    assert gpu.launch_count() == launches


@pytest.mark.parametrize("L", [12, 16, 24])
def test_gates_on_wires_of_their_own_run_in_layers(gpu, L):
    gates = _circuit(L, 8, 3)[0]
    wires = np.array([[2 * k % 8, 2 * k % 8 + 1] for k in (0, 0, 1, 1, 2, 2, 3, 3)], np.int32)   # two layers of four
    psi = np.zeros(1 << L, complex)
    psi[1] = 1
    gpu.reset_launch_count()
    gpu.enable_kernel_timing(True)
    gpu.apply_quantum_circuit(gates, wires, psi)
    launches = gpu.kernel_time(0)[1]
    gpu.enable_kernel_timing(False)
    assert gpu.launch_count() == 2 and launches == 2
