"""Device states that do not begin at a multiple of their amplitude's size, as views into a
buffer of single numbers do: complex128 entry points stage them and give what aligned states
give, bit for bit; entry points that cannot stage refuse them on the host, before any launch."""
import ctypes as C

import numpy as np
import pytest

from helpers import crandn, haar_unitary

pytestmark = pytest.mark.gpu


def _at_offset(values, off):
    """Device copy of a complex array that begins `off` real numbers into a buffer."""
    import torch
    flat = torch.from_numpy(np.ascontiguousarray(values)).view(-1)
    flat = torch.view_as_real(flat).reshape(-1).to("cuda")
    buf = torch.zeros(flat.numel() + 4, dtype=flat.dtype, device="cuda")
    buf[off:off + flat.numel()] = flat
    view = buf[off:off + flat.numel()]
    assert view.data_ptr() % (2 * flat.element_size()) == off % 2 * flat.element_size()
    torch.cuda.synchronize()
    return view


def _values(view):
    v = view.cpu().numpy()
    return v[0::2] + 1j * v[1::2]


@pytest.mark.parametrize("L", [3, 9, 10, 12, 14])
@pytest.mark.parametrize("off_in,off_out", [(1, 0), (0, 1), (1, 1)])
def test_circuits_take_states_at_any_address(gpu, L, off_in, off_out):
    from rqcopt_hpc_b200.abi import Statevector
    rng = np.random.default_rng(L)
    gates = np.stack([haar_unitary(rng) for _ in range(7)])
    wires = np.array([rng.choice(L, 2, replace=False) for _ in range(7)], np.int32)
    psi = crandn(1 << L, rng)
    ref = gpu.apply_quantum_circuit(gates, wires, psi)
    a, b = _at_offset(psi, off_in), _at_offset(np.zeros(1 << L, complex), off_out)
    assert gpu.lib().apply_quantum_circuit(gates.ctypes.data, 7, wires.ctypes.data, C.byref(Statevector(a.data_ptr(), L)),
                                           C.byref(Statevector(b.data_ptr(), L))) == 0
    assert np.array_equal(_values(b), ref)
    assert np.array_equal(_values(a), psi)


def test_backward_pass_takes_states_at_any_address(gpu):
    from rqcopt_hpc_b200.abi import Statevector
    rng = np.random.default_rng(1)
    L, V = 9, haar_unitary(rng)
    psi, dout = crandn(1 << L, rng), crandn(1 << L, rng)
    ref, dref = gpu.apply_gate_backward(V, 2, 7, psi, dout)
    a, b, c = _at_offset(psi, 1), _at_offset(dout, 1), _at_offset(np.zeros(1 << L, complex), 1)
    dV = np.zeros((4, 4), complex)
    sv = [C.byref(Statevector(x.data_ptr(), L)) for x in (a, b, c)]
    gpu.lib().apply_gate_backward(np.ascontiguousarray(V).ctypes.data, 2, 7, *sv, dV.ctypes.data)
    assert np.array_equal(_values(c), ref) and np.array_equal(dV, dref)


def test_entries_that_cannot_stage_refuse_unaligned_states(gpu):
    from rqcopt_hpc_b200.abi import Statevector
    rng = np.random.default_rng(2)
    L, V = 10, np.ascontiguousarray(haar_unitary(rng))
    wires = np.array([[1, 4]], np.int32)
    psi = crandn(1 << L, rng)
    small = [_at_offset(psi.astype(np.complex64), off) for off in (0, 1)]
    gpu.reset_launch_count()
    for a, b in [(1, 0), (0, 1)]:
        assert gpu.lib().rqcopt_apply_quantum_circuit_c64(V.ctypes.data, 1, wires.ctypes.data, small[a].data_ptr(),
                                                          small[b].data_ptr(), L) == -6
    assert gpu.launch_count() == 0
    f = gpu.lib().rqcopt_apply_gate_backward_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_int, C.c_int] + [C.POINTER(Statevector)] * 3 + [C.c_void_p, C.c_void_p]
    dV = np.zeros((4, 4), complex)
    for odd in range(3):
        t = [_at_offset(psi, int(k == odd)) for k in range(3)]
        sv = [C.byref(Statevector(x.data_ptr(), L)) for x in t]
        assert f(V.ctypes.data, 1, 4, *sv, dV.ctypes.data, None) == -6
        assert np.array_equal(_values(t[2]), psi)
