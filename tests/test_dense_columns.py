"""Dense targets summed over a range of columns: a short range picks its columns on the host and
leaves the matrix there, a long one copies it; the same sums either way."""
import os
import subprocess
import sys

import numpy as np
import pytest

from helpers import crandn, haar_unitary, rel_err

pytestmark = pytest.mark.gpu

PROBE = """
import sys
import numpy as np, torch
sys.path[:0] = [{root!r}, {tests!r}]
from rqcopt_hpc_b200 import gpu
from helpers import crandn, haar_unitary
rng = np.random.default_rng(0)
L = 12
u = crandn((1 << L, 1 << L), rng)
g, w = haar_unitary(rng)[None], np.array([[3, 8]], np.int32)
gpu.set_column_range(0, 4)
gpu.circuit_unitary_target(gpu.Target(circuit=(g, w)), g, w, L)   # the engine's own memory
free = torch.cuda.mem_get_info()[0]
gpu.circuit_unitary_target(gpu.Target(dense=u), g, w, L)
print(free - torch.cuda.mem_get_info()[0])
"""


def test_a_short_range_leaves_the_matrix_on_the_host(gpu):
    tests = os.path.dirname(os.path.abspath(__file__))
    p = subprocess.run([sys.executable, "-c", PROBE.format(root=os.path.dirname(tests), tests=tests)], capture_output=True,
                       text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    assert int(p.stdout.split()[-1]) < 64 << 20   # the matrix has 256 MB


@pytest.mark.parametrize("L", [8, 9, 10])
def test_ranges_of_any_length_agree(gpu, oracle, L):
    rng = np.random.default_rng(L)
    u = np.ascontiguousarray(crandn((1 << L, 1 << L), rng) / 2 ** (L / 2))
    gates = np.stack([haar_unitary(rng) for _ in range(5)])
    wires = np.array([rng.choice(L, 2, replace=False) for _ in range(5)], np.int32)
    target = gpu.Target(dense=u)
    edge = (1 << L) // 16
    try:
        for begin, end in [(0, 1), (5, 5 + edge), (5, 6 + edge), (7, 0), (0, 0)]:
            gpu.set_column_range(begin, end)
            f, dg = gpu.circuit_unitary_target_and_gradient(target, gates, wires, L)
            cols = np.arange(begin, end or 1 << L)
            e = np.zeros((len(cols), 1 << L), complex)
            e[np.arange(len(cols)), cols] = 1
            out = np.stack([oracle.apply_quantum_circuit(gates, wires, c) for c in e]) if len(cols) <= 64 else None
            if out is not None:   # f = -sum of conj(U e) . (C e)
                ref = -np.sum(u[:, cols].T.conj() * out)
                assert abs(f - ref) <= 1e-12 * len(cols)
            gpu.set_gates_per_pass(1)
            f1, dg1 = gpu.circuit_unitary_target_and_gradient(target, gates, wires, L)
            gpu.set_autotune(True)
            assert abs(f - f1) <= 1e-12 * len(cols) and rel_err(dg, dg1) <= 1e-12
    finally:
        gpu.set_column_range(0, 0)
        gpu.set_autotune(True)
