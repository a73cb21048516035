"""rqcopt_batch_footprint counts what a problem holds: with its size grow the work items of both
precisions and the list of its columns (one per orbit of its wire symmetries)."""
import pytest

from rqcopt_hpc_b200 import batch

COLUMN = 8     # bytes of a listed column, {state, weight}


def _orbits(L):
    """Orbits of the basis states under the shifts by two wires (the periodic brickwall)."""
    seen, n = set(), 0
    for b in range(1 << L):
        if b in seen:
            continue
        n += 1
        for _ in range(L // 2):
            seen.add(b)
            b = (b >> 2) | ((b & 3) << (L - 2))
    return n


@pytest.mark.parametrize("L", [12, 14])
def test_columns_are_counted(L):
    # at 10 or more qubits every size has as many work items: the difference is the columns'
    assert batch.footprint(L, 5) - batch.footprint(10, 5) >= COLUMN * (_orbits(L) - _orbits(10))


def test_sizes_out_of_range_have_no_footprint():
    assert batch.footprint(16, 5) == 0 and batch.footprint(8, 0) == 0 and batch.footprint(8, 17) == 0
