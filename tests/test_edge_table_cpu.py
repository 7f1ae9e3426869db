"""CPU test of the mesh-edge table's sizes (csrc/edges.cu): its slots are a power
of two with two or more per side, at any triangle count, and the counts beyond
which the table is not built are told (no allocation is made here)."""
import subprocess
import sys

import pytest

CODE = """
import ctypes, sys
from cutanddisplacejulia_b200 import _lib
L = ctypes.CDLL(_lib.LIB_PATH)
work, fits = L._ZN3cad14edge_work_intsEl, L._ZN3cad15edge_table_fitsEl
work.restype, fits.restype = ctypes.c_size_t, ctypes.c_bool
n = ctypes.c_int64(int(sys.argv[1]))
print(work(n), fits(n))
"""


@pytest.mark.parametrize("n", [1, 10, 11, 1000, 357913941, 357913942, 715827882, 1 << 40])
def test_slots_and_limit(cad, n):
    # in a process of its own: a size that overflows must not hang the tests
    out = subprocess.run([sys.executable, "-c", CODE, str(n)], capture_output=True, text=True, timeout=60, check=True)
    ints, fits = out.stdout.split()
    slots = 64
    while slots < 6 * n:
        slots *= 2
    assert int(ints) == slots + 9 * n + (3 * n + 255) // 256 + 2
    assert (fits == "True") == (6 * n <= 2 ** 31)
