"""Column weights of the allocation-free entry point's matrix when its entries are not 0 and 1: sums
of the entries, of any size and sign, whose largest and whose equality the search plans by
(csrc/grand_prep.cuh on the emulated device against tests/host_guided.cpp's own sums)."""
import subprocess

import numpy as np
import pytest

from library_s_grand_gb300 import synth
from test_guided_host import guided  # noqa: F401  (fixture)
from test_host_kernels import _write_code

BIG = 2**30


@pytest.mark.parametrize("entries", [
    {(3, 5): BIG + 7}, {(3, 5): 2**31 - 1}, {(3, 5): -BIG - 9}, {(3, 5): -2**31},
    {(3, 5): -2**31, (4, 6): 2**31 - 1}, {(3, 5): BIG, (4, 6): -BIG}, "negative", "zero and negative",
], ids=str)
def test_weights_are_sums_of_the_entries(guided, tmp_path, entries):  # noqa: F811
    h = synth.BB_CODES[72]().hz.copy()
    if entries == "negative":
        h = -h
    elif entries == "zero and negative":
        h = -h
        h[:, 7] = 0
    else:
        for (r, c), v in entries.items():
            h[:, c] = 0
            h[r, c] = v
    _write_code(str(tmp_path / "code"), h, 0, 0, (3, 256, 0, 64, 10, -1), [], Ho=np.abs(h) & 1)
    p = subprocess.run([guided, str(tmp_path / "code"), "prep"], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
