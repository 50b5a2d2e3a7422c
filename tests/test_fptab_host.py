"""The FP64 far field's table-driven e^{ix} and e^x (fptab.cuh) compiled for the
host, against long double over their ranges: arguments spread over their
logarithm, and the seams between two table entries.

Bounds: the reduced argument is at most pi/128 (ln2/128), so what is added to a
table value is below 2^-5.3 (2^-6.5 of the result) and each of the four roundings
before the last one below 2^-59 (2^-60), the series' remainder below 2^-57.8
(2^-65): half a unit in the last place and 2^-56 for e^{ix}, 0.52 units for e^x.
The long double reference itself is 2^-12 of a unit off."""
import os
import subprocess
import tempfile

import pytest

from test_ffmath_host import _nvcc

HERE = os.path.dirname(os.path.abspath(__file__))


def test_table_functions_against_long_double():
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc not available")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "fptab")
        subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-ffp-contract=off",
                        "-o", exe, os.path.join(HERE, "fptab_check.cu")], check=True, capture_output=True)
        out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    vals = dict(zip(out[0::2], map(float, out[1::2])))
    assert vals["expi"] <= 1.0, vals
    assert vals["exp"] <= 0.52, vals
    assert vals["bad"] == 0, vals
