"""Codes outside 0..2 are refused by sodagpu_predict, wherever they are.  They are
counted on the device while the genomic values are formed, so the table kernel
(dgv.cuh) sees them too: a table holds the 243 sums of five SNPs' codes, and the
bytes of the index that other codes give go up to 255."""
import os
import re

import numpy as np
import pytest

import sodabayes_gb300 as sg
from sodabayes_gb300 import SodaGpuError, _abi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_an_index_of_any_codes_stays_inside_its_table():
    """The kernel's index arithmetic for four individuals in a word, over random bytes: what the shared array must hold."""
    txt = open(os.path.join(ROOT, "sodabayes_gb300", "csrc", "dgv.cuh")).read()
    entries = int(re.search(r"DGV_TAB = (\d+);", txt).group(1))
    row = re.search(r"__shared__ long long s_t\[DGV_CHUNK\]\[DGV_TAB( \+ 1)?\];", txt)
    entries += 1 if row.group(1) else 0
    rng = np.random.default_rng(1)
    words = rng.integers(0, 1 << 32, size=(5, 200000), dtype=np.uint64)
    idx = np.zeros(200000, dtype=np.uint64)
    for d in range(4, -1, -1):
        idx = (idx * 3 + words[d]) & 0xFFFFFFFF
    top = max(int(np.max((idx >> (8 * b)) & 0xFF)) for b in range(4))
    assert top == 255 and top < entries


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [-1, 3, 127, -128])
def test_codes_outside_the_range_are_refused_wherever_they_are(gpu_lib, bad):
    """Also in the last of the 40 SNPs whose tables are in shared memory together."""
    rng = np.random.default_rng(5)
    codes = rng.binomial(2, 0.4, size=(130, 45)).astype(np.int8)
    freq = np.full(45, 0.4)
    for where in (slice(35, 40), slice(0, 5), slice(0, 45)):
        c = codes.copy()
        c[::3, where] = bad
        with pytest.raises(SodaGpuError) as e:
            sg.predict(codes=c, freq=freq, mu=0.0, effects=np.ones(45))
        assert e.value.code == _abi.E_ARG
