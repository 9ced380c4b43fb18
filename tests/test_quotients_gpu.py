"""The branch-free FP64 quotients against the division operator, bit for bit."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pagani-toolkit_b200", "csrc")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mismatches(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("quotients") / "quotients.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                    "-shared", f"-I{CSRC}", os.path.join(HERE, "quotients.cu"), "-o", so], check=True)
    f = ct.CDLL(so).quotient_mismatches
    f.restype, f.argtypes = ct.c_longlong, [ct.c_int, ct.c_ulonglong, ct.c_longlong]
    return f


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
def test_quotients_equal_the_division_operator(mismatches, kind):
    """(1 + x) / (1 - x) and (m - 1) / (m + 1) of the Fisher transform; a
    vector's entries, of any exponent, by its norm; a sum by the edge count."""
    assert mismatches(kind, 12345 + kind, 1 << 28) == 0


@pytest.mark.parametrize("weighted", [False, True])
def test_fisher_transform_of_r_next_to_zero(ctx, weighted):
    """Series of small integers, whose sums of products often cancel: r of a
    few 1e-17, where 1 - r has a mantissa of ones."""
    rng = np.random.default_rng(12)
    bold = rng.integers(-2, 3, (12, 257)).astype(np.float32)
    z, _ = O.zscore(bold)
    d = (1.0 - O.corr_packed(z, weighted=weighted)).view(np.uint64)
    assert ((d & np.uint64(2 ** 52 - 1)) == np.uint64(2 ** 52 - 1)).sum() >= 10
    with ctx.cohort(257, fisher=True, weighted=weighted) as c:
        c.add(bold)
        packed = c.packed()
    assert np.array_equal(packed, O.cohort_keys([bold], fisher=True, weighted=weighted).astype(np.float32))
