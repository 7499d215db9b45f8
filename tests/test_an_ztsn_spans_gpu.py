"""wrap_An_ZtSn_ww__run where its counts come in spans of several 1920-column
blocks, against the C oracle, bit for bit: spans with a shorter last one, the
longest span with every bit on (34 blocks, 65280 in 16 bits), more blocks than a
grid's z dimension has, rows in ranges, and the scratch that the counts take."""
import numpy as np
import pytest

import kernel_cases as kc
import test_an_ztsn_gpu as base
from lakcluster_c_gb300 import abi

pytestmark = pytest.mark.gpu


def _packed(rng, rows, ncols):
    w = rng.integers(0, 256, (rows, abi.bsize(ncols)), dtype=np.uint8)
    w[:, ncols // 8:] = 0
    return w


def _handles(rng, n, m, B, nS, ones_row=False):
    A, Z = _packed(rng, n, m), _packed(rng, nS * (B + 1), m)
    if ones_row:
        A[0, : m // 8] = Z[0, : m // 8] = Z[-1, : m // 8] = 255
    An = abi.MHandle(None, nrows=n, ncols=m, wX=A)
    MZ = abi.MHandle(None, nrows=Z.shape[0], ncols=m, wX=Z)
    MZ.s.ncols_per_z, MZ.s.min_d, MZ.s.mlt_d = B + 1, -2.75, float(2 ** B) / 3.3
    return An, MZ, abi.MHandle(np.ones((nS, 16), np.uint8))


@pytest.mark.parametrize("n,m,B,nS", [(2050, 1920 * 80 - 8, 32, 1), (5000, 1920 * 69 + 8, 16, 3), (3, 1920 * 65537, 1, 1)])
def test_spans_equal_oracle(gpu_lib, n, m, B, nS):
    h = _handles(np.random.default_rng(n + B), n, m, B, nS, ones_row=True)
    want = base._call("oracle", abi.SPACING_a, abi.SPACING_a, *h)
    got = base._call("gpu", abi.SPACING_a, abi.SPACING_a, *h)
    assert got.tobytes() == want.tobytes()
    assert gpu_lib.lakgb_device_status() == 0


def test_row_ranges_equal_oracle(gpu_lib):
    n, m, B, nS = 8192, 1920 * 69 - 8, 32, 33
    rng = np.random.default_rng(9)
    An, Z, St = _handles(rng, n, m, B, nS)
    got = base._call("gpu", abi.SPACING_a, abi.SPACING_a, An, Z, St).reshape(nS, n)
    some = np.zeros(n, np.uint8)
    some[rng.permutation(n)[:200]] = 1
    some[[0, 5119, 5120, n - 1]] = 1  # the ends of the ranges
    An.set_masks(mr_j=some)
    want = base._call("oracle", abi.SPACING_a, abi.SPACING_a, An, Z, St).reshape(nS, n)
    k = some.astype(bool)
    assert got[:, k].tobytes() == want[:, k].tobytes()
    assert gpu_lib.lakgb_device_status() == 0


def test_scratch_of_the_counts(gpu_lib):
    """4096 rows x 99 planes x 69 blocks: 56 MB as a count per block."""
    import ctypes as C
    gpu_lib.lakgb_pool_high_water.argtypes, gpu_lib.lakgb_pool_high_water.restype = [C.c_int], C.c_longlong
    n, m, B, nS = 4096, 1920 * 69 - 8, 32, 3
    An, Z, St = _handles(np.random.default_rng(4), n, m, B, nS)
    base._call("gpu", abi.SPACING_a, abi.SPACING_a, An, Z, St)
    gpu_lib.lakgb_pool_high_water(1)
    base._call("gpu", abi.SPACING_a, abi.SPACING_a, An, Z, St)
    inputs = An.wX.nbytes + Z.wX.nbytes + 8 * n * nS
    # (at most 1216 tiles of 128 x 64 counts, and small arrays)
    assert gpu_lib.lakgb_pool_high_water(0) < inputs + 1216 * 128 * 64 * 2 + (4 << 20)
