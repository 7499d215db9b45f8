"""The tensor-core counts of 128 x 64 tiles (small Grams split over blocks, and
the SNP x SNP product) against the C oracle, bit for bit, where they can go
wrong: partial tiles, one row, partial and several 1920-column blocks, masks,
weights whose products with the counts round, unit weights and none, symmetric
calls, several covariate columns and SNP blocks."""
import ctypes as C

import numpy as np
import pytest

import kernel_cases as kc
from lakcluster_c_gb300 import abi

pytestmark = pytest.mark.gpu
SPLIT, AUTO = 3, 2


def _handle(rng, n, m, keep):
    k = lambda s: (rng.random(s) < keep).astype(np.uint8) | (np.arange(s) == 0)  # noqa: E731
    return abi.MHandle((rng.random((n, m)) < 0.35).astype(np.uint8), mr_j=k(n), mc_j=k(m))


@pytest.mark.parametrize("nA,nZ,m,keep", [(1, 1, 1, 1.0), (128, 64, 1920, 1.0), (129, 65, 1921, 0.8), (127, 200, 128, 1.0),
                                          (300, 63, 5777, 0.6), (33, 900, 3839, 0.9)])
@pytest.mark.parametrize("symmetric", [False, True])
def test_split_gram_equals_oracle(gpu_lib, nA, nZ, m, keep, symmetric):
    rng = np.random.default_rng(nA + 7 * nZ + m)
    MA = _handle(rng, nA, m, keep)
    MZ = MA if symmetric else _handle(rng, nZ, m, keep)
    MZ.set_masks(mc_j=np.unpackbits(MA.mc_j)[:m])
    P = abi.psize(m)
    gpu_lib.lakgb_set_gram_impl(SPLIT)
    try:
        for w in (abi.calc_A_ajdk(0.02 + 0.96 * rng.random(P)), abi.calc_A_ajdk(np.full(P, 0.5)), None):
            for t in (abi.TYPE_pm, abi.TYPE_00):
                args = (symmetric, t, abi.SPACING_b, abi.SPACING_j, MA, MZ, w, None, None)
                want, got = kc.call_gram("oracle", *args), kc.call_gram("gpu", *args)
                assert np.array_equal(got.view(np.uint64), want.view(np.uint64)), (t, w is None)
        assert gpu_lib.lakgb_device_status() == 0
    finally:
        gpu_lib.lakgb_set_gram_impl(AUTO)


@pytest.mark.parametrize("nA,nY,m,nt,keep", [(1, 1, 1, 1, 1.0), (128, 64, 1920, 1, 1.0), (130, 70, 1921, 3, 0.7),
                                             (2100, 33, 300, 1, 0.9), (40, 4000, 2500, 2, 0.8), (5000, 130, 90, 1, 0.5)])
def test_snp_product_equals_oracle(gpu_lib, nA, nY, m, nt, keep):
    rng = np.random.default_rng(3 * nA + nY + m)
    At, Yt, Tt = _handle(rng, nA, m, keep), _handle(rng, nY, m, keep), _handle(rng, nt, m, 1.0)
    pat = np.unpackbits(At.mc_j)[:m]
    for M in (Yt, Tt):
        M.set_masks(mc_j=pat)
    wa, wy = (abi.calc_A_ajdk(0.05 + 0.9 * rng.random(abi.psize(n))) for n in (nA, nY))
    la, ly = (abi.LHandle.from_matrix(rng.integers(-m, m + 1, (n, nt)).astype(np.float64)) for n in (nA, nY))
    out = []
    for fn, thread in ((kc.load_backend("oracle").lako_AtTYn_vv, ()),
                       (gpu_lib.wrap_AtTYn_vv__run, (C.byref(C.c_int(0)), None, None))):
        o = abi.LHandle(nA * nY * nt)
        p = o.ptr
        fn(*thread, abi.SPACING_a, abi.SPACING_a, abi.SPACING_a, At.ptr, Tt.ptr, Yt.ptr, kc_dp(wa), kc_dp(wy), la.ptr,
           ly.ptr, C.byref(p))
        out.append(o.buf.copy())
    assert gpu_lib.lakgb_device_status() == 0
    assert np.array_equal(out[1].view(np.uint64), out[0].view(np.uint64))


def kc_dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))
