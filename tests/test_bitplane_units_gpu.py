"""wrap_At_T_YnWt_S_Zn_ww__run on the tensor cores against the C oracle, bit for
bit, where its split can go wrong: pair tiles of 128 and units of 256 / B Wn
rows with remainders, 128-patient chunks and 1920-patient blocks, several
covariate columns, masks, and products whose terms exceed the scratch (several
batches, sums carried from one to the next)."""
import ctypes as C

import numpy as np
import pytest

import kernel_cases as kc
from lakcluster_c_gb300 import abi

pytestmark = pytest.mark.gpu


def _mask(rng, n, keep):
    m = (rng.random(n) < keep).astype(np.uint8)
    m[rng.integers(0, n)] = 1
    return m


def _handles(rng, snps, ny, nw, B, nt, keep, mlt):
    bits = lambda *s: (rng.random(s) < 0.4).astype(np.uint8)  # noqa: E731
    ks, ky, kw = _mask(rng, snps, keep), _mask(rng, ny, keep), _mask(rng, nw, keep)
    h = dict(At=abi.MHandle(bits(snps, ny), mr_j=ks, mc_j=ky), Zt=abi.MHandle(bits(snps, nw), mr_j=ks, mc_j=kw),
             Tt=abi.MHandle(bits(nt, ny), mc_j=ky), St=abi.MHandle(bits(nt, nw), mc_j=kw),
             Yn=abi.MHandle(np.zeros((ny, 16), np.uint8), mr_j=ky), Wn=abi.MHandle(np.zeros((nw, 16), np.uint8), mr_j=kw))
    planes = np.zeros(((B + 1) * int(kw.sum()), abi.bsize(ny)), np.uint8)
    w = (ny + 7) // 8
    packed = np.packbits(ky)
    planes[:, :w] = rng.integers(0, 256, (planes.shape[0], w), dtype=np.uint8) & packed
    planes[0, :w] = packed
    X = abi.MHandle(None, nrows=planes.shape[0], ncols=ny, wX=planes, mc_j=ky)
    X.s.ncols_per_z, X.s.min_d, X.s.mlt_d = B + 1, -37.7, mlt
    h["X"] = X
    h["w"] = abi.calc_A_ajdk(0.05 + 0.9 * rng.random(abi.psize(snps)))
    return h


def _call(fn, h, snps, nt, thread):
    out = abi.LHandle(snps * nt)
    p = out.ptr
    fn(*thread, abi.SPACING_a, abi.SPACING_a, h["At"].ptr, h["Tt"].ptr, h["Yn"].ptr, h["Wn"].ptr, h["St"].ptr,
       h["Zt"].ptr, h["w"].ctypes.data_as(C.POINTER(C.c_double)), h["X"].ptr, C.byref(p))
    return out.buf.copy()


@pytest.mark.parametrize("snps,ny,nw,B,nt,keep,mlt", [
    (1, 1, 1, 32, 1, 1.0, 1.7), (127, 127, 7, 32, 1, 1.0, 3.1e7), (129, 129, 8, 32, 2, 0.9, 1.0),
    (300, 500, 9, 16, 3, 0.7, 6.0e3), (128, 1920, 17, 16, 1, 1.0, 1.1e-9), (2000, 1921, 40, 8, 1, 0.8, 0.3),
    (257, 2100, 33, 8, 2, 0.6, 5.5e40), (20000, 100, 520, 32, 1, 1.0, 2.0e6), (9000, 60, 400, 32, 3, 0.95, 2.3e6)])
def test_tensor_bitplane_equals_oracle(gpu_lib, snps, ny, nw, B, nt, keep, mlt):
    rng = np.random.default_rng(snps + 3 * ny + nw + B)
    h = _handles(rng, snps, ny, nw, B, nt, keep, mlt)
    want = _call(kc.load_backend("oracle").lako_At_T_YnWt_S_Zn_ww, h, snps, nt, ())
    got = _call(gpu_lib.wrap_At_T_YnWt_S_Zn_ww__run, h, snps, nt, (C.byref(C.c_int(0)), None, None))
    assert gpu_lib.lakgb_device_status() == 0
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))


@pytest.mark.parametrize("ny,nw,B", [(383, 28, 8), (384, 29, 8), (385, 14, 16), (769, 15, 16), (1537, 7, 32),
                                     (3841, 6, 32)])
def test_units_of_224_planes_and_steps_of_384_patients(gpu_lib, ny, nw, B):
    test_tensor_bitplane_equals_oracle(gpu_lib, 130, ny, nw, B, 2, 0.9, 2.9)
