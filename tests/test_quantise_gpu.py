"""The quantisation kernels (lakgb_xcalc_noalloc) against a numpy restatement of
xcalc.c:25-34,130,150 at the sizes where they can go wrong: partial and exact
row groups (256 rows, 1920-bit padding), plane rows that are not 16-byte
aligned, one to 62 bits (the fixed-point and the FP64 form), values on integer
boundaries, far from zero, of mixed magnitude, infinite and NaN.  Planes and
scalars are compared exactly."""
import ctypes as C

import numpy as np
import pytest

from test_zz_no_alloc import NoAllocArgs, _bind

pytestmark = pytest.mark.gpu


def _values(rng, kind, shape):
    x = rng.standard_normal(shape) * 50.0
    if kind == "integers":
        x = rng.integers(-9, 10, shape).astype(np.float64)
    elif kind == "offset":
        x = 1e9 + x * 1e-3
    elif kind == "mixed":
        x = x * np.exp(rng.standard_normal(shape) * 20.0)
    elif kind == "equal":
        x = np.full(shape, -3.25)
    elif kind == "inf":
        x[0, 1] = np.inf
    elif kind == "nan":
        x[rng.random(shape) < 0.1] = np.nan
        x[0, 0] = 1.0
    elif kind == "nan first":
        x[0, 0] = np.nan
    return x


def _reference(x, B, d):
    """x: retained columns x retained rows, in order.  min, max, mlt, values."""
    flat = x.ravel()
    mn = mx = flat[0]
    if not np.isnan(flat[0]):
        mn, mx = np.nanmin(flat), np.nanmax(flat)
    with np.errstate(all="ignore"):
        if mn >= mx:
            mx = mn + 1.0
        lo, hi = mn - 0.0625 * (mx - mn), mx + 0.0625 * (mx - mn)
        mlt = float(d) / (hi - lo)
        y = mlt * (x - lo)
    v = np.zeros(x.shape, np.uint64)
    fin = np.isfinite(y) & (y >= 1.0) & (y < float(d))
    v[fin] = y[fin].astype(np.uint64)
    v[np.isnan(y) | (y >= float(d))] = d - 1   # a conversion out of range, cropped
    v = np.clip(v, np.uint64(1), np.uint64(d - 1))
    return lo, hi, (mlt if np.isfinite(mlt) and mlt > 0 else 1.0), v


@pytest.mark.parametrize("rows,cols,B,d,kind,pad", [
    (1, 1, 32, 1 << 32, "normal", 0), (31, 3, 8, 1 << 8, "normal", 0), (255, 7, 16, 1 << 16, "integers", 4),
    (256, 40, 32, 1 << 32, "offset", 0), (257, 5, 32, 1 << 32, "mixed", 12), (1919, 9, 33, 1 << 33, "normal", 0),
    (1920, 4, 38, (1 << 38) - 5, "mixed", 0), (1921, 6, 39, 1 << 39, "normal", 0), (4100, 13, 62, 1 << 62, "normal", 4),
    (300, 700, 32, 1 << 32, "equal", 0), (700, 30, 32, 1 << 32, "inf", 0), (700, 30, 32, 1 << 32, "nan", 0),
    (700, 30, 16, 1 << 16, "nan first", 0), (90, 11, 5, 33, "integers", 0), (64, 64, 7, 64, "integers", 0),
    (2500, 33, 8, 1 << 32, "normal", 0)])
def test_quantise_matches_numpy(gpu_lib, rows, cols, B, d, kind, pad):
    import torch
    lib = _bind(gpu_lib)
    rng = np.random.default_rng(rows * 7 + cols + B)
    x = _values(rng, kind, (cols, rows))
    kr, kc = rng.random(rows) < 0.8, rng.random(cols) < 0.8
    kr[0] = kc[0] = True
    r, k = np.nonzero(kr)[0].astype(np.int64), np.nonzero(kc)[0].astype(np.int64)
    off = np.where(kr, np.arange(rows), -1).astype(np.int64)
    row_bytes = (rows + 1919) // 1920 * 240 + pad      # a multiple of 4; of 16 only for pad 0
    row0 = np.zeros(row_bytes, np.uint8)
    row0[: (rows + 7) // 8] = np.packbits(kr)
    lo, hi, mlt, v = _reference(x[np.ix_(kc, kr)], B, d)
    bits = np.zeros((len(k), B + 1, 8 * row_bytes), np.uint8)
    for b in range(B):
        bits[:, B - b, np.nonzero(kr)[0]] = (v >> np.uint64(b)).astype(np.uint8) & 1
    want = np.packbits(bits, axis=2)
    want[0, 0] = row0
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x.ravel(), off, r, k * rows, row0)]
    planes = torch.full((want.size + 64,), 0xA7, dtype=torch.uint8, device="cuda")
    out = (C.c_double * 3)()
    for shift in (0, 4):   # 16-byte aligned planes, then 4-byte aligned ones
        planes.fill_(0xA7)
        torch.cuda.synchronize()
        a = NoAllocArgs(dev[0].data_ptr(), dev[1].data_ptr(), rows, dev[2].data_ptr(), len(r), dev[3].data_ptr(), len(k),
                        dev[4].data_ptr(), B, d, row_bytes, planes.data_ptr() + shift,
                        C.cast(out, C.POINTER(C.c_double)), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert lib.lakgb_xcalc_noalloc(C.byref(a)) == 0
        got = planes.cpu().numpy()
        assert np.array_equal(np.array(out[:]), np.array([lo, hi, mlt]), equal_nan=True)
        assert np.array_equal(got[shift:shift + want.size].reshape(want.shape), want)
        assert (got[:shift] == 0xA7).all() and (got[shift + want.size:] == 0xA7).all()
