"""Performance cases: the work that users of this package have it do, through
its public entry points (whole solves and the C entry points below them), at
the sizes of the repository's own configurations and around them.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same
ranges, ``prepare(case, seed)`` makes what a caller has in hand before the
call, ``run(state)`` makes the call and returns its outputs, ``work(case)``
counts the bytes and operations a call cannot do without (one multiply and
add of a bit pair = 2 flops) and ``exact(case, seed)`` evaluates the outputs
in 64-bit floating point with plain torch.

Every input is synthetic and made on the GPU from the seed: Bernoulli
genotype bits with a minor-allele frequency per SNP, a planted bicluster in
the cases of a solve, normal scores.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from lakcluster_c_gb300 import abi, gram_pass, serve, solve
from lakcluster_c_gb300._lib import load

BLOCK = abi.POPLENGTH
DEV = "cuda"

# ---------------------------------------------------------------------------
# the cases


def listed():
    return [
        # The smallest whole solve in use: cases only, Bernoulli(0.5), one bin
        # (the configuration that the CPU program also runs in seconds).
        # Elimination steps over a few hundred rows: launches and latency.
        dict(name="solve_cases_1024", op="solve", cases=1024, controls=0, cols=1024, bins=1, covariates=1, b_mlt=32,
             gamma=0.05, qc="YnWt", maf_lo=0.5, maf_hi=0.5),
        # The ordinary whole solve: case/control study, 2 covariate bins.
        dict(name="solve_case_control", op="solve", cases=4096, controls=4096, cols=16384, bins=2, covariates=1,
             b_mlt=32, gamma=0.05, qc="YnWt", maf_lo=0.05, maf_hi=0.5),
        # Permutation nulls of a study, solved together on one GPU.
        dict(name="null_solves_batch", op="null_batch", instances=8, rows_lo=1024, rows_hi=4096, cols_lo=4096,
             cols_hi=8192, workers=8, gamma=0.05),
        # The Gram pass of a large study, operands in HBM, one launch per
        # product (row bins half as high as the largest configuration's).
        dict(name="gram_pass_large", op="gram_pass", cases=16384, controls=16384, cols=131072, bins=3, grouped=False,
             maf_lo=0.01, maf_hi=0.5),
        # The Gram pass of the ordinary study as one grouped launch.
        dict(name="gram_pass_grouped", op="gram_pass", cases=4096, controls=4096, cols=16384, bins=2, grouped=True,
             maf_lo=0.05, maf_hi=0.5),
        # One low-rank update Gram of an elimination step: every retained row
        # pair over the few hundred SNPs just removed.
        dict(name="gram_update", op="gram_update", rows_a=2018, rows_z=2025, cols=820, keep=0.9, type="pm"),
        # One Gram through the reference's entry point, host buffers in and
        # out, masked rows and columns, ragged sizes.
        dict(name="gram_host", op="gram_host", rows_a=2010, rows_z=2031, cols=16384, keep=0.9, symmetric=False),
        # Row terms (allele-frequency moments) of a study's bin, host buffers.
        dict(name="row_terms_host", op="row_terms", rows=8192, cols=65536, keep=0.95),
        # Quantisation of a score matrix into bit planes on device buffers.
        dict(name="quantise_device", op="quantise", rows=4096, cols=4001, b_mlt=32, keep=0.97),
        # The bit-plane loop product behind the SNP scores, host buffers.
        dict(name="loop_product_host", op="loop_product", snps=4096, rows_y=1024, rows_w=1000, b_mlt=32, covariates=1,
             keep=0.95),
        # SNP x SNP product of an elimination step: retained SNPs against the
        # SNPs just removed, over a bin's rows.
        dict(name="snp_product_host", op="snp_product", snps=7800, snps_y=410, rows=2018, covariates=1, keep=0.95),
        # Input pipeline: PLINK .bed records to the sorted allele matrix.
        dict(name="bed_to_b16_host", op="bed", snps=60000, patients=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["solve", "null_batch", "gram_pass", "gram_pass", "gram_update", "gram_host", "row_terms",
                     "quantise", "loop_product", "snp_product", "bed"])
    if op == "solve":
        # covariate columns and the SNP x SNP column strategy multiply the
        # work, so their SNP range ends lower
        covariates = rng.choice([1, 1, 1, 2, 3])
        qc = rng.choice(["YnWt", "YnWt", "YnWt", "ZtSWn"])
        cols_hi = 1024 if qc == "ZtSWn" else (16384 if covariates == 1 else 4096)
        rows_hi = 1024 if qc == "ZtSWn" else (4096 if covariates == 1 else 2048)
        return dict(op=op, cases=_log_int(rng, 256, rows_hi), controls=_log_int(rng, 256, rows_hi),
                    cols=_log_int(rng, 512, cols_hi), bins=rng.choice([1, 2, 3]), covariates=covariates,
                    b_mlt=rng.choice([16, 32]), gamma=rng.choice([0.05, 0.08, 0.125]), qc=qc, maf_lo=0.05, maf_hi=0.5)
    if op == "null_batch":
        lo, clo = _log_int(rng, 512, 1500), _log_int(rng, 2048, 5000)
        return dict(op=op, instances=rng.randint(4, 8), rows_lo=lo, rows_hi=2 * lo, cols_lo=clo, cols_hi=2 * clo - 1,
                    workers=rng.choice([4, 8]), gamma=0.05)
    if op == "gram_pass":
        grouped = rng.random() < 0.5
        return dict(op=op, cases=_log_int(rng, 1024, 16000), controls=_log_int(rng, 1024, 16000),
                    cols=_log_int(rng, 4096, 131072), bins=rng.choice([1, 2, 3]), grouped=grouped,
                    maf_lo=rng.choice([0.01, 0.05]), maf_hi=0.5)
    if op == "gram_update":
        return dict(op=op, rows_a=_log_int(rng, 40, 8192), rows_z=_log_int(rng, 40, 8192), cols=_log_int(rng, 60, 4000),
                    keep=rng.choice([1.0, 0.9, 0.6]), type=rng.choice(["pm", "pm", "pm", "00"]))
    if op == "gram_host":
        sym = rng.random() < 0.4
        n = _log_int(rng, 200, 5000)
        return dict(op=op, rows_a=n, rows_z=n if sym else _log_int(rng, 200, 5000), cols=_log_int(rng, 1000, 65536),
                    keep=rng.choice([1.0, 0.9, 0.6]), symmetric=sym)
    if op == "row_terms":
        return dict(op=op, rows=_log_int(rng, 200, 24000), cols=_log_int(rng, 2000, 65536), keep=rng.choice([1.0, 0.95, 0.6]))
    if op == "quantise":
        return dict(op=op, rows=_log_int(rng, 150, 6000), cols=_log_int(rng, 150, 6000), b_mlt=rng.choice([8, 16, 32]),
                    keep=rng.choice([1.0, 0.97, 0.6]))
    if op == "loop_product":
        return dict(op=op, snps=_log_int(rng, 200, 12000), rows_y=_log_int(rng, 150, 2000), rows_w=_log_int(rng, 150, 1200),
                    b_mlt=rng.choice([16, 32, 32]), covariates=rng.choice([1, 1, 2]), keep=rng.choice([1.0, 0.95, 0.6]))
    if op == "snp_product":
        return dict(op=op, snps=_log_int(rng, 400, 16000), snps_y=_log_int(rng, 30, 800), rows=_log_int(rng, 300, 8000),
                    covariates=rng.choice([1, 1, 2]), keep=rng.choice([1.0, 0.95, 0.6]))
    return dict(op="bed", snps=_log_int(rng, 3000, 60000), patients=_log_int(rng, 1000, 8192))


# ---------------------------------------------------------------------------
# inputs


def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * int(seed) + salt)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV)


def _pack(bits, nbytes):
    """(rows, n) bool -> (rows, nbytes) uint8, MSB first, zero padded."""
    rows, n = bits.shape
    if n < 8 * nbytes:
        bits = torch.nn.functional.pad(bits, (0, 8 * nbytes - n))
    w = torch.tensor([128, 64, 32, 16, 8, 4, 2, 1], dtype=torch.uint8, device=DEV)
    return (bits.reshape(rows, nbytes, 8).to(torch.uint8) * w).sum(dim=2, dtype=torch.uint8)


def _bernoulli(g, rows, p, nbytes, chunk=4096):
    """Packed rows of bits that are set with the column probabilities p."""
    out = torch.empty((rows, nbytes), dtype=torch.uint8, device=DEV)
    step = max(1, min(chunk, (1 << 28) // max(1, p.numel())))
    for r in range(0, rows, step):
        n = min(step, rows - r)
        out[r:r + n] = _pack(_rand(g, n, p.numel()) < p, nbytes)
    return out


def _unpack(packed, n):
    """(rows, bytes) uint8 -> (rows, n) float32 of 0 / 1."""
    sh = torch.tensor([7, 6, 5, 4, 3, 2, 1, 0], dtype=torch.uint8, device=DEV)
    return ((packed.unsqueeze(2) >> sh) & 1).reshape(packed.shape[0], -1)[:, :n].to(torch.float32)


def _maf(g, cols, lo=0.05, hi=0.5):
    return lo + (hi - lo) * _rand(g, cols)


def _ajdk(p):
    """The 15 x P allele weights alpha^j D^k of the blocks' mean frequencies
    (row j + 5 k), and the block frequencies' alpha and D."""
    pad = (-p.numel()) % BLOCK
    n = torch.full((p.numel() // BLOCK + (1 if pad else 0),), float(BLOCK), dtype=torch.float64, device=DEV)
    if pad:
        n[-1] = BLOCK - pad
    f = torch.nn.functional.pad(p.double(), (0, pad)).reshape(-1, BLOCK).sum(1) / n
    a, d = f - (1 - f), 1.0 / torch.clamp(4.0 * f * (1 - f), min=0.01)
    return torch.stack([a ** j * d ** k for k in range(3) for j in range(5)])


def _keep(g, n, frac):
    """A mask that retains that share of n, drawn at random."""
    m = torch.zeros(n, dtype=torch.bool, device=DEV)
    m[torch.randperm(n, generator=g, device=DEV)[: max(1, round(frac * n))]] = True
    return m


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _handle(packed, ncols, row_keep=None, col_keep=None):
    """The M_handle of packed rows, with the rows and columns still retained."""
    return abi.MHandle(None, nrows=packed.shape[0], ncols=ncols, wX=_host(packed),
                       mr_j=None if row_keep is None else _host(row_keep).astype(np.uint8),
                       mc_j=None if col_keep is None else _host(col_keep).astype(np.uint8))


def _threads():
    return C.byref(C.c_int(0)), None, None


def _dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


# ---------------------------------------------------------------------------
# whole solves


def _split_bins(packed, bins, g):
    b = torch.randint(0, bins, (packed.shape[0],), generator=g, device=DEV)
    b[:2 * bins] = torch.arange(2 * bins, device=DEV) % bins  # no bin is empty
    return [_host(packed[b == k]) for k in range(bins)]


def _planted(g, packed, cols, nbytes):
    """A bicluster of 1/16 of the rows and 1/32 of the SNPs with 5 % flips."""
    rows, k = packed.shape[0], max(2, packed.shape[0] // 16)
    kc = max(16, cols // 32) // 8 * 8
    pat = _rand(g, kc) < 0.5
    packed[:k, : kc // 8] = _pack(pat ^ (_rand(g, k, kc) < 0.05), kc // 8)
    return packed[torch.randperm(rows, generator=g, device=DEV)]


def _solve_problem(cases, controls, cols, bins, covariates, b_mlt, gamma, qc, maf_lo, maf_hi, seed):
    g = _gen(seed)
    nbytes = (cols + 15) // 16 * 2
    p = _maf(g, cols, maf_lo, maf_hi)
    A = _split_bins(_planted(g, _bernoulli(g, cases, p, nbytes), cols, nbytes), bins, g)
    Z = _split_bins(_bernoulli(g, controls, p, nbytes), bins, g) if controls else None
    T = S = None
    if covariates > 1:
        def cov(x):
            t = _rand(g, x.shape[0], covariates) < 0.5
            t[:, 0] = True
            return _host(t).astype(np.uint8)
        T, S = [cov(a) for a in A], [cov(z) for z in (Z or [a[:0] for a in A])]
    return solve.Problem(A, Z, gamma=gamma, B_MLT=b_mlt, T_bins=T, S_bins=S, qc_strategy=qc, packed_ncols=cols)


def _take_result(lib, res):
    n6, n2 = 6 * res.iterations, 2 * res.n_xdrop
    try:
        return dict(trace=np.ctypeslib.as_array(res.trace, (n6,)).copy(),
                    xdrop_a=np.ctypeslib.as_array(res.xdrop_a, (n2,)).copy(),
                    xdrop_b=np.ctypeslib.as_array(res.xdrop_b, (n2,)).copy())
    finally:
        lib.lakgb_bcc_result_free(C.byref(res))


def _run_solve(s):
    res = solve.BccResult()
    if s.lib.lakgb_bcc_solve(C.byref(s.prob), C.byref(res)) != 0:
        raise RuntimeError("lakgb_bcc_solve failed")
    return _take_result(s.lib, res)


def _null_sizes(c):
    n = c["instances"]
    f = [i / max(1, n - 1) for i in range(n)]
    rows = [int(round(c["rows_lo"] * (c["rows_hi"] / c["rows_lo"]) ** x)) for x in f]
    cols = [int(round(c["cols_lo"] * (c["cols_hi"] / c["cols_lo"]) ** f[(5 * i + 2) % n])) for i in range(n)]
    return list(zip(rows, cols))


def _prepare_null_batch(c, seed):
    ps = [_solve_problem(r // 2, r - r // 2, m, 1, 1, 32, c["gamma"], "YnWt", 0.05, 0.5, 64 * seed + i)
          for i, (r, m) in enumerate(_null_sizes(c))]
    lib = serve.bind(load())
    lib.lakgb_bcc_solve_many.argtypes = [C.POINTER(solve.BccProblem), C.c_int, C.POINTER(solve.BccResult),
                                         C.POINTER(C.c_int), C.c_int, C.c_longlong]
    lib.lakgb_bcc_solve_many.restype = C.c_int
    arr = (solve.BccProblem * len(ps))(*[p.prob for p in ps])
    return dict(ps=ps, arr=arr, lib=lib, workers=c["workers"])


def _run_null_batch(s):
    n = len(s["ps"])
    res, rcs = (solve.BccResult * n)(), (C.c_int * n)()
    if s["lib"].lakgb_bcc_solve_many(s["arr"], n, res, rcs, s["workers"], 0) != 0:
        raise RuntimeError("lakgb_bcc_solve_many: a solve failed")
    return [_take_result(s["lib"], r) for r in res]


# ---------------------------------------------------------------------------
# Grams on device buffers


def _bin_sizes(n, bins):
    """Bins of unequal size, as covariate categories make them."""
    w = [1.0 + 0.07 * k for k in range(bins)]
    s = [int(n * x / sum(w)) for x in w]
    s[-1] += n - sum(s)
    return s


def _mask_sums(w, mask):
    c = _unpack(mask.reshape(1, -1), 8 * mask.numel()).reshape(-1, BLOCK).sum(1).double()
    return float((w[5] * c).sum()), float((w[7] * c).sum()), c


def _row_term(packed, mask, w6):
    """Row sums sum_b w_b (2 popcount(row & mask) - popcount(mask)) per row."""
    out = []
    for r in range(0, packed.shape[0], 2048):
        x = _unpack(packed[r:r + 2048] & mask, 8 * packed.shape[1]).reshape(-1, packed.shape[1] // 240, BLOCK).sum(2)
        out.append((2.0 * x.double() - _unpack(mask.reshape(1, -1), 8 * mask.numel()).reshape(1, -1, BLOCK).sum(2)) @ w6)
    return torch.cat(out) if out else torch.zeros(0, dtype=torch.float64, device=DEV)


def _gram_pass_inputs(c, seed):
    g = _gen(seed, 1)
    cols, rb = c["cols"], abi.bsize(c["cols"])
    p = _maf(g, cols, c["maf_lo"], c["maf_hi"])
    w = _ajdk(p)
    mask = _pack(torch.ones((1, cols), dtype=torch.bool, device=DEV), rb)[0]
    x = dict(w=w, mask=mask, rows={}, lf={})
    for key, n in (("A", c["cases"]), ("Z", c["controls"])):
        for b, m in enumerate(_bin_sizes(n, c["bins"])):
            x["rows"][key, b] = _bernoulli(g, m, p, rb)
            x["lf"][key, b] = _row_term(x["rows"][key, b], mask, w[6])
    return x


def _gram_args(wA, wZ, mask, w, sums, lfA, lfZ, idx, out, symmetric=False, a_rows=None, z_rows=None, type_flag=abi.TYPE_pm):
    """lakgb_gram_args over device tensors; outputs at the rows' own indices
    (stride = A rows).  `idx` is an int32 arange at least as long as the rows."""
    a = gram_pass.GramArgs()
    a_rows = idx if a_rows is None else a_rows
    z_rows = idx if z_rows is None else z_rows
    a.wA, a.a_rowb, a.nA, a.a_row_bytes = wA.data_ptr(), a_rows.data_ptr(), lfA.numel(), wA.shape[1]
    a.wZ, a.z_rowb, a.nZ, a.z_row_bytes = wZ.data_ptr(), z_rows.data_ptr(), lfZ.numel(), wZ.shape[1]
    a.mask, a.P, a.D, a.type_flag = mask.data_ptr(), wA.shape[1] // 240, w[5].data_ptr(), type_flag
    a.a0d1, a.a2d1 = sums[0], sums[1]
    if type_flag == abi.TYPE_pm:
        a.lfA, a.lfZ = lfA.data_ptr(), lfZ.data_ptr()
    a.out_r = a.out_c2 = idx.data_ptr()
    a.out_c = a.out_r2 = idx.data_ptr()
    a.out_stride, a.out, a.symmetric = lfA.numel(), out.data_ptr(), int(symmetric)
    return a


def _prepare_gram_pass(c, seed):
    x = _gram_pass_inputs(c, seed)
    lib = load()
    lib.lakgb_gram_device.argtypes = [C.POINTER(gram_pass.GramArgs)]
    lib.lakgb_gram_device.restype = C.c_int
    sums = _mask_sums(x["w"], x["mask"])
    x["idx"] = torch.arange(max(t.shape[0] for t in x["rows"].values()), dtype=torch.int32, device=DEV)
    x["out"], args = [], []
    for kind, b1, b2, sym in gram_pass.products(c["bins"]):
        k1, k2 = ("A", b1), (("Z" if kind == "AnZt" else "A"), b2)
        n = x["rows"][k1].shape[0] * x["rows"][k2].shape[0]
        x["out"].append(torch.empty(n, dtype=torch.float64, device=DEV))
        args.append(_gram_args(x["rows"][k1], x["rows"][k2], x["mask"], x["w"], sums, x["lf"][k1], x["lf"][k2],
                               x["idx"], x["out"][-1], sym))
    x["lib"], x["args"], x["group"] = lib, args, None
    x["stream"] = torch.cuda.current_stream().cuda_stream
    for a in args:
        a.stream = x["stream"]
    if c["grouped"]:
        x["arr"] = (gram_pass.GramArgs * len(args))(*args)
        torch.cuda.synchronize()
        x["group"] = _Group(lib, lib.lakgb_gram_group_create(C.cast(x["arr"], C.c_void_p), len(args)))
    return x


class _Group:
    """A grouped Gram's handle, destroyed with the state that holds it."""

    def __init__(self, lib, h):
        if not h:
            raise RuntimeError("lakgb_gram_group_create failed")
        self.lib, self.h = lib, h

    def __del__(self):
        torch.cuda.synchronize()
        self.lib.lakgb_gram_group_destroy(self.h)


def _run_gram_device(x):
    if x["group"] is not None:
        if x["lib"].lakgb_gram_group_run(x["group"].h, C.c_void_p(x["stream"] or None)) != 0:
            raise RuntimeError("lakgb_gram_group_run failed")
    else:
        for a in x["args"]:
            if x["lib"].lakgb_gram_device(C.byref(a)) != 0:
                raise RuntimeError("lakgb_gram_device failed")
    return x["out"]


def _gram_exact(wA, wZ, mask, w, sums, lfA, lfZ, type_flag=abi.TYPE_pm):
    """The Gram in float64: per block, integer counts by an exact matrix
    product of 0 / 1 values, then the weighted sum over the blocks."""
    acc = torch.zeros((wA.shape[0], wZ.shape[0]), dtype=torch.float64, device=DEV)
    for b in range(mask.numel() // 240):
        s = slice(240 * b, 240 * b + 240)
        a, z = _unpack(wA[:, s] & mask[s], BLOCK).half(), _unpack(wZ[:, s] & mask[s], BLOCK).half()
        c = (a @ z.T).double()  # <= 1920: exact in half
        if type_flag == abi.TYPE_pm:
            c = a.float().sum(1).double()[:, None] + z.float().sum(1).double()[None, :] - 2.0 * c
        acc += w[5][b] * c
    if type_flag == abi.TYPE_pm:
        acc = sums[0] - 2.0 * acc - ((lfA[:, None] + lfZ[None, :]) - sums[1])
    return acc.T.reshape(-1)  # element (i, k) at i + k * rows of A


def _exact_gram_pass(c, seed):
    x = _gram_pass_inputs(c, seed)
    sums = _mask_sums(x["w"], x["mask"])
    out = []
    for kind, b1, b2, _ in gram_pass.products(c["bins"]):
        k1, k2 = ("A", b1), (("Z" if kind == "AnZt" else "A"), b2)
        out.append(_gram_exact(x["rows"][k1], x["rows"][k2], x["mask"], x["w"], sums, x["lf"][k1], x["lf"][k2]))
    return out


def _work_gram_pass(c):
    a, z = _bin_sizes(c["cases"], c["bins"]), _bin_sizes(c["controls"], c["bins"])
    pairs = sum(a[b1] * (z if kind == "AnZt" else a)[b2] for kind, b1, b2, _ in gram_pass.products(c["bins"]))
    return {"bytes": (c["cases"] + c["controls"]) * abi.bsize(c["cols"]) + 8 * pairs, "flops": 2.0 * pairs * c["cols"]}


def _gram_update_inputs(c, seed):
    g = _gen(seed, 2)
    cols, rb = c["cols"], abi.bsize(c["cols"])
    p = _maf(g, cols)
    x = dict(w=_ajdk(p), mask=_pack(_keep(g, cols, c["keep"]).reshape(1, -1), rb)[0])
    for k, n in (("A", c["rows_a"]), ("Z", c["rows_z"])):
        stored = max(n, int(n / c["keep"]))  # the retained rows are some of the stored ones
        x["w" + k] = _bernoulli(g, stored, p, rb)
        x["r" + k] = torch.sort(torch.randperm(stored, generator=g, device=DEV)[:n])[0].to(torch.int32)
        x["lf" + k] = _row_term(x["w" + k][x["r" + k].long()], x["mask"], x["w"][6])
    x["type"] = abi.TYPE_pm if c["type"] == "pm" else abi.TYPE_00
    return x


def _prepare_gram_update(c, seed):
    x = _gram_update_inputs(c, seed)
    lib = load()
    lib.lakgb_gram_device.argtypes = [C.POINTER(gram_pass.GramArgs)]
    lib.lakgb_gram_device.restype = C.c_int
    x["idx"] = torch.arange(max(c["rows_a"], c["rows_z"]), dtype=torch.int32, device=DEV)
    x["out"] = [torch.empty(c["rows_a"] * c["rows_z"], dtype=torch.float64, device=DEV)]
    a = _gram_args(x["wA"], x["wZ"], x["mask"], x["w"], _mask_sums(x["w"], x["mask"]), x["lfA"], x["lfZ"], x["idx"],
                   x["out"][0], a_rows=x["rA"], z_rows=x["rZ"], type_flag=x["type"])
    a.stream = torch.cuda.current_stream().cuda_stream
    x["lib"], x["args"], x["group"] = lib, [a], None
    return x


def _exact_gram_update(c, seed):
    x = _gram_update_inputs(c, seed)
    return [_gram_exact(x["wA"][x["rA"].long()], x["wZ"][x["rZ"].long()], x["mask"], x["w"],
                        _mask_sums(x["w"], x["mask"]), x["lfA"], x["lfZ"], x["type"])]


# ---------------------------------------------------------------------------
# entry points on host buffers


def _gram_host_inputs(c, seed):
    g = _gen(seed, 3)
    cols, rb = c["cols"], abi.bsize(c["cols"])
    p = _maf(g, cols)
    x = dict(w=_ajdk(p), ck=_keep(g, cols, c["keep"]))
    x["mask"] = _pack(x["ck"].reshape(1, -1), rb)[0]
    for k, n in (("A", c["rows_a"]), ("Z", c["rows_z"])):
        if k == "Z" and c["symmetric"]:
            x["wZ"], x["kZ"] = x["wA"], x["kA"]
        else:
            x["w" + k], x["k" + k] = _bernoulli(g, n, p, rb), _keep(g, n, c["keep"])
        lf = torch.zeros((n, abi.AJDK_TOT), dtype=torch.float64, device=DEV)
        lf[:, 6] = _row_term(x["w" + k], x["mask"], x["w"][6])
        x["lf" + k] = lf
    return x


def _prepare_gram_host(c, seed):
    x = _gram_host_inputs(c, seed)
    MA = _handle(x["wA"], c["cols"], x["kA"], x["ck"])
    MZ = MA if c["symmetric"] else _handle(x["wZ"], c["cols"], x["kZ"], x["ck"])
    lf = [abi.LHandle.from_matrix(_host(x["lf" + k]), abi.SPACING_b, abi.SPACING_a) for k in "AZ"]
    out = abi.LHandle(MA.rpop_b * MZ.rpop_b)
    return dict(fn=load().wrap_AnAt_vv__run if c["symmetric"] else load().wrap_AnZt_vv__run, MA=MA, MZ=MZ, lf=lf,
                w=_host(x["w"]), out=out, outp=out.ptr)


def _run_gram_host(s):
    s["fn"](*_threads(), abi.TYPE_pm, abi.SPACING_b, abi.SPACING_b, s["MA"].ptr, s["MZ"].ptr, _dp(s["w"]),
            s["lf"][0].ptr, s["lf"][1].ptr, C.byref(s["outp"]))
    return s["out"].buf


def _exact_gram_host(c, seed):
    x = _gram_host_inputs(c, seed)
    a, z = torch.nonzero(x["kA"])[:, 0], torch.nonzero(x["kZ"])[:, 0]
    o = _gram_exact(x["wA"][a], x["wZ"][z], x["mask"], x["w"], _mask_sums(x["w"], x["mask"]), x["lfA"][a, 6], x["lfZ"][z, 6])
    full = torch.zeros((c["rows_z"], c["rows_a"]), dtype=torch.float64, device=DEV)
    full[z[:, None], a[None, :]] = o.reshape(z.numel(), a.numel())
    return full.reshape(-1)


def _row_terms_inputs(c, seed):
    g = _gen(seed, 4)
    cols, rb = c["cols"], abi.bsize(c["cols"])
    p = _maf(g, cols)
    return dict(w=_ajdk(p), ck=_keep(g, cols, c["keep"]), W=_bernoulli(g, c["rows"], p, rb), kr=_keep(g, c["rows"], c["keep"]))


def _prepare_row_terms(c, seed):
    x = _row_terms_inputs(c, seed)
    M = _handle(x["W"], c["cols"], x["kr"], x["ck"])
    out = abi.LHandle(c["rows"] * abi.AJDK_TOT)
    return dict(lib=load(), M=M, w=_host(x["w"]), out=out, outp=out.ptr)


def _run_row_terms(s):
    s["lib"].wrap_An_ajdk_v(*_threads(), abi.TYPE_pm, abi.SPACING_a, s["M"].ptr, _dp(s["w"]), C.byref(s["outp"]))
    return s["out"].buf


def _exact_row_terms(c, seed):
    x = _row_terms_inputs(c, seed)
    mask = _pack(x["ck"].reshape(1, -1), x["W"].shape[1])[0]
    o = torch.stack([_row_term(x["W"], mask, x["w"][k]) for k in range(abi.AJDK_TOT)])
    o[:, ~x["kr"]] = 0.0
    return o.reshape(-1)


class _NoallocArgs(C.Structure):
    _fields_ = [("lf", C.c_void_p), ("row_off_a", C.c_void_p), ("nrows_a", C.c_int), ("rows_j", C.c_void_p),
                ("n_rows_j", C.c_int), ("cols_j", C.c_void_p), ("n_cols_j", C.c_int), ("row0", C.c_void_p),
                ("b_mlt", C.c_int), ("d_mlt", C.c_longlong), ("brows", C.c_longlong), ("planes", C.c_void_p),
                ("min_max_mlt", C.c_void_p), ("stream", C.c_void_p)]


def _quantise_inputs(c, seed):
    g = _gen(seed, 5)
    lf = 300.0 * torch.randn(c["rows"] * c["cols"], generator=g, device=DEV, dtype=torch.float64)
    return lf, _keep(g, c["rows"], c["keep"]), _keep(g, c["cols"], c["keep"])


def _prepare_quantise(c, seed):
    """Column-major scores lf[r + c * rows], retained rows and columns."""
    lf, kr, kc = _quantise_inputs(c, seed)
    n = c["rows"]
    r, k = torch.nonzero(kr)[:, 0], torch.nonzero(kc)[:, 0]
    brows = abi.bsize(n)
    s = dict(lib=load(), lf=lf, off=torch.where(kr, torch.arange(n, device=DEV), -1), r=r, k=k * n,
             row0=_pack(kr.reshape(1, -1), brows)[0], mmm=np.zeros(3),
             planes=torch.empty(((c["b_mlt"] + 1) * k.numel(), brows), dtype=torch.uint8, device=DEV))
    s["lib"].lakgb_xcalc_noalloc.argtypes = [C.POINTER(_NoallocArgs)]
    s["lib"].lakgb_xcalc_noalloc.restype = C.c_int
    s["a"] = _NoallocArgs(lf.data_ptr(), s["off"].data_ptr(), n, s["r"].data_ptr(), r.numel(), s["k"].data_ptr(),
                          k.numel(), s["row0"].data_ptr(), c["b_mlt"], 1 << c["b_mlt"], brows, s["planes"].data_ptr(),
                          s["mmm"].ctypes.data, torch.cuda.current_stream().cuda_stream)
    return s


def _run_quantise(s):
    if s["lib"].lakgb_xcalc_noalloc(C.byref(s["a"])) != 0:
        raise RuntimeError("lakgb_xcalc_noalloc failed")
    return dict(planes=s["planes"], min_max_mlt=s["mmm"])


def _exact_quantise(c, seed):
    lf, kr, kc = _quantise_inputs(c, seed)
    x = lf.reshape(c["cols"], c["rows"])[kc][:, kr]
    mn, mx = float(x.min()), float(x.max())
    lo, hi = mn - 0.0625 * (mx - mn), mx + 0.0625 * (mx - mn)
    return dict(planes=None, min_max_mlt=np.array([lo, hi, (1 << c["b_mlt"]) / (hi - lo)]))


def _loop_inputs(c, seed):
    """SNP rows over cases (At) and controls (Zt), covariates, and the bit
    planes of a score matrix over the cases, per retained control."""
    g = _gen(seed, 6)
    ny, nw, B = c["rows_y"], c["rows_w"], c["b_mlt"]
    ky, kw, ks = _keep(g, ny, c["keep"]), _keep(g, nw, c["keep"]), _keep(g, c["snps"], c["keep"])
    p = _maf(g, c["snps"])
    x = dict(ky=ky, kw=kw, ks=ks, w=_ajdk(p))
    x["At"] = _pack(_rand(g, c["snps"], ny) < p[:, None], abi.bsize(ny))
    x["Zt"] = _pack(_rand(g, c["snps"], nw) < p[:, None], abi.bsize(nw))
    ones = torch.ones((1, max(ny, nw)), dtype=torch.bool, device=DEV)
    extra = _rand(g, c["covariates"] - 1, max(ny, nw)) < 0.5
    tt = torch.cat([ones, extra])
    x["Tt"], x["St"] = _pack(tt[:, :ny], abi.bsize(ny)), _pack(tt[:, :nw], abi.bsize(nw))
    # scores of the retained controls in [1, 2^B), quantised; plane k of a
    # control holds bit B - k, and one leading plane marks the retained cases
    m = int(kw.sum())
    v = (2.0 ** (B - 1) * (1.0 + 0.2 * torch.randn((m, ny), generator=g, device=DEV, dtype=torch.float64)))
    q = torch.clamp(v, 1.0, 2.0 ** B - 1.0).to(torch.int64) * ky
    x["q"] = q
    planes = torch.zeros(((B + 1) * m, abi.bsize(ny)), dtype=torch.uint8, device=DEV)
    for k in range(1, B + 1):
        planes[k::B + 1] = _pack(((q >> (B - k)) & 1).bool(), abi.bsize(ny))
    planes[0] = _pack(ky.reshape(1, -1), abi.bsize(ny))[0]
    x["planes"] = planes
    x["min"], x["mlt"] = -900.0, 2.0 ** B / 1800.0
    return x


def _prepare_loop(c, seed):
    x = _loop_inputs(c, seed)
    ny, nw, n = c["rows_y"], c["rows_w"], c["snps"]
    s = dict(lib=load(), w=_host(x["w"]))
    s["At"], s["Zt"] = _handle(x["At"], ny, x["ks"], x["ky"]), _handle(x["Zt"], nw, x["ks"], x["kw"])
    s["Tt"], s["St"] = _handle(x["Tt"], ny, None, x["ky"]), _handle(x["St"], nw, None, x["kw"])
    empty = torch.zeros((1, abi.bsize(16)), dtype=torch.uint8, device=DEV)
    s["Yn"], s["Wn"] = (_handle(empty.expand(r, -1), 16, k) for r, k in ((ny, x["ky"]), (nw, x["kw"])))
    s["X"] = _handle(x["planes"], ny, None, x["ky"])
    s["X"].s.ncols_per_z, s["X"].s.min_d, s["X"].s.mlt_d = c["b_mlt"] + 1, x["min"], x["mlt"]
    s["out"] = abi.LHandle(n * c["covariates"])
    s["outp"] = s["out"].ptr
    return s


def _run_loop(s):
    s["lib"].wrap_At_T_YnWt_S_Zn_ww__run(*_threads(), abi.SPACING_a, abi.SPACING_a, s["At"].ptr, s["Tt"].ptr, s["Yn"].ptr,
                                         s["Wn"].ptr, s["St"].ptr, s["Zt"].ptr, _dp(s["w"]), s["X"].ptr, C.byref(s["outp"]))
    return s["out"].buf


def _exact_loop(c, seed):
    x = _loop_inputs(c, seed)
    ny, nw = c["rows_y"], c["rows_w"]
    y, k = torch.nonzero(x["ky"])[:, 0], torch.nonzero(x["kw"])[:, 0]
    a_all = x["w"][1].repeat_interleave(BLOCK)[: c["snps"]]
    at, zt = (2.0 * _unpack(x[n], m).double() - 1.0 for n, m in (("At", ny), ("Zt", nw)))
    tt, stt = (2.0 * _unpack(x[n], m).double() - 1.0 for n, m in (("Tt", ny), ("St", nw)))
    q = x["q"].double()
    out = torch.zeros((c["covariates"], c["snps"]), dtype=torch.float64, device=DEV)
    for t in range(c["covariates"]):
        row = at[:, y] * tt[t, y]
        base, tbase = row.sum(1) * x["min"] * x["mlt"], float(tt[t, y].sum()) * x["min"] * x["mlt"]
        X = (base[:, None] + row @ q[:, y].T) / x["mlt"] - a_all[:, None] * (tbase + q[:, y] @ tt[t, y])[None, :] / x["mlt"]
        out[t] = (X * stt[t, k] * (zt[:, k] - a_all[:, None])).sum(1)
    out[:, ~x["ks"]] = 0.0
    return out.reshape(-1)


def _snp_inputs(c, seed):
    g = _gen(seed, 7)
    n, m, r, t = c["snps"], c["snps_y"], c["rows"], c["covariates"]
    pa, py = _maf(g, n), _maf(g, m)
    x = dict(wa=_ajdk(pa), wy=_ajdk(py), kr=_keep(g, r, c["keep"]), ka=_keep(g, n, c["keep"]))
    x["At"], x["Yt"] = (_pack(_rand(g, q.numel(), r) < q[:, None], abi.bsize(r)) for q in (pa, py))
    tt = _rand(g, t, r) < 0.5
    tt[0] = True
    x["Tt"] = _pack(tt, abi.bsize(r))
    pm = lambda w: (2.0 * _unpack(w, r).double() - 1.0) * x["kr"]  # noqa: E731
    x["a"], x["y"], x["t"] = pm(x["At"]), pm(x["Yt"]), pm(x["Tt"])
    x["lfa"], x["lfy"] = x["a"] @ x["t"].T, x["y"] @ x["t"].T
    return x


def _prepare_snp(c, seed):
    x = _snp_inputs(c, seed)
    s = dict(lib=load(), wa=_host(x["wa"]), wy=_host(x["wy"]), At=_handle(x["At"], c["rows"], x["ka"], x["kr"]),
             Yt=_handle(x["Yt"], c["rows"], None, x["kr"]), Tt=_handle(x["Tt"], c["rows"], None, x["kr"]),
             la=abi.LHandle.from_matrix(_host(x["lfa"])), ly=abi.LHandle.from_matrix(_host(x["lfy"])))
    s["out"] = abi.LHandle(c["snps"] * c["snps_y"] * c["covariates"])
    s["outp"] = s["out"].ptr
    return s


def _run_snp(s):
    s["lib"].wrap_AtTYn_vv__run(*_threads(), abi.SPACING_a, abi.SPACING_a, abi.SPACING_a, s["At"].ptr, s["Tt"].ptr,
                                s["Yt"].ptr, _dp(s["wa"]), _dp(s["wy"]), s["la"].ptr, s["ly"].ptr, C.byref(s["outp"]))
    return s["out"].buf


def _exact_snp(c, seed):
    x = _snp_inputs(c, seed)
    aa, ay = (w[1].repeat_interleave(BLOCK)[:n] for w, n in ((x["wa"], c["snps"]), (x["wy"], c["snps_y"])))
    out = torch.zeros((c["covariates"], c["snps_y"], c["snps"]), dtype=torch.float64, device=DEV)
    for t in range(c["covariates"]):
        o = (x["a"] * x["t"][t]) @ x["y"].T - x["lfa"][:, t:t + 1] * ay - aa[:, None] * x["lfy"][:, t]
        o += aa[:, None] * float(x["t"][t].sum()) * ay
        o[~x["ka"]] = 0.0
        out[t] = o.T
    return out.reshape(-1)


class _BedParams(C.Structure):
    _fields_ = [(n, C.c_double) for n in ("snp_mss", "snp_maf", "snp_I_opt", "pat_mss")]


class _BedResult(C.Structure):
    _fields_ = [("n_snp", C.c_int), ("n_fam", C.c_int), ("n_snp_retain", C.c_int), ("n_pat_retain", C.c_int),
                ("n_allele", C.c_int), ("row_bytes", C.c_longlong)] + [(n, C.POINTER(C.c_int)) for n in (
                    "snp", "pat", "order")] + [(n, C.POINTER(C.c_double)) for n in ("freq", "maf", "mss", "I")] + [
                        ("A_n", C.POINTER(C.c_ubyte))]


def _prepare_bed(c, seed):
    """Hardy-Weinberg genotypes with 0.2 % missing calls.  Of the SNPs, an
    eighth are rare (MAF U[0.005, 0.02]) and a sixteenth miss 3 % of their
    calls; a 64th of the patients miss a tenth of theirs: the filters drop
    these and keep the others (MAF U[0.08, 0.5])."""
    g = _gen(seed, 8)
    n, m = c["snps"], c["patients"]
    nb = (m + 3) // 4
    rec = np.empty((n, nb), np.uint8)
    w = torch.tensor([1, 4, 16, 64], dtype=torch.uint8, device=DEV)
    bad = 0.1 * (torch.arange(4 * nb, device=DEV) % 64 == 17)
    for r in range(0, n, 16384):
        k = min(16384, n - r)
        snp = torch.arange(r, r + k, device=DEV)[:, None]
        q = torch.where(snp % 8 == 3, 0.005 + 0.015 * _rand(g, k, 1), 0.08 + 0.42 * _rand(g, k, 1))
        miss = torch.where(snp % 16 == 9, 0.03, 0.002) + bad
        u = _rand(g, k, 4 * nb)
        v = torch.where(u < q * q, 0, torch.where(u < q * q + 2 * q * (1 - q), 2, 3)).to(torch.uint8)
        v = torch.where(_rand(g, k, 4 * nb) < miss, 1, v).to(torch.uint8)
        v[:, m:] = 0
        rec[r:r + k] = (v.reshape(k, nb, 4) * w).sum(2, dtype=torch.uint8).cpu().numpy()
    lib = load()
    lib.lakgb_bed_to_b16_mem.argtypes = [C.c_void_p, C.c_int, C.c_int, C.POINTER(_BedParams), C.POINTER(_BedResult)]
    lib.lakgb_bed_to_b16_mem.restype = C.c_int
    lib.lakgb_bed_result_free.argtypes = [C.POINTER(_BedResult)]
    return dict(lib=lib, rec=rec, n=n, m=m, prm=_BedParams(0.01, 0.05, 0.01, 0.04))


def _run_bed(s):
    r = _BedResult()
    if s["lib"].lakgb_bed_to_b16_mem(s["rec"].ctypes.data, s["n"], s["m"], C.byref(s["prm"]), C.byref(r)) != 0:
        raise RuntimeError("lakgb_bed_to_b16_mem failed")
    arr = lambda p, n: np.ctypeslib.as_array(p, (n,)).copy() if n else np.zeros(0)  # noqa: E731
    try:
        return dict(A_n=arr(r.A_n, r.n_allele * r.row_bytes), snp=arr(r.snp, r.n_snp_retain), pat=arr(r.pat, r.n_pat_retain),
                    order=arr(r.order, r.n_allele), freq=arr(r.freq, r.n_allele), maf=arr(r.maf, r.n_allele))
    finally:
        s["lib"].lakgb_bed_result_free(C.byref(r))


# ---------------------------------------------------------------------------


def _prepare_solve(c, seed):
    return _solve_problem(c["cases"], c["controls"], c["cols"], c["bins"], c["covariates"], c["b_mlt"], c["gamma"],
                          c["qc"], c["maf_lo"], c["maf_hi"], seed)


def _solve_work(rows_a, rows_z, cols, b_mlt, covariates):
    pairs = rows_a * (rows_a + rows_z)
    return {"bytes": (rows_a + rows_z) * cols / 8.0 + 8.0 * pairs,
            "flops": 2.0 * pairs * cols * (1 + b_mlt * covariates)}


_PREPARE = {"solve": _prepare_solve, "null_batch": _prepare_null_batch, "gram_pass": _prepare_gram_pass,
            "gram_update": _prepare_gram_update, "gram_host": _prepare_gram_host, "row_terms": _prepare_row_terms,
            "quantise": _prepare_quantise, "loop_product": _prepare_loop, "snp_product": _prepare_snp, "bed": _prepare_bed}
_RUN = {"solve": _run_solve, "null_batch": _run_null_batch, "gram_pass": _run_gram_device,
        "gram_update": _run_gram_device, "gram_host": _run_gram_host, "row_terms": _run_row_terms,
        "quantise": _run_quantise, "loop_product": _run_loop, "snp_product": _run_snp, "bed": _run_bed}
_EXACT = {"gram_pass": _exact_gram_pass, "gram_update": _exact_gram_update, "gram_host": _exact_gram_host,
          "row_terms": _exact_row_terms, "quantise": _exact_quantise, "loop_product": _exact_loop,
          "snp_product": _exact_snp}


def prepare(case, seed):
    return case["op"], _PREPARE[case["op"]](case, seed)


def run(state):
    op, s = state
    return _RUN[op](s)


def exact(case, seed):
    f = _EXACT.get(case["op"])
    return f(case, seed) if f else None


def work(case):
    c, op = case, case["op"]
    if op == "solve":
        return _solve_work(c["cases"], c["controls"], c["cols"], c["b_mlt"], c["covariates"])
    if op == "null_batch":
        each = [_solve_work(r // 2, r - r // 2, m, 32, 1) for r, m in _null_sizes(c)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if op == "gram_pass":
        return _work_gram_pass(c)
    if op in ("gram_update", "gram_host"):
        pairs = float(c["rows_a"]) * c["rows_z"]
        return {"bytes": (c["rows_a"] + c["rows_z"]) * abi.bsize(c["cols"]) + 8.0 * pairs, "flops": 2.0 * pairs * c["cols"]}
    if op == "row_terms":
        return {"bytes": c["rows"] * (abi.bsize(c["cols"]) + 8.0 * abi.AJDK_TOT),
                "flops": 2.0 * c["rows"] * (c["cols"] + abi.AJDK_TOT * abi.psize(c["cols"]))}
    if op == "quantise":
        return {"bytes": 8.0 * c["rows"] * c["cols"] + (c["b_mlt"] + 1.0) * c["cols"] * abi.bsize(c["rows"]),
                "flops": 4.0 * c["rows"] * c["cols"]}
    if op == "loop_product":
        planes = c["rows_w"] * (c["b_mlt"] + 1.0)
        return {"bytes": c["snps"] * (abi.bsize(c["rows_y"]) + abi.bsize(c["rows_w"])) + planes * abi.bsize(c["rows_y"])
                + 8.0 * c["snps"] * c["covariates"], "flops": 2.0 * c["snps"] * planes * c["rows_y"] * c["covariates"]}
    if op == "snp_product":
        pairs = float(c["snps"]) * c["snps_y"] * c["covariates"]
        return {"bytes": (c["snps"] + c["snps_y"]) * abi.bsize(c["rows"]) + 8.0 * pairs, "flops": 2.0 * pairs * c["rows"]}
    return {"bytes": c["snps"] * c["patients"] * (0.25 + 3.0 / 8.0), "flops": 3.0 * c["snps"] * c["patients"]}
