"""GPU parity at the benchmark's shapes and on the kernel-selection boundaries: golden
fixtures, the 4096x4096 single-MatVec config, Llama FFN shapes, columns that take the
register-load kernel instead of the TMA-fed one, activations with outliers / zeros / inf,
and size-independent properties (linearity, row-shard reassembly) at full size."""
import os

import numpy as np
import pytest

import oracle as O
from conftest import CASES, case_id, case_ok, make_w, to_product_blob

pytestmark = pytest.mark.gpu
TOL = 1e-3
GOLD = os.path.join(os.path.dirname(__file__), "golden", "golden_small.npz")


def check(y, ob, x, refs=("scalar", "simd")):
    den = O.sum_abs_wx(ob, x)
    for name in refs:
        ref = O.matvec(ob, x) if name == "scalar" else O.matvec_simd(ob, x, 0)
        err = np.abs(y.astype(np.float64) - ref.astype(np.float64))
        assert np.all(err <= TOL * den + 1e-30), f"{name}: worst {np.max(err / np.maximum(den, 1e-30)):.3e}"
    return float(np.max(np.abs(y.astype(np.float64) - O.matvec_simd(ob, x, 0)) / np.maximum(den, 1e-30)))


def test_golden_fixtures_on_device(wv):
    g = np.load(GOLD)
    q = wv.quant
    for rows, cols in ((8, 512), (3, 100)):
        x = g[f"x_{rows}x{cols}"]
        for c in CASES:
            if not case_ok(c, rows, cols):
                continue
            f, bw, dt = c
            k = f"{case_id(c)}_{rows}x{cols}"
            blob = q.Blob(q.Format(O.FMT[f]), rows, cols, g[k + "_raw"], g[k + "_scales"], g[k + "_mins"], bw or 0, dt)
            assert np.array_equal(q.Unpack(blob).view(np.uint32), g[k + "_unpack"].view(np.uint32)), k
            y = np.zeros(rows, np.float32)
            q.MatVec(blob, x, y)
            ob = O.Blob(O.FMT[f], rows, cols, g[k + "_raw"], g[k + "_scales"], g[k + "_mins"], blob.BlockWeights if f != "none" else 1, dt)
            if f == "BinaryPacked":
                ob.block_weights = 128 if bw == 128 else 32
            den = O.sum_abs_wx(ob, x)
            assert np.all(np.abs(y.astype(np.float64) - g[k + "_y_scalar"]) <= TOL * den + 1e-30), k


@pytest.mark.parametrize("case", CASES, ids=case_id)
def test_single_matvec_4096x4096(wv, case):
    """The single Dense MatVec config (4096x4096, W ~ N(0,0.02^2) seed 0, x ~ N(0,1) seed 1) for every layout."""
    f, bw, dt = case
    rows = cols = 4096
    w = np.random.default_rng(0).normal(0, 0.02, (rows, cols)).astype(np.float32)
    x = np.random.default_rng(1).normal(0, 1, cols).astype(np.float32)
    q = wv.quant
    blob = q.Pack(q.Format(O.FMT[f]), w, rows, cols, bw, dt)          # device packer
    ob = O.Blob(O.FMT[f], rows, cols, blob.Raw, blob.Scales, blob.Mins, blob.BlockWeights, dt)
    assert np.array_equal(q.Unpack(blob).view(np.uint32), O.unpack(ob).view(np.uint32))
    y = np.zeros(rows, np.float32)
    wv.dense.MatVecPackedBlob(blob, x, y)
    check(y, ob, x)


@pytest.mark.parametrize("fmt", ["Q4_K", "Q8_0", "Q4_0", "IQ2_XS", "IQ4_NL", "BinaryPacked"])
@pytest.mark.parametrize("shape", [(4096, 14336), (14336, 4096)], ids=["4096x14336", "14336x4096"])
def test_ffn_shapes_full_size(wv, fmt, shape):
    rows, cols = shape
    bw = 128 if fmt == "BinaryPacked" else 0
    w = np.random.default_rng(2).normal(0, 0.02, rows * cols).astype(np.float32)
    x = np.random.default_rng(22).normal(0, 1, cols).astype(np.float32)
    q = wv.quant
    blob = q.Pack(q.Format(O.FMT[fmt]), w, rows, cols, bw)
    ob = O.Blob(O.FMT[fmt], rows, cols, blob.Raw, blob.Scales, blob.Mins, blob.BlockWeights)
    assert np.array_equal(blob.Raw, O.pack(fmt, w, rows, cols, bw).raw), "device packer differs from the reference packer at full size"
    y = np.zeros(rows, np.float32)
    q.MatVec(blob, x, y)
    check(y, ob, x, refs=("simd",))
    # linearity: W(2x + x2) == 2 Wx + W x2 within tolerance (no oracle involved)
    x2 = np.random.default_rng(23).normal(0, 1, cols).astype(np.float32)
    y2, y3 = np.zeros(rows, np.float32), np.zeros(rows, np.float32)
    q.MatVec(blob, x2, y2)
    q.MatVec(blob, (2 * x + x2).astype(np.float32), y3)
    den = O.sum_abs_wx(ob, np.abs(2 * x) + np.abs(x2))
    assert np.all(np.abs(y3.astype(np.float64) - (2.0 * y + y2)) <= 3 * TOL * den)


_FULL = ("Q4_K", "Q8_0", "Q4_0", "IQ2_XS", "IQ4_NL", "BinaryPacked")   # covered by test_ffn_shapes_full_size (packer equality, linearity)
_REST = [c for c in CASES if not (c[0] in _FULL and (c[0] != "BinaryPacked" or c[1] == 128))]


def _device_packed(wv, f, bw, dt, w, rows, cols):
    """Blob packed by the device packer (byte-identical to the reference packer: test_pack_unpack_matvec and
    test_ffn_shapes_full_size) and the oracle's view of the same bytes."""
    q = wv.quant
    blob = q.Pack(q.Format(O.FMT[f]), w, rows, cols, bw, dt)
    ob = O.Blob(O.FMT[f], rows, cols, blob.Raw, blob.Scales, blob.Mins, blob.BlockWeights if f != "none" else 1, dt)
    return blob, ob


@pytest.mark.parametrize("case", _REST, ids=case_id)
@pytest.mark.parametrize("shape", [(4096, 14336), (14336, 4096)], ids=["4096x14336", "14336x4096"])
def test_ffn_shapes_every_layout(wv, case, shape):
    """The benchmark's two shapes for every layout the benchmark times there (the six formats of
    test_ffn_shapes_full_size apart): outputs against the SIMD-path oracle on the benchmark's own inputs."""
    f, bw, dt = case
    rows, cols = shape
    w = np.random.default_rng(2).normal(0, 0.02, rows * cols).astype(np.float32)
    x = np.random.default_rng(1).normal(0, 1, cols).astype(np.float32)
    blob, ob = _device_packed(wv, f, 64 if f == "AffinePacked" else bw, dt, w, rows, cols)
    y = np.zeros(rows, np.float32)
    wv.quant.MatVec(blob, x, y)
    check(y, ob, x, refs=("simd",))


@pytest.mark.parametrize("fmt", ["Q4_K", "Q8_0"])
@pytest.mark.parametrize("shape", [(8192, 8192), (1024, 8192), (28672, 8192), (8192, 28672)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_70b_block_shapes_full_size(wv, fmt, shape):
    """The projection shapes of the 70B decoder block (Q/O 8192x8192, K/V 1024x8192, gate/up 28672x8192,
    down 8192x28672) at full size, weights seed 5."""
    rows, cols = shape
    w = np.random.default_rng(5).normal(0, 0.02, rows * cols).astype(np.float32)
    x = np.random.default_rng(6).normal(0, 1, cols).astype(np.float32)
    blob, ob = _device_packed(wv, fmt, 0, 1, w, rows, cols)
    y = np.zeros(rows, np.float32)
    wv.quant.MatVec(blob, x, y)
    check(y, ob, x, refs=("simd",))


@pytest.mark.parametrize("cols", [8192, 1056, 4608, 17408, 28672])
@pytest.mark.parametrize("fmt", ["Q4_K", "Q5_1", "IQ3_S", "Q8_0"])
def test_kernel_selection_boundaries(wv, fmt, cols):
    """8192 and 4608: TMA-fed kernel with partial column warps; 1056 (cols % 512 != 0), 17408 and
    28672 (more than 16 column warps): register-load kernel with the activation scratch."""
    rows = 97
    w, x = make_w(cols, rows, cols)
    ob = O.pack(fmt, w, rows, cols)
    blob = to_product_blob(wv, ob)
    y = np.zeros(rows, np.float32)
    wv.quant.MatVec(blob, x, y)
    check(y, ob, x)


@pytest.mark.parametrize("fmt", ["Q4_0", "Q4_K", "Q6_K", "IQ1_S", "TernaryPacked", "AffinePacked"])
def test_activation_edge_cases(wv, fmt):
    rows, cols = 64, 4096
    w, x = make_w(31, rows, cols)
    ob = O.pack(fmt, w, rows, cols, 64 if fmt == "AffinePacked" else 0)
    blob = to_product_blob(wv, ob)
    y = np.zeros(rows, np.float32)
    # outliers 1e4 times the typical magnitude, tiny values, an all-zero block, signed zeros
    xo = x.copy()
    xo[[5, 700, 2049]] = [3.0e4, -1.0e4, 2.5e4]
    xo[64:96] = 0.0
    xo[128:160] *= 1e-30
    xo[200] = -0.0
    wv.quant.MatVec(blob, xo, y)
    check(y, ob, xo)
    # zero input gives exactly zero
    wv.quant.MatVec(blob, np.zeros(cols, np.float32), y)
    assert np.all(y == 0)
    # inf / NaN in x poison the outputs (the reference's f32 arithmetic does too) and do not hang
    xn = x.copy()
    xn[10] = np.inf
    wv.quant.MatVec(blob, xn, y)
    assert not np.all(np.isfinite(y))
    from welvet_b200 import _lib
    assert _lib.lib().wv_device_status() == 0


def test_lm_head_slice_row_shard(wv):
    """One rank's 1/8 shard of a 128256x8192 head (16032 rows), Q8_0 and Q4_K: the shard GEMV equals
    the oracle on the same rows."""
    import ctypes as C
    from welvet_b200 import _lib
    L = _lib.lib()
    rows_full, cols, world, rank = 128256, 8192, 8, 3
    lo, hi = C.c_int(), C.c_int()
    _lib.check(L.wv_shard_range(rows_full, rank, world, C.byref(lo), C.byref(hi)))
    n = hi.value - lo.value
    assert n == 16032
    w = np.random.default_rng(5).normal(0, 0.02, n * cols).astype(np.float32)
    x = np.random.default_rng(6).normal(0, 1, cols).astype(np.float32)
    for fmt in ("Q8_0", "Q4_K"):
        blob = wv.quant.Pack(wv.quant.Format(O.FMT[fmt]), w, n, cols)
        ob = O.Blob(O.FMT[fmt], n, cols, blob.Raw, blob.Scales, blob.Mins, blob.BlockWeights)
        y = np.zeros(n, np.float32)
        wv.quant.MatVec(blob, x, y)
        check(y, ob, x, refs=("simd",))


def test_concurrent_host_callers(wv):
    """Callers may be concurrent threads (the reference's goroutines): the synchronous entry serialises
    on its staging buffers and every caller gets its own result."""
    import threading
    rows, cols = 512, 2048
    q = wv.quant
    jobs = []
    for i, f in enumerate(["Q4_K", "Q8_0", "Q4_0", "IQ2_XS"]):
        w, x = make_w(70 + i, rows, cols)
        ob = O.pack(f, w, rows, cols)
        jobs.append((to_product_blob(wv, ob), ob, x))
    for b, _, x in jobs:                       # warm: uploads happen once
        q.MatVec(b, x, np.zeros(rows, np.float32))
    want = [(lambda y: (q.MatVec(b, x, y), y)[1])(np.zeros(rows, np.float32)) for b, _, x in jobs]
    out = [[None] * 20 for _ in jobs]
    errs = []

    def worker(j):
        try:
            b, _, x = jobs[j]
            for k in range(20):
                y = np.zeros(rows, np.float32)
                q.MatVec(b, x, y)
                out[j][k] = y
        except Exception as e:  # noqa: BLE001
            errs.append(e)
    ts = [threading.Thread(target=worker, args=(j,)) for j in range(len(jobs))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errs, errs
    for j in range(len(jobs)):
        for k in range(20):
            assert np.array_equal(out[j][k].view(np.uint32), want[j].view(np.uint32))


@pytest.mark.parametrize("dt,rows,cols,batch", [(1, 1, 1024, 1), (1, 149, 1032, 1), (1, 296, 5000, 1), (1, 700, 8192, 2), (1, 2400, 1024, 1), (1, 33, 8200, 1), (1, 9, 1016, 1),
                                                (2, 7, 2048, 1), (2, 148, 2056, 3), (2, 2368, 4104, 1), (2, 2369, 2048, 1), (2, 1500, 2048, 2), (3, 301, 8192, 1), (3, 60, 5000, 5)])
def test_plain_rows_at_the_limits_of_the_ring_kernel(wv, dt, rows, cols, batch):
    """FormatNone rows at the edges of the ring kernel's range (row bytes, columns, slices that do not divide the row, rows of W above
    and below its limit, several rows of x, x that is not 16-byte aligned) against float64: float32 products and sums, so at most
    cols + 8 roundings of 2^-24 of sum |w x|, of which random signs leave a fraction; the bound is 64 of them."""
    import torch
    from welvet_b200 import _lib
    L, key = _lib.lib(), 0x7000 + rows * 16 + dt
    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    w = torch.randn(rows * cols, device="cuda", generator=gen) * 0.02
    torch.cuda.synchronize()
    _lib.check(L.wv_pack_upload_dev(key, 0, dt, 0, w.data_ptr(), rows, cols, None))
    d = torch.zeros(rows, cols, device="cuda")
    _lib.check(L.wv_unpack_dev(key, d.data_ptr(), None))
    buf = torch.randn(batch * cols + 1, device="cuda", generator=gen)
    torch.cuda.synchronize()
    try:
        for off in (0, 1):
            x = buf[off : off + batch * cols]
            y = torch.full((batch, rows), float("nan"), device="cuda")
            torch.cuda.synchronize()
            _lib.check(L.wv_matvec_dev(key, x.data_ptr(), y.data_ptr(), batch, cols, rows, None))
            torch.cuda.synchronize()
            xd = x.reshape(batch, cols).double()
            err = (y.double() - xd @ d.double().T).abs()
            assert bool((err <= 64 * 2.0 ** -24 * (xd.abs() @ d.double().abs().T)).all())
        assert L.wv_device_status() == 0
    finally:
        L.wv_blob_evict(key)


@pytest.mark.parametrize("dt,rows,cols", [(1, 4096, 4096), (1, 2500, 5000), (1, 2500, 3000), (1, 2400, 8192), (2, 2400, 2056), (2, 4096, 4096), (3, 3001, 8192)])
def test_plain_rows_do_not_depend_on_the_launch(wv, dt, rows, cols):
    """FormatNone: a row's bits are the same in the whole matrix, in a shard of its rows and with any number of rows of x, on either
    side of the line between the two kernels (2368 rows, counted once for every row of x)."""
    import torch
    from welvet_b200 import _lib
    L, check = _lib.lib(), _lib.check
    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    w = torch.randn(rows, cols, device="cuda", generator=gen) * 0.02
    x = torch.randn(3, cols, device="cuda", generator=gen)
    cuts = [0, 7, rows // 3, rows // 3 + 1200, rows]
    keys = [0x7100 + i for i in range(len(cuts))]
    torch.cuda.synchronize()

    def call(key, n, batch):
        y = torch.full((batch, n), float("nan"), device="cuda")
        torch.cuda.synchronize()
        check(L.wv_matvec_dev(key, x.data_ptr(), y.data_ptr(), batch, cols, n, None))
        torch.cuda.synchronize()
        return y
    try:
        check(L.wv_pack_upload_dev(keys[-1], 0, dt, 0, w.data_ptr(), rows, cols, None))
        for key, a, b in zip(keys, cuts, cuts[1:]):
            check(L.wv_pack_upload_dev(key, 0, dt, 0, w[a].data_ptr(), b - a, cols, None))
        whole = call(keys[-1], rows, 3)
        assert torch.equal(call(keys[-1], rows, 1), whole[:1])
        for batch in (1, 2, 3):
            parts = [call(key, b - a, batch) for key, a, b in zip(keys, cuts, cuts[1:])]
            assert torch.equal(torch.cat(parts, 1), whole[:batch])
        assert L.wv_device_status() == 0
    finally:
        for key in keys:
            L.wv_blob_evict(key)


@pytest.mark.parametrize("dt,rows,cols,row", [(1, 2000, 4096, 1), (1, 2000, 4096, 3), (1, 2000, 6144, 5), (2, 1000, 8192, 2), (2, 40, 2048, 1)])
def test_plain_rows_after_a_wait_that_runs_out(wv, hooks, dt, rows, cols, row):
    """The ring kernel of FormatNone with a copy that never comes: the call is reported, the rows that were not summed are NaN and
    the others have their bits; the next call is sound."""
    import torch
    from welvet_b200 import _lib
    L, check, key = _lib.lib(), _lib.check, 0x7200
    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    w, x = torch.randn(rows, cols, device="cuda", generator=gen) * 0.02, torch.randn(cols, device="cuda", generator=gen)
    torch.cuda.synchronize()
    check(L.wv_pack_upload_dev(key, 0, dt, 0, w.data_ptr(), rows, cols, None))

    def call():
        y = torch.zeros(rows, device="cuda")
        torch.cuda.synchronize()
        check(L.wv_matvec_dev(key, x.data_ptr(), y.data_ptr(), 1, cols, rows, None))
        torch.cuda.synchronize()
        return y, L.wv_device_status()
    try:
        want, status = call()
        assert status == 0
        hooks.wv_set_ring_stall(row, 2000)
        try:
            y, status = call()
        finally:
            hooks.wv_set_ring_stall(0, 0)
        assert status == _lib.WV_ETIMEOUT
        assert bool(y.isnan().any()) and (bool((~y.isnan()).any()) or row == 1) and bool((y.isnan() | (y == want)).all())
        y, status = call()
        assert status == 0 and torch.equal(y, want)
    finally:
        L.wv_blob_evict(key)


@pytest.mark.parametrize("fmt,cols", [("Q5_K", 16384), ("Q5_K", 16128), ("Q6_K", 15872), ("Q6_K", 30720), ("Q5_1", 15104), ("Q8_0", 12672)])
def test_widths_where_the_staged_x_has_no_padding(wv, fmt, cols):
    """The one-row kernel at the widths where only an unpadded copy of x leaves three stages (and next to them), alone, with a residual
    and with the RMSNorm in its prologue, aligned and unaligned, against float64 over the dequantised weights: an activation is off
    by at most 1 / 65024 of its chunk's largest, to which come 2^-20 of sum |w x| for the float32 steps."""
    import ctypes as C

    import torch
    from welvet_b200 import _lib
    from welvet_b200.decode import MatVecFusedCUDA, RMSNormCUDA
    L, check, key, rows = _lib.lib(), _lib.check, 0x7300, 1400
    gen = torch.Generator(device="cuda").manual_seed(cols)
    w = torch.randn(rows * cols, device="cuda", generator=gen) * 0.02
    torch.cuda.synchronize()
    check(L.wv_pack_upload_dev(key, O.FMT[fmt], 1, 0, w.data_ptr(), rows, cols, None))
    try:
        d = torch.zeros(rows, cols, device="cuda")
        check(L.wv_unpack_dev(key, d.data_ptr(), None))
        buf = torch.randn(cols + 1, device="cuda", generator=gen)
        gamma = 1 + 0.1 * torch.randn(cols, device="cuda", generator=gen)
        res = torch.randn(rows, device="cuda", generator=gen)
        torch.cuda.synchronize()
        d = d.double()

        def close(y, x, plus=0.0):
            x = x.double()
            step = x.abs().view(-1, 32).amax(1).repeat_interleave(32) / 65024
            return bool(((y.double() - plus - d @ x).abs() <= d.abs() @ (1.01 * step + 2.0 ** -20 * x.abs()) + 1e-6).all())
        for off in (0, 1):
            x = buf[off:off + cols]
            y, z, n, xn = (torch.full((k,), float("nan"), device="cuda") for k in (rows, rows, rows, cols))
            torch.cuda.synchronize()
            check(L.wv_matvec_dev(key, x.data_ptr(), y.data_ptr(), 1, cols, rows, None))
            check(L.wv_matvec_dev_add(key, x.data_ptr(), res.data_ptr(), z.data_ptr(), cols, rows, None))
            RMSNormCUDA(x.data_ptr(), gamma.data_ptr(), xn.data_ptr(), 1, cols, 1e-5)
            if cols <= 16384:      # the norm needs the whole row of x at once
                MatVecFusedCUDA((C.c_uint64 * 1)(key), x.data_ptr(), (C.c_void_p * 1)(n.data_ptr()), cols, (C.c_int * 1)(rows), dnorm_gamma=gamma.data_ptr(), norm_eps=1e-5)
            torch.cuda.synchronize()
            assert close(y, x) and close(z, x, res.double())
            assert cols > 16384 or close(n, xn)
        assert L.wv_device_status() == 0
    finally:
        L.wv_blob_evict(key)
