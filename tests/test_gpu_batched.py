"""Batched Dense MatVec (several activation rows against one packed matrix) on the tcgen05 kernel: every packed
format, batches around the padding and tiling edges, rows that do not fill the last 128-row tile, against the oracle's
SIMD-path GEMV per activation row within 1e-3 * sum |w x|, and the small-batch GEMM configuration at full size."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle as O
from conftest import CASES, case_id, case_ok, to_product_blob

pytestmark = pytest.mark.gpu
TOL = 1e-3


def _run(wv, ob, x):
    """x: [batch, cols] -> y [batch, rows] through wv_matvec_dev with device buffers."""
    L = wv._lib.lib()
    blob = to_product_blob(wv, ob)
    key = wv.quant.EnsureResident(blob)
    dx = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    dy = torch.full((x.shape[0], ob.rows), float("nan"), device="cuda")
    wv._lib.check(L.wv_matvec_dev(key, dx.data_ptr(), dy.data_ptr(), x.shape[0], ob.cols, ob.rows, None))
    torch.cuda.synchronize()
    assert L.wv_device_status() == 0
    return dy.cpu().numpy(), blob


def _check(ob, x, y, rows_checked=None):
    cache = O.SimdCache(ob)
    worst = 0.0
    for m in (range(x.shape[0]) if rows_checked is None else rows_checked):
        ref = np.zeros(ob.rows, np.float32)
        cache.matvec(np.ascontiguousarray(x[m]), ref, 0)
        den = O.sum_abs_wx(ob, x[m])
        err = np.abs(y[m].astype(np.float64) - ref)
        assert np.all(err <= TOL * den + 1e-30), (m, float(np.max(err / np.maximum(den, 1e-30))))
        worst = max(worst, float(np.max(err / np.maximum(den, 1e-30))))
    return worst


@pytest.mark.parametrize("case", [c for c in CASES if c[0] != "none"], ids=case_id)
@pytest.mark.parametrize("batch", [2, 16, 17, 100])
def test_batched_every_format(wv, case, batch):
    f, bw, dt = case
    rows, cols = 300, 1024            # three row tiles, the last one 44 rows; four column splits
    w = np.random.default_rng(21).normal(0, 0.02, rows * cols).astype(np.float32)
    ob = O.pack(f, w, rows, cols, bw, dt)
    x = np.random.default_rng(22).normal(0, 1, (batch, cols)).astype(np.float32)
    x[0, ::5] *= 50.0                 # a row with outliers, and one scaled far down
    x[-1] *= 1e-20
    y, _ = _run(wv, ob, x)
    assert np.all(np.isfinite(y))
    _check(ob, x, y)


@pytest.mark.parametrize("fmt", ["Q8_0", "Q4_K"])
@pytest.mark.parametrize("batch", [1, 4, 16, 64, 256, 300])
def test_small_batch_gemm_configuration(wv, fmt, batch):
    """M activation rows x 4096 against W 4096 x 4096 in Q8_0 and in the 4-bit k-quant, N(0, 0.02^2) seed 3."""
    rows = cols = 4096
    rng = np.random.default_rng(3)
    w = rng.normal(0, 0.02, rows * cols).astype(np.float32)
    x = rng.normal(0, 1, (batch, cols)).astype(np.float32)
    ob = O.pack(fmt, w, rows, cols)
    y, blob = _run(wv, ob, x)
    picks = sorted({0, batch // 2, batch - 1})
    worst = _check(ob, x, y, picks)
    assert worst < TOL
    if batch > 1:
        # every row agrees with the batch-1 kernel's result for that row within the two kernels' error budgets
        L = wv._lib.lib()
        key = wv.quant.EnsureResident(blob)
        dx = torch.from_numpy(x).cuda()
        one = torch.zeros(rows, device="cuda")
        for m in picks:
            wv._lib.check(L.wv_matvec_dev(key, dx.data_ptr() + 4 * m * cols, one.data_ptr(), 1, cols, rows, None))
            torch.cuda.synchronize()
            den = O.sum_abs_wx(ob, x[m])
            assert np.all(np.abs(y[m].astype(np.float64) - one.cpu().numpy()) <= 2 * TOL * den + 1e-30)


def test_batched_wide_and_tall_shapes(wv):
    for rows, cols, batch in ((14336, 4096, 8), (4096, 14336, 33), (128, 32768, 5), (1000, 256, 256)):
        w = np.random.default_rng(rows).normal(0, 0.02, rows * cols).astype(np.float32)
        ob = O.pack("Q4_K", w, rows, cols)
        x = np.random.default_rng(cols).normal(0, 1, (batch, cols)).astype(np.float32)
        y, _ = _run(wv, ob, x)
        _check(ob, x, y, [0, batch - 1])


def test_dense_forward_batched(wv):
    """dense.Forward with a batch: bias and activation after the batched GEMV, as for batch 1."""
    d = wv.dense
    rows, cols, batch = 512, 2048, 24
    w = np.random.default_rng(5).normal(0, 0.02, rows * cols).astype(np.float32)
    layer = d.NewConfigured(cols, rows, d.ActivationSilu, wv.quant.DTypeFloat32, wv.quant.Format.FormatQ4_K, w)
    st = layer.Weights
    st.Bias = np.random.default_rng(6).normal(0, 0.1, rows)
    x = np.random.default_rng(7).normal(0, 1, (batch, cols)).astype(np.float32)
    pre, post = d.Forward(layer, x)
    ob = O.Blob(O.FMT["Q4_K"], rows, cols, st.Packed.Raw, st.Packed.Scales, st.Packed.Mins, st.Packed.BlockWeights)
    for m in (0, batch - 1):
        ref = O.matvec_simd(ob, x[m]).astype(np.float64) + st.Bias
        den = O.sum_abs_wx(ob, x[m])
        assert np.all(np.abs(pre[m] - ref) <= TOL * den + 1e-6)
        pm = pre[m].astype(np.float64)
        assert np.allclose(post[m], pm / (1 + np.exp(-pm)), rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("rows,cols,batch,nbias", [(333, 512, 1, 333), (512, 1024, 8, 600), (130, 254, 5, 7), (257, 512, 3, 0)])
def test_dense_forward_bias_and_activations(wv, rows, cols, batch, nbias):
    """Bias and activation behind the GEMV against the float64 passes of dense.Activate: biases shorter and longer than a row, every
    activation. The sum is the same bits; the activation may round to the neighbouring float32 (float64 functions of a few
    units in the last place each; 1 + tanh(v) loses its leading digits for negative v, hence the term in |v|)."""
    d = wv.dense
    rng = np.random.default_rng(rows)
    layer = d.NewConfigured(cols, rows, d.ActivationLinear, wv.quant.DTypeFloat32, wv.quant.Format.FormatQ5_0, rng.normal(0, 0.1, rows * cols).astype(np.float32))
    x = rng.normal(0, 1, (batch, cols)).astype(np.float32)
    y = d.Forward(layer, x)[0].astype(np.float64)
    if nbias:
        layer.Weights.Bias = rng.normal(0, 1, nbias)
        y[:, :nbias] += layer.Weights.Bias[:rows]
    for act in d._ACTIVATIONS:
        layer.Activation = act
        pre, post = d.Forward(layer, x)
        assert pre.dtype == post.dtype == np.float32 and (pre is post) == (act == d.ActivationLinear and not nbias)
        np.testing.assert_array_equal(pre, y.astype(np.float32))
        p = pre.astype(np.float64)
        ref = d.Activate(p, act)
        assert np.all(np.abs(post - ref) <= 2.0 ** -23 * np.abs(ref) + 2.0 ** -49 * np.abs(p) + 1e-45), act


@pytest.mark.parametrize("as_type", [float, np.float32, np.int64, int])
def test_dense_forward_activation_value_types(wv, as_type):
    """An activation equal to one of the eight values is that activation, whatever numeric type a program read it into."""
    d = wv.dense
    rng = np.random.default_rng(3)
    layer = d.NewConfigured(64, 24, d.ActivationLinear, wv.quant.DTypeFloat32, wv.quant.Format.FormatQ8_0, rng.normal(0, 1, 24 * 64).astype(np.float32))
    x = rng.standard_normal((3, 64), np.float32)
    y = d.Forward(layer, x)[0]
    layer.Activation = as_type(d.ActivationReLU2)
    pre, post = d.Forward(layer, x)
    np.testing.assert_array_equal(pre, y)
    np.testing.assert_array_equal(post, np.where(y < 0, 0, y.astype(np.float64) ** 2).astype(np.float32))


@pytest.mark.parametrize("rows,cols,batch", [(32, 32, 65537), (160, 64, 27000)])
def test_dense_forward_bias_and_activation_of_large_batches(wv, rows, cols, batch):
    """More rows than a grid has in y, and more results than the pinned buffer takes at a time (4 Mi floats): every row is the plain
    product's row with the bias added in float64 and rounded, and its ReLU (both exact)."""
    d = wv.dense
    rng = np.random.default_rng(batch)
    layer = d.NewConfigured(cols, rows, d.ActivationLinear, wv.quant.DTypeFloat32, wv.quant.Format.FormatQ8_0, rng.normal(0, 0.1, rows * cols).astype(np.float32))
    x = rng.standard_normal((batch, cols), np.float32)
    y = d.Forward(layer, x)[0]
    layer.Weights.Bias, layer.Activation = rng.normal(0, 1, rows), d.ActivationReLU
    pre, post = d.Forward(layer, x)
    np.testing.assert_array_equal(pre, (y + layer.Weights.Bias).astype(np.float32))
    np.testing.assert_array_equal(post, np.maximum(pre, 0))


def test_calls_that_fail_between_two_launches(wv):
    """Rows wider than FormatNone takes: x is on its way to the device when the GEMV's launch is refused. Both host calls report it
    and the staging slot serves the next call."""
    d, none = wv.dense, wv.quant.Format.FormatNone
    rng = np.random.default_rng(11)
    wide = d.NewConfigured(32768, 4, d.ActivationLinear, wv.quant.DTypeFloat32, none, rng.normal(0, 1, 4 * 32768).astype(np.float32))
    layer = d.NewConfigured(64, 24, d.ActivationLinear, wv.quant.DTypeFloat32, none, rng.normal(0, 1, 24 * 64).astype(np.float32))
    x = rng.standard_normal((40, 64), np.float32)
    want = d.Forward(layer, x)[0]
    for act in (d.ActivationLinear, d.ActivationReLU):
        wide.Activation = layer.Activation = act
        for batch in (1, 40):
            with pytest.raises(wv._lib.WelvetError) as e:
                d.Forward(wide, np.ones((batch, 32768), np.float32))
            assert e.value.code == wv._lib.WV_ESHAPE
            pre, post = d.Forward(layer, x)
            np.testing.assert_array_equal(pre, want)
            np.testing.assert_array_equal(post, want if act == d.ActivationLinear else np.maximum(want, 0))


def test_host_pointer_calls_from_threads(wv):
    """wv_matvec (host pointers in and out) from six threads at once, as goroutines call Dense in the reference: the
    staging slots keep the calls apart, every result equals the single-threaded one bit for bit."""
    import threading
    q = wv.quant
    rng = np.random.default_rng(31)
    jobs = []
    for i, (fmt, rows, cols) in enumerate((("Q4_K", 512, 4096), ("Q8_0", 300, 2048), ("IQ3_S", 1000, 1024), ("Q4_0", 96, 14336),
                                           ("Q6_K", 700, 2048), ("BinaryPacked", 256, 4096))):
        w = rng.normal(0, 0.02, rows * cols).astype(np.float32)
        blob = q.Pack(q.Format["Format" + fmt], w, rows, cols)
        x = rng.normal(0, 1, cols).astype(np.float32)
        want = np.zeros(rows, np.float32)
        q.MatVec(blob, x, want)
        jobs.append((blob, x, want))
    errors = []

    def worker(job):
        blob, x, want = job
        try:
            for _ in range(50):
                y = np.full(blob.Rows, np.nan, np.float32)
                q.MatVec(blob, x, y)
                if not np.array_equal(y.view(np.uint32), want.view(np.uint32)):
                    errors.append("mismatch")
                    return
        except Exception as e:   # noqa: BLE001
            errors.append(repr(e))
    threads = [threading.Thread(target=worker, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]
    assert wv._lib.lib().wv_device_status() == 0


@pytest.mark.parametrize("case", [c for c in CASES if c[0] != "none"], ids=case_id)
@pytest.mark.parametrize("shape", [(130, 96), (40, 544), (200, 1056), (140, 1536), (129, 4352)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_batched_column_orders(wv, case, shape):
    """Chunk counts that leave the four producer groups unequal runs, a part of a load unit or nothing at all, rows that do
    not start on a load unit (17 and 33 chunks), and one and two rounds of stages (batches up to 64 and beyond)."""
    rows, cols = shape
    if not case_ok(case, rows, cols):
        pytest.skip("layout needs aligned cols")
    f, bw, dt = case
    w = np.random.default_rng(cols).normal(0, 0.02, rows * cols).astype(np.float32)
    ob = O.pack(f, w, rows, cols, bw, dt)
    wd = O.unpack(ob).reshape(rows, cols).astype(np.float64)
    for batch in (6, 64, 65, 256):
        x = np.random.default_rng(batch).normal(0, 1, (batch, cols)).astype(np.float32)
        y, _ = _run(wv, ob, x)
        # two operands rounded to 11 bits, as derived beside the kernel
        assert np.all(np.abs(y - x.astype(np.float64) @ wd.T) <= 9.9e-4 * (np.abs(x).astype(np.float64) @ np.abs(wd).T) + 1e-30), batch


@pytest.mark.parametrize("fmt", ["Q4_0", "Q4_K", "IQ3_S", "TernaryPacked", "IQ1_S"])
def test_batched_non_finite_parameters(wv, fmt):
    """A row whose scales are infinite or NaN comes out non-finite, as its dequantised weights are; its neighbours do not."""
    rows, cols, batch = 130, 512, 9
    w = np.random.default_rng(1).normal(0, 0.02, rows * cols).astype(np.float32)
    ob = O.pack(fmt, w, rows, cols)
    per_row = (len(ob.scales) if len(ob.scales) else len(ob.raw)) // rows
    for r, bad in ((3, np.inf), (77, np.nan)):
        if len(ob.scales):
            ob.scales[r * per_row] = bad
        else:
            ob.raw[r * per_row:r * per_row + 4] = np.frombuffer(np.float32(bad).tobytes(), np.uint8)     # the first block's scale
    x = np.random.default_rng(2).normal(0, 1, (batch, cols)).astype(np.float32)
    y, _ = _run(wv, ob, x)
    assert not np.any(np.isfinite(y[:, [3, 77]]))
    assert np.all(np.isfinite(np.delete(y, [3, 77], axis=1)))


@pytest.mark.parametrize("fmt,header,mid_code", [("Q6_K", 24, 32), ("Q4_K", 40, 0)])
def test_batched_scale_that_overflows(wv, fmt, header, mid_code):
    """A super-block whose d is finite and whose group scale d * byte is not: the group's weights of code zero are NaN, as
    dequantisation defines them, and so is the row; the rows beside it keep their values."""
    rows, cols, batch = 130, 512, 9
    w = np.random.default_rng(3).normal(0, 0.02, rows * cols).astype(np.float32)
    ob = O.pack(fmt, w, rows, cols)
    bits = {32: 6, 0: 4}[mid_code]
    per_row = len(ob.raw) // rows
    blk = ob.raw[5 * per_row:5 * per_row + header + 32 * bits]
    blk[:4] = np.frombuffer(np.float32(3e38).tobytes(), np.uint8)
    blk[8:24] = 1                                    # every group d / 255 ...
    blk[8] = 255                                     # ... but the first: infinite
    code = np.array([mid_code >> (i % bits) & 1 for i in range(256 * bits)], np.uint8)
    blk[header:] = np.packbits(code, bitorder="little")
    wd = O.unpack(ob).reshape(rows, cols)
    assert np.all(np.isnan(wd[5, :16])) and np.all(np.isfinite(wd[5, 16:]))
    x = np.random.default_rng(4).normal(0, 1, (batch, cols)).astype(np.float32)
    y, _ = _run(wv, ob, x)
    assert np.all(np.isnan(y[:, 5])) and np.all(np.isfinite(np.delete(y, 5, axis=1)))


def _packed(wv, fmt, rows, cols, seed):
    w = np.random.default_rng(seed).normal(0, 0.02, rows * cols).astype(np.float32)
    blob = wv.quant.Pack(wv.quant.Format(O.FMT[fmt]), w, rows, cols)
    return wv.quant.EnsureResident(blob), blob


def test_batched_calls_on_many_streams(wv):
    """Batched calls in flight on 20 streams at once (more than the library keeps buffers for), each with activations of its
    own: every one gives the bits it gives alone."""
    rows, cols, batch, n = 20000, 2048, 24, 20
    L = wv._lib.lib()
    key, _keep = _packed(wv, "Q8_0", rows, cols, 30)
    x = torch.randn(n, batch, cols, device="cuda", generator=torch.Generator("cuda").manual_seed(31))
    alone, y = torch.zeros(n, batch, rows, device="cuda"), torch.zeros(n, batch, rows, device="cuda")
    for i in range(n):
        wv._lib.check(L.wv_matvec_dev(key, x[i].data_ptr(), alone[i].data_ptr(), batch, cols, rows, None))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(n)]
    for _ in range(3):
        y.zero_()
        torch.cuda.synchronize()
        for i, s in enumerate(streams):
            wv._lib.check(L.wv_matvec_dev(key, x[i].data_ptr(), y[i].data_ptr(), batch, cols, rows, s.cuda_stream))
        torch.cuda.synchronize()
        assert torch.equal(alone, y)
    assert L.wv_device_status() == 0


def test_batched_calls_in_graphs(wv):
    """Two captured batched calls replayed on two streams while the stream they were captured on makes larger calls: the
    graphs' buffers are their own, and outlive the growth of the stream's."""
    rows, cols = 20000, 2048
    L = wv._lib.lib()
    key, _keep = _packed(wv, "Q4_K", rows, cols, 32)
    gen = torch.Generator("cuda").manual_seed(33)
    side = torch.cuda.Stream()
    jobs = []
    for batch in (8, 20):
        x, y = torch.randn(batch, cols, device="cuda", generator=gen), torch.zeros(batch, rows, device="cuda")
        with torch.cuda.stream(side):
            wv._lib.check(L.wv_matvec_dev(key, x.data_ptr(), y.data_ptr(), batch, cols, rows, side.cuda_stream))
        torch.cuda.synchronize()
        want = y.clone()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            wv._lib.check(L.wv_matvec_dev(key, x.data_ptr(), y.data_ptr(), batch, cols, rows, torch.cuda.current_stream().cuda_stream))
        jobs.append((g, x, y, want))
    xb, yb = torch.randn(256, cols, device="cuda", generator=gen), torch.zeros(256, rows, device="cuda")
    wv._lib.check(L.wv_matvec_dev(key, xb.data_ptr(), yb.data_ptr(), 256, cols, rows, side.cuda_stream))
    torch.cuda.synchronize()
    wantb = yb.clone()
    streams = [torch.cuda.Stream() for _ in jobs]
    for _ in range(3):
        yb.zero_()
        for _, _, y, _ in jobs:
            y.zero_()
        torch.cuda.synchronize()
        for (g, _, _, _), s in zip(jobs, streams):
            with torch.cuda.stream(s):
                g.replay()
        wv._lib.check(L.wv_matvec_dev(key, xb.data_ptr(), yb.data_ptr(), 256, cols, rows, side.cuda_stream))
        torch.cuda.synchronize()
        assert torch.equal(yb, wantb) and all(torch.equal(y, want) for _, _, y, want in jobs)
    assert L.wv_device_status() == 0


@pytest.mark.parametrize("slice_", [1, 2, 5])
@pytest.mark.parametrize("batch", [9, 100])
def test_batched_wait_that_runs_out(wv, hooks, slice_, batch):
    """A producer warp that never hands its slice over: the waits of the others run out, the call ends with the time-out
    status, copies and MMAs that were in flight are waited for, and the next call is as good as any."""
    rows, cols = 300, 14336
    key, _keep = _packed(wv, "Q4_0", rows, cols, 40)
    x = torch.randn(batch, cols, device="cuda", generator=torch.Generator("cuda").manual_seed(41))
    y = [torch.zeros(batch, rows, device="cuda") for _ in range(3)]

    def call(i):
        wv._lib.check(hooks.wv_matvec_dev(key, x.data_ptr(), y[i].data_ptr(), batch, cols, rows, None))
        torch.cuda.synchronize()
        return hooks.wv_device_status()

    assert call(0) == 0
    hooks.wv_set_tcg_stall(slice_, 2000)
    try:
        assert call(1) != 0
    finally:
        hooks.wv_set_tcg_stall(0, 0)
    assert call(2) == 0 and torch.equal(y[0], y[2])


@pytest.mark.parametrize("shape", [(40, 14336), (300, 14336), (70, 4352), (129, 8192)], ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("fmt", ["Q8_0", "Q4_K", "AffinePacked"])
def test_batched_few_rows_many_columns(wv, fmt, shape):
    """One to three row tiles whose columns are split over more CTAs than a portable cluster holds; the last split shorter than
    the others, or not."""
    rows, cols = shape
    w = np.random.default_rng(cols).normal(0, 0.02, rows * cols).astype(np.float32)
    ob = O.pack(fmt, w, rows, cols)
    wd = O.unpack(ob).reshape(rows, cols).astype(np.float64)
    for batch in (6, 33, 256):
        x = np.random.default_rng(batch).normal(0, 1, (batch, cols)).astype(np.float32)
        y, _ = _run(wv, ob, x)
        assert np.all(np.abs(y - x.astype(np.float64) @ wd.T) <= 9.9e-4 * (np.abs(x).astype(np.float64) @ np.abs(wd).T) + 1e-30), batch


@pytest.mark.parametrize("group,cols", [(32, 1920), (96, 1920), (160, 1920), (256, 2048), (96, 1056)])
def test_batched_affine_groups(wv, group, cols):
    """Groups of one, three, five and eight chunks: inside a producer's load unit, across two units, and (1056 columns, 33 chunks)
    chunk by chunk."""
    rows = 200
    w = np.random.default_rng(group).normal(0, 0.02, rows * cols).astype(np.float32)
    ob = O.pack("AffinePacked", w, rows, cols, group)
    wd = O.unpack(ob).reshape(rows, cols).astype(np.float64)
    for batch in (6, 70):
        x = np.random.default_rng(batch).normal(0, 1, (batch, cols)).astype(np.float32)
        y, _ = _run(wv, ob, x)
        assert np.all(np.abs(y - x.astype(np.float64) @ wd.T) <= 9.9e-4 * (np.abs(x).astype(np.float64) @ np.abs(wd).T) + 1e-30), batch


def test_batched_graphs_come_and_go(wv):
    """Graphs captured and dropped one after another, each with more rows than the last, so that no buffer given back is large
    enough for the next; then one with few rows, which reuses one, and a larger call outside a capture, which frees the rest."""
    rows, cols = 1024, 2048
    L = wv._lib.lib()
    key, _keep = _packed(wv, "Q8_0", rows, cols, 34)
    side = torch.cuda.Stream()
    gen = torch.Generator("cuda").manual_seed(35)
    x, y = torch.zeros(6, cols, device="cuda"), torch.zeros(6, rows, device="cuda")
    wv._lib.check(L.wv_matvec_dev(key, x.data_ptr(), y.data_ptr(), 6, cols, rows, side.cuda_stream))      # the kernel is loaded before any capture
    for batch in (8, 40, 120, 16, 250):
        x, y = torch.randn(batch, cols, device="cuda", generator=gen), torch.zeros(batch, rows, device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            wv._lib.check(L.wv_matvec_dev(key, x.data_ptr(), y.data_ptr(), batch, cols, rows, torch.cuda.current_stream().cuda_stream))
        g.replay()
        torch.cuda.synchronize()
        got = y.clone()
        g.reset()
        del g
        y.zero_()
        wv._lib.check(L.wv_matvec_dev(key, x.data_ptr(), y.data_ptr(), batch, cols, rows, side.cuda_stream))
        torch.cuda.synchronize()
        assert torch.equal(got, y), batch
    assert L.wv_device_status() == 0


@pytest.mark.parametrize("fmt,rows,cols", [("Q4_0", 333, 512), ("Q4_K", 700, 2048), ("Q8_0", 130, 254)])
def test_dense_forward_one_row_again_and_again(wv, fmt, rows, cols):
    """A layer with bias and activation called row by row: from the second call on one graph launch serves it. New x and new bias values
    every time, two activations and two bias lengths in turn, a larger batch that moves the slot's buffers and a matrix that is
    evicted and uploaded again in between. The bits are the plain product's plus the bias."""
    d = wv.dense
    rng = np.random.default_rng(rows)
    layer = d.NewConfigured(cols, rows, d.ActivationReLU, wv.quant.DTypeFloat32, wv.quant.Format["Format" + fmt], rng.normal(0, 0.1, rows * cols).astype(np.float32))
    for step in range(30):
        x = rng.standard_normal((40 if step == 12 else 1, cols), np.float32)
        if step % 10 == 0:
            layer.Activation = (d.ActivationReLU, d.ActivationLeakyReLU, d.ActivationReLU)[step // 10]
        bias = rng.normal(0, 1, rows if step < 24 else 7)
        layer.Weights.Bias, act = None, layer.Activation
        layer.Activation = d.ActivationLinear
        want = d.Forward(layer, x)[0].astype(np.float64)
        want[:, :len(bias)] += bias
        layer.Weights.Bias, layer.Activation = bias, act
        if step == 16:
            wv._lib.lib().wv_blob_evict(wv.quant.EnsureResident(layer.Weights.Packed))
        pre, post = d.Forward(layer, x)
        np.testing.assert_array_equal(pre, want.astype(np.float32))
        np.testing.assert_array_equal(post, d.Activate(pre, act).astype(np.float32))


@pytest.mark.parametrize("n,batch", [(256, 8), (1024, 33), (4096, 6), (1280, 256)])
def test_batched_calls_in_a_chain(wv, n, batch):
    """Each batched call's X is the Y of the call right before it on the stream, with another batched call behind: the kernel that rounds
    X lets the next one start before its own wait. The same bits as with a synchronisation behind every call."""
    L, check = wv._lib.lib(), wv._lib.check
    gen = torch.Generator(device="cuda").manual_seed(n)
    keys = [0x7400, 0x7401, 0x7402]
    x = torch.randn(batch, n, device="cuda", generator=gen)
    stream = torch.cuda.Stream()

    def chain(wait):
        ys = [torch.full((batch, n), float("nan"), device="cuda") for _ in range(12)]
        torch.cuda.synchronize()
        for i, y in enumerate(ys):
            check(L.wv_matvec_dev(keys[i % 3], (ys[i - 1] if i else x).data_ptr(), y.data_ptr(), batch, n, n, stream.cuda_stream))
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return torch.stack(ys)
    try:
        for key, f in zip(keys, ("Q8_0", "Q4_K", "Q4_0")):
            w = torch.randn(n, n, device="cuda", generator=gen) / n ** 0.5
            torch.cuda.synchronize()
            check(L.wv_pack_upload_dev(key, O.FMT[f], 1, 0, w.data_ptr(), n, n, None))
        want = chain(True)
        assert bool(want.isfinite().all())
        for _ in range(5):
            assert torch.equal(chain(False), want)
        assert L.wv_device_status() == 0
    finally:
        for key in keys:
            L.wv_blob_evict(key)


@pytest.mark.parametrize("fmt", ["Q4_0", "Q5_K", "Q8_0", "IQ3_S"])
@pytest.mark.parametrize("shape", [(130, 256), (129, 4352)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_batched_rounds_of_stages(wv, fmt, shape):
    """Either side of the line between two rounds of pipeline stages and one (192 rows), as in test_batched_column_orders."""
    rows, cols = shape
    ob = O.pack(fmt, np.random.default_rng(cols).normal(0, 0.02, rows * cols).astype(np.float32), rows, cols)
    wd = O.unpack(ob).reshape(rows, cols).astype(np.float64)
    for batch in (177, 192, 193, 208):
        x = np.random.default_rng(batch).normal(0, 1, (batch, cols)).astype(np.float32)
        y, _ = _run(wv, ob, x)
        assert np.all(np.abs(y - x.astype(np.float64) @ wd.T) <= 9.9e-4 * (np.abs(x).astype(np.float64) @ np.abs(wd).T) + 1e-30), batch


@pytest.mark.parametrize("batch", [1, 3, 8])
def test_dense_forward_non_finite_and_threads(wv, batch):
    """Bias and activation on the device with infinities and NaN in x and in the bias, from four threads at once: where the float64
    passes of dense.Activate give an infinity or a NaN the device does, elsewhere the bounds of the test above hold."""
    import threading
    d, rows, cols = wv.dense, 300, 512
    errors = []

    def worker(seed):
        try:
            rng = np.random.default_rng(seed)
            layer = d.NewConfigured(cols, rows, d.ActivationLinear, wv.quant.DTypeFloat32, wv.quant.Format.FormatQ4_0, rng.normal(0, 0.1, rows * cols).astype(np.float32))
            x = rng.normal(0, 1, (batch, cols)).astype(np.float32)
            if seed % 2:
                x[-1, 7] = (np.inf, np.nan)[seed // 2]
            y = d.Forward(layer, x)[0].astype(np.float64)
            bias = rng.normal(0, 3, rows)
            bias[[3, 50, 299]], bias[[7, 8]] = (np.inf, -np.inf, np.nan), (3e38, -3e38)
            layer.Weights.Bias = bias
            with np.errstate(all="ignore"):
                want = (y + bias).astype(np.float32)
                for act in d._ACTIVATIONS * 3:
                    layer.Activation = act
                    pre, post = d.Forward(layer, x)
                    np.testing.assert_array_equal(pre, want)
                    p = pre.astype(np.float64)
                    ref = d.Activate(p, act).astype(np.float32)
                    ok = np.isfinite(ref)
                    np.testing.assert_array_equal(post[~ok], ref[~ok])
                    exact = d.Activate(p, act)[ok]
                    assert np.all(np.abs(post[ok] - exact) <= 2.0 ** -23 * np.abs(exact) + 2.0 ** -49 * np.abs(p[ok]) + 1e-45), act
        except BaseException as e:      # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=worker, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_host_calls_with_scratch_from_threads(wv):
    """Widths whose kernel takes scratch for the activation records (an odd number of chunks), replayed from graphs of several slots
    while other calls go round the shared scratch ring more than once: every call's bits are those of the first."""
    import threading
    d, L, check = wv.dense, wv._lib.lib(), wv._lib.check
    rows, cols, errors = 40, 16352, []
    gen = torch.Generator(device="cuda").manual_seed(1)
    w, x, y = (torch.randn(n, device="cuda", generator=gen) for n in (rows * cols, cols, rows))
    torch.cuda.synchronize()
    check(L.wv_pack_upload_dev(0x7500, O.FMT["Q4_0"], 1, 0, w.data_ptr(), rows, cols, None))
    stream = torch.cuda.Stream()

    def worker(seed):
        try:
            rng = np.random.default_rng(seed)
            layer = d.NewConfigured(cols, rows, d.ActivationLinear, wv.quant.DTypeFloat32, wv.quant.Format.FormatQ4_0, rng.normal(0, 0.1, rows * cols).astype(np.float32))
            xs = rng.standard_normal((4, 1, cols), np.float32)
            bias = rng.normal(0, 1, rows)
            want = [d.Forward(layer, v)[0] for v in xs]
            for i in range(400):
                layer.Weights.Bias, layer.Activation = (bias, d.ActivationReLU) if i % 3 == 0 else (None, d.ActivationLinear)
                pre, post = d.Forward(layer, xs[i % 4])
                np.testing.assert_array_equal(pre, (want[i % 4] + bias).astype(np.float32) if i % 3 == 0 else want[i % 4])
                np.testing.assert_array_equal(post, np.maximum(pre, 0) if i % 3 == 0 else pre)
        except BaseException as e:      # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=worker, args=(s,)) for s in range(3)]
    for t in threads:
        t.start()
    for i in range(1200):
        check(L.wv_matvec_dev(0x7500, x.data_ptr(), y.data_ptr(), 1, cols, rows, stream.cuda_stream))
        if i % 50 == 49:
            stream.synchronize()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    L.wv_blob_evict(0x7500)
    assert not errors, errors[0]
