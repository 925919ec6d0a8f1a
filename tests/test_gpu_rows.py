"""Two to five activation rows: every packed layout on whichever kernel takes it, batches that fill a CTA's rows unevenly,
bands of less than a tile, one and several column warps, and rows up to and beyond the width that leaves the integer-dot
rows kernel room for its records."""
import numpy as np
import pytest

import oracle as O
from conftest import CASES, case_id, case_ok, make_w
from test_gpu_batched import _run

pytestmark = pytest.mark.gpu

# rows x cols: fewer rows than SMs, a partial last tile, one column warp, a partial last column warp (1280 = 40 chunks),
# 4608 (formats that the tensor pipe takes up to 4096), 6144, 14336 (row by row); the smallest run row by row in most batches
SHAPES = [(5, 512), (300, 1024), (149, 1280), (450, 4096), (40, 4608), (64, 6144), (40, 14336)]


def _bound(ob, x):
    """float32 scales and sums over at most 16 column warps (64 roundings are ample), and an activation off by at most
    amax / 65024 of its 32-column chunk under 16-bit records."""
    wd = np.abs(O.unpack(ob).reshape(ob.rows, ob.cols).astype(np.float64))
    amax = np.abs(x).reshape(-1, 32).max(1).repeat(32)
    return wd @ (np.abs(x) * 64 * 2.0 ** -24 + amax / 65024) + 1e-30


@pytest.mark.parametrize("case", [c for c in CASES if c[0] != "none"], ids=case_id)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_rows_every_format(wv, case, shape):
    rows, cols = shape
    if not case_ok(case, rows, cols):
        pytest.skip("layout needs aligned cols")
    f, bw, dt = case
    w, _ = make_w(rows + cols, rows, cols)
    ob = O.pack(f, w, rows, cols, bw, dt)
    wd = O.unpack(ob).reshape(rows, cols).astype(np.float64)
    rng = np.random.default_rng(cols)
    for batch in (2, 3, 5):
        x = rng.normal(0, 1, (batch, cols)).astype(np.float32)
        x[-1] *= 1e-20
        x[0, ::97] *= 1e4             # outliers: 24-bit records for this row only
        y, _ = _run(wv, ob, x)
        for m in range(batch):
            err = np.abs(y[m] - wd @ x[m].astype(np.float64))
            assert np.all(err <= 2 * _bound(ob, x[m])), (batch, m, float(np.max(err / _bound(ob, x[m]))))


def test_rows_keep_their_own_infinities(wv):
    """A non-finite activation makes its own row's outputs NaN and leaves the others alone."""
    rows, cols = 64, 2048
    w, _ = make_w(3, rows, cols)
    ob = O.pack("Q4_K", w, rows, cols)
    x = np.random.default_rng(4).normal(0, 1, (4, cols)).astype(np.float32)
    clean, _ = _run(wv, ob, x)
    x[2, 700] = np.inf
    y, _ = _run(wv, ob, x)
    assert np.all(np.isnan(y[2])) and np.array_equal(y[[0, 1, 3]], clean[[0, 1, 3]])


@pytest.mark.parametrize("fmt,cols", [("Q4_K", 2048), ("Q6_K", 2048), ("TernaryPacked", 2048), ("IQ3_S", 2048), ("Q4_0", 4608), ("Q5_0", 4608)])
@pytest.mark.parametrize("bad", [np.inf, -np.inf])
def test_infinite_activations_give_nan(wv, fmt, cols, bad):
    """An infinity among ordinary values, in the formats without a min (whose sums hold nothing that is NaN by itself) as
    well: the rows kernel and the one-row kernel make the row's outputs NaN, never a number or an infinity of some sign."""
    rows = 40
    w, _ = make_w(9, rows, cols)
    ob = O.pack(fmt, w, rows, cols)
    x = np.random.default_rng(10).normal(0, 1, (4, cols)).astype(np.float32)
    x[2, 700] = bad
    y, _ = _run(wv, ob, x)
    assert np.all(np.isnan(y[2])) and np.all(np.isfinite(y[[0, 1, 3]]))
    one, _ = _run(wv, ob, x[2:3])
    assert np.all(np.isnan(one))


@pytest.mark.parametrize("fmt,rows,cols,batch", [("Q4_K", 24, 4096, 4), ("Q6_K", 29, 1024, 5), ("IQ3_XXS", 74, 6144, 2), ("Q4_K", 64, 6144, 3), ("TernaryPacked", 42, 4096, 4)])
def test_few_rows_of_w_run_row_by_row(wv, fmt, rows, cols, batch):
    """Where all activation rows' CTAs fit on the chip side by side the batch is that many one-row launches in one: the same
    bits as one at a time."""
    w, _ = make_w(rows, rows, cols)
    ob = O.pack(fmt, w, rows, cols)
    x = np.random.default_rng(rows).normal(0, 1, (batch, cols)).astype(np.float32)
    y, _ = _run(wv, ob, x)
    one = np.concatenate([_run(wv, ob, x[m:m + 1])[0] for m in range(batch)])
    assert np.array_equal(y, one)


@pytest.mark.parametrize("fmt", ["TernaryPacked", "IQ1_S", "Q4_0"])
def test_two_rows_of_wide_matrices_run_one_by_one(wv, fmt):
    rows, cols = 1200, 9216
    w, _ = make_w(2, rows, cols)
    ob = O.pack(fmt, w, rows, cols)
    x = np.random.default_rng(3).normal(0, 1, (2, cols)).astype(np.float32)
    y, _ = _run(wv, ob, x)
    assert np.array_equal(y, np.concatenate([_run(wv, ob, x[m:m + 1])[0] for m in range(2)]))


@pytest.mark.parametrize("fmt", ["TernaryPacked", "Q4_K"])
def test_two_rows_of_a_streamed_wide_matrix_keep_their_precision(wv, fmt):
    """More than 64 MB of codes at 9216 columns: two rows stay on the integer-dot kernel, whose error the tensor cores' TF32
    (2.9e-4 of the result's norm) exceeds."""
    n, block, cols = {"TernaryPacked": 112, "Q4_K": 56}[fmt], 256, 9216
    w = np.random.default_rng(5).normal(0, 0.02, block * cols).astype(np.float32)
    ob = O.pack(fmt, w, block, cols)          # rows are whole groups: a block of them, repeated
    big = O.Blob(ob.format, n * block, cols, np.tile(ob.raw, n), np.tile(ob.scales, n), np.tile(ob.mins, n), ob.block_weights, ob.dtype)
    x = np.random.default_rng(6).normal(0, 1, (2, cols)).astype(np.float32)
    y, _ = _run(wv, big, x)
    ref = np.tile(x.astype(np.float64) @ O.unpack(ob).reshape(block, cols).astype(np.float64).T, n)
    # 16-bit records: an activation is off by amax / 65024 of its chunk at most, some 5e-5 of its size on the average
    assert np.linalg.norm(y - ref) <= 1e-4 * np.linalg.norm(ref)


# a band of one row in some CTAs, widths with two row groups (2048 to 8192, where 4-bit formats have no room for their ring)
# and with one (8704)
WIDE_SHAPES = [(100, 2048), (100, 7168), (100, 8192), (100, 8704)]


@pytest.mark.parametrize("case", [c for c in CASES if c[0] != "none"], ids=case_id)
@pytest.mark.parametrize("shape", WIDE_SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_rows_four_to_a_cta(wv, case, shape):
    """Four activation rows: all of a CTA's record slots in use, each against float64."""
    rows, cols = shape
    if not case_ok(case, rows, cols):
        pytest.skip("layout needs aligned cols")
    f, bw, dt = case
    w, _ = make_w(rows + cols, rows, cols)
    ob = O.pack(f, w, rows, cols, bw, dt)
    wd = O.unpack(ob).reshape(rows, cols).astype(np.float64)
    x = np.random.default_rng(cols).normal(0, 1, (4, cols)).astype(np.float32)
    x[3] *= 1e3
    x[1, ::97] *= 1e4             # outliers: 24-bit records for this row only
    y, _ = _run(wv, ob, x)
    for m in range(4):
        err = np.abs(y[m] - wd @ x[m].astype(np.float64))
        assert np.all(err <= 2 * _bound(ob, x[m])), (m, float(np.max(err / _bound(ob, x[m]))))
