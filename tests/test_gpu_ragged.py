"""Rows that do not start on a chunk or vector boundary: the chunk-wise ragged kernels at the sizes where a row's first and
last chunk are shared with its neighbours in every way, and at rows too wide for shared memory."""
import numpy as np
import pytest

import oracle as O
from conftest import CASES, case_id, case_ok, make_w, to_product_blob

pytestmark = pytest.mark.gpu

# one chunk or less, one more than a chunk, half-chunk boundaries, more chunks than lanes, more rows than warps in the
# grid, shared memory just below 48 KB (11500, before any wider row), above it and at its limit (49150), and (49154) x
# read from global memory
SHAPES = [(7, 5), (40, 33), (37, 48), (19, 1022), (9, 1070), (9001, 46), (4, 11500), (5, 20001), (3, 49150), (3, 49154)]


@pytest.mark.parametrize("case", [c for c in CASES if c[1] == 0], ids=case_id)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_ragged_rows(wv, case, shape):
    rows, cols = shape
    if not case_ok(case, rows, cols):
        pytest.skip("layout needs aligned cols")
    f, bw, dt = case
    w, x = make_w(rows * 7 + cols, rows, cols)
    ob = O.pack(f, w, rows, cols, bw, dt)
    y = np.zeros(rows, np.float32)
    wv.dense.MatVecPackedBlob(to_product_blob(wv, ob), x, y)
    wd = O.unpack(ob).reshape(rows, cols).astype(np.float64)
    ref, den = wd @ x, np.abs(wd) @ np.abs(x)
    # float32: at most 24 roundings inside a chunk and over the lanes plus one per 1024 columns, each 2^-24 of sum |w x|;
    # twice that for the formats with a min, whose |code * scale| may exceed |w|
    assert np.all(np.abs(y - ref) <= 2 * (24 + cols / 1024) * 2.0 ** -24 * den + 1e-30)


def test_ragged_batch_and_neighbours(wv):
    """Batch rows, and a neighbour's non-finite scale that shares a chunk but no half of it with the row."""
    rows, cols, batch = 5, 48, 3
    w, _ = make_w(5, rows, cols)
    X = np.random.default_rng(6).normal(0, 1, (batch, cols)).astype(np.float32)
    ob = O.pack("IQ3_S", w, rows, cols)
    ob.scales[0:3] = np.inf          # row 0 is groups 0 - 2; group 3, in the same chunk as group 2, is row 1's
    st = wv.weights.FromBlob(to_product_blob(wv, ob))
    pre, _ = wv.dense.Forward(wv.dense.Layer(cols, rows, wv.dense.ActivationLinear, st), X)
    wd = O.unpack(ob).reshape(rows, cols).astype(np.float64)[1:]
    ref, den = X @ wd.T, np.abs(X) @ np.abs(wd).T
    assert np.all(np.isfinite(pre[:, 1:])) and np.all(np.abs(pre[:, 1:] - ref) <= 50 * 2.0 ** -24 * den)
    assert not np.any(np.isfinite(pre[:, 0]))


def _raw_rows(wv, ob, X):
    st = wv.weights.FromBlob(to_product_blob(wv, ob))
    pre, _ = wv.dense.Forward(wv.dense.Layer(ob.cols, ob.rows, wv.dense.ActivationLinear, st), X)
    wd = O.unpack(ob).reshape(ob.rows, ob.cols).astype(np.float64)
    return pre, wd


@pytest.mark.parametrize("fmt", ["TernaryPacked", "Q4_1"])
def test_ragged_neighbours_infinite_weights(wv, fmt):
    """A group that two rows share, in which the neighbour's weights are infinite and this row's are not: a ternary group of
    infinite scale where this row has zeros, and codes of 15 times a scale of 1e38 beside codes of 0."""
    rows, cols = 4, 40                     # weights 32 - 39 are row 0's, 40 - 47 row 1's
    w, _ = make_w(8, rows, cols)
    X = np.random.default_rng(9).normal(0, 1, (2, cols)).astype(np.float32)
    ob = O.pack(fmt, w, rows, cols)
    if fmt == "TernaryPacked":
        ob.scales[2] = np.inf
        ob.raw[8:12] = [0x55, 0x55, 0xAA, 0xAA]
    else:
        ob.raw[24:28] = np.frombuffer(np.float32(1e38).tobytes(), np.uint8)
        ob.raw[32:48] = [0] * 4 + [255] * 12
    pre, wd = _raw_rows(wv, ob, X)
    assert np.all(np.isfinite(wd[[0, 3]])) and np.any(np.isinf(wd[1]))
    assert not np.any(np.isfinite(pre[:, 1]))
    for r in (0, 3):
        assert np.all(np.abs(pre[:, r] - X @ wd[r]) <= 100 * 2.0 ** -24 * (np.abs(X) @ np.abs(wd[r])))


@pytest.mark.parametrize("fmt", ["Q8_0", "Q6_K", "IQ3_S", "IQ4_NL", "IQ4_XS", "TernaryPacked"])
def test_ragged_large_activations(wv, fmt):
    """Activations of 1e37: the products with the weights are far from float32's limit, those with the bare codes are not."""
    rows, cols = 20, 1022
    w, _ = make_w(11, rows, cols)
    X = (1e37 * np.random.default_rng(12).normal(0, 1, (2, cols))).astype(np.float32)
    pre, wd = _raw_rows(wv, O.pack(fmt, w, rows, cols), X)
    ref, den = X.astype(np.float64) @ wd.T, np.abs(X.astype(np.float64)) @ np.abs(wd).T
    assert den.max() < 3e38
    assert np.all(np.isfinite(pre)) and np.all(np.abs(pre - ref) <= 100 * 2.0 ** -24 * den)


# 8, 16 and 32 lanes per row: widths on both sides of 8 and 16 units (chunks: 225 / 226, 481 / 482; vectors of 4 elements: 29 / 30,
# 61 / 62; of 8: 57 / 58, 121 / 122), and rows enough for fewer lanes than units; rows that leave a warp's last rows empty
LANE_SHAPES = [(65, 29), (33, 30), (37, 57), (38, 58), (39, 61), (41, 62), (65, 121), (33, 122), (70, 225), (71, 226), (30, 481), (29, 482),
               (1579, 1022), (3157, 514), (3159, 1030)]


@pytest.mark.parametrize("case", [c for c in CASES if c[1] == 0], ids=case_id)
def test_ragged_lanes_per_row(wv, case):
    f, bw, dt = case
    for rows, cols in LANE_SHAPES:
        if not case_ok(case, rows, cols):
            continue
        w, _ = make_w(rows + cols, rows, cols)
        X = np.random.default_rng(cols).normal(0, 1, (3, cols)).astype(np.float32)
        pre, wd = _raw_rows(wv, O.pack(f, w, rows, cols, bw, dt), X)
        # float32: a lane adds at most cols / 32 + 8 products in a row, then 8 sums; a weight with a min has two more roundings
        assert np.all(np.abs(pre - X @ wd.T) <= (cols / 32 + 30) * 2.0 ** -24 * (np.abs(X) @ np.abs(wd).T) + 1e-30), (rows, cols)
