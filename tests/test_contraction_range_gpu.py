"""Tensor-core contractions of the histogram path where the operands of one sum span more than fp16 halves of one scale do: every result
is as accurate as its own terms ask for, against the fp32 FMA contractions."""
import numpy as np
import pytest

import golden_util
from test_hist_contractions_gpu import SHAPES
from test_product_gpu import inputs_for, run_gpu

pytestmark = pytest.mark.gpu


def problem(name, signed=False):
    cfg = dict(SHAPES[name])
    cfg["n_virtual"] = 2 * cfg["E"] + cfg["Npe"]
    x, anchors, W, pe, dY = inputs_for(cfg)
    if signed:
        return cfg, x, anchors, W.reshape(-1, cfg["O"]), pe, dY
    # positive terms: a sum is as large as its terms, so that fp32 sums of n terms in any order agree to sqrt(n) * 2^-24 of themselves
    return cfg, x, anchors, np.abs(W).reshape(-1, cfg["O"]) + np.float32(0.1), pe, np.abs(dY) + np.float32(0.1)


def both(cfg, x, anchors, W, pe, dY):
    W, dY = W.astype(np.float32).reshape(-1), dY.astype(np.float32)
    return run_gpu(cfg, x, anchors, W, pe, dY, 2), run_gpu(cfg, x, anchors, W, pe, dY, 3)


def assert_each_close(a, b, rel, what):
    a, b = a.astype(np.float64), b.astype(np.float64)
    assert np.isfinite(b).all() and (b >= 0).all() and (b > 0).any()
    assert (np.abs(a - b) <= rel * b).all(), f"{what}: {np.max(np.abs(a - b) / np.where(b > 0, b, 1)):.1e}"


@pytest.mark.parametrize("decades", [8, 14, 30])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_rows_and_queries_of_any_size(name, decades):
    """Table rows and queries' gradients of very different size: a query that selects small rows only has their sum, a table row
    that small gradients reach only has theirs.  (Up to n = 3e5 terms: sqrt(n) * 2^-24 = 3e-5 at the very most, 1e-5 for these sizes.)"""
    cfg, x, anchors, W, pe, dY = problem(name)
    rng = np.random.default_rng(decades)
    W = W * 10.0 ** -(decades * rng.random((W.shape[0], 1)))
    dY = dY * 10.0 ** -(decades * rng.random(dY.shape[:2] + (1,)))
    W[1], dY[:, 3] = 0.0, 0.0
    got, want = both(cfg, x, anchors, W, pe, dY)
    assert_each_close(got["y"], want["y"], 1e-5, "y")
    assert_each_close(got["dW"], want["dW"], 1e-5, "dW")


@pytest.mark.parametrize("decades", [5, 7, 12])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_outputs_of_any_size(name, decades):
    """Outputs of very different size, gradients the other way round: all terms of a row dot are of one size, whichever of its
    factors is small."""
    cfg, x, anchors, W, pe, dY = problem(name)
    size = 10.0 ** (decades * np.random.default_rng(decades).uniform(-1, 1, cfg["O"]))
    got, want = both(cfg, x, anchors, W * size, pe, dY / size)
    assert_each_close(got["y"], want["y"], 1e-5, "y")
    assert_each_close(got["dW"], want["dW"], 1e-5, "dW")
    # (differences of row dots: of terms of both signs, so that they are of the dots' own size)
    cfg, x, anchors, W, pe, dY = problem(name, signed=True)
    got, want = both(cfg, x, anchors, W * size, pe, dY / size)
    golden_util.assert_close(got["dX"], want["dX"], 1e-5, "dX")
    if cfg["Npe"]:
        golden_util.assert_close(got["dPE"], want["dPE"], 1e-5, "dPE")


@pytest.mark.parametrize("small", [1e-10, 1e-13, 1e-20])
@pytest.mark.parametrize("operand", ["W", "dY"])
def test_one_small_element(operand, small):
    """Rows and columns of one large element and small ones, and one small element alone."""
    cfg, x, anchors, W, pe, dY = problem("parts_and_slices")
    a = W if operand == "W" else dY.reshape(-1, cfg["O"])
    a[:, 17] *= small    # small in its row
    a[40, 17] = 3.0      # and in its column, but for this one
    a[:, 250] = 0.0
    a[7, 250] = small
    a[1100, 5] = small
    got, want = both(cfg, x, anchors, W, pe, dY)
    for k in ("y", "dW"):
        assert_each_close(got[k], want[k], 1e-5, k)
    cfg, x, anchors, W, pe, dY = problem("parts_and_slices", signed=True)
    (W if operand == "W" else dY.reshape(-1, cfg["O"]))[:, 17] *= small
    (dY.reshape(-1, cfg["O"]) if operand == "W" else W)[:, 17] /= small
    got, want = both(cfg, x, anchors, W, pe, dY)
    golden_util.assert_close(got["dX"], want["dX"], 1e-5, "dX")


def test_small_elements_in_different_rows_of_neighbouring_columns():
    """Columns of one tile with small elements in different parts of a slice, in memory that held NaN before (where a column has none its
    second halves are not written)."""
    import torch

    cfg, x, anchors, W, pe, dY = problem("parts_and_slices")
    rows = dY.reshape(-1, cfg["O"])
    for k in range(9):   # 128 rows, 16 columns at a time
        rows[128 * k + 5, 16 * k + 3] = 1e-10
        W[200 * k + 7, 16 * k + 4] = 1e-10
    junk = torch.full((256 << 20,), float("nan"), device="cuda")   # (freed, and likely to be the calls' scratch)
    del junk
    got, want = both(cfg, x, anchors, W, pe, dY)
    for k in ("y", "dW"):
        assert_each_close(got[k], want[k], 1e-5, k)
    assert np.isfinite(got["dX"]).all()


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_what_is_not_finite_stays_in_its_column(value):
    cfg, x, anchors, W, pe, dY = problem("parts_and_slices")
    base = run_gpu(cfg, x, anchors, W.reshape(-1), pe, dY, 2)
    W[5, 33] = value
    W[9, 33] = 1e-30
    got = run_gpu(cfg, x, anchors, W.reshape(-1), pe, dY, 2)
    kept = np.arange(cfg["O"]) != 33
    assert np.array_equal(got["y"][..., kept], base["y"][..., kept])
    assert not np.isfinite(got["y"][..., 33]).any()
    assert np.array_equal(got["dW"], base["dW"])
