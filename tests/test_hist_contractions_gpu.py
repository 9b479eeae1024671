"""The fp16-split tensor-core contractions of the histogram path (hist_gemm_sm100.cu) at the edges of their tiles, slices and
parts, and their scales."""
import numpy as np
import pytest

import golden_util
from test_product_gpu import inputs_for, run_gpu

pytestmark = pytest.mark.gpu

SHAPES = {
    # table narrower than a box of the tensor map, rows of 12 outputs (padded to 16 in the fp16 copies)
    "one_small_table": dict(seed=801, B=1, S=40, E=6, Nt=1, Nc=4, Npe=1, O=12),
    # KT = 2304: 36 blocks of 64, in several parts; 1170 rows: two slices in the table gradient, the last tile of 256 half empty
    "parts_and_slices": dict(seed=802, B=9, S=130, E=6, Nt=9, Nc=8, Npe=0, O=260),
    # more than one tile along every extent and one row, one column past a tile; a contraction of 65 elements (rows)
    "one_past": dict(seed=803, B=1, S=257, E=5, Nt=17, Nc=4, Npe=2, O=260),
    "one_block": dict(seed=804, B=1, S=64, E=5, Nt=4, Nc=4, Npe=0, O=64),
}


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_contractions_match_the_fma_contractions(name):
    """Both sum up to n = 300000 fp32 terms a cell in different orders: sqrt(n) * 2^-24 = 3e-5 of the largest at the very most,
    1e-5 as everywhere for these sizes."""
    cfg = dict(SHAPES[name])
    cfg["n_virtual"] = 2 * cfg["E"] + cfg["Npe"]
    x, anchors, W, pe, dY = inputs_for(cfg)
    got, want = run_gpu(cfg, x, anchors, W, pe, dY, 2), run_gpu(cfg, x, anchors, W, pe, dY, 3)
    for k in want:
        golden_util.assert_close(got[k], want[k], 1e-5, k)


@pytest.mark.parametrize("e", [0, 40, 100])
def test_scales_are_exact(e):
    """Powers of two on the tables and on the output gradients pass through: the same bits, scaled.  Magnitudes of 2^100 leave
    the range in which the two scales of a row dot may be multiplied in any order, and one row and one column are zero."""
    cfg = dict(SHAPES["one_past"])
    cfg["n_virtual"] = 2 * cfg["E"] + cfg["Npe"]
    x, anchors, W, pe, dY = inputs_for(cfg)
    W, dY = W.copy(), dY.copy()
    W.reshape(-1, cfg["O"])[3] = 0.0
    W.reshape(-1, cfg["O"])[:, 5] = 0.0
    dY[:, 7] = 0.0
    base = run_gpu(cfg, x, anchors, W, pe, dY, 2)
    up, down = np.float32(2.0 ** e), np.float32(2.0 ** -e)
    got = run_gpu(cfg, x, anchors, W * up, pe, dY * down, 2)
    assert np.array_equal(got["y"], base["y"] * up)
    assert np.array_equal(got["dW"], base["dW"] * down)
    # (the routed sums are shared-memory and L2 additions in any order: fp32 rounding of a few hundred terms)
    golden_util.assert_close(got["dX"], base["dX"], 1e-5, "dX")
    assert not base["y"][..., 5].any()


def test_rows_of_very_different_size_keep_their_own_precision():
    """Table rows and output gradients whose magnitudes differ by 10^6 from row to row: every row of the table gradient and every
    query's output is as accurate as its own size asks for (an element 2^-20 below its column's largest still has 22 bits)."""
    cfg = dict(SHAPES["parts_and_slices"])
    cfg["n_virtual"] = 2 * cfg["E"]
    x, anchors, W, pe, dY = inputs_for(cfg)
    rng = np.random.default_rng(5)
    O = cfg["O"]
    W = (W.reshape(-1, O) * 10.0 ** -(6 * rng.random((W.size // O, 1)))).astype(np.float32).reshape(-1)
    dY = (dY * 10.0 ** -(6 * rng.random(dY.shape[:2] + (1,)))).astype(np.float32)
    got, want = run_gpu(cfg, x, anchors, W, pe, dY, 2), run_gpu(cfg, x, anchors, W, pe, dY, 3)
    for k, width in (("y", O), ("dW", O)):
        a, b = got[k].reshape(-1, width).astype(np.float64), want[k].reshape(-1, width).astype(np.float64)
        size = np.abs(b).max(axis=1)
        assert (np.abs(a - b).max(axis=1) <= 1e-5 * size).all(), k
