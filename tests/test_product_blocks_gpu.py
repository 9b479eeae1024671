"""Histogram path of product layers: blocks over (detector, part of the sequence, sequence) where all three have several values, with
every number of key-query anchors a detector can have, against the oracle."""
import numpy as np
import pytest

import golden_util
from oracle import lut_oracle as orc
from test_product_gpu import compare, expand_pe, inputs_for, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [2, 3], ids=["tensor_cores", "fma"])
@pytest.mark.parametrize("Npe", [0, 2])
@pytest.mark.parametrize("B,S,Nc", [(3, 131, 8), (2, 300, 5), (1, 515, 9), (5, 9, 8)])
def test_blocks_of_detectors_parts_and_sequences(B, S, Nc, Npe, variant):
    cfg = dict(seed=1300 + S, B=B, S=S, E=12, Nt=Nc + 1, Nc=Nc, O=8, Npe=Npe, n_virtual=24 + Npe)
    x, anchors, W, pe, dY = inputs_for(cfg)
    anchors = anchors.reshape(Nc + 1, Nc, 2)
    rng = np.random.default_rng(S)
    for t in range(Nc + 1):   # detector t: t anchors that compare a key with a query (either end first), the others keys or queries alone
        for k in range(Nc):
            key, query = rng.integers(0, 12, 2), 12 + rng.integers(0, 12, 2)
            anchors[t, k] = ((key[0], query[0]) if k % 2 else (query[0], key[0])) if k < t else (key if k % 3 else query)
        if Npe:
            anchors[t, Nc - 1, 1] = 24 + t % Npe
    pe3 = expand_pe(cfg, pe)
    y = orc.product_forward(W, x, pe3, anchors, Nc + 1, Nc, 8, Npe)
    dX, dW, dPE = orc.product_backward(W, x, pe3, anchors, dY, Nc + 1, Nc, Npe)
    got = run_gpu(cfg, x, anchors, W, pe, dY, variant)
    # a table cell sums up to n pairs in fp32, in different orders on both sides: about sqrt(n) * 2^-24 of the sum for each
    golden_util.assert_close(got["dW"], dW, 2 * (B * S * (S - 1) / 2) ** 0.5 * 2.0 ** -24, "dW")
    compare(cfg, got, dict(y=y, dX=dX, dW=got["dW"], dPE=dPE))


# counters of 8 bits up to 256 tokens (counts up to 255: every key on one row), of 16 bits from 257 on; ten bits of a count and eleven
@pytest.mark.parametrize("S", [255, 256, 257, 1024, 1025, 1500])
def test_counts_of_one_row(S):
    cfg = dict(seed=1400, B=1, S=S, E=4, Nt=3, Nc=4, O=4, Npe=0, n_virtual=8)
    x, anchors, W, pe, dY = inputs_for(cfg)
    x[...] = np.float32(0.25)   # no difference at all: every pair takes row 0
    x[0, S // 2:, 0] = 1.0      # but those with a later query's (or key's) element 0
    ref_y = orc.product_forward(W, x, expand_pe(cfg, pe), anchors, 3, 4, 4, 0)
    for variant in (2, 3):
        got = run_gpu(cfg, x, anchors, W, pe, dY, variant)
        # a query's sum: counts times at most 16 rows a detector, each to fp32 accuracy or that of the split of its operands (2^-22)
        bound = 3 * S * np.abs(W).max() * 2.0 ** -21 + S * 2.0 ** -24 * np.abs(ref_y)   # and the oracle's own fp32 order
        assert (np.abs(got["y"].astype(np.float64) - ref_y) <= bound).all(), variant
