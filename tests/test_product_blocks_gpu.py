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
