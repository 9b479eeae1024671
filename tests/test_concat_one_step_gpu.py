"""Concatenation layers whose rows are one step of a lane group, with at least a block per SM: every group width with vector and scalar
columns, two tokens to more than a warp of pairs, odd and even lengths, with and without a positional part, both kinds of update, against
the oracle."""
import numpy as np
import pytest

import golden_util
from oracle import lut_oracle as orc
from test_concat_gpu import compare, expand_pe, inputs_for, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("policy", ["dense", "internal"])
@pytest.mark.parametrize("S,Npe", [(2, 2), (3, 0), (8, 2), (33, 3)])
@pytest.mark.parametrize("O", [1, 4, 7, 8, 12, 16, 28, 31, 32, 36, 64])
def test_rows_of_one_step(O, S, Npe, policy):
    cfg = dict(seed=1500 + O, B=60, S=S, E=10, Nt=5, Nc=2, Npe=Npe, O=O)
    if policy == "internal":
        cfg.update(policy="internal", ext_lr=0.03125)
    x, anchors, W, pe, dY = inputs_for(cfg)
    dY[:, :, ::5] = 0.0   # (not part of the table gradient)
    pe3 = expand_pe(cfg, pe)
    y, st = orc.concat_forward(W, x, pe3, anchors, 5, 2, O, Npe)
    dX, dW, dPE = orc.concat_backward(W, dY, anchors, st, 10, 2, Npe, forward_group_size=32)
    ref = dict(y=y, y_eval=y, dX=dX, dPE=dPE, idx=st["idx"], min_k=st["min_k"], min_delta=st["min_delta"],
               pidx=st["pidx"], pmin=st["pmin"], pmin_k=st["pmin_k"])
    got = run_gpu(cfg, x, anchors, W, pe, dY)
    # cells of the tables and of the positional embeddings sum up to n terms in fp32, in different orders on both sides: about
    # sqrt(n) * 2^-24 of the sum for each
    n = 60 * S * (S - 1) / 2
    rel = max(1e-5, 2 * n ** 0.5 * 2.0 ** -24)
    if policy == "internal":
        ref["W_after"] = W - np.float32(cfg["ext_lr"]) * dW.reshape(W.shape)
        # (the update rounds once per term, on a weight of up to |W| beside the sum)
        bound = 0.03125 * rel * np.abs(dW).max() + 2.0 ** -24 * (np.abs(W).max() + 0.03125 * np.abs(dW).max()) * 2 * n ** 0.5
        assert np.abs(got["W_after"].astype(np.float64).reshape(-1) - ref["W_after"].reshape(-1)).max() <= bound
        ref["W_after"] = got["W_after"]
    else:
        golden_util.assert_close(got["dW"], dW, rel, "dW")
        ref["dW"] = got["dW"]
    if Npe:
        golden_util.assert_close(got["dPE"], dPE, rel, "dPE")
        ref["dPE"] = got["dPE"]
    compare(cfg, got, ref)
