"""Input gradient of rows that one step of a lane group covers: every group width with vector and scalar columns, detectors one
short of a round of 32, a round, and one past; detectors without a used anchor; added to dX and written."""
import numpy as np
import pytest

from cases import nonseq_fc_inputs
from oracle import lut_oracle as orc
from spiky_b200._native import DX_WRITE
from test_nonseq_fc_gpu import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("write", [0, DX_WRITE], ids=["add", "write"])
@pytest.mark.parametrize("Nt", [31, 32, 33])
@pytest.mark.parametrize("O", [1, 2, 3, 4, 7, 8, 12, 15, 16, 31, 32, 36, 64, 100, 128, 33, 132])
def test_input_gradient_matches_oracle(O, Nt, write):
    cfg = dict(seed=900 + O, B=19, I=40, Nt=Nt, Nc=4, O=O)
    x, anchors, W, dY = nonseq_fc_inputs(cfg)
    # row 0 of the first table is no sample's row and no sample's neighbour (its first bit is always set, with a wide margin):
    # what slots without a detector read there must reach nothing
    x = np.clip(x, -1, 1)
    x[:, 0] = 9.0
    anchors = anchors.reshape(Nt, 4, 2)
    anchors[anchors == 0] = 1
    anchors[0, 0] = (0, 1)
    anchors[5] = -1   # nothing to flip
    W = W.reshape(Nt, 16, O)
    W[0, 0] = np.inf
    W[5, 0] = 1.0
    W[5, 1:] = np.nan
    got = run_gpu(cfg, x, anchors, W.reshape(-1), dY, dw_variant=write)
    y, idx, md, mk = orc.nonseq_fc_forward(W.reshape(-1), x, anchors, Nt, 4, O, 0.0, True, 32)
    assert (idx[:, 0] & 1).all() and (mk[:, 0] != 0).all()
    assert (mk[:, 5] == -1).all()
    W0, k0, pairs = W.copy(), mk.copy(), anchors.copy()   # (the oracle always flips a bit: a table of zeros has no gradient)
    W0[5], k0[:, 5], pairs[5] = 0, 0, 1
    want, _ = orc.nonseq_fc_backward(W0.reshape(-1), dY, pairs, idx, md, k0, 40, 4, 1.0, -1.0, 32)
    # per detector: each product of dY with a difference of rows carries the difference's rounding and at most 4 roundings of a lane's
    # sum; every term then enters a cell of dX with one rounding per term of that cell.  Surrogate |u'| <= 1 / 2.
    bound = np.zeros((19, 40))
    terms = np.zeros((19, 40))
    Wf, dYr, mk, idx = np.where(np.isfinite(W), W, 0.0).astype(np.float64), dY.reshape(19, O).astype(np.float64), mk.reshape(19, Nt), idx.reshape(19, Nt)
    for b in range(19):
        for t in np.flatnonzero(mk[b] >= 0):
            row, alt = Wf[t, idx[b, t]], Wf[t, idx[b, t] ^ (1 << mk[b, t])]
            mass = 0.5 * (np.abs(dYr[b]) * (np.abs(row) + np.abs(alt))).sum()
            for cell in anchors[t, mk[b, t]]:
                bound[b, cell] += mass
                terms[b, cell] += 1
    bound *= 2.0 ** -24 * (5 + terms)
    assert np.isfinite(got["dX"]).all()
    err = np.abs(got["dX"].astype(np.float64) - want.reshape(19, 40))
    assert (err <= bound).all()
    assert np.abs(want).max() > 1e3 * bound.max()
