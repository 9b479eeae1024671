"""Workspace of the row-list table gradient: one that is sized for the largest batch does for every smaller one."""
import ctypes

import pytest

from spiky_b200 import _native


@pytest.mark.parametrize("detectors,anchors", [(50, 7), (64, 6), (16, 8), (9, 1), (3, 11), (3, 12)])
def test_row_list_workspace_grows_with_the_batch(detectors, anchors):
    cfg = _native.LayerCfg(n_inputs=30, n_outputs=33, n_detectors=detectors, n_anchors=anchors, seq_len=1, forward_group=32, backward_group=32,
                           int_rescaler=1.0, lr_meta=1.0)
    short = 2048 // (1 << anchors) * 128   # up to here the sort takes short slices
    batches = sorted({b for c in (1, 128, 256, 1024, short, 2 * short, 4096, 1 << 17) for b in range(max(1, c - 2), c + 130)})
    need = [_native.lib().lutb_nonseq_fc_table_grad_rows_workspace(ctypes.byref(cfg), b) for b in batches]
    assert all(n > 0 for n in need)
    assert need == sorted(need)
