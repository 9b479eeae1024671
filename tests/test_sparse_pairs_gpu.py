"""Sparse layers whose rows are read two synapses at a time, and runs of samples: row lengths and forward groups on both sides of
the rule, a table array that starts off 8 bytes, batches that end inside a run, against the oracle."""
import numpy as np
import pytest
import torch

import synth
from test_sparse_staged_gpu import check, oracle_layer, run_layer

pytestmark = pytest.mark.gpu


def make(projection, fg, per, batch):
    from spiky_b200.lut_layer import PointSamplingPolicy, PointSamplingType, ProjectionLUTLayer, SynapseMeta

    layer = ProjectionLUTLayer(
        (14, 14), (12, 12), 4, 36, per, (5, 5), projection,
        synapse_meta=SynapseMeta(min_weight=-1.0, max_weight=1.0, initial_noise_level=0.1, initial_weight=-0.05),
        detectors_sampling_policy=PointSamplingPolicy(PointSamplingType.Grid, grid_h=6, grid_w=6, stride_h=2, stride_w=2, pad_h=2, pad_w=2),
        _forward_group_size=fg, random_seed=3, device="cuda:0")
    return layer, synth.sparse_images(5, (batch, 196)), synth.normal(6, (batch, 144))


# rows of 2, 6, 8, 9, 12, 16, 20, 32 synapses; groups that end inside a row: even (pairs), odd (one at a time)
@pytest.mark.parametrize("fg", [3, 6, 32])
@pytest.mark.parametrize("projection", [(1, 2), (2, 3), (2, 4), (3, 3), (3, 4), (4, 4), (4, 5), (4, 8)])
def test_row_lengths_and_groups(projection, fg):
    layer, x, dY = make(projection, fg, 35, 21)   # chunks of 32 and of 3 detectors
    check(run_layer(layer, x, dY), oracle_layer(layer, x, dY, 4), f"{projection} in groups of {fg}")


def test_tables_off_eight_bytes():
    layer, x, dY = make((4, 4), 32, 9, 50)
    want = oracle_layer(layer, x, dY, 4)
    W = layer._weights.data
    moved = torch.empty(W.numel() + 1, device=W.device)[1:]
    moved.copy_(W)
    layer._weights.data = moved
    assert layer._weights.data_ptr() % 8 == 4
    check(run_layer(layer, x, dY), want, "tables off eight bytes")


def test_layers_of_pairs_are_marked():
    assert make((4, 4), 32, 9, 1)[0]._lut_dm._sparse.pair_rows == 1
    assert make((3, 3), 32, 9, 1)[0]._lut_dm._sparse.pair_rows == 0
    assert make((4, 4), 3, 9, 1)[0]._lut_dm._sparse.pair_rows == 0


# one sample a run up to 16 of them, the last run not full
@pytest.mark.parametrize("batch", [1, 793, 1585, 3173, 6341, 12645])
def test_runs_of_samples(batch):
    layer, x, dY = make((4, 4), 32, 9, batch)
    got, want = run_layer(layer, x, dY), oracle_layer(layer, x, dY, 4)
    assert np.array_equal(got["idx"], want["idx"])
    for k in ("y", "y_eval", "dX"):   # the bound of `check`, a sample's sums have the same few terms whatever the batch
        assert np.abs(got[k] - want[k]).max() <= 1e-5 * np.abs(want[k]).max(), k
    # a cell of dW sums up to `batch` values of dY in fp32, in any order
    idx = want["idx"]
    most = max(np.bincount(idx[:, t], minlength=16).max() for t in range(idx.shape[1]))
    assert np.abs(got["dW"].astype(np.float64) - want["dW"]).max() <= 2 * 2.0 ** -24 * most * most * np.abs(dY).max()


@pytest.mark.parametrize("batch", [1, 793, 1585, 3173, 6341, 12645])
def test_table_gradient_of_runs_is_exact(batch):
    """Output gradients on a grid of 2^-6 of which any sum of a batch is an fp32 number: a run of samples that is left out or counted
    twice shows in every cell, whatever the order of the sums."""
    layer, x, dY = make((4, 4), 32, 9, batch)
    dY = np.round(np.clip(dY, -4, 4) * 64) / 64
    dY = dY.astype(np.float32)
    assert batch * 4 * 64 < 2 ** 24
    got, want = run_layer(layer, x, dY), oracle_layer(layer, x, dY, 4)
    assert np.array_equal(got["idx"], want["idx"])
    assert np.abs(want["dW"]).max() > 0 and np.array_equal(got["dW"], want["dW"])
