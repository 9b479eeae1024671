"""Edges of the staged inference kernels: the ordered anchor lists of the comparison, pairs of detectors in the int8 sums, the
ring of the fp32 kernel."""
import numpy as np
import pytest
import torch

import synth
from oracle import lut_oracle as orc
from test_inference_gpu import make_problem

pytestmark = pytest.mark.gpu


def row_indices(x, anchors, Nc, eps):
    """The oracle's rule on the GPU (the problems are large): bit k set where the difference is above the dead band."""
    idx = torch.zeros(x.shape[0], anchors.shape[0], dtype=torch.int32, device=x.device)
    for k in range(Nc):
        a = anchors[:, k].long()
        used = (a >= 0).all(dim=1)
        d = x[:, a[:, 0].clamp_min(0)] - x[:, a[:, 1].clamp_min(0)]
        up = (d > 0) & used if eps == 0 else (d.abs() >= eps) & (d > 0) & used
        idx |= up.int() << k
    return idx


# a row tile per SM is where the lists start to be used: 8 * 148 rows; rows of 8192 inputs and one past take another kernel (eight of
# them do not fit shared memory: see test_ordered_anchor_lists_of_long_rows)
@pytest.mark.parametrize("shape", [(1184, 8192, 517, 8), (1190, 8193, 517, 8), (1187, 3200, 1030, 6), (2500, 40, 2047, 5), (1200, 33, 513, 1)])
@pytest.mark.parametrize("eps", [0.0, 0.4])
def test_ordered_anchor_lists_give_the_same_indices(shape, eps):
    from spiky_b200.inference import LUTInference

    B, I, Nt, Nc = shape
    g = torch.Generator(device="cuda").manual_seed(B + I)
    x = torch.randint(-3, 4, (B, I), device="cuda", generator=g).float() / 4   # ties, and differences on the dead band's edge
    x[5, ::3] = float("inf")
    x[6, ::2] = float("-inf")
    x[7, ::4] = float("nan")
    x[8] *= 1e-42   # subnormal differences
    anchors = torch.randint(0, I, (Nt, Nc, 2), device="cuda", generator=g, dtype=torch.int32)
    anchors[3, 0] = -1
    anchors[4, Nc - 1, 1] = -1
    anchors[Nt - 1] = I - 1
    O = 36
    layer = LUTInference(I, O, Nt, Nc, anchors, torch.randn(Nt * (1 << Nc) * O, device="cuda", generator=g), cmp_eps=eps)
    y = layer(x)
    idx = row_indices(x, anchors, Nc, np.float32(eps).item())
    assert torch.equal(layer.last_indices, idx)
    W = layer.tables.view(Nt, 1 << Nc, O)
    rows = [0, 5, 6, 7, 8, B // 2, B - 1]
    want = torch.stack([W[torch.arange(Nt, device="cuda"), idx[b].long()].double().sum(0) for b in rows])
    # 12 rows of a run are added in fp32, the runs in double
    assert (y[rows] - want).abs().max() <= 16 * 2.0 ** -24 * want.abs().max() * 12


# eight rows with their anchors' ends in one block of an SM from 3200 inputs on, up to the longest that fit its shared memory, and one past
@pytest.mark.parametrize("inputs", [3201, 5000, 7231, 7232, 7233])
def test_ordered_anchor_lists_of_long_rows(inputs):
    test_ordered_anchor_lists_give_the_same_indices((1187, inputs, 1030, 8), 0.0)


# rows on both sides of where the lists start to be used
@pytest.mark.parametrize("rows", [1000, 1184, 1301])
@pytest.mark.parametrize("eps", [0.0, 0.4])
@pytest.mark.parametrize("tables", ["fp32", "int8"])
def test_zeros_of_both_signs_are_equal(tables, eps, rows):
    """Anchors over inputs that are +0, -0 or a number on either end (the lists may swap the ends): a pair of zeros sets no bit,
    and the same row has the same indices in any batch."""
    from spiky_b200.inference import LUTInference

    I, Nt, Nc, O = 48, 1030, 8, 40   # (int8 lists need rows of eight)
    g = torch.Generator(device="cuda").manual_seed(rows)
    values = torch.tensor([0.0, -0.0, 0.0, -0.0, 0.75, -0.75], device="cuda")
    x = values[torch.randint(0, 6, (rows, I), device="cuda", generator=g)]
    x[::7] = 0.0
    x[::7, ::2] = -0.0
    anchors = torch.randint(0, I, (Nt, Nc, 2), device="cuda", generator=g, dtype=torch.int32)
    W = torch.randn(Nt * (1 << Nc) * O, device="cuda", generator=g)
    if tables == "int8":
        layer = LUTInference(I, O, Nt, Nc, anchors, (W * 40).clamp(-128, 127).to(torch.int8), torch.ones(Nt, device="cuda"), cmp_eps=eps)
    else:
        layer = LUTInference(I, O, Nt, Nc, anchors, W, cmp_eps=eps)
    layer(x)
    idx = layer.last_indices.clone()
    assert torch.equal(idx, row_indices(x, anchors, Nc, np.float32(eps).item()))
    assert not idx[::7].any()
    layer(x[:300])
    assert torch.equal(layer.last_indices, idx[:300])


@pytest.mark.parametrize("block", [1, 2, 5, 32, 255, 1024])
@pytest.mark.parametrize("spread", ["none", "some", "all"])
def test_int8_sums_of_detector_pairs(block, spread):
    """Truncation blocks of odd and even lengths (a pair never crosses one), scales that share an exponent range and blocks of
    scales that do not, in one call; samples past the batch in the last tile."""
    from spiky_b200.inference import LUTInference

    B, I, Nt, Nc, O = 300, 64, 1027, 4, 72
    x, anchors, q, s = make_problem(970 + block, B, I, Nt, Nc, O)
    q[:64] = -128   # the byte without a counterpart
    if spread == "some":
        s[3 * block:4 * block:2] *= np.float32(2.0 ** 9)
    if spread == "all":
        s[::2] *= np.float32(2.0 ** -12)
    s[11] = 0.0
    layer = LUTInference(I, O, Nt, Nc, torch.from_numpy(anchors), torch.from_numpy(q), torch.from_numpy(s), int_rescaler=0.05,
                         backward_group_size=block)
    acc = layer.partial(torch.from_numpy(x).cuda()).cpu().numpy()
    want, ridx = orc.infer_int8(q, s, x, anchors, Nt, Nc, O, backward_group_size=block, int_rescaler=0.05, exact=True)
    assert np.array_equal(layer.last_indices.cpu().numpy(), ridx)
    assert np.array_equal(acc, want)


@pytest.mark.parametrize("shape", [(1, 512, 8, 64), (1025, 513, 1, 36), (2049, 535, 8, 100), (700, 1025, 3, 132)])
def test_fp32_ring(shape):
    """One sample, one past a tile, tables of two rows, an odd detector at the end of a run, column slices that end inside one."""
    from spiky_b200 import _native
    from spiky_b200.inference import LUTInference

    B, Nt, Nc, O = shape
    I = 50
    g = torch.Generator(device="cuda").manual_seed(B)
    x = torch.randn(B, I, device="cuda", generator=g)
    anchors = torch.from_numpy(synth.anchor_pairs(5, Nt, Nc, I)).cuda()
    W = torch.randn(Nt * (1 << Nc) * O, device="cuda", generator=g)
    layer = LUTInference(I, O, Nt, Nc, anchors, W)
    y = layer(x)
    idx = row_indices(x, anchors.view(Nt, Nc, 2), Nc, 0.0)
    assert torch.equal(layer.last_indices, idx)
    want = torch.zeros(B, O, dtype=torch.float64, device="cuda")
    W = W.view(Nt, 1 << Nc, O).double()
    for t in range(Nt):
        want += W[t, idx[:, t].long()]
    assert (y - want).abs().max() <= 16 * 2.0 ** -24 * want.abs().max() * 12
    assert _native.device_wait_errors() == 0
