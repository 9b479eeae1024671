"""CUDA path of the non-sequence fully connected layer, called through the C ABI, against
(1) the golden vectors recorded from the reference and (2) the CPU oracle on larger seeded inputs.

Bar: indices, min-margin anchors, min deltas and every fixed-point (int32) result bit-exact;
fp32 outputs and gradients within 1e-5 of the tensor's scale (summation order only)."""
import numpy as np
import pytest
import torch

import golden_util
import synth
from cases import nonseq_fc_inputs
from oracle import lut_oracle as orc

pytestmark = pytest.mark.gpu
REL = 1e-5


def make_dm(cfg):
    from spiky_b200.lut_data_manager import LUTDataManagerF, LUTDataManagerI

    args = (cfg["I"], cfg["O"], cfg["Nt"], cfg["Nc"], 1, 0, 0, cfg.get("G", 32), cfg.get("Gb", 32))
    dm = LUTDataManagerI(*args, cfg.get("int_rescaler", 0.001)) if cfg.get("int_mode") else LUTDataManagerF(*args)
    dm.register_synapse_meta(learning_rate=cfg.get("lr_meta", 1.0), min_synaptic_weight=-1.0, max_synaptic_weight=1.0,
                             initial_noise_level=0.0, initial_weight=0.0)
    dm.initialize_neurons(True)
    dm.to_device(0)
    return dm


def run_gpu(cfg, x, anchors, W, dY, dw_variant=0):
    dev = torch.device("cuda:0")
    dm = make_dm(cfg)
    B, I, Nt, O = cfg["B"], cfg["I"], cfg["Nt"], cfg["O"]
    tW = torch.from_numpy(W).to(dev)
    tx = torch.from_numpy(x).reshape(-1).to(dev)
    ta = torch.from_numpy(anchors).reshape(-1).to(dev)
    eps = cfg.get("cmp_eps", 0.0)
    out = {}
    y_eval = torch.zeros(B * O, device=dev)
    idx_eval = torch.zeros(B * Nt, dtype=torch.int32, device=dev)
    dm.forward_step(tW, B, tx, ta, y_eval, idx_eval, eps, None, None, None)
    y = torch.zeros(B * O, device=dev)
    idx = torch.zeros(B * Nt, dtype=torch.int32, device=dev)
    md = torch.zeros(B * Nt, device=dev)
    mk = torch.zeros(B * Nt, dtype=torch.int32, device=dev)
    dm.forward_step(tW, B, tx, ta, y, idx, eps, None, md, mk)
    dX = torch.zeros(B * I, device=dev)
    internal = cfg.get("policy") == "internal"
    dW = None if internal else torch.zeros_like(tW)
    dm.backward_backprop(tW, B, torch.from_numpy(dY).reshape(-1).to(dev), ta, idx, md, mk, dX,
                         cfg["ext_lr"] if internal else -1.0, dW, None, dw_variant=dw_variant)
    torch.cuda.synchronize()
    out.update(y_eval=y_eval.cpu().numpy().reshape(B, O), idx_eval=idx_eval.cpu().numpy().reshape(B, Nt),
               y=y.cpu().numpy().reshape(B, O), idx=idx.cpu().numpy().reshape(B, Nt),
               min_delta=md.cpu().numpy().reshape(B, Nt), min_k=mk.cpu().numpy().reshape(B, Nt),
               dX=dX.cpu().numpy().reshape(B, I))
    if internal:
        out["W_after"] = tW.cpu().numpy()
    else:
        out["dW"] = dW.cpu().numpy()
    return out


def compare(cfg, got, ref):
    assert np.array_equal(got["idx"], ref["idx"]) and np.array_equal(got["idx_eval"], ref["idx"])
    assert np.array_equal(got["min_k"], ref["min_k"])
    assert np.array_equal(got["min_delta"].view(np.int32), ref["min_delta"].view(np.int32))
    keys = ["y", "y_eval", "dX"] + (["W_after"] if "W_after" in ref else ["dW"])
    for k in keys:
        if cfg.get("int_mode"):
            assert np.array_equal(got[k], ref[k]), f"{k}: fixed-point results must be bit-exact"
        else:
            golden_util.assert_close(got[k], ref[k], REL, k)


@pytest.mark.parametrize("name", golden_util.names("fc_"))
def test_nonseq_fc_matches_reference_golden(name):
    cfg, ref = golden_util.load(name)
    x, anchors, W, dY = nonseq_fc_inputs(cfg)
    compare(cfg, run_gpu(cfg, x, anchors, W, dY), ref)


def oracle_reference(cfg, x, anchors, W, dY):
    kw = dict(int_mode=cfg.get("int_mode", False), int_rescaler=cfg.get("int_rescaler", 0.001))
    y, idx, md, mk = orc.nonseq_fc_forward(W, x, anchors, cfg["Nt"], cfg["Nc"], cfg["O"], cfg.get("cmp_eps", 0.0),
                                           True, cfg.get("Gb", 32), **kw)
    dX, dW = orc.nonseq_fc_backward(W, dY, anchors, idx, md, mk, cfg["I"], cfg["Nc"], cfg.get("lr_meta", 1.0), -1.0,
                                    cfg.get("G", 32), **kw)
    return dict(y=y, y_eval=y, idx=idx, min_delta=md, min_k=mk, dX=dX, dW=dW)


ORACLE_CASES = {
    # the single-layer benchmark configuration at full size (batch 256 x 784 -> 64 tables x 6 pairs -> 32)
    "c1_full_f32": dict(seed=500, B=256, I=784, Nt=64, Nc=6, O=32),
    "c1_full_i32": dict(seed=501, B=256, I=784, Nt=64, Nc=6, O=32, int_mode=True),
    "c1_sparse_images": dict(seed=502, B=64, I=784, Nt=64, Nc=6, O=32, sparse_input=True),
    # output rows wider than one warp pass, table of 256 rows, odd batch
    "ffn_like": dict(seed=503, B=67, I=256, Nt=16, Nc=8, O=1024),
    "ffn_like_i32": dict(seed=504, B=33, I=256, Nt=16, Nc=8, O=640, int_mode=True, int_rescaler=0.01),
    # outputs not a multiple of 4 (scalar path), many detectors
    "ragged": dict(seed=505, B=19, I=333, Nt=150, Nc=5, O=10),
    "ragged_i32": dict(seed=506, B=19, I=333, Nt=150, Nc=5, O=10, int_mode=True, G=3, Gb=7),
    # every lane-group width of the vectorised forward gather: 1, 2, 4, 8 (c1), 16 (c5), 32 float4 per row, two chunks
    "rows_of_4": dict(seed=510, B=37, I=64, Nt=45, Nc=5, O=4),
    "rows_of_8": dict(seed=511, B=37, I=64, Nt=45, Nc=5, O=8),
    "rows_of_16": dict(seed=512, B=37, I=64, Nt=45, Nc=5, O=16),
    "rows_of_128": dict(seed=513, B=21, I=64, Nt=33, Nc=5, O=128),
    "rows_of_260": dict(seed=514, B=21, I=64, Nt=33, Nc=5, O=260),
    # one sample; more detectors than threads of a row group; inputs not a multiple of 4
    "one_sample": dict(seed=515, B=1, I=50, Nt=300, Nc=7, O=12),
    "odd_inputs": dict(seed=516, B=13, I=4099, Nt=64, Nc=8, O=32, normal_input=True),
    # input rows so long that fewer rows are staged together (2, then 1), and rows that do not fit shared memory at all
    "inputs_10k": dict(seed=517, B=5, I=10001, Nt=20, Nc=5, O=8, normal_input=True),
    "inputs_20k": dict(seed=518, B=3, I=20002, Nt=20, Nc=5, O=8, normal_input=True),
    "inputs_60k": dict(seed=519, B=3, I=60001, Nt=20, Nc=5, O=8, normal_input=True),
    # a slice of the large inference layer (4096 inputs, 8 pairs, 64 outputs)
    "c5_slice": dict(seed=507, B=40, I=4096, Nt=512, Nc=8, O=64, normal_input=True),
    "nan_inputs": dict(seed=508, B=8, I=32, Nt=8, Nc=4, O=8, nan_input=True),
}


@pytest.mark.parametrize("name", sorted(ORACLE_CASES))
def test_nonseq_fc_matches_oracle(name):
    cfg = ORACLE_CASES[name]
    x, anchors, W, dY = nonseq_fc_inputs(cfg)
    if cfg.get("nan_input"):
        x[:, 3] = np.nan  # NaN deltas: bit 0, never the minimum unless first (reference compare semantics)
    ref = oracle_reference(cfg, x, anchors, W, dY)
    got = run_gpu(cfg, x, anchors, W, dY)
    if cfg.get("nan_input"):
        assert np.array_equal(got["idx"], ref["idx"]) and np.array_equal(got["min_k"], ref["min_k"])
        return
    compare(cfg, got, ref)


def test_large_batch_properties():
    """Full-size batch of the single-layer configuration: size-independent properties.
    (1) duplicating the batch doubles dW and leaves per-sample outputs unchanged;
    (2) dX rows sum to zero (+du and -du per detector); (3) two runs give identical indices."""
    cfg = dict(seed=600, B=8192, I=784, Nt=64, Nc=6, O=32)
    x, anchors, W, dY = nonseq_fc_inputs(cfg)
    a = run_gpu(cfg, x, anchors, W, dY)
    cfg2 = dict(cfg, B=2 * cfg["B"])
    b = run_gpu(cfg2, np.concatenate([x, x]), anchors, W, np.concatenate([dY, dY]))
    assert np.array_equal(b["idx"][: cfg["B"]], a["idx"]) and np.array_equal(b["idx"][cfg["B"]:], a["idx"])
    golden_util.assert_close(b["y"][: cfg["B"]], a["y"], 1e-6, "y")
    golden_util.assert_close(b["dW"], 2.0 * a["dW"], REL, "dW linearity")
    assert np.abs(a["dX"].astype(np.float64).sum(axis=1)).max() <= 1e-4 * np.abs(a["dX"]).max()
    sample = slice(0, 64)
    ref = oracle_reference(dict(cfg, B=64), x[sample], anchors, W, dY[sample])
    assert np.array_equal(a["idx"][sample], ref["idx"])
    golden_util.assert_close(a["y"][sample], ref["y"], REL, "y vs oracle")
    golden_util.assert_close(a["dX"][sample], ref["dX"], REL, "dX vs oracle")


def test_runtime_errors_mirror_reference():
    dm = make_dm(dict(I=8, O=4, Nt=4, Nc=2))
    dev = torch.device("cuda:0")
    w = torch.zeros(4 * 4 * 4, device=dev)
    with pytest.raises(RuntimeError):  # dtype mismatch -> RuntimeError like checkTensor
        dm.forward_step(w, 1, torch.zeros(8, device=dev, dtype=torch.float64), torch.zeros(16, dtype=torch.int32, device=dev),
                        torch.zeros(4, device=dev), torch.zeros(4, dtype=torch.int32, device=dev))
    with pytest.raises(ValueError):  # backward before any forward -> "no active context"
        dm.backward_backprop(w, 1, torch.zeros(4, device=dev), torch.zeros(16, dtype=torch.int32, device=dev),
                             torch.zeros(4, dtype=torch.int32, device=dev), torch.zeros(4, device=dev),
                             torch.zeros(4, dtype=torch.int32, device=dev), torch.zeros(8, device=dev), -1.0,
                             torch.zeros_like(w))
    with pytest.raises(ValueError):
        dm.forward_step(w, 0, torch.zeros(8, device=dev), torch.zeros(16, dtype=torch.int32, device=dev),
                        torch.zeros(4, device=dev), torch.zeros(4, dtype=torch.int32, device=dev))


@pytest.mark.parametrize("name", ["c1_full_f32", "ragged", "ffn_like"])
def test_sorted_table_gradient_is_bit_exact_and_deterministic(name):
    """LUTB_DW_SORTED adds every cell's contributions in ascending sample order with one fp32 rounding each,
    the order of the reference's host loop: dW equals the oracle's bit for bit, run after run."""
    cfg = ORACLE_CASES[name]
    x, anchors, W, dY = nonseq_fc_inputs(cfg)
    ref = oracle_reference(cfg, x, anchors, W, dY)
    a = run_gpu(cfg, x, anchors, W, dY, dw_variant=3)
    b = run_gpu(cfg, x, anchors, W, dY, dw_variant=3)
    assert np.array_equal(a["dW"], ref["dW"])
    assert np.array_equal(a["dW"], b["dW"])
    golden_util.assert_close(a["dX"], ref["dX"], REL, "dX")


def test_sorted_variant_rejects_missing_workspace():
    import ctypes
    from spiky_b200 import _native

    dm = make_dm(dict(I=8, O=4, Nt=4, Nc=2))
    cfg = dm._cfg()
    L = _native.lib()
    need = L.lutb_nonseq_fc_backward_workspace(ctypes.byref(cfg), 16, 3)
    assert need > 0 and L.lutb_nonseq_fc_backward_workspace(ctypes.byref(cfg), 16, 1) == 0
    dev = torch.device("cuda:0")
    t = lambda n, dt=torch.float32: torch.zeros(n, dtype=dt, device=dev)
    p = lambda z: ctypes.c_void_p(z.data_ptr())
    rc = L.lutb_nonseq_fc_backward(ctypes.byref(cfg), 16, p(t(64)), p(t(64)), p(t(16, torch.int32)), p(t(64, torch.int32)),
                                   p(t(64)), p(t(64, torch.int32)), p(t(128)), p(t(64)), -1.0, 3, None, 0, None)
    assert rc == -4 and b"workspace" in L.lutb_last_error()


@pytest.mark.parametrize("rows,I,Nt,Nc", [(1, 5, 1, 1), (8, 64, 33, 6), (9, 63, 257, 7), (700, 100, 300, 2), (2403, 30, 390, 6),
                                          (2500, 40, 24, 3), (8, 3200, 40, 4), (17, 3201, 40, 5), (19, 4096, 600, 8),
                                          (520, 4096, 770, 6), (523, 7232, 769, 7), (523, 7233, 769, 7), (17, 6400, 40, 5),
                                          (17, 6401, 40, 3), (400, 6401, 450, 6), (5, 9000, 31, 8)])
def test_check_detectors_row_and_detector_splits(rows, I, Nt, Nc):
    """Eight rows with one or two threads a detector (in one or two blocks per SM; 3200 and 7232 inputs are the longest that
    leave room for two and for one), fewer rows for longer inputs, anchor lists read two at a time or one by one, unused
    anchor pairs, an input that is not 16-byte aligned."""
    import ctypes
    from spiky_b200 import _native

    x = synth.normal(960, (rows, I))
    anchors = synth.anchor_pairs(961, Nt, Nc, max(I, 2)).reshape(Nt, Nc, 2).copy()
    if Nc > 2:
        anchors[::3, 1] = -1
    cfg = _native.LayerCfg(n_inputs=I, n_outputs=4, n_detectors=Nt, n_anchors=Nc, seq_len=1, pos_dim=0, forward_group=32,
                           backward_group=32, int_mode=0, sliced_product=0, cmp_eps=0.0, reserved0=0.0, int_rescaler=1.0,
                           lr_meta=1.0)
    ridx, rmd, rmk = orc.check_detectors(x, anchors.reshape(-1), Nt, Nc, 0.0, True)
    ta = torch.from_numpy(anchors.reshape(-1)).cuda()
    for shift in (0, 1):
        store = torch.zeros(rows * I + shift, device="cuda")
        tx = store[shift:]
        tx.copy_(torch.from_numpy(x).reshape(-1))
        idx = torch.empty(rows * Nt, dtype=torch.int32, device="cuda")
        md, mk = torch.empty(rows * Nt, device="cuda"), torch.empty_like(idx)
        p = [ctypes.c_void_p(t.data_ptr()) for t in (tx, ta, idx, md, mk)]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        L = _native.lib()
        _native.check(L.lutb_check_detectors(ctypes.byref(cfg), rows, p[0], p[1], p[2], p[3], p[4], stream))
        assert np.array_equal(idx.cpu().numpy(), ridx.reshape(-1)) and np.array_equal(mk.cpu().numpy(), rmk.reshape(-1))
        assert np.array_equal(md.cpu().numpy().view(np.int32), rmd.reshape(-1).view(np.int32))
        idx.fill_(-7)
        _native.check(L.lutb_check_detectors(ctypes.byref(cfg), rows, p[0], p[1], p[2], None, None, stream))
        assert np.array_equal(idx.cpu().numpy(), ridx.reshape(-1))


@pytest.mark.parametrize("B,I,Nt,Nc,O", [(1, 7, 1, 1, 1), (9, 33, 5, 4, 4), (70, 100, 33, 6, 12), (600, 50, 70, 5, 33),
                                         (2400, 64, 64, 6, 32), (2403, 37, 16, 8, 64), (2500, 2052, 20, 3, 132),
                                         (2400, 63, 40, 4, 5), (19000, 24, 9, 4, 8), (2500, 40, 40, 4, 1), (33, 40, 40, 4, 2),
                                         (2500, 60, 35, 4, 2), (2500, 60, 35, 4, 3)])
def test_input_gradient_kernel_splits(B, I, Nt, Nc, O):
    """Lane groups of every width, rows of several steps, few samples (32 detectors a block) and many; the input gradient
    added to what is there and written over what is there (with rows that fit shared memory and longer ones)."""
    import ctypes
    from spiky_b200 import _native

    x = synth.normal(970, (B, I))
    anchors = synth.anchor_pairs(971, Nt, Nc, I)
    W = synth.normal(972, (Nt * (1 << Nc) * O,), 0.0, 0.05)
    dY = synth.normal(973, (B, O))
    _, idx, md, mk = orc.nonseq_fc_forward(W, x, anchors, Nt, Nc, O)
    want, dW = orc.nonseq_fc_backward(W, dY, anchors, idx, md, mk, I, Nc)
    cfg = _native.LayerCfg(n_inputs=I, n_outputs=O, n_detectors=Nt, n_anchors=Nc, seq_len=1, pos_dim=0, forward_group=32,
                           backward_group=32, int_mode=0, sliced_product=0, cmp_eps=0.0, reserved0=0.0, int_rescaler=1.0,
                           lr_meta=1.0)
    tW, tdY, ta, ti, tm, tk = [torch.from_numpy(np.ascontiguousarray(v)).reshape(-1).cuda() for v in (W, dY, anchors, idx, md, mk)]
    L, stream = _native.lib(), torch.cuda.current_stream().cuda_stream
    for variant, start in ((0, 1.0), (_native.DX_WRITE, float("nan"))):
        dX, gW = torch.full((B * I,), start, device="cuda"), torch.zeros_like(tW)
        _native.check(L.lutb_nonseq_fc_backward(ctypes.byref(cfg), B, tW.data_ptr(), tdY.data_ptr(), ta.data_ptr(), ti.data_ptr(),
                                                tm.data_ptr(), tk.data_ptr(), dX.data_ptr(), gW.data_ptr(), -1.0, variant, None, 0,
                                                stream))
        got = dX.cpu().numpy().reshape(B, I)
        if variant == 0:
            # (adding to 1 rounds every partial sum at 2^-24)
            assert np.abs(got - 1.0 - want).max() <= 1e-5 * np.abs(want).max() + 2.0 ** -24 * 4 * Nt
        else:
            golden_util.assert_close(got, want, 1e-5, "dX")
        if B < 10000:
            golden_util.assert_close(gW.cpu().numpy(), dW.reshape(-1), 1e-5, "dW")


@pytest.mark.parametrize("B,O", [(21, O) for O in (1, 2, 3, 7, 10, 17, 31, 33, 45, 63, 65, 130, 4, 36, 132)] +
                         [(900, 65), (900, 127), (900, 131), (5, 16385)])
def test_forward_gather_widths(B, O):
    """Rows of every lane group, one, two and four columns a lane, several column chunks, aligned and not; detectors that end
    inside a group of 32."""
    from spiky_b200.lut_data_manager import LUTDataManagerF

    I, Nt, Nc = 40, 37, 4
    x = synth.normal(980, (B, I))
    anchors = synth.anchor_pairs(981, Nt, Nc, I)
    W = synth.normal(982, (Nt * (1 << Nc) * O,), 0.0, 0.05)
    want, idx, md, mk = orc.nonseq_fc_forward(W, x, anchors, Nt, Nc, O)
    dm = LUTDataManagerF(I, O, Nt, Nc, 1, 0, 0, 32, 32)
    dm.register_synapse_meta(1.0, -1.0, 1.0, 0.0, 0.0)
    dm.initialize_neurons(True)
    dm.to_device(0)
    y = torch.zeros(B * O, device="cuda")
    ti = torch.empty(B * Nt, dtype=torch.int32, device="cuda")
    dm.forward_step(torch.from_numpy(W).cuda(), B, torch.from_numpy(x).reshape(-1).cuda(),
                    torch.from_numpy(anchors).reshape(-1).cuda(), y, ti)
    assert np.array_equal(ti.cpu().numpy(), idx.reshape(-1))
    golden_util.assert_close(y.cpu().numpy().reshape(B, O), want, 1e-5, "y")


def test_forward_gather_of_very_wide_scalar_rows():
    """More columns than a grid has chunks of 32 for: two samples, one detector, 2.1 M outputs that are no multiple of four."""
    from spiky_b200.lut_data_manager import LUTDataManagerF

    O = 65535 * 32 + 5
    dm = LUTDataManagerF(4, O, 1, 1, 1, 0, 0, 32, 32)
    dm.register_synapse_meta(1.0, -1.0, 1.0, 0.0, 0.0)
    dm.initialize_neurons(True)
    dm.to_device(0)
    W = torch.randn(2 * O, device="cuda")
    x = torch.tensor([1.0, 0.0, 0.0, 0.0, -1.0, 0.0, 0.0, 0.0], device="cuda")
    y, idx = torch.zeros(2 * O, device="cuda"), torch.empty(2, dtype=torch.int32, device="cuda")
    dm.forward_step(W, 2, x, torch.tensor([0, 1], dtype=torch.int32, device="cuda"), y, idx)
    assert idx.tolist() == [1, 0]
    assert torch.equal(y.view(2, O), W.view(2, O).flip(0))


def test_input_gradient_of_very_many_detectors():
    """More groups of 32 detectors than a grid has rows (few samples): 2.1 M detectors of two rows."""
    import ctypes
    from spiky_b200 import _native

    B, I, Nt = 2, 5000, 65535 * 32 + 33
    g = torch.Generator(device="cuda").manual_seed(3)
    W = torch.randn(Nt, 2, 4, device="cuda", generator=g)
    dY = torch.randn(B, 4, device="cuda", generator=g)
    first = torch.randint(0, I, (Nt,), device="cuda", generator=g)
    anchors = torch.stack([first, (first + 1) % I], 1).int().contiguous()
    idx = torch.randint(0, 2, (B, Nt), device="cuda", generator=g, dtype=torch.int32)
    md = torch.randn(B, Nt, device="cuda", generator=g)
    mk = torch.zeros(B, Nt, dtype=torch.int32, device="cuda")
    dX = torch.zeros(B, I, device="cuda")
    cfg = _native.LayerCfg(n_inputs=I, n_outputs=4, n_detectors=Nt, n_anchors=1, seq_len=1, pos_dim=0, forward_group=32,
                           backward_group=32, int_mode=0, sliced_product=0, cmp_eps=0.0, reserved0=0.0, int_rescaler=1.0,
                           lr_meta=1.0)
    _native.check(_native.lib().lutb_nonseq_fc_backward(
        ctypes.byref(cfg), B, W.data_ptr(), dY.data_ptr(), anchors.data_ptr(), idx.data_ptr(), md.data_ptr(), mk.data_ptr(),
        dX.data_ptr(), None, _native.SKIP_TABLE_GRADIENT, 0, None, 0, torch.cuda.current_stream().cuda_stream))
    sign = 2.0 * idx.double() - 1.0
    dot = sign * torch.einsum("bo,to->bt", dY.double(), (W[:, 1] - W[:, 0]).double())
    du = torch.where(md > 0, 0.5, -0.5) / (1.0 + md.double().abs()) ** 2 * dot
    want = torch.zeros(B, I, dtype=torch.float64, device="cuda")
    for b in range(B):
        want[b].index_add_(0, anchors[:, 0].long(), du[b])
        want[b].index_add_(0, anchors[:, 1].long(), -du[b])
    # a cell sums about 840 fp32 terms
    golden_util.assert_close(dX.cpu().numpy(), want.cpu().numpy(), 1e-5, "dX")
