"""Product-mode layers on two streams at once: the results of a run one after the other."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("native", [True, False], ids=["native", "python"])
@pytest.mark.parametrize("kept", [True, False], ids=["kept", "counted_again"])
def test_layers_on_two_streams(native, kept):
    from spiky_b200.lut_data_manager import _LUTDataManager
    from spiky_b200.lut_layer import LUTLayer, SynapseMeta

    layers, xs = [], []
    for k in range(2):
        layer = LUTLayer(64, 8, 16, 64, sequence_length=160, concatenation_product=False, positional_dim=2,
                         synapse_meta=SynapseMeta(min_weight=-1.0, max_weight=1.0), random_seed=3 + k, device="cuda:0")
        with torch.no_grad():
            layer._weights.normal_(0.0, 0.3, generator=torch.Generator(device="cuda").manual_seed(k))
        if not native:
            layer.backward_step = layer.backward_step   # (a replaced method selects the Python route)
        layers.append(layer)
        xs.append(torch.rand((16, 160, 64), device="cuda", generator=torch.Generator(device="cuda").manual_seed(9 + k)))
    dy = torch.linspace(-1.0, 1.0, 16 * 160 * 64, device="cuda").view(16, 160, 64)

    def one(k):
        x = xs[k].clone().requires_grad_()
        layers[k]._weights.grad = layers[k]._positional_embeddings.grad = None
        y = layers[k](x)
        y.backward(dy)
        return [y.detach(), x.grad, layers[k]._weights.grad, layers[k]._positional_embeddings.grad]

    saved = _LUTDataManager.product_keep_limit
    if not kept:
        _LUTDataManager.product_keep_limit = 0
    try:
        want = [one(k) for k in range(2)]
        streams = [torch.cuda.Stream() for _ in range(2)]
        for _ in range(5):
            for s in streams:
                s.wait_stream(torch.cuda.current_stream())
            got = []
            for k, s in enumerate(streams):
                with torch.cuda.stream(s):
                    got.append(one(k))
            for s in streams:
                torch.cuda.current_stream().wait_stream(s)
            torch.cuda.synchronize()
            for a, b in zip(got, want):
                assert torch.equal(a[0], b[0]) and torch.equal(a[2], b[2])   # (no sums in any order there)
                for u, v in zip(a[1:], b[1:]):
                    assert (u - v).abs().max() <= 1e-5 * v.abs().max()
    finally:
        _LUTDataManager.product_keep_limit = saved
