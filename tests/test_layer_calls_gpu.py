"""The native host side of layer calls (host/layer_calls.cpp) against the Python route, which an instance attribute that
replaces one of the layer's methods selects."""
import gc
import weakref

import pytest
import torch

pytestmark = pytest.mark.gpu

KINDS = ["fc", "fc_sparse_policy", "fc_internal", "projection", "projection_internal", "concat", "concat_no_pe", "concat_unified",
         "product", "product_no_pe", "product_unified", "product_sliced"]


def make(kind, seed=3):
    from spiky_b200.lut_layer import GradientPolicy, GradientType, LUTLayer, PointSamplingPolicy, PointSamplingType, ProjectionLUTLayer, SynapseMeta
    policy = GradientPolicy(GradientType.Internal if "internal" in kind else GradientType.Sparse if "sparse_policy" in kind else GradientType.Dense)
    meta = dict(synapse_meta=SynapseMeta(min_weight=-1.0, max_weight=1.0), weights_gradient_policy=policy, random_seed=seed, device="cuda:0")
    if kind.startswith("projection"):
        layer = ProjectionLUTLayer((14, 14), (10, 10), 4, 9, 3, (5, 5), (3, 3),
                                   detectors_sampling_policy=PointSamplingPolicy(PointSamplingType.RandomUniform), **meta)
        shape = (6, 1, 14, 14)
    elif kind.startswith("fc"):
        layer, shape = LUTLayer(20, 5, 9, 12, **meta), (6, 1, 20)
    else:
        npe = 0 if "no_pe" in kind else 20 if "sliced" in kind else 2
        layer = LUTLayer(20, 4, 5, 12, sequence_length=9, concatenation_product=kind.startswith("concat"), positional_dim=npe,
                         unified_pe="unified" in kind or "sliced" in kind, sliced_product_mode="sliced" in kind, **meta)
        shape = (3, 9, 20)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        layer._weights.normal_(0.0, 0.3, generator=gen)
    if "internal" in kind:
        layer.set_external_learning_rate_hook(lambda w: 0.125)
    return layer, torch.rand(shape, device="cuda", generator=gen), gen


def python_route(layer):
    layer.backward_step = layer.backward_step
    return layer


def passed(layer, x, dy=None, gen=None, grad_x=True):
    x = x.detach().requires_grad_(grad_x)
    y = layer(x)
    if dy is None:
        dy = torch.randn(y.shape, device="cuda", generator=gen)
    y.backward(dy)
    out = [y.detach(), x.grad] + [None if p.grad is None else p.grad.to_dense() for p in layer.parameters()] + [p.detach() for p in layer.parameters()]
    return out, dy


def close(a, b):
    assert (a is None) == (b is None)
    if a is not None:
        assert a.shape == b.shape and (a - b).abs().max() <= 1e-5 * max(b.abs().max().item(), 1e-30)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("how", ["plain", "strided", "no_input_gradient", "evaluation"])
def test_native_route_equals_the_python_route(kind, how):
    layer, x, gen = make(kind)
    other = python_route(make(kind)[0])
    if how == "strided":
        x = torch.cat([x, x + 1], dim=-1)[..., ::2]
        assert not x.is_contiguous()
    if how == "evaluation":
        with torch.no_grad():
            close(layer.eval()(x), other.eval()(x))   # (concatenation mode adds its outputs up in L2, in any order)
        return
    a, dy = passed(layer, x, gen=gen, grad_x=how != "no_input_gradient")
    b, _ = passed(other, x, dy, grad_x=how != "no_input_gradient")
    for u, v in zip(a, b):
        close(u, v)
    with torch.no_grad():   # training mode without a graph
        close(layer(x), other(x))


@pytest.mark.parametrize("kind", ["fc", "projection", "concat", "product"])
def test_graph_machinery(kind):
    layer, x, gen = make(kind)
    other = python_route(make(kind)[0])
    packed = []
    for l in (layer, other):
        seen = []

        def pack(t):
            seen.append(tuple(t.shape))
            return t.clone()
        xs = x.detach().requires_grad_()
        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
            y = l(xs)
        packed.append(seen)
        assert type(y.grad_fn).__name__ and y.grad_fn.name().startswith("_LUTFunctionBackward")
        dy = torch.ones_like(y)
        g1, = torch.autograd.grad(y, xs, dy, retain_graph=True)
        g2, = torch.autograd.grad(y, xs, dy)
        close(g2, g1)
        with pytest.raises(RuntimeError, match="second time"):
            torch.autograd.grad(y, xs, dy)
    assert packed[0] == packed[1] and len(packed[0]) > 0
    # an input changed in place after the forward pass is noticed
    xs = (x.detach() + 0).requires_grad_() * 1.0
    y = layer(xs)
    xs.add_(1.0)
    with pytest.raises(RuntimeError, match="inplace"):
        y.sum().backward()


def test_what_was_refused_stays_refused():
    layer, x, gen = make("fc")
    with pytest.raises(ValueError):
        layer(x[..., :7])
    with pytest.raises(AssertionError):
        layer(x.cpu())
    with pytest.raises(RuntimeError):
        layer(x.double())
    with pytest.raises(ValueError, match="batch_size"):
        layer(x[:0])
    with pytest.raises(RuntimeError):
        torch.vmap(layer)(x.unsqueeze(0))
    internal, xi, _ = make("fc_internal")
    internal._external_lr_hook = None
    with pytest.raises(ValueError, match="external_learning_rate_hook"):
        internal(xi.requires_grad_()).sum().backward()
    with pytest.raises(RuntimeError):
        with torch.autograd.forward_ad.dual_level():
            layer(torch.autograd.forward_ad.make_dual(x.detach(), torch.ones_like(x)))


def test_replaced_parts_are_called():
    """Replaced methods and hooks, also those set between the two passes."""
    layer, x, gen = make("fc")
    called = []
    y = layer(x)
    real = layer.backward_step
    layer.backward_step = lambda *a, **k: (called.append("backward"), real(*a, **k))[1]
    y.sum().backward()
    layer._set_lookup_indices_callback(lambda *a: called.append("indices"))
    layer(x)
    dm, layer.backward_step = layer._lut_dm, real
    forward = dm.forward_step
    dm.forward_step = lambda *a, **k: (called.append("manager"), forward(*a, **k))[1]
    layer(x)
    assert [c for c in called if c != "indices"] == ["backward", "manager"] and called.count("indices") == 2


def test_product_histogram_crosses_between_the_routes():
    """What a native forward pass leaves is found by a Python backward pass, and the other way round."""
    want = None
    for first, second in ((False, False), (False, True), (True, False), (True, True)):
        layer, x, gen = make("product")
        x = x.requires_grad_()
        dy = torch.ones(3, 9, 12, device="cuda")
        if first:
            python_route(layer)
        y = layer(x)
        assert layer._lut_dm._kept_histogram is not None
        layer.__dict__.pop("backward_step", None)
        if second:
            python_route(layer)
        y.backward(dy)
        assert layer._lut_dm._kept_histogram is None
        got = [x.grad, layer._weights.grad, layer._positional_embeddings.grad]
        want = want or got
        for u, v in zip(got, want):
            close(u, v)


@pytest.mark.parametrize("route", [lambda layer: layer, python_route], ids=["native", "python"])
@pytest.mark.parametrize("way", ["strided", "offloaded", "other_stream"])
def test_a_kept_histogram_is_of_its_own_call(route, way):
    """Two forward passes, then the backward pass of the first one: the histogram that the second left is of other inputs, also where
    the inputs that a pass reads are copies whose memory is free again after it."""
    xs = [make("product")[1], make("product", seed=4)[1]]
    dy = torch.linspace(-1.0, 1.0, 3 * 9 * 12, device="cuda").view(3, 9, 12)

    def graph(layer, x):
        if way == "strided":
            wide = torch.empty(3, 9, 40, device="cuda")
            wide[..., ::2] = x
            return layer(wide[..., ::2].requires_grad_())
        if way == "offloaded":   # what comes back lies wherever there is room
            with torch.autograd.graph.save_on_cpu():
                return layer(x.clone().requires_grad_())
        return layer(x.clone().requires_grad_())

    want = route(make("product")[0])
    graph(want, xs[0]).backward(dy)
    layer = route(make("product")[0])
    y = graph(layer, xs[0])
    if way == "other_stream":
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            graph(layer, xs[0])
        torch.cuda.current_stream().wait_stream(s)
    else:
        with torch.no_grad():
            graph(layer, xs[1])
    y.backward(dy)
    close(layer._weights.grad, want._weights.grad)
    close(layer._positional_embeddings.grad, want._positional_embeddings.grad)
    assert layer._lut_dm._kept_histogram is None   # and nothing of the inputs is kept after it


def test_a_kept_histogram_keeps_no_graph():
    layer, x, gen = make("product")
    for route in (layer, python_route(make("product")[0])):
        class Mark(torch.autograd.Function):
            @staticmethod
            def forward(ctx, x, mark):
                ctx.mark = mark
                return x.clone()

        mark = type("Mark", (), {})()
        alive = weakref.ref(mark)
        y = route(Mark.apply(x.clone().requires_grad_(), mark))
        assert route._lut_dm._kept_histogram is not None
        del y, mark
        gc.collect()
        assert alive() is None


def test_native_route_after_a_transform():
    layer, x, gen = make("fc")
    torch.vmap(lambda t: t + 1)(x)
    assert not isinstance(layer(x.requires_grad_()).grad_fn, torch.autograd.function.BackwardCFunction)   # (the Python route's node)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: layer(t).sum())(x)   # as before any of it: the Python route's answer while one is active


@pytest.mark.parametrize("kind", KINDS)
def test_a_layer_that_keeps_its_output(kind):
    """It is freed with it, and the node shows what it has saved, and the layer."""
    layer, x, gen = make(kind)
    x = x.requires_grad_()
    other = python_route(make(kind)[0])
    y = other(x)
    shapes = [tuple(t.shape) for t in y.grad_fn.saved_tensors]
    layer.last = layer(x)
    node = layer.last.grad_fn
    assert [tuple(t.shape) for t in node.saved_tensors] == shapes and node.saved_tensors[0] is x
    assert node.layer is layer and node.name() == "_LUTFunctionBackward" and node.next_functions[0][0] is not None
    alive = weakref.ref(layer)
    del layer, node
    gc.collect()
    assert alive() is None


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("backward", ["native", "python"])
def test_backward_after_the_layer_has_gone(kind, backward):
    layer, x, gen = make(kind)
    want, dy = passed(make(kind)[0], x, gen=gen)
    x = x.detach().requires_grad_()
    y = layer(x)
    if backward == "python":   # a gradient that the native route leaves
        class Sub(torch.Tensor):
            pass
        y.register_hook(lambda g: g.as_subclass(Sub))
    parameters = list(layer.parameters())
    alive = weakref.ref(layer)
    del layer
    gc.collect()
    assert alive() is None
    y.backward(dy)
    got = [y.detach(), x.grad] + [None if p.grad is None else p.grad.to_dense() for p in parameters] + [p.detach() for p in parameters]
    for u, v in zip(got, want):
        close(u if u is None else u.as_subclass(torch.Tensor), v)
