"""Host-side logic of the network glue (mem_efficient_blr_b200/networks.py) with dense linears on CPU: the static
key/value cache, the rotary embedding and the prefill / decode split must agree with each other."""
import pytest
import torch

from mem_efficient_blr_b200 import networks as nw


def _small():
    return nw.LlamaShape(layers=2, d=64, heads=4, ffn=128, vocab=97, b=4, rank_attn=16, rank_mlp=16)


def test_decode_step_continues_a_prefill():
    """Prefill of T - 1 tokens followed by one decode step at slot T - 1 of a cache of length T gives the logits of a
    prefill of all T tokens."""
    T, B = 9, 3
    ids = torch.randint(0, 97, (B, T), generator=torch.Generator().manual_seed(1))
    full = nw.LlamaDecoder(_small(), "dense", batch=B, cache_len=T, device="cpu", dtype=torch.float32, seed=3)
    want = full.prefill(ids)
    step = nw.LlamaDecoder(_small(), "dense", batch=B, cache_len=T, device="cpu", dtype=torch.float32, seed=3)
    step.prefill(ids[:, :T - 1])
    got = step.decode_step(ids[:, T - 1:], torch.tensor([T - 1]))
    assert got.shape == (B, 97)
    assert torch.allclose(got, want, atol=1e-4, rtol=1e-4)
    # the caches of the two runs hold the same keys and values
    for a, b in zip(full.kcache + full.vcache, step.kcache + step.vcache):
        assert torch.allclose(a, b, atol=1e-5)


def test_same_seed_gives_same_network_and_structured_list():
    a = nw.LlamaDecoder(_small(), "dense", batch=1, cache_len=4, device="cpu", dtype=torch.float32, seed=5)
    b = nw.LlamaDecoder(_small(), "dense", batch=1, cache_len=4, device="cpu", dtype=torch.float32, seed=5)
    for pa, pb in zip(a.parameters(), b.parameters()):
        assert torch.equal(pa, pb)
    assert len(a.structured_linears()) == 2 * 7


def test_vit_shapes_and_rank_rule():
    s = nw.ViTShape()
    # ranks chosen for about half of the dense parameters: R (I + O + b^2) ~ I O / 2, multiples of 16
    for name, (i, o) in {"qkv": (768, 2304), "intermediate": (768, 3072), "output": (3072, 768)}.items():
        r = s.ranks[name]
        assert r % 16 == 0 and 0.45 < r * (i + o + s.b ** 2) / (i * o) < 0.55
    small = nw.ViTShape(layers=1, d=64, heads=4, mlp=128, image=32, patch=16, b=4, ranks={"qkv": 16, "intermediate": 16, "output": 16})
    m = nw.ViTEncoder(small, "dense", device="cpu", dtype=torch.float32)
    out = m(torch.randn(2, 3, 32, 32))
    assert out.shape == (2, 5, 64) and len(m.structured_linears()) == 3


def test_ideal_order_index_and_dense_folding_on_cpu():
    """The block-major (right_ideal) order against the oracle's re-ordering, and a dense layer that absorbs it."""
    from mem_efficient_blr_b200 import monarch_kernels as mk
    from oracle import blr_oracle as orc
    b, S, O = 4, 6, 5
    g = torch.Generator().manual_seed(0)
    y_int = torch.randn(3, S * b, generator=g)
    y_ideal = orc.monarch_ideal_order(y_int, b)
    idx = mk.ideal_order_index(S * b, b)
    assert torch.equal(y_ideal[..., idx], y_int)
    W = torch.randn(O, S * b, generator=g)
    Wf = mk.fold_ideal_order_into_dense(W, b)
    assert torch.allclose(y_ideal @ Wf.T, y_int @ W.T, atol=1e-6)


# ------------------------------------------------------------------------------------------------ fused passes and replaced modules
def _tiny(kind, depth=2):
    if kind == "vit":
        s = nw.ViTShape(layers=depth, d=64, heads=4, mlp=128, image=32, patch=16, b=4, ranks={"qkv": 16, "intermediate": 16, "output": 16})
        net = nw.ViTEncoder(s, "dense", device="cpu", dtype=torch.float32)
        return net, net.layers, (torch.randn(2, 3, 32, 32, generator=torch.Generator().manual_seed(1)),)
    s = nw.DiTShape(layers=depth, d=64, heads=4, mlp=128, latent=8, classes=10, b=4, freq=32, ranks={"qkv": 16, "fc1": 16, "adaln": 16})
    net = nw.DiTDenoiser(s, "dense", device="cpu", dtype=torch.float32)
    g = torch.Generator().manual_seed(1)
    return net, net.blocks, (torch.randn(3, 4, 8, 8, generator=g), torch.tensor([5, 400, 999]), torch.tensor([0, 7, 10]))


def _bent(t):
    """Another value that a norm behind it does not undo."""
    return t + 0.5 * t.roll(1, -1)


class _Wrapped(torch.nn.Module):
    def __init__(self, m):
        super().__init__()
        self.m = m

    def forward(self, *a, **k):
        return _bent(self.m(*a, **k))


def _subclass(m):
    m.__class__ = type("Own" + type(m).__name__, (type(m),), {"forward": lambda self, *a, **k: _bent(super(type(self), self).forward(*a, **k))})


class _Drop(torch.nn.Module):
    def forward(self, x, *rest):
        return x


def _affine(d):
    n = nw.LayerNorm(d, eps=1e-6).requires_grad_(False)
    n.weight.copy_(torch.linspace(0.5, 2, d))
    n.bias.copy_(torch.linspace(-1, 1, d))
    return n


def _put(layers, i, m):
    layers[i] = m


# what a caller may have done to a network, by the layer list and the network: each changes the result
REPLACED = {
    "subclass with a forward of its own": lambda net, layers, mp: _subclass(layers[1]),
    "forward put on the object": lambda net, layers, mp: mp.setattr(layers[1], "forward", lambda *a, f=layers[1].forward: _bent(f(*a)), raising=False),
    "method patched on the class": lambda net, layers, mp: mp.setattr(type(layers[1]), "forward", lambda self, *a, f=type(layers[1]).forward: _bent(f(self, *a))),
    "layer dropped": lambda net, layers, mp: _put(layers, 1, _Drop()),
    "layer wrapped": lambda net, layers, mp: _put(layers, 0, _Wrapped(layers[0])),
    "hook": lambda net, layers, mp: layers[1].register_forward_hook(lambda m, a, out: _bent(out)),
    "pre-hook": lambda net, layers, mp: layers[1].register_forward_pre_hook(lambda m, a: (_bent(a[0]), *a[1:])),
    "hook on an inner norm": lambda net, layers, mp: _norms(layers[1])[1].register_forward_hook(lambda m, a, out: _bent(out)),
    "subclass of an inner norm": lambda net, layers, mp: _subclass(_norms(layers[1])[0]),
    "subclass of the last norm": lambda net, layers, mp: _subclass(net.ln if hasattr(net, "ln") else net.final_norm),
    "affine last norm": lambda net, layers, mp: setattr(net, "ln" if hasattr(net, "ln") else "final_norm", _affine(64)),
    "affine inner norm": lambda net, layers, mp: setattr(layers[1], "ln2" if hasattr(net, "ln") else "norm2", _affine(64)),
}


def _norms(layer):
    return (layer.ln1, layer.ln2) if hasattr(layer, "ln1") else (layer.norm1, layer.norm2)


def _stand_ins(monkeypatch):
    """The fused operators as torch computes them, so that the fused passes run without a device; how often each was called."""
    from mem_efficient_blr_b200 import ops
    F, calls = torch.nn.functional, {"add_layernorm": 0, "gated_add_modulate": 0}

    def add_layernorm(x, y, w, b, eps, or_none=False):
        if or_none and (x.shape != y.shape or x.dtype != y.dtype):
            return None
        calls["add_layernorm"] += 1
        return x + y, F.layer_norm(x + y, x.shape[-1:], w, b, eps)

    def layernorm_modulate(x, shift, scale, eps):
        return F.layer_norm(x, x.shape[-1:], None, None, eps) * (1 + scale.unsqueeze(1)) + shift.unsqueeze(1)

    def gated_add_modulate(x, gate, y, shift, scale, eps):
        calls["gated_add_modulate"] += 1
        t = x + gate.unsqueeze(1) * y
        return t, layernorm_modulate(t, shift, scale, eps)

    for f in (add_layernorm, layernorm_modulate, gated_add_modulate):
        monkeypatch.setattr(ops, f.__name__, f)
    return calls


@pytest.mark.parametrize("kind", ["vit", "dit"])
def test_fused_pass_of_a_stock_network(kind, monkeypatch):
    """Seven layers (modulations in calls of three, three and one): the fused pass runs, and gives the layer-by-layer result."""
    calls = _stand_ins(monkeypatch)
    net, layers, inputs = _tiny(kind, 7)
    monkeypatch.setattr(nw, "_one_kernel", lambda x: False)
    want = net(*inputs)
    assert not any(calls.values())
    monkeypatch.setattr(nw, "_one_kernel", lambda x: True)
    got = net(*inputs)
    assert calls["add_layernorm" if kind == "vit" else "gated_add_modulate"] == 14
    assert torch.allclose(got, want, atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("what", list(REPLACED) + ["hook on all modules", "pre-hook on all modules"])
@pytest.mark.parametrize("kind", ["vit", "dit"])
def test_replaced_or_hooked_modules_are_called(kind, what, monkeypatch):
    """Whatever a caller put in a layer's place, on it or around it takes part also where the fused operators could run."""
    _stand_ins(monkeypatch)
    net, layers, inputs = _tiny(kind)
    stock = net(*inputs)
    handle = None
    if what in REPLACED:
        REPLACED[what](net, layers, monkeypatch)
    elif what == "hook on all modules":
        handle = torch.nn.modules.module.register_module_forward_hook(lambda m, a, out: _bent(out) if type(m).__name__ in ("ViTLayer", "DiTBlock", "LayerNorm") else None)
    else:
        handle = torch.nn.modules.module.register_module_forward_pre_hook(lambda m, a: (_bent(a[0]), *a[1:]) if type(m).__name__ in ("ViTLayer", "DiTBlock") else None)
    try:
        monkeypatch.setattr(nw, "_one_kernel", lambda x: False)
        want = net(*inputs)
        monkeypatch.setattr(nw, "_one_kernel", lambda x: True)
        got = net(*inputs)
    finally:
        if handle is not None:
            handle.remove()
    assert torch.allclose(got, want, atol=1e-5, rtol=1e-5)
    assert not torch.allclose(want, stock, atol=1e-3)


def test_replaced_linears_of_a_fused_call_are_called(monkeypatch):
    """Subclasses and hooked layers keep their own call in structured_multi and linear_act; stock ones go to the fused operators."""
    new = lambda: nw.BlastTorchLinear(64, 64, 4, 16, device="cpu", dtype=torch.float32, generator=torch.Generator().manual_seed(2))
    monkeypatch.setattr(nw.BlastTorchLinear, "U_device_ok", lambda self: True)
    monkeypatch.setattr(nw.bk, "blast_multi_torch_layout", lambda x, layers, *a, **k: ["fused"] * len(layers))
    x = torch.ones(2, 64)
    assert nw.structured_multi([new(), new()], x) == ["fused", "fused"] and nw.linear_act(new(), x, "gelu") == "fused"

    class Own(nw.BlastTorchLinear):
        def forward(self, x):
            return -x

    own = Own(64, 64, 4, 16, device="cpu", dtype=torch.float32)
    hooked = new()
    hooked.forward = lambda x: x
    bumped = nw.make_linear("dense", 64, 64, 0, 0, False, "cpu", torch.float32, None)
    assert torch.equal(nw.structured_multi([own], x)[0], -x) and torch.equal(nw.structured_multi([hooked, bumped], x)[0], x)
    assert torch.equal(nw.linear_act(own, x, "gelu"), torch.nn.functional.gelu(-x))
    seen = []
    stock = new()
    stock.register_forward_pre_hook(lambda m, a: seen.append(a[0].shape))
    monkeypatch.setattr(nw.bk, "blast_torch_layout", lambda x, *f: x)
    assert torch.equal(nw.structured_multi([stock], x)[0], x) and seen == [x.shape]


@pytest.mark.parametrize("y", [lambda x: x[:, :1], lambda x: x.double(), lambda x: x.transpose(0, 1).contiguous().transpose(0, 1), lambda x: x[:1].expand(3, -1, -1)],
                         ids=["broadcast", "dtype", "strides", "expanded"])
def test_add_norm_takes_what_an_addition_takes(y, monkeypatch):
    """Terms that the fused operator refuses (another shape or dtype) are added as before; strides are the operator's to repair."""
    calls = _stand_ins(monkeypatch)
    monkeypatch.setattr(nw, "_one_kernel", lambda x: True)
    x = torch.randn(3, 5, 64, generator=torch.Generator().manual_seed(1))
    norm = nw.LayerNorm(64).to(torch.promote_types(x.dtype, y(x).dtype)).requires_grad_(False)
    t, out = nw.add_norm(x, y(x), norm)
    assert torch.equal(t, x + y(x)) and t.dtype == (x + y(x)).dtype and torch.equal(out, norm(t))
    assert calls["add_layernorm"] == (y(x).shape == x.shape and y(x).dtype == x.dtype)


def test_encoder_projection_whose_weight_is_no_parameter(monkeypatch):
    """Sharding and offloading wrappers put a plain tensor in the parameter's place: the projection is then called as it is."""
    from mem_efficient_blr_b200 import _lib

    class Direct:
        def attention(self, *a):
            raise AssertionError("not on parameters that are not there")

    shape = nw.ViTShape(layers=1, d=64, heads=4, mlp=128, image=32, patch=16, b=4)
    layer = nw.ViTLayer(shape, "dense", "cpu", torch.float32, torch.Generator().manual_seed(1))
    h = torch.randn(2, 5, 64)
    want = layer.attention(h)
    weight = layer.attn_out.weight.data.clone()
    del layer.attn_out.weight
    layer.attn_out.weight = weight
    monkeypatch.setattr(_lib, "direct", lambda: Direct())
    monkeypatch.setattr(nw, "_factors16", lambda m: ("U", "Vt", "S", None))
    assert torch.equal(layer.attention(h), want)
