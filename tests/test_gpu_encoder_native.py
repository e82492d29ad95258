"""The encoder layer's halves as one native call each: the same bits as the calls they stand for, and none of it where a module is not stock."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _net(nw, dtype=torch.float16):
    shape = nw.ViTShape(layers=2, d=256, heads=4, mlp=512, image=64, patch=16, b=16, ranks={"qkv": 32, "intermediate": 48, "output": 48})
    net = nw.ViTEncoder(shape, "blast", device=DEV, dtype=dtype, seed=4)
    for layer in net.layers:
        layer.qkv.bias.data.normal_()
        layer.output.bias = None
    return net, torch.randn(3, 3, 64, 64, device=DEV, dtype=dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_same_bits_as_call_by_call(monkeypatch, dtype):
    from mem_efficient_blr_b200 import _lib, networks as nw
    net, img = _net(nw, dtype)
    calls = []
    for name in ("attention", "mlp"):
        f = getattr(_lib.direct(), name)
        monkeypatch.setattr(_lib.direct(), name, lambda *a, f=f: calls.append(1) or f(*a))
    got = net(img)
    assert len(calls) == 4
    monkeypatch.setattr(_lib, "direct", lambda: None)
    assert torch.equal(got, net(img)) and len(calls) == 4


@pytest.mark.parametrize("which", ["qkv", "attn_out", "intermediate", "output"])
def test_hooked_and_replaced_modules_are_called(which):
    from mem_efficient_blr_b200 import networks as nw
    net, img = _net(nw)
    want, seen = net(img), []
    m = getattr(net.layers[1], which)
    handle = m.register_forward_hook(lambda m, a, out: seen.append(1) and None)
    got = net(img)
    assert seen
    if which == "intermediate":  # (its activation is then torch's, on a rounded result: one rounding of 2^-11 more in each of two layers)
        assert (got - want).float().norm() < 2e-3 * want.float().norm()
    else:
        assert torch.equal(got, want)
    handle.remove()

    class Twice(type(m)):
        def forward(self, x, *a):
            return 2 * super().forward(x, *a)
    m.__class__ = Twice
    assert not torch.equal(net(img), want)


def test_few_rows_and_gradients_go_the_general_way():
    from mem_efficient_blr_b200 import _lib, networks as nw
    net, _ = _net(nw)
    layer, lin = nw._factors16(net.layers[0].qkv), net.layers[0].attn_out
    d, h = _lib.direct(), torch.randn(1, 16, 256, device=DEV).half()
    assert d.attention(h, layer, 4, lin.weight, lin.bias) is None
    h = torch.randn(1, 17, 256, device=DEV).half()
    assert d.attention(h, layer, 3, lin.weight, lin.bias) is None and d.attention(h, layer[:3], 4, lin.weight, lin.bias) is None
    assert d.mlp(h, layer, layer, 0) is None  # 768 values against 256
    y = d.attention(h, layer, 4, lin.weight, lin.bias)
    assert y.shape == h.shape
    assert d.attention(h.requires_grad_(), layer, 4, lin.weight, lin.bias) is None
    with torch.no_grad():
        assert torch.equal(d.attention(h, layer, 4, lin.weight, lin.bias), y)


def test_a_profile_names_the_halves():
    from mem_efficient_blr_b200 import networks as nw
    net, img = _net(nw)
    net(img)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU], record_shapes=True) as prof:
        net(img)
    for name in ("attention", "mlp"):
        events = [e for e in prof.events() if e.name == f"blr_b200_ext::{name}"]
        assert len(events) == 2 and all(list(e.input_shapes[0]) == [3, 17, 256] for e in events)
