"""The direct calls of the torch extension (eager route of the Python layer) against the general route on the same inputs,
for the shapes of x they take, the ones they decline, and the errors of the general route behind them."""
import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def L():
    from mem_efficient_blr_b200 import _lib
    assert _lib.direct() is not None, "the torch extension is not built"
    return _lib


def _inputs(kind, base):
    """x views of one (48, 512) matrix: (taken by the direct call, x)."""
    return {"plain": (True, base[:5]), "strided": (True, base[:10:2]), "lead": (True, base[:6].view(2, 3, 512)),
            "row": (True, base[7:8]), "many": (True, base), "misaligned": (False, torch.cat((base, base), 1)[:5, 4:516]),
            "transposed": (False, base[:5].t().contiguous().t()), "empty": (False, base[:0]), "one_dim": (False, base[3])}[kind]


@pytest.mark.parametrize("kind", ["plain", "strided", "lead", "row", "many", "misaligned", "transposed", "empty", "one_dim"])
def test_direct_and_general_route_agree(L, monkeypatch, kind):
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    import mem_efficient_blr_b200.dense_kernels as dk
    import mem_efficient_blr_b200.low_rank_kernels as lk
    import mem_efficient_blr_b200.monarch_kernels as mk
    from mem_efficient_blr_b200 import ops
    x0, U, Vt, S = (t.to(DEV) for t in orc.make_blast_inputs(48, 512, 768, 4, 128, torch.float16, seed=1))
    taken, x = _inputs(kind, x0.reshape(48, 512))
    w = lambda *s: (torch.randn(*s, generator=torch.Generator().manual_seed(2)) / 16).half().to(DEV)
    part, bmm = orc.blast_to_partial_layout(U, Vt, S), orc.blast_to_bmm_layout(U, Vt, S)
    q8 = (*bq.quantize_blast_factors(U, Vt, 8), S)
    bias = w(768)
    calls = [
        lambda: bk.blast_torch_layout(x, U, Vt, S),
        lambda: bk.triton_blast_partial_grouped_fp16(x, *(t.contiguous() for t in part)),
        lambda: bk.triton_blast_bmm_fp16(x, *(t.contiguous() for t in bmm)),
        lambda: bq.blast_wq(x, *q8, 8),
        lambda: mk.triton_monarch_right_fp16(x, w(4, 128, 64), w(4, 192, 64)),
        lambda: mk.triton_monarch_right_left_fp16(x, w(4, 128, 64), w(4, 64, 192)),
        lambda: mk.monarch_torch_layout(x, w(4, 64, 128), w(4, 192, 64), True),
        lambda: lk.triton_low_rank_fp16(x, w(512, 64), w(64, 768)),
        lambda: lk.low_rank_torch_layout(x, w(64, 512), w(768, 64)),
        lambda: dk.triton_dense_fp16(x, w(512, 768)),
        lambda: dk.dense_torch_layout(x, w(768, 512)),
        lambda: bk.blast_multi_torch_layout(x, [(U, Vt, S)], biases=[bias])[0],
        lambda: bq.blast_wq_multi(x, [q8], 8, biases=[bias])[0],
        lambda: ops.layernorm(x, w(512), None, 1e-6),
        lambda: ops.rmsnorm(x, w(512), 1e-6),
    ]
    if kind == "one_dim":
        calls = calls[:4]   # (the others never took a single vector)
    d = L.direct()
    assert (d.blast(x, U, Vt, S, 0, 0, 256, 4, 128) is not None) == taken
    if kind in ("empty",):
        calls = calls[:11]
    got = [c() for c in calls]
    monkeypatch.setattr(L, "_direct", None)
    for c, g in zip(calls, got):
        want = c()
        assert g.shape == want.shape and g.dtype == want.dtype
        assert torch.allclose(g, want, rtol=1e-2, atol=1e-3)   # (the cluster kernel's sums have no fixed order)


def test_direct_calls_leave_errors_to_the_general_route(L):
    import mem_efficient_blr_b200.blast_kernels as bk
    x, U, Vt, S = (t.to(DEV) for t in orc.make_blast_inputs(4, 512, 768, 4, 128, torch.float16, seed=1))
    x = x.reshape(4, 512)
    with pytest.raises(AssertionError):
        bk.blast_torch_layout(x, U, Vt[:, :64].contiguous(), S)          # ranks differ
    with pytest.raises(RuntimeError, match="one 16-bit dtype"):
        bk.blast_torch_layout(x, U.bfloat16(), Vt, S)
    with pytest.raises(RuntimeError, match="contiguous"):
        bk.blast_torch_layout(x, U.transpose(1, 2).contiguous().transpose(1, 2), Vt, S)
    with pytest.raises(RuntimeError, match="CUDA"):
        bk.blast_torch_layout(x.cpu(), U, Vt, S)
    with pytest.raises(RuntimeError, match="multiple"):                  # the library's own checks come through
        bk.blast_torch_layout(torch.zeros(2, 48, device=DEV).half(), torch.zeros(4, 12, 20, device=DEV).half(),
                              torch.zeros(4, 20, 12, device=DEV).half(), torch.zeros(4, 4, 20, device=DEV).half())


def _calls():
    """One small call of every operator on x (..., 64)."""
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    import mem_efficient_blr_b200.dense_kernels as dk
    import mem_efficient_blr_b200.low_rank_kernels as lk
    import mem_efficient_blr_b200.monarch_kernels as mk
    g = torch.Generator().manual_seed(5)
    w = lambda *s: (torch.randn(*s, generator=g) / 8).half().to(DEV)
    U, Vt, S = w(4, 24, 32), w(4, 32, 16), w(4, 4, 32)
    q8 = (*bq.quantize_blast_factors(U, Vt, 8), S)
    m1, m2, V, Ul, W = w(4, 32, 16), w(4, 24, 32), w(32, 64), w(96, 32), w(96, 64)
    return {"blast": lambda x: bk.blast_torch_layout(x, U, Vt, S), "blast_wq": lambda x: bq.blast_wq(x, *q8, 8),
            "monarch": lambda x: mk.monarch_torch_layout(x, m1, m2), "low_rank": lambda x: lk.low_rank_torch_layout(x, V, Ul),
            "dense": lambda x: dk.dense_torch_layout(x, W)}


OPS = ["blast", "blast_wq", "monarch", "low_rank", "dense"]


@pytest.mark.parametrize("op", OPS)
def test_a_jit_trace_holds_the_operator(L, op):
    """The result must depend on the traced input: a call past the tracer would be a constant of the graph."""
    call = _calls()[op]
    x, other = torch.randn(2, 3, 64, device=DEV).half().unbind(0)
    traced = torch.jit.trace(call, (x,), check_trace=False)
    assert f"blr_b200_ext::{op}" in str(traced.graph)
    assert torch.allclose(traced(other), call(other), rtol=1e-2, atol=1e-3)


@pytest.mark.filterwarnings("ignore:There is a performance drop")
@pytest.mark.parametrize("op", OPS)
def test_vmap_takes_the_operators(L, op):
    call = _calls()[op]
    x = torch.randn(2, 5, 64, device=DEV).half()
    assert torch.allclose(torch.vmap(call)(x), torch.stack([call(x[0]), call(x[1])]), rtol=1e-2, atol=1e-3)


@pytest.mark.parametrize("op", OPS)
def test_modes_and_lazy_negation_see_the_operator(L, op):
    from torch.overrides import TorchFunctionMode
    seen = []

    class Watch(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    call = _calls()[op]
    x = torch.randn(3, 64, device=DEV).half()
    with Watch():
        call(x)
    assert any(f"blr_b200_ext.{op}" in s for s in seen)
    assert torch.allclose(call(torch._neg_view(x)), -call(x), rtol=1e-2, atol=1e-3)


@pytest.mark.parametrize("op", OPS)
def test_a_profile_names_the_operator(L, op):
    call = _calls()[op]
    x = torch.randn(3, 64, device=DEV).half()
    call(x)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU], record_shapes=True) as prof:
        call(x)
    events = [e for e in prof.events() if e.name == f"blr_b200_ext::{op}"]
    assert len(events) == 1 and list(events[0].input_shapes[0]) == [3, 64]


@pytest.mark.parametrize("op", OPS)
def test_autograd_learns_of_the_operator(L, op):
    """No operator here has a derivative; a result that depends on a leaf has to say so instead of looking like a constant."""
    call = _calls()[op]
    x = torch.randn(3, 64, device=DEV).half().requires_grad_()
    assert call(x).grad_fn is not None
    with torch.no_grad():
        assert call(x).grad_fn is None
    assert call(x.detach()).grad_fn is None


def test_arguments_that_are_no_numbers_are_errors_of_the_general_route(L):
    """... and not a SystemError of the interpreter over an exception that the direct call left behind."""
    import mem_efficient_blr_b200.blast_kernels as bk
    from mem_efficient_blr_b200 import ops
    x, U, Vt, S = (t.to(DEV) for t in orc.make_blast_inputs(4, 64, 96, 4, 32, torch.float16, seed=1))
    for call in (lambda: bk.blast_torch_layout(x, U, Vt, S, flags="none"), lambda: ops.layernorm(x, None, None, "small")):
        with pytest.raises((TypeError, ValueError, RuntimeError)):
            call()
