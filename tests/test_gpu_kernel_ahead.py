"""Calls on what the kernel directly ahead of them in the stream writes, against the same call once everything has finished."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rn(seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return lambda *s, fan=1: (torch.randn(*s, generator=g, device=DEV) / fan ** 0.5).half()


def _few(N, bits, b, P, Q, R):
    from mem_efficient_blr_b200 import _lib
    return _lib.load().blr_debug_few_tokens_route(N, bits, 0, b, P, Q, R)


def _same_after(make, call):
    """make() enqueues a long kernel of this library and returns what it writes; call(that) right behind it, other values each time."""
    made = []
    for _ in range(3):
        torch.cuda.synchronize()
        t = make()
        got = call(t)
        torch.cuda.synchronize()
        assert torch.equal(got, call(t)) and not any(torch.equal(t, m) for m in made)
        made.append(t.clone())


@pytest.mark.parametrize("bits,N,P,Q,R", [(8, 4, 1024, 256, 512), (8, 4, 64, 64, 256), (4, 4, 64, 64, 256), (8, 100, 64, 64, 256), (16, 100, 64, 64, 256), (16, 500, 64, 64, 256)])
def test_residual_and_bias(bits, N, P, Q, R):
    """The additions of the last kernel; first through the GEMMs at 4 tokens, then through the two decode launches."""
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    import mem_efficient_blr_b200.dense_kernels as dk
    b, P, Q, R, K = 16, 64, 256, 256, 8192
    rn = _rn(bits + N)
    x, U, V, S, W = rn(N, b * P), rn(b, Q, R, fan=R), rn(b, R, P, fan=P), rn(b, b, R), rn(b * Q, K, fan=K)
    layer = (U, V, S) if bits == 16 else (*bq.quantize_blast_factors(U, V, bits), S)
    multi = bk.blast_multi_torch_layout if bits == 16 else lambda x, l, **k: bq.blast_wq_multi(x, l, bits, 0, **k)
    _same_after(lambda: dk.dense_torch_layout(rn(N, K), W), lambda r: multi(x, [layer], residuals=[r])[0])
    _same_after(lambda: dk.dense_torch_layout(rn(1, K), W), lambda t: multi(x, [layer], biases=[t.view(-1)])[0])


@pytest.mark.parametrize("bits,N", [(16, 9), (16, 16), (16, 17), (16, 300), (8, 9), (4, 16), (8, 17), (4, 300), (8, 900)])
def test_factors(bits, N):
    """Layers that go through the GEMMs: each of U, V and S (quantised layers: with their scales) from right ahead, the other two old."""
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    import mem_efficient_blr_b200.dense_kernels as dk
    b, P, Q, R, K = 16, 256, 688, 1024, 4096
    assert N > 16 or _few(N, bits, b, P, Q, R) == 2
    rn = _rn(bits + N)
    x, U, V, S = rn(N, b * P), rn(b, Q, R, fan=R), rn(b, R, P, fan=P), rn(b, b, R)

    def made(n, W):   # a long GEMM, whose result is the factor
        return lambda: dk.dense_torch_layout(rn(n, K), W)
    to_u, to_v, to_s = made(b * Q, rn(R, K, fan=K * R)), made(b * R, rn(P, K, fan=K * P)), made(b * b, rn(R, K, fan=K))
    if bits == 16:
        _same_after(to_u, lambda t: bk.blast_torch_layout(x, t.view(b, Q, R), V, S))
        _same_after(to_v, lambda t: bk.blast_torch_layout(x, U, t.view(b, R, P), S))
        _same_after(to_s, lambda t: bk.blast_torch_layout(x, U, V, t.view(b, b, R)))
        return
    Uq, us, Vq, vs = bq.quantize_blast_factors(U, V, bits)
    _same_after(to_s, lambda t: bq.blast_wq(x, Uq, us, Vq, vs, t.view(b, b, R), bits))
    # the stored bytes and scales of the layer, re-quantised into the same memory ahead of each call
    for t, q, s in ((V, Vq, vs), (U, Uq, us)):
        for k in range(3):
            new = bq.quantize_blast_factors(*((U, rn(*V.shape, fan=P)) if t is V else (rn(*U.shape, fan=R), V)), bits)
            torch.cuda.synchronize()
            q.copy_(new[2 if t is V else 0])
            s.copy_(new[3 if t is V else 1])
            got = bq.blast_wq(x, Uq, us, Vq, vs, S, bits)
            torch.cuda.synchronize()
            assert torch.equal(got, bq.blast_wq(x, Uq, us, Vq, vs, S, bits))


def test_positions():
    """Decode positions counted up on the device right ahead of each append, with no synchronisation between the steps."""
    from mem_efficient_blr_b200 import ops
    B, H, S, hd = 4, 8, 512, 64
    rn = _rn(3)
    ang = torch.rand(S, hd // 2, device=DEV)
    cos, sin, kc = ang.cos(), ang.sin(), torch.zeros(B, H, S, hd, device=DEV, dtype=torch.float16)
    vc, pos, want_k, want_v = torch.zeros_like(kc), torch.full((1,), -1, device=DEV), torch.zeros_like(kc), torch.zeros_like(kc)
    steps = [(rn(B, H * hd), rn(B, H * hd), rn(B, H * hd)) for _ in range(S)]
    for q, k, v in steps:
        pos.add_(1)
        ops.rope_append(q, k, v, cos, sin, pos, kc, vc, 1)
    for s, (_, k, v) in enumerate(steps):
        a, b = k.view(B, H, 2, hd // 2).float().unbind(2)
        want_k[:, :, s] = torch.cat((a * cos[s] - b * sin[s], b * cos[s] + a * sin[s]), -1).half()
        want_v[:, :, s] = v.view(B, H, hd)
    assert torch.equal(vc, want_v) and (kc - want_k).abs().max() <= 2 ** -8  # (values below 8 of 11 bits: the other neighbour)
