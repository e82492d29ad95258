"""Layers that go through the tensor-core GEMMs at 16 tokens or fewer: edges of tiles, stages and couplings against the oracle, through the operators and, with
bias and residual in the last GEMM's epilogue, through blr_blast_multi.  Every shape is checked to go that way."""
import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _close(got, want):
    got = got.reshape(want.shape).float().cpu()
    assert orc.rel_fro(got, want) < 1e-2  # (two roundings to 11 | 8 bits, as in the other tests of these kernels)
    assert (got - want).abs().max() < 0.05 * want.abs().max()  # a wrong row, column or tile is not drowned in the norm of the rest


def _multi(x, layer, bits, bias, res):
    """One layer with bias and residual by the C entry."""
    from mem_efficient_blr_b200 import _lib as L, ops
    n = x.shape[0]
    U, us, Vt, vs, S = layer if bits != 16 else (layer[0], None, layer[1], None, layer[2])
    b, Q, R, P = U.shape[0], U.shape[1], S.shape[2], x.shape[1] // U.shape[0]
    out = torch.empty(n, b * Q, dtype=x.dtype, device=DEV)
    arr = (L.BlastProblem * 1)()
    arr[0].U, arr[0].V, arr[0].S = U.data_ptr(), Vt.data_ptr(), S.data_ptr()
    if bits != 16:
        arr[0].u_scale, arr[0].v_scale = us.data_ptr(), vs.data_ptr()
    arr[0].bias, arr[0].residual, arr[0].ldr, arr[0].out, arr[0].ldo = bias.data_ptr(), res.data_ptr(), res.stride(0), out.data_ptr(), out.stride(0)
    ws, st = ops._ws(x, n, b, R)
    L.check(L.load().blr_blast_multi(x.data_ptr(), x.stride(0), 0, L.ACT_NONE, n, L.dtype_code(x.dtype), 1, arr, b * R, R, 1, bits, 0, b, P, Q, R, ws.data_ptr(),
                                     ws.numel(), st))
    L.workspace_status(torch.device(DEV))
    return out


def _additions(N, O, dtype):
    g = torch.Generator().manual_seed(1)
    return torch.randn(O, generator=g).to(dtype), torch.randn(N, O, generator=g).to(dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,bits,b,P,Q,R", [
    (4, 8, 16, 1056, 136, 480),    # the fewest tokens; ragged contractions, a second tile of 8 rows
    (4, 4, 15, 1056, 264, 224),    # blocks that are no multiple of a coupling CTA's
    (5, 8, 13, 1056, 136, 480),
    (8, 4, 16, 608, 72, 512),      # the most ranks at 8 tokens
    (9, 8, 5, 1248, 1032, 800),
    (15, 8, 13, 544, 520, 544),
    (16, 8, 16, 1024, 64, 1024),   # the longest chain that comes here
    (16, 4, 13, 416, 1032, 1056),
])
def test_quantised(N, bits, b, P, Q, R, dtype):
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    from mem_efficient_blr_b200 import _lib
    assert _lib.load().blr_debug_few_tokens_route(N, bits, 0, b, P, Q, R) == 2
    x, U, Vt, S = orc.make_blast_inputs(N, b * P, b * Q, b, R, dtype, seed=N + Q + R)
    q = bq.quantize_blast_factors(U.to(DEV), Vt.to(DEV), bits, 0)
    want = orc.blast_wq(x, *[t.cpu() for t in q], S, bits, 0)[0].reshape(N, b * Q)
    xd, layer = x.reshape(N, b * P).to(DEV), (*q, S.to(DEV))
    _close(bq.blast_wq(xd, *layer, bits), want)
    bias, res = _additions(N, b * Q, dtype)
    _close(_multi(xd, layer, bits, bias.to(DEV), res.to(DEV)), want + bias.float() + res.float())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,b,P,Q,R", [
    (9, 12, 1272, 520, 520),       # the fewest tokens, the longest chain at them
    (11, 13, 328, 904, 1016),      # ragged everywhere, blocks that are no multiple of a coupling CTA's
    (12, 5, 1400, 1544, 648),
    (16, 3, 1480, 3640, 664),      # few blocks
    (16, 6, 1280, 904, 520),
    (16, 16, 72, 136, 520),        # in-blocks of little more than a stage, a second tile of 8 rows
    (16, 16, 688, 256, 1488),      # more CTAs than SMs
])
def test_16_bits(N, b, P, Q, R, dtype):
    import mem_efficient_blr_b200.blast_kernels as bk
    from mem_efficient_blr_b200 import _lib
    assert _lib.load().blr_debug_few_tokens_route(N, 16, 0, b, P, Q, R) == 2
    x, U, Vt, S = orc.make_blast_inputs(N, b * P, b * Q, b, R, dtype, seed=N + Q + R)
    want = orc.blast(x, U, Vt, S)[0].reshape(N, b * Q)
    xd, layer = x.reshape(N, b * P).to(DEV), tuple(t.to(DEV) for t in (U, Vt, S))
    _close(bk.blast_torch_layout(xd, *layer), want)
    _close(bk.triton_blast_partial_grouped_fp16(xd, *[t.to(DEV) for t in orc.blast_to_partial_layout(U, Vt, S)]), want)
    bias, res = _additions(N, b * Q, dtype)
    _close(_multi(xd, layer, 16, bias.to(DEV), res.to(DEV)), want + bias.float() + res.float())


@pytest.mark.parametrize("N,bits,b,P,Q,R", [
    (16, 8, 5, 704, 88, 1344), (12, 4, 12, 288, 552, 1408),   # front grids of two waves
    (16, 16, 2, 856, 1080, 1064), (12, 16, 9, 904, 368, 712),
])
def test_where_the_two_launches_decline(N, bits, b, P, Q, R):
    """Whichever of the paths serves the layer, plain and with additions."""
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    x, U, Vt, S = orc.make_blast_inputs(N, b * P, b * Q, b, R, torch.float16, seed=N + Q + R)
    xd, bias, res = x.reshape(N, b * P).to(DEV), *_additions(N, b * Q, torch.float16)
    if bits == 16:
        want, layer = orc.blast(x, U, Vt, S)[0].reshape(N, b * Q), tuple(t.to(DEV) for t in (U, Vt, S))
        _close(bk.blast_torch_layout(xd, *layer), want)
        _close(bk.triton_blast_partial_grouped_fp16(xd, *[t.to(DEV) for t in orc.blast_to_partial_layout(U, Vt, S)]), want)
    else:
        q = bq.quantize_blast_factors(U.to(DEV), Vt.to(DEV), bits, 0)
        want, layer = orc.blast_wq(x, *[t.cpu() for t in q], S, bits, 0)[0].reshape(N, b * Q), (*q, S.to(DEV))
        _close(bq.blast_wq(xd, *layer, bits), want)
    _close(_multi(xd, layer, bits, bias.to(DEV), res.to(DEV)), want + bias.float() + res.float())
