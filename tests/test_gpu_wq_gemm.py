"""The GEMMs on stored int8 / int4 weights (csrc/umma_wq.cu): edges of their tiles against the oracle, through the operators."""
import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _layer(N, b, P, Q, R, bits, group, dtype):
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    x, U, Vt, S = orc.make_blast_inputs(N, b * P, b * Q, b, R, dtype, seed=N + Q + R)
    Uq, us, Vq, vs = bq.quantize_blast_factors(U.to(DEV), Vt.to(DEV), bits, group)
    want = orc.blast_wq(x, Uq.cpu(), us.cpu(), Vq.cpu(), vs.cpu(), S, bits, group)[0].reshape(N, b * Q)
    return x.reshape(N, b * P).to(DEV), (Uq, us, Vq, vs, S.to(DEV)), want


def _close(got, want):
    got = got.reshape(want.shape).float().cpu()
    assert orc.rel_fro(got, want) < 1e-2  # (two roundings to 11 | 8 bits: observed 4e-4 | 3e-3)
    assert (got - want).abs().max() < 0.05 * want.abs().max()  # a wrong row, column or tile is not drowned in the norm of the rest


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits,group", [(8, 0), (4, 0), (8, 128), (4, 128)])
@pytest.mark.parametrize("N,b,P,Q,R", [
    (17, 2, 128, 8, 128),      # one tile of 8 rows of 128; two stages of the first GEMM
    (48, 16, 128, 136, 384),   # a second tile of 8 rows
    (256, 3, 256, 128, 128),   # the most tokens of one MMA
    (257, 4, 128, 264, 640),   # two MMAs side by side
    (384, 16, 128, 256, 256),  # the most tokens of a CTA
    (385, 5, 128, 72, 128),    # two shares
    (700, 9, 128, 200, 1152),
])
def test_tiles_above_16_tokens(N, b, P, Q, R, bits, group, dtype):
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    x, layer, want = _layer(N, b, P, Q, R, bits, group, dtype)
    _close(bq.blast_wq(x, *layer, bits, group), want)
    g = torch.Generator().manual_seed(1)
    bias, res = torch.randn(b * Q, generator=g).to(dtype), torch.randn(N, b * Q, generator=g).to(dtype)
    _close(bq.blast_wq_multi(x, [layer], bits, group, biases=[bias.to(DEV)], residuals=[res.to(DEV)])[0], want + bias.float() + res.float())
    _close(bq.blast_wq_multi(x, [layer], bits, group, biases=[bias.to(DEV)], out_act="gelu")[0], torch.nn.functional.gelu(want + bias.float()))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("N,b,P,Q,R", [
    (4, 2, 32, 8, 32),         # the fewest tokens and ranks
    (5, 3, 96, 136, 96),       # ranks and contraction beyond a stage, a second tile of 8 rows
    (8, 16, 64, 72, 512),
    (9, 16, 256, 688, 1024),
    (15, 13, 96, 40, 544),     # in-blocks that are no multiple of the out-blocks of a coupling CTA
    (16, 16, 1024, 64, 1024),  # the longest chain that comes here
])
def test_up_to_16_tokens(N, b, P, Q, R, bits, dtype):
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    x, layer, want = _layer(N, b, P, Q, R, bits, 0, dtype)
    _close(bq.blast_wq(x, *layer, bits), want)
    g = torch.Generator().manual_seed(1)
    bias, res = torch.randn(b * Q, generator=g).to(dtype), torch.randn(N, b * Q, generator=g).to(dtype)
    _close(bq.blast_wq_multi(x, [layer], bits, 0, biases=[bias.to(DEV)], residuals=[res.to(DEV)])[0], want + bias.float() + res.float())
    # rows of a wider matrix
    wide = torch.zeros(N, b * P + 8, dtype=dtype, device=DEV)
    wide[:, :b * P] = x
    _close(bq.blast_wq(wide[:, :b * P], *layer, bits), want)


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("N", [513, 1024, 1025])
def test_where_large_layers_are_widened(N, bits, monkeypatch):
    """A million weights: inside the GEMMs up to 1024 tokens, in a pass beyond, plain and with a bias; the same bits either way."""
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    from mem_efficient_blr_b200 import ops
    x, layer, _ = _layer(N, 8, 256, 264, 256, bits, 0, torch.float16)
    widened = []
    monkeypatch.setattr(ops, "dequantize_sym", lambda *a, f=ops.dequantize_sym: widened.append(1) or f(*a))
    got = bq.blast_wq(x, *layer, bits)
    assert bool(widened) == (N > 1024)
    widened.clear()
    bias = torch.randn(8 * 264, device=DEV).half()
    fused = bq.blast_wq_multi(x, [layer], bits, 0, biases=[bias])[0]
    assert bool(widened) == (N > 1024)
    Uw, Vw = (ops.dequantize_sym(q, s, bits, 0, torch.float16) for q, s in (layer[:2], layer[2:4]))
    want = bk.blast_torch_layout(x, Uw, Vw, layer[4])
    assert torch.equal(got, want)
    assert orc.rel_fro(fused.float().cpu(), (want.float() + bias.float()).cpu()) < 2e-3  # (one rounding more or less, 2^-11)
