"""16-bit weights as the rows of the GEMMs' tiles (csrc/umma_wq.cu): edges of rows, tokens and shares against the oracle, through the operators."""
import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _close(got, want):
    got = got.reshape(want.shape).float().cpu()
    assert orc.rel_fro(got, want) < 1e-2  # (two roundings to 11 | 8 bits: observed 4e-4 | 3e-3)
    assert (got - want).abs().max() < 0.05 * want.abs().max()  # a wrong row, column or tile is not drowned in the norm of the rest


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,b,P,Q,R", [
    (17, 2, 72, 8, 136),       # 8 rows of a tile, a ragged contraction
    (130, 16, 48, 136, 264),   # a second tile of 8 rows; in-blocks shorter than a stage
    (256, 4, 128, 264, 640),   # the most tokens of one MMA
    (257, 4, 256, 1024, 1024), # two MMAs side by side, or two shares
    (384, 16, 256, 688, 1024), # the most tokens of a CTA
    (385, 16, 256, 256, 1024), # two shares
    (1000, 9, 128, 384, 256),
])
def test_blast(N, b, P, Q, R, dtype):
    import mem_efficient_blr_b200.blast_kernels as bk
    x, U, Vt, S = orc.make_blast_inputs(N, b * P, b * Q, b, R, dtype, seed=N + Q + R)
    want = orc.blast(x, U, Vt, S)[0].reshape(N, b * Q)
    xd, layer = x.reshape(N, b * P).to(DEV), tuple(t.to(DEV) for t in (U, Vt, S))
    _close(bk.blast_torch_layout(xd, *layer), want)
    _close(bk.triton_blast_partial_grouped_fp16(xd, *[t.to(DEV) for t in orc.blast_to_partial_layout(U, Vt, S)]), want)
    g = torch.Generator().manual_seed(1)
    bias, res = torch.randn(b * Q, generator=g).to(dtype), torch.randn(N, b * Q, generator=g).to(dtype)
    _close(bk.blast_multi_torch_layout(xd, [layer], biases=[bias.to(DEV)], residuals=[res.to(DEV)])[0], want + bias.float() + res.float())
    _close(bk.blast_multi_torch_layout(xd, [layer], biases=[bias.to(DEV)], out_act="gelu_tanh")[0],
           torch.nn.functional.gelu(want + bias.float(), approximate="tanh"))


@pytest.mark.parametrize("N,I,O,b,rank", [(40, 512, 1024, 4, 512), (128, 1024, 2752, 4, 1536), (300, 768, 1600, 4, 1024)])
def test_monarch(N, I, O, b, rank):
    """Rank / b a multiple of 128, or not: runs of outputs a plane apart."""
    import mem_efficient_blr_b200.monarch_kernels as mk
    x, w1, w2 = orc.make_monarch_inputs(N, I, O, b, rank, torch.float16, seed=N)
    want = orc.monarch(x, w1, w2)[0].reshape(N, O)
    w1k = orc.monarch_w1_to_kernel_layout(w1).to(DEV)
    _close(mk.triton_monarch_right_fp16(x.to(DEV), w1k, w2.to(DEV)), want)
    _close(mk.monarch_torch_layout(x.to(DEV), w1.to(DEV), w2.to(DEV)), want)


@pytest.mark.parametrize("N,I,O,R", [(17, 4096, 264, 256), (200, 2048, 1000, 1024), (400, 768, 3072, 128)])
def test_low_rank(N, I, O, R):
    import mem_efficient_blr_b200.low_rank_kernels as lk
    g = torch.Generator(device=DEV).manual_seed(N)
    x, V, U = (torch.randn(*s, generator=g, device=DEV).half() for s in ((N, I), (R, I), (O, R)))
    V, U = V / I ** 0.5, U / R ** 0.5
    want = ((x.float() @ V.float().t()).half().float() @ U.float().t()).cpu()
    _close(lk.low_rank_torch_layout(x, V, U), want)
    _close(lk.triton_low_rank_fp16(x, V.t().contiguous(), U.t().contiguous()), want)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,b,P,Q,R", [
    (9, 16, 256, 688, 1024),
    (11, 3, 72, 136, 520),     # ragged contractions, a second tile of 8 rows, ranks beyond a coupling CTA's
    (12, 13, 688, 40, 1488),   # the longest chain that comes here
    (16, 2, 1280, 8, 512),
])
def test_blast_up_to_16_tokens(N, b, P, Q, R, dtype):
    import mem_efficient_blr_b200.blast_kernels as bk
    x, U, Vt, S = orc.make_blast_inputs(N, b * P, b * Q, b, R, dtype, seed=N + Q + R)
    want = orc.blast(x, U, Vt, S)[0].reshape(N, b * Q)
    xd, layer = x.reshape(N, b * P).to(DEV), tuple(t.to(DEV) for t in (U, Vt, S))
    _close(bk.blast_torch_layout(xd, *layer), want)
    _close(bk.triton_blast_partial_grouped_fp16(xd, *[t.to(DEV) for t in orc.blast_to_partial_layout(U, Vt, S)]), want)
    g = torch.Generator().manual_seed(1)
    bias, res = torch.randn(b * Q, generator=g).to(dtype), torch.randn(N, b * Q, generator=g).to(dtype)
    _close(bk.blast_multi_torch_layout(xd, [layer], biases=[bias.to(DEV)], residuals=[res.to(DEV)])[0], want + bias.float() + res.float())


@pytest.mark.parametrize("N", [20, 128, 700])
def test_factors_that_the_call_before_writes(N):
    """The first factor comes from a GEMM of this library right ahead of the call, a long one: no stage may read it before that has finished."""
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.dense_kernels as dk
    b, P, Q, R, K = 16, 128, 64, 256, 4096
    g = torch.Generator(device=DEV).manual_seed(N)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV).half()
    x, U, S, B = rn(N, b * P), rn(b, Q, R) / R ** 0.5, rn(b, b, R), rn(P, K) / (K * P) ** 0.5
    for _ in range(3):
        A = rn(b * R, K)
        want = bk.blast_torch_layout(x, U, (V := dk.dense_torch_layout(A, B)).view(b, R, P).clone(), S)
        A2 = rn(b * R, K)
        torch.cuda.synchronize()
        V2 = dk.dense_torch_layout(A2, B)
        got = bk.blast_torch_layout(x, U, V2.view(b, R, P), S)
        torch.cuda.synchronize()
        assert torch.equal(got, bk.blast_torch_layout(x, U, V2.view(b, R, P), S)) and not torch.equal(got, want)
