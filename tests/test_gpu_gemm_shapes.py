"""GPU parity of the tensor-core GEMM with TMA stores (csrc/umma_pair.cu) and its neighbour at the edges of their tiles and of the
choice between them: ragged last tiles, one and several waves, CTA pairs, store chunks of a permuted output, bias and activation."""
import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [
    # N, I, O                  what runs
    (129, 48, 4096 * 8),       # short contraction, a token tile of one
    (2100, 128, 1000),         # ... with a ragged last tile of columns
    (3000, 184, 104),          # ... one tile per block
    (2500, 688, 5000),         # pairs, ragged in both directions
    (5001, 1000, 2056),        # pairs, a narrow last tile of 8 columns
    (600, 4096, 1024),         # one wave of narrow tiles
])
def test_dense_shapes(shape, dtype):
    import mem_efficient_blr_b200.dense_kernels as dk
    N, I, O = shape
    x, Wt = orc.make_dense_inputs(N, I, O, dtype, seed=N)
    xd, Wd = x.reshape(N, I).to(DEV), Wt.to(DEV)
    want = xd.float() @ Wd.float().t()
    for got in (dk.dense_torch_layout(xd, Wd), dk.triton_dense_fp16(xd, Wd.t().contiguous())):
        assert orc.rel_fro(got.float().cpu(), want.cpu()) < 1e-2
        assert (got.float() - want).abs().max() < 0.05 * want.abs().max()


@pytest.mark.parametrize("act", [None, "gelu", "gelu_tanh"])
@pytest.mark.parametrize("shape", [
    # N, I, O, b, R
    (700, 768, 3072, 16, 288),    # Q = 192: single CTAs, additions in the epilogue
    (1300, 512, 800, 4, 256),     # Q = 200: a ragged tile
    (400, 1024, 16 * 264, 16, 704),  # pairs with additions
])
def test_bias_residual_and_activation(shape, act):
    import mem_efficient_blr_b200.blast_kernels as bk
    N, I, O, b, R = shape
    x, U, Vt, S = orc.make_blast_inputs(N, I, O, b, R, torch.float16, seed=N)
    g = torch.Generator().manual_seed(1)
    bias = torch.randn(O, generator=g).half()
    res = torch.randn(N, O, generator=g).half() if N <= 512 else None
    want = orc.blast(x, U, Vt, S)[0].reshape(N, O) + bias.float()
    if act is not None:
        want = torch.nn.functional.gelu(want, approximate="tanh" if act == "gelu_tanh" else "none")
    if res is not None:
        want = want + res.float()
    dev = lambda t: None if t is None else t.to(DEV)
    got = bk.blast_multi_torch_layout(dev(x.reshape(N, I)), [(dev(U), dev(Vt), dev(S))], biases=[dev(bias)], residuals=[dev(res)], out_act=act)[0]
    assert orc.rel_fro(got.float().cpu(), want) < 1e-2


@pytest.mark.parametrize("per", [64, 128, 96, 24])
def test_monarch_with_grouped_columns(per):
    """The first GEMM's output is permuted in runs of `per` columns: whole store chunks or not."""
    import mem_efficient_blr_b200.monarch_kernels as mk
    N, b = 900, 4
    x, w1, w2 = orc.make_monarch_inputs(N, 512, 640, b, b * per, torch.float16, seed=per)
    ref = orc.monarch(x, w1, w2)
    ref = ref[0] if isinstance(ref, tuple) else ref
    got = mk.triton_monarch_right_fp16(x.reshape(N, -1).to(DEV), orc.monarch_w1_to_kernel_layout(w1).contiguous().to(DEV), w2.to(DEV))
    assert orc.rel_fro(got.float().cpu(), ref.reshape(N, -1)) < 1e-2


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [
    # N, I, O, R
    (900, 11000, 264, 1488),   # three slices, the last one ragged
    (500, 16392, 264, 1032),   # a rank tile of 8 columns
    (1601, 16384, 512, 776),
])
def test_low_rank_in_slices(shape, dtype):
    """The first stage's contraction in slices with fp32 planes, both layouts of its weights."""
    import mem_efficient_blr_b200.low_rank_kernels as lk
    N, I, O, R = shape
    g = torch.Generator(device=DEV).manual_seed(N)
    x, V, U = (torch.randn(*s, generator=g, device=DEV).to(dtype) for s in ((N, I), (R, I), (O, R)))
    V, U = V / I ** 0.5, U / R ** 0.5
    want = (x.float() @ V.float().t()).to(dtype).float() @ U.float().t()
    for got in (lk.low_rank_torch_layout(x, V, U), lk.triton_low_rank_fp16(x, V.t().contiguous(), U.t().contiguous())):
        assert orc.rel_fro(got.float().cpu(), want.cpu()) < 1e-2
