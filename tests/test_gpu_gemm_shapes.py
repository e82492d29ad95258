"""GPU parity of the tensor-core GEMM with TMA stores (csrc/umma_pair.cu) and its neighbour at the edges of their tiles and of the
choice between them: ragged last tiles, one and several waves, CTA pairs, store chunks of a permuted output, bias and activation.
Every shape names the kernel it is there for: DIRECT (csrc/umma_gemm.cu), SINGLE or PAIRS (csrc/umma_pair.cu), checked against the rule."""
import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DIRECT, SINGLE, PAIRS = 0, 1, 2


def _route(G, M, K, N, run=0, additions=False):
    """The kernel of a shape; calls without additions run in both layouts of the weights here, and are meant for one kernel."""
    from mem_efficient_blr_b200 import _lib
    lib = _lib.load()
    kernel = lib.blr_debug_gemm_route(G, M, K, N, run, int(additions))
    if not additions:
        assert lib.blr_debug_gemm_choice(G, M, K, N, run, 0, _lib.MMAJOR, 16, None) == kernel
    return kernel


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [
    # N, I, O, kernel
    (129, 48, 4096 * 8, SINGLE),   # short contraction, a token tile of one
    (2100, 128, 1000, DIRECT),     # one wave, a ragged last tile of columns
    (2100, 128, 2312, SINGLE),     # ... several waves, a last tile of 8 columns
    (3000, 184, 104, DIRECT),      # one tile per block
    (2500, 688, 5000, DIRECT),     # ragged in both directions
    (5001, 1000, 2056, DIRECT),    # a narrow last tile of 8 columns
    (2500, 2504, 2056, PAIRS),     # all of that and a ragged contraction; a pair's second CTA with 68 tokens
    (2400, 2504, 2056, PAIRS),     # ... and with none
    (600, 4096, 1024, DIRECT),     # one wave of narrow tiles
])
def test_dense_shapes(shape, dtype):
    import mem_efficient_blr_b200.dense_kernels as dk
    N, I, O, kernel = shape
    assert _route(1, O, I, N) == kernel
    x, Wt = orc.make_dense_inputs(N, I, O, dtype, seed=N)
    xd, Wd = x.reshape(N, I).to(DEV), Wt.to(DEV)
    want = xd.float() @ Wd.float().t()
    for got in (dk.dense_torch_layout(xd, Wd), dk.triton_dense_fp16(xd, Wd.t().contiguous())):
        assert orc.rel_fro(got.float().cpu(), want.cpu()) < 1e-2
        assert (got.float() - want).abs().max() < 0.05 * want.abs().max()


@pytest.mark.parametrize("act", [None, "gelu", "gelu_tanh"])
@pytest.mark.parametrize("shape", [
    # N, I, O, b, R, kernel of the last GEMM
    (700, 768, 3072, 16, 288, DIRECT),         # Q = 192
    (1250, 768, 3072, 16, 288, SINGLE),        # ... several waves, a ragged token tile
    (1300, 512, 800, 4, 256, DIRECT),          # Q = 200: a ragged tile
    (4900, 512, 800, 4, 256, SINGLE),
    (400, 1024, 16 * 520, 16, 288, SINGLE),    # a residual; a last tile of 8 columns
    (400, 1024, 16 * 264, 16, 704, DIRECT),
    (3152, 512, 2048, 4, 1024, DIRECT),        # several waves of a long contraction
    (400, 1024, 16 * 512, 16, 1304, PAIRS),    # a residual, a ragged contraction and token tile
    (1000, 1024, 16 * 264, 16, 1600, PAIRS),   # a last tile of 8 columns
])
def test_bias_residual_and_activation(shape, act):
    import mem_efficient_blr_b200.blast_kernels as bk
    N, I, O, b, R, kernel = shape
    assert _route(b, O // b, R, N, additions=True) == kernel
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
    # a wrong column or row is not drowned in the norm of the rest
    assert (got.float().cpu() - want).abs().max() < 0.05 * want.abs().max()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [
    # N, I, O, b, R, kernel of the first GEMM
    (1250, 768, 512, 16, 104, SINGLE),     # one ragged tile per block
    (2500, 10016, 512, 4, 512, PAIRS),
])
def test_first_stages_plain_and_rounded(shape, dtype):
    """The intermediates as they are or rounded to integers by the GEMM's epilogue."""
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    N, I, O, b, R, kernel = shape
    assert _route(b, R, I // b, N) == kernel
    x, U, Vt, S = orc.make_blast_inputs(N, I, O, b, R, dtype, seed=N)
    x = x.reshape(N, I) * 4
    bmm = [t.to(DEV) for t in orc.blast_to_bmm_layout(U, Vt, S)]
    assert orc.rel_fro(bk.triton_blast_bmm_fp16(x.to(DEV), *bmm).float().cpu(), orc.blast(x, U, Vt, S)[0]) < 1e-2
    assert orc.rel_fro(bq.triton_blast_bmm_int8_fp16(x.to(DEV), *bmm).float().cpu(), orc.blast_act_int8(x, U, Vt, S)[0]) < 3e-2


@pytest.mark.parametrize("shape", [
    # N, I, rank / b, kernel of the first GEMM
    (900, 512, 64, DIRECT), (900, 512, 128, DIRECT), (900, 512, 96, DIRECT), (900, 512, 24, DIRECT),
    (4800, 512, 64, SINGLE), (4800, 512, 128, SINGLE), (4800, 512, 96, DIRECT),
    (2500, 4 * 2504, 128, PAIRS),
])
def test_monarch_with_grouped_columns(shape):
    """The first GEMM's output is permuted in runs of `per` columns: whole store chunks or not."""
    import mem_efficient_blr_b200.monarch_kernels as mk
    N, I, per, kernel = shape
    b = 4
    assert _route(b, b * per, I // b, N, run=per) == kernel
    x, w1, w2 = orc.make_monarch_inputs(N, I, 640, b, b * per, torch.float16, seed=per)
    ref = orc.monarch(x, w1, w2)
    ref = ref[0] if isinstance(ref, tuple) else ref
    got = mk.triton_monarch_right_fp16(x.reshape(N, -1).to(DEV), orc.monarch_w1_to_kernel_layout(w1).contiguous().to(DEV), w2.to(DEV))
    ref = ref.reshape(N, -1)
    assert orc.rel_fro(got.float().cpu(), ref) < 1e-2
    assert (got.float().cpu() - ref).abs().max() < 0.05 * ref.abs().max()


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


@pytest.mark.parametrize("bits", [16, 8, 4])
@pytest.mark.parametrize("shape", [
    # N, I, O, b, R: fewer tokens than a tile has rows, whose other rows are not copied
    (17, 1024, 16 * 40, 16, 128),     # the fewest; tiles of 32 and 64 rows, a ragged one
    (31, 512, 4 * 1000, 4, 192),      # a ragged box of tokens, tiles of several widths
    (64, 512, 4 * 992, 4, 1024),
    (112, 4 * 704, 4 * 104, 4, 320),
    (127, 4 * 256, 4 * 2696, 4, 128), # one row short of a tile
    (129, 4 * 256, 4 * 1352, 4, 128), # one more
])
def test_fewer_tokens_than_rows(shape, bits):
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    N, I, O, b, R = shape
    x, U, Vt, S = orc.make_blast_inputs(N, I, O, b, R, torch.float16, seed=N)
    xd, Ud, Vd, Sd = (t.to(DEV) for t in (x.reshape(N, I), U, Vt, S))
    if bits == 16:
        want = orc.blast(x, U, Vt, S)[0].reshape(N, O)
        calls = [lambda: bk.blast_torch_layout(xd, Ud, Vd, Sd),
                 lambda: bk.triton_blast_partial_grouped_fp16(xd, *[t.to(DEV) for t in orc.blast_to_partial_layout(U, Vt, S)])]
    else:
        Uq, us, Vq, vs = bq.quantize_blast_factors(Ud, Vd, bits)
        want = orc.blast_wq(x, Uq.cpu(), us.cpu(), Vq.cpu(), vs.cpu(), S, bits)[0].reshape(N, O)
        calls = [lambda: bq.blast_wq(xd, Uq, us, Vq, vs, Sd, bits)]
    for call in calls:
        got = call().reshape(N, O).float().cpu()
        assert orc.rel_fro(got, want) < 1e-2  # (the bound of the other tests of the pipeline: two roundings to 11 bits, observed 3e-4)
        assert (got - want).abs().max() < 0.05 * want.abs().max()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kernel,width,weights,b,Q,R,N,additions", [
    # every (kernel, tile width, kind of weights) that the choice returns for the last GEMM of a call, Q x R weights a block: ragged in rows,
    # contraction and tokens, most with several tiles
    (DIRECT, 32, "K", 2, 16, 72, 18, False),
    (DIRECT, 64, "K", 4, 624, 72, 18, False),
    (DIRECT, 96, "K", 9, 656, 72, 20, False),
    (DIRECT, 128, "K", 8, 1952, 72, 17, False),
    (DIRECT, 160, "K", 16, 1160, 72, 18, False),
    (DIRECT, 192, "K", 16, 1448, 72, 18, False),
    (DIRECT, 224, "K", 9, 3264, 72, 18, False),
    (DIRECT, 256, "K", 8, 4040, 72, 19, False),
    (DIRECT, 64, "M", 2, 72, 72, 18, False),
    (DIRECT, 128, "M", 16, 608, 72, 17, False),
    (DIRECT, 192, "M", 6, 3088, 72, 17, False),
    (DIRECT, 256, "M", 8, 3576, 72, 19, False),
    (DIRECT, 64, "int8", 2, 72, 96, 17, False),
    (DIRECT, 128, "int8", 9, 1040, 96, 17, True),
    (DIRECT, 192, "int8", 16, 1168, 96, 17, True),
    (DIRECT, 256, "int8", 8, 3696, 96, 17, False),
    (DIRECT, 64, "int4", 2, 72, 96, 17, False),
    (DIRECT, 128, "int4", 8, 1168, 96, 17, False),
    (DIRECT, 192, "int4", 9, 2120, 96, 17, True),
    (DIRECT, 256, "int4", 16, 1800, 96, 17, False),
    (SINGLE, 32, "K", 16, 24, 208, 1187, True),
    (SINGLE, 64, "K", 9, 120, 208, 2063, True),
    (SINGLE, 96, "K", 6, 72, 72, 3302, True),
    (SINGLE, 128, "K", 16, 264, 80, 516, False),
    (SINGLE, 160, "K", 16, 136, 72, 1215, False),
    (SINGLE, 192, "K", 16, 1248, 72, 130, True),
    (SINGLE, 224, "K", 9, 200, 72, 2213, False),
    (SINGLE, 256, "K", 8, 3568, 72, 134, True),
    (SINGLE, 64, "M", 8, 56, 72, 2314, False),
    (SINGLE, 128, "M", 16, 264, 72, 522, False),
    (SINGLE, 192, "M", 16, 1192, 72, 130, False),
    (SINGLE, 256, "M", 16, 1928, 72, 129, False),
    (PAIRS, 64, "K", 16, 40, 608, 1259, False),
    (PAIRS, 128, "K", 16, 264, 360, 581, True),
    (PAIRS, 192, "K", 16, 520, 728, 135, True),
    (PAIRS, 256, "K", 16, 784, 784, 130, True),
    (PAIRS, 128, "M", 16, 296, 360, 521, False),
    (PAIRS, 256, "M", 16, 648, 712, 135, False),
])
def test_every_kernel_width_and_kind_of_weights(kernel, width, weights, b, Q, R, N, additions, dtype):
    import ctypes
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    from mem_efficient_blr_b200 import _lib
    bits, tile = {"int8": 8, "int4": 4}.get(weights, 16), ctypes.c_int()
    lib = _lib.load()
    layout = _lib.MMAJOR if weights == "M" else _lib.KMAJOR
    assert lib.blr_debug_gemm_choice(b, Q, R, N, 0, int(additions), layout, bits, ctypes.byref(tile)) == kernel and tile.value == width
    x, U, Vt, S = orc.make_blast_inputs(N, b * 32, b * Q, b, R, dtype, seed=N + width)
    xd, Ud, Vd, Sd = (t.to(DEV) for t in (x.reshape(N, -1), U, Vt, S))
    bias = torch.randn(b * Q, generator=torch.Generator().manual_seed(1)).to(dtype) if additions else None
    if bits != 16:
        Uq, us, Vq, vs = bq.quantize_blast_factors(Ud, Vd, bits)
        want = orc.blast_wq(x, Uq.cpu(), us.cpu(), Vq.cpu(), vs.cpu(), S, bits)[0]
        got = (bq.blast_wq_multi(xd, [(Uq, us, Vq, vs, Sd)], bits, 0, biases=[bias.to(DEV)])[0] if additions else bq.blast_wq(xd, Uq, us, Vq, vs, Sd, bits))
    else:
        want = orc.blast(x, U, Vt, S)[0]
        if weights == "M":
            got = bk.triton_blast_partial_grouped_fp16(xd, *[t.to(DEV) for t in orc.blast_to_partial_layout(U, Vt, S)])
        elif additions:
            got = bk.blast_multi_torch_layout(xd, [(Ud, Vd, Sd)], biases=[bias.to(DEV)])[0]
        else:
            got = bk.blast_torch_layout(xd, Ud, Vd, Sd)
    want = want.reshape(N, -1) + (0 if bias is None else bias.float())
    got = got.reshape(N, -1).float().cpu()
    assert orc.rel_fro(got, want) < 1e-2  # (two roundings to 11 | 8 bits: observed 5e-4 | 4e-3, the largest element 6e-4 | 5e-3 of the largest value)
    # a wrong row, column or tile is not drowned in the norm of the rest
    assert (got - want).abs().max() < 0.05 * want.abs().max()
