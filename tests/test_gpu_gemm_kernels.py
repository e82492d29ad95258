"""Each GEMM kernel on shapes that it, and not the one with the weights as the rows of its tiles (csrc/umma_wq.cu), takes, and that one at every number of shares:
the last GEMM of a call against the oracle, the kernel checked against the choice."""
import ctypes

import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DIRECT, SINGLE, PAIRS = 0, 1, 2


def _call(dtype, weights, b, Q, R, N, additions, seed, P=32):
    """(result, reference) of a BLAST call whose last GEMM has b groups of Q rows over R."""
    import mem_efficient_blr_b200.blast_kernels as bk
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    bits = {"int8": 8, "int4": 4}.get(weights, 16)
    x, U, Vt, S = orc.make_blast_inputs(N, b * P, b * Q, b, R, dtype, seed=seed)
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
    return got.reshape(N, -1).float().cpu(), want.reshape(N, -1) + (0 if bias is None else bias.float())


def _close(got, want):
    assert orc.rel_fro(got, want) < 1e-2  # (two roundings to 11 | 8 bits, as in test_gpu_gemm_shapes.py)
    # a wrong row, column or tile is not drowned in the norm of the rest
    assert (got - want).abs().max() < 0.05 * want.abs().max()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kernel,width,weights,b,Q,R,N,additions", [
    (DIRECT, 32, "K", 2, 88, 360, 900, False),
    (DIRECT, 64, "K", 2, 928, 360, 385, False),
    (DIRECT, 96, "K", 6, 280, 264, 600, False),
    (DIRECT, 128, "K", 2, 296, 136, 2063, False),
    (DIRECT, 256, "K", 9, 952, 72, 400, False),
    (DIRECT, 64, "M", 2, 712, 520, 400, False),
    (DIRECT, 128, "M", 2, 1760, 264, 513, False),
    # quantised: blocks of outputs that are no multiple of 8
    (DIRECT, 64, "int8", 6, 268, 352, 17, False),
    (DIRECT, 128, "int8", 4, 3308, 352, 17, True),
    (DIRECT, 192, "int8", 6, 1124, 224, 500, True),
    (DIRECT, 256, "int8", 8, 1836, 288, 400, False),
    (DIRECT, 64, "int4", 2, 548, 224, 130, False),
    (DIRECT, 128, "int4", 8, 660, 352, 300, False),
    (DIRECT, 192, "int4", 8, 2860, 224, 200, True),
    (DIRECT, 256, "int4", 8, 1988, 352, 200, False),
    (SINGLE, 192, "K", 6, 2232, 264, 390, True),
    (SINGLE, 256, "K", 9, 1544, 104, 385, True),
    (PAIRS, 192, "K", 8, 1176, 520, 385, True),
    (PAIRS, 256, "K", 16, 960, 1048, 385, True),
    (PAIRS, 256, "M", 8, 1912, 1048, 385, False),
])
def test_tokens_as_the_rows(kernel, width, weights, b, Q, R, N, additions, dtype):
    from mem_efficient_blr_b200 import _lib
    lib, tile, bits = _lib.load(), ctypes.c_int(), {"int8": 8, "int4": 4}.get(weights, 16)
    layout = _lib.MMAJOR if weights == "M" else _lib.KMAJOR
    assert lib.blr_debug_gemm_choice(b, Q, R, N, 0, int(additions), layout, bits, ctypes.byref(tile)) == kernel and tile.value == width
    assert lib.blr_debug_gemm_rows(b, Q, R, N, 0, int(additions), layout, bits) == 0
    _close(*_call(dtype, weights, b, Q, R, N, additions, N + width))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("weights,shares,N,b,Q,R", [
    # 16 bits: every number of shares, ragged rows, contraction and tokens
    ("K", 1, 24, 9, 1072, 928), ("K", 1, 349, 16, 1016, 760), ("K", 2, 17, 3, 104, 928), ("K", 2, 362, 9, 848, 80), ("K", 3, 377, 4, 1224, 328),
    ("K", 4, 364, 16, 168, 696), ("K", 5, 379, 4, 816, 328), ("K", 6, 84, 3, 352, 432), ("K", 6, 375, 2, 328, 216),
    ("M", 1, 381, 16, 1144, 472), ("M", 2, 348, 16, 416, 920), ("M", 3, 309, 9, 592, 312), ("M", 4, 50, 2, 96, 96), ("M", 5, 338, 9, 304, 496),
    ("M", 6, 365, 9, 64, 328),
    ("int8", 7, 333, 2, 136, 160), ("int4", 3, 800, 16, 264, 352),
])
def test_weights_as_the_rows(weights, shares, N, b, Q, R, dtype):
    from mem_efficient_blr_b200 import _lib
    bits = {"int8": 8, "int4": 4}.get(weights, 16)
    assert _lib.load().blr_debug_gemm_rows(b, Q, R, N, 0, 0, _lib.MMAJOR if weights == "M" else _lib.KMAJOR, bits) == shares
    _close(*_call(dtype, weights, b, Q, R, N, False, N + Q))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [2056, 4104, 8192, 8200])
def test_rmsnorm_of_long_rows(d, dtype):
    """Rows of two and four pieces a thread, and longer ones, which are read twice."""
    from mem_efficient_blr_b200 import ops
    g = torch.Generator().manual_seed(d)
    x, w = (torch.randn(3, d, generator=g) * 3).to(dtype), (1 + 0.1 * torch.randn(d, generator=g)).to(dtype)
    want = x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-5) * w.float()
    got = ops.rmsnorm(x.to(DEV), w.to(DEV), 1e-5).float().cpu()
    # (one rounding to 11 | 8 bits, on top of a few of fp32)
    assert ((got - want).abs() <= want.abs() * (2 ** -11 if dtype == torch.float16 else 2 ** -8) * 1.01 + 2 ** -24).all()
