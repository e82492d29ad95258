"""GPU parity of the two-launch path for any layout of 16-bit factors (csrc/skinny.cu), 1..16 tokens, at the edges of its tiles:
rank and output tiles with remainders, in-blocks cut into slices, one and both token tiles, all ways z is formed."""
import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOKENS = (1, 3, 8, 9, 16)


def _check(run, ref):
    got, again = run(), run()
    torch.cuda.synchronize()
    assert torch.equal(got, again)   # every sum has a fixed order
    assert orc.rel_fro(got.float().cpu().reshape(ref.shape), ref) < 1e-2


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [
    # I, O, b, R
    (16, 16, 2, 8),              # everything smaller than a tile
    (344 * 4, 104 * 4, 4, 72),   # remainders in the slice, the rank and the outputs
    (1568 * 2, 40 * 2, 2, 1000), # in-blocks of four slices
    (48 * 16, 688 * 16, 16, 136),
    (96 * 6, 264 * 6, 6, 1288),
    (128 * 9, 512 * 9, 9, 256),  # out-blocks of 16 tiles whose clusters would not all be resident with a tile per CTA
    (144 * 12, 40 * 12, 12, 1840), # clusters of two
])
def test_blast_layouts(shape, dtype):
    import mem_efficient_blr_b200.blast_kernels as bk
    I, O, b, R = shape
    for N in TOKENS:
        x, U, Vt, S = orc.make_blast_inputs(N, I, O, b, R, dtype, seed=N)
        ref = orc.blast(x, U, Vt, S)[0]
        xd = x.to(DEV)
        part, bmm = ([t.to(DEV) for t in f(U, Vt, S)] for f in (orc.blast_to_partial_layout, orc.blast_to_bmm_layout))
        _check(lambda: bk.triton_blast_partial_grouped_fp16(xd, *part), ref)
        _check(lambda: bk.triton_blast_bmm_fp16(xd, *bmm), ref)


@pytest.mark.parametrize("shape", [(512, 640, 4, 64), (512, 1056, 4, 96), (3136, 640, 2, 144), (1024, 768, 16, 256)])
def test_monarch_layouts(shape):
    import mem_efficient_blr_b200.monarch_kernels as mk
    I, O, b, R = shape
    for N in TOKENS:
        x, w1, w2 = orc.make_monarch_inputs(N, I, O, b, R, torch.float16, seed=N)
        ref = orc.monarch(x, w1, w2)[0]
        xd, w1d, w2d, w2l = (t.to(DEV) for t in (x, orc.monarch_w1_to_kernel_layout(w1), w2, orc.monarch_w2_to_left_layout(w2)))
        _check(lambda: mk.triton_monarch_right_fp16(xd, w1d, w2d), ref)
        _check(lambda: mk.triton_monarch_right_left_fp16(xd, w1d, w2l), ref)
        _check(lambda: mk.triton_monarch_right_ideal_fp16(xd, w1d, w2d), orc.monarch_ideal_order(ref, b))


@pytest.mark.parametrize("shape", [
    # I, O, R
    (16, 16, 8), (1008, 1008, 200), (11008, 272, 72), (6160, 512, 128),
    # a width whose eighths are odd: the grid-wide kernel (csrc/stream_kernel.cu)
    (8, 8, 8), (1000, 1008, 200), (11008, 264, 72),
])
def test_low_rank_layouts(shape):
    import mem_efficient_blr_b200.low_rank_kernels as lk
    I, O, R = shape
    for N in TOKENS:
        x, Vt, Ut = orc.make_low_rank_inputs(N, I, O, R, torch.float16, seed=N)
        ref = orc.low_rank(x, Vt, Ut)[0].reshape(N, O)
        xd, V, U = (t.to(DEV) for t in (x, Vt.t().contiguous(), Ut.t().contiguous()))
        _check(lambda: lk.triton_low_rank_fp16(xd, V, U), ref)


def test_rounded_intermediates():
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    x, U, Vt, S = orc.make_blast_inputs(5, 512, 768, 4, 128, torch.float16, seed=7)
    x = x * 4
    ref, _, _ = orc.blast_act_int8(x, U, Vt, S)
    xd, bmm = x.to(DEV), [t.to(DEV) for t in orc.blast_to_bmm_layout(U, Vt, S)]
    assert orc.rel_fro(bq.triton_blast_bmm_int8_fp16(xd, *bmm).float().cpu(), ref) < 3e-2


@pytest.mark.parametrize("shape", [(344 * 4, 104 * 4, 4, 72), (1568 * 2, 40 * 2, 2, 1000), (8192, 264 * 8, 8, 256)])
def test_fused_single_layer(shape):
    """down(silu(x) * m) + bias + residual in the two launches."""
    import mem_efficient_blr_b200.blast_kernels as bk
    I, O, b, R = shape
    for N in (1, 4, 8):
        x, U, Vt, S = orc.make_blast_inputs(N, I, O, b, R, torch.float16, seed=N)
        g = torch.Generator().manual_seed(N)
        xm, bias, res = (torch.randn(*s, generator=g).half() for s in ((N, I), (O,), (N, O)))
        x = x.reshape(N, I)
        xe = (torch.nn.functional.silu(x.float()).half().float() * xm.float()).half()
        ref = orc.blast(xe, U, Vt, S)[0].reshape(N, O) + bias.double() + res.double()
        xd, xmd, bd, rd, Ud, Vd, Sd = (t.to(DEV) for t in (x, xm, bias, res, U, Vt, S))
        _check(lambda: bk.blast_multi_torch_layout(xd, [(Ud, Vd, Sd)], x_mul=xmd, biases=[bd], residuals=[rd])[0], ref)


@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("shape", [(4096, 4096, 16, 1024), (1032 * 8, 264 * 8, 8, 1240)])
def test_fused_layers(shape, k):
    """Layers on one x in the two launches, each with additions of its own."""
    import mem_efficient_blr_b200.blast_kernels as bk
    I, O, b, R = shape
    for N in (k + 1, 8, 16):
        sets = [orc.make_blast_inputs(N, I, O, b, R, torch.float16, seed=10 * N + i) for i in range(k)]
        x = sets[0][0].reshape(N, I)
        g = torch.Generator().manual_seed(N)
        bias = [torch.randn(O, generator=g).half() if i != 1 else None for i in range(k)]
        dev = lambda t: None if t is None else t.to(DEV)
        outs = bk.blast_multi_torch_layout(dev(x), [tuple(dev(t) for t in s[1:]) for s in sets], biases=[dev(t) for t in bias])
        for s, t, got in zip(sets, bias, outs):
            ref = orc.blast(x, *s[1:])[0].reshape(N, O)
            ref = ref if t is None else ref + t.double()
            assert orc.rel_fro(got.float().cpu(), ref) < 1e-2
