"""GPU parity of the coupling kernel above 16 tokens (csrc/couple.cu) at the edges of its tiles: block counts around 8 and
16, a rank tile with a remainder, one token tile and more than a CTA's share of them, both ways the factors are fetched."""
import pytest
import torch

from oracle import blr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

SHAPES = [
    # N, b, b_out, R
    (17, 2, 2, 8),         # one piece of 8 ranks
    (32, 8, 8, 72),        # eight blocks: one step of in-blocks; a rank tile of 8
    (33, 9, 9, 64),        # nine blocks: the second step mostly empty; a token tile of one
    (48, 16, 16, 136),     # few tiles: out-blocks shared out over two CTAs
    (257, 16, 3, 200),     # a slice of the out-blocks
    (700, 12, 12, 1032),   # more token tiles than CTAs of a rank tile
    (1500, 5, 5, 256),
    (33, 4, 4, 72),        # few tiles of 4, 6 and 8 blocks: the sums on the CUDA cores, out-blocks shared out unevenly
    (65, 6, 6, 136),
    (40, 8, 3, 64),
    (33, 3, 2, 72),        # ... of 2 and 3 blocks
    (1030, 2, 2, 640),     # 330 tiles of two blocks: one step of in-blocks again
    (17, 5, 5, 8),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", SHAPES)
def test_coupling_edges(shape, dtype):
    import mem_efficient_blr_b200.blast_kernels as bk
    N, b, bo, R = shape
    x, U, Vt, S = orc.make_blast_inputs(N, 16 * b, 24 * b, b, R, dtype, seed=N + b)
    ref = orc.blast(x, U, Vt, S)[0].reshape(N, -1)
    xd, Ud, Vd, Sd = (t.to(DEV) for t in (x.reshape(N, -1), U[:bo].contiguous(), Vt, S[:bo].contiguous()))
    got = bk.blast_output_blocks(xd, Ud, Vd, Sd)
    assert orc.rel_fro(got.float().cpu(), ref[:, :bo * 24]) < 1e-2
    if bo == b:  # the factors of a rank contiguous
        got = bk.triton_blast_bmm_fp16(xd, *(t.to(DEV) for t in orc.blast_to_bmm_layout(U, Vt, S)))
        assert orc.rel_fro(got.float().cpu(), ref) < 1e-2


def test_coupling_rounds_like_the_reference():
    import mem_efficient_blr_b200.blast_sym_quant_kernels as bq
    x, U, Vt, S = orc.make_blast_inputs(300, 256, 384, 16, 128, torch.float16, seed=3)
    x = x * 4
    ref, _, _ = orc.blast_act_int8(x, U, Vt, S)
    got = bq.triton_blast_bmm_int8_fp16(x.to(DEV), *(t.to(DEV) for t in orc.blast_to_bmm_layout(U, Vt, S)))
    assert orc.rel_fro(got.float().cpu(), ref) < 3e-2
