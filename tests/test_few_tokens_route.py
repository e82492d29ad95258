"""Which layers go through the tensor-core GEMMs at 16 tokens or fewer (pure host logic; the calls themselves: test_gpu_wq_gemm.py, test_gpu_rows_gemm.py)."""
import pytest

from mem_efficient_blr_b200 import _lib


def _route(n, bits, b, inp, out, R, host=0):
    return _lib.load().blr_debug_few_tokens_route(n, bits, host, b, inp // b, out // b, R)


@pytest.mark.parametrize("bits", [16, 8, 4])
@pytest.mark.parametrize("shape", [(16, 4096, 11008, 1024), (16, 4096, 4096, 1024), (8, 6144, 6144, 512)])
def test_calls_from_host_buffers_keep_the_fewer_launches(bits, shape):
    assert _route(16, bits, *shape) and not any(_route(n, bits, *shape, host=1) for n in range(1, 17))
