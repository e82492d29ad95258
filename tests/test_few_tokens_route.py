"""Which layers go through the tensor-core GEMMs at 16 tokens or fewer (pure host logic; the calls themselves: test_gpu_wq_gemm.py, test_gpu_rows_gemm.py)."""
import pytest

from mem_efficient_blr_b200 import _lib


def _route(n, bits, b, inp, out, R, host=0):
    return _lib.load().blr_debug_few_tokens_route(n, bits, host, b, inp // b, out // b, R)


@pytest.mark.parametrize("bits", [16, 8, 4])
@pytest.mark.parametrize("shape", [(16, 4096, 11008, 1024), (16, 4096, 4096, 1024), (8, 6144, 6144, 512)])
def test_calls_from_host_buffers_keep_the_fewer_launches(bits, shape):
    assert _route(16, bits, *shape) and not any(_route(n, bits, *shape, host=1) for n in range(1, 17))


@pytest.mark.parametrize("n,bits,b,P,Q,R", [
    (4, 8, 2, 1408, 1760, 64),     # few CTAs: 5.9 us on the two-launch path, 9.4 as GEMMs
    (5, 8, 2, 1088, 3848, 256),    # 6.3 | 9.1
    (9, 4, 16, 224, 144, 1536),    # more CTAs than SMs: 13.0 | 17.4
    (9, 16, 3, 216, 832, 1208),    # 7.3 | 10.2
    (12, 16, 2, 728, 40, 928),     # 7.3 | 10.0
    (9, 16, 8, 184, 88, 1024),     # 7.4 | 9.4
    (9, 16, 16, 328, 480, 1328),   # 15.4 | 18.3
])
def test_layers_that_the_two_launches_serve_faster(n, bits, b, P, Q, R):
    assert _route(n, bits, b, b * P, b * Q, R) == 1


@pytest.mark.parametrize("n,bits,b,P,Q,R", [
    (9, 8, 16, 256, 688, 1024), (16, 4, 16, 256, 688, 1024),   # 15.9 | 12.3, 16.2 | 12.2
    (16, 8, 16, 192, 48, 288),                                 # 9.3 | 7.9
    (9, 16, 16, 256, 688, 1024), (16, 16, 16, 256, 256, 1024), (16, 16, 16, 688, 256, 1488), (16, 16, 8, 768, 768, 512),
])
def test_layers_that_the_gemms_serve_faster(n, bits, b, P, Q, R):
    assert _route(n, bits, b, b * P, b * Q, R) == 2


def test_tokens_and_sizes_that_never_go_there():
    assert [_route(n, 8, 8, 6144, 6144, 512) > 0 for n in range(1, 17)] == [n >= 4 for n in range(1, 17)]
    assert [_route(n, 8, 8, 6144, 6144, 544) > 0 for n in range(1, 17)] == [n >= 9 for n in range(1, 17)]
    assert [_route(n, 16, 16, 4096, 4096, 512) > 0 for n in range(1, 17)] == [n >= 9 for n in range(1, 17)]
    assert [_route(n, 16, 16, 11008, 4096, 1488) > 0 for n in range(1, 17)] == [n >= 12 for n in range(1, 17)]
    assert not any(_route(n, 16, 16, 4096, 4096, 504) for n in range(1, 17))
    assert not any(_route(n, 4, 16, 16 * 1056, 4096, 1024) for n in range(1, 17))


def test_the_benchmark_names_the_kernels_of_its_points():
    import bench
    assert [(bits, n, bench.group_of(bits, n), bench.launches_of(bits, n)) for bits in (8, 4) for n in (1, 4, 16)] == [
        (bits, n, "gemms" if n == 16 else "two_launch", 2 if n == 1 else 3) for bits in (8, 4) for n in (1, 4, 16)]
