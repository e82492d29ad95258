"""Which GEMMs take the weights as the rows of their tiles (pure host logic; the numbers of shares are those of 148 SMs)."""
import pytest

from mem_efficient_blr_b200 import _lib

K, M = _lib.KMAJOR, _lib.MMAJOR


def _shares(G, rows, contraction, n, layout, bits=16, run=0):
    return _lib.load().blr_debug_gemm_rows(G, rows, contraction, n, run, 0, layout, bits)


@pytest.mark.parametrize("G,rows,contraction,n,layout", [
    (1, 768, 3072, 60, K), (1, 768, 3072, 218, K), (1, 4096, 11008, 27, K), (1, 4096, 4096, 384, K),   # long rows of a single block
    (1, 7048, 3344, 49, M), (1, 984, 3256, 36, M),                                                   # output-contiguous rows off 32 bytes
    (1, 11000, 1224, 340, M), (1, 10664, 792, 340, K),                                               # results off 32 bytes
])
def test_where_narrow_tiles_were_measured_ahead(G, rows, contraction, n, layout):
    assert _shares(G, rows, contraction, n, layout) == 0


@pytest.mark.parametrize("G,rows,contraction,n,layout", [
    (16, 688, 1024, 128, K), (16, 688, 1488, 128, M), (4, 2752, 1536, 128, M), (1, 4096, 1024, 128, M), (16, 1024, 688, 24, K), (1, 7040, 3344, 49, M),
    (2, 808, 1672, 49, K), (1, 11000, 1224, 49, M), (8, 1000, 512, 340, K),
])
def test_where_the_weights_are_the_rows(G, rows, contraction, n, layout):
    assert _shares(G, rows, contraction, n, layout) > 0


def test_quantised_weights_wherever_the_copies_can_store():
    for n in (17, 333, 1000, 5000):
        assert _shares(16, 688, 1024, n, K, 8) >= (n + 383) // 384 and _shares(16, 688, 1024, n, K, 4) >= (n + 383) // 384
        assert _shares(4, 1002, 1024, n, K, 8) == 0 and _shares(4, 64, 128, n, K, 8, run=16) == 0
    assert _shares(16, 688, 1024, 385, K) == 0   # (16-bit weights: up to the tokens of one CTA)
