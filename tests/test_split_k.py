"""Split counts of the weight-gradient products."""
import pytest

from param_decomp_b200.ops.site_linear import _split_k_for


@pytest.mark.parametrize("M,N", [(8, 8), (256, 256), (768, 1024), (512, 4096), (4096, 768), (4096, 14336)])
def test_no_split_is_empty_and_short_products_stay_whole(M, N):
    for K in (*range(1, 2048, 37), 2047):
        assert _split_k_for(M, N, K) == 1
    for K in range(2048, 40000, 61):
        s, blocks = _split_k_for(M, N, K), (K + 63) // 64
        per = -(-blocks // s)  # what the kernel gives each split
        assert 1 <= s <= 8 and (s - 1) * per < blocks, (K, s)
