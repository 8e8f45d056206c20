"""Rules that choose between two forms of a product by its sizes, against what both were measured to take on a B200."""
import pytest

from inf_engine_b200 import kernels


# both products of a few tokens' experts, us: (hidden, intermediate, blocks of a few rows, through the ring)
@pytest.mark.parametrize("hidden,inter,blocks,ring", [(256, 256, 10.5, 11.6), (512, 256, 13.0, 13.5), (1024, 512, 58.0, 36.2), (1024, 1024, 37.4, 25.0), (2048, 2048, 82.2, 60.1)])
def test_experts_through_the_ring(hidden, inter, blocks, ring):
    assert kernels.moe_ring_pays(hidden, inter) == (ring < blocks)


# a block-diagonal product, us: (rows, k of a block, tiles of 64 rows, a warp an output)
@pytest.mark.parametrize("m,k,tiles,warps", [(8, 256, 15.3, 5.1), (16, 256, 15.4, 8.7), (1, 64, 4.7, 2.6), (8, 64, 4.7, 3.4), (16, 64, 4.9, 5.7),
                                             (4, 16, 2.1, 2.8), (16, 16, 2.2, 5.4), (16, 512, 36.7, 24.8), (17, 256, 15.7, 16.0)])
def test_gate_products_of_a_few_rows(m, k, tiles, warps):
    assert kernels.diag_rows_pay(m, k) == (warps < tiles)


# float32-arithmetic attention, us: (requests with few rows, requests, head size, one launch for all, two)
@pytest.mark.parametrize("n_small,n_requests,hd,one,two", [(4, 4, 64, 134, 21), (2, 3, 64, 170, 98), (8, 9, 96, 3449, 1597), (2, 3, 20, 74, 81),
                                                           (8, 9, 20, 487, 517), (4, 4, 20, 64, 15)])
def test_a_launch_of_its_own_for_decode_tokens(n_small, n_requests, hd, one, two):
    from inf_engine_b200.parts.attention import ordered_rows_pay
    assert ordered_rows_pay(n_small, n_requests, hd, hd) == (two < one)
    assert not ordered_rows_pay(0, n_requests, hd, hd)
