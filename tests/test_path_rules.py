"""Rules that choose between two forms of a product by its sizes, against what both were measured to take on a B200."""
import pytest

from inf_engine_b200 import kernels


# both products of a few tokens' experts, us: (hidden, intermediate, blocks of a few rows, through the ring)
@pytest.mark.parametrize("hidden,inter,blocks,ring", [(256, 256, 10.5, 11.6), (512, 256, 13.0, 13.5), (1024, 512, 58.0, 36.2), (1024, 1024, 37.4, 25.0), (2048, 2048, 82.2, 60.1)])
def test_experts_through_the_ring(hidden, inter, blocks, ring):
    assert kernels.moe_ring_pays(hidden, inter) == (ring < blocks)
