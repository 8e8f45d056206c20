"""The gated delta rule's library compiles for head sizes whose outputs outgrow the first operands of the chunked form's last
kernel (narrow keys, wide values); a size that does not compile is a model that does not start."""
import pytest

from inf_engine_b200.csrc.build import build_library


@pytest.mark.parametrize("dk,dv", [(32, 128)])
def test_narrow_keys_and_wide_values_compile(dk, dv):
    assert build_library(f"gated_delta_k{dk}_v{dv}", ["gated_delta.cu"], {"IE_GD_DK": dk, "IE_GD_DV": dv}, verbose=False).is_file()
