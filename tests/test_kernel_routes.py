"""Which kernel a call goes to, where the sizes decide it on the host: no GPU is needed."""
import pytest

from vitna_anchor_b200 import ops


# (tokens, q and k heads, v heads, their sizes, taps): what the slices of channels were measured to be slower or faster at than a block a token
@pytest.mark.parametrize("sizes,sliced", [
    ((64, 16, 32, 128, 128, 4), False), ((65, 1, 2, 16, 16, 4), False), ((400, 2, 4, 32, 64, 4), False), ((592, 2, 2, 20, 12, 4), False), ((1183, 2, 2, 20, 12, 4), False),
    ((200, 3, 9, 64, 64, 4), False), ((65, 3, 9, 64, 64, 2), False), ((400, 1, 1, 512, 64, 4), False), ((400, 1, 1, 1024, 64, 4), False), ((4000, 1, 2, 64, 64, 5), False),
    ((65, 4, 16, 128, 128, 4), True), ((400, 3, 9, 64, 64, 4), True), ((600, 2, 4, 32, 64, 4), True), ((600, 1, 1, 1024, 64, 4), True), ((1185, 1, 2, 16, 16, 4), True)])
def test_delta_rule_preparation(sizes, sliced):
    assert (ops.lib().vk_delta_prepare_slices(*sizes) > 0) == sliced
