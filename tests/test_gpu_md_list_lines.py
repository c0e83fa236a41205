"""The list builds where the line between a warp a leaf and a thread an atom lies
for each leaf width: the lists are exactly the pairs within r_c + skin."""
import pytest

from test_gpu_md_list_widths import _check

pytestmark = pytest.mark.gpu


# 152 SMs: 76, 77 blocks of 256 (leaves of 1), 152, 153 (of 2), 305 (of 16, 32)
@pytest.mark.parametrize("n,apl", [(19456, 1), (19458, 1), (38912, 2), (38914, 2), (77840, 16),
                                   (77856, 32)])
def test_lists_at_the_lines(nd, oracle, n, apl):
    side = (n / 0.83) ** (1.0 / 3.0)
    _check(nd, oracle, nd.synth.uniform_positions_mindist(n, n, side, 0.8), side, apl)
