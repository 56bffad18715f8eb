"""The state-space scan of prompt blocks (state_space.cu): thread blocks per SM, and blocks of more rows than it keeps step
sizes for at a time."""
import numpy as np
import pytest

from nerva_b200.session import CudaHfDecodeSequenceSession, SmokeStatus
from tests import vamidra_models as M
from tests import vamidra_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("state,blocks", [(16, 2), (128, 2), (129, 1), (256, 1)])
def test_thread_blocks_per_sm(built_lib, state, blocks):
    assert built_lib.nerva_b200_state_space_scan_blocks_per_sm(state) >= blocks


@pytest.mark.parametrize("state", [128, 200])
@pytest.mark.parametrize("count", [256, 257, 320, 577])
def test_blocks_of_more_rows_than_steps_are_kept_for(built_lib, state, count):
    cfg = M.config([M.space(ff=0, heads=4, groups=2, state=state, norm_groups=1)])
    w = M.weights(cfg)
    tokens = M.tokens(cfg, count)
    s = CudaHfDecodeSequenceSession(M.checkpoint(cfg, w), count, compute="bfloat16")
    assert s.status == SmokeStatus.OK, s.error
    got = s.append(tokens, range(count), reset=True)
    assert M.worst_position(got, O.forward(cfg, w, tokens)) < 2 * M.TOLERANCE["bfloat16"]
    assert np.array_equal(got, s.append(tokens, range(count), reset=True))
    s.destroy()
