"""GPU: flux weights and kappa sums by blocks.

The kappa kernel takes 32 steps per block and adds partial sums over the
children; the flux kernel takes 32 children per block.  Step and child counts
around those against the oracle at the bars of the recrossing tests."""
import pytest

from conftest import rel_err
from test_gpu_recross import run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntraj,steps", [(2, 31), (32, 32), (34, 33), (66, 65)])
def test_blocks_match_oracle(require_gpu, ntraj, steps):
    (num, den, w, q, p, st), (onum, oden, ow, oq, op) = run_pair(ntraj, 4, steps)
    assert not st.any() and len(num) == steps
    assert rel_err(w, ow) <= 1e-12
    assert abs(den - oden) <= 1e-12 * abs(oden)
    assert rel_err(num / den, onum / oden) <= 1e-9
