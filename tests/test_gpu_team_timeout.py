"""A bounded wait that gives up in one CTA of a team is known to all of them after
the team's next barrier: nobody ever completes the barrier that is waited for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [2, 4, 8])
def test_a_timeout_in_one_cta_reaches_the_team(size):
    from ps_claude_opt_b200 import native

    for rank in list(range(size)) + [size]:  # the last: none waits
        st = np.full(size, -1, dtype=np.int32)
        native._check(native.lib().ps_probe_team_timeout(1000, size, rank, st.ctypes.data_as(native._ip)))
        assert st.tolist() == [4 if rank < size else 0] * size  # PS_DEVSTAT_TIMEOUT
