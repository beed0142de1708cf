"""After a timeout a CTA waits, with a limit, for the last copy it issued on each
barrier before its shared memory is released: the wait ends at once where that
copy has landed or none was issued, and runs out where it has not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("uses", [0, 1, 2, 3, 7, 8])
def test_wait_is_for_the_last_copy(uses):
    from ps_claude_opt_b200 import native

    st = np.full(1, -1, dtype=np.int32)
    for done in range(max(0, uses - 1), uses + 1):
        native._check(native.lib().ps_probe_last_wait(1000, uses, done, st.ctypes.data_as(native._ip)))
        assert st[0] == (0 if done == uses else 4)  # PS_DEVSTAT_TIMEOUT
