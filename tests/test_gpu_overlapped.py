"""Launches that come up while the one before them on the stream still writes what they read:
the forward transform's compact input. Inputs change from call to call at one shape, so that the buffers keep their addresses and a
value kept from the call before would show; everything against the oracle."""
import numpy as np
import pytest

from zs_b200 import wire

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trace_log,log_blowup,n_cols", [(3, 1, 5), (9, 2, 40), (12, 3, 3), (16, 1, 2)])
def test_transform_reads_the_pass_before(orc, trace_log, log_blowup, n_cols):
    from zs_b200 import native
    rng = np.random.default_rng(41 * trace_log + n_cols)
    inputs = [wire.columns(list(rng.integers(0, 2**31 - 1, (n_cols, 1 << trace_log, 4), dtype=np.uint32)))
              for _ in range(3)]
    want = [orc.commit_columns(b, n_cols, trace_log, log_blowup) for b in inputs]
    for _ in range(3):
        assert [native.commit_columns(b, trace_log, log_blowup) for b in inputs] == want
