"""Launches that come up while the one before them on the stream still writes what they read:
the forward transform's compact input and the sum-check tables that a fold's own launch leaves.
Inputs change from call to call at one shape, so that the buffers keep their addresses and a
value kept from the call before would show; everything against the oracle."""
import numpy as np
import pytest

from zs_b200 import wire

pytestmark = pytest.mark.gpu
NINE_POINTS = [([0, 1, 2, 0, 1, 2, 0, 1], 3), ([2], 5)]  # one point per pass: the fold has its own launch


@pytest.mark.parametrize("trace_log,log_blowup,n_cols", [(3, 1, 5), (9, 2, 40), (12, 3, 3), (16, 1, 2)])
def test_transform_reads_the_pass_before(orc, trace_log, log_blowup, n_cols):
    from zs_b200 import native
    rng = np.random.default_rng(41 * trace_log + n_cols)
    inputs = [wire.columns(list(rng.integers(0, 2**31 - 1, (n_cols, 1 << trace_log, 4), dtype=np.uint32)))
              for _ in range(3)]
    want = [orc.commit_columns(b, n_cols, trace_log, log_blowup) for b in inputs]
    for _ in range(3):
        assert [native.commit_columns(b, trace_log, log_blowup) for b in inputs] == want


@pytest.mark.parametrize("level,k,m,terms", [(3, 12, 3, NINE_POINTS), (7, 8, 41, [([0, 40], 5), ([7], 1)])])
def test_rounds_read_the_fold_before(orc, level, k, m, terms):
    from zs_b200 import native
    es = 1 if level == 3 else 16
    rng = np.random.default_rng(43 * k + m)
    inputs = [rng.bytes(m * (1 << k) * es) for _ in range(2)]
    want = [orc.binius_prove(level, t, k, m, terms) for t in inputs]
    for _ in range(3):
        assert [native.binius_prove_combination(8 if level == 3 else 128, t, k, m, terms) for t in inputs] == want
