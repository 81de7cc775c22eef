"""Column trees at the sizes where their launches change: one subtree, a subtree and its
top, each of the wide launches (2^17, 2^20 and 2^21 digests in the set) and sets of more
than 64 trees, roots against the oracle."""
import numpy as np
import pytest

from zs_b200 import wire

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trace_log,log_blowup,n_cols", [
    (0, 1, 1), (1, 1, 3), (7, 1, 1), (8, 1, 2), (11, 1, 1), (13, 3, 1), (7, 2, 65), (9, 2, 64), (11, 2, 15),
    (11, 2, 16), (15, 2, 1), (18, 2, 1), (19, 2, 1), (12, 2, 130)])
def test_column_tree_launches(orc, trace_log, log_blowup, n_cols):
    from zs_b200 import native
    rng = np.random.default_rng(31 * trace_log + n_cols)
    cols = rng.integers(0, 2**31 - 1, (n_cols, 1 << trace_log, 4), dtype=np.uint32)
    b = wire.columns(list(cols))
    assert native.commit_columns(b, trace_log, log_blowup) == orc.commit_columns(b, n_cols, trace_log, log_blowup)
