"""The circle LDE at every number of layers of its middle pass (one chunk, two equal or
unequal chunks, a split above 2^10), each blowup, ragged column counts: all values against
the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_rows,log_blowup,n_cols", [
    (10, 2, 3), (11, 0, 3), (11, 2, 5), (12, 1, 2), (13, 2, 3), (14, 3, 2), (15, 1, 7), (16, 2, 3), (17, 2, 2),
    (17, 0, 1), (18, 1, 3), (18, 2, 1), (19, 2, 1), (19, 0, 2), (21, 1, 1)])
def test_lde_matches_oracle(orc, log_rows, log_blowup, n_cols):
    from zs_b200 import native
    rng = np.random.default_rng(17 * log_rows + log_blowup)
    trace = rng.integers(0, 2**31 - 1, (n_cols, 1 << log_rows), dtype=np.uint32)
    trace[0, ::5] = 0
    trace[0, 1::5] = 2**31 - 2
    gammas = rng.integers(0, 2**31 - 1, (n_cols, 4), dtype=np.uint32)
    alphas = rng.integers(0, 2**31 - 1, (1, 4), dtype=np.uint32)
    want = orc.circle_commit(trace, log_blowup, gammas, alphas, keep_lde=True)
    plan = native.CommitPlan(n_cols, log_rows, log_blowup, 1)
    plan.set_challenges(gammas, alphas)
    plan.upload(trace)
    plan.run()
    got = plan.results()
    assert np.array_equal(plan.lde(), want["lde"])
    assert got["lde_root"] == want["lde_root"]
    assert np.array_equal(got["final_layer"], want["final_layer"])
    plan.close()
