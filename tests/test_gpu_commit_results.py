"""A commit plan's results where their copies change: final layers of up to 256 KB come back in
one copy with the roots, larger ones in their own; without folds; and with any output left out.
Against the oracle."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cols,log_rows,log_blowup,n_folds", [
    (3, 9, 2, 0), (2, 12, 1, 1), (2, 13, 1, 0), (1, 14, 1, 0), (2, 13, 2, 1), (5, 10, 2, 12), (1, 16, 1, 16)])
def test_results_at_every_copy(orc, n_cols, log_rows, log_blowup, n_folds):
    from zs_b200 import native
    rng = np.random.default_rng(71 * log_rows + n_folds)
    trace = rng.integers(0, 2**31 - 1, (n_cols, 1 << log_rows), dtype=np.uint32)
    gammas = rng.integers(0, 2**31 - 1, (n_cols, 4), dtype=np.uint32)
    alphas = rng.integers(0, 2**31 - 1, (n_folds, 4), dtype=np.uint32)
    want = orc.circle_commit(trace, log_blowup, gammas, alphas)
    plan = native.CommitPlan(n_cols, log_rows, log_blowup, n_folds)
    plan.set_challenges(gammas, alphas)
    plan.upload(trace)
    plan.run()
    for left_out in range(8):
        root = np.full(32, 0xa5, dtype=np.uint8)
        layers = np.full((n_folds, 32), 0xa5, dtype=np.uint8)
        final = np.full(want["final_layer"].shape, 0xa5a5a5a5, dtype=np.uint32)
        pointers = [root.ctypes.data_as(native.u8p), layers.ctypes.data_as(native.u8p),
                    final.ctypes.data_as(native.u32p)]
        for bit in range(3):
            if left_out >> bit & 1:
                pointers[bit] = None
        native.check(native.lib().zs_m31_commit_plan_results(plan._h, ctypes.c_void_p(0), *pointers), "results")
        assert (bytes(root) == want["lde_root"]) if not left_out & 1 else (root == 0xa5).all()
        assert np.array_equal(layers, want["layer_roots"]) if not left_out & 2 else (layers == 0xa5).all()
        assert np.array_equal(final, want["final_layer"]) if not left_out & 4 else (final == 0xa5a5a5a5).all()
    plan.close()
