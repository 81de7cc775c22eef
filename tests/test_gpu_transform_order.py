"""The host transforms are ordered after what the caller has queued on the default stream: an
asynchronous copy into the input, still behind other work when the call is made, is part of it.
Outputs against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cols,log_n", [(1, 10), (12, 16), (5, 18)])
@pytest.mark.parametrize("inverse", [False, True])
def test_pending_copy_into_the_input(orc, n_cols, log_n, inverse):
    import torch
    from zs_b200 import native
    call, oracle_call = (native.circle_ifft, orc.circle_ifft) if inverse else (native.circle_fft, orc.circle_fft)
    rng = np.random.default_rng(61 * log_n + n_cols)
    x = rng.integers(0, 2**31 - 1, (n_cols, 1 << log_n), dtype=np.uint32)
    want = np.stack([oracle_call(c) for c in x])
    d = torch.from_numpy(x.view(np.int32)).cuda()
    pinned = torch.zeros((n_cols, 1 << log_n), dtype=torch.int32).pin_memory()
    host = pinned.numpy().view(np.uint32)
    a = torch.randn(4096, 4096, device="cuda")
    for _ in range(3):
        pinned.zero_()
        torch.cuda.synchronize()
        for _ in range(40):  # tens of milliseconds of work before the copy
            a = torch.tanh(a @ a)
        pinned.copy_(d, non_blocking=True)
        assert np.array_equal(call(host), want)
    torch.cuda.synchronize()
