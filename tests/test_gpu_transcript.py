"""The device's transcript steps at every alignment of the transcript: separators that put
the FRI roots and samples across block (64 bytes) and chunk (1024 bytes) boundaries and on
stacks of one to three subtrees, proof bytes against the oracle's."""
import pytest

from zs_b200 import wire
from zs_b200 import workload as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sep_len", [0, 1, 2, 3, 15, 31, 32, 46, 47, 48, 63, 64, 200, 300, 400, 500, 555, 601, 640, 702,
                                     777, 1007, 1500, 2031, 3300, 7000])
@pytest.mark.parametrize("trace_log", [5, 9])
def test_transcript_alignment(orc, trace_log, sep_len):
    from zs_b200 import native
    tr, pi = wl.seeded_fib(trace_log, 77 + sep_len)
    params = wire.StarkParams(trace_log, 2, 5, 3).encode()
    sep = bytes((7 * k + sep_len) & 0xff for k in range(sep_len))
    b = wire.columns(tr)
    assert native.prove(wl.AIR_SEEDED_FIB, params, pi, b, b"", sep) == \
        orc.prove(wl.AIR_SEEDED_FIB, params, pi, b"", b, sep)
