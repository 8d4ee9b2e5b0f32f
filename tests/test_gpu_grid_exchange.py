"""The bounded waits of the one-launch solves (needs a B200).

Their blocks wait for words and sums of other blocks.  The library's self-test makes one block of a
small cooperative launch leave before it sends its word or adds to a sum: the others must give up
after the stated limit and the error must reach the host.  So must an error that one block reports
while the block that stores the solve's state knows nothing of it.  Up to 32 blocks read one
another's words, more go through block 0; block 0 itself can be the one that leaves.
"""
import ctypes as C
import time

import pytest

pytestmark = pytest.mark.gpu

NONE, NO_WORD, NO_SUM, REPORTS = range(4)


def _run(blocks, who, failure, limit_s):
    from phast_b200 import _lib
    err, passed = C.c_int(-1), C.c_int(-1)
    t0 = time.perf_counter()
    st = _lib.load().phastb_test_grid_exchange(blocks, who, failure, limit_s, C.byref(err), C.byref(passed))
    return st, err.value, passed.value, time.perf_counter() - t0


@pytest.mark.parametrize("blocks", [1, 2, 32, 33, 148])
def test_exchange_passes(blocks):
    from phast_b200 import _lib
    assert _run(blocks, 0, NONE, 1.0)[:3] == (_lib.OK, 0, blocks)


@pytest.mark.parametrize("blocks,who", [(8, 0), (8, 5), (100, 0), (100, 70)])
@pytest.mark.parametrize("failure", [NO_WORD, NO_SUM])
def test_wait_runs_out(blocks, who, failure):
    from phast_b200 import _lib
    st, err, passed, secs = _run(blocks, who, failure, 0.02)
    assert (st, err, passed) == (_lib.ERR_CUDA, 1, 0) and secs < 5.0
    assert _run(blocks, who, NONE, 1.0)[:3] == (_lib.OK, 0, blocks)  # the context stays usable


@pytest.mark.parametrize("blocks,who", [(8, 5), (100, 70)])
def test_reported_failure_survives_the_state(blocks, who):
    from phast_b200 import _lib
    assert _run(blocks, who, REPORTS, 1.0)[:3] == (_lib.ERR_CUDA, 1, blocks)
