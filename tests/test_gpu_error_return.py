"""A row-sharded fit whose all-reduce fails returns its error although the stream holds work that does not end
soon (a collective that waits for a peer: here a host function on the stream)."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_error_does_not_wait_for_a_stalled_stream(lib):
    cuda = ctypes.CDLL("libcuda.so.1")
    stall = ctypes.CFUNCTYPE(None, ctypes.c_void_p)(lambda _: time.sleep(5.0))
    rng = np.random.default_rng(0)
    X, Y = rng.standard_normal((100, 40)), rng.standard_normal((100, 2))

    def fail(buf, count, stream):
        if count > 40:
            assert cuda.cuLaunchHostFunc(ctypes.c_void_p(stream), stall, None) == 0
            raise RuntimeError("peer lost")
    lib.pls_model2_fast(X, Y, [3])
    t = time.perf_counter()
    with pytest.raises(RuntimeError, match="peer lost"):
        lib.pls_model2_fast(X, Y, [3], allreduce=fail)
    assert time.perf_counter() - t < 4.0   # two seconds, not five
    assert lib.pls_model2_fast(X, Y, [3])["n_components"] == 3
