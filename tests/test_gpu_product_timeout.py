"""The bounded waits of the transform's tensor-core product (csrc/fj_expand.cu):
one that runs out reaches a host-memory call's status, and the device stays
usable. The kernel waits ~1 ms for operands that are never sent and returns."""
import threading

import numpy as np
import pytest

from test_gpu_expand import _case, _run

pytestmark = pytest.mark.gpu


def test_timeout_reaches_the_call_s_flag(lib):
    case = _case(300, 200, 150, seed=3)
    before = _run(case)
    for _ in range(3):
        assert lib.ccfj_self_test_product_timeout(None) == 0, lib.ccfj_last_error()
        assert lib.ccfj_device_status(None) == 0  # not a transform's timeout
        assert np.array_equal(_run(case), before)  # nor a later call's


def test_flags_of_calls_in_other_threads(lib):
    """Calls that run beside timeouts of another thread report none."""
    case = _case(300, 200, 150, seed=3)
    want = _run(case)
    wrong, stop = [], threading.Event()

    def calls():
        while not stop.is_set():
            try:
                if not np.array_equal(_run(case), want):
                    wrong.append("bits")
            except Exception as e:  # noqa: BLE001
                wrong.append(repr(e))

    threads = [threading.Thread(target=calls) for _ in range(3)]
    for t in threads:
        t.start()
    try:
        status = [lib.ccfj_self_test_product_timeout(None) for _ in range(40)]
    finally:
        stop.set()
        for t in threads:
            t.join()
    assert status == [0] * 40 and not wrong
