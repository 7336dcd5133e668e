"""Tensor parallelism, rank 0's side of a step (csrc/engine.cu wait_workers): it goes on when every worker has come as far as the step's
plan, and raises when one reported a failure, died or stays behind -- before anything of the step is used."""
import multiprocessing
import os
import threading
import time

import numpy as np
import pytest

from vllm_tgis_adapter_b200.engine import _lib


class Shared:
    def __init__(self):
        self.counters, self.failed, self.pids = np.zeros(16, np.uint64), np.zeros(16, np.int32), np.full(16, os.getpid(), np.int32)

    def wait(self, tp, seq, timeout):
        lib = _lib.load_library()
        rc = lib.tgis_k_tp_wait(self.counters.ctypes.data, self.failed.ctypes.data, self.pids.ctypes.data, tp, seq, timeout)
        return rc, _lib.last_error(lib) if rc else ""


def test_goes_on_once_every_worker_is_there():
    s = Shared()
    s.counters[1:4] = 7   # (entry 0, rank 0's own, is not looked at)
    assert s.wait(4, 7, 5.0)[0] == 0
    s.counters[2] = 6

    def later():
        time.sleep(0.2)
        s.counters[2] = 7

    t = threading.Thread(target=later)
    t.start()
    at = time.monotonic()
    assert s.wait(4, 7, 5.0)[0] == 0 and time.monotonic() - at > 0.1
    t.join()


@pytest.mark.parametrize("worker", [1, 3])
def test_a_worker_whose_results_are_not_valid_ends_the_step(worker):
    """Such a worker raises its flag and leaves its counter at the step before."""
    s = Shared()
    s.counters[1:4] = 7
    s.counters[worker], s.failed[worker] = 6, 1
    rc, message = s.wait(4, 7, 5.0)
    assert rc != 0 and f"rank {worker} reported a failure" in message


def test_a_dead_or_late_worker_ends_the_step():
    gone = multiprocessing.get_context("spawn").Process(target=time.sleep, args=(0,))
    gone.start()
    gone.join()
    s = Shared()
    s.pids[1] = gone.pid
    rc, message = s.wait(2, 1, 5.0)
    assert rc != 0 and "died" in message
    s.pids[1] = os.getpid()
    rc, message = s.wait(2, 1, 0.2)
    assert rc != 0 and "did not finish a step" in message
