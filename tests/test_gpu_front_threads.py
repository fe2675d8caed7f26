"""The operators of the Python front end leave the interpreter lock to other threads while the library waits."""
import threading
import time

import pytest
import torch

import portdnn_b200 as pd

pytestmark = pytest.mark.gpu


def test_a_waiting_launch_lets_other_threads_run():
    """Some 2500 launches behind half a second of other work fill the launch queue, and the next one waits for
    most of that time.  A second thread, which asks for a millisecond's sleep again and again, goes on."""
    x, done, gaps = torch.zeros(64, device="cuda"), threading.Event(), []
    pd.pointwise(pd.ACT_RELU, x, out=x)
    torch.cuda.synchronize()

    def beat():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(1e-3)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    other = threading.Thread(target=beat)
    other.start()
    began = time.perf_counter()
    torch.cuda._sleep(1_000_000_000)  # clock cycles: 0.5 s at the highest clock
    for _ in range(2500):
        pd.pointwise(pd.ACT_RELU, x, out=x)
    issued = time.perf_counter() - began
    torch.cuda.synchronize()
    done.set()
    other.join()
    assert issued > 0.25  # the launches did wait
    assert max(gaps) < 0.5 * issued
