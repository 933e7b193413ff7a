"""The interpreter is free for other threads while a native call allocates and launches.
"""
import threading
import time

import pytest
import torch


@pytest.mark.gpu
def test_other_threads_run_during_a_call(cuda, tmp_path):
    """A call that waits for room in the launch queue (the GPU sleeps for about a
    second) does not hold the interpreter: another thread keeps ticking."""
    from libcpab_gb300 import Cpab
    T = Cpab([7], backend='pytorch', device='gpu', basis_dir=str(tmp_path))
    theta = torch.zeros(1, T.get_theta_dim(), device=cuda)
    pts = torch.rand(1, 64, device=cuda)
    for _ in range(3):
        T.transform_grid(pts, theta)
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.002)

    other = threading.Thread(target=tick)
    other.start()
    longest = 0.0
    try:
        torch.cuda._sleep(1_500_000_000)
        begin = time.perf_counter()
        while longest < 0.2 and time.perf_counter() - begin < 0.6:
            t0 = time.perf_counter()
            T.transform_grid(pts, theta)
            longest = max(longest, time.perf_counter() - t0)
    finally:
        stop.set()
        other.join()
        torch.cuda.synchronize()
    if longest < 0.2:
        pytest.skip('no call waited')
    gaps = [b - a for a, b in zip(ticks, ticks[1:])]
    assert max(gaps) < 0.1
