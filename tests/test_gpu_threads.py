"""Contexts on several host threads at once."""
import threading
import time

import numpy as np
import pytest

from helpers import gpu_system, random_system
from test_gpu_parity import random_system_fast

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,prec,engine,kcs", [(64, 0, "auto", (5, 40)),   # k rows in FP64
                                               (64, 1, "auto", (4, 16)),   # k rows in FP32
                                               (64, 1, "tc", (4, 25)),
                                               (64, 1, "simt", (4, 40)),
                                               (6001, 1, "auto", (16, 21))])  # mesh
def test_kernels_of_different_shared_memory(n, prec, engine, kcs):
    """Threads launch the same k-space kernels with the shared memory of different
    kc (steps with uploaded noise: launch by launch, no graph): each launch gets its
    own size, whatever another thread asked for last."""
    steps = 200 if n < 1000 else 20
    xi = np.zeros((steps, 3, 3, n))
    sims = []
    for k in range(10):
        ini, g = random_system(n, seed=n, rc_frac=0.3, phi=0.02) if n < 1000 else random_system_fast(n, n, 0.10, 0.02)
        g["kc"] = kcs[k % 2]
        sims.append(gpu_system(ini, g, prec, noise=1))
        if prec:
            sims[-1].set_kspace_engine(engine)
    failed, end = [], time.monotonic() + 2.0

    def work(s):
        try:
            while time.monotonic() < end and not failed:
                s.step(steps, 1e-15, xi=xi)
        except Exception as e:
            failed.append(e)

    th = [threading.Thread(target=work, args=(s,)) for s in sims]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not failed, failed[0]
