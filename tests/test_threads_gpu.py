"""A thread in an op does not hold the interpreter: the others run while its launches wait for room in the queue."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("name", ["qk", "sapa_fused", "deform_sapa_fused", "module"])
def test_other_threads_run(name):
    import sapa_b200 as sp
    q, k, v, o = (torch.randn(*s, device=DEV) for s in ((1, 8, 16, 16), (1, 8, 8, 8), (1, 8, 8, 8), (1, 36, 16, 16)))
    m = sp.SAPA(32, embedding_dim=16).to(DEV)
    y, x = torch.randn(1, 32, 16, 16, device=DEV), torch.randn(1, 32, 8, 8, device=DEV)
    call = {"qk": lambda: sp.qk(q, k, 5, 2), "sapa_fused": lambda: sp.sapa_fused(q, k, v, 5, 2),
            "deform_sapa_fused": lambda: sp.deform_sapa_fused(q, k, v, o, 9, 2, 2), "module": lambda: m(y, x)}[name]
    with torch.no_grad():
        call()
    torch.cuda.synchronize()
    done = []

    def work():
        with torch.no_grad():
            torch.cuda._sleep(int(1e9))      # half a second at 2 GHz, in which the queue (about a thousand launches) fills
            for _ in range(2500):
                call()
        done.append(True)
    thread = threading.Thread(target=work)
    thread.start()
    longest, last = 0.0, time.perf_counter()
    while not done and thread.is_alive():
        time.sleep(0.001)      # a spinning thread would cost every call of the other one a switch interval
        now = time.perf_counter()
        longest, last = max(longest, now - last), now
    thread.join()
    torch.cuda.synchronize()
    assert done and longest < 0.15
