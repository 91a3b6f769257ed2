"""-m gpu: a closed model's pool goes with the last array of it; other models' takes and gives do not wait for that."""
import threading
import time

import pytest

import test_gpu_result_pool as R

pytestmark = pytest.mark.gpu


def test_other_models_go_on_while_a_pool_goes(cuda, pkg):
    m = R.model(pkg)
    take, give = m.lib.c.pb200_result_take, m.lib.c.pb200_result_give
    block = take(m.h, 4096)                          # its slab stays
    goes, stop, ops = [], threading.Event(), []

    def close_others():
        for _ in range(6):
            o = R.model(pkg)
            b = take(o.h, R.POOL)
            o.close()
            t = time.perf_counter()
            assert give(b) == 0                      # the last of that pool
            goes.append((t, time.perf_counter()))
        stop.set()
    th = threading.Thread(target=close_others)
    th.start()
    while not stop.is_set():
        t = time.perf_counter()
        b = take(m.h, 4096)
        assert b and give(b) == 0
        ops.append((t, time.perf_counter()))
    th.join()
    assert len(goes) == 6
    longest = max(b - a for a, b in goes)
    inside = sum(1 for a, b in ops for s, e in goes if s <= a and b <= e)
    print("a pool goes in up to", longest, "s;", inside, "takes and gives meanwhile")
    assert longest > 2e-4 and inside >= 20           # held up, each of the six would have let one or two by
    assert give(block) == 0
    m.close()
