"""Threads that refine instances of different K on their own contexts: the
kernels' limit of dynamic shared memory is one for the process, and a launch for a
small K must not lower it under another thread's launch for a large one."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOOPS = 400


@pytest.mark.parametrize("metric,Ks", [("TV", (16, 600)), ("TM", (16, 600))])
def test_threads_with_different_K(fp, orc, metric, Ks):
    hg = fp.generate(fp.GenSpec.column_net(600, 500, 2, 6, seed=93))
    want = {K: orc.run_oracle(hg, K, metric, 1) for K in Ks}
    assert all(o["status"] == 0 for o in want.values())
    failed = []

    def work(K):
        try:
            eng = fp.Engine(0)
            eng.set_sm_limit(48)   # both grids fit the device together
            with eng.instance(hg, K, metric) as inst:
                inst.initial_partition()
                for _ in range(LOOPS):
                    inst.reset_state()
                    inst.refine(1)
                np.testing.assert_array_equal(inst.partition(), want[K]["part_vec"])
            eng.close()
        except Exception as e:
            failed.append((K, repr(e)[:300]))

    threads = [threading.Thread(target=work, args=(K,)) for K in Ks]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
