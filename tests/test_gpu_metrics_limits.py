"""fp_metrics at the part counts where its shared memory crosses the 48 KB that
a launch may have without the opt-in (static and dynamic together: K = 3008 on;
dynamic alone: K = 3073 on) and at the largest K, and with instances of several K
alive at once (the kernel has one limit for all of them), against the oracle."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hg(fp):
    return fp.generate(fp.GenSpec.column_net(6000, 2500, 2, 16, seed=91))


def expected(orc, hg, K):
    return orc.run_oracle(hg, K, "TV", 0)["metrics_init"]


@pytest.mark.parametrize("K", (3007, 3008, 3072, 3073, 4096))
def test_metrics_at_shared_memory_limits(orc, gpu_engine, hg, K):
    with gpu_engine.instance(hg, K, "TV") as inst:
        inst.initial_partition()
        for _ in range(2):
            assert inst.metrics() == expected(orc, hg, K)


@pytest.mark.parametrize("Ks", ((4096, 3100, 16), (16, 3100, 4096), (3100, 4096, 3008)), ids=lambda k: "-".join(map(str, k)))
def test_metrics_of_instances_alive_together(orc, gpu_engine, hg, Ks):
    insts = []
    try:
        for K in Ks:
            insts.append(gpu_engine.instance(hg, K, "TV"))
            insts[-1].initial_partition()
        for i in (0, 1, 2, 1, 0):
            assert insts[i].metrics() == expected(orc, hg, Ks[i])
    finally:
        for inst in insts:
            inst.close()


@pytest.mark.parametrize("K", (16, 700))
def test_metrics_under_changed_sm_limits(fp, orc, hg, K):
    eng = fp.Engine(0)   # (its own context: the limit is the context's)
    try:
        with eng.instance(hg, K, "TV") as inst:
            inst.initial_partition()
            for sms in (1, 7, 0):   # limits set after the instance was made
                eng.set_sm_limit(sms)
                assert inst.metrics() == expected(orc, hg, K)
    finally:
        eng.close()
