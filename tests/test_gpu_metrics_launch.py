"""fp_metrics as one launch (K up to 512) and as two (csrc/fp_metrics.cu) against
the oracle: repeated calls (each leaves its scratch zeroed), a changed state
between them, and fewer nets than a CTA takes."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noe", (3, 3000))
@pytest.mark.parametrize("K", (2, 33, 512, 513, 1500))
def test_metrics_launches_match_oracle(fp, orc, gpu_engine, K, noe):
    hg = fp.generate(fp.GenSpec.column_net(4000, noe, 2, 16, seed=K))
    o = orc.run_oracle(hg, K, "TV", 1)
    with gpu_engine.instance(hg, K, "TV") as inst:
        inst.initial_partition()
        for _ in range(3):
            assert inst.metrics() == o["metrics_init"]
        assert inst.last_launches() == (1 if K <= 512 else 2)
        if o["status"] == 0:
            inst.refine(1)
            for _ in range(2):
                assert inst.metrics() == o["metrics_final"]
