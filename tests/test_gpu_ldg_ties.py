"""The LDG argmax where it can go wrong: many parts of one count whose order is
decided by size and first sighting (unit weights, small nets), K on both sides
of a warp's width, and every evaluation class (one warp, one CTA, the whole
grid) on the same instance, against the CPU oracle, whose results are integers
(compared for equality)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (light, super) work bounds: None leaves the defaults; small ones send most
# vertices of these instances to the CTA and the whole-grid evaluation
CLASSES = [None, (12, 40), (0, 8)]


@pytest.mark.parametrize("classes", CLASSES, ids=["default", "mixed", "grid"])
@pytest.mark.parametrize("K", [2, 31, 32, 33, 300])
@pytest.mark.parametrize("metric", ["TV", "MSV", "MSRV"])
def test_gpu_ldg_ties_match_oracle(fp, orc, gpu_engine, metric, K, classes):
    hg = fp.generate(fp.GenSpec.column_net(900, 800, 2, 7, seed=41 + K))
    o = orc.run_oracle(hg, K, metric, 3)
    assert o["status"] == 0
    with gpu_engine.instance(hg, K, metric) as inst:
        if classes:
            inst.set_classes(*classes)
        inst.initial_partition()
        inst.refine(3)
        ln, pt, ct = inst.lists()
        np.testing.assert_array_equal(inst.partition(), o["part_vec"])
        np.testing.assert_array_equal(inst.moves(3), o["moves"])
        np.testing.assert_array_equal(ln, o["ep_len"])
        np.testing.assert_array_equal(orc.flat_lists(hg, ln, pt), orc.flat_lists(hg, o["ep_len"], o["ep_part"]))
        np.testing.assert_array_equal(ct, o["ep_cnt"])
        assert inst.metrics() == o["metrics_final"]
