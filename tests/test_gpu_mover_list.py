"""A position decided again several times in one window (a mover, then staying
home, then a mover again) keeps its one entry in the window's mover list, which
has room for one entry per position: light vertices redone by their warps, medium
and whole-grid ones by a CTA, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("classes", [None, (4, 40), (0, 0)], ids=["light", "medium", "grid"])
@pytest.mark.parametrize("K", [3, 8])
@pytest.mark.parametrize("name", ["mixed", "uniform"])
def test_redone_movers_keep_their_entry(fp, orc, gpu_engine, name, K, classes):
    if name == "mixed":
        hg = fp.generate(fp.GenSpec.zipf(12000, 8000, 2.2, 2, 2000, seed=56))
    else:
        hg = fp.generate(fp.GenSpec.column_net(3000, 3100, 2, 16, seed=53))
    o = orc.run_oracle(hg, K, "MSV", 2, eps_factor=1.03)
    assert o["status"] == 0
    with gpu_engine.instance(hg, K, "MSV", 1.03) as inst:
        if classes:
            inst.set_classes(*classes)
        inst.initial_partition()
        inst.refine(2)
        ln, pt, ct = inst.lists()
        np.testing.assert_array_equal(inst.partition(), o["part_vec"])
        np.testing.assert_array_equal(inst.moves(2), o["moves"])
        np.testing.assert_array_equal(ln, o["ep_len"])
        np.testing.assert_array_equal(orc.flat_lists(hg, ln, pt), orc.flat_lists(hg, o["ep_len"], o["ep_part"]))
        np.testing.assert_array_equal(ct, o["ep_cnt"])
        assert inst.metrics() == o["metrics_final"]
        if classes is None:   # (windows of whole-grid vertices hold few positions)
            assert inst.stats()["relisted"] > 0
