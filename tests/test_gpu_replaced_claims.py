"""Windows whose list of replaced moves' claims is full: the change without room
ends the window in front of it, and the next window decides it anew, so results
do not depend on the room (none, one entry, a few, all), for light, medium and
whole-grid vertices, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("classes", [None, (4, 40), (0, 0)], ids=["light", "medium", "grid"])
@pytest.mark.parametrize("room", [0, 1, 64, 700])
@pytest.mark.parametrize("metric", ["TV", "MSV", "MSRV"])
def test_gpu_full_list_matches_oracle(fp, orc, gpu_engine, metric, room, classes):
    hg = fp.generate(fp.GenSpec.zipf(3001, 2900, 2.2, 2, 1500, seed=52))
    K = 8
    o = orc.run_oracle(hg, K, metric, 2, eps_factor=1.03, records=True)
    assert o["status"] == 0
    with gpu_engine.instance(hg, K, metric, 1.03) as inst:
        if classes:
            inst.set_classes(*classes)
        inst.set_decision_log(True)
        inst.initial_partition()
        inst.refine(2)
        roomy = inst.stats()["cut_size"]
        inst.debug_replaced_room(room)
        inst.reset_state()
        inst.refine(2)
        ln, pt, ct = inst.lists()
        np.testing.assert_array_equal(inst.partition(), o["part_vec"])
        np.testing.assert_array_equal(inst.moves(2), o["moves"])
        np.testing.assert_array_equal(ln, o["ep_len"])
        np.testing.assert_array_equal(orc.flat_lists(hg, ln, pt), orc.flat_lists(hg, o["ep_len"], o["ep_part"]))
        np.testing.assert_array_equal(ct, o["ep_cnt"])
        assert inst.metrics() == o["metrics_final"]
        d = inst.decisions()
        for k in ("dest", "gain", "loss", "moved"):
            np.testing.assert_array_equal(d[k], o[f"rec_{k}"], err_msg=k)
        if room == 0 and metric != "MSRV":
            assert inst.stats()["cut_size"] > roomy   # windows ended at a change without room
        with pytest.raises(fp.FastPartError):
            inst.debug_replaced_room(-1)
