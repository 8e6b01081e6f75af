"""MSM's max-message parts as a list and as a mask (csrc/fp_spec_msg.cu): part
counts around the words of the mask, many parts tied at the maximum and few,
against the oracle, decision records of a last pass included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log", [False, True], ids=["", "records"])
@pytest.mark.parametrize("K", [2, 31, 32, 33, 257, 512, 700])
@pytest.mark.parametrize("name", ["uniform", "mixed"])
def test_msm_max_parts_match_oracle(fp, orc, gpu_engine, name, K, log):
    if name == "uniform":   # few nets per part: most parts send the same number of messages
        hg = fp.generate(fp.GenSpec.column_net(1294, 728, 2, 16, seed=61))
    else:
        hg = fp.generate(fp.GenSpec.zipf(4000, 3900, 2.2, 2, 2000, seed=62))
    o = orc.run_oracle(hg, K, "MSM", 3, records=True)
    if o["status"] != 0:
        pytest.skip("the reference's behaviour is undefined on this instance")
    with gpu_engine.instance(hg, K, "MSM") as inst:
        inst.set_decision_log(log)
        inst.initial_partition()
        inst.refine(3)
        ln, pt, ct = inst.lists()
        np.testing.assert_array_equal(inst.partition(), o["part_vec"])
        np.testing.assert_array_equal(inst.moves(3), o["moves"])
        np.testing.assert_array_equal(orc.flat_lists(hg, ln, pt), orc.flat_lists(hg, o["ep_len"], o["ep_part"]))
        np.testing.assert_array_equal(ct, o["ep_cnt"])
        assert inst.metrics() == o["metrics_final"]
        if log:
            d = inst.decisions()
            for k in ("dest", "gain", "loss", "moved"):
                np.testing.assert_array_equal(d[k], o[f"rec_{k}"], err_msg=k)
