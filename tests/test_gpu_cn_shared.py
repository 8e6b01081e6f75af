"""CN windows whose acting nets share large nets, against the CPU oracle: few
nets of many pins over most vertices, many small nets around them, so that
several acting nets of one window move pins of the same large net (their order
decides its list), at K around the bounds on its number of parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [3, 4, 16, 64])
@pytest.mark.parametrize("big", [(3, 2000), (40, 200), (400, 24)], ids=["huge", "large", "mid"])
def test_gpu_cn_shared_nets_match_oracle(fp, orc, gpu_engine, K, big):
    rng = np.random.default_rng(61 + K)
    nov, (nbig, size) = 4000, big
    # vertices in a large net lie on one or two small nets more, pairs and triples
    nets = [rng.choice(nov, size=size, replace=False) for _ in range(nbig)]
    nets += [rng.choice(nov, size=int(s), replace=False) for s in rng.integers(2, 4, 5000)]
    order = rng.permutation(len(nets))
    nets = [nets[i].astype(np.uint32) for i in order]
    nptr = np.concatenate([[0], np.cumsum([n.size for n in nets])]).astype(np.uint32)
    hg = fp.Hypergraph.from_nets(nov, nptr, np.concatenate(nets))
    o = orc.run_oracle(hg, K, "CN", 3, records=True)
    assert o["status"] == 0
    with gpu_engine.instance(hg, K, "CN") as inst:
        inst.set_decision_log(True)
        inst.initial_partition()
        inst.refine(3)
        ln, pt, ct = inst.lists()
        np.testing.assert_array_equal(inst.partition(), o["part_vec"])
        np.testing.assert_array_equal(inst.moves(3), o["moves"])
        np.testing.assert_array_equal(ln, o["ep_len"])
        np.testing.assert_array_equal(orc.flat_lists(hg, ln, pt), orc.flat_lists(hg, o["ep_len"], o["ep_part"]))
        np.testing.assert_array_equal(ct, o["ep_cnt"])
        assert inst.metrics() == o["metrics_final"]
        d = inst.decisions()
        for k in ("dest", "gain", "loss", "moved"):
            np.testing.assert_array_equal(d[k], o[f"rec_{k}"], err_msg=k)


@pytest.mark.parametrize("log", [False, True])
@pytest.mark.parametrize("K", [2, 33, 100])
@pytest.mark.parametrize("metric", ["TM", "MSM"])
def test_gpu_message_metrics_skip_only_what_cannot_move(fp, orc, gpu_engine, metric, K, log):
    """Most vertices on no net, several max-message parts, whole-grid teams."""
    hg = fp.generate(fp.GenSpec.zipf(3000, 2500, 2.1, 2, 600, beta=1.5, seed=71 + K))
    o = orc.run_oracle(hg, K, metric, 3, records=True)
    assert o["status"] == 0
    with gpu_engine.instance(hg, K, metric) as inst:
        inst.set_classes(16, 60)
        inst.set_decision_log(log)
        inst.initial_partition()
        inst.refine(3)
        ln, pt, ct = inst.lists()
        np.testing.assert_array_equal(inst.partition(), o["part_vec"])
        np.testing.assert_array_equal(inst.moves(3), o["moves"])
        np.testing.assert_array_equal(orc.flat_lists(hg, ln, pt), orc.flat_lists(hg, o["ep_len"], o["ep_part"]))
        assert inst.metrics() == o["metrics_final"]
        if log:
            d = inst.decisions()
            for k in ("dest", "gain", "loss", "moved"):
                np.testing.assert_array_equal(d[k], o[f"rec_{k}"], err_msg=k)
