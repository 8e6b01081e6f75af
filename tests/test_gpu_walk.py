"""Windows whose decisions change with the part sizes (the LDG engine's walk),
against the CPU oracle: unit weights with most vertices on no net (each takes
the least-loaded part, which its own kind moves), ties of small nets, more
candidates than a staged row holds, windows around the staged chunk sizes, and
vertices of every evaluation class.  Integer results, compared for equality,
decision records included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graphs(fp):
    G = fp.GenSpec
    return {
        # 2/3 of the vertices lie on no net, hubs on most nets
        "zipf_unit": G.zipf(2500, 2300, 2.1, 2, 800, beta=1.5, seed=51),
        "mixed_unit": G.zipf(3001, 2900, 2.2, 2, 1500, seed=52),
        "colnet_unit": G.column_net(3000, 3100, 2, 16, seed=53),
        # degree weights: vertices without nets are left out of the positions
        "zipf_degree": G.zipf(6000, 5000, 2.1, 2, 900, beta=1.5, weight_rule=1, seed=54),
    }


@pytest.mark.parametrize("window", [(0, 4), (1, 1), (33, 2), (2048, 4)], ids=lambda w: f"w{w[0]}x{w[1]}")
@pytest.mark.parametrize("K", [3, 64, 100])
@pytest.mark.parametrize("name", ["zipf_unit", "mixed_unit", "colnet_unit", "zipf_degree"])
@pytest.mark.parametrize("metric", ["TV", "MSV", "MSRV"])
def test_gpu_walk_matches_oracle(fp, orc, gpu_engine, metric, name, K, window):
    hg = fp.generate(graphs(fp)[name])
    if window == (33, 2):   # some vertices without nets weigh nothing, others do; shuffled order
        rng = np.random.default_rng(7)
        hg.weights = rng.integers(0, 3, hg.nov).astype(np.int32)
        hg.ordering = rng.permutation(hg.nov).astype(np.int32)
    o = orc.run_oracle(hg, K, metric, 2, eps_factor=1.03, records=True)
    if o["status"] != 0:
        pytest.skip("the reference's behaviour is undefined on this instance")
    with gpu_engine.instance(hg, K, metric, 1.03) as inst:
        inst.set_window(*window)
        if window == (2048, 4):
            inst.set_classes(24, 400)
        inst.set_decision_log(True)
        inst.initial_partition()
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


@pytest.mark.parametrize("metric", ["TV", "MSV"])
def test_gpu_changes_taken_at_once_match_oracle(fp, orc, gpu_engine, metric):
    """Windows of thousands of positions with few changed decisions: all of
    them are redone at once and the window is validated again."""
    hg = fp.generate(fp.GenSpec.zipf(100_003, 60_000, 2.1, 2, 10_000, beta=1.5, weight_rule=1, seed=7))
    K = 256 if metric == "TV" else 64
    o = orc.run_oracle(hg, K, metric, 2)
    assert o["status"] == 0
    with gpu_engine.instance(hg, K, metric) as inst:
        inst.set_window(8192, 4)
        inst.initial_partition()
        inst.refine(2)
        ln, pt, ct = inst.lists()
        np.testing.assert_array_equal(inst.partition(), o["part_vec"])
        np.testing.assert_array_equal(inst.moves(2), o["moves"])
        np.testing.assert_array_equal(orc.flat_lists(hg, ln, pt), orc.flat_lists(hg, o["ep_len"], o["ep_part"]))
        np.testing.assert_array_equal(ct, o["ep_cnt"])
        assert inst.metrics() == o["metrics_final"]
