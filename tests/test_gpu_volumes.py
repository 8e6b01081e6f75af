"""Volumes inside a window of the MSV / MSRV engine (csrc/fp_spec.cu) against
the oracle: accept tests taken again from listed terms where the max-volume
parts change in the window -- one part or several at the maximum, more changes
than a window keeps (15), under MSRV with listed parts off the old maximum --
movers that touch more parts than a list holds (64), and K from 2 to 700 (where
the terms are staged).  Partition, moves, metrics and decision records are
equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def broad(fp, seed):
    """4000 vertices; 30 lie on 200 nets each, of half of them as the source:
    their moves change the volumes of most parts."""
    rng = np.random.default_rng(seed)
    nov, nets = 4000, []
    for h in rng.choice(nov, size=30, replace=False):
        rest = np.setdiff1d(np.arange(nov), [h])
        for i in range(200):
            others = rng.choice(rest, size=int(rng.integers(1, 4)), replace=False)
            nets.append(np.concatenate([[h], others] if i % 2 else [others, [h]]).astype(np.uint32))
    for _ in range(3000):
        k = int(rng.integers(2, 6))
        nets.append(rng.choice(nov, size=k, replace=False).astype(np.uint32))
    nptr = np.cumsum([0] + [len(n) for n in nets]).astype(np.uint32)
    return fp.Hypergraph.from_nets(nov, nptr, np.concatenate(nets))


CASES = [
    ("uniform_K2", lambda fp: fp.generate(fp.GenSpec.column_net(3000, 3000, 2, 8, seed=1)), 2, 1.05),
    ("uniform_K3", lambda fp: fp.generate(fp.GenSpec.column_net(4000, 4000, 2, 12, seed=2)), 3, 1.1),
    ("uniform_K8", lambda fp: fp.generate(fp.GenSpec.column_net(6000, 6000, 2, 16, seed=3)), 8, 1.03),
    ("uniform_K33", lambda fp: fp.generate(fp.GenSpec.column_net(6000, 6000, 2, 16, seed=4)), 33, 1.05),
    ("zipf_K64", lambda fp: fp.generate(fp.GenSpec.zipf(8000, 8000, 2.2, 2, 1500, 0.0, 0, seed=5)), 64, 1.05),
    ("zipfw_K128", lambda fp: fp.generate(fp.GenSpec.zipf(20000, 20000, 2.1, 2, 3000, 1.5, 1, seed=6)), 128, 1.05),
    ("broad_K200", lambda fp: broad(fp, 7), 200, 1.05),
    ("broad_K400", lambda fp: broad(fp, 8), 400, 1.2),
    ("uniform_K700", lambda fp: fp.generate(fp.GenSpec.column_net(6000, 6000, 2, 16, seed=9)), 700, 1.5),
]


@pytest.mark.parametrize("window", (None, (16384, 4)), ids=("", "long"))
@pytest.mark.parametrize("metric", ("MSV", "MSRV"))
@pytest.mark.parametrize("name,mk,K,eps", CASES, ids=[c[0] for c in CASES])
def test_volumes_in_a_window_match_oracle(fp, orc, gpu_engine, name, mk, K, eps, metric, window):
    hg, passes = mk(fp), 3
    o = orc.run_oracle(hg, K, metric, passes, eps, records=True)
    with gpu_engine.instance(hg, K, metric, eps) as inst:
        if window:
            inst.set_window(*window)
        inst.set_decision_log(True)
        inst.initial_partition()
        if o["status"] != 0:
            with pytest.raises(fp.FastPartError):
                inst.refine(passes)
            return
        inst.refine(passes)
        np.testing.assert_array_equal(inst.partition(), o["part_vec"], err_msg=f"{name} {metric}")
        assert list(inst.moves(passes)) == list(o["moves"]), (name, metric)
        assert inst.metrics() == o["metrics_final"], (name, metric)
        d = inst.decisions()
        for k in ("dest", "gain", "loss", "moved"):
            np.testing.assert_array_equal(d[k], o[f"rec_{k}"], err_msg=k)
