"""The commit of the CN engine (csrc/fp_spec_cn.cu) against the oracle: windows
that move few pins (their nets spread over the warps), nets shared by
acting nets whose lists are staged (up to 256 parts) and not, up to K parts per
list, and as many acting nets on one net as are staged (256) or more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def shared(fp, n_small, seed, nov=3000):
    """n_small nets of two or three pins, all of them on nets of nov / 2 pins and
    more, so that most acting nets share those."""
    rng = np.random.default_rng(seed)
    nets = [rng.choice(nov, size=int(rng.integers(2, 4)), replace=False) for _ in range(n_small)]
    nets += [rng.choice(nov, size=nov // 2 + 100 * i, replace=False) for i in range(4)]
    rng.shuffle(nets)
    nptr = np.cumsum([0] + [len(n) for n in nets]).astype(np.uint32)
    return fp.Hypergraph.from_nets(nov, nptr, np.concatenate(nets).astype(np.uint32))


CASES = [
    ("shared_K8", lambda fp: shared(fp, 3000, 1), 8),
    ("shared_K255", lambda fp: shared(fp, 2500, 2), 255),
    ("shared_K256", lambda fp: shared(fp, 2500, 3), 256),
    ("shared_K300", lambda fp: shared(fp, 2500, 4), 300),
    ("shared_K900", lambda fp: shared(fp, 2500, 5), 900),
    ("uniform_small_nets", lambda fp: fp.generate(fp.GenSpec.column_net(40000, 40000, 2, 3, seed=6)), 16),
    ("zipf", lambda fp: fp.generate(fp.GenSpec.zipf(20000, 20000, 2.1, 2, 5000, 1.5, 1, seed=7)), 64),
]


@pytest.mark.parametrize("window", (None, (16384, 4)), ids=("", "long"))
@pytest.mark.parametrize("name,mk,K", CASES, ids=[c[0] for c in CASES])
def test_cn_commit_matches_oracle(fp, orc, gpu_engine, name, mk, K, window):
    hg, passes = mk(fp), 3
    o = orc.run_oracle(hg, K, "CN", passes)
    if o["status"] != 0:
        pytest.skip("the reference's behaviour is undefined on this instance")
    with gpu_engine.instance(hg, K, "CN") as inst:
        if window:
            inst.set_window(*window)
        inst.initial_partition()
        inst.refine(passes)
        ln, pt, ct = inst.lists()
        np.testing.assert_array_equal(inst.partition(), o["part_vec"], err_msg=name)
        np.testing.assert_array_equal(ln, o["ep_len"])
        np.testing.assert_array_equal(orc.flat_lists(hg, ln, pt), orc.flat_lists(hg, o["ep_len"], o["ep_part"]))
        np.testing.assert_array_equal(ct, o["ep_cnt"])
        assert list(inst.moves(passes)) == list(o["moves"])
        assert inst.metrics() == o["metrics_final"]
