"""The window forms of the LDG device streams (csrc/fp_stream.cu) against the
host streams: windows with no, a few and more than 32 positions with long lists
(a team of CTAs each, or a CTA each), windows shorter and longer than the grid
has CTAs, changed decisions walked or not, and a TV part limit that the stream
runs into.  Every field of the state is equal, or both refuse."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("part_vec", "ep_ends", "ep_parts", "ep_cnt", "part_sizes", "marker", "send", "recv")


def hubs(fp, nhub, every, seed, noe=1500, nov=6000):
    """nhub vertices of some noe * 15 / nhub nets each, one in `every` of the
    visiting order's first vertices; the other pins are spread."""
    rng = np.random.default_rng(seed)
    ids = np.arange(nhub) * every
    rest = np.setdiff1d(np.arange(nov), ids)
    nets = [np.concatenate([rng.choice(ids, size=min(15, nhub), replace=False),
                            rng.choice(rest, size=int(rng.integers(40, 90)), replace=False)]).astype(np.uint32)
            for _ in range(noe)]
    nptr = np.cumsum([0] + [len(n) for n in nets]).astype(np.uint32)
    hg = fp.Hypergraph.from_nets(nov, nptr, np.concatenate(nets))
    hg.weights = np.ascontiguousarray(np.diff(hg.vptr).astype(np.int32))
    return hg


CASES = [
    ("hubs100_row", lambda fp: hubs(fp, 100, 1, 1), 64),      # > 32 in a window
    ("hubs100_spread", lambda fp: hubs(fp, 100, 20, 2), 64),  # a few in a window
    ("hubs3_K200", lambda fp: hubs(fp, 3, 700, 3), 200),      # one per window, 500 nets or more
    ("hubs40_K2", lambda fp: hubs(fp, 40, 7, 4), 2),
    ("uniform20k", lambda fp: fp.generate(fp.GenSpec.column_net(20000, 20000, 2, 6, seed=5)), 8),   # long windows
]


@pytest.mark.parametrize("walk", (False, True))
@pytest.mark.parametrize("metric", ("TV", "MSRV", "CN"))
@pytest.mark.parametrize("name,mk,K", CASES, ids=[c[0] for c in CASES])
def test_stream_windows_match_host_stream(fp, gpu_engine, name, mk, K, metric, walk):
    hg = mk(fp)
    hg.weights = np.ascontiguousarray(np.diff(hg.vptr).astype(np.int32))
    want = fp.stream_partition(hg, K, metric)
    with gpu_engine.instance(hg, K, metric) as inst:
        inst.set_stream("device")
        inst.set_stream_walk(walk)
        inst.initial_partition()
        assert inst.streamed_on_device()
        got = inst.get_state()
    for f in FIELDS:
        np.testing.assert_array_equal(got[f], want[f], err_msg=f"{name} {metric} {f}")


@pytest.mark.parametrize("walk", (False, True))
@pytest.mark.parametrize("eps", (1.05, 1.5, 4.0))
def test_tv_part_limit_refused_alike(fp, gpu_engine, eps, walk):
    """With a capacity above TV's part limit a vertex may choose a part above
    the limit: the reference would use part -1, host and device refuse."""
    hg = hubs(fp, 40, 7, 6)

    def run(where):
        with gpu_engine.instance(hg, 8, "TV", eps) as inst:
            inst.set_stream(where)
            inst.set_stream_walk(walk)
            try:
                inst.initial_partition()
            except Exception as e:
                return type(e), str(e)
            return inst.get_state()["part_vec"].tolist()

    host, dev = run("host"), run("device")
    assert host == dev
