"""Performance cases: the calls a user of the partitioner makes, over the sizes it is used at.

Every case runs through the package's public entry points.  The hypergraphs
come from the seeded generator with the repository's own distributions:

  mix      the requests of the mixed batch (``serving.mixed_batch``): Zipf(2.2)
           net sizes up to 2,000 pins, uniformly drawn pins, unit weights,
           K a power of two up to 512
  uniform  the column-net pattern of the ``uniform16k`` workload: nets of 2-16
           pins, unit weights, K = 8, C = (W / K) * 1.03
  zipf     the ``zipf4m`` workload at smaller sizes: Zipf(2.1) net sizes up to
           10,000 pins, Zipf(1.5) vertex popularity (a few hub vertices on most
           nets, most vertices on none), vertex weight = degree, K = 256;
           ``unit`` runs it with unit weights, the reference's own setting

and four kinds of call:

  refine   ``reset_state`` (host -> device state), ``refine(passes)``, the six
           metrics and the part vector back on the host
  metrics  the six metrics of a given partition
  stream   the streaming initial partition, the metrics and the part vector
  inverse  the net -> pins transpose of a vertex -> nets CSR, host to host
"""
import math

import numpy as np

import fastpartitioner_gb300 as fp

ORDER = tuple(fp.OUTPUT_ORDER)


def _refine(name, graph, nov, noe, K, metric, passes, unit=1, eps=1.05):
    return dict(name=name, kind="refine", graph=graph, nov=nov, noe=noe, unit=unit, K=K, metric=metric, passes=passes,
                eps=eps)


def listed():
    return [
        # the smallest call: the metrics of a partition somebody hands in, where
        # launches and the synchronisation are all there is
        dict(name="metrics_1k", kind="metrics", graph="mix", nov=1000, noe=1000, unit=1, K=16),
        # the CPU-sized workload of the reference, whole schedule of five passes
        _refine("refine_tv_uniform16k", "uniform", 16384, 16384, 8, "TV", 5, eps=1.03),
        # a small request of the mixed batch under the send-volume metric
        _refine("refine_msv_mix10k", "mix", 10007, 10000, 64, "MSV", 3),
        # the benchmark's hypergraph with unit weights, the reference's setting
        _refine("refine_tv_zipf16k_unit", "zipf", 16384, 16384, 64, "TV", 1),
        # the benchmark's hypergraph and K, each of the six metrics
        _refine("refine_cn_zipf256k", "zipf", 262144, 262144, 256, "CN", 3, unit=0),
        _refine("refine_tv_zipf1m", "zipf", 1048576, 1048576, 256, "TV", 3, unit=0),
        _refine("refine_tm_zipf256k", "zipf", 262144, 262144, 256, "TM", 5, unit=0),
        _refine("refine_msm_zipf1m", "zipf", 1048576, 1048576, 256, "MSM", 10, unit=0),
        _refine("refine_msv_zipf256k", "zipf", 262144, 262144, 256, "MSV", 3, unit=0),
        _refine("refine_msrv_zipf256k", "zipf", 262144, 262144, 256, "MSRV", 10, unit=0),
        # where the initial partition comes from
        dict(name="stream_tv_zipf256k", kind="stream", graph="zipf", nov=262144, noe=262144, unit=0, K=256,
             metric="TV"),
        # a driver's file as vertices -> nets, turned into nets -> pins
        dict(name="inverse_zipf1m", kind="inverse", graph="zipf", nov=1048576, noe=1048576),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["refine"] * 6 + ["metrics", "stream", "inverse"])
    ratio = math.exp(rng.uniform(math.log(0.5), math.log(1.5)))
    if kind == "inverse":
        nov = _log(rng, 1000, 700000)
        return dict(kind=kind, graph=rng.choice(["mix", "uniform", "zipf"]), nov=nov, noe=max(1, int(nov * ratio)))
    K = rng.choice([2, 5, 8, 16, 24, 32, 64, 100, 128, 256, 512])
    if kind == "metrics":
        nov = _log(rng, 1000, 700000)
        return dict(kind=kind, graph=rng.choice(["mix", "uniform", "zipf"]), nov=nov, noe=max(1, int(nov * ratio)),
                    unit=1, K=K)
    if kind == "stream":
        nov = _log(rng, 1000, 170000)
        return dict(kind=kind, graph="zipf", nov=nov, noe=max(1, int(nov * ratio)), unit=0, K=max(K, 16),
                    metric=rng.choice(["TV", "MSV", "MSRV"]))
    metric = rng.choice(["CN", "TV", "TM", "MSM", "MSV", "MSRV"])
    graph = rng.choice(["mix", "uniform", "zipf", "zipf_unit"])
    unit = int(graph != "zipf")
    passes = rng.choice([1, 2, 3])
    if unit and metric in ("TV", "MSV"):
        # most decisions break ties on part sizes: the costliest refinements
        nov = _log(rng, 1000, 6000 if graph == "zipf_unit" else 12000)
        passes = 1 if graph == "zipf_unit" else passes
    elif metric in ("MSV", "MSRV", "TM", "CN"):
        nov = _log(rng, 1000, 150000)
    else:
        nov = _log(rng, 1000, 500000)
    return dict(kind="refine", graph="zipf" if graph == "zipf_unit" else graph, nov=nov,
                noe=max(1, int(nov * ratio)), unit=unit, K=K, metric=metric, passes=passes,
                eps=rng.choice([1.03, 1.05, 1.1]))


def _shape(case):
    """(alpha, lo, hi, beta) of the case's net sizes and vertex popularity."""
    if case["graph"] == "uniform":
        return 0.0, 2, 16, 0.0
    if case["graph"] == "mix":
        return 2.2, 2, min(2000, case["nov"]), 0.0
    return 2.1, 2, min(10000, case["nov"]), 1.5


def _hypergraph(case, seed):
    alpha, lo, hi, beta = _shape(case)
    if alpha == 0.0:
        spec = fp.GenSpec.column_net(case["nov"], case["noe"], lo, hi, seed=seed)
    else:
        spec = fp.GenSpec.zipf(case["nov"], case["noe"], alpha, lo, hi, beta=beta,
                               weight_rule=0 if case.get("unit", 1) else 1, seed=seed)
    hg = fp.generate(spec)
    if case["kind"] == "inverse":
        # a file of a fixed number of pins (the arrays' sizes belong to the case,
        # not to the seed): the nets beyond it are empty
        nptr = np.minimum(hg.nptr, _file_pins(case))
        hg = fp.Hypergraph.from_nets(hg.nov, nptr, hg.npins[:nptr[-1]])
    return hg


def _file_pins(case):
    return int(0.7 * case["noe"] * _mean_size(case))


def _given_partition(hg, K, seed):
    """A partition as another tool would hand it over: a part per vertex drawn
    at random, and the per-net lists of parts with their pin counts."""
    part = np.random.default_rng(seed).integers(0, K, hg.nov).astype(np.int32)
    net = np.repeat(np.arange(hg.noe, dtype=np.int64), np.diff(hg.nptr.astype(np.int64)))
    keys, counts = np.unique(net * K + part[hg.npins], return_counts=True)
    lens = np.bincount(keys // K, minlength=hg.noe)
    starts = hg.nptr[:-1].astype(np.int64)
    at = np.repeat(starts - np.concatenate([[0], np.cumsum(lens)[:-1]]), lens) + np.arange(keys.size)
    parts = np.full(hg.pins, -1, np.int32)
    cnt = np.zeros(hg.pins, np.int32)
    parts[at] = keys % K
    cnt[at] = counts
    return part, dict(part_vec=part, ep_starts=starts, ep_ends=lens, ep_parts=parts, ep_cnt=cnt)


def prepare(case, seed):
    hg = _hypergraph(case, seed)
    engine = fp.Engine(0)
    state = dict(kind=case["kind"], engine=engine, hg=hg, passes=case.get("passes", 0))
    if case["kind"] == "inverse":
        return state
    inst = engine.instance(hg, case["K"], case.get("metric", "CN"), case.get("eps", 1.05))
    state["inst"] = inst
    if case["kind"] == "refine":
        inst.initial_partition()
    elif case["kind"] == "metrics":
        inst.set_state(**_given_partition(hg, case["K"], seed)[1])
    return state


def _metrics(inst):
    m = inst.metrics()
    return np.array([m[k] for k in ORDER], np.int64)


def run(state):
    if state["kind"] == "inverse":
        hg = state["hg"]
        row_ptr, col_ind = state["engine"].create_inverse(hg.nov, hg.noe, hg.vptr, hg.vnets)
        return {"row_ptr_inv": row_ptr.view(np.int32), "col_ind_inv": col_ind.view(np.int32)}
    inst = state["inst"]
    if state["kind"] == "metrics":
        return {"metrics": _metrics(inst)}
    if state["kind"] == "stream":
        inst.initial_partition()
    else:
        inst.reset_state()
        inst.refine(state["passes"])
    return {"metrics": _metrics(inst), "part_sizes": inst.part_sizes(), "part_vec": inst.partition()}


def _mean_size(case):
    alpha, lo, hi, _ = _shape(case)
    if alpha == 0.0:
        return 0.5 * (lo + hi)
    s = np.arange(1, (1 << 20) + 1, dtype=np.float64)
    mass = s ** -alpha
    tail = float((1 << 20) ** (1.0 - alpha)) / (alpha - 1.0)
    mean = float((mass * np.clip(s, lo, hi)).sum()) + tail * hi
    return mean / (float(mass.sum()) + tail)


def work(case):
    """Bytes: every array the call has to read or write, once.  Flops: one
    integer operation per (vertex, net) pair and pass."""
    nov, noe = case["nov"], case["noe"]
    pins = int(noe * _mean_size(case))
    if case["kind"] == "inverse":
        pins = _file_pins(case)
        return {"bytes": 4 * (nov + 1) + 4 * pins + 4 * (noe + 1) + 4 * pins, "flops": pins}
    lists = 4 * noe + 8 * pins
    if case["kind"] == "metrics":
        return {"bytes": 4 * (noe + 1) + 4 * noe + 4 * nov + lists, "flops": pins}
    csr = 4 * (nov + 1) + 4 * pins + 4 * (noe + 1) + 4 * noe + 4 * nov
    if case["kind"] == "stream":
        return {"bytes": csr + lists + 4 * nov, "flops": pins}
    # the state goes up once, is read, and the part vector is written and read back
    return {"bytes": csr + 2 * (lists + 4 * nov) + 8 * nov, "flops": pins * case["passes"]}


def exact(case, seed):
    """The metrics of a given partition and the transpose, in 64-bit numpy; a
    refinement or stream has no closed form."""
    if case["kind"] == "inverse":
        hg = _hypergraph(case, seed)
        owner = np.repeat(np.arange(hg.nov, dtype=np.uint32), np.diff(hg.vptr.astype(np.int64)))
        order = np.argsort(hg.vnets, kind="stable")
        nptr = np.concatenate([[0], np.cumsum(np.bincount(hg.vnets, minlength=hg.noe))])
        return {"row_ptr_inv": nptr.astype(np.int32), "col_ind_inv": owner[order].astype(np.int32)}
    if case["kind"] != "metrics":
        return None
    hg, K = _hypergraph(case, seed), case["K"]
    part, _ = _given_partition(hg, K, seed)
    net = np.repeat(np.arange(hg.noe, dtype=np.int64), np.diff(hg.nptr.astype(np.int64)))
    keys = np.unique(net * K + part[hg.npins])
    e, p = keys // K, keys % K
    lam = np.bincount(e, minlength=hg.noe)
    src = part[hg.src].astype(np.int64)[e]
    sent = p != src                                    # one volume unit per net and receiving part
    send = np.bincount(src[sent], minlength=K)
    recv = np.bincount(p[sent], minlength=K)
    pairs = np.unique(src[sent] * K + p[sent])         # one message per pair of parts
    msgs = np.bincount(pairs // K, minlength=K)
    value = {"TV": (lam - 1).sum(), "CN": (lam > 1).sum(), "TM": pairs.size, "MSM": msgs.max(), "MSV": send.max(),
             "MSRV": (send + recv).max()}
    return {"metrics": np.array([value[k] for k in ORDER], np.int64)}
