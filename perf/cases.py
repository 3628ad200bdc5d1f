"""What the framework is timed on: label propagation over CGR-compressed graphs
through the package's public entry points, and the calls on either side of it
(compressing a graph, decoding one, going from a compressed graph to labels in
one go).

A case is a dict of plain values:
  call      "run"      init_labels + run(iters) + labels of a kept Propagator
            "step"     set_labels + iterate + labels, one iteration end to end
            "oneshot"  LabelPropagator(graph).run(iters) + get_labels: create included
            "encode"   HostGraph.compress on the GPU, the compressed arrays copied out
            "decode"   lpa_decode_csr into the caller's arrays
            "batch"    Batch.run + every graph's labels
  graph     "road" (width x height grid), "rmat" (n vertices, edge factor 16),
            "copy" (n vertices, out-degree 30), or for a batch "mixed": graphs
            of lo..hi vertices, road grids and R-MAT (edge factor 8) in turn
  thresh    degrees below it stay in the plain CSR (0: everything compressed)
  cms       degrees from it on are counted by the sketch (0: exact)
  plan      "fixed" (the default dispatch), "learned", "twopass"
  budget    device bytes for the bitstream and scratch out of core (0: resident)
Every graph, and the labels of a "step", come from the seed.
"""
import ctypes as C
import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np

import lpa_b200 as L

# iterations of a kept handle that settle the learned plan (fixed, explorations, trials)
LEARN_ITERS = 10


def listed():
    return [
        # the smallest calls: a road grid of 131k vertices, tens of us of
        # device work per iteration, where launches and latency count
        dict(name="road-362", call="run", graph="road", width=362, height=362, thresh=0, cms=0, plan="fixed", iters=20,
             early=False, budget=0),
        # road network of 2M vertices, stopping when nothing changes
        dict(name="road-1404", call="run", graph="road", width=1404, height=1404, thresh=0, cms=0, plan="fixed",
             iters=30, early=True, budget=0),
        # a social graph with the default dispatch and the sketch for hubs
        dict(name="rmat-18-fixed", call="run", graph="rmat", n=1 << 18, thresh=32, cms=1024, plan="fixed", iters=20,
             early=False, budget=0),
        # the large social graph, learned dispatch (what the benchmark runs)
        dict(name="rmat-22-learned", call="run", graph="rmat", n=1 << 22, thresh=32, cms=1024, plan="learned", iters=20,
             early=False, budget=0),
        # a web-like graph (runs of equal labels, many intervals), odd vertex count
        dict(name="copy-4m-learned", call="run", graph="copy", n=3999999, thresh=16, cms=4096, plan="learned", iters=10,
             early=False, budget=0),
        # one iteration end to end, labels in from and out to the host: a
        # caller that keeps the labels itself; two-pass kernels
        dict(name="rmat-20-step", call="step", graph="rmat", n=1 << 20, thresh=32, cms=1024, plan="twopass", iters=1,
             early=False, budget=0),
        # no sketch and no plain CSR: exact counts of every hub, ragged size,
        # the driver program's flow from a compressed graph to labels
        dict(name="rmat-17-oneshot", call="oneshot", graph="rmat", n=150001, thresh=16, cms=0, plan="fixed", iters=20,
             early=False, budget=0),
        # a bitstream larger than the device budget, copied range by range
        dict(name="rmat-20-stream", call="run", graph="rmat", n=1000003, thresh=32, cms=1024, plan="fixed", iters=5,
             early=False, budget=64 << 20),
        # compressing a graph (the encode direction)
        dict(name="rmat-20-encode", call="encode", graph="rmat", n=1 << 20, thresh=32, cms=0, plan="fixed", iters=1,
             early=False, budget=0),
        # decoding one (the decode direction)
        dict(name="copy-1m-decode", call="decode", graph="copy", n=1000001, thresh=16, cms=0, plan="fixed", iters=1,
             early=False, budget=0),
        # many uneven graphs together, each with its own convergence test:
        # joined into one graph, and run from the device queue
        dict(name="batch-lockstep", call="batch", graph="mixed", graphs=48, lo=1000, hi=65536, thresh=16, cms=0,
             plan="learned", iters=30, early=True, budget=0),
        dict(name="batch-queue", call="batch", graph="mixed", graphs=32, lo=1000, hi=32768, thresh=16, cms=0,
             plan="queue", iters=30, early=True, budget=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes log-uniform up to the listed ones, odd ones among them."""
    call = rng.choice(["run"] * 6 + ["step", "step", "oneshot", "oneshot", "encode", "decode", "batch", "batch"])
    c = dict(call=call, cms=0, plan="fixed", iters=1, early=False, budget=0)
    if call == "batch":
        c.update(graph="mixed", graphs=rng.randint(3, 40), lo=1000, hi=_log(rng, 2000, 32768), iters=rng.randint(5, 30),
                 early=True, plan=rng.choice(["learned", "fixed", "queue"]), thresh=rng.choice([0, 8, 16, 32]),
                 cms=rng.choice([0, 0, 256]))
        return c
    kind = rng.choice(["road", "rmat", "rmat", "copy"])
    if kind == "road":
        c.update(graph="road", width=_log(rng, 24, 1400), height=_log(rng, 24, 1400), thresh=rng.choice([0, 0, 0, 4]))
    elif kind == "rmat":
        c.update(graph="rmat", n=_log(rng, 1000, 1 << (21 if call in ("run", "step") else 19)),
                 thresh=rng.choice([0, 8, 16, 32, 64]))
    else:
        c.update(graph="copy", n=_log(rng, 2000, 2000000 if call in ("run", "step") else 500000),
                 thresh=rng.choice([0, 16, 16, 64]))
    if kind != "road" and call in ("run", "step", "oneshot"):
        c["cms"] = rng.choice([0, 128, 1024, 4096])
    if call in ("run", "oneshot"):
        c["iters"] = rng.randint(4, 20)
        c["early"] = call == "run" and rng.random() < 0.4
    if call in ("run", "step"):
        c["plan"] = rng.choice(["fixed", "learned", "twopass"])
        if kind == "rmat" and c["n"] > 200000 and rng.random() < 0.15:
            c["budget"] = 64 << 20
    return c


def _graph(case, seed):
    if case["graph"] == "road":
        return L.HostGraph.road(case["width"], case["height"], seed=seed)
    if case["graph"] == "copy":
        return L.HostGraph.copy_model(case["n"], 30, seed=seed)
    return L.HostGraph.rmat(max(8, math.ceil(math.log2(case["n"]))), 16.0, seed=seed, n_limit=case["n"])


def _batch(case, seed):
    rng = np.random.default_rng(case["graphs"] + case["hi"])  # the sizes are the case's, the graphs the seed's
    sizes = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["graphs"])).astype(int)

    def make(i):
        n = int(sizes[i])
        if i % 2 == 0:
            side = max(4, int(round(math.sqrt(n))))
            g = L.HostGraph.road(side, side, seed=seed + i)
        else:
            g = L.HostGraph.rmat(max(8, math.ceil(math.log2(n))), 8.0, seed=seed + i, n_limit=n)
        return g.compress(case["thresh"], 128, threads=1)

    with ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        return list(ex.map(make, range(case["graphs"])))


def _opts(case):
    o = dict(device=0, cms_threshold=case["cms"], stream_budget=case["budget"])
    if case["plan"] == "learned":
        o["dispatch"] = L.Dispatch.LEARNED
    elif case["plan"] == "twopass":
        o.update(dispatch=L.Dispatch.FORCE, force_variant=int(L.Variant.TWO_PASS))
    elif case["plan"] == "queue":
        o["batch_mode"] = L.BatchMode.QUEUE
    return o


def _buffers(case):
    """Arrays of the caller's, large enough for any graph of the case (zeros past its end)."""
    n, arcs = _limits(case)
    if case["call"] == "decode":
        return {"row": np.zeros(n + 1, np.uint64), "clm": np.zeros(arcs, np.uint32)}
    return {"words": np.zeros(arcs * 3 // 4 + n, np.uint32), "offsets": np.zeros(n + 1, np.uint64),
            "vertices": np.zeros(n, np.uint32), "small_graph": np.zeros(min(arcs, n * case["thresh"]), np.uint32),
            "small_offset": np.zeros(n + 1, np.uint32)}


def prepare(case, seed):
    st = {"case": case}
    if case["call"] == "batch":
        st["b"] = L.Batch(_batch(case, seed), **_opts(case))
        if case["plan"] == "learned":
            st["b"].run(LEARN_ITERS, early_exit=False)
        return st
    g = _graph(case, seed)
    if case["call"] == "encode":
        st.update(g=g, out=_buffers(case))  # the uncompressed graph
        return st
    g.compress(case["thresh"], 128)
    st["g"] = g
    if case["call"] == "oneshot":
        return st
    if case["call"] == "decode":
        st["out"] = _buffers(case)
    p = st["p"] = L.Propagator(g, **_opts(case))
    if case["plan"] == "learned":
        p.run(LEARN_ITERS)
        p.init_labels()
    if case["call"] == "step":  # labels part-way through a propagation: few of them, shared by neighbours
        p.run(int(np.random.default_rng(seed).integers(1, 4)))
        st["labels"] = p.labels()
    return st


def _copy_out(dst, src, count):
    if count:
        dst[:count] = np.ctypeslib.as_array(src, shape=(int(count),))


def run(st):
    case = st["case"]
    if case["call"] == "run":
        p = st["p"]
        p.init_labels()
        n = p.run(case["iters"], early_exit=case["early"])
        changed = np.zeros(case["iters"], np.uint64)
        changed[:n] = p.changed_history(n)
        return {"labels": p.labels(), "iters": n, "changed": changed}
    if case["call"] == "step":
        p = st["p"]
        p.set_labels(st["labels"])
        changed = p.iterate()
        return {"labels": p.labels(), "changed": changed}
    if case["call"] == "oneshot":
        p = L.LabelPropagator(st["g"], **_opts(case))
        p.run(case["iters"])
        return {"labels": p.get_labels()}
    if case["call"] == "encode":
        d, out = st["g"].compress(case["thresh"], 128, device=0).desc(), st["out"]
        n, n_c = d.num_vertices, d.num_compressed
        _copy_out(out["words"], d.words, d.num_words)
        _copy_out(out["offsets"], d.offsets, n_c + 1)
        _copy_out(out["vertices"], d.vertices, n)
        _copy_out(out["small_graph"], d.small_graph, d.num_small_arcs)
        _copy_out(out["small_offset"], d.small_offset, n - n_c + 1 if n > n_c else 0)
        return out
    if case["call"] == "decode":
        out = st["out"]
        status = L.lib().lpa_decode_csr(st["p"]._h, out["row"].ctypes.data_as(C.POINTER(C.c_uint64)),
                                        out["clm"].ctypes.data_as(C.POINTER(C.c_uint32)))
        if status:
            raise L.LpaError(status, "lpa_decode_csr")
        return out
    b = st["b"]
    iters = b.run(case["iters"], early_exit=case["early"])
    return {"iters": iters, "labels": np.concatenate([b.labels(i) for i in range(len(b.n))])}


def _limits(case):
    """(vertices, most arcs) of a case's graph."""
    if case["graph"] == "road":
        n = case["width"] * case["height"]
        return n, 6 * n
    n = case["n"]
    if case["graph"] == "copy":
        return n, 30 * n
    return n, 2 * 16 * (1 << max(8, math.ceil(math.log2(n))))


def _sizes(case):
    """(vertices, arcs, compressed bytes): generator averages, so that no graph has to be built."""
    if case["graph"] == "road":
        n = case["width"] * case["height"]
        return n, 2.83 * n, 1.95 * 2.83 * n
    if case["graph"] == "copy":
        return case["n"], 26.4 * case["n"], 1.7 * 26.4 * case["n"]
    if case["graph"] == "mixed":
        lo, hi = case["lo"], case["hi"]
        n = case["graphs"] * (hi - lo) / math.log(hi / lo)
        return n, 8.5 * n, 1.5 * 8.5 * n
    n = case["n"]
    arcs = n * min(31.0, 20.0 + 0.6 * math.log2(n))
    return n, arcs, 1.45 * arcs


def work(case):
    n, arcs, stream = _sizes(case)
    once = stream + 12 * n  # the compressed graph, its degrees, labels in and out
    if case["call"] == "encode":
        b = 4 * arcs + 8 * n + stream + 4 * n
    elif case["call"] == "decode":
        b = stream + 4 * arcs + 8 * n
    else:
        b = case["iters"] * once
    return {"bytes": float(b), "flops": 0.0}


def exact(case, seed):
    """Every output is a whole number, fixed by the update rule or the format: no 64-bit value to stand beside it."""
    return None
