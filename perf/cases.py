"""The work that programs have this library do, as cases that can be timed.

A case is a dict of plain values; prepare() makes what a program holds before
the call (the graph in device memory, the handle, the roots), run() makes one
pass through the public entry points and returns its results.  Parents of the
parallel traversal depend on which neighbour wins a race, so they are returned
only where the caller asked for the deterministic tree (min_parent); depths,
edge and vertex counts and component labels are always the same.

kinds
  root        one BFS the way the reference's main loop runs a trial: clear,
              run_beamer, count, results to host arrays
  trial       the same with the validation of the tree (--check_results)
  roots       k BFSs back to back, every root's depths and parents left in
              the caller's device arrays (run_many_into)
  packed      many small graphs in one CSR, one root in each, one launch
  batch       up to 64 roots per pass over the graph, every root's depths and
              parents written by the run
  components  connected components, labels left in device memory (host=True:
              labels and sizes copied to host arrays)
"""
import ctypes
import random

import numpy as np
import torch

import beedrill_b200 as bd
from beedrill_b200 import policy

ORDERS = {"insertion": bd.ORDER_INSERTION, "sorted": bd.ORDER_SORTED, "degree": bd.ORDER_DEGREE,
          "hub": bd.ORDER_HUB}


def _case(kind, graph, *, scale=0, edge_factor=16, rows=0, cols=0, parts=0, order="hub", roots=1,
          alg="beamer_hybrid", min_parent=False, learned=False, host=False, name=None):
    case = {"kind": kind, "graph": graph, "scale": scale, "edge_factor": edge_factor, "rows": rows,
            "cols": cols, "parts": parts, "order": order, "roots": roots, "alg": alg,
            "min_parent": min_parent, "learned": learned, "host": host}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one query on a small graph: nothing but call latency, launches and levels
        _case("root", "rmat", scale=10, order="insertion", host=True, name="root-s10"),
        # the usual validation run: 8 trials at scale 16 in file order, deterministic trees
        _case("roots", "rmat", scale=16, order="insertion", roots=8, min_parent=True,
              name="roots-s16-x8-min-parent"),
        # the reference's top-down algorithms (remote_writes, migrating_threads)
        _case("roots", "rmat", scale=19, edge_factor=13, order="degree", roots=5, alg="top_down",
              name="roots-s19-x5-top-down"),
        # the Graph500 loop, one root per launch, on a graph larger than L2
        _case("roots", "rmat", scale=22, roots=64, name="roots-s22-x64"),
        # high diameter: thousands of levels of a few hundred vertices (road-like graphs)
        _case("roots", "grid", rows=1021, cols=1031, order="insertion", roots=1,
              name="root-grid-1021x1031"),
        # one trial with its check, as the command line runs it
        _case("trial", "rmat", scale=20, order="hub", name="trial-s20-check"),
        # many small graphs of mixed size at once
        _case("packed", "packed", parts=128, order="insertion", name="packed-128"),
        # a small batch on a small graph: latency again
        _case("batch", "rmat", scale=12, edge_factor=9, roots=16, order="degree", name="batch-s12-x16"),
        # four full groups replayed as one graph
        _case("batch", "rmat", scale=20, roots=256, name="batch-s20-x256"),
        # the headline: 64 roots at scale 24 under the learned push/pull policy
        _case("batch", "rmat", scale=24, roots=64, learned=True, name="batch-s24-x64-learned"),
        # a batch whose wavefronts never line up
        _case("batch", "grid", rows=509, cols=523, order="insertion", roots=64, learned=True,
              name="batch-grid-509x523-x64"),
        # components of a graph of some millions of vertices
        _case("components", "rmat", scale=22, order="insertion", name="components-s22"),
    ]


def draw(rng: random.Random):
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["root", "roots", "roots", "trial", "packed", "batch", "batch", "components"])
    order = rng.choice(["insertion", "sorted", "degree", "hub", "hub"])
    learned = rng.random() < 0.5
    edge_factor = rng.randint(4, 33)
    if kind == "packed":
        return _case("packed", "packed", parts=log_int(5, 160), order="insertion")
    if kind == "root":
        return _case("root", "rmat", scale=rng.randint(8, 16), edge_factor=edge_factor, order=order,
                     host=True)
    if kind == "trial":
        return _case("trial", "rmat", scale=rng.randint(10, 20), edge_factor=edge_factor,
                     order=order)
    if rng.random() < 0.3:
        shape = {"graph": "grid", "rows": log_int(37, 700), "cols": log_int(37, 700),
                 "order": rng.choice(["insertion", "hub"])}
    else:
        shape = {"graph": "rmat", "scale": rng.randint(10, 20), "edge_factor": edge_factor,
                 "order": order}
    graph = shape.pop("graph")
    if kind == "components":
        return _case("components", graph, host=shape.get("scale", 99) <= 14, **shape)
    if kind == "roots":
        if graph == "rmat":
            shape["alg"] = rng.choice(["beamer_hybrid", "beamer_hybrid", "beamer_hybrid",
                                       "top_down"])
        return _case("roots", graph, roots=log_int(1, 4 if graph == "grid" else 48),
                     min_parent=rng.random() < 0.4, **shape)
    return _case("batch", graph, roots=log_int(3, 130), learned=learned,
                 min_parent=rng.random() < 0.2, **shape)


def _graph(case, seed):
    order = ORDERS[case["order"]]
    if case["graph"] == "rmat":
        return bd.Graph.rmat(case["scale"], case["edge_factor"], seed=seed, order=order)
    if case["graph"] == "grid":
        return bd.Graph.grid(case["rows"], case["cols"], 0.01, seed, order=order)
    raise ValueError(case["graph"])


def _parts(case):
    """(scale, edge factor) of each graph of a packed case."""
    rng = np.random.default_rng(case["parts"])
    return list(zip(rng.integers(10, 17, case["parts"]).tolist(),
                    rng.integers(4, 33, case["parts"]).tolist()))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "packed":
        graphs = [bd.Graph.rmat(sc, ef, seed=seed * 1009 + i, order=ORDERS[case["order"]])
                  for i, (sc, ef) in enumerate(_parts(case))]
        g, base = bd.Graph.concat(graphs)
        s["roots"] = np.array([int(p.pick_roots(seed + i, 1)[0]) + int(base[i])
                               for i, p in enumerate(graphs)], np.int64)
        for p in graphs:
            p.close()
    else:
        g = _graph(case, seed)
        s["roots"] = g.pick_roots(seed, case["roots"])
    s["graph"], s["n"] = g, g.num_vertices()
    if kind == "components":
        s["handle"] = bd.Components(g)
    elif kind == "batch":
        s["handle"] = bd.BatchedBFS(g, case["roots"], materialize=True,
                                    min_parent=case["min_parent"])
        if case["learned"]:
            policy.Policy.load(policy.BATCHED_PATH).install(s["handle"])
    else:
        s["handle"] = bd.HybridBFS(g, alg=case["alg"], min_parent=case["min_parent"])
    if kind == "roots":
        s["depth"] = torch.empty((case["roots"], s["n"]), dtype=torch.int32, device="cuda")
        s["parent"] = torch.empty((case["roots"], s["n"]), dtype=torch.int64, device="cuda")
    return s


class _DeviceArray:
    """An array in a handle's device memory, for torch.as_tensor; the tensor
    keeps this object, and with it the handle that owns the memory."""

    def __init__(self, handle, address, shape, typestr):
        self.handle = handle
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr,
                                         "data": (address, False), "version": 3}


def _view(handle, address, shape, typestr):
    return torch.as_tensor(_DeviceArray(handle, address, shape, typestr), device="cuda")


def _single_depths(handle, n):
    d, p = ctypes.c_void_p(), ctypes.c_void_p()
    status = bd.lib().bd_bfs_device_ptrs(handle._h, ctypes.byref(d), ctypes.byref(p))
    if status != bd.BD_OK:
        raise bd.BeedrillError(status, "device_ptrs")
    return _view(handle, d.value, (n,), "<i4")


def _batch_rows(handle, count, n, with_parents):
    """The rows of all roots as one [count, n] array (they lie one after another)."""
    d0, p0 = handle.device_results(0)
    d1, p1 = handle.device_results(count - 1)
    if d1 - d0 != 4 * n * (count - 1) or p1 - p0 != 8 * n * (count - 1):
        raise RuntimeError("result rows are not consecutive")
    depth = _view(handle, d0, (count, n), "<i4")
    return [depth, _view(handle, p0, (count, n), "<i8")] if with_parents else [depth]


def run(s):
    case, h, roots, n = s["case"], s["handle"], s["roots"], s["n"]
    kind = case["kind"]
    if kind == "root":
        h.clear()
        h.run_beamer(int(roots[0]), 15, 18)
        edges = h.count_num_traversed_edges()
        h.parents()  # what the program is after; which parent wins is a race
        return [h.depths(), edges]
    if kind == "trial":
        h.clear()
        h.run_beamer(int(roots[0]), 15, 18)
        ok = h.check(int(roots[0]))
        return [_single_depths(h, n), ok, h.count_num_traversed_edges()]
    if kind == "roots":
        _, edges, reached, _ = h.run_many_into(roots, s["depth"].data_ptr(), s["parent"].data_ptr())
        out = [s["depth"], edges, reached]
        return out + [s["parent"]] if case["min_parent"] else out
    if kind == "packed":
        st = h.run_multi(roots)
        return [_single_depths(h, n), st.traversed_edges, st.reached]
    if kind == "batch":
        h.run(roots)
        edges, reached = h.counts()
        return _batch_rows(h, len(roots), n, case["min_parent"]) + [edges, reached]
    if kind == "components":
        st = h.run()
        if case["host"]:
            return [h.labels(), h.sizes(), st.num_components]
        p = ctypes.c_void_p()
        status = bd.lib().bd_components_device_labels(h._h, ctypes.byref(p))
        if status != bd.BD_OK:
            raise bd.BeedrillError(status, "device_labels")
        return [_view(h, p.value, (n,), "<i8"), st.num_components]
    raise ValueError(kind)


def _size(case):
    """(vertices, undirected edges); RMAT edges counted before the duplicates go."""
    if case["graph"] == "rmat":
        return 1 << case["scale"], case["edge_factor"] << case["scale"]
    if case["graph"] == "grid":
        r, c = case["rows"], case["cols"]
        return r * c, int(0.99 * (r * (c - 1) + (r - 1) * c))
    return (sum(1 << s for s, _ in _parts(case)), sum(f << s for s, f in _parts(case)))


def work(case):
    """The graph read once (int64 offsets, two uint32 arcs per edge) and every
    result written once: per root an int32 depth and an int64 parent of every
    vertex, or an int64 label.  Integer work only."""
    n, m = _size(case)
    graph = 8 * (n + 1) + 8 * m
    if case["kind"] == "components":
        return {"bytes": graph + 16 * n, "flops": 0}
    return {"bytes": graph + 12 * n * (1 if case["kind"] == "packed" else case["roots"]),
            "flops": 0}


def _plain_depths(src, dst, n, root):
    depth = torch.full((n,), -1, dtype=torch.int64, device=src.device)
    depth[root] = 0
    level = 0
    while True:
        hit = dst[(depth[src] == level) & (depth[dst] < 0)]
        if hit.numel() == 0:
            return depth
        level += 1
        depth[hit] = level


def exact(case, seed):
    """Depths by a plain level-synchronous search over the edge list, for the
    cases where that is quick; the other outputs are counts and trees."""
    kind = case["kind"]
    if kind in ("components", "packed") or case["graph"] != "rmat" or case["roots"] > 16:
        return None
    g = _graph(case, seed)
    roots = g.pick_roots(seed, case["roots"])
    n = g.num_vertices()
    src, dst = (torch.from_numpy(a).cuda() for a in g.edges())
    src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    depth = torch.stack([_plain_depths(src, dst, n, int(r)) for r in roots])
    g.close()
    if kind in ("root", "trial"):
        return [depth[0]] + [None] * (2 if kind == "trial" else 1)
    return [depth] + [None] * (3 if case["min_parent"] else 2)
