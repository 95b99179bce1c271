"""The calls whose time matters to a user of this framework.

Each case is one call, or the few calls that belong together, as a program
makes them: a whole solve from host arrays, a solve on a graph that stays on
the device, a new frame of capacities, the reference's two-call drop-in, a
batch, a matching, a solve in the caller's own device buffers.  The graphs
are the benchmark's families (GENRMF, layered, R-MAT, graph-cut grids,
bipartite matching) in the sizes that the tests and the benchmark use.

Every output is unique for its input: the maximum-flow value, and the two
extreme minimum cuts (vertex sides and per-arc indicators).  A maximum
preflow itself (excess, labels, arc flows) is not, and is not returned.
"""
from __future__ import annotations

import ctypes as C
from collections import deque

import numpy as np
import torch

import wbpr_gb300 as W
from wbpr_gb300 import workloads


def listed():
    return [
        # the smallest whole call: host arrays in, value out, nothing kept
        dict(name="call_tiny", op="call", family="genrmf", a=4, b=5, layout="bcsr", algo="vc"),
        # the reference's preflow() / push_relabel() pair on its RCSR host arrays, default algorithm
        dict(name="dropin_layered", op="dropin", family="layered", a=11, b=37, layout="rcsr", algo="tc"),
        # the benchmark's small GENRMF, thread-centric on the reference's default layout
        dict(name="solve_genrmf_tc", op="solve", family="genrmf", a=8, b=16, layout="rcsr", algo="tc"),
        # a hard mid-size GENRMF: many rounds over few vertices
        dict(name="solve_genrmf_vc", op="solve", family="genrmf", a=16, b=40, layout="bcsr", algo="vc"),
        # new capacities on a kept topology, then the value and the source side of the cut
        dict(name="recap_layered", op="recap", family="layered", a=32, b=256, layout="bcsr", algo="vc"),
        # one frame of a graph-cut layer: forward, and both extreme subgradients
        dict(name="grid_fwd_bwd", op="adjoint", family="grid", a=512, b=512, layout="bcsr", algo="vc"),
        # a solve in the caller's own device buffers, without allocation
        dict(name="noalloc_rmat", op="noalloc", family="rmat", a=13, b=16, layout="bcsr", algo="vc"),
        # a power-law graph of ordinary size on the reference's default layout, with the sink side of the cut
        dict(name="cut_rmat_rcsr", op="cut", family="rmat", a=17, b=11, layout="rcsr", algo="vc"),
        # many uneven instances in one launch
        dict(name="batch_uneven", op="batch", family="mixed", a=512, b=0, layout="bcsr", algo="vc"),
        # unit-capacity bipartite matching at the benchmark's size
        dict(name="matching_2m", op="solve", family="bipartite", a=2000000, b=2000000, layout="bcsr", algo="vc"),
        # the headline workload on a kept graph, and the whole call from page-locked host arrays
        dict(name="solve_rmat22", op="solve", family="rmat", a=22, b=16, layout="bcsr", algo="vc"),
        dict(name="call_rmat22", op="call", family="rmat", a=22, b=16, layout="bcsr", algo="vc"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(lo * (hi / lo) ** rng.random() + 0.5))


def _sizes(rng, family, small=False):
    if family == "genrmf":
        return _log_int(rng, 4, 8 if small else 18), _log_int(rng, 4, 16 if small else 48)
    if family == "layered":
        return _log_int(rng, 4, 16 if small else 40), _log_int(rng, 12, 64 if small else 320)
    if family == "grid":
        return _log_int(rng, 17, 90 if small else 500), _log_int(rng, 17, 90 if small else 500)
    if family == "bipartite":
        return _log_int(rng, 900, 9000 if small else 2000000), _log_int(rng, 900, 9000 if small else 2000000)
    return _log_int(rng, 9, 13 if small else 20), _log_int(rng, 5, 16)


def draw(rng):
    op = rng.choice(["call", "call", "solve", "solve", "solve", "recap", "adjoint", "noalloc", "dropin", "cut", "batch"])
    layout, algo = rng.choice(["bcsr", "bcsr", "rcsr"]), rng.choice(["vc", "vc", "tc"])
    small = op in ("noalloc", "dropin")
    if op == "batch":
        return dict(op=op, family="mixed", a=_log_int(rng, 21, 500), b=0, layout="bcsr", algo="vc")
    if op == "adjoint":
        family = "grid"
    elif op == "recap":
        family = rng.choice(["layered", "genrmf", "grid", "rmat"])
    else:
        family = rng.choice(["genrmf", "layered", "grid", "bipartite", "rmat", "rmat"])
    if op == "noalloc":
        layout = "bcsr"
    if op == "dropin":
        layout = "rcsr"
    a, b = _sizes(rng, family, small)
    return dict(op=op, family=family, a=a, b=b, layout=layout, algo=algo)


def _graph(case, seed):
    a, b, f = case["a"], case["b"], case["family"]
    if f == "genrmf":
        return W.gen_genrmf(a, b, 1, 10000, seed)
    if f == "layered":
        return W.gen_layered(a, b, 3, 6, 1, 1000, seed)
    if f == "grid":
        return W.gen_grid(a, b, seed)
    if f == "bipartite":
        return W.gen_bipartite(a, b, 2.0, 4096, seed)
    return W.gen_rmat(a, b, seed=seed)


def _page_locked(x):
    return torch.from_numpy(np.ascontiguousarray(x, np.int32)).pin_memory()


def prepare(case, seed):
    op = case["op"]
    s = {"op": op, "algo": case["algo"], "layout": case["layout"]}
    if op == "batch":
        # a batch solver is kept as a serving program keeps it
        s["batch"] = W.Batch(workloads.config3(case["a"], seed))
        return s
    g = _graph(case, seed)
    if op == "call":
        s["pinned"] = [_page_locked(x) for x in (g.off, g.dst, g.cap)]
        s["graph"] = W.Graph(g.n, *(t.numpy() for t in s["pinned"]), g.s, g.t)
    elif op == "dropin":
        s["graph"] = g
        s["reverse"] = W.build_rcsr(g)
    elif op == "noalloc":
        off, dst, cap, back = W.build_bcsr(g)
        s["n"], s["arcs"], s["s"], s["t"] = g.n, 2 * g.m, g.s, g.t
        s["row"] = torch.from_numpy(off).cuda()
        s["arc"] = torch.from_numpy(np.stack([dst, cap], 1)).cuda()
        s["arx"] = torch.from_numpy(np.stack([back, cap], 1)).cuda()
    else:
        s["cap"] = g.cap
        s["device"] = W.DeviceGraph(g, case["layout"])
    return s


def run(s):
    op, algo = s["op"], s["algo"]
    if op == "call":
        return {"flow": W.maxflow(s["graph"], algo, s["layout"])}
    if op == "solve":
        return {"flow": int(s["device"].solve(algo).flow)}
    if op == "cut":
        flow = int(s["device"].solve(algo).flow)
        return {"flow": flow, "sink_side": s["device"].cut_sides(0)}
    if op == "recap":
        s["device"].set_capacities(s["cap"])
        flow = int(s["device"].solve(algo).flow)
        return {"flow": flow, "source_side": s["device"].cut_sides(1)}
    if op == "adjoint":
        s["device"].set_capacities(s["cap"])
        flow = int(s["device"].solve(algo).flow)
        return {"flow": flow, "sink_grad": s["device"].mincut_adjoint(0)[0], "source_grad": s["device"].mincut_adjoint(1)[0]}
    if op == "batch":
        return {"flows": s["batch"].solve()[0]}
    if op == "dropin":
        state = W.rcsr_preflow(s["graph"], *s["reverse"])
        flow, _, _ = W.rcsr_push_relabel(W.ALGOS[algo], s["graph"], state, *s["reverse"])
        return {"flow": flow}
    flow = C.c_int64(-1)
    status = W.lib().wbpr_solve_bcsr_noalloc(s["n"], s["arcs"], s["row"].data_ptr(), s["arc"].data_ptr(), s["arx"].data_ptr(),
                                             s["s"], s["t"], W.ALGOS[algo], torch.cuda.current_stream().cuda_stream, C.byref(flow))
    if status:
        raise RuntimeError(W.status_str(status))
    return {"flow": flow.value}


def _size(family, a, b):
    """(vertices, arcs) of a family's graph; the random ones on average."""
    if family == "genrmf":
        return a * a * b, 4 * a * (a - 1) * b + a * a * (b - 1)
    if family == "layered":
        return a * b + 2, 4.5 * a * b
    if family == "grid":
        return a * b + 2, 6 * a * b
    if family == "bipartite":
        return a + b + 2, 6.4 * a + b
    return 2 ** a, 0.96 * b * 2 ** a


def work(case):
    """The graph (offsets, heads, capacities) read once and the answer written once; one operation an arc."""
    op, a, b = case["op"], case["a"], case["b"]
    if op == "batch":  # half GENRMF, half layered: about 11,000 vertices and 50,000 arcs an instance
        return {"bytes": a * (11000 * 4 + 50000 * 8 + 8), "flops": a * 50000}
    n, m = _size(case["family"], a, b)
    out = {"cut": n, "recap": n, "adjoint": 2 * m}.get(op, 0) + 8
    return {"bytes": 4 * (n + 1) + 8 * m + out, "flops": m}


def _max_flow(g):
    """The maximum flow and both extreme minimum cuts, by shortest augmenting paths (Dinic) in Python integers."""
    n, m = g.n, len(g.dst)
    tail = np.repeat(np.arange(n), np.diff(g.off)).tolist()
    head, left = g.dst.tolist(), g.cap.tolist() + [0] * m  # arc i and its reverse m + i
    end = head + tail
    out = [[] for _ in range(n)]
    for i in range(m):
        out[tail[i]].append(i)
        out[head[i]].append(m + i)
    twin = list(range(m, 2 * m)) + list(range(m))

    def levels(root, backwards):
        d = [-1] * n
        d[root] = 0
        q = deque([root])
        while q:
            u = q.popleft()
            for i in out[u]:
                if d[end[i]] < 0 and left[twin[i] if backwards else i] > 0:
                    d[end[i]] = d[u] + 1
                    q.append(end[i])
        return d

    flow = 0
    while True:
        d = levels(g.s, False)
        if d[g.t] < 0:
            break
        at, path, u = [0] * n, [], g.s
        while True:
            if u == g.t:
                p = min(left[i] for i in path)
                flow += p
                for i in path:
                    left[i] -= p
                    left[twin[i]] += p
                k = next(k for k, i in enumerate(path) if left[i] == 0)
                u = end[twin[path[k]]]
                del path[k:]
                continue
            while at[u] < len(out[u]):
                i = out[u][at[u]]
                if left[i] > 0 and d[end[i]] == d[u] + 1:
                    break
                at[u] += 1
            if at[u] < len(out[u]):
                path.append(out[u][at[u]])
                u = end[path[-1]]
            elif path:
                u = end[twin[path.pop()]]
                at[u] += 1
            else:
                break
    return flow, np.array(levels(g.t, True)) >= 0, np.array(levels(g.s, False)) >= 0


def exact(case, seed):
    op, a, b = case["op"], case["a"], case["b"]
    if op == "batch" or _size(case["family"], a, b)[1] > 12000:
        return None  # too long in Python
    g = _graph(case, seed)
    flow, sink_side, source_side = _max_flow(g)
    tail = np.repeat(np.arange(g.n), np.diff(g.off))
    if op == "cut":
        return {"flow": flow, "sink_side": sink_side.astype(np.int8)}
    if op == "recap":
        return {"flow": flow, "source_side": source_side.astype(np.int8)}
    if op == "adjoint":
        return {"flow": flow, "sink_grad": (~sink_side[tail] & sink_side[g.dst]).astype(np.int8),
                "source_grad": (source_side[tail] & ~source_side[g.dst]).astype(np.int8)}
    return {"flow": flow}
