"""Performance cases of the counting path: what a program that uses this
package has it do, each through a public entry point of ``Context``.

A case names a graph family with its sizes, the entry point (``entry``), the
dispatch option and the tuning entry of ``tuning.json`` (0 = the defaults).
``listed()`` gives the fixed cases, ``draw(rng)`` one more case of the same
ranges.  Inputs come from the package's seeded generators (``synth``), so
another seed is another graph of the same family.

Entries:
  device   ``count`` over an edge list in device memory (torch tensors)
  host     ``count`` over pinned host arrays, the copy to the device included
  packed   ``count_batch_packed`` over many graphs in device memory
  batch    ``count_batch`` over a list of graphs in host memory
  text     ``count_text`` over `u v sign` lines in host memory
  export   ``build_forward_csr``: host edge list to a host forward CSR
  csr      ``count_triangles`` over a host forward CSR
  vertex   ``vertex_counts``: per-source counts of a host edge list
"""
import math

import numpy as np
import torch

import signed_triangle_counting_b200 as stc
from signed_triangle_counting_b200 import autotune, synth


def listed():
    return [
        # The smallest call: a 100,000-edge random graph (workload 1), where
        # launches and synchronisations are the time.
        dict(name="er_100k", entry="device", family="er", n=10_000, m=100_000, p=0.7,
             dispatch="fixed", tuning=0),
        # A planar mesh of a million points (workload 2): short lists, the
        # graph build is the time.
        dict(name="delaunay_1m", entry="device", family="delaunay", n=1_000_000, m=0, p=0.6,
             dispatch="fixed", tuning=2),
        # A power-law graph of odd sizes under the default tuning, as a first
        # call on an unknown graph is.
        dict(name="rmat_odd_20m", entry="device", family="rmat", n=1_499_977, m=20_000_003, p=0.5,
             dispatch="fixed", tuning=0),
        # The benchmark's workload (3): RMAT scale 24, edge factor 16, the
        # largest graph counted.
        dict(name="rmat_24", entry="device", family="rmat", n=1 << 24, m=16 << 24, p=0.5,
             dispatch="fixed", tuning=3),
        # Hubs with millions of neighbours over a sparse backbone (workload
        # 5), under the learned dispatch tables.
        dict(name="skew_64m", entry="device", family="skew", n=64 << 20, m=128 << 20, p=0.8,
             dispatch="learned", tuning=5),
        # A share of the batched workload (4): many graphs of very different
        # sizes, resident, counted in one call.
        dict(name="batch_128", entry="packed", family="mixed", n=1_000_000, m=128, p=0.0,
             dispatch="fixed", tuning=4),
        # A request of a few dozen small graphs from host memory.
        dict(name="batch_small_48", entry="batch", family="mixed", n=20_000, m=48, p=0.0,
             dispatch="fixed", tuning=0),
        # A text file's bytes (1.8 million lines) through the device parser.
        dict(name="text_1800k", entry="text", family="rmat", n=120_011, m=1_800_001, p=0.5,
             dispatch="fixed", tuning=0),
        # End to end from pinned host memory: the copy, then the whole path.
        dict(name="host_rmat_21", entry="host", family="rmat", n=1 << 21, m=16 << 21, p=0.5,
             dispatch="fixed", tuning=3),
        # The forward CSR returned to the host, for programs that go on with
        # their own code.
        dict(name="export_er_4m", entry="export", family="er", n=262_147, m=4_194_301, p=0.5,
             dispatch="fixed", tuning=0),
        # Counting a forward CSR that the program already holds.
        dict(name="csr_rmat_19", entry="csr", family="rmat", n=400_009, m=16 << 19, p=0.5,
             dispatch="fixed", tuning=0),
        # Per-vertex counts.
        dict(name="vertex_rmat_20", entry="vertex", family="rmat", n=1 << 20, m=16 << 20, p=0.5,
             dispatch="fixed", tuning=0),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["er", "delaunay", "rmat", "rmat", "skew", "packed", "batch", "text", "host",
                       "export", "csr", "vertex"])
    dispatch = rng.choice(["fixed", "fixed", "fixed", "learned"])
    p = round(rng.uniform(0.3, 0.9), 3)
    if kind == "er":
        n = _log_uniform(rng, 1_000, 2_000_000)
        return dict(entry="device", family="er", n=n, m=rng.randint(2, 16) * n + rng.randint(0, n - 1),
                    p=p, dispatch=dispatch, tuning=0)
    if kind == "delaunay":
        return dict(entry="device", family="delaunay", n=_log_uniform(rng, 1_000, 1_000_000), m=0,
                    p=p, dispatch=dispatch, tuning=rng.choice([0, 2]))
    if kind == "rmat":
        n = _log_uniform(rng, 2_000, 8_000_000)
        return dict(entry="device", family="rmat", n=n, m=rng.randint(4, 16) * n + rng.randint(0, n),
                    p=p, dispatch=dispatch, tuning=rng.choice([0, 3]))
    if kind == "skew":
        n = _log_uniform(rng, 300_000, 32_000_000)
        return dict(entry="device", family="skew", n=n, m=2 * n + rng.randint(0, n), p=p,
                    dispatch=dispatch, tuning=rng.choice([0, 5]))
    if kind == "packed":
        return dict(entry="packed", family="mixed", n=_log_uniform(rng, 30_000, 1_000_000),
                    m=_log_uniform(rng, 8, 128), p=0.0, dispatch=dispatch, tuning=rng.choice([0, 4]))
    if kind == "batch":
        return dict(entry="batch", family="mixed", n=_log_uniform(rng, 2_000, 100_000),
                    m=_log_uniform(rng, 2, 64), p=0.0, dispatch=dispatch, tuning=0)
    n = _log_uniform(rng, 2_000, {"text": 200_000, "host": 2_000_000}.get(kind, 700_000))
    return dict(entry=kind, family="er" if kind == "export" else "rmat", n=n,
                m=rng.randint(4, 16) * n + rng.randint(0, n), p=p,
                dispatch=dispatch if kind in ("text", "host", "csr") else "fixed",
                tuning=rng.choice([0, 3]) if kind == "host" else 0)


# One context per (dispatch, tuning), kept by the program for all its graphs.
_contexts = {}


def _context(case):
    key = (case["dispatch"], case["tuning"])
    if key not in _contexts:
        ctx = stc.Context(0)
        if case["tuning"]:
            ctx.set_tuning(autotune.tuning_for(case["tuning"]))
        if case["dispatch"] == "learned":
            ctx.load_dispatch_model()
        _contexts[key] = ctx
    return _contexts[key]


def _scale(n):
    return max(1, (n - 1).bit_length())


def _edges(case, seed):
    """The case's edge list as host arrays (src, dst, sign)."""
    n, m, p, seed = case["n"], case["m"], case["p"], 7 + seed
    if case["family"] == "er":
        el = synth.er(seed, n, min(m, n * (n - 1) // 4), p)
    elif case["family"] == "delaunay":
        el = synth.delaunay(seed, n, 0.2, p)
    elif case["family"] == "rmat":
        el = synth.rmat(seed, _scale(n), n, m, p_pos=p)
    else:
        el = synth.skew(seed, n, m, 32, max(1, n // 671), max(2, n // 7), p)
    if case["entry"] in ("export", "vertex") and max(el.src.max(), el.dst.max()) < n - 1:
        # These outputs have a size that follows from the ids: the top id is
        # always used (ER edges are distinct, so their number is fixed too).
        el.dst[0] = n - 1
    return el.src, el.dst, el.sign


def _specs(case, seed):
    """Recipes of the batched workload's families with n in [1e3, case n]."""
    rng = np.random.default_rng(7 + seed)
    specs = []
    for _ in range(case["m"]):
        n = int(round(math.exp(rng.uniform(math.log(1_000), math.log(case["n"])))))
        kind = int(rng.integers(3))
        specs.append(dict(seed=int(rng.integers(1 << 62)), n=n, kind=kind,
                          rmat_scale=_scale(n) if kind == 1 else 0, m_target=(4 * n, 8 * n, 0)[kind],
                          p_pos=float(rng.uniform(0.3, 0.9))))
    return specs


def _text(src, dst, sign):
    """`u v sign` lines as bytes."""
    width = 10
    rows = np.empty((len(src), 2 * width + 5), np.uint8)
    keep = np.zeros(rows.shape, bool)
    for at, ids in ((0, src), (width + 1, dst)):
        x = ids.astype(np.int64)
        for k in range(width - 1, -1, -1):
            rows[:, at + k] = 48 + x % 10
            keep[:, at + k] = (x > 0) | (k == width - 1)
            x //= 10
        rows[:, at + width] = 32
        keep[:, at + width] = True
    rows[:, -3], rows[:, -2], rows[:, -1] = 45, 49, 10
    keep[:, -3], keep[:, -2], keep[:, -1] = sign < 0, True, True
    return rows[keep].tobytes()


def _to_device(src, dst, sign):
    dev = torch.device("cuda", 0)
    return (torch.from_numpy(src.view(np.int32)).to(dev), torch.from_numpy(dst.view(np.int32)).to(dev),
            torch.from_numpy(sign).to(dev))


def prepare(case, seed):
    ctx, entry = _context(case), case["entry"]
    state = dict(ctx=ctx, entry=entry, dispatch=case["dispatch"])
    if entry == "device" and case["family"] == "rmat":
        dev = torch.device("cuda", 0)
        edges = (torch.empty(case["m"], dtype=torch.int32, device=dev),
                 torch.empty(case["m"], dtype=torch.int32, device=dev),
                 torch.empty(case["m"], dtype=torch.int8, device=dev))
        ctx.synth_rmat_device(7 + seed, _scale(case["n"]), case["n"], case["m"], 0.57, 0.19, 0.19,
                              case["p"], *edges)
        state["edges"] = edges
    elif entry == "device":
        state["edges"] = _to_device(*_edges(case, seed))
    elif entry == "packed":
        el, state["offsets"] = synth.batch_packed(_specs(case, seed))
        state["edges"] = _to_device(el.src, el.dst, el.sign)
    elif entry == "batch":
        els = [synth.batch_graph(s) for s in _specs(case, seed)]
        state["graphs"] = [(el.src, el.dst, el.sign) for el in els]
    elif entry == "text":
        state["text"] = _text(*_edges(case, seed))
    elif entry == "host":
        pinned = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).pin_memory()
                  for a in _edges(case, seed)]
        state["pinned"] = pinned
        state["edges"] = (pinned[0].numpy().view(np.uint32), pinned[1].numpy().view(np.uint32),
                          pinned[2].numpy())
    elif entry == "csr":
        state["csr"] = ctx.build_forward_csr(*_edges(case, seed))
    else:
        state["edges"] = _edges(case, seed)
    torch.cuda.synchronize()
    return state


def run(state):
    ctx, entry, dispatch = state["ctx"], state["entry"], state["dispatch"]
    if entry in ("device", "host"):
        return ctx.count(*state["edges"], dispatch=dispatch).as_tuple()
    if entry == "packed":
        return np.array([c.as_tuple() for c in ctx.count_batch_packed(
            *state["edges"], state["offsets"], dispatch=dispatch)], np.int64)
    if entry == "batch":
        return np.array([c.as_tuple() for c in ctx.count_batch(state["graphs"], dispatch=dispatch)],
                        np.int64)
    if entry == "text":
        counts, lines, n = ctx.count_text(state["text"], dispatch=dispatch)
        return (*counts.as_tuple(), lines, n)
    if entry == "export":
        csr = ctx.build_forward_csr(*state["edges"])
        return dict(n=csr.n, m=csr.m, offsets=csr.offsets.view(np.int64),
                    edges=csr.edges.view(np.int32), signs=csr.signs, fdeg=csr.fdeg.view(np.int32),
                    rank=csr.rank.view(np.int32))
    if entry == "csr":
        return ctx.count_triangles(state["csr"], dispatch=dispatch).as_tuple()
    return ctx.vertex_counts(*state["edges"]).view(np.int64)


def _edge_count(case):
    """Input edges (expected, where the seed decides)."""
    if case["family"] == "delaunay":
        return 2.4 * case["n"]
    if case["family"] == "mixed":  # n log-uniform in [1e3, N]: mean (N - 1e3) / ln(N / 1e3)
        lo, hi = 1_000, max(1_001, case["n"])
        return case["m"] * (hi - lo) / math.log(hi / lo) * (4 + 8 + 2.4) / 3
    return float(case["m"])


def work(case):
    """Every input read once (9 bytes an edge: two ids and a sign), every
    output written once; the counting itself is integer work."""
    m, n, entry = _edge_count(case), case["n"], case["entry"]
    read = 9.0 * m
    if entry == "text":
        read = m * (2 * len(str(n)) + 4)
    elif entry == "csr":
        read = 5.0 * m + 16.0 * n
    written = {"export": 5.0 * m + 16.0 * n, "vertex": 32.0 * n, "packed": 32.0 * case["m"],
               "batch": 32.0 * case["m"]}.get(entry, 32.0)
    return {"bytes": read + written, "flops": 0.0}


def _count_plain(src, dst, sign):
    """Counts (t0, t1, t2, t3) in plain numpy: every pair of out-neighbours
    of a vertex (edges from lower to higher (degree, id)) looked up among the
    edges; None where there are too many pairs."""
    lo, hi = np.minimum(src, dst).astype(np.int64), np.maximum(src, dst).astype(np.int64)
    _, first = np.unique((lo << 32) | hi, return_index=True)
    first = first[lo[first] != hi[first]]
    lo, hi, neg = lo[first], hi[first], (sign[first] < 0).astype(np.int64)
    n = int(hi.max(initial=-1)) + 1
    deg = np.bincount(lo, minlength=n) + np.bincount(hi, minlength=n)
    rank = np.empty(n, np.int64)
    rank[np.lexsort((np.arange(n), deg))] = np.arange(n)
    a, b = np.minimum(rank[lo], rank[hi]), np.maximum(rank[lo], rank[hi])
    order = np.argsort((a << 32) | b)
    a, b, neg = a[order], b[order], neg[order]
    keys = (a << 32) | b
    left = np.searchsorted(a, a, side="right") - np.arange(len(a)) - 1  # later heads of the same tail
    total = int(left.sum())
    if total > 60_000_000:
        return None
    by = np.zeros(4, np.int64)
    step = max(1, int(len(a) * min(1.0, 4_000_000 / max(1, total))))
    for s in range(0, len(a), step):
        cnt = left[s:s + step]
        i = np.repeat(np.arange(s, s + len(cnt)), cnt)
        j = i + 1 + np.arange(len(i)) - np.repeat(np.cumsum(cnt) - cnt, cnt)
        want = (b[i] << 32) | b[j]
        at = np.minimum(np.searchsorted(keys, want), len(keys) - 1)
        hit = keys[at] == want
        by += np.bincount(neg[i][hit] + neg[j][hit] + neg[at][hit], minlength=4)
    return tuple(int(x) for x in by[::-1])


def exact(case, seed):
    entry = case["entry"]
    if entry == "batch":
        per = [_count_plain(el.src, el.dst, el.sign)
               for el in (synth.batch_graph(s) for s in _specs(case, seed))]
        return None if any(t is None for t in per) else np.array(per, np.int64)
    if entry not in ("device", "host", "csr") or _edge_count(case) > 3_000_000:
        return None
    return _count_plain(*_edges(case, seed))
