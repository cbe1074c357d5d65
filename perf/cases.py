"""The work whose time this framework is judged by, one dict per case.

A user of the engine builds a resident graph (Kernel 1), searches it from
Graph500 roots one at a time (results left in HBM, or in page-locked host
memory as the Graph500 rule wants), searches 64 or 128 roots as one batch,
checks the trees, or asks for scipy's (FIFO) parents.  The listed cases take
each of these through the public entry points at the sizes of the drivers, the
tests and the benchmark (R-MAT scales 12 to 23, directed Erdos-Renyi graphs of
mean degree 8, 4-neighbour grids); draw() gives more of the same ranges, with
vertex counts that are no power of two among them.

A case's graph is one of
  rmat  the Graph500 R-MAT graph of ceil(log2(n)) levels, cut to its first n
        vertices (n a power of two: the benchmark's own graph)
  er    directed uniform random graph, n * degree edges before duplicates
  grid  the side x side 4-neighbour grid (n = side * side)
"""
import ctypes
import math

import numpy as np
import torch

from ceregraphs_gb300 import _lib, generators
from ceregraphs_gb300.engine import Graph

DIRECTIONS = {"auto": _lib.CG_DIR_AUTO, "topdown": _lib.CG_DIR_TOPDOWN}


def listed():
  return [
      # One search of a small graph, results left on the device: the smallest
      # call, all launch and round latency (a service's lookups).
      dict(name="search-rmat-4k", do="search", graph="rmat", n=1 << 12, degree=16,
           direction="auto"),
      # A mid-size graph of a ragged vertex count, searched top-down: what the
      # single-search driver runs unless told otherwise.
      dict(name="search-rmat-100k-topdown", do="search", graph="rmat", n=100_003, degree=16,
           direction="topdown"),
      # The benchmark's graph (scale 23), one Graph500 root.
      dict(name="search-rmat-8m", do="search", graph="rmat", n=1 << 23, degree=16,
           direction="auto"),
      # A directed graph (separate in- and out-lists) without hubs, ragged n.
      dict(name="search-er-3m", do="search", graph="er", n=3_000_001, degree=8,
           direction="auto"),
      # A deep search of tiny frontiers: up to 2044 rounds on a road-like grid.
      dict(name="search-grid-1m", do="search", graph="grid", n=1023 * 1023, degree=4,
           direction="auto"),
      # The Graph500 rule: levels and parents in page-locked host memory when
      # the call returns.
      dict(name="host-rmat-1m", do="host", graph="rmat", n=1 << 20, degree=16,
           direction="auto"),
      # 64 roots as one batch on a graph that fits the L2 cache.
      dict(name="batch64-rmat-256k", do="batch", graph="rmat", n=1 << 18, degree=16, roots=64),
      # The benchmark's batch: 64 Graph500 roots at scale 23.
      dict(name="batch64-rmat-8m", do="batch", graph="rmat", n=1 << 23, degree=16, roots=64),
      # A wide batch (128 lanes, some of them empty) on a directed graph.
      dict(name="batch100-er-1m", do="batch", graph="er", n=1_000_003, degree=8, roots=100),
      # scipy's parents (the reference driver's host check) for one search.
      dict(name="fifo-rmat-1m", do="fifo", graph="rmat", n=1 << 20, degree=16),
      # The Graph500 tree checks and edge counts of a batch of searches.
      dict(name="validate16-rmat-1m", do="validate", graph="rmat", n=1 << 20, degree=16, roots=16),
      # Kernel 1 from an edge list on the device, then the first search of it:
      # what a program that meets each graph once pays.
      dict(name="build-rmat-1m", do="build", graph="rmat", n=1 << 20, degree=16),
  ]


def _log_uniform(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  """One more case: sizes log-uniform over the range of each kind of work."""
  do = rng.choice(["search", "search", "host", "batch", "batch", "fifo", "validate", "build"])
  graph = "rmat"
  if do in ("search", "batch", "fifo", "validate"):
    graph = rng.choice(["rmat", "rmat", "er"] + (["grid"] if do == "search" else []))
  top = {"search": 1 << 23, "host": 1 << 21, "batch": 1 << 22, "fifo": 1 << 21,
         "validate": 1 << 20, "build": 1 << 21}[do]
  n = _log_uniform(rng, 1 << 12, min(top, 1 << 22) if graph == "er" else top)
  degree = rng.choice([8, 16, 32]) if graph == "rmat" else rng.choice([4, 8, 12])
  if graph == "grid":
    side = _log_uniform(rng, 64, 1023)
    n, degree = side * side, 4
  elif rng.random() < 0.3:
    n = 1 << max(12, n.bit_length() - 1)  # benchmarks use powers of two, data does not
  case = dict(do=do, graph=graph, n=n, degree=degree)
  if do in ("search", "host"):
    case["direction"] = rng.choice(["auto", "auto", "topdown"])
  if do == "batch":
    case["roots"] = rng.choice([64, rng.randint(4, 64), rng.randint(65, 128)])
  if do == "validate":
    case["roots"] = rng.randint(1, 16)
  return case


# ---- inputs ------------------------------------------------------------------
def _levels(n):
  return max(1, (n - 1).bit_length())


def _edges(case, seed):
  """(src, dst, flags) of a random graph as device tensors."""
  n, degree = case["n"], case["degree"]
  if case["graph"] == "rmat":
    u, v = generators.rmat_edges_device(_levels(n), degree, seed)
    if n != 1 << _levels(n):
      keep = (u < n) & (v < n)
      u, v = u[keep], v[keep]
    return u, v, _lib.CG_EDGES_SYMMETRIZE | _lib.CG_EDGES_DROP_LOOPS
  gen = torch.Generator(device="cuda").manual_seed(seed)
  u, v = (torch.randint(0, n, (n * degree,), generator=gen, device="cuda", dtype=torch.int32)
          for _ in range(2))
  return u, v, _lib.CG_EDGES_DROP_LOOPS


def _from_edges(n, src, dst, flags):
  h = ctypes.c_void_p()
  _lib.check(_lib.load().cg_graph_from_edges(n, len(src), ctypes.c_void_p(src.data_ptr()),
                                             ctypes.c_void_p(dst.data_ptr()), flags,
                                             ctypes.byref(h)), "cg_graph_from_edges")
  return Graph.from_handle(h)


def _graph(case, seed):
  if case["graph"] == "grid":
    return Graph(generators.grid2d(math.isqrt(case["n"])))
  src, dst, flags = _edges(case, seed)
  torch.cuda.synchronize()
  return _from_edges(case["n"], src, dst, flags)


def _roots(case, g, seed, k):
  """k distinct vertices that have neighbours (the Graph500 choice of roots)."""
  rng = np.random.default_rng([seed, 1])
  degree = np.diff(g.export_offsets())
  return rng.choice(np.nonzero(degree)[0], size=k, replace=False).tolist()


def prepare(case, seed):
  do, n = case["do"], case["n"]
  state = dict(do=do, n=n)
  k = case.get("roots", 1)
  shape = (k, n) if do in ("batch", "validate") else (n,)
  if do == "host":
    state["levels"], state["parents"] = (torch.empty(n, dtype=torch.int32, pin_memory=True)
                                         for _ in range(2))
  else:
    state["levels"] = torch.empty(shape, dtype=torch.int32, device="cuda")
    state["parents"] = torch.empty(shape, dtype=torch.int32, device="cuda")
  if do == "build":
    src, dst, flags = _edges(case, seed)
    state.update(edges=(src, dst, flags), root=int(src[int((src != dst).nonzero()[0])]))
    torch.cuda.synchronize()
    return state
  g = state["g"] = _graph(case, seed)
  state["roots"] = _roots(case, g, seed, k)
  state["root"] = state["roots"][0]
  if "direction" in case:
    g.set_options(direction=DIRECTIONS[case["direction"]])
  if do == "batch":
    g.set_options(lane_words=1 if k <= 64 else 2)
  if do == "fifo":
    g.set_options(parent_rule=_lib.CG_PARENT_FIFO)
  if do == "validate":
    # the searches' own results, the last one damaged in a few vertices so
    # that the checks have something to report
    g.msbfs_device(state["roots"], state["levels"], state["parents"])
    g.last_stats()
    at = torch.from_numpy(np.random.default_rng([seed, 2]).integers(0, n, size=5)).cuda()
    state["parents"][k - 1, at] = state["parents"][k - 1, at] + 1
  torch.cuda.synchronize()
  return state


# ---- one pass ------------------------------------------------------------------
def run(state):
  do = state["do"]
  levels, parents = state["levels"], state["parents"]
  if do in ("search", "fifo"):
    state["g"].bfs_device(state["root"], levels, parents)
    return {"levels": levels, "parents": parents}
  if do == "host":
    _, _, stats = state["g"].bfs(state["root"], levels, parents)
    return {"levels": levels, "parents": parents, "rounds": stats["rounds"],
            "visited": stats["visited"]}
  if do == "batch":
    state["g"].msbfs_device(state["roots"], levels, parents)
    return {"levels": levels, "parents": parents}
  if do == "validate":
    found = state["g"].validate(state["roots"], levels, parents)
    edges = state["g"].count_edges(levels, len(state["roots"]))
    return {"failures": np.array([[f[c]["failures"] for c in _lib.CG_CHECK_NAMES]
                                  for f in found]),
            "first": np.array([[f[c]["first"] for c in _lib.CG_CHECK_NAMES] for f in found]),
            "edges": edges}
  src, dst, flags = state["edges"]
  g = _from_edges(state["n"], src, dst, flags)
  offsets = g.export_offsets()
  g.bfs_device(state["root"], levels, parents)
  nnz = g.nnz
  g.close()  # waits for the search
  return {"nnz": nnz, "offsets": offsets, "levels": levels, "parents": parents}


# ---- what a pass cannot do without ----------------------------------------------
def _entries(case):
  """About the stored entries of the case's graph (duplicates merged)."""
  n, degree = case["n"], case["degree"]
  if case["graph"] == "grid":
    return 4 * n
  if case["graph"] == "er":
    return n * degree
  full = 1 << _levels(n)
  # an R-MAT edge stays with probability about (n / 2^levels)^0.81 (= 0.57 at a half)
  return 2 * 0.93 * full * degree * (n / full) ** 0.81


def work(case):
  """Each list entry, offset and output once (SpMV over the reached part)."""
  n, k, nnz = case["n"], case.get("roots", 1), _entries(case)
  adjacency, outputs = 4 * nnz + 8 * (n + 1), 8 * n * k
  if case["do"] == "build":  # edge list in, lists and offsets out, then the search
    m = nnz / 2 / 0.93
    return {"bytes": 8 * m + adjacency + adjacency + outputs, "flops": 0}
  return {"bytes": adjacency + outputs, "flops": 0}


# ---- the same in plain numpy ------------------------------------------------------
def _host_lists(case, seed):
  """(dst, src) of the stored entries, without this repository's code."""
  n, degree = case["n"], case["degree"]
  if case["graph"] == "rmat":
    m = degree << _levels(n)
    rng = np.random.default_rng(seed)
    u, v = np.zeros(m, dtype=np.int64), np.zeros(m, dtype=np.int64)
    for level in range(_levels(n)):
      r, bit = rng.random(m), 1 << (_levels(n) - 1 - level)
      ab = 0.57 + 0.19
      u += bit * (r >= ab)
      v += bit * (((r >= 0.57) & (r < ab)) | (r >= ab + 0.19))
    keep = (u < n) & (v < n) & (u != v)
    u, v = u[keep], v[keep]
    u, v = np.concatenate([u, v]), np.concatenate([v, u])
  elif case["graph"] == "er":
    gen = torch.Generator(device="cuda").manual_seed(seed)
    u, v = (torch.randint(0, n, (n * degree,), generator=gen, device="cuda", dtype=torch.int32)
            .cpu().numpy().astype(np.int64) for _ in range(2))
    u, v = u[u != v], v[u != v]
  else:
    side = math.isqrt(n)
    i = np.arange(n, dtype=np.int64)
    r, d = i[i % side < side - 1], i[i < n - side]
    u = np.concatenate([r, r + 1, d, d + side])
    v = np.concatenate([r + 1, r, d + side, d])
  key = np.unique(v * n + u)
  return key // n, key % n


def _host_search(n, dst, src, root):
  """Levels, and the lowest-numbered in-neighbour one level up."""
  level = np.full(n, -1, dtype=np.int64)
  level[root] = depth = 0
  while True:
    new = dst[(level[src] == depth) & (level[dst] < 0)]
    if not len(new):
      break
    depth += 1
    level[new] = depth
  parent = np.full(n, -1, dtype=np.int64)
  up = (level[src] >= 0) & (level[src] + 1 == level[dst])
  first = np.unique(dst[up], return_index=True)  # entries are sorted by (dst, src)
  parent[first[0]] = src[up][first[1]]
  parent[root] = root
  return level, parent


def exact(case, seed):
  """Searches of up to 2^17 vertices, in numpy; None for the other cases."""
  n = case["n"]
  if case["do"] != "search" or n > 1 << 17 or (case["graph"] == "grid" and n > 200 * 200):
    return None
  dst, src = _host_lists(case, seed)
  rng = np.random.default_rng([seed, 1])
  degree = np.bincount(dst, minlength=n)
  root = rng.choice(np.nonzero(degree)[0], size=1, replace=False).tolist()[0]
  level, parent = _host_search(n, dst, src, root)
  return {"levels": level, "parents": parent}
