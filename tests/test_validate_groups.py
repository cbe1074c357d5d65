"""The grouped tree checks at the edges of their ranges: searches per group,
in-lists around the thread / warp / chunk limits, levels around the byte limit."""
import numpy as np
import pytest

from ceregraphs_gb300 import generators
from ceregraphs_gb300.preprocess import from_edges

CHECKS = ("root", "tree", "edges", "span", "tree_edge", "lowest")


def _degrees_graph(n, seed):
  """Directed graph with in-degrees at 1, 32/33, 128/129, 512/513, 1024/1025
  and 2000 among random ones."""
  rng = np.random.default_rng(seed)
  src, dst = [], []
  for v, d in enumerate([1, 31, 32, 33, 127, 128, 129, 511, 512, 513, 1024, 1025, 2000]):
    at = v * 37 + 5
    src.append(rng.choice(n, size=d, replace=False))
    dst.append(np.full(d, at))
  src.append(rng.integers(0, n, 4 * n))
  dst.append(rng.integers(0, n, 4 * n))
  return from_edges(n, np.concatenate(src), np.concatenate(dst), drop_self_loops=True)


def _path(n):
  i = np.arange(n - 1)
  return from_edges(n, i, i + 1, symmetrize=True)


def _damage(lv, pa, n, rng, many):
  """Random mistakes in levels and parents, some far out of range."""
  lv, pa = lv.copy(), pa.copy()
  at = rng.integers(0, n, many)
  lv[at] = rng.choice([-1, -5, 0, 1, 2, 3, 125], size=many)
  at = rng.integers(0, n, many)
  pa[at] = rng.choice([-1, -2, 0, n - 1, n, n + 9, 2 ** 31 - 1], size=many)
  at = rng.integers(0, n, many)
  pa[at] = rng.integers(0, n, many)
  return lv, pa


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 4, 5, 8, 9, 16, 17, 35])
@pytest.mark.parametrize("kind", ["degrees", "rmat", "path126", "path127"])
def test_groups_match_oracle(built_lib, oracle_mod, kind, k):
  import torch
  from ceregraphs_gb300.engine import Graph
  a = {"degrees": lambda: _degrees_graph(3001, 3), "rmat": lambda: generators.rmat(11, 16, 4),
       # from vertex 0 the deepest level is 125 (the last that fits) or 126
       "path126": lambda: _path(126), "path127": lambda: _path(127)}[kind]()
  rng = np.random.default_rng(k)
  out_off, out_idx = a.out_lists()
  roots = [0] + rng.integers(0, a.n, k - 1).tolist()
  L, P = np.empty((k, a.n), np.int32), np.empty((k, a.n), np.int32)
  for i, r in enumerate(roots):
    L[i], P[i], _ = oracle_mod.bfs(out_off, out_idx, a.in_off, a.in_idx, r)
    if i % 3 != 1:  # some searches stay clean
      L[i], P[i] = _damage(L[i], P[i], a.n, rng, 1 + 7 * (i % 3))
  with Graph(a) as g:
    for _ in range(2):  # a second call on the kept workspace
      got = g.validate(roots, torch.from_numpy(L).cuda(), torch.from_numpy(P).cuda())
      for i, r in enumerate(roots):
        want = oracle_mod.validation_counts(a.in_off, a.in_idx, r, L[i], P[i])
        for c in CHECKS:
          assert (got[i][c]["failures"], got[i][c]["first"]) == want[c], (i, c, got[i], want)


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 15, 16, 17])
def test_edge_counts_of_groups(built_lib, k):
  import torch
  from ceregraphs_gb300.engine import Graph
  rng = np.random.default_rng(k)
  for a in (_degrees_graph(3001, 3), generators.rmat(11, 16, 4)):
    L = rng.integers(-1, 4, (k, a.n)).astype(np.int32)
    with Graph(a) as g:
      got = g.count_edges(torch.from_numpy(L).cuda(), k)
    dst = np.repeat(np.arange(a.n), np.diff(a.in_off))
    for i in range(k):
      seen = L[i] >= 0
      want = int(np.sum(seen[dst] & (a.in_idx <= dst))) if a.symmetric else int(seen[a.in_idx].sum())
      assert got[i] == want


@pytest.mark.gpu
@pytest.mark.parametrize("k", [4, 7, 16])
def test_large_graph_matches_oracle(built_lib, oracle_mod, k):
  # from 2^19 vertices on lists go to chunks later, and chunks are longer
  import torch
  from ceregraphs_gb300.engine import Graph
  a = _degrees_graph((1 << 19) + 3, 5)
  rng = np.random.default_rng(k)
  out_off, out_idx = a.out_lists()
  special = [v * 37 + 5 for v in range(13)]
  roots = [0] + rng.integers(0, a.n, k - 1).tolist()
  L, P = np.empty((k, a.n), np.int32), np.empty((k, a.n), np.int32)
  for i, r in enumerate(roots):
    L[i], P[i], _ = oracle_mod.bfs(out_off, out_idx, a.in_off, a.in_idx, r)
    if i % 3 == 1:
      continue
    L[i], P[i] = _damage(L[i], P[i], a.n, rng, 20)
    for j, v in enumerate(special):  # any in-neighbour, the last one, none of them
      nb = a.in_idx[a.in_off[v]:a.in_off[v + 1]]
      P[i][v] = (int(rng.choice(nb)), int(nb[-1]), int(rng.integers(0, a.n)))[(i + j) % 3]
      L[i][int(rng.choice(nb))] = int(rng.integers(0, 9))
  with Graph(a) as g:
    got = g.validate(roots, torch.from_numpy(L).cuda(), torch.from_numpy(P).cuda())
    for i, r in enumerate(roots):
      want = oracle_mod.validation_counts(a.in_off, a.in_idx, r, L[i], P[i])
      for c in CHECKS:
        assert (got[i][c]["failures"], got[i][c]["first"]) == want[c], (i, c, got[i], want)


def _caterpillar(spine, leaves):
  i, j = np.arange(spine - 1), np.arange(spine * leaves)
  return from_edges(spine * (leaves + 1), np.concatenate([i, j // leaves]),
                    np.concatenate([i + 1, spine + j]), symmetrize=True)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["grid200", "caterpillar"])
def test_deep_searches_side_by_side(built_lib, kind):
  """The checks of a small deep graph, whose levels pass a byte, fill the GPU with
  several searches at once: eight times the searches, which take nearly eight
  times as long one after another, take less than half of that."""
  import time
  import torch
  from ceregraphs_gb300.engine import Graph
  a = generators.grid2d(200) if kind == "grid200" else _caterpillar(3000, 30)
  with Graph(a) as g:
    took = {}
    for k in (8, 64):
      roots = list(range(k))
      lv, pa = (torch.empty((k, a.n), dtype=torch.int32, device="cuda") for _ in range(2))
      for i, r in enumerate(roots):
        g.bfs_device(r, lv[i], pa[i])
      g.last_stats()
      assert int(lv.max()) > 126
      times = []
      for _ in range(15):
        t0 = time.perf_counter()
        found = g.validate(roots, lv, pa)  # waits
        times.append(time.perf_counter() - t0)
      took[k] = sorted(times)[len(times) // 2]
      assert all(f[c]["failures"] == 0 for f in found for c in CHECKS)
  assert took[64] < 4 * took[8], took


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(3001, 32), (3001, 70), (100_003, 64)])
def test_groups_side_by_side_match_oracle(built_lib, oracle_mod, n, k):
  """Full groups of 16 searches run side by side on small graphs: all of them, the
  last of fewer searches alone, and (100,003 vertices) three at a time."""
  import torch
  from ceregraphs_gb300.engine import Graph
  a = _degrees_graph(n, 9)
  rng = np.random.default_rng(k)
  out_off, out_idx = a.out_lists()
  roots = [0] + rng.integers(0, a.n, k - 1).tolist()
  L, P = np.empty((k, a.n), np.int32), np.empty((k, a.n), np.int32)
  for i, r in enumerate(roots):
    L[i], P[i], _ = oracle_mod.bfs(out_off, out_idx, a.in_off, a.in_idx, r)
    if i % 3 != 1:
      L[i], P[i] = _damage(L[i], P[i], a.n, rng, 1 + 7 * (i % 3))
  L[20, 7] = 126  # past a byte: the second group's searches one at a time
  with Graph(a) as g:
    for _ in range(2):
      got = g.validate(roots, torch.from_numpy(L).cuda(), torch.from_numpy(P).cuda())
      for i, r in enumerate(roots):
        want = oracle_mod.validation_counts(a.in_off, a.in_idx, r, L[i], P[i])
        for c in CHECKS:
          assert (got[i][c]["failures"], got[i][c]["first"]) == want[c], (i, c, got[i], want)


@pytest.mark.gpu
def test_groups_of_a_small_graph_take_little_longer_than_one(built_lib):
  """Four groups in turn take more than three times as long as one; the GPU has
  room for all of a small graph's at once."""
  import time
  import torch
  from ceregraphs_gb300.engine import Graph
  a = generators.rmat(12, 16, 4)
  with Graph(a) as g:
    took = {}
    for k in (16, 64):
      roots = np.nonzero(np.diff(a.in_off))[0][:k].tolist()
      lv, pa = (torch.empty((k, a.n), dtype=torch.int32, device="cuda") for _ in range(2))
      g.msbfs_device(roots, lv, pa)
      g.last_stats()
      times = []
      for _ in range(15):
        t0 = time.perf_counter()
        g.validate(roots, lv, pa)  # waits
        times.append(time.perf_counter() - t0)
      took[k] = sorted(times)[len(times) // 2]
  assert took[64] < 2.5 * took[16], took
