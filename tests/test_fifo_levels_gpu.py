"""FIFO parents where the pass changes its way: lists around the thread / warp /
chunk limits on both sides, levels of one vertex, runs of small levels of
every length between wide ones, more levels than are summed or fit a byte."""
import numpy as np
import pytest

from ceregraphs_gb300 import _lib
from ceregraphs_gb300.engine import Graph
from ceregraphs_gb300.preprocess import from_edges

pytestmark = pytest.mark.gpu


def _layers(widths, degree, rng, both):
  first = np.concatenate([[0], np.cumsum(widths)])
  ids = rng.permutation(int(first[-1]))  # queue order and id order differ
  src, dst = [], []
  for i, w in enumerate(widths[:-1]):
    nxt = widths[i + 1]
    k = max(degree, -(-nxt // w))
    src.append(first[i] + np.repeat(np.arange(w), k))
    dst.append(first[i + 1] + rng.integers(0, nxt, w * k))
    src.append(first[i] + rng.integers(0, w, nxt))  # every vertex has a parent
    dst.append(first[i + 1] + np.arange(nxt))
  src, dst = ids[np.concatenate(src)], ids[np.concatenate(dst)]
  return from_edges(int(first[-1]), src, dst, symmetrize=both), int(ids[0])


CASES = {
    "one_then_wide": ([1, 1, 9000, 1, 1, 20000, 3], 2),
    "hubs_push": ([1, 3, 12000, 40, 9000], 2),          # out-lists of thousands
    "hubs_pull": ([1, 9000, 2, 9000, 5], 3),            # in-lists of thousands
    "limits": ([1, 40, 1300, 33, 1056, 32, 1024, 31], 1),
    "small_runs": ([1, 9000, 50, 9000, 50, 60, 9000, 50, 60, 70, 9000, 10, 10, 10, 10, 9000], 2),
    "small_edge": ([1, 8191, 8192, 8193, 8192, 100, 100, 100, 100], 2),
    "deep": ([1] + [9, 30] * 40 + [9000] + [7] * 10, 2),
    "very_deep": ([1] + [4] * 300 + [9000, 2, 2, 2, 9000], 2),
}


@pytest.mark.parametrize("both", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_fifo_parents_of_layered_graphs(built_lib, oracle_mod, name, both):
  widths, degree = CASES[name]
  rng = np.random.default_rng(len(name))
  a, root = _layers(widths, degree, rng, both)
  with Graph(a) as g:
    g.set_options(parent_rule=_lib.CG_PARENT_FIFO)
    for r in [root, root] + rng.integers(0, a.n, 3).tolist():  # the kept state, too
      lv, pa, st = g.bfs(r)
      rl, _, _ = oracle_mod.bfs(*a.out_lists(), a.in_off, a.in_idx, r)
      assert st["status"] == 0 and np.array_equal(lv, rl)
      assert np.array_equal(pa, oracle_mod.fifo_parents(a.in_off, a.in_idx, rl, r))


@pytest.mark.parametrize("levels", [2, 63, 64, 65, 255, 256, 257, 4000])
def test_levels_listed_in_id_order(built_lib, oracle_mod, levels):
  """The listing's passes (one up to 64 levels, one for each 8 bits beyond), on a
  ragged number of vertices with levels all over the ids and half of them unreached."""
  rng = np.random.default_rng(levels)
  per = max(1, 12_345 // levels)
  widths = [1] + [int(w) for w in rng.integers(1, 2 * per + 1, levels - 1)]
  a, root = _layers(widths, 2, rng, False)
  src = np.repeat(np.arange(a.n), np.diff(a.out_lists()[0]))
  n = 2 * a.n + 77
  ids = rng.permutation(n)
  a = from_edges(n, ids[src], ids[a.out_lists()[1]])
  root = int(ids[root])
  rl, _, _ = oracle_mod.bfs(*a.out_lists(), a.in_off, a.in_idx, root)
  assert rl.max() == levels - 1
  with Graph(a) as g:
    g.set_options(parent_rule=_lib.CG_PARENT_FIFO)
    for _ in range(2):
      lv, pa, _ = g.bfs(root)
      assert np.array_equal(lv, rl)
      assert np.array_equal(pa, oracle_mod.fifo_parents(a.in_off, a.in_idx, rl, root))


def test_more_levels_than_two_bytes(built_lib):
  """Two vertices a level, each with edges to both of the next: all of a level have
  the same parent, the lower vertex of the level before."""
  rng = np.random.default_rng(8)
  depth = 66_000
  n = 2 * depth + 1000
  ids = rng.permutation(n)
  root, pairs = int(ids[0]), ids[1:2 * depth + 1].reshape(depth, 2)
  src = np.concatenate([[root, root]] + [pairs[:-1, i] for i in (0, 0, 1, 1)])
  dst = np.concatenate([pairs[0]] + [pairs[1:, i] for i in (0, 1, 0, 1)])
  want = np.full(n, -1, dtype=np.int32)
  want[root], want[pairs[0]] = root, root
  want[pairs[1:]] = pairs[:-1].min(axis=1)[:, None]
  with Graph(from_edges(n, src, dst)) as g:
    g.set_options(parent_rule=_lib.CG_PARENT_FIFO)
    lv, pa, st = g.bfs(root)
    assert st["rounds"] == depth + 1
    assert np.array_equal(lv[pairs], np.repeat(np.arange(1, depth + 1), 2).reshape(depth, 2))
    assert np.array_equal(pa, want)


def test_hubs_past_the_counted_levels(built_lib, oracle_mod):
  """Long lists on levels whose entries are not counted (from 64 on)."""
  rng = np.random.default_rng(3)
  a, root = _layers([1] + [5] * 70 + [6000, 12, 6000, 3, 5000, 40, 40, 40, 2000], 3, rng, True)
  with Graph(a) as g:
    g.set_options(parent_rule=_lib.CG_PARENT_FIFO)
    lv, pa, _ = g.bfs(root)
    rl, _, _ = oracle_mod.bfs(*a.out_lists(), a.in_off, a.in_idx, root)
    assert rl.max() > 70 and np.array_equal(lv, rl)
    assert np.array_equal(pa, oracle_mod.fifo_parents(a.in_off, a.in_idx, rl, root))
