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
