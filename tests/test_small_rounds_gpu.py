"""Searches whose rounds one block runs alone: frontiers and edge counts around
the limits of such runs, and runs longer than one wait's time limit."""
import numpy as np
import pytest

from ceregraphs_gb300 import _lib
from ceregraphs_gb300.engine import Graph
from ceregraphs_gb300.preprocess import from_edges

pytestmark = pytest.mark.gpu


def _layers(widths, degree, seed):
  """Directed layers of the given widths; each vertex has `degree` targets in
  the next layer (all of a layer of one; the first vertex is the root)."""
  rng = np.random.default_rng(seed)
  first = np.concatenate([[0], np.cumsum(widths)])
  src, dst = [], []
  for i, w in enumerate(widths[:-1]):
    nxt = widths[i + 1]
    if w == 1:
      src.append(np.full(nxt, first[i]))
      dst.append(first[i + 1] + np.arange(nxt))
      continue
    src.append(first[i] + np.repeat(np.arange(w), degree))
    dst.append(first[i + 1] + rng.integers(0, nxt, w * degree))
  return from_edges(int(first[-1]), np.concatenate(src), np.concatenate(dst))


def _check(oracle_mod, a, g, root):
  lv, pa, st = g.bfs(root)
  rl, rp, rounds = oracle_mod.bfs(*a.out_lists(), a.in_off, a.in_idx, root)
  assert st["status"] == 0 and st["rounds"] == rounds
  assert st["visited"] == int((rl >= 0).sum())
  assert np.array_equal(lv, rl) and np.array_equal(pa, rp)


@pytest.mark.parametrize("direction", [_lib.CG_DIR_AUTO, _lib.CG_DIR_TOPDOWN])
@pytest.mark.parametrize("width,degree", [(639, 3), (640, 3), (641, 3), (700, 2), (1279, 3),
                                          (1280, 3), (1281, 3), (2500, 1), (512, 4), (513, 4),
                                          (1023, 4), (1024, 4), (1025, 4), (40, 100)])
def test_frontiers_around_the_limits(built_lib, oracle_mod, width, degree, direction):
  # up to the width and down again, so runs start, end and start anew
  widths = [1, 3, 60, 500, width, width, width, 5, 1, 900, width, 30, 30, 1]
  a = _layers(widths, degree, width)
  with Graph(a) as g:
    g.set_options(direction=direction)
    for root in (0, 1, a.n - 1):
      _check(oracle_mod, a, g, root)


def test_run_longer_than_the_time_limit(built_lib, oracle_mod):
  i = np.arange(7999)
  a = from_edges(8000, i, i + 1, symmetrize=True)
  with Graph(a) as g:
    g.set_options(wait_timeout_ms=8)  # the search takes longer
    _check(oracle_mod, a, g, 0)


@pytest.mark.parametrize("block_size,blocks_per_sm", [(64, 0), (256, 1), (512, 1)])
def test_other_block_shapes(built_lib, oracle_mod, block_size, blocks_per_sm):
  a = _layers([1, 200, 1000, 1300, 20, 1], 3, 5)
  with Graph(a) as g:
    g.set_options(block_size=block_size, blocks_per_sm=blocks_per_sm)
    _check(oracle_mod, a, g, 0)
