"""Searches whose rounds a team of blocks runs: plateaus of frontiers above what
one block takes, growth past the team's limits, uneven shares, long runs."""
import numpy as np
import pytest

from ceregraphs_gb300 import _lib
from ceregraphs_gb300.engine import Graph
from ceregraphs_gb300.preprocess import from_edges

pytestmark = pytest.mark.gpu


def _layers(widths, degree, seed, hubs=()):
  """Directed layers; each vertex has `degree` targets in the next layer (all of
  it from a layer of one).  hubs: (layer, vertices, targets each) of additional
  edges from the layer's first vertices."""
  rng = np.random.default_rng(seed)
  first = np.concatenate([[0], np.cumsum(widths)])
  src, dst = [], []
  for i, w in enumerate(widths[:-1]):
    nxt = widths[i + 1]
    if w == 1:
      src.append(np.full(nxt, first[i]))
      dst.append(first[i + 1] + np.arange(nxt))
      continue
    # in-degrees as even as they can be: the next layer's vertices in turn
    src.append(first[i] + np.repeat(np.arange(w), degree))
    dst.append(first[i + 1] + rng.permutation(np.arange(w * degree) % nxt))
  for layer, count, targets in hubs:
    for h in range(count):
      src.append(np.full(targets, first[layer] + h))
      dst.append(first[layer + 1] + (h * targets + np.arange(targets)) % widths[layer + 1])
  # (vertices without edges make up the size from which teams run)
  n = max(int(first[-1]), 1 << 16)
  return from_edges(n, np.concatenate(src), np.concatenate(dst))


def _check(oracle_mod, a, g, root=0):
  lv, pa, st = g.bfs(root)
  rl, rp, rounds = oracle_mod.bfs(*a.out_lists(), a.in_off, a.in_idx, root)
  assert st["status"] == 0 and st["rounds"] == rounds
  assert st["visited"] == int((rl >= 0).sum())
  assert np.array_equal(lv, rl) and np.array_equal(pa, rp)


@pytest.mark.parametrize("direction", [_lib.CG_DIR_AUTO, _lib.CG_DIR_TOPDOWN])
@pytest.mark.parametrize("width,degree", [(341, 3), (342, 3), (512, 2), (513, 2), (600, 3),
                                          (1000, 4), (1279, 3), (1025, 1)])
def test_plateaus(built_lib, oracle_mod, width, degree, direction):
  up = [1] + [v for v in (40, 70, 120, 200, 300, 450, 700, 1000) if v < width]
  widths = up + [width] * 12 + up[:2:-1] + [60] * 2 + up[3:] + [width] * 9
  a = _layers(widths, degree, width)
  with Graph(a) as g:
    g.set_options(direction=direction)
    _check(oracle_mod, a, g)


def test_growth_past_the_limits_and_back(built_lib, oracle_mod):
  widths = [1, 50, 100, 200] + [int(400 * 1.15 ** i) for i in range(26)]
  widths += widths[::-1][1:-2]
  for degree in (2, 3):
    a = _layers(widths, degree, degree)
    with Graph(a) as g:
      g.set_options(direction=_lib.CG_DIR_TOPDOWN)
      _check(oracle_mod, a, g)


@pytest.mark.parametrize("widths,hubs", [
    ([1, 50, 300] + [700] * 8 + [4000, 1500, 700], [(10, 40, 90)]),    # one block claims most
    ([1, 50, 300] + [700] * 8 + [5000], [(10, 3, 1500)]),               # claims without out-edges
    ([1, 50, 300] + [700] * 9 + [1300000], [(11, 1, 1300000)]),         # out-degrees past 20 bits
])
def test_uneven_shares(built_lib, oracle_mod, widths, hubs):
  a = _layers(widths, 2, 7, hubs)
  with Graph(a) as g:
    for direction in (_lib.CG_DIR_AUTO, _lib.CG_DIR_TOPDOWN):
      g.set_options(direction=direction)
      _check(oracle_mod, a, g)


def test_runs_longer_than_a_session_and_the_time_limit(built_lib, oracle_mod):
  a = _layers([1, 50, 300] + [600] * 1700, 2, 11)
  with Graph(a) as g:
    _check(oracle_mod, a, g)
    for ms in (4, 1):  # the search takes longer
      g.set_options(wait_timeout_ms=ms)
      for _ in range(3):
        _check(oracle_mod, a, g)


@pytest.mark.parametrize("cap", [10, 16, 17, 40])
def test_level_cap_inside_a_run(built_lib, oracle_mod, cap):
  a = _layers([1, 50, 300] + [600] * 60, 2, 13)
  with Graph(a) as g:
    g.set_options(level_cap=cap)
    with pytest.raises(_lib.CgError) as e:
      g.bfs(0)
    assert e.value.status == _lib.CG_ERR_LEVEL_CAP
    g.set_options(level_cap=0)
    _check(oracle_mod, a, g)


@pytest.mark.parametrize("block_size", [64, 192, 512])
def test_square_grid(built_lib, oracle_mod, block_size):
  side = 601
  v = np.arange(side * side).reshape(side, side)
  src = np.concatenate([v[:, :-1].ravel(), v[:-1].ravel()])
  dst = np.concatenate([v[:, 1:].ravel(), v[1:].ravel()])
  a = from_edges(side * side, src, dst, symmetrize=True)
  with Graph(a) as g:
    g.set_options(block_size=block_size)
    for root in (0, side * side // 2):
      _check(oracle_mod, a, g, root)
