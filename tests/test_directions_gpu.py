"""Searches in a direction of the caller's choice: the grid and the split of the
work that the library picks for them."""
import time

import numpy as np
import pytest

from ceregraphs_gb300 import _lib, generators
from ceregraphs_gb300.engine import Graph

pytestmark = pytest.mark.gpu


def _searched(g, root, lv, pa, **options):
  """Median time of a search, in seconds."""
  import torch
  g.set_options(**options)
  times = []
  for _ in range(12):
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    g.bfs_device(root, lv, pa)
    torch.cuda.synchronize()
    times.append(time.perf_counter() - t0)
  assert g.last_stats()["status"] == 0
  return sorted(times)[len(times) // 2]


def _graph(scale, degree):
  g, _ = generators.rmat_device(scale, degree, 3, export=False)
  with_edges = np.nonzero(np.diff(g.export_offsets()))[0]
  return g, int(with_edges[len(with_edges) // 2])


CASES = [
    ("bottomup", 20, 4, dict(direction=_lib.CG_DIR_BOTTOMUP)),
    ("bottomup", 21, 16, dict(direction=_lib.CG_DIR_BOTTOMUP)),
    ("switch at once", 20, 4, dict(direction=_lib.CG_DIR_TAU, tau_switch_count=0)),
    ("switch late", 17, 128, dict(direction=_lib.CG_DIR_TAU)),
]


@pytest.mark.parametrize("name,scale,degree,options", CASES)
def test_default_grid_is_near_the_best(built_lib, name, scale, degree, options):
  """No more than 15% over the best of 1, 2 and 3 blocks an SM."""
  import torch
  g, root = _graph(scale, degree)
  with g:
    lv, pa = (torch.empty(g.n, dtype=torch.int32, device="cuda") for _ in range(2))
    best = min(_searched(g, root, lv, pa, blocks_per_sm=b, **options) for b in (1, 2, 3))
    assert _searched(g, root, lv, pa, blocks_per_sm=0, **options) < 1.15 * best


@pytest.mark.parametrize("options", [CASES[0][3], CASES[2][3]])
def test_early_pull_rounds_split_the_hubs(built_lib, options):
  """The hubs' lists are scanned to their ends in a pull round before its time: a
  search of pull rounds takes seven to eight times the direction-optimizing
  one, twelve and more where they go to few warps."""
  import torch
  g, root = _graph(20, 4)
  with g:
    lv, pa = (torch.empty(g.n, dtype=torch.int32, device="cuda") for _ in range(2))
    auto = _searched(g, root, lv, pa, direction=_lib.CG_DIR_AUTO)
    want = lv.clone(), pa.clone()
    assert _searched(g, root, lv, pa, **options) < 10 * auto
    assert torch.equal(lv, want[0]) and torch.equal(pa, want[1])


def test_large_graphs_of_bounded_degree(built_lib):
  """Bottom-up searches of 4 M vertices of bounded degree, which run in the common
  kernel, against direction-optimizing ones, which run in the team's."""
  import ctypes
  import torch
  n, m = 1 << 22, 5_000_000
  gen = torch.Generator(device="cuda").manual_seed(1)
  src, dst = (torch.randint(0, n, (m,), generator=gen, device="cuda", dtype=torch.int32)
              for _ in range(2))
  torch.cuda.synchronize()
  h = ctypes.c_void_p()
  _lib.check(_lib.load().cg_graph_from_edges(n, m, ctypes.c_void_p(src.data_ptr()),
                                             ctypes.c_void_p(dst.data_ptr()),
                                             _lib.CG_EDGES_DROP_LOOPS, ctypes.byref(h)), "build")
  with Graph.from_handle(h) as g:
    lv, pa = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    for root in range(0, n, n // 7):
      g.set_options(direction=_lib.CG_DIR_AUTO)
      g.bfs_device(root, lv, pa)
      rounds = g.last_stats()["rounds"]
      want = lv.clone(), pa.clone()
      g.set_options(direction=_lib.CG_DIR_BOTTOMUP)
      g.bfs_device(root, lv, pa)
      assert g.last_stats()["rounds"] == rounds
      assert torch.equal(lv, want[0]) and torch.equal(pa, want[1])
