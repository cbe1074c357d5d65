"""Where a team of blocks runs a search's small rounds: the searches that have one and
those just below the limits, a degree-ordered copy, a captured search, every
direction."""
import ctypes

import numpy as np
import pytest

from ceregraphs_gb300 import _lib
from ceregraphs_gb300.engine import Graph
from test_team_rounds_gpu import _check, _layers

pytestmark = pytest.mark.gpu

UP = (40, 70, 120, 200, 300, 450, 700, 1000)


def _plateau(width, degree, n=1 << 16):
  up = [1] + [v for v in UP if v < width]
  a = _layers(up + [width] * 12 + up[:2:-1] + [60] * 2, degree, width)
  assert a.n == n
  return a


def _runs(g):
  runs = ctypes.c_int32(-1)
  _lib.check(_lib.load().cg_test_team_runs(g.handle, ctypes.byref(runs)), "cg_test_team_runs")
  return runs.value


# a run on one block becomes the team's after four rounds of more than 1,024 edges
# (a layer loses the few edges that are drawn twice)
@pytest.mark.parametrize("width,degree,team", [(341, 3, False), (360, 3, True), (512, 2, False),
                                               (530, 2, True), (600, 3, True), (1000, 4, True),
                                               (1279, 3, True)])
def test_plateaus_above_the_limit_are_the_teams(built_lib, oracle_mod, width, degree, team):
  a = _plateau(width, degree)
  with Graph(a) as g:
    _check(oracle_mod, a, g)
    assert (_runs(g) > 0) == team


@pytest.mark.parametrize("width,team", [(1024, False), (1025, True)])
def test_limit_of_the_team(built_lib, oracle_mod, width, team):
  a = _layers([1] + [width] * 12, 1, width)  # `width` edges a round, one a vertex
  with Graph(a) as g:
    _check(oracle_mod, a, g)
    assert (_runs(g) > 0) == team


def test_hub_graphs_and_short_runs_have_no_team(built_lib, oracle_mod):
  hubs = _layers([1, 40, 300] + [600] * 8 + [60] + [600] * 4, 3, 5)  # in-lists of 30
  assert 1024 * (np.diff(hubs.in_off) * (np.diff(hubs.in_off) > 8)).sum() > hubs.nnz
  short = _layers([1, 40, 300, 700, 700, 700, 100], 3, 5)  # three rounds of 2,100 edges
  for a in (hubs, short):
    with Graph(a) as g:
      _check(oracle_mod, a, g)
      assert _runs(g) == 0


def test_long_runs_are_handed_out_again(built_lib, oracle_mod):
  a = _layers([1, 50, 300] + [600] * 400, 2, 11)
  with Graph(a) as g:
    _check(oracle_mod, a, g)
    assert _runs(g) >= 400 // 64


@pytest.mark.parametrize("direction,tau,team", [
    (_lib.CG_DIR_AUTO, -1, True), (_lib.CG_DIR_TOPDOWN, -1, True), (_lib.CG_DIR_BOTTOMUP, -1, False),
    (_lib.CG_DIR_TAU, -1, True), (_lib.CG_DIR_TAU, 1 << 15, True), (_lib.CG_DIR_TAU, 400, False)])
@pytest.mark.parametrize("reordered", [False, True])
def test_team_in_every_direction_and_on_a_relabelled_copy(built_lib, oracle_mod, direction, tau,
                                                          team, reordered):
  a = _plateau(700, 3)
  with Graph(a) as g, g.reorder() as copy:
    h = copy if reordered else g
    h.set_options(direction=direction, tau_switch_count=tau)
    for root in (0, 5):
      _check(oracle_mod, a, h, root)
      assert (_runs(h) > 0) == team


@pytest.mark.parametrize("reordered", [False, True])
def test_team_in_a_capture(built_lib, oracle_mod, reordered):
  import torch
  a = _plateau(700, 3)
  roots = [0, 3]
  with Graph(a) as g, g.reorder() as copy:
    h = copy if reordered else g
    out = torch.empty((4, a.n), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    exe = h.capture(lambda: [h.bfs_device(r, out[2 * i], out[2 * i + 1])
                             for i, r in enumerate(roots)])
    for _ in range(3):
      out.fill_(7)
      torch.cuda.synchronize()
      exe.launch()
      assert h.last_stats()["status"] == 0 and _runs(h) > 0
      for i, r in enumerate(roots):
        rl, rp, _ = oracle_mod.bfs(*a.out_lists(), a.in_off, a.in_idx, r)
        assert np.array_equal(out[2 * i].cpu().numpy(), rl)
        assert np.array_equal(out[2 * i + 1].cpu().numpy(), rp)
    exe.close()
