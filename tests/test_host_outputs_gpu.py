"""One search into page-locked host buffers that do not start on 16 bytes."""
import numpy as np
import pytest

from ceregraphs_gb300 import _lib, generators
from ceregraphs_gb300.engine import Graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [40, 41])  # 1,600 and 1,681 vertices
@pytest.mark.parametrize("rule", [_lib.CG_PARENT_LOWEST, _lib.CG_PARENT_FIFO])
@pytest.mark.parametrize("offsets", [(0, 0), (1, 0), (0, 2), (3, 1)])
def test_unaligned_page_locked_outputs(built_lib, side, rule, offsets):
  import torch
  a = generators.grid2d(side)
  with Graph(a) as g:
    g.set_options(parent_rule=rule)
    want_l, want_p, _ = g.bfs(7)
    bufs = [torch.full((a.n + 8,), 99, dtype=torch.int32, pin_memory=True) for _ in range(2)]
    lv, pa = (b[o:o + a.n] for b, o in zip(bufs, offsets))
    g.bfs(7, lv, pa)
    assert np.array_equal(lv.numpy(), want_l) and np.array_equal(pa.numpy(), want_p)
    for b, o in zip(bufs, offsets):  # nothing beside them
      assert (b[:o] == 99).all() and (b[o + a.n:] == 99).all()
