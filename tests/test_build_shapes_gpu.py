"""Graph construction from device edge lists at the edges of its ranges: vertex
counts around powers of two, empty and loop-only lists, long runs of rows
without entries, hubs, and every flag, against the host construction."""
import ctypes

import numpy as np
import pytest

from ceregraphs_gb300 import _lib, preprocess
from ceregraphs_gb300.engine import Graph

pytestmark = pytest.mark.gpu


def _lists(n, kind, rng):
  if kind == "random":
    return rng.integers(0, n, 5 * n + 7), rng.integers(0, n, 5 * n + 7)
  if kind == "loops":
    v = rng.integers(0, n, 50)
    return v, v
  if kind == "ends":  # only the first and the last vertices: long gaps
    v = np.concatenate([np.arange(min(n, 3)), np.arange(max(0, n - 3), n)])
    return rng.choice(v, 40), rng.choice(v, 40)
  if kind == "hub":
    return np.concatenate([np.zeros(n, np.int64), rng.integers(0, n, n)]), \
        np.concatenate([np.arange(n), np.full(n, n - 1)])
  return np.array([n - 1]), np.array([0])  # one edge


@pytest.mark.parametrize("flags", range(8))
@pytest.mark.parametrize("n", [1, 2, 3, 64, 65, 127, 128, 129, 4096, 4097, 200_000])
def test_build_matches_host(built_lib, n, flags):
  import torch
  sym, drop = bool(flags & 1), bool(flags & 2)
  rng = np.random.default_rng(n + flags)
  for kind in ("random", "loops", "ends", "hub", "one"):
    src, dst = (x.astype(np.int32) for x in _lists(n, kind, rng))
    ds, dd = torch.from_numpy(src).cuda(), torch.from_numpy(dst).cuda()
    torch.cuda.synchronize()
    h = ctypes.c_void_p()
    _lib.check(_lib.load().cg_graph_from_edges(n, len(src), ctypes.c_void_p(ds.data_ptr()),
                                               ctypes.c_void_p(dd.data_ptr()), flags,
                                               ctypes.byref(h)), "from_edges")
    with Graph.from_handle(h) as g:
      a = g.export()
    want = preprocess.from_edges(n, src, dst, symmetrize=sym, drop_self_loops=drop)
    assert a.nnz == want.nnz
    assert np.array_equal(a.in_off, want.in_off) and np.array_equal(a.in_idx, want.in_idx), kind
    if flags & 4 or sym:
      assert a.symmetric == want.symmetric
    oo, oi = a.out_lists()
    wo, wi = want.out_lists()
    assert np.array_equal(oo, wo) and np.array_equal(oi, wi), kind
