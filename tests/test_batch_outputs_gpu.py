"""Batched outputs at the edges of the output pass: vertex counts around tiles
and residues of 16-byte rows, outputs that start off 16 bytes, lane counts
around words, in-degrees around the light limit, positions to the last entry,
levels past one batch of planes."""
import numpy as np
import pytest

from ceregraphs_gb300.engine import Graph
from ceregraphs_gb300.preprocess import from_edges

pytestmark = pytest.mark.gpu


def _graph(n, seed, chain):
  """Directed: random edges, a chain through the first vertices (deep levels),
  and vertices of in-degree 31, 32, 33, 64 whose parents sit anywhere in the list."""
  rng = np.random.default_rng(seed)
  src, dst = [rng.integers(0, n, 3 * n)], [rng.integers(0, n, 3 * n)]
  c = min(chain, n - 1)
  src.append(np.arange(c))
  dst.append(np.arange(c) + 1)
  for i, d in enumerate([31, 32, 33, 64]):
    if n > 200:
      src.append(rng.choice(n, size=d, replace=False))
      dst.append(np.full(d, n - 1 - i))
  return from_edges(n, np.concatenate(src), np.concatenate(dst), drop_self_loops=True)


def _sparse(n, seed):
  """Half the vertices get no edge; long light lists from a few sources."""
  rng = np.random.default_rng(seed)
  m = 16 * (n // 2)
  return from_edges(n, rng.integers(0, n, m), rng.integers(0, max(1, n // 2), m), symmetrize=False,
                    drop_self_loops=True)


def _run(oracle_mod, a, k, offsets, rng, lane_words):
  import torch
  roots = rng.integers(0, a.n, k).tolist()
  if k > 2:
    roots[1] = roots[0]  # the same root twice
  with Graph(a) as g:
    g.set_options(lane_words=lane_words)
    store = [torch.full((k * a.n + 8,), -9, dtype=torch.int32, device="cuda") for _ in range(2)]
    out = [s[o:o + k * a.n].view(k, a.n) for s, o in zip(store, offsets)]
    torch.cuda.synchronize()
    g.msbfs_device(roots, *out)
    st = g.last_stats()
    assert st["status"] == 0
    hosts = [s.cpu().numpy() for s in store]
  want = [oracle_mod.bfs(*a.out_lists(), a.in_off, a.in_idx, r) for r in roots]
  for h, o, which in zip(hosts, offsets, (0, 1)):
    assert np.all(h[:o] == -9) and np.all(h[o + k * a.n:] == -9)  # nothing written outside
    got = h[o:o + k * a.n].reshape(k, a.n)
    for i in range(k):
      assert np.array_equal(got[i], want[i][which]), (which, i)
  assert st["visited"] == sum(int((w[0] >= 0).sum()) for w in want)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 27, 28, 29, 31, 32, 33, 56, 57, 63, 64, 65, 1000, 1001,
                               1002, 1003, 4096])
def test_sizes(built_lib, oracle_mod, n):
  rng = np.random.default_rng(n)
  for a in (_graph(n, n, 20), _sparse(n, n)):
    for k, lane_words in ((5, 1), (64, 1), (100, 2)):
      _run(oracle_mod, a, k, (0, 0), rng, lane_words)


@pytest.mark.parametrize("offsets", [(1, 1), (2, 2), (3, 3), (0, 1), (3, 2), (4, 0)])
@pytest.mark.parametrize("n", [999, 1000, 1002])
def test_outputs_off_16_bytes(built_lib, oracle_mod, n, offsets):
  _run(oracle_mod, _graph(n, 7, 10), 40, offsets, np.random.default_rng(n), 1)


@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128])
def test_lane_counts(built_lib, oracle_mod, k):
  _run(oracle_mod, _graph(515, 3, 30), k, (0, 0), np.random.default_rng(k), 1 if k <= 64 else 2)
