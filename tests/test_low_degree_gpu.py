"""Searches of low-degree graphs (no list of more than 16 edges), which every
strategy runs as vertex levels on one cluster or the whole grid: labels against
the oracle and the reported statistics, at the edges of the kernel's variants
(4, 8 and 16 lanes a list), with frontiers that stay on the cluster, move to
the grid and back, and need compact queue room."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bfs_mod():
    import back40computing_b200 as b
    return b


def _regular(n, degree, seed, directed=False):
    """Union of random permutations: out-degree exactly `degree` (twice that when undirected)."""
    rng = np.random.default_rng(seed)
    rows = np.tile(np.arange(n), degree)
    cols = np.concatenate([rng.permutation(n) for _ in range(degree)])
    if not directed:
        rows, cols = np.concatenate([rows, cols]), np.concatenate([cols, rows])
    return bfs_mod().from_coo(n, rows.astype(np.int32), cols.astype(np.int32))


GRAPHS = {
    "path": lambda b: b.from_coo(3000, np.r_[:2999, 1:3000].astype(np.int32), np.r_[1:3000, :2999].astype(np.int32)),
    "one_vertex": lambda b: b.from_coo(1, [], []),
    "grid2d_tall": lambda b: b.grid2d(333),
    "grid3d_37": lambda b: b.grid3d(37),
    "grid3d_81": lambda b: b.grid3d(81),                      # leaves the cluster and comes back
    "degree4_random": lambda b: _regular(200_003, 2, 1),       # levels of most of the graph: compact room
    "degree8_directed": lambda b: _regular(100_001, 8, 2, True),
    "degree16": lambda b: _regular(60_001, 8, 3),
    "degree17": lambda b: _regular(5_001, 17, 4, True),        # one above: the strategies' own kernels
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("strategy", [0, 1, 2, 3])
def test_low_degree_matches_oracle(cuda_device, oracle, name, strategy):
    b = bfs_mod()
    g = GRAPHS[name](b)
    deg = np.diff(g.row_offsets)
    prob = b.CsrProblem(False).from_graph(g)
    for src in sorted({0, g.nodes // 2, g.nodes - 1}):
        ref, _ = oracle.bfs(g, src)
        d = int(ref.max())
        edges = int(deg[ref >= 0].sum())
        last = bool((deg[ref == d] > 0).any())
        depth = {0: {d}, 1: {d + last}, 2: {d}, 3: {d, d + last}}[strategy]
        queued = {0: int((ref >= 0).sum())}.get(strategy, 1 + edges)
        for instrument, sizing in ((False, 1.0), (True, 1.3)):
            en = b.make_enactor(strategy, INSTRUMENT=instrument)
            b.check(prob.Reset(en.GetFrontierType(), sizing))
            b.check(en.EnactSearch(prob, src))
            assert oracle.first_mismatch(prob.labels(), ref) == -1, (name, src, instrument)
            stats = en.GetStatistics()
            assert stats[1] in depth
            if instrument and name != "degree17":
                assert stats[0] == queued and 0.0 < stats[2] <= 1.0
