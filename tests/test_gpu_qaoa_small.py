"""Batched QAOA instances of up to 12 qubits, which stay in shared memory: every
qubit count, tile widths of the mixer's two parts, depths 1 to 16, no edges and
many, against the CPU oracle; graphs against plain launches, and a replayed graph
over another list of edges of the same shape.

Tolerances. Against the oracle: an operation rounds each component at most twice
(u = 2^-24), a layer has n mixer gates and one phase, there and back, and C is at
most W: 16 sqrt(2) u p (n + 1) W on the energy, W more on dE/dgamma (its factor
W - 2C), n on dE/dbeta (a sum over the qubits). Graph against plain launches: the
same kernels on the same data."""
import numpy as np
import pytest

import oracle as O
from quantumforge_gb300 import PauliSum
from quantumforge_gb300 import workloads as W
from quantumforge_gb300.qaoa import QaoaBatch

pytestmark = pytest.mark.gpu


def instance(rng, n, edges):
    pairs = [(u, v) for u in range(n) for v in range(u)]
    return n, [(*pairs[i], 1.0) for i in rng.permutation(len(pairs))[:edges]]


def check(got, want, problems):
    for a, b in zip(got, want):
        assert (a == b).all()


@pytest.mark.parametrize("sizes,edges,p", [(range(2, 13), 1, 1), (range(2, 13), 12, 4), ((12, 11, 12, 9), 60, 3), ((5, 12), 0, 2),
                                           ((12, 4, 10), 18, 16), ((12,) * 40, 18, 2)])
@pytest.mark.parametrize("tile", [None, 4, 7, 8, 9, 11, 12])
def test_resident_instances_match_the_oracle(backend, sizes, edges, p, tile):
    rng = np.random.default_rng(edges + p)
    problems = [instance(rng, n, edges) for n in sizes]
    gam, bet = rng.uniform(0, np.pi, (len(problems), p)), rng.uniform(-np.pi, np.pi, (len(problems), p))
    tiles = None if tile is None else {n: tile for n in range(2, 13)}
    cost, grad = QaoaBatch(problems, p, tile_qubits=tiles, backend=backend, use_graph=False).run(gam, bet)
    again = QaoaBatch(problems, p, tile_qubits=tiles, backend=backend, use_graph=True).run(gam, bet)
    check(again, (cost, grad), problems)
    for i, (n, ed) in enumerate(problems):
        ops = W.qaoa_param_circuit(n, ed, p)
        e, g = O.adjoint_uncompute(ops, n, np.concatenate([2 * gam[i], 2 * bet[i]]), PauliSum.maxcut(ed).array()) if ed else (0.0, 0.0)
        tol = 16.0 * np.sqrt(2.0) * 2.0**-24 * p * (n + 1) * (len(ed) + 1)
        assert abs(cost[i] - e) <= tol
        assert np.abs(grad[i] - 2 * g).max() <= tol * (len(ed) + n + 1)


def test_graph_of_another_edge_count(backend):
    """Same instances' sizes and depth, more edges: the layout behind them moves."""
    rng = np.random.default_rng(3)
    gam, bet = rng.uniform(0, np.pi, (6, 2)), rng.uniform(-np.pi, np.pi, (6, 2))
    for edges in (8, 30, 8):
        problems = [instance(rng, n, edges) for n in (14, 13, 12, 11, 10, 9)]
        got = QaoaBatch(problems, 2, backend=backend, use_graph=True).run(gam, bet)
        check(got, QaoaBatch(problems, 2, backend=backend, use_graph=False).run(gam, bet), problems)


@pytest.mark.parametrize("n,count", [(13, 7), (14, 40), (16, 3)])
@pytest.mark.parametrize("where", ["low", "high", "across", "any"])
def test_cut_values_of_tiled_instances(backend, n, count, where):
    """Edges inside a tile's low 12 bits, above them, between the two and mixed, more
    runs of tiles than CTAs and fewer, against the oracle (tolerance as above)."""
    rng = np.random.default_rng(n + count)
    pairs = [(u, v) for u in range(n) for v in range(u)]
    pairs = [(u, v) for u, v in pairs if where == "any" or where == ("low" if u < 12 else "high" if v >= 12 else "across")]
    problems = []
    for _ in range(count):
        if pairs:
            problems.append((n, [(*pairs[i], 1.0) for i in rng.permutation(len(pairs))[: int(rng.integers(1, 20))]]))
    if not problems:
        return
    gam, bet = rng.uniform(0, np.pi, (len(problems), 1)), rng.uniform(-np.pi, np.pi, (len(problems), 1))
    cost, grad = QaoaBatch(problems, 1, backend=backend).run(gam, bet)
    for i in (0, len(problems) // 2, len(problems) - 1):
        ed = problems[i][1]
        e, g = O.adjoint_uncompute(W.qaoa_param_circuit(n, ed, 1), n, np.array([2 * gam[i, 0], 2 * bet[i, 0]]),
                                   PauliSum.maxcut(ed).array())
        tol = 16.0 * np.sqrt(2.0) * 2.0**-24 * (n + 1) * (len(ed) + 1)
        assert abs(cost[i] - e) <= tol and np.abs(grad[i] - 2 * g).max() <= tol * (len(ed) + n + 1)
