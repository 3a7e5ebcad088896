"""Batched QAOA instances of up to 12 qubits that stay in shared memory, against
the per-instance kernel at the tile width (10) whose float32 sums they keep:
every qubit count, depths 1 to 16, no edges and many, batches that mix both
kernels, and a replayed graph over another list of edges of the same shape.

Tolerance: the float32 operations are the same, only double sums are ordered
differently: at most 2^n terms whose moduli add up to at most 2 W n."""
import numpy as np
import pytest

from quantumforge_gb300.qaoa import QaoaBatch

pytestmark = pytest.mark.gpu


def instance(rng, n, edges):
    pairs = [(u, v) for u in range(n) for v in range(u)]
    return n, [(*pairs[i], 1.0) for i in rng.permutation(len(pairs))[:edges]]


def check(got, want, problems):
    for i, (n, edges) in enumerate(problems):
        tol = 2.0**-53 * 2**n * 2 * (len(edges) + 1) * n
        assert abs(got[0][i] - want[0][i]) <= tol
        assert np.abs(got[1][i] - want[1][i]).max() <= tol


@pytest.mark.parametrize("sizes,edges,p", [(range(2, 13), 1, 1), (range(2, 13), 12, 4), ((12, 11, 12, 9), 60, 3), ((5, 12), 0, 2),
                                           ((12, 4, 10), 18, 16), ((12,) * 200, 18, 2)])
@pytest.mark.parametrize("graph", [False, True])
def test_resident_instances_match_the_tiled_kernel(backend, sizes, edges, p, graph):
    rng = np.random.default_rng(edges + p)
    problems = [instance(rng, n, edges) for n in sizes]
    gam, bet = rng.uniform(0, np.pi, (len(problems), p)), rng.uniform(-np.pi, np.pi, (len(problems), p))
    want = QaoaBatch(problems, p, tile_qubits={n: 10 for n in range(2, 13)}, backend=backend, use_graph=False).run(gam, bet)
    check(QaoaBatch(problems, p, backend=backend, use_graph=graph).run(gam, bet), want, problems)
    half = QaoaBatch(problems, p, tile_qubits={n: 10 for n in range(7, 13)}, backend=backend, use_graph=graph).run(gam, bet)
    check(half, want, problems)


def test_graph_of_another_edge_count(backend):
    """Same instances' sizes and depth, more edges: the layout behind them moves."""
    rng = np.random.default_rng(3)
    gam, bet = rng.uniform(0, np.pi, (6, 2)), rng.uniform(-np.pi, np.pi, (6, 2))
    for edges in (8, 30, 8):
        problems = [instance(rng, n, edges) for n in (14, 13, 12, 11, 10, 9)]
        got = QaoaBatch(problems, 2, backend=backend, use_graph=True).run(gam, bet)
        check(got, QaoaBatch(problems, 2, backend=backend, use_graph=False).run(gam, bet), problems)
