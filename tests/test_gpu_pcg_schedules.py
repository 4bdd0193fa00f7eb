"""The persistent PCG and the default choice between it and the phases, at
sizes where the cluster kernel's split can go wrong: one and several groups of
32 nodes a CTA, one CTA and sixteen, windows cut by the cloth's ends (cloths
3 crossings wide or high), the largest cloth a cluster holds and one more row,
batches whose small cloths leave CTAs without nodes, and one of more 128-node
blocks than two an SM, whose phases run a thread per node. Every schedule sums
in the same order, so the results are the same bits.
"""
import numpy as np
import pytest

from pkg import gpu_available, ys
from test_gpu_pcg_persistent import _specs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not gpu_available():
        pytest.skip("no CUDA device")


def _run(sides, schedule, graphed, mode):
    b = ys.ClothBatch(_specs(sides, 3))
    if schedule == "phases":
        b.set_pcg_schedule(False)
    elif schedule == "persistent":
        b.set_pcg_schedule(True, 1024, 16)
    b.use_graphs(graphed)
    N = b.total_nodes
    ext = 1e-4 * np.random.default_rng(4).standard_normal((N, 5))
    out, stats = [], []
    for k in range(2):
        st = b.step(1e-3, ext if k else None, tol=1e-10)
        assert all(s["ok"] for s in st)
        stats += [(s["cg_iterations"], s["cg_error"]) for s in st]
        out += list(b.get_state().values())
    if mode:  # a solve with A^T as well
        rng = np.random.default_rng(5)
        g = {k: rng.standard_normal((N, c)) for k, c in dict(LPos=3, LVel=3, EPos=2, EVel=2, EPosBar=2).items()}
        adj = ys.Adjoint(b, "exact")
        gs, gp, _ = adj.step_back(1e-3, g, None, tol=1e-10)
        adj.close()
        out += list(gs.values()) + list(gp.values())
    b.close()
    return out, stats


@pytest.mark.parametrize("sides", [[(3, 3)], [(3, 11), (4, 8)], [(3, 171)], [(170, 3)], [(23, 22)], [(33, 31), (3, 3)],
                                   [(64, 64)], [(64, 65)], [(17, 17)] * 24, [(41, 41)] + [(7, 9)] * 20,
                                   [(3, 5), (12, 11)] * 160])
@pytest.mark.parametrize("graphed", [False, True])
def test_schedules_give_the_same_bits(sides, graphed):
    ref, it = _run(sides, "phases", False, not graphed)
    for schedule in ("persistent", "default"):
        got, n = _run(sides, schedule, graphed, not graphed)
        assert n == it, schedule
        for a, c in zip(ref, got):
            assert np.array_equal(a, c), schedule


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("sides", [[(3, 3)], [(23, 22), (5, 9)]])
@pytest.mark.parametrize("kact", [1, 3, 4])
def test_directions_solved_together(sides, mode, kact):
    """The directions' solves of a tangent step in one launch, and one by one in phases."""
    outs = []
    for persistent in (False, True):
        b = ys.ClothBatch(_specs(sides, 5))
        b.set_pcg_schedule(persistent, 1024, 16)
        b.tangent_enable(mode)
        K, nl, nc = b.n_tangents, sum(w + h for w, h in sides), len(sides)
        rng = np.random.default_rng(2)
        b.tangent_seed(rng.standard_normal((K, nl)) * 1e-4, rng.standard_normal((K, nl)) * 1e2,
                       rng.standard_normal((K, nl)) * 1e-6, rng.standard_normal((K, nc)) * 1e-5,
                       rng.standard_normal((K, nc)) * 1e-2)
        for _ in range(2):
            assert all(s["ok"] for s in b.step_tangent(1e-3, tol=1e-12, kact=kact))
        outs.append((b.get_state(), b.tangent_get_state()))
        b.close()
    for a, c in zip(*outs):
        for k in a:
            assert np.array_equal(a[k], c[k]), k
